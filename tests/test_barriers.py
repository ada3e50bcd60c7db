"""Barriers that need the lanes of a warp together (the aligned cluster barrier, named
CTA barriers by their instruction) stand in one helper each, which brings the lanes
together first: loops and branches before a barrier may have left them apart."""
import os
import re

CUDA = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sc23-ad_gb300", "csrc", "cuda")


def _lines(pattern):
    found = []
    for name in sorted(os.listdir(CUDA)):
        with open(os.path.join(CUDA, name), encoding="utf-8") as f:
            lines = f.read().split("\n")
        found += [(name, k, lines) for k, line in enumerate(lines) if re.search(pattern, line) and not line.lstrip().startswith("//")]
    return found


def test_cluster_barrier_has_one_helper():
    found = _lines(r"barrier\.cluster\.")
    assert [f[0] for f in found] == ["common.cuh"]
    name, k, lines = found[0]
    assert lines[k - 1].strip() == "__syncwarp();"
