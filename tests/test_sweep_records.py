"""The memory that a sweep's records take (host/sweep_plan.cpp, compiled by itself):
a chain of rows, which needs a record of a KiB or more a row, runs by blocks up to
the limit and level by level beyond it; a grid's records are a few times its
triangle and have no limit of their own."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HOST = os.path.join(ROOT, "sc23-ad_gb300", "csrc", "host")
DRIVER = """
#include <cstdio>
#include <cstdlib>
#include "sweep_plan.hpp"
using namespace sagb;
int main(int, char **a) {  // rows, columns of the grid, bytes of a value, limit (0: its default)
    const int n = atoi(a[1]), w = atoi(a[2]), es = atoi(a[3]);
    std::vector<int> rptr(1, 0), cind;
    for (int i = 0; i < n; i++) {
        if (w > 1 && i >= w) cind.push_back(i - w);
        if (w > 1 ? i % w > 0 : i > 0) cind.push_back(i - 1);
        cind.push_back(i);
        rptr.push_back((int)cind.size());
    }
    std::vector<char> val(cind.size() * es, 0);
    SweepLimits lim;
    lim.sms = 152;
    lim.smem = 227 * 1024;
    lim.integer = es == 4;
    if (atoll(a[4])) lim.record_bytes = atoll(a[4]);
    const SweepPlan p = build_sweep_plan(rptr.data(), cind.data(), val.data(), es, n, lim);
    printf("%d %d %lld %lld\\n", p.ok(), p.levels != nullptr, p.ok() ? p.stream.back() * p.quads * 512ll : 0,
           (long long)cind.size() * (4 + es) + 4ll * n);
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("records")
    (d / "driver.cpp").write_text(DRIVER)
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I" + HOST, str(d / "driver.cpp")]
                          + [os.path.join(HOST, f) for f in ("sweep_plan.cpp", "schedule.cpp", "tri_cost.cpp")] + ["-o", str(d / "driver")])

    def ask(*args):
        out = subprocess.run([str(d / "driver"), *map(str, args)], capture_output=True, text=True, check=True).stdout.split()
        return [int(v) for v in out]

    return ask


@pytest.mark.parametrize("es", [4, 8])
def test_a_chain_of_rows(plan, es):
    ok, _, used, own = plan(3000, 1, es, 64 << 20)
    assert ok and used >= 1024 * 3000 > 8 * own
    assert plan(3000, 1, es, used)[0] == 1
    assert plan(3000, 1, es, used - 1)[:2] == [0, 1]


def test_a_chain_beyond_the_default(plan):
    assert plan(2200000, 1, 4, 0)[:2] == [0, 1]


@pytest.mark.parametrize("es", [4, 8])
def test_a_grid(plan, es):
    ok, _, used, own = plan(181 * 181, 181, es, 1)
    assert ok and used <= 4 * own
