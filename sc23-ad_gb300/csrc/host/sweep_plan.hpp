// The plan of a triangular sweep by blocks of rows (kernel: cuda/trsv.cu, k_sweep).
//
// The rows are cut into `blocks` contiguous blocks, one CTA each.  A row reads
// rows of its own block, which stay in the CTA's shared memory, and rows of
// earlier blocks ("imports"), which the CTA copies into shared memory as they
// are published, in groups of up to 32 that no two steps share (a group that
// waited for the imports of later steps would put the CTA that many steps
// further behind).  A block's rows are taken in the order of the dependency
// levels of the whole triangle, one step per level that has rows in the block,
// so a block runs behind the blocks it reads by about one publication latency
// and a sweep takes about levels * step + blocks * latency.
//
// Everything static about a step is packed at setup in the order in which the
// CTA's warps consume it.  Warp w of a block reads one stream of records, each
// 32 lanes of `quads` 16-byte quads (quad q of lane k at q * 32 + k).  A record
// holds `lines` pairs of entries a lane for up to 32 / G rows of one step, G =
// 2^lg lanes a row, the same G in all records of a plan:
//   quad 0           {control word, place to publish at (-1: none), inverse diagonal (4 or 8 bytes)}
//   quads 1 ..       4-byte values: {slot byte offset, value, slot byte offset, value}
//                    8-byte values: {value, value}, and after them one quad of slot numbers of 16 bits
// control word: slot of the row (16 bits), 1 when its row goes on in the next
// record (1), barriers before the record (1), barriers before that one (7),
// import groups that it is the first of its warp to need (7).  Lane g of a row
// holds entries g, g + G, ... in the row's order; missing entries read a slot of
// zero; missing rows write to a spare slot; the parts of a row before its last
// one have an inverse diagonal of zero.  Slots: the block's rows, its
// imports, the zero, the spare.
#pragma once
#include <cstdint>
#include <memory>
#include <vector>

#include "tri_cost.hpp"

namespace sagb {

struct SweepQuad {
    uint32_t v[4];
};

struct SweepLimits {
    int sms = 1;                 // CTAs that run at the same time
    int smem = 0;                // bytes of shared memory of a CTA
    bool integer = false;        // 4-byte integers (else floating point)
    int lanes_log = -1;          // log2 of a row's lanes where the order of its sum is given
    int lanes = 1;               // a row's lanes in the kernels that go level by level
    // Records may take this much memory, or kSweepRecordShare times the triangle's own if
    // that is more.  A record has room for 32 lanes: where a level has one or two rows
    // (tridiagonal and narrow band matrices) a row takes 1 to 1.5 KiB of it instead of 20
    // bytes, and a matrix of tens of millions of rows all of a GPU's memory.  (Levels of
    // 2D and 3D grids: 1.3 to 4 times the triangle, up to 9 where small.)
    int64_t record_bytes = 2ll << 30;
};

constexpr int kSweepImporters = 8;   // most warps that fetch imports (a power of two)
constexpr int kSweepGroup = 32;      // most imports that become usable together
constexpr int kSweepMaxWarps = 8;
constexpr int kSweepStage = 4;         // records of a warp in shared memory
constexpr int kSweepMaxSlots = 65535;
constexpr int kSweepAhead = 24;        // records prefetched into the L2
constexpr int kSweepRecordShare = 8;

// bytes of shared memory beside the slots: block, epoch and the importers'
// progress (128), the records on their way
inline int sweep_fixed_smem(int warps, int quads) { return 128 + warps * kSweepStage * quads * 512; }

struct SweepPlan {
    int n = 0, nlev = 0, max_level_rows = 0;
    int64_t nnz_off = 0;
    int blocks = 0, warps = 0, importers = 0, lg = 0, lines = 0, quads = 0;  // importers: a power of two
    int virt = 0;  // each lane stands for 2^virt (SweepLimits::lanes_log)
    int max_slots = 0;                    // largest block (rows, imports, zero and spare)
    std::vector<int> row0;                // first row of each block (blocks + 1)
    std::vector<int> steps;               // steps (and barriers) of each block
    // each block's imported rows in the order of first use, in groups that a
    // step needs first: group k of a block fills import slots grp[k] .. grp[k+1]
    // (rows by their places: block by block, level by level, so that the rows
    // of one level, which are published and polled together, are neighbours)
    std::vector<int> imp_ptr, imp_place;
    std::vector<int> grp_ptr, grp;        // (grp_ptr: blocks + 1; a block's grp has one entry more than groups)
    std::vector<int64_t> stream;          // first record of (block, warp) (blocks * warps + 1)
    std::unique_ptr<SweepQuad[]> data;    // the streams one after the other
    // without blocks: the rows level by level, for k_tri_cta (one_cta) or k_tri
    std::unique_ptr<TriSchedule> levels;
    bool one_cta = false;
    bool ok() const { return blocks > 0; }
};

// The plan of the LD sweep rptr / cind / vals (off-diagonal entries, then the
// inverse diagonal last in each row); es: bytes of a value (4 or 8).
// level_hint (optional): a level per row in which every dependency has a lower
// level.  Without blocks (ok() false) when a block cannot be made to fit, when
// several blocks are needed and some row reads a later one, when the records would
// take too much memory, or when a kernel that goes level by level costs less.
SweepPlan build_sweep_plan(const int *rptr, const int *cind, const void *vals, int es, int n,
                           const SweepLimits &lim, const int *level_hint = nullptr);

}  // namespace sagb
