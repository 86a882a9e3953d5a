// Spread form of launch-ordered plans: the work of every call of a launch as
// one list of independent tiles, one thread block per tile.
//
// The rank form (gpumpi_plan_kernel) gives each rank one block, which runs
// its rank's share of one call after another.  A launch of 8 ranks then uses
// 8 of 152 SMs, a communicator of 256 ranks finishes long after one of 4, and
// six one-element calls take six times one call's latency.  In a
// launch-ordered plan nothing of that is needed: the calls touch disjoint
// memory and every input was complete when the launch started, so any block
// may do any piece of any call.  The results are those of the rank form, bit
// for bit: copies are copies, and a fold takes its inputs in rank order.
//
// Measured (rank form -> spread form, one launch, back to back): Allreduce of 8
// ranks of 16 MiB 2515 -> 46 us; the 16-communicator batch of Bcast, Allreduce and
// Alltoall at 1 element per rank 81 -> 13.3 us (with a wait after each 86 -> 22), at
// 301 326 -> 17.3 us, at 2^15 477 -> 319 us, at 100003 (rank buffers aligned to their
// elements only) 1909 -> 1047 us, at 2^20 11.55 -> 9.81 ms.
#pragma once

#include <stdint.h>
#include <string.h>

#include <vector>

#include "gpumpi.h"
#include "rt.cuh"

namespace gm {

constexpr int SP_T = 256;               // threads of a block
constexpr u32 SP_RING = 50 * 1024;      // staging bytes of a block
constexpr int SP_TAB = 256;             // ranks whose buffer addresses fit in shared memory
constexpr int SP_MAX_RANKS = 3072;   // a gather tile holds 16 bytes of every rank
constexpr u32 SP_SMEM = SP_RING + 2 * SP_TAB * (u32)sizeof(char*);
constexpr int SP_WARPS = SP_T / 32;
constexpr u32 SP_PART = SP_RING / SP_WARPS;   // a warp's part of the ring
constexpr u32 SP_CHUNK = 128;
// With more than SP_TAB ranks a fold keeps the sources' addresses at the end of
// its shared memory; that leaves each warp this much of the ring.
__host__ __device__ constexpr u32 fold_table(u32 nsrc) { return SP_SMEM - nsrc * (u32)sizeof(char*); }
__host__ __device__ constexpr u32 rows_part(u32 nsrc) {
    return nsrc <= 2 * SP_TAB ? SP_PART : fold_table(nsrc) / SP_WARPS / 16 * 16;
}
__host__ __device__ constexpr u32 passes_half(u32 nsrc) { return fold_table(nsrc) / 32 * 16; }
constexpr int SP_MAX_STAGES = 8;
constexpr int SP_BLOCKS_PER_SM = 4;     // 216 KiB of dynamic shared memory, 64 registers a thread

// What the tiles of one SpreadCall do.  Units of a copy are `ub` bytes.
enum SpreadKind : int {
    // Blocks of `nu` units: block q of every destination row comes from source
    // q.  A tile is `per` units of one block for `group` rows: loaded once,
    // stored to each (Bcast: one source; Allgather).
    SP_FAN = 0,
    // The same blocks when they are short: a tile is `per` units of the
    // sequence of all rows, each loaded and stored by one thread; with `group` 1,
    // `per` chunks of SP_CHUNK units, each of one block and moved by one warp.
    SP_COPY = 1,
    // Fold of `nu` elements over all sources in rank order, written to every
    // destination.  A tile is `per` elements: the block loads them from all
    // sources into shared memory at once, then thread i folds element i.
    SP_GATHER = 2,
    // The same fold for long vectors: a tile is `per` rows of one 16-byte
    // vector per thread, every thread streams its own vectors of one source
    // after another through its part of a ring in shared memory.
    SP_STREAM = 3,
    // Copies of longer blocks of any alignment (Alltoall, Allgather, Bcast): a
    // row is a piece of `per` bytes of one block for `group` destinations, a
    // tile is `rows` rows.  Each warp loads its rows by bulk copies of the
    // 16-byte units they touch, `stages` rows ahead, and stores them from the
    // ring, shifted to each destination's alignment.  `nu` is in bytes.
    SP_MOVE = 4,
    // The fold again, of buffers aligned to their elements only, of very many
    // ranks or in finer pieces.  Each warp folds chunks of `per` elements, a tile is `rows`
    // chunks; `batch` sources are loaded at a time, `ub` bytes apart.  With `group`
    // 1 a tile is one chunk, folded by the whole block in passes over the sources.
    SP_ROWS = 5,
};

struct alignas(16) SpreadCall {
    const char* const* src;     // [nsrc]
    char* const* dst;           // [ndst]
    u64 nu;
    u64 rs;                     // SP_GATHER: bytes between the starts of two tiles; Alltoall: between a source's blocks
    u64 off;                    // folds: bytes added to every address
    u32 first_tile, ntiles;
    int kind;
    int fn;                     // folds: element type and operator
    u32 nsrc, ndst;
    u32 per, group;
    u32 ub;
    u32 rows;                   // SP_MOVE: rows of a tile; SP_ROWS: chunks
    u32 stages;                 // SP_MOVE: stages of a warp's part of the ring
    u32 batch;                  // SP_ROWS: sources of a group
    u32 tile_bytes;             // folds: traffic of a tile
    u32 cold;                   // SP_MOVE to several destinations: the results do not fit L2
};

// The tiles of a plan, level by level: the calls of a level touch disjoint
// memory, those of the next may use their results.  A level is a launch.
struct SpreadLevel {
    u32 first_call, ncalls, ntiles;
};

struct SpreadArgs {
    SpreadCall one;             // the call of a launch with a single SpreadCall
    Job* job;                   // error words and the limit of every wait
    const SpreadCall* calls;
    u32 ncalls;
    u32 ntiles;
    u32 overlap;                // touches nothing that the launches since the last one without this mark touch
};

// A launch whose calls and addresses are parameters of the kernel (4.5 KiB).
constexpr int SP_PARAM_RANKS = 256;
constexpr int SP_PARAM_CALLS = 3;   // a fold's whole vectors and its edges
struct SpreadParams {
    SpreadCall calls[SP_PARAM_CALLS];         // src / dst: indexes into ptrs
    void* ptrs[2 * SP_PARAM_RANKS];
    u32 ncalls;
    u32 ntiles;
};

// The schedule of each collective that the tiles carry out, spread over the GPU
// instead of the ranks' blocks: from the root to every rank, a segment of the fold
// written where it is wanted, the vectors of all peer blocks over every thread.  A
// call that names it runs as one that names none, so that what gpumpi_autotune
// returns is not slower than no tuning (16 communicators of 4..256 ranks, 2^20
// elements each: rank blocks 10.9 ms, tiles 9.8; 2^15: 466 and 318 us; 1 element:
// 80 and 13 us).
inline int tiles_schedule(int op) {
    switch (op) {
        case GPUMPI_COLL_BCAST: return 1;
        case GPUMPI_COLL_REDUCE: return 2;
        case GPUMPI_COLL_ALLREDUCE: return 3;
        case GPUMPI_COLL_BARRIER: return 0;
        default: return 4;
    }
}

// What the calls of a level amount to.
struct SpreadLoad {
    int calls = 0;
    double bytes = 0;     // read and written
    double folded = 0;    // elements of their folds' results
    void count(const gpumpi_coll_desc& d, int nranks, int esize);
};

// Collects the tiles of descriptors for one launch.
struct SpreadBuilder {
    std::vector<SpreadCall> calls;      // src / dst hold indexes into ptrs until image()
    std::vector<void*> ptrs;
    std::vector<SpreadLevel> levels;

    // True when the spread form covers the call (schedule left to the runtime or
    // the tiles' own, no flag rounds, element type with the operator, no NULL buffer).
    static bool covers(const gpumpi_coll_desc& d, int nranks, int esize);
    // Append the call's tiles, sized for the level it is part of.
    void add(const gpumpi_coll_desc& d, int nranks, int esize, const SpreadLoad& level);
    void end_level();
    // Device image (calls, addresses) of bytes() bytes, and the arguments of each level's launch.
    size_t bytes() const;
    static size_t max_bytes(int nranks);   // at most so many of them belong to one call
    void image(char* host, char* dev, SpreadArgs* args);
    // The same as kernel parameters; false when they hold too few ranks.
    bool params(SpreadParams* p) const;
};

}  // namespace gm

extern "C" __global__ void gpumpi_spread_kernel(const __grid_constant__ gm::SpreadArgs A);
extern "C" __global__ void gpumpi_spread_params_kernel(const __grid_constant__ gm::SpreadParams A);
