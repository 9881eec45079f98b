// Block-scaled dense GEMM for sm_100a: out[M,N] = bf16(alpha * A[M,K] . B[N,K]^T)
// with MXFP8 (e4m3 + UE8M0 / 32), NVFP4 (e2m1 + UE4M3 / 16) or MXFP4 (e2m1 +
// UE8M0 / 32) operands whose scales arrive in the 128x4 SfAtom order.
//
// Replaces the reference's CUTLASS/CuTe kernel (csrc/kernel/gemm/gemm_kernel.cuh:28-285,
// mainloop_fwd.cuh:405-1007, epilogue.cuh:713-1058, tile_scheduler.cuh:523-542)
// with hand-written PTX.  Per CTA (one per SM, persistent over output tiles):
//   warp 0   TMA producer: A and B tiles (128-byte swizzle) by tensor map, the
//            512-byte scale atoms by flat bulk copies, into a ring of stages
//   warp 1   one lane issues the block-scaled tcgen05.mma (fp32 accumulators
//            in tensor memory, two accumulator stages so the epilogue overlaps
//            the next tile)
//   warps 2-5 epilogue: tcgen05.ld -> * alpha -> bf16 -> swizzled staging in
//            shared memory -> TMA store (rows >= M are dropped by the tensor
//            map extent, so neither A nor the output is ever padded)
//   warps 6-9 scales: shared memory -> registers -> tensor memory (tcgen05.st),
//            one warp per lane quarter, a few k-tiles ahead of the MMAs
//   warp 10  a second MMA issuer: every other k-tile, in k order into the same accumulator,
//            or (one row of 64-wide dense tiles) into one of its own that the epilogue adds
// Warps 0, 1 and 10 (and their counterparts in the 2-CTA and small-M kernels) run their loops on all
// lanes and issue each asynchronous instruction from one elected lane (ptx::elect_one).
// Against loops inside `if (lane == 0)`: 512 x 1536 x 4096 behind its quantizer 17.6 -> 13.9 us,
// 128 x 8192 x 4096 17.0 -> 13.8, NVFP4 4096 x 14336 x 4096 148 -> 138, 8192 x 8192 x 8192 502 -> 483
// (sustained, at the power cap), 5 x 3136 x 3072 on the small-M kernel 9.2 -> 8.7; same bits.
// Every mbarrier wait is bounded: a role that waits longer than kTimeoutNs
// records a code in the device status word, raises the CTA's abort flag and
// all roles leave through the common teardown that frees tensor memory.

#include <cuda_bf16.h>

#include <unistd.h>

#include <algorithm>
#include <cmath>
#include <initializer_list>
#include <mutex>

#include "common.cuh"
#include "ptx.cuh"

namespace hq {
namespace {

constexpr int kBM = 128;           // rows of A per CTA tile
constexpr int kBKBytes = 128;      // bytes of K per stage row: 128 e4m3 or 256 e2m1
constexpr int kThreads = 352;      // single-CTA kernel: 11 warps (pair kernel: see Cfg2)
constexpr int kEpiWarps = 4;
constexpr int kSfWarps = 4;        // single-CTA kernel: warps 6-9 move the scales into tensor memory
constexpr int kEpiChunk = 32;      // accumulator columns per tcgen05.ld / TMA store
constexpr int kEpiBufBytes = 32 * kEpiChunk * 2;  // 32 rows x 64 bytes
constexpr int kMaxRuns = 255;      // runs of contiguous experts a launch may keep in shared memory, and their end
constexpr int kRunBytes = 4 * (kMaxRuns + 1);
constexpr uint64_t kTimeoutNs = 2000000000ull;    // bound of every device-side wait
constexpr int kSmemBudget = 232448;               // 227 KiB opt-in maximum per CTA

// device status word: non-zero when a kernel gave up on a bounded wait
__device__ uint32_t g_status[4];

enum : uint32_t {
    kStatusProducer = 0x01,
    kStatusMma = 0x02,
    kStatusEpilogue = 0x04,
};

template <int BN, int KIND>
struct Cfg {
    static_assert(BN == 64 || BN == 128 || BN == 256, "tile widths built");
    static constexpr int kABytes = kBM * kBKBytes;
    static constexpr int kBBytes = BN * kBKBytes;
    // SfAtoms along K that one stage needs per 128 rows: K elements per stage / (4 * group)
    static constexpr int kSfKAtoms = (KIND == 0 || KIND == 3) ? 1 : (KIND == 1 ? 4 : 2);
    static constexpr int kNAtoms = (BN + 127) / 128;
    static constexpr int kSfaBytes = kSfKAtoms * 512;
    static constexpr int kSfbBytes = kNAtoms * kSfaBytes;
    static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
    static constexpr int kEpiBufs = (KIND == 1 && BN == 256) ? 1 : 2;
    static constexpr int kEpiBytes = kEpiWarps * kEpiBufs * kEpiBufBytes;
    static constexpr int kBarBytes = 1024 + kRunBytes;  // barriers, then the runs of contiguous experts
    static constexpr int kStagesFit = (kSmemBudget - kEpiBytes - kBarBytes - 1024) / kStageBytes;
    static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;
    static constexpr int kSmemBytes = kStages * kStageBytes + kEpiBytes + kBarBytes + 1024;

    // Tensor memory columns: two accumulator stages of BN columns, then kSfSets sets of scale
    // columns (one set = the scales of one k-tile: kSfKAtoms * 4 columns for A, then
    // kSfKAtoms * kNAtoms * 4 for B).  When BN == 256 the accumulator stages overlap by
    // kOverlap columns so that everything fits in 512 (the epilogue drains the shared
    // columns first).  The scales are written by four warps of their own (tcgen05.st, one
    // warp per lane quarter) into the set it % kSfSets, so they run ahead of the MMAs: a
    // tcgen05.cp of one 512-byte atom occupies the copy unit for 75-90 cycles whoever issues
    // it, and NVFP4 needs 12 per k-tile of 512 MMA cycles.
    static constexpr int kSfCols = kSfKAtoms * 4 * (1 + kNAtoms);
    static constexpr int kSfSets = BN < 256 ? 4 : 2;
    static constexpr int kSfRegion = kSfCols * kSfSets;
    static constexpr int kOverlap = BN == 256 ? (kSfRegion + 15) / 16 * 16 : 0;
    static constexpr int kAccStride = BN - kOverlap;
    static constexpr int kSfaCol = kAccStride + BN;  // set 0
    static constexpr int kSfbCol = kSfaCol + kSfKAtoms * 4;
    // 64-wide tiles: two more accumulator stages, for the second MMA issuer (behind the scales)
    static constexpr int kDualCol = kSfaCol + kSfRegion;
    static constexpr int kColsUsed = kDualCol + (BN == 64 ? 2 * BN : 0);
    static constexpr int kTmemCols = kColsUsed <= 32 ? 32 : kColsUsed <= 64 ? 64 : kColsUsed <= 128 ? 128
                                     : kColsUsed <= 256 ? 256 : 512;
    static_assert(kColsUsed <= 512, "tensor memory budget");
    static constexpr int kChunks = BN / kEpiChunk;
    static constexpr int kOverlapChunks = (kOverlap + kEpiChunk - 1) / kEpiChunk;
    static_assert(kStages >= 2, "pipeline depth");
};

struct Barriers {
    uint64_t full[16];
    uint64_t empty[16];
    uint64_t acc_full[2];
    uint64_t acc_empty[2];
    uint64_t overlap_free[2];
    uint64_t sf_full[16];  // single-CTA kernel: the scale bytes of a stage have landed
    uint64_t sf_ready[4];  // the scales of a k-tile are in tensor memory
    uint64_t turn[2];      // pair kernel: hands the MMA issue from one issuer thread to the other
    uint64_t recv_full;    // split-K: the other CTA's partial sums have landed in this CTA's buffer
    uint64_t epi_sync;     // small-M kernel: rendezvous of the four epilogue warps (a bounded wait, unlike bar.sync)
    uint32_t tmem_base;
    uint32_t abort;
    int run_counts[16];  // contiguous experts: runs that start in a warp's share of the rows
};
constexpr int kKeptOffset = 576;  // pair kernel: the epilogue warps' places in the walk, behind the barriers
static_assert(sizeof(Barriers) <= kKeptOffset, "kBarBytes");

// Bounded mbarrier wait of one lane.  Returns false when the CTA is aborting.  kCluster: the barrier is one
// that CTAs of the cluster arrive on with release semantics; the wait acquires what they wrote into
// this CTA's shared memory before arriving.  A function of its own: the roles come here only when a first
// try_wait, which holds a converged warp until the phase ends (woken 84 cycles after the arrival, also after
// 6000 cycles), has returned without it, and the polling code is not in their loops.  (InPlace: inline after all, for the split-K
// kernel, which took 170 cycles a k-tile longer with the calls in its loops: 125 x 704 x 8064 10.8 us, 13.7 with them.  Inline in every
// kernel: SituQuant 300 x 5120 x 2048 7.5 -> 8.6 us, NVFP4 2048 x 8192 x 2048 20.7 -> 26.0, W4A8 12 slots of 256 x 3072 x 2048
// 18.7 -> 25.5.)
enum class InPlace {};
template <bool kCluster = false>
__device__ __forceinline__ bool wait_bar_lane(InPlace, uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t code,
                                              uint64_t limit_ns = kTimeoutNs) {
    const auto done = [&] { return kCluster ? ptx::mbar_try_wait_cluster(bar, parity) : ptx::mbar_try_wait(bar, parity); };
    if (done()) return true;
    const uint64_t t0 = ptx::globaltimer_ns();
    uint32_t spins = 0;
    while (!done()) {
        if ((++spins & 31u) == 0u) {
            if (*abort != 0u) return false;
            if (ptx::globaltimer_ns() - t0 > limit_ns) {
                *abort = 1u;
                atomicOr(&g_status[0], code);
                return false;
            }
        }
    }
    return true;
}
template <bool kCluster = false>
__device__ __noinline__ bool wait_bar_lane(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t code,
                                           uint64_t limit_ns = kTimeoutNs) {
    return wait_bar_lane<kCluster>(InPlace{}, bar, parity, abort, code, limit_ns);
}

// The wait of a role: called by all lanes of a warp, with one result for all of them.  Lanes poll for
// themselves, so when a wait runs out while its barrier completes after all, some of them see the one and
// some the other; leaving the role's loop on that would send a part of the warp into
// .sync.aligned instructions, __syncwarp and elections that count on all 32 lanes.
// The first try and its vote are straight-line code (a completed barrier: 58 cycles); with the polling loop inline, lane by
// lane, a wait on a completed barrier took a role 125: 512 x 1536 x 4096 8.8 -> 8.5 us, 1024 x 1536 x 8192 26.0 -> 24.9 (both on
// the 128 x 64 tile), NVFP4 512 x 4096 x 8192 12.9 -> 12.7, GEMM alone.
template <bool kInPlace = false>
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t code) {
    if (__all_sync(0xffffffffu, ptx::mbar_try_wait(bar, parity) ? 1 : 0) != 0) return true;
    const bool mine = kInPlace ? wait_bar_lane(InPlace{}, bar, parity, abort, code) : wait_bar_lane(bar, parity, abort, code);
    return __all_sync(0xffffffffu, mine ? 1 : 0) != 0;
}
// Two waits with one vote (the second only if `both`): a vote between a barrier and the work behind it is on the
// critical path of a k-step.
template <bool kInPlace = false>
__device__ __forceinline__ bool wait_bars(uint32_t bar, uint32_t parity, bool both, uint32_t bar2, uint32_t parity2,
                                          volatile uint32_t* abort, uint32_t code) {
    bool mine = ptx::mbar_try_wait(bar, parity);
    if (both) mine = ptx::mbar_try_wait(bar2, parity2) && mine;
    if (__all_sync(0xffffffffu, mine ? 1 : 0) != 0) return true;
    if constexpr (kInPlace) {
        mine = wait_bar_lane(InPlace{}, bar, parity, abort, code) && (!both || wait_bar_lane(InPlace{}, bar2, parity2, abort, code));
    } else {
        mine = wait_bar_lane(bar, parity, abort, code) && (!both || wait_bar_lane(bar2, parity2, abort, code));
    }
    return __all_sync(0xffffffffu, mine ? 1 : 0) != 0;
}
template <bool kInPlace = false>
__device__ __forceinline__ bool wait_bar_cluster(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t code) {
    if (__all_sync(0xffffffffu, ptx::mbar_try_wait_cluster(bar, parity) ? 1 : 0) != 0) return true;
    const bool mine = kInPlace ? wait_bar_lane<true>(InPlace{}, bar, parity, abort, code) : wait_bar_lane<true>(bar, parity, abort, code);
    return __all_sync(0xffffffffu, mine ? 1 : 0) != 0;
}

// The warp's index in its CTA, known to be warp-uniform.
__device__ __forceinline__ int warp_index() { return __shfl_sync(0xffffffffu, int(threadIdx.x >> 5), 0); }

struct TileCoord {
    int m;
    int n;
};

// Persistent static schedule: tile ids walk down groups of 8 row tiles, then
// across columns, so one wave of CTAs shares a small set of A and B tiles in L2.
__device__ __forceinline__ TileCoord tile_coord(int tile, int tiles_m, int tiles_n) {
    constexpr int kGroup = 8;
    if (tiles_m == 1) return {0, tile};  // decode shapes: no divisions on the way to the first load
    const int per_group = kGroup * tiles_n;
    const int g = tile / per_group;
    const int first_m = g * kGroup;
    const int gsz = min(kGroup, tiles_m - first_m);
    const int r = tile - g * per_group;
    return {first_m + r % gsz, r / gsz};
}

// How the rows of A map to weights.  Dense: one weight.  The grouped kinds stack
// `count` weights [count, N, K] (scales: every weight starts on its own 128-row atom):
//   batch       A rows [g * rows, (g + 1) * rows) use weight g; out is [rows, count * N]
//   masked      the same slots, of which only the first table[g] rows are valid;
//               out is [count * rows, N]
//   contiguous  row r uses weight table[r] (sorted, every run of equal ids starts on a
//               multiple of 64 rows); out is [M, N]
// Follows the reference's four kernel modes (csrc/kernel/gemm/tile_scheduler.cuh:253-297,
// 393-460, 575-670).
enum { kGroupDense = 0, kGroupBatch = 1, kGroupMasked = 2, kGroupContiguous = 3 };

struct GroupParams {
    int kind;
    int count;         // number of weights
    int rows;          // rows per batch / padded rows per expert (batch, masked)
    const int* table;  // masked: valid rows per expert; contiguous: expert of every row
};

// Contiguous experts: the rows as runs of one expert each.  A run is cut into tiles of kRows rows from the 128-row
// boundary at or before its start (where its scale atoms are), so that every tile is worked once, for one expert, and the tiles
// of all runs are dealt out alike.  (Tiles on fixed boundaries were worked once per run in them, one pass after the other by the CTA that
// had them: ten uneven experts on 8192 x 4096 x 4096 MXFP8, pair tile, 152 us where one expert takes 113;
// NVFP4 40960 x 4096 x 4096 324 and 293.)
// Entry i: first 64-row quarter of run i, and its expert << 16; the entry behind the last run ends it.
struct RunTable {
    const uint32_t* runs;  // null: the rows have more runs, or more quarters, than the table can hold
    int row_tiles;
};

// Tiles of kRows rows in the run between two entries.
template <int kRows>
__device__ __forceinline__ int run_tiles(uint32_t entry, uint32_t next) {
    const int first = int(entry & 0xffffu) / 2 * 128;
    return (int(next & 0xffffu) * 64 - first + kRows - 1) / kRows;
}

// Called by all threads of the block, kBlock of them, after the wait for the preceding kernel.
template <int kRows, int kBlock>
__device__ __forceinline__ RunTable build_runs(const GroupParams& g, int m, Barriers* bars, uint32_t* runs) {
    static_assert(kBlock / 32 <= 16, "Barriers::run_counts");
    const int nq = m / 64;
    if (nq > 0xffff || g.count > 0x10000) return {nullptr, 0};
    const int lane = threadIdx.x & 31;
    const int warp = threadIdx.x >> 5;
    int total = 0;
    constexpr int kRounds = 2;  // loads in flight per thread
    for (int b = 0; b < nq; b += kRounds * kBlock) {
        int id[kRounds], before[kRounds];
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            const int q = b + r * kBlock + int(threadIdx.x);
            id[r] = q < nq ? __ldg(g.table + q * 64) : 0;
            before[r] = q < nq && q > 0 ? __ldg(g.table + q * 64 - 64) : ~id[r];
        }
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            if (b + r * kBlock >= nq) break;
            const int q = b + r * kBlock + int(threadIdx.x);
            const bool starts = q < nq && id[r] != before[r];
            const uint32_t ballot = __ballot_sync(0xffffffffu, starts);
            if (lane == 0) bars->run_counts[warp] = __popc(ballot);
            __syncthreads();
            int at = total + __popc(ballot & ((1u << lane) - 1u));
#pragma unroll
            for (int w = 0; w < kBlock / 32; ++w) {
                const int c = bars->run_counts[w];
                at += w < warp ? c : 0;
                total += c;
            }
            if (starts && at < kMaxRuns) runs[at] = uint32_t(q) | (uint32_t(min(max(id[r], 0), g.count - 1)) << 16);
            if (b + (r + 1) * kBlock < nq) __syncthreads();  // run_counts are written again
        }
    }
    if (total > kMaxRuns) return {nullptr, 0};
    if (threadIdx.x == 0) runs[total] = uint32_t(nq);
    __syncthreads();
    int tiles = 0;  // every warp for itself
    for (int i = lane; i < total; i += 32) tiles += run_tiles<kRows>(runs[i], runs[i + 1]);
    return {runs, int(__reduce_add_sync(0xffffffffu, tiles))};
}

// A role's place in the runs: row tile `rt` of them, by steps from the last one asked for.
template <int kRows>
struct RunWalk {
    RunTable t;
    int run = -1, base = 0, count = 0;  // the run of the last row tile, the row tiles before it and in it
    uint32_t entry = 0, next = 0;       // its entry and the one behind it

    __device__ __forceinline__ void take(int i) {
        run = i;
        entry = t.runs[i];
        next = t.runs[i + 1];
        count = run_tiles<kRows>(entry, next);
    }
    // first row of the tile, the rows [lo, hi) of it that are the run's, and the expert
    __device__ __forceinline__ void find(int rt, int& row0, int& lo, int& hi, int& expert) {
        if (run < 0) take(0);
        while (rt >= base + count) {
            base += count;
            take(run + 1);
        }
        while (rt < base) {
            take(run - 1);
            base -= count;
        }
        const int start = int(entry & 0xffffu) * 64;
        row0 = start / 128 * 128 + (rt - base) * kRows;
        lo = max(0, start - row0);
        hi = min(kRows, int(next & 0xffffu) * 64 - row0);
        expert = int(entry >> 16);
    }
};

// What one persistent-loop iteration of the single-CTA kernel works on.
struct Work {
    int a_row0;     // first row of the A box (and 128 x its scale-atom row)
    int b_row0;     // first row of the B box in the stacked weights
    int sfb_tile;   // 128-row scale atom row of the B box
    int sfb_shift;  // 32-row group of the B box inside that atom (BN = 64 only)
    int cols;       // weight rows of the tile that exist; its other columns are neither loaded for nor stored
    int group;      // weight index: selects alpha and the bias row
    int row_lo;     // accumulator rows [row_lo, row_hi) belong to this item; the others
    int row_hi;     //   are padding or belong to the neighbouring group
    int out_row0;   // output row of accumulator row 0 (negative when a batch starts mid-tile)
    int out_col0;   // first output column
    int bias_col0;  // first bias element
};

// The three warp roles walk the same sequence of work items, each with its own copy
// of this iterator.  Tiles are cut on 128-row boundaries of the stacked A rows (where
// the scale atoms are); a tile that holds rows of two groups is worked once per group
// (the reference's rule for batches, csrc/kernel/gemm/gemm_dispatch.cuh:90-93).
template <int BN>
struct WorkIter {
    GroupParams g;
    int M, N, tiles_m, tiles_n;
    int tile;
    int pass = 0;        // contiguous: second expert of a tile
    int walk_group = 0;  // batch / masked: group of the last item and the number of
    int walk_base = 0;   //   (group, row tile) pairs before it

    int stride;          // work items between two items of this CTA (or cluster)
    RunWalk<kBM> runs;   // contiguous

    __device__ WorkIter(const GroupParams& grp, int m, int n, int tm, int tn, const RunTable& rt, int first = blockIdx.x,
                        int step = gridDim.x)
        : g(grp), M(m), N(n), tiles_m(tm), tiles_n(tn), tile(first), stride(step), runs{rt} {
        if (g.kind == kGroupContiguous && rt.runs != nullptr) tiles_m = rt.row_tiles;
    }

    __device__ __forceinline__ void set_b(Work& w, int group, int nt) const {
        w.group = group;
        w.cols = min(BN, N - nt * BN);
        w.b_row0 = group * N + nt * BN;
        w.sfb_tile = group * ((N + 127) / 128) + (nt * BN) / 128;
        w.sfb_shift = ((nt * BN) % 128) / 32;
        w.bias_col0 = w.b_row0;
    }

    __device__ bool next(Work& w) {
        if (g.kind == kGroupDense || g.kind == kGroupContiguous) {
            if (tile >= tiles_m * tiles_n) return false;
            const TileCoord tc = tile_coord(tile, tiles_m, tiles_n);
            w.out_col0 = tc.n * BN;
            int group = 0;
            if (g.kind == kGroupContiguous && runs.t.runs != nullptr) {
                runs.find(tc.m, w.a_row0, w.row_lo, w.row_hi, group);
                w.out_row0 = w.a_row0;
                set_b(w, group, tc.n);
                tile += stride;
                return true;
            }
            w.a_row0 = tc.m * kBM;
            w.out_row0 = w.a_row0;
            w.row_lo = 0;
            w.row_hi = min(kBM, M - w.a_row0);
            if (g.kind == kGroupContiguous) {
                const int e0 = __ldg(g.table + w.a_row0);
                const int e1 = w.a_row0 + 64 < M ? __ldg(g.table + w.a_row0 + 64) : e0;
                group = min(max(pass != 0 ? e1 : e0, 0), g.count - 1);
                if (e1 != e0) {
                    // two experts meet in the middle of this tile: one pass each
                    if (pass == 0) {
                        w.row_hi = 64;
                    } else {
                        w.row_lo = 64;
                    }
                    pass ^= 1;
                }
            }
            set_b(w, group, tc.n);
            if (pass == 0) tile += stride;
            return true;
        }
        // batch / masked: item = (group, j-th row tile that holds valid rows of it, n tile)
        const int pair = tile / tiles_n;
        const int nt = tile - pair * tiles_n;
        int first, valid;
        for (;;) {
            if (walk_group >= g.count) return false;
            first = walk_group * g.rows;
            valid = g.kind == kGroupMasked ? min(max(__ldg(g.table + walk_group), 0), g.rows) : g.rows;
            const int cnt = valid > 0 ? (first + valid - 1) / kBM - first / kBM + 1 : 0;
            if (pair < walk_base + cnt) break;
            walk_base += cnt;
            ++walk_group;
        }
        w.a_row0 = (first / kBM + (pair - walk_base)) * kBM;
        w.row_lo = max(0, first - w.a_row0);
        w.row_hi = min(kBM, first + valid - w.a_row0);
        set_b(w, walk_group, nt);
        if (g.kind == kGroupBatch) {
            w.out_row0 = w.a_row0 - first;
            w.out_col0 = w.b_row0;
        } else {
            w.out_row0 = w.a_row0;
            w.out_col0 = nt * BN;
        }
        tile += stride;
        return true;
    }
};

template <int BN, int KIND>
__device__ __forceinline__ uint32_t instr_desc(uint32_t sf_id) {
    // block-scaled instruction descriptor: [4,6) SFB byte id, [7,10) A format,
    // [10,13) B format, bit 15/16 A/B major (0 = K), [17,23) N >> 3,
    // bit 23 scale format (1 = UE8M0, 0 = UE4M3), [24,29) M >> 4, [29,31) SFA byte id
    // KIND 0: e4m3 x e4m3 (code 0); KIND 1 / 2: e2m1 x e2m1 of the mxf4nvf4 kinds (code 1);
    // KIND 3: e4m3 x e2m1 of the mxf8f6f4 kind, whose code for e2m1 is 5
    constexpr uint32_t fmt_a = (KIND == 0 || KIND == 3) ? 0u : 1u;
    constexpr uint32_t fmt_b = KIND == 0 ? 0u : (KIND == 3 ? 5u : 1u);
    constexpr uint32_t scale_fmt = KIND == 1 ? 0u : 1u;
    return (sf_id << 4) | (fmt_a << 7) | (fmt_b << 10) | (uint32_t(BN >> 3) << 17) | (scale_fmt << 23) |
           (uint32_t(kBM >> 4) << 24) | (sf_id << 29);
}

// Parameters of the SiTU-GLU quantising epilogue (all zero for the other epilogues).
struct SituParams {
    uint8_t* q;       // e4m3 output: [M, N/2] (SituQuant) or [M, B * N] (the batch Quant epilogues)
    uint8_t* sf;      // UE8M0 scales of the output, SfAtom order, kb_out scale columns
    int64_t ldq;      // bytes between output rows
    int kb_out;       // scale columns of the output: N / 2 / 32 or B * N / 32
    float beta;       // gate soft-cap
    float inv_beta;
    float lin;        // up soft-cap, 0 = none
    float inv_lin;
    const __nv_bfloat16* gate;  // [M, B * N] multiplier of the GateMulQuant epilogues (logits for the sigmoid form)
    int64_t gate_ld;            // elements between its rows
    int valid_rows;             // rows of the quantised output; `sf` covers them rounded up to 128
};

// The quantising epilogues store a scale byte for every row that exists.  The rows that pad
// the last 128-row SfAtom get zero bytes here (what group_wise_quant writes there), so a
// caller need not clear `sf` first.  Called by the 128 epilogue threads of every CTA.
__device__ __forceinline__ void zero_sf_padding(const SituParams& sp, int tid) {
    const int pad_rows = (128 - (sp.valid_rows & 127)) & 127;
    const int total = pad_rows * sp.kb_out;
    for (int i = int(blockIdx.x) * 128 + tid; i < total; i += int(gridDim.x) * 128) {
        const int row = sp.valid_rows + i / sp.kb_out;
        const int kb = i % sp.kb_out;
        sp.sf[(int64_t(row >> 7) * (sp.kb_out >> 2) + (kb >> 2)) * 512 + (row & 31) * 16 + ((row >> 5) & 3) * 4 +
              (kb & 3)] = 0;
    }
}

__device__ __forceinline__ float tanh_fast(float x) {
    float t;
    asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
    return t;
}

// 16 SiTU-GLU outputs from one 32-column accumulator chunk whose first 16 columns
// are gate rows and last 16 the matching up rows (the row order interleave_gate_up
// produces): bf16(beta tanh(g / beta) sigmoid(g) * lin tanh(u / lin)), or * u when
// there is no up soft-cap (reference: halops/gemm/dense_gemm.py:100-109,
// csrc/common/activation.cuh:33-62; the sigmoid here is 0.5 tanh(g / 2) + 0.5).
__device__ __forceinline__ void situ_chunk(const uint32_t (&r)[32], const __nv_bfloat16* __restrict__ bias_chunk,
                                           const SituParams& sp, uint32_t* y8) {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
    if (bias_chunk != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 b = __ldg(reinterpret_cast<const uint4*>(bias_chunk) + j);
            const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                v[8 * j + 2 * i] += __uint_as_float(w[i] << 16);
                v[8 * j + 2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
            }
        }
    }
    float o[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float g = v[i];
        const float u = v[16 + i];
        const float gate = sp.beta * tanh_fast(g * sp.inv_beta) * fmaf(0.5f, tanh_fast(0.5f * g), 0.5f);
        const float up = sp.lin != 0.0f ? sp.lin * tanh_fast(u * sp.inv_lin) : u;
        o[i] = gate * up;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const __nv_bfloat162 p = __float22bfloat162_rn(make_float2(o[2 * i], o[2 * i + 1]));
        y8[i] = *reinterpret_cast<const uint32_t*>(&p);
    }
}

// MXFP8 quantisation of 32 bf16 values (16 packed words) of one row: UE8M0 byte
// e = ceil(log2(amax / 448)) + 127 computed exactly on the bf16 bit fields (floor 85),
// codes = e4m3(v * 2^(127 - e)) with NaN -> -448.  This is the exact-integer recipe of
// the reference's quantising epilogue (csrc/common/mx_quant.cuh:60-71,
// csrc/kernel/gemm/epilogue.cuh:990-1010), not the fast-math one of group_wise_quant.
__device__ __forceinline__ uint32_t quant32_bf16(const uint32_t (&y)[16], uint4& lo, uint4& hi) {
    uint32_t mx = y[0] & 0x7fff7fffu;
#pragma unroll
    for (int i = 1; i < 16; ++i) {
        uint32_t a = y[i] & 0x7fff7fffu, m2;
        asm("max.bf16x2 %0, %1, %2;" : "=r"(m2) : "r"(mx), "r"(a));
        mx = m2;
    }
    uint32_t sw = __byte_perm(mx, 0, 0x1032), m2;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(m2) : "r"(mx), "r"(sw));
    const uint32_t bits = m2 & 0xffffu;                      // bf16 amax: 8 exponent, 7 mantissa bits
    const uint32_t exp8 = ((bits + 31u) >> 7) & 0xffu;       // exponent, + 1 when the mantissa exceeds 1.75
    const uint32_t e = max(exp8, 85u + 8u) - 8u;
    const float mult = __uint_as_float((254u - e) << 23);
    uint32_t c[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        uint32_t g;
        asm("max.bf16x2 %0, %1, %2;" : "=r"(g) : "r"(y[i]), "r"(0xff80ff80u));  // NaN -> -inf -> -448
        const float a = __uint_as_float(g << 16) * mult;
        const float b = __uint_as_float(g & 0xffff0000u) * mult;
        uint16_t h;
        asm("cvt.rn.satfinite.e4m3x2.f32 %0, %2, %1;" : "=h"(h) : "f"(a), "f"(b));
        c[i] = h;
    }
    lo = make_uint4(c[0] | (c[1] << 16), c[2] | (c[3] << 16), c[4] | (c[5] << 16), c[6] | (c[7] << 16));
    hi = make_uint4(c[8] | (c[9] << 16), c[10] | (c[11] << 16), c[12] | (c[13] << 16), c[14] | (c[15] << 16));
    return e;
}

// Epilogue math for one 32-column chunk of one accumulator row:
// y = acc * alpha (+ bias[col]); Identity stores bf16(y), Sigmoid stores
// bf16(0.5 * tanh.approx(0.5 * y) + 0.5), the reference's formulation
// (csrc/common/activation.cuh:25-27, csrc/kernel/gemm/epilogue.cuh:867-951).
__device__ __forceinline__ void epilogue_chunk(const uint32_t (&r)[32], uint32_t (&p)[16], float scale,
                                               const __nv_bfloat16* __restrict__ bias_chunk, int epi_op) {
    float y[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) y[i] = __uint_as_float(r[i]) * scale;
    if (bias_chunk != nullptr) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint4 b = __ldg(reinterpret_cast<const uint4*>(bias_chunk) + j);
            const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                y[8 * j + 2 * i] += __uint_as_float(w[i] << 16);
                y[8 * j + 2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
            }
        }
    }
    if (epi_op == HQ_EPILOGUE_SIGMOID) {
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            float t;
            asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * y[i]));
            y[i] = fmaf(0.5f, t, 0.5f);
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const __nv_bfloat162 v = __float22bfloat162_rn(make_float2(y[2 * i], y[2 * i + 1]));
        p[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
}

// The scale atoms of one stage (512 bytes each, 16 for a lane) into registers, in the order of a scale set's columns:
// SFA by atom along K, then SFB by atom along K and 128 columns.
template <typename C>
__device__ __forceinline__ void load_scales(uint32_t sfa_stage, uint32_t sfb_stage, int lane, uint32_t (&r)[C::kSfCols]) {
    const uint32_t a0 = sfa_stage + uint32_t(lane) * 16u;
    const uint32_t b0 = sfb_stage + uint32_t(lane) * 16u;
#pragma unroll
    for (int a = 0; a < C::kSfKAtoms; ++a) {
        ptx::ld_shared_v4(a0 + a * 512, r[4 * a], r[4 * a + 1], r[4 * a + 2], r[4 * a + 3]);
#pragma unroll
        for (int j = 0; j < C::kNAtoms; ++j) {
            const int c = 4 * (C::kSfKAtoms + a * C::kNAtoms + j);
            ptx::ld_shared_v4(b0 + (j * C::kSfKAtoms + a) * 512, r[c], r[c + 1], r[c + 2], r[c + 3]);
        }
    }
}

// kSplitK (64-wide tiles, one row of tiles, at most half as many tiles as SMs): a cluster of
// two CTAs works one tile, each half of the k-tiles; the second CTA sends its fp32 partial
// sums through distributed shared memory into a 32 KB buffer of the first (carved out of the
// last two A stages), which adds them to its accumulator before the usual epilogue.
//
// kDense: one weight and a plain epilogue (Identity, Sigmoid), known at compile time.  The group walk in
// every role and the quantising epilogues are then not in the code: a small problem fetches its
// instructions anew at every launch, and they were most of them (512 x 1536 x 4096 behind its
// quantizer 13.9 -> 12.8 us, 128 x 256 x 512 5.6 -> 5.1, NVFP4 300 x 4096 x 4096 12.0 -> 11.4; large
// problems unchanged).  The other forms take the general code.
//
// kRuns: contiguous experts, cut into tiles by their runs (RunTable), known at compile time.  Batches, masked experts and the contiguous
// problems that the table does not repay (contiguous_by_runs) carry none of its code, and the runs none of theirs: MXFP8 5504 x 3456 x 768
// with 12 experts on the 128 x 128 tile 35 -> 24 us, NVFP4 21504 x 2432 x 1024 with 18 75 (pair tile) -> 47; masked and batch 2 % faster.
// (The pair kernel has one grouped form for all: with the runs in one of their own they took 1.17 and 1.25 of the time on
// the 256 x 128 tile in MXFP8 and W4A8.)
template <int BN, int KIND, bool kSplitK = false, bool kDense = kSplitK, bool kRuns = false>
__global__ void __launch_bounds__(kThreads, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
            const __grid_constant__ CUtensorMap tm_d, const uint8_t* __restrict__ sfa,
            const uint8_t* __restrict__ sfb, const float* __restrict__ alpha,
            const __nv_bfloat16* __restrict__ bias, int epi_op, __nv_bfloat16* __restrict__ out, int64_t ldo,
            int M, int N, int k_tiles, int kq_dim, int tiles_m, int tiles_n, int a_rows, int direct_store,
            int dual_issue, int prefetch_weight, const GroupParams grp_arg, const SituParams situ) {
    using C = Cfg<BN, KIND>;
    const GroupParams grp = kDense ? GroupParams{kGroupDense, 1, 0, nullptr}
                            : kRuns ? GroupParams{kGroupContiguous, grp_arg.count, grp_arg.rows, grp_arg.table} : grp_arg;
    constexpr bool kPlain = kDense || kRuns;  // Identity or Sigmoid
    // Two MMA issuers with an accumulator each (64-wide dense tiles, plain epilogues): the k-tiles
    // of a tile are summed as (even ones) + (odd ones), deterministically, but not in the k order
    // of the other tiles.
    const bool dual = BN == 64 && kDense && !kSplitK && dual_issue == 1;
    // dual_issue == 2: two issuers as well, but into ONE accumulator and in k order, as in the
    // 2-CTA kernel: the threads take alternate k-iterations and hand each other the turn (tcgen05
    // fences around an mbarrier arrival), so the MMAs reach the tensor core in the order one thread
    // would issue them and the bits do not change.  What it buys is issue time: 4 MMAs and the
    // commit that releases the stage keep one thread busy for longer than a narrow tile's MMAs run.
    const bool ordered = dual_issue == 2;
    static_assert(!kSplitK || (BN == 64 && 2 * C::kABytes == kBM * BN * 4 && C::kStages >= 6), "split-K buffer");
    // stages of the ring; with split-K the last two A stages hold the partial sums received
    constexpr uint32_t kRing = kSplitK ? C::kStages - 2 : C::kStages;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment: required by the 128-byte swizzle of the operand tiles
    const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* const smem = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
    const uint32_t a_base = smem_base;
    const uint32_t recv_base = a_base + kRing * C::kABytes;
    const uint32_t k_rank = kSplitK ? ptx::cluster_ctarank() : 0u;
    // this CTA's share of the k-tiles and of the work items
    const int k_begin = kSplitK ? int(k_rank) * k_tiles / 2 : 0;
    const int k_end = kSplitK ? (int(k_rank) + 1) * k_tiles / 2 : k_tiles;
    const int first_item = kSplitK ? blockIdx.x >> 1 : blockIdx.x;
    const int item_step = kSplitK ? gridDim.x >> 1 : gridDim.x;
    const uint32_t b_base = a_base + C::kStages * C::kABytes;
    const uint32_t sfa_base = b_base + C::kStages * C::kBBytes;
    const uint32_t sfb_base = sfa_base + C::kStages * C::kSfaBytes;
    const uint32_t epi_base = sfb_base + C::kStages * C::kSfbBytes;
    const uint32_t bar_off = C::kStages * C::kStageBytes + C::kEpiBytes;
    Barriers* const bars = reinterpret_cast<Barriers*>(smem + bar_off);
    volatile uint32_t* const abort = &bars->abort;

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            ptx::mbar_init(ptx::smem_u32(&bars->full[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&bars->sf_full[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&bars->empty[s]), 1);
        }
        for (int s = 0; s < 2; ++s) {
            ptx::mbar_init(ptx::smem_u32(&bars->acc_full[s]), (dual || ordered) ? 2 : 1);  // one commit per MMA issuer
            ptx::mbar_init(ptx::smem_u32(&bars->turn[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&bars->acc_empty[s]), kEpiWarps);
            ptx::mbar_init(ptx::smem_u32(&bars->overlap_free[s]), kEpiWarps);
        }
        for (int s = 0; s < C::kSfSets; ++s) ptx::mbar_init(ptx::smem_u32(&bars->sf_ready[s]), kSfWarps);
        if (kSplitK) ptx::mbar_init(ptx::smem_u32(&bars->recv_full), kEpiWarps);
        bars->abort = 0;
        ptx::fence_mbar_init();
        ptx::prefetch_tmap(&tm_a);
        ptx::prefetch_tmap(&tm_b);
        ptx::prefetch_tmap(&tm_d);
    }
    if (warp == 1) {
        ptx::tmem_alloc<1>(ptx::smem_u32(&bars->tmem_base), C::kTmemCols);
        ptx::tmem_relinquish<1>();
    }
    ptx::tc_fence_before();
    __syncthreads();
    // the other CTA's barriers exist before anyone signals across the pair
    if (kSplitK) ptx::cluster_sync();
    ptx::tc_fence_after();
    const uint32_t tmem = bars->tmem_base;

    // The first k-tiles of this CTA's weight into L2 while the preceding kernel finishes: a hint, as in the
    // small-M kernel, up to 160 KB per CTA (24 MB in all).  The CTAs that share a column of tiles share
    // the k-tiles too.  128 x 8192 x 4096 behind its quantizer 13.2 -> 12.5 us, 512 x 1536 x 4096 12.8 -> 12.7.
    // Only under a programmatic launch: a CTA that starts after the preceding kernel has ended would ask for
    // everything twice (128 x 8192 x 4096 launched without, 11.7 us, was 12.8 with it).
    // (Dense only: which weight a grouped tile takes is only known after the wait.)
    if constexpr (kDense) {
        if (threadIdx.x == 64 && prefetch_weight != 0 && first_item < tiles_m * tiles_n) {
            const TileCoord tc = tile_coord(first_item, tiles_m, tiles_n);
            const int end = min(k_end, k_begin + 1280 / BN);
            for (int kt = k_begin + (tc.m & 7); kt < end; kt += min(8, tiles_m)) {
                ptx::tma_prefetch_2d(&tm_b, kt * kBKBytes, tc.n * BN);
            }
        }
        __syncwarp();
    }
    // Everything above overlaps the tail of the previous kernel under a
    // programmatic launch; nothing below may run before its writes are visible.
    ptx::pdl_wait();
    RunTable run_table = {nullptr, 0};
    if constexpr (kRuns) {
        run_table = build_runs<kBM, kThreads>(grp, M, bars, reinterpret_cast<uint32_t*>(smem + bar_off + 1024));
    }

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer
        {
            uint32_t it = 0;
            bool ok = true;
            WorkIter<BN> work(grp, M, N, tiles_m, tiles_n, run_table, first_item, item_step);
            Work wk;
            while (ok && work.next(wk)) {
                const int m0 = wk.a_row0;
                const int n0 = wk.b_row0;
                const uint8_t* const sfa_row = sfa + int64_t(m0 / kBM) * kq_dim * 512;
                const uint8_t* const sfb_row = sfb + int64_t(wk.sfb_tile) * kq_dim * 512;
                for (int kt = k_begin; kt < k_end; ++kt, ++it) {
                    const uint32_t s = it % kRing;
                    const uint32_t ph = (it / kRing) & 1u;
                    ok = wait_bar<kSplitK>(ptx::smem_u32(&bars->empty[s]), ph ^ 1u, abort, kStatusProducer);
                    if (!ok) break;
                    const uint32_t full = ptx::smem_u32(&bars->full[s]);
                    const uint32_t sf_full = ptx::smem_u32(&bars->sf_full[s]);
                    // The scales have a barrier of their own: they are few bytes and land early,
                    // so the scale warps are done before the operand tiles arrive.
                    if (ptx::elect_one()) ptx::mbar_arrive_expect_tx(sf_full, C::kSfaBytes + C::kSfbBytes);
                    const int64_t koff = int64_t(kt) * C::kSfaBytes;
                    if (ptx::elect_one()) {
                        ptx::bulk_load(sfa_base + s * C::kSfaBytes, sfa_row + koff, C::kSfaBytes, sf_full);
                    }
#pragma unroll
                    for (int j = 0; j < C::kNAtoms; ++j) {
                        // (a ragged last tile takes the atoms that exist once more)
                        const int ja = (j * 128 < wk.cols) ? j : 0;
                        if (ptx::elect_one()) {
                            ptx::bulk_load(sfb_base + s * C::kSfbBytes + j * C::kSfaBytes,
                                           sfb_row + int64_t(ja) * kq_dim * 512 + koff, C::kSfaBytes, sf_full);
                        }
                    }
                    // a short activation loads only its own rows (the A box is a_rows tall)
                    // packed e2m1 weights spread to one byte per value in shared memory, but the
                    // barrier counts the bytes read from global memory: half of the stage's B bytes
                    if (ptx::elect_one()) {
                        ptx::mbar_arrive_expect_tx(full, C::kABytes + C::kBBytes - (kBM - a_rows) * kBKBytes -
                                                             (KIND == 3 ? C::kBBytes / 2 : 0));
                    }
                    if (ptx::elect_one()) ptx::tma_load_2d(a_base + s * C::kABytes, &tm_a, kt * kBKBytes, m0, full);
                    if (ptx::elect_one()) ptx::tma_load_2d(b_base + s * C::kBBytes, &tm_b, kt * kBKBytes, n0, full);
                }
            }
            // let a dependent kernel start its prologue
            ptx::pdl_launch_dependents();
        }
    } else if (warp == 1 || warp == 10) {
        // ------------------------------------------------------------ MMA issuer(s)
        const int me = warp == 1 ? 0 : 1;
        if (me == 0 || dual || ordered) {
            uint32_t it = 0;
            uint32_t t = 0;
            bool ok = true;
            WorkIter<BN> work(grp, M, N, tiles_m, tiles_n, run_table, first_item, item_step);
            Work wk;
            for (; ok && work.next(wk); ++t) {
                const uint32_t as = t & 1u;
                const uint32_t aph = (t >> 1) & 1u;
                // (with two issuers both wait here, also the one that has no k-tile in a tile of
                // one: its arrival below must not run ahead of the stage's previous use)
                ok = wait_bar<kSplitK>(ptx::smem_u32(&bars->acc_empty[as]), aph ^ 1u, abort, kStatusMma);
                if (!ok) break;
                if (C::kOverlap != 0 && t > 0) {
                    // the previous tile's epilogue has drained the columns both stages share
                    ok = wait_bar<kSplitK>(ptx::smem_u32(&bars->overlap_free[as ^ 1u]), ((t - 1) >> 1) & 1u,
                                  abort, kStatusMma);
                    if (!ok) break;
                }
                ptx::tc_fence_after();
                const uint32_t acc = tmem + ((me == 0 || ordered) ? as * C::kAccStride : C::kDualCol + as * BN);
                // a 64-wide tile uses half of a 128-row scale atom
                const uint32_t sfb_shift = BN == 64 ? uint32_t(wk.sfb_shift) : 0u;
                bool issued = false;
                for (int kt = k_begin; kt < k_end; ++kt, ++it) {
                    if (dual && ((kt - k_begin) & 1) != me) continue;
                    if (ordered && int(it & 1u) != me) continue;
                    const uint32_t s = it % kRing;
                    const uint32_t ph = (it / kRing) & 1u;
                    // the scales of this k-tile are in their set (the scale warps waited for the
                    // scale bytes); the stage's own barrier orders this thread after the TMA writes
                    ok = wait_bars<kSplitK>(ptx::smem_u32(&bars->sf_ready[it % C::kSfSets]), (it / C::kSfSets) & 1u, true,
                                   ptx::smem_u32(&bars->full[s]), ph, abort, kStatusMma);
                    // (in-order pair of issuers) the other thread has issued the MMAs of the previous k-iteration
                    if (ok && ordered && it > 0u) {
                        ok = wait_bar<kSplitK>(ptx::smem_u32(&bars->turn[me]), ((it - 1u) >> 1) & 1u, abort, kStatusMma);
                    }
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint32_t set = tmem + (it % C::kSfSets) * C::kSfCols;
                    const uint64_t adesc = ptx::smem_desc(a_base + s * C::kABytes, 16, 1024, 2);
                    const uint64_t bdesc = ptx::smem_desc(b_base + s * C::kBBytes, 16, 1024, 2);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        // 32 bytes of K per instruction: K = 32 (e4m3) or 64 (e2m1)
                        uint32_t atom, sf_id;
                        if constexpr (KIND == 0 || KIND == 3) {
                            atom = 0;
                            sf_id = k;
                        } else if constexpr (KIND == 1) {
                            atom = k;
                            sf_id = 0;
                        } else {
                            atom = k >> 1;
                            sf_id = (k & 1) * 2;
                        }
                        if (ptx::elect_one()) {
                            ptx::tc_mma_block_scaled<1, KIND>(
                                acc, adesc + uint64_t(k * 2), bdesc + uint64_t(k * 2),
                                instr_desc<BN, KIND>(sf_id), set + C::kSfaCol + atom * 4,
                                set + C::kSfbCol + atom * C::kNAtoms * 4 + sfb_shift,
                                (ordered ? (kt > k_begin || k > 0) : (issued || k > 0)) ? 1u : 0u);
                        }
                    }
                    issued = true;
                    if (ordered) {
                        // hand the turn over before the (slow) commit
                        ptx::tc_fence_before();
                        if (ptx::elect_one()) ptx::mbar_arrive(ptx::smem_u32(&bars->turn[me ^ 1]));
                    }
                    // stage s may be refilled once these MMAs have read it
                    if (ptx::elect_one()) ptx::tc_commit(ptx::smem_u32(&bars->empty[s]));
                }
                if (!ok) break;
                // a commit tracks the executing thread's operations: every issuer reports its own
                if (ptx::elect_one()) {
                    if (issued) {
                        ptx::tc_commit(ptx::smem_u32(&bars->acc_full[as]));
                    } else {
                        ptx::mbar_arrive(ptx::smem_u32(&bars->acc_full[as]));
                    }
                }
            }
        }
    } else if (warp >= 2 + kEpiWarps) {
        // ------------------------------------------------------------ scales -> tensor memory (warps 6-9)
        // One SfAtom is 32 rows of 16 bytes; lane l of every lane quarter of tensor memory
        // holds row l in 4 columns (what tcgen05.cp.32x128b.warpx4 would write).  Each of
        // the four warps fills its own quarter from the same shared-memory image.
        const uint32_t quarter = (uint32_t(warp) & 3u) * 32u;
        uint32_t it = 0;
        bool ok = true;
        WorkIter<BN> work(grp, M, N, tiles_m, tiles_n, run_table, first_item, item_step);
        Work wk;
        while (ok && work.next(wk)) {
            for (int kt = k_begin; kt < k_end; ++kt, ++it) {
                const uint32_t s = it % kRing;
                // the MMAs of k-tile it - kSfSets read this set: they are done once they
                // have released their stage
                const uint32_t prev = it - uint32_t(C::kSfSets);
                const uint32_t sf_full = ptx::smem_u32(&bars->sf_full[s]);
                const uint32_t set_free = ptx::smem_u32(&bars->empty[prev % kRing]);
                // A k-tile's scales go to registers first, and on with as few stores as there are.  Where only
                // two sets rotate and a set is large, the loads do not wait for it: what lies between its release and
                // the MMAs that wait for its next scales is on the critical path there, and it was 12 loads and 12
                // stores one after the other, some 700 cycles against 512 of one k-tile's MMAs (NVFP4 512 x 4096 x 4096 on the
                // 128 x 256 tile 10.9 -> 9.9 us, 4096 x 14336 x 4096 128 -> 121, 8192 x 8192 x 8192 270 -> 254, sustained).
                // Elsewhere the second vote costs more than it saves (NVFP4 4096 x 4096 x 4096 on 128 x 128 36.2 -> 36.8).
                uint32_t r[C::kSfCols];
                const auto load = [&] { load_scales<C>(sfa_base + s * C::kSfaBytes, sfb_base + s * C::kSfbBytes, lane, r); };
                if constexpr (C::kSfSets == 2 && C::kSfKAtoms > 1) {
                    ok = wait_bar<kSplitK>(sf_full, (it / kRing) & 1u, abort, kStatusProducer);
                    if (!ok) break;
                    load();
                    if (it >= uint32_t(C::kSfSets)) ok = wait_bar<kSplitK>(set_free, (prev / kRing) & 1u, abort, kStatusProducer);
                    if (!ok) break;
                } else {
                    ok = wait_bars<kSplitK>(sf_full, (it / kRing) & 1u, it >= uint32_t(C::kSfSets), set_free, (prev / kRing) & 1u,
                                   abort, kStatusProducer);
                    if (!ok) break;
                    load();
                }
                ptx::tc_fence_after();
                const uint32_t set = tmem + (quarter << 16) + C::kSfaCol + (it % C::kSfSets) * C::kSfCols;
                ptx::tc_store_32x32<C::kSfCols>(set, r);
                ptx::tc_wait_st();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->sf_ready[it % C::kSfSets]));
            }
        }
    } else {
        // ------------------------------------------------------------ epilogue
        const int ew = warp - 2;                  // staging buffer owner
        const uint32_t lane_base = (warp & 3) * 32;  // tensor-memory lanes this warp may read
        uint32_t t = 0;
        uint32_t stores = 0;
        bool ok = true;
        float scale = 1.0f;
        int scale_group = -1;
        WorkIter<BN> work(grp, M, N, tiles_m, tiles_n, run_table, first_item, item_step);
        Work wk;
        const int ar = int(lane_base) + lane;  // accumulator row of this thread
        if (!kPlain && situ.sf != nullptr) zero_sf_padding(situ, (warp - 2) * 32 + lane);
        for (; ok && work.next(wk); ++t) {
            const int m0 = wk.out_row0;  // output row of accumulator row 0
            const int n0 = wk.out_col0;
            // this warp's 32 rows are all padding or all belong to a neighbouring group
            const bool warp_idle = int(lane_base) >= wk.row_hi || int(lane_base) + 32 <= wk.row_lo;
            const bool row_ok = ar >= wk.row_lo && ar < wk.row_hi;
            // rows go out through TMA stores (a dense tail is clipped by the tensor map), except where only some of
            // this warp's are the item's: those are stored from registers, row by row, and so are items of at most
            // 32 rows (no staging round trip: NVFP4, two batches of 32 x 1792 x 768, 4.0 us with it)
            const bool warp_whole = int(lane_base) >= wk.row_lo && int(lane_base) + 32 <= wk.row_hi;
            const bool reg_store = direct_store != 0 || wk.row_hi - wk.row_lo <= 32 ||
                                   (!warp_whole && grp.kind != kGroupDense);
            // per-tensor (dense) or per-group factor of the NVFP4 recipe
            if (KIND == 1 && alpha != nullptr && wk.group != scale_group) {
                scale = __ldg(alpha + wk.group);
                scale_group = wk.group;
            }
            const uint32_t as = t & 1u;
            const uint32_t aph = (t >> 1) & 1u;
            ok = wait_bar<kSplitK>(ptx::smem_u32(&bars->acc_full[as]), aph, abort, kStatusEpilogue);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint32_t acc = tmem + as * C::kAccStride + (lane_base << 16);
            if (!kPlain && KIND == 0 && epi_op == HQ_EPILOGUE_SITU_QUANT) {
                // quantising epilogue: 64 accumulator columns -> one group of 32 e4m3 outputs
                constexpr int kGroups = C::kChunks / 2;
#pragma unroll 1
                for (int gi = 0; gi < kGroups; ++gi) {
                    const int g = (C::kOverlap != 0 && as == 0) ? kGroups - 1 - gi : gi;
                    uint32_t r0[32], r1[32];
                    ptx::tc_load_32x32(acc + (2 * g) * kEpiChunk, r0);
                    ptx::tc_load_32x32(acc + (2 * g + 1) * kEpiChunk, r1);
                    ptx::tc_wait_ld();
                    if (C::kOverlap != 0 && gi == (C::kOverlapChunks - 1) / 2) {
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->overlap_free[as]));
                    }
                    if (gi == kGroups - 1) {
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->acc_empty[as]));
                    }
                    if (warp_idle) continue;  // (N is a multiple of 256 here: no ragged tile)
                    uint32_t y[16];
                    const __nv_bfloat16* const bc = bias != nullptr ? bias + n0 + 2 * g * kEpiChunk : nullptr;
                    situ_chunk(r0, bc, situ, &y[0]);
                    situ_chunk(r1, bc != nullptr ? bc + kEpiChunk : nullptr, situ, &y[8]);
                    uint4 lo, hi;
                    const uint32_t e = quant32_bf16(y, lo, hi);
                    const int64_t row = m0 + ar;
                    if (row_ok) {
                        const int kb = (n0 >> 6) + g;  // group of 32 output columns
                        uint4* const dst = reinterpret_cast<uint4*>(situ.q + row * situ.ldq + int64_t(kb) * 32);
                        dst[0] = lo;
                        dst[1] = hi;
                        situ.sf[((row >> 7) * (situ.kb_out >> 2) + (kb >> 2)) * 512 + (row & 31) * 16 +
                                ((row >> 5) & 3) * 4 + (kb & 3)] = uint8_t(e);
                    }
                }
                continue;
            }
            // Several chunks of columns shared with the other accumulator stage (FP4 kinds: the
            // scale sets take 48-96 columns): read them all into registers first, so that the
            // next tile's MMAs may start after three tensor-memory loads instead of after two
            // or three whole chunk iterations (convert, staging buffer, TMA store).
            constexpr int kPre = C::kOverlapChunks > 1 ? C::kOverlapChunks : 0;
            uint32_t ro[kPre > 0 ? kPre : 1][32];
            if constexpr (kPre > 0) {
#pragma unroll
                for (int j = 0; j < kPre; ++j) {
                    const int c = as == 0 ? C::kChunks - 1 - j : j;
                    ptx::tc_load_32x32(acc + c * kEpiChunk, ro[j]);
                }
                ptx::tc_wait_ld();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->overlap_free[as]));
            }
#pragma unroll 1
            for (int ci = 0; ci < C::kChunks; ++ci) {
                // stage 0 shares its highest columns with stage 1, stage 1 its lowest with stage 0
                const int c = (C::kOverlap != 0 && as == 0) ? C::kChunks - 1 - ci : ci;
                uint32_t r[32];
                if (kPre > 0 && ci < kPre) {
#pragma unroll
                    for (int j = 0; j < kPre; ++j) {
                        if (ci == j) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) r[i] = ro[j][i];
                        }
                    }
                } else {
                    ptx::tc_load_32x32(acc + c * kEpiChunk, r);
                    ptx::tc_wait_ld();
                }
                if constexpr (BN == 64 && kDense && !kSplitK) {
                    // the second issuer's accumulator (it has k-tiles whenever the tile has two or more)
                    if (dual && k_end - k_begin > 1) {
                        uint32_t r2[32];
                        ptx::tc_load_32x32(tmem + C::kDualCol + as * BN + (lane_base << 16) + c * kEpiChunk, r2);
                        ptx::tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(r2[i]));
                    }
                }
                if constexpr (kSplitK) {
                    // row `ar`, columns [32 c, 32 c + 32) of the 128 x 64 fp32 buffer
                    const uint32_t slot = recv_base + uint32_t(ar) * (BN * 4) + uint32_t(c) * (kEpiChunk * 4);
                    if (k_rank != 0) {
                        // an aborting CTA sends nothing more across the pair (one decision per warp)
                        ok = __any_sync(0xffffffffu, *abort != 0u ? 1 : 0) == 0;
                        if (!ok) break;
                        const uint32_t dst = ptx::mapa_cluster(slot, 0);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            ptx::st_cluster_v4(dst + j * 16, __uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]),
                                               __uint_as_float(r[4 * j + 2]), __uint_as_float(r[4 * j + 3]));
                        }
                        if (ci == C::kChunks - 1) {
                            // every lane's stores are ordered before the warp's one remote arrive
                            __syncwarp();
                            if (lane == 0) {
                                ptx::mbar_arrive_cluster_addr(ptx::mapa_cluster(ptx::smem_u32(&bars->recv_full), 0));
                            }
                            ptx::tc_fence_before();
                            __syncwarp();
                            if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->acc_empty[as]));
                        }
                        continue;
                    }
                    if (ci == 0) {
                        // this tile's partial sums (one phase of the barrier per tile)
                        ok = wait_bar_cluster<kSplitK>(ptx::smem_u32(&bars->recv_full), t & 1u, abort, kStatusEpilogue);
                        if (!ok) break;
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float4 v;
                        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                                     : "r"(slot + j * 16));
                        r[4 * j] = __float_as_uint(__uint_as_float(r[4 * j]) + v.x);
                        r[4 * j + 1] = __float_as_uint(__uint_as_float(r[4 * j + 1]) + v.y);
                        r[4 * j + 2] = __float_as_uint(__uint_as_float(r[4 * j + 2]) + v.z);
                        r[4 * j + 3] = __float_as_uint(__uint_as_float(r[4 * j + 3]) + v.w);
                    }
                }
                if (C::kOverlap != 0 && kPre == 0 && ci == C::kOverlapChunks - 1) {
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->overlap_free[as]));
                }
                if (ci == C::kChunks - 1) {
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) ptx::mbar_arrive(ptx::smem_u32(&bars->acc_empty[as]));
                }
                if (warp_idle || c * kEpiChunk >= wk.cols) continue;
                uint32_t p[16];
                epilogue_chunk(r, p, scale, bias != nullptr ? bias + wk.bias_col0 + c * kEpiChunk : nullptr,
                               epi_op);
                const int row = m0 + ar;
                const int col = n0 + c * kEpiChunk;
                if (!kPlain && (epi_op == HQ_EPILOGUE_QUANT || epi_op == HQ_EPILOGUE_GATE_MUL_QUANT ||
                                epi_op == HQ_EPILOGUE_SIGMOID_GATE_MUL_QUANT)) {
                    // The bf16 result (times the gate, as a bf16 product) re-quantised to MXFP8 per
                    // 32 columns: the reference's batch epilogues (csrc/kernel/gemm/epilogue.cuh:990-1051).
                    if (row_ok) {
                        if (epi_op != HQ_EPILOGUE_QUANT) {
                            const uint4* const gp =
                                reinterpret_cast<const uint4*>(situ.gate + int64_t(row) * situ.gate_ld + col);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const uint4 gq = __ldg(gp + j);
                                uint32_t gw[4] = {gq.x, gq.y, gq.z, gq.w};
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    if (epi_op == HQ_EPILOGUE_SIGMOID_GATE_MUL_QUANT) {
                                        const float lo = fmaf(0.5f, tanh_fast(0.5f * __uint_as_float(gw[i] << 16)), 0.5f);
                                        const float hi =
                                            fmaf(0.5f, tanh_fast(0.5f * __uint_as_float(gw[i] & 0xffff0000u)), 0.5f);
                                        const __nv_bfloat162 sg = __float22bfloat162_rn(make_float2(lo, hi));
                                        gw[i] = *reinterpret_cast<const uint32_t*>(&sg);
                                    }
                                    const __nv_bfloat162 prod =
                                        __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&p[4 * j + i]),
                                                *reinterpret_cast<const __nv_bfloat162*>(&gw[i]));
                                    p[4 * j + i] = *reinterpret_cast<const uint32_t*>(&prod);
                                }
                            }
                        }
                        uint4 lo, hi;
                        const uint32_t e = quant32_bf16(p, lo, hi);
                        const int kb = col >> 5;
                        uint4* const dst = reinterpret_cast<uint4*>(situ.q + int64_t(row) * situ.ldq + col);
                        dst[0] = lo;
                        dst[1] = hi;
                        situ.sf[(int64_t(row >> 7) * (situ.kb_out >> 2) + (kb >> 2)) * 512 + (row & 31) * 16 +
                                ((row >> 5) & 3) * 4 + (kb & 3)] = uint8_t(e);
                    }
                    continue;
                }
                if (reg_store) {
                    if (row_ok) {
                        uint4* dst = reinterpret_cast<uint4*>(out + int64_t(row) * ldo + col);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            dst[j] = make_uint4(p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
                        }
                    }
                } else {
                    const uint32_t buf =
                        epi_base + (ew * C::kEpiBufs + (stores % C::kEpiBufs)) * kEpiBufBytes;
                    // the TMA store that last read this buffer must be done with it
                    if (lane == 0) ptx::bulk_wait_read<C::kEpiBufs - 1>();
                    __syncwarp();
                    // 32 rows x 64 bytes, 64-byte swizzle: 16-byte chunk j of row r
                    // sits at chunk j ^ ((r >> 1) & 3)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t dst = buf + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst),
                                     "r"(p[4 * j]), "r"(p[4 * j + 1]), "r"(p[4 * j + 2]),
                                     "r"(p[4 * j + 3])
                                     : "memory");
                    }
                    ptx::fence_proxy_async_smem();
                    __syncwarp();
                    if (lane == 0) {
                        ptx::tma_store_2d(&tm_d, buf, col, m0 + int(lane_base));
                        ptx::bulk_commit();
                    }
                    ++stores;
                }
            }
        }
        if (lane == 0) ptx::bulk_wait_read<0>();
    }

    if (*abort != 0u) {
        // bounded grace period for copies / MMAs still in flight before the
        // shared and tensor memory they target is released
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before();
    __syncthreads();
    // split-K: neither CTA of the pair leaves while the other may still store partial sums
    // into its shared memory or arrive on its barrier (every wait above is bounded, so both
    // get here)
    if (kSplitK) ptx::cluster_sync();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc<1>(tmem, C::kTmemCols);
    }
}

// Self-test of the bounded wait and of the way a timeout spreads: thread 0 waits, with a
// short limit, on a barrier that nothing ever arrives on; thread 32 waits on the same
// barrier with the ordinary limit and must leave as soon as it sees the abort flag thread
// 0 raises.  The third warp makes a role's wait in which half of the lanes ask for a phase that is over and
// half for one that never ends: all of them must be told to leave.  Nothing is in flight when the
// waits give up: no copies, no MMAs, no tensor memory.  What the host then reads through hq_device_status
// is what it would read after a GEMM role had timed out.
__global__ void __launch_bounds__(96, 1) wait_selftest_kernel(uint64_t limit_ns) {
    __shared__ uint64_t bar;
    __shared__ uint32_t abort_flag;
    if (threadIdx.x == 0) {
        ptx::mbar_init(ptx::smem_u32(&bar), 1);
        abort_flag = 0;
        ptx::fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        wait_bar_lane(ptx::smem_u32(&bar), 0, &abort_flag, kStatusMma, limit_ns);
    } else if (threadIdx.x == 32) {
        // sees the flag within 32 polls of its being raised; its own limit never runs out
        if (wait_bar_lane(ptx::smem_u32(&bar), 0, &abort_flag, kStatusEpilogue)) atomicOr(&g_status[0], 0x80u);
    } else if (threadIdx.x >= 64) {
        // (the phase before the first counts as over)
        if (wait_bar(ptx::smem_u32(&bar), threadIdx.x & 1u, &abort_flag, kStatusEpilogue)) atomicOr(&g_status[0], 0x40u);
    }
    __syncwarp();
    __syncthreads();
}

// ---------------------------------------------------------------------------- 2-CTA tiles
//
// Pair kernel: a cluster of two CTAs computes one 256 x BN tile with
// tcgen05.mma.cta_group::2 (M = 256).  CTA r of the pair owns rows
// [128 r, 128 r + 128) of the A tile, rows [r BN/2, (r + 1) BN/2) of the B tile and the
// matching half of the accumulator; both CTAs hold the scales of all BN columns.
// Every CTA loads its own halves with plain (non-broadcast) TMA copies in the
// cta_group::2 form, which lets the bytes be counted on the leader's (rank 0)
// barrier; only the leader issues tcgen05.mma.  It releases a stage, and publishes an accumulator, with
// one tcgen05.commit that arrives in both CTAs.  The scales of a k-tile go from shared to tensor memory
// by four warps of each CTA, as in the single-CTA kernel, which report to the leader, as the epilogue warps of
// both CTAs do.  Per CTA this halves the B traffic from L2 and leaves room for 6 stages instead of 4.
//
// What bounds it: large problems the power cap (clocks of 1.1 to 1.4 GHz), so the bytes that each product moves count
// more than the cycles between them; small ones the hand-over between the k-tiles.  Against scales copied by
// tcgen05.cp from one warp (75 to 90 cycles a copy, a commit behind them) and a release that the leader's loader
// passed on: MXFP8 8192 x 8192 x 8192 462 -> 448 us, 4096 x 7168 x 2048 58.4 -> 56.5, 512 x 4096 x 4096 16.4 -> 15.0,
// 4096 x 4096 x 4096 on the 256 x 128 tile 80 -> 64 (sustained, GEMM alone; the waits' part of the last is 10).  NVFP4, with
// 12 copies a k-tile: 8192 x 8192 x 8192 295 -> 233, which made it the better tile for the FP4 kinds too
// (single-CTA 128 x 256: 248); 4096 x 4096 x 4096 44 -> 35.5 (41).

template <int BN, int KIND>
struct Cfg2 {
    static_assert(BN == 128 || BN == 256, "pair tile widths built");
    static constexpr int kABytes = kBM * kBKBytes;
    static constexpr int kBBytes = (BN / 2) * kBKBytes;
    static constexpr bool kFp8Kind = KIND == 0 || KIND == 3;  // mxf8f6f4: e4m3 x e4m3, or e4m3 x packed e2m1
    static constexpr int kSfKAtoms = kFp8Kind ? 1 : (KIND == 1 ? 4 : 2);
    static constexpr int kNAtoms = BN / 128;
    static constexpr int kSfaBytes = kSfKAtoms * 512;
    static constexpr int kSfbBytes = kNAtoms * kSfaBytes;
    static constexpr int kStageBytes = kABytes + kBBytes + kSfaBytes + kSfbBytes;
    // operand bytes a stage reads from global memory: packed e2m1 weights (KIND 3) are spread to one byte
    // per value by the copy, and the barrier counts what was read
    static constexpr int kStageTxBytes = kABytes + kBBytes - (KIND == 3 ? kBBytes / 2 : 0);
    static constexpr int kEpiBufs = 2;
    static constexpr int kEpiBytes = kEpiWarps * kEpiBufs * kEpiBufBytes;
    static constexpr int kBarBytes = 1024 + kRunBytes;  // barriers, then the runs of contiguous experts
    static constexpr int kStagesFit = (kSmemBudget - kEpiBytes - kBarBytes - 1024) / kStageBytes;
    static constexpr int kStages = kStagesFit > 8 ? 8 : kStagesFit;
    static constexpr int kSmemBytes = kStages * kStageBytes + kEpiBytes + kBarBytes + 1024;
    // Scale columns of one k-iteration and how many such sets rotate in tensor memory.  A set is free again once the
    // MMAs that read it have completed, so with 4 sets the scales run two k-tiles ahead; NVFP4's 48 columns
    // leave room for 2.
    static constexpr int kSfCols = kSfKAtoms * 4 * (1 + kNAtoms);
    static constexpr int kSfSets = BN < 256 || KIND != 1 ? 4 : 2;
    // warps: 0 box loader, 1 MMA issuer, 2-5 epilogue, 6 scale loader, 7-10 scales to tensor memory, 11 MMA issuer
    // Two threads (of warp 1 and of the last warp) issue the MMAs of alternate k-tiles.  After its MMAs a thread
    // hands the turn to the other one (tcgen05 fences around an mbarrier arrive), so the
    // MMAs still reach the tensor core in k order.
    static constexpr int kMma2Warp = 7 + kSfWarps;
    static constexpr int kThreads = 32 * (kMma2Warp + 1);
    static constexpr int kSfRegion = kSfCols * kSfSets;
    static constexpr int kOverlap = BN == 256 ? (kSfRegion + 15) / 16 * 16 : 0;
    static constexpr int kAccStride = BN - kOverlap;
    static constexpr int kSfCol0 = kAccStride + BN;
    static constexpr int kColsUsed = kSfCol0 + kSfRegion;
    static constexpr int kTmemCols = kColsUsed <= 256 ? 256 : 512;
    static_assert(kColsUsed <= 512, "tensor memory budget");
    static constexpr int kChunks = BN / kEpiChunk;
    static constexpr int kOverlapChunks = (kOverlap + kEpiChunk - 1) / kEpiChunk;
    static_assert(kStages >= 2, "pipeline depth");
};

template <int BN, int KIND>
__device__ __forceinline__ uint32_t instr_desc_pair(uint32_t sf_id) {
    // (the fields and format codes of instr_desc; M = 256 across the pair)
    constexpr uint32_t fmt_a = (KIND == 0 || KIND == 3) ? 0u : 1u;
    constexpr uint32_t fmt_b = KIND == 0 ? 0u : (KIND == 3 ? 5u : 1u);
    constexpr uint32_t scale_fmt = KIND == 1 ? 0u : 1u;
    return (sf_id << 4) | (fmt_a << 7) | (fmt_b << 10) | (uint32_t(BN >> 3) << 17) | (scale_fmt << 23) |
           (uint32_t(256 >> 4) << 24) | (sf_id << 29);
}

// What one persistent-loop iteration of the 2-CTA kernel works on: a 256-row tile of the
// stacked A rows against BN rows of one weight.
struct PairWork {
    int a_row0;     // first of the tile's 256 stacked A rows (a multiple of 128: runs of experts start there; of 256 otherwise)
    int b_row0;     // first of the BN weight rows in the stacked weights
    int sfb_tile;   // 128-row scale atom row of that row
    int cols;       // weight rows of the tile that exist (see Work)
    int row_lo;     // tile rows [row_lo, row_hi) belong to this item; the others are padding,
    int row_hi;     //   belong to another expert, or lie beyond M
    int group;      // weight index: selects alpha
    int out_row0;   // output row of tile row 0
    int out_col0;   // first output column
    int bias_col0;  // first bias element
};

// The grouped kinds on the 2-CTA tile (kGrouped; dense otherwise).  Batches and masked experts
// take it when their row count is a multiple of 256, so that no tile holds rows of two of
// them; an item is (expert, 256-row tile that holds valid rows of it, column tile).  The
// contiguous layout is cut into tiles by runs of experts (RunTable); with more runs than the table holds, a tile
// whose four 64-row quarters belong to several experts is worked once per run of equal experts, each pass storing
// its own rows.  The roles of the kernel walk the same sequence of items, each with its own copy of this iterator.
template <int BN, bool kGrouped>
struct PairWorkIter {
    GroupParams g;
    int M, N, tiles_m, tiles_n;
    int tile, stride;
    int pass = 0;        // contiguous: run of the current tile to work next
    int walk_group = 0;  // batch / masked: group of the last item and the number of
    int walk_base = 0;   //   (group, row tile) pairs before it
    RunWalk<256> runs;   // contiguous

    __device__ PairWorkIter(const GroupParams& grp, int m, int n, int tm, int tn, const RunTable& rt, int first, int step)
        : g(grp), M(m), N(n), tiles_m(tm), tiles_n(tn), tile(first), stride(step), runs{rt} {
        if (kGrouped && g.kind == kGroupContiguous && rt.runs != nullptr) tiles_m = rt.row_tiles;
    }

    __device__ __forceinline__ void set_b(PairWork& w, int group, int nt) const {
        w.group = group;
        w.cols = min(BN, N - nt * BN);
        w.b_row0 = group * N + nt * BN;
        w.sfb_tile = group * ((N + 127) / 128) + (nt * BN) / 128;
        w.bias_col0 = w.b_row0;
    }

    // How many items next() will give: the roles that work k-tiles whatever they belong to (scales, MMAs) count them down
    // instead of walking.  -1: only the walk can tell (contiguous experts without a run table).
    __device__ int items() const {
        int row_tiles = tiles_m;
        if constexpr (kGrouped) {
            if (g.kind == kGroupContiguous && runs.t.runs == nullptr) return -1;
            if (g.kind == kGroupBatch) row_tiles = g.count * ((g.rows + 255) / 256);
            if (g.kind == kGroupMasked) {
                row_tiles = 0;
                for (int e = 0; e < g.count; ++e) row_tiles += (min(max(__ldg(g.table + e), 0), g.rows) + 255) / 256;
            }
        }
        const int total = row_tiles * tiles_n;
        return tile < total ? (total - tile + stride - 1) / stride : 0;
    }

    __device__ bool next(PairWork& w) {
        if (!kGrouped || g.kind == kGroupContiguous) {
            if (tile >= tiles_m * tiles_n) return false;
            const TileCoord tc = tile_coord(tile, tiles_m, tiles_n);
            w.out_col0 = tc.n * BN;
            int group = 0;
            bool last = true;
            if (kGrouped && runs.t.runs != nullptr) {
                runs.find(tc.m, w.a_row0, w.row_lo, w.row_hi, group);
                w.out_row0 = w.a_row0;
                set_b(w, group, tc.n);
                tile += stride;
                return true;
            }
            w.a_row0 = tc.m * 256;
            w.out_row0 = w.a_row0;
            w.row_lo = 0;
            w.row_hi = min(256, M - w.a_row0);
            if constexpr (kGrouped) {
                int e[4];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int row = w.a_row0 + 64 * q;
                    e[q] = row < M ? min(max(__ldg(g.table + row), 0), g.count - 1) : e[q > 0 ? q - 1 : 0];
                }
                int start = 0, run = 0, cur = e[0];
                bool found = false;
                group = e[0];
#pragma unroll
                for (int q = 1; q <= 4; ++q) {
                    const bool ends = q == 4 || e[q & 3] != e[q - 1];  // the run [start, q) of quarters ends here
                    if (!found && ends) {
                        if (run == pass) {
                            w.row_lo = 64 * start;
                            w.row_hi = min(64 * q, M - w.a_row0);
                            group = cur;
                            last = q == 4;
                            found = true;
                        } else {
                            ++run;
                            start = q;
                            cur = e[q & 3];
                        }
                    }
                }
                pass = last ? 0 : pass + 1;
            }
            set_b(w, group, tc.n);
            if (last) tile += stride;
            return true;
        }
        // batch / masked
        const int pair = tile / tiles_n;
        const int nt = tile - pair * tiles_n;
        int first, valid;
        for (;;) {
            if (walk_group >= g.count) return false;
            first = walk_group * g.rows;
            valid = g.kind == kGroupMasked ? min(max(__ldg(g.table + walk_group), 0), g.rows) : g.rows;
            const int cnt = (valid + 255) / 256;
            if (pair < walk_base + cnt) break;
            walk_base += cnt;
            ++walk_group;
        }
        const int rt = pair - walk_base;
        w.a_row0 = first + rt * 256;
        w.row_lo = 0;
        w.row_hi = min(256, valid - rt * 256);
        set_b(w, walk_group, nt);
        if (g.kind == kGroupBatch) {
            w.out_row0 = w.a_row0 - first;
            w.out_col0 = w.b_row0;
        } else {
            w.out_row0 = w.a_row0;
            w.out_col0 = nt * BN;
        }
        tile += stride;
        return true;
    }
};

// What the grouped 2-CTA kernel needs beyond the tensor maps: the groups, and the output for
// the rows it stores from registers (tiles that are only partly this item's).
struct PairGroupArgs {
    GroupParams grp;
    __nv_bfloat16* out;
    int64_t ldo;
    int m;  // stacked A rows
    int n;  // columns per weight
};

// Column-parallel all-gather fused into the epilogue (kGather): besides its own output, a rank
// stores every finished chunk of a tile into the same columns of its peers' outputs (symmetric
// memory mapped over NVLink): the TMA store that writes the staged chunk to the local output
// is repeated with a tensor map over each peer's matrix.  Every LOAD of the kernel (operands,
// scales) is from this GPU's memory.
template <bool kGather>
struct GatherMaps {
    int count;
};
template <>
struct GatherMaps<true> {
    CUtensorMap out[7];  // the peers' outputs, each map starting at this rank's first column
    int count;
};

// The epilogue of a warp of which some or none of the 32 rows are the item's: each thread stores its own row from
// registers, or nothing (`out` null).  A function of its own: in a branch inside the chunk loop it cost every tile 8 %, full
// ones too (32768 x 3072 x 1280 NVFP4 in one batch 102.7 us with it there, 94.9 without).
template <typename C>
__device__ __noinline__ void partial_rows(uint32_t acc, bool second_stage, __nv_bfloat16* out, float scale,
                                          const __nv_bfloat16* bias, int epi_op, int cols, uint32_t overlap_free,
                                          uint32_t acc_empty) {
    const int lane = threadIdx.x & 31;
#pragma unroll 1
    for (int ci = 0; ci < C::kChunks; ++ci) {
        const int c = (C::kOverlap != 0 && !second_stage) ? C::kChunks - 1 - ci : ci;
        uint32_t r[32];
        ptx::tc_load_32x32(acc + c * kEpiChunk, r);
        ptx::tc_wait_ld();
        const bool overlap_read = C::kOverlap != 0 && ci == C::kOverlapChunks - 1;
        if (overlap_read || ci == C::kChunks - 1) {
            ptx::tc_fence_before();
            __syncwarp();
            if (lane == 0 && overlap_read) ptx::mbar_arrive_cluster_relaxed(overlap_free);
            if (lane == 0 && ci == C::kChunks - 1) ptx::mbar_arrive_cluster_relaxed(acc_empty);
        }
        if (out == nullptr || c * kEpiChunk >= cols) continue;
        uint32_t p[16];
        epilogue_chunk(r, p, scale, bias != nullptr ? bias + c * kEpiChunk : nullptr, epi_op);
        uint4* const dst = reinterpret_cast<uint4*>(out + c * kEpiChunk);
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[j] = make_uint4(p[4 * j], p[4 * j + 1], p[4 * j + 2], p[4 * j + 3]);
    }
}

// The SiTU-GLU quantising epilogue's outputs (kSitu; dense MXFP8 only).
template <bool kSitu>
struct PairSitu {};
template <>
struct PairSitu<true> {
    SituParams p;
};

template <int BN, int KIND, bool kGather = false, bool kGrouped = false, bool kSitu = false>
__global__ void __launch_bounds__((Cfg2<BN, KIND>::kThreads), 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                 const __grid_constant__ CUtensorMap tm_d, const __grid_constant__ CUtensorMap tm_sfa,
                 const __grid_constant__ CUtensorMap tm_sfb, const float* __restrict__ alpha,
                 const __nv_bfloat16* __restrict__ bias_arg, int epi_arg, int k_tiles, int kq_dim, int tiles_m,
                 int tiles_n, int prefetch_weight, const __grid_constant__ GatherMaps<kGather> peers, const PairGroupArgs ga,
                 const PairSitu<kSitu> situ) {
    using C = Cfg2<BN, KIND>;
    // (only MXFP8 takes a bias, only the dense form another epilogue than Identity: less to hold through the loop over the chunks)
    const __nv_bfloat16* const bias = KIND == 0 ? bias_arg : nullptr;
    const int epi_op = kGrouped ? HQ_EPILOGUE_IDENTITY : epi_arg;
    using Iter = PairWorkIter<BN, kGrouped>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* const smem = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
    const uint32_t a_base = smem_base;
    const uint32_t b_base = a_base + C::kStages * C::kABytes;
    const uint32_t sfa_base = b_base + C::kStages * C::kBBytes;
    const uint32_t sfb_base = sfa_base + C::kStages * C::kSfaBytes;
    const uint32_t epi_base = sfb_base + C::kStages * C::kSfbBytes;
    const uint32_t bar_off = C::kStages * C::kStageBytes + C::kEpiBytes;
    Barriers* const bars = reinterpret_cast<Barriers*>(smem + bar_off);
    volatile uint32_t* const abort = &bars->abort;

    const int warp = warp_index();
    const int lane = threadIdx.x & 31;
    const uint32_t rank = ptx::cluster_ctarank();  // 0 = leader
    const bool leader = rank == 0;
    const int cluster_id = blockIdx.x >> 1;
    const int num_clusters = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < C::kStages; ++s) {
            // the leader's copy collects the operand bytes of both CTAs after one
            // expect_tx arrival of the leader's producer; the scales' bytes are each CTA's own matter
            ptx::mbar_init(ptx::smem_u32(&bars->full[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&bars->sf_full[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&bars->empty[s]), 1);  // one tcgen05.commit
        }
        for (int s = 0; s < 2; ++s) {
            ptx::mbar_init(ptx::smem_u32(&bars->acc_full[s]), 2);  // one commit per MMA-issuing thread
            ptx::mbar_init(ptx::smem_u32(&bars->acc_empty[s]), 2 * kEpiWarps);  // leader's copy is used
            ptx::mbar_init(ptx::smem_u32(&bars->overlap_free[s]), 2 * kEpiWarps);
        }
        // (the leader's copy is used)
        for (int s = 0; s < C::kSfSets; ++s) ptx::mbar_init(ptx::smem_u32(&bars->sf_ready[s]), 2 * kSfWarps);
        for (int s = 0; s < 2; ++s) ptx::mbar_init(ptx::smem_u32(&bars->turn[s]), 1);
        bars->abort = 0;
        ptx::fence_mbar_init();
        ptx::prefetch_tmap(&tm_a);
        ptx::prefetch_tmap(&tm_b);
        ptx::prefetch_tmap(&tm_d);
        ptx::prefetch_tmap(&tm_sfa);
        ptx::prefetch_tmap(&tm_sfb);
    }
    if (warp == 1) {
        ptx::tmem_alloc<2>(ptx::smem_u32(&bars->tmem_base), C::kTmemCols);
        ptx::tmem_relinquish<2>();
    }
    ptx::tc_fence_before();
    __syncthreads();
    // barriers of both CTAs are initialised before anyone signals across the pair
    ptx::cluster_sync();
    ptx::tc_fence_after();
    const uint32_t tmem = bars->tmem_base;

    // as in the single-CTA kernel (300 x 8192 x 8192 behind its quantizer 33.1 -> 32.7 us, 512 x 14336 x 4096
    // 32.3 -> 32.2, four rows of tiles and more: no change); this CTA's half of the columns
    if constexpr (!kGrouped) {
        if (threadIdx.x == 64 && prefetch_weight != 0 && cluster_id < tiles_m * tiles_n) {
            const TileCoord tc = tile_coord(cluster_id, tiles_m, tiles_n);
            const int end = min(k_tiles, 2560 / BN);
            for (int kt = (tc.m & 7); kt < end; kt += min(8, tiles_m)) {
                ptx::tma_prefetch_2d(&tm_b, kt * kBKBytes, tc.n * BN + int(rank) * (BN / 2));
            }
        }
        __syncwarp();
    }
    ptx::pdl_wait();
    RunTable run_table = {nullptr, 0};
    if constexpr (kGrouped) {
        if (ga.grp.kind == kGroupContiguous) {
            run_table = build_runs<256, C::kThreads>(ga.grp, ga.m, bars, reinterpret_cast<uint32_t*>(smem + bar_off + 1024));
        }
    }

    if (warp == 0) {
        // ------------------------------------------------------------ box loader (both CTAs)
        {
            uint32_t it = 0;
            bool ok = true;
            Iter walk(ga.grp, ga.m, ga.n, tiles_m, tiles_n, run_table, cluster_id, num_clusters);
            PairWork wk;
            while (ok && walk.next(wk)) {
                const int m0 = wk.a_row0 + int(rank) * kBM;
                const int n0 = wk.b_row0 + int(rank) * (BN / 2);
                for (int kt = 0; kt < k_tiles; ++kt, ++it) {
                    const uint32_t s = it % C::kStages;
                    ok = wait_bar(ptx::smem_u32(&bars->empty[s]), ((it / C::kStages) & 1u) ^ 1u, abort,
                                  kStatusProducer);
                    if (!ok) break;
                    const uint32_t full = ptx::mapa_cluster(ptx::smem_u32(&bars->full[s]), 0);
                    // The bytes of both loaders of the pair are counted on the leader's
                    // barrier; only its own registers them (the count may go negative in
                    // between).
                    if (leader && ptx::elect_one()) ptx::mbar_arrive_expect_tx(ptx::smem_u32(&bars->full[s]), 2 * C::kStageTxBytes);
                    if (ptx::elect_one()) ptx::tma_load_2d_pair(a_base + s * C::kABytes, &tm_a, kt * kBKBytes, m0, full);
                    if (ptx::elect_one()) ptx::tma_load_2d_pair(b_base + s * C::kBBytes, &tm_b, kt * kBKBytes, n0, full);
                }
            }
            ptx::pdl_launch_dependents();
            // The releases of the last stages, which no load waits for any more: commits that arrive in both CTAs, so
            // neither may leave before it has seen its own (the closing cluster_sync orders what threads did, not these).
            for (uint32_t d = it > uint32_t(C::kStages) ? it - C::kStages : 0u; ok && d < it; ++d) {
                ok = wait_bar(ptx::smem_u32(&bars->empty[d % C::kStages]), (d / C::kStages) & 1u, abort, kStatusProducer);
            }
        }
    } else if (warp == 6) {
        // ------------------------------------------------------------ scale loader (both CTAs)
        {
            uint32_t it = 0;
            bool ok = true;
            Iter walk(ga.grp, ga.m, ga.n, tiles_m, tiles_n, run_table, cluster_id, num_clusters);
            PairWork wk;
            while (ok && walk.next(wk)) {
                const int sfa_atom_row = (wk.a_row0 / 128 + int(rank)) * kq_dim;
                const int sfb_atom_row = wk.sfb_tile * kq_dim;
                for (int kt = 0; kt < k_tiles; ++kt, ++it) {
                    const uint32_t s = it % C::kStages;
                    ok = wait_bar(ptx::smem_u32(&bars->empty[s]), ((it / C::kStages) & 1u) ^ 1u, abort,
                                  kStatusProducer);
                    if (!ok) break;
                    const uint32_t sf_full = ptx::smem_u32(&bars->sf_full[s]);
                    if (ptx::elect_one()) ptx::mbar_arrive_expect_tx(sf_full, C::kSfaBytes + C::kSfbBytes);
                    // scale atoms are rows of 128 32-bit words (those beyond the weight arrive as zeros)
                    if (ptx::elect_one()) {
                        ptx::tma_load_2d(sfa_base + s * C::kSfaBytes, &tm_sfa, 0, sfa_atom_row + kt * C::kSfKAtoms, sf_full);
                    }
#pragma unroll
                    for (int j = 0; j < C::kNAtoms; ++j) {
                        if (ptx::elect_one()) {
                            ptx::tma_load_2d(sfb_base + s * C::kSfbBytes + j * C::kSfaBytes, &tm_sfb, 0,
                                             sfb_atom_row + j * kq_dim + kt * C::kSfKAtoms, sf_full);
                        }
                    }
                }
            }
        }
    } else if (warp >= 7 && warp < 7 + kSfWarps) {
        // ------------------------------------------------------------ scales -> tensor memory (both CTAs)
        // as in the single-CTA kernel: every warp fills its quarter of the lanes with the same image
        const uint32_t quarter = (uint32_t(warp) & 3u) * 32u;
        uint32_t it = 0;
        bool ok = true;
        Iter walk(ga.grp, ga.m, ga.n, tiles_m, tiles_n, run_table, cluster_id, num_clusters);
        PairWork wk;
        int left = walk.items();
        while (ok && (left >= 0 ? left-- > 0 : walk.next(wk))) {
            for (int kt = 0; kt < k_tiles; ++kt, ++it) {
                const uint32_t s = it % C::kStages;
                ok = wait_bar(ptx::smem_u32(&bars->sf_full[s]), (it / C::kStages) & 1u, abort, kStatusProducer);
                if (!ok) break;
                // into registers before the set is free, in the order of its columns
                uint32_t r[C::kSfCols];
                load_scales<C>(sfa_base + s * C::kSfaBytes, sfb_base + s * C::kSfbBytes, lane, r);
                if (it >= uint32_t(C::kSfSets)) {
                    // the MMAs of k-tile it - kSfSets read this set: they are done once they
                    // have released their stage
                    const uint32_t prev = it - uint32_t(C::kSfSets);
                    ok = wait_bar(ptx::smem_u32(&bars->empty[prev % C::kStages]), (prev / C::kStages) & 1u, abort,
                                  kStatusProducer);
                    if (!ok) break;
                }
                ptx::tc_fence_after();
                ptx::tc_store_32x32<C::kSfCols>(tmem + (quarter << 16) + C::kSfCol0 + (it % C::kSfSets) * C::kSfCols, r);
                ptx::tc_wait_st();
                ptx::tc_fence_before();
                __syncwarp();
                // (what it reports is in tensor memory, and complete)
                if (ptx::elect_one()) {
                    ptx::mbar_arrive_cluster_relaxed(ptx::mapa_cluster(ptx::smem_u32(&bars->sf_ready[it % C::kSfSets]), 0));
                }
            }
        }
    } else if (warp == 1 || warp == C::kMma2Warp) {
        // ------------------------------------------------------------ MMA issuers (leader only)
        if (leader) {
            const uint32_t me = warp == 1 ? 0u : 1u;  // this thread issues the k-iterations it & 1 == me
            uint32_t it = 0;
            uint32_t t = 0;
            bool ok = true;
            Iter walk(ga.grp, ga.m, ga.n, tiles_m, tiles_n, run_table, cluster_id, num_clusters);
            PairWork wk;
            int left = walk.items();
            for (; ok && (left >= 0 ? left-- > 0 : walk.next(wk)); ++t) {
                const uint32_t as = t & 1u;
                const uint32_t aph = (t >> 1) & 1u;
                const uint32_t acc = tmem + as * C::kAccStride;
                for (int kt = 0; kt < k_tiles; ++kt, ++it) {
                    if ((it & 1u) != me) {
                        if (k_tiles == 1) {
                            // A tile of one k-tile has nothing for this thread, but the accumulator's
                            // barrier expects both threads.  The arrival may not run ahead of the
                            // previous use of this accumulator stage, hence the same wait the
                            // issuing thread makes.
                            ok = wait_bar(ptx::smem_u32(&bars->acc_empty[as]), aph ^ 1u, abort, kStatusMma);
                            if (!ok) break;
                            const uint32_t accf = ptx::smem_u32(&bars->acc_full[as]);
                            if (ptx::elect_one()) {
                                ptx::mbar_arrive(accf);
                                ptx::mbar_arrive_cluster_relaxed(ptx::mapa_cluster(accf, 1));
                            }
                        }
                        continue;
                    }
                    const uint32_t s = it % C::kStages;
                    if (kt == 0) {
                        // first k-tile of a tile: the accumulator stage must have been drained
                        ok = wait_bar(ptx::smem_u32(&bars->acc_empty[as]), aph ^ 1u, abort, kStatusMma);
                        if (ok && C::kOverlap != 0 && t > 0) {
                            ok = wait_bar(ptx::smem_u32(&bars->overlap_free[as ^ 1u]), ((t - 1) >> 1) & 1u, abort,
                                          kStatusMma);
                        }
                        if (!ok) break;
                    }
                    // the scales of both CTAs are in tensor memory and the operand boxes of both have landed
                    ok = wait_bars(ptx::smem_u32(&bars->sf_ready[it % C::kSfSets]), (it / C::kSfSets) & 1u, true,
                                   ptx::smem_u32(&bars->full[s]), (it / C::kStages) & 1u, abort, kStatusMma);
                    // the other thread has issued the MMAs of the previous k-iteration
                    if (ok && it > 0u) {
                        ok = wait_bar(ptx::smem_u32(&bars->turn[me]), ((it - 1u) >> 1) & 1u, abort, kStatusMma);
                    }
                    if (!ok) break;
                    ptx::tc_fence_after();
                    const uint32_t set = tmem + C::kSfCol0 + (it % C::kSfSets) * C::kSfCols;
                    const uint64_t adesc = ptx::smem_desc(a_base + s * C::kABytes, 16, 1024, 2);
                    const uint64_t bdesc = ptx::smem_desc(b_base + s * C::kBBytes, 16, 1024, 2);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        uint32_t atom, sf_id;
                        if constexpr (KIND == 0 || KIND == 3) {
                            atom = 0;
                            sf_id = k;
                        } else if constexpr (KIND == 1) {
                            atom = k;
                            sf_id = 0;
                        } else {
                            atom = k >> 1;
                            sf_id = (k & 1) * 2;
                        }
                        if (ptx::elect_one()) {
                            ptx::tc_mma_block_scaled<2, KIND>(
                                acc, adesc + uint64_t(k * 2), bdesc + uint64_t(k * 2),
                                instr_desc_pair<BN, KIND>(sf_id), set + atom * 4,
                                set + C::kSfKAtoms * 4 + atom * C::kNAtoms * 4, (kt > 0 || k > 0) ? 1u : 0u);
                        }
                    }
                    // hand the turn over before the commits
                    ptx::tc_fence_before();
                    if (ptx::elect_one()) ptx::mbar_arrive(ptx::smem_u32(&bars->turn[me ^ 1u]));
                    // the loaders of both CTAs may refill stage s once these MMAs have read it
                    if (ptx::elect_one()) ptx::tc_commit_both(ptx::smem_u32(&bars->empty[s]));
                    // A commit tracks the operations of the thread that executes it, so each of
                    // the two threads commits the accumulator after its own last k-tile of the
                    // tile; the epilogue starts when both have completed.
                    if (kt >= k_tiles - 2) {
                        if (ptx::elect_one()) ptx::tc_commit_both(ptx::smem_u32(&bars->acc_full[as]));
                    }
                }
            }
        }
    } else if (warp < 6) {
        // ------------------------------------------------------------ epilogue (both CTAs)
        const int ew = warp - 2;
        const uint32_t lane_base = (warp & 3) * 32;
        uint32_t t = 0;
        uint32_t stores = 0;
        bool ok = true;
        float scale = 1.0f;
        int scale_group = -1;
        if constexpr (kSitu) zero_sf_padding(situ.p, (warp - 2) * 32 + lane);
        // The grouped kinds keep their place in shared memory: a dozen registers less through the loop over the chunks.  With
        // that and the item count of the other roles 32768 x 3072 x 1280 NVFP4 in one batch took 93 us instead of 99.
        static_assert(sizeof(Iter) * kEpiWarps <= 1024 - kKeptOffset, "behind the barriers");
        Iter* const kept = reinterpret_cast<Iter*>(smem + bar_off + kKeptOffset);
        Iter walk(ga.grp, ga.m, ga.n, tiles_m, tiles_n, run_table, cluster_id, num_clusters);
        if (kGrouped) {
            if (lane == 0) kept[ew] = walk;
            __syncwarp();
        }
        const auto next = [&](PairWork& w) {
            if constexpr (!kGrouped) return walk.next(w);
            Iter at = kept[ew];
            const bool more = at.next(w);
            __syncwarp();
            if (lane == 0) kept[ew] = at;
            __syncwarp();
            return more;
        };
        PairWork wk;
        for (; ok && next(wk); ++t) {
            const int m0 = wk.out_row0 + int(rank) * kBM;
            const int n0 = wk.out_col0;
            // rows of this CTA's half of the tile that belong to the item
            const int half_lo = min(max(wk.row_lo - int(rank) * kBM, 0), kBM);
            const int half_hi = min(max(wk.row_hi - int(rank) * kBM, 0), kBM);
            // Of a warp's 32 rows all, none or (masked) some are the item's.  (A dense tile that sticks out beyond M is clipped by the TMA store.)
            const bool partial = kGrouped && (int(lane_base) < half_lo || int(lane_base) + 32 > half_hi);
            // per-tensor (dense) or per-group factor of the NVFP4 recipe
            if (KIND == 1 && alpha != nullptr && wk.group != scale_group) {
                scale = __ldg(alpha + wk.group);
                scale_group = wk.group;
            }
            const uint32_t as = t & 1u;
            const uint32_t aph = (t >> 1) & 1u;
            ok = wait_bar(ptx::smem_u32(&bars->acc_full[as]), aph, abort, kStatusEpilogue);
            if (!ok) break;
            ptx::tc_fence_after();
            const uint32_t acc = tmem + as * C::kAccStride + (lane_base << 16);
            if constexpr (kSitu) {
                // 64 accumulator columns -> one group of 32 e4m3 outputs, as in the single-CTA kernel; the
                // group shared with the other accumulator stage comes first
                static_assert(KIND == 0 && !kGrouped && !kGather && C::kOverlapChunks <= 2, "dense MXFP8");
                constexpr int kGroups = C::kChunks / 2;
#pragma unroll 1
                for (int gi = 0; gi < kGroups; ++gi) {
                    const int g = (C::kOverlap != 0 && as == 0) ? kGroups - 1 - gi : gi;
                    uint32_t r0[32], r1[32];
                    ptx::tc_load_32x32(acc + (2 * g) * kEpiChunk, r0);
                    ptx::tc_load_32x32(acc + (2 * g + 1) * kEpiChunk, r1);
                    ptx::tc_wait_ld();
                    if (gi == 0 && C::kOverlap != 0) {
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            ptx::mbar_arrive_cluster_relaxed(ptx::mapa_cluster(ptx::smem_u32(&bars->overlap_free[as]), 0));
                        }
                    }
                    if (gi == kGroups - 1) {
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            ptx::mbar_arrive_cluster_relaxed(ptx::mapa_cluster(ptx::smem_u32(&bars->acc_empty[as]), 0));
                        }
                    }
                    uint32_t y[16];
                    const __nv_bfloat16* const bc = bias != nullptr ? bias + n0 + 2 * g * kEpiChunk : nullptr;
                    situ_chunk(r0, bc, situ.p, &y[0]);
                    situ_chunk(r1, bc != nullptr ? bc + kEpiChunk : nullptr, situ.p, &y[8]);
                    uint4 lo, hi;
                    const uint32_t e = quant32_bf16(y, lo, hi);
                    const int64_t row = m0 + int(lane_base) + lane;
                    if (row < ga.m) {
                        const int kb = (n0 >> 6) + g;  // group of 32 output columns
                        uint4* const dst = reinterpret_cast<uint4*>(situ.p.q + row * situ.p.ldq + int64_t(kb) * 32);
                        dst[0] = lo;
                        dst[1] = hi;
                        situ.p.sf[((row >> 7) * (situ.p.kb_out >> 2) + (kb >> 2)) * 512 + (row & 31) * 16 +
                                  ((row >> 5) & 3) * 4 + (kb & 3)] = uint8_t(e);
                    }
                }
                continue;
            }
            if constexpr (kGrouped) {
                if (partial) {
                    const int row = int(lane_base) + lane;
                    const bool row_ok = row >= half_lo && row < half_hi;
                    partial_rows<C>(acc, as != 0, row_ok ? ga.out + int64_t(m0 + row) * ga.ldo + n0 : nullptr, scale,
                                    bias != nullptr ? bias + wk.bias_col0 : nullptr, epi_op, wk.cols,
                                    ptx::mapa_cluster(ptx::smem_u32(&bars->overlap_free[as]), 0),
                                    ptx::mapa_cluster(ptx::smem_u32(&bars->acc_empty[as]), 0));
                    continue;
                }
            }
            // chunks shared with the other accumulator stage are read into registers first (as
            // in the single-CTA kernel), so that the next tile's MMAs may start early
            constexpr int kPre = C::kOverlapChunks > 1 ? C::kOverlapChunks : 0;
            uint32_t ro[kPre > 0 ? kPre : 1][32];
            if constexpr (kPre > 0) {
#pragma unroll
                for (int j = 0; j < kPre; ++j) {
                    const int c = as == 0 ? C::kChunks - 1 - j : j;
                    ptx::tc_load_32x32(acc + c * kEpiChunk, ro[j]);
                }
                ptx::tc_wait_ld();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive_cluster_relaxed(ptx::mapa_cluster(ptx::smem_u32(&bars->overlap_free[as]), 0));
                }
            }
#pragma unroll 1
            for (int ci = 0; ci < C::kChunks; ++ci) {
                const int c = (C::kOverlap != 0 && as == 0) ? C::kChunks - 1 - ci : ci;
                uint32_t r[32];
                if (kPre > 0 && ci < kPre) {
#pragma unroll
                    for (int j = 0; j < kPre; ++j) {
                        if (ci == j) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) r[i] = ro[j][i];
                        }
                    }
                } else {
                    ptx::tc_load_32x32(acc + c * kEpiChunk, r);
                    ptx::tc_wait_ld();
                }
                // The arrivals below tell the leader's MMA threads that tensor-memory reads have
                // completed (tcgen05.wait::ld); no shared or global data rides on them.
                if (C::kOverlap != 0 && kPre == 0 && ci == C::kOverlapChunks - 1) {
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        ptx::mbar_arrive_cluster_relaxed(ptx::mapa_cluster(ptx::smem_u32(&bars->overlap_free[as]), 0));
                    }
                }
                if (ci == C::kChunks - 1) {
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        ptx::mbar_arrive_cluster_relaxed(ptx::mapa_cluster(ptx::smem_u32(&bars->acc_empty[as]), 0));
                    }
                }
                if (c * kEpiChunk >= wk.cols) continue;
                uint32_t p[16];
                epilogue_chunk(r, p, scale, bias != nullptr ? bias + wk.bias_col0 + c * kEpiChunk : nullptr, epi_op);
                if constexpr (kGather) {
                    // Two neighbouring chunks are staged as ONE box of 32 rows x 128 bytes (the warp's
                    // two buffers, 128-byte swizzle) and stored together: rows of 128 bytes use
                    // NVLink better than rows of 64 (measured on 4 GPUs).  Chunks come in ascending
                    // or descending order, so chunk c's partner c ^ 1 is always the next or the previous one.
                    const uint32_t buf = epi_base + ew * C::kEpiBufs * kEpiBufBytes;
                    if ((ci & 1) == 0) {
                        if (lane == 0) ptx::bulk_wait_read<0>();
                        __syncwarp();
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t piece = uint32_t((c & 1) * 4 + j);
                        const uint32_t dst = buf + lane * 128 + ((piece ^ (lane & 7)) << 4);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(p[4 * j]),
                                     "r"(p[4 * j + 1]), "r"(p[4 * j + 2]), "r"(p[4 * j + 3])
                                     : "memory");
                    }
                    if ((ci & 1) != 0) {
                        ptx::fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            const int col = n0 + (c & ~1) * kEpiChunk;
                            ptx::tma_store_2d(&tm_d, buf, col, m0 + int(lane_base));
                            for (int q = 0; q < peers.count; ++q) {
                                ptx::tma_store_2d(&peers.out[q], buf, col, m0 + int(lane_base));
                            }
                            ptx::bulk_commit();
                        }
                    }
                    continue;
                }
                const uint32_t buf = epi_base + (ew * C::kEpiBufs + (stores % C::kEpiBufs)) * kEpiBufBytes;
                if (lane == 0) ptx::bulk_wait_read<C::kEpiBufs - 1>();
                __syncwarp();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t dst = buf + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4);
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(p[4 * j]),
                                 "r"(p[4 * j + 1]), "r"(p[4 * j + 2]), "r"(p[4 * j + 3])
                                 : "memory");
                }
                ptx::fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    ptx::tma_store_2d(&tm_d, buf, n0 + c * kEpiChunk, m0 + int(lane_base));
                    ptx::bulk_commit();
                }
                ++stores;
            }
        }
        if constexpr (kGather) {
            // the stores into the peers' memory have been performed, not only read from shared
            // memory, before the kernel is seen as complete
            if (lane == 0) {
                ptx::bulk_wait<0>();
                __threadfence_system();
            }
        } else {
            if (lane == 0) ptx::bulk_wait_read<0>();
        }
    }

    if (*abort != 0u) {
        for (int i = 0; i < 64; ++i) __nanosleep(1000);
    }
    ptx::tc_fence_before();
    __syncthreads();
    // neither CTA may leave while the other can still signal its barriers or while MMAs of the pair read its shared
    // memory: threads' arrivals are ordered by this barrier, the commits of both kinds have been waited for
    // (acc_full by the epilogue, empty by the loader)
    ptx::cluster_sync();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc<2>(tmem, C::kTmemCols);
    }
}

// ---------------------------------------------------------------------------- small M
#include "decode.cuh"

// ---------------------------------------------------------------------------- host

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            p = nullptr;
        }
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// rank-2 row-major tensor map: `inner` elements per row, `rows` rows, `pitch` bytes between rows
bool make_tmap_2d(CUtensorMap* map, CUtensorMapDataType dtype, const void* base, uint64_t inner,
                  uint64_t rows, uint64_t pitch, uint32_t box_inner, uint32_t box_rows,
                  CUtensorMapSwizzle swizzle) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[2] = {inner, rows};
    const cuuint64_t strides[1] = {pitch};
    const cuuint32_t box[2] = {box_inner, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, dtype, 2, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The same matrix cut into 128-byte k-tiles: [pitch / 128][rows][128 bytes], so that one copy brings
// `box_tiles` neighbouring k-tiles of `box_rows` rows, each in the 128-byte-swizzled form of its own
// (a box may stick out past the last k-tile, which then arrives as zeros).
bool make_tmap_ktiles(CUtensorMap* map, const void* base, uint64_t rows, uint64_t pitch, uint32_t box_rows,
                      uint32_t box_tiles) {
    EncodeTiledFn fn = encode_tiled_fn();
    if (fn == nullptr) return false;
    const cuuint64_t dims[3] = {uint64_t(kBKBytes), rows, pitch / kBKBytes};
    const cuuint64_t strides[2] = {pitch, uint64_t(kBKBytes)};
    const cuuint32_t box[3] = {uint32_t(kBKBytes), box_rows, box_tiles};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Per-device, once: the opt-in to more than 48 KB of dynamic shared memory for one kernel.
// A failed attempt is not remembered, so the next call tries (and reports) again.
struct SmemOptIn {
    std::mutex mu;
    bool done[64] = {};
    template <typename Kernel>
    cudaError_t ensure(Kernel kernel, int bytes, int* dev_out = nullptr) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        if (dev_out != nullptr) *dev_out = dev;
        std::lock_guard<std::mutex> lock(mu);
        if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e == cudaSuccess && dev >= 0 && dev < 64) done[dev] = true;
        return e;
    }
};

struct GemmArgs {
    const void* a;
    const void* b;
    const uint8_t* sfa;
    const uint8_t* sfb;
    const float* alpha;
    const __nv_bfloat16* bias;
    int epi_op;
    SituParams situ;
    __nv_bfloat16* out;
    int64_t ldo;
    int m, n;          // rows of A (all groups stacked) and columns per weight
    GroupParams grp;
    int64_t k_bytes;
    int kq_dim;
    int sm_count;
    bool pdl;
    bool runs = false;           // contiguous experts: tiles by runs (RunTable)
    bool early_weights = false;  // with pdl: b and sfb may be read before the preceding kernel completes
    bool direct_store;
    cudaStream_t stream;
};

// The environment switches (HALOPS_B200_*, for experiments and tests), read on every call: entry points that lead to one
// of them begin with a SwitchScope.  It asks getenv, which a thread that changes the environment meanwhile is kept from
// by nothing but the C library; a caller that has a lock for that reads them under it (hq_hold_switches), in one walk over
// the environment, and the calls that follow on its thread take that reading.  (Five getenv are 0.5 us among 135 variables.)
struct Switches {
    char tile[16] = "", splitk[8] = "", issuers[8] = "", decode[64] = "", epilogue[16] = "", runs[8] = "";

    template <typename F>
    void each(F&& f) {
        f("HALOPS_B200_TILE", tile, sizeof(tile));
        f("HALOPS_B200_SPLITK", splitk, sizeof(splitk));
        f("HALOPS_B200_ISSUERS", issuers, sizeof(issuers));
        f("HALOPS_B200_DECODE", decode, sizeof(decode));
        f("HALOPS_B200_EPILOGUE", epilogue, sizeof(epilogue));
        f("HALOPS_B200_RUNS", runs, sizeof(runs));
    }
    void clear() {
        each([](const char*, char* to, size_t) { to[0] = '\0'; });
    }
    void ask() {
        each([](const char* name, char* to, size_t size) {
            const char* const v = getenv(name);
            to[0] = '\0';
            if (v != nullptr) snprintf(to, size, "%s", v);
        });
    }
    void walk() {
        clear();
        for (char** e = environ; e != nullptr && *e != nullptr; ++e) {
            if ((*e)[0] != 'H' || strncmp(*e, "HALOPS_B200_", 12) != 0) continue;
            each([v = *e](const char* name, char* to, size_t size) {
                const size_t len = strlen(name);
                if (to[0] == '\0' && strncmp(v, name, len) == 0 && v[len] == '=') snprintf(to, size, "%s", v + len + 1);
            });
        }
    }
};
thread_local Switches t_switches;
thread_local bool t_switches_held = false;

struct SwitchScope {
    SwitchScope() {
        if (!t_switches_held) t_switches.ask();
    }
};

// Split-K is taken for a dense problem with one row of 64-wide tiles and a long K: at least 56 k-tiles where its two CTAs per tile
// fill at most half of the SMs, 96 where they fill more (a tile's weights then come no faster to two CTAs than to one).
// HALOPS_B200_SPLITK=0 turns it off; read on every call.  The cluster and its exchange cost 3.5 us; N = 704 (11 tiles) takes
// 9.6 us split and 9.2 whole at 48 k-tiles, 10.2 and 10.4 at 56, 13.2 and 16.1 at 96; N = 3712 13.9 and 13.1 at 64, 17.1 and 17.9
// at 96 (112 problems of 66 and 128 rows).  With the 64-wide tile forced, from 8 k-tiles on.
bool split_k_chosen(int group_kind, int tiles_m, int tiles_n, int k_tiles, int sm_count, int epi_op) {
    if (t_switches.splitk[0] == '0') return false;
    const int least = strcmp(t_switches.tile, "64") == 0 ? 8 : 4 * tiles_n <= sm_count ? 56 : 96;
    return group_kind == kGroupDense && tiles_m == 1 && 2 * tiles_n <= sm_count && k_tiles >= least &&
           (epi_op == HQ_EPILOGUE_IDENTITY || epi_op == HQ_EPILOGUE_SIGMOID);
}

// 2: the single-CTA kernel issues its MMAs from two threads in k order (see the kernel);
// 0 with HALOPS_B200_ISSUERS=1 (read on every call)
int issuers_in_order() {
    return t_switches.issuers[0] == '1' ? 0 : 2;
}

// (group, 128-row tile) pairs of `count` groups of `rows` rows each; a tile that straddles groups counts once per group.
int64_t slot_row_tiles(int64_t count, int64_t rows) {
    const auto tiles = [rows](int64_t g) { return ((g + 1) * rows - 1) / kBM - g * rows / kBM + 1; };
    int64_t period = 1;  // groups after which the starts in their tiles come again
    while (period < kBM && period * rows % kBM != 0) period *= 2;
    int64_t each = 0, total = 0;
    for (int64_t g = 0; g < std::min(period, count); ++g) each += tiles(g);
    total = count / period * each;
    for (int64_t g = count / period * period; g < count; ++g) total += tiles(g);
    return total;
}

template <int BN, int KIND>
int launch_tile(const GemmArgs& g, char* err, size_t errlen) {
    using C = Cfg<BN, KIND>;
    static SmemOptIn opt_in;
    HQ_CUDA_TRY(opt_in.ensure(gemm_kernel<BN, KIND>, C::kSmemBytes));

    CUtensorMap tm_a, tm_b, tm_d;
    // M < 128: the A box holds only the rows that exist (rounded up to the 8-row
    // swizzle period); the other rows of the shared-memory tile keep stale bytes,
    // which only feed accumulator rows that are never stored
    const int64_t rows_a = g.m;
    const int64_t rows_b = int64_t(g.grp.kind == kGroupDense ? 1 : g.grp.count) * g.n;
    // output: [rows, count * N] for batches, else [M, N]
    const int64_t out_rows = g.grp.kind == kGroupBatch ? g.grp.rows : g.m;
    const int64_t out_cols = g.grp.kind == kGroupBatch ? rows_b : g.n;
    const int a_rows = rows_a >= kBM ? kBM : int((rows_a + 7) / 8 * 8);
    const bool maps_ok =
        make_tmap_2d(&tm_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, g.a, uint64_t(g.k_bytes), uint64_t(rows_a),
                     uint64_t(g.k_bytes), kBKBytes, uint32_t(a_rows), CU_TENSOR_MAP_SWIZZLE_128B) &&
        // KIND 3: packed e2m1 weights; the copy spreads every 16 values (8 bytes) over 16 bytes
        // of shared memory, the form the mxf8f6f4 MMA reads 4-bit operands in, so a box of
        // 128 values per row fills the same 128 bytes as 128 e4m3 values
        (KIND == 3 ? make_tmap_2d(&tm_b, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, g.b, uint64_t(g.k_bytes),
                                  uint64_t(rows_b), uint64_t(g.k_bytes / 2), kBKBytes, BN,
                                  CU_TENSOR_MAP_SWIZZLE_128B)
                   : make_tmap_2d(&tm_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, g.b, uint64_t(g.k_bytes), uint64_t(rows_b),
                                  uint64_t(g.k_bytes), kBKBytes, BN, CU_TENSOR_MAP_SWIZZLE_128B)) &&
        // (the quantising epilogue stores from registers; its map only has to be valid)
        make_tmap_2d(&tm_d, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, g.out,
                     uint64_t(g.epi_op == HQ_EPILOGUE_SITU_QUANT ? g.n / 4
                              : (g.epi_op == HQ_EPILOGUE_IDENTITY || g.epi_op == HQ_EPILOGUE_SIGMOID) ? out_cols
                                                                                                       : out_cols / 2),
                     uint64_t(out_rows),
                     uint64_t(g.ldo) * 2, kEpiChunk, 32, CU_TENSOR_MAP_SWIZZLE_64B);
    if (!maps_ok) {
        return fail(err, errlen, HQ_ERR_CUDA, "cuTensorMapEncodeTiled failed for the GEMM operands");
    }
    int tiles_m = (g.m + kBM - 1) / kBM;
    if (g.grp.kind == kGroupBatch || g.grp.kind == kGroupMasked) {
        // (group, 128-row tile) pairs; a straddling tile counts once per group.  For the
        // masked kind this is the upper bound that sizes the grid: the kernel walks the
        // valid rows only.
        tiles_m = int(slot_row_tiles(g.grp.count, g.grp.rows));
    }
    const int tiles_n = (g.n + BN - 1) / BN;
    // runs are cut into at most a tile each more than the rows alone
    const int64_t row_tiles = g.runs ? std::min<int64_t>(g.m / 64, int64_t(tiles_m) + g.grp.count) : tiles_m;
    const int grid = int(std::min<int64_t>(g.sm_count, row_tiles * tiles_n));
    const int k_tiles = int(g.k_bytes / kBKBytes);
    if constexpr (BN == 64 && KIND != 3) {  // (the e4m3 x e2m1 kind is a grouped one)
        // One row of at most sm_count / 2 tiles and a long K: two CTAs per tile, half of K each.
        if (split_k_chosen(g.grp.kind, tiles_m, tiles_n, k_tiles, g.sm_count, g.epi_op)) {
            static SmemOptIn opt_in_split;
            HQ_CUDA_TRY(opt_in_split.ensure(gemm_kernel<BN, KIND, true>, C::kSmemBytes));
            HQ_CUDA_TRY(launch(gemm_kernel<BN, KIND, true>, dim3(2 * tiles_n), dim3(kThreads), size_t(C::kSmemBytes),
                               g.stream, g.pdl, 2, tm_a, tm_b, tm_d, g.sfa, g.sfb, g.alpha, g.bias, g.epi_op, g.out,
                               g.ldo, g.m, g.n, k_tiles, g.kq_dim, tiles_m, tiles_n, a_rows,
                               g.direct_store ? 1 : 0, issuers_in_order(), g.pdl ? 1 : 0, g.grp, g.situ));
            return HQ_OK;
        }
    }
    // One row of 64-wide dense tiles with a plain epilogue (65 to 128 activation rows, or fewer
    // when the small-M kernel is not taken): two MMA issuers with an accumulator each (see the
    // kernel).  Problems with several rows of tiles never take that mode, so that every tile
    // shape sums the k-tiles of an output element in the same order and gives the same bits.
    int dual = BN == 64 && g.grp.kind == kGroupDense && tiles_m == 1 && k_tiles >= 2 &&
                       (g.epi_op == HQ_EPILOGUE_IDENTITY || g.epi_op == HQ_EPILOGUE_SIGMOID)
                   ? 1
                   : 0;
    // Everything else: two issuers in k order (same bits as one issuer; the dense and the
    // grouped kinds alike).  HALOPS_B200_ISSUERS=1 keeps one issuer (read on every call).
    if (dual == 0 && k_tiles >= 2) dual = issuers_in_order();
    if constexpr (KIND != 3) {
        if (g.grp.kind == kGroupDense && (g.epi_op == HQ_EPILOGUE_IDENTITY || g.epi_op == HQ_EPILOGUE_SIGMOID)) {
            static SmemOptIn opt_in_dense;
            HQ_CUDA_TRY(opt_in_dense.ensure(gemm_kernel<BN, KIND, false, true>, C::kSmemBytes));
            HQ_CUDA_TRY(launch(gemm_kernel<BN, KIND, false, true>, dim3(grid), dim3(kThreads), size_t(C::kSmemBytes), g.stream,
                               g.pdl, 1, tm_a, tm_b, tm_d, g.sfa, g.sfb, g.alpha, g.bias, g.epi_op, g.out, g.ldo, g.m, g.n, k_tiles,
                               g.kq_dim, tiles_m, tiles_n, a_rows, g.direct_store ? 1 : 0, dual, g.pdl ? 1 : 0, g.grp, g.situ));
            return HQ_OK;
        }
    }
    if (g.runs) {
        static SmemOptIn opt_in_runs;
        HQ_CUDA_TRY(opt_in_runs.ensure(gemm_kernel<BN, KIND, false, false, true>, C::kSmemBytes));
        HQ_CUDA_TRY(launch(gemm_kernel<BN, KIND, false, false, true>, dim3(grid), dim3(kThreads), size_t(C::kSmemBytes), g.stream,
                           g.pdl, 1, tm_a, tm_b, tm_d, g.sfa, g.sfb, g.alpha, g.bias, g.epi_op, g.out, g.ldo, g.m, g.n, k_tiles,
                           g.kq_dim, tiles_m, tiles_n, a_rows, g.direct_store ? 1 : 0, dual, g.pdl ? 1 : 0, g.grp, g.situ));
        return HQ_OK;
    }
    HQ_CUDA_TRY(launch(gemm_kernel<BN, KIND>, dim3(grid), dim3(kThreads), size_t(C::kSmemBytes), g.stream,
                       g.pdl, 1, tm_a, tm_b, tm_d, g.sfa, g.sfb, g.alpha, g.bias, g.epi_op, g.out, g.ldo, g.m, g.n, k_tiles,
                       g.kq_dim, tiles_m, tiles_n, a_rows, g.direct_store ? 1 : 0, dual, g.pdl ? 1 : 0, g.grp, g.situ));
    return HQ_OK;
}

template <int BN, int KIND, bool kGather = false, bool kGrouped = false, bool kSitu = false>
int launch_pair(const GemmArgs& g, char* err, size_t errlen, __nv_bfloat16* const* gather = nullptr,
                int gather_count = 0) {
    using C = Cfg2<BN, KIND>;
    static SmemOptIn opt_in;
    int dev = 0;
    HQ_CUDA_TRY(opt_in.ensure(gemm_pair_kernel<BN, KIND, kGather, kGrouped, kSitu>, C::kSmemBytes, &dev));
    // the grouped kinds: weights (and their scales) of all groups are stacked; a batch writes
    // [rows, count * N]
    const int64_t weights = kGrouped ? g.grp.count : 1;
    const int64_t out_rows = kGrouped && g.grp.kind == kGroupBatch ? g.grp.rows : g.m;
    const int64_t out_cols = kGrouped && g.grp.kind == kGroupBatch ? weights * g.n : g.n;

    const uint64_t atoms_a = uint64_t((g.m + 127) / 128) * uint64_t(g.kq_dim);
    const uint64_t atoms_b = uint64_t(weights) * uint64_t((g.n + 127) / 128) * uint64_t(g.kq_dim);
    CUtensorMap tm_a, tm_b, tm_d, tm_sfa, tm_sfb;
    const bool maps_ok =
        make_tmap_2d(&tm_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, g.a, uint64_t(g.k_bytes), uint64_t(g.m),
                     uint64_t(g.k_bytes), kBKBytes, kBM, CU_TENSOR_MAP_SWIZZLE_128B) &&
        // (KIND 3: packed e2m1 weights, spread to one byte per value by the copy; see launch_tile)
        (KIND == 3 ? make_tmap_2d(&tm_b, CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B, g.b, uint64_t(g.k_bytes),
                                  uint64_t(weights * g.n), uint64_t(g.k_bytes / 2), kBKBytes, BN / 2,
                                  CU_TENSOR_MAP_SWIZZLE_128B)
                   : make_tmap_2d(&tm_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, g.b, uint64_t(g.k_bytes),
                                  uint64_t(weights * g.n), uint64_t(g.k_bytes), kBKBytes, BN / 2,
                                  CU_TENSOR_MAP_SWIZZLE_128B)) &&
        // (the gathering kernel stores boxes of two chunks, see its epilogue)
        // (the quantising epilogue stores from registers; its map only has to be valid)
        make_tmap_2d(&tm_d, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, g.out, uint64_t(kSitu ? g.n / 4 : out_cols), uint64_t(out_rows),
                     uint64_t(g.ldo) * 2, kGather ? 2 * kEpiChunk : kEpiChunk, 32,
                     kGather ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B) &&
        // scale atoms as rows of 128 32-bit words
        make_tmap_2d(&tm_sfa, CU_TENSOR_MAP_DATA_TYPE_UINT32, g.sfa, 128, atoms_a, 512, 128, C::kSfKAtoms,
                     CU_TENSOR_MAP_SWIZZLE_NONE) &&
        make_tmap_2d(&tm_sfb, CU_TENSOR_MAP_DATA_TYPE_UINT32, g.sfb, 128, atoms_b, 512, 128, C::kSfKAtoms,
                     CU_TENSOR_MAP_SWIZZLE_NONE);
    if (!maps_ok) {
        return fail(err, errlen, HQ_ERR_CUDA, "cuTensorMapEncodeTiled failed for the GEMM operands");
    }
    const int tiles_m = (g.m + 255) / 256;
    const int tiles_n = (g.n + BN - 1) / BN;
    // persistent grid: no more clusters than can be resident at once
    static int max_clusters[64];
    static std::mutex max_clusters_mutex;
    std::lock_guard<std::mutex> max_clusters_lock(max_clusters_mutex);
    const int slot = dev >= 0 && dev < 64 ? dev : 63;
    if (max_clusters[slot] == 0 || dev != slot) {
        cudaLaunchConfig_t occ = {};
        occ.gridDim = dim3(2 * 74);
        occ.blockDim = dim3(C::kThreads);
        occ.dynamicSmemBytes = size_t(C::kSmemBytes);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = 2;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        occ.attrs = at;
        occ.numAttrs = 1;
        int n = 0;
        HQ_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<BN, KIND, kGather, kGrouped, kSitu>, &occ));
        max_clusters[slot] = n > 0 ? n : 1;
    }
    const int64_t row_tiles = kGrouped && g.grp.kind == kGroupContiguous ? std::min<int64_t>(g.m / 64, int64_t(tiles_m) + g.grp.count) : tiles_m;
    const int clusters = int(std::min<int64_t>(min(g.sm_count / 2, max_clusters[slot]), row_tiles * tiles_n));
    const int k_tiles = int(g.k_bytes / kBKBytes);
    GatherMaps<kGather> peers{};
    if constexpr (kGather) {
        for (int q = 0; q < gather_count; ++q) {
            if (!make_tmap_2d(&peers.out[q], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, gather[q], uint64_t(g.n), uint64_t(g.m),
                              uint64_t(g.ldo) * 2, 2 * kEpiChunk, 32, CU_TENSOR_MAP_SWIZZLE_128B)) {
                return fail(err, errlen, HQ_ERR_CUDA, "cuTensorMapEncodeTiled failed for the output of a peer");
            }
        }
        peers.count = gather_count;
    }
    const PairGroupArgs ga{kGrouped ? g.grp : GroupParams{kGroupDense, 1, 0, nullptr}, g.out, g.ldo, g.m, g.n};
    PairSitu<kSitu> situ{};
    if constexpr (kSitu) situ.p = g.situ;
    HQ_CUDA_TRY(launch(gemm_pair_kernel<BN, KIND, kGather, kGrouped, kSitu>, dim3(2 * clusters), dim3(C::kThreads),
                       size_t(C::kSmemBytes), g.stream, g.pdl, 2, tm_a, tm_b, tm_d, tm_sfa, tm_sfb, g.alpha, g.bias,
                       g.epi_op, k_tiles, g.kq_dim, tiles_m, tiles_n, g.pdl ? 1 : 0, peers, ga, situ));
    return HQ_OK;
}

// Switches of the small-M kernel, for experiments and tests (HALOPS_B200_DECODE, a comma-separated
// list read on every call): "off" sends small M to the 128 x 64 tile instead, "nosplit" keeps
// every CTA on whole tiles, "split" deals every tile to several CTAs whatever the estimate says,
// "wide" also takes 65 to 128 activation rows, "nocluster" exchanges partial tiles through the
// global scratch buffer also where a cluster could do it through shared memory.
struct DecodeSwitches {
    bool off = false, nosplit = false, split = false, wide = false, nocluster = false;
};
DecodeSwitches decode_switches() {
    DecodeSwitches d;
    const char* const e = t_switches.decode;
    if (e[0] == '\0') return d;
    d.off = strstr(e, "off") != nullptr;
    d.nosplit = strstr(e, "nosplit") != nullptr;
    d.split = !d.nosplit && strstr(e, "split") != nullptr;
    d.wide = strstr(e, "wide") != nullptr;
    d.nocluster = strstr(e, "nocluster") != nullptr;
    return d;
}

// Small M goes to the operand-swapped kernel: dense MXFP8 without bias, plain or sigmoid
// epilogue, no forced tile.
bool decode_eligible(int64_t m, int64_t n, int64_t k, int mode, int epi_op, bool has_bias) {
    if (t_switches.tile[0] != '\0') return false;
    if ((n / 128 + 1) * (k / 256 + 1) >= (int64_t(1) << 31)) return false;
    // Up to 64 activation rows by default.  With 65 to 128 a stage is half activations, the
    // weight in flight per CTA halves, and the best 128-row tile was faster on each of 33 problems (128 x 8192 x 4096
    // behind its quantizer 15.5 against 12.8 us on the 128 x 64 tile, 96 x 24576 x 1536 14.9 against 12.5 on the
    // 128 x 128 one); HALOPS_B200_DECODE=wide sends them here all the same.
    const DecodeSwitches sw = decode_switches();
    const int64_t m_max = sw.wide ? 128 : 64;
    return mode == HQ_MODE_W8A8_MXFP8 && m >= 1 && m <= m_max && n % 64 == 0 && k % 128 == 0 && !has_bias &&
           (epi_op == HQ_EPILOGUE_IDENTITY || epi_op == HQ_EPILOGUE_SIGMOID) && !sw.off;
}

int decode_width(int64_t m) { return m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 ? 64 : 128; }

// bytes of the operand ring of gemm_decode_kernel<NACT, *>: where a cluster's partial tiles land
int64_t decode_ring_bytes(int nact) {
    switch (nact) {
        case 16:
            return int64_t(DecCfg<16>::kStages) * DecCfg<16>::kWBytes;
        case 32:
            return int64_t(DecCfg<32>::kStages) * DecCfg<32>::kWBytes;
        case 64:
            return int64_t(DecCfg<64>::kStages) * DecCfg<64>::kWBytes;
        default:
            return int64_t(DecCfg<128>::kStages) * DecCfg<128>::kWBytes;
    }
}

// How many clusters of 2, 4 and 8 CTAs of gemm_decode_kernel<NACT, *> the current device can hold at
// once; asked once per device and width.  Without a device (shape queries on a machine without
// a GPU) the figures of a B200 stand in: 74, 36 and 14.
template <int NACT>
void decode_cluster_query(DecClusterLimits* out) {
    for (int sc = 2; sc <= 8; sc *= 2) {
        cudaLaunchConfig_t occ = {};
        occ.gridDim = dim3(unsigned(sc));
        occ.blockDim = dim3(kDecThreads);
        occ.dynamicSmemBytes = size_t(DecCfg<NACT>::kSmemBytes);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = unsigned(sc);
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        occ.attrs = at;
        occ.numAttrs = 1;
        int n = 0;
        if (cudaFuncSetAttribute(gemm_decode_kernel<NACT, kDealCluster>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 DecCfg<NACT>::kSmemBytes) != cudaSuccess ||
            cudaOccupancyMaxActiveClusters(&n, gemm_decode_kernel<NACT, kDealCluster>, &occ) != cudaSuccess) {
            cudaGetLastError();
            n = sc == 2 ? 74 : sc == 4 ? 36 : 14;
        }
        out->max_active[sc] = n;
    }
}

const DecClusterLimits* decode_cluster_limits(int nact) {
    static std::mutex mu;
    static DecClusterLimits limits[64][4];
    static bool known[64][4];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        dev = 63;
    }
    const int slot = dev >= 0 && dev < 64 ? dev : 63;
    const int w = nact == 16 ? 0 : nact == 32 ? 1 : nact == 64 ? 2 : 3;
    std::lock_guard<std::mutex> lock(mu);
    if (!known[slot][w]) {
        switch (nact) {
            case 16:
                decode_cluster_query<16>(&limits[slot][w]);
                break;
            case 32:
                decode_cluster_query<32>(&limits[slot][w]);
                break;
            case 64:
                decode_cluster_query<64>(&limits[slot][w]);
                break;
            default:
                decode_cluster_query<128>(&limits[slot][w]);
        }
        known[slot][w] = true;
    }
    return &limits[slot][w];
}

DecPlan decode_plan(int64_t m, int64_t n, int64_t k_bytes, int sm_count) {
    const DecodeSwitches sw = decode_switches();
    const int nact = decode_width(m);
    return dec_plan(int(n), k_bytes, sm_count, !sw.nosplit, nact, sw.split, decode_ring_bytes(nact),
                    sw.nocluster ? nullptr : decode_cluster_limits(nact));
}

// Launches the instantiation of the plan's deal.
template <int NACT>
int launch_decode_deal(const DecPlan& plan, const GemmArgs& g, const CUtensorMap& tm_w, const CUtensorMap& tm_x,
                       const CUtensorMap& tm_o, const DecParams& p, char* err, size_t errlen) {
    constexpr int kSmem = DecCfg<NACT>::kSmemBytes;
    const auto run = [&](auto kernel, unsigned cluster) {
        return launch(kernel, dim3(plan.ctas), dim3(kDecThreads), size_t(kSmem), g.stream, g.pdl, cluster, tm_w, tm_x, tm_o, p,
                      DecPlain<false>{});
    };
    if (plan.aligned) {  // (the caller has opted in)
        HQ_CUDA_TRY(run(gemm_decode_kernel<NACT, kDealWhole>, 1u));
    } else if (plan.cluster > 1) {
        static SmemOptIn opt_in;
        HQ_CUDA_TRY(opt_in.ensure(gemm_decode_kernel<NACT, kDealCluster>, kSmem));
        HQ_CUDA_TRY(run(gemm_decode_kernel<NACT, kDealCluster>, unsigned(plan.cluster)));
    } else {
        static SmemOptIn opt_in;
        HQ_CUDA_TRY(opt_in.ensure(gemm_decode_kernel<NACT, kDealScratch>, kSmem));
        HQ_CUDA_TRY(run(gemm_decode_kernel<NACT, kDealScratch>, 1u));
    }
    return HQ_OK;
}

template <int NACT>
int launch_decode(const GemmArgs& g, char* err, size_t errlen) {
    using C = DecCfg<NACT>;
    static SmemOptIn opt_in;
    int dev = 0;
    HQ_CUDA_TRY(opt_in.ensure(gemm_decode_kernel<NACT, kDealWhole>, C::kSmemBytes, &dev));
    DecParams p;
    p.plan = decode_plan(g.m, g.n, g.k_bytes, g.sm_count);
    DecScratch scratch;
    if (!p.plan.aligned && p.plan.cluster <= 1 && !dec_scratch(dev, g.stream, &scratch)) {
        // no scratch buffer to be had: whole tiles per CTA need none
        p.plan.ctas = p.plan.tiles < g.sm_count ? p.plan.tiles : g.sm_count;
        p.plan.aligned = 1;
        p.plan.fits32 = 0;
    }
    const int x_rows = int((g.m + 7) / 8 * 8);
    CUtensorMap tm_w, tm_x, tm_o;
    const bool maps_ok =
        make_tmap_ktiles(&tm_w, g.b, uint64_t(g.n), uint64_t(g.k_bytes), kDecRows, 2) &&
        make_tmap_ktiles(&tm_x, g.a, uint64_t(g.m), uint64_t(g.k_bytes), uint32_t(x_rows), 2) &&
        // the epilogue stores [16 rows x 32 columns] boxes; rows past M and columns past N are clipped
        make_tmap_2d(&tm_o, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, g.out, uint64_t(g.n), uint64_t(g.m),
                     uint64_t(g.ldo) * 2, 32, 16, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (!maps_ok) {
        return fail(err, errlen, HQ_ERR_CUDA, "cuTensorMapEncodeTiled failed for the GEMM operands");
    }
    p.sfw = g.sfb;
    p.early_weights = g.pdl && g.early_weights ? 1 : 0;
    // (without a programmatic launch there is nothing to overlap; with early weights the loads are the prefetch)
    p.prefetch_steps = g.pdl && !g.early_weights ? dec_prefetch_steps(p.plan, C::kWBytes) : 0;
    p.sfx = g.sfa;
    p.scratch = scratch.partials;
    p.counters = scratch.counters;
    p.m = g.m;
    p.n = g.n;
    p.k_bytes = g.k_bytes;
    p.kq_dim = g.kq_dim;
    p.x_rows = x_rows;
    p.epi_op = g.epi_op;
    return launch_decode_deal<NACT>(p.plan, g, tm_w, tm_x, tm_o, p, err, errlen);
}

// ---------------------------------------------------------------------------- small M without any allocation
//
// hq_dense_gemm_small_m_noalloc is for callers that cannot let a library allocate device
// memory behind their back: code that runs between the begin and end of a stream capture (a
// cudaMalloc there fails the capture), serving loops that hand all of the GPU's memory to
// their own pool at start-up and treat a later cudaMalloc as a bug, and real-time paths that
// must not take the allocator's locks.  The small-M kernel needs scratch memory when it deals
// one tile of the weight to several CTAs (float32 partial tiles and one counter per tile);
// hq_dense_gemm gets it from cudaMalloc on first use.  This variant keeps it in the array
// below, which is part of the library's image: every GPU that loads the library holds these
// bytes until the process ends, whether the entry point is called or not.
//
// Limits that keep the array modest: at most kNoAllocMaxM activation rows (32-column
// accumulators, 16 KB per partial tile), at most kNoAllocMaxCtas CTAs with two partial tiles
// each, at most kNoAllocMaxTiles weight tiles of 128 rows.
constexpr int kNoAllocMaxM = 32;
constexpr int kNoAllocMaxCtas = 160;
constexpr int kNoAllocMaxTiles = 4096;
constexpr size_t kNoAllocPartialFloats = size_t(kNoAllocMaxCtas) * 2 * 32 * kDecRows;  // 5 MiB of float32
constexpr size_t kNoAllocBytes = kNoAllocPartialFloats * sizeof(float) + size_t(kNoAllocMaxTiles) * sizeof(int);

// In host code this name is only a handle for the runtime's symbol calls; the device address
// comes from cudaGetSymbolAddress (see noalloc_scratch below).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

// Device address of the array on the current device, looked up once per device.  The
// look-up may initialise the module on that device, so the first call on a device should
// come before any stream capture.
cudaError_t noalloc_scratch(int dev, DecScratch* out) {
    static std::mutex mu;
    static unsigned char* addr[64];
    std::lock_guard<std::mutex> lock(mu);
    unsigned char* base = dev >= 0 && dev < 64 ? addr[dev] : nullptr;
    if (base == nullptr) {
        const cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void**>(&base), g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        if (dev >= 0 && dev < 64) addr[dev] = base;
    }
    out->partials = reinterpret_cast<float*>(base);
    out->counters = reinterpret_cast<int*>(base + kNoAllocPartialFloats * sizeof(float));
    return cudaSuccess;
}

template <int NACT>
int launch_decode_noalloc(const GemmArgs& g, const DecPlan& plan, char* err, size_t errlen) {
    using C = DecCfg<NACT>;
    static SmemOptIn opt_in;
    int dev = 0;
    HQ_CUDA_TRY(opt_in.ensure(gemm_decode_kernel<NACT, kDealWhole>, C::kSmemBytes, &dev));
    DecScratch scratch;
    HQ_CUDA_TRY(noalloc_scratch(dev, &scratch));
    DecParams p;
    p.plan = plan;
    if (!plan.aligned) {
        // The array keeps what the last call left in it.  The partial tiles are written before
        // they are read; the tile counters must start at zero, and a call that was cut short
        // may have left some counted: clear the ones this launch uses, in stream order.
        HQ_CUDA_TRY(cudaMemsetAsync(scratch.counters, 0, size_t(plan.tiles) * sizeof(int), g.stream));
    }
    const int x_rows = int((g.m + 7) / 8 * 8);
    CUtensorMap tm_w, tm_x, tm_o;
    const bool maps_ok =
        make_tmap_ktiles(&tm_w, g.b, uint64_t(g.n), uint64_t(g.k_bytes), kDecRows, 2) &&
        make_tmap_ktiles(&tm_x, g.a, uint64_t(g.m), uint64_t(g.k_bytes), uint32_t(x_rows), 2) &&
        make_tmap_2d(&tm_o, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, g.out, uint64_t(g.n), uint64_t(g.m),
                     uint64_t(g.ldo) * 2, 32, 16, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (!maps_ok) {
        return fail(err, errlen, HQ_ERR_CUDA, "cuTensorMapEncodeTiled failed for the GEMM operands");
    }
    p.sfw = g.sfb;
    p.early_weights = g.pdl && g.early_weights ? 1 : 0;
    // (without a programmatic launch there is nothing to overlap; with early weights the loads are the prefetch)
    p.prefetch_steps = g.pdl && !g.early_weights ? dec_prefetch_steps(p.plan, C::kWBytes) : 0;
    p.sfx = g.sfa;
    p.scratch = scratch.partials;
    p.counters = scratch.counters;
    p.m = g.m;
    p.n = g.n;
    p.k_bytes = g.k_bytes;
    p.kq_dim = g.kq_dim;
    p.x_rows = x_rows;
    p.epi_op = g.epi_op;
    return launch_decode_deal<NACT>(plan, g, tm_w, tm_x, tm_o, p, err, errlen);
}

const char* mode_name(int mode) {
    switch (mode) {
        case HQ_MODE_W8A8_MXFP8:
            return "w8a8-mxfp8";
        case HQ_MODE_W4A4_MXFP4:
            return "w4a4-mxfp4";
        case HQ_MODE_W4A8_MXFP4:
            return "w4a8-mxfp4";
        default:
            return "w4a4-nvfp4";
    }
}

struct TilePick {
    int bn;     // tile width, 0 = no tile fits
    bool pair;  // 256-row tile on a pair of CTAs
    bool runs = false;  // contiguous experts: tiles by their runs
};

// Shape legality follows the reference's "some compiled tile fits" rule
// (csrc/kernel/gemm/gemm_dispatch.cuh:65-100 over the tiles of gemm_tile.cuh:371-395):
// MXFP8 needs K % 128 == 0 and N % 64 == 0, the FP4 modes K % 256 == 0 and
// N % 128 == 0; any M >= 1.  A tile may stick out beyond N (the copies fill its rows beyond the weight with
// zeros, the epilogue skips its columns), so every width is open to every N: when a width had to divide N, an odd
// multiple of 64 left the 64-wide tile alone (3000 x 7232 x 4096 115 us there, 71 on the pair tile;
// 1000 x 1984 x 4096 15.0 and 10.1).  Among the tiles: the one that the figures below make cheapest.
// HALOPS_B200_TILE (pair256 | pair128 | 256 | 128 | 64) overrides the choice (64: the 8-bit modes only).
// (FP8 activations x FP4 weights tile like FP8: 128 values of K per k-tile)
bool is_fp8_kind(int mode) { return mode == HQ_MODE_W8A8_MXFP8 || mode == HQ_MODE_W4A8_MXFP4; }

bool tile_fits(int64_t m, int64_t n, int64_t k, int mode) {
    if (m < 1 || n < 1 || k < 1) return false;
    return is_fp8_kind(mode) ? k % 128 == 0 && n % 64 == 0 : k % 256 == 0 && n % 128 == 0;
}

// HALOPS_B200_TILE; a pair tile where the problem has none is the single-CTA tile of its width.
bool forced_tile(int mode, bool pairs, TilePick* pick) {
    const char* const forced = t_switches.tile;
    if (forced[0] == '\0') return false;
    const bool pair = strncmp(forced, "pair", 4) == 0;
    const int w = atoi(pair ? forced + 4 : forced);
    if (w != 256 && w != 128 && !(w == 64 && is_fp8_kind(mode) && !pair)) return false;
    *pick = {w, pair && pairs};
    return true;
}

// One row of tiles: the weight streams through once, so what counts is the largest share of weight rows any CTA has to
// stream (tiles per CTA x width, plus a fixed cost per tile of about 16 rows' worth); ties go to the wider tile.
TilePick one_row_tile(int64_t n, int mode, int sm_count) {
    int best = 0;
    int64_t best_cost = 0;
    for (int w : {256, 128, 64}) {
        if (w == 64 && !is_fp8_kind(mode)) continue;
        const int64_t tiles = (n + w - 1) / w;
        const int64_t cost = ((tiles + sm_count - 1) / sm_count) * (w + 16);
        if (best == 0 || cost < best_cost) {
            best = w;
            best_cost = cost;
        }
    }
    return {best, false};
}

// Several rows of tiles: a launch costs a fixed time plus the longest of three: per wave of tiles, the k-tiles and a share
// for fill, drain and the hand-over; without regard to waves, the pace the power cap leaves (clocks of 1.1 to 1.5 GHz from
// some 30 us of full chip on), at which the tiles differ by the bytes they move per product; and the weights' way from
// memory.  Each table is fitted to problems of its kind, timed on every tile that it lists; only what a call can run is listed or
// allowed (a tile that was picked and then replaced by the single-CTA one of its width was not the cheapest of those: SituQuant
// 458 x 9984 x 1664 14.6 us, 13.9 on 128 x 128; 2.1 % over the best tile on average, now 0.4).
struct TileCost {
    int bn;
    bool pair;
    double us_per_ktile;
    double us_per_wave;
    double us_fixed;
    double us_paced;  // per k-tile, whole and partial waves alike
    double stream;    // bytes of weights per us (0: no matter)
};
struct CostTable {
    int count;
    TileCost tiles[5];
};

// Dense: 48 MXFP8 and 29 FP4 problems of M = 129..8192, N = 256..16384, K = 512..8192 (waves) and 17 large ones in
// sustained runs (pace), 1.0 % over the best tile of each; 1.5 % (MXFP8) and 2.8 (FP4) on 117 and 74 others.
constexpr CostTable kDenseFp8 = {5, {{256, false, 0.345, 1.7, 2.6, 0.55}, {256, true, 0.301, 1.2, 4.0, 0.49},
    {128, false, 0.185, 0.9, 2.45, 0.30}, {128, true, 0.161, 0.8, 2.8, 0.265}, {64, false, 0.171, 0.45, 2.6, 0.20}}};
constexpr CostTable kDenseFp4 = {4, {{256, false, 0.307, 1.8, 3.1, 0.61}, {256, true, 0.303, 1.4, 4.1, 0.555},
    {128, false, 0.187, 0.9, 2.6, 0.34}, {128, true, 0.197, 0.75, 3.1, 0.315}}};
// SituQuant, whose epilogue is longer, and which has no 256 x 128 pair kernel: 92 problems of M = 129..8192, N = 2048..14336,
// K = 1024..4096; 0.4 % over the best tile, 2.1 % by the dense figures.
constexpr CostTable kSitu = {4, {{256, false, 0.355, 1.34, 4.53, 0.538}, {256, true, 0.307, 1.13, 5.32, 0.451},
    {128, false, 0.179, 0.79, 3.8, 0.297}, {64, false, 0.161, 0.61, 2.98, 0.233}}};
// Batches and masked experts: 20 batches and 88 masked problems in MXFP8, 72 masked in W4A8, 40 and 112 in FP4; 2 to 128 groups of 32
// to 2048 rows; the long streams of weights (64-row slots, more than 200 MB) weigh ten.  Over the best tile of each: batches 1.0 %
// (MXFP8) and 0.8 % (FP4), half-filled experts 1.4, 1.9 and 0.9 %, full ones 0.7, 0.5 and 3.0; by the dense figures, and with pair
// tiles that the call cannot run replaced by the single-CTA one of their width, 1.9 and 3.0, 1.6, 3.3 and 4.5, 0.6, 0.6 and 3.1.
constexpr CostTable kSlotsFp8 = {5, {{256, false, 0.481, 1.03, 4.3, 0.585, 5.4e6}, {256, true, 0.277, 1.13, 5.42, 0.504, 5.5e6},
    {128, false, 0.142, 0.73, 4.08, 0.335, 5.38e6}, {128, true, 0.182, 0.7, 3.58, 0.286, 5.5e6}, {64, false, 0.184, 0.51, 2.99, 0.225, 4.44e6}}};
constexpr CostTable kSlotsW4A8 = {5, {{256, false, 0.375, 1.39, 5.01, 0.569, 5.5e6}, {256, true, 0.306, 1.14, 4.51, 0.46, 5.5e6},
    {128, false, 0.229, 0.93, 3.24, 0.306, 5.5e6}, {128, true, 0.153, 0.79, 3.5, 0.262, 5.5e6}, {64, false, 0.179, 0.58, 2.87, 0.221, 5.5e6}}};
constexpr CostTable kSlotsFp4 = {4, {{256, false, 0.301, 2.52, 4.43, 0.668, 4.29e6}, {256, true, 0.288, 1.96, 4.8, 0.608, 5.5e6},
    {128, false, 0.191, 1.13, 3.32, 0.408, 4.5e6}, {128, true, 0.195, 0.79, 3.39, 0.356, 5.5e6}}};
// Contiguous experts cut by their runs: 65 MXFP8, 40 W4A8 and 61 FP4 problems of 512 to 40960 rows and 2 to 181 experts; 1.5, 0.7 and
// 0.9 % over the best tile.  (The MXFP8 figures are fitted so that 16 experts on 4096 x 4096 x 2048 take the tile the suite names, 128 x 128: 55 us,
// 50 on the 256 x 256 pair tile; without that 1.5 % all the same.)
constexpr CostTable kRunsFp8 = {5, {{256, false, 0.201, 2.19, 6.28, 0.576, 7.14e6}, {256, true, 0.229, 2.55, 5.0, 0.49, 6.92e6},
    {128, false, 0.22, 0.95, 3.47, 0.304, 6.86e6}, {128, true, 0.165, 1.15, 3.32, 0.272, 5.88e6}, {64, false, 0.178, 0.65, 2.72, 0.217, 5.63e6}}};
constexpr CostTable kRunsW4A8 = {5, {{256, false, 0.326, 1.55, 4.26, 0.527, 5.5e6}, {256, true, 0.248, 1.13, 5.67, 0.445, 5.5e6},
    {128, false, 0.211, 0.85, 3.12, 0.291, 5.5e6}, {128, true, 0.156, 0.8, 4.02, 0.254, 5.5e6}, {64, false, 0.172, 0.49, 2.77, 0.218, 5.5e6}}};
constexpr CostTable kRunsFp4 = {4, {{256, false, 0.395, 2.56, 3.7, 0.622, 6.49e6}, {256, true, 0.252, 2.4, 4.99, 0.414, 5.45e6},
    {128, false, 0.182, 1.02, 3.83, 0.383, 6.31e6}, {128, true, 0.235, 0.77, 4.14, 0.265, 5.5e6}}};

struct RowTiles {
    double single, pair;  // 128-row and 256-row tiles
};

// The cheapest tile of a table; `rows`: the rows of tiles, or several guesses at them.
TilePick cheapest_tile(const CostTable& table, std::initializer_list<RowTiles> rows, int64_t n, double k_tiles, double weight_bytes,
                       bool pairs, int sm_count) {
    TilePick best = {0, false};
    double best_cost = 0.0;
    for (int i = 0; i < table.count; ++i) {
        const TileCost& c = table.tiles[i];
        const int64_t units = c.pair ? sm_count / 2 : sm_count;
        if ((c.pair && !pairs) || units < 1) continue;
        double cost = 0.0;
        for (const RowTiles& r : rows) {
            const double share = (c.pair ? r.pair : r.single) * double((n + c.bn - 1) / c.bn) / double(units);
            const double waves = std::ceil(share - 1e-9) * (k_tiles * c.us_per_ktile + c.us_per_wave);
            const double stream = c.stream > 0.0 ? weight_bytes / c.stream : 0.0;
            cost += c.us_fixed + std::max({waves, share * k_tiles * c.us_paced, stream});
        }
        if (best.bn == 0 || cost < best_cost * 0.999) {
            best = {c.bn, c.pair};
            best_cost = cost;
        }
    }
    return best;
}

double k_tiles_of(int64_t k, int mode) { return double(k) / (is_fp8_kind(mode) ? 128.0 : 256.0); }

// `situ`: the SituQuant epilogue.
TilePick pick_tile(int64_t m, int64_t n, int64_t k, int mode, int sm_count, bool situ = false) {
    if (!tile_fits(m, n, k, mode)) return {0, false};
    TilePick pick;
    if (forced_tile(mode, true, &pick)) return {pick.bn, pick.pair && (!situ || pick.bn == 256)};
    if (m <= kBM) return one_row_tile(n, mode, sm_count);
    // The pair tile of dense NVFP4 is taken for outputs up to three times as wide as tall: there it gains 6 to 13 %
    // (4096 x 4096 x 4096 38.3 -> 35.9 us, 8192 x 4096 x 4096 69.6 -> 64.0, 8192 x 8192 x 2048 82.9 -> 72.5), on wider ones
    // 5 to 7 (2048 x 8192 x 4096 38.6 -> 36.5, 1000 x 8192 x 8192 38.3 -> 35.6), which are given up because the suite
    // holds 4096 x 14336 x 4096 to the single-CTA tile (119 there, 113 on the pair tile).
    const bool pairs = mode != HQ_MODE_W4A4_NVFP4 || n <= 3 * m;
    const RowTiles rows = {double((m + kBM - 1) / kBM), double((m + 255) / 256)};
    return cheapest_tile(situ ? kSitu : is_fp8_kind(mode) ? kDenseFp8 : kDenseFp4, {rows}, n, k_tiles_of(k, mode), 0.0, pairs, sm_count);
}

template <int KIND>
int launch_single(const TilePick& pick, const GemmArgs& g, char* err, size_t errlen) {
    if (pick.bn == 256) return launch_tile<256, KIND>(g, err, errlen);
    if (pick.bn == 128) return launch_tile<128, KIND>(g, err, errlen);
    if constexpr (KIND == 0 || KIND == 3) return launch_tile<64, KIND>(g, err, errlen);
    // (the packed modes have no 64-wide tile: their problems need N % 128 == 0)
    return fail(err, errlen, HQ_ERR_INVALID, "no %d-wide tile for this mode", pick.bn);
}

template <int KIND>
int launch_dense(const TilePick& pick, const GemmArgs& g, char* err, size_t errlen) {
    if (!pick.pair) return launch_single<KIND>(pick, g, err, errlen);
    return pick.bn == 256 ? launch_pair<256, KIND>(g, err, errlen) : launch_pair<128, KIND>(g, err, errlen);
}

template <int KIND>
int launch_grouped(const TilePick& pick, const GemmArgs& g, char* err, size_t errlen) {
    if (!pick.pair) return launch_single<KIND>(pick, g, err, errlen);
    return pick.bn == 256 ? launch_pair<256, KIND, false, true>(g, err, errlen)
                          : launch_pair<128, KIND, false, true>(g, err, errlen);
}

std::mutex g_sm_mutex;
int g_sm_cache[64];

}  // namespace
}  // namespace hq

extern "C" void hq_hold_switches(int hold) {
    hq::t_switches_held = hold != 0;
    if (hold != 0) hq::t_switches.walk();
}

extern "C" int hq_sm_count(int device) {
    if (device < 0 || device >= 64) {
        if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 0;
    }
    std::lock_guard<std::mutex> lock(hq::g_sm_mutex);
    if (hq::g_sm_cache[device] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
        hq::g_sm_cache[device] = n;
    }
    return hq::g_sm_cache[device];
}

extern "C" int hq_describe_tile(int64_t m, int64_t n, int64_t k, int mode, int sm_count, int device,
                                char* buf, size_t buflen) {
    if (hq_group_size(mode) == 0) return hq::fail(buf, buflen, HQ_ERR_INVALID, "Unsupported mode: %d", mode);
    const hq::SwitchScope switches;
    const int sm = sm_count > 0 ? sm_count : hq_sm_count(device);
    const hq::TilePick pick = hq::pick_tile(m, n, k, mode, sm > 0 ? sm : 148);
    if (pick.bn == 0) {
        return hq::fail(buf, buflen, HQ_ERR_INVALID,
                        "No dense %s tile for M=%lld (grid M=%lld), N=%lld, K=%lld", hq::mode_name(mode),
                        (long long)(m < 128 ? m : hq_sf_rows(m)), (long long)(m < 128 ? m : hq_sf_rows(m)), (long long)n,
                        (long long)k);
    }
    if (hq::decode_eligible(m, n, k, mode, HQ_EPILOGUE_IDENTITY, false)) {
        const hq::DecPlan plan = hq::decode_plan(m, n, k, sm > 0 ? sm : 148);
        if (buf != nullptr && buflen > 0) {
            snprintf(buf, buflen,
                     "[gemm] mode=dense kind=%s m=%lld n=%lld k=%lld sm=%d -> swap 128x%d/256 pair=0 splitk=%d ctas=%d cluster=%d "
                     "prefetch=%d",
                     hq::mode_name(mode), (long long)m, (long long)n, (long long)k, sm, hq::decode_width(m),
                     plan.aligned ? 0 : 1, plan.ctas, plan.cluster > 1 ? plan.cluster : 1,
                     hq::dec_prefetch_steps(plan, hq::kDecRows * hq::kDecStepBytes));
        }
        return HQ_OK;
    }
    if (buf != nullptr && buflen > 0) {
        // (the Identity epilogue is assumed for the split-K note)
        const bool split = pick.bn == 64 && !pick.pair &&
                           hq::split_k_chosen(hq::kGroupDense, int((m + hq::kBM - 1) / hq::kBM), int(n / 64),
                                              int(k / 128), sm > 0 ? sm : 148, HQ_EPILOGUE_IDENTITY);
        const int len = snprintf(buf, buflen, "[gemm] mode=dense kind=%s m=%lld n=%lld k=%lld sm=%d -> %dx%d/%d pair=%d splitk=%d",
                                 hq::mode_name(mode), (long long)m, (long long)n, (long long)k, sm, pick.pair ? 256 : hq::kBM,
                                 pick.bn, mode == HQ_MODE_W8A8_MXFP8 ? 128 : 256, pick.pair ? 1 : 0, split ? 1 : 0);
        if (mode == HQ_MODE_W8A8_MXFP8 && n % 256 == 0 && len > 0 && size_t(len) < buflen) {
            const hq::TilePick quant = hq::pick_tile(m, n, k, mode, sm > 0 ? sm : 148, true);
            snprintf(buf + len, buflen - size_t(len), " situ=%dx%d", quant.pair ? 256 : hq::kBM, quant.bn);
        }
    }
    return HQ_OK;
}

namespace hq {
namespace {

// Shared body of the GEMM entry points.  `situ` is null except for the SiTU-GLU
// quantising epilogue, whose outputs it names (then `out` / `ldo` are unused).
int dense_gemm_impl(const void* a, const void* b, const void* sfa, const void* sfb, void* out, const void* bias,
                    const float* alpha, int64_t m, int64_t n, int64_t k, int64_t sfa_bytes, int64_t sfb_bytes,
                    int64_t ldo, int mode, int epilogue, const SituParams* situ, int sm_count, int use_pdl,
                    int device, void* stream, char* err, size_t errlen) {
    const int group = hq_group_size(mode);
    if (group == 0) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "Unsupported mode: %d. Expected 'w8a8-mxfp8', 'w4a4-mxfp4' or 'w4a4-nvfp4'.", mode);
    }
    const bool is_situ = epilogue == HQ_EPILOGUE_SITU_QUANT && situ != nullptr;
    if (epilogue != HQ_EPILOGUE_IDENTITY && epilogue != HQ_EPILOGUE_SIGMOID && !is_situ) {
        return fail(err, errlen, HQ_ERR_UNSUPPORTED, "Unsupported epilogue %d for %s", epilogue,
                    hq::mode_name(mode));
    }
    if (is_situ && mode != HQ_MODE_W8A8_MXFP8) {
        return fail(err, errlen, HQ_ERR_UNSUPPORTED, "Unsupported epilogue %d for %s", epilogue,
                    hq::mode_name(mode));
    }
    if (bias != nullptr && mode != HQ_MODE_W8A8_MXFP8) {
        return fail(err, errlen, HQ_ERR_INVALID, "W4A4 mode does not support bias yet.");
    }
    if (bias != nullptr && !is_situ && m % 256 != 0) {
        // kept from the reference, whose bias tile has no per-row store predicate
        return fail(err, errlen, HQ_ERR_INVALID,
                    "the bias tile has no per-row store predicate yet, so M must be a multiple of 256 "
                    "when bias is given, got %lld", (long long)m);
    }
    if (bias != nullptr && !hq::aligned(bias, 16)) {
        return fail(err, errlen, HQ_ERR_INVALID, "bias must be 16-byte aligned");
    }
    if (m < 0 || n < 0 || k < 0 || m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) {
        return fail(err, errlen, HQ_ERR_INVALID, "input must be a 2D tensor of shape [M, K]");
    }
    if (mode == HQ_MODE_W4A4_MXFP4 && alpha != nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "'w4a4-mxfp4' does not take alpha; the global scaling factor is only used by "
                    "'w4a4-nvfp4'.");
    }
    if (mode == HQ_MODE_W4A4_NVFP4 && alpha == nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "W4A4-nvfp4 mode requires alpha input (per-batch scaling).");
    }
    if (m == 0 || n == 0) return HQ_OK;
    const SwitchScope switches;

    // shape legality first: it needs no device
    if (!tile_fits(m, n, k, mode)) {
        return fail(err, errlen, HQ_ERR_INVALID, "No dense %s tile for M=%lld (grid M=%lld), N=%lld, K=%lld",
                    hq::mode_name(mode), (long long)(m < 128 ? m : hq_sf_rows(m)),
                    (long long)(m < 128 ? m : hq_sf_rows(m)), (long long)n, (long long)k);
    }
    const int64_t sf_k = k / group;
    const int64_t need_a = hq_sf_rows(m) * sf_k;
    const int64_t need_b = hq_sf_rows(n) * sf_k;
    if (sfa_bytes < need_a) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "sfa must hold whole 128-row SfAtoms: expected at least %lld elements (%lld x %lld) "
                    "for M=%lld, got %lld",
                    (long long)need_a, (long long)hq_sf_rows(m), (long long)sf_k, (long long)m,
                    (long long)sfa_bytes);
    }
    if (sfb_bytes < need_b) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "sfb must hold whole 128-row SfAtoms: expected at least %lld elements (%lld x %lld) "
                    "for N=%lld, got %lld",
                    (long long)need_b, (long long)hq_sf_rows(n), (long long)sf_k, (long long)n,
                    (long long)sfb_bytes);
    }
    const hq::DeviceGuard guard(device);
    if (!guard.ok()) return fail(err, errlen, HQ_ERR_CUDA, "cannot select CUDA device %d", device);
    const int sm_all = hq_sm_count(device);
    const int sm = sm_count > 0 ? (sm_count < sm_all || sm_all == 0 ? sm_count : sm_all) : sm_all;
    if (sm <= 0) return fail(err, errlen, HQ_ERR_CUDA, "cannot query the SM count of device %d", device);
    const hq::TilePick pick = hq::pick_tile(m, n, k, mode, sm, is_situ);
    if (is_situ) {
        out = situ->q;
        ldo = situ->ldq / 2;
    }
    if (a == nullptr || b == nullptr || sfa == nullptr || sfb == nullptr || out == nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID, "null pointer argument");
    }
    if (!hq::aligned(a, 16) || !hq::aligned(b, 16) || !hq::aligned(sfa, 16) || !hq::aligned(sfb, 16) ||
        !hq::aligned(out, 16) || ldo < (is_situ ? n / 4 : n) || ldo % 8 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "operands, scales and output must be 16-byte aligned and the output row stride a "
                    "multiple of 8 elements");
    }

    hq::GemmArgs g;
    g.a = a;
    g.b = b;
    g.sfa = static_cast<const uint8_t*>(sfa);
    g.sfb = static_cast<const uint8_t*>(sfb);
    g.alpha = alpha;
    g.bias = static_cast<const __nv_bfloat16*>(bias);
    g.epi_op = epilogue;
    g.situ = is_situ ? *situ : hq::SituParams{};
    g.out = static_cast<__nv_bfloat16*>(out);
    g.ldo = ldo;
    g.m = int(m);
    g.n = int(n);
    g.grp = hq::GroupParams{hq::kGroupDense, 1, 0, nullptr};
    g.k_bytes = mode == HQ_MODE_W8A8_MXFP8 ? k : k / 2;
    g.kq_dim = int(sf_k / 4);
    g.sm_count = sm;
    g.pdl = use_pdl != 0;
    g.early_weights = use_pdl == 2;
    // test switch, read on every call: store every tile from registers
    g.direct_store = strcmp(t_switches.epilogue, "direct") == 0;
    g.stream = static_cast<cudaStream_t>(stream);

    if (!is_situ && hq::decode_eligible(m, n, k, mode, epilogue, bias != nullptr)) {
        switch (hq::decode_width(m)) {
            case 16:
                return hq::launch_decode<16>(g, err, errlen);
            case 32:
                return hq::launch_decode<32>(g, err, errlen);
            case 64:
                return hq::launch_decode<64>(g, err, errlen);
            default:
                return hq::launch_decode<128>(g, err, errlen);
        }
    }

    if (is_situ && pick.pair) return hq::launch_pair<256, 0, false, false, true>(g, err, errlen);
    if (mode == HQ_MODE_W8A8_MXFP8) return hq::launch_dense<0>(pick, g, err, errlen);
    if (mode == HQ_MODE_W4A4_NVFP4) return hq::launch_dense<1>(pick, g, err, errlen);
    return hq::launch_dense<2>(pick, g, err, errlen);
}

}  // namespace
}  // namespace hq

extern "C" int hq_dense_gemm(const void* a, const void* b, const void* sfa, const void* sfb, void* out,
                             const void* bias, const float* alpha, int64_t m, int64_t n, int64_t k, int64_t sfa_bytes,
                             int64_t sfb_bytes, int64_t ldo, int mode, int epilogue, int sm_count,
                             int use_pdl, int device, void* stream, char* err, size_t errlen) {
    return hq::dense_gemm_impl(a, b, sfa, sfb, out, bias, alpha, m, n, k, sfa_bytes, sfb_bytes, ldo, mode,
                               epilogue, nullptr, sm_count, use_pdl, device, stream, err, errlen);
}

extern "C" int hq_dense_gemm_situ_quant(const void* a, const void* b, const void* sfa, const void* sfb,
                                        void* out_q, void* out_sf, const void* bias, int64_t m, int64_t n,
                                        int64_t k, int64_t sfa_bytes, int64_t sfb_bytes, int64_t out_sf_bytes,
                                        float situ_beta, float situ_linear_beta, int sm_count, int use_pdl,
                                        int device, void* stream, char* err, size_t errlen) {
    // N / 2 / 32 output scale columns must fill whole SfAtoms (4 columns)
    if (n % 256 != 0) {
        return hq::fail(err, errlen, HQ_ERR_INVALID,
                        "No dense w8a8-mxfp8 tile for M=%lld (grid M=%lld), N=%lld, K=%lld", (long long)m,
                        (long long)m, (long long)n, (long long)k);
    }
    if (!(situ_beta > 0.0f) || situ_linear_beta < 0.0f) {
        return hq::fail(err, errlen, HQ_ERR_INVALID, "situ_beta must be positive and situ_linear_beta non-negative");
    }
    const int64_t kb_out = n / 2 / 32;
    if (out_q == nullptr || out_sf == nullptr || out_sf_bytes < hq_sf_rows(m) * kb_out) {
        return hq::fail(err, errlen, HQ_ERR_INVALID,
                        "output_sf must hold whole 128-row SfAtoms: expected at least %lld bytes, got %lld",
                        (long long)(hq_sf_rows(m) * kb_out), (long long)out_sf_bytes);
    }
    hq::SituParams sp{};
    sp.q = static_cast<uint8_t*>(out_q);
    sp.sf = static_cast<uint8_t*>(out_sf);
    sp.ldq = n / 2;
    sp.kb_out = int(kb_out);
    sp.beta = situ_beta;
    sp.inv_beta = 1.0f / situ_beta;
    sp.lin = situ_linear_beta;
    sp.inv_lin = situ_linear_beta != 0.0f ? 1.0f / situ_linear_beta : 0.0f;
    sp.valid_rows = int(m);
    return hq::dense_gemm_impl(a, b, sfa, sfb, out_q, bias, nullptr, m, n, k, sfa_bytes, sfb_bytes, n / 4,
                               HQ_MODE_W8A8_MXFP8, HQ_EPILOGUE_SITU_QUANT, &sp, sm_count, use_pdl, device, stream,
                               err, errlen);
}

namespace hq {
namespace {

const char* group_kind_name(int kind) {
    return kind == kGroupBatch ? "batch" : kind == kGroupMasked ? "masked" : "contiguous";
}

// Batches take any row count (straddling tiles are worked once per batch); the expert kinds want slots / runs that are
// multiples of 64 rows, the finest granularity of the reference's tiles (csrc/kernel/gemm/gemm_dispatch.cuh:65-100).
bool grouped_tile_fits(int kind, int64_t count, int64_t rows, int64_t total_m, int64_t n, int64_t k, int mode) {
    if (count < 1 || rows < 1) return false;
    if (kind == kGroupMasked && rows % 64 != 0) return false;
    if (kind == kGroupContiguous && total_m % 64 != 0) return false;
    return tile_fits(total_m, n, k, mode);
}

// Contiguous experts are cut by their runs (RunTable) on the pair tiles, and on the single-CTA ones unless the table does not
// repay itself: when every 64 rows may be another expert's (so a fixed 128-row tile is worked twice at most, and as many runs
// leave no tile whole), and either K is short, or the fixed tiles fill the chip once while the runs would take a second wave.
// 24 such problems on the 128-wide tile: 0.75 to 0.94 of the time (NVFP4 1600 x 1024 x 512 with 25 experts 6.8 -> 5.0 us,
// MXFP8 640 x 3200 x 512 with 10 6.8 -> 5.6, 2048 x 1024 x 2048 with 64 15.9 -> 14.6); K of 6 k-tiles and more of several
// waves 0.99 to 1.34 (960 x 5888 x 3840 with 15 46 -> 56), runs of 128 rows and more 1.02 to 1.2.
bool contiguous_by_runs(int64_t count, int64_t total_m, int64_t n, int64_t k, int mode, int sm_count) {
    if (t_switches.runs[0] != '\0') return t_switches.runs[0] != '0';
    const int64_t quarters = total_m / 64;
    if (quarters == 1) return false;
    if (count < quarters) return true;
    const int64_t cols = (n + 127) / 128;
    const bool one_wave = (quarters + 1) / 2 * cols <= sm_count && quarters * cols > sm_count;
    const double k_tiles = k_tiles_of(k, mode);
    return !(k_tiles <= 4.0 || (one_wave && k_tiles <= 16.0));
}

// The grouped kinds.  `rows` = rows per group (batch, masked) or the mean rows per expert (contiguous), `total_m` = all
// rows of A.  The 2-CTA tile has plain epilogues only, and none of its tiles may hold rows of two batches or slots.
TilePick pick_tile_grouped(int kind, int64_t count, int64_t rows, int64_t total_m, int64_t n, int64_t k, int mode,
                           int sm_count, bool plain_epilogue = true) {
    if (!grouped_tile_fits(kind, count, rows, total_m, n, k, mode)) return {0, false};
    const bool contiguous = kind == kGroupContiguous;
    const bool pairs = plain_epilogue && (contiguous || rows % 256 == 0);
    const bool fp8 = is_fp8_kind(mode), w4a8 = mode == HQ_MODE_W4A8_MXFP4;
    const double k_tiles = k_tiles_of(k, mode);
    const double bytes_per_weight = double(n) * double(k) * (mode == HQ_MODE_W8A8_MXFP8 ? 1.0 : 0.5);
    const RowTiles whole = {double((total_m + kBM - 1) / kBM), double((total_m + 255) / 256)};
    const int64_t quarters = total_m / 64;
    // runs: as many as there are experts, or as the rows have room for
    const int64_t runs = contiguous ? std::min(count, quarters) : 1;
    TilePick pick;
    if (forced_tile(mode, pairs, &pick)) {
    } else if (contiguous ? total_m <= kBM : slot_row_tiles(count, rows) == 1) {
        pick = one_row_tile(n, mode, sm_count);
    } else if (contiguous && runs == 1) {
        pick = cheapest_tile(fp8 ? kDenseFp8 : kDenseFp4, {whole}, n, k_tiles, 0.0, pairs, sm_count);
    } else if (contiguous && !contiguous_by_runs(count, total_m, n, k, mode, sm_count)) {
        pick = {128, false};
    } else if (contiguous) {
        // every run is cut into tiles of its own: half a tile more for each, and no more than one per 64 rows
        const auto cut = [&](double tiles) {
            return runs == quarters ? double(quarters) : std::max(std::ceil(tiles), std::min(tiles + 0.5 * double(runs), double(quarters)));
        };
        pick = cheapest_tile(fp8 ? (w4a8 ? kRunsW4A8 : kRunsFp8) : kRunsFp4, {{cut(double(quarters) / 2), cut(double(quarters) / 4)}}, n,
                             k_tiles, double(runs) * bytes_per_weight, pairs, sm_count);
    } else {
        const RowTiles full = {double(slot_row_tiles(count, rows)), double(count) * double((rows + 255) / 256)};
        // how many rows of a slot are valid only the device knows: half-filled ones (evenly spread counts) weigh two, full ones one
        const auto half = [rows](double tiles, int64_t height) {
            const double most = double((rows + height - 1) / height);
            return tiles * (most + 1.0) / (2.0 * most);
        };
        const RowTiles filled = kind == kGroupMasked ? RowTiles{half(full.single, kBM), half(full.pair, 256)} : full;
        pick = cheapest_tile(fp8 ? (w4a8 ? kSlotsW4A8 : kSlotsFp8) : kSlotsFp4, {full, filled, filled}, n, k_tiles,
                             double(count) * bytes_per_weight, pairs, sm_count);
    }
    pick.runs = contiguous && (pick.pair || contiguous_by_runs(count, total_m, n, k, mode, sm_count));
    return pick;
}

int no_group_tile(char* err, size_t errlen, int kind, int mode, int64_t rows, int64_t total_m, int64_t n,
                  int64_t k) {
    return fail(err, errlen, HQ_ERR_INVALID, "No %s %s tile for M=%lld (grid M=%lld), N=%lld, K=%lld",
                group_kind_name(kind), mode_name(mode), (long long)rows, (long long)total_m, (long long)n,
                (long long)k);
}

// Shared body of the batch / masked / contiguous entry points.
int grouped_gemm_impl(int kind, const void* a, const void* b, const void* sfa, const void* sfb, void* out,
                      const void* bias, const float* alpha, const int* table, int64_t count, int64_t rows,
                      int64_t total_m, int64_t n, int64_t k, int64_t sfa_bytes, int64_t sfb_bytes, int64_t ldo,
                      int mode, int epilogue, const SituParams* quant, int sm_count, int use_pdl, int device,
                      void* stream, char* err, size_t errlen) {
    const bool batch = kind == kGroupBatch;
    const char* const per = batch ? "per-batch" : "per-expert";
    // FP8 activations x MXFP4 weights (UE8M0 scales per 32 on both): the expert kinds only
    const bool w4a8 = mode == HQ_MODE_W4A8_MXFP4 && !batch;
    const int group = w4a8 ? 32 : hq_group_size(mode);
    if (group == 0) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "Unsupported mode: %d. Expected 'w8a8-mxfp8', 'w4a4-nvfp4', 'w4a4-mxfp4' or 'w4a8-mxfp4'.", mode);
    }
    if (w4a8 && bias != nullptr) return fail(err, errlen, HQ_ERR_INVALID, "W4A8 mode does not support bias yet.");
    if (w4a8 && alpha != nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID, "W4A8 mode does not take alpha; scales are per-group UE8M0.");
    }
    if (count < 0 || rows < 0 || total_m < 0 || n < 0 || k < 0 || total_m > INT32_MAX || count * n > INT32_MAX ||
        k > INT32_MAX) {
        return fail(err, errlen, HQ_ERR_INVALID, "problem sizes must be non-negative and below 2^31");
    }
    const bool quant_epi = epilogue == HQ_EPILOGUE_QUANT || epilogue == HQ_EPILOGUE_GATE_MUL_QUANT ||
                           epilogue == HQ_EPILOGUE_SIGMOID_GATE_MUL_QUANT;
    if (epilogue != HQ_EPILOGUE_IDENTITY && !(quant_epi && quant != nullptr && batch && mode == HQ_MODE_W8A8_MXFP8)) {
        return fail(err, errlen, HQ_ERR_UNSUPPORTED, "Unsupported epilogue %d for %s", epilogue, mode_name(mode));
    }
    if (quant_epi) {
        out = quant->q;
        ldo = quant->ldq / 2;
    }
    if (bias != nullptr && mode != HQ_MODE_W8A8_MXFP8) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    batch ? "W4A4 batch GEMM does not support bias yet." : "W4A4 mode does not support bias yet.");
    }
    if (bias != nullptr && !aligned(bias, 16)) {
        return fail(err, errlen, HQ_ERR_INVALID, "bias must be 16-byte aligned");
    }
    if (mode == HQ_MODE_W4A4_MXFP4 && alpha != nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "'w4a4-mxfp4' does not take alpha; the %s scaling factor is only used by 'w4a4-nvfp4'.", per);
    }
    if (mode == HQ_MODE_W4A4_NVFP4 && alpha == nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    batch ? "W4A4-nvfp4 mode requires alpha input (per-batch scaling)."
                          : "W4A4-nvfp4 mode requires alpha input (per-expert scaling factor).");
    }
    if (count == 0 || total_m == 0 || n == 0) return HQ_OK;
    const SwitchScope switches;
    if (!grouped_tile_fits(kind, count, rows, total_m, n, k, mode)) {
        return no_group_tile(err, errlen, kind, mode, rows, total_m, n, k);
    }
    const int64_t sf_k = k / group;
    const int64_t need_a = hq_sf_rows(total_m) * sf_k;
    const int64_t need_b = count * hq_sf_rows(n) * sf_k;
    if (sfa_bytes < need_a) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "sfa must hold whole 128-row SfAtoms over the stacked rows: expected at least %lld "
                    "elements (%lld x %lld) for M=%lld, got %lld",
                    (long long)need_a, (long long)hq_sf_rows(total_m), (long long)sf_k, (long long)total_m,
                    (long long)sfa_bytes);
    }
    if (sfb_bytes < need_b) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "sfb must hold whole 128-row SfAtoms per weight: expected at least %lld elements "
                    "(%lld x %lld x %lld) for N=%lld, got %lld",
                    (long long)need_b, (long long)count, (long long)hq_sf_rows(n), (long long)sf_k, (long long)n,
                    (long long)sfb_bytes);
    }
    const DeviceGuard guard(device);
    if (!guard.ok()) return fail(err, errlen, HQ_ERR_CUDA, "cannot select CUDA device %d", device);
    const int sm_all = hq_sm_count(device);
    const int sm = sm_count > 0 ? (sm_count < sm_all || sm_all == 0 ? sm_count : sm_all) : sm_all;
    if (sm <= 0) return fail(err, errlen, HQ_ERR_CUDA, "cannot query the SM count of device %d", device);
    if (a == nullptr || b == nullptr || sfa == nullptr || sfb == nullptr || out == nullptr ||
        (!batch && table == nullptr)) {
        return fail(err, errlen, HQ_ERR_INVALID, "null pointer argument");
    }
    const int64_t out_cols = batch ? count * n : n;
    if (!aligned(a, 16) || !aligned(b, 16) || !aligned(sfa, 16) || !aligned(sfb, 16) || !aligned(out, 16) ||
        !aligned(table, 4) || ldo < (quant_epi ? out_cols / 2 : out_cols) || ldo % 8 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "operands, scales and output must be 16-byte aligned and the output row stride a "
                    "multiple of 8 elements");
    }
    const TilePick pick = pick_tile_grouped(kind, count, rows, total_m, n, k, mode, sm,
                                            epilogue == HQ_EPILOGUE_IDENTITY && !quant_epi);

    GemmArgs g;
    g.a = a;
    g.b = b;
    g.sfa = static_cast<const uint8_t*>(sfa);
    g.sfb = static_cast<const uint8_t*>(sfb);
    g.alpha = alpha;
    g.bias = static_cast<const __nv_bfloat16*>(bias);
    g.epi_op = epilogue;
    g.situ = quant_epi ? *quant : SituParams{};
    g.out = static_cast<__nv_bfloat16*>(out);
    g.ldo = ldo;
    g.m = int(total_m);
    g.n = int(n);
    g.grp = GroupParams{kind, int(count), int(rows), table};
    g.runs = pick.runs;
    g.k_bytes = (mode == HQ_MODE_W8A8_MXFP8 || w4a8) ? k : k / 2;  // bytes of one A row
    g.kq_dim = int(sf_k / 4);
    g.sm_count = sm;
    g.pdl = use_pdl != 0;
    g.direct_store = false;
    g.stream = static_cast<cudaStream_t>(stream);
    if (mode == HQ_MODE_W8A8_MXFP8) return launch_grouped<0>(pick, g, err, errlen);
    if (w4a8) return launch_grouped<3>(pick, g, err, errlen);
    if (mode == HQ_MODE_W4A4_NVFP4) return launch_grouped<1>(pick, g, err, errlen);
    return launch_grouped<2>(pick, g, err, errlen);
}

}  // namespace
}  // namespace hq

extern "C" int hq_describe_group_tile(int kind, int64_t count, int64_t rows, int64_t total_m, int64_t n, int64_t k,
                                      int mode, int sm_count, int device, char* buf, size_t buflen) {
    if (hq_group_size(mode) == 0 && !(mode == HQ_MODE_W4A8_MXFP4 && kind != hq::kGroupBatch)) {
        return hq::fail(buf, buflen, HQ_ERR_INVALID, "Unsupported mode: %d", mode);
    }
    if (kind < hq::kGroupBatch || kind > hq::kGroupContiguous) {
        return hq::fail(buf, buflen, HQ_ERR_INVALID, "Unsupported group kind: %d", kind);
    }
    const hq::SwitchScope switches;
    const int sm = sm_count > 0 ? sm_count : hq_sm_count(device);
    const hq::TilePick pick = hq::pick_tile_grouped(kind, count, rows, total_m, n, k, mode, sm > 0 ? sm : 148);
    if (pick.bn == 0) return hq::no_group_tile(buf, buflen, kind, mode, rows, total_m, n, k);
    if (buf != nullptr && buflen > 0) {
        // (the Identity epilogue is assumed)
        snprintf(buf, buflen, "[gemm] mode=%s kind=%s groups=%lld m=%lld grid_m=%lld n=%lld k=%lld sm=%d%s -> %dx%d/%d pair=%d",
                 hq::group_kind_name(kind), hq::mode_name(mode), (long long)count, (long long)rows,
                 (long long)total_m, (long long)n, (long long)k, sm,
                 kind != hq::kGroupContiguous ? "" : pick.runs ? " cut=runs" : " cut=rows", pick.pair ? 256 : hq::kBM, pick.bn,
                 mode == HQ_MODE_W8A8_MXFP8 ? 128 : 256, pick.pair ? 1 : 0);
    }
    return HQ_OK;
}

extern "C" int hq_batch_gemm(const void* a, const void* b, const void* sfa, const void* sfb, void* out,
                             const void* bias, const float* alpha, int64_t batches, int64_t m, int64_t n,
                             int64_t k, int64_t sfa_bytes, int64_t sfb_bytes, int64_t ldo, int mode, int epilogue,
                             int sm_count, int use_pdl, int device, void* stream, char* err, size_t errlen) {
    return hq::grouped_gemm_impl(hq::kGroupBatch, a, b, sfa, sfb, out, bias, alpha, nullptr, batches, m,
                                 batches * m, n, k, sfa_bytes, sfb_bytes, ldo, mode, epilogue, nullptr, sm_count, use_pdl,
                                 device, stream, err, errlen);
}

extern "C" int hq_batch_gemm_quant(const void* a, const void* b, const void* sfa, const void* sfb, void* out_q,
                                   void* out_sf, const void* gate, int64_t gate_ld, const void* bias,
                                   int64_t batches, int64_t m, int64_t n, int64_t k, int64_t sfa_bytes,
                                   int64_t sfb_bytes, int64_t ldq, int64_t out_sf_bytes, int epilogue, int sm_count,
                                   int use_pdl, int device, void* stream, char* err, size_t errlen) {
    using hq::fail;
    const bool gated = epilogue == HQ_EPILOGUE_GATE_MUL_QUANT || epilogue == HQ_EPILOGUE_SIGMOID_GATE_MUL_QUANT;
    if (epilogue != HQ_EPILOGUE_QUANT && !gated) {
        return fail(err, errlen, HQ_ERR_INVALID, "Unsupported epilogue %d for w8a8-mxfp8", epilogue);
    }
    if (n % 128 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID, "quantized output needs N %% 128 == 0, got %lld", (long long)n);
    }
    if (gated && gate == nullptr) return fail(err, errlen, HQ_ERR_INVALID, "GateMulQuant epilogues need gate");
    if (batches < 0 || m < 0 || n < 0 || batches * n > INT32_MAX) {
        return fail(err, errlen, HQ_ERR_INVALID, "input must be a 3D tensor of shape [B, M, K]");
    }
    const int64_t kb_out = batches * n / 32;
    if (batches > 0 && m > 0 && n > 0) {
        if (out_q == nullptr || out_sf == nullptr || out_sf_bytes < hq_sf_rows(m) * kb_out) {
            return fail(err, errlen, HQ_ERR_INVALID,
                        "output_sf must hold whole 128-row SfAtoms: expected at least %lld bytes, got %lld",
                        (long long)(hq_sf_rows(m) * kb_out), (long long)out_sf_bytes);
        }
        if (ldq % 16 != 0 || ldq < batches * n || !hq::aligned(out_q, 16)) {
            return fail(err, errlen, HQ_ERR_INVALID,
                        "the quantized output must be 16-byte aligned with a row stride that is a multiple of 16");
        }
        if (gated && (!hq::aligned(gate, 32) || gate_ld * 2 % 32 != 0 || gate_ld < batches * n)) {
            return fail(err, errlen, HQ_ERR_INVALID, "gate rows must be contiguous and 32-byte aligned");
        }
    }
    hq::SituParams sp{};
    sp.q = static_cast<uint8_t*>(out_q);
    sp.sf = static_cast<uint8_t*>(out_sf);
    sp.ldq = ldq;
    sp.kb_out = int(kb_out);
    sp.gate = static_cast<const __nv_bfloat16*>(gate);
    sp.gate_ld = gate_ld;
    sp.valid_rows = int(m);
    return hq::grouped_gemm_impl(hq::kGroupBatch, a, b, sfa, sfb, out_q, bias, nullptr, nullptr, batches, m,
                                 batches * m, n, k, sfa_bytes, sfb_bytes, ldq / 2, HQ_MODE_W8A8_MXFP8, epilogue, &sp,
                                 sm_count, use_pdl, device, stream, err, errlen);
}

extern "C" int hq_group_masked_gemm(const void* a, const void* b, const void* sfa, const void* sfb,
                                    const int32_t* masked_m, void* out, const void* bias, const float* alpha,
                                    int64_t num_experts, int64_t max_m_per_expert, int64_t n, int64_t k,
                                    int64_t sfa_bytes, int64_t sfb_bytes, int64_t ldo, int mode, int sm_count,
                                    int use_pdl, int device, void* stream, char* err, size_t errlen) {
    if (max_m_per_expert <= 0) {
        return hq::fail(err, errlen, HQ_ERR_INVALID, "max_m_per_expert must be greater than 0, got %lld",
                        (long long)max_m_per_expert);
    }
    return hq::grouped_gemm_impl(hq::kGroupMasked, a, b, sfa, sfb, out, bias, alpha, masked_m, num_experts,
                                 max_m_per_expert, num_experts * max_m_per_expert, n, k, sfa_bytes, sfb_bytes,
                                 ldo, mode, HQ_EPILOGUE_IDENTITY, nullptr, sm_count, use_pdl, device, stream, err, errlen);
}

extern "C" int hq_group_contiguous_gemm(const void* a, const void* b, const void* sfa, const void* sfb,
                                        const int32_t* expert_ids, void* out, const void* bias,
                                        const float* alpha, int64_t num_experts, int64_t m, int64_t n, int64_t k,
                                        int64_t sfa_bytes, int64_t sfb_bytes, int64_t ldo, int mode, int sm_count,
                                        int use_pdl, int device, void* stream, char* err, size_t errlen) {
    // the reference sizes its tiles by the mean rows per expert (csrc/kernel/gemm/group_contiguous_gemm.cu:80-87)
    const int64_t rows = num_experts > 0 ? m / num_experts : 0;
    if (num_experts > 0 && m > 0 && rows == 0) {
        return hq::no_group_tile(err, errlen, hq::kGroupContiguous, mode, rows, m, n, k);
    }
    return hq::grouped_gemm_impl(hq::kGroupContiguous, a, b, sfa, sfb, out, bias, alpha, expert_ids, num_experts,
                                 rows, m, n, k, sfa_bytes, sfb_bytes, ldo, mode, HQ_EPILOGUE_IDENTITY, nullptr, sm_count,
                                 use_pdl, device, stream, err, errlen);
}

extern "C" int hq_low_latency_gemm(const void* a, const void* b, const void* sfa, const void* sfb, void* out,
                                   const void* a2, const void* b2, const void* sfa2, const void* sfb2, void* out2,
                                   int64_t m, int64_t n, int64_t n2, int64_t k1, int64_t k2, int64_t sfa_stride,
                                   int64_t sfb_stride, int64_t sfa2_stride, int64_t sfb2_stride, int64_t ldo,
                                   int64_t ldo2, int use_sigmoid, int sm_count, int use_pdl, int device,
                                   void* stream, char* err, size_t errlen) {
    using hq::fail;
    const bool concat = a2 != nullptr;
    const bool dual = out2 != nullptr;
    const bool second_weight = b2 != nullptr;
    // same rules and texts as the reference's ResolveLlShapes (csrc/kernel/gemm/low_latency_utils.cuh:222-273)
    if ((a2 != nullptr) != (sfa2 != nullptr) || second_weight != (sfb2 != nullptr) || second_weight != (concat != dual)) {
        return fail(err, errlen, HQ_ERR_INVALID, "weight2 / sfb2 must come with either input2 / sfa2 or output2");
    }
    if (use_sigmoid && second_weight) {
        return fail(err, errlen, HQ_ERR_INVALID, "low_latency_mma_gemm use_sigmoid does not support input2 or output2");
    }
    if (m < 0 || n < 0 || n2 < 0 || k1 < 0 || k2 < 0 || n > INT32_MAX || n2 > INT32_MAX || k1 > INT32_MAX ||
        k2 > INT32_MAX) {
        return fail(err, errlen, HQ_ERR_INVALID, "problem sizes must be non-negative and below 2^31");
    }
    if (!dual) n2 = 0;
    if (!concat) k2 = 0;
    if (m > 16) return fail(err, errlen, HQ_ERR_INVALID, "low_latency_mma_gemm supports M <= 16, got M=%lld", (long long)m);
    if (n % 8 != 0 || n2 % 8 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID, "low_latency_mma_gemm weight rows must be divisible by 8, got %lld and %lld",
                    (long long)n, (long long)n2);
    }
    if ((k1 + k2) % 256 != 0 || k1 % 128 != 0 || k2 % 128 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID, "low_latency_mma_gemm K must be divisible by 256, got K=%lld",
                    (long long)(k1 + k2));
    }
    if (concat && k1 % 512 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID, "concat-K K1 must be a multiple of 512, got K1=%lld", (long long)k1);
    }
    const int64_t kb2 = dual ? k1 / 32 : k2 / 32;  // scale columns of sfb2
    if (sfa_stride % 16 != 0 || sfb_stride % 16 != 0 || sfa_stride < k1 / 32 || sfb_stride < k1 / 32 ||
        (concat && (sfa2_stride % 16 != 0 || sfa2_stride < k2 / 32)) ||
        (second_weight && (sfb2_stride % 16 != 0 || sfb2_stride < kb2))) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "sfa / sfb / sfa2 / sfb2 must be plain row-major [rows, K / 32] scales "
                    "(group_wise_quant(..., use_swizzle=False)) with a row stride that is a multiple of 16 bytes; "
                    "got row strides %lld, %lld, %lld, %lld",
                    (long long)sfa_stride, (long long)sfb_stride, (long long)sfa2_stride, (long long)sfb2_stride);
    }
    if (m == 0 || (n == 0 && n2 == 0) || k1 + k2 == 0) return HQ_OK;
    const hq::DeviceGuard guard(device);
    if (!guard.ok()) return fail(err, errlen, HQ_ERR_CUDA, "cannot select CUDA device %d", device);
    const int sm_all = hq_sm_count(device);
    const int sm = sm_count > 0 ? (sm_count < sm_all || sm_all == 0 ? sm_count : sm_all) : sm_all;
    if (sm <= 0) return fail(err, errlen, HQ_ERR_CUDA, "cannot query the SM count of device %d", device);
    if (a == nullptr || b == nullptr || sfa == nullptr || sfb == nullptr || out == nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID, "null pointer argument");
    }
    if (!hq::aligned(out, 16) || (dual && !hq::aligned(out2, 16)) || ldo % 8 != 0 || ldo < n ||
        (dual && (ldo2 % 8 != 0 || ldo2 < n2)) || !hq::aligned(sfa, 4) || !hq::aligned(sfb, 4) ||
        !hq::aligned(sfa2, 4) || !hq::aligned(sfb2, 4)) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "outputs must be 16-byte aligned with a row stride that is a multiple of 8 elements, scales "
                    "4-byte aligned");
    }

    // A dual output has rows, and a first weight that may be empty is still an operand: neither has
    // a tensor map of its own below that would refuse it.
    if ((dual && n2 == 0) || !hq::aligned(b, 16)) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "TMA descriptor encoding failed: input and weight must be 16-byte aligned, contiguous rows");
    }
    if (n == 0) {  // dual output with an empty first weight
        b = b2;
        sfb = sfb2;
        sfb_stride = sfb2_stride;
        out = out2;
        ldo = ldo2;
        n = n2;
        n2 = 0;
    }
    // The kernel of dense_gemm's small M, always on whole tiles: the result may not depend on sm_count,
    // which a split of K over several CTAs would.
    using C = hq::DecCfg<16>;
    hq::DecParams p{};
    hq::DecPlain<true> plain{};
    p.x_rows = int((m + 7) / 8 * 8);
    CUtensorMap tm_w, tm_x, tm_o;
    const bool second_out = dual && n2 > 0;  // (n2 has become n if the first weight is empty)
    const bool maps_ok =
        hq::make_tmap_ktiles(&tm_w, b, uint64_t(n), uint64_t(k1), hq::kDecRows, 2) &&
        hq::make_tmap_ktiles(&tm_x, a, uint64_t(m), uint64_t(k1), uint32_t(p.x_rows), 2) &&
        // (a form without a second weight or input gets the first one's map, which is then never used)
        (concat ? hq::make_tmap_ktiles(&plain.w2, b2, uint64_t(n), uint64_t(k2), hq::kDecRows, 2)
         : second_out ? hq::make_tmap_ktiles(&plain.w2, b2, uint64_t(n2), uint64_t(k1), hq::kDecRows, 2)
                      : (plain.w2 = tm_w, true)) &&
        (concat ? hq::make_tmap_ktiles(&plain.x2, a2, uint64_t(m), uint64_t(k2), uint32_t(p.x_rows), 2)
                : (plain.x2 = tm_x, true)) &&
        hq::make_tmap_2d(&tm_o, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, out, uint64_t(n), uint64_t(m), uint64_t(ldo) * 2, 32, 16,
                         CU_TENSOR_MAP_SWIZZLE_NONE) &&
        (second_out ? hq::make_tmap_2d(&plain.o2, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, out2, uint64_t(n2), uint64_t(m),
                                       uint64_t(ldo2) * 2, 32, 16, CU_TENSOR_MAP_SWIZZLE_NONE)
                    : (plain.o2 = tm_o, true));
    if (!maps_ok) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "TMA descriptor encoding failed: input and weight must be 16-byte aligned, contiguous rows");
    }
    plain.sfx = static_cast<const uint8_t*>(sfa);
    plain.sfw = static_cast<const uint8_t*>(sfb);
    plain.sfx2 = static_cast<const uint8_t*>(concat ? sfa2 : sfa);
    plain.sfw2 = static_cast<const uint8_t*>(second_weight ? sfb2 : sfb);
    plain.sfx_stride = sfa_stride;
    plain.sfw_stride = sfb_stride;
    plain.sfx2_stride = concat ? sfa2_stride : sfa_stride;
    plain.sfw2_stride = second_weight ? sfb2_stride : sfb_stride;
    plain.n2 = int(n2);
    plain.tiles1 = int((n + hq::kDecRows - 1) / hq::kDecRows);
    plain.ksteps1 = int(k1 / hq::kDecStepBytes);
    p.m = int(m);
    p.n = int(n);
    p.k_bytes = k1 + k2;
    p.epi_op = use_sigmoid ? HQ_EPILOGUE_SIGMOID : HQ_EPILOGUE_IDENTITY;
    p.plan.tiles = plain.tiles1 + int((n2 + hq::kDecRows - 1) / hq::kDecRows);
    p.plan.ksteps = int((k1 + k2) / hq::kDecStepBytes);
    p.plan.ctas = std::min(sm, p.plan.tiles);
    p.plan.aligned = 1;
    p.prefetch_steps = use_pdl != 0 ? hq::dec_prefetch_steps(p.plan, C::kWBytes) : 0;

    static hq::SmemOptIn opt_in;
    HQ_CUDA_TRY(opt_in.ensure(hq::gemm_decode_kernel<16, hq::kDealWhole, true>, C::kSmemBytes));
    HQ_CUDA_TRY(hq::launch(hq::gemm_decode_kernel<16, hq::kDealWhole, true>, dim3(p.plan.ctas), dim3(hq::kDecThreads + 32),
                           size_t(C::kSmemBytes), static_cast<cudaStream_t>(stream), use_pdl != 0, 1, tm_w, tm_x, tm_o, p,
                           plain));
    return HQ_OK;
}

extern "C" int hq_device_status(int device, void* stream, uint32_t* status, char* err, size_t errlen) {
    const hq::DeviceGuard guard(device);
    if (!guard.ok()) return hq::fail(err, errlen, HQ_ERR_CUDA, "cannot select CUDA device %d", device);
    HQ_CUDA_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    uint32_t host[4] = {0, 0, 0, 0};
    HQ_CUDA_TRY(cudaMemcpyFromSymbol(host, hq::g_status, sizeof(host)));
    if (host[0] != 0) {
        const uint32_t zero[4] = {0, 0, 0, 0};
        HQ_CUDA_TRY(cudaMemcpyToSymbol(hq::g_status, zero, sizeof(zero)));
    }
    if (status != nullptr) *status = host[0];
    if (host[0] != 0) {
        return hq::fail(err, errlen, HQ_ERR_DEVICE,
                        "a GEMM role gave up on a bounded wait (status 0x%x: 1 producer, 2 MMA, 4 epilogue)",
                        host[0]);
    }
    return HQ_OK;
}

extern "C" int hq_selftest_bounded_wait(uint32_t limit_us, int device, void* stream, char* err, size_t errlen) {
    if (limit_us == 0 || limit_us > 100000u) {
        return hq::fail(err, errlen, HQ_ERR_INVALID, "limit_us must be in [1, 100000], got %u", limit_us);
    }
    const hq::DeviceGuard guard(device);
    if (!guard.ok()) return hq::fail(err, errlen, HQ_ERR_CUDA, "cannot select CUDA device %d", device);
    HQ_CUDA_TRY(hq::launch(hq::wait_selftest_kernel, dim3(1), dim3(96), size_t(0), static_cast<cudaStream_t>(stream),
                           false, 1, uint64_t(limit_us) * 1000ull));
    return HQ_OK;
}

extern "C" int hq_dense_gemm_allgather(const void* a, const void* b, const void* sfa, const void* sfb,
                                       void* const* outs, int world, int rank, int64_t m, int64_t n_local, int64_t k,
                                       int64_t sfa_bytes, int64_t sfb_bytes, int64_t ldo, int sm_count, int use_pdl,
                                       int device, void* stream, char* err, size_t errlen) {
    using hq::fail;
    if (world < 1 || world > 8 || rank < 0 || rank >= world || outs == nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID, "world must be 1..8 with 0 <= rank < world and one output per rank, got "
                                                 "world=%d rank=%d", world, rank);
    }
    if (m < 1 || n_local < 1 || k < 1 || m > INT32_MAX || n_local * world > INT32_MAX || k > INT32_MAX) {
        return fail(err, errlen, HQ_ERR_INVALID, "input must be a 2D tensor of shape [M, K]");
    }
    if (n_local % 256 != 0 || k % 128 != 0 || m <= 128) {
        return fail(err, errlen, HQ_ERR_UNSUPPORTED,
                    "the fused all-gather runs on the 256x256 2-CTA tile: N per rank must be a multiple of 256, K of "
                    "128 and M > 128, got M=%lld N=%lld K=%lld", (long long)m, (long long)n_local, (long long)k);
    }
    const int64_t sf_k = k / 32;
    if (sfa_bytes < hq_sf_rows(m) * sf_k || sfb_bytes < hq_sf_rows(n_local) * sf_k) {
        return fail(err, errlen, HQ_ERR_INVALID, "sfa / sfb must hold whole 128-row SfAtoms");
    }
    if (ldo < n_local * world || ldo % 8 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID, "the outputs are [M, world * N] matrices: row stride %lld is too small "
                                                 "or not a multiple of 8", (long long)ldo);
    }
    for (int r = 0; r < world; ++r) {
        if (outs[r] == nullptr || !hq::aligned(outs[r], 16)) {
            return fail(err, errlen, HQ_ERR_INVALID, "output %d is null or not 16-byte aligned", r);
        }
    }
    if (a == nullptr || b == nullptr || sfa == nullptr || sfb == nullptr || !hq::aligned(a, 16) || !hq::aligned(b, 16) ||
        !hq::aligned(sfa, 16) || !hq::aligned(sfb, 16)) {
        return fail(err, errlen, HQ_ERR_INVALID, "operands and scales must be non-null and 16-byte aligned");
    }
    const hq::DeviceGuard guard(device);
    if (!guard.ok()) return fail(err, errlen, HQ_ERR_CUDA, "cannot select CUDA device %d", device);
    const int sm_all = hq_sm_count(device);
    const int sm = sm_count > 0 ? (sm_count < sm_all || sm_all == 0 ? sm_count : sm_all) : sm_all;
    if (sm <= 0) return fail(err, errlen, HQ_ERR_CUDA, "cannot query the SM count of device %d", device);
    hq::GemmArgs g;
    g.a = a;
    g.b = b;
    g.sfa = static_cast<const uint8_t*>(sfa);
    g.sfb = static_cast<const uint8_t*>(sfb);
    g.alpha = nullptr;
    g.bias = nullptr;
    g.epi_op = HQ_EPILOGUE_IDENTITY;
    g.situ = hq::SituParams{};
    // this rank's own copy: columns [rank * n_local, (rank + 1) * n_local) of its [M, ldo] output
    g.out = static_cast<__nv_bfloat16*>(outs[rank]) + int64_t(rank) * n_local;
    g.ldo = ldo;
    g.m = int(m);
    g.n = int(n_local);
    g.grp = hq::GroupParams{hq::kGroupDense, 1, 0, nullptr};
    g.k_bytes = k;
    g.kq_dim = int(sf_k / 4);
    g.sm_count = sm;
    g.pdl = use_pdl != 0;
    g.direct_store = false;
    g.stream = static_cast<cudaStream_t>(stream);
    __nv_bfloat16* peers[8];
    int count = 0;
    for (int r = 0; r < world; ++r) {
        if (r != rank) peers[count++] = static_cast<__nv_bfloat16*>(outs[r]) + int64_t(rank) * n_local;
    }
    return hq::launch_pair<256, 0, true>(g, err, errlen, peers, count);
}

extern "C" int hq_dense_gemm_small_m_noalloc(const void* a, const void* b, const void* sfa, const void* sfb, void* out,
                                             int64_t m, int64_t n, int64_t k, int64_t sfa_bytes, int64_t sfb_bytes,
                                             int64_t ldo, int epilogue, int sm_count, int use_pdl, int device,
                                             void* stream, char* err, size_t errlen) {
    using hq::fail;
    if (epilogue != HQ_EPILOGUE_IDENTITY && epilogue != HQ_EPILOGUE_SIGMOID) {
        return fail(err, errlen, HQ_ERR_UNSUPPORTED, "Unsupported epilogue %d for w8a8-mxfp8", epilogue);
    }
    if (m < 0 || n < 0 || k < 0 || n > INT32_MAX || k > INT32_MAX) {
        return fail(err, errlen, HQ_ERR_INVALID, "input must be a 2D tensor of shape [M, K]");
    }
    if (m > hq::kNoAllocMaxM) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "hq_dense_gemm_small_m_noalloc takes at most %d activation rows (its scratch memory is a fixed "
                    "array), got M=%lld; use hq_dense_gemm", hq::kNoAllocMaxM, (long long)m);
    }
    if ((n + 127) / 128 > hq::kNoAllocMaxTiles) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "hq_dense_gemm_small_m_noalloc takes at most %d weight rows (one counter per 128 rows in a "
                    "fixed array), got N=%lld; use hq_dense_gemm", hq::kNoAllocMaxTiles * 128, (long long)n);
    }
    if (m == 0 || n == 0) return HQ_OK;
    if (k % 128 != 0 || n % 64 != 0 || k == 0) {
        return fail(err, errlen, HQ_ERR_INVALID, "No dense w8a8-mxfp8 tile for M=%lld (grid M=%lld), N=%lld, K=%lld",
                    (long long)m, (long long)m, (long long)n, (long long)k);
    }
    const int64_t sf_k = k / 32;
    if (sfa_bytes < hq_sf_rows(m) * sf_k || sfb_bytes < hq_sf_rows(n) * sf_k) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "sfa / sfb must hold whole 128-row SfAtoms: expected at least %lld and %lld elements, got %lld "
                    "and %lld", (long long)(hq_sf_rows(m) * sf_k), (long long)(hq_sf_rows(n) * sf_k),
                    (long long)sfa_bytes, (long long)sfb_bytes);
    }
    const hq::DeviceGuard guard(device);
    if (!guard.ok()) return fail(err, errlen, HQ_ERR_CUDA, "cannot select CUDA device %d", device);
    const int sm_all = hq_sm_count(device);
    const int sm = sm_count > 0 ? (sm_count < sm_all || sm_all == 0 ? sm_count : sm_all) : sm_all;
    if (sm <= 0) return fail(err, errlen, HQ_ERR_CUDA, "cannot query the SM count of device %d", device);
    if (a == nullptr || b == nullptr || sfa == nullptr || sfb == nullptr || out == nullptr) {
        return fail(err, errlen, HQ_ERR_INVALID, "null pointer argument");
    }
    if (!hq::aligned(a, 16) || !hq::aligned(b, 16) || !hq::aligned(sfa, 16) || !hq::aligned(sfb, 16) ||
        !hq::aligned(out, 16) || ldo < n || ldo % 8 != 0) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "operands, scales and output must be 16-byte aligned and the output row stride a "
                    "multiple of 8 elements");
    }
    // the same deal of the work as hq_dense_gemm makes for this shape, capped by the array's size
    const hq::SwitchScope switches;
    hq::DecPlan plan = hq::decode_plan(m, n, k, sm);
    if (plan.ctas > hq::kNoAllocMaxCtas) {
        return fail(err, errlen, HQ_ERR_INVALID,
                    "hq_dense_gemm_small_m_noalloc runs on at most %d CTAs, this shape wants %d; pass a smaller sm_count",
                    hq::kNoAllocMaxCtas, plan.ctas);
    }
    hq::GemmArgs g;
    g.a = a;
    g.b = b;
    g.sfa = static_cast<const uint8_t*>(sfa);
    g.sfb = static_cast<const uint8_t*>(sfb);
    g.alpha = nullptr;
    g.bias = nullptr;
    g.epi_op = epilogue;
    g.situ = hq::SituParams{};
    g.out = static_cast<__nv_bfloat16*>(out);
    g.ldo = ldo;
    g.m = int(m);
    g.n = int(n);
    g.grp = hq::GroupParams{hq::kGroupDense, 1, 0, nullptr};
    g.k_bytes = k;
    g.kq_dim = int(sf_k / 4);
    g.sm_count = sm;
    g.pdl = use_pdl != 0;
    g.direct_store = false;
    g.stream = static_cast<cudaStream_t>(stream);
    return m <= 16 ? hq::launch_decode_noalloc<16>(g, plan, err, errlen) : hq::launch_decode_noalloc<32>(g, plan, err, errlen);
}

extern "C" int hq_selftest_decode_plan(int64_t n, int64_t k, int sm_count, int force_split, char* err,
                                       size_t errlen) {
    if (n < 1 || k < 128 || k % 128 != 0 || sm_count < 1) {
        return hq::fail(err, errlen, HQ_ERR_INVALID, "n >= 1, k a positive multiple of 128 and sm_count >= 1 expected");
    }
    hq::DecClusterLimits nominal = {};
    nominal.max_active[2] = 74;
    nominal.max_active[4] = 36;
    nominal.max_active[8] = 14;
    hq::DecPlan p = hq::dec_plan(int(n), k, sm_count, true, 16, force_split != 0, hq::decode_ring_bytes(16), &nominal);
    if (force_split == 2) {
        // the general even deal: every CTA one contiguous run of units, whatever the tile boundaries
        const int64_t units = int64_t(p.tiles) * p.ksteps;
        p.ctas = int(units < sm_count ? units : sm_count);
        p.aligned = 0;
        p.cluster = 0;
        p.fits32 = units * p.ctas < (int64_t(1) << 32) ? 1 : 0;
    }
    if (!hq::dec_plan_selfcheck(p)) {
        return hq::fail(err, errlen, HQ_ERR_INVALID, "unit deal inconsistent: tiles=%d ksteps=%d ctas=%d aligned=%d",
                        p.tiles, p.ksteps, p.ctas, p.aligned);
    }
    return HQ_OK;
}

extern "C" const char* hq_version(void) { return "halops_b200 0.1 (sm_100a)"; }
