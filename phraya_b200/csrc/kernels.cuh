// kernels.cuh -- parameter blocks and launchers shared by the engine's .cu files.
#pragma once

#include "common.cuh"

namespace phr {

// Work list of one extension pass. Pairs are referenced through `order` (sorted by
// bucket and length); task i covers order[task_first[i] .. task_first[i] + task_count[i])
// and is run by one warp split into groups of task_group[i] lanes (one pair per group).
struct TaskList {
    const uint32_t* order;
    const uint32_t* task_first;
    const uint8_t* task_count;
    const uint8_t* task_group;
    const uint32_t* range;   // device {begin, end} of the tasks this launch runs
};

struct ExtendParams {
    const PairDesc* desc;
    PairOut* out;
    const uint32_t* packed2;    // 2-bit arena
    const uint32_t* bytes;      // byte arena (raw input, as words)
    char* text;                 // CIGAR staging text
    const uint64_t* text_off;   // per-pair staging offset
    TaskList tasks;
    uint32_t* queue_head;       // persistent-kernel work counter (zeroed before launch)
    uint8_t* scratch;           // per-warp slots
    uint64_t slot_bytes;
    uint32_t* redo_list;        // pairs whose scratch need exceeded the slot / band
    uint32_t* redo_count;
    unsigned long long* redo_need_max;
    unsigned long long* redo_need;   // need of redo_list[k] (same index), may be NULL
    const uint64_t* task_off;   // when set: task t uses scratch + task_off[t] ...
    const uint64_t* task_len;   // ... with task_len[t] bytes (redo passes); else per-warp slots
    const uint64_t* task_need;  // estimated scratch need per task (main pass), may be NULL
    const uint32_t* pair_list;  // when set: the launch's tasks are these pairs, 32 lanes each
    int32_t engine;             // phr_engine
    int32_t full_band;          // Myers: store every block (no band)
    int32_t band_base;          // Myers: band half-width base
    phr_affine_costs costs;
    uint32_t* error_flag;       // set on an internal inconsistency (bounded loops ran out)
    int32_t big_min;            // linear WFA: pairs with qn+tn >= big_min run one per CTA (0: off)
    uint32_t big_smem;          // dynamic shared memory of the CTA-per-pair kernel (bytes)
    unsigned long long* work;   // [0] banded Myers block-columns, [1] pairs sent to redo,
                                // [2] WFA wavefront diagonals, [3] WFA LCP word compares
    int32_t lane_ckpt;          // banded Myers lane kernel: checkpoints + recomputed segments (1)
                                // or every column's records (0)
};

// task_group values marking a redo task for wfa.cu's CTA-per-pair kernel, the register tiles
// of one CTA and those of one warp (added to the lanes per pair, at most 32)
constexpr uint8_t kBigTask = 0x80;
constexpr uint8_t kCtaTileTask = 0xC0;
constexpr uint8_t kWarpTileTask = 0x40;
constexpr uint8_t kOtherKernel = 0xC0;   // mask of the three
constexpr int kBigThreads = 512;         // threads of a register-tile CTA (one CTA per SM)
// most threads per CTA of wfa.cu's gap-affine CTA-per-pair kernel, and its default (one CTA
// per SM; the "wfa_affine_big_threads" setting launches 512 or 256, two or four per SM)
constexpr int kBigAffineThreads = 1024;
// Largest "wfa_big_smem". A kernel's limit of dynamic shared memory belongs to the process, so
// every launch sets this one, whatever the context's own size: contexts of different sizes set
// and launched side by side otherwise.
constexpr int kBigSmemMax = 200 << 10;
constexpr uint32_t kBigMinFrameCells = 4096;  // smallest shared frame pair worth staging

// Shared-memory words the CTA-per-pair kernel needs for the two sequences of a pair:
// each is staged by a bulk copy from the 16-byte boundary at or below its first word
// (up to 3 leading words) to the next 16-byte boundary, plus one zero word after it
// (32-bit windows read one word past the last symbol), each copy starting 16-byte
// aligned in shared memory.
__host__ __device__ __forceinline__ uint64_t big_seq_words(int qn, int tn, int mode) {
    const int per = mode == 0 ? 16 : 4;
    return static_cast<uint64_t>((qn + per - 1) / per) + static_cast<uint64_t>((tn + per - 1) / per) + 16;
}

// A WFA pair long enough that one warp would be latency-bound on it: unless the register
// tiles take it (tile_warps below), it runs one per CTA of wfa.cu's kernels, in a redo pass.
__host__ __device__ __forceinline__ bool big_pair(int32_t engine, int32_t big_min, int qn, int tn) {
    return big_min > 0 && (engine == PHR_ENGINE_WFA_LINEAR || engine == PHR_ENGINE_WFA_AFFINE) && qn + tn >= big_min;
}

// Whether the gap-affine CTA kernel stages a big pair's sequences in its shared memory;
// longer ones are read from global memory.
__host__ __device__ __forceinline__ bool big_staged(uint32_t big_smem, int qn, int tn, int mode) {
    return (big_seq_words(qn, tn, mode) + 2ull * kBigMinFrameCells) * 4 <= big_smem;
}

// First-pass scratch estimate of one WFA pair: room for scores up to 64 + qn/8 (linear:
// 4 bytes of history per cell plus two value frames; affine: three layers of 8-byte
// cells). A pair that needs more overflows and is redone with what it asks for.
__host__ __device__ __forceinline__ uint64_t wfa_region_est(int qn, int tn, bool affine) {
    const uint64_t L = static_cast<uint64_t>(qn + tn);
    const uint64_t s = 64 + static_cast<uint64_t>(qn) / 8;
    if (affine) return (160ull << 10) + 512ull * L;
    const uint64_t cells = s + 2 * (s * s / 2);
    return 16 * L + 4 * cells + 4096;
}

// ---------------------------------------------------------------------------
// Lane-per-pair banded Myers (global mode, 2-bit pairs; myers_lane.cu).
//
// Band of one pair: every cell (i, j) of an alignment of cost ed satisfies
// |i - j| + |(m - i) - (n - j)| <= ed, i.e. its diagonal d = j - i lies in
// [min(0, n-m) - h, max(0, n-m) + h] with h = (ed - |n - m|) / 2. With E >= ed the
// band is [dmin, dmax] below (one spare diagonal each side for the rounding of h).
// A warp runs 32 pairs; its window covers the union of their bands and holds
// P = ceil((dmax - dmin + 127) / 64) query blocks of 64 rows per column (at most nb).
// ---------------------------------------------------------------------------
constexpr int kLaneMaxSlots = 8;
// Records of kLaneColGroup consecutive columns of one lane and slot are adjacent. One
// column per group measured fastest on B200: grouping two or four columns halves the
// traceback's sector reads but the forward pass's interleaved stores cost more.
constexpr int kLaneColGroup = 1;

struct LaneBand {
    int E;
    int dmin, dmax;
};

__host__ __device__ __forceinline__ LaneBand lane_band(int m, int n, int band_base) {
    const int delta = n - m;
    const int ad = delta < 0 ? -delta : delta;
    int E = band_base + ad + (m >> 4);
    if (E > m + n) E = m + n;
    const int h = (E - ad) >> 1;
    LaneBand b;
    b.E = E;
    b.dmin = (delta < 0 ? delta : 0) - h - 1;
    b.dmax = (delta > 0 ? delta : 0) + h + 1;
    return b;
}

__host__ __device__ __forceinline__ int lane_slots(int dmin, int dmax, int nb) {
    const int p = (dmax - dmin + 127 + 63) / 64;
    return p < nb ? p : nb;
}

// Whether a fitting-mode batch of n pairs gives its 2-bit pairs of up to kLaneMaxSlots blocks
// a lane each (every block in the window: nothing is banded) instead of a group of lanes.
// A lane takes the latency of its whole pair, so the batch has to fill the chip's lanes:
// windows of 100-300 bp, lanes against groups: 20,000 0.47 / 0.51 ms, 50,000 0.59 / 1.00,
// 200,000 1.12 / 3.21 (12,000, with lanes 20 % slower on large batches than now, 0.46 / 0.43).
constexpr uint64_t kFitLaneMin = 16384;
__host__ __device__ __forceinline__ bool fit_lanes(int32_t engine, uint64_t n, int32_t lane_ckpt) {
    return engine == PHR_ENGINE_MYERS_FIT && n >= kFitLaneMin && lane_ckpt;
}

// Columns per traceback segment of the checkpointed lane kernel: the forward pass keeps
// the window's {VP, VN} after every kSegCols-th column and the horizontal deltas that
// entered each block, the traceback recomputes one segment's columns of the two blocks its
// path is in. (Recomputing every block of the window, 8 columns took 13.43 ms per 1,000,000
// pairs of 64-2048 bp, 4 columns 13.76, 2 columns 15.90.)
constexpr int kSegCols = 8;

// Scratch of one lane task, then one reverse-run list of (m_max + n_max + 2) words per
// lane. Record mode: 16-byte {VP, HP} records [column group][slot][lane][column in
// group] of every column. Checkpoint mode: 16-byte {VP, VN} states [checkpoint][slot]
// [lane] after columns kSegCols, 2 kSegCols, ... below n_max, then the deltas that
// entered each block, two bits a column, [segment][slot][lane], and the query blocks' two
// bit planes [block][lane].
__host__ __device__ __forceinline__ uint64_t lane_ckpt_bytes(int n_max, int P) {
    const uint64_t nck = n_max > 0 ? static_cast<uint64_t>((n_max - 1) / kSegCols) : 0;
    return (nck * P * 512 + 255) & ~255ull;
}

__host__ __device__ __forceinline__ uint64_t lane_hin_bytes(int n_max, int P) {
    return (static_cast<uint64_t>((n_max + kSegCols - 1) / kSegCols) * P * 64 + 255) & ~255ull;
}

__host__ __device__ __forceinline__ uint64_t lane_rec_bytes(int n_max, int m_max, int P, int ckpt) {
    const uint64_t ng = static_cast<uint64_t>((n_max + kLaneColGroup - 1) / kLaneColGroup);
    return ckpt ? lane_ckpt_bytes(n_max, P) + lane_hin_bytes(n_max, P) + static_cast<uint64_t>((m_max + 63) / 64) * 512
                : ((ng * kLaneColGroup * P * 512 + 255) & ~255ull);
}

__host__ __device__ __forceinline__ uint64_t lane_task_need(int n_max, int m_max, int P, int ckpt = 0) {
    const uint64_t rec = lane_rec_bytes(n_max, m_max, P, ckpt);
    const uint64_t runs = (32ull * static_cast<uint64_t>(m_max + n_max + 2) * 4 + 255) & ~255ull;
    return rec + runs;
}

// Scratch of one pair in the warp-group Myers kernel with every block stored (redo).
__host__ __device__ __forceinline__ uint64_t myers_full_need(int m, int n) {
    const uint64_t nb = static_cast<uint64_t>((m + 63) >> 6);
    uint64_t need = (static_cast<uint64_t>(n) * nb * 16 + 15) & ~15ull;
    if (nb > 32) need += (static_cast<uint64_t>(n) + 15) & ~15ull;
    need += (static_cast<uint64_t>(m + n + 2) * 4 + 15) & ~15ull;
    return need;
}

// ---------------------------------------------------------------------------
// Linear WFA in register tiles, one CTA per long pair (wfa_tile.cu).
// ---------------------------------------------------------------------------
constexpr int kTileSteps = 8;                                  // scores a tile advances between barriers
constexpr int kTileRegs = 8;                                   // most diagonals per lane
constexpr int kTileMax = 32 * kTileRegs;                       // most diagonals of a tile
constexpr uint32_t kTileCtlBytes = 768;                         // a team's control block in shared memory

// The pool of a main-pass launch: bytes [0, pool_end) of the scratch buffer, taken by
// atomicAdd on pool_used. pool_used NULL (redo passes): every pair has its own region.
// A launch of one CTA per pair leaves a pair past step `defer_at` (0: never) where it is once
// no more than a quarter of the SMs have a pair, and lists it; a second launch with a
// cluster of CTAs per pair (resume) takes it up. One SM per pair to the end measured, for
// 1,000 long reads with a few unrelated windows of 10-40 kb among them, 50.7 ms, with
// clusters 22.8 ms; 200 gap-affine pairs of 4-16 kb 14.1 against 8.8 ms; one 10 kb
// pair (score 1,143, linear) 0.85 against 0.49 ms.
struct TileLaunch {
    unsigned long long* pool_used;
    uint64_t pool_end;
    uint32_t chunk;
    int32_t defer_at;
    int32_t sm_count;
    uint32_t* defer_count;
    unsigned long long* defer_list;   // region / 256 << 32 | pair
};

// Below this step a band is too narrow for more than one SM (one pair alone: left at step 96
// 0.49 ms, at 256 0.49, at 512 0.55).
constexpr int32_t kTileDeferStep = 256;

// How far a deferred pair got, kept in the last kTileHeadBytes of its fixed part.
struct TileHead {
    int32_t u, step, v0;   // block to go on with, its first step less one, the match run at score 0
};
constexpr uint64_t kTileHeadBytes = 256;

constexpr uint64_t kRecordAlign = 256;
__host__ __device__ __forceinline__ uint64_t tile_align(uint64_t v) { return (v + kRecordAlign - 1) & ~(kRecordAlign - 1); }
__host__ __device__ __forceinline__ uint64_t tile_runs_bytes(int qn, int tn) {
    return tile_align(4 * (static_cast<uint64_t>(qn) + tn + 2));
}
__host__ __device__ __forceinline__ uint64_t tile_table_bytes(int qn, int tn) {
    return tile_align(4 * ((static_cast<uint64_t>(qn) + tn) / kTileSteps + 3));
}
// What a pair takes before its first record: edits, CIGAR runs and two tables.
__host__ __device__ __forceinline__ uint64_t tile_fixed_bytes(int qn, int tn) {
    return 2 * tile_runs_bytes(qn, tn) + 2 * tile_table_bytes(qn, tn) + kTileHeadBytes;
}
// Upper bound of the records of scores up to s: block u holds 16 (u + 1) diagonals of 4
// bytes of value and at most 8 / 3 of ops, plus rounding to tiles and the narrow tiles of
// small bands.
__host__ __device__ __forceinline__ uint64_t tile_hist_bytes(int64_t s) {
    const uint64_t u = static_cast<uint64_t>(s) / kTileSteps + 1;
    return u * 3328 + 54 * u * (u + 1);
}
// The gap-affine tiles' counterparts. Steps are scores over g = gcd of the costs; an edit
// costs at least one, a mismatch two.
__host__ __device__ __forceinline__ uint64_t aff_tile_steps(int qn, int tn) {
    return 2 * (static_cast<uint64_t>(qn) + tn) + 16;
}
__host__ __device__ __forceinline__ uint64_t aff_tile_table_bytes(int qn, int tn) {
    return tile_align(4 * (aff_tile_steps(qn, tn) / kTileSteps + 3));
}
__host__ __device__ __forceinline__ uint64_t aff_tile_fixed_bytes(int qn, int tn) {
    return 2 * tile_runs_bytes(qn, tn) + 4 * aff_tile_table_bytes(qn, tn) + kTileHeadBytes;
}
// Block u: up to 16 (u + 1) diagonals at 28 bytes of values and at most 8 of ops.
__host__ __device__ __forceinline__ uint64_t aff_tile_hist_bytes(int64_t steps) {
    const uint64_t u = static_cast<uint64_t>(steps) / kTileSteps + 1;
    return u * 8320 + 288 * u * (u + 1);
}
// Costs the gap-affine tiles are specialised for, as (O + E) / g; 0: none. (2, 4, 1) gives 5,
// (4, 6, 2) gives 4.
__host__ __device__ __forceinline__ int aff_tile_open(phr_affine_costs c) {
    const int E = c.gap_extend;
    if (E <= 0 || c.mismatch != 2 * E || c.gap_open <= 0 || c.gap_open > (1 << 20)) return 0;
    const int oe = c.gap_open / E + 1;
    return c.gap_open % E == 0 && (oe == 4 || oe == 5) ? oe : 0;
}

// Score a pair is given room for at first: a quarter of the query for DNA, half for bytes
// (protein). Records come from a pool, so one pair may take more.
__host__ __device__ __forceinline__ int64_t tile_score_est(int qn, int mode) {
    return 64 + static_cast<int64_t>(qn) / (mode == 0 ? 4 : 2);
}
constexpr uint32_t kTileChunk = 64 << 10;   // first chunk a CTA takes from the pool, bytes
constexpr uint32_t kWarpTileChunk = 16 << 10;   // the same for a one-warp team
constexpr int kWarpTileThreads = 256;           // threads per CTA of the one-warp teams' kernel
constexpr uint32_t kWarpTileSmem = 12 << 10;    // shared memory of a one-warp team

// How many warps a WFA pair's register tiles get: 0 (the warp-group kernels, or wfa.cu's
// CTA kernel), 1, or kBigThreads / 32 (one CTA, long pairs). One warp: pairs from long_min
// on, and byte pairs (protein, which mostly differ a lot) from kWarpTileBytesMin on, where
// the warp-group kernel's frames in global memory cost more than a warp per pair: 5,000
// protein pairs of 200-800 at 30 % measured 1.9 + 1.6 ms (two passes) before and 0.78 ms
// now (linear). `open` is aff_tile_open for gap-affine pairs. Offsets are kept times 256
// (linear) or 1024 in 32 bits, hence the upper limits; longer pairs run one per CTA of
// wfa.cu's kernels (big_pair).
constexpr int kWarpTileBytesMin = 128;
constexpr int kTileMaxQuery = 1 << 22;   // a linear pair's query is shorter, its target below 2^27
__host__ __device__ __forceinline__ int tile_warps(int32_t engine, int open, int32_t big_min, int32_t long_min, int qn,
                                                   int tn, int mode) {
    const int64_t len = static_cast<int64_t>(qn) + tn;
    if (big_min <= 0 || tn >= (1 << 27)) return 0;
    if (engine == PHR_ENGINE_WFA_LINEAR) {
        if (qn >= kTileMaxQuery) return 0;
    } else if (engine != PHR_ENGINE_WFA_AFFINE || open == 0 || qn >= (1 << 20)) {
        return 0;
    }
    if (len >= big_min) return kBigThreads / 32;
    return len >= (mode == 0 ? long_min : kWarpTileBytesMin) ? 1 : 0;
}

void launch_myers(const ExtendParams& p, int grid, int block, cudaStream_t st);
constexpr int kLaneThreads = 256;   // most threads per block of the lane kernel
// Launch of the lane kernel over `warps` scratch slots, one per warp: never more warps than
// slots, whatever the block size of the other kernels.
struct LaneGrid {
    int blocks, threads;
};
__host__ __forceinline__ LaneGrid lane_grid(uint64_t warps, int sm_count, int blocks_per_sm) {
    const uint64_t per_block = warps < kLaneThreads / 32 ? warps : kLaneThreads / 32;
    const uint64_t most = static_cast<uint64_t>(sm_count) * blocks_per_sm, want = warps / per_block;
    return LaneGrid{static_cast<int>(want < most ? want : most), static_cast<int>(32 * per_block)};
}
void launch_myers_lane(const ExtendParams& p, LaneGrid g, cudaStream_t st);
// Resident blocks per SM of the lane kernel in each mode (its shared memory per warp).
int myers_lane_blocks_per_sm(int ckpt);
void launch_wfa_linear(const ExtendParams& p, int grid, int block, cudaStream_t st);
// Tasks per SM above which they run first in the kernel for short pairs alone, whose second
// launch and tail of the longest pairs need time to pay: pairs of 100-300 bp at 0-5 %, with
// it / without, 20,000 0.23 / 0.14 ms, 60,000 0.38 / 0.37, 90,000 0.52 / 0.55, 150,000
// 0.79 / 0.91, 1,000,000 4.43 / 5.72.
constexpr uint32_t kShortAffineMin = 512;
// The same for linear pairs (four a task): with it / without, 20,000 0.10 / 0.17 ms, 100,000
// 0.25 / 0.36, 1,000,000 2.08 / 3.01; below, the warps of one launch hold every task.
constexpr uint32_t kShortLinearMin = 16;
// The launch's linear or (costs aff_tile_open knows) gap-affine pairs, those of few symbols and
// edits, in `blocks_per_sm` CTAs a SM at most; the pairs it leaves go to left[0 .. *n_left).
// 0 CTAs: no room in the `scratch_bytes` of p.scratch, nothing launched.
int launch_wfa_short(const ExtendParams& p, uint64_t scratch_bytes, int sms, int blocks_per_sm, uint32_t* left,
                     uint32_t* n_left, cudaStream_t st);
void launch_wfa_affine(const ExtendParams& p, int grid, int block, cudaStream_t st);
void launch_wfa_linear_big(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st);
// The largest cluster of the resume kernels that the device can hold: 16 (not a portable size),
// 8, 4, or 1 for none. All of them are CTAs of kBigThreads threads, one per SM.
int wfa_cluster_fit(uint32_t smem);
// The size for `pairs` deferred pairs where up to `most` CTAs are allowed: the fewer the pairs,
// the more SMs each.
__host__ __forceinline__ int wfa_cluster_size(uint32_t pairs, int sm_count, int most) {
    const uint32_t sms = static_cast<uint32_t>(sm_count);
    const int want = pairs <= sms / 16 ? 16 : pairs <= sms / 8 ? 8 : 4;
    return want < most ? want : most;
}
// Deferred pairs of both symbol modes' launches, `ctas` (4, 8 or 16) CTAs per pair.
void launch_wfa_linear_resume(const ExtendParams& p, const TileLaunch& a, int pairs, int ctas, int mode, cudaStream_t st);
void launch_wfa_affine_resume(const ExtendParams& p, const TileLaunch& a, int pairs, int ctas, int mode, cudaStream_t st);
void launch_wfa_affine_cta_tiles(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st);
void launch_wfa_affine_warp_tiles(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st);
void launch_wfa_linear_tile(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st);
void launch_wfa_linear_long(const ExtendParams& p, int grid, int mode, cudaStream_t st);
void launch_wfa_affine_big(const ExtendParams& p, int grid, int threads, int mode, cudaStream_t st);

}  // namespace phr
