// wfa_tile.cuh -- what the register-tile WFA kernels share: the pair's sequences, tile
// geometry, record space, CIGAR runs and text, and the loop of a team over its pairs
// (wfa_tile.cu linear, wfa_affine_tile.cu gap-affine; the method is described there).
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "kernels.cuh"

namespace phr {
namespace {

constexpr int kNeg = -(1 << 30);   // an unset value word (any negative word is)
constexpr int kStay = 16;          // a block's diagonals moved are kept plus this
constexpr uint64_t kNoBase = ~0ull;

template <class S>
constexpr int sym_shift() {  // log2 of the bits per symbol
    return S::kBits == 2 ? 1 : 3;
}

// Symbols before the first set bit of x (kPerWord when x is zero): the bits below it are
// counted, one operation of the slow pipe instead of a reversal and a leading-zero count.
template <class S>
__device__ __forceinline__ int first_diff(uint32_t x) {
    return __popc((x - 1) & ~x) >> sym_shift<S>();
}

// Symbols before the first difference of three consecutive words.
template <class S>
__device__ __forceinline__ int first_diff3(uint32_t d0, uint32_t d1, uint32_t d2) {
    int n = first_diff<S>(d0);
    n += d0 == 0 ? first_diff<S>(d1) : 0;
    n += (d0 | d1) == 0 ? first_diff<S>(d2) : 0;
    return n;
}

// The CTA's dynamic shared memory: every access names it, so that loads through a call
// stay shared-memory loads.
extern __shared__ __align__(16) uint8_t tile_sm[];

// A pair's sequences: in shared memory as overlapping word pairs (entry i holds words i and
// i + 1, so one 64-bit load gives the 32 bits at any offset), or in global memory.
template <class S, bool STAGED>
struct PairSeq {
    uint32_t q2, t2;      // byte offsets in tile_sm (staged)
    const uint32_t* q;    // global words (otherwise)
    const uint32_t* t;
    __device__ __forceinline__ static uint64_t entry(uint32_t w2, uint32_t i) {
        return *reinterpret_cast<const uint64_t*>(tile_sm + w2 + i * 8);
    }
    __device__ __forceinline__ static uint32_t win(uint32_t w2, const uint32_t* w, int pos) {
        const uint32_t i = static_cast<uint32_t>(pos) / S::kPerWord;
        if constexpr (STAGED) {
            const uint64_t e = entry(w2, i);
            return __funnelshift_r(static_cast<uint32_t>(e), static_cast<uint32_t>(e >> 32),
                                   static_cast<uint32_t>(pos) << sym_shift<S>());
        } else {
            return __funnelshift_r(w[i], w[i + 1], static_cast<uint32_t>(pos) << sym_shift<S>());
        }
    }
    // XOR of the symbols from query position p and target position j on
    __device__ __forceinline__ uint32_t diff(int p, int j) const { return win(q2, q, p) ^ win(t2, t, j); }
    // three consecutive words from position pos on
    __device__ __forceinline__ static void win3(uint32_t w2, const uint32_t* w, int pos, uint32_t (&o)[3]) {
        const uint32_t i = static_cast<uint32_t>(pos) / S::kPerWord;
        const uint32_t sh = static_cast<uint32_t>(pos) << sym_shift<S>();
        uint32_t a, b, c, d;
        if constexpr (STAGED) {
            const uint64_t e = entry(w2, i), f = entry(w2, i + 2);
            a = static_cast<uint32_t>(e), b = static_cast<uint32_t>(e >> 32);
            c = static_cast<uint32_t>(f), d = static_cast<uint32_t>(f >> 32);
        } else {
            a = w[i], b = w[i + 1], c = w[i + 2], d = w[i + 3];
        }
        o[0] = __funnelshift_r(a, b, sh);
        o[1] = __funnelshift_r(b, c, sh);
        o[2] = __funnelshift_r(c, d, sh);
    }
    // symbols query and target share from (p, j) on, at most three words
    __device__ __forceinline__ int run3(int p, int j) const {
        uint32_t a[3], b[3];
        win3(q2, q, p, a);
        win3(t2, t, j, b);
        return first_diff3<S>(a[0] ^ b[0], a[1] ^ b[1], a[2] ^ b[2]);
    }
};

// Offset where the match run of diagonal k ends that goes on at offset v, at most hi. Three
// words a round, loaded together: runs between two edits mostly end in the first.
template <class S, bool STAGED>
__device__ __forceinline__ int extend_run(const PairSeq<S, STAGED>& sq, int v, int k, int hi, uint32_t& words) {
    while (v < hi) {
        ++words;
        const int n = sq.run3(v, v - k);
        v += n;
        if (n < 3 * S::kPerWord) break;
    }
    return min(v, hi);
}

// Longest common prefix from (p, j), at most lim, by the whole warp (warp-uniform
// arguments): one word first, then 32 words per round.
template <class S, bool STAGED>
__device__ __forceinline__ int warp_lcp(const PairSeq<S, STAGED>& sq, int p, int j, int lim) {
    if (lim <= 0) return 0;
    const uint32_t x0 = sq.diff(p, j);
    if (x0 != 0 || lim <= S::kPerWord) return min(first_diff<S>(x0), lim);
    const int lane = lane_id();
    for (int n = S::kPerWord; n < lim; n += 32 * S::kPerWord) {
        const int o = n + lane * S::kPerWord;
        const uint32_t x = o < lim ? sq.diff(p + o, j + o) : 0u;
        const unsigned b = __ballot_sync(PHR_FULL_MASK, x != 0);
        if (b) {
            const int src = __ffs(b) - 1;
            const int f = __shfl_sync(PHR_FULL_MASK, first_diff<S>(x), src);
            return min(n + src * S::kPerWord + f, lim);
        }
    }
    return lim;
}

// Diagonals a tile of R per lane keeps.
__host__ __device__ constexpr int tile_use(int R) { return 32 * R - 2 * kTileSteps; }

// Tiles of R diagonals per lane over a pair: diagonal 0 sits in the middle of tile nb.
template <int R>
struct TileGeom {
    static constexpr int use = tile_use(R);
    int qn, tn, nb;
    __device__ __forceinline__ TileGeom(int q, int t) : qn(q), tn(t), nb(t / use + 2) {}
    __device__ __forceinline__ int tile_of(int k) const { return static_cast<int>(static_cast<uint32_t>(k + use / 2 + nb * use) / use); }
    __device__ __forceinline__ int first(int g) const { return (g - nb) * use - use / 2; }   // first kept diagonal
    // first / last tile of a band of `half` diagonals to each side
    __device__ __forceinline__ int lo(int half) const { return tile_of(-min(half, tn)); }
    __device__ __forceinline__ int hi(int half) const { return tile_of(min(half, qn)); }
};

// Diagonals per lane for bands of `half` diagonals to each side, at most RMAX: few while the band is narrow, so that a
// team's warps share it and a score's chain is short; more as it widens, since the
// overlap of 16 diagonals per tile weighs less.
template <int W, int RMAX>
__device__ __forceinline__ int tile_regs(int half, int qn, int tn) {
    const int width = min(half, qn) + min(half, tn) + 1;
    if constexpr (W == 1) {
        // one warp does a block's tiles one after the other: the fewest diagonals computed
        // (tiles grow to both sides of diagonal 0: five of R = 4 beat three of R = 8)
        return width <= tile_use(1) ? 1
               : width <= tile_use(2) ? 2
               : RMAX == 4 || width <= tile_use(4) ? 4
               : width <= tile_use(8) || width > 5 * tile_use(4) ? 8 : 4;
    } else {
        // a tile per warp before tiles widen
        return width <= W * tile_use(1) ? 1
               : width <= W * tile_use(2) ? 2
               : RMAX == 4 || width <= W * tile_use(4) ? 4 : 8;
    }
}

// Calls f with R (1, 2, 4 or 8, at most RMAX) as a compile-time constant.
template <int RMAX, class F>
__device__ __forceinline__ void with_regs(int R, F&& f) {
    if (R == 1) f(std::integral_constant<int, 1>{});
    else if (R == 2) f(std::integral_constant<int, 2>{});
    else if (RMAX == 4 || R == 4) f(std::integral_constant<int, 4>{});
    else f(std::integral_constant<int, RMAX>{});
}

// A team's control block in shared memory. Its record chunks, of growing size, are taken from
// the launch's pool once and used again for each of the team's pairs.
constexpr int kMaxChunks = 40;
struct TileMin {   // what all of a team's warps reduce into
    unsigned long long end_key[2];   // smallest end cell, by parity of the score block
    int32_t reach;                   // furthest query offset
};
struct TileCtl {
    TileMin min;
    unsigned long long base[2];      // record block of this / the next kTileSteps scores
    unsigned long long cursor, chunk_end;   // free part of the record chunk in hand, bytes of P.scratch
    unsigned long long chunk[kMaxChunks];   // where the team's chunks start
    uint32_t chunk_size[kMaxChunks];        // in units of 256 bytes
    int32_t n_chunks, cur_chunk;
    uint32_t task;
    uint32_t defer[2];   // leave the pair to a cluster, by parity of the block
    uint32_t n_runs;
    uint32_t text_len[kBigThreads / 32];
};
static_assert(sizeof(TileCtl) <= kTileCtlBytes, "control block");

// Teams: one warp, the warps of one CTA (W = kCtaWarps), or those of a cluster of CTAs, whose
// control block is the first CTA's.
constexpr int kCtaWarps = kBigThreads / 32;

template <int W>
__device__ __forceinline__ void team_sync() {
    if constexpr (W == 1) {
        __syncwarp();
    } else if constexpr (W == kCtaWarps) {
        __syncthreads();
    } else {
        cooperative_groups::this_cluster().sync();
    }
}
template <int W>
__device__ __forceinline__ int team_rank() {   // CTA within the cluster
    return W <= kCtaWarps ? 0 : static_cast<int>(cooperative_groups::this_cluster().block_rank());
}
template <int W>
__device__ __forceinline__ int team_tid() {
    return W == 1 ? lane_id() : team_rank<W>() * kBigThreads + static_cast<int>(threadIdx.x);
}
// The thread that takes record space: the first CTA's last warp, which has a tile least often.
template <int W>
constexpr int alloc_tid() {
    return 32 * ((W < kCtaWarps ? W : kCtaWarps) - 1);
}

// Where a team reduces: its shared memory; a cluster in global memory (64-bit atomic minima
// on another CTA's shared memory lost updates), behind the pair's head.
template <int W>
__device__ __forceinline__ TileMin* team_min(TileCtl* sh, uint8_t* region, uint64_t fixed) {
    if constexpr (W <= kCtaWarps)
        return &sh->min;
    else
        return reinterpret_cast<TileMin*>(region + fixed - kTileHeadBytes / 2);
}

// Record block u of a pair: where it starts, in units of kRecordAlign bytes of P.scratch (30
// bits: any offset in a GPU's memory), and log2 of its tiles' diagonals per lane (1..8).
__device__ __forceinline__ uint32_t table_entry(uint64_t base, int R) {
    return static_cast<uint32_t>(base / kRecordAlign) << 2 | static_cast<uint32_t>(31 - __clz(R));
}
__device__ __forceinline__ uint64_t entry_base(uint32_t e) { return static_cast<uint64_t>(e >> 2) * kRecordAlign; }
__device__ __forceinline__ int entry_regs(uint32_t e) { return 1 << (e & 3u); }

// Record space for `bytes`, kNoBase when there is none (one thread of the team). New chunks
// double from A.chunk up to 256 times that.
__device__ __forceinline__ unsigned long long grab_records(const TileLaunch& A, TileCtl* sh, uint64_t bytes) {
    bytes = tile_align(bytes);   // table_entry's unit
    while (sh->cursor + bytes > sh->chunk_end) {
        const int i = sh->cur_chunk + 1;
        if (!A.pool_used || i >= kMaxChunks) return kNoBase;
        if (i >= sh->n_chunks) {
            const uint64_t size = max(static_cast<uint64_t>(A.chunk) << min(i, 8), bytes);
            const uint64_t o = atomicAdd(A.pool_used, static_cast<unsigned long long>(size));
            if (o + size > A.pool_end) return kNoBase;
            sh->chunk[i] = o;
            sh->chunk_size[i] = static_cast<uint32_t>(size >> 8);
            sh->n_chunks = i + 1;
        }
        sh->cur_chunk = i;
        sh->cursor = sh->chunk[i];
        sh->chunk_end = sh->cursor + (static_cast<uint64_t>(sh->chunk_size[i]) << 8);
    }
    const uint64_t o = sh->cursor;
    sh->cursor = o + bytes;
    return o;
}

// Lists a pair for a redo pass with `need` bytes of scratch of its own (one thread).
__device__ __forceinline__ void tile_redo(const ExtendParams& P, uint32_t pid, uint64_t need) {
    const uint32_t i = atomicAdd(P.redo_count, 1u);
    P.redo_list[i] = pid;
    atomicMax(P.redo_need_max, static_cast<unsigned long long>(need));
    if (P.redo_need) P.redo_need[i] = need;
}

// Forward-order CIGAR runs from the path's edits (edits[i], i = 1 .. n_edits: the match run
// after the edit << 2 | op, 1 mismatch, 2 query-extra, 3 target-extra) and the match run v0
// before the first, 32 edits at a time; returns their number. One warp.
__device__ uint32_t path_runs(const uint32_t* edits, uint32_t* cigar, int n_edits, int v0) {
    const int lane = lane_id();
    uint32_t nr = 0;
    if (v0 > 0) {
        if (lane == 0) cigar[0] = static_cast<uint32_t>(v0) << 2;
        nr = 1;
    }
    auto edit = [&](int i) -> uint32_t { return i <= n_edits ? edits[i] : 0u; };
    uint32_t word = edit(1 + lane);
    uint32_t last_op = 0;   // op and length so far of an edit run that goes on into this chunk (0: none)
    uint32_t open = 0;
    for (int base = 1; base <= n_edits; base += 32) {
        const uint32_t next = edit(base + 32 + lane);
        const uint32_t ops = word & 3u, my_n = word >> 2;
        // an edit run starts where a match came before or the op changes
        const uint32_t prev_op = __shfl_up_sync(PHR_FULL_MASK, ops, 1);
        const uint32_t prev_n = __shfl_up_sync(PHR_FULL_MASK, my_n, 1);
        const uint32_t first_next = __shfl_sync(PHR_FULL_MASK, next & 3u, 0);
        uint32_t next_op = __shfl_down_sync(PHR_FULL_MASK, ops, 1);
        if (lane == 31) next_op = first_next;
        const bool in = base + lane <= n_edits;
        const bool start = lane == 0 ? ops != last_op : (prev_n > 0 || prev_op != ops);
        const bool end = in && (my_n > 0 || base + lane == n_edits || next_op != ops);
        const unsigned starts = __ballot_sync(PHR_FULL_MASK, in && start);
        const unsigned ends = __ballot_sync(PHR_FULL_MASK, end);
        const unsigned match = __ballot_sync(PHR_FULL_MASK, in && my_n > 0);
        const unsigned below = (1u << lane) - 1u;
        const unsigned mine = starts & (below | (1u << lane));   // starts at or below this lane
        const uint32_t len = mine ? static_cast<uint32_t>(lane - (31 - __clz(mine)) + 1) : open + lane + 1;
        uint32_t at = nr + __popc(ends & below) + __popc(match & below);
        if (end) cigar[at++] = (len << 2) | (ops == 1 ? 1u : ops == 2 ? 3u : 2u);
        if (in && my_n > 0) cigar[at] = my_n << 2;
        nr += __popc(ends) + __popc(match);
        const bool closed = (ends >> 31) & 1u;
        open = closed ? 0u : __shfl_sync(PHR_FULL_MASK, len, 31);
        last_op = closed ? 0u : __shfl_sync(PHR_FULL_MASK, ops, 31);
        word = next;
    }
    return nr;
}

// Writes the runs as CIGAR text, a contiguous share per warp of the team; returns the
// text's length. `sh_len` holds a length per warp.
template <int W>
__device__ uint32_t format_runs(const uint32_t* runs, uint32_t nr, char* out, uint32_t* sh_len) {
    const int lane = lane_id();
    const int warp = W == 1 ? 0 : static_cast<int>(threadIdx.x) >> 5;
    const uint32_t share = (nr + W - 1) / W;
    const uint32_t from = min(nr, warp * share), to = min(nr, from + share);
    uint32_t base = 0, total = 0;
    if constexpr (W > 1) {
        uint32_t mine = 0;
        for (uint32_t c = from + lane; c < to; c += 32) mine += ndigits(runs[c] >> 2) + 1;
        mine = __reduce_add_sync(PHR_FULL_MASK, mine);
        if (lane == 0) sh_len[warp] = mine;
        team_sync<W>();
        for (int i = 0; i < W; ++i) {
            const uint32_t l = sh_len[i];
            if (i < warp) base += l;
            total += l;
        }
    }
    for (uint32_t c0 = from; c0 < to; c0 += 32) {
        const uint32_t c = c0 + lane;
        uint32_t len = 0, run = 0;
        if (c < to) {
            run = runs[c];
            len = ndigits(run >> 2) + 1;
        }
        const uint32_t incl = group_incl_scan(len, 32);
        if (c < to) {
            char* p = out + base + incl - len;
            uint32_t v = run >> 2;
            for (int dd = static_cast<int>(len) - 2; dd >= 0; --dd) {
                p[dd] = static_cast<char>('0' + v % 10);
                v /= 10;
            }
            p[len - 1] = op_char(run & 3);
        }
        base += __shfl_sync(PHR_FULL_MASK, incl, 31);
    }
    return W == 1 ? base : total;
}

// Stages a sequence as overlapping word pairs.
__device__ __forceinline__ void stage_pairs(uint64_t* dst, const uint32_t* src, int words, int tid, int nthr) {
    for (int i = tid; i < words; i += nthr) {
        const uint32_t a = __ldg(src + i), b = __ldg(src + i + 1);
        dst[i] = (static_cast<uint64_t>(b) << 32) | a;
    }
}

// Persistent loop of one team of W warps over the launch's tasks (W > kCtaWarps: over the
// deferred pairs); Algo aligns a pair.
template <class S, int W, class Algo>
__device__ __forceinline__ void tile_team(const ExtendParams& P, const TileLaunch& A, uint32_t sm_off, uint32_t sm_bytes) {
    constexpr bool kResume = W > kCtaWarps;
    const int tid = team_tid<W>();
    TileCtl* sh = reinterpret_cast<TileCtl*>(tile_sm + sm_off);
    if constexpr (kResume) sh = cooperative_groups::this_cluster().map_shared_rank(sh, 0);
    const uint32_t body_off = sm_off + kTileCtlBytes;
    uint8_t* body = tile_sm + body_off;
    const uint32_t body_bytes = sm_bytes - kTileCtlBytes;
    const uint32_t first = kResume ? 0u : P.tasks.range[0], last = kResume ? *A.defer_count : P.tasks.range[1];
    if (tid == 0) sh->n_chunks = 0;
    for (;;) {
        if (tid == 0) sh->task = first + atomicAdd(P.queue_head, 1u);
        team_sync<W>();
        const uint32_t task = sh->task;
        team_sync<W>();
        if (task >= last) break;
        uint32_t pid;
        if constexpr (kResume) {
            pid = static_cast<uint32_t>(A.defer_list[task]);
        } else {
            if (P.task_off && (P.tasks.task_group[task] & kOtherKernel) != (W == 1 ? kWarpTileTask : kCtaTileTask)) continue;
            pid = P.tasks.order[P.tasks.task_first[task]];
        }
        const PairDesc d = P.desc[pid];
        if (d.mode != (S::kBits == 2 ? 0 : 1)) continue;
        // the pair's fixed part and records: its own region (redo), or the team's chunks. A
        // cluster takes new chunks for every pair: what one of its CTAs has read before, and
        // may hold in its L1, is never written again.
        const uint64_t fixed = Algo::fixed_bytes(d.qn, d.tn);
        if (tid == 0) {
            sh->cur_chunk = -1;
            sh->cursor = sh->chunk_end = 0;
            if (kResume) sh->n_chunks = 0;
            if (P.task_off) {
                sh->cursor = P.task_off[task];
                sh->chunk_end = sh->cursor + (P.task_len[task] & ~15ull);
            }
            if (!kResume) sh->base[0] = grab_records(A, sh, fixed);
        }
        team_sync<W>();
        const unsigned long long at = kResume ? (A.defer_list[task] >> 32) * 256 : sh->base[0];
        team_sync<W>();
        if (at == kNoBase) {   // uniform over the team
            if (tid == 0) tile_redo(P, pid, fixed + Algo::hist_bytes(Algo::score_est(d.qn, d.mode)));
            continue;
        }
        uint8_t* region = P.scratch + at;
        const uint32_t* gq = (S::kBits == 2 ? P.packed2 : P.bytes) + d.q_word;
        const uint32_t* gt = (S::kBits == 2 ? P.packed2 : P.bytes) + d.t_word;
        const int qw = (d.qn + S::kPerWord - 1) / S::kPerWord, tw = (d.tn + S::kPerWord - 1) / S::kPerWord;
        // lanes on diagonals outside [-tn, qn] read up to a tile past a sequence's end
        constexpr int pad = kTileMax / S::kPerWord + 2;
        const uint64_t seq_bytes = (static_cast<uint64_t>(qw) + tw + 2 * pad) * 8;
        if (seq_bytes + 4 * kTileMax * 4 <= body_bytes) {
            uint64_t* q2 = reinterpret_cast<uint64_t*>(body);
            uint64_t* t2 = q2 + qw + pad;
            constexpr int nthr = W == 1 ? 32 : kBigThreads;   // each CTA of a cluster stages both
            const int t = W == 1 ? tid : static_cast<int>(threadIdx.x);
            stage_pairs(q2, gq, qw, t, nthr);
            stage_pairs(t2, gt, tw, t, nthr);
            team_sync<W>();
            const PairSeq<S, true> sq{body_off, body_off + (qw + pad) * 8, gq, gt};
            const int fcap = static_cast<int>((body_bytes - seq_bytes) / 4);
            Algo::template pair<S, true, W>(P, A, pid, d, sq, region, reinterpret_cast<int32_t*>(body + seq_bytes), fcap, sh);
        } else {
            const PairSeq<S, false> sq{0, 0, gq, gt};
            const int fcap = static_cast<int>(body_bytes / 4);
            Algo::template pair<S, false, W>(P, A, pid, d, sq, region, reinterpret_cast<int32_t*>(body), fcap, sh);
        }
    }
}

// Whether most SMs have run out of pairs (one thread): each CTA that found the queue empty
// has moved its head past the end.
__device__ __forceinline__ bool tile_sms_idle(const ExtendParams& P, const TileLaunch& A) {
    const int past = static_cast<int>(*reinterpret_cast<const volatile uint32_t*>(P.queue_head) + P.tasks.range[0] -
                                      P.tasks.range[1]);
    const int busy = static_cast<int>(gridDim.x) - max(past, 0);
    return busy * 4 <= A.sm_count;
}

// Leaves a pair for the cluster launch: what it has stays where it is, so the team starts
// over with new chunks (one thread).
__device__ __forceinline__ void tile_defer(const ExtendParams& P, const TileLaunch& A, TileCtl* sh, uint32_t pid,
                                           uint8_t* region, uint64_t fixed, const TileHead& head) {
    *reinterpret_cast<TileHead*>(region + fixed - kTileHeadBytes) = head;
    const uint32_t i = atomicAdd(A.defer_count, 1u);
    A.defer_list[i] = static_cast<unsigned long long>((region - P.scratch) / 256) << 32 | pid;
    sh->n_chunks = 0;
}

// Launch of `teams` clusters of `ctas` CTAs each.
struct ClusterLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr = {};
    template <class K>
    ClusterLaunch(K kernel, int teams, int ctas, uint32_t smem, cudaStream_t st) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBigSmemMax);
        if (ctas > 8) cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cfg.gridDim = dim3(static_cast<unsigned>(teams * ctas));
        cfg.blockDim = dim3(kBigThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = static_cast<unsigned>(ctas);
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
    ClusterLaunch(const ClusterLaunch&) = delete;
};

// Launches a cluster kernel, `ctas` CTAs per team, at most as many teams as fit at once.
template <class K>
inline void launch_clusters(K kernel, const ExtendParams& p, const TileLaunch& a, int pairs, int ctas, cudaStream_t st) {
    const int most = a.sm_count / ctas > 0 ? a.sm_count / ctas : 1;
    ClusterLaunch l(kernel, pairs < most ? pairs : most, ctas, p.big_smem, st);
    cudaLaunchKernelEx(&l.cfg, kernel, p, a);
}

// Whether the device can hold one such cluster.
template <class K>
inline bool cluster_fits(K kernel, int ctas, uint32_t smem) {
    ClusterLaunch l(kernel, 1, ctas, smem, nullptr);
    int n = 0;
    const bool ok = cudaOccupancyMaxActiveClusters(&n, kernel, &l.cfg) == cudaSuccess && n > 0;
    cudaGetLastError();   // a size the device does not know is an answer, not a failure
    return ok;
}

}  // namespace
}  // namespace phr
