// wfa_tile.cu -- linear WFA of long pairs, wavefronts in register tiles (sm_100a).
//
// Semantics are those of wfa_linear_group (wfa.cu): fill_wfa wfa_simd.rs:231-345,
// fill_wfa_fitting_impl :360-482, traceback_wfa :959-1130; every value, op and tie-break
// is the same.
//
// What bounds it: a score's cells are a short dependent chain (three neighbours, one
// compare of 16 bases), so a pair is bound by that chain's latency while its wavefront is
// narrow and by the integer pipes once it is wide, one SM per pair. 200 pairs of 4-16 kb at
// up to 10 % divergence: 165 M band diagonals in 2.1 ms, 84 instructions a diagonal with the
// tiles' overlap, idle lanes and the traceback (issue 49 % on single CTAs, 27 % on
// clusters). 500 such pairs: 2.5 ms a call; with the kernel before it (one barrier per score,
// ~200 instructions per cell, frames and history of 32-bit words, a second pass for every
// pair that outgrew its first scratch) 15.2 ms.
//
// Tiles. A warp holds 32 R consecutive diagonals, lane l the diagonals l, l + 32, ... of
// the tile (neighbours are then one lane away, and the 32 lanes' sequence reads of one
// step fall on neighbouring words), and advances them kTileSteps scores in registers.
// A cell depends on its two neighbours one score back, so after h scores the outer h
// diagonals on each side are wrong: tiles overlap by kTileSteps diagonals on each side
// and only the inner ones are kept, and the team meets at one barrier per kTileSteps
// scores. R grows with the band from 1 to 8 (tile_regs): a narrow band is shared by all
// warps, a wide one recomputes few diagonals. 16 warps at 128 registers (one CTA per SM)
// measured 3.4 ms where two CTAs per SM at 64 registers, which spill, took 5.2 ms.
//
// History. The path through (score, diagonal) space is fixed by each cell's op alone, so
// two bits per cell are stored, plus, every kTileSteps scores, each diagonal's value word:
// the offset and the diagonal it came from kTileSteps scores before (carried along in the
// low bits of the value, where it costs nothing: the op bits above it decide every tie).
// The traceback then takes one dependent step per kTileSteps scores, and the blocks it
// passed are expanded in parallel, each from its own start offset, with every match run
// the longest common prefix again. Records come from a pool shared by the pairs of a
// launch, so a divergent pair uses what the others leave (a pair that still runs out is
// redone with scratch of its own).
#include "wfa_tile.cuh"

namespace phr {
namespace {

// A value word: offset << 8 | op << 6 | diagonals moved since the block's start + kStay.
constexpr int kLinRegs = 8;   // most diagonals per lane

// Record words of a tile's kTileSteps scores (two bits a cell), and the scores per word.
__host__ __device__ constexpr int rec_words(int R) { return R < 2 ? 1 : R * kTileSteps / 16; }
__host__ __device__ constexpr int rec_steps(int R) { return kTileSteps / rec_words(R); }

// Value words of a block of n tiles.
template <int R>
__device__ __forceinline__ uint64_t frame_bytes(int n) {
    return (static_cast<uint64_t>(n) * tile_use(R) * 4 + 127) & ~127ull;
}

// Advances tile g of one warp by kTileSteps scores, s0 + 1 .. s0 + kTileSteps. `cur` holds
// the value words of score s0 for diagonals [cur_lo, cur_hi); the kept diagonals' words go
// to `nxt` and `saved` (from diagonal nxt_lo on; one array when they are the same) and the
// ops to `rec`. FAR: `cur` was written by other SMs. Returns the smallest (score << 32 |
// k + tn) of a kept end cell, ~0 when there is none.
template <class S, bool STAGED, int R, bool FAR>
__device__ __forceinline__ unsigned long long lin_tile(const PairSeq<S, STAGED>& sq, const TileGeom<R>& G, int g, int s0,
                                                       bool fitting, const int32_t* cur, int cur_lo, int cur_hi,
                                                       int32_t* nxt, int32_t* saved, int nxt_lo, uint32_t* rec,
                                                       uint32_t& extra) {
    const int lane = lane_id();
    const int qn = G.qn, tn = G.tn;
    const int k0 = G.first(g) - kTileSteps + lane;   // this lane's first diagonal
    const int tk0 = tn + k0;
    int x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int k = k0 + 32 * r;
        x[r] = (k >= cur_lo && k < cur_hi) ? ((FAR ? __ldcg(cur + (k - cur_lo)) : cur[k - cur_lo]) & ~255) | kStay : kNeg;
    }
    // end cells: diagonal qn - tn alone (global), or any from there on (fitting)
    const int kend = qn - tn;
    const bool may_end = G.first(g) + G.use > kend && (fitting || G.first(g) <= kend);   // warp-uniform
    const int up_src = (lane + 31) & 31, dn_src = (lane + 1) & 31;
    unsigned long long best_key = ~0ull;
    uint32_t ops = 0;
#pragma unroll(R < 4 ? 4 / R : 1)
    for (int h = 0; h < kTileSteps; ++h) {
        uint32_t more = 0, acc = 0;
        int prev_up = kNeg;   // lane 31 of the slot below
        int old = x[0];
        int dn = __shfl_sync(PHR_FULL_MASK, x[0], dn_src);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            constexpr int kLast = R - 1;
            const int up_rot = __shfl_sync(PHR_FULL_MASK, old, up_src);
            const int dn_next = r < kLast ? __shfl_sync(PHR_FULL_MASK, x[r < kLast ? r + 1 : r], dn_src) : kNeg;
            const int up = lane == 0 ? prev_up : up_rot;
            const int down = lane == 31 ? dn_next : dn;
            prev_up = up_rot;
            dn = dn_next;
            // candidates in order [mismatch, ins, del], the LAST maximal one wins: the op
            // above the move decides ties
            const int best = __viaddmax_s32(up, (1 << 8) + (2 << 6) + 1,
                                            __viaddmax_s32(old, (1 << 8) + (1 << 6), down + (3 << 6) - 1));
            old = x[r < kLast ? r + 1 : r];
            const int pos = best >> 8;
            const int k = k0 + 32 * r;
            const int lo = __viaddmax_s32(k0, 32 * r, 0), hi = __viaddmin_s32(tk0, 32 * r, qn);
            const int lim = pos >= lo ? hi - pos : -1;   // symbols left on the diagonal; < 0: invalid cell
            int p, j;
            if constexpr (STAGED) {
                p = lim >= 0 ? pos : lo;   // reads stay within the staged padding
                j = p - k;
            } else {
                p = lim >= 0 ? pos : 0;
                j = lim >= 0 ? pos - k : 0;
            }
            const int n = min(first_diff<S>(sq.diff(p, j)), lim);
            x[r] = lim >= 0 ? ((p + n) << 8) + (best & 63) : kNeg;
            acc += static_cast<uint32_t>(best & (3 << 6)) << (2 * r);
            if (n == S::kPerWord) more |= 1u << r;
        }
        while (more) {   // match runs longer than one word
            const int r = __ffs(more) - 1;
            more &= more - 1;
            int v = x[0];
#pragma unroll
            for (int i = 1; i < R; ++i) v = r == i ? x[i] : v;
            const int k = k0 + 32 * r;
            v = (extend_run<S, STAGED>(sq, v >> 8, k, min(qn, tn + k), extra) << 8) + (v & 63);
#pragma unroll
            for (int i = 0; i < R; ++i) x[i] = r == i ? v : x[i];
        }
        if (may_end) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int in_tile = 32 * r + lane;
                const int k = k0 + 32 * r;
                if (x[r] >= (qn << 8) && in_tile >= kTileSteps && in_tile < kTileSteps + tile_use(R) &&
                    (fitting ? k >= kend : k == kend)) {
                    const unsigned long long key =
                        (static_cast<unsigned long long>(s0 + h + 1) << 32) | static_cast<unsigned>(k + tn);
                    best_key = min(best_key, key);
                }
            }
        }
        constexpr int kPer = rec_steps(R);   // scores per record word
        ops |= (acc >> 6) << (2 * R * (h % kPer));
        if ((h + 1) % kPer == 0) {
            rec[(h / kPer) * 32 + lane] = ops;
            ops = 0;
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int in_tile = 32 * r + lane;
        if (in_tile >= kTileSteps && in_tile < kTileSteps + tile_use(R)) {
            const int i = k0 + 32 * r - nxt_lo;
            nxt[i] = x[r];
            if (saved != nxt) saved[i] = x[r];
        }
    }
    return best_key;
}

// Diagonals of the bands of scores 1 .. s (the reference's scan ranges).
__device__ __forceinline__ uint64_t tile_band_cells(int qn, int tn, int64_t s) {
    auto tri = [&](int64_t x) { return s <= x ? s * (s + 1) / 2 : x * (x + 1) / 2 + (s - x) * x; };
    return static_cast<uint64_t>(s + tri(qn) + tri(tn));
}

// A team's share of the launch's scratch.
struct TileScratch {
    uint32_t* edits;    // the path's edits (one per score), each with the match run after it
    uint32_t* cigar;    // forward-order CIGAR runs
    int32_t* kpath;     // diagonal of the path after score kTileSteps u
    uint32_t* table;    // record block u (table_entry)
};

// Where block u of a pair keeps its value words and ops.
struct BlockAt {
    const int32_t* frame;    // value words from diagonal lo on
    const uint32_t* rec;     // ops, tile after tile
    int lo, glo;
};
template <int R>
__device__ __forceinline__ BlockAt block_at(const uint8_t* scratch, const uint32_t* table, int qn, int tn, int u) {
    const TileGeom<R> G(qn, tn);
    const int s_hi = (u + 1) * kTileSteps;
    BlockAt b;
    b.glo = G.lo(s_hi);
    b.lo = G.first(b.glo);
    const uint8_t* base = scratch + entry_base(table[u]);
    b.frame = reinterpret_cast<const int32_t*>(base);
    b.rec = reinterpret_cast<const uint32_t*>(base + frame_bytes<R>(G.hi(s_hi) - b.glo + 1));
    return b;
}

// Ops of block u's scores up to h_top (the last is kTileSteps - 1 but in the path's last
// block), the path at diagonal k after it; moves k to the block's start. Within a block the
// path moves at most one diagonal per score, and a tile's overlap is valid to exactly that
// depth, so the tile that keeps diagonal k holds the whole stretch. One lane.
template <int R>
__device__ __forceinline__ uint32_t block_ops(const BlockAt& b, const TileGeom<R>& G, int h_top, int& k) {
    const int g = G.tile_of(k);
    const int base = G.first(g) - kTileSteps;
    const uint32_t* rec = b.rec + static_cast<int64_t>(g - b.glo) * rec_words(R) * 32;
    uint32_t ops = 0;
#pragma unroll
    for (int h = kTileSteps - 1; h >= 0; --h) {
        if (h > h_top) continue;
        const int at = k - base;
        const uint32_t w = rec[(h / rec_steps(R)) * 32 + (at & 31)];
        const uint32_t op = (w >> (2 * ((h % rec_steps(R)) * R + (at >> 5)))) & 3u;
        ops |= op << (2 * h);
        k += op < 2 ? 0 : static_cast<int>(op) * 2 - 5;   // 2: from diagonal k - 1, 3: from k + 1
    }
    return ops;
}

// Follows the path back from block u_top's start (kpath[u_top]) block by block: the value
// word of the path's cell after block u says how far it moved in it. The words of the next
// blocks are fetched ahead for the 64 diagonals the path can have reached by then, so that
// the chain is a lookup per block and not a memory round trip. One warp; leaves kpath.
__device__ void walk_blocks(const uint8_t* scratch, const TileScratch& sc, int qn, int tn, int u_top) {
    constexpr int kAhead = 4;
    const int lane = lane_id();
    int k = sc.kpath[u_top];
    int w0[kAhead], w1[kAhead], mid[kAhead];
    auto fetch = [&](int u, int c, int& a, int& b) {   // words of diagonals c - 32 + lane, c + lane
        a = b = 0;
        if (u < 0) return;
        const uint32_t e = sc.table[u];
        with_regs<kLinRegs>(entry_regs(e), [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const TileGeom<R> G(qn, tn);
            const int s_hi = (u + 1) * kTileSteps;
            const int glo = G.lo(s_hi), lo = G.first(glo), hi = G.first(G.hi(s_hi) + 1);
            const int32_t* f = reinterpret_cast<const int32_t*>(scratch + entry_base(e));
            const int ka = c - 32 + lane, kb = c + lane;
            if (ka >= lo && ka < hi) a = f[ka - lo];
            if (kb >= lo && kb < hi) b = f[kb - lo];
        });
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i) {
        mid[i] = k;
        fetch(u_top - 1 - i, k, w0[i], w1[i]);
    }
    for (int u0 = u_top - 1; u0 >= 0; u0 -= kAhead) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int u = u0 - i;
            if (u >= 0) {
                const int o = k - mid[i] + 32;   // 0..63: at most kTileSteps diagonals a block
                const int a = __shfl_sync(PHR_FULL_MASK, w0[i], o & 31);
                const int b = __shfl_sync(PHR_FULL_MASK, w1[i], o & 31);
                k -= ((o < 32 ? a : b) & 63) - kStay;
                if (lane == 0) sc.kpath[u] = k;
                mid[i] = k;
                fetch(u - kAhead, k, w0[i], w1[i]);
            }
        }
    }
}

// Expands the path's blocks, one per thread of the team: their ops, and from the block's
// start offset the match run after every score.
template <class S, bool STAGED, int W>
__device__ void expand_blocks(const PairSeq<S, STAGED>& sq, const uint8_t* scratch, const TileScratch& sc, int qn, int tn,
                              int s_end, int k_end, int v0) {
    const int tid = W == 1 ? lane_id() : static_cast<int>(threadIdx.x);
    const int u_top = (s_end - 1) / kTileSteps;
    for (int u = tid; u <= u_top; u += 32 * W) {
        const int h_top = u == u_top ? (s_end - 1) % kTileSteps : kTileSteps - 1;
        int k = u == u_top ? k_end : sc.kpath[u + 1];
        uint32_t ops = 0;
        with_regs<kLinRegs>(entry_regs(sc.table[u]), [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            ops = block_ops<R>(block_at<R>(scratch, sc.table, qn, tn, u), TileGeom<R>(qn, tn), h_top, k);
        });
        int p = v0;
        if (u > 0)
            with_regs<kLinRegs>(entry_regs(sc.table[u - 1]), [&](auto rc) {
                const BlockAt b = block_at<decltype(rc)::value>(scratch, sc.table, qn, tn, u - 1);
                p = b.frame[k - b.lo] >> 8;
            });
        uint32_t words = 0;
        for (int h = 0; h <= h_top; ++h) {
            const uint32_t op = (ops >> (2 * h)) & 3u;
            p += op != 3;
            k += op == 2 ? 1 : op == 3 ? -1 : 0;
            const int e = extend_run<S, STAGED>(sq, p, k, min(qn, tn + k), words);
            sc.edits[u * kTileSteps + h + 1] = static_cast<uint32_t>(max(e - p, 0)) << 2 | op;
            p = max(e, p);
        }
    }
}

// The wavefront of a team's pair between two score blocks.
struct TileWave {
    const int32_t* cur;       // values of score s0, diagonals [cur_lo, cur_hi)
    int cur_lo, cur_hi;
    int u, s0;                // score block, its first score less one
    int state;                // 0 running, 1 end found, 2 out of records, 3 every score done, 4 deferred
    unsigned long long end;
    uint32_t extra;           // word compares beyond a cell's first
};

template <int R>
__device__ __forceinline__ uint64_t block_bytes(const TileGeom<R>& G, int u) {
    const int s_hi = (u + 1) * kTileSteps;
    const int n = G.hi(s_hi) - G.lo(s_hi) + 1;
    return frame_bytes<R>(n) + static_cast<uint64_t>(n) * rec_words(R) * 128;
}

// Score blocks of a pair while its tiles hold R diagonals per lane: the team's warps share
// the block's tiles, the last warp's first lane takes the next block's record space.
template <class S, bool STAGED, int W, int R>
__device__ __forceinline__ void lin_blocks(const ExtendParams& P, const TileLaunch& A, const PairSeq<S, STAGED>& sq,
                                           int qn, int tn, bool fitting, uint32_t* table, int32_t* frames, int fcap,
                                           TileCtl* sh, TileMin* tm, TileWave& w) {
    constexpr bool kFar = W > kCtaWarps;   // a cluster's values go through L2
    const int tid = team_tid<W>();
    const int warp = W == 1 ? 0 : tid >> 5;
    const TileGeom<R> G(qn, tn);
    do {
        const int s_hi = w.s0 + kTileSteps;
        const int glo = G.lo(s_hi), ghi = G.hi(s_hi);
        const int nxt_lo = G.first(glo), nxt_hi = G.first(ghi + 1);
        const unsigned long long base = sh->base[w.u & 1];
        if (base == kNoBase) {
            w.state = 2;
            return;
        }
        // the next score's values: in shared memory while they fit, else only in the record
        int32_t* saved = reinterpret_cast<int32_t*>(P.scratch + base);
        int32_t* nxt = !kFar && nxt_hi - nxt_lo <= fcap / 2 ? frames + ((w.u + 1) & 1) * (fcap / 2) : saved;
        uint32_t* rec = reinterpret_cast<uint32_t*>(P.scratch + base + frame_bytes<R>(ghi - glo + 1));
        unsigned long long key = ~0ull;
        for (int g = glo + warp; g <= ghi; g += W)
            key = min(key, lin_tile<S, STAGED, R, kFar>(sq, G, g, w.s0, fitting, w.cur, w.cur_lo, w.cur_hi, nxt, saved, nxt_lo,
                                                  rec + (g - glo) * rec_words(R) * 32, w.extra));
        if (key != ~0ull) atomicMin(&tm->end_key[w.u & 1], key);
        const bool more = tile_regs<W, kLinRegs>(s_hi + kTileSteps, qn, tn) == R;
        if (tid == alloc_tid<W>()) {
            table[w.u] = table_entry(base, R);
            uint64_t bytes = 0;
            if (more)
                bytes = block_bytes<R>(G, w.u + 1);
            else
                with_regs<kLinRegs>(tile_regs<W, kLinRegs>(s_hi + kTileSteps, qn, tn),
                          [&](auto rc) { bytes = block_bytes(TileGeom<decltype(rc)::value>(qn, tn), w.u + 1); });
            sh->base[(w.u + 1) & 1] = grab_records(A, sh, bytes);
            if (W == kCtaWarps && A.defer_at > 0) sh->defer[w.u & 1] = tile_sms_idle(P, A);
        }
        team_sync<W>();
        w.cur = nxt;
        w.cur_lo = nxt_lo;
        w.cur_hi = nxt_hi;
        w.s0 = s_hi;
        w.end = kFar ? __ldcg(&tm->end_key[w.u & 1]) : tm->end_key[w.u & 1];
        ++w.u;
        if (w.end != ~0ull)
            w.state = 1;
        else if (s_hi >= qn + tn)
            w.state = 3;
        else if (W == kCtaWarps && A.defer_at > 0 && s_hi >= A.defer_at && sh->defer[(w.u - 1) & 1])
            w.state = 4;
        if (!more) return;
    } while (w.state == 0);
}

template <class S, bool STAGED, int W>
__device__ void lin_tile_pair(const ExtendParams& P, const TileLaunch& A, uint32_t pid, const PairDesc& d,
                              const PairSeq<S, STAGED>& sq, uint8_t* region, int32_t* frames, int fcap, TileCtl* sh) {
    constexpr bool kResume = W > kCtaWarps;
    constexpr int W1 = W < kCtaWarps ? W : kCtaWarps;   // the traceback is the first CTA's
    const int tid = team_tid<W>();
    const int warp = W == 1 ? 0 : tid >> 5;
    const int qn = d.qn, tn = d.tn;
    const bool fitting = tn > qn + qn / 2 + 10;
    const int max_s = qn + tn;

    TileScratch sc;
    uint64_t at = 0;
    sc.edits = reinterpret_cast<uint32_t*>(region);
    at += tile_runs_bytes(qn, tn);
    sc.cigar = reinterpret_cast<uint32_t*>(region + at);
    at += tile_runs_bytes(qn, tn);
    sc.kpath = reinterpret_cast<int32_t*>(region + at);
    at += tile_table_bytes(qn, tn);
    sc.table = reinterpret_cast<uint32_t*>(region + at);

    // ---- s = 0, or where the pair was left ----
    const uint64_t fixed = tile_fixed_bytes(qn, tn);
    const TileHead head = kResume ? *reinterpret_cast<const TileHead*>(region + fixed - kTileHeadBytes) : TileHead{};
    const int v0 = kResume ? head.v0 : warp_lcp<S, STAGED>(sq, 0, 0, min(qn, tn));
    bool done = !kResume && (fitting ? v0 >= qn : qn == tn && v0 == qn);   // wfa_simd.rs:277-283
    TileMin* tm = team_min<W>(sh, region, fixed);
    int s_end = 0, k_end = 0;
    TileWave w = {frames, 0, 1, 0, 0, 0, ~0ull, 0u};
    if (kResume) {
        w.u = head.u;
        w.s0 = head.step;
        with_regs<kLinRegs>(entry_regs(sc.table[w.u - 1]), [&](auto rc) {
            const TileGeom<decltype(rc)::value> G(qn, tn);
            w.cur_lo = G.first(G.lo(w.s0));
            w.cur_hi = G.first(G.hi(w.s0) + 1);
        });
        w.cur = reinterpret_cast<const int32_t*>(P.scratch + entry_base(sc.table[w.u - 1]));
    }
    if (!done) {
        if (tid == alloc_tid<W>()) {
            tm->end_key[0] = tm->end_key[1] = ~0ull;
            if (kResume) {
                // block u's space was taken for the narrower team's tiles
                uint64_t bytes = 0;
                with_regs<kLinRegs>(tile_regs<W, kLinRegs>(w.s0 + kTileSteps, qn, tn),
                                    [&](auto rc) { bytes = block_bytes(TileGeom<decltype(rc)::value>(qn, tn), w.u); });
                sh->base[w.u & 1] = grab_records(A, sh, bytes);
            } else {
                frames[0] = v0 << 8;
                sh->base[0] = grab_records(A, sh, block_bytes(TileGeom<1>(qn, tn), 0));
            }
        }
        team_sync<W>();
        while (w.state == 0)
            with_regs<kLinRegs>(tile_regs<W, kLinRegs>(w.s0 + kTileSteps, qn, tn), [&](auto rc) {
                lin_blocks<S, STAGED, W, decltype(rc)::value>(P, A, sq, qn, tn, fitting, sc.table, frames, fcap, sh, tm, w);
            });
        if (w.state == 1) {
            s_end = static_cast<int>(w.end >> 32);
            k_end = static_cast<int>(w.end & 0xffffffffu) - tn;
            done = s_end <= max_s;
        }
        if (w.state == 4) {   // uniform over the team
            if (tid == alloc_tid<W>()) tile_defer(P, A, sh, pid, region, fixed, TileHead{w.u, w.s0, v0});
            if (P.work && w.extra) atomicAdd(P.work + 3, static_cast<unsigned long long>(w.extra));
            team_sync<W>();
            return;
        }
        if (w.state == 2) {   // uniform over the team
            // Scratch for the redo: the final score from the furthest query offset reached
            // so far (the wavefront advances about in proportion to the score) plus a
            // quarter, at least twice the scores reached, at most the whole search.
            if (tid == 0) tm->reach = 0;
            team_sync<W>();
            int vm = 0;
            for (int i = tid; i < w.cur_hi - w.cur_lo; i += 32 * W) vm = max(vm, w.cur[i] >> 8);
            vm = __reduce_max_sync(PHR_FULL_MASK, vm);
            if ((tid & 31) == 0) atomicMax(&tm->reach, vm);
            team_sync<W>();
            if (tid == 0) {
                int64_t s2 = 2LL * w.s0 + 64;
                const int64_t reach = kResume ? __ldcg(&tm->reach) : tm->reach;
                if (reach > 0) {
                    int64_t est = static_cast<int64_t>(w.s0) * qn / reach;
                    est += est / 4 + 64;
                    s2 = ::max(s2, est);
                }
                s2 = ::min(static_cast<int64_t>(max_s) + 1, s2);
                tile_redo(P, pid, fixed + tile_hist_bytes(s2));
            }
        }
    }
    const bool overflow = w.state == 2;
    const int s0 = w.s0;
    const uint32_t extra = w.extra;
    if (P.work) {   // work counters: band diagonals, word compares of match extension
        const int sc_done = done ? s_end : ::min(s0, max_s);
        if (tid == 0) {
            const unsigned long long cells = static_cast<unsigned long long>(tile_band_cells(qn, tn, sc_done));
            atomicAdd(P.work + 2, cells);
            atomicAdd(P.work + 3, cells + 1);
        }
        if (extra) atomicAdd(P.work + 3, static_cast<unsigned long long>(extra));
    }
    if (!overflow && team_rank<W>() == 0) {   // uniform over each CTA
        uint32_t nr = 0, tl = 0;
        if (done) {
            if (warp == 0) {
                if (s_end > 0) {
                    // the last block is walked score by score, those below block by block
                    const int u_top = (s_end - 1) / kTileSteps;
                    int k = k_end;
                    with_regs<kLinRegs>(entry_regs(sc.table[u_top]), [&](auto rc) {
                        constexpr int R = decltype(rc)::value;
                        block_ops<R>(block_at<R>(P.scratch, sc.table, qn, tn, u_top), TileGeom<R>(qn, tn),
                                     (s_end - 1) % kTileSteps, k);
                    });
                    if (tid == 0) sc.kpath[u_top] = k;
                    __syncwarp();
                    walk_blocks(P.scratch, sc, qn, tn, u_top);
                }
            }
            team_sync<W1>();
            if (s_end > 0) expand_blocks<S, STAGED, W1>(sq, P.scratch, sc, qn, tn, s_end, k_end, v0);
            team_sync<W1>();
            if (warp == 0) {
                const uint32_t n = path_runs(sc.edits, sc.cigar, s_end, v0);
                if (tid == 0) sh->n_runs = n;
            }
            team_sync<W1>();
            nr = sh->n_runs;
            tl = format_runs<W1>(sc.cigar, nr, P.text + P.text_off[pid], sh->text_len);
        }
        if (tid == 0) {
            PairOut o = {};
            o.status = done ? PHR_OK : PHR_ALIGNMENT_FAILED;
            if (done) {
                o.ed = s_end;
                o.t_consumed = fitting ? qn - k_end : tn;
                o.n_runs = nr;
                o.text_len = tl;
            }
            P.out[pid] = o;
        }
    }
    team_sync<W>();   // shared memory is reused by the team's next pair
}

struct LinearTiles {
    __device__ static uint64_t fixed_bytes(int qn, int tn) { return tile_fixed_bytes(qn, tn); }
    __device__ static uint64_t hist_bytes(int64_t s) { return tile_hist_bytes(s); }
    __device__ static int64_t score_est(int qn, int mode) { return tile_score_est(qn, mode); }
    template <class S, bool STAGED, int W>
    __device__ static void pair(const ExtendParams& P, const TileLaunch& A, uint32_t pid, const PairDesc& d,
                                const PairSeq<S, STAGED>& sq, uint8_t* region, int32_t* frames, int fcap, TileCtl* sh) {
        lin_tile_pair<S, STAGED, W>(P, A, pid, d, sq, region, frames, fcap, sh);
    }
};

template <class S>
__global__ void __launch_bounds__(kBigThreads, 1) wfa_linear_big_kernel(ExtendParams P, TileLaunch A) {
    tile_team<S, kBigThreads / 32, LinearTiles>(P, A, 0, P.big_smem);
}

// Deferred pairs, a cluster of C CTAs per pair.
template <class S, int C>
__global__ void __launch_bounds__(kBigThreads, 1) wfa_linear_resume_kernel(ExtendParams P, TileLaunch A) {
    tile_team<S, C * kCtaWarps, LinearTiles>(P, A, 0, P.big_smem);
}

// One warp per pair: kWarpTileThreads / 32 teams per CTA, two CTAs per SM.
template <class S>
__global__ void __launch_bounds__(kWarpTileThreads, 2) wfa_linear_tile_kernel(ExtendParams P, TileLaunch A) {
    tile_team<S, 1, LinearTiles>(P, A, (threadIdx.x >> 5) * kWarpTileSmem, kWarpTileSmem);
}

}  // namespace

void launch_wfa_linear_resume(const ExtendParams& p, const TileLaunch& a, int pairs, int ctas, int mode, cudaStream_t st) {
    auto go = [&](auto kernel) { launch_clusters(kernel, p, a, pairs, ctas, st); };
    if (mode == 0)
        ctas == 16 ? go(wfa_linear_resume_kernel<Seq2, 16>) : ctas == 8 ? go(wfa_linear_resume_kernel<Seq2, 8>) : go(wfa_linear_resume_kernel<Seq2, 4>);
    else
        ctas == 16 ? go(wfa_linear_resume_kernel<SeqB, 16>) : ctas == 8 ? go(wfa_linear_resume_kernel<SeqB, 8>) : go(wfa_linear_resume_kernel<SeqB, 4>);
}
int wfa_cluster_fit(uint32_t smem) {
    return cluster_fits(wfa_linear_resume_kernel<Seq2, 16>, 16, smem)  ? 16
           : cluster_fits(wfa_linear_resume_kernel<Seq2, 8>, 8, smem) ? 8
           : cluster_fits(wfa_linear_resume_kernel<Seq2, 4>, 4, smem) ? 4
                                                                      : 1;
}
void launch_wfa_linear_tile(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st) {
    constexpr int smem = kWarpTileThreads / 32 * static_cast<int>(kWarpTileSmem);
    if (mode == 0) {
        cudaFuncSetAttribute(wfa_linear_tile_kernel<Seq2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        wfa_linear_tile_kernel<Seq2><<<grid, kWarpTileThreads, smem, st>>>(p, a);
    } else {
        cudaFuncSetAttribute(wfa_linear_tile_kernel<SeqB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        wfa_linear_tile_kernel<SeqB><<<grid, kWarpTileThreads, smem, st>>>(p, a);
    }
}

void launch_wfa_linear_big(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st) {
    if (mode == 0) {
        cudaFuncSetAttribute(wfa_linear_big_kernel<Seq2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBigSmemMax);
        wfa_linear_big_kernel<Seq2><<<grid, kBigThreads, p.big_smem, st>>>(p, a);
    } else {
        cudaFuncSetAttribute(wfa_linear_big_kernel<SeqB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBigSmemMax);
        wfa_linear_big_kernel<SeqB><<<grid, kBigThreads, p.big_smem, st>>>(p, a);
    }
}

}  // namespace phr
