// wfa_affine_tile.cu -- gap-affine WFA of long and byte pairs in register tiles (sm_100a).
//
// Semantics are those of wfa_affine_group (wfa.cu): fill_wfa_affine_generic
// wfa_simd.rs:581-779, affine_pos_valid :563-569, affine_traceback :785-886; every value,
// op and tie-break is the same. The method is wfa_tile.cu's; what differs:
//
// * Scores are walked in steps of g = gcd(X, O, E). A lane keeps, per diagonal, M of the
//   last (O + E) / g steps and I and D of the last one (X / g = 2 and E / g = 1: the costs
//   (2, 4, 1) and (4, 6, 2) and their multiples; other costs stay in wfa.cu).
// * The I and D candidates of a step are formed on their source diagonal, the larger of
//   "open" and "extend" first, so that one value per gap layer crosses lanes.
// * Only a value at the query's or the target's end has an invalid successor, so validity
//   is one comparison on the rare side and the common case takes the plain maximum.
// * A path cell's predecessor may lie O + E steps back, so a block of kTileSteps steps
//   is entered from one of O + E + 2 states (M of the last steps, I, D); each value word
//   carries the state and the diagonal its path entered the block with, and a block keeps
//   all those rows for its last step.
//
// What bounds it: instruction issue on the SM that holds a pair and, once the rows outgrow
// shared memory, their trip through L2. 40 pairs of 4-16 kb at up to 10 %, mostly on clusters:
// 125 instructions a band diagonal with overlap, idle lanes and traceback, issue 36 % (48 % on
// single CTAs); the kernel before it took 285, a barrier per score and a second pass for
// most pairs. 200 such pairs: 64.5 -> 9.7 ms a call.
#include "wfa_tile.cuh"

namespace phr {
namespace {

// A value word: offset << 10 | two tie / op bits << 8 | entry state << 5 | diagonals moved
// since the block's start + kStay.
constexpr int kOne = 1 << 10;
constexpr int kTag = 3 << 8;
constexpr int kAffRegs = 4;   // most diagonals per lane
constexpr int kUnset = kNeg + kStay;   // (moves of an unset word do not reach the tag bits)

// Half-width of the band of step t: a gap of length L costs open + L - 1 steps.
__device__ __forceinline__ int aff_half(int t, int open) { return max(t - open + 1, 0); }

// The value rows of a block's last step: M of the last `open` steps, then I, then D.
struct AffRows {
    const int32_t* base;
    int lo, width;   // diagonals [lo, lo + width) of every row
};

template <int R, int OES>
__device__ __forceinline__ uint64_t aff_frame_bytes(int tiles) {
    return (static_cast<uint64_t>(tiles) * tile_use(R) * 4 * (OES + 2) + 127) & ~127ull;
}

// Advances tile g of one warp by kTileSteps steps, t0 + 1 .. t0 + kTileSteps. `cur` holds
// the rows of step t0; the kept diagonals' rows go to `nxt` and `saved` (one array when
// they are the same) and the ops, eight steps of four bits per diagonal, to `rec`. FAR:
// `cur` was written by other SMs. Returns
// the smallest (step << 32 | (k + tn) << 2 | layer) of a kept end cell, ~0 without one.
template <class S, bool STAGED, int R, int OES, bool FAR>
__device__ __forceinline__ unsigned long long aff_tile(const PairSeq<S, STAGED>& sq, const TileGeom<R>& G, int g, int t0,
                                                       bool fitting, const AffRows& cur, int32_t* nxt, int32_t* saved,
                                                       int nxt_lo, int nxt_w, uint32_t* rec, uint32_t& extra) {
    constexpr int XS = 2, RM = OES;
    const int lane = lane_id();
    const int qn = G.qn, tn = G.tn;
    const int k0 = G.first(g) - kTileSteps + lane;   // this lane's first diagonal
    // where this lane's diagonal ends in the target: no offset is beyond the query's end, and
    // a bound just past that stays within a value word whatever the target's length
    const int tk0 = min(tn + k0, qn + 1);
    int M[RM][R], I[R], D[R];
    uint32_t ops[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int i = k0 + 32 * r - cur.lo;
        const bool in = i >= 0 && i < cur.width;
        auto row = [&](int a) -> int {
            const int32_t* at = cur.base + static_cast<int64_t>(a) * cur.width + i;
            const int v = in ? (FAR ? __ldcg(at) : *at) : kUnset;
            return v < 0 ? kUnset : (v & ~1023) | (a << 5) | kStay;
        };
#pragma unroll
        for (int a = 0; a < RM; ++a) M[a][r] = row(a);
        I[r] = row(RM);
        D[r] = row(RM + 1);
        ops[r] = 0;
    }
    const int kend = qn - tn;
    const bool may_end = G.first(g) + G.use > kend && (fitting || G.first(g) <= kend);   // warp-uniform
    const int up_src = (lane + 31) & 31, dn_src = (lane + 1) & 31;
    const int q_last = (qn << 10) | 1023;   // no offset beyond the query's end
    unsigned long long best_key = ~0ull;
#pragma unroll(R < 4 ? 4 / R : 1)
    for (int h = 0; h < kTileSteps; ++h) {
        int to_up[R], to_dn[R];   // the I candidate of diagonal k + 1, the D candidate of k - 1
#pragma unroll
        for (int r = 0; r < R; ++r) {
            // [open from M, extend], open first on a tie
            int a = M[OES - 1][r] + kOne + (1 << 8) + 1, e = I[r] + kOne + 1;
            int c = max(a, e);
            if (c > q_last) {
                if (a > q_last) a = kUnset;
                if (e > q_last) e = kUnset;
                c = max(a, e);
            }
            to_up[r] = c;
            a = M[OES - 1][r] + (2 << 8) - 1, e = D[r] - 1;
            c = max(a, e);
            const int t_last = ((tk0 + 32 * r - 1) << 10) | 1023;   // no offset beyond the target's end
            if (c > t_last) {
                if (a > t_last) a = kUnset;
                if (e > t_last) e = kUnset;
                c = max(a, e);
            }
            to_dn[r] = c;
        }
        uint32_t more = 0;
        int nM[R];
        int prev_up = kUnset;
        int dn = __shfl_sync(PHR_FULL_MASK, to_dn[0], dn_src);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            constexpr int kLast = R - 1;
            const int up_rot = __shfl_sync(PHR_FULL_MASK, to_up[r], up_src);
            const int dn_next = r < kLast ? __shfl_sync(PHR_FULL_MASK, to_dn[r < kLast ? r + 1 : r], dn_src) : kUnset;
            const int ins = lane == 0 ? prev_up : up_rot;
            const int del = lane == 31 ? dn_next : dn;
            prev_up = up_rot;
            dn = dn_next;
            I[r] = ins & ~kTag;
            D[r] = del & ~kTag;
            // [mismatch, close I, close D], the first on a tie
            const int k = k0 + 32 * r;
            const int hi = __viaddmin_s32(tk0, 32 * r, qn);
            int mis = M[XS - 1][r] + kOne + (3 << 8);
            if (mis > ((hi << 10) | 1023)) mis = kUnset;
            const int m = __viaddmax_s32(I[r], 2 << 8, __viaddmax_s32(D[r], 1 << 8, mis));
            const int pos = m >> 10;
            const int lo = __viaddmax_s32(k0, 32 * r, 0);
            const int lim = m >= 0 ? hi - pos : -1;
            int p, j;
            if constexpr (STAGED) {
                p = max(pos, lo);   // an unset cell reads within the staged padding
                j = p - k;
            } else {
                p = m >= 0 ? pos : 0;
                j = m >= 0 ? pos - k : 0;
            }
            const int n = min(first_diff<S>(sq.diff(p, j)), lim);
            nM[r] = (m & ~kTag) + (n << 10);   // an unset cell stays negative
            if (n == S::kPerWord) more |= 1u << r;
            ops[r] = (ops[r] >> 4) | (((static_cast<uint32_t>(m) & kTag) | ((static_cast<uint32_t>(ins | del) & kTag) << 2)) << 20);
        }
        while (more) {   // match runs longer than one word
            const int r = __ffs(more) - 1;
            more &= more - 1;
            int v = nM[0];
#pragma unroll
            for (int i = 1; i < R; ++i) v = r == i ? nM[i] : v;
            const int k = k0 + 32 * r;
            v = (extend_run<S, STAGED>(sq, v >> 10, k, min(qn, tn + k), extra) << 10) + (v & 1023);
#pragma unroll
            for (int i = 0; i < R; ++i) nM[i] = r == i ? v : nM[i];
        }
        if (may_end) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int in_tile = 32 * r + lane;
                const int k = k0 + 32 * r;
                const int end = qn << 10;
                // end cell: value == qn in layer order M, I, D
                const int layer = nM[r] >= end ? 0 : I[r] >= end ? 1 : D[r] >= end ? 2 : 3;
                if (layer < 3 && in_tile >= kTileSteps && in_tile < kTileSteps + tile_use(R) &&
                    (fitting ? k >= kend : k == kend)) {
                    const unsigned long long key = (static_cast<unsigned long long>(t0 + h + 1) << 32) |
                                                   (static_cast<unsigned>(k + tn) << 2) | static_cast<unsigned>(layer);
                    best_key = min(best_key, key);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int a = RM - 1; a > 0; --a) M[a][r] = M[a - 1][r];
            M[0][r] = nM[r];
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        rec[r * 32 + lane] = ops[r];
        const int in_tile = 32 * r + lane;
        if (in_tile >= kTileSteps && in_tile < kTileSteps + tile_use(R)) {
            const int i = k0 + 32 * r - nxt_lo;
#pragma unroll
            for (int a = 0; a < RM + 2; ++a) {
                const int v = a < RM ? M[a < RM ? a : 0][r] : a == RM ? I[r] : D[r];
                nxt[static_cast<int64_t>(a) * nxt_w + i] = v;
                if (saved != nxt) saved[static_cast<int64_t>(a) * nxt_w + i] = v;
            }
        }
    }
    return best_key;
}

// A team's share of the launch's scratch.
struct AffScratch {
    uint32_t* edits;    // the path's edits, each with the match run after it
    uint32_t* cigar;    // forward-order CIGAR runs
    int32_t* entry;     // diagonal and state the path enters block u with: (k + tn) << 3 | state
    uint32_t* list;     // block u's edits in path order, three bits each (op, match run follows), count << 24
    uint32_t* start;    // edits before block u
    uint32_t* table;    // record block u (table_entry)
};

// Where block u of a pair keeps its rows and ops.
template <int R>
struct AffBlock {
    AffRows rows;
    const uint32_t* rec;
    int glo;
    TileGeom<R> G;
    template <int OES>
    __device__ __forceinline__ static AffBlock at(const uint8_t* scratch, const uint32_t* table, int qn, int tn, int u) {
        AffBlock b = {{nullptr, 0, 0}, nullptr, 0, TileGeom<R>(qn, tn)};
        const int half = aff_half((u + 1) * kTileSteps, OES);
        b.glo = b.G.lo(half);
        const int ghi = b.G.hi(half);
        const uint8_t* base = scratch + entry_base(table[u]);
        b.rows.base = reinterpret_cast<const int32_t*>(base);
        b.rows.lo = b.G.first(b.glo);
        b.rows.width = b.G.first(ghi + 1) - b.rows.lo;
        b.rec = reinterpret_cast<const uint32_t*>(base + aff_frame_bytes<R, OES>(ghi - b.glo + 1));
        return b;
    }
};

// Follows the path back through one block from its step h (1 .. kTileSteps) in `layer` on
// diagonal k to its entry; returns the edits in path order (AffScratch::list) and leaves
// the entry's diagonal and state. One thread. (The tile that keeps diagonal k holds the
// whole stretch: see block_ops in wfa_tile.cu.)
template <int R, int OES>
__device__ __forceinline__ uint32_t aff_block_edits(const AffBlock<R>& b, int h, int layer, int& k, int& state) {
    const int g = b.G.tile_of(k);
    const int base = b.G.first(g) - kTileSteps;
    const uint32_t* rec = b.rec + static_cast<int64_t>(g - b.glo) * R * 32;
    uint32_t list = 0, count = 0;
    uint32_t run_after = 0;   // a match run follows the next edit found
    while (h > 0) {
        const uint32_t nib = rec[k - base] >> (4 * (h - 1));
        if (layer == 0) {
            const uint32_t op = nib & 3u;   // 3 mismatch, 2 close I, 1 close D
            if (op == 3) {
                list = list << 3 | 4u | 1u;
                ++count;
                h -= 2;
            } else {
                layer = op == 2 ? 1 : 2;
                run_after = 4u;
            }
        } else {
            list = list << 3 | run_after | (layer == 1 ? 2u : 3u);
            ++count;
            run_after = 0;
            k += layer == 1 ? -1 : 1;
            if (nib & (layer == 1 ? 4u : 8u)) {   // opened from M
                h -= OES;
                layer = 0;
            } else {
                h -= 1;
            }
        }
    }
    state = layer == 0 ? -h : OES + layer - 1;
    return list | count << 24;
}

// The wavefront of a team's pair between two blocks.
struct AffWave {
    AffRows cur;              // rows of step t0
    int u, t0;                // block, its first step less one
    int state;                // 0 running, 1 end found, 2 out of records, 3 every score done, 4 deferred
    unsigned long long end;
    uint32_t extra;           // word compares beyond a cell's first
};

template <int OES, int R>
__device__ __forceinline__ uint64_t aff_block_bytes(const TileGeom<R>& G, int u) {
    const int half = aff_half((u + 1) * kTileSteps, OES);
    const int n = G.hi(half) - G.lo(half) + 1;
    return aff_frame_bytes<R, OES>(n) + static_cast<uint64_t>(n) * R * 128;
}

// Blocks of a pair while its tiles hold R diagonals per lane (see lin_blocks).
template <class S, bool STAGED, int W, int R, int OES>
__device__ __forceinline__ void aff_blocks(const ExtendParams& P, const TileLaunch& A, const PairSeq<S, STAGED>& sq,
                                           int qn, int tn, bool fitting, int64_t max_t, uint32_t* table, int32_t* frames,
                                           int fcap, TileCtl* sh, TileMin* tm, AffWave& w) {
    constexpr bool kFar = W > kCtaWarps;   // a cluster's rows go through L2
    const int tid = team_tid<W>();
    const int warp = W == 1 ? 0 : tid >> 5;
    const TileGeom<R> G(qn, tn);
    do {
        const int half = aff_half(w.t0 + kTileSteps, OES);
        const int glo = G.lo(half), ghi = G.hi(half);
        const int nxt_lo = G.first(glo), nxt_w = G.first(ghi + 1) - nxt_lo;
        const unsigned long long base = sh->base[w.u & 1];
        if (base == kNoBase) {
            w.state = 2;
            return;
        }
        // the next rows: in shared memory while they fit, else only in the record
        int32_t* saved = reinterpret_cast<int32_t*>(P.scratch + base);
        int32_t* nxt = !kFar && nxt_w * (OES + 2) <= fcap / 2 ? frames + ((w.u + 1) & 1) * (fcap / 2) : saved;
        uint32_t* rec = reinterpret_cast<uint32_t*>(P.scratch + base + aff_frame_bytes<R, OES>(ghi - glo + 1));
        unsigned long long key = ~0ull;
        for (int g = glo + warp; g <= ghi; g += W)
            key = min(key, aff_tile<S, STAGED, R, OES, kFar>(sq, G, g, w.t0, fitting, w.cur, nxt, saved, nxt_lo, nxt_w,
                                                       rec + (g - glo) * R * 32, w.extra));
        if (key != ~0ull) atomicMin(&tm->end_key[w.u & 1], key);
        const int next_R = tile_regs<W, kAffRegs>(aff_half(w.t0 + 2 * kTileSteps, OES), qn, tn);
        if (tid == alloc_tid<W>()) {
            table[w.u] = table_entry(base, R);
            uint64_t bytes = 0;
            if (next_R == R)
                bytes = aff_block_bytes<OES>(G, w.u + 1);
            else
                with_regs<kAffRegs>(next_R, [&](auto rc) {
                    bytes = aff_block_bytes<OES>(TileGeom<decltype(rc)::value>(qn, tn), w.u + 1);
                });
            sh->base[(w.u + 1) & 1] = grab_records(A, sh, bytes);
            if (W == kCtaWarps && A.defer_at > 0) sh->defer[w.u & 1] = tile_sms_idle(P, A);
        }
        team_sync<W>();
        w.cur = AffRows{nxt, nxt_lo, nxt_w};
        w.t0 += kTileSteps;
        w.end = kFar ? __ldcg(&tm->end_key[w.u & 1]) : tm->end_key[w.u & 1];
        ++w.u;
        if (w.end != ~0ull)
            w.state = 1;
        else if (w.t0 >= max_t)
            w.state = 3;
        else if (W == kCtaWarps && A.defer_at > 0 && w.t0 >= A.defer_at && sh->defer[(w.u - 1) & 1])
            w.state = 4;
        if (next_R != R) return;
    } while (w.state == 0);
}

template <class S, bool STAGED, int W, int OES>
__device__ void aff_tile_pair(const ExtendParams& P, const TileLaunch& A, uint32_t pid, const PairDesc& d,
                              const PairSeq<S, STAGED>& sq, uint8_t* region, int32_t* frames, int fcap, TileCtl* sh) {
    constexpr bool kResume = W > kCtaWarps;
    constexpr int W1 = W < kCtaWarps ? W : kCtaWarps;   // the traceback is the first CTA's
    const int tid = team_tid<W>();
    const int warp = W == 1 ? 0 : tid >> 5;
    const int qn = d.qn, tn = d.tn;
    const bool fitting = tn > qn + qn / 2 + 10;
    const int g = P.costs.gap_extend;   // score of a step
    const int64_t max_t = (static_cast<int64_t>(qn + tn) * max(P.costs.mismatch, 1) + P.costs.gap_open +
                           P.costs.gap_extend + 4) / g;

    AffScratch sc;
    const uint64_t tab = aff_tile_table_bytes(qn, tn);
    sc.edits = reinterpret_cast<uint32_t*>(region);
    sc.cigar = reinterpret_cast<uint32_t*>(region + tile_runs_bytes(qn, tn));
    uint8_t* tables = region + 2 * tile_runs_bytes(qn, tn);
    sc.entry = reinterpret_cast<int32_t*>(tables);
    sc.list = reinterpret_cast<uint32_t*>(tables + tab);
    sc.start = reinterpret_cast<uint32_t*>(tables + 2 * tab);
    sc.table = reinterpret_cast<uint32_t*>(tables + 3 * tab);

    // ---- s = 0: endpoint (wfa_simd.rs:618-650) on diagonal 0 alone; or where the pair was left ----
    const uint64_t fixed = aff_tile_fixed_bytes(qn, tn);
    const TileHead head = kResume ? *reinterpret_cast<const TileHead*>(region + fixed - kTileHeadBytes) : TileHead{};
    const int v0 = kResume ? head.v0 : warp_lcp<S, STAGED>(sq, 0, 0, min(qn, tn));
    bool done = !kResume && v0 == qn && (fitting ? qn <= tn : qn == tn);
    TileMin* tm = team_min<W>(sh, region, fixed);
    int t_end = 0, k_end = 0, layer_end = 0;
    AffWave w = {{frames, 0, 1}, 0, 0, 0, ~0ull, 0u};
    if (kResume) {
        w.u = head.u;
        w.t0 = head.step;
        with_regs<kAffRegs>(entry_regs(sc.table[w.u - 1]), [&](auto rc) {
            w.cur = AffBlock<decltype(rc)::value>::template at<OES>(P.scratch, sc.table, qn, tn, w.u - 1).rows;
        });
    }
    if (!done) {
        if (tid == alloc_tid<W>()) {
            tm->end_key[0] = tm->end_key[1] = ~0ull;
            if (!kResume)
                for (int a = 0; a < OES + 2; ++a) frames[a] = a == 0 ? v0 << 10 : kUnset;
            uint64_t bytes = 0;
            with_regs<kAffRegs>(tile_regs<W, kAffRegs>(aff_half(w.t0 + kTileSteps, OES), qn, tn), [&](auto rc) {
                bytes = aff_block_bytes<OES>(TileGeom<decltype(rc)::value>(qn, tn), w.u);
            });
            sh->base[w.u & 1] = grab_records(A, sh, bytes);
        }
        team_sync<W>();
        while (w.state == 0)
            with_regs<kAffRegs>(tile_regs<W, kAffRegs>(aff_half(w.t0 + kTileSteps, OES), qn, tn), [&](auto rc) {
                aff_blocks<S, STAGED, W, decltype(rc)::value, OES>(P, A, sq, qn, tn, fitting, max_t, sc.table, frames,
                                                                  fcap, sh, tm, w);
            });
        if (w.state == 1) {
            t_end = static_cast<int>(w.end >> 32);
            k_end = static_cast<int>((w.end & 0xffffffffu) >> 2) - tn;
            layer_end = static_cast<int>(w.end & 3u);
            done = t_end <= max_t;
        }
        if (w.state == 4) {   // uniform over the team
            if (tid == alloc_tid<W>()) tile_defer(P, A, sh, pid, region, fixed, TileHead{w.u, w.t0, v0});
            if (P.work && w.extra) atomicAdd(P.work + 3, static_cast<unsigned long long>(w.extra));
            team_sync<W>();
            return;
        }
        if (w.state == 2) {   // uniform over the team
            // Scratch for the redo from the furthest query offset so far, as in wfa_tile.cu.
            if (tid == 0) tm->reach = 0;
            team_sync<W>();
            int vm = 0;
            for (int i = tid; i < w.cur.width; i += 32 * W) vm = max(vm, w.cur.base[i] >> 10);
            vm = __reduce_max_sync(PHR_FULL_MASK, vm);
            if ((tid & 31) == 0) atomicMax(&tm->reach, vm);
            team_sync<W>();
            if (tid == 0) {
                int64_t s2 = 2LL * w.t0 + 64;
                const int64_t reach = kResume ? __ldcg(&tm->reach) : tm->reach;
                if (reach > 0) {
                    int64_t est = static_cast<int64_t>(w.t0) * qn / reach;
                    est += est / 4 + 64;
                    s2 = ::max(s2, est);
                }
                s2 = ::min(max_t + 1, s2);
                tile_redo(P, pid, fixed + aff_tile_hist_bytes(s2));
            }
        }
    }
    const bool overflow = w.state == 2;
    if (P.work) {   // work counters: M-band diagonals, word compares of match extension
        if (tid == 0) {
            // bands of steps 1 .. T: one diagonal, from step OES on one more on each side
            const int64_t T = done ? t_end : ::min(static_cast<int64_t>(w.t0), max_t);
            const int64_t H = ::max(T - OES + 1, static_cast<int64_t>(0));
            auto tri = [&](int64_t x) { return H <= x ? H * (H + 1) / 2 : x * (x + 1) / 2 + (H - x) * x; };
            const unsigned long long cells = static_cast<unsigned long long>(T + tri(qn) + tri(tn));
            atomicAdd(P.work + 2, cells);
            atomicAdd(P.work + 3, cells + 1);
        }
        if (w.extra) atomicAdd(P.work + 3, static_cast<unsigned long long>(w.extra));
    }
    if (!overflow && team_rank<W>() == 0) {   // uniform over each CTA
        uint32_t nr = 0, tl = 0, n_edits = 0;
        if (done) {
            const int u_top = (t_end - 1) / kTileSteps;
            const int h_end = t_end - u_top * kTileSteps;
            auto regs_of = [&](int u) { return entry_regs(sc.table[u]); };
            if (t_end > 0) {
                if (tid == 0) {
                    // the entry of every block: the last one step by step, those below by their
                    // value words
                    int k = k_end, state = 0;
                    with_regs<kAffRegs>(regs_of(u_top), [&](auto rc) {
                        constexpr int R = decltype(rc)::value;
                        const AffBlock<R> b = AffBlock<R>::template at<OES>(P.scratch, sc.table, qn, tn, u_top);
                        aff_block_edits<R, OES>(b, h_end, layer_end, k, state);
                    });
                    sc.entry[u_top] = (k + tn) << 3 | state;
                    for (int u = u_top - 1; u >= 0; --u) {
                        int word = 0;
                        with_regs<kAffRegs>(regs_of(u), [&](auto rc) {
                            constexpr int R = decltype(rc)::value;
                            const AffRows r = AffBlock<R>::template at<OES>(P.scratch, sc.table, qn, tn, u).rows;
                            word = r.base[static_cast<int64_t>(state) * r.width + (k - r.lo)];
                        });
                        k -= (word & 31) - kStay;
                        state = (word >> 5) & 7;
                        sc.entry[u] = (k + tn) << 3 | state;
                    }
                }
                team_sync<W1>();
                // the edits of every block, one block per thread
                for (int u = tid; u <= u_top; u += 32 * W1) {
                    int k = k_end, h = h_end, layer = layer_end, state = 0;
                    if (u < u_top) {
                        const int e = sc.entry[u + 1];
                        k = (e >> 3) - tn;
                        const int s = e & 7;
                        layer = s < OES ? 0 : s - OES + 1;
                        h = s < OES ? kTileSteps - s : kTileSteps;
                    }
                    with_regs<kAffRegs>(regs_of(u), [&](auto rc) {
                        constexpr int R = decltype(rc)::value;
                        const AffBlock<R> b = AffBlock<R>::template at<OES>(P.scratch, sc.table, qn, tn, u);
                        sc.list[u] = aff_block_edits<R, OES>(b, h, layer, k, state);
                    });
                }
                team_sync<W1>();
                if (warp == 0) {   // edits before each block
                    uint32_t total = 0;
                    for (int c = 0; c <= u_top; c += 32) {
                        const int u = c + lane_id();
                        const uint32_t n = u <= u_top ? sc.list[u] >> 24 : 0u;
                        const uint32_t incl = group_incl_scan(n, 32);
                        if (u <= u_top) sc.start[u] = total + incl - n;
                        total += __shfl_sync(PHR_FULL_MASK, incl, 31);
                    }
                    if (tid == 0) sh->n_runs = total;
                }
                team_sync<W1>();
                n_edits = sh->n_runs;
                // from each block's entry offset, the match runs after its edits
                for (int u = tid; u <= u_top; u += 32 * W1) {
                    const int e = sc.entry[u];
                    int k = (e >> 3) - tn, p = v0;
                    if (u > 0)
                        with_regs<kAffRegs>(regs_of(u - 1), [&](auto rc) {
                            constexpr int R = decltype(rc)::value;
                            const AffRows r = AffBlock<R>::template at<OES>(P.scratch, sc.table, qn, tn, u - 1).rows;
                            p = r.base[static_cast<int64_t>(e & 7) * r.width + (k - r.lo)] >> 10;
                        });
                    const uint32_t list = sc.list[u];
                    uint32_t* out = sc.edits + sc.start[u] + 1;
                    uint32_t words = 0;
                    for (uint32_t i = 0; i < list >> 24; ++i) {
                        const uint32_t ed = list >> (3 * i);
                        const uint32_t op = ed & 3u;
                        p += op != 3;
                        k += op == 2 ? 1 : op == 3 ? -1 : 0;
                        int run = 0;
                        if (ed & 4u) {
                            run = max(extend_run<S, STAGED>(sq, p, k, min(qn, tn + k), words) - p, 0);
                            p += run;
                        }
                        out[i] = static_cast<uint32_t>(run) << 2 | op;
                    }
                }
            }
            team_sync<W1>();
            if (warp == 0) {
                const uint32_t n = path_runs(sc.edits, sc.cigar, static_cast<int>(n_edits), v0);
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
                o.ed = static_cast<int32_t>(n_edits);   // levenshtein_from_cigar: X + I/D lengths
                o.t_consumed = qn - k_end;
                o.affine_score = t_end * g;
                o.n_runs = nr;
                o.text_len = tl;
            }
            P.out[pid] = o;
        }
    }
    team_sync<W>();   // shared memory is reused by the team's next pair
}

template <int OES>
struct AffineTiles {
    __device__ static uint64_t fixed_bytes(int qn, int tn) { return aff_tile_fixed_bytes(qn, tn); }
    __device__ static uint64_t hist_bytes(int64_t s) { return aff_tile_hist_bytes(s); }
    __device__ static int64_t score_est(int qn, int mode) { return tile_score_est(qn, mode); }
    template <class S, bool STAGED, int W>
    __device__ static void pair(const ExtendParams& P, const TileLaunch& A, uint32_t pid, const PairDesc& d,
                                const PairSeq<S, STAGED>& sq, uint8_t* region, int32_t* frames, int fcap, TileCtl* sh) {
        aff_tile_pair<S, STAGED, W, OES>(P, A, pid, d, sq, region, frames, fcap, sh);
    }
};

template <class S, int OES>
__global__ void __launch_bounds__(kBigThreads, 1) wfa_affine_big_tile_kernel(ExtendParams P, TileLaunch A) {
    tile_team<S, kBigThreads / 32, AffineTiles<OES>>(P, A, 0, P.big_smem);
}

// Deferred pairs, a cluster of C CTAs per pair.
template <class S, int OES, int C>
__global__ void __launch_bounds__(kBigThreads, 1) wfa_affine_resume_kernel(ExtendParams P, TileLaunch A) {
    tile_team<S, C * kCtaWarps, AffineTiles<OES>>(P, A, 0, P.big_smem);
}

// One warp per pair: kWarpTileThreads / 32 teams per CTA, two CTAs per SM.
template <class S, int OES>
__global__ void __launch_bounds__(kWarpTileThreads, 2) wfa_affine_tile_kernel(ExtendParams P, TileLaunch A) {
    tile_team<S, 1, AffineTiles<OES>>(P, A, (threadIdx.x >> 5) * kWarpTileSmem, kWarpTileSmem);
}

template <class S, int OES>
void launch_cta(const ExtendParams& p, const TileLaunch& a, int grid, cudaStream_t st) {
    cudaFuncSetAttribute(wfa_affine_big_tile_kernel<S, OES>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBigSmemMax);
    wfa_affine_big_tile_kernel<S, OES><<<grid, kBigThreads, p.big_smem, st>>>(p, a);
}

template <class S, int OES>
void launch_warps(const ExtendParams& p, const TileLaunch& a, int grid, cudaStream_t st) {
    constexpr int smem = kWarpTileThreads / 32 * static_cast<int>(kWarpTileSmem);
    cudaFuncSetAttribute(wfa_affine_tile_kernel<S, OES>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    wfa_affine_tile_kernel<S, OES><<<grid, kWarpTileThreads, smem, st>>>(p, a);
}

}  // namespace

void launch_wfa_affine_resume(const ExtendParams& p, const TileLaunch& a, int pairs, int ctas, int mode, cudaStream_t st) {
    auto go = [&](auto kernel) { launch_clusters(kernel, p, a, pairs, ctas, st); };
    auto by_size = [&](auto sc, auto oc) {
        using S = decltype(sc);
        constexpr int kO = decltype(oc)::value;
        ctas == 16 ? go(wfa_affine_resume_kernel<S, kO, 16>) : ctas == 8 ? go(wfa_affine_resume_kernel<S, kO, 8>) : go(wfa_affine_resume_kernel<S, kO, 4>);
    };
    const std::integral_constant<int, 4> o4;
    const std::integral_constant<int, 5> o5;
    if (aff_tile_open(p.costs) == 4)
        mode == 0 ? by_size(Seq2{}, o4) : by_size(SeqB{}, o4);
    else
        mode == 0 ? by_size(Seq2{}, o5) : by_size(SeqB{}, o5);
}
void launch_wfa_affine_cta_tiles(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st) {
    const bool four = aff_tile_open(p.costs) == 4;
    if (mode == 0)
        four ? launch_cta<Seq2, 4>(p, a, grid, st) : launch_cta<Seq2, 5>(p, a, grid, st);
    else
        four ? launch_cta<SeqB, 4>(p, a, grid, st) : launch_cta<SeqB, 5>(p, a, grid, st);
}
void launch_wfa_affine_warp_tiles(const ExtendParams& p, const TileLaunch& a, int grid, int mode, cudaStream_t st) {
    const bool four = aff_tile_open(p.costs) == 4;
    if (mode == 0)
        four ? launch_warps<Seq2, 4>(p, a, grid, st) : launch_warps<Seq2, 5>(p, a, grid, st);
    else
        four ? launch_warps<SeqB, 4>(p, a, grid, st) : launch_warps<SeqB, 5>(p, a, grid, st);
}

}  // namespace phr
