// wfa.cu -- wavefront alignment, linear and gap-affine, with traceback (sm_100a).
//
// Semantics restated from phraya-align/src/wfa_simd.rs:
//   linear   fill_wfa :231-345, fill_wfa_fitting_impl :360-482, fitting_end_k :940-955,
//            traceback_wfa_with_tend :959-1041 / traceback_wfa :1044-1130
//   affine   fill_wfa_affine_generic :581-779, affine_pos_valid :563-569,
//            affine_traceback :785-886, levenshtein_from_cigar :893-908,
//            fill_wfa_affine_fitting_impl :919-935
//
// GPU design. One pair per group of G lanes; the diagonals of a wavefront are dealt to
// the group's lanes round-robin (diagonal k goes to lane (k + tn) mod G, the same lane
// for every layer and score, so a cell's I/D/M values never cross lanes within a step).
// Match runs are extended with 16-base (2-bit) or 4-byte word compares (common.cuh lcp).
//
// The reference keeps full-width frames (qn+tn+1 diagonals per score). Only cells
// reachable from the origin can ever be set, so each frame is stored over its
// reachable band only: linear [-min(s,tn), min(s,qn)] (the reference's own scan
// range); affine per layer, the union of its source bands shifted by the move, clipped
// to [-tn, qn]. Cells outside a band are UNSET in the reference too, so every stored
// value, op code and tie-break is identical.
//
// History per cell is what the traceback needs: the post-extension value (input to
// later scores) and the pre-extension candidate `raw` with its op code. In both
// tracebacks the match-run start is exactly `raw` (linear: edit_start = pred_pos+1 for
// ops 1/2 and pred_pos for op 3 == the winning candidate; affine: raw of each m_op).

#include "kernels.cuh"
#include "wfa_tile.cuh"

namespace phr {
namespace {

constexpr int32_t UNSET = INT32_MIN;

__device__ __forceinline__ uint64_t align16(uint64_t v) { return (v + 15) & ~15ull; }

template <class S>
__device__ __forceinline__ const uint32_t* seq_base(const ExtendParams& P, uint64_t word) {
    return (S::kBits == 2 ? P.packed2 : P.bytes) + word;
}

// Group-cooperative CIGAR formatting of `nr` reverse-order runs; returns text length.
__device__ uint32_t format_group(const uint32_t* runs, uint32_t nr, char* out, int G) {
    const int gl = lane_id() & (G - 1);
    const uint32_t nrmax = __reduce_max_sync(PHR_FULL_MASK, nr);
    const uint32_t rounds = (nrmax + G - 1) / G;
    uint32_t base = 0;
    for (uint32_t rr = 0; rr < rounds; ++rr) {
        const uint32_t c = rr * G + gl;
        uint32_t len = 0, run = 0;
        if (c < nr) {
            run = runs[nr - 1 - c];
            len = ndigits(run >> 2) + 1;
        }
        const uint32_t incl = group_incl_scan(len, G);
        if (c < nr) {
            char* p = out + base + incl - len;
            uint32_t v = run >> 2;
            const uint32_t nd = len - 1;
            for (int dd = static_cast<int>(nd) - 1; dd >= 0; --dd) {
                p[dd] = static_cast<char>('0' + v % 10);
                v /= 10;
            }
            p[nd] = op_char(run & 3);
        }
        base += __shfl_sync(PHR_FULL_MASK, incl, G - 1, G);
    }
    return base;
}

__device__ __forceinline__ void report_redo(const ExtendParams& P, uint32_t pid, uint64_t need) {
    const uint32_t k = atomicAdd(P.redo_count, 1u);
    P.redo_list[k] = pid;
    atomicMax(P.redo_need_max, static_cast<unsigned long long>(need));
    if (P.redo_need) P.redo_need[k] = need;
}

// 32 bits holding symbols [pos, pos + kPerWord) of a sequence in shared or global memory.
template <class S>
__device__ __forceinline__ uint32_t window_any(const uint32_t* base, int32_t pos) {
    const uint32_t w = static_cast<uint32_t>(pos) / S::kPerWord;
    const uint32_t sh = (static_cast<uint32_t>(pos) % S::kPerWord) * S::kBits;
    return __funnelshift_r(base[w], base[w + 1], sh);
}

// extend closure (wfa_simd.rs:252-262) for a valid position (0 <= qp <= qn, 0 <= qp-k <= tn).
// `words` counts the word compares (the LCP work of the roofline).
template <class S>
__device__ __forceinline__ int32_t extend_valid(const uint32_t* q, int32_t qn, const uint32_t* t, int32_t tn,
                                                int32_t qp, int32_t k, uint32_t& words) {
    const int32_t tp = qp - k;
    const int32_t lim = min(qn - qp, tn - tp);
    int32_t n = 0;
    while (n < lim) {
        ++words;
        const uint32_t x = window_any<S>(q, qp + n) ^ window_any<S>(t, tp + n);
        if (x != 0) return qp + min(n + static_cast<int32_t>(__ffs(x) - 1) / S::kBits, lim);
        n += S::kPerWord;
    }
    return qp + lim;
}

// ===========================================================================
// Linear WFA
// ===========================================================================
// cells stored before frame s: sum_{s'<s} (min(s',qn) + min(s',tn) + 1)
__device__ __forceinline__ uint64_t tri_min(int64_t s, int64_t x) {  // sum_{s'=0}^{s-1} min(s', x)
    if (s <= 0) return 0;
    if (s - 1 <= x) return static_cast<uint64_t>((s - 1) * s / 2);
    return static_cast<uint64_t>(x * (x + 1) / 2 + (s - 1 - x) * x);
}
__device__ __forceinline__ uint64_t lin_base(int64_t s, int64_t qn, int64_t tn) {
    return static_cast<uint64_t>(s) + tri_min(s, qn) + tri_min(s, tn);
}

// Traceback (wfa_simd.rs:959-1041) from (qn, t_end) over the history words raw << 2 | op of
// every score's band, into reverse-order runs. One thread.
__device__ __forceinline__ void lin_trace(RunWriter& rw, const uint32_t* hr, int qn, int tn, int t_end, int s_end) {
    int qi = qn, ti = t_end, k = qi - ti, ss = s_end;
    while (qi > 0 || ti > 0) {
        if (ss < 0) break;
        if (ss == 0) {
            const int mm = min(qi, ti);
            rw.push(0, static_cast<uint32_t>(mm));
            qi -= mm;
            ti -= mm;
            break;
        }
        const int lo = -min(ss, tn);
        const uint32_t aux = hr[lin_base(ss, qn, tn) + (k - lo)];
        const uint32_t op = aux & 3;
        const int32_t edit_start = static_cast<int32_t>(aux >> 2);
        const int mc = qi - edit_start;
        if (mc > 0) {
            rw.push(0, static_cast<uint32_t>(mc));
            qi -= mc;
            ti -= mc;
        }
        if (op == 1) {
            rw.push(1, 1);
            --qi;
            --ti;
        } else if (op == 2) {
            rw.push(3, 1);  // 'D': query advances
            --qi;
            k -= 1;
        } else if (op == 3) {
            rw.push(2, 1);  // 'I': target advances
            --ti;
            k += 1;
        }
        --ss;
    }
    rw.flush();
}

template <class S>
__device__ void wfa_linear_group(const ExtendParams& P, const PairDesc& d, uint32_t pid, bool act, int G,
                                 uint8_t* region, uint64_t region_bytes) {
    const int gl = lane_id() & (G - 1);
    const int qn = act ? d.qn : 0, tn = act ? d.tn : 0;
    const bool fitting = act && tn > qn + qn / 2 + 10;
    const uint32_t* qb = seq_base<S>(P, d.q_word);
    const uint32_t* tb = seq_base<S>(P, d.t_word);

    // region: [runs (qn+tn+2) u32][two value frames of qn+tn+1 int32][hr u32 cells]
    // Later scores only read the previous frame's values, so values live in two
    // ping-pong frames; the traceback reads only hr = raw << 2 | op of every frame.
    uint32_t* runs = reinterpret_cast<uint32_t*>(region);
    const uint64_t runs_bytes = align16(static_cast<uint64_t>(qn + tn + 2) * 4);
    const uint64_t frame_bytes = align16(static_cast<uint64_t>(qn + tn + 1) * 4);
    const uint64_t fixed = runs_bytes + 2 * frame_bytes;
    const uint64_t cell_cap = region_bytes > fixed ? (region_bytes - fixed) / 4 : 0;
    int32_t* hv_frames = reinterpret_cast<int32_t*>(region + runs_bytes);
    uint32_t* hr = reinterpret_cast<uint32_t*>(region + fixed);
    auto hvf = [&](int sc) -> int32_t* { return hv_frames + (sc & 1) * (frame_bytes / 4); };

    // largest score whose frames fit: lin_base(s+1) <= cell_cap
    const int max_s = qn + tn;
    uint32_t wf_cells = 0, lcp_words = 0;   // work counters: band diagonals, LCP word compares
    bool alive = act;
    bool done = false, overflow = false;
    int s_end = 0, t_end = 0;

    // ---- s = 0 ----
    if (alive) {
        if (lin_base(1, qn, tn) > cell_cap) {
            overflow = true;
            alive = false;
        }
    }
    if (alive && gl == 0) {
        const int32_t v = extend_valid<S>(qb, qn, tb, tn, 0, 0, lcp_words);
        hvf(0)[0] = v;
        hr[0] = 0;
    }
    __syncwarp();
    if (alive) {
        const int32_t v0 = hvf(0)[0];
        if (!fitting) {
            if (qn - tn == 0 && v0 == qn) {  // wfa_simd.rs:277-283 (perfect match only on diagonal 0)
                done = true;
                s_end = 0;
                t_end = tn;
            }
        } else {
            // fitting_end_k over the only set diagonal k = 0 (t_end = qn)
            if (qn <= tn && v0 >= qn) {
                done = true;
                s_end = 0;
                t_end = qn;
            }
        }
    }
    int s = 1;
    for (;;) {
        const bool run = alive && !done && s <= max_s;
        if (!__any_sync(PHR_FULL_MASK, run)) break;
        int lo = 0, hi = -1;
        uint64_t base = 0, pbase = 0;
        int plo = 0, phi = -1;
        if (run) {
            lo = -min(s, tn);
            hi = min(s, qn);
            plo = -min(s - 1, tn);
            phi = min(s - 1, qn);
            base = lin_base(s, qn, tn);
            pbase = lin_base(s - 1, qn, tn);
            if (base + static_cast<uint64_t>(hi - lo + 1) > cell_cap) {
                overflow = true;
                alive = false;
            }
        }
        const bool go = run && alive;
        int best_end_k = INT32_MAX;
        if (go && gl == 0) wf_cells += static_cast<uint32_t>(hi - lo + 1);
        if (go) {
            const int32_t* pv_frame = hvf(s - 1);
            int32_t* cur_frame = hvf(s);
            // lane gl handles diagonals k with (k + tn) mod G == gl (G is a power of two)
            int k = lo + ((gl - lo - tn) & (G - 1));
            for (; k <= hi; k += G) {
                int32_t best_pos = UNSET;
                uint32_t best_op = 0;
                bool have = false;
                // candidates in order [mismatch, ins, del]; the LAST maximal one wins
                if (k >= plo && k <= phi) {
                    const int32_t pv = pv_frame[k - plo];
                    if (pv != UNSET) {
                        best_pos = pv + 1;
                        best_op = 1;
                        have = true;
                    }
                }
                if (k > -tn && k - 1 >= plo && k - 1 <= phi) {
                    const int32_t pv = pv_frame[k - 1 - plo];
                    if (pv != UNSET) {
                        const int32_t c = pv + 1;
                        if (!have || c >= best_pos) {
                            best_pos = c;
                            best_op = 2;
                            have = true;
                        }
                    }
                }
                if (k < qn && k + 1 >= plo && k + 1 <= phi) {
                    const int32_t pv = pv_frame[k + 1 - plo];
                    if (pv != UNSET) {
                        if (!have || pv >= best_pos) {
                            best_pos = pv;
                            best_op = 3;
                            have = true;
                        }
                    }
                }
                int32_t val = UNSET;
                uint32_t aux = 0;
                if (have) {
                    const int32_t j = best_pos - k;
                    if (!(best_pos < 0 || best_pos > qn || j < 0 || j > tn)) {
                        val = extend_valid<S>(qb, qn, tb, tn, best_pos, k, lcp_words);
                        aux = (static_cast<uint32_t>(best_pos) << 2) | best_op;
                    }
                }
                cur_frame[k - lo] = val;
                hr[base + (k - lo)] = aux;
                if (val != UNSET) {
                    if (!fitting) {
                        if (k == qn - tn && val >= qn) best_end_k = k;
                    } else if (k >= qn - tn && k <= qn && val >= qn) {
                        best_end_k = min(best_end_k, k);
                    }
                }
            }
        }
        // reduce the end diagonal over the group (min k = max t_end)
        int kk = best_end_k;
        for (int o = 1; o < G; o <<= 1) kk = min(kk, __shfl_xor_sync(PHR_FULL_MASK, kk, o, G));
        __syncwarp();
        if (go && kk != INT32_MAX) {
            done = true;
            s_end = s;
            t_end = qn - kk;
        }
        if (run) ++s;
    }
    {
        const unsigned cw = __reduce_add_sync(PHR_FULL_MASK, wf_cells), lw = __reduce_add_sync(PHR_FULL_MASK, lcp_words);
        if (lane_id() == 0 && P.work) {
            atomicAdd(P.work + 2, static_cast<unsigned long long>(cw));
            atomicAdd(P.work + 3, static_cast<unsigned long long>(lw));
        }
    }
    const bool failed = act && !done && !overflow;  // loop exhausted: AlignmentFailed
    if (act && overflow && gl == 0) {
        // retry with room for twice the scores reached so far (capped at the full search)
        const int64_t s2 = ::min(static_cast<long long>(max_s) + 1, 2LL * s + 64);
        const uint64_t need = fixed + lin_base(s2, qn, tn) * 4 + 64;
        report_redo(P, pid, need);
    }

    // ---- traceback, one walk per group ----
    RunWriter rw;
    rw.init(runs, static_cast<uint32_t>(qn + tn + 2));
    const bool trace = act && done;
    if (trace && gl == 0) lin_trace(rw, hr, qn, tn, t_end, s_end);
    const uint32_t nr = __shfl_sync(PHR_FULL_MASK, rw.n, lane_id() & ~(G - 1));
    const bool ovf = __shfl_sync(PHR_FULL_MASK, rw.overflow ? 1 : 0, lane_id() & ~(G - 1)) != 0;
    __syncwarp();
    const uint32_t nr_fmt = (trace && !ovf) ? nr : 0;
    char* out = act ? P.text + P.text_off[pid] : nullptr;
    const uint32_t tl = format_group(runs, nr_fmt, out, G);
    if (act && gl == 0) {
        if (trace && !ovf) {
            PairOut o;
            o.status = PHR_OK;
            o.ed = s_end;
            o.t_consumed = t_end;
            o.affine_score = 0;
            o.n_runs = nr;
            o.text_len = tl;
            P.out[pid] = o;
        } else if (failed) {
            PairOut o = {};
            o.status = PHR_ALIGNMENT_FAILED;
            P.out[pid] = o;
        } else if (trace && ovf) {
            atomicOr(P.error_flag, 2u);
        }
    }
}

// Bulk asynchronous copies (the TMA unit's untiled cp.async.bulk, no multicast) of the
// pair's sequences into shared memory, completing on an mbarrier.
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return done != 0;
}
// `bytes` (a positive multiple of 16) from 16-byte aligned global memory to 16-byte
// aligned shared memory; completion is counted on `bar`.
__device__ __forceinline__ void bulk_copy_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}
// Bounded wait for phase `parity` of `bar` (each try itself blocks for a while); false
// when the limit ran out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity) {
    for (int it = 0; it < (1 << 22); ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Stages a pair's two sequences in the CTA's shared memory `sm`, each followed by one
// zero word (32-bit windows read one word past the last symbol): one bulk copy per
// sequence from the 16-byte boundary at or below its first word to the next 16-byte
// boundary after its last (the arenas are 256-byte aligned and hold four padding words
// after every sequence, so both ends stay inside them). Called by every thread of the
// CTA; returns the first free word after the staged sequences (16-byte aligned). A pair
// too long for the shared memory (big_staged) is read in place: 0 is returned and the
// output pointers are the global ones.
template <class S>
__device__ uint32_t stage_pair_cta(const ExtendParams& P, const PairDesc& d, uint32_t* sm, uint64_t* bar,
                                   uint32_t& phase, uint32_t** sq_out, uint32_t** st_out) {
    const int tid = threadIdx.x;
    const uint32_t* gq = seq_base<S>(P, d.q_word);
    const uint32_t* gt = seq_base<S>(P, d.t_word);
    if (!big_staged(P.big_smem, d.qn, d.tn, S::kBits == 2 ? 0 : 1)) {
        // too long for shared memory: read in place (each sequence is followed by padding
        // words in its arena, and every match extension is clamped to the sequence ends)
        *sq_out = const_cast<uint32_t*>(gq);
        *st_out = const_cast<uint32_t*>(gt);
        return 0;
    }
    const int qw = (d.qn + S::kPerWord - 1) / S::kPerWord;
    const int tw = (d.tn + S::kPerWord - 1) / S::kPerWord;
    const int lead_q = static_cast<int>((reinterpret_cast<uintptr_t>(gq) & 15) >> 2);
    const int lead_t = static_cast<int>((reinterpret_cast<uintptr_t>(gt) & 15) >> 2);
    const uint32_t t_base = static_cast<uint32_t>(lead_q + qw + 1 + 3) & ~3u;
    uint32_t* sq = sm + lead_q;
    uint32_t* st = sm + t_base + lead_t;
    const uint32_t nb_q = static_cast<uint32_t>((lead_q + qw + 3) & ~3) * 4;
    const uint32_t nb_t = static_cast<uint32_t>((lead_t + tw + 3) & ~3) * 4;
    if (tid == 0) {
        // order this CTA's earlier shared-memory accesses before the async writes
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        mbar_expect_tx(bar, nb_q + nb_t);
        if (nb_q) bulk_copy_g2s(sm, gq - lead_q, nb_q, bar);
        if (nb_t) bulk_copy_g2s(sm + t_base, gt - lead_t, nb_t, bar);
    }
    if (!mbar_wait_bounded(bar, phase)) {
        atomicOr(P.error_flag, 32u);
        mbar_wait_bounded(bar, phase);  // the copies may still land: wait once more, bounded
    }
    phase ^= 1u;
    if (tid == 0) {
        sq[qw] = 0u;
        st[tw] = 0u;
    }
    *sq_out = sq;
    *st_out = st;
    return (t_base + static_cast<uint32_t>(lead_t + tw + 1) + 3) & ~3u;
}

// ===========================================================================
// Gap-affine WFA
// ===========================================================================
struct LayerBand {
    int lo, hi;          // empty when lo > hi
    uint64_t base;       // first cell of this layer/score in the cell arrays
};

// Frame directory entry per score s: M, I, D bands.
struct AffDir {
    LayerBand L[3];
};


// Directory entry of one score with 32-bit cell indices, kept in a per-group shared
// ring for the recurrence (which looks back at most max(X, O + E) scores).
struct SBand {
    int lo, hi;
    uint32_t base;
};
struct SDir {
    SBand L[3];
};
constexpr int kAffRing = 16;          // scores per ring (power of two)
constexpr int kAffRingGroups = 4;     // rings per warp: groups of 8 or more lanes

// affine_pos_valid (wfa_simd.rs:563-569); UNSET and UNSET + 1 are negative, so invalid.
__device__ __forceinline__ bool pos_ok(int32_t pos, int k, int qn, int tn) {
    return static_cast<uint32_t>(pos) <= static_cast<uint32_t>(qn) &&
           static_cast<uint32_t>(pos) - static_cast<uint32_t>(k) <= static_cast<uint32_t>(tn);
}

// CIGAR text and record of a pair whose group leader has walked its runs into `rw`.
__device__ __forceinline__ void wfa_result(const ExtendParams& P, uint32_t pid, bool act, int G, bool trace, bool failed,
                                              const RunWriter& rw, const uint32_t* runs, uint32_t n_edit, int s_end,
                                              int t_end) {
    const int gl = lane_id() & (G - 1);
    const int leader = lane_id() & ~(G - 1);
    const uint32_t nr = __shfl_sync(PHR_FULL_MASK, rw.n, leader);
    const bool ovf = __shfl_sync(PHR_FULL_MASK, rw.overflow ? 1 : 0, leader) != 0;
    const uint32_t ned = __shfl_sync(PHR_FULL_MASK, n_edit, leader);
    __syncwarp();
    const uint32_t nr_fmt = (trace && !ovf) ? nr : 0;
    char* out = act ? P.text + P.text_off[pid] : nullptr;
    const uint32_t tl = format_group(runs, nr_fmt, out, G);
    if (act && gl == 0) {
        if (trace && !ovf) {
            PairOut o;
            o.status = PHR_OK;
            o.ed = static_cast<int32_t>(ned);  // levenshtein_from_cigar: X + I/D lengths
            o.t_consumed = t_end;
            o.affine_score = s_end;
            o.n_runs = nr;
            o.text_len = tl;
            P.out[pid] = o;
        } else if (failed) {
            PairOut o = {};
            o.status = PHR_ALIGNMENT_FAILED;
            P.out[pid] = o;
        } else if (trace && ovf) {
            atomicOr(P.error_flag, 2u);
        }
    }
}

// Traceback (wfa_simd.rs:785-886) of a finished affine wavefront and the pair's result:
// history in `auxs` through the score directory below `dir_top`. Called by all lanes of
// the warp; the leader of each group of G lanes walks its pair.
// With row_g > 0 the history is the register kernel's: one word per (score, k) at
// auxs[(score / row_g) * row_w + k - row_lo] holding raw << 4 | dop << 3 | iop << 2 | mop
// (all three layers' history of the cell), no directory read. With `folded` the same
// words are laid out per score over its M band, found through the directory (the CTA
// kernel).
__device__ void affine_finish(const ExtendParams& P, uint32_t pid, bool act, int G, int qn, int tn, int X, int O,
                              int E, uint32_t* runs, const uint32_t* auxs, const AffDir* dir_top, bool done,
                              bool failed, int s_end, int t_end, int k_end, int layer_end, bool folded = false) {
    const int gl = lane_id() & (G - 1);
    auto dir_at = [&](int64_t sc) -> const AffDir& { return dir_top[-1 - sc]; };
    auto aux_at = [&](int ss, int layer, int k) -> uint32_t {
        if (folded) {
            // one word per diagonal of the score's M band (the CTA kernel's layout)
            const LayerBand& b = dir_at(ss).L[0];
            const uint32_t w = auxs[b.base + (k - b.lo)];
            return layer == 0 ? (((w >> 4) << 2) | (w & 3u)) : (w >> (layer + 1)) & 1u;
        }
        const LayerBand& b = dir_at(ss).L[layer];
        return auxs[b.base + (k - b.lo)];
    };
    RunWriter rw;
    rw.init(runs, static_cast<uint32_t>(qn + tn + 2));
    const bool trace = act && done;
    uint32_t n_edit = 0;
    if (trace && gl == 0) {
        int qi = qn, ti = t_end, k = k_end, ss = s_end, layer = layer_end;
        int guard = 4 * (qn + tn) + 16;
        while ((qi > 0 || ti > 0) && guard-- > 0) {
            if (ss == 0) {
                const int mm = min(qi, ti);
                rw.push(0, static_cast<uint32_t>(mm));
                qi -= mm;
                ti -= mm;
                break;
            }
            if (layer == 0) {
                const uint32_t aux = aux_at(ss, 0, k);
                const uint32_t mop = aux & 3;
                const int32_t raw = static_cast<int32_t>(aux >> 2);
                const int mc = max(qi - raw, 0);
                if (mc > 0) {
                    rw.push(0, static_cast<uint32_t>(mc));
                    qi -= mc;
                    ti -= mc;
                }
                if (mop == 0) {
                    rw.push(1, 1);
                    --qi;
                    --ti;
                    ++n_edit;
                    ss -= X;
                } else {
                    layer = static_cast<int>(mop);
                }
            } else if (layer == 1) {
                rw.push(3, 1);  // ins (query-extra) -> 'D'
                --qi;
                ++n_edit;
                if (aux_at(ss, 1, k) == 0) {
                    ss -= O + E;
                    layer = 0;
                } else {
                    ss -= E;
                }
                k -= 1;
            } else {
                rw.push(2, 1);  // del (target-extra) -> 'I'
                --ti;
                ++n_edit;
                if (aux_at(ss, 2, k) == 0) {
                    ss -= O + E;
                    layer = 0;
                } else {
                    ss -= E;
                }
                k += 1;
            }
        }
        if (guard < 0) atomicOr(P.error_flag, 4u);
        rw.flush();
    }
    wfa_result(P, pid, act, G, trace, failed, rw, runs, n_edit, s_end, t_end);
}

template <class S>
__device__ void wfa_affine_group(const ExtendParams& P, const PairDesc& d, uint32_t pid, bool act, int G,
                                 uint8_t* region, uint64_t region_bytes, SDir* ring, unsigned long long* work) {
    const int gl = lane_id() & (G - 1);
    const int qn = act ? d.qn : 0, tn = act ? d.tn : 0;
    const bool fitting = act && tn > qn + qn / 2 + 10;
    const int X = P.costs.mismatch, O = P.costs.gap_open, E = P.costs.gap_extend;
    const uint32_t* qb = seq_base<S>(P, d.q_word);
    const uint32_t* tb = seq_base<S>(P, d.t_word);
    const int64_t hard_max_s = static_cast<int64_t>(qn + tn) * max(X, 1) + O + E + 4;
    __syncwarp();
    const bool use_ring = ring != nullptr && O + E < kAffRing && X < kAffRing;

    // region: [runs][values: cap int32][aux: cap uint32][... directory growing down]
    // The recurrence reads values only; keeping them apart from the traceback's aux words
    // doubles the cells each cached sector holds. Directory entry of score s is
    // dir_top[-1 - s], in the last quarter of the region.
    uint32_t* runs = reinterpret_cast<uint32_t*>(region);
    const uint64_t runs_bytes = align16(static_cast<uint64_t>(qn + tn + 2) * 4);
    const uint64_t rest = region_bytes > runs_bytes ? region_bytes - runs_bytes : 0;
    const uint64_t dir_cap = (rest / 4) / sizeof(AffDir);
    // cell indices stay 32-bit: a region never holds more than 2^32 - 1 cells here
    const uint64_t cell_bytes = rest - rest % sizeof(AffDir) - dir_cap * sizeof(AffDir);
    const uint64_t cell_cap = min(static_cast<uint64_t>((cell_bytes / 8) & ~3ull), static_cast<uint64_t>(0xFFFFFFFFu));
    int32_t* vals = reinterpret_cast<int32_t*>(region + runs_bytes);
    uint32_t* auxs = reinterpret_cast<uint32_t*>(vals + cell_cap);
    AffDir* dir_top = reinterpret_cast<AffDir*>(region + runs_bytes + rest - (rest % sizeof(AffDir)));
    auto dir_at = [&](int64_t sc) -> AffDir& { return dir_top[-1 - sc]; };
    auto fits = [&](uint64_t ncells, int64_t nscores) -> bool {
        return ncells <= cell_cap && static_cast<uint64_t>(nscores) <= dir_cap;
    };
    auto band_of = [&](int64_t sc, int layer) -> SBand {
        if (use_ring) return ring[sc & (kAffRing - 1)].L[layer];
        const LayerBand& b = dir_at(sc).L[layer];
        return SBand{b.lo, b.hi, static_cast<uint32_t>(b.base)};
    };

    bool alive = act;
    bool done = false, overflow = false;
    int s_end = 0, t_end = 0, k_end = 0, layer_end = 0;
    uint32_t used = 0;
    uint32_t wf_cells = 0, lcp_words = 0;   // work counters: M-band diagonals, LCP word compares

    if (alive && (dir_cap < 1 || cell_cap < 1 || !fits(1, 1))) {
        overflow = true;
        alive = false;
    }
    // ---- s = 0: m0[0] = extend(0, 0) ----
    if (alive && gl == 0) {
        AffDir e;
        e.L[0].lo = 0;
        e.L[0].hi = 0;
        e.L[0].base = 0;
        e.L[1].lo = 1;
        e.L[1].hi = 0;
        e.L[1].base = 1;
        e.L[2].lo = 1;
        e.L[2].hi = 0;
        e.L[2].base = 1;
        dir_at(0) = e;
        if (use_ring) ring[0] = SDir{{{0, 0, 0u}, {1, 0, 1u}, {1, 0, 1u}}};
        vals[0] = extend_valid<S>(qb, qn, tb, tn, 0, 0, lcp_words);
        auxs[0] = 0;
    }
    __syncwarp();
    if (alive) {
        used = 1;
        const int v0 = vals[0];
        // endpoint (wfa_simd.rs:618-650) on frame 0: only diagonal 0 is set
        if (!fitting) {
            if (qn - tn == 0 && v0 == qn) {
                done = true;
                t_end = tn;
                k_end = 0;
                layer_end = 0;
            }
        } else if (qn <= tn && v0 == qn) {
            done = true;
            t_end = qn;
            k_end = 0;
            layer_end = 0;
        }
    }
    const SBand none = {1, 0, 0u};
    // every reachable score is a sum of X, O + E and E: a multiple of g = gcd(X, O, E).
    // Other scores have empty wavefronts (and are never looked up nor traced back), so
    // the loop visits multiples of g only.
    int g = 0;
    for (int v : {X, O, E}) {
        int a = g, b = v < 0 ? -v : v;
        while (b) {
            const int t = a % b;
            a = b;
            b = t;
        }
        g = a;
    }
    const int step = g > 0 ? g : 1;
    int64_t s = step;
    for (;;) {
        const bool run = alive && !done && s <= hard_max_s;
        if (!__any_sync(PHR_FULL_MASK, run)) break;
        SBand bI = none, bD = none, bM = none;
        SBand sMo = none, sIe = none, sDe = none, sMx = none;
        bool go = run;
        if (go) {
            const int64_t so = s - O - E, se = s - E, sx = s - X;
            if (so >= 0) sMo = band_of(so, 0);
            if (se >= 0) {
                sIe = band_of(se, 1);
                sDe = band_of(se, 2);
            }
            if (sx >= 0) sMx = band_of(sx, 0);
            // I: from M[so] (k-1) and I[se] (k-1): bands shifted by +1
            int lo = INT32_MAX, hi = INT32_MIN;
            if (sMo.lo <= sMo.hi) { lo = min(lo, sMo.lo + 1); hi = max(hi, sMo.hi + 1); }
            if (sIe.lo <= sIe.hi) { lo = min(lo, sIe.lo + 1); hi = max(hi, sIe.hi + 1); }
            bI.lo = max(lo, -tn);
            bI.hi = min(hi, qn);
            // D: from M[so] (k+1) and D[se] (k+1): shifted by -1
            lo = INT32_MAX;
            hi = INT32_MIN;
            if (sMo.lo <= sMo.hi) { lo = min(lo, sMo.lo - 1); hi = max(hi, sMo.hi - 1); }
            if (sDe.lo <= sDe.hi) { lo = min(lo, sDe.lo - 1); hi = max(hi, sDe.hi - 1); }
            bD.lo = max(lo, -tn);
            bD.hi = min(hi, qn);
            // M: from M[sx] (k), I[s] (k), D[s] (k)
            lo = INT32_MAX;
            hi = INT32_MIN;
            if (sMx.lo <= sMx.hi) { lo = min(lo, sMx.lo); hi = max(hi, sMx.hi); }
            if (bI.lo <= bI.hi) { lo = min(lo, bI.lo); hi = max(hi, bI.hi); }
            if (bD.lo <= bD.hi) { lo = min(lo, bD.lo); hi = max(hi, bD.hi); }
            bM.lo = max(lo, -tn);
            bM.hi = min(hi, qn);
            if (gl == 0 && bM.lo <= bM.hi) wf_cells += static_cast<uint32_t>(bM.hi - bM.lo + 1);
            const uint32_t wI = bI.lo <= bI.hi ? static_cast<uint32_t>(bI.hi - bI.lo + 1) : 0;
            const uint32_t wD = bD.lo <= bD.hi ? static_cast<uint32_t>(bD.hi - bD.lo + 1) : 0;
            const uint32_t wM = bM.lo <= bM.hi ? static_cast<uint32_t>(bM.hi - bM.lo + 1) : 0;
            bI.base = used;
            bD.base = used + wI;
            bM.base = used + wI + wD;
            if (!fits(static_cast<uint64_t>(used) + wI + wD + wM, s + 1)) {
                overflow = true;
                alive = false;
                go = false;
            } else {
                used += wI + wD + wM;
            }
        }
        int best_end_k = INT32_MAX, best_end_layer = 0;
        if (go && bM.lo <= bM.hi) {
            // union band == M band (it contains the I and D bands); lane gl takes the
            // diagonals k with (k + tn) mod G == gl (G is a power of two)
            const int lo = bM.lo, hi = bM.hi;
            for (int k = lo + ((gl - lo - tn) & (G - 1)); k <= hi; k += G) {
                int32_t ins = UNSET, del = UNSET;
                if (k >= bI.lo && k <= bI.hi) {
                    int32_t best = UNSET, iop = 0;
                    if (k - 1 >= sMo.lo && k - 1 <= sMo.hi) {
                        const int32_t c = vals[sMo.base + (k - 1 - sMo.lo)] + 1;
                        if (pos_ok(c, k, qn, tn) && c > best) { best = c; iop = 0; }
                    }
                    if (k - 1 >= sIe.lo && k - 1 <= sIe.hi) {
                        const int32_t c = vals[sIe.base + (k - 1 - sIe.lo)] + 1;
                        if (pos_ok(c, k, qn, tn) && c > best) { best = c; iop = 1; }
                    }
                    ins = best;
                    vals[bI.base + (k - bI.lo)] = ins;
                    auxs[bI.base + (k - bI.lo)] = static_cast<uint32_t>(iop);
                }
                if (k >= bD.lo && k <= bD.hi) {
                    int32_t best = UNSET, dop = 0;
                    if (k + 1 >= sMo.lo && k + 1 <= sMo.hi) {
                        const int32_t c = vals[sMo.base + (k + 1 - sMo.lo)];
                        if (pos_ok(c, k, qn, tn) && c > best) { best = c; dop = 0; }
                    }
                    if (k + 1 >= sDe.lo && k + 1 <= sDe.hi) {
                        const int32_t c = vals[sDe.base + (k + 1 - sDe.lo)];
                        if (pos_ok(c, k, qn, tn) && c > best) { best = c; dop = 1; }
                    }
                    del = best;
                    vals[bD.base + (k - bD.lo)] = del;
                    auxs[bD.base + (k - bD.lo)] = static_cast<uint32_t>(dop);
                }
                // M (wfa_simd.rs:743-765): [mismatch-extend, ins close, del close], strict >
                int32_t best = UNSET;
                uint32_t mop = 0;
                if (k >= sMx.lo && k <= sMx.hi) {
                    const int32_t c = vals[sMx.base + (k - sMx.lo)] + 1;
                    if (pos_ok(c, k, qn, tn)) { best = c; mop = 0; }
                }
                if (pos_ok(ins, k, qn, tn) && ins > best) { best = ins; mop = 1; }
                if (pos_ok(del, k, qn, tn) && del > best) { best = del; mop = 2; }
                int32_t mval = UNSET;
                uint32_t aux = 0;
                if (best != UNSET) {
                    mval = extend_valid<S>(qb, qn, tb, tn, best, k, lcp_words);
                    aux = (static_cast<uint32_t>(best) << 2) | mop;
                }
                vals[bM.base + (k - bM.lo)] = mval;
                auxs[bM.base + (k - bM.lo)] = aux;
                // endpoint candidates: value == qn in layer order m, ins, del
                const int layer = mval == qn ? 0 : ins == qn ? 1 : del == qn ? 2 : -1;
                if (layer >= 0) {
                    if (!fitting) {
                        if (k == qn - tn) { best_end_k = k; best_end_layer = layer; }
                    } else if (k >= qn - tn && k < best_end_k) {
                        best_end_k = k;
                        best_end_layer = layer;
                    }
                }
            }
        }
        if (go && gl == 0) {
            AffDir e;
            e.L[0] = LayerBand{bM.lo, bM.hi, bM.base};
            e.L[1] = LayerBand{bI.lo, bI.hi, bI.base};
            e.L[2] = LayerBand{bD.lo, bD.hi, bD.base};
            dir_at(s) = e;
            if (use_ring) ring[s & (kAffRing - 1)] = SDir{{bM, bI, bD}};
        }
        // group min over (k, layer): smallest k wins (largest t_end)
        int kk = best_end_k, ll = best_end_layer;
        for (int o = 1; o < G; o <<= 1) {
            const int ok = __shfl_xor_sync(PHR_FULL_MASK, kk, o, G);
            const int ol = __shfl_xor_sync(PHR_FULL_MASK, ll, o, G);
            if (ok < kk) { kk = ok; ll = ol; }
        }
        __syncwarp();
        if (go && kk != INT32_MAX) {
            done = true;
            s_end = static_cast<int>(s);
            t_end = qn - kk;
            k_end = kk;
            layer_end = ll;
        }
        if (run) s += step;
    }
    {
        const unsigned cw = __reduce_add_sync(PHR_FULL_MASK, wf_cells), lw = __reduce_add_sync(PHR_FULL_MASK, lcp_words);
        if (lane_id() == 0) {
            work[0] += cw;
            work[1] += lw;
        }
    }
    const bool failed = act && !done && !overflow;
    if (act && overflow && gl == 0) {
        // retry with 4x the room used so far (bounded by every diagonal of every score)
        const uint64_t full = runs_bytes + 4ull * static_cast<uint64_t>(hard_max_s + 1) * sizeof(AffDir) +
                              static_cast<uint64_t>(hard_max_s + 1) * 3ull * static_cast<uint64_t>(qn + tn + 1) * 8ull + 4096;
        // the directory gets a quarter of the region, the cells the rest
        const uint64_t grow = runs_bytes + 4ull * (static_cast<uint64_t>(used) * 8 + static_cast<uint64_t>(s + 1) * sizeof(AffDir)) +
                              4096;
        report_redo(P, pid, min(full, grow));
    }

    affine_finish(P, pid, act, G, qn, tn, X, O, E, runs, auxs, dir_top, done, failed, s_end, t_end, k_end,
                  layer_end);
}

// ===========================================================================
// Gap-affine WFA, one CTA per long pair
// ===========================================================================
// The warp-group kernel above runs a long, divergent pair with 32 lanes over bands of
// thousands of diagonals per score, and only a few hundred such pairs exist in a batch:
// most SMs idle. Here a CTA of kBigAffineThreads threads takes one pair; the recurrence, band
// rules, candidate order and tie-breaks are those of wfa_affine_group (values, ops and
// the end cell are identical), the diagonals of each score are dealt to the CTA's
// threads, both sequences sit in shared memory (bulk copies) while they fit, and one
// warp walks the traceback.
// Memory: the recurrence reads values at most max(X, O + E) scores back, so the M, I and
// D values live in a ring of that many score slots, indexed by diagonal; what every
// score keeps is one 32-bit history word per diagonal of its M band (the M source and
// the M value before extension, plus the I and D extend bits; the bands of I and D lie
// inside M's) and a directory entry with the three bands: 4 bytes per cell instead of
// 8 per cell and layer.
template <class S>
__device__ void wfa_affine_cta(const ExtendParams& P, const PairDesc& d, uint32_t pid, uint8_t* region,
                               uint64_t region_bytes, uint32_t* sm, uint64_t* bar, uint32_t& phase, int* sh_red) {
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int qn = d.qn, tn = d.tn;
    const bool fitting = tn > qn + qn / 2 + 10;
    const int X = P.costs.mismatch, O = P.costs.gap_open, E = P.costs.gap_extend;
    const int64_t hard_max_s = static_cast<int64_t>(qn + tn) * max(X, 1) + O + E + 4;
    uint32_t *qb, *tb;
    stage_pair_cta<S>(P, d, sm, bar, phase, &qb, &tb);

    int g = 0;
    for (int v : {X, O, E}) {
        int a = g, b = v < 0 ? -v : v;
        while (b) {
            const int t = a % b;
            a = b;
            b = t;
        }
        g = a;
    }
    const int step = g > 0 ? g : 1;
    // value ring: slot (score / step) % ring_n, layers M, I, D, indexed by k + tn
    const int ring_n = max(max(X, O + E), 1) / step + 1;
    const uint64_t ring_w = static_cast<uint64_t>(qn + tn + 1);

    // region: [runs][value ring][history words ...][... directory growing down]
    uint32_t* runs = reinterpret_cast<uint32_t*>(region);
    const uint64_t runs_bytes = align16(static_cast<uint64_t>(qn + tn + 2) * 4);
    const uint64_t ring_bytes = align16(static_cast<uint64_t>(ring_n) * 3 * ring_w * 4);
    const uint64_t fixed = runs_bytes + ring_bytes;
    const uint64_t rest = region_bytes > fixed ? region_bytes - fixed : 0;
    const uint64_t dir_cap = (rest / 8) / sizeof(AffDir);
    const uint64_t cell_bytes = rest - rest % sizeof(AffDir) - dir_cap * sizeof(AffDir);
    const uint64_t cell_cap = min(static_cast<uint64_t>((cell_bytes / 4) & ~3ull), static_cast<uint64_t>(0xFFFFFFFFu));
    int32_t* ring = reinterpret_cast<int32_t*>(region + runs_bytes);
    uint32_t* auxs = reinterpret_cast<uint32_t*>(region + fixed);
    AffDir* dir_top = reinterpret_cast<AffDir*>(region + fixed + rest - (rest % sizeof(AffDir)));
    auto dir_at = [&](int64_t sc) -> AffDir& { return dir_top[-1 - sc]; };
    auto val = [&](int64_t sc, int layer, int k) -> int32_t* {
        return ring + (static_cast<uint64_t>((sc / step) % ring_n) * 3 + layer) * ring_w + (k + tn);
    };
    auto fits = [&](uint64_t ncells, int64_t nscores) -> bool {
        return ncells <= cell_cap && static_cast<uint64_t>(nscores) <= dir_cap;
    };
    auto band_of = [&](int64_t sc, int layer) -> SBand {
        const LayerBand& b = dir_at(sc).L[layer];
        return SBand{b.lo, b.hi, static_cast<uint32_t>(b.base)};
    };

    bool done = false, overflow = false;
    int s_end = 0, t_end = 0, k_end = 0, layer_end = 0;
    uint32_t used = 0;
    uint32_t wf_cells = 0, lcp_words = 0;
    int32_t reach = 0;  // furthest query offset this thread's cells reached (redo sizing)
    if (region_bytes <= fixed || dir_cap < 1 || cell_cap < 1 || !fits(1, 1)) overflow = true;
    // ---- s = 0 ----
    if (!overflow && tid == 0) {
        AffDir e;
        e.L[0] = LayerBand{0, 0, 0};
        e.L[1] = LayerBand{1, 0, 0};
        e.L[2] = LayerBand{1, 0, 0};
        dir_at(0) = e;
        *val(0, 0, 0) = extend_valid<S>(qb, qn, tb, tn, 0, 0, lcp_words);
        auxs[0] = 0;
    }
    __syncthreads();
    if (!overflow) {
        used = 1;
        const int v0 = *val(0, 0, 0);
        reach = v0;
        if (!fitting) {
            if (qn - tn == 0 && v0 == qn) {
                done = true;
                t_end = tn;
            }
        } else if (qn <= tn && v0 == qn) {
            done = true;
            t_end = qn;
        }
    }
    const SBand none = {1, 0, 0u};
    int64_t s = step;
    // every thread computes the same bands and counters from the directory, so control
    // flow is uniform across the CTA
    while (!done && !overflow && s <= hard_max_s) {
        SBand bI = none, bD = none, bM = none;
        SBand sMo = none, sIe = none, sDe = none, sMx = none;
        const int64_t so = s - O - E, se = s - E, sx = s - X;
        if (so >= 0) sMo = band_of(so, 0);
        if (se >= 0) {
            sIe = band_of(se, 1);
            sDe = band_of(se, 2);
        }
        if (sx >= 0) sMx = band_of(sx, 0);
        int lo = INT32_MAX, hi = INT32_MIN;
        if (sMo.lo <= sMo.hi) { lo = min(lo, sMo.lo + 1); hi = max(hi, sMo.hi + 1); }
        if (sIe.lo <= sIe.hi) { lo = min(lo, sIe.lo + 1); hi = max(hi, sIe.hi + 1); }
        bI.lo = max(lo, -tn);
        bI.hi = min(hi, qn);
        lo = INT32_MAX;
        hi = INT32_MIN;
        if (sMo.lo <= sMo.hi) { lo = min(lo, sMo.lo - 1); hi = max(hi, sMo.hi - 1); }
        if (sDe.lo <= sDe.hi) { lo = min(lo, sDe.lo - 1); hi = max(hi, sDe.hi - 1); }
        bD.lo = max(lo, -tn);
        bD.hi = min(hi, qn);
        lo = INT32_MAX;
        hi = INT32_MIN;
        if (sMx.lo <= sMx.hi) { lo = min(lo, sMx.lo); hi = max(hi, sMx.hi); }
        if (bI.lo <= bI.hi) { lo = min(lo, bI.lo); hi = max(hi, bI.hi); }
        if (bD.lo <= bD.hi) { lo = min(lo, bD.lo); hi = max(hi, bD.hi); }
        bM.lo = max(lo, -tn);
        bM.hi = min(hi, qn);
        if (tid == 0 && bM.lo <= bM.hi) wf_cells += static_cast<uint32_t>(bM.hi - bM.lo + 1);
        const uint32_t wM = bM.lo <= bM.hi ? static_cast<uint32_t>(bM.hi - bM.lo + 1) : 0;
        bM.base = used;
        bI.base = bD.base = used;  // their history bits sit in M's words
        if (!fits(static_cast<uint64_t>(used) + wM, s + 1)) {
            overflow = true;
            break;
        }
        used += wM;
        int best_end_k = INT32_MAX, best_end_layer = 0;
        // (an empty band has lo = INT32_MAX, where lo + tid would wrap: its k loop starts
        // past hi)
        const int k0 = wM > 0 ? bM.lo + tid : 1, k1 = wM > 0 ? bM.hi : 0;
        // ring rows of this score's sources and of the score itself, indexed by diagonal
        // (the slot arithmetic once per score, not per cell; a negative score's row is
        // never read: its band is empty)
        auto row = [&](int64_t sc, int layer) -> int32_t* {
            return sc < 0 ? nullptr : val(sc, layer, 0);
        };
        const int32_t* rMo = row(so, 0);
        const int32_t* rIe = row(se, 1);
        const int32_t* rDe = row(se, 2);
        const int32_t* rMx = row(sx, 0);
        int32_t* cM = row(s, 0);
        int32_t* cI = row(s, 1);
        int32_t* cD = row(s, 2);
        for (int k = k0; k <= k1; k += nthr) {
            int32_t ins = UNSET, del = UNSET;
            uint32_t iop = 0, dop = 0;
            if (k >= bI.lo && k <= bI.hi) {
                int32_t best = UNSET;
                if (k - 1 >= sMo.lo && k - 1 <= sMo.hi) {
                    const int32_t c = rMo[k - 1] + 1;
                    if (pos_ok(c, k, qn, tn) && c > best) { best = c; iop = 0; }
                }
                if (k - 1 >= sIe.lo && k - 1 <= sIe.hi) {
                    const int32_t c = rIe[k - 1] + 1;
                    if (pos_ok(c, k, qn, tn) && c > best) { best = c; iop = 1; }
                }
                ins = best;
                cI[k] = ins;
            }
            if (k >= bD.lo && k <= bD.hi) {
                int32_t best = UNSET;
                if (k + 1 >= sMo.lo && k + 1 <= sMo.hi) {
                    const int32_t c = rMo[k + 1];
                    if (pos_ok(c, k, qn, tn) && c > best) { best = c; dop = 0; }
                }
                if (k + 1 >= sDe.lo && k + 1 <= sDe.hi) {
                    const int32_t c = rDe[k + 1];
                    if (pos_ok(c, k, qn, tn) && c > best) { best = c; dop = 1; }
                }
                del = best;
                cD[k] = del;
            }
            int32_t best = UNSET;
            uint32_t mop = 0;
            if (k >= sMx.lo && k <= sMx.hi) {
                const int32_t c = rMx[k] + 1;
                if (pos_ok(c, k, qn, tn)) { best = c; mop = 0; }
            }
            if (pos_ok(ins, k, qn, tn) && ins > best) { best = ins; mop = 1; }
            if (pos_ok(del, k, qn, tn) && del > best) { best = del; mop = 2; }
            int32_t mval = UNSET;
            uint32_t aux = (dop << 3) | (iop << 2);
            if (best != UNSET) {
                mval = extend_valid<S>(qb, qn, tb, tn, best, k, lcp_words);
                aux |= (static_cast<uint32_t>(best) << 4) | mop;
                reach = max(reach, mval);
            }
            cM[k] = mval;
            auxs[bM.base + (k - bM.lo)] = aux;
            const int layer = mval == qn ? 0 : ins == qn ? 1 : del == qn ? 2 : -1;
            if (layer >= 0) {
                if (!fitting) {
                    if (k == qn - tn) { best_end_k = k; best_end_layer = layer; }
                } else if (k >= qn - tn && k < best_end_k) {
                    best_end_k = k;
                    best_end_layer = layer;
                }
            }
        }
        if (tid == 0) {
            AffDir e;
            e.L[0] = LayerBand{bM.lo, bM.hi, bM.base};
            e.L[1] = LayerBand{bI.lo, bI.hi, bI.base};
            e.L[2] = LayerBand{bD.lo, bD.hi, bD.base};
            dir_at(s) = e;
        }
        // CTA min over (k, layer): smallest k wins (largest t_end); one key per thread
        const long long key = best_end_k == INT32_MAX
                                  ? LLONG_MAX
                                  : static_cast<long long>(best_end_k) * 4 + best_end_layer;  // layer < 4
        long long wkey = key;
        for (int o = 16; o > 0; o >>= 1) wkey = min(wkey, __shfl_xor_sync(PHR_FULL_MASK, wkey, o));
        long long* red = reinterpret_cast<long long*>(sh_red);
        if ((tid & 31) == 0) red[tid >> 5] = wkey;
        __syncthreads();  // this score's cells, directory entry and partial minima are visible
        long long best = LLONG_MAX;
        for (int w = 0; w < nthr / 32; ++w) best = min(best, red[w]);
        __syncthreads();  // `red` and the ring slot of s - ring_n * step are rewritten next
        if (best != LLONG_MAX) {
            done = true;
            s_end = static_cast<int>(s);
            k_end = static_cast<int>(best >> 2);   // floor(best / 4), also for negative k
            layer_end = static_cast<int>(best & 3);
            t_end = qn - k_end;
        }
        s += step;
    }
    if (P.work) {
        if (tid == 0) atomicAdd(P.work + 2, static_cast<unsigned long long>(wf_cells));
        if (lcp_words) atomicAdd(P.work + 3, static_cast<unsigned long long>(lcp_words));
    }
    const bool failed = !done && !overflow;
    if (overflow) {  // CTA-uniform
        // Scratch for the redo: extrapolate the final score from the furthest query offset
        // reached so far (the wavefront advances about in proportion to the score), plus a
        // quarter as margin, and the history from the cells so far (bands grow linearly,
        // so cells grow with the square of the score); at least four times what was used,
        // at most the whole search.
        long long* red = reinterpret_cast<long long*>(sh_red);
        int32_t wr = reach;
        for (int o = 16; o > 0; o >>= 1) wr = max(wr, __shfl_xor_sync(PHR_FULL_MASK, wr, o));
        if ((tid & 31) == 0) red[tid >> 5] = wr;
        __syncthreads();
        if (tid == 0) {
            int64_t rmax = 0;
            for (int w = 0; w < nthr / 32; ++w) rmax = ::max(rmax, static_cast<int64_t>(red[w]));
            const uint64_t full_cells = static_cast<uint64_t>(hard_max_s / step + 1) * ring_w;
            uint64_t s_est = static_cast<uint64_t>(hard_max_s) + 1, cells = full_cells;
            if (rmax > 0 && s > step) {
                uint64_t e = static_cast<uint64_t>(s) * static_cast<uint64_t>(qn) / static_cast<uint64_t>(rmax);
                e += e / 4 + 64;
                if (e < s_est) {
                    s_est = e;
                    const double r = static_cast<double>(e) / static_cast<double>(s);
                    cells = ::min(full_cells, static_cast<uint64_t>(static_cast<double>(used) * r * r) + 1024);
                }
            }
            cells = ::max(cells, static_cast<uint64_t>(4ull * used + 1024));
            const uint64_t need_rest =
                ::max(static_cast<uint64_t>(cells * 4 * 8 / 7 + 4096), static_cast<uint64_t>(8 * (s_est + 1) * sizeof(AffDir))) + 64;
            report_redo(P, pid, fixed + need_rest + 4096);
        }
    }
    __syncthreads();
    if (tid < 32)
        affine_finish(P, pid, true, 32, qn, tn, X, O, E, runs, auxs, dir_top, done, failed, s_end, t_end, k_end,
                      layer_end, true);
    __syncthreads();
}

template <class S>
__global__ void __launch_bounds__(kBigAffineThreads, 1) wfa_affine_big_kernel(ExtendParams P) {
    extern __shared__ __align__(16) uint32_t big_sm[];
    __shared__ uint32_t sh_task;
    __shared__ __align__(8) long long sh_red[kBigAffineThreads / 32];
    __shared__ __align__(8) uint64_t sh_bar;
    uint32_t phase = 0;  // parity of sh_bar's current phase, the same in every thread
    if (threadIdx.x == 0) mbar_init(&sh_bar, 1);
    __syncthreads();
    for (;;) {
        if (threadIdx.x == 0) sh_task = P.tasks.range[0] + atomicAdd(P.queue_head, 1u);
        __syncthreads();
        const uint32_t task = sh_task;
        __syncthreads();
        if (task >= P.tasks.range[1]) break;
        if ((P.tasks.task_group[task] & kOtherKernel) != kBigTask) continue;
        const uint32_t pid = P.tasks.order[P.tasks.task_first[task]];
        const PairDesc d = P.desc[pid];
        if (d.mode != (S::kBits == 2 ? 0 : 1)) continue;
        wfa_affine_cta<S>(P, d, pid, P.scratch + P.task_off[task], P.task_len[task] & ~15ull, big_sm, &sh_bar, phase,
                          reinterpret_cast<int*>(sh_red));
    }
}

// ===========================================================================
// Linear WFA, one CTA per pair (pairs beyond the register tiles' offsets)
// ===========================================================================
// Queries of 2^22 symbols and targets of 2^27 do not fit the value words of wfa_tile.cu. Such
// a pair is latency-bound on one warp (every cell is a chain of dependent loads), so
// kBigThreads threads share its diagonals. The sequences are read in place; the two value
// frames live in shared memory while they fit, then in the region's global frames, the
// layout of wfa_linear_group, so scratch needs and the redo rule are identical.
// What bounds it is the match runs, a thread's word compares one after the other: 4.2 Mb
// pairs of 4, 200 and 2,000 mismatches 23.7, 25.0 and 31.7 ms (with the sequences' staging
// code in the same kernel, which pairs of this size never took, 23.3, 24.3 and 31.5).
template <class S>
__device__ void wfa_linear_cta(const ExtendParams& P, const PairDesc& d, uint32_t pid, uint8_t* region,
                               uint64_t region_bytes, int32_t* sfr, uint32_t fcap, int* sh_end) {
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int qn = d.qn, tn = d.tn;
    const bool fitting = tn > qn + qn / 2 + 10;
    const uint32_t* sq = seq_base<S>(P, d.q_word);
    const uint32_t* st = seq_base<S>(P, d.t_word);

    // ---- region layout, as in wfa_linear_group ----
    uint32_t* runs = reinterpret_cast<uint32_t*>(region);
    const uint64_t runs_bytes = align16(static_cast<uint64_t>(qn + tn + 2) * 4);
    const uint64_t frame_bytes = align16(static_cast<uint64_t>(qn + tn + 1) * 4);
    const uint64_t fixed = runs_bytes + 2 * frame_bytes;
    const uint64_t cell_cap = region_bytes > fixed ? (region_bytes - fixed) / 4 : 0;
    int32_t* gfr = reinterpret_cast<int32_t*>(region + runs_bytes);
    uint32_t* hr = reinterpret_cast<uint32_t*>(region + fixed);
    bool global_frames = false;
    auto frame = [&](int sc) -> int32_t* {
        return global_frames ? gfr + (sc & 1) * (frame_bytes / 4) : sfr + (sc & 1) * fcap;
    };

    if (tid < 3) sh_end[tid] = INT32_MAX;
    const int max_s = qn + tn;
    bool done = false, overflow = lin_base(1, qn, tn) > cell_cap;
    uint64_t wf_cells = 0;   // band diagonals of the scores computed
    uint32_t lcp_words = 0;  // this thread's word compares of match extension
    int s_end = 0, t_end = 0, s = 1;
    __syncthreads();
    if (!overflow) {
        if (tid == 0) {
            frame(0)[0] = extend_valid<S>(sq, qn, st, tn, 0, 0, lcp_words);
            hr[0] = 0;
        }
        __syncthreads();
        const int32_t v0 = frame(0)[0];
        if (!fitting) {
            if (qn - tn == 0 && v0 == qn) {  // wfa_simd.rs:277-283
                done = true;
                t_end = tn;
            }
        } else if (qn <= tn && v0 >= qn) {
            done = true;
            t_end = qn;
        }
        for (; !done && s <= max_s; ++s) {
            const int lo = -min(s, tn), hi = min(s, qn);
            const int plo = -min(s - 1, tn), phi = min(s - 1, qn);
            const uint64_t base = lin_base(s, qn, tn);
            const int width = hi - lo + 1;
            if (base + static_cast<uint64_t>(width) > cell_cap) {
                overflow = true;
                break;
            }
            wf_cells += static_cast<uint64_t>(width);
            if (!global_frames && static_cast<uint32_t>(width) > fcap) {
                // frames outgrow shared memory: continue on the region's global frames
                const int32_t* src = frame(s - 1);
                int32_t* dst = gfr + ((s - 1) & 1) * (frame_bytes / 4);
                for (int i = tid; i < phi - plo + 1; i += nthr) dst[i] = src[i];
                global_frames = true;
                __syncthreads();
            }
            const int32_t* pv_frame = frame(s - 1);
            int32_t* cur_frame = frame(s);
            if (tid == 0) sh_end[(s + 1) % 3] = INT32_MAX;
            int my_end = INT32_MAX;
            for (int k = lo + tid; k <= hi; k += nthr) {
                // candidates in order [mismatch, ins, del]; the LAST maximal one wins
                auto prev = [&](int pk) { return pk >= plo && pk <= phi ? pv_frame[pk - plo] : UNSET; };
                const int32_t mis = prev(k), ins = k > -tn ? prev(k - 1) : UNSET, del = k < qn ? prev(k + 1) : UNSET;
                int32_t best_pos = UNSET;
                uint32_t best_op = 0;
                if (mis != UNSET) best_pos = mis + 1, best_op = 1;
                if (ins != UNSET && ins + 1 >= best_pos) best_pos = ins + 1, best_op = 2;
                if (del != UNSET && del >= best_pos) best_pos = del, best_op = 3;
                int32_t val = UNSET;
                uint32_t aux = 0;
                const int32_t j = best_pos - k;
                if (best_op != 0 && best_pos <= qn && j >= 0 && j <= tn) {
                    val = extend_valid<S>(sq, qn, st, tn, best_pos, k, lcp_words);
                    aux = (static_cast<uint32_t>(best_pos) << 2) | best_op;
                }
                cur_frame[k - lo] = val;
                hr[base + (k - lo)] = aux;
                if (val >= qn && (fitting ? k >= qn - tn : k == qn - tn)) my_end = min(my_end, k);
            }
            my_end = __reduce_min_sync(PHR_FULL_MASK, my_end);
            if ((tid & 31) == 0 && my_end != INT32_MAX) atomicMin(&sh_end[s % 3], my_end);
            __syncthreads();
            const int kk = sh_end[s % 3];
            if (kk != INT32_MAX) {
                done = true;
                s_end = s;
                t_end = qn - kk;
            }
        }
    }
    if (P.work) {  // work counters: band diagonals (the same in every thread), LCP word compares
        if (tid == 0) atomicAdd(P.work + 2, static_cast<unsigned long long>(wf_cells));
        if (lcp_words) atomicAdd(P.work + 3, static_cast<unsigned long long>(lcp_words));
    }
    if (overflow) {  // CTA-uniform
        // Scratch for the redo: extrapolate the final score from the furthest query offset
        // of the last score (the wavefront advances about in proportion to the score) plus a
        // quarter; at least twice the scores reached, at most the whole search.
        int vm = 0;
        if (s >= 2) {
            const int32_t* pf = frame(s - 1);
            const int plo = -min(s - 1, tn), phi = min(s - 1, qn);
            for (int k = plo + tid; k <= phi; k += nthr) vm = max(vm, pf[k - plo]);
        }
        vm = __reduce_max_sync(PHR_FULL_MASK, vm);
        __syncthreads();  // every thread is done with the end flags
        if (tid == 0) sh_end[0] = 0;
        __syncthreads();
        if ((tid & 31) == 0) atomicMax(&sh_end[0], vm);
        __syncthreads();
        if (tid == 0) {
            const int64_t reach = sh_end[0];
            int64_t s2 = 2LL * s + 64;
            if (reach > 0) {
                int64_t est = static_cast<int64_t>(s) * qn / reach;
                est += est / 4 + 64;
                s2 = ::max(s2, est);
            }
            s2 = ::min(static_cast<int64_t>(max_s) + 1, s2);
            report_redo(P, pid, fixed + lin_base(s2, qn, tn) * 4 + 64);
        }
    }

    // ---- traceback by thread 0, formatting by warp 0 ----
    if (tid < 32) {
        RunWriter rw;
        rw.init(runs, static_cast<uint32_t>(qn + tn + 2));
        if (done && tid == 0) lin_trace(rw, hr, qn, tn, t_end, s_end);
        wfa_result(P, pid, true, 32, done, !done && !overflow, rw, runs, static_cast<uint32_t>(s_end), 0,
                   t_end);
    }
    __syncthreads();  // shared memory and the task slot are reused by the next pair
}

template <class S>
__global__ void __launch_bounds__(kBigThreads, 2) wfa_linear_long_kernel(ExtendParams P) {
    extern __shared__ __align__(16) int32_t long_frames[];
    __shared__ uint32_t sh_task;
    __shared__ int sh_end[3];
    for (;;) {
        if (threadIdx.x == 0) sh_task = P.tasks.range[0] + atomicAdd(P.queue_head, 1u);
        __syncthreads();
        const uint32_t task = sh_task;
        __syncthreads();
        if (task >= P.tasks.range[1]) break;
        if ((P.tasks.task_group[task] & kOtherKernel) != kBigTask) continue;
        const uint32_t pid = P.tasks.order[P.tasks.task_first[task]];
        const PairDesc d = P.desc[pid];
        if (d.mode != (S::kBits == 2 ? 0 : 1)) continue;
        wfa_linear_cta<S>(P, d, pid, P.scratch + P.task_off[task], P.task_len[task] & ~15ull, long_frames, P.big_smem / 8,
                          sh_end);
    }
}

// ===========================================================================
// WFA, one short pair per warp, wavefronts in registers
// ===========================================================================
// Gap-affine: every reachable cell of score s lies on a diagonal |k| <= (s - O) / E (a gap of length L
// costs O + L E), so 32 R lanes hold whole wavefronts while that bound stays inside them: R
// is 1 for diagonals -16..15, then 2, 4 and 8. A lane keeps M of the last (O + E) / g steps and
// I and D of the last one, as in wfa_affine_tile.cu (X / g = 2, E / g = 1): the larger of
// "open" and "extend" is formed on its source diagonal and crosses lanes as one value, tie
// tags in the two low bits decide as the reference's candidate order does, and an offset at
// a sequence's end is the only one with an invalid successor. What a step costs is
// instructions (about 60 and the longest match run); the cells are computed exactly as in
// wfa_affine_group, so values, ops and the end cell are identical. Only the traceback's aux
// words are stored, one row per step. A pair whose band would leave the window runs through
// wfa_affine_group in the same warp.
// Before, four values crossed lanes per cell, validity was a range test per candidate and
// wide bands stepped five slots of which some lay outside: 1,000,000 pairs of 100-300 bp at
// 0-5 %, costs (4, 6, 2), 8.57 -> 5.72 ms (6,213 -> about 3,950 warp instructions a pair),
// and 4.43 in wfa_short_kernel; 300,000 at 0-10 % 6.88 -> 4.24, at 0-20 %
// 27.1 -> 17.7, of 300-480 bp 6.62 -> 4.14.
// With 4 slots at most, pairs whose band passes 128 diagonals are done twice: 7.97 at 0-10 %.
constexpr int kRegMaxLen = 1024;  // qlen + tlen below which a pair tries the register path
constexpr int kRegSlots = 8;      // most diagonals per lane here
constexpr int kRegFewSlots = 4;   // and in the kernel for short pairs alone
// History rows of diagonals -16..15 kept in the warp's shared memory: those of the first
// kRegShRows steps, which hold the whole history of most short pairs.
constexpr int kRegShRows = 32;
// A short pair's sequences as overlapping word pairs, each with room for reads from
// diagonals outside the pair.
constexpr int kRegSeqPad = kRegSlots + 4;
constexpr int kRegSeqEntries = kRegMaxLen / 16 + 2 + 2 * kRegSeqPad;
constexpr int kRegWarpSmem = kRegShRows * 128 + kRegSeqEntries * 8;

// What the steps of a pair share.
struct RegPair {
    int qn, tn;
    bool fitting;
    int64_t max_t;
    uint32_t* rows;       // global history: `win` words a step, diagonals -win / 2 on
    int win;
    uint64_t row_cap;
    uint32_t* sh_hist;
    uint32_t extra;       // word compares beyond a cell's first
    uint32_t cells;       // diagonals of the bands
    int t;                // last step done
    int end_k, end_layer; // end cell, end_layer < 0: none yet
};

// Steps of a pair while its band stays inside 32 R lanes; false when it would leave them.
template <class S, int R, int OES>
__device__ __forceinline__ bool reg_steps(const PairSeq<S, true>& sq, RegPair& C, int (&M)[OES][R], int (&I)[R],
                                          int (&D)[R]) {
    constexpr int kUnset = kNeg;
    const int lane = lane_id();
    const int qn = C.qn, tn = C.tn;
    const int k0 = lane - 16 * R;
    const int kend = qn - tn;
    const int q_last = (qn << 2) | 3;
    const int up_src = (lane + 31) & 31, dn_src = (lane + 1) & 31;
#pragma unroll 1
    while (C.t < C.max_t) {
        const int t = C.t + 1;
        const int half = max(t - OES + 1, 0);
        const int blo = max(-tn, -half), bhi = min(qn, half);
        if (blo < -16 * R || bhi > 16 * R - 1 || static_cast<uint64_t>(t) >= C.row_cap) return false;
        C.cells += static_cast<uint32_t>(bhi - blo + 1);
        int to_up[R], to_dn[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            // [open from M, extend], open first on a tie
            int a = M[OES - 1][r] + 4 + 1, e = I[r] + 4;
            int c = max(a, e);
            if (c > q_last) c = max(a > q_last ? kUnset : a, e > q_last ? kUnset : e);
            to_up[r] = c;
            const int t_last = ((tn + k0 + 32 * r - 1) << 2) | 3;
            a = M[OES - 1][r] + 1, e = D[r];
            c = max(a, e);
            if (c > t_last) c = max(a > t_last ? kUnset : a, e > t_last ? kUnset : e);
            to_dn[r] = c;
        }
        uint32_t more = 0;
        int nM[R];
        uint32_t aux[R];
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
            I[r] = ins & ~3;
            D[r] = del & ~3;
            // [mismatch, close I, close D], the first on a tie
            const int k = k0 + 32 * r;
            const int hi = min(qn, tn + k);
            int mis = M[1][r] + 4 + 3;
            if (mis > ((hi << 2) | 3)) mis = kUnset;
            const int m = __viaddmax_s32(I[r], 2, __viaddmax_s32(D[r], 1, mis));
            const int pos = m >> 2;
            const int lim = m >= 0 ? hi - pos : -1;
            const int p = max(pos, max(k, 0));   // an unset cell reads within the staged padding
            const int n = min(first_diff<S>(sq.diff(p, p - k)), lim);
            nM[r] = (m & ~3) + (n << 2);         // an unset cell stays negative
            if (n == S::kPerWord) more |= 1u << r;
            // raw << 4 | D extends << 3 | I extends << 2 | M's source (0 mismatch, 1 I, 2 D)
            aux[r] = (static_cast<uint32_t>(m & ~3) << 2) | (static_cast<uint32_t>(~m) & 3u) |
                     ((static_cast<uint32_t>(~ins) & 1u) << 2) | ((static_cast<uint32_t>(~del) & 1u) << 3);
        }
        while (more) {   // match runs longer than one word
            const int r = __ffs(more) - 1;
            more &= more - 1;
            int v = nM[0];
#pragma unroll
            for (int i = 1; i < R; ++i) v = r == i ? nM[i] : v;
            const int k = k0 + 32 * r;
            v = extend_run<S, true>(sq, v >> 2, k, min(qn, tn + k), C.extra) << 2;
#pragma unroll
            for (int i = 0; i < R; ++i) nM[i] = r == i ? v : nM[i];
        }
        // end cell: value == qn in layer order M, I, D; smallest k (largest t_end)
        bool any = false;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int k = k0 + 32 * r;
            any |= max(nM[r], max(I[r], D[r])) >= (qn << 2) && (C.fitting ? k >= kend : k == kend);
        }
        if (__any_sync(PHR_FULL_MASK, any)) {
            int best = INT32_MAX;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int k = k0 + 32 * r;
                const int layer = nM[r] >= (qn << 2) ? 0 : I[r] >= (qn << 2) ? 1 : D[r] >= (qn << 2) ? 2 : 3;
                if (layer < 3 && (C.fitting ? k >= kend : k == kend)) best = min(best, (k + tn) * 4 + layer);
            }
            best = __reduce_min_sync(PHR_FULL_MASK, best);
            C.end_k = (best >> 2) - tn;
            C.end_layer = best & 3;
        }
        uint32_t* row = C.rows + static_cast<uint64_t>(t) * C.win + C.win / 2;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int k = k0 + 32 * r;
            if (t < kRegShRows && static_cast<unsigned>(k + 16) < 32u)
                C.sh_hist[t * 32 + k + 16] = aux[r];
            else
                row[k] = aux[r];
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int a = OES - 1; a > 0; --a) M[a][r] = M[a - 1][r];
            M[0][r] = nM[r];
        }
        C.t = t;
        if (C.end_layer >= 0) return true;
    }
    return true;
}

// Linear scores of a pair while its band stays inside 32 R lanes: a step is a score, the band
// of score s |k| <= s; candidates [mismatch, I, D], the LAST maximal one wins, and a cell whose
// winner lies outside the sequences is invalid, as in wfa_linear_group.
template <class S, int R>
__device__ __forceinline__ bool lin_steps(const PairSeq<S, true>& sq, RegPair& C, int (&x)[R]) {
    const int lane = lane_id();
    const int qn = C.qn, tn = C.tn;
    const int k0 = lane - 16 * R;
    const int kend = qn - tn;
    const int up_src = (lane + 31) & 31, dn_src = (lane + 1) & 31;
#pragma unroll 1
    while (C.t < C.max_t) {
        const int t = C.t + 1;
        const int blo = -min(t, tn), bhi = min(t, qn);
        if (blo < -16 * R || bhi > 16 * R - 1 || static_cast<uint64_t>(t) >= C.row_cap) return false;
        C.cells += static_cast<uint32_t>(bhi - blo + 1);
        uint32_t more = 0;
        int nx[R];
        int prev_up = kNeg;
        int dn = __shfl_sync(PHR_FULL_MASK, x[0], dn_src);
        uint32_t* row = C.rows + static_cast<uint64_t>(t) * C.win + C.win / 2;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            constexpr int kLast = R - 1;
            const int up_rot = __shfl_sync(PHR_FULL_MASK, x[r], up_src);
            const int dn_next = r < kLast ? __shfl_sync(PHR_FULL_MASK, x[r < kLast ? r + 1 : r], dn_src) : kNeg;
            const int up = lane == 0 ? prev_up : up_rot;
            const int down = lane == 31 ? dn_next : dn;
            prev_up = up_rot;
            dn = dn_next;
            const int m = __viaddmax_s32(up, 4 + 2, __viaddmax_s32(x[r], 4 + 1, down + 3));   // raw << 2 | op
            const int k = k0 + 32 * r;
            const int pos = m >> 2;
            const int lim = m >= 0 ? min(qn, tn + k) - pos : -1;
            const int p = lim >= 0 ? pos : max(k, 0);   // an unset cell reads within the staged padding
            const int n = min(first_diff<S>(sq.diff(p, p - k)), lim);
            nx[r] = lim >= 0 ? (m & ~3) + (n << 2) : kNeg;
            if (n == S::kPerWord) more |= 1u << r;
            if (t < kRegShRows && static_cast<unsigned>(k + 16) < 32u)
                C.sh_hist[t * 32 + k + 16] = static_cast<uint32_t>(m);
            else
                row[k] = static_cast<uint32_t>(m);
        }
        while (more) {   // match runs longer than one word
            const int r = __ffs(more) - 1;
            more &= more - 1;
            int v = nx[0];
#pragma unroll
            for (int i = 1; i < R; ++i) v = r == i ? nx[i] : v;
            const int k = k0 + 32 * r;
            v = extend_run<S, true>(sq, v >> 2, k, min(qn, tn + k), C.extra) << 2;
#pragma unroll
            for (int i = 0; i < R; ++i) nx[i] = r == i ? v : nx[i];
        }
        bool any = false;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            x[r] = nx[r];
            const int k = k0 + 32 * r;
            any |= x[r] >= (qn << 2) && (C.fitting ? k >= kend : k == kend);
        }
        C.t = t;
        if (__any_sync(PHR_FULL_MASK, any)) {   // smallest k (largest t_end)
            int best = INT32_MAX;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int k = k0 + 32 * r;
                if (x[r] >= (qn << 2) && (C.fitting ? k >= kend : k == kend)) best = min(best, k);
            }
            C.end_k = __reduce_min_sync(PHR_FULL_MASK, best);
            C.end_layer = 0;
            return true;
        }
    }
    return true;
}

// A row of 32 A lanes as one of 32 B (both centred on diagonal 0).
template <int A, int B>
__device__ __forceinline__ void reg_widen(const int (&x)[A], int (&y)[B]) {
    if constexpr (A == 1) {
        const int lane = lane_id();
        const int a = __shfl_sync(PHR_FULL_MASK, x[0], (lane + 16) & 31);
#pragma unroll
        for (int i = 0; i < B; ++i) y[i] = (i == B / 2 - 1 && lane >= 16) || (i == B / 2 && lane < 16) ? a : kNeg;
    } else {
        constexpr int kOff = (B - A) / 2;
#pragma unroll
        for (int i = 0; i < B; ++i) y[i] = kNeg;
#pragma unroll
        for (int i = 0; i < A; ++i) y[kOff + i] = x[i];
    }
}

// The steps of a pair from a state of 32 R lanes on, widened as the band grows.
template <class S, int R, int RMAX, int OES>
__device__ __forceinline__ bool reg_search(const PairSeq<S, true>& sq, RegPair& C, int (&M)[OES][R], int (&I)[R],
                                           int (&D)[R]) {
    if (reg_steps<S, R, OES>(sq, C, M, I, D)) return true;
    if constexpr (R < RMAX) {
        constexpr int N = 2 * R;
        int Mn[OES][N], In[N], Dn[N];
#pragma unroll
        for (int a = 0; a < OES; ++a) reg_widen<R, N>(M[a], Mn[a]);
        reg_widen<R, N>(I, In);
        reg_widen<R, N>(D, Dn);
        return reg_search<S, N, RMAX, OES>(sq, C, Mn, In, Dn);
    } else {
        return false;
    }
}

template <class S, int R, int RMAX>
__device__ __forceinline__ bool lin_search(const PairSeq<S, true>& sq, RegPair& C, int (&x)[R]) {
    if (lin_steps<S, R>(sq, C, x)) return true;
    if constexpr (R < RMAX) {
        int y[2 * R];
        reg_widen<R, 2 * R>(x, y);
        return lin_search<S, 2 * R, RMAX>(sq, C, y);
    } else {
        return false;
    }
}

// Path of a finished pair from its history (lane 0), its text and record. OES 0: linear.
template <int OES>
__device__ __forceinline__ void reg_finish(const ExtendParams& P, uint32_t pid, const RegPair& C, uint32_t* runs, int g) {
    RunWriter rw;
    rw.init(runs, static_cast<uint32_t>(C.qn + C.tn + 2));
    const bool trace = C.end_layer >= 0;
    uint32_t n_edit = 0;
    if (trace && lane_id() == 0) {
        int qi = C.qn, ti = C.qn - C.end_k, k = C.end_k, t = C.t, layer = C.end_layer;
        int guard = 4 * (C.qn + C.tn) + 16;
        while ((qi > 0 || ti > 0) && guard-- > 0) {
            if (t == 0) {
                const int mm = min(qi, ti);
                rw.push(0, static_cast<uint32_t>(mm));
                qi -= mm;
                ti -= mm;
                break;
            }
            const uint32_t w = t < kRegShRows && static_cast<unsigned>(k + 16) < 32u
                                   ? C.sh_hist[t * 32 + k + 16]
                                   : C.rows[static_cast<uint64_t>(t) * C.win + C.win / 2 + k];
            if constexpr (OES == 0) {
                const int mc = max(qi - static_cast<int>(w >> 2), 0);
                rw.push(0, static_cast<uint32_t>(mc));
                qi -= mc;
                ti -= mc;
                const uint32_t op = w & 3u;   // 1 mismatch, 2 I (query-extra -> 'D'), 3 D (target-extra -> 'I')
                rw.push(op == 1 ? 1 : op == 2 ? 3 : 2, 1);
                if (op != 3) --qi;
                if (op != 2) --ti;
                k += op == 2 ? -1 : op == 3 ? 1 : 0;
                --t;
                continue;
            }
            if (layer == 0) {
                const int mc = max(qi - static_cast<int>(w >> 4), 0);
                rw.push(0, static_cast<uint32_t>(mc));
                qi -= mc;
                ti -= mc;
                layer = static_cast<int>(w & 3u);
                if (layer == 0) {
                    rw.push(1, 1);
                    --qi;
                    --ti;
                    ++n_edit;
                    t -= 2;
                    continue;
                }
            }
            ++n_edit;
            const bool ins = layer == 1;   // query-extra -> 'D'; target-extra -> 'I'
            const bool open = ((w >> (layer + 1)) & 1u) == 0;
            rw.push(ins ? 3 : 2, 1);
            if (ins) --qi, --k;
            else --ti, ++k;
            t -= open ? OES : 1;
            if (open) layer = 0;
        }
        if (guard < 0) atomicOr(P.error_flag, 4u);
        rw.flush();
    }
    wfa_result(P, pid, true, 32, trace, !trace, rw, runs, OES == 0 ? static_cast<uint32_t>(C.t) : n_edit, C.t * g,
                  C.qn - C.end_k);
}

// Returns true when the pair's band left the window: nothing is written for it and the
// caller runs it another way.
template <class S, int RMAX, int OES>
__device__ bool wfa_reg(const ExtendParams& P, const PairDesc& d, uint32_t pid, uint8_t* region,
                               uint64_t region_bytes, uint32_t sm_off, unsigned long long* work) {
    const int lane = lane_id();
    const int qn = d.qn, tn = d.tn;
    const int X = P.costs.mismatch, O = P.costs.gap_open, E = P.costs.gap_extend;
    const int g = OES == 0 ? 0 : E;   // affine score of a step
    const int qw = (qn + 15) / 16, tw = (tn + 15) / 16;
    uint64_t* q2 = reinterpret_cast<uint64_t*>(tile_sm + sm_off + kRegShRows * 128);
    uint64_t* t2 = q2 + qw + kRegSeqPad;
    stage_pairs(q2, seq_base<S>(P, d.q_word), qw, lane, 32);
    stage_pairs(t2, seq_base<S>(P, d.t_word), tw, lane, 32);
    __syncwarp();
    const PairSeq<S, true> sq{sm_off + kRegShRows * 128, sm_off + kRegShRows * 128 + (qw + kRegSeqPad) * 8, nullptr, nullptr};

    // region: [runs][history rows: a word per diagonal of the window]; row r holds step r, so the
    // traceback needs no directory
    uint32_t* runs = reinterpret_cast<uint32_t*>(region);
    const uint64_t runs_bytes = align16(static_cast<uint64_t>(qn + tn + 2) * 4);
    const uint64_t rest = region_bytes > runs_bytes ? region_bytes - runs_bytes : 0;
    RegPair C = {};
    C.qn = qn;
    C.tn = tn;
    C.fitting = tn > qn + qn / 2 + 10;
    C.max_t = qn + tn;
    if constexpr (OES != 0) C.max_t = (static_cast<int64_t>(qn + tn) * max(X, 1) + O + E + 4) / E;
    C.rows = reinterpret_cast<uint32_t*>(region + runs_bytes);
    C.win = 32 * RMAX;
    C.row_cap = rest / (C.win * 4);
    C.sh_hist = reinterpret_cast<uint32_t*>(tile_sm + sm_off);
    C.end_layer = -1;
    // ---- s = 0: M[0][0] = extend(0, 0) ----
    const int v0 = warp_lcp<S, true>(sq, 0, 0, min(qn, tn));
    if (v0 == qn && (C.fitting ? qn <= tn : qn == tn)) C.end_layer = 0;
    if (lane == 0) C.sh_hist[16] = 0;   // row 0, diagonal 0
    bool inside = C.row_cap >= 2;
    if (inside && C.end_layer < 0) {
        if constexpr (OES == 0) {
            int x[1] = {lane == 16 ? v0 << 2 : kNeg};
            inside = lin_search<S, 1, RMAX>(sq, C, x);
        } else {
            int M[OES][1], I[1] = {kNeg}, D[1] = {kNeg};
#pragma unroll
            for (int a = 0; a < OES; ++a) M[a][0] = kNeg;
            if (lane == 16) M[0][0] = v0 << 2;
            inside = reg_search<S, 1, RMAX, OES>(sq, C, M, I, D);
        }
    }
    {
        const unsigned extra = __reduce_add_sync(PHR_FULL_MASK, C.extra);
        if (lane == 0) {
            work[0] += C.cells;
            work[1] += C.cells + extra + 1;
        }
    }
    __syncwarp();
    if (!inside) return true;
    reg_finish<OES>(P, pid, C, runs, g);
    return false;
}

// Persistent kernel: warps pull tasks; each task's groups split the warp's slot evenly.
constexpr int kAffGroupSmem = kAffRingGroups * kAffRing * static_cast<int>(sizeof(SDir));
constexpr int kAffWarpSmem = kAffGroupSmem > kRegWarpSmem ? kAffGroupSmem : kRegWarpSmem;
constexpr int kAffBlockSmem = 8 * kAffWarpSmem;   // of the largest block (the limit set for every size, as kBigSmemMax)

constexpr uint32_t kTaskGrab = 4;   // tasks a warp takes at a time

template <class S, bool kAffine>
__global__ void __launch_bounds__(256, kAffine ? 2 : 4) wfa_kernel(ExtendParams P) {
    extern __shared__ __align__(16) uint8_t wfa_smem[];
    const int lane = lane_id();
    const uint64_t warp_global = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    // One counter hands out every task, and an addition to one address costs about a
    // nanosecond (300,000 equal pairs of 100-300 bp with three of them a pair: 1.00 ms; with
    // one a four tasks, and the work counters' sums kept per warp: 0.45). Gap-affine tasks of
    // a pair each are taken by fours where a warp gets 128 or more, so that the last ones of
    // the launch wait for little; linear tasks hold up to 16 pairs and lose 4 % by the same.
    __shared__ unsigned long long sh_work[kAffine ? 8 : 1][2];
    unsigned long long* work = sh_work[kAffine ? threadIdx.x >> 5 : 0];
    if (kAffine && lane == 0) work[0] = work[1] = 0;
    const uint32_t grab =
        kAffine && P.tasks.range[1] - P.tasks.range[0] >= 32 * kTaskGrab * (gridDim.x * blockDim.x / 32) ? kTaskGrab : 1;
    uint32_t next = 0, batch_end = 0;
    for (;; ++next) {
        if (!kAffine || next == batch_end) {
            if (lane == 0) next = P.tasks.range[0] + atomicAdd(P.queue_head, grab);
            next = __shfl_sync(PHR_FULL_MASK, next, 0);
            if (next >= P.tasks.range[1]) break;
            batch_end = min(next + grab, P.tasks.range[1]);
        }
        const uint32_t task = next;   // (of one pair and 32 lanes with a pair list)
        uint8_t* slot = P.task_off ? P.scratch + P.task_off[task] : P.scratch + warp_global * P.slot_bytes;
        const uint64_t slot_bytes = P.task_off ? P.task_len[task] : P.slot_bytes;
        const uint8_t tg = P.pair_list ? 32 : P.tasks.task_group[task];
        if (tg & kOtherKernel) continue;  // a redo task of another kernel
        const int G = tg;
        const int count = P.pair_list ? 1 : P.tasks.task_count[task];
        const int grp = lane / G;
        bool act = grp < count;
        const uint32_t pid = P.pair_list ? P.pair_list[task] : act ? P.tasks.order[P.tasks.task_first[task] + grp] : 0;
        PairDesc d = {};
        if (act) d = P.desc[pid];
        // pairs of the other symbol mode run in the other instantiation
        act = act && d.mode == (S::kBits == 2 ? 0 : 1);
        // long pairs that the register tiles do not take run one per CTA: deferred from the main
        // pass to the redo passes, where wfa_linear_long_kernel / wfa_affine_big_kernel take them
        if (act && !P.task_off && big_pair(P.engine, P.big_min, d.qn, d.tn)) {
            if ((lane & (G - 1)) == 0)
                report_redo(P, pid, wfa_region_est(d.qn, d.tn, kAffine));
            act = false;
        }
        if (!__any_sync(PHR_FULL_MASK, act)) continue;
        // redo tasks hold one pair, which gets the whole task region
        const uint64_t region_bytes = (P.task_off ? slot_bytes : slot_bytes / (32 / G)) & ~15ull;
        uint8_t* region = slot + static_cast<uint64_t>(grp) * region_bytes;
        // a task whose estimated need exceeds the slot goes straight to a redo pass
        if (!P.task_off && !P.pair_list && P.task_need && P.task_need[task] > slot_bytes) {
            if (act && (lane & (G - 1)) == 0) report_redo(P, pid, P.task_need[task] / (32 / G));
            continue;
        }
        if constexpr (kAffine && S::kBits == 2) {
            // short 2-bit pairs of one warp each, costs with a register specialisation:
            // wavefronts in registers (redo passes and wide bands take the group kernel)
            if (G == 32 && !P.task_off && act && d.qn + d.tn < kRegMaxLen) {
                const uint32_t sm_off = (threadIdx.x >> 5) * static_cast<uint32_t>(kAffWarpSmem);
                const int open = aff_tile_open(P.costs);
                bool wide = true;  // the band left the register window (or no specialisation)
                if (open == 4) wide = wfa_reg<S, kRegSlots, 4>(P, d, pid, region, region_bytes, sm_off, work);
                else if (open == 5) wide = wfa_reg<S, kRegSlots, 5>(P, d, pid, region, region_bytes, sm_off, work);
                if (!wide) continue;
                // otherwise the group kernel below takes the pair in place (no redo pass)
            }
        }
        if (kAffine) {
            // per warp: one directory ring per group of >= 4 lanes
            uint8_t* wsm = wfa_smem + static_cast<size_t>(threadIdx.x >> 5) * kAffWarpSmem;
            SDir* ring = 32 / G <= kAffRingGroups ? reinterpret_cast<SDir*>(wsm) + grp * kAffRing : nullptr;
            wfa_affine_group<S>(P, d, pid, act, G, region, region_bytes, ring, work);
        }
        else
            wfa_linear_group<S>(P, d, pid, act, G, region, region_bytes);
    }
    if (kAffine && lane == 0 && P.work) {
        atomicAdd(P.work + 2, work[0]);
        atomicAdd(P.work + 3, work[1]);
    }
}

// Bytes of a warp's region in the kernel below: runs and rows of its widest band's steps.
constexpr uint64_t kShortSlot = ((kRegMaxLen + 2) * 4 + 15) / 16 * 16 + (16 * kRegFewSlots + 16) * (32 * kRegFewSlots * 4);
__host__ __device__ constexpr int short_blocks(int oes) { return oes == 0 ? 4 : 3; }

// The register path alone, for batches that fill the chip: without the group path's registers
// and code three CTAs fit an SM where wfa_kernel has two, which the stalls on the steps' own
// dependences need (general kernel: an instruction in 52 % of the cycles). A pair that is too
// long or too wide goes to wfa_kernel by `left`. 1,000,000 pairs of 100-300 bp at 0-5 %:
// gap-affine 5.72 -> 4.45 ms; four CTAs, with spills, 4.54.
// OES 0: linear pairs, whose tasks hold several pairs; the warp takes one after the other.
// wfa_linear_group's lanes waited for the longest of four pairs and kept frames in global
// memory (12 of 32 lanes busy): 3.01 -> 2.08 ms; 300,000 at 0-10 % 2.06 -> 1.28, of
// 300-480 bp 2.19 -> 1.35, of 20-60 bp 0.30 -> 0.28.
template <int OES>
__global__ void __launch_bounds__(256, short_blocks(OES)) wfa_short_kernel(ExtendParams P, uint32_t* left, uint32_t* n_left) {
    constexpr uint32_t kGrab = OES == 0 ? 1 : kTaskGrab;
    __shared__ unsigned long long sh_work[8][2];
    const int lane = lane_id();
    unsigned long long* work = sh_work[threadIdx.x >> 5];
    if (lane == 0) work[0] = work[1] = 0;
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    uint8_t* region = P.scratch + warp * kShortSlot;
    const uint32_t sm_off = (threadIdx.x >> 5) * static_cast<uint32_t>(kRegWarpSmem);
    const uint32_t end = P.tasks.range[1];
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = P.tasks.range[0] + atomicAdd(P.queue_head, kGrab);
        base = __shfl_sync(PHR_FULL_MASK, base, 0);
        if (base >= end) break;
        // the pairs of the tasks taken (consecutive in `order`), a lane each
        uint32_t first = P.tasks.task_first[base];
        const uint32_t last = min(base + kGrab, end) - 1;
        const uint32_t stop = P.tasks.task_first[last] + P.tasks.task_count[last];
        for (; first < stop; first += 32) {
            const uint32_t n = min(stop - first, 32u);
            uint32_t pid_l = 0;
            bool ok_l = false;
            PairDesc d_l = {};
            if (static_cast<uint32_t>(lane) < n) {
                pid_l = P.tasks.order[first + lane];
                d_l = P.desc[pid_l];
                ok_l = d_l.mode == 0 && d_l.qn + d_l.tn < kRegMaxLen;
            }
            for (uint32_t i = 0; i < n; ++i) {
                PairDesc d = {};
                d.qn = __shfl_sync(PHR_FULL_MASK, d_l.qn, i);
                d.tn = __shfl_sync(PHR_FULL_MASK, d_l.tn, i);
                d.q_word = __shfl_sync(PHR_FULL_MASK, d_l.q_word, i);
                d.t_word = __shfl_sync(PHR_FULL_MASK, d_l.t_word, i);
                const uint32_t pid = __shfl_sync(PHR_FULL_MASK, pid_l, i);
                bool wide = __shfl_sync(PHR_FULL_MASK, ok_l ? 0 : 1, i) != 0;
                if (!wide) wide = wfa_reg<Seq2, kRegFewSlots, OES>(P, d, pid, region, kShortSlot, sm_off, work);
                if (wide && lane == 0) left[atomicAdd(n_left, 1u)] = pid;
            }
        }
    }
    if (lane == 0 && P.work) {
        atomicAdd(P.work + 2, work[0]);
        atomicAdd(P.work + 3, work[1]);
    }
}

}  // namespace

void launch_wfa_linear(const ExtendParams& p, int grid, int block, cudaStream_t st) {
    wfa_kernel<Seq2, false><<<grid, block, 0, st>>>(p);
}
void launch_wfa_linear_bytes(const ExtendParams& p, int grid, int block, cudaStream_t st) {
    wfa_kernel<SeqB, false><<<grid, block, 0, st>>>(p);
}
void launch_wfa_linear_long(const ExtendParams& p, int grid, int mode, cudaStream_t st) {
    auto go = [&](auto kernel) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBigSmemMax);
        kernel<<<grid, kBigThreads, p.big_smem, st>>>(p);
    };
    mode == 0 ? go(wfa_linear_long_kernel<Seq2>) : go(wfa_linear_long_kernel<SeqB>);
}
void launch_wfa_affine_big(const ExtendParams& p, int grid, int threads, int mode, cudaStream_t st) {
    if (mode == 0) {
        cudaFuncSetAttribute(wfa_affine_big_kernel<Seq2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBigSmemMax);
        wfa_affine_big_kernel<Seq2><<<grid, threads, p.big_smem, st>>>(p);
    } else {
        cudaFuncSetAttribute(wfa_affine_big_kernel<SeqB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBigSmemMax);
        wfa_affine_big_kernel<SeqB><<<grid, threads, p.big_smem, st>>>(p);
    }
}

int launch_wfa_short(const ExtendParams& p, uint64_t scratch_bytes, int sms, int blocks_per_sm, uint32_t* left,
                     uint32_t* n_left, cudaStream_t st) {
    const int smem = 8 * kRegWarpSmem;
    const int oes = p.engine == PHR_ENGINE_WFA_LINEAR ? 0 : aff_tile_open(p.costs);
    const uint64_t fit = scratch_bytes / (8 * kShortSlot);
    const int grid = static_cast<int>(std::min<uint64_t>(static_cast<uint64_t>(sms) * std::min(blocks_per_sm, short_blocks(oes)), fit));
    if (grid == 0) return 0;
    auto* kernel = oes == 0 ? wfa_short_kernel<0> : oes == 4 ? wfa_short_kernel<4> : wfa_short_kernel<5>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    kernel<<<grid, 256, smem, st>>>(p, left, n_left);
    return grid;
}
void launch_wfa_affine(const ExtendParams& p, int grid, int block, cudaStream_t st) {
    const int smem = (block / 32) * kAffWarpSmem;
    cudaFuncSetAttribute(wfa_kernel<Seq2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAffBlockSmem);
    wfa_kernel<Seq2, true><<<grid, block, smem, st>>>(p);
}
void launch_wfa_affine_bytes(const ExtendParams& p, int grid, int block, cudaStream_t st) {
    const int smem = (block / 32) * kAffWarpSmem;
    cudaFuncSetAttribute(wfa_kernel<SeqB, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kAffBlockSmem);
    wfa_kernel<SeqB, true><<<grid, block, smem, st>>>(p);
}

}  // namespace phr
