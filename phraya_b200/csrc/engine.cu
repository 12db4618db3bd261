// engine.cu -- extension batch driver: pair preparation (suffixes, 2-bit packing),
// length-bucketed task lists, persistent-kernel launches with overflow redo passes,
// and packing of the CIGAR text into the caller's arena.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <unordered_set>

#include "engine.cuh"

namespace phr {

// ---------------------------------------------------------------------------
// DeviceArena
// ---------------------------------------------------------------------------
cudaError_t DeviceArena::reserve(size_t need) {
    if (need <= cap) return cudaSuccess;
    auto alloc = [&](size_t bytes) -> cudaError_t {
        void* p = nullptr;
        cudaError_t e = stream ? cudaMallocAsync(&p, bytes, stream) : cudaMalloc(&p, bytes);
        base = static_cast<char*>(p);
        return e;
    };
    if (base) {
        if (stream)
            cudaFreeAsync(base, stream);
        else
            cudaFree(base);
    }
    base = nullptr;
    cap = 0;
    size_t want = std::max(need + need / 4, static_cast<size_t>(64) << 20);
    cudaError_t e = alloc(want);
    if (e != cudaSuccess) {
        cudaGetLastError();
        e = alloc(need);
        if (e != cudaSuccess) {
            base = nullptr;
            return e;
        }
        want = need;
    }
    cap = want;
    used = 0;
    return cudaSuccess;
}

void Ctx::bind_stream() {
    for (DeviceArena* a : {&arena, &scratch, &io, &pipe, &seeds}) a->stream = stream;
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
        uint64_t keep = ~0ull;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    cudaGetLastError();
}

void* DeviceArena::take(size_t bytes, size_t align) {
    size_t off = (used + align - 1) / align * align;
    if (off + bytes > cap) return nullptr;
    used = off + bytes;
    return base + off;
}

DeviceArena::~DeviceArena() {
    if (base) cudaFree(base);
}

void Ctx::begin_kernel(const char* name, cudaEvent_t* a) {
    if (cudaEventCreate(a) != cudaSuccess) {
        *a = nullptr;
        return;
    }
    cudaEventRecord(*a, stream);
}

void Ctx::end_kernel(const char* name, cudaEvent_t a) {
    cudaEvent_t b;
    if (cudaEventCreate(&b) != cudaSuccess) {
        cudaEventDestroy(a);
        return;
    }
    cudaEventRecord(b, stream);
    pending.push_back({name, a, b});
}

void Ctx::resolve_timings() {
    for (auto& p : pending) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
            auto& t = timings[p.name];
            t.first += 1;
            t.second += ms;
        }
        cudaEventDestroy(p.a);
        cudaEventDestroy(p.b);
    }
    pending.clear();
}

Ctx::~Ctx() {
    for (auto& p : pending) {
        cudaEventDestroy(p.a);
        cudaEventDestroy(p.b);
    }
    if (d_counters) cudaFree(d_counters);
    if (h_pinned) cudaFreeHost(h_pinned);
    if (copy_in) cudaStreamDestroy(copy_in);
    if (copy_out) cudaStreamDestroy(copy_out);
    if (stream) cudaStreamDestroy(stream);
}

phr_status set_error(Ctx* ctx, phr_status st, const std::string& msg) {
    if (ctx) ctx->last_error = msg;
    return st;
}

phr_status cuda_status(Ctx* ctx, cudaError_t e, const char* what) {
    std::string msg = std::string(what) + ": " + cudaGetErrorString(e);
    if (e == cudaErrorMemoryAllocation) return set_error(ctx, PHR_ERR_OOM, msg);
    return set_error(ctx, PHR_ERR_CUDA, msg);
}

namespace {

constexpr uint32_t kInvalidKey = 0xFFFFFFFFu;
// key segments of the register-tile pairs (log2 lanes is 0..5): one warp, one CTA per pair
constexpr uint32_t kWarpTileSeg = 6, kTileSeg = 7;

__device__ __forceinline__ int next_pow2_cap32(int v) {
    int g = 1;
    while (g < v && g < 32) g <<= 1;
    return g;
}

struct PrepParams {
    DevPairs in;
    int32_t engine;
    phr_affine_costs costs;
    PairDesc* desc;
    PairOut* out;
    uint64_t* w2;      // 2-bit words per pair -> scanned in place to offsets
    uint64_t* wb;      // byte words per pair
    uint64_t* tb;      // text bound per pair
};

// Suffix lengths, seed validation, arena sizes of pair i.
__device__ __forceinline__ void prep_pair(const PrepParams& P, uint64_t i) {
    const uint32_t ql = P.in.q_len[i], tl = P.in.t_len[i];
    uint32_t qs = P.in.q_seed ? P.in.q_seed[i] : 0, ts = P.in.t_seed ? P.in.t_seed[i] : 0;
    if (P.engine == PHR_ENGINE_MYERS_GLOBAL) qs = ts = 0;
    PairDesc d = {};
    const bool invalid = qs > ql || ts > tl;
    d.qs = static_cast<int32_t>(qs);
    d.ts = static_cast<int32_t>(ts);
    d.qn = invalid ? 0 : static_cast<int32_t>(ql - qs);
    d.tn = invalid ? 0 : static_cast<int32_t>(tl - ts);
    d.trivial = (invalid || d.qn == 0 || d.tn == 0) ? 1 : 0;
    d.mode = 0;
    P.desc[i] = d;
    PairOut o = {};
    o.status = invalid ? PHR_INVALID_INPUT : -1;  // -1: not yet produced
    P.out[i] = o;
    const uint64_t qn = d.qn, tn = d.tn;
    P.w2[i] = d.trivial ? 0 : (qn + 15) / 16 + 4 + (tn + 15) / 16 + 4;
    P.wb[i] = d.trivial ? 0 : (qn + 3) / 4 + 4 + (tn + 3) / 4 + 4;
    P.tb[i] = 2 * (qn + tn) + 16;
}

__global__ void prep_sizes_kernel(PrepParams P) {
    const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (i < P.in.n) prep_pair(P, i);
}

__device__ __forceinline__ uint32_t code2(uint8_t b, bool& pure) {
    switch (b) {
        case 'A': return 0;
        case 'C': return 1;
        case 'G': return 2;
        case 'T': return 3;
        default: pure = false; return 0;
    }
}

// The first `keep` (0..4) of four ASCII bytes -> their 2-bit codes (A, C, G, T = 0..3) in
// the low 8 bits (the other bytes' codes are zero); `pure` turns false unless those bytes
// are all A, C, G or T. The code of A/C/G/T is bits 1-2 of the byte XOR bits 2-3 (0x41,
// 0x43, 0x47, 0x54 -> 0, 1, 2, 3); a byte is one of them exactly when the letter of its
// code ('A', 'C', 'G', 'T' picked by one byte permute) is the byte itself.
__device__ __forceinline__ uint32_t code2x4m(uint32_t x, int keep, bool& pure) {
    const uint32_t bytes = keep >= 4 ? 0xFFFFFFFFu : (1u << (8 * keep)) - 1u;
    const uint32_t c = ((x >> 1) ^ (x >> 2)) & 0x03030303u;
    const uint32_t sel = (c & 0x3u) | ((c >> 4) & 0x30u) | ((c >> 8) & 0x300u) | ((c >> 12) & 0x3000u);
    if (((__byte_perm(0x54474341u, 0u, sel) ^ x) & bytes) != 0) pure = false;
    uint32_t cm = c & bytes;
    cm |= cm >> 6;
    cm |= cm >> 12;
    return cm & 0xFFu;
}

// Writes "<n><op>" at p, returns its length.
__device__ uint32_t write_count_op(char* p, uint32_t n, char op) {
    const uint32_t nd = ndigits(n);
    for (int d = static_cast<int>(nd) - 1; d >= 0; --d) {
        p[d] = static_cast<char>('0' + n % 10);
        n /= 10;
    }
    p[nd] = op;
    return nd + 1;
}

struct PackParams {
    DevPairs in;
    int32_t engine;
    phr_affine_costs costs;
    PairDesc* desc;
    PairOut* out;
    const uint64_t* w2_off;
    const uint64_t* wb_off;
    const uint64_t* text_off;
    uint32_t* arena2;
    uint32_t* arenab;
    char* text;
    uint32_t* keys;
    uint32_t* vals;
    int wfa_g_short, wfa_g_long;
    int wfa_long_min;   // qn + tn from which a WFA pair gets wfa_g_long lanes
    int band_base;      // Myers band half-width base
    int big_min;        // qn + tn from which a linear WFA pair runs in register tiles
    int lane_ckpt;      // mode of the lane-per-pair Myers kernel
};

// 2-bit packing (16 bases per word) of both suffixes; a pair holding any byte other
// than A/C/G/T is also copied word-aligned to the byte arena and runs the byte path.
// Trivial pairs (an empty suffix) get their final result here. One warp per pair.
__device__ __forceinline__ void pack_pair(const PackParams& P, uint64_t i, int lane) {
    PairDesc d = P.desc[i];
    if (d.trivial) {
        if (lane == 0) {
            PairOut o = P.out[i];
            P.keys[i] = kInvalidKey;
            P.vals[i] = static_cast<uint32_t>(i);
            if (o.status == PHR_INVALID_INPUT) {
                o.ed = 0;
                o.t_consumed = 0;
                o.text_len = 0;
                P.out[i] = o;
                return;
            }
            char* t = P.text + P.text_off[i];
            uint32_t len = 0;
            o.status = PHR_OK;
            o.affine_score = 0;
            const int qn = d.qn, tn = d.tn;
            if (P.engine == PHR_ENGINE_MYERS_GLOBAL) {
                if (qn == 0) {
                    o.ed = tn;
                    if (tn > 0) len = write_count_op(t, tn, 'I');
                } else {
                    o.ed = qn;
                    len = write_count_op(t, qn, 'D');
                }
                o.t_consumed = tn;
            } else if (qn == 0) {
                o.ed = 0;  // wfa_simd.rs:194-203 / :365-367 / :592-601, :3793-3795
                o.t_consumed = 0;
            } else {      // tn == 0: every query base is query-extra
                o.ed = qn;
                len = write_count_op(t, qn, 'D');
                o.t_consumed = 0;
                if (P.engine == PHR_ENGINE_WFA_AFFINE) o.affine_score = P.costs.gap_open + qn * P.costs.gap_extend;
            }
            o.n_runs = len ? 1 : 0;
            o.text_len = len;
            P.out[i] = o;
        }
        return;
    }
    const uint8_t* qsrc = P.in.seq + P.in.q_off[i] + d.qs;
    const uint8_t* tsrc = (P.in.t_seq ? P.in.t_seq : P.in.seq) + P.in.t_off[i] + d.ts;
    const uint64_t w2 = P.w2_off[i];
    const uint64_t q2w = (d.qn + 15) / 16 + 4;
    bool pure = true;
    // bytes a lane may read with aligned 32-bit loads: those of the batch arena (targets
    // from a separate arena take the byte loop)
    const uintptr_t ok_lo = reinterpret_cast<uintptr_t>(P.in.seq);
    const uintptr_t ok_hi = ok_lo + P.in.seq_bytes;
    // query words then target words, dealt to the warp's lanes as one list
    const int nwq = (d.qn + 15) / 16, nwt = (d.tn + 15) / 16;
    for (int x = lane; x < nwq + nwt; x += 32) {
        const int side = x >= nwq;
        const int w = side ? x - nwq : x;
        const uint8_t* src = side ? tsrc : qsrc;
        const bool wide = !(side && P.in.t_seq);
        const int len = side ? d.tn : d.qn;
        uint32_t* dst = P.arena2 + w2 + (side ? q2w : 0);
        uint32_t word = 0;
        const int p0 = w * 16;
        const int lim = min(16, len - p0);
        const uint8_t* cp = src + p0;
        const uintptr_t a0 = reinterpret_cast<uintptr_t>(cp) & ~static_cast<uintptr_t>(3);
        if (wide && a0 >= ok_lo && a0 + 20 <= ok_hi) {
            // 16 bases from five aligned words, four bases per step; in the last word of a
            // sequence the bytes past its end are read (inside the arena) but neither
            // coded nor checked
            const uint32_t* wp = reinterpret_cast<const uint32_t*>(a0);
            const uint32_t sh = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(cp) & 3) * 8;
            uint32_t v[5];
#pragma unroll
            for (int j = 0; j < 5; ++j) v[j] = __ldg(wp + j);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int keep = min(max(lim - 4 * j, 0), 4);  // bytes of this group inside the sequence
                word |= code2x4m(__funnelshift_r(v[j], v[j + 1], sh), keep, pure) << (8 * j);
            }
        } else {
            for (int b = 0; b < lim; ++b) word |= code2(cp[b], pure) << (2 * b);
        }
        dst[w] = word;
    }
    pure = __all_sync(PHR_FULL_MASK, pure);
    if (pure) {
        d.mode = 0;
        d.q_word = w2;
        d.t_word = w2 + q2w;
    } else {
        const uint64_t wb = P.wb_off[i];
        const uint64_t qbw = (d.qn + 3) / 4 + 4;
        for (int side = 0; side < 2; ++side) {
            const uint8_t* src = side ? tsrc : qsrc;
            const int len = side ? d.tn : d.qn;
            uint32_t* dst = P.arenab + wb + (side ? qbw : 0);
            const int nw = (len + 3) / 4;
            for (int w = lane; w < nw; w += 32) {
                uint32_t word = 0;
                const int p0 = w * 4;
                const int lim = min(4, len - p0);
                for (int b = 0; b < lim; ++b) word |= static_cast<uint32_t>(src[p0 + b]) << (8 * b);
                dst[w] = word;
            }
        }
        d.mode = 1;
        d.q_word = wb;
        d.t_word = wb + qbw;
    }
    if (lane == 0) {
        P.desc[i] = d;
        int G;
        uint32_t len;
        if (P.engine == PHR_ENGINE_MYERS_FIT || P.engine == PHR_ENGINE_MYERS_GLOBAL) {
            G = next_pow2_cap32((d.qn + 63) / 64);
            // global 2-bit pairs whose band fits the lane kernel's window: one lane each
            if (P.engine == PHR_ENGINE_MYERS_GLOBAL && d.mode == 0) {
                const LaneBand b = lane_band(d.qn, d.tn, P.band_base);
                if (lane_slots(b.dmin, b.dmax, (d.qn + 63) / 64) <= kLaneMaxSlots - 2) G = 1;
            }
            const uint32_t nb = static_cast<uint32_t>((d.qn + 63) / 64);
            len = static_cast<uint32_t>(d.tn) * nb;
            if (fit_lanes(P.engine, P.in.n, P.lane_ckpt) && d.mode == 0 && nb <= kLaneMaxSlots) {
                G = 1;   // a warp's pairs of one block count, for the last block's score
                len = nb << 22 | min(static_cast<uint32_t>(d.tn), (1u << 22) - 1u);
            }
        } else {
            G = (d.qn + d.tn < P.wfa_long_min) ? P.wfa_g_short : P.wfa_g_long;
            len = static_cast<uint32_t>(d.qn + d.tn);
        }
        // register-tile pairs form segments of their own after the warp-group ones
        const int tw = tile_warps(P.engine, aff_tile_open(P.costs), P.big_min, P.wfa_long_min, d.qn, d.tn, d.mode);
        const uint32_t glog = tw == 0 ? static_cast<uint32_t>(__ffs(G) - 1) : tw == 1 ? kWarpTileSeg : kTileSeg;
        const uint32_t lk = 0x0FFFFFFFu - min(len, 0x0FFFFFFFu);  // longest first within a bucket
        P.keys[i] = (static_cast<uint32_t>(d.mode) << 31) | (glog << 28) | lk;
        P.vals[i] = static_cast<uint32_t>(i);
    }
}

__global__ void pack_kernel(PackParams P) {
    const uint64_t warp = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5;
    if (warp < P.in.n) pack_pair(P, warp, threadIdx.x & 31);
}

struct TaskBuild {
    const uint32_t* keys;      // sorted
    const uint32_t* order;     // sorted pair ids
    uint64_t n;
    uint32_t* head;            // scratch: segment head positions
    uint32_t* flag;
    uint32_t* tidx;
    uint32_t* task_first;
    uint8_t* task_count;
    uint8_t* task_group;
    uint32_t* ranges;          // {0, split, split, n_tasks}
    uint32_t* split_min;
    uint32_t* g1_min;          // first 2-bit task of more than one lane per pair
    const PairDesc* desc;
    int32_t engine;
    int32_t band_base;
    unsigned long long* need_max;
    uint64_t* task_need;          // per task
    unsigned int* need_hist;      // 64 buckets by bit length of the need
    int32_t big_min;              // WFA pairs for wfa.cu's CTA-per-pair kernels (not in the main
                                  // pass, so not in its slot statistics)
    int32_t lane_ckpt;            // lane kernel mode (its scratch need)
    uint32_t* tile_min;           // [4] first one-warp register-tile task of each symbol mode, first CTA one
    uint32_t* tile_ranges;        // {begin, end} of each of the four
    unsigned long long* tile_need;   // scratch wanted by the register-tile pairs: sum, largest
};

__device__ __forceinline__ bool key_tile(uint32_t k) { return ((k >> 28) & 7u) >= kWarpTileSeg; }
__device__ __forceinline__ int key_group(uint32_t k) { return key_tile(k) ? 32 : 1 << ((k >> 28) & 7); }
__device__ __forceinline__ uint32_t key_seg(uint32_t k) { return k >> 28; }

__global__ void task_head_kernel(TaskBuild T) {
    const uint64_t p = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (p >= T.n) return;
    const uint32_t k = T.keys[p];
    T.head[p] = (p == 0 || key_seg(T.keys[p - 1]) != key_seg(k)) ? static_cast<uint32_t>(p) : 0u;
}

__global__ void task_flag_kernel(TaskBuild T) {
    const uint64_t p = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (p >= T.n) return;
    const uint32_t k = T.keys[p];
    const uint32_t per = 32 / key_group(k);
    T.flag[p] = (k != kInvalidKey && ((p - T.head[p]) % per) == 0) ? 1u : 0u;
}

__device__ __forceinline__ uint64_t myers_need_est(int m, int n, int G, int band_base) {
    const int nb = (m + 63) >> 6;
    int E = min(band_base + abs(m - n) + (m >> 4), max(m, n));
    int W = min((2 * (E + 2) + 1 + 63) / 64 + 1, nb);
    uint64_t need = ((static_cast<uint64_t>(n) * W * 16) + 15) & ~15ull;  // 16-byte VP/HP records
    if (nb > G) need += (static_cast<uint64_t>(n) + 15) & ~15ull;
    need += (static_cast<uint64_t>(m + n + 2) * 4 + 15) & ~15ull;
    return need;
}

// Task of sorted position p; called by whole warps.
__device__ __forceinline__ void task_fill(const TaskBuild& T, uint64_t p) {
    // every lane stays to the warp-level reductions at the end; lanes without a task
    // contribute nothing to them
    const bool has_task = p < T.n && T.flag[p];
    uint64_t need = 0, tile_need = 0;
    uint32_t t_split = 0xFFFFFFFFu, t_g1 = 0xFFFFFFFFu, t_tile = 0xFFFFFFFFu;
    if (has_task) {
        const uint32_t k = T.keys[p];
        const int G = key_group(k);
        const uint32_t per = 32 / G;
        uint32_t cnt = 0;
        uint64_t region = 0;
        // lane-kernel tasks (global Myers, 2-bit, one lane per pair): window over the union band
        const bool fit = fit_lanes(T.engine, T.n, T.lane_ckpt);
        const bool lane_task = (T.engine == PHR_ENGINE_MYERS_GLOBAL || fit) && G == 1 && !((k >> 31) & 1);
        int dmin = 0x7fffffff, dmax = static_cast<int>(0x80000000), n_max = 0, m_max = 0;
        for (uint32_t c = 0; c < per && p + c < T.n; ++c) {
            const uint32_t kc = T.keys[p + c];
            if (kc == kInvalidKey || key_seg(kc) != key_seg(k)) break;
            const PairDesc d = T.desc[T.order[p + c]];
            if (lane_task) {
                const LaneBand b = lane_band(d.qn, d.tn, T.band_base);
                dmin = min(dmin, b.dmin);
                dmax = max(dmax, b.dmax);
                n_max = max(n_max, d.tn);
                m_max = max(m_max, d.qn);
            } else if (T.engine == PHR_ENGINE_MYERS_FIT || T.engine == PHR_ENGINE_MYERS_GLOBAL)
                need += myers_need_est(d.qn, d.tn, G, T.band_base);
            else if (key_tile(k))
                tile_need = T.engine == PHR_ENGINE_WFA_AFFINE
                                ? aff_tile_fixed_bytes(d.qn, d.tn) +
                                      tile_align(aff_tile_hist_bytes(tile_score_est(d.qn, d.mode)))
                                : tile_fixed_bytes(d.qn, d.tn) + tile_align(tile_hist_bytes(tile_score_est(d.qn, d.mode)));
            else if (!big_pair(T.engine, T.big_min, d.qn, d.tn))
                region = max(region, wfa_region_est(d.qn, d.tn, T.engine == PHR_ENGINE_WFA_AFFINE));
            ++cnt;
        }
        if (T.engine != PHR_ENGINE_MYERS_FIT && T.engine != PHR_ENGINE_MYERS_GLOBAL) need = region * per;
        if (lane_task && cnt) {
            const int nb = (m_max + 63) >> 6;
            need = lane_task_need(n_max, m_max, fit ? nb : lane_slots(dmin, dmax, nb), T.lane_ckpt);
        }
        const uint32_t t = T.tidx[p];
        T.task_first[t] = static_cast<uint32_t>(p);
        T.task_count[t] = static_cast<uint8_t>(cnt);
        T.task_group[t] = static_cast<uint8_t>(G);
        T.task_need[t] = need;
        if ((k >> 31) & 1) t_split = t;
        else if (G > 1) t_g1 = t;
        if (key_tile(k)) t_tile = t;
    }
    // one atomic per warp and value instead of one per task (a million tasks would
    // otherwise queue on the same three addresses)
    uint64_t nmax = need;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nmax = max(nmax, __shfl_xor_sync(PHR_FULL_MASK, nmax, o));
    t_split = __reduce_min_sync(PHR_FULL_MASK, t_split);
    t_g1 = __reduce_min_sync(PHR_FULL_MASK, t_g1);
    if (__any_sync(PHR_FULL_MASK, tile_need != 0)) {
        uint64_t sum = tile_need;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(PHR_FULL_MASK, sum, o);
        const uint32_t kind = has_task ? key_seg(T.keys[p]) : 0u;   // mode << 3 | segment
        for (int m = 0; m < 4; ++m) {
            const bool mine = kind == ((m & 1) << 3 | (m < 2 ? kWarpTileSeg : kTileSeg));
            const uint32_t f = __reduce_min_sync(PHR_FULL_MASK, mine ? t_tile : 0xFFFFFFFFu);
            if ((threadIdx.x & 31) == 0 && f != 0xFFFFFFFFu) atomicMin(T.tile_min + m, f);
        }
        uint64_t most = tile_need;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) most = max(most, __shfl_xor_sync(PHR_FULL_MASK, most, o));
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(T.tile_need, static_cast<unsigned long long>(sum));
            atomicMax(T.tile_need + 1, static_cast<unsigned long long>(most));
        }
    }
    const int bucket = need ? 64 - __clzll(need) : 64;   // 64: no histogram entry
    const uint32_t same = __match_any_sync(PHR_FULL_MASK, bucket);
    const int lane = threadIdx.x & 31;
    if (bucket < 64 && lane == __ffs(same) - 1) atomicAdd(&T.need_hist[bucket], static_cast<unsigned>(__popc(same)));
    if (lane == 0) {
        if (nmax) atomicMax(T.need_max, static_cast<unsigned long long>(nmax));
        if (t_split != 0xFFFFFFFFu) atomicMin(T.split_min, t_split);
        if (t_g1 != 0xFFFFFFFFu) atomicMin(T.g1_min, t_g1);
    }
}

__global__ void task_fill_kernel(TaskBuild T) {
    task_fill(T, blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x);
}

// Task ranges from the number of tasks and the reduced first tasks. One thread.
__device__ __forceinline__ void task_ranges(const TaskBuild& T, uint32_t nt) {
    const uint32_t split = min(__ldcg(T.split_min), nt);
    // segments of each mode in key order: warp groups, one-warp tiles, CTA tiles
    for (int m = 0; m < 2; ++m) {
        const uint32_t begin = m ? split : 0, end = m ? nt : split;
        const uint32_t cta = min(__ldcg(T.tile_min + 2 + m), end), warp = min(__ldcg(T.tile_min + m), cta);
        T.ranges[2 * m] = begin;
        T.ranges[2 * m + 1] = warp;
        T.tile_ranges[2 * m] = warp;
        T.tile_ranges[2 * m + 1] = cta;
        T.tile_ranges[4 + 2 * m] = cta;
        T.tile_ranges[4 + 2 * m + 1] = end;
    }
    // lane-kernel range {0, g1} and warp-group 2-bit range {g1, split} (global Myers)
    const uint32_t g1 = min(__ldcg(T.g1_min), split);
    T.ranges[28] = 0;
    T.ranges[29] = g1;
    T.ranges[30] = g1;
    T.ranges[31] = split;
}

__global__ void task_finalize_kernel(TaskBuild T) {
    task_ranges(T, T.n > 0 ? T.tidx[T.n - 1] + T.flag[T.n - 1] : 0);
}

// ---------------------------------------------------------------------------
// Small batches: one CTA does what the scans, the sort and the task build do for a large
// one, a thread per pair. A call on a few pairs is bound by its launches, copies and
// waits: 31 launches and 8 copies of 0.1 ms of kernels took 0.25 ms.
// ---------------------------------------------------------------------------
constexpr int kSmallPairs = 1024;
constexpr int kTinyPairs = 32;      // few enough to be packed by the same CTA, a warp each

// Exclusive sum over the CTA's kSmallPairs threads; `sh` holds a value per warp.
__device__ __forceinline__ uint64_t cta_excl_sum(uint64_t v, uint64_t* sh, uint64_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t up = __shfl_up_sync(PHR_FULL_MASK, incl, o);
        if (lane >= o) incl += up;
    }
    __syncthreads();   // sh may still be read from the last call
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    uint64_t before = 0, all = 0;
    for (int w = 0; w < kSmallPairs / 32; ++w) {
        const uint64_t x = sh[w];
        if (w < warp) before += x;
        all += x;
    }
    *total = all;
    return before + incl - v;
}

// Sorts the keys (stable: pair ids break ties) and builds the task list.
__device__ void small_tasks(const TaskBuild& T, const uint32_t* keys_in, uint32_t* keys_out, uint32_t* order_out,
                            uint64_t* sh_sort, uint64_t* sh_sum) {
    const int t = threadIdx.x, n = static_cast<int>(T.n);
    int m = 32;
    while (m < n) m <<= 1;
    sh_sort[t] = t < n ? static_cast<uint64_t>(keys_in[t]) << 32 | static_cast<uint32_t>(t) : ~0ull;
    __syncthreads();
    for (int k = 2; k <= m; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int o = t ^ j;
            if (t < m && o > t) {
                const uint64_t a = sh_sort[t], b = sh_sort[o];
                if ((a > b) == ((t & k) == 0)) {
                    sh_sort[t] = b;
                    sh_sort[o] = a;
                }
            }
            __syncthreads();
        }
    const uint32_t key = static_cast<uint32_t>(sh_sort[t] >> 32);
    const uint32_t id = static_cast<uint32_t>(sh_sort[t]);
    const bool first = t < n && (t == 0 || key_seg(static_cast<uint32_t>(sh_sort[t > 0 ? t - 1 : 0] >> 32)) != key_seg(key));
    if (t < n) {
        keys_out[t] = key;
        order_out[t] = id;
    }
    // start of this position's segment: the last `first` at or before it
    int head = first ? t : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) head = max(head, __shfl_up_sync(PHR_FULL_MASK, head, o));
    __syncthreads();
    if ((t & 31) == 31) sh_sum[t >> 5] = static_cast<uint64_t>(head);
    __syncthreads();
    for (int w = 0; w < t >> 5; ++w) head = max(head, static_cast<int>(sh_sum[w]));
    const uint32_t per = 32 / key_group(key);
    const bool task = t < n && key != kInvalidKey && ((t - head) % per) == 0;
    uint64_t nt = 0;
    const uint64_t at = cta_excl_sum(task ? 1 : 0, sh_sum, &nt);
    if (t < n) {
        T.flag[t] = task ? 1u : 0u;
        T.tidx[t] = static_cast<uint32_t>(at);
    }
    __syncthreads();
    task_fill(T, t);
    __syncthreads();
    if (t == 0) task_ranges(T, static_cast<uint32_t>(nt));
}

struct SmallBuild {
    PrepParams prep;
    PackParams pack;
    TaskBuild tasks;
    uint64_t *w2o, *wbo, *tbo;
    uint32_t* cnt;       // counter block, set up here
    uint32_t *keys_s, *order;
};

// Counter block, pair descriptors and arena offsets; tiny batches are packed and their
// tasks built as well.
__global__ void __launch_bounds__(kSmallPairs) small_build_kernel(SmallBuild B, bool tiny) {
    __shared__ uint64_t sh_sort[kSmallPairs];
    __shared__ uint64_t sh_sum[32];
    const int t = threadIdx.x, n = static_cast<int>(B.prep.in.n);
    if (t < 64) {   // the "first task" counters start at their maximum
        const bool is_min = t == 4 || t == 20 || (t >= 40 && t < 44);
        B.cnt[t] = is_min ? 0xFFFFFFFFu : 0u;
        B.tasks.need_hist[t] = 0;
    }
    uint64_t w2 = 0, wb = 0, tb = 0, total;
    if (t < n) {
        prep_pair(B.prep, t);
        w2 = B.prep.w2[t];
        wb = B.prep.wb[t];
        tb = B.prep.tb[t];
    }
    w2 = cta_excl_sum(w2, sh_sum, &total);
    wb = cta_excl_sum(wb, sh_sum, &total);
    tb = cta_excl_sum(tb, sh_sum, &total);
    if (t < n) {
        B.w2o[t] = w2;
        B.wbo[t] = wb;
        B.tbo[t] = tb;
    }
    if (!tiny) return;
    __syncthreads();
    if ((t >> 5) < n) pack_pair(B.pack, t >> 5, t & 31);
    __syncthreads();
    small_tasks(B.tasks, B.pack.keys, B.keys_s, B.order, sh_sort, sh_sum);
}

__global__ void __launch_bounds__(kSmallPairs) small_tasks_kernel(SmallBuild B) {
    __shared__ uint64_t sh_sort[kSmallPairs];
    __shared__ uint64_t sh_sum[32];
    small_tasks(B.tasks, B.pack.keys, B.keys_s, B.order, sh_sort, sh_sum);
}

// Redo pass task list: one pair per task, in redo order.
__global__ void redo_tasks_kernel(const uint32_t* redo_list, const uint32_t* redo_count, const PairDesc* desc,
                                  int32_t engine, int aff_open, int wfa_g_short, int wfa_g_long, int wfa_long_min, int32_t big_min,
                                  uint32_t* task_first, uint8_t* task_count, uint8_t* task_group,
                                  uint32_t* ranges) {
    const uint32_t n = *redo_count;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) {
        ranges[0] = 0;
        ranges[1] = n;
    }
    if (t >= n) return;
    const PairDesc d = desc[redo_list[t]];
    int G;
    if (engine == PHR_ENGINE_MYERS_FIT || engine == PHR_ENGINE_MYERS_GLOBAL)
        G = next_pow2_cap32((d.qn + 63) / 64);
    else
        G = (d.qn + d.tn < wfa_long_min) ? wfa_g_short : wfa_g_long;
    task_first[t] = t;
    task_count[t] = 1;
    task_group[t] = static_cast<uint8_t>(G);
    const int tw = tile_warps(engine, aff_open, big_min, wfa_long_min, d.qn, d.tn, d.mode);
    if (tw > 1) task_group[t] = kCtaTileTask | 32;
    else if (tw == 1) task_group[t] = kWarpTileTask | 32;
    else if (big_pair(engine, big_min, d.qn, d.tn)) task_group[t] = kBigTask | 32;
}

struct FinishParams {
    uint64_t n;
    int32_t engine;
    const PairDesc* desc;
    const PairOut* out;
    const uint64_t* text_off;
    const char* text;
    uint64_t* cig_off;       // exclusive scan of text_len
    phr_alignment* aln;
    char* cigar;
    uint64_t cigar_capacity;
    uint32_t* error_flag;
    uint64_t cigar_base;
    int per_warp;            // pairs a warp writes (1..32)
    const uint32_t* redo_count;
    uint64_t* total;         // text bytes of all pairs
};

__global__ void text_len_kernel(const PairOut* out, uint64_t n, uint64_t* len) {
    const uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const PairOut o = out[i];
    len[i] = (o.status == PHR_OK) ? o.text_len : 0;
}

// Copies len bytes with one warp: words at the destination's 4-byte boundaries, funnelled
// from the source's, single bytes at both ends (and for short texts). Reads stay within the
// source's aligned words.
__device__ __forceinline__ void copy_text(char* dst, const char* src, uint32_t len, int lane) {
    if (len < 96) {
        for (uint32_t c = lane; c < len; c += 32) dst[c] = src[c];
        return;
    }
    const uint32_t head = static_cast<uint32_t>(-reinterpret_cast<intptr_t>(dst)) & 3u;
    if (static_cast<uint32_t>(lane) < head) dst[lane] = src[lane];
    const char* s = src + head;
    uint32_t* d = reinterpret_cast<uint32_t*>(dst + head);
    const uint32_t words = (len - head) / 4;
    const uint32_t sh = (static_cast<uint32_t>(reinterpret_cast<uintptr_t>(s)) & 3u) * 8;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(reinterpret_cast<uintptr_t>(s) & ~static_cast<uintptr_t>(3));
    if (sh == 0) {
#pragma unroll 4
        for (uint32_t i = lane; i < words; i += 32) d[i] = w[i];
    } else {
#pragma unroll 4
        for (uint32_t i = lane; i < words; i += 32) d[i] = __funnelshift_r(w[i], w[i + 1], sh);
    }
    const uint32_t done = head + 4 * words;
    if (done + lane < len) dst[done + lane] = src[done + lane];
}

// Packs CIGAR text and writes the phr_alignment records. One warp per F.per_warp
// consecutive pairs: lane l writes pair first + l's record (the warp's records are
// contiguous), then the lanes copy the pairs' texts one pair after the other. 32 pairs per
// warp in a large batch; fewer when there are few pairs, whose texts then are copied side
// by side (500 texts of ~3 kB: 0.60 ms with 32 per warp and byte copies, below 0.01 ms now).
__device__ __forceinline__ void finish_pairs(const FinishParams& F, uint64_t first, int lane) {
    const uint64_t i = first + lane;
    uint64_t off = 0, toff = 0;
    uint32_t len = 0;
    bool copy = false;
    if (lane < F.per_warp && i < F.n) {
        const PairOut o = F.out[i];
        if (o.status == -1) {
            atomicOr(F.error_flag, 8u);
        } else {
            const PairDesc d = F.desc[i];
            off = F.cig_off[i];
            toff = F.text_off[i];
            len = (o.status == PHR_OK) ? o.text_len : 0;
            copy = off + len <= F.cigar_capacity;
            if (!copy) atomicOr(F.error_flag, 16u);
            phr_alignment a;
            a.status = o.status;
            a.edit_distance = o.status == PHR_OK ? static_cast<uint32_t>(o.ed) : 0;
            a.cigar_off = F.cigar_base + off;
            a.cigar_len = len;
            a.affine_score = o.status == PHR_OK ? static_cast<uint32_t>(o.affine_score) : 0;
            if (F.engine == PHR_ENGINE_MYERS_GLOBAL) {
                a.query_start = 0;
                a.query_end = static_cast<uint32_t>(d.qn);
                a.target_start = 0;
                a.target_end = static_cast<uint32_t>(d.tn);
            } else if (o.status != PHR_OK) {
                a.query_start = a.query_end = a.target_start = a.target_end = 0;
            } else {
                a.query_start = static_cast<uint32_t>(d.qs);
                a.query_end = static_cast<uint32_t>(d.qs + d.qn);
                a.target_start = static_cast<uint32_t>(d.ts);
                a.target_end = static_cast<uint32_t>(d.ts + o.t_consumed);
            }
            F.aln[i] = a;
        }
    }
    const unsigned todo = __ballot_sync(PHR_FULL_MASK, copy && len > 0);
    for (unsigned m = todo; m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        const uint32_t lj = __shfl_sync(PHR_FULL_MASK, len, j);
        const uint64_t oj = __shfl_sync(PHR_FULL_MASK, off, j);
        const uint64_t tj = __shfl_sync(PHR_FULL_MASK, toff, j);
        copy_text(F.cigar + oj, F.text + tj, lj, lane);
    }
}

// Launched before the host knows how the pass went: nothing is written when pairs are to be
// redone or the text does not fit (the host looks at both next).
__device__ __forceinline__ bool finish_blocked(const FinishParams& F) {
    return __ldcg(F.redo_count) != 0 || __ldcg(F.total) > F.cigar_capacity;
}

__global__ void finish_kernel(FinishParams F) {
    const uint64_t first =
        ((blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5) * static_cast<uint64_t>(F.per_warp);
    if (first >= F.n || finish_blocked(F)) return;
    finish_pairs(F, first, threadIdx.x & 31);
}

// The tail of a small batch in one CTA: text offsets and total, and with `texts` the records
// and texts too.
__global__ void __launch_bounds__(kSmallPairs) small_tail_kernel(FinishParams F, uint64_t* tlen, bool texts) {
    __shared__ uint64_t sh_sum[32];
    const int t = threadIdx.x;
    uint64_t len = 0, total = 0;
    if (t < static_cast<int>(F.n)) {
        const PairOut o = F.out[t];
        len = o.status == PHR_OK ? o.text_len : 0;
    }
    const uint64_t off = cta_excl_sum(len, sh_sum, &total);
    if (t < static_cast<int>(F.n)) {
        tlen[t] = len;
        F.cig_off[t] = off;
    }
    if (t == 0) *F.total = total;
    __threadfence_block();
    __syncthreads();
    if (!texts || *F.redo_count != 0 || total > F.cigar_capacity) return;
    const uint64_t first = static_cast<uint64_t>(t >> 5) * F.per_warp;   // per_warp covers n with 32 warps
    if (first < F.n) finish_pairs(F, first, t & 31);
}

__global__ void total_kernel(const uint64_t* off, const uint64_t* len, uint64_t n, uint64_t* total) {
    *total = n ? off[n - 1] + len[n - 1] : 0;
}

inline unsigned blocks_for(uint64_t n, unsigned t) { return static_cast<unsigned>((n + t - 1) / t); }

}  // namespace

namespace {
__global__ void sum_lengths_kernel(const uint32_t* a, const uint32_t* b, uint64_t n, unsigned long long* out) {
    unsigned long long acc = 0;
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        acc += static_cast<unsigned long long>(a[i]) + b[i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(PHR_FULL_MASK, acc, o);
    if ((threadIdx.x & 31) == 0 && acc) atomicAdd(out, acc);
}

// The same for few lengths, one CTA: no counter to clear first.
__global__ void sum_lengths_small_kernel(const uint32_t* a, const uint32_t* b, uint32_t n, unsigned long long* out) {
    __shared__ unsigned long long sh[32];
    unsigned long long acc = 0;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) acc += static_cast<unsigned long long>(a[i]) + b[i];
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(PHR_FULL_MASK, acc, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (unsigned w = 1; w < blockDim.x / 32; ++w) acc += sh[w];
        *out = acc;
    }
}
}  // namespace

uint64_t device_length_sum(Ctx* ctx, const uint32_t* a, const uint32_t* b, uint64_t n, cudaError_t* err) {
    *err = cudaSuccess;
    if (!ctx->d_counters) {
        *err = cudaMalloc(&ctx->d_counters, 256);
        if (*err != cudaSuccess) return 0;
    }
    if (!ctx->h_pinned) {
        *err = cudaMallocHost(&ctx->h_pinned, kPinnedBytes);
        if (*err != cudaSuccess) return 0;
    }
    unsigned long long* d = reinterpret_cast<unsigned long long*>(ctx->d_counters);
    unsigned long long* h = static_cast<unsigned long long*>(ctx->h_pinned);
    cudaStream_t st = ctx->stream;
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>((n + 255) / 256, 4ull * ctx->sm_count));
    if (n <= 16384) {
        KernelScope ks(ctx, "sum_lengths");
        sum_lengths_small_kernel<<<1, 1024, 0, st>>>(a, b, static_cast<uint32_t>(n), d);
    } else {
        if ((*err = cudaMemsetAsync(d, 0, 8, st)) != cudaSuccess) return 0;
        KernelScope ks(ctx, "sum_lengths");
        sum_lengths_kernel<<<std::max(1u, grid), 256, 0, st>>>(a, b, n, d);
    }
    if ((*err = cudaMemcpyAsync(h, d, 8, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return 0;
    if ((*err = cudaStreamSynchronize(st)) != cudaSuccess) return 0;
    return *h;
}

size_t extend_arena_need(uint64_t n, uint64_t seq_bytes, uint64_t sum_qt) {
    size_t s = 0;
    auto add = [&](size_t b) { s += (b + 511) / 256 * 256; };
    add(n * sizeof(PairDesc));
    add(n * sizeof(PairOut));
    add(n * 8 * 3);                       // w2, wb, tb (scanned in place)
    add(n * 8 * 3);                       // scan outputs
    add((sum_qt / 16 + 12 * n + 64) * 4);  // 2-bit arena
    add((sum_qt / 4 + 12 * n + 64) * 4);   // byte arena
    add(2 * sum_qt + 16 * n + 64);        // text staging
    add(n * 4 * 4);                       // keys/vals (2x for sort)
    add(n * 4 * 6);                       // task build scratch
    add(n * 6);                           // task count/group
    add(n * 8 * 2);                       // text len + cigar offsets
    add(n * 4);                           // redo list
    add(n * 8 * 4 + 256);                 // task needs, redo needs, redo task offsets/lengths
    add(64ull << 20);                     // CUB temp
    add(4096);
    return s;
}

phr_status run_extend(Ctx* ctx, phr_engine engine, const DevPairs& in, phr_affine_costs costs, DevResults* res,
                      uint64_t sum_qt) {
    const uint64_t n = in.n;
    cudaStream_t st = ctx->stream;
    res->cigar_used = 0;
    if (n == 0) return PHR_OK;
    if (n > 0xFFFFFFF0ull) return set_error(ctx, PHR_ERR_ARG, "too many pairs in one batch");
    HostScope hs_setup(ctx, "host:extend_setup");
    DeviceArena& A = ctx->arena;
    A.reset();
    PHR_CUDA_TRY(ctx, A.reserve(extend_arena_need(n, in.seq_bytes, sum_qt)));
    auto take = [&](size_t b) { return A.take(b); };
    PairDesc* desc = static_cast<PairDesc*>(take(n * sizeof(PairDesc)));
    PairOut* pout = static_cast<PairOut*>(take(n * sizeof(PairOut)));
    uint64_t* w2 = static_cast<uint64_t*>(take(n * 8));
    uint64_t* wb = static_cast<uint64_t*>(take(n * 8));
    uint64_t* tb = static_cast<uint64_t*>(take(n * 8));
    uint64_t* w2o = static_cast<uint64_t*>(take(n * 8));
    uint64_t* wbo = static_cast<uint64_t*>(take(n * 8));
    uint64_t* tbo = static_cast<uint64_t*>(take(n * 8));
    // per sequence ceil(len/16)+4 (2-bit) / ceil(len/4)+4 (byte) words: <= len/16 + 5 per sequence
    uint32_t* arena2 = static_cast<uint32_t*>(take((sum_qt / 16 + 12 * n + 64) * 4));
    uint32_t* arenab = static_cast<uint32_t*>(take((sum_qt / 4 + 12 * n + 64) * 4));
    char* text = static_cast<char*>(take(2 * sum_qt + 16 * n + 64));
    uint32_t* keys = static_cast<uint32_t*>(take(n * 4));
    uint32_t* vals = static_cast<uint32_t*>(take(n * 4));
    uint32_t* keys_s = static_cast<uint32_t*>(take(n * 4));
    uint32_t* order = static_cast<uint32_t*>(take(n * 4));
    uint32_t* head = static_cast<uint32_t*>(take(n * 4));
    uint32_t* head_s = static_cast<uint32_t*>(take(n * 4));
    uint32_t* flag = static_cast<uint32_t*>(take(n * 4));
    uint32_t* tidx = static_cast<uint32_t*>(take(n * 4));
    uint32_t* task_first = static_cast<uint32_t*>(take(n * 4));
    uint32_t* redo_list = static_cast<uint32_t*>(take(n * 4));
    uint8_t* task_count = static_cast<uint8_t*>(take(n));
    uint8_t* task_group = static_cast<uint8_t*>(take(n));
    uint64_t* tlen = static_cast<uint64_t*>(take(n * 8));
    uint64_t* cigoff = static_cast<uint64_t*>(take(n * 8));
    uint64_t* task_need = static_cast<uint64_t*>(take(n * 8));
    unsigned long long* redo_need = static_cast<unsigned long long*>(take(n * 8));
    uint64_t* rtask_off = static_cast<uint64_t*>(take(n * 8));
    uint64_t* rtask_len = static_cast<uint64_t*>(take(n * 8));
    // counters: [0..3] ranges, [4] split_min, [5] queue head 0, [6] queue head 1,
    // [7] redo count, [8..9] need max (u64), [10] error flag, [12..13] total (u64), [14..17] redo ranges,
    // [20] first multi-lane 2-bit task, [21] queue head of the kernel for short WFA pairs, [22..23] range of
    // the pairs it left (from 0), [24..25] CTA-kernel queue heads, [26] lane-kernel queue head,
    // [28..31] lane-kernel and warp-group 2-bit ranges (global Myers), [32..39] work counters (u64),
    // [40..43] first register-tile task of each kind (one warp 2-bit / bytes, CTA 2-bit / bytes),
    // [44..51] their ranges, [52..55] their scratch need: sum, largest (u64), [56..59] their queue
    // heads, [60..61] pool bytes taken (u64), [62] deferred register-tile pairs, [63] their queue head
    // The histogram of the tasks' needs follows, so that one copy brings both back.
    uint32_t* cnt = static_cast<uint32_t*>(take(512));
    if (!cnt) return set_error(ctx, PHR_ERR_OOM, "device arena exhausted");
    unsigned int* need_hist = cnt + 64;
    if (!ctx->h_pinned) PHR_CUDA_TRY(ctx, cudaMallocHost(&ctx->h_pinned, kPinnedBytes));
    const uint32_t* h_cnt = static_cast<const uint32_t*>(ctx->h_pinned);   // the host's copy of both
    auto read_counters = [&](size_t bytes) -> cudaError_t {
        const cudaError_t e = cudaMemcpyAsync(ctx->h_pinned, cnt, bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    };
    unsigned long long* need_max = reinterpret_cast<unsigned long long*>(cnt + 8);
    uint64_t* total = reinterpret_cast<uint64_t*>(cnt + 12);
    const unsigned T = 256;
    uint64_t pass_budget = std::min(ctx->scratch_budget, ctx->pass_budget);
    const bool small = n <= kSmallPairs;
    // lanes per short WFA pair: affine and linear tune separately
    const int g_short = engine == PHR_ENGINE_WFA_AFFINE ? ctx->tune.wfa_affine_group_short : ctx->tune.wfa_group_short;
    const PrepParams pp{in, engine, costs, desc, pout, w2, wb, tb};
    const PackParams pk{in, engine, costs, desc, pout, w2o, wbo, tbo, arena2, arenab, text, keys, vals,
                        g_short, ctx->tune.wfa_group_long, ctx->tune.wfa_long_min,
                        ctx->tune.myers_band_base, ctx->tune.wfa_big_min, ctx->tune.myers_lane_ckpt};
    TaskBuild tbp{keys_s, order, n, small ? head_s : head, flag, tidx, task_first, task_count, task_group, cnt, cnt + 4,
                  cnt + 20, desc, engine, ctx->tune.myers_band_base, need_max, task_need, need_hist,
                  ctx->tune.wfa_big_min, ctx->tune.myers_lane_ckpt, cnt + 40, cnt + 44, reinterpret_cast<unsigned long long*>(cnt + 52)};
    size_t t_need = 0, tn_ = 0;
    void* tmp = nullptr;
    if (small) {
        const SmallBuild sb{pp, pk, tbp, w2o, wbo, tbo, cnt, keys_s, order};
        const bool tiny = n <= kTinyPairs;
        {
            KernelScope ks(ctx, "small_build");
            small_build_kernel<<<1, kSmallPairs, 0, st>>>(sb, tiny);
        }
        if (!tiny) {
            {
                KernelScope ks(ctx, "pack");
                pack_kernel<<<blocks_for(n * 32, T), T, 0, st>>>(pk);
            }
            KernelScope ks(ctx, "small_tasks");
            small_tasks_kernel<<<1, kSmallPairs, 0, st>>>(sb);
        }
    } else {
        PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt, 0, 512, st));   // the histogram follows the counters
        PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 4, 0xFF, 4, st));
        PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 20, 0xFF, 4, st));
        PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 40, 0xFF, 16, st));
        // CUB temp sizes
        size_t t_sort = 0, t_scan = 0, t_max = 0, t_scan32 = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, t_sort, keys, keys_s, vals, order, static_cast<int>(n), 0, 32, st);
        cub::DeviceScan::ExclusiveSum(nullptr, t_scan, w2, w2o, static_cast<int>(n), st);
        cub::DeviceScan::InclusiveScan(nullptr, t_max, head, head_s, cub::Max(), static_cast<int>(n), st);
        cub::DeviceScan::ExclusiveSum(nullptr, t_scan32, flag, tidx, static_cast<int>(n), st);
        t_need = std::max({t_sort, t_scan, t_max, t_scan32});
        tmp = take(t_need);
        if (!tmp) return set_error(ctx, PHR_ERR_OOM, "device arena exhausted (cub)");
        {
            KernelScope ks(ctx, "prep_sizes");
            prep_sizes_kernel<<<blocks_for(n, T), T, 0, st>>>(pp);
        }
        tn_ = t_need;
        cub::DeviceScan::ExclusiveSum(tmp, tn_, w2, w2o, static_cast<int>(n), st);
        tn_ = t_need;
        cub::DeviceScan::ExclusiveSum(tmp, tn_, wb, wbo, static_cast<int>(n), st);
        tn_ = t_need;
        cub::DeviceScan::ExclusiveSum(tmp, tn_, tb, tbo, static_cast<int>(n), st);
        {
            KernelScope ks(ctx, "pack");
            pack_kernel<<<blocks_for(n * 32, T), T, 0, st>>>(pk);
        }
        tn_ = t_need;
        cub::DeviceRadixSort::SortPairs(tmp, tn_, keys, keys_s, vals, order, static_cast<int>(n), 0, 32, st);
        {
            KernelScope ks(ctx, "task_head");
            task_head_kernel<<<blocks_for(n, T), T, 0, st>>>(tbp);
        }
        tn_ = t_need;
        cub::DeviceScan::InclusiveScan(tmp, tn_, head, head_s, cub::Max(), static_cast<int>(n), st);
        tbp.head = head_s;
        {
            KernelScope ks(ctx, "task_flag");
            task_flag_kernel<<<blocks_for(n, T), T, 0, st>>>(tbp);
        }
        tn_ = t_need;
        cub::DeviceScan::ExclusiveSum(tmp, tn_, flag, tidx, static_cast<int>(n), st);
        {
            KernelScope ks(ctx, "task_fill");
            task_fill_kernel<<<blocks_for(n, T), T, 0, st>>>(tbp);
        }
        {
            KernelScope ks(ctx, "task_finalize");
            task_finalize_kernel<<<1, 1, 0, st>>>(tbp);
        }
    }

    // Main-pass slot: the smallest power of two that covers 99.5 % of the tasks (and no
    // less than the largest task when that still fits a full grid); tasks needing more
    // are deferred to the redo passes, which size scratch per task.
    PHR_CUDA_TRY(ctx, read_counters(512));
    uint64_t h_need = 0;
    std::memcpy(&h_need, h_cnt + 8, 8);
    unsigned int h_hist[64];
    std::memcpy(h_hist, h_cnt + 64, sizeof(h_hist));
    uint32_t h_ranges[4];
    std::memcpy(h_ranges, h_cnt, sizeof(h_ranges));
    const bool lanes = engine == PHR_ENGINE_MYERS_GLOBAL || fit_lanes(engine, n, ctx->tune.myers_lane_ckpt);
    const uint32_t n_lane = lanes ? h_cnt[29] - h_cnt[28] : 0;
    const uint32_t n_group2 = lanes ? h_cnt[31] - h_cnt[30] : h_ranges[1] - h_ranges[0];
    const uint32_t n_groupb = h_ranges[3] - h_ranges[2];
    const bool any_2bit = h_ranges[2] > 0, any_bytes = h_cnt[51] > h_ranges[2];
    PHR_CUDA_TRY(ctx, cudaGetLastError());
    hs_setup.stop();
    uint32_t n_tile[4], n_tiles = 0;
    for (int i = 0; i < 4; ++i) n_tiles += n_tile[i] = h_cnt[45 + 2 * i] - h_cnt[44 + 2 * i];
    uint64_t tile_need[2];   // sum, largest
    std::memcpy(tile_need, h_cnt + 52, 16);
    {
        uint64_t n_tasks = 0;  // tasks of the main pass with a scratch need
        for (int b = 0; b < 64; ++b) n_tasks += h_hist[b];
        const uint64_t full_grid_warps =
            static_cast<uint64_t>(ctx->sm_count) * ctx->tune.max_blocks_per_sm * (ctx->tune.block_threads / 32);
        if (h_need * full_grid_warps > ctx->scratch_budget && n_tasks > 0) {
            uint64_t acc = 0, slot = 4096;
            for (int b = 0; b < 64; ++b) {
                acc += h_hist[b];
                slot = b >= 63 ? ~0ull : (1ull << b);
                if (acc * 1000 >= n_tasks * 995) break;
            }
            h_need = std::min(h_need, std::max<uint64_t>(slot, 64 << 10));
        }
    }

    const bool is_myers = engine == PHR_ENGINE_MYERS_FIT || engine == PHR_ENGINE_MYERS_GLOBAL;
    ExtendParams P{};
    P.desc = desc;
    P.out = pout;
    P.packed2 = arena2;
    P.bytes = arenab;
    P.text = text;
    P.text_off = tbo;
    P.scratch = nullptr;
    P.redo_list = redo_list;
    P.redo_count = cnt + 7;
    P.redo_need_max = need_max;
    P.redo_need = redo_need;
    P.task_need = task_need;
    P.engine = engine;
    P.full_band = 0;
    P.band_base = ctx->tune.myers_band_base;
    P.lane_ckpt = ctx->tune.myers_lane_ckpt;
    P.costs = costs;
    P.error_flag = cnt + 10;
    P.big_min = ctx->tune.wfa_big_min;
    P.big_smem = static_cast<uint32_t>(ctx->tune.wfa_big_smem);
    P.work = reinterpret_cast<unsigned long long*>(cnt + 32);

    const int block = ctx->tune.block_threads;
    // main pass (per_task false): per-warp slots of `slot` bytes; redo passes: per-task
    // scratch (P.task_off / P.task_len set by the caller, `per_task_total` bytes in all,
    // `n_tasks_hint` tasks)
    uint64_t tile_pool = 0;   // of the main pass
    int cluster_max = 1;      // most CTAs that a long pair left by its own is given
    if (n_tile[2] + n_tile[3] > 0 && ctx->tune.wfa_cluster_max > 1) {
        if (ctx->cluster_fit == 0) ctx->cluster_fit = wfa_cluster_fit(P.big_smem);
        cluster_max = std::min(ctx->cluster_fit, ctx->tune.wfa_cluster_max);
    }
    auto launch_pass = [&](const uint32_t* ord, const uint32_t* tfirst, const uint8_t* tcount, const uint8_t* tgroup,
                           const uint32_t* range0, const uint32_t* range1, uint64_t slot, int full_band,
                           bool per_task = false, uint64_t per_task_total = 0,
                           uint64_t n_tasks_hint = 0) -> phr_status {
        const uint64_t warps_per_block = block / 32;
        uint64_t grid = static_cast<uint64_t>(ctx->sm_count) * ctx->tune.max_blocks_per_sm;
        uint64_t pool = 0;
        if (!per_task) {
            slot = std::max<uint64_t>((slot + 255) & ~255ull, 4096);
            // grid: resident blocks per SM, no more warps than tasks, shrunk to the scratch budget
            grid = std::max<uint64_t>(1, std::min<uint64_t>(grid, (h_ranges[3] + warps_per_block - 1) / warps_per_block));
            while (grid > 1 && grid * warps_per_block * slot > ctx->scratch_budget) grid = (grid + 1) / 2;
            // The register-tile pairs run after the group kernels and reuse the buffer from its
            // start. Teams keep their chunks from pair to pair and chunks grow by doubling:
            // twice what the pairs in flight want; a small batch gets room for any divergence.
            pool = 0;
            if (n_tiles > 0) {
                const uint64_t teams = n_tile[0] + n_tile[1] > 0 ? 16ull * ctx->sm_count : ctx->sm_count;
                pool = std::min<uint64_t>(2 * tile_need[0], 2 * teams * tile_need[1]);
                pool = std::max<uint64_t>(pool, std::min<uint64_t>(16 * tile_need[0], 1ull << 30)) + (1 << 20);
                pool = std::min<uint64_t>(pool, pass_budget);
            }
            const uint64_t slots = grid * warps_per_block * slot;
            cudaError_t e = ctx->scratch.reserve(std::max(slots, pool));
            // the pool is what is wanted, not what is needed: where the device has less to give,
            // pairs that do not fit follow in redo passes, which then keep to the same
            while (e == cudaErrorMemoryAllocation && pool > std::max<uint64_t>(slots, 64 << 20)) {
                cudaGetLastError();
                pass_budget = pool /= 2;
                e = ctx->scratch.reserve(std::max(slots, pool));
            }
            PHR_CUDA_TRY(ctx, e);
            tile_pool = pool;
        } else {
            grid = std::max<uint64_t>(1, std::min<uint64_t>(grid, (n_tasks_hint + warps_per_block - 1) / warps_per_block));
            PHR_CUDA_TRY(ctx, ctx->scratch.reserve(per_task_total));
        }
        P.scratch = reinterpret_cast<uint8_t*>(ctx->scratch.base);
        P.slot_bytes = slot;
        P.full_band = full_band;
        P.tasks.order = ord;
        P.tasks.task_first = tfirst;
        P.tasks.task_count = tcount;
        P.tasks.task_group = tgroup;
        // the queue heads start at zero with the counter block
        if (per_task) PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 5, 0, 8, st));
        static const char* const names[2][3][2] = {
            {{"myers", "myers_bytes"}, {"wfa_linear", "wfa_linear_bytes"}, {"wfa_affine", "wfa_affine_bytes"}},
            {{"myers_redo", "myers_bytes_redo"}, {"wfa_linear_redo", "wfa_linear_bytes_redo"},
             {"wfa_affine_redo", "wfa_affine_bytes_redo"}}};
        const int ek = is_myers ? 0 : engine == PHR_ENGINE_WFA_LINEAR ? 1 : 2;
        const char* kname = names[per_task][ek][0];
        const char* kname_b = names[per_task][ek][1];
        if (!per_task && lanes) range0 = cnt + 30;
        if (!per_task && n_lane > 0) {
            // 2-bit pairs of one lane each (tasks [0, g1)); the warp-group kernel
            // below takes the remaining 2-bit tasks [g1, split)
            const LaneGrid lg = lane_grid(grid * warps_per_block, ctx->sm_count, myers_lane_blocks_per_sm(P.lane_ckpt));
            P.tasks.range = cnt + 28;
            P.queue_head = cnt + 26;
            {
                KernelScope ks(ctx, "myers_lane");
                launch_myers_lane(P, lg, st);
            }
        }
        P.tasks.range = range0;
        const uint32_t short_min = engine == PHR_ENGINE_WFA_LINEAR ? kShortLinearMin : kShortAffineMin;
        if (!per_task && (engine == PHR_ENGINE_WFA_LINEAR || (engine == PHR_ENGINE_WFA_AFFINE && aff_tile_open(costs) != 0)) &&
            P.big_min > 0 && n_group2 > short_min * static_cast<uint32_t>(ctx->sm_count)) {
            // most short pairs of a large batch end in the kernel for them alone, the rest
            // follow below from its list
            P.queue_head = cnt + 21;
            KernelScope ks(ctx, kname);
            if (launch_wfa_short(P, grid * warps_per_block * slot, ctx->sm_count, ctx->tune.max_blocks_per_sm, head, cnt + 23,
                                 st) > 0) {
                P.pair_list = head;
                P.tasks.range = cnt + 22;
            }
        }
        P.queue_head = cnt + 5;
        if (per_task ? any_2bit : n_group2 > 0) {
            KernelScope ks(ctx, kname);
            if (is_myers)
                launch_myers(P, static_cast<int>(grid), block, st);
            else if (engine == PHR_ENGINE_WFA_LINEAR)
                launch_wfa_linear(P, static_cast<int>(grid), block, st);
            else
                launch_wfa_affine(P, static_cast<int>(grid), block, st);
        }
        P.pair_list = nullptr;
        P.tasks.range = range1;
        P.queue_head = cnt + 6;
        if (per_task ? any_bytes : n_groupb > 0) {
            KernelScope ks(ctx, kname_b);
            if (is_myers)
                launch_myers_bytes(P, static_cast<int>(grid), block, st);
            else if (engine == PHR_ENGINE_WFA_LINEAR)
                launch_wfa_linear_bytes(P, static_cast<int>(grid), block, st);
            else
                launch_wfa_affine_bytes(P, static_cast<int>(grid), block, st);
        }
        const bool tiles = engine == PHR_ENGINE_WFA_LINEAR ||
                           (engine == PHR_ENGINE_WFA_AFFINE && aff_tile_open(costs) != 0);
        if (tiles && P.big_min > 0 && (per_task ? n_tasks_hint : n_tiles) > 0) {
            // register tiles: long pairs one CTA each (one per SM), the others a warp each
            if (per_task) PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 56, 0, 16, st));
            static const char* const tile_names[2][4] = {
                {"wfa_linear_tile", "wfa_linear_tile_bytes", "wfa_linear_big", "wfa_linear_big_bytes"},
                {"wfa_affine_tile", "wfa_affine_tile_bytes", "wfa_affine_big", "wfa_affine_big_bytes"}};
            const bool affine = engine == PHR_ENGINE_WFA_AFFINE;
            for (int i = 3; i >= 0; --i) {   // the longest first
                const uint64_t nt = per_task ? (((i & 1) ? any_bytes : any_2bit) ? n_tasks_hint : 0) : n_tile[i];
                if (nt == 0) continue;
                const bool cta = i >= 2;
                const TileLaunch tl{per_task ? nullptr : reinterpret_cast<unsigned long long*>(cnt + 60), pool,
                                    cta ? kTileChunk : kWarpTileChunk,
                                    per_task || !cta || cluster_max == 1 ? 0 : kTileDeferStep, ctx->sm_count,
                                    cnt + 62, reinterpret_cast<unsigned long long*>(rtask_off)};
                const uint64_t most = static_cast<uint64_t>(ctx->sm_count) *
                                      (cta ? 1 : std::min(ctx->tune.max_blocks_per_sm, 2));
                const uint64_t ctas = cta ? nt : (nt + kWarpTileThreads / 32 - 1) / (kWarpTileThreads / 32);
                P.tasks.range = per_task ? ((i & 1) ? range1 : range0) : cnt + 44 + 2 * i;
                P.queue_head = cnt + 56 + i;
                const int tile_grid = static_cast<int>(std::min(ctas, most));
                KernelScope ks(ctx, tile_names[affine][i]);
                if (affine)
                    (cta ? launch_wfa_affine_cta_tiles : launch_wfa_affine_warp_tiles)(P, tl, tile_grid, i & 1, st);
                else
                    (cta ? launch_wfa_linear_big : launch_wfa_linear_tile)(P, tl, tile_grid, i & 1, st);
            }
        }
        // (no linear pair is beyond the tiles in a batch of fewer symbols than their limit)
        const bool aff = engine == PHR_ENGINE_WFA_AFFINE;
        if (per_task && (aff || (engine == PHR_ENGINE_WFA_LINEAR && sum_qt >= static_cast<uint64_t>(kTileMaxQuery))) &&
            P.big_min > 0 && n_tasks_hint > 0) {
            // long pairs the register tiles do not take, one CTA each. Gap-affine:
            // kBigAffineThreads / wfa_affine_big_threads CTAs per SM; linear: two (one when the
            // tune keeps fewer blocks resident)
            const int aff_threads = ctx->tune.wfa_affine_big_threads;
            const uint64_t per_sm = aff ? kBigAffineThreads / aff_threads : ctx->tune.max_blocks_per_sm >= 4 ? 2 : 1;
            const int big_grid = static_cast<int>(std::min<uint64_t>(n_tasks_hint, ctx->sm_count * per_sm));
            PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 24, 0, 8, st));
            for (int mode = 0; mode < 2; ++mode) {
                if (!(mode ? any_bytes : any_2bit)) continue;
                P.tasks.range = mode ? range1 : range0;
                P.queue_head = cnt + 24 + mode;
                if (aff) {
                    KernelScope ks(ctx, mode ? "wfa_affine_big_bytes" : "wfa_affine_big");
                    launch_wfa_affine_big(P, big_grid, aff_threads, mode, st);
                } else {
                    KernelScope ks(ctx, mode ? "wfa_linear_long_bytes" : "wfa_linear_long");
                    launch_wfa_linear_long(P, big_grid, mode, st);
                }
            }
        }
        PHR_CUDA_TRY(ctx, cudaGetLastError());
        return PHR_OK;
    };

    phr_status s = launch_pass(order, task_first, task_count, task_group, cnt + 0, cnt + 2, h_need, 0);
    if (s != PHR_OK) return s;
    if (n_tile[2] + n_tile[3] > 0) {
        // long pairs left by the CTA kernels when most SMs had run out of pairs: a cluster each
        PHR_CUDA_TRY(ctx, read_counters(256));
        const uint32_t h_defer = h_cnt[62];
        if (h_defer > 0) {
            const TileLaunch tl{reinterpret_cast<unsigned long long*>(cnt + 60), tile_pool, kTileChunk, 0, ctx->sm_count, cnt + 62,
                                reinterpret_cast<unsigned long long*>(rtask_off)};
            const int ctas = wfa_cluster_size(h_defer, ctx->sm_count, cluster_max);
            for (int mode = 0; mode < 2; ++mode) {
                if (n_tile[2 + mode] == 0) continue;
                PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 63, 0, 4, st));
                P.queue_head = cnt + 63;
                const bool affine = engine == PHR_ENGINE_WFA_AFFINE;
                KernelScope ks(ctx, affine ? "wfa_affine_resume" : "wfa_linear_resume");
                (affine ? launch_wfa_affine_resume : launch_wfa_linear_resume)(P, tl, static_cast<int>(h_defer), ctas, mode, st);
            }
            PHR_CUDA_TRY(ctx, cudaGetLastError());
        }
    }

    // Redo passes: each pair that did not fit its slot (or, for Myers, whose edit distance
    // left the stored band) runs again alone, with scratch sized for it: pairs are packed
    // into passes of at most the workspace budget, one variable-size region per task.
    uint32_t* rlist = redo_list;
    uint32_t* rlist2 = head;  // reuse: free after task build
    P.task_need = nullptr;
    std::vector<uint32_t> h_list;
    std::vector<unsigned long long> h_rneed;
    std::unordered_set<uint32_t> clamped;
    // a pair that still overflows the whole budget ends with status PHR_ERR_OOM (the
    // other pairs of the call go on)
    static const PairOut kOomOut = {PHR_ERR_OOM, 0, 0, 0, 0, 0};
    uint64_t n_oom = 0;
    // Text offsets, their total, the records and texts; nothing is written while pairs wait for
    // a redo pass or when the text does not fit.
    FinishParams F{n, engine, desc, pout, tbo, text, cigoff, res->aln, res->cigar, res->cigar_capacity, cnt + 10,
                   res->cigar_base, 32, cnt + 7, total};
    auto launch_tail = [&]() {
        const bool texts = small && sum_qt <= (64u << 10);   // little enough for one CTA to copy
        if (small) {
            FinishParams f = F;
            f.per_warp = static_cast<int>((n + 31) / 32);
            KernelScope ks(ctx, "small_tail");
            small_tail_kernel<<<1, kSmallPairs, 0, st>>>(f, tlen, texts);
        } else {
            {
                KernelScope ks(ctx, "text_len");
                text_len_kernel<<<blocks_for(n, T), T, 0, st>>>(pout, n, tlen);
            }
            tn_ = t_need;
            cub::DeviceScan::ExclusiveSum(tmp, tn_, tlen, cigoff, static_cast<int>(n), st);
            KernelScope ks(ctx, "total");
            total_kernel<<<1, 1, 0, st>>>(cigoff, tlen, n, total);
        }
        if (texts) return;
        FinishParams f = F;
        // at least 16 warps per SM before a warp takes more than one pair
        while (f.per_warp > 1 && (n + f.per_warp - 1) / f.per_warp < 16ull * ctx->sm_count) f.per_warp /= 2;
        KernelScope ks(ctx, "finish");
        finish_kernel<<<blocks_for((n + f.per_warp - 1) / f.per_warp * 32, T), T, 0, st>>>(f);
    };
    // a batch this small is finished before the host knows whether pairs are to be redone: one
    // wait less when there are none, a few microseconds of work in vain otherwise
    const bool ahead = n <= (1u << 16);
    bool tail_done = false;
    HostScope hs_redo(ctx, "host:redo");
    for (int round = 0; round < 12; ++round) {
        if (ahead) launch_tail();
        PHR_CUDA_TRY(ctx, read_counters(256));
        const uint32_t h_redo = h_cnt[7];
        tail_done = ahead && h_redo == 0;
        if (h_redo == 0) break;
        if (round == 11) return set_error(ctx, PHR_ERR_CAPACITY, "extension did not fit after repeated redo passes");
        h_list.resize(h_redo);
        h_rneed.resize(h_redo);
        PHR_CUDA_TRY(ctx, cudaMemcpyAsync(h_list.data(), rlist, h_redo * 4, cudaMemcpyDeviceToHost, st));
        PHR_CUDA_TRY(ctx, cudaMemcpyAsync(h_rneed.data(), redo_need, h_redo * 8, cudaMemcpyDeviceToHost, st));
        PHR_CUDA_TRY(ctx, cudaStreamSynchronize(st));
        PHR_CUDA_TRY(ctx, cudaMemsetAsync(cnt + 7, 0, 4, st));
        // largest first, packed into passes within the budget
        std::vector<uint32_t> idx(h_redo);
        for (uint32_t i = 0; i < h_redo; ++i) idx[i] = i;
        std::sort(idx.begin(), idx.end(), [&](uint32_t a, uint32_t b) { return h_rneed[a] > h_rneed[b]; });
        if (const char* tp = std::getenv("PHRAYA_EXTEND_TRACE")) {
            // one line per redo round: engine round pairs budget, then the eight largest
            // needs as qn:tn:need_bytes
            if (FILE* f = std::fopen(tp, "a")) {
                std::fprintf(f, "engine %d round %d pairs %u budget %llu", static_cast<int>(engine), round, h_redo,
                             static_cast<unsigned long long>(ctx->scratch_budget));
                for (uint32_t i = 0; i < std::min<uint32_t>(h_redo, 8); ++i) {
                    PairDesc hd{};
                    PHR_CUDA_TRY(ctx, cudaMemcpy(&hd, desc + h_list[idx[i]], sizeof(PairDesc), cudaMemcpyDeviceToHost));
                    std::fprintf(f, " %d:%d:%llu", hd.qn, hd.tn, h_rneed[idx[i]]);
                }
                std::fprintf(f, "\n");
                std::fclose(f);
            }
        }
        size_t pos = 0;
        while (pos < idx.size()) {
            std::vector<uint32_t> pl;
            std::vector<uint64_t> po, pn;
            uint64_t tot = 0;
            while (pos < idx.size()) {
                uint64_t need = (std::max<uint64_t>(h_rneed[idx[pos]], 4096) + 255) & ~255ull;
                bool clamp = false;
                if (need > ctx->scratch_budget) {
                    // first-pass needs are estimates: try once with the whole budget
                    if (clamped.count(h_list[idx[pos]])) {
                        PHR_CUDA_TRY(ctx, cudaMemcpyAsync(pout + h_list[idx[pos]], &kOomOut, sizeof(PairOut),
                                                          cudaMemcpyHostToDevice, st));
                        ++n_oom;
                        ++pos;
                        continue;
                    }
                    clamp = true;
                    need = ctx->scratch_budget & ~255ull;
                }
                if (!pl.empty() && tot + need > pass_budget) break;  // this pair opens the next pass
                // the whole-budget try is spent only once the pair is placed in a pass
                if (clamp) clamped.insert(h_list[idx[pos]]);
                pl.push_back(h_list[idx[pos]]);
                po.push_back(tot);
                pn.push_back(need);
                tot += need;
                ++pos;
            }
            const uint32_t m = static_cast<uint32_t>(pl.size());
            if (m == 0) continue;
            PHR_CUDA_TRY(ctx, cudaMemcpyAsync(rlist2, pl.data(), m * 4, cudaMemcpyHostToDevice, st));
            PHR_CUDA_TRY(ctx, cudaMemcpyAsync(rtask_off, po.data(), m * 8, cudaMemcpyHostToDevice, st));
            PHR_CUDA_TRY(ctx, cudaMemcpyAsync(rtask_len, pn.data(), m * 8, cudaMemcpyHostToDevice, st));
            PHR_CUDA_TRY(ctx, cudaMemcpyAsync(cnt + 18, &m, 4, cudaMemcpyHostToDevice, st));
            {
                KernelScope ks(ctx, "redo_tasks");
                redo_tasks_kernel<<<blocks_for(m, T), T, 0, st>>>(rlist2, cnt + 18, desc, engine,
                                                                 aff_tile_open(costs), g_short, ctx->tune.wfa_group_long,
                                                                 ctx->tune.wfa_long_min,
                                                                 P.big_min, task_first, task_count, task_group,
                                                                 cnt + 14);
            }
            // byte-mode and 2-bit pairs share this list: both launches walk all of it
            PHR_CUDA_TRY(ctx, cudaMemcpyAsync(cnt + 16, cnt + 14, 8, cudaMemcpyDeviceToDevice, st));
            P.redo_list = rlist;   // fresh overflows of this pass are appended here
            P.task_off = rtask_off;
            P.task_len = rtask_len;
            // synchronise before the scratch buffer may be reallocated for this pass
            PHR_CUDA_TRY(ctx, cudaStreamSynchronize(st));
            s = launch_pass(rlist2, task_first, task_count, task_group, cnt + 14, cnt + 16, 0, 1, true, tot, m);
            P.task_off = nullptr;
            P.task_len = nullptr;
            if (s != PHR_OK) return s;
            PHR_CUDA_TRY(ctx, cudaStreamSynchronize(st));
        }
    }

    hs_redo.stop();
    if (n_oom) ctx->counters["scratch_oom_pairs"] += n_oom;
    if (const char* tp = std::getenv("PHRAYA_EXTEND_TRACE")) {
        // one line per pair of qlen + tlen >= 65536: its final status and distance
        std::vector<PairDesc> hd(n);
        std::vector<PairOut> ho(n);
        PHR_CUDA_TRY(ctx, cudaMemcpyAsync(hd.data(), desc, n * sizeof(PairDesc), cudaMemcpyDeviceToHost, st));
        PHR_CUDA_TRY(ctx, cudaMemcpyAsync(ho.data(), pout, n * sizeof(PairOut), cudaMemcpyDeviceToHost, st));
        PHR_CUDA_TRY(ctx, cudaStreamSynchronize(st));
        if (FILE* f = std::fopen(tp, "a")) {
            for (uint64_t i = 0; i < n; ++i)
                if (static_cast<int64_t>(hd[i].qn) + hd[i].tn >= 65536)
                    std::fprintf(f, "engine %d pair %llu %d:%d seed %d:%d status %d ed %d\n", static_cast<int>(engine),
                                 static_cast<unsigned long long>(i), hd[i].qn, hd[i].tn, hd[i].qs, hd[i].ts,
                                 ho[i].status, ho[i].ed);
            std::fclose(f);
        }
    }
    HostScope hs_tail(ctx, "host:extend_tail");
    if (!tail_done) {
        launch_tail();
        PHR_CUDA_TRY(ctx, read_counters(256));
    }
    uint64_t h_total = 0;
    std::memcpy(&h_total, h_cnt + 12, 8);
    if (h_total > res->cigar_capacity)
        return set_error(ctx, PHR_ERR_CAPACITY, "CIGAR arena too small: need " + std::to_string(h_total) + " bytes");
    const uint32_t h_err = h_cnt[10];
    unsigned long long h_work[4];
    std::memcpy(h_work, h_cnt + 32, sizeof(h_work));
    if (h_work[0]) ctx->counters["myers_lane_block_columns"] += h_work[0];
    if (h_work[1]) ctx->counters["myers_lane_redo_pairs"] += h_work[1];
    if (h_work[2] || h_work[3]) {
        const std::string e = engine == PHR_ENGINE_WFA_AFFINE ? "wfa_affine" : "wfa_linear";
        ctx->counters[e + "_cells"] += h_work[2];
        ctx->counters[e + "_lcp_words"] += h_work[3];
    }
    PHR_CUDA_TRY(ctx, cudaGetLastError());
    if (ctx->timing) ctx->resolve_timings();
    if (h_err) return set_error(ctx, PHR_ERR_CUDA, "internal consistency check failed (flags " + std::to_string(h_err) + ")");
    res->cigar_used = h_total;
    return PHR_OK;
}

}  // namespace phr
