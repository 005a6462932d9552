// Prefill attention: any number of queries per sequence, causal (right-aligned to the cache end) or full. The canonical
// arithmetic is that of decode (top of attention.cu): a query's scores, softmax scalars, accumulators and split merge
// are the same operations on the same operands in the same order, only laid out over threads for many queries at once.
//
// What bounds it: the fp32 pipe. The key-by-key order keeps the tensor cores out: a (query, key) pair costs 128 fma + 31
// add for the score, 128 mul + 128 fma for the accumulation (head_dim 128) and about 25 for the exponential, 440 fp32
// operations, and an SM retires 128 a clock: 0.82 ms for 32 heads x 2048 causal tokens. Next to it stand shared-memory
// reads: a 16-byte load costs the SM 2 clocks when neighbouring lanes share addresses and 4 when they do not.
//
// Work split: a CTA of 128 threads takes QB = TQ * 1024 / D query rows that share one kv head (row = (query head in the
// group, query), so that short chunks fill a CTA across the heads of the group) and walks the keys in blocks of KB inside
// the fixed splits. Per block:
//   A  scores: a thread owns TQ rows x 2 keys and evaluates their whole dot products, virtual lanes 2I and 2I+1 riding in
//      one f32x2 and the xor tree evaluated depth first (ten registers a score); every K element it converts serves TQ
//      rows, every query element two keys;
//   B  softmax scalars: a warp takes QB / 4 rows, lane = key: prefix maximum (skipped when no score of the block exceeds
//      its row's running maximum), one exponential per score, factors to shared memory;
//   C  accumulation: a thread owns TQ rows x 8 dims and walks the block's keys in order.
// K is refilled (cp.async) once the scores exist, V is double buffered. Up to three CTAs share an SM, so that one computes
// while another waits at a barrier.
//
// Measured (bf16, D = 128, 32 query / 8 kv heads, causal): 2048 tokens 1231 us (the 0.82 ms of fp32 operations are two
// thirds of it), before 4442 us with eight lanes per key stream; 2 x 512 tokens 175 us, before 740 us.
#include "attn_common.cuh"

namespace bi {
namespace {

constexpr int PF_THREADS = 128;
constexpr int PF_SMEM_MAX = 227 * 1024;                           // what a CTA may have

template <typename T, int DL, int TQ> struct PF {
    static constexpr int D = 32 * DL;
    static constexpr int QB = TQ * PF_THREADS * 8 / D;            // query rows per CTA
    static constexpr int RG = QB / 4 < 4 ? QB / 4 : 4;            // rows whose softmax scalars a warp evaluates together
    static constexpr int KB = DL == 8 ? 64 : 32;                  // keys per block
    static constexpr int KROW = D * (int)sizeof(T);
    static constexpr int KPITCH = KROW + 16;                      // 16 keys read at one column land on distinct banks
    static constexpr int QPITCH = D * 4 + 16;
    static constexpr int SPITCH = KB + 4;                         // floats
    static constexpr int PPITCH = QB + RG;                        // floats; a vector of RG floats per key, no two keys of a store phase on one bank
    static constexpr int KOFF = QB * QPITCH;
    static constexpr int VOFF = KOFF + KB * KPITCH;
    static constexpr int SOFF = VOFF + 2 * KB * KROW;
    static constexpr int POFF = SOFF + QB * SPITCH * 4;
    static constexpr int COFF = POFF + KB * PPITCH * 4;
    static constexpr int MOFF = COFF + KB * PPITCH * 4;           // running maximum of the split, per row
    static constexpr int NOFF = MOFF + QB * 4;                    // keys a row sees
    static constexpr int TOFF = (NOFF + QB * 4 + 15) / 16 * 16;   // merged accumulators, touched once per split
    static constexpr int SMEM = TOFF + PF_THREADS * TQ * 8 * 4;
};

// The 2 * DL dims of virtual lanes 2I and 2I+1 of a K row in shared memory as pairs (x[2I][d], x[2I+1][d]).
template <typename T, int DL>
__device__ __forceinline__ void key_pairs(const uint8_t* row, int I, uint64_t (&k2)[DL]) {
    if constexpr (sizeof(T) == 4) {
        const float* f = reinterpret_cast<const float*>(row) + I * 2 * DL;
        float x[2 * DL];
#pragma unroll
        for (int i = 0; i < 2 * DL; i += (DL == 1 ? 2 : 4)) {
            if constexpr (DL == 1) {
                const float2 w = *reinterpret_cast<const float2*>(f);
                x[0] = w.x; x[1] = w.y;
            } else {
                const float4 w = *reinterpret_cast<const float4*>(f + i);
                x[i] = w.x; x[i + 1] = w.y; x[i + 2] = w.z; x[i + 3] = w.w;
            }
        }
#pragma unroll
        for (int d = 0; d < DL; ++d) k2[d] = ptx::pack2(x[d], x[DL + d]);
    } else {
        uint32_t w[DL];                                            // word i: dims 2i, 2i+1 of the two lanes' run
        const uint8_t* p = row + I * 4 * DL;
        if constexpr (DL == 1) w[0] = *reinterpret_cast<const uint32_t*>(p);
        else if constexpr (DL == 2) { const uint2 v = *reinterpret_cast<const uint2*>(p); w[0] = v.x; w[1] = v.y; }
        else {
#pragma unroll
            for (int i = 0; i < DL; i += 4) {
                const uint4 v = *reinterpret_cast<const uint4*>(p + i * 4);
                w[i] = v.x; w[(i + 1) % DL] = v.y; w[(i + 2) % DL] = v.z; w[(i + 3) % DL] = v.w;
            }
        }
        if constexpr (DL == 1) k2[0] = ptx::pack2(word_lo<T>(w[0]), word_hi<T>(w[0]));
        else {
#pragma unroll
            for (int d = 0; d < DL; ++d) {
                const uint32_t a = w[d / 2], b = w[(DL + d) / 2];
                k2[d] = (d & 1) ? ptx::pack2(word_hi<T>(a), word_hi<T>(b)) : ptx::pack2(word_lo<T>(a), word_lo<T>(b));
            }
        }
    }
}

// Packed partial sums (part_{2I}, part_{2I+1}) of TQ rows against two keys.
template <typename T, int DL, int TQ, int I>
__device__ __forceinline__ void score_leaf(const uint8_t* ka, const uint8_t* kb, const uint8_t* qr, uint64_t (&out)[TQ][2]) {
    uint64_t k2[2][DL];
    key_pairs<T, DL>(ka, I, k2[0]);
    key_pairs<T, DL>(kb, I, k2[1]);
#pragma unroll
    for (int iq = 0; iq < TQ; ++iq) {
        const uint8_t* qp = qr + iq * PF<T, DL, TQ>::QPITCH + I * 8 * DL;
        uint64_t q2[DL];
        if constexpr (DL == 1) q2[0] = *reinterpret_cast<const uint64_t*>(qp);
        else {
#pragma unroll
            for (int d = 0; d < DL; d += 2) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(qp + d * 8);
                q2[d] = w.x; q2[(d + 1) % DL] = w.y;
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint64_t p = ptx::fma2_rn(q2[0], k2[j][0], ptx::pack2(0.0f, 0.0f));
#pragma unroll
            for (int d = 1; d < DL; ++d) p = ptx::fma2_rn(q2[d], k2[j][d], p);
            out[iq][j] = p;
        }
    }
}
// The xor tree over the sixteen pairs: stride 8 is tree level 16, then 8, 4, 2 (level 1 is the sum inside the pair).
template <typename T, int DL, int TQ, int STRIDE, int I>
__device__ __forceinline__ void score_node(const uint8_t* ka, const uint8_t* kb, const uint8_t* qr, uint64_t (&out)[TQ][2]) {
    uint64_t b[TQ][2];
    if constexpr (STRIDE == 8) {
        score_leaf<T, DL, TQ, I>(ka, kb, qr, out);
        score_leaf<T, DL, TQ, I + 8>(ka, kb, qr, b);
    } else {
        score_node<T, DL, TQ, STRIDE * 2, I>(ka, kb, qr, out);
        score_node<T, DL, TQ, STRIDE * 2, I + STRIDE>(ka, kb, qr, b);
    }
#pragma unroll
    for (int iq = 0; iq < TQ; ++iq)
#pragma unroll
        for (int j = 0; j < 2; ++j) out[iq][j] = ptx::add2_rn(out[iq][j], b[iq][j]);
}

// N consecutive floats (N = 1, 2 or 4) of shared memory, aligned to their size.
template <int N> __device__ __forceinline__ void ld_vec(const float* p, float (&v)[N]) {
    if constexpr (N == 4) { const float4 w = *reinterpret_cast<const float4*>(p); v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w; }
    else if constexpr (N == 2) { const float2 w = *reinterpret_cast<const float2*>(p); v[0] = w.x; v[1] = w.y; }
    else v[0] = *p;
}
template <int N> __device__ __forceinline__ void st_vec(float* p, const float (&v)[N]) {
    if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    else if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else *p = v[0];
}

// Eight consecutive dims of a V row as four pairs of consecutive dims.
template <typename T>
__device__ __forceinline__ void value_pairs(const uint8_t* p, uint64_t (&v2)[4]) {
    if constexpr (sizeof(T) == 4) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p), b = *reinterpret_cast<const ulonglong2*>(p + 16);
        v2[0] = a.x; v2[1] = a.y; v2[2] = b.x; v2[3] = b.y;
    } else {
        const uint4 w = *reinterpret_cast<const uint4*>(p);
        v2[0] = ptx::pack2(word_lo<T>(w.x), word_hi<T>(w.x));
        v2[1] = ptx::pack2(word_lo<T>(w.y), word_hi<T>(w.y));
        v2[2] = ptx::pack2(word_lo<T>(w.z), word_hi<T>(w.z));
        v2[3] = ptx::pack2(word_lo<T>(w.w), word_hi<T>(w.w));
    }
}

// Row block of a CTA. Blocks that see the most keys (the last queries, when causal) are dealt first.
struct RowBlock {
    long long R, r0;                                               // rows per (batch, kv head); the block's first
    int bh, rows;
    __device__ __forceinline__ RowBlock(int B, int Hkv, int G, int Tq, int QB) {
        R = (long long)G * Tq;
        const int nb = (int)((R + QB - 1) / QB);
        const int t = (int)(blockIdx.x / (unsigned)(B * Hkv));
        bh = (int)(blockIdx.x % (unsigned)(B * Hkv));
        const int rb = nb % G == 0 ? (t % G) * (nb / G) + (nb / G - 1 - t / G) : nb - 1 - t;
        r0 = (long long)rb * QB;
        rows = (int)min((long long)QB, R - r0);
    }
};

// One row by one warp, key by key over the n keys it sees, as the canonical arithmetic is written: lane = virtual lane, with
// its DL dims of q, k, v and the accumulator. For rows the tiled phases cannot keep apart (below).
template <typename T, int DL>
__device__ __forceinline__ void literal_row(const T* q, const T* k, const T* v, T* out, int n, int64_t sl, float scale, int split) {
    const int d0 = (threadIdx.x & 31) * DL;
    float qf[DL], A[DL], M = -INFINITY, L = 0.0f;
#pragma unroll
    for (int d = 0; d < DL; ++d) { qf[d] = mul_rn(Cvt<T>::up(q[d0 + d]), scale); A[d] = 0.0f; }
    for (int j0 = 0; j0 < n; j0 += split) {
        float m = -INFINITY, l = 0.0f, acc[DL];
#pragma unroll
        for (int d = 0; d < DL; ++d) acc[d] = 0.0f;
        const int j1 = min(n, j0 + split);
        for (int j = j0; j < j1; ++j) {
            const T *kr = k + (int64_t)j * sl + d0, *vr = v + (int64_t)j * sl + d0;
            float s = 0.0f;
#pragma unroll
            for (int d = 0; d < DL; ++d) s = fma_rn(qf[d], Cvt<T>::up(kr[d]), s);
#pragma unroll
            for (int off = 16; off; off >>= 1) s = add_rn(s, __shfl_xor_sync(0xffffffffu, s, off));
            const float e = expf_canon(-fabsf(sub_rn(s, m)));
            const bool rises = s >= m;
            const float c = rises ? e : 1.0f, p = rises ? 1.0f : e;
            m = fmaxf(m, s);
            l = fma_rn(l, c, p);
#pragma unroll
            for (int d = 0; d < DL; ++d) acc[d] = fma_rn(acc[d], c, mul_rn(p, Cvt<T>::up(vr[d])));
        }
        float c_old, c_new;
        merge_coeffs(M, L, m, l, c_old, c_new);
#pragma unroll
        for (int d = 0; d < DL; ++d) A[d] = merge_acc(A[d], c_old, acc[d], c_new);
    }
#pragma unroll
    for (int d = 0; d < DL; ++d) out[d0 + d] = Cvt<T>::down(div_canon(A[d], L));
}

// The rows of this CTA that hold NaN in `ms`, by literal_row. Everything is worked out again from the launch's arguments, so
// that the kernel keeps no register for it through its loops.
template <typename T, int DL, int TQ>
__device__ __noinline__ void literal_rows(const float* ms, const T* q, const T* k, const T* v, T* out, int B, int Hkv, int G, int Tq, int L,
                                          int64_t sb, int64_t sh, int64_t sl, float scale, int split) {
    constexpr int D = 32 * DL, QB = PF<T, DL, TQ>::QB;
    const RowBlock w(B, Hkv, G, Tq, QB);
    for (int row = threadIdx.x >> 5; row < w.rows; row += PF_THREADS / 32) {
        if (ms[row] == ms[row]) continue;
        const int64_t at = ((int64_t)w.bh * w.R + w.r0 + row) * D, kv = (int64_t)(w.bh / Hkv) * sb + (int64_t)(w.bh % Hkv) * sh;
        literal_row<T, DL>(q + at, k + kv, v + kv, out + at, L - Tq + (int)((w.r0 + row) % Tq) + 1, sl, scale, split);
    }
}

template <typename T, int DL, int TQ>
__global__ void __launch_bounds__(PF_THREADS, TQ == 4 && (DL == 2 || DL == 4) && sizeof(T) == 2 ? 3 : 2) prefill_kernel(
    const T* __restrict__ q, const T* __restrict__ k, const T* __restrict__ v, T* __restrict__ out, int B, int Hkv, int G, int Tq,
    int L, KvLayout lay, float scale, int causal, int split, int rows16) {
    using C = PF<T, DL, TQ>;
    constexpr int D = C::D, QB = C::QB, KB = C::KB, RG = C::RG;
    extern __shared__ __align__(16) uint8_t sm[];
    uint8_t* const qs = sm;
    uint8_t* const ks = sm + C::KOFF;
    uint8_t* const vs = sm + C::VOFF;
    float* const ss = reinterpret_cast<float*>(sm + C::SOFF);
    float* const ps = reinterpret_cast<float*>(sm + C::POFF);
    float* const cs = reinterpret_cast<float*>(sm + C::COFF);
    float* const ms = reinterpret_cast<float*>(sm + C::MOFF);
    int* const ns = reinterpret_cast<int*>(sm + C::NOFF);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    ptx::grid_dep_wait();     // everything before this kernel has completed and is visible

    const RowBlock block(B, Hkv, G, Tq, QB);
    const long long R = block.R, r0 = block.r0;
    const int bh = block.bh, rows = block.rows, b = bh / Hkv, hk = bh % Hkv;
    const T* const kbase = k + (int64_t)b * lay.sb + (int64_t)hk * lay.sh;
    const T* const vbase = v + (int64_t)b * lay.sb + (int64_t)hk * lay.sh;
    const T* const qbase = q + ((int64_t)bh * R + r0) * D;         // rows of a (batch, kv head) are contiguous in q and out

    for (int i = tid; i < QB; i += PF_THREADS)
        ns[i] = i < rows ? (causal ? L - Tq + (int)((r0 + i) % Tq) + 1 : L) : 0;
    for (int i = tid; i < QB * D; i += PF_THREADS) {               // pre-scaled queries, in the order score_leaf reads them
        const int row = i / D, d = i % D;
        const int lanep = d / (2 * DL), w = d % (2 * DL);          // pair I, place in its run
        const float x = row < rows ? mul_rn(Cvt<T>::up(qbase[i]), scale) : 0.0f;
        *reinterpret_cast<float*>(qs + row * C::QPITCH + (lanep * 2 * DL + (w % DL) * 2 + w / DL) * 4) = x;
    }
    __syncthreads();
    int nmax = 0;
    for (int i = lane; i < QB; i += 32) nmax = max(nmax, ns[i]);
    nmax = __reduce_max_sync(0xffffffffu, nmax);

    // Rows [key0, key0 + cnt) of K or V to shared memory; rows past the end re-read the last one.
    auto fetch = [&](uint8_t* dst, int pitch, const T* base, int key0, int cnt) {
        if (rows16) {
            constexpr int SEGS = C::KROW / 16;
            const uint32_t d0 = ptx::smem_u32(dst);
#pragma unroll
            for (int i = tid; i < KB * SEGS; i += PF_THREADS) {
                const int row = i / SEGS, seg = i % SEGS;
                const uint8_t* g = reinterpret_cast<const uint8_t*>(base + (int64_t)(key0 + min(row, cnt - 1)) * lay.sl) + seg * 16;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d0 + row * pitch + seg * 16), "l"(g) : "memory");
            }
        } else {
            for (int i = tid; i < KB * D; i += PF_THREADS) {
                const int row = i / D, d = i % D;
                *reinterpret_cast<T*>(dst + row * pitch + d * (int)sizeof(T)) = base[(int64_t)(key0 + min(row, cnt - 1)) * lay.sl + d];
            }
        }
    };

    // accumulation tile of this thread: rows tq .. tq+3, dims td .. td+7
    constexpr int DG = D / 8;
    const int tq = (tid / DG) * TQ, td = (tid % DG) * 8;
    uint64_t acc[TQ][4];
    // merged accumulators of the thread: pairs (2i, 2i+1) of its TQ x 4 at tot[i * PF_THREADS]
    ulonglong2* const tot = reinterpret_cast<ulonglong2*>(sm + C::TOFF) + tid;
    float l[TQ], Mt[TQ], Lt[TQ];
#pragma unroll
    for (int i = 0; i < TQ; ++i) {
        l[i] = 0.0f; Mt[i] = -INFINITY; Lt[i] = 0.0f;
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
#pragma unroll
        for (int j = 0; j < 2; ++j) tot[(i * 2 + j) * PF_THREADS] = make_ulonglong2(0, 0);
    }

    fetch(ks, C::KPITCH, kbase, 0, min(KB, min(split, nmax)));
    fetch(vs, C::KROW, vbase, 0, min(KB, min(split, nmax)));
    asm volatile("cp.async.commit_group;" ::: "memory");
    int buf = 0;
    for (int j0 = 0; j0 < nmax; j0 += split) {
        const int j1 = min(nmax, j0 + split);
        for (int j = j0; j < j1; j += KB) {
            const int cnt = min(KB, j1 - j);
            if (j == j0 && tid < QB) ms[tid] = -INFINITY;
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            // ---- A: scores
#pragma unroll 1
            for (int tile = tid; tile < QB * KB / (2 * TQ); tile += PF_THREADS) {
                const int kg = tile % (KB / 2), qg = tile / (KB / 2);
                uint64_t o[TQ][2];
                score_node<T, DL, TQ, 1, 0>(ks + kg * C::KPITCH, ks + (kg + KB / 2) * C::KPITCH, qs + qg * TQ * C::QPITCH, o);
#pragma unroll
                for (int iq = 0; iq < TQ; ++iq)
#pragma unroll
                    for (int jj = 0; jj < 2; ++jj) {
                        float d0, d1;
                        ptx::unpack2(o[iq][jj], d0, d1);
                        ss[(qg * TQ + iq) * C::SPITCH + kg + jj * (KB / 2)] = add_rn(d0, d1);
                    }
            }
            __syncthreads();
            {   // the block after this one
                const bool same = j + KB < j1;
                const int jn = same ? j + KB : j1, je = same ? j1 : min(nmax, j1 + split);
                if (jn < nmax) {
                    fetch(ks, C::KPITCH, kbase, jn, min(KB, je - jn));
                    fetch(vs + (buf ^ 1) * KB * C::KROW, C::KROW, vbase, jn, min(KB, je - jn));
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
            // ---- B: softmax scalars, RG rows at a time (independent chains; their factors leave in one store per key)
            for (int rr = warp * (QB / 4); rr < (warp + 1) * (QB / 4); rr += RG) {
#pragma unroll
                for (int half = 0; half < KB / 32; ++half) {
                    const int key = half * 32 + lane;
                    float p4[RG], c4[RG], s4[RG], m4[RG];
                    bool on4[RG], rise = false;
                    ld_vec<RG>(ms + rr, m4);
#pragma unroll
                    for (int u = 0; u < RG; ++u) {
                        s4[u] = ss[(rr + u) * C::SPITCH + key];
                        on4[u] = key < cnt && j + key < ns[rr + u];
                        rise |= on4[u] && s4[u] > m4[u];
                    }
                    if (__any_sync(0xffffffffu, rise)) {                 // inclusive prefix maxima over the lanes
                        float x[RG], y[RG];
#pragma unroll
                        for (int u = 0; u < RG; ++u) x[u] = on4[u] ? s4[u] : -INFINITY;
#pragma unroll
                        for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
                            for (int u = 0; u < RG; ++u) y[u] = __shfl_up_sync(0xffffffffu, x[u], off);
#pragma unroll
                            for (int u = 0; u < RG; ++u) if (lane >= off) x[u] = fmaxf(x[u], y[u]);
                        }
#pragma unroll
                        for (int u = 0; u < RG; ++u) y[u] = fmaxf(m4[u], x[u]);
                        if (lane == 31) st_vec<RG>(ms + rr, y);
#pragma unroll
                        for (int u = 0; u < RG; ++u) {                   // running maximum before this key
                            const float up = __shfl_up_sync(0xffffffffu, x[u], 1);
                            if (lane > 0) m4[u] = fmaxf(m4[u], up);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < RG; ++u) {
                        const float e = expf_canon(-fabsf(sub_rn(s4[u], m4[u])));
                        const bool rises = s4[u] >= m4[u];
                        c4[u] = on4[u] && rises ? e : 1.0f;
                        p4[u] = on4[u] ? (rises ? 1.0f : e) : 0.0f;
                    }
                    st_vec<RG>(ps + key * C::PPITCH + rr, p4);
                    st_vec<RG>(cs + key * C::PPITCH + rr, c4);
                    if (KB > 32) __syncwarp();                           // the running maximum, before the next half reads it
                }
            }
            __syncthreads();
            // ---- C: accumulation, key by key
            const uint8_t* const vb = vs + buf * KB * C::KROW + td * (int)sizeof(T);
#pragma unroll 8
            for (int i = 0; i < cnt; ++i) {
                float p[TQ], c[TQ];
                ld_vec<TQ>(ps + i * C::PPITCH + tq, p);
                ld_vec<TQ>(cs + i * C::PPITCH + tq, c);
                uint64_t v2[4], t2[4];
                value_pairs<T>(vb + i * C::KROW, v2);
#pragma unroll
                for (int iq = 0; iq < TQ; ++iq) {
                    const uint64_t p2 = ptx::pack2(p[iq], p[iq]), c2 = ptx::pack2(c[iq], c[iq]);
                    l[iq] = fma_rn(l[iq], c[iq], p[iq]);
#pragma unroll
                    for (int d = 0; d < 4; ++d) t2[d] = ptx::mul2_rn(p2, v2[d]);
#pragma unroll
                    for (int d = 0; d < 4; ++d) acc[iq][d] = ptx::fma2_rn(acc[iq][d], c2, t2[d]);
                }
            }
            buf ^= 1;
        }
        // ---- the split's end: fold it into the running state of every row that saw a key of it
#pragma unroll
        for (int iq = 0; iq < TQ; ++iq) {
            if (j0 < ns[tq + iq]) {
                float c_old, c_new;
                merge_coeffs(Mt[iq], Lt[iq], ms[tq + iq], l[iq], c_old, c_new);
                const uint64_t o2 = ptx::pack2(c_old, c_old), n2 = ptx::pack2(c_new, c_new);
#pragma unroll
                for (int d = 0; d < 2; ++d) {
                    ulonglong2 x = tot[(iq * 2 + d) * PF_THREADS];
                    x.x = ptx::fma2_rn(x.x, o2, ptx::mul2_rn(acc[iq][2 * d], n2));
                    x.y = ptx::fma2_rn(x.y, o2, ptx::mul2_rn(acc[iq][2 * d + 1], n2));
                    tot[(iq * 2 + d) * PF_THREADS] = x;
                }
            }
#pragma unroll
            for (int d = 0; d < 4; ++d) acc[iq][d] = 0;
            l[iq] = 0.0f;
        }
        __syncthreads();                                                 // ms is read above, reset by the next split
    }

    bool poisoned = false;
#pragma unroll
    for (int iq = 0; iq < TQ; ++iq) {
        if (tq + iq >= rows) continue;
        bool nan = false;
        T* o = out + ((int64_t)bh * R + r0 + tq + iq) * D + td;
        alignas(16) T w[8];
#pragma unroll
        for (int d = 0; d < 4; ++d) {
            float a0, a1;
            const ulonglong2 x = tot[(iq * 2 + d / 2) * PF_THREADS];
            ptx::unpack2((d & 1) ? x.y : x.x, a0, a1);
            nan |= a0 != a0 || a1 != a1;
            w[2 * d] = Cvt<T>::down(div_canon(a0, Lt[iq]));
            w[2 * d + 1] = Cvt<T>::down(div_canon(a1, Lt[iq]));
        }
        if (rows16) {
#pragma unroll
            for (int i = 0; i < (int)sizeof(w) / 16; ++i) reinterpret_cast<uint4*>(o)[i] = reinterpret_cast<const uint4*>(w)[i];
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = w[i];
        }
        if (nan) ms[tq + iq] = NAN;                                      // a running maximum is never NaN
        poisoned |= nan;
    }
    // Phase C folds a key that a row does not see into it with weight 0: no change, unless the key's value holds an infinity
    // or NaN, whose product with 0 stays in the accumulator as NaN to the end. Rows that end with one are computed again
    // without their unseen keys, so that no later token reaches a row. (Skipping unseen keys in phase C, or looking for such
    // values there, cost 2-8 % of every launch and up to 39 % where a row block straddles two heads.)
    if (causal && __syncthreads_or(poisoned))
        literal_rows<T, DL, TQ>(ms, q, k, v, out, B, Hkv, G, Tq, L, lay.sb, lay.sh, lay.sl, scale, split);
}

template <typename T, int DL, int TQ>
int launch_prefill_tq(const void* q, const void* k, const void* v, void* out, int64_t B, int64_t Hq, int64_t Hkv,
                   int64_t Tq, int64_t L, const KvLayout& lay, float scale, int causal, int split, cudaStream_t st) {
    using C = PF<T, DL, TQ>;
    static_assert(C::SMEM <= PF_SMEM_MAX, "more shared memory than a CTA may have");
    const int64_t G = Hq / Hkv;
    const int64_t blocks = B * Hkv * ((G * Tq + C::QB - 1) / C::QB);
    if (blocks > 0x7fffffffLL) return fail(BI_ERR_UNSUPPORTED, "bi_attn_prefill: grid too large");
    const int64_t per16 = 16 / (int64_t)sizeof(T);
    const int rows16 = aligned(k, 16) && aligned(v, 16) && aligned(out, 16) && lay.sb % per16 == 0 && lay.sh % per16 == 0 && lay.sl % per16 == 0;
    constexpr auto kern = prefill_kernel<T, DL, TQ>;
    if (!opt_in_smem<kern>()) return fail_cuda("bi_attn_prefill smem attr", cudaErrorInvalidValue);
    // More CTAs than SMs are launched plainly: two or three lie on an SM, unevenly when they are let in beside a running kernel, in
    // long prompts too, whose blocks differ in keys. Linear and attention of 512 tokens, 32 / 8 heads of 128: 143 us so, 120 plainly
    // (1400 tokens 675 and 683); norm, linear and 512 tokens of 14 / 2 heads of 64 89 and 63, held to two an SM 75. Held to one,
    // 100 tokens of 32 / 8 heads in a row take 18.1 us, 18.5 plainly (eagerly 18.9 and 21.0).
    const bool overlapped = pdl_enabled() && blocks <= sm_count();
    launch_kernel(overlapped, kern, dim3((unsigned)blocks), dim3(PF_THREADS), overlapped ? spread_smem<kern>(blocks, C::SMEM) : C::SMEM, st,
        static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), static_cast<T*>(out), (int)B, (int)Hkv,
        (int)G, (int)Tq, (int)L, lay, scale, causal, split, rows16);
    return check_launch("bi_attn_prefill");
}

template <typename T, int DL>
int launch_prefill(const void* q, const void* k, const void* v, void* out, int64_t B, int64_t Hq, int64_t Hkv,
                   int64_t Tq, int64_t L, const KvLayout& lay, float scale, int causal, int split, cudaStream_t st) {
    // Rows per thread: four give every loaded operand the most use and win while at least two CTAs per SM are left
    // (32 heads x 2048 tokens: 1231 us with four, 1420 with two, 1908 with one); with fewer CTAs the block's serial
    // chain is what counts and shorter row blocks are faster (8 heads x 16 queries over 1000 keys: 119 / 75 / 56 us). Four
    // rows of fp32 with 256 dims would take 240 KB of shared memory.
    const int64_t rows = (Hq / Hkv) * Tq, sms = sm_count();
    if (split > 1 << 30) split = 1 << 30;                  // the most keys there are: sums with a split stay in 32 bits
    auto ctas = [&](int qb) { return B * Hkv * ((rows + qb - 1) / qb); };
    if constexpr (PF<T, DL, 4>::SMEM <= PF_SMEM_MAX) {
        if (ctas(PF<T, DL, 4>::QB) >= 2 * sms) return launch_prefill_tq<T, DL, 4>(q, k, v, out, B, Hq, Hkv, Tq, L, lay, scale, causal, split, st);
    }
    if (ctas(PF<T, DL, 2>::QB) >= sms / 2) return launch_prefill_tq<T, DL, 2>(q, k, v, out, B, Hq, Hkv, Tq, L, lay, scale, causal, split, st);
    return launch_prefill_tq<T, DL, 1>(q, k, v, out, B, Hq, Hkv, Tq, L, lay, scale, causal, split, st);
}

}  // namespace
}  // namespace bi

extern "C" int bi_attn_prefill(const void* q, const void* k, const void* v, void* out, int64_t B, int64_t Hq,
                               int64_t Hkv, int64_t Tq, int64_t L, int64_t D, int64_t kv_sb, int64_t kv_sh,
                               int64_t kv_sl, float scale, int causal, int split_size, int dtype, void* stream) {
    using namespace bi;
    KvLayout lay{kv_sb, kv_sh, kv_sl};
    int rc = check_attention("bi_attn_prefill", q, k, v, out, B, Hq, Hkv, Tq, L, D, lay, split_size, dtype);
    if (rc || B == 0) return rc;
    if (causal && Tq > L) return fail(BI_ERR_BAD_ARG, "bi_attn_prefill: causal needs Tq <= L (Tq=%lld L=%lld)", (long long)Tq, (long long)L);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    BI_DISPATCH_T_DL(launch_prefill, q, k, v, out, B, Hq, Hkv, Tq, L, lay, scale, causal, split_size, st);
}

