// RMSNorm: one CTA of 256 threads per row, or, for many rows, a warp that stands for those threads.
//
// Canonical order per row (identical to the Metal kernel of the reference,
// mlx_batch_invariant/kernels/rmsnorm.py:19-47):
//   thread t:  ss_t = 0; for i = t, t+256, ...: ss_t = fma(x_i, x_i, ss_t)
//   tree:      for s = 128, 64, ..., 1: red[t] = red[t] + red[t+s]  (t < s)
//   inv  = 1 / sqrt(red[0] / float(D) + eps)
//   out_i = T((x_i * inv) * w_i)          two fp32 multiplies, one rounding
// How many rows share the launch never enters: a row sees only its own CTA, or its own warp.
//
// bi_add_rms_norm is the same kernel with a residual add in front: sum_i = T(x_i + delta_i) (fp32 add, one
// rounding -- what an elementwise add of two T arrays gives), written out, and the norm runs over the
// rounded sums exactly as if they had been read back from memory.
//
// A decode batch is one wave of CTAs, each a chain of memory and barrier latencies: the weight is fetched beside the row, the
// residual's and the row's pieces before the first is stored, and the tree's upper three levels are one barrier instead of
// three (64 / 1 rows of 4096 with the residual in the decoder's step: 4.4 / 4.2 -> 3.2 / 2.7 us).
//
// Data movement is free to differ from the reference: the row is staged in
// shared memory with 16-byte loads, each thread then walks its stride-256
// elements there, results are written back in place and leave with 16-byte
// stores. Rows too long for shared memory, or not 16-byte aligned, take the
// same arithmetic straight from global memory.
#include <type_traits>
#include "bi_common.cuh"
#include "bi_ptx.cuh"

namespace bi {
namespace {

constexpr int TG = 256;

__device__ __forceinline__ float block_tree_sum(float ss, float* red, int t) {
    red[t] = ss;
    __syncthreads();
    if (t < 32) {
        // levels 128, 64 and 32 over the eight values whose tree ends in red[t]: the same pairs, without a barrier a level
        float a[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = add_rn(red[t + 32 * i], red[t + 32 * i + 128]);
        float v = add_rn(add_rn(a[0], a[2]), add_rn(a[1], a[3]));
        v = add_rn(v, __shfl_down_sync(0xffffffffu, v, 16));
        v = add_rn(v, __shfl_down_sync(0xffffffffu, v, 8));
        v = add_rn(v, __shfl_down_sync(0xffffffffu, v, 4));
        v = add_rn(v, __shfl_down_sync(0xffffffffu, v, 2));
        v = add_rn(v, __shfl_down_sync(0xffffffffu, v, 1));
        if (t == 0) red[0] = v;
    }
    __syncthreads();
    return red[0];
}

// `delta` may be the destination of a peer gather whose arrival nobody has waited for yet: the CTA then first
// waits (bounded, 2 s) until every peer's flag has reached *epoch; on expiry it records a code and goes on.
struct NormAwait {
    const uint32_t* flags;
    const uint32_t* epoch;
    int rank, world;
    int32_t* status;
};

template <typename T, bool STAGED, bool HAS_W, bool HAS_RES>
__global__ void __launch_bounds__(TG) rms_norm_kernel(const T* x, const T* __restrict__ delta, const T* __restrict__ w,
                                                      T* sum_out, T* __restrict__ out, int D, float eps, NormAwait aw) {
    ptx::grid_dep_wait_and_launch();
    extern __shared__ uint4 stage_raw[];
    __shared__ float red[TG];
    const int t = threadIdx.x;
    if (HAS_RES && aw.flags != nullptr) {
        if (t < aw.world && t != aw.rank) {
            const uint32_t epoch = *aw.epoch;
            uint64_t t0;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
            while (true) {
                uint32_t seen;
                asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(aw.flags + t) : "memory");
                if ((int32_t)(seen - epoch) >= 0) break;
                uint64_t now;
                asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
                if (now - t0 > 2000000000ull) {
                    if (aw.status) atomicCAS(aw.status, 0, (int)(0x20000 | (t << 8) | (epoch & 0xff)));
                    break;
                }
            }
        }
        __syncthreads();
    }
    const size_t row = blockIdx.x;
    const T* xr = x + row * (size_t)D;
    T* orow = out + row * (size_t)D;
    T* xs = reinterpret_cast<T*>(stage_raw);

    if (STAGED) {
        constexpr int VEC = 16 / sizeof(T);
        const uint4* src = reinterpret_cast<const uint4*>(xr);
        if (HAS_RES) {
            // x + delta, rounded to T, goes to shared memory for the norm and to sum_out (which may be x)
            const uint4* dsrc = reinterpret_cast<const uint4*>(delta + row * (size_t)D);
            uint4* sdst = reinterpret_cast<uint4*>(sum_out + row * (size_t)D);
            auto put = [&](int i, uint4 a, const uint4& b) {
                T* av = reinterpret_cast<T*>(&a);
                const T* bv = reinterpret_cast<const T*>(&b);
#pragma unroll
                for (int j = 0; j < VEC; ++j) av[j] = Cvt<T>::down(add_rn(Cvt<T>::up(av[j]), Cvt<T>::up(bv[j])));
                stage_raw[i] = a;
                sdst[i] = a;
            };
            for (int i = t; i < D / VEC; i += 2 * TG) {              // the loads of two pieces before the first store
                const bool two = i + TG < D / VEC;
                const uint4 a0 = src[i], b0 = dsrc[i];
                uint4 a1 = a0, b1 = b0;
                if (two) { a1 = src[i + TG]; b1 = dsrc[i + TG]; }
                put(i, a0, b0);
                if (two) put(i + TG, a1, b1);
            }
        } else {
            for (int i = t; i < D / VEC; i += TG) stage_raw[i] = __ldg(src + i);
        }
    } else if (HAS_RES) {
        const T* dr = delta + row * (size_t)D;
        T* sr = sum_out + row * (size_t)D;
        for (int i = t; i < D; i += TG) sr[i] = Cvt<T>::down(add_rn(Cvt<T>::up(xr[i]), Cvt<T>::up(dr[i])));
        // each thread reads back only what it wrote
    }
    const T* xin = STAGED ? xs : (HAS_RES ? sum_out + row * (size_t)D : xr);

    // Rows of up to 256 * KEEP elements keep the thread's values in registers between the two passes (the second
    // pass then reads neither shared nor global memory for x); longer rows read them again.
    constexpr int KEEP = 16;
    const bool keep = D <= TG * KEEP;
    float kept[KEEP];
    T wk[HAS_W ? KEEP : 1];                       // fetched beside the row: behind the reduction their latency stood alone
    float ss = 0.0f;
    if (keep) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j)
            if (HAS_W && t + j * TG < D) wk[j] = w[t + j * TG];
    }
    if (STAGED) __syncthreads();                  // the row is staged
    if (keep) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j) {
            const int i = t + j * TG;
            kept[j] = i < D ? Cvt<T>::up(xin[i]) : 0.0f;
            if (i < D) ss = fma_rn(kept[j], kept[j], ss);
        }
    } else {
        for (int i = t; i < D; i += TG) {
            float v = Cvt<T>::up(xin[i]);
            ss = fma_rn(v, v, ss);
        }
    }
    const float total = block_tree_sum(ss, red, t);
    const float inv = rsqrt_canon(add_rn(div_canon(total, (float)D), eps));

    if (keep) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j) {
            const int i = t + j * TG;
            if (i < D) {
                const float v = mul_rn(kept[j], inv);
                const float wi = HAS_W ? Cvt<T>::up(wk[HAS_W ? j : 0]) : 1.0f;
                const T o = Cvt<T>::down(mul_rn(v, wi));
                if (STAGED) xs[i] = o; else orow[i] = o;
            }
        }
    } else {
        for (int i = t; i < D; i += TG) {
            float v = mul_rn(Cvt<T>::up(xin[i]), inv);
            float wi = HAS_W ? Cvt<T>::up(w[i]) : 1.0f;
            T o = Cvt<T>::down(mul_rn(v, wi));
            if (STAGED) xs[i] = o; else orow[i] = o;
        }
    }
    if (STAGED) {
        constexpr int VEC = 16 / sizeof(T);
        __syncthreads();
        uint4* dst = reinterpret_cast<uint4*>(orow);
        for (int i = t; i < D / VEC; i += TG) dst[i] = stage_raw[i];
    }
}

// A warp per row, for many rows: lane l owns virtual threads 8 l ... 8 l + 7, whose stride-256 elements are exactly pieces
// l, l + 32, ... of eight elements of the row, and the tree is shuffles: levels 128, 64, 32 halve the eight values a lane
// holds (it keeps the half its lane bit names and adds its partner's), 16 and 8 add whole lanes, 4, 2, 1 meet over the same
// three lane bits -- the canonical pairs, whose order inside an add is free.
__device__ __forceinline__ float warp_tree_sum(const float (&ss)[8], int lane) {
    float h4[4], h2[2], h;
    const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) {                        // red[t] + red[t + 128]
        const float got = __shfl_xor_sync(0xffffffffu, b16 ? ss[e] : ss[e + 4], 16);
        h4[e] = add_rn(b16 ? ss[e + 4] : ss[e], got);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {                        // 64
        const float got = __shfl_xor_sync(0xffffffffu, b8 ? h4[e] : h4[e + 2], 8);
        h2[e] = add_rn(b8 ? h4[e + 2] : h4[e], got);
    }
    {                                                    // 32
        const float got = __shfl_xor_sync(0xffffffffu, b4 ? h2[0] : h2[1], 4);
        h = add_rn(b4 ? h2[1] : h2[0], got);
    }
    h = add_rn(h, __shfl_xor_sync(0xffffffffu, h, 2));   // 16
    h = add_rn(h, __shfl_xor_sync(0xffffffffu, h, 1));   // 8
    h = add_rn(h, __shfl_xor_sync(0xffffffffu, h, 16));  // 4: the value kept by the other half
    h = add_rn(h, __shfl_xor_sync(0xffffffffu, h, 8));   // 2
    h = add_rn(h, __shfl_xor_sync(0xffffffffu, h, 4));   // 1
    return h;
}

// 16-bit rows of up to 16 KB: the row waits in shared memory, brought by cp.async in two halves (a lane reads only what it
// copied itself, so nothing but its own wait stands between the copies and the sums). What bounds it: memory, by the bytes in
// flight. With the row in registers 16 to 20 warps fit an SM (160 KB in flight, and 2400 rows of bf16 took a second wave);
// staged, 26 rows of 8 KB do (13 CTAs of 16 KB and the 1 KB that a CTA is charged: 3848 rows a wave), and longer rows no
// longer fall back to a CTA per row, which spends its time on load, five barriers and store in series. Neither rows nor
// results in L2, bf16: 4093 x 4096 16.7 -> 14.4 us (6000: 23.8 -> 19.0; 2400: 12.9 -> 9.7, fp16 9.0 -> 9.5), 4093 x 896 7.1 ->
// 5.1 us, 4093 x 8192 34.9 -> 26.5 us, 32768 x 64 29.8 -> 18.3 us. Two rows a CTA: four are up to 5 % slower from 6144 elements
// on (4093 x 6144 20.4 against 21.4 us) and up to 25 % faster below 512 (32768 x 128 18.3 against 14.1). With results in L2,
// one piece of copies instead of two halves, and loops unrolled by four, were 5 to 20 % slower.
constexpr int STAGED_ROWS = 2;                           // 14 CTAs below: a cap of 72 registers, no occupancy is lost to them
constexpr size_t STAGED_ROW_MAX = 16 * 1024;
template <typename T, bool HAS_W>
__global__ void __launch_bounds__(32 * STAGED_ROWS, 14) rms_norm_staged_warp_kernel(const T* x, const T* __restrict__ w, T* out, long long rows,
                                                                                    int D, float eps) {
    static_assert(sizeof(T) == 2 && STAGED_ROWS * STAGED_ROW_MAX <= 48 * 1024, "a piece of eight elements is one 16-byte word; no shared-memory opt-in");
    ptx::grid_dep_wait_and_launch();
    extern __shared__ uint4 stage_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long row = (long long)blockIdx.x * STAGED_ROWS + wid;
    if (row >= rows) return;
    const int n = D >> 3, half = (n >> 6) << 5;          // pieces of the row; whole rounds of the warp in front of the second wait
    const size_t at = (size_t)row * (size_t)D;
    uint4* const buf = stage_raw + (size_t)wid * (size_t)n;
    const uint4* const src = reinterpret_cast<const uint4*>(x + at);
    const uint32_t buf_s = (uint32_t)__cvta_generic_to_shared(buf);
    auto fetch = [&](int i) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buf_s + (uint32_t)i * 16u), "l"(src + i) : "memory"); };
#pragma unroll 8
    for (int i = lane; i < half; i += 32) fetch(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 8
    for (int i = half + lane; i < n; i += 32) fetch(i);
    asm volatile("cp.async.commit_group;" ::: "memory");
    float ss[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) ss[e] = 0.0f;
    auto add = [&](int i) {
        const uint4 v = buf[i];
        const T* a = reinterpret_cast<const T*>(&v);
#pragma unroll
        for (int e = 0; e < 8; ++e) { const float f = Cvt<T>::up(a[e]); ss[e] = fma_rn(f, f, ss[e]); }
    };
    asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll 8
    for (int i = lane; i < half; i += 32) add(i);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll 8
    for (int i = half + lane; i < n; i += 32) add(i);
    const float h = warp_tree_sum(ss, lane);
    const float inv = rsqrt_canon(add_rn(div_canon(h, (float)D), eps));
    uint4* const dst = reinterpret_cast<uint4*>(out + at);
#pragma unroll 8
    for (int i = lane; i < n; i += 32) {
        uint4 v = buf[i], wv = make_uint4(0u, 0u, 0u, 0u);
        if (HAS_W) wv = reinterpret_cast<const uint4*>(w)[i];
        T* a = reinterpret_cast<T*>(&v);
        const T* b = reinterpret_cast<const T*>(&wv);
#pragma unroll
        for (int e = 0; e < 8; ++e) a[e] = Cvt<T>::down(mul_rn(mul_rn(Cvt<T>::up(a[e]), inv), HAS_W ? Cvt<T>::up(b[e]) : 1.0f));
        dst[i] = v;
    }
}

// fp32 rows of up to 1024 elements: the row stays in the lane's registers from the load to the store (two 16-byte words a
// piece; 4093 x 896, results in L2: 6.3 us, staged like the 16-bit rows 7.8).
constexpr int WARP_ROWS = 4;
constexpr int WARP_ROW_MAX = 1024;                       // longest row kept in registers
template <bool HAS_W>
__global__ void __launch_bounds__(32 * WARP_ROWS) rms_norm_warp_kernel(const float* x, const float* __restrict__ w, float* out, long long rows,
                                                                       int D, float eps) {
    using T = float;
    ptx::grid_dep_wait();      // the next kernel is let in at the end: fp32 linears have no weights to fetch ahead (4093 x 896 6.1 -> 5.2 us)
    constexpr int PIECES = WARP_ROW_MAX / 256;          // eight elements of a lane each
    constexpr int Q = sizeof(T) / 2;                     // 16-byte words per piece
    struct Piece { uint4 q[Q]; };
    const int lane = threadIdx.x & 31;
    const long long row = (long long)blockIdx.x * WARP_ROWS + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int n = D >> 3;
    auto load = [&](const T* base, int i) {
        Piece r;
#pragma unroll
        for (int k = 0; k < Q; ++k) r.q[k] = reinterpret_cast<const uint4*>(base)[i * Q + k];
        return r;
    };
    auto store = [&](T* base, int i, const Piece& r) {
#pragma unroll
        for (int k = 0; k < Q; ++k) reinterpret_cast<uint4*>(base)[i * Q + k] = r.q[k];
    };
    const size_t at = (size_t)row * (size_t)D;
    Piece v[PIECES];
#pragma unroll
    for (int j = 0; j < PIECES; ++j)
        if (j * 32 + lane < n) v[j] = load(x + at, j * 32 + lane);
    float ss[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) ss[e] = 0.0f;
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const int i = j * 32 + lane;
        if (i < n) {
            const T* a = reinterpret_cast<const T*>(&v[j]);
#pragma unroll
            for (int e = 0; e < 8; ++e) { const float f = Cvt<T>::up(a[e]); ss[e] = fma_rn(f, f, ss[e]); }
        }
    }
    const float h = warp_tree_sum(ss, lane);
    const float inv = rsqrt_canon(add_rn(div_canon(h, (float)D), eps));
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const int i = j * 32 + lane;
        if (i < n) {
            T* a = reinterpret_cast<T*>(&v[j]);
            Piece wp;
            if (HAS_W) wp = load(w, i);
            const T* b = reinterpret_cast<const T*>(&wp);
#pragma unroll
            for (int e = 0; e < 8; ++e) a[e] = Cvt<T>::down(mul_rn(mul_rn(Cvt<T>::up(a[e]), inv), HAS_W ? Cvt<T>::up(b[e]) : 1.0f));
            store(out + at, i, v[j]);
        }
    }
}

// LayerNorm, one CTA of 256 threads per row, in the manner of the RMSNorm above (the reference lists a
// batch-invariant LayerNorm as future work, README.md:261-263 there; this is its canonical order here):
//   thread t:  s_t = 0;  for i = t, t+256, ...: s_t = s_t + x_i           tree 128..1 -> mean = sum / float(D)
//   thread t:  q_t = 0;  for i = t, t+256, ...: d = x_i - mean; q_t = fma(d, d, q_t)   tree -> var = q / float(D)
//   inv = 1 / sqrt(var + eps);  out_i = T((((x_i - mean) * inv) * w_i) + b_i)   (w, b optional; one rounding)
template <typename T, bool HAS_W, bool HAS_B>
__global__ void __launch_bounds__(TG) layer_norm_kernel(const T* __restrict__ x, const T* __restrict__ w, const T* __restrict__ b,
                                                        T* __restrict__ out, int D, float eps) {
    if (gridDim.x < 64) ptx::grid_dep_launch();
    ptx::grid_dep_wait();     // everything before this kernel has completed and is visible
    __shared__ float red[TG];
    const int t = threadIdx.x;
    const T* xr = x + (size_t)blockIdx.x * (size_t)D;
    T* orow = out + (size_t)blockIdx.x * (size_t)D;
    constexpr int KEEP = 16;                     // rows of up to 4096 elements stay in registers after the first read
    const bool keep = D <= TG * KEEP;
    float kept[KEEP];
    float s = 0.0f;
    if (keep) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j) {
            const int i = t + j * TG;
            kept[j] = i < D ? Cvt<T>::up(xr[i]) : 0.0f;
            if (i < D) s = add_rn(s, kept[j]);
        }
    } else {
        for (int i = t; i < D; i += TG) s = add_rn(s, Cvt<T>::up(xr[i]));
    }
    const float mean = div_canon(block_tree_sum(s, red, t), (float)D);
    ptx::grid_dep_launch();                      // the row is read (600 rows of 4096, a chain of norms: let in at the start 5.3 us, here 4.8; in front of a linear 14.0 and 14.1)
    __syncthreads();                             // red[] is reused by the second reduction
    float q = 0.0f;
    if (keep) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j) {
            const int i = t + j * TG;
            if (i < D) { const float d = sub_rn(kept[j], mean); q = fma_rn(d, d, q); }
        }
    } else {
        for (int i = t; i < D; i += TG) { const float d = sub_rn(Cvt<T>::up(xr[i]), mean); q = fma_rn(d, d, q); }
    }
    const float var = div_canon(block_tree_sum(q, red, t), (float)D);
    const float inv = rsqrt_canon(add_rn(var, eps));
    auto finish = [&](float xv, int i) {
        float y = mul_rn(sub_rn(xv, mean), inv);
        if (HAS_W) y = mul_rn(y, Cvt<T>::up(w[i]));
        if (HAS_B) y = add_rn(y, Cvt<T>::up(b[i]));
        orow[i] = Cvt<T>::down(y);
    };
    if (keep) {
#pragma unroll
        for (int j = 0; j < KEEP; ++j) {
            const int i = t + j * TG;
            if (i < D) finish(kept[j], i);
        }
    } else {
        for (int i = t; i < D; i += TG) finish(Cvt<T>::up(xr[i]), i);
    }
}

template <typename T>
int launch_layer_norm(const void* x, const void* w, const void* b, void* out, int64_t rows, int64_t D, float eps, cudaStream_t st) {
    const T* xp = static_cast<const T*>(x);
    const T* wp = static_cast<const T*>(w);
    const T* bp = static_cast<const T*>(b);
    T* op = static_cast<T*>(out);
    dim3 grid((unsigned)rows), block(TG);
    if (w && b) launch_overlapped(layer_norm_kernel<T, true, true>, grid, block, 0, st, xp, wp, bp, op, (int)D, eps);
    else if (w) launch_overlapped(layer_norm_kernel<T, true, false>, grid, block, 0, st, xp, wp, bp, op, (int)D, eps);
    else if (b) launch_overlapped(layer_norm_kernel<T, false, true>, grid, block, 0, st, xp, wp, bp, op, (int)D, eps);
    else launch_overlapped(layer_norm_kernel<T, false, false>, grid, block, 0, st, xp, wp, bp, op, (int)D, eps);
    return check_launch("bi_layer_norm");
}

template <typename T>
int launch(const void* x, const void* delta, const void* w, void* sum_out, void* out, int64_t rows, int64_t D, float eps,
           cudaStream_t st, const NormAwait& aw = NormAwait{nullptr, nullptr, 0, 0, nullptr}) {
    const size_t row_bytes = (size_t)D * sizeof(T);
    const bool staged = row_bytes % 16 == 0 && row_bytes <= 160 * 1024 && aligned(x, 16) && aligned(out, 16) &&
                        (!delta || (aligned(delta, 16) && aligned(sum_out, 16)));
    const T* xp = static_cast<const T*>(x);
    const T* dp = static_cast<const T*>(delta);
    const T* wp = static_cast<const T*>(w);
    T* sp = static_cast<T*>(sum_out);
    T* op = static_cast<T*>(out);
    // A warp per row once there are rows enough for it, by times over rows and results that are not in L2. 16-bit rows of up to
    // 16 KB from 512 on: there it is faster at every width (bf16, 256 / 511 rows by a CTA -> by a warp: 4096 4.0 / 4.9 -> 3.9 /
    // 4.6 us, 896 3.2 / 3.8 -> 3.4 / 3.5, 8192 5.5 / 7.9 -> 5.6 / 6.7, 6144 4.7 / 6.4 -> 4.9 / 5.8). fp32 rows of up to 4 KB from
    // 1024 on (results in L2, 896: 5.7 -> 4.1 us); longer ones leave too few warps in flight (4093 x 4096: 26.5 against 34.7 us
    // staged). With the residual's second stream the CTA per row is not slower.
    if (staged && !delta && D % 8 == 0 && (!w || aligned(w, 16))) {
        if constexpr (sizeof(T) == 2) {
            if (row_bytes <= STAGED_ROW_MAX && rows >= 512) {
                auto kern = w ? rms_norm_staged_warp_kernel<T, true> : rms_norm_staged_warp_kernel<T, false>;
                const dim3 wgrid((unsigned)((rows + STAGED_ROWS - 1) / STAGED_ROWS)), wblock(32 * STAGED_ROWS);
                launch_overlapped(kern, wgrid, wblock, STAGED_ROWS * row_bytes, st, xp, wp, op, (long long)rows, (int)D, eps);
                return check_launch("bi_rms_norm");
            }
        } else if (D <= WARP_ROW_MAX && rows >= 1024) {
            auto kern = w ? rms_norm_warp_kernel<true> : rms_norm_warp_kernel<false>;
            const dim3 wgrid((unsigned)((rows + WARP_ROWS - 1) / WARP_ROWS)), wblock(32 * WARP_ROWS);
            launch_overlapped(kern, wgrid, wblock, 0, st, xp, wp, op, (long long)rows, (int)D, eps);
            return check_launch("bi_rms_norm");
        }
    }
    dim3 grid((unsigned)rows), block(TG);
#define BI_RMS_LAUNCH2(ST, HW, HR)                                                                  \
    do {                                                                                            \
        auto kern = rms_norm_kernel<T, ST, HW, HR>;                                                 \
        size_t smem = ST ? row_bytes : 0;                                                           \
        if (smem > 48 * 1024) {                                                                     \
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                                 (int)smem);                                        \
            if (e != cudaSuccess) return fail_cuda("rms_norm smem attr", e);                               \
        }                                                                                           \
        launch_overlapped_unless(aw.flags != nullptr, kern, grid, block, smem, st, xp, dp, wp, sp, op, (int)D, eps, aw);                       \
    } while (0)
#define BI_RMS_LAUNCH(ST, HW) do { if (delta) BI_RMS_LAUNCH2(ST, HW, true); else BI_RMS_LAUNCH2(ST, HW, false); } while (0)
    if (staged) { if (w) BI_RMS_LAUNCH(true, true); else BI_RMS_LAUNCH(true, false); }
    else        { if (w) BI_RMS_LAUNCH(false, true); else BI_RMS_LAUNCH(false, false); }
#undef BI_RMS_LAUNCH
#undef BI_RMS_LAUNCH2
    return check_launch(delta ? "bi_add_rms_norm" : "bi_rms_norm");
}

}  // namespace
}  // namespace bi

extern "C" int bi_rms_norm(const void* x, const void* w, void* out, int64_t rows, int64_t D, float eps,
                           int dtype, void* stream) {
    using namespace bi;
    if (!dtype_ok(dtype)) return fail(BI_ERR_UNSUPPORTED, "bi_rms_norm: dtype %d", dtype);
    if (rows < 0 || D <= 0 || D > INT32_MAX) return fail(BI_ERR_BAD_ARG, "bi_rms_norm: rows=%lld D=%lld", (long long)rows, (long long)D);
    if (rows == 0) return BI_OK;
    if (!x || !out) return fail(BI_ERR_BAD_ARG, "bi_rms_norm: null pointer");
    if (rows > 0x7fffffffLL) return fail(BI_ERR_UNSUPPORTED, "bi_rms_norm: rows=%lld exceeds the grid limit", (long long)rows);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case BI_F32: return launch<float>(x, nullptr, w, nullptr, out, rows, D, eps, st);
        case BI_F16: return launch<__half>(x, nullptr, w, nullptr, out, rows, D, eps, st);
        default:     return launch<__nv_bfloat16>(x, nullptr, w, nullptr, out, rows, D, eps, st);
    }
}

extern "C" int bi_add_rms_norm(const void* x, const void* delta, const void* w, void* sum_out, void* out, int64_t rows,
                               int64_t D, float eps, int dtype, void* stream) {
    using namespace bi;
    if (!dtype_ok(dtype)) return fail(BI_ERR_UNSUPPORTED, "bi_add_rms_norm: dtype %d", dtype);
    if (rows < 0 || D <= 0 || D > INT32_MAX) return fail(BI_ERR_BAD_ARG, "bi_add_rms_norm: rows=%lld D=%lld", (long long)rows, (long long)D);
    if (rows == 0) return BI_OK;
    if (!x || !delta || !sum_out || !out) return fail(BI_ERR_BAD_ARG, "bi_add_rms_norm: null pointer");
    if (out == sum_out || out == x || out == delta) return fail(BI_ERR_BAD_ARG, "bi_add_rms_norm: out must not alias x, delta or sum_out");
    if (rows > 0x7fffffffLL) return fail(BI_ERR_UNSUPPORTED, "bi_add_rms_norm: rows=%lld exceeds the grid limit", (long long)rows);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case BI_F32: return launch<float>(x, delta, w, sum_out, out, rows, D, eps, st);
        case BI_F16: return launch<__half>(x, delta, w, sum_out, out, rows, D, eps, st);
        default:     return launch<__nv_bfloat16>(x, delta, w, sum_out, out, rows, D, eps, st);
    }
}

extern "C" int bi_add_rms_norm_awaiting(const void* x, const void* delta, const void* w, void* sum_out, void* out, int64_t rows,
                                        int64_t D, float eps, int dtype, void* stream, const uint32_t* flags,
                                        const uint32_t* epoch, int rank, int world, int32_t* status) {
    using namespace bi;
    if (!dtype_ok(dtype)) return fail(BI_ERR_UNSUPPORTED, "bi_add_rms_norm_awaiting: dtype %d", dtype);
    if (rows < 0 || D <= 0 || D > INT32_MAX) return fail(BI_ERR_BAD_ARG, "bi_add_rms_norm_awaiting: rows=%lld D=%lld", (long long)rows, (long long)D);
    if (rows == 0) return BI_OK;
    if (!x || !delta || !sum_out || !out) return fail(BI_ERR_BAD_ARG, "bi_add_rms_norm_awaiting: null pointer");
    if (out == sum_out || out == x || out == delta) return fail(BI_ERR_BAD_ARG, "bi_add_rms_norm_awaiting: out must not alias x, delta or sum_out");
    if (rows > 0x7fffffffLL) return fail(BI_ERR_UNSUPPORTED, "bi_add_rms_norm_awaiting: rows=%lld exceeds the grid limit", (long long)rows);
    if (flags && (!epoch || world < 1 || world > 8 || rank < 0 || rank >= world))
        return fail(BI_ERR_BAD_ARG, "bi_add_rms_norm_awaiting: bad gather to wait for (rank %d of %d)", rank, world);
    const NormAwait aw{flags, epoch, rank, world, status};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case BI_F32: return launch<float>(x, delta, w, sum_out, out, rows, D, eps, st, aw);
        case BI_F16: return launch<__half>(x, delta, w, sum_out, out, rows, D, eps, st, aw);
        default:     return launch<__nv_bfloat16>(x, delta, w, sum_out, out, rows, D, eps, st, aw);
    }
}

extern "C" int bi_layer_norm(const void* x, const void* w, const void* b, void* out, int64_t rows, int64_t D, float eps,
                             int dtype, void* stream) {
    using namespace bi;
    if (!dtype_ok(dtype)) return fail(BI_ERR_UNSUPPORTED, "bi_layer_norm: dtype %d", dtype);
    if (rows < 0 || D <= 0 || D > INT32_MAX) return fail(BI_ERR_BAD_ARG, "bi_layer_norm: rows=%lld D=%lld", (long long)rows, (long long)D);
    if (rows == 0) return BI_OK;
    if (!x || !out) return fail(BI_ERR_BAD_ARG, "bi_layer_norm: null pointer");
    if (rows > 0x7fffffffLL) return fail(BI_ERR_UNSUPPORTED, "bi_layer_norm: rows=%lld exceeds the grid limit", (long long)rows);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case BI_F32: return launch_layer_norm<float>(x, w, b, out, rows, D, eps, st);
        case BI_F16: return launch_layer_norm<__half>(x, w, b, out, rows, D, eps, st);
        default:     return launch_layer_norm<__nv_bfloat16>(x, w, b, out, rows, D, eps, st);
    }
}
