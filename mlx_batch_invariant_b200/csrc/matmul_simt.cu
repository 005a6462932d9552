// CUDA-core matmul with the K-group contract, and the split-path combine kernel.
//
// Canonical order per output element on this path:
//   for each K group g (256 wide, ascending):  acc = 0;
//       for k ascending inside the group:      acc = fma(a[m,k], b[k,n], acc)
//   total = 0;  total = total + acc_g          (plain fp32 adds, g ascending)
//   out = T(total)                             (one rounding)
// Operands are upcast to fp32 exactly; every product/sum is a single fp32 fma.
// It serves fp32 inputs (Blackwell tensor cores have no full-precision fp32
// mode) and 16-bit weights whose rows cannot be described to TMA. Which path a
// weight takes depends on the weight alone, never on the batch.
//
// Two launch shapes, as in the reference (mlx_batch_invariant/kernels/matmul.py:279-314):
// fused (one CTA walks all groups and folds) and split (grid.z = group, raw fp32
// partials, then combine_kernel folds them). Both perform the same sequence of
// operations on every element.
#include <type_traits>
#include "bi_common.cuh"
#include "bi_ptx.cuh"
#include "matmul_internal.cuh"

namespace bi {
namespace {

struct QuantArgs {
    const uint32_t* w;   // [N, K*bits/32]
    const void* scales;  // [N, K/gs]
    const void* biases;
    int bits, gs;
    const void* out_bias;  // optional [N] bias of the linear layer (dense and quantized alike), in T
};

// Affine dequantization of one code: fma in fp32, then one rounding to the staged type T.
template <typename T>
__device__ __forceinline__ float dequant_code(uint32_t code, float s, float b) {
    return Cvt<T>::up(Cvt<T>::down(fma_rn((float)code, s, b)));
}

// A piece, four consecutive k of one row, as it lies in memory: what a thread holds from its fetch to its store into the stage.
template <typename T> struct Raw4 { T v[4]; };
template <typename T> struct RawCodes { uint32_t codes; T scale, bias; };
__device__ __forceinline__ float4 widen(const float4& r) { return r; }
template <typename T> __device__ __forceinline__ float4 widen(const Raw4<T>& r) {
    return make_float4(Cvt<T>::up(r.v[0]), Cvt<T>::up(r.v[1]), Cvt<T>::up(r.v[2]), Cvt<T>::up(r.v[3]));
}
template <typename T> __device__ __forceinline__ float4 widen(const RawCodes<T>& r, int bits) {
    const uint32_t mask = (1u << bits) - 1u;
    const float s = Cvt<T>::up(r.scale), b = Cvt<T>::up(r.bias);
    return make_float4(dequant_code<T>(r.codes & mask, s, b), dequant_code<T>((r.codes >> bits) & mask, s, b),
                       dequant_code<T>((r.codes >> 2 * bits) & mask, s, b), dequant_code<T>((r.codes >> 3 * bits) & mask, s, b));
}

// V consecutive floats of shared memory (V = 1, 2, 4, aligned to their size).
template <int V> __device__ __forceinline__ void ld_floats(const float* p, float* v) {
    if constexpr (V == 4) { const float4 w = *reinterpret_cast<const float4*>(p); v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w; }
    else if constexpr (V == 2) { const float2 w = *reinterpret_cast<const float2*>(p); v[0] = w.x; v[1] = w.y; }
    else v[0] = *p;
}

// A thread's W rows (or columns) of an operand tile lie in runs of four (the last may be shorter), each run one stripe of
// `lanes` such runs after the one before. place(): tile row of element u of thread idx; ld_tile(): all of them at one k.
template <int W> __host__ __device__ constexpr int run_len(int r) { return W - 4 * r < 4 ? W - 4 * r : 4; }
template <int W> __device__ __forceinline__ int place(int idx, int u, int lanes) {
    return lanes * 4 * (u / 4) + idx * run_len<W>(u / 4) + u % 4;
}
template <int W, int R = 0> __device__ __forceinline__ void ld_tile(const float* row, int idx, int lanes, int sw, float* v) {
    if constexpr (4 * R < W) {
        ld_floats<run_len<W>(R)>(row + ((lanes * 4 * R + idx * run_len<W>(R)) ^ sw), v + 4 * R);
        ld_tile<W, R + 1>(row, idx, lanes, sw, v);
    }
}

// A CTA owns BM x BN outputs (BM = MG * TM, BN = NL * TN); thread (mg, nl) holds a TM x TN tile of them. Operand tiles lie
// k-major in shared memory ([k][row]): the TN values of a k are read as consecutive registers, so that the accumulators and
// the operand of every fma can sit in different register banks (k-contiguous tiles, read four k at a time, ran at 60 % of
// the fp32 pipe with the issue slots lost to operand conflicts). A stage is fetched into registers while the one before is
// multiplied and then stored transposed; the row index is swizzled with k / 4 so that a warp's stores meet no bank conflict
// and groups of four rows stay together. k runs in order inside every accumulator; past the end of the operands the
// stages hold zeros (fma(0, 0, acc) leaves acc). Bound by the fp32 pipe from about 16 rows on, below by the stream of weights.
// VEC: fp32 operands with k contiguous and 16-byte aligned rows, fetched as float4. Otherwise element by element (16-bit
// operands, any strides); of packed weights the four codes of a piece share a word and a quantization group (groups and K
// are multiples of 32). A fetched piece is widened or unpacked only when it is stored: done at the fetch, every load is
// waited for before the next one, code by code. At M = 1, widened at the fetch / at the store: bf16 row-major [896, 4864]
// 82 / 21 us, bf16 [4096, 515] 82 / 21 us, fp32 on 4-bit [4096, 512] 85 / 24 us; at M = 256 1040 / 560 us for the last's kin
// [4096, 4096].
template <typename T, int TM, int TN, int MG, int NL, bool SPLIT, bool QUANT, bool VEC>
__global__ void __launch_bounds__(MG * NL, (SPLIT ? (TM * TN > 64 ? 256 : (MG * NL == 64 && TM * TN == 64 ? 320 : 512)) : 256) / (MG * NL))
simt_matmul_kernel(const T* __restrict__ a, const T* __restrict__ b, QuantArgs qa, void* __restrict__ outp, int M, int N, int K,
                   int64_t a_sm, int64_t a_sk, int64_t b_sk, int64_t b_sn) {
    ptx::grid_dep_wait();     // everything before this kernel has completed and is visible
    constexpr int BM = MG * TM, BN = NL * TN, THREADS = MG * NL;
    constexpr int SLAB = 16, SWZ = 3;                                       // k per stage; row ^= (k / 4) << SWZ
    constexpr int PA = (BM + 31) / 32 * 32, PB = (BN + 31) / 32 * 32;       // row pitches of the k-major tiles
    __shared__ __align__(16) float As[2][SLAB][PA];
    __shared__ __align__(16) float Bs[2][SLAB][PB];
    const int tid = threadIdx.x;
    const int nl = tid % NL, mg = tid / NL;
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    const int g0 = SPLIT ? (int)blockIdx.z : 0;
    const int kbeg = g0 * GROUP_K, kend = SPLIT ? min(K, kbeg + GROUP_K) : K;
    const int nslab = (kend - kbeg + SLAB - 1) / SLAB;
    constexpr int SEGS = SLAB / 4;                                          // float4 pieces of a row
    constexpr int STEP = THREADS / SEGS;                                    // rows between a thread's pieces
    constexpr int FA = (BM + STEP - 1) / STEP, FB = (BN + STEP - 1) / STEP; // pieces a thread fetches of either operand

    // The thread's first piece is row `pr`, k offset 4 * `seg`; the others are STEP rows apart.
    const int pr = tid / SEGS, seg = tid % SEGS;
    using Raw = std::conditional_t<VEC, float4, Raw4<T>>;
    using RawB = std::conditional_t<QUANT, RawCodes<T>, Raw>;
    Raw fa[FA];
    RawB fb[FB];
    const T zero = Cvt<T>::down(0.0f);
    auto piece = [&](int row, int tile_rows, int first, int limit, const T* base, int64_t s_row, int64_t s_k, int k) -> Raw {
        if constexpr (VEC) {
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row < tile_rows && first + row < limit && k < kend) v = __ldg(reinterpret_cast<const float4*>(base + (int64_t)(first + row) * s_row + k));
            return v;
        } else {
            Raw v{{zero, zero, zero, zero}};
            if (row < tile_rows && first + row < limit && k < kend) {
                const T* p = base + (int64_t)(first + row) * s_row + (int64_t)k * s_k;
                v.v[0] = p[0];
                if (k + 1 < kend) v.v[1] = p[s_k];
                if (k + 2 < kend) v.v[2] = p[2 * s_k];
                if (k + 3 < kend) v.v[3] = p[3 * s_k];
            }
            return v;
        }
    };
    const int word_shift = qa.bits == 4 ? 3 : 2, group_shift = 31 - __clz(qa.gs);       // QUANT: k per word, per quantization group
    auto codes = [&](int row, int k) {
        RawCodes<T> r{0u, zero, zero};
        const int n = n0 + row;
        if (row < BN && n < N && k < kend) {
            r.codes = qa.w[(int64_t)n * (K >> word_shift) + (k >> word_shift)] >> ((k & ((1 << word_shift) - 1)) * qa.bits);
            const int64_t e = (int64_t)n * (K >> group_shift) + (k >> group_shift);
            r.scale = static_cast<const T*>(qa.scales)[e];
            r.bias = static_cast<const T*>(qa.biases)[e];
        }
        return r;
    };
    auto fetch = [&](int s) {
        const int k = s < nslab ? kbeg + s * SLAB + seg * 4 : kend;
#pragma unroll
        for (int f = 0; f < FA; ++f) fa[f] = piece(pr + f * STEP, BM, m0, M, a, a_sm, a_sk, k);
#pragma unroll
        for (int f = 0; f < FB; ++f) {
            if constexpr (QUANT) fb[f] = codes(pr + f * STEP, k);
            else fb[f] = piece(pr + f * STEP, BN, n0, N, b, b_sn, b_sk, k);
        }
    };
    auto store = [&](int buf) {
        auto put = [&](float* d, int pitch, const float4& v) { d[0] = v.x; d[pitch] = v.y; d[2 * pitch] = v.z; d[3 * pitch] = v.w; };
#pragma unroll
        for (int f = 0; f < FA; ++f)
            if (BM % STEP == 0 || pr + f * STEP < BM) put(&As[buf][seg * 4][(pr + f * STEP) ^ (seg << SWZ)], PA, widen(fa[f]));
#pragma unroll
        for (int f = 0; f < FB; ++f)
            if (BN % STEP == 0 || pr + f * STEP < BN) {
                float4 w;
                if constexpr (QUANT) w = widen(fb[f], qa.bits);
                else w = widen(fb[f]);
                put(&Bs[buf][seg * 4][(pr + f * STEP) ^ (seg << SWZ)], PB, w);
            }
    };

    // Accumulators as pairs of columns (two independent fma per instruction; a's value rides in both halves).
    constexpr int TP = TN / 2;
    uint64_t acc[TM][TP], total[SPLIT ? 1 : TM][SPLIT ? 1 : TP];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TP; ++j) {
            acc[i][j] = 0;
            if constexpr (!SPLIT) total[i][j] = 0;
        }

    fetch(0);
    for (int s = 0; s < nslab; ++s) {
        const int buf = s & 1;
        store(buf);
        __syncthreads();                                            // slab s visible; slab s - 1 was read before the barrier of s
        fetch(s + 1);
#pragma unroll
        for (int k = 0; k < SLAB; ++k) {
            const int sw = (k >> 2) << SWZ;
            float av[TM], bv[TN];
            ld_tile<TM>(&As[buf][k][0], mg, MG, sw, av);
            ld_tile<TN>(&Bs[buf][k][0], nl, NL, sw, bv);
            uint64_t b2[TP];
#pragma unroll
            for (int j = 0; j < TP; ++j) b2[j] = ptx::pack2(bv[2 * j], bv[2 * j + 1]);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const uint64_t a2 = ptx::pack2(av[i], av[i]);
#pragma unroll
                for (int j = 0; j < TP; ++j) acc[i][j] = ptx::fma2_rn(a2, b2[j], acc[i][j]);
            }
        }
        if constexpr (!SPLIT) {
            if ((s + 1) % (GROUP_K / SLAB) == 0 || s + 1 == nslab) {   // a K group is complete
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TP; ++j) { total[i][j] = ptx::add2_rn(total[i][j], acc[i][j]); acc[i][j] = 0; }
            }
        }
    }

#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + place<TM>(mg, i, MG);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + place<TN>(nl, j, NL);
            if (n >= N) continue;
            float lo, hi;
            ptx::unpack2(SPLIT ? acc[i][j / 2] : total[SPLIT ? 0 : i][SPLIT ? 0 : j / 2], lo, hi);
            const float r = (j & 1) ? hi : lo;
            if constexpr (SPLIT) static_cast<float*>(outp)[((int64_t)g0 * M + m) * N + n] = r;
            else static_cast<T*>(outp)[(int64_t)m * N + n] = round_out<T>(r, static_cast<const T*>(qa.out_bias), n);
        }
    }
}

// Up to eight rows of fp32: a stream of the weight. Thread nl owns column n0 + nl of all TM rows; the stages keep k
// contiguous, as in memory, and are filled by 16-byte cp.async two stages ahead (4096 x 4096 at M = 1: 15.3 us with the
// combine launch, of which 10.4 us are the weight's bytes; 22.5 us with the register-fetched stages of the tile kernel).
constexpr int STREAM_N = 128, STREAM_SLAB = 32, STREAM_PITCH = STREAM_SLAB + 4, STREAM_STAGES = 3;
template <int TM, bool SPLIT>
__global__ void __launch_bounds__(STREAM_N) simt_stream_kernel(const float* __restrict__ a, const float* __restrict__ b, QuantArgs qa,
                                                               float* __restrict__ out, int M, int N, int K, int64_t a_sm, int64_t b_sn) {
    ptx::grid_dep_wait();     // everything before this kernel has completed and is visible
    extern __shared__ __align__(16) float stream_smem[];
    constexpr int ROWS = TM + STREAM_N, SEGS = STREAM_SLAB / 4;
    const int tid = threadIdx.x, n0 = blockIdx.x * STREAM_N;
    const int g0 = SPLIT ? (int)blockIdx.z : 0;
    const int kbeg = g0 * GROUP_K, kend = SPLIT ? min(K, kbeg + GROUP_K) : K;
    const int nslab = (kend - kbeg + STREAM_SLAB - 1) / STREAM_SLAB;
    auto fill = [&](int s) {
        if (s < nslab) {
            const uint32_t d0 = ptx::smem_u32(stream_smem + (s % STREAM_STAGES) * ROWS * STREAM_PITCH);
            for (int e = tid; e < ROWS * SEGS; e += STREAM_N) {
                const int r = e / SEGS, k = kbeg + s * STREAM_SLAB + (e % SEGS) * 4;
                const bool isa = r < TM;
                const int i = isa ? r : n0 + r - TM;
                const bool ok = i < (isa ? M : N) && k < kend;
                const float* src = ok ? (isa ? a + (int64_t)i * a_sm : b + (int64_t)i * b_sn) + k : a;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d0 + (r * STREAM_PITCH + (e % SEGS) * 4) * 4), "l"(src), "r"(ok ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[TM], total[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) { acc[i] = 0.0f; total[i] = 0.0f; }
    for (int s = 0; s < STREAM_STAGES - 1; ++s) fill(s);
    for (int s = 0; s < nslab; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STREAM_STAGES - 2) : "memory");
        __syncthreads();                                            // slab s visible; everyone is done with slab s - 1
        fill(s + STREAM_STAGES - 1);
        const float* const st = stream_smem + (s % STREAM_STAGES) * ROWS * STREAM_PITCH;
#pragma unroll 2
        for (int k4 = 0; k4 < STREAM_SLAB; k4 += 4) {
            float bv[4];
            ld_floats<4>(st + (TM + tid) * STREAM_PITCH + k4, bv);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                float av[4];
                ld_floats<4>(st + i * STREAM_PITCH + k4, av);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) acc[i] = fma_rn(av[kk], bv[kk], acc[i]);
            }
        }
        if (!SPLIT && ((s + 1) % (GROUP_K / STREAM_SLAB) == 0 || s + 1 == nslab)) {      // a K group is complete
#pragma unroll
            for (int i = 0; i < TM; ++i) { total[i] = add_rn(total[i], acc[i]); acc[i] = 0.0f; }
        }
    }
    const int n = n0 + tid;
    if (n >= N) return;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        if (i >= M) break;
        if (SPLIT) out[((int64_t)g0 * M + i) * N + n] = acc[i];
        else out[(int64_t)i * N + n] = round_out<float>(total[i], static_cast<const float*>(qa.out_bias), n);
    }
}

// out[idx] = T(((0 + p_0[idx]) + p_1[idx]) + ...): the fold of the split path
// (reference: bi_matmul_combine, mlx_batch_invariant/kernels/matmul.py:226-234).
// PUSH: the output is this rank's column slice of a gathered activation: out[m, n] goes to column rank * N + n of
// every rank's [M, world * N] destination, and the launch ends with the gather's handshake (peer_push.cuh) -- the
// fold and the all-gather that follows it are one kernel, the local slice never exists in memory.
template <typename T, int VEC, bool PUSH>
__global__ void __launch_bounds__(256) combine_kernel(const float* __restrict__ part, T* __restrict__ out, int G,
                                                      int64_t MN, const T* __restrict__ bias, int64_t N, PushSink sink) {
    ptx::grid_dep_wait_and_launch();
    const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * VEC;
    if (i0 < MN) {
        float total[VEC];
#pragma unroll
        for (int v = 0; v < VEC; ++v) total[v] = 0.0f;
        for (int g = 0; g < G; ++g) {
            const float* p = part + (int64_t)g * MN + i0;
            if (VEC == 4) {
                const float4 x = *reinterpret_cast<const float4*>(p);
                total[0] = add_rn(total[0], x.x); total[1 % VEC] = add_rn(total[1 % VEC], x.y);
                total[2 % VEC] = add_rn(total[2 % VEC], x.z); total[3 % VEC] = add_rn(total[3 % VEC], x.w);
            } else {
                total[0] = add_rn(total[0], p[0]);
            }
        }
        if (PUSH) {
            // VEC consecutive outputs stay inside one row (N % VEC == 0 is checked by the launcher)
            const int64_t m = i0 / N, n = i0 - m * N;
            const int64_t o = m * N * sink.world + (int64_t)sink.rank * N + n;
            T vals[VEC];
#pragma unroll
            for (int v = 0; v < VEC; ++v) vals[v] = round_out<T>(total[v], bias, bias ? n + v : 0);
            for (int r = 0; r < sink.world; ++r) {
                T* d = static_cast<T*>(sink.dst.p[r]) + o;
#pragma unroll
                for (int v = 0; v < VEC; ++v) d[v] = vals[v];
            }
        } else {
#pragma unroll
            for (int v = 0; v < VEC; ++v) out[i0 + v] = round_out<T>(total[v], bias, bias ? (i0 + v) % N : 0);
        }
    }
    if (PUSH) push_handshake(sink);
}

template <typename T>
int combine_t(const float* part, void* out, int G, int64_t MN, cudaStream_t st, const void* bias_v, int64_t N,
              const PushSink* sink = nullptr) {
    const T* bias = static_cast<const T*>(bias_v);
    const bool vec_ok = MN % 4 == 0 && aligned(part, 16) && (!sink || N % 4 == 0);
    const PushSink none{};
#define BI_COMBINE(VEC, THREADS_)                                                                                        \
    do {                                                                                                                 \
        const unsigned blocks_ = (unsigned)(((THREADS_) + 255) / 256);                                                  \
        if (sink) launch_overlapped_unless(true, combine_kernel<T, VEC, true>, dim3(blocks_), dim3(256), 0, st, part, (T*)nullptr, G, MN, bias, N, *sink); \
        else launch_overlapped(combine_kernel<T, VEC, false>, dim3(blocks_), dim3(256), 0, st, part, static_cast<T*>(out), G, MN, bias, N, none); \
    } while (0)
    if (vec_ok && MN >= (1 << 20)) {
        BI_COMBINE(4, MN / 4);
    } else {
        // few outputs: one per thread, so that enough loads are in flight to cover the L2 latency
        // (4096x14336 at M = 16: 31.1 -> 28.3 us for matmul + combine)
        BI_COMBINE(1, MN);
    }
#undef BI_COMBINE
    return check_launch("matmul combine");
}

// The fold of the split path for a decoder's qkv projection, with bi_rope_append's work done on the folded values
// before they ever reach memory. One thread per element, as in combine_kernel (enough loads in flight to cover the
// L2 latency): it folds its column, rounds to T (the bits combine_kernel would have stored), leaves the value in shared
// memory for the thread that holds the other half of the rotation pair (a block of 256 consecutive elements covers
// whole heads: 256 % D == 0), and then repeats rope_append_kernel's arithmetic: q and k heads rotated, v heads
// copied, positions outside the cache skipped with a status code.
template <typename T>
__global__ void __launch_bounds__(256) combine_rope_kernel(const float* __restrict__ part, int G, int64_t MN, RopeSink r) {
    ptx::grid_dep_launch();       // at once: the attention behind it is one CTA an SM (decoder step of 4 sequences 3504 -> 3482 us)
    ptx::grid_dep_wait();
    __shared__ T rounded[256];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = i < MN;
    float total = 0.0f;
    if (live)
        for (int g = 0; g < G; ++g) total = add_rn(total, part[(int64_t)g * MN + i]);
    const T x = Cvt<T>::down(total);
    rounded[threadIdx.x] = x;
    __syncthreads();
    if (!live) return;
    const int H = r.Hq + 2 * r.Hkv, half = r.D / 2;
    const int d = (int)(i % r.D);
    const int h = (int)((i / r.D) % H);
    const int64_t bt = i / ((int64_t)r.D * H);
    const int t = (int)(bt % r.T);
    const int b = (int)(bt / r.T);
    const int64_t pos = r.pos0[0] + t;
    if (pos < 0 || pos >= r.capacity) {
        if (r.status) atomicCAS(r.status, 0, (int)(0x30000 | (int)(pos & 0xffff)));
        return;
    }
    if (h >= r.Hq + r.Hkv) {                               // v: stored as is
        static_cast<T*>(r.v_cache)[(int64_t)b * r.c_sb + (int64_t)(h - r.Hq - r.Hkv) * r.c_sh + pos * r.c_sl + d] = x;
        return;
    }
    const float other = Cvt<T>::up(rounded[d < half ? threadIdx.x + half : threadIdx.x - half]);
    const float rot = d < half ? -other : other;
    const T o = Cvt<T>::down(add_rn(mul_rn(Cvt<T>::up(x), r.cos_table[pos * r.D + d]), mul_rn(rot, r.sin_table[pos * r.D + d])));
    if (h < r.Hq) static_cast<T*>(r.q_out)[(((int64_t)b * r.Hq + h) * r.T + t) * r.D + d] = o;
    else          static_cast<T*>(r.k_cache)[(int64_t)b * r.c_sb + (int64_t)(h - r.Hq) * r.c_sh + pos * r.c_sl + d] = o;
}

// Tiles of a launch: TM x TN outputs per thread, MG x NL threads, all 128 columns wide. `cost`: time per fma relative to
// the last one (4096 x 4096 at M = 128, split: 134 / 105 / 95 us): a smaller thread tile reads shared memory more often,
// but wastes fewer rows of a small batch. Taller thread tiles (12 and 16 rows) and 256-thread CTAs measured no faster.
struct SimtTile { int tm, tn, mg, nl; double cost; };
constexpr SimtTile SIMT_TILES[] = {{8, 4, 2, 32, 1.41}, {8, 8, 4, 16, 1.10}, {8, 8, 8, 16, 1.0}};
constexpr int SIMT_NTILES = sizeof(SIMT_TILES) / sizeof(SIMT_TILES[0]);
constexpr int STREAM_M_MAX = 8;

int simt_tile(int64_t M) {
    int best = 0;
    double least = 0;
    for (int i = 0; i < SIMT_NTILES; ++i) {
        const int64_t bm = SIMT_TILES[i].tm * SIMT_TILES[i].mg;
        const double c = SIMT_TILES[i].cost * (double)((M + bm - 1) / bm * bm);
        if (i == 0 || c < least) { best = i; least = c; }
    }
    return best;
}

struct SimtArgs {
    const void *a, *b;
    QuantArgs qa;
    void* dst;
    int64_t M, N, K, a_sm, a_sk, b_sk, b_sn;
    bool split;
    cudaStream_t st;
};

// How a grid lies on the SMs decides its time where it is less than a wave (spread_smem). Up to a CTA an SM it is held to that;
// of two CTAs an SM up the fullest ones were slower than an idle machine's spread, so these are launched plainly, and grids of
// a wave up again beside the kernel in front; so are packed weights, whose codes come through the L1 that the hold takes from (64 x
// 896 -> 4864, 4 bits 70.0 us, held 71.6). us a call in chains, let in without regard / plainly / so: fp32 128 x 2048 -> 2048
// 52.5 / 31 / 30.4, 9 x 2048 -> 2048 19.5 / 14.7 / 13.8, 64 x 2048 -> 2048 behind a 16-bit linear 60 / 26 / 23.8; eagerly 100 x 4096 ->
// 4096 93 / 97 / 93.
template <auto KERNEL, bool HOLD, typename... Args>
void launch_simt(dim3 grid, int threads, size_t smem, cudaStream_t st, Args... args) {
    const int64_t ctas = (int64_t)grid.x * grid.y * grid.z;
    bool overlapped = pdl_enabled();
    if (HOLD && overlapped && ctas <= sm_count()) smem = spread_smem<KERNEL>(ctas, smem);
    else if (overlapped) overlapped = ctas >= (int64_t)resident_ctas<KERNEL>(threads, smem) * sm_count();
    launch_kernel(overlapped, KERNEL, grid, dim3(threads), smem, st, args...);
}

template <int TM, bool SPLIT>
int simt_columns(dim3 grid, size_t smem, const SimtArgs& p) {
    constexpr auto kern = simt_stream_kernel<TM, SPLIT>;
    if (!opt_in_smem<kern>()) return fail_cuda("matmul (cuda-core path) smem attr", cudaErrorInvalidValue);
    launch_simt<kern, true>(grid, STREAM_N, smem, p.st, static_cast<const float*>(p.a), static_cast<const float*>(p.b), p.qa, static_cast<float*>(p.dst), (int)p.M,
                      (int)p.N, (int)p.K, p.a_sm, p.b_sn);
    return check_launch("matmul (cuda-core path)");
}

template <int TM>
int simt_stream(const SimtArgs& p) {
    const int64_t G = (p.K + GROUP_K - 1) / GROUP_K;
    if (p.split && G > 65535) return fail(BI_ERR_UNSUPPORTED, "matmul (cuda-core path): K=%lld too large", (long long)p.K);
    dim3 grid((unsigned)((p.N + STREAM_N - 1) / STREAM_N), 1, p.split ? (unsigned)G : 1u);
    constexpr size_t smem = (size_t)STREAM_STAGES * (TM + STREAM_N) * STREAM_PITCH * sizeof(float);
    return p.split ? simt_columns<TM, true>(grid, smem, p) : simt_columns<TM, false>(grid, smem, p);
}

template <typename T, int TM, int TN, int MG, int NL, bool SPLIT, bool QUANT, bool VEC>
void simt_tiles(dim3 grid, const SimtArgs& p) {
    launch_simt<simt_matmul_kernel<T, TM, TN, MG, NL, SPLIT, QUANT, VEC>, !QUANT>(grid, MG * NL, 0, p.st, static_cast<const T*>(p.a), static_cast<const T*>(p.b),
                                                                                  p.qa, p.dst, (int)p.M, (int)p.N, (int)p.K, p.a_sm, p.a_sk, p.b_sk, p.b_sn);
}

template <typename T, bool QUANT, bool VEC, int I>
int simt_launch(int tile, const SimtArgs& p) {
    if constexpr (I < SIMT_NTILES) {
        if (tile != I) return simt_launch<T, QUANT, VEC, I + 1>(tile, p);
        constexpr SimtTile t = SIMT_TILES[I];
        constexpr int bm = t.tm * t.mg, bn = t.tn * t.nl;
        const int64_t G = (p.K + GROUP_K - 1) / GROUP_K, gy = (p.M + bm - 1) / bm;
        if (gy > 65535 || (p.split && G > 65535)) return fail(BI_ERR_UNSUPPORTED, "matmul (cuda-core path): M=%lld K=%lld too large", (long long)p.M, (long long)p.K);
        dim3 grid((unsigned)((p.N + bn - 1) / bn), (unsigned)gy, p.split ? (unsigned)G : 1u);
        if (p.split) simt_tiles<T, t.tm, t.tn, t.mg, t.nl, true, QUANT, VEC>(grid, p);
        else simt_tiles<T, t.tm, t.tn, t.mg, t.nl, false, QUANT, VEC>(grid, p);
        return check_launch("matmul (cuda-core path)");
    }
    return fail(BI_ERR_UNSUPPORTED, "matmul (cuda-core path): no tile %d", tile);
}

template <typename T, bool QUANT>
int simt_t(const void* a, const void* b, const QuantArgs& qa, void* out, float* part, int64_t M, int64_t N,
           int64_t K, int64_t a_sm, int64_t a_sk, int64_t b_sk, int64_t b_sn, bool split, cudaStream_t st) {
    const SimtArgs p{a, b, qa, split ? static_cast<void*>(part) : out, M, N, K, a_sm, a_sk, b_sk, b_sn, split, st};
    int rc;
    if constexpr (sizeof(T) == 4 && !QUANT) {
        const bool vec = a_sk == 1 && b_sk == 1 && K % 4 == 0 && (M == 1 || a_sm % 4 == 0) && (N == 1 || b_sn % 4 == 0) && aligned(a, 16) && aligned(b, 16);
        if (vec && M <= STREAM_M_MAX) rc = M <= 1 ? simt_stream<1>(p) : (M <= 2 ? simt_stream<2>(p) : (M <= 4 ? simt_stream<4>(p) : simt_stream<8>(p)));
        else rc = vec ? simt_launch<T, QUANT, true, 0>(simt_tile(M), p) : simt_launch<T, QUANT, false, 0>(simt_tile(M), p);
    } else {
        rc = simt_launch<T, QUANT, false, 0>(simt_tile(M), p);
    }
    if (rc || !split) return rc;
    return combine_t<T>(part, out, (int)((K + GROUP_K - 1) / GROUP_K), M * N, st, qa.out_bias, N);
}

}  // namespace

double simt_waves(int64_t M, int64_t N) {
    const SimtTile& t = SIMT_TILES[simt_tile(M)];
    const int64_t bm = t.tm * t.mg, bn = t.tn * t.nl, resident = sm_count() * (256 / (t.mg * t.nl));   // launch bounds: 256 threads an SM
    return (double)((M + bm - 1) / bm * ((N + bn - 1) / bn)) / (double)resident;
}

int launch_combine_rope(const float* part, int G, int64_t MN, int dtype, cudaStream_t st, const RopeSink& rope) {
    if (rope.D > 256 || 256 % rope.D != 0) return fail(BI_ERR_UNSUPPORTED, "matmul + rope: head_dim %d (must divide 256)", rope.D);
    const int64_t blocks = (MN + 255) / 256;
    if (blocks > 0x7fffffffLL) return fail(BI_ERR_UNSUPPORTED, "matmul + rope: too large");
    switch (dtype) {
        case BI_F32: launch_overlapped(combine_rope_kernel<float>, dim3((unsigned)blocks), dim3(256), 0, st, part, G, MN, rope); break;
        case BI_F16: launch_overlapped(combine_rope_kernel<__half>, dim3((unsigned)blocks), dim3(256), 0, st, part, G, MN, rope); break;
        default:     launch_overlapped(combine_rope_kernel<__nv_bfloat16>, dim3((unsigned)blocks), dim3(256), 0, st, part, G, MN, rope); break;
    }
    return check_launch("matmul fold + rope");
}

int launch_combine(const float* part, void* out, int G, int64_t MN, int dtype, cudaStream_t st, const void* bias, int64_t N,
                   const PushSink* sink) {
    switch (dtype) {
        case BI_F32: return combine_t<float>(part, out, G, MN, st, bias, N, sink);
        case BI_F16: return combine_t<__half>(part, out, G, MN, st, bias, N, sink);
        default:     return combine_t<__nv_bfloat16>(part, out, G, MN, st, bias, N, sink);
    }
}

int launch_simt_matmul(const void* a, const void* b, void* out, float* part, int64_t M, int64_t N, int64_t K,
                       int64_t a_sm, int64_t a_sk, int64_t b_sk, int64_t b_sn, int dtype, bool split,
                       cudaStream_t st, const void* bias) {
    QuantArgs qa{nullptr, nullptr, nullptr, 0, 0, bias};
    switch (dtype) {
        case BI_F32: return simt_t<float, false>(a, b, qa, out, part, M, N, K, a_sm, a_sk, b_sk, b_sn, split, st);
        case BI_F16: return simt_t<__half, false>(a, b, qa, out, part, M, N, K, a_sm, a_sk, b_sk, b_sn, split, st);
        default:     return simt_t<__nv_bfloat16, false>(a, b, qa, out, part, M, N, K, a_sm, a_sk, b_sk, b_sn, split, st);
    }
}

int launch_simt_qmm(const void* x, const uint32_t* w, const void* scales, const void* biases, void* out, float* part,
                    int64_t M, int64_t N, int64_t K, int64_t x_sm, int gs, int bits, int dtype, bool split,
                    cudaStream_t st) {
    QuantArgs qa{w, scales, biases, bits, gs, nullptr};
    switch (dtype) {
        case BI_F32: return simt_t<float, true>(x, nullptr, qa, out, part, M, N, K, x_sm, 1, 1, K, split, st);
        case BI_F16: return simt_t<__half, true>(x, nullptr, qa, out, part, M, N, K, x_sm, 1, 1, K, split, st);
        default:     return simt_t<__nv_bfloat16, true>(x, nullptr, qa, out, part, M, N, K, x_sm, 1, 1, K, split, st);
    }
}

}  // namespace bi
