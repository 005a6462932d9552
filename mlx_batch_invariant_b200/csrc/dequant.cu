// Affine-quantized weight -> the 16-bit weight the tensor-core kernels multiply: w[n, k] = T(fma(float(code), scale, bias)).
//
// Used in front of the SM-pair matmul (matmul_pair.cu), whose batch is tall enough that unpacking a weight once per
// call is cheaper than unpacking it once per batch tile inside the matmul. Bound by memory: a thread turns eight codes
// (4 or 8 bytes) into one 16-byte store, four independent pieces at a time so that the loads overlap; a warp reads 128
// or 256 and writes 512 consecutive bytes.
#include "bi_common.cuh"
#include "bi_ptx.cuh"
#include "matmul_internal.cuh"
#include "matmul_tc_common.cuh"

namespace bi {
namespace {

constexpr int DQ_THREADS = 256, DQ_PIECES = 4;

template <typename T, int QBITS>
__global__ void __launch_bounds__(DQ_THREADS)
dequant_kernel(const uint32_t* __restrict__ codes, const T* __restrict__ scales, const T* __restrict__ biases, uint4* __restrict__ out,
               unsigned pieces, unsigned group_shift) {
    ptx::grid_dep_wait_and_launch();
    constexpr int WORDS = QBITS / 4;                          // 32-bit words behind eight codes
    const unsigned i0 = blockIdx.x * (DQ_THREADS * DQ_PIECES) + threadIdx.x;
    uint32_t w[DQ_PIECES][WORDS];
    float s[DQ_PIECES], b[DQ_PIECES];
#pragma unroll
    for (int j = 0; j < DQ_PIECES; ++j) {
        const unsigned i = i0 + j * DQ_THREADS;
        if (i < pieces) {
#pragma unroll
            for (int k = 0; k < WORDS; ++k) w[j][k] = __ldg(codes + (size_t)i * WORDS + k);
            // rows are whole numbers of quantization groups, so entry and piece are both flat indices
            s[j] = Cvt<T>::up(scales[i >> group_shift]);
            b[j] = Cvt<T>::up(biases[i >> group_shift]);
        }
    }
#pragma unroll
    for (int j = 0; j < DQ_PIECES; ++j) {
        const unsigned i = i0 + j * DQ_THREADS;
        if (i < pieces) out[i] = dequant8<T, QBITS>(w[j], ptx::pack2(s[j], s[j]), ptx::pack2(b[j], b[j]));
    }
}

template <typename T>
int launch_t(const TcQuant& q, void* out, unsigned pieces, cudaStream_t st) {
    const unsigned shift = q.gs == 32 ? 2 : (q.gs == 64 ? 3 : 4);            // pieces of eight per quantization group
    const dim3 grid((pieces + DQ_THREADS * DQ_PIECES - 1) / (DQ_THREADS * DQ_PIECES));
    const T *s = static_cast<const T*>(q.scales), *b = static_cast<const T*>(q.biases);
    launch_overlapped(q.bits == 4 ? dequant_kernel<T, 4> : dequant_kernel<T, 8>, grid, dim3(DQ_THREADS), 0, st, q.codes, s, b,
                      static_cast<uint4*>(out), pieces, shift);
    return check_launch("weight dequantization");
}

}  // namespace

int launch_dequant(const TcQuant& q, void* out, int64_t N, int64_t K, int dtype, cudaStream_t st) {
    const unsigned pieces = (unsigned)(N * K / 8);
    return dtype == BI_BF16 ? launch_t<__nv_bfloat16>(q, out, pieces, st) : launch_t<__half>(q, out, pieces, st);
}

}  // namespace bi
