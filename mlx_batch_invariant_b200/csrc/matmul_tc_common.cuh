// Pieces shared by the tensor-core matmul kernels: bounded barrier waits, the affine dequantizer and the
// tensor-map encoders.
#pragma once
#include <cuda.h>
#include "bi_common.cuh"
#include "bi_ptx.cuh"

namespace bi {
namespace {

constexpr int BLOCK_N = 128;  // weight rows of an operand tile (the MMA's M, per CTA)
constexpr int BLOCK_K = 64;   // elements per tile along K: 128 bytes = one swizzle row
constexpr int UMMA_K = 16;
constexpr uint64_t WAIT_LIMIT_NS = 2000000000ull;
#ifndef BI_EPI_SLEEP_NS
#define BI_EPI_SLEEP_NS 100
#endif

enum { ROLE_TMA = 1, ROLE_MMA = 2, ROLE_EPI = 3, ROLE_DEQ = 4 };

struct Ctl {
    int32_t* status;
    volatile int* abort_flag;  // shared memory
};

__device__ __forceinline__ void report(const Ctl& c, int role, int idx) {
    *c.abort_flag = 1;
    if (c.status) atomicCAS(c.status, 0, (int)(0x10000 | (role << 8) | (idx & 0xff)));
}

// Wait for barrier phase `parity` to complete. Gives up after WAIT_LIMIT_NS or when another
// role has raised the abort flag; returns false then. CLUSTER: the arrivals come from the other CTA of a pair.
template <bool CLUSTER = false>
__device__ __forceinline__ bool wait_bounded(uint32_t bar, uint32_t parity, const Ctl& c, int role, int idx) {
    if (role == ROLE_EPI || role == ROLE_DEQ) {
        // whole warps wait here; back off so they do not take issue slots from the TMA and MMA threads
        for (int i = 0; i < 2048; ++i) {
            if ((CLUSTER ? ptx::mbar_try_wait_cluster(bar, parity) : ptx::mbar_try_wait(bar, parity))) return true;
            __nanosleep(BI_EPI_SLEEP_NS);
        }
    } else {
        for (int i = 0; i < 4096; ++i)
            if ((CLUSTER ? ptx::mbar_try_wait_cluster(bar, parity) : ptx::mbar_try_wait(bar, parity))) return true;
    }
    const uint64_t t0 = ptx::globaltimer_ns();
    while (true) {
        for (int i = 0; i < 256; ++i)
            if ((CLUSTER ? ptx::mbar_try_wait_cluster(bar, parity) : ptx::mbar_try_wait(bar, parity))) return true;
        if (*c.abort_flag) return false;
        if (ptx::globaltimer_ns() - t0 > WAIT_LIMIT_NS) { report(c, role, idx); return false; }
    }
}

template <typename T> struct Pack2;
template <> struct Pack2<__nv_bfloat16> {
    static __device__ __forceinline__ uint32_t rn(float lo, float hi) {
        __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x = lo (low address)
        return *reinterpret_cast<uint32_t*>(&v);
    }
};
template <> struct Pack2<__half> {
    static __device__ __forceinline__ uint32_t rn(float lo, float hi) {
        __half2 v = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<uint32_t*>(&v);
    }
};

// The T value of a 16-bit word, widened.
template <typename T> __device__ __forceinline__ float word16_up(uint32_t w) {
    const unsigned short h = (unsigned short)w;
    T v;
    *reinterpret_cast<unsigned short*>(&v) = h;
    return Cvt<T>::up(v);
}

// Byte offset, inside a chunk's packed codes, of 16-byte piece `piece` of weight row `row` (pieces count along the
// row's bytes of the chunk). The codes lie as boxes of 128 rows x span bytes under the TMA swizzle of that span:
// the piece index inside a span is XORed with bits [7, 7 + log2(span / 16)) of the byte address.
__device__ __forceinline__ uint32_t raw_piece_offset(int row, int piece, int span) {
    const int per = span >> 4;                         // pieces per row of one box: 2, 4 or 8
    const int box = piece / per, pb = piece - box * per;
    const int sw = ((row * span) >> 7) & (per - 1);
    return (uint32_t)(box * (BLOCK_N * span) + row * span + ((pb ^ sw) << 4));
}

// Eight consecutive codes -> eight T values, one 16-byte swizzle chunk.
//   value = T(fma(float(code), scale, bias))   fp32 fma, one rounding.
// float(code) is formed exactly without an integer->float conversion: a byte permute drops the code
// into the low mantissa byte of 2^23 (0x4B0000cc = 8388608 + cc) and 2^23 is subtracted, which is
// exact. The subtract and the fma run as packed f32x2 instructions: two independent IEEE
// round-to-nearest operations each, same bits as the scalar forms.
template <typename T, int QBITS>
__device__ __forceinline__ uint4 dequant8(const uint32_t* words, uint64_t s2, uint64_t b2) {
    const uint64_t neg_magic = ptx::pack2(-8388608.0f, -8388608.0f);
    uint32_t src_even[4], src_odd[4];  // register + byte index holding codes 2i and 2i+1
    uint32_t o[4];
    if (QBITS == 4) {
        const uint32_t lo = words[0] & 0x0F0F0F0Fu;          // bytes: codes 0, 2, 4, 6
        const uint32_t hi = (words[0] >> 4) & 0x0F0F0F0Fu;   // bytes: codes 1, 3, 5, 7
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            src_even[i] = __byte_perm(lo, 0x4B000000u, 0x7540u + i);
            src_odd[i] = __byte_perm(hi, 0x4B000000u, 0x7540u + i);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            src_even[i] = __byte_perm(words[i >> 1], 0x4B000000u, 0x7540u + 2 * (i & 1));
            src_odd[i] = __byte_perm(words[i >> 1], 0x4B000000u, 0x7540u + 2 * (i & 1) + 1);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint64_t v = ptx::pack2(__uint_as_float(src_even[i]), __uint_as_float(src_odd[i]));
        v = ptx::add2_rn(v, neg_magic);
        v = ptx::fma2_rn(v, s2, b2);
        float x, y;
        ptx::unpack2(v, x, y);
        o[i] = Pack2<T>::rn(x, y);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// The same values from packed 16-bit arithmetic, where that is exact. fma.rn.T rounds code * scale + bias once; the canonical
// sequence rounds it to fp32 and then to T. The two agree whenever the fp32 fma is exact, that is when all bits of the
// product (code bits + the scale's) and of the bias lie within 24 binary places of each other -- a bound on the difference
// of the two exponents, which every group of an ordinary weight keeps (the bias is a few steps of the scale) -- or when the
// bias or the scale is zero. Groups outside it and scales that are subnormal or too large to be shifted as below (infinities
// and NaN among them) take dequant8. A bias that is infinite or NaN passes beside a large scale: the products are finite, so
// either form gives that bias back.
// Why: eight 4-bit codes take 15 instructions (a shift, two masks, four permutes, four multiplies, four fmas) instead of 23,
// none of them a conversion and half of them on the FP32 pipe instead of the integer one. Packed weights of group 64 that are
// not in L2, without -> with, 1 / 64 rows: 4 bits, 4096 -> 14336 25.3 -> 23.6 / 39.0 -> 35.5 us, 14336 -> 4096 27.8 -> 25.1 /
// 51.3 -> 47.9 us; 8 bits 26.4 -> 25.2 / 38.8 -> 36.2, 27.7 -> 25.9 / 53.3 -> 51.1 us. The test itself counts: as scalar
// code for each half it cost 0.5 to 1 us of that. Where every warp meets a group that takes dequant8 a call is 3 - 8 % slower
// than without all this at 1 and 16 rows (4096 -> 14336, 4 bits 25.7 -> 27.5 us, 8 bits 26.4 -> 28.7 us), and not at 64.
// The tile body (more than 64 rows) keeps dequant8: its long layers were up to 8 % slower with this (4096 -> 28672 at 100
// rows: 101 against 110 us), its short ones 6 - 12 % faster.
template <typename T> struct Half2;
template <> struct Half2<__nv_bfloat16> {
    static constexpr uint32_t UP = 0x7F007F00u, DOWN = 0x42804280u;    // 2^127 and 2^6: an integer as a bit pattern is itself times 2^-133
    static constexpr int MANT = 7, EXP = 255, EXP_LO = 1, EXP_HI = 240;
    static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
    static __device__ __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
};
template <> struct Half2<__half> {
    static constexpr uint32_t UP = 0x78007800u, DOWN = 0x60006000u;    // 2^15 and 2^9: ... times 2^-24
    static constexpr int MANT = 10, EXP = 31, EXP_LO = 1, EXP_HI = 20;
    static __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) { uint32_t r; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b)); return r; }
    static __device__ __forceinline__ uint32_t fma(uint32_t a, uint32_t b, uint32_t c) { uint32_t r; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c)); return r; }
};
// Two scales and two biases as the 16-bit words they are in memory. With scale exponent es and bias exponent eb (M = stored
// mantissa bits, Q = code bits) the sum's bits lie between 2^(min(es, eb) - M) and 2^(max(es + Q + 1, eb + 1) + 1). Bit 14 of
// each half says that a difference is not negative. ZEROS: a bias or scale of zero leaves nothing to round, wherever the
// other lies.
template <typename T, int QBITS, bool ZEROS>
__device__ __forceinline__ bool dequant_exact(uint32_t scales, uint32_t biases) {
    using H = Half2<T>;
    constexpr uint32_t BOTH = 0x00010001u, TOP = 0x4000u * BOTH, EXPS = H::EXP * BOTH;
    constexpr uint32_t BELOW = (24 - H::MANT - QBITS - 2) * BOTH, ABOVE = (24 - H::MANT - 2) * BOTH;     // how far the bias may lie
    const uint32_t es = (scales >> H::MANT) & EXPS, eb = (biases >> H::MANT) & EXPS;
    const uint32_t in_range = (es + (TOP - H::EXP_LO * BOTH)) & ((TOP + H::EXP_HI * BOTH) - es);
    uint32_t near = (eb - es + (TOP + BELOW)) & (es - eb + (TOP + ABOVE));
    if (!ZEROS) return (in_range & near & TOP) == TOP;
    const uint32_t magnitudes = 0x7fff7fffu;
    const uint32_t bias0 = ~((biases & magnitudes) + magnitudes) >> 1, scale0 = ~((scales & magnitudes) + magnitudes) >> 1;
    return (((in_range & (near | bias0)) | scale0) & TOP) == TOP;
}
template <typename T> __device__ __forceinline__ uint32_t dequant_scale(uint32_t scale2) { return Half2<T>::mul(scale2, Half2<T>::DOWN); }
template <int SEL> __device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b) {   // a selector nibble with bit 3 set gives the byte's sign, eight times
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "n"(SEL));
    return r;
}
// scale2: dequant_scale() of the scale in both halves; bias2: the bias in both halves. Codes are turned into T exactly: the
// bit pattern of a small integer is a subnormal number (8-bit codes reach the first normal binade, which continues it).
template <typename T, int QBITS>
__device__ __forceinline__ uint4 dequant8_packed(const uint32_t* words, uint32_t scale2, uint32_t bias2) {
    using H = Half2<T>;
    uint32_t c[4];
    if (QBITS == 4) {
        const uint32_t lo = words[0] & 0x0F0F0F0Fu, hi = (words[0] >> 4) & 0x0F0F0F0Fu;      // codes 0, 2, 4, 6 and 1, 3, 5, 7; sign bits zero
        c[0] = prmt<0xC480>(lo, hi); c[1] = prmt<0xD591>(lo, hi); c[2] = prmt<0xE6A2>(lo, hi); c[3] = prmt<0xF7B3>(lo, hi);
    } else {
        c[0] = prmt<0x4140>(words[0], 0u); c[1] = prmt<0x4342>(words[0], 0u);
        c[2] = prmt<0x4140>(words[1], 0u); c[3] = prmt<0x4342>(words[1], 0u);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] = H::fma(H::mul(c[i], H::UP), scale2, bias2);
    return make_uint4(c[0], c[1], c[2], c[3]);
}

// ---- host side -----------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

[[maybe_unused]] EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// 2-D row-major tensor [rows, cols] with `ld` elements between rows; box = [box_rows, box_cols].
[[maybe_unused]] int make_map(CUtensorMap* m, CUtensorMapDataType dt, size_t esize, const void* base, uint64_t cols, uint64_t rows,
             uint64_t ld, uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle sw) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(BI_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t gdim[2] = {cols, rows};
    cuuint64_t gstr[1] = {ld * esize};
    cuuint32_t box[2] = {box_cols, box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(m, dt, 2, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BI_ERR_CUDA, "cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
    return BI_OK;
}

// The same tensor seen as [K/64 blocks][rows][inner elements] (needs K % 64 == 0; inner = the elements that hold
// 64 values of K: 64 for 16-bit data, 8 or 16 words for packed codes): a box of `depth` blocks lands as `depth`
// consecutive K-step tiles of box_rows x (inner * esize) bytes.
[[maybe_unused]] int make_map3(CUtensorMap* m, CUtensorMapDataType dt, size_t esize, const void* base, uint64_t kblocks, uint64_t rows,
              uint64_t ld, uint32_t box_rows, uint32_t depth, uint32_t inner = BLOCK_K,
              CUtensorMapSwizzle sw = CU_TENSOR_MAP_SWIZZLE_128B) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(BI_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t gdim[3] = {(cuuint64_t)inner, rows, kblocks};
    cuuint64_t gstr[2] = {ld * esize, (cuuint64_t)inner * esize};
    cuuint32_t box[3] = {(cuuint32_t)inner, box_rows, depth};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(m, dt, 3, const_cast<void*>(base), gdim, gstr, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(BI_ERR_CUDA, "cuTensorMapEncodeTiled (3-D) failed with CUresult %d", (int)r);
    return BI_OK;
}

}  // namespace
}  // namespace bi
