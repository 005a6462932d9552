// Shared by the decode and prefill attention kernels: the K/V layout, the split merge and the conversion of packed
// 16-bit pairs. The canonical arithmetic they are part of is stated at the top of attention.cu.
#pragma once
#include "bi_common.cuh"
#include "bi_ptx.cuh"

namespace bi {

// Fold one split's (m, l) into the running (M, L) and return the two factors
// the accumulators are folded with:  A_d = fma(A_d, c_old, acc_d * c_new).
__device__ __forceinline__ void merge_coeffs(float& M, float& L, float m, float l, float& c_old, float& c_new) {
    const float M_new = fmaxf(M, m);
    c_old = expf_canon(sub_rn(M, M_new));
    c_new = expf_canon(sub_rn(m, M_new));
    L = fma_rn(L, c_old, mul_rn(l, c_new));
    M = M_new;
}
__device__ __forceinline__ float merge_acc(float A, float c_old, float acc, float c_new) {
    return fma_rn(A, c_old, mul_rn(acc, c_new));
}

struct KvLayout {
    int64_t sb, sh, sl;  // element strides of k and v: batch (or page, when paged), kv head, key
    // Paged cache (table != nullptr): k and v are pools of pages [page, kv head, key in page, D]; keys
    // [i * page_size, (i + 1) * page_size) of sequence b live in page table[b * table_stride + i].
    const int32_t* table;
    int page_size, table_stride;
};

// two T values (consecutive dims) packed in one 32-bit word -> fp32, for 16-bit T
template <typename T> __device__ __forceinline__ float word_lo(uint32_t w);
template <typename T> __device__ __forceinline__ float word_hi(uint32_t w);
template <> __device__ __forceinline__ float word_lo<__nv_bfloat16>(uint32_t w) { return __uint_as_float(w << 16); }
template <> __device__ __forceinline__ float word_hi<__nv_bfloat16>(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }
template <> __device__ __forceinline__ float word_lo<__half>(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xFFFFu))); }
template <> __device__ __forceinline__ float word_hi<__half>(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }

// Validation common to the attention entry points (defined in attention.cu).
int check_attention(const char* op, const void* q, const void* k, const void* v, const void* out, int64_t B, int64_t Hq,
                    int64_t Hkv, int64_t Tq, int64_t L, int64_t D, const KvLayout& lay, int split, int dtype);

}  // namespace bi

// FN<T, D / 32>(...) for the call's dtype and head_dim (D is 32, 64, 128 or 256, dtype a bi_dtype: check_attention).
#define BI_DISPATCH_T_DL(FN, ...)                                                        \
    do {                                                                                 \
        const int dl_ = (int)(D / 32);                                                   \
        if (dtype == BI_F32) {                                                           \
            if (dl_ == 1) return FN<float, 1>(__VA_ARGS__);                              \
            if (dl_ == 2) return FN<float, 2>(__VA_ARGS__);                              \
            if (dl_ == 4) return FN<float, 4>(__VA_ARGS__);                              \
            return FN<float, 8>(__VA_ARGS__);                                            \
        } else if (dtype == BI_F16) {                                                    \
            if (dl_ == 1) return FN<__half, 1>(__VA_ARGS__);                             \
            if (dl_ == 2) return FN<__half, 2>(__VA_ARGS__);                             \
            if (dl_ == 4) return FN<__half, 4>(__VA_ARGS__);                             \
            return FN<__half, 8>(__VA_ARGS__);                                           \
        } else {                                                                         \
            if (dl_ == 1) return FN<__nv_bfloat16, 1>(__VA_ARGS__);                      \
            if (dl_ == 2) return FN<__nv_bfloat16, 2>(__VA_ARGS__);                      \
            if (dl_ == 4) return FN<__nv_bfloat16, 4>(__VA_ARGS__);                      \
            return FN<__nv_bfloat16, 8>(__VA_ARGS__);                                    \
        }                                                                                \
    } while (0)
