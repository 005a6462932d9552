// Tensor-core matmul on pairs of SMs, for batches that fill tall tiles (prefill):   out[M, N] = x[M, K] @ W[N, K]^T
//
// Two CTAs of a cluster share one tile of 256 weight rows x up to 256 batch rows through
// tcgen05.mma.cta_group::2: each holds 128 weight rows and half of the batch rows in its shared memory, the
// instruction reads both halves of both, and CTA r's tensor memory receives weight rows 128 r ... 128 r + 127 for
// all batch rows. An SM therefore fetches 128 + bm/2 rows per K step for 128 x bm outputs.
//
// The arithmetic is that of matmul_tc.cu: sixteen K = 16 steps per 256-wide group in ascending k into a fresh fp32
// accumulator, the group partials added in ascending g by plain fp32 adds from an exact 0, one rounding. The group
// totals live in the registers of eight epilogue warps (each thread one weight row, half of the batch tile), while
// the MMAs of the next group fill the other of two accumulators of 256 tensor-memory columns.
//
// The finished tile leaves through shared memory: pieces of 16 batch rows x 128 weight rows in a ring of four for each half,
// one TMA store each. Stored from the registers, 64 bytes a warp instruction, a tile kept the epilogue warps for 9 us, in
// which the MMAs stood still after two groups: 1900 x 4096 -> 14336 at bm = 256 248 us so, 212 us staged. Outputs whose rows
// are no whole 16-byte units are still stored that way.
//
// What bounds it: a K step of 64 takes 0.2 us or 0.12 us + 0.9 ns per batch row of the tile, whichever is more (bm = 64 / 128 /
// 256: 0.20 / 0.22 / 0.35, of which the MMAs alone 0.07 / 0.14 / 0.27): at small tiles the chain commit -> drain -> arrival ->
// next group of the two accumulators, at 256 rows the tensor pipe under the power cap; 8 - 10 us a launch. One SM per tile
// (128 x 128, matmul_tc.cu) takes 0.46 us a step for a quarter of the pair's outputs. fp16 1900 x 4096 -> 14336: 241 -> 170 us at
// bm = 224 (1313 TFLOP/s), bf16 1024 x 4096 -> 4096 60 -> 40 us, 1024 x 14336 -> 4096 179 -> 112 us at bm = 128.
//
// Every wait is bounded; a wait that runs out records a code in the status word, raises the CTA's abort flag, and the
// pair meets at the cluster barrier (which every warp reaches) before tensor memory is freed.
#include <type_traits>
#include "bi_common.cuh"
#include "bi_ptx.cuh"
#include "matmul_internal.cuh"
#include "matmul_tc_common.cuh"

namespace bi {
namespace {

constexpr int PAIR_SMEM_LIMIT = 227 * 1024;
constexpr int PAIR_MAX_SLOTS = 8;
constexpr int PAIR_BAR_BYTES = 512;
constexpr int PAIR_TMEM_COLS = 512;
constexpr int PAIR_ACC_STRIDE = 256;           // columns between the two accumulators
constexpr int W_BYTES = BLOCK_N * BLOCK_K * 2; // one weight operand tile
constexpr int EPI0 = 4;                        // warps 0-3 issue (setmaxnreg works on whole warpgroups), 4-11 fold
constexpr int PAIR_THREADS = 32 * (EPI0 + 8);
constexpr int PAIR_MAX_BM = 256;
// Output staging: pieces of 16 batch rows x 128 weight rows, four for each half of the batch tile
constexpr int OUT_ROWS = 16, OUT_BUFS = 4;
constexpr int OUT_PIECE = OUT_ROWS * BLOCK_N * 2;
constexpr int OUT_BYTES = 2 * OUT_BUFS * OUT_PIECE;
// Registers per thread after the split: 128 x 64 + 256 x 216 = 63488 of the 384 x 168 = 64512 launched.
constexpr int REGS_LAUNCH = 168, REGS_ISSUE = 64, REGS_EPI = 216;
static_assert(128 * REGS_ISSUE + 256 * REGS_EPI <= PAIR_THREADS * REGS_LAUNCH, "a split above the launch's registers never completes");

struct PairParams {
    void* out;
    const void* bias;     // optional [N] in T, added to the rounded output
    int32_t* status;
    Await await;
    int M, N, K, G;
    int bm;               // batch rows per tile: a multiple of 32, at most 256
    int m_tiles, units;
    int box3d;            // K % 64 == 0: the tensor maps are [K/64][rows][64] views (else 2-D, one K step per slot)
    int slots;            // ring depth
    int x_bytes;          // shared-memory bytes of a CTA's activation tile (bm / 2 rows of one K step)
    int static_w;         // no kernel still in flight writes the weight: it is read before they are done
};

__device__ __forceinline__ uint32_t cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// `addr` (shared memory of this CTA) as it is seen in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// The accumulator's reads are what this arrival reports: they are complete (tcgen05.wait::ld) and ordered by the tcgen05
// fences on both sides. Nothing that was written is handed over, so no release at cluster scope, which made every arrival
// wait for a fence of the whole memory system: 0.5 - 1 us on the way from a drained accumulator to the next group's
// MMAs (fp16 1900 x 4096 -> 14336: 213 us with it, 178 without; bf16 1024 x 14336 -> 4096 at bm = 128: 166 and 112).
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Boxes of this GPU's memory into this CTA's shared memory; completion is signalled on `bar`, which may be the peer's.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const void* tmap, int c0, int c1, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* tmap, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
// Operand descriptor words (K-major tile, 128-byte swizzle: ptx::smem_desc_sw128): the high word is a constant, the low
// word holds the tile's address in 16-byte units.
constexpr uint32_t DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr) { return ((addr & 0x3FFFFu) >> 4) | (1u << 16); }
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint32_t da, uint32_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(da), "r"(db), "r"(idesc), "r"(accumulate), "n"(DESC_HI)
        : "memory");
}
// All MMAs issued so far arrive, when complete, on the barrier at this shared-memory offset in both CTAs.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void half_sync(int half) { asm volatile("bar.sync %0, 128;" ::"r"(1 + half) : "memory"); }
template <int R> __device__ __forceinline__ void regs_inc() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R)); }
template <int R> __device__ __forceinline__ void regs_dec() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R)); }

template <typename T, int KS, bool STAGED>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
pair_matmul_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   const __grid_constant__ CUtensorMap tmap_out, const PairParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
    // weight tiles, then activation tiles (each a multiple of 1024 bytes), then barriers
    const int S = p.slots;
    const uint32_t x_ring = smem_base + (uint32_t)(S * KS) * W_BYTES;
    const uint32_t out_base = x_ring + (uint32_t)(S * KS * p.x_bytes);
    const uint32_t bar_base = out_base + OUT_BYTES;
    auto bar_full = [&](int s) { return bar_base + 8u * s; };                              // first CTA: both CTAs' tiles landed
    auto bar_empty = [&](int s) { return bar_base + 8u * (PAIR_MAX_SLOTS + s); };          // MMAs of the slot complete
    auto bar_tfull = [&](int b) { return bar_base + 8u * (2 * PAIR_MAX_SLOTS + b); };      // accumulator complete
    auto bar_tempty = [&](int b) { return bar_base + 8u * (2 * PAIR_MAX_SLOTS + 2 + b); }; // first CTA: both CTAs drained it
    uint8_t* misc = smem_gen + (bar_base - smem_base) + 8 * (2 * PAIR_MAX_SLOTS + 4);
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(misc);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(misc + 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cta_rank();
    const Ctl ctl{p.status, abort_flag};

    if (threadIdx.x == 0) {
        *abort_flag = 0;
        for (int i = 0; i < PAIR_MAX_SLOTS; ++i) {
            ptx::mbar_init(bar_full(i), 1);
            ptx::mbar_init(bar_empty(i), 1);
        }
        for (int b = 0; b < 2; ++b) {
            ptx::mbar_init(bar_tfull(b), 1);
            ptx::mbar_init(bar_tempty(b), 16);
        }
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_w);
        ptx::prefetch_tensormap(&tmap_x);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot))), "r"(PAIR_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    ptx::tc_fence_before();
    __syncthreads();
    cluster_sync_all();                    // both CTAs' barriers exist before either signals the other's
    ptx::tc_fence_after();
    if (!p.static_w) ptx::grid_dep_wait();
    const uint32_t tmem_base = 0;          // the whole of tensor memory was allocated: it starts at column 0

    const int n_clusters = (int)(gridDim.x >> 1), first = (int)(blockIdx.x >> 1);
    const int xh = p.bm >> 1;                                        // batch rows of this CTA's activation tile
    // Units are dealt round-robin with the batch tiles of a weight tile next to each other, so that the clusters
    // running at one time share few weight rows and all of x in L2.
    auto unit_n0 = [&](int u) { return (u / p.m_tiles) * (2 * BLOCK_N) + (int)rank * BLOCK_N; };
    auto unit_m0 = [&](int u) { return (u % p.m_tiles) * p.bm; };

    if (warp < EPI0) regs_dec<REGS_ISSUE>();
    if (warp == 1 && p.static_w) ptx::grid_dep_wait();               // no bounded wait counts the time of the kernels in front
    if (warp == 0) {
        // ------------------------------------------------------------ TMA: weight and activation tiles
        const bool leader = ptx::elect_one();
        bool ok = true;
        if (p.await.flags != nullptr) {
            // the activation is still arriving from the other ranks: lane r watches rank r's flag
            const uint32_t epoch = *p.await.epoch;
            const uint64_t t0 = ptx::globaltimer_ns();
            bool arrived = true;
            if (lane < p.await.world && lane != p.await.rank) {
                uint32_t seen;
                do {
                    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.await.flags + lane) : "memory");
                    if ((int32_t)(seen - epoch) >= 0) break;
                    if (ptx::globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
                        *abort_flag = 1;
                        if (p.status) atomicCAS(p.status, 0, (int)(0x20000 | (lane << 8) | (epoch & 0xff)));
                        arrived = false;
                        break;
                    }
                } while (true);
            }
            if (!__all_sync(0xffffffffu, arrived)) ok = false;
            asm volatile("fence.proxy.async.global;" ::: "memory");
        }
        const uint32_t tx = 2u * (uint32_t)(KS * (p.x_bytes + W_BYTES));
        const uint32_t full0 = map_to_rank(bar_full(0), 0);
        int s = 0, filled = 0;
        uint32_t ph = 1;                                             // an untouched barrier passes the odd phase
        auto load_w = [&](int sl, int n0, int k) {                   // all K steps of a slot in one box per operand
            const uint32_t wt = smem_base + (uint32_t)(sl * KS) * W_BYTES, bar = full0 + 8u * (uint32_t)sl;
            if (rank == 0) ptx::mbar_expect_tx(bar_full(sl), tx);
            if (KS > 1 || p.box3d) tma_load_3d_pair(wt, &tmap_w, 0, n0, k >> 6, bar);
            else tma_load_2d_pair(wt, &tmap_w, k, n0, bar);
        };
        auto load_x = [&](int sl, int m0, int k) {
            const uint32_t xt = x_ring + (uint32_t)(sl * KS * p.x_bytes), bar = full0 + 8u * (uint32_t)sl;
            if (KS > 1 || p.box3d) tma_load_3d_pair(xt, &tmap_x, 0, m0, k >> 6, bar);
            else tma_load_2d_pair(xt, &tmap_x, k, m0, bar);
        };
        // The kernels in front may still be running: the slots of the first unit get their weights, then those kernels are
        // waited for, and the loop below finds so many weights there.
        int ahead = 0;
        if (p.static_w) {
            ahead = min(S, (p.K + KS * BLOCK_K - 1) / (KS * BLOCK_K));
            if (ok && leader)
                for (int i = 0; i < ahead; ++i) load_w(i, unit_n0(first), i * KS * BLOCK_K);
            __syncwarp();
            ptx::grid_dep_wait();
        }
        for (int u = first; u < p.units; u += n_clusters) {
            const int n0 = unit_n0(u), m0 = unit_m0(u) + (int)rank * xh;
            for (int k = 0; k < p.K; k += KS * BLOCK_K) {
                ok = ok && wait_bounded(bar_empty(s), ph, ctl, ROLE_TMA, 8 + s);
                if (ok && leader) {
                    if (ahead <= 0) load_w(s, n0, k);
                    load_x(s, m0, k);
                }
                --ahead;
                __syncwarp();
                filled += ok ? 1 : 0;
                if (++s == S) { s = 0; ph ^= 1u; }
            }
        }
        ptx::grid_dep_launch();                                      // the last loads are on their way: the next kernel may start
        // Every slot's last use has to be over before this CTA may go away: the copies have landed (also after an
        // abort, when no MMA will read them) and no commit is still to arrive here.
        const int from = max(0, filled - S);
        for (int i = from; i < filled; ++i) {
            const int sl = i % S;
            const uint32_t par = (uint32_t)(i / S) & 1u;             // parity of that fill's phase, on both barriers
            const uint64_t t0 = ptx::globaltimer_ns();
            const uint64_t limit = ok ? WAIT_LIMIT_NS : WAIT_LIMIT_NS / 16;
            while (!ptx::mbar_try_wait(bar_empty(sl), par)) {
                if (!ok && rank == 0 && ptx::mbar_try_wait(bar_full(sl), par)) break;
                if (ptx::globaltimer_ns() - t0 > limit) break;
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (first CTA of the pair)
        if (rank == 0) {
            const bool leader = ptx::elect_one();
            constexpr uint32_t FMT = std::is_same<T, __nv_bfloat16>::value ? 1u : 0u;
            const uint32_t IDESC = (1u << 4) | (FMT << 7) | (FMT << 10) | ((uint32_t)(p.bm >> 3) << 17) |
                                   ((uint32_t)(2 * BLOCK_N >> 4) << 24);
            const uint32_t da0 = desc_lo(smem_base), db0 = desc_lo(x_ring);
            const uint32_t xstep = (uint32_t)p.x_bytes >> 4;
            constexpr uint32_t WSTEP = W_BYTES >> 4;
            int s = 0, job = 0;
            uint32_t ph = 0;
            bool ok = true;
            // No early exit: after a failed wait the loops run on without waiting or issuing. Ring positions and
            // descriptors are then functions of the launch alone, which the compiler can keep in uniform registers
            // (with a break on a waited-for value they live in per-thread registers and every MMA pays for moving its
            // operands: measured 160 cycles per instruction, more than the instruction takes).
            for (int u = first; u < p.units; u += n_clusters) {
                for (int g = 0; g < p.G; ++g, ++job) {
                    const int buf = job & 1;
                    ok = ok && wait_bounded<true>(bar_tempty(buf), (uint32_t)((job >> 1) & 1) ^ 1u, ctl, ROLE_MMA, 32 + buf);
                    ptx::tc_fence_after();                           // the epilogue's reads of this accumulator
                    const uint32_t d = tmem_base + (uint32_t)(buf * PAIR_ACC_STRIDE);
                    const int kend = min(p.K, (g + 1) * GROUP_K);
                    for (int k = g * GROUP_K; k < kend; k += KS * BLOCK_K) {
                        ok = ok && wait_bounded(bar_full(s), ph, ctl, ROLE_MMA, s);
                        __syncwarp();
                        const uint32_t da = da0 + (uint32_t)(s * KS) * WSTEP, db = db0 + (uint32_t)(s * KS) * xstep;
                        const uint32_t be = bar_empty(s), tf = bar_tfull(buf);
                        const uint32_t acc0 = k > g * GROUP_K ? 1u : 0u;
                        const bool last = k + KS * BLOCK_K >= kend;
                        if (kend - k >= KS * BLOCK_K) {
                            if (ok && leader) {
#pragma unroll
                                for (int j = 0; j < KS; ++j) {
                                    const uint32_t a = da + (uint32_t)j * WSTEP, b = db + (uint32_t)j * xstep;
                                    umma_pair(d, a, b, IDESC, j ? 1u : acc0);
                                    umma_pair(d, a + 2, b + 2, IDESC, 1u);
                                    umma_pair(d, a + 4, b + 4, IDESC, 1u);
                                    umma_pair(d, a + 6, b + 6, IDESC, 1u);
                                }
                                commit_pair(be);
                                if (last) commit_pair(tf);
                            }
                        } else {                                     // the end of K: only the K = 16 steps that hold elements
                            const int n16 = (kend - k + UMMA_K - 1) / UMMA_K;
                            if (ok && leader) {
                                for (int i = 0; i < n16; ++i)
                                    umma_pair(d, da + (uint32_t)(i >> 2) * WSTEP + 2u * (uint32_t)(i & 3), db + (uint32_t)(i >> 2) * xstep + 2u * (uint32_t)(i & 3),
                                              IDESC, (acc0 | (uint32_t)i) ? 1u : 0u);
                                commit_pair(be);
                                commit_pair(tf);
                            }
                        }
                        __syncwarp();
                        if (++s == S) { s = 0; ph ^= 1u; }
                    }
                }
            }
        }
    } else if (warp >= EPI0) {
        // ------------------------------------------------------------ epilogue: totals in registers
        regs_inc<REGS_EPI>();
        if (p.static_w) ptx::grid_dep_wait();                        // before the first store
        constexpr int CH = PAIR_MAX_BM / 2 / 16;                     // 16-column pieces of half a batch tile
        static_assert(CH % 4 == 0, "read in blocks of 32 columns, two at a time");
        const int quad = warp & 3, half = (warp - EPI0) >> 2;
        const uint32_t lane_base = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * xh);
        T* out = static_cast<T*>(p.out);
        const T* bias = static_cast<const T*>(p.bias);
        const uint32_t tempty0 = map_to_rank(bar_tempty(0), 0), tempty1 = map_to_rank(bar_tempty(1), 0);
        const uint32_t stage = out_base + (uint32_t)(half * OUT_BUFS * OUT_PIECE);
        int job = 0;
        uint32_t piece = 0;                                          // pieces this half has staged
        bool ok = true;
        // No early exit here either: the four warps of a half meet at a barrier for every piece they store.
        for (int u = first; u < p.units; u += n_clusters) {
            float tot[CH * 16];
#pragma unroll
            for (int j = 0; j < CH * 16; ++j) tot[j] = 0.0f;
            const int m0 = unit_m0(u) + half * xh;
            const int cols = min(xh, p.M - m0);                      // batch rows that exist (may be <= 0)
            for (int g = 0; g < p.G; ++g, ++job) {
                const int buf = job & 1;
                ok = ok && wait_bounded(bar_tfull(buf), (uint32_t)(job >> 1) & 1u, ctl, ROLE_EPI, 16 + buf);
                if (!ok) continue;
                ptx::tc_fence_after();
                const uint32_t acc = lane_base + (uint32_t)(buf * PAIR_ACC_STRIDE);
#pragma unroll
                for (int c = 0; c < CH / 2; c += 2) {                // warp-uniform conditions; two blocks of 32 columns share a wait
                    if (c * 32 < cols) {
                        uint32_t v0[32], v1[32];
                        const bool two = (c + 1) * 32 < cols;
                        ptx::tmem_ld_32x32(acc + c * 32, v0);
                        if (two) ptx::tmem_ld_32x32(acc + c * 32 + 32, v1);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) tot[c * 32 + j] = add_rn(tot[c * 32 + j], __uint_as_float(v0[j]));
                        if (two) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) tot[c * 32 + 32 + j] = add_rn(tot[c * 32 + 32 + j], __uint_as_float(v1[j]));
                        }
                    }
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) arrive_cluster(buf ? tempty1 : tempty0);
            }
            const int n = unit_n0(u) + quad * 32 + lane;
            if (STAGED) {                                            // outputs whose rows are whole 16-byte units: through shared memory and TMA
                const T* b = n < p.N ? bias : nullptr;
#pragma unroll
                for (int c = 0; c < CH; ++c) {
                    if (c * 16 < cols) {                             // the same in the four warps of a half
                        const uint32_t dst = stage + (piece & (OUT_BUFS - 1)) * OUT_PIECE;
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            ptx::st_shared(dst + (uint32_t)(j * BLOCK_N * 2 + (quad * 32 + lane) * 2), round_out<T>(tot[c * 16 + j], b, n));
                        ptx::fence_proxy_async_smem();
                        // before the barrier all but the last two copies have read their piece: the next piece is free after it
                        if (quad == 0 && lane == 0) ptx::bulk_wait_read<OUT_BUFS - 2>();
                        half_sync(half);
                        if (ok && quad == 0 && lane == 0) ptx::tma_store_2d(&tmap_out, unit_n0(u), m0 + c * 16, dst);
                        ++piece;
                    }
                }
            } else if (ok && n < p.N) {
                T* dst = out + (long long)m0 * p.N + n;
#pragma unroll
                for (int j = 0; j < CH * 16; ++j)
                    if (j < cols) dst[(long long)j * p.N] = round_out<T>(tot[j], bias, n);
            }
        }
        if (quad == 0 && lane == 0) ptx::bulk_wait_all();
    }

    __syncwarp();
    ptx::tc_fence_before();
    __syncthreads();
    cluster_sync_all();                    // neither CTA leaves while the other may still signal it or read its operands
    if (warp == 1) {
        ptx::tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(PAIR_TMEM_COLS) : "memory");
    }
}

template <typename T, int KS, bool STAGED>
int launch_pair_t(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mo, const PairParams& p, int smem, cudaStream_t st) {
    auto kern = pair_matmul_kernel<T, KS, STAGED>;
    static bool attr_done[64] = {false};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!attr_done[dev]) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM_LIMIT);
        if (e != cudaSuccess) return fail_cuda("matmul smem attr", e);
        attr_done[dev] = true;
    }
    const int clusters = sm_count() / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2u * (unsigned)(p.units < clusters ? p.units : clusters));
    cfg.blockDim = dim3(PAIR_THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled(p.await.flags != nullptr) ? 2 : 1;
    cudaLaunchKernelEx(&cfg, kern, mw, mx, mo, p);
    return check_launch("matmul (tensor-core path, SM pairs)");
}

}  // namespace

int launch_pair_matmul(const void* x, int64_t x_ld, const void* w, int64_t w_ld, void* out, int64_t M, int64_t N, int64_t K, int dtype,
                       const TcShape& shape, int32_t* status, cudaStream_t st) {
    const int bm = shape.bm;
    if (bm < 32 || bm > PAIR_MAX_BM || bm % 32) return fail(BI_ERR_BAD_ARG, "matmul: batch tile %d of a pair of SMs", bm);
    PairParams p{};
    p.out = out; p.bias = shape.bias; p.status = status; p.await = shape.await;
    p.M = (int)M; p.N = (int)N; p.K = (int)K;
    p.G = (int)((K + GROUP_K - 1) / GROUP_K);
    p.static_w = shape.static_w && !shape.await.flags ? 1 : 0;
    p.bm = bm;
    p.m_tiles = (int)((M + bm - 1) / bm);
    const int64_t units = (N + 2 * BLOCK_N - 1) / (2 * BLOCK_N) * p.m_tiles;
    if (units >= (1LL << 30)) return fail(BI_ERR_UNSUPPORTED, "matmul: %lld work units exceed the kernel's 32-bit unit index", (long long)units);
    p.units = (int)units;
    p.x_bytes = bm / 2 * BLOCK_K * 2;                       // a multiple of 2 KB
    p.box3d = K % BLOCK_K == 0 ? 1 : 0;
    const int limit = PAIR_SMEM_LIMIT - 1024 - PAIR_BAR_BYTES - OUT_BYTES;
    const int ks = p.box3d ? 2 : 1;                         // two K steps per slot: half the handshakes (bm = 128: 349 -> 321 us); four measure the same
    const int slot_bytes = ks * (W_BYTES + p.x_bytes);
    const int fit = limit / slot_bytes;
    p.slots = fit < PAIR_MAX_SLOTS ? fit : PAIR_MAX_SLOTS;
    const int smem = 1024 + PAIR_BAR_BYTES + OUT_BYTES + p.slots * slot_bytes;

    const CUtensorMapDataType dt = dtype == BI_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap mw, mx, mo{};
    int rc = BI_OK;
    const bool staged = N % 8 == 0 && aligned(out, 16);
    if (staged) rc = make_map(&mo, dt, 2, out, (uint64_t)N, (uint64_t)M, (uint64_t)N, BLOCK_N, OUT_ROWS, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc) return rc;
    if (p.box3d) {
        rc = make_map3(&mx, dt, 2, x, (uint64_t)(K / BLOCK_K), (uint64_t)M, (uint64_t)x_ld, (uint32_t)(bm / 2), (uint32_t)ks);
        if (!rc) rc = make_map3(&mw, dt, 2, w, (uint64_t)(K / BLOCK_K), (uint64_t)N, (uint64_t)w_ld, BLOCK_N, (uint32_t)ks);
    } else {
        rc = make_map(&mx, dt, 2, x, (uint64_t)K, (uint64_t)M, (uint64_t)x_ld, BLOCK_K, (uint32_t)(bm / 2), CU_TENSOR_MAP_SWIZZLE_128B);
        if (!rc) rc = make_map(&mw, dt, 2, w, (uint64_t)K, (uint64_t)N, (uint64_t)w_ld, BLOCK_K, BLOCK_N, CU_TENSOR_MAP_SWIZZLE_128B);
    }
    if (rc) return rc;
#define BI_PAIR_LAUNCH_KS(TT, STAGED) (ks == 2 ? launch_pair_t<TT, 2, STAGED>(mw, mx, mo, p, smem, st) : launch_pair_t<TT, 1, STAGED>(mw, mx, mo, p, smem, st))
#define BI_PAIR_LAUNCH(TT) (staged ? BI_PAIR_LAUNCH_KS(TT, true) : BI_PAIR_LAUNCH_KS(TT, false))
    return dtype == BI_BF16 ? BI_PAIR_LAUNCH(__nv_bfloat16) : BI_PAIR_LAUNCH(__half);
#undef BI_PAIR_LAUNCH_KS
#undef BI_PAIR_LAUNCH
}

}  // namespace bi
