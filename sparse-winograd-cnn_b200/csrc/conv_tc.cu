// TF32 tensor-core path of the Winograd-domain product (sm_100a only): tcgen05.mma with
// accumulators in TMEM, operands staged by TMA into 128B-swizzled shared memory, the
// A^T m A output transform done by the epilogue warps straight from TMEM.
//
// Work unit = 128 tiles (one TMEM lane per tile) x 64 output channels x all 16 Winograd
// positions.  The 16 positions are walked one Winograd row i (four positions j) at a time:
// four 128x64 fp32 accumulators (256 TMEM columns) per row, double-buffered across rows
// (512 columns), so the epilogue of row i overlaps the MMAs of row i+1 and V is read from
// memory exactly once per 64 output channels.  Nothing but Y is written.
//
// Warp roles (384 threads = 3 warpgroups): warp 0 = TMA producer, warp 1 = TMEM owner + MMA issuer
// (warps 2-3 idle), warps 4..11 = epilogue (two warps per TMEM lane quarter, 32 columns each).  The
// control warpgroup hands most of its registers to the epilogue warpgroups (setmaxnreg), which keep
// 128 output values per thread live.
// Every mbarrier wait is bounded; on expiry the kernel records where it gave up, drains
// and returns (status readable through wg2x2_last_device_status).
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstring>

#include "wg_common.cuh"

namespace wg {

constexpr int kBlockM = 128;            // tiles per unit (TMEM lanes)
constexpr int kBlockN = 64;             // output channels per unit
constexpr int kBlockK = 32;             // tf32 elements per stage along C: 128 bytes = one swizzle row
constexpr int kStages = 8;
constexpr int kABytes = kBlockM * kBlockK * 4;   // 16 KB
constexpr int kBBytes = kBlockN * kBlockK * 4;   //  8 KB
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kTcThreads = 320;           // gradient GEMM kernels: producer, MMA issuer, 8 epilogue warps
constexpr int kFwdThreads = 384;          // forward kernel: one control warpgroup + two epilogue warpgroups
constexpr int kEpiWarps = 8;
constexpr uint32_t kTmemCols = 512;
constexpr int kCtrlBytes = 1024;                   // barriers, TMEM pointer, abort flag, per-role block masks
constexpr int kEpiStageBytes = 32 * 32 * 4;        // per epilogue warp: 32 tiles x 32 channels, for coalesced NHWC stores
constexpr int kSmemBytes = kStages * kStageBytes + 1024 /*alignment slack*/ + kCtrlBytes + kEpiWarps * kEpiStageBytes;
constexpr uint32_t kSpinLimit = 40u * 1000 * 1000;   // try_wait polls before a wait gives up (~ a second)

__device__ unsigned int g_tc_status[2];  // [0] = 0 ok / 1 timeout, [1] = where (role<<8 | detail)
__device__ unsigned int g_tc_diag[32];   // after a timeout: per role (where >> 8), the wait it was in when it gave up or was told to

#ifdef WG_TC_TRACE   // development aid: cycle stamps of CTA 0's roles, read back by wg2x2_debug_read_trace
__device__ long long g_tc_trace[4096];
#define TC_TRACE(slot) do { if (blockIdx.x == 0 && (slot) < 4096) g_tc_trace[(slot)] = clock64(); } while (0)
#else
#define TC_TRACE(slot) do { } while (0)
#endif

// ---------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait.  Returns false when it gave up (or when another role already did).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag, unsigned where,
                                          uint32_t limit = kSpinLimit)
{
    for (uint32_t it = 0; it < limit; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 1023) == 1023 && *abort_flag) { g_tc_diag[(where >> 8) & 31] = where | (parity << 16) | 0x40000000u; return false; }
    }
    *abort_flag = 1;
    g_tc_diag[(where >> 8) & 31] = where | (parity << 16) | 0x80000000u;
    g_tc_status[1] = where;
    g_tc_status[0] = 1;
    return false;
}

// The same wait for a role in which all 32 lanes of a warp poll: lanes can leave the polling loop in different
// iterations, and what follows (tcgen05.ld / tcgen05.st / tcgen05.wait) is .sync.aligned, which a diverged
// warp must not execute.  The vote brings the lanes back together and makes the outcome (and so every
// break out of the role's loop) the same for all of them.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag, unsigned where,
                                               uint32_t limit = kSpinLimit)
{
    const bool ok = mbar_wait(bar, parity, abort_flag, where, limit);
    return __all_sync(0xffffffffu, ok);
}

// After a wait that gave up: copies and MMAs already in flight get about a millisecond to end before the CTA hands back its memories
__device__ __forceinline__ void let_them_land()
{
    for (int it = 0; it < 1000; ++it) __nanosleep(1000);
}

// true in exactly one lane of the (converged) warp
__device__ __forceinline__ bool elect_one()
{
    uint32_t pred;
    asm volatile(
        "{\n\t.reg .pred P;\n\t"
        "elect.sync _|P, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, P;\n\t}"
        : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols)
{
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish()
{
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols)
{
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] * B[smem], M=128, N=kBlockN, K=8 (tf32)
__device__ __forceinline__ void umma_tf32(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// mbarrier arrives once all MMAs issued so far by this thread have completed
__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 lanes x 8 consecutive 32-bit columns -> 8 registers per thread
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *r)
{
    uint32_t u[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(taddr));
#pragma unroll
    for (int q = 0; q < 8; ++q) r[q] = __uint_as_float(u[q]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle, rows 128 B apart,
// 8-row groups 1024 B apart (SBO), LBO unused (1), descriptor version 1 (sm_100).
__device__ __forceinline__ uint64_t make_desc_k_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;                 // leading byte offset (ignored for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset
    d |= (uint64_t)1 << 46;                 // version
    d |= (uint64_t)2 << 61;                 // SWIZZLE_128B
    return d;
}

// The 16 per-position block masks of one unit: 16 independent loads, parked in shared memory
// so that the role's loop reads them without another trip to L2.
__device__ __forceinline__ void load_unit_masks(const unsigned long long *masks, int nKB, int kb, unsigned long long *dst)
{
    unsigned long long m[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) m[t] = __ldg(masks + (long long)t * nKB + kb);
#pragma unroll
    for (int t = 0; t < 16; ++t) dst[t] = m[t];
}

// Instruction descriptor: D=f32, A=B=tf32, both K-major, N and M as given
__host__ __device__ constexpr uint32_t make_idesc_tf32(int M, int N)
{
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ---------------------------------------------------------------------------------------
// Weight preparation: W (16,C,K) -> Wp (16,K,C) rounded to TF32 (round-to-nearest), plus a
// 64-bit map mask[t][kb] whose bit cc is set when the 64x32 block (out-channels kb*64..,
// in-channels cc*32..) of position t has any non-zero weight.  Layers with more than 64
// chunks (C > 2048) keep every bit set: nothing is skipped there.
// A CTA takes 64 out-channels x 256 in-channels of one position: one byte of a map word, which it alone writes (so that the
// map needs no clearing first), the first CTA along C also the bytes beyond the last one.
// ---------------------------------------------------------------------------------------
constexpr int kPackC = 256;
constexpr int kPackThreads = 1024;        // four blocks at a time
// byte `group` of the map word: bit r = block r of the group; nbytes: bytes of a word that the CTAs along the chunks write
__device__ __forceinline__ void store_map_byte(unsigned long long *word, int group, int ngroups, int nCC, unsigned bits)
{
    unsigned char *b = reinterpret_cast<unsigned char *>(word);
    if (nCC > 64) {
        if (group == 0) *word = ~0ull;
        return;
    }
    b[group] = (unsigned char)bits;
    if (group == 0)
        for (int g = ngroups; g < 8; ++g) b[g] = 0;
}
__global__ void __launch_bounds__(kPackThreads) pack_weights_kernel(const float *__restrict__ Wt, float *__restrict__ Wp,
                                                                      unsigned long long *__restrict__ masks, int C, int K, int nKB, int nCC)
{
    after_previous_kernel(Wt, Wp, masks);
    __shared__ float tile[kPackThreads / 128][32][33];
    __shared__ int live;
    if (threadIdx.x == 0) live = 0;
    __syncthreads();
    const int t = blockIdx.z, kb = blockIdx.x;
    const int tx = threadIdx.x & 31, ty = (threadIdx.x >> 5) & 3, part = threadIdx.x >> 7;   // 128 threads turn a 32 x 32 half of a block
    const int k0 = kb * 64 + 32 * (part & 1);
#pragma unroll 1
    for (int r0 = 0; r0 < kPackC / 32; r0 += kPackThreads / 256) {
        const int r = r0 + (part >> 1), c0 = blockIdx.y * kPackC + r * 32;
        int nz = 0;
        float w[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = c0 + ty + 4 * q, k = k0 + tx;
            w[q] = (c < C && k < K) ? __ldg(Wt + ((long long)t * C + c) * K + k) : 0.f;
        }
        if (r0) __syncthreads();           // the turned values of the round before have been read
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            uint32_t u;
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(w[q]));
            w[q] = __uint_as_float(u);
            nz |= (w[q] != 0.f);
            tile[part][ty + 4 * q][tx] = w[q];
        }
        if (__any_sync(0xffffffffu, nz) && tx == 0) atomicOr(&live, 1 << r);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int k = k0 + ty + 4 * q, c = c0 + tx;
            if (c < C && k < K) Wp[((long long)t * K + k) * C + c] = tile[part][tx][ty + 4 * q];
        }
        if (blockIdx.y * kPackC + (r0 + kPackThreads / 256) * 32 >= C) break;
    }
    __syncthreads();
    if (threadIdx.x == 0) store_map_byte(masks + (long long)t * nKB + kb, blockIdx.y, gridDim.y, nCC, (unsigned)live);
}

// ---------------------------------------------------------------------------------------
// Main kernel
// ---------------------------------------------------------------------------------------
struct TcParams {
    float *Y;
    // optional epilogue extras: Y = acc * out_scale[k] + out_shift[k] (+ residual, same shape and layout as Y)
    const float *out_scale, *out_shift, *residual;
    int res_relu;            // the residual passes through a ReLU first
    const unsigned long long *masks;
    long long P;
    int nH, nW, C, K, outH, outW;
    int nMT, nKB, nCC;   // m-tiles, 64-channel blocks, 32-channel chunks
    int tpu;             // tiles per unit (<= 128): chosen so that the units divide evenly over the SMs
    int units;
    uint32_t spin_limit;    // polls before a wait gives up (wg2x2_set_wait_limit)
    int drop_load;          // >= 0: the producer of CTA 0 leaves out its drop_load-th stage (wg2x2_test_drop_load), else -1
};

// EXTRAS: compile the optional epilogue affine map and residual addition in (kept out of the plain kernel,
// whose store loops are the critical path of the HBM-bound shapes).
template <int LAYOUT, bool EXTRAS>
__global__ void __launch_bounds__(kFwdThreads, 1)
conv_fwd_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB, const TcParams prm)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;                 // 1024-B aligned operand stages
    uint8_t *gen_base = smem_raw + (base - raw);
    const uint32_t bars = base + kStages * kStageBytes;           // barrier block
    uint64_t *bars_gen = reinterpret_cast<uint64_t *>(gen_base + kStages * kStageBytes);
    // barrier layout (8 B each): full[kStages], empty[kStages], acc_full[2], acc_empty[2], then tmem ptr, abort flag
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kStages + s); };
    auto accf_bar = [&](int b) { return bars + 8u * (2 * kStages + b); };
    auto acce_bar = [&](int b) { return bars + 8u * (2 * kStages + 2 + b); };
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(bars_gen + 2 * kStages + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bars_gen + 2 * kStages + 5);
    unsigned long long *role_masks = reinterpret_cast<unsigned long long *>(bars_gen + 2 * kStages + 8);  // 2 x 16 words
    float *epi_stage_all = reinterpret_cast<float *>(gen_base + kStages * kStageBytes + kCtrlBytes);

    // (broadcast from lane 0: the compiler then treats the warp index, and all that is derived from it, as warp-uniform)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(accf_bar(b), 1); mbar_init(acce_bar(b), kEpiWarps); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc(smem_u32((const void *)tmem_ptr_slot), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_slot, 0);
    // (set-up touched no global memory; from here on the kernel reads and writes it)
    wait_for_previous_kernel(kNumSMs / 2);

    const int nCC = prm.nCC;

    // 384 threads x 168 registers at launch: the control warpgroup drops to 40 registers per thread and the
    // two epilogue warpgroups rise to 232 (each inside its own branch, so that no code is shared between them)
    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 0) {
        // ------------------------------ TMA producer ------------------------------------
        if (lane == 0) {
            int s = 0; uint32_t ph = 0;
            bool ok = true;
            int tr = 0; (void)tr;
            int nload = 0;
            for (int u = blockIdx.x; u < prm.units && ok; u += gridDim.x) {
                const int mt = u / prm.nKB, kb = u % prm.nKB;
                const int p0 = mt * prm.tpu, k0 = kb * kBlockN;
                load_unit_masks(prm.masks, prm.nKB, kb, role_masks);
                for (int t = 0; t < 16 && ok; ++t) {
                    const unsigned long long mk = role_masks[t];
                    for (int cc = 0; cc < nCC; ++cc) {
                        if (cc > 0 && cc < 64 && !((mk >> cc) & 1ull)) continue;   // all-zero weight block: nothing to add
                        if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, 0x100u | s, prm.spin_limit)) { ok = false; break; }
                        TC_TRACE(tr); ++tr;
                        // test hook: this stage is never filled (nothing is put in flight), so the issuer's wait on it runs out
                        if (blockIdx.x == 0 && nload++ == prm.drop_load) { ok = false; break; }
                        mbar_expect_tx(full_bar(s), kStageBytes);
                        const uint32_t a_dst = base + s * kStageBytes;
                        tma_load_3d(a_dst, &mapA, full_bar(s), cc * kBlockK, p0, t);
                        tma_load_3d(a_dst + kABytes, &mapB, full_bar(s), cc * kBlockK, k0, t);
                        if (++s == kStages) { s = 0; ph ^= 1u; }
                    }
                }
            }
            if (!ok) {
                // give copies already in flight about a millisecond to land before the CTA
                // hands its shared memory back
                for (int it = 0; it < 1000; ++it) __nanosleep(1000);
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer --------------------------------------
        // The whole warp walks the loop with warp-uniform values, so that descriptors and addresses live in uniform
        // registers; one elected lane issues the MMAs and the commits.  (Issued by a lone lane from per-thread
        // registers, an MMA takes several times as many issue slots, and the epilogue warps compete for them.)
        {
            constexpr uint32_t idesc = make_idesc_tf32(kBlockM, kBlockN);
            const bool leader = elect_one();
            int s = 0; uint32_t ph = 0;
            uint32_t acc_use[2] = {0, 0};
            bool ok = true;
            int tr = 0; (void)tr;
            for (int u = blockIdx.x; u < prm.units && ok; u += gridDim.x) {
                const int kb = u % prm.nKB;
                __syncwarp();
                if (lane < 16) role_masks[16 + lane] = __ldg(prm.masks + (long long)lane * prm.nKB + kb);
                __syncwarp();
                for (int i = 0; i < 4 && ok; ++i) {
                    const int buf = i & 1;
                    // the epilogue must have drained this accumulator buffer
                    if (!mbar_wait_warp(acce_bar(buf), (acc_use[buf] & 1u) ^ 1u, abort_flag, 0x200u | buf, prm.spin_limit)) { ok = false; break; }
                    acc_use[buf]++;
                    tc_fence_after();
                    for (int j = 0; j < 4 && ok; ++j) {
                        const int t = 4 * i + j;
                        const unsigned long long mk = role_masks[16 + t];
                        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * 4 * kBlockN + j * kBlockN);
                        for (int cc = 0; cc < nCC; ++cc) {
                            if (cc > 0 && cc < 64 && !((mk >> cc) & 1ull)) continue;
                            if (!mbar_wait_warp(full_bar(s), ph, abort_flag, 0x300u | s, prm.spin_limit)) { ok = false; break; }
                            if (leader) TC_TRACE(512 + tr);
                            tc_fence_after();
                            const uint32_t a_addr = base + s * kStageBytes;
                            const uint64_t adesc = make_desc_k_sw128(a_addr);
                            const uint64_t bdesc = make_desc_k_sw128(a_addr + kABytes);
                            if (leader) {
#pragma unroll
                                for (int kk = 0; kk < kBlockK / 8; ++kk)   // 32 bytes (8 tf32) further along K per step
                                    umma_tf32(d_tmem, adesc + 2u * kk, bdesc + 2u * kk, idesc, (cc > 0 || kk > 0) ? 1u : 0u);
                                umma_commit(empty_bar(s));
                            }
                            __syncwarp();
                            if (leader) TC_TRACE(1024 + tr);
                            ++tr;
                            if (++s == kStages) { s = 0; ph ^= 1u; }
                        }
                    }
                    if (ok && leader) umma_commit(accf_bar(buf));
                    __syncwarp();
                }
            }
        }
    }
    } else {
        // ------------------------------ epilogue ----------------------------------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 232;");
        const int ew = warp - 4;
        const int q = warp & 3;            // TMEM lane quarter this warp may read
        const int half = ew >> 2;          // which 32 of the 64 columns
        uint32_t acc_use[2] = {0, 0};
        bool ok = true;
        int tr = 0; (void)tr;
        for (int u = blockIdx.x; u < prm.units && ok; u += gridDim.x) {
            const int mt = u / prm.nKB, kb = u % prm.nKB;
            float y[4][32];                // [2a+e][column]
#pragma unroll
            for (int o = 0; o < 4; ++o)
#pragma unroll
                for (int c = 0; c < 32; ++c) y[o][c] = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int buf = i & 1;
                if (ok && !mbar_wait_warp(accf_bar(buf), acc_use[buf] & 1u, abort_flag, 0x400u | (ew << 4) | buf, prm.spin_limit)) ok = false;
                acc_use[buf]++;
                if (ok) {
                    if (ew == 0 && lane == 0) TC_TRACE(1536 + 4 * tr);
                    tc_fence_after();
                    const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 4 * kBlockN + half * 32);
#pragma unroll
                    for (int ch = 0; ch < 4; ++ch) {
                        float m[4][8];
#pragma unroll
                        for (int j = 0; j < 4; ++j) tmem_ld8(taddr + (uint32_t)(j * kBlockN + ch * 8), m[j]);
                        tmem_ld_wait();
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            float z0, z1;
                            at_cols(m[0][c], m[1][c], m[2][c], m[3][c], z0, z1);
                            // rows: AT[0] = [1,1,1,0], AT[1] = [0,1,-1,-1]
                            if (i <= 2) { y[0][ch * 8 + c] += z0; y[1][ch * 8 + c] += z1; }
                            if (i == 1) { y[2][ch * 8 + c] += z0; y[3][ch * 8 + c] += z1; }
                            if (i >= 2) { y[2][ch * 8 + c] -= z0; y[3][ch * 8 + c] -= z1; }
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acce_bar(buf));
                    if (ew == 0 && lane == 0) TC_TRACE(1536 + 4 * tr + 1);
                    ++tr;
                }
            }
            if (!ok) break;
            if (ew == 0 && lane == 0) TC_TRACE(1536 + 4 * (tr - 1) + 2);
            // ---- store the 2x2 outputs of this thread's tile for its 32 channels ----
            const long long p = (long long)mt * prm.tpu + q * 32 + lane;
            const bool tile_ok = (q * 32 + lane < prm.tpu) && p < prm.P;
            const int tw = (int)(p % prm.nW), th = (int)((p / prm.nW) % prm.nH), b = (int)(p / ((long long)prm.nW * prm.nH));
            const int kbase = kb * kBlockN + half * 32;
            if (LAYOUT == WG2X2_NHWC) {
                if (kbase + 32 <= prm.K && (prm.K & 3) == 0) {
                    // Coalesced path: the warp turns its 32 tiles x 32 channels through shared memory
                    // so that 8 consecutive lanes write one full 128-byte line (4 lines per instruction).
                    float *stg = epi_stage_all + ew * (kEpiStageBytes / 4);
                    float4 sc4 = make_float4(1.f, 1.f, 1.f, 1.f), sh4 = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (EXTRAS && prm.out_scale) {   // this lane always stores channels kbase + 4*(lane&7) .. +3
                        sc4 = __ldg(reinterpret_cast<const float4 *>(prm.out_scale + kbase) + (lane & 7));
                        sh4 = __ldg(reinterpret_cast<const float4 *>(prm.out_shift + kbase) + (lane & 7));
                    }
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int h = 2 * th + a, w = 2 * tw + e;
                            const long long my_off = (tile_ok && h < prm.outH && w < prm.outW)
                                ? (((long long)b * prm.outH + h) * prm.outW + w) * prm.K + kbase : -1;
                            __syncwarp();
#pragma unroll
                            for (int c8 = 0; c8 < 8; ++c8)   // 16-byte chunk c8 of row `lane`, XOR-swizzled against bank conflicts
                                *reinterpret_cast<float4 *>(stg + lane * 32 + ((c8 ^ (lane & 7)) << 2)) =
                                    make_float4(y[2 * a + e][4 * c8], y[2 * a + e][4 * c8 + 1], y[2 * a + e][4 * c8 + 2], y[2 * a + e][4 * c8 + 3]);
                            __syncwarp();
                            // residual values first (8 independent loads in flight), then the stores
                            long long off[8];
                            float4 rs[8];
#pragma unroll
                            for (int r = 0; r < 8; ++r) {
                                off[r] = __shfl_sync(0xffffffffu, my_off, 4 * r + (lane >> 3));
                                rs[r] = make_float4(0.f, 0.f, 0.f, 0.f);
                                if (EXTRAS && prm.residual && off[r] >= 0) rs[r] = __ldg(reinterpret_cast<const float4 *>(prm.residual + off[r]) + (lane & 7));
                                if (EXTRAS && prm.res_relu) rs[r] = relu_nan(rs[r]);
                            }
#pragma unroll
                            for (int r = 0; r < 8; ++r) {
                                const int row = 4 * r + (lane >> 3), ch = lane & 7;
                                float4 v = *reinterpret_cast<const float4 *>(stg + row * 32 + ((ch ^ (row & 7)) << 2));
                                if (off[r] >= 0) {
                                    if (EXTRAS && prm.out_scale) {
                                        v.x = fmaf(v.x, sc4.x, sh4.x); v.y = fmaf(v.y, sc4.y, sh4.y);
                                        v.z = fmaf(v.z, sc4.z, sh4.z); v.w = fmaf(v.w, sc4.w, sh4.w);
                                    }
                                    if (EXTRAS) { v.x += rs[r].x; v.y += rs[r].y; v.z += rs[r].z; v.w += rs[r].w; }
                                    *reinterpret_cast<float4 *>(prm.Y + off[r] + 4 * ch) = v;
                                }
                            }
                        }
                } else if (tile_ok) {
#pragma unroll
                    for (int a = 0; a < 2; ++a)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int h = 2 * th + a, w = 2 * tw + e;
                            if (h >= prm.outH || w >= prm.outW) continue;
                            const long long o = (((long long)b * prm.outH + h) * prm.outW + w) * prm.K + kbase;
#pragma unroll
                            for (int c = 0; c < 32; ++c)
                                if (kbase + c < prm.K) {
                                    float v = y[2 * a + e][c];
                                    if (EXTRAS && prm.out_scale) v = fmaf(v, __ldg(prm.out_scale + kbase + c), __ldg(prm.out_shift + kbase + c));
                                    if (EXTRAS && prm.residual) v += prm.res_relu ? relu_nan(__ldg(prm.residual + o + c)) : __ldg(prm.residual + o + c);
                                    prm.Y[o + c] = v;
                                }
                        }
                }
            } else if (tile_ok) {
                // NCHW: the two pixels of a tile row are adjacent in memory; with an even row
                // length consecutive lanes write consecutive, fully covered 8-byte pairs.
                const bool pair = (prm.outW & 1) == 0;
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const int h = 2 * th + a;
                    if (h >= prm.outH) continue;
                    const long long cstride = (long long)prm.outH * prm.outW;
                    const long long o0 = (((long long)b * prm.K + kbase) * prm.outH + h) * prm.outW + 2 * tw;
#pragma unroll
                    for (int cg = 0; cg < 32; cg += 8) {
                        // residual values of 8 channels first (independent loads in flight), then the stores
                        float2 rs[8];
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            rs[c] = make_float2(0.f, 0.f);
                            if (EXTRAS && prm.residual && kbase + cg + c < prm.K) {
                                const float *rp = prm.residual + o0 + (cg + c) * cstride;
                                if (pair) rs[c] = __ldg(reinterpret_cast<const float2 *>(rp));
                                else { rs[c].x = __ldg(rp); if (2 * tw + 1 < prm.outW) rs[c].y = __ldg(rp + 1); }
                                if (prm.res_relu) rs[c] = make_float2(relu_nan(rs[c].x), relu_nan(rs[c].y));
                            }
                        }
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            if (kbase + cg + c >= prm.K) continue;
                            float v0 = y[2 * a][cg + c], v1 = y[2 * a + 1][cg + c];
                            if (EXTRAS && prm.out_scale) {
                                const float s1 = __ldg(prm.out_scale + kbase + cg + c), b1 = __ldg(prm.out_shift + kbase + cg + c);
                                v0 = fmaf(v0, s1, b1); v1 = fmaf(v1, s1, b1);
                            }
                            if (EXTRAS) { v0 += rs[c].x; v1 += rs[c].y; }
                            float *dst = prm.Y + o0 + (cg + c) * cstride;
                            if (pair) *reinterpret_cast<float2 *>(dst) = make_float2(v0, v1);
                            else { dst[0] = v0; if (2 * tw + 1 < prm.outW) dst[1] = v1; }
                        }
                    }
                }
            }
            if (ew == 0 && lane == 0) TC_TRACE(1536 + 4 * (tr - 1) + 3);
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
    if (threadIdx.x == 0) TC_TRACE(4095);
}

// ---------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------
// Poll limit of the bounded waits and the one-shot test hook, handed to every launch through its parameters.
static std::atomic<uint32_t> g_wait_limit{kSpinLimit};
static std::atomic<int> g_drop_load{-1};

int tc_set_wait_limit(long long polls)
{
    if (polls < 0 || polls > 0xFFFFFFFFLL) return WG2X2_ERR_BAD_ARG;
    g_wait_limit.store(polls == 0 ? kSpinLimit : (uint32_t)polls);
    return WG2X2_OK;
}
int tc_test_drop_load(int nth)
{
    g_drop_load.store(nth < 0 ? -1 : nth);
    return WG2X2_OK;
}
static uint32_t wait_limit() { return g_wait_limit.load(); }
static int take_drop_load() { return g_drop_load.exchange(-1); }   // consumed by the next launch that looks at it

// Smallest possible exercise of the bounded wait: one thread waits on a barrier nobody arrives on.
__global__ void wait_probe_kernel(uint32_t limit, unsigned where)
{
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&bar), 1);
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        mbar_wait(smem_u32(&bar), 0, &abort_flag, where, limit);
    }
}
int tc_wait_probe(long long polls, unsigned where, cudaStream_t st)
{
    if (polls <= 0 || polls > (long long)kSpinLimit) return WG2X2_ERR_BAD_ARG;
    wait_probe_kernel<<<1, 32, 0, st>>>((uint32_t)polls, where);
    return launch_status();
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn_raw()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// cuTensorMapEncodeTiled behind a small per-thread cache keyed by every argument: a layer that is called again on
// the same buffers (the usual case: a network's activations live at fixed addresses from step to step) finds its
// maps instead of encoding up to five of them per launch, which matters where a launch is only a few microseconds
// of GPU time.  A tensor map holds no state but its arguments, so a hit is exact.
struct MapKey {
    const void *ptr;
    cuuint64_t dims[5], strides[4];
    cuuint32_t box[5], estr[5];
    int rank, dtype, interleave, swizzle, promo, oob;
};
static CUresult encode_cached(CUtensorMap *map, CUtensorMapDataType dtype, cuuint32_t rank, void *ptr, const cuuint64_t *dims,
                              const cuuint64_t *strides, const cuuint32_t *box, const cuuint32_t *estr, CUtensorMapInterleave il,
                              CUtensorMapSwizzle sw, CUtensorMapL2promotion promo, CUtensorMapFloatOOBfill oob)
{
    constexpr int kEntries = 64;
    struct Entry { MapKey key; CUtensorMap map; bool used; };
    thread_local Entry cache[kEntries];
    thread_local int next = 0;
    if (rank < 1 || rank > 5) return CUDA_ERROR_INVALID_VALUE;
    MapKey k;
    memset(&k, 0, sizeof(k));
    k.ptr = ptr; k.rank = (int)rank; k.dtype = (int)dtype; k.interleave = (int)il; k.swizzle = (int)sw; k.promo = (int)promo; k.oob = (int)oob;
    for (cuuint32_t d = 0; d < rank; ++d) { k.dims[d] = dims[d]; k.box[d] = box[d]; k.estr[d] = estr[d]; }
    for (cuuint32_t d = 0; d + 1 < rank; ++d) k.strides[d] = strides[d];
    for (int e = 0; e < kEntries; ++e)
        if (cache[e].used && memcmp(&cache[e].key, &k, sizeof(k)) == 0) { *map = cache[e].map; return CUDA_SUCCESS; }
    EncodeTiledFn fn = encode_fn_raw();
    if (!fn) return CUDA_ERROR_NOT_SUPPORTED;
    CUresult r = fn(map, dtype, rank, ptr, dims, strides, box, estr, il, sw, promo, oob);
    // a driver call on a thread that has not yet run anything on the device finds no context (an autograd thread whose
    // first call is this one): have the runtime bind it and ask again
    if ((r == CUDA_ERROR_INVALID_CONTEXT || r == CUDA_ERROR_NOT_INITIALIZED) && cudaFree(nullptr) == cudaSuccess)
        r = fn(map, dtype, rank, ptr, dims, strides, box, estr, il, sw, promo, oob);
    if (r == CUDA_SUCCESS) {
        Entry &en = cache[next];
        next = (next + 1) % kEntries;
        en.key = k; en.map = *map; en.used = true;
    }
    return r;
}
static EncodeTiledFn encode_fn() { return encode_fn_raw() ? &encode_cached : nullptr; }

// Dense fp32 map with unit element strides, for the kernels of the other source files
bool tensor_map_f32(CUtensorMap *map, int rank, const float *ptr, const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box,
                    CUtensorMapSwizzle swizzle)
{
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    EncodeTiledFn fn = encode_fn();
    return fn && fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank, const_cast<float *>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The status word of the current device, for those kernels' bounded waits (NULL: it cannot be had)
unsigned int *tc_status_word()
{
    static std::atomic<unsigned int *> known[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    unsigned int *p = known[dev].load(std::memory_order_acquire);
    if (!p) {
        void *a = nullptr;
        if (cudaGetSymbolAddress(&a, g_tc_status) != cudaSuccess) return nullptr;
        p = static_cast<unsigned int *>(a);
        known[dev].store(p, std::memory_order_release);
    }
    return p;
}
uint32_t tc_wait_limit() { return wait_limit(); }

// 3-D map over a (16, rows, C) fp32 tensor, C contiguous: box = 32 x box_rows x 1, 128-B swizzle,
// out-of-range elements read as zero.
static bool make_map(CUtensorMap *map, const float *ptr, int C, long long rows, int box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)C, (cuuint64_t)rows, 16};
    cuuint64_t strides[2] = {(cuuint64_t)C * 4, (cuuint64_t)rows * C * 4};
    cuuint32_t box[3] = {(cuuint32_t)kBlockK, (cuuint32_t)box_rows, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

size_t prepared_weights_bytes(int C, int K)
{
    const size_t w = align_up((size_t)16 * K * C * sizeof(float), 256);
    const size_t f = align_up((size_t)16 * cdiv(K, kBlockN) * sizeof(unsigned long long), 256);
    return w + f;
}

bool tc_shape_supported(int C, int K) { return C % 4 == 0 && C >= 4 && K >= 1; }

int weights_prepare(const float *Wt, int C, int K, void *prepared, size_t bytes, cudaStream_t st)
{
    if (!Wt || !prepared || C <= 0 || K <= 0) return WG2X2_ERR_BAD_ARG;
    if (!tc_shape_supported(C, K)) return WG2X2_ERR_UNSUPPORTED;
    if (bytes < prepared_weights_bytes(C, K)) return WG2X2_ERR_WORKSPACE;
    if (reinterpret_cast<uintptr_t>(prepared) & 255u) return WG2X2_ERR_BAD_ARG;
    const int nKB = cdiv(K, kBlockN), nCC = cdiv(C, kBlockK);
    float *Wp = static_cast<float *>(prepared);
    unsigned long long *masks = reinterpret_cast<unsigned long long *>(static_cast<unsigned char *>(prepared) +
                                                                       align_up((size_t)16 * K * C * sizeof(float), 256));
    return launch(pack_weights_kernel, dim3(nKB, cdiv(C, kPackC), 16), kPackThreads, 0, st, Wt, Wp, masks, C, K, nKB, nCC);
}

// Launcher.  `contr` = contraction length C, `ncols` = output channels K; A is (16, P, contr), Bop is
// (16, ncols, contr), both contraction-contiguous.
static int tc_launch(int layout, const float *A, const float *Bop, const unsigned long long *masks, float *out, long long P,
                     int nH, int nW, int contr, int ncols, int outH, int outW, const float *out_scale, const float *out_shift,
                     const float *residual, int res_relu, cudaStream_t st)
{
    if (P > 0x7fffffffLL - kBlockM) return WG2X2_ERR_UNSUPPORTED;
    TcParams prm;
    prm.Y = out;
    prm.out_scale = out_scale; prm.out_shift = out_shift; prm.residual = residual; prm.res_relu = res_relu;
    prm.masks = masks;
    prm.P = P; prm.nH = nH; prm.nW = nW; prm.C = contr; prm.K = ncols; prm.outH = outH; prm.outW = outW;
    prm.nKB = cdiv(ncols, kBlockN);
    prm.nCC = cdiv(contr, kBlockK);
    // Tiles per unit: 128 fills every TMEM lane, but a unit count that is not a multiple of the SM
    // count leaves SMs idle in the last round.  When there is more than one round of work, shrink
    // the units a little so that they divide evenly (the TMA box still brings 128 rows; the extra
    // rows are the neighbouring unit's and cost L2 bandwidth only).
    prm.tpu = kBlockM;
    const long long min_units = cdivll(P, kBlockM) * prm.nKB;
    if (min_units > kNumSMs) {
        const long long rounds = cdivll(min_units, kNumSMs);
        const long long want_mt = (rounds * kNumSMs) / prm.nKB;
        if (want_mt > 0) {
            const long long t = cdivll(P, want_mt);
            if (t >= 32 && t <= kBlockM) prm.tpu = (int)t;
        }
    }
    prm.nMT = (int)cdivll(P, prm.tpu);
    prm.units = prm.nMT * prm.nKB;
    prm.spin_limit = wait_limit();
    prm.drop_load = take_drop_load();
    CUtensorMap mapA, mapB;
    if (!make_map(&mapA, A, contr, P, kBlockM)) return WG2X2_ERR_LAUNCH;
    if (!make_map(&mapB, Bop, contr, ncols, kBlockN)) return WG2X2_ERR_LAUNCH;
    const int grid = prm.units < kNumSMs ? prm.units : kNumSMs;
    const bool extras = out_scale || residual;
    auto *kernel = layout == WG2X2_NHWC ? (extras ? conv_fwd_tc_kernel<WG2X2_NHWC, true> : conv_fwd_tc_kernel<WG2X2_NHWC, false>)
                                        : (extras ? conv_fwd_tc_kernel<WG2X2_NCHW, true> : conv_fwd_tc_kernel<WG2X2_NCHW, false>);
    return launch(kernel, dim3((unsigned)grid), kFwdThreads, kSmemBytes, st, mapA, mapB, prm);
}

int conv_fwd_tc_prepared(const float *V, const void *prepared, float *Y, int B, int nH, int nW, int C, int K, int outH, int outW,
                         int layout, const float *out_scale, const float *out_shift, const float *residual, int res_relu, cudaStream_t st)
{
    if (!V || !prepared || !Y) return WG2X2_ERR_BAD_ARG;
    if ((out_scale == nullptr) != (out_shift == nullptr)) return WG2X2_ERR_BAD_ARG;
    if (out_scale && ((reinterpret_cast<uintptr_t>(out_scale) & 15u) || (reinterpret_cast<uintptr_t>(out_shift) & 15u))) return WG2X2_ERR_BAD_ARG;
    if (residual && (reinterpret_cast<uintptr_t>(residual) & 15u)) return WG2X2_ERR_BAD_ARG;
    if (!tc_shape_supported(C, K)) return WG2X2_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(V) & 15u) || (reinterpret_cast<uintptr_t>(Y) & 15u)) return WG2X2_ERR_BAD_ARG;
    const unsigned long long *masks = reinterpret_cast<const unsigned long long *>(
        static_cast<const unsigned char *>(prepared) + align_up((size_t)16 * K * C * sizeof(float), 256));
    return tc_launch(layout, V, static_cast<const float *>(prepared), masks, Y, (long long)B * nH * nW, nH, nW, C, K, outH, outW,
                     out_scale, out_shift, residual, res_relu, st);
}

bool conv_fwd_wide_preferred(long long P, int C, int K);
size_t conv_fwd_wide_workspace_bytes(long long P, int K);
int conv_fwd_tc_wide(const float *V, const void *prepared, float *Y, int B, int nH, int nW, int C, int K, int outH, int outW,
                     int layout, const float *out_scale, const float *out_shift, const float *residual, int res_relu, void *ws,
                     size_t ws_bytes, cudaStream_t st);

size_t conv_fwd_tc_workspace_bytes(int B, int nH, int nW, int C, int K)
{
    if (C <= 0 || K <= 0 || B <= 0 || nH <= 0 || nW <= 0) return 0;
    size_t n = prepared_weights_bytes(C, K);
    if (conv_fwd_wide_preferred((long long)B * nH * nW, C, K)) n += conv_fwd_wide_workspace_bytes((long long)B * nH * nW, K);
    return n;
}

int conv_fwd_tc(const float *V, const float *Wt, float *Y, int B, int nH, int nW, int C, int K, int outH, int outW, int layout,
                void *ws, size_t ws_bytes, cudaStream_t st)
{
    if (!tc_shape_supported(C, K)) return WG2X2_ERR_UNSUPPORTED;
    if (!ws || ws_bytes < prepared_weights_bytes(C, K)) return WG2X2_ERR_WORKSPACE;
    const int s = weights_prepare(Wt, C, K, ws, ws_bytes, st);
    if (s != WG2X2_OK) return s;
    const size_t pb = prepared_weights_bytes(C, K);
    if (conv_fwd_wide_preferred((long long)B * nH * nW, C, K) && ws_bytes >= pb + conv_fwd_wide_workspace_bytes((long long)B * nH * nW, K))
        return conv_fwd_tc_wide(V, ws, Y, B, nH, nW, C, K, outH, outW, layout, nullptr, nullptr, nullptr, 0,
                                static_cast<char *>(ws) + pb, ws_bytes - pb, st);
    return conv_fwd_tc_prepared(V, ws, Y, B, nH, nW, C, K, outH, outW, layout, nullptr, nullptr, nullptr, 0, st);
}

void dw_reduce_launch(const float *partial, const float *mask, float *dW, long long n, int splits, cudaStream_t st);  // conv_ffma.cu

#include "conv_tc_bwd.cuh"
#include "conv_tc_cluster.cuh"
#include "conv_tc_fused.cuh"
#include "conv_tc_pair.cuh"
#include "stem_tc.cuh"
#include "conv1x1_tc.cuh"

#if defined(WG_TC_TRACE) || defined(WG_TC_DIAG)   // development builds only
extern "C" int wg2x2_debug_read_diag(unsigned int *host)
{
    cudaDeviceSynchronize();
    return cudaMemcpyFromSymbol(host, g_tc_diag, sizeof(unsigned int) * 32) == cudaSuccess ? 0 : -1;
}
#endif
#ifdef WG_TC_TRACE
extern "C" int wg2x2_debug_read_trace(long long *host, int n)
{
    cudaDeviceSynchronize();
    return cudaMemcpyFromSymbol(host, g_tc_trace, sizeof(long long) * (n < 4096 ? n : 4096)) == cudaSuccess ? 0 : -1;
}
#endif

int tc_last_device_status(cudaStream_t st, unsigned int *where)
{
    if (cudaStreamSynchronize(st) != cudaSuccess) return WG2X2_ERR_LAUNCH;
    unsigned int h[2] = {0, 0};
    if (cudaMemcpyFromSymbol(h, g_tc_status, sizeof(h)) != cudaSuccess) return WG2X2_ERR_LAUNCH;
    if (where) *where = h[1];
    if (h[0]) {
        const unsigned int z[2] = {0, 0};
        cudaMemcpyToSymbol(g_tc_status, z, sizeof(z));
        return WG2X2_ERR_TIMEOUT;
    }
    return WG2X2_OK;
}

}  // namespace wg

extern "C" int wg2x2_conv1x1_preferred(int B, int C, int K, int HW)
{
    return (B > 0 && C > 0 && K > 0 && HW > 0 && wg::conv1x1_preferred(B, C, K, HW)) ? 1 : 0;
}
extern "C" int wg2x2_conv1x1(const float *X, const float *W, float *Y, int B, int C, int K, int HW, void *stream)
{
    return wg::conv1x1(X, W, Y, B, C, K, HW, (cudaStream_t)stream);
}

extern "C" int wg2x2_stem_prepared_floats(void) { return wg::kStWtFloats; }

extern "C" int wg2x2_stem_prepare(const float *W, float *Wp, void *stream) { return wg::stem_prepare(W, Wp, (cudaStream_t)stream); }

extern "C" int wg2x2_stem7x7s2_pool(const float *X, const float *Wp, float *Y, float *Y_relu, const float *relu_scale,
                                    const float *relu_shift, int B, int H, int W, void *stream)
{
    return wg::stem_pool(X, Wp, Y, Y_relu, relu_scale, relu_shift, B, H, W, (cudaStream_t)stream);
}
