// FP32 (CUDA-core) kernels of the Winograd-domain product: the exact-arithmetic path (max rel err <= 1e-5 against
// float64) that the tensor-core path is validated against, and the default precision of the layer wrappers.
//
//   conv_fwd_ffma : Y    = A^T (V_t . W_t) A         rows = tiles, columns = out-channels, contraction over in-channels
//   conv_dv_ffma  : dV_t = (A dY A^T)_t . W_t^T      rows = tiles, columns = in-channels,  contraction over out-channels
//   conv_dw_ffma  : dW_t = V_t^T . (A dY A^T)_t      rows = in-channels, columns = out-channels, contraction over tiles (split)
//
// One structure for all three.  A CTA owns one block of rows x 32 columns of all sixteen products and has sixteen warps, one
// per Winograd position: a warp computes its position's product, 8 * MT rows (MT = 8, 4, 2) x 32 columns, MT x 8 values per
// thread.  Operands arrive by TMA, two stages of 16 contraction
// steps (by 4-byte asynchronous copies where a row is not a multiple of 16 bytes).  Nothing is shared between positions, so the forward kernel's loop has no CTA-wide barrier; its sixteen products
// meet in shared memory once, at the end, where A^T m A is applied.  The gradients of Y enter the other two as dM = A dY A^T:
// the four pixels of every tile are staged once per CTA, and eight of the sixteen warps in turn (the first and the second
// half on alternate stages) turn the next stage's pixels into its sixteen operand tiles while all of them compute.  No
// product tensor M or dM is ever written to memory.
//
// Bound: the FP32 pipe (128 FMA per SM and clock).  Per 4 contraction steps a warp with MT = 8 issues 256 FMAs against 16
// shared-memory loads of 16 bytes.  (The packed fma.rn.f32x2 is no faster: 2.5 clocks each with its operands in the best
// order, 3.8 otherwise, against 1.14 for a plain FMA of half the work, measured with four warps per scheduler.)
#include <cuda.h>

#include "wg_common.cuh"

namespace wg {

constexpr int kFfWarps = 16;              // one per Winograd position
constexpr int kFfThreads = 32 * kFfWarps;
constexpr int kFfKC = 16;                 // contraction steps per stage
constexpr int kFfN = 32;                  // columns per CTA
constexpr int kFfB = kFfKC * kFfN;        // floats of a position's B tile
constexpr int kFfCtrl = 2048;             // alignment slack, then two barriers per warp
template <int MT> struct FfTile {
    static constexpr int M = 8 * MT;                    // rows per CTA
    static constexpr int A = M * kFfKC;                 // floats of a position's A tile
    static constexpr int kMP = kFfN + 4;                // pitch of a row of products in shared memory (forward)
    static constexpr int kRawRows = 4 * M * kFfKC;      // floats of the staged pixels: dV ...
    static constexpr int kRawCols = 4 * kFfKC * kFfN;   // ... and dW
    static constexpr int kOperands = 2 * kFfWarps * (A + kFfB);
    static constexpr int kFold = kFfWarps * M * kMP;
    static constexpr int kFwdBytes = kFfCtrl + (kOperands > kFold ? kOperands : kFold) * (int)sizeof(float);
    static constexpr int kDvBytes = kFfCtrl + (kOperands + 2 * kRawRows > kFold ? kOperands + 2 * kRawRows : kFold) * (int)sizeof(float);
    static constexpr int kDwBytes = kFfCtrl + (kOperands + 2 * kRawCols > kFold ? kOperands + 2 * kRawCols : kFold) * (int)sizeof(float);
    static_assert(kFwdBytes <= 232448 && kDvBytes <= 232448 && kDwBytes <= 232448, "shared memory per CTA");
};

// index of image-like tensor element (b, h, w, ch) for a tensor with `Cn` channels
template <int LAYOUT>
static __device__ __forceinline__ long long img_index(int b, int h, int w, int ch, int Hh, int Ww, int Cn)
{
    return LAYOUT == WG2X2_NHWC ? (((long long)b * Hh + h) * Ww + w) * Cn + ch
                                : (((long long)b * Cn + ch) * Hh + h) * Ww + w;
}

struct FfGrid {
    long long P;
    int nH, nW, H, W;      // tile grid and true image size
};
static __device__ __forceinline__ void decode_tile(const FfGrid &g, long long p, int &b, int &th, int &tw)
{
    if (g.P <= 0x7fffffffLL) {
        const unsigned q = (unsigned)p, r = q / (unsigned)g.nW;
        tw = (int)(q - r * (unsigned)g.nW);
        b = (int)(r / (unsigned)g.nH);
        th = (int)(r - (unsigned)b * (unsigned)g.nH);
    } else {
        tw = (int)(p % g.nW);
        th = (int)((p / g.nW) % g.nH);
        b = (int)(p / ((long long)g.nW * g.nH));
    }
}

// asynchronous copies to shared memory; what lies beyond the matrix (ok == false, or beyond `have` floats) arrives as zeros
static __device__ __forceinline__ void cp16(float *dst, const float *src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
static __device__ __forceinline__ void cp4(float *dst, const float *src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
// four floats, `have` of them in the matrix (a source that is not read still has to be an address of it: `any`)
template <bool VEC>
static __device__ __forceinline__ void copy4(float *dst, const float *src, int have, const float *any)
{
    if (VEC) {
        cp16(dst, have > 0 ? src : any, have > 0);
    } else {
#pragma unroll
        for (int q = 0; q < 4; ++q) cp4(dst + q, have > q ? src + q : any, have > q);
    }
}
static __device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
static __device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// TMA boxes of a (16, rows, columns) matrix, and the warp's wait for one.  The wait is bounded as everywhere in this library;
// one that runs out leaves a note in the status word and gives the copy a last millisecond, and the warp goes on (its results are then
// incomplete).
static __device__ __forceinline__ uint32_t ff_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
static __device__ __forceinline__ void ff_tma(float *dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2)
{
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(ff_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
static __device__ __forceinline__ void ff_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
static __device__ __forceinline__ void ff_wait(uint32_t bar, uint32_t parity, unsigned int *status, uint32_t limit)
{
    for (uint32_t it = 0; it < limit; ++it) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return;
    }
    status[1] = 0x1E00u;
    status[0] = 1;
    for (int it = 0; it < 1000; ++it) __nanosleep(1000);
}
struct FfWait {
    unsigned int *status;      // the library's status word
    uint32_t limit;            // polls before a wait gives up
};
// the dynamic shared memory, on the boundary the swizzles want, and the warp's two barriers
static __device__ __forceinline__ float *ff_shared(uint32_t &bar)
{
    extern __shared__ __align__(16) uint8_t ff_smem[];
    const uint32_t a = ff_u32(ff_smem), up = (a + 1023u) & ~1023u;
    bar = up + 16u * (threadIdx.x >> 5);
    if ((threadIdx.x & 31) == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar + 8));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncwarp();
    return reinterpret_cast<float *>(ff_smem + (up - a) + 1024);
}

template <bool VEC>
static __device__ __forceinline__ float4 load4(const float *p, int have)
{
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (VEC) {
        if (have > 0) v = __ldg(reinterpret_cast<const float4 *>(p));
    } else {
        if (have > 0) v.x = __ldg(p);
        if (have > 1) v.y = __ldg(p + 1);
        if (have > 2) v.z = __ldg(p + 2);
        if (have > 3) v.w = __ldg(p + 3);
    }
    return v;
}
template <bool VEC>
static __device__ __forceinline__ void store4(float *p, int have, float a, float b, float c, float d)
{
    if (VEC) {
        if (have > 0) *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, d);
    } else {
        if (have > 0) p[0] = a;
        if (have > 1) p[1] = b;
        if (have > 2) p[2] = c;
        if (have > 3) p[3] = d;
    }
}

// ------------------------------------------------------------------------------------------
// Operand tiles in shared memory.
//   "by rows"  [row][16 steps]  : the 16-byte group g of row r sits at g ^ ((r >> 1) & 3)  (TMA's 64-byte swizzle)
//   "by steps" [step][columns]  : B with its 16-byte group g of step k at g ^ (k & 7)      (the 128-byte swizzle); A of dW plainly
// The XORs keep the rows of an access on different banks.
// ------------------------------------------------------------------------------------------
static __device__ __forceinline__ int at_row(int r, int g) { return r * kFfKC + ((g ^ ((r >> 1) & 3)) << 2); }
static __device__ __forceinline__ int at_step(int k, int g) { return k * kFfN + ((g ^ (k & 7)) << 2); }

// Without TMA: a warp's copy of rows row0 .. row0 + ROWS - 1, steps k .. k + 15 of src[row][K] (steps contiguous), by rows
template <int ROWS>
static __device__ __forceinline__ void copy_rows(float *dst, const float *src, long long row0, long long rows, int K, int k)
{
    const int lane = threadIdx.x & 31, g = lane & 3;
    for (int r = lane >> 2; r < ROWS; r += 8)
        copy4<false>(dst + at_row(r, g), src + (row0 + r) * K + k + 4 * g, row0 + r < rows ? K - k - 4 * g : 0, src);
}
// and of steps k .. k + 15, columns c0 .. of src[step][cols] (columns contiguous), by steps
template <int COLS, bool SWIZZLE>
static __device__ __forceinline__ void copy_steps(float *dst, const float *src, long long k, long long kend, int c0, int cols)
{
    constexpr int G = COLS / 4;
    for (int e = threadIdx.x & 31; e < kFfKC * G; e += 32) {
        const int s = e / G, g = e % G, c = c0 + 4 * g;
        copy4<false>(dst + (SWIZZLE ? at_step(s, g) : s * COLS + 4 * g), src + (k + s) * cols + c, k + s < kend ? cols - c : 0, src);
    }
}

// ------------------------------------------------------------------------------------------
// The product of one warp.  Lane (lm = lane >> 2, ln = lane & 3) owns MT rows and 8 columns of the block:
//   A by rows: rows lm + 8 m           A by steps: rows 4 lm + (m & 3) of every 32 (MT = 2: 2 lm + m)
//   B by rows: columns ln + 4 n        B by steps: columns 4 ln + (n & 3) of every 16
// ------------------------------------------------------------------------------------------
template <int MT, bool A_ROWS, bool B_ROWS>
struct WarpTile {
    float acc[MT][8];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < 8; ++n) acc[m][n] = 0.f;
    }
    // one step with the operands in registers
    __device__ __forceinline__ void step(const float *B, int k, const float (&a)[MT])
    {
        const int ln = threadIdx.x & 3;
        const float4 b0 = *reinterpret_cast<const float4 *>(B + at_step(k, ln)), b1 = *reinterpret_cast<const float4 *>(B + at_step(k, ln + 4));
        const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < 8; ++n) acc[m][n] = fmaf(a[m], b[n], acc[m][n]);
    }
    __device__ __forceinline__ void chunk(const float *A, const float *B)
    {
        const int lm = (threadIdx.x & 31) >> 2, ln = threadIdx.x & 3;
        if (A_ROWS && B_ROWS) {
#pragma unroll
            for (int g = 0; g < kFfKC / 4; ++g) {
                float4 b[8];
#pragma unroll
                for (int n = 0; n < 8; ++n) b[n] = *reinterpret_cast<const float4 *>(B + at_row(ln + 4 * n, g));
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    const float4 a = *reinterpret_cast<const float4 *>(A + at_row(lm + 8 * m, g));
#pragma unroll
                    for (int n = 0; n < 8; ++n) acc[m][n] = fmaf(a.x, b[n].x, acc[m][n]);
#pragma unroll
                    for (int n = 0; n < 8; ++n) acc[m][n] = fmaf(a.y, b[n].y, acc[m][n]);
#pragma unroll
                    for (int n = 0; n < 8; ++n) acc[m][n] = fmaf(a.z, b[n].z, acc[m][n]);
#pragma unroll
                    for (int n = 0; n < 8; ++n) acc[m][n] = fmaf(a.w, b[n].w, acc[m][n]);
                }
            }
        } else if (A_ROWS) {
#pragma unroll
            for (int g = 0; g < kFfKC / 4; ++g) {
                float4 a4[MT];
#pragma unroll
                for (int m = 0; m < MT; ++m) a4[m] = *reinterpret_cast<const float4 *>(A + at_row(lm + 8 * m, g));
                float a[MT];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
#pragma unroll
                    for (int m = 0; m < MT; ++m) a[m] = q == 0 ? a4[m].x : q == 1 ? a4[m].y : q == 2 ? a4[m].z : a4[m].w;
                    step(B, 4 * g + q, a);
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < kFfKC; ++k) {
                float a[MT];
                if (MT >= 4) {
#pragma unroll
                    for (int h = 0; h < MT / 4; ++h) {
                        const float4 v = *reinterpret_cast<const float4 *>(A + k * 8 * MT + 32 * h + 4 * lm);
                        a[4 * h] = v.x; a[4 * h + 1] = v.y; a[4 * h + 2] = v.z; a[4 * h + 3] = v.w;
                    }
                } else {
                    const float2 v = *reinterpret_cast<const float2 *>(A + k * 8 * MT + 2 * lm);
                    a[0] = v.x; a[1] = v.y;
                }
                step(B, k, a);
            }
        }
    }
    // the block of products to shared memory, [row][column] with a pitch of kMP
    __device__ __forceinline__ void put(float *d) const
    {
        const int lm = (threadIdx.x & 31) >> 2, ln = threadIdx.x & 3;
        constexpr int MP = FfTile<MT>::kMP;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            float *r = d + (A_ROWS ? lm + 8 * m : (MT >= 4 ? 32 * (m >> 2) + 4 * lm + (m & 3) : 2 * lm + m)) * MP;
            if (B_ROWS) {
#pragma unroll
                for (int n = 0; n < 8; ++n) r[ln + 4 * n] = acc[m][n];
            } else {
                *reinterpret_cast<float4 *>(r + 4 * ln) = make_float4(acc[m][0], acc[m][1], acc[m][2], acc[m][3]);
                *reinterpret_cast<float4 *>(r + 16 + 4 * ln) = make_float4(acc[m][4], acc[m][5], acc[m][6], acc[m][7]);
            }
        }
    }
};

// ------------------------------------------------------------------------------------------
// Forward
// ------------------------------------------------------------------------------------------
template <int MT, bool VEC, int LAYOUT>
__global__ void __launch_bounds__(kFfThreads, 1) conv_fwd_ffma_kernel(const __grid_constant__ CUtensorMap mapV,
                                                                       const __grid_constant__ CUtensorMap mapW, const float *__restrict__ V,
                                                                       const float *__restrict__ Wt, float *__restrict__ Y, FfGrid g, int C,
                                                                       int K, FfWait wt)
{
    after_previous_kernel(V, Wt, Y);
    using T = FfTile<MT>;
    uint32_t bar;
    float *smem = ff_shared(bar);
    const int t = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long p0 = (long long)blockIdx.x * T::M;
    const int k0 = blockIdx.y * kFfN;
    WarpTile<MT, true, false> w;
    w.clear();
    {
        float *stage = smem + t * 2 * (T::A + kFfB);
        auto fetch = [&](int buf, int c) {
            float *A = stage + buf * (T::A + kFfB), *B = A + T::A;
            if (VEC) {
                if (lane == 0) {
                    ff_expect(bar + 8 * buf, (T::A + kFfB) * 4);
                    ff_tma(A, &mapV, bar + 8 * buf, c, (int)p0, t);
                    ff_tma(B, &mapW, bar + 8 * buf, k0, c, t);
                }
            } else {
                copy_rows<T::M>(A, V + (long long)t * g.P * C, p0, g.P, C, c);
                copy_steps<kFfN, true>(B, Wt + (long long)t * C * K, c, C, k0, K);
                cp_commit();
            }
        };
        fetch(0, 0);
        int buf = 0;
        uint32_t ph = 0;
#pragma unroll 1
        for (int c = 0; c < C; c += kFfKC) {
            if (VEC) ff_wait(bar + 8 * buf, ph, wt.status, wt.limit); else cp_wait_all();
            __syncwarp();                  // this stage has landed for every lane, and every lane is done with the other one
            if (c + kFfKC < C) fetch(buf ^ 1, c + kFfKC);
            w.chunk(stage + buf * (T::A + kFfB), stage + buf * (T::A + kFfB) + T::A);
            buf ^= 1;
            ph ^= (uint32_t)(buf == 0);
        }
    }
    __syncthreads();                       // every warp is done with its stages: the products take their place
    w.put(smem + t * T::M * T::kMP);
    __syncthreads();
    // A^T m A: one tile x 4 channels at a time.  NHWC: channels fastest over the threads (128-byte runs of Y), NCHW: tiles
    // fastest (pairs of pixels along the image row).
    for (int e = threadIdx.x; e < T::M * (kFfN / 4); e += kFfThreads) {
        const int row = LAYOUT == WG2X2_NHWC ? e >> 3 : e % T::M;
        const int c4 = LAYOUT == WG2X2_NHWC ? e & 7 : e / T::M;
        const long long p = p0 + row;
        const int k = k0 + 4 * c4;
        if (p >= g.P || k >= K) continue;
        float4 y[2][2];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float4 m[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                m[j] = *reinterpret_cast<const float4 *>(smem + ((4 * i + j) * T::M + row) * T::kMP + 4 * c4);
            const float4 z0 = m[0] + m[1] + m[2], z1 = m[1] - m[2] - m[3];
            if (i == 0) { y[0][0] = z0; y[0][1] = z1; }
            if (i == 1) { y[0][0] = y[0][0] + z0; y[0][1] = y[0][1] + z1; y[1][0] = z0; y[1][1] = z1; }
            if (i == 2) { y[0][0] = y[0][0] + z0; y[0][1] = y[0][1] + z1; y[1][0] = y[1][0] - z0; y[1][1] = y[1][1] - z1; }
            if (i == 3) { y[1][0] = y[1][0] - z0; y[1][1] = y[1][1] - z1; }
        }
        int b, th, tw;
        decode_tile(g, p, b, th, tw);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const int h = 2 * th + a, x = 2 * tw + s;
                if (h >= g.H || x >= g.W) continue;
                float *dst = Y + img_index<LAYOUT>(b, h, x, k, g.H, g.W, K);
                if (LAYOUT == WG2X2_NHWC && VEC) {
                    *reinterpret_cast<float4 *>(dst) = y[a][s];
                } else {
                    const long long sk = LAYOUT == WG2X2_NHWC ? 1 : (long long)g.H * g.W;
                    dst[0] = y[a][s].x;
                    if (k + 1 < K) dst[sk] = y[a][s].y;
                    if (k + 2 < K) dst[2 * sk] = y[a][s].z;
                    if (k + 3 < K) dst[3 * sk] = y[a][s].w;
                }
            }
    }
}

// The sixteen dM values of four channels from the four pixels of a tile: put(t, value)
template <typename Get, typename Put>
static __device__ __forceinline__ void build_dm(Get pixel, Put put)
{
    const float4 g00 = pixel(0), g01 = pixel(1), g10 = pixel(2), g11 = pixel(3);
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 u0 = i == 0 ? g00 : i == 1 ? g00 + g10 : i == 2 ? g00 - g10 : z - g10;
        const float4 u1 = i == 0 ? g01 : i == 1 ? g01 + g11 : i == 2 ? g01 - g11 : z - g11;
        put(4 * i, u0);
        put(4 * i + 1, u0 + u1);
        put(4 * i + 2, u0 - u1);
        put(4 * i + 3, z - u1);
    }
}

// The loop of the two gradient kernels.  At the top of stage n the pixels of stage n + 1 and this stage's other operand have
// landed and dM of stage n is built; then the copies of the next stages are issued, half of the warps build dM of stage
// n + 1, and everybody computes stage n.
template <typename CopyRaw, typename CopyOther, typename WaitOther, typename Build, typename Compute>
static __device__ __forceinline__ void gradient_loop(int nstages, CopyRaw copy_raw, CopyOther copy_other, WaitOther wait_other, Build build,
                                                     Compute compute)
{
    if (nstages <= 0) return;
    copy_raw(0, 0);
    copy_other(0, 0);
    cp_commit();
    cp_wait_all();
    __syncthreads();
    if (nstages > 1) copy_raw(1, 1);
    cp_commit();
    if (threadIdx.x < kFfThreads / 2) build(0);
#pragma unroll 1
    for (int n = 0; n < nstages; ++n) {
        const int buf = n & 1;
        cp_wait_all();
        __syncthreads();
        if (n + 2 < nstages) copy_raw(buf, n + 2);
        if (n + 1 < nstages) {
            copy_other(buf ^ 1, n + 1);
            if ((threadIdx.x < kFfThreads / 2) == ((n & 1) != 0)) build(buf ^ 1);
        }
        cp_commit();
        wait_other(buf, (uint32_t)(n >> 1) & 1u);
        compute(buf);
    }
}

// The gradient kernels' results leave through shared memory: rows of 32 columns, 16 bytes per thread.  first: index of the
// block's first element in the position's plane; finish(offset, values) applies a mask.
template <int MT, bool VEC, typename Warp, typename Finish>
static __device__ __forceinline__ void store_block(const Warp &w, float *smem, float *plane, long long row0, long long rows, int col0, int cols,
                                                   Finish finish)
{
    using T = FfTile<MT>;
    __syncthreads();                       // every warp is done with its operands
    float *d = smem + (threadIdx.x >> 5) * T::M * T::kMP;
    w.put(d);
    __syncwarp();
    const int lane = threadIdx.x & 31, c = col0 + 4 * (lane & 7);
#pragma unroll
    for (int r = lane >> 3; r < T::M; r += 4) {
        if (row0 + r >= rows || c >= cols) continue;
        const long long o = (row0 + r) * cols + c;
        float4 v = *reinterpret_cast<const float4 *>(d + r * T::kMP + 4 * (lane & 7));
        v = finish(o, cols - c, v);
        store4<VEC>(plane + o, cols - c, v.x, v.y, v.z, v.w);
    }
}

// ------------------------------------------------------------------------------------------
// dV_t[p][c] = sum_k dM_t[p][k] W_t[c][k]   (optionally zeroed where the saved V <= 0)
// ------------------------------------------------------------------------------------------
template <int MT, bool VEC, int LAYOUT>
__global__ void __launch_bounds__(kFfThreads, 1) conv_dv_ffma_kernel(const __grid_constant__ CUtensorMap mapW, const float *__restrict__ Vsaved,
                                                                      const float *__restrict__ Wt, const float *__restrict__ dY,
                                                                      float *__restrict__ dV, FfGrid g, int C, int K, int relu, FfWait wt)
{
    after_previous_kernel(Vsaved, Wt, dY, dV);
    using T = FfTile<MT>;
    uint32_t bar;
    float *As = ff_shared(bar), *Bs = As + 2 * kFfWarps * T::A, *raw = Bs + 2 * kFfWarps * kFfB;
    const int t = threadIdx.x >> 5;
    const long long p0 = (long long)blockIdx.x * T::M;
    const int c0 = blockIdx.y * kFfN;
    const int half_id = threadIdx.x & (kFfThreads / 2 - 1);
    WarpTile<MT, true, true> w;
    w.clear();

    // Pixels: [pixel 2a + e][row][16 channels] for NHWC, [pixel][16 channels][row] for NCHW.  A thread copies for one row: both
    // pixels (a = 0, 1) of one e and one group of four channels (NHWC), or one pixel's share of the channels (NCHW).
    constexpr int RT = LAYOUT == WG2X2_NHWC ? T::M * 4 * 2 : 4 * T::M;             // threads that copy one e x group / one pixel each
    const int ce = LAYOUT == WG2X2_NHWC ? (threadIdx.x / (T::M * 4)) & 1 : 0, cpix = (threadIdx.x / T::M) & 3;
    const int crow = LAYOUT == WG2X2_NHWC ? (threadIdx.x >> 2) % T::M : threadIdx.x % T::M, cg = threadIdx.x & 3;
    const float *src = dY;
    bool ok0 = false, ok1 = false;
    if (threadIdx.x < RT || LAYOUT == WG2X2_NCHW) {
        const long long p = p0 + crow;
        if (p < g.P) {
            int b, th, tw;
            decode_tile(g, p, b, th, tw);
            if (LAYOUT == WG2X2_NHWC) {
                ok0 = 2 * tw + ce < g.W;
                ok1 = ok0 && 2 * th + 1 < g.H;
                src = dY + img_index<LAYOUT>(b, 2 * th, 2 * tw + ce, 4 * cg, g.H, g.W, K);
            } else {
                ok0 = 2 * th + (cpix >> 1) < g.H && 2 * tw + (cpix & 1) < g.W;
                src = dY + img_index<LAYOUT>(b, 2 * th + (cpix >> 1), 2 * tw + (cpix & 1), 0, g.H, g.W, K);
            }
        }
    }
    auto copy_raw = [&](int buf, int n) {
        float *d = raw + buf * T::kRawRows;
        const int k = n * kFfKC;
        if (LAYOUT == WG2X2_NHWC) {
            if (threadIdx.x < RT) {
                const int have = K - k - 4 * cg;
                copy4<VEC>(d + (ce * T::M + crow) * kFfKC + 4 * cg, src + k, ok0 ? have : 0, dY);
                copy4<VEC>(d + ((2 + ce) * T::M + crow) * kFfKC + 4 * cg, src + (long long)g.W * K + k, ok1 ? have : 0, dY);
            }
        } else {
            // the threads beyond 4 x M take further channels of the same pixels
            constexpr int S = kFfThreads / (4 * T::M);
            for (int q = threadIdx.x / (4 * T::M); q < kFfKC; q += S) {
                const bool ok = ok0 && k + q < K;
                cp4(d + (cpix * kFfKC + q) * T::M + crow, ok ? src + (long long)(k + q) * g.H * g.W : dY, ok);
            }
        }
    };
    auto copy_other = [&](int buf, int n) {
        float *B = Bs + (buf * kFfWarps + t) * kFfB;
        if (!VEC) {
            copy_rows<kFfN>(B, Wt + (long long)t * C * K, c0, C, K, n * kFfKC);
        } else if ((threadIdx.x & 31) == 0) {
            ff_expect(bar + 8 * buf, kFfB * 4);
            ff_tma(B, &mapW, bar + 8 * buf, n * kFfKC, c0, t);
        }
    };
    auto wait_other = [&](int buf, uint32_t ph) { if (VEC) ff_wait(bar + 8 * buf, ph, wt.status, wt.limit); };
    auto build = [&](int buf) {
        const float *r = raw + buf * T::kRawRows;
        float *d = As + buf * kFfWarps * T::A;
        for (int e = half_id; e < T::M * (kFfKC / 4); e += kFfThreads / 2) {
            const int row = LAYOUT == WG2X2_NHWC ? e >> 2 : e % T::M, gq = LAYOUT == WG2X2_NHWC ? e & 3 : e / T::M;
            build_dm([&](int pix) {
                if (LAYOUT == WG2X2_NHWC) return *reinterpret_cast<const float4 *>(r + (pix * T::M + row) * kFfKC + 4 * gq);
                const float *q = r + (pix * kFfKC + 4 * gq) * T::M + row;
                return make_float4(q[0], q[T::M], q[2 * T::M], q[3 * T::M]);
            }, [&](int pos, float4 v) { *reinterpret_cast<float4 *>(d + pos * T::A + at_row(row, gq)) = v; });
        }
    };
    auto compute = [&](int buf) { w.chunk(As + (buf * kFfWarps + t) * T::A, Bs + (buf * kFfWarps + t) * kFfB); };
    gradient_loop(cdiv(K, kFfKC), copy_raw, copy_other, wait_other, build, compute);
    const long long plane = (long long)t * g.P * C;
    store_block<MT, VEC>(w, As, dV + plane, p0, g.P, c0, C, [&](long long o, int have, float4 v) {
        if (!relu) return v;
        const float4 s = load4<VEC>(Vsaved + plane + o, have);
        return make_float4(s.x > 0.f ? v.x : 0.f, s.y > 0.f ? v.y : 0.f, s.z > 0.f ? v.z : 0.f, s.w > 0.f ? v.w : 0.f);
    });
}

// ------------------------------------------------------------------------------------------
// dW_t[c][k] = sum_p V_t[p][c] dM_t[p][k], contraction over P split across gridDim.z CTAs.
// With one split the result (times the mask) goes straight to dW; otherwise each split writes
// its partial sum to scratch memory and conv_dw_reduce_kernel adds them in a fixed order.
// ------------------------------------------------------------------------------------------
template <int MT, bool VEC, int LAYOUT>
__global__ void __launch_bounds__(kFfThreads, 1) conv_dw_ffma_kernel(const __grid_constant__ CUtensorMap mapV, const float *__restrict__ V,
                                                                      const float *__restrict__ dY, const float *__restrict__ mask,
                                                                      float *__restrict__ out, FfGrid g, int C, int K, int chunks_per_split,
                                                                      int direct, FfWait wt)
{
    after_previous_kernel(V, dY, mask, out);
    using T = FfTile<MT>;
    uint32_t bar;
    float *As = ff_shared(bar), *Bs = As + 2 * kFfWarps * T::A, *raw = Bs + 2 * kFfWarps * kFfB;
    const int t = threadIdx.x >> 5;
    const int ktiles = cdiv(K, kFfN);
    const int c0 = (blockIdx.x / ktiles) * T::M, k0 = (blockIdx.x % ktiles) * kFfN;
    const long long pbeg = (long long)blockIdx.z * chunks_per_split * kFfKC;
    const long long pend = min(g.P, pbeg + (long long)chunks_per_split * kFfKC);
    const int half_id = threadIdx.x & (kFfThreads / 2 - 1);
    WarpTile<MT, false, false> w;
    w.clear();

    // Pixels: [pixel][tile][32 channels] for NHWC (a thread: one pixel of one tile, four channels), [pixel][channel][tile] for
    // NCHW (a thread: four channels of one pixel of one tile)
    const int cpix = threadIdx.x >> 7, cp = LAYOUT == WG2X2_NHWC ? (threadIdx.x >> 3) & 15 : threadIdx.x & 15;
    const int cg = LAYOUT == WG2X2_NHWC ? threadIdx.x & 7 : (threadIdx.x >> 4) & 7;
    auto copy_raw = [&](int buf, int n) {
        float *d = raw + buf * T::kRawCols;
        const long long p = pbeg + (long long)n * kFfKC + cp;
        int b = 0, th = 0, tw = 0;
        bool ok = p < pend;
        if (ok) {
            decode_tile(g, p, b, th, tw);
            ok = 2 * th + (cpix >> 1) < g.H && 2 * tw + (cpix & 1) < g.W;
        }
        if (LAYOUT == WG2X2_NHWC) {
            const int k = k0 + 4 * cg;
            copy4<VEC>(d + (cpix * kFfKC + cp) * kFfN + 4 * cg, dY + img_index<LAYOUT>(b, 2 * th + (cpix >> 1), 2 * tw + (cpix & 1), k, g.H, g.W, K),
                       ok ? K - k : 0, dY);
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int k = k0 + cg + 8 * q;
                const bool in = ok && k < K;
                cp4(d + (cpix * kFfN + cg + 8 * q) * kFfKC + cp,
                    in ? dY + img_index<LAYOUT>(b, 2 * th + (cpix >> 1), 2 * tw + (cpix & 1), k, g.H, g.W, K) : dY, in);
            }
        }
    };
    auto copy_other = [&](int buf, int n) {
        float *A = As + (buf * kFfWarps + t) * T::A;
        const long long p = pbeg + (long long)n * kFfKC;
        if (!VEC) {
            copy_steps<T::M, false>(A, V + (long long)t * g.P * C, p, pend, c0, C);
        } else if ((threadIdx.x & 31) == 0) {      // (splits are whole stages, so a box that reaches beyond pend reaches beyond P)
            ff_expect(bar + 8 * buf, T::A * 4);
            ff_tma(A, &mapV, bar + 8 * buf, c0, (int)p, t);
        }
    };
    auto wait_other = [&](int buf, uint32_t ph) { if (VEC) ff_wait(bar + 8 * buf, ph, wt.status, wt.limit); };
    auto build = [&](int buf) {
        const float *r = raw + buf * T::kRawCols;
        float *d = Bs + buf * kFfWarps * kFfB;
        if (half_id < kFfKC * (kFfN / 4)) {
            const int p = LAYOUT == WG2X2_NHWC ? half_id >> 3 : half_id & 15, gq = LAYOUT == WG2X2_NHWC ? half_id & 7 : half_id >> 4;
            build_dm([&](int pix) {
                if (LAYOUT == WG2X2_NHWC) return *reinterpret_cast<const float4 *>(r + (pix * kFfKC + p) * kFfN + 4 * gq);
                const float *q = r + (pix * kFfN + 4 * gq) * kFfKC + p;
                return make_float4(q[0], q[kFfKC], q[2 * kFfKC], q[3 * kFfKC]);
            }, [&](int pos, float4 v) { *reinterpret_cast<float4 *>(d + pos * kFfB + at_step(p, gq)) = v; });
        }
    };
    auto compute = [&](int buf) { w.chunk(As + (buf * kFfWarps + t) * T::A, Bs + (buf * kFfWarps + t) * kFfB); };
    gradient_loop((int)cdivll(pend - pbeg, kFfKC), copy_raw, copy_other, wait_other, build, compute);
    const long long plane = (long long)t * C * K;
    float *dst = (direct ? out : out + (long long)blockIdx.z * 16 * C * K) + plane;
    store_block<MT, VEC>(w, As, dst, c0, C, k0, K, [&](long long o, int have, float4 v) {
        if (!direct || !mask) return v;
        const float4 s = load4<VEC>(mask + plane + o, have);
        return make_float4(v.x * s.x, v.y * s.y, v.z * s.z, v.w * s.w);
    });
}

__global__ void __launch_bounds__(256) conv_dw_reduce_kernel(const float *__restrict__ partial, const float *__restrict__ mask,
                                                               float *__restrict__ dW, long long n, int splits)
{
    after_previous_kernel(partial, mask, dW);
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (long long)gridDim.x * blockDim.x) {
        float s = 0.f;
        for (int sp = 0; sp < splits; ++sp) s += partial[(long long)sp * n + idx];
        if (mask) s *= __ldg(mask + idx);
        dW[idx] = s;
    }
}

// W with the pruning mask applied, four values at a time where both are on 16-byte boundaries
template <int VEC>
__global__ void __launch_bounds__(256) mask_weights_kernel(const float *__restrict__ Wt, const float *__restrict__ mask, float *__restrict__ out,
                                                             long long n)
{
    after_previous_kernel(Wt, mask, out);
    for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * VEC; i < n; i += (long long)gridDim.x * blockDim.x * VEC) {
        if (VEC == 4) {
            const float4 w = __ldg(reinterpret_cast<const float4 *>(Wt + i)), m = __ldg(reinterpret_cast<const float4 *>(mask + i));
            *reinterpret_cast<float4 *>(out + i) = make_float4(w.x * m.x, w.y * m.y, w.z * m.z, w.w * m.w);
        } else {
            out[i] = __ldg(Wt + i) * __ldg(mask + i);
        }
    }
}

int weights_mask(const float *Wt, const float *mask, float *out, int C, int K, cudaStream_t st)
{
    const long long n = 16LL * C * K;         // a multiple of 4
    const bool vec = ((reinterpret_cast<uintptr_t>(Wt) | reinterpret_cast<uintptr_t>(mask) | reinterpret_cast<uintptr_t>(out)) & 15u) == 0;
    const int blocks = (int)min((long long)kNumSMs * 16, cdivll(n, vec ? 1024 : 256));
    return launch(vec ? mask_weights_kernel<4> : mask_weights_kernel<1>, dim3((unsigned)blocks), 256, 0, st, Wt, mask, out, n);
}

void dw_reduce_launch(const float *partial, const float *mask, float *dW, long long n, int splits, cudaStream_t st)
{
    const int blocks = (int)min((long long)kNumSMs * 8, cdivll(n, 256));
    launch(conv_dw_reduce_kernel, dim3((unsigned)blocks), 256, 0, st, partial, mask, dW, n, splits);
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// Rows per thread of a product with `rows` x `cols` results: the block height whose last wave over the SMs wastes least.  A CTA
// of 64 rows takes 1, one of 32 rows 0.55, one of 16 rows 0.32 (less reuse per shared-memory load); one CTA runs per SM.
static int ff_rows_per_thread(long long rows, int cols)
{
    const long long nc = cdiv(cols, kFfN);
    const double t8 = (double)cdivll(cdivll(rows, 64) * nc, kNumSMs), t4 = 0.55 * (double)cdivll(cdivll(rows, 32) * nc, kNumSMs),
                 t2 = 0.32 * (double)cdivll(cdivll(rows, 16) * nc, kNumSMs);
    return t8 <= t4 && t8 <= t2 ? 8 : (t4 <= t2 ? 4 : 2);
}

// conv_tc.cu: the tensor-map cache, the status word of the bounded waits on the current device and their poll limit
bool tensor_map_f32(CUtensorMap *map, int rank, const float *ptr, const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box,
                    CUtensorMapSwizzle swizzle);
unsigned int *tc_status_word();
uint32_t tc_wait_limit();
static FfWait ff_wait_args() { return FfWait{tc_status_word(), tc_wait_limit()}; }

// A (16, rows, cols) matrix, columns contiguous: box of box_cols x box_rows of one position
static bool ff_map(CUtensorMap *m, const float *p, long long cols, long long rows, int box_cols, int box_rows, CUtensorMapSwizzle swizzle)
{
    const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, 16}, strides[2] = {(cuuint64_t)cols * 4, (cuuint64_t)rows * cols * 4};
    const cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1};
    return tensor_map_f32(m, 3, p, dims, strides, box, swizzle);
}
// 16-byte rows on 16-byte boundaries: what TMA and the vector accesses ask for
static bool ff_vec(long long P, int C, int K) { return C % 4 == 0 && K % 4 == 0 && P <= 0x7fffffffLL - 64; }

int conv_fwd_ffma(const float *V, const float *Wt, float *Y, int B, int nH, int nW, int C, int K, int outH, int outW,
                  int layout, cudaStream_t st)
{
    const FfGrid g{(long long)B * nH * nW, nH, nW, outH, outW};
    if (cdivll(g.P, 16) > 0x7fffffffLL || cdiv(K, kFfN) > 65535) return WG2X2_ERR_UNSUPPORTED;
    const bool vec = ff_vec(g.P, C, K) && aligned16(V) && aligned16(Wt) && aligned16(Y);
    const int mt = ff_rows_per_thread(g.P, K);
    const dim3 grid((unsigned)cdivll(g.P, 8 * mt), cdiv(K, kFfN));
    CUtensorMap mapV = {}, mapW = {};
    if (vec && (!ff_map(&mapV, V, C, g.P, kFfKC, 8 * mt, CU_TENSOR_MAP_SWIZZLE_64B) ||
                !ff_map(&mapW, Wt, K, C, kFfN, kFfKC, CU_TENSOR_MAP_SWIZZLE_128B)))
        return WG2X2_ERR_LAUNCH;
    const FfWait wt = ff_wait_args();
    if (!wt.status) return WG2X2_ERR_LAUNCH;
#define WG_FF(MT, VEC, L) launch(conv_fwd_ffma_kernel<MT, VEC, L>, grid, kFfThreads, FfTile<MT>::kFwdBytes, st, mapV, mapW, V, Wt, Y, g, C, K, wt)
#define WG_FF_L(MT, VEC) (layout == WG2X2_NHWC ? WG_FF(MT, VEC, WG2X2_NHWC) : WG_FF(MT, VEC, WG2X2_NCHW))
#define WG_FF_V(MT) (vec ? WG_FF_L(MT, true) : WG_FF_L(MT, false))
    return mt == 8 ? WG_FF_V(8) : mt == 4 ? WG_FF_V(4) : WG_FF_V(2);
#undef WG_FF
}

int conv_dv_ffma(const float *V, const float *Wt, const float *dY, float *dV, int B, int H, int W, int C, int K, int layout,
                 int relu, cudaStream_t st)
{
    const FfGrid g{(long long)B * ((H + 1) / 2) * ((W + 1) / 2), (H + 1) / 2, (W + 1) / 2, H, W};
    if (cdivll(g.P, 16) > 0x7fffffffLL || cdiv(C, kFfN) > 65535) return WG2X2_ERR_UNSUPPORTED;
    const bool vec = ff_vec(g.P, C, K) && (!relu || aligned16(V)) && aligned16(Wt) && aligned16(dY) && aligned16(dV);
    const int mt = ff_rows_per_thread(g.P, C);
    const dim3 grid((unsigned)cdivll(g.P, 8 * mt), cdiv(C, kFfN));
    CUtensorMap mapW = {};
    if (vec && !ff_map(&mapW, Wt, K, C, kFfKC, kFfN, CU_TENSOR_MAP_SWIZZLE_64B)) return WG2X2_ERR_LAUNCH;
    const FfWait wt = ff_wait_args();
    if (!wt.status) return WG2X2_ERR_LAUNCH;
#define WG_FF(MT, VEC, L) launch(conv_dv_ffma_kernel<MT, VEC, L>, grid, kFfThreads, FfTile<MT>::kDvBytes, st, mapW, V, Wt, dY, dV, g, C, K, relu, wt)
    return mt == 8 ? WG_FF_V(8) : mt == 4 ? WG_FF_V(4) : WG_FF_V(2);
#undef WG_FF
}

// Rows of dW per CTA: 64, or fewer where there are fewer in-channels
static int dw_rows_per_thread(int C) { return C > 32 ? 8 : (C > 16 ? 4 : 2); }

// Number of P-splits of the dW kernel: as many CTAs as one wave over the SMs holds; two splits where the blocks alone fill
// more than half of it (the wave is as long either way, and two sums of half the length are the more accurate ones).
int conv_dw_splits(long long P, int C, int K)
{
    const long long tiles = (long long)cdiv(C, 8 * dw_rows_per_thread(C)) * cdiv(K, kFfN);
    const long long chunks = cdivll(P, kFfKC);
    long long s = tiles >= kNumSMs ? 1 : (2 * tiles > kNumSMs ? 2 : kNumSMs / tiles);
    if (s > chunks) s = chunks;
    if (s < 1) s = 1;
    // every split must own at least one chunk
    const long long cps = cdivll(chunks, s);
    return (int)cdivll(chunks, cps);
}

size_t conv_dw_scratch_bytes(long long P, int C, int K)
{
    const int s = conv_dw_splits(P, C, K);
    return s > 1 ? (size_t)s * 16 * C * K * sizeof(float) : 0;
}

int conv_dw_ffma(const float *V, const float *dY, const float *mask, float *dW, int B, int H, int W, int C, int K, int layout,
                 float *scratch, int splits, cudaStream_t st)
{
    const FfGrid g{(long long)B * ((H + 1) / 2) * ((W + 1) / 2), (H + 1) / 2, (W + 1) / 2, H, W};
    const int cps = (int)cdivll(cdivll(g.P, kFfKC), splits);
    const int mt = dw_rows_per_thread(C);
    const long long gx = (long long)cdiv(C, 8 * mt) * cdiv(K, kFfN);
    if (gx > 0x7fffffffLL || splits > 65535) return WG2X2_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)gx, 1, splits);
    const int direct = splits == 1;
    float *out = direct ? dW : scratch;
    const bool vec = ff_vec(g.P, C, K) && aligned16(V) && aligned16(dY) && aligned16(out) && (!mask || aligned16(mask));
    CUtensorMap mapV = {};
    if (vec && !ff_map(&mapV, V, C, g.P, 8 * mt, kFfKC, CU_TENSOR_MAP_SWIZZLE_NONE)) return WG2X2_ERR_LAUNCH;
    const FfWait wt = ff_wait_args();
    if (!wt.status) return WG2X2_ERR_LAUNCH;
#define WG_FF(MT, VEC, L) launch(conv_dw_ffma_kernel<MT, VEC, L>, grid, kFfThreads, FfTile<MT>::kDwBytes, st, mapV, V, dY, mask, out, g, C, K, cps, direct, wt)
    const int s = mt == 8 ? WG_FF_V(8) : mt == 4 ? WG_FF_V(4) : WG_FF_V(2);
#undef WG_FF
#undef WG_FF_L
#undef WG_FF_V
    if (s != WG2X2_OK) return s;
    if (!direct) dw_reduce_launch(scratch, mask, dW, (long long)16 * C * K, splits, st);
    return launch_status();
}

}  // namespace wg
