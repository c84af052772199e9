// Shared device helpers for the Winograd F(2x2,3x3) kernels: the three small transforms in
// separable form, plus launch bookkeeping.  Position index t = 4*i + j everywhere.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdlib.h>

#include <initializer_list>
#include <mutex>

#include "../../include/winograd2x2_b200.h"

namespace wg {

constexpr int kNumSMs = 148;  // B200: grids of grid-stride kernels are sized in multiples of this

__host__ __device__ inline int cdiv(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline long long cdivll(long long a, long long b) { return (a + b - 1) / b; }

__device__ __forceinline__ float4 operator+(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ float4 operator-(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }

// max(x, 0) that keeps NaN, as torch.relu does (fmaxf gives the other value), for the ReLUs that stand in for one of the network's
__device__ __forceinline__ float relu_nan(float x)
{
    float y;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float4 relu_nan(float4 a) { return make_float4(relu_nan(a.x), relu_nan(a.y), relu_nan(a.z), relu_nan(a.w)); }

// ---- B^T d B, separable: 16 adds for the rows, 16 for the columns -----------------------
// B^T = [[1,0,-1,0],[0,1,1,0],[0,-1,1,0],[0,1,0,-1]]
template <typename T>
__device__ __forceinline__ void bt_d_b(const T (&d)[4][4], T (&v)[4][4])
{
    T r[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        r[0][x] = d[0][x] - d[2][x];
        r[1][x] = d[1][x] + d[2][x];
        r[2][x] = d[2][x] - d[1][x];
        r[3][x] = d[1][x] - d[3][x];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[i][0] = r[i][0] - r[i][2];
        v[i][1] = r[i][1] + r[i][2];
        v[i][2] = r[i][2] - r[i][1];
        v[i][3] = r[i][1] - r[i][3];
    }
}

// ---- A^T m A -----------------------------------------------------------------------------
// A^T = [[1,1,1,0],[0,1,-1,-1]]; column step: z[e] from one row of m
__device__ __forceinline__ void at_cols(float m0, float m1, float m2, float m3, float &z0, float &z1)
{
    z0 = m0 + m1 + m2;
    z1 = m1 - m2 - m3;
}
// row step: given the column-transformed pair of Winograd row i, add into y[a][e]
__device__ __forceinline__ void at_rows_accum(int i, float z0, float z1, float (&y)[2][2])
{
    // AT[0] = [1,1,1,0], AT[1] = [0,1,-1,-1]
    if (i == 0) { y[0][0] += z0; y[0][1] += z1; }
    if (i == 1) { y[0][0] += z0; y[0][1] += z1; y[1][0] += z0; y[1][1] += z1; }
    if (i == 2) { y[0][0] += z0; y[0][1] += z1; y[1][0] -= z0; y[1][1] -= z1; }
    if (i == 3) { y[1][0] -= z0; y[1][1] -= z1; }
}

// ---- A dY A^T : the 16 Winograd-domain gradients of a 2x2 output block ---------------------
// dM[i][j] = sum_{a,e} AT[a][i] AT[e][j] g[a][e]
__device__ __forceinline__ void a_g_at(float g00, float g01, float g10, float g11, float (&dm)[4][4])
{
    // rows over a: u[i][e]
    float u[4][2];
    u[0][0] = g00;        u[0][1] = g01;
    u[1][0] = g00 + g10;  u[1][1] = g01 + g11;
    u[2][0] = g00 - g10;  u[2][1] = g01 - g11;
    u[3][0] = -g10;       u[3][1] = -g11;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        dm[i][0] = u[i][0];
        dm[i][1] = u[i][0] + u[i][1];
        dm[i][2] = u[i][0] - u[i][1];
        dm[i][3] = -u[i][1];
    }
}
// B^T as compile-time coefficients (for the gather in the input-transform gradient)
__host__ __device__ constexpr int bt_coef(int i, int y)
{
    return (i == 0) ? (y == 0 ? 1 : (y == 2 ? -1 : 0))
         : (i == 1) ? ((y == 1 || y == 2) ? 1 : 0)
         : (i == 2) ? (y == 1 ? -1 : (y == 2 ? 1 : 0))
                    : (y == 1 ? 1 : (y == 3 ? -1 : 0));
}

// How the NCHW kernels that walk tiles with lane = channel cut an image: bands of R tile rows, and, where a band is a single
// row, segments of S tiles along it.  `blocks`: CTAs per band (images x channel blocks).  A small problem is cut until the
// grid gives every SM a few CTAs (a warp's tiles are a serial chain of loads: 3 x 27 x 27 x 32 channels took 25 us in 6 CTAs,
// whatever the bytes); eight warps share a block's tiles, so segments end at 8.
struct BandCut {
    int R, nbands, S, nsegs;
};
inline BandCut cut_bands(int nH, int nW, long long blocks, int max_rows)
{
    BandCut c;
    c.R = max_rows < 1 ? 1 : (max_rows > nH ? nH : max_rows);
    while (c.R > 1 && blocks * cdiv(nH, c.R) < 3LL * kNumSMs) --c.R;
    c.nbands = cdiv(nH, c.R);
    c.R = cdiv(nH, c.nbands);                 // bands of even height
    c.nbands = cdiv(nH, c.R);
    c.nsegs = 1;
    if (c.R == 1)
        while (cdiv(nW, c.nsegs) > 8 && blocks * c.nbands * c.nsegs < 3LL * kNumSMs) ++c.nsegs;
    c.S = cdiv(nW, c.nsegs);
    c.nsegs = cdiv(nW, c.S);
    return c;
}

// Staging for those kernels: each of eight warps copies four of 32 channel planes (nch of them exist) to rows of shared memory,
// `n` floats per channel at src(i) / dst[i], four channels at a time so that as many loads are in flight.
template <typename Src>
__device__ __forceinline__ void stage_channels(const float *__restrict__ plane0, long long plane, int nch, int n, float *dst0, int pitch, Src src)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float *p = plane0 + warp * plane;
    float *d = dst0 + warp * pitch;
    for (int i = lane; i < n; i += 32) {
        const int o = src(i);
        float v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = warp + 8 * q < nch ? __ldg(p + 8 * q * plane + o) : 0.f;
#pragma unroll
        for (int q = 0; q < 4; ++q) d[8 * q * pitch + i] = v[q];
    }
}

// ---- 64 channels of an NCHW image in shared memory as [pixel][channel], for kernels with two channels per lane ----
constexpr int kPairCB = 64, kPairPitch = kPairCB + 2;   // channels per CTA; floats of a pixel in shared memory

// Stage rows gy0 .. gy0 + rows - 1 of 64 channels: slot (row, x) receives pixel (gy0 + row, x - gx0), PW slots a row, zeros outside
// the image.  Asynchronous copies, all in flight at once: staged through registers, the few loads that a warp had open at a
// time were what the kernel waited for (34 against 29 us at 128 x 256 x 14 x 14).  inv = ceil(2^20 / PW).
__device__ __forceinline__ void stage_pairs(const float *__restrict__ X, float *S, int b, int c0, int C, int H, int W, int gy0, int gx0, int rows, int PW,
                                            unsigned inv)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nch = min(kPairCB, C - c0) - warp;          // channels warp, warp + 8, ... of the block: (nch + 7) / 8 of them exist
    const long long HW8 = 8LL * H * W;
    const float *plane = X + ((long long)b * C + c0 + warp) * H * W;
    for (int i = lane; i < rows * PW; i += 32) {
        const int r = (int)(((unsigned)i * inv) >> 20), x = i - r * PW - gx0, y = gy0 + r;
        const bool in = y >= 0 && y < H && x >= 0 && x < W;
        const float *src = plane + (in ? (long long)y * W + x : 0);
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(S + i * kPairPitch + warp);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const bool ok = in && 8 * q < nch;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 32u * q), "l"(ok ? src + q * HW8 : X), "r"(ok ? 4 : 0) : "memory");
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

// The band height of the kernels that stage so (bands of 2 R + extra rows): least work of the busiest SM (a tile is 146 issue slots, a
// staged pixel 10 per 64 channels, and a CTA costs something of its own), shared memory for three CTAs per SM.  0: too few CTAs to
// fill the GPU.
inline int pair_rows(int B, int C, int nH, int nW, int W, int extra)
{
    const long long per_band = (long long)B * cdiv(C, kPairCB);
    int best = 0;
    double t = 1e300;
    for (int R = 1; R <= nH; ++R) {
        if (R > 1 && (2 * R + extra) * (2 * nW + extra) * kPairPitch * 4 > 72 * 1024) break;
        const long long ctas = per_band * cdiv(nH, R);
        if (ctas < 2LL * kNumSMs) continue;
        const double u = (double)cdivll(ctas, kNumSMs) * ((2.0 * R + extra) * W * 10 + (double)R * nW * 146 + 1500);
        if (u < t) { t = u; best = R; }
    }
    return best ? cdiv(nH, cdiv(nH, best)) : 0;
}

inline int launch_status()
{
    return cudaGetLastError() == cudaSuccess ? WG2X2_OK : WG2X2_ERR_LAUNCH;
}

// ---- launches ------------------------------------------------------------------------------
// Every kernel goes out with programmatic stream serialisation: its CTAs may be scheduled while the kernel before it in the
// stream still runs its last ones, and wait there (after_previous_kernel) until that kernel has completed and its writes are
// visible.  A layer is up to seven kernels of a few microseconds; what a boundary between two of them costs otherwise -- launch
// latency, scheduling, set-up -- is one to two microseconds each.  Not during graph capture; WG2X2_PDL=0 turns it off.
//
// When the next kernel may come in: at once where this grid is small (max_ctas), else when its CTAs have ended.  Let in
// early beside a grid that occupies the SMs, the next one's CTAs pile up on those that have room or finish first, and a
// kernel of only one wave then runs unbalanced (16.8 against 14.4 us for the 64 x 256 x 14 x 14 input transform).
__device__ __forceinline__ void wait_for_previous_kernel(unsigned max_ctas)
{
    if (gridDim.x * gridDim.y * gridDim.z <= max_ctas) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// First statement of a kernel that touches global memory only through the given pointers.  The pointers pass through the
// wait, so that no load from them can be moved in front of it.
template <typename... P>
__device__ __forceinline__ void after_previous_kernel(P &...p)
{
    wait_for_previous_kernel(kNumSMs);
    (void)std::initializer_list<int>{([](P &q) { asm volatile("" : "+l"(q)::"memory"); }(p), 0)...};
}

// Dynamic shared memory above 48 KB has to be granted to a kernel, per device and for the whole process.  A kernel may be launched
// with other sizes by several threads at once, so a grant is only ever raised: one thread at a time looks at it and sets it.  What a
// thread has seen granted it need not ask for again.
inline bool grant_smem(const void *kernel, size_t bytes)
{
    struct Entry { const void *kernel; int dev; size_t bytes; };
    thread_local Entry seen[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    Entry &e = seen[(reinterpret_cast<uintptr_t>(kernel) >> 4) & 63];
    if (e.kernel == kernel && e.dev == dev && e.bytes >= bytes) return true;
    static std::mutex one_at_a_time;
    const std::lock_guard<std::mutex> lock(one_at_a_time);
    cudaFuncAttributes now;
    if (cudaFuncGetAttributes(&now, kernel) != cudaSuccess) return false;
    size_t granted = now.maxDynamicSharedSizeBytes < 0 ? 0 : (size_t)now.maxDynamicSharedSizeBytes;
    if (granted < bytes) {
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess) return false;
        granted = bytes;
    }
    e = Entry{kernel, dev, granted};
    return true;
}

template <typename... KernelArgs, typename... Args>
int launch(void (*kernel)(KernelArgs...), dim3 grid, int threads, size_t smem, cudaStream_t st, Args &&...args)
{
    if (smem > 48 * 1024 && !grant_smem(reinterpret_cast<const void *>(kernel), smem)) return WG2X2_ERR_LAUNCH;
    static const bool pdl_env = [] { const char *e = getenv("WG2X2_PDL"); return !(e && e[0] == '0'); }();
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &capturing) != cudaSuccess) return WG2X2_ERR_LAUNCH;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_env && capturing == cudaStreamCaptureStatusNone ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KernelArgs>(args)...) == cudaSuccess ? launch_status() : WG2X2_ERR_LAUNCH;
}

}  // namespace wg
