// Input transform (+ Winograd-domain ReLU) and its gradient.  HBM-bound kernels:
//   forward  : reads |X| once from HBM (the 4x overlap between neighbouring tiles is served
//              by L1/L2 or by the shared-memory stage), writes 16 planes of V = 4|X|
//   backward : reads dV (and V when the ReLU mask is asked for), writes dX; a gather, so it
//              is deterministic and needs neither atomics nor scratch memory.
#include "wg_common.cuh"

namespace wg {

template <int VEC> struct Vec;
template <> struct Vec<4> { using type = float4; };
template <> struct Vec<1> { using type = float; };

__device__ __forceinline__ float4 ldg(const float4 *p) { return __ldg(p); }
__device__ __forceinline__ float ldg(const float *p) { return __ldg(p); }
__device__ __forceinline__ float4 zero_of(float4) { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float zero_of(float) { return 0.f; }
__device__ __forceinline__ float4 fma_of(float4 a, float4 s, float4 b) { return make_float4(fmaf(a.x, s.x, b.x), fmaf(a.y, s.y, b.y), fmaf(a.z, s.z, b.z), fmaf(a.w, s.w, b.w)); }
__device__ __forceinline__ float fma_of(float a, float s, float b) { return fmaf(a, s, b); }
__device__ __forceinline__ float4 relu_of(float4 a) { return make_float4(fmaxf(a.x, 0.f), fmaxf(a.y, 0.f), fmaxf(a.z, 0.f), fmaxf(a.w, 0.f)); }
__device__ __forceinline__ float relu_of(float a) { return fmaxf(a, 0.f); }
// the components of a value to p[0], p[pitch], ... (by name: indexing through a pointer would put the value on the stack)
__device__ __forceinline__ void put_lanes(float *p, int pitch, float4 v) { p[0] = v.x; p[pitch] = v.y; p[2 * pitch] = v.z; p[3 * pitch] = v.w; }
__device__ __forceinline__ void put_lanes(float *p, int, float v) { p[0] = v; }
__device__ __forceinline__ float4 keep_where_pos(float4 g, float4 m) { return make_float4(m.x > 0.f ? g.x : 0.f, m.y > 0.f ? g.y : 0.f, m.z > 0.f ? g.z : 0.f, m.w > 0.f ? g.w : 0.f); }
__device__ __forceinline__ float keep_where_pos(float g, float m) { return m > 0.f ? g : 0.f; }

// The ReLU mask as bits: 16 per tile and channel, bit t set where position t of V is positive.  [P][C] of them, 1/32 of V, is what
// the backward pass reads instead of V itself (64 x 64 x 56 x 56: 6.4 MB for 205).
typedef unsigned short signs_t;
__device__ __forceinline__ signs_t signs_of(const float (&v)[4][4])
{
    unsigned m = 0;
#pragma unroll
    for (int t = 0; t < 16; ++t) m |= v[t >> 2][t & 3] > 0.f ? 1u << t : 0u;
    return (signs_t)m;
}
__device__ __forceinline__ void put_signs(signs_t *s, const float4 (&v)[4][4])
{
    unsigned m[4] = {0, 0, 0, 0};
#pragma unroll
    for (int t = 0; t < 16; ++t) {
        const float4 x = v[t >> 2][t & 3];
        m[0] |= x.x > 0.f ? 1u << t : 0u;
        m[1] |= x.y > 0.f ? 1u << t : 0u;
        m[2] |= x.z > 0.f ? 1u << t : 0u;
        m[3] |= x.w > 0.f ? 1u << t : 0u;
    }
    *reinterpret_cast<uint2 *>(s) = make_uint2(m[0] | (m[1] << 16), m[2] | (m[3] << 16));
}
__device__ __forceinline__ void put_signs(signs_t *s, const float (&v)[4][4]) { *s = signs_of(v); }

// ------------------------------------------------------------------------------------------
// Forward, NHWC.  One thread = one tile x VEC channels; consecutive threads walk the channel
// axis first, so each of the 16 plane stores of a warp is one contiguous run.
// ------------------------------------------------------------------------------------------
template <int VEC, bool AFFINE, bool SIGNS>
__global__ void __launch_bounds__(256) imtrans_fwd_nhwc_kernel(const float *__restrict__ X, float *__restrict__ V, signs_t *__restrict__ signs,
                                                                 int B, int H, int W, int C, int nH, int nW, int relu,
                                                                 const float *__restrict__ scale, const float *__restrict__ shift)
{
    after_previous_kernel(X, V, signs, scale, shift);
    using T = typename Vec<VEC>::type;
    const int CV = C / VEC;
    const long long total = (long long)B * nH * nW * CV;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int cv = (int)(idx % CV);
    const long long p = idx / CV;
    const int tw = (int)(p % nW);
    const int th = (int)((p / nW) % nH);
    const int b = (int)(p / ((long long)nW * nH));

    const T *Xv = reinterpret_cast<const T *>(X);
    // optional per-channel affine map of the pixels (an inference-form BatchNorm in front of the
    // transform); the zero padding stays zero
    T sc = zero_of(T()), sh = zero_of(T());
    if (AFFINE) { sc = ldg(reinterpret_cast<const T *>(scale) + cv); sh = ldg(reinterpret_cast<const T *>(shift) + cv); }
    T d[4][4];
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        const int fy = 2 * th - 1 + y;
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int fx = 2 * tw - 1 + x;
            const bool in = (fy >= 0) && (fy < H) && (fx >= 0) && (fx < W);
            T v = in ? ldg(Xv + (((long long)b * H + fy) * W + fx) * CV + cv) : zero_of(T());
            if (AFFINE && in) v = fma_of(v, sc, sh);
            d[y][x] = v;
        }
    }
    T v[4][4];
    bt_d_b(d, v);
    T *Vv = reinterpret_cast<T *>(V);
    const long long plane = (long long)B * nH * nW * CV;
    const long long off = p * CV + cv;
    if (SIGNS) put_signs(signs + off * VEC, v);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            Vv[(long long)(4 * i + j) * plane + off] = relu ? relu_of(v[i][j]) : v[i][j];
}

// ------------------------------------------------------------------------------------------
// Forward, NCHW.  The image axis W is contiguous and tiles overlap along it, so a CTA stages
// the 4 input rows of one tile row, for CCH channels and TSEG tiles, in shared memory
// (coalesced along W), then computes with the channel index fastest across a warp so that
// the plane stores are contiguous along C.
// ------------------------------------------------------------------------------------------
constexpr int kCCH = 32;                       // channels per CTA
constexpr int kTSEG = 32;                      // tiles along W per CTA
constexpr int kRowPitch = 2 * kTSEG + 2;       // 66 pixels feed 32 tiles
constexpr int kChanPitch = 4 * kRowPitch + 1;  // odd, so 32 channels hit 32 different banks

__global__ void __launch_bounds__(256) imtrans_fwd_nchw_kernel(const float *__restrict__ X, float *__restrict__ V, signs_t *__restrict__ signs,
                                                                 int B, int H, int W, int C, int nH, int nW, int relu,
                                                                 const float *__restrict__ scale, const float *__restrict__ shift)
{
    after_previous_kernel(X, V, signs, scale, shift);
    __shared__ float S[kCCH * kChanPitch];
    const int nseg = cdiv(nW, kTSEG);
    int bx = blockIdx.x;
    const int seg = bx % nseg; bx /= nseg;
    const int th = bx % nH;
    const int b = bx / nH;
    const int c0 = blockIdx.y * kCCH;
    const int tw0 = seg * kTSEG;
    const int tid = threadIdx.x;

    for (int idx = tid; idx < kCCH * 4 * kRowPitch; idx += 256) {
        const int x = idx % kRowPitch;
        const int y = (idx / kRowPitch) & 3;
        const int c = idx / (4 * kRowPitch);
        const int gx = 2 * tw0 - 1 + x, gy = 2 * th - 1 + y;
        float val = 0.f;
        if (c0 + c < C && gx >= 0 && gx < W && gy >= 0 && gy < H) {
            val = __ldg(X + (((long long)b * C + c0 + c) * H + gy) * W + gx);
            if (scale) val = fmaf(val, __ldg(scale + c0 + c), __ldg(shift + c0 + c));
        }
        S[c * kChanPitch + y * kRowPitch + x] = val;
    }
    __syncthreads();

    const int c = tid & 31;
    const long long plane = (long long)B * nH * nW * C;
#pragma unroll 1
    for (int it = 0; it < kTSEG / 8; ++it) {
        const int twl = (tid >> 5) + 8 * it;
        const int tw = tw0 + twl;
        if (tw >= nW || c0 + c >= C) continue;
        float d[4][4], v[4][4];
#pragma unroll
        for (int y = 0; y < 4; ++y)
#pragma unroll
            for (int x = 0; x < 4; ++x) d[y][x] = S[c * kChanPitch + y * kRowPitch + 2 * twl + x];
        bt_d_b(d, v);
        const long long off = (((long long)b * nH + th) * nW + tw) * C + c0 + c;
        if (signs) signs[off] = signs_of(v);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                V[(long long)(4 * i + j) * plane + off] = relu ? fmaxf(v[i][j], 0.f) : v[i][j];
    }
}

// ------------------------------------------------------------------------------------------
// Forward, NCHW, image rows up to 128 pixels (every Winograd layer of a ResNet).  A CTA owns one
// image, 32 channels and a band of R tile rows.  For one channel the 2R+2 input rows of the band
// are one contiguous run of memory, so the fill is a plain coalesced copy into shared memory
// (one run per channel, odd pitch between channels); then each warp walks tiles with lane =
// channel, which makes the shared-memory reads conflict-free and every plane store one
// contiguous 128-byte run along C.  Borders and padding are predicates on warp-uniform
// coordinates.  Rows are re-read (2R+2)/2R times, from L2.
// ------------------------------------------------------------------------------------------
constexpr int kBandFloats = 384;   // at most this many input floats per channel in shared memory

template <bool AFFINE, bool SIGNS>
__global__ void __launch_bounds__(256) imtrans_fwd_nchw_band_kernel(const float *__restrict__ X, float *__restrict__ V, signs_t *__restrict__ signs,
                                                                      int B, int H, int W, int C, int nH, int nW, int relu,
                                                                      int R, int nbands, int pitch,
                                                                      const float *__restrict__ scale, const float *__restrict__ shift)
{
    after_previous_kernel(X, V, signs, scale, shift);
    extern __shared__ float S[];   // [32 channels][pitch]
    const int band = blockIdx.x % nbands;
    const int b = blockIdx.x / nbands;
    const int c0 = blockIdx.y * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int th0 = band * R;
    const int rows_tile = min(R, nH - th0);
    const int gy0 = 2 * th0 - 1;                                  // first input row of the band (may be -1)
    const int lo = max(gy0, 0), hi = min(gy0 + 2 * rows_tile + 2, H);
    const int nfill = (hi - lo) * W;

    for (int cc = warp; cc < 32; cc += 8) {
        if (c0 + cc >= C) break;
        const float *src = X + (((long long)b * C + c0 + cc) * H + lo) * W;
        float *dst = S + cc * pitch + (lo - gy0) * W;
        for (int i = lane; i < nfill; i += 32) dst[i] = __ldg(src + i);
    }
    __syncthreads();

    const long long plane = (long long)B * nH * nW * C;
    const bool c_ok = c0 + lane < C;
    const float *Sc = S + lane * pitch;
    const int ntiles = rows_tile * nW;
    const float sc = (AFFINE && c_ok) ? __ldg(scale + c0 + lane) : 1.f;
    const float sh = (AFFINE && c_ok) ? __ldg(shift + c0 + lane) : 0.f;
    for (int q = warp; q < ntiles; q += 8) {
        const int tr = q / nW, tw = q - tr * nW;
        float d[4][4], v[4][4];
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const int gy = gy0 + 2 * tr + y;
            const bool row_ok = (gy >= 0) && (gy < H);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int gx = 2 * tw - 1 + x;
                const bool in = row_ok && gx >= 0 && gx < W && c_ok;
                d[y][x] = in ? (AFFINE ? fmaf(Sc[(2 * tr + y) * W + gx], sc, sh) : Sc[(2 * tr + y) * W + gx]) : 0.f;
            }
        }
        bt_d_b(d, v);
        if (c_ok) {
            const long long off = (((long long)b * nH + th0 + tr) * nW + tw) * C + c0 + lane;
            if (SIGNS) signs[off] = signs_of(v);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    V[(long long)(4 * i + j) * plane + off] = relu ? fmaxf(v[i][j], 0.f) : v[i][j];
        }
    }
}

// The same for small problems: a segment of S tiles of one tile row per CTA (cut_bands).  (A kernel of its own: as a variant of
// the one above it cost that one eight registers and 7 % of its speed.)
template <bool AFFINE, bool SIGNS>
__global__ void __launch_bounds__(256) imtrans_fwd_nchw_row_kernel(const float *__restrict__ X, float *__restrict__ V, signs_t *__restrict__ signs,
                                                                     int B, int H, int W, int C, int nH, int nW, int relu,
                                                                     int S_, int nsegs, int pitch,
                                                                     const float *__restrict__ scale, const float *__restrict__ shift)
{
    after_previous_kernel(X, V, signs, scale, shift);
    extern __shared__ float S[];   // [32 channels][pitch]
    const int seg = blockIdx.x % nsegs, th = (blockIdx.x / nsegs) % nH, b = blockIdx.x / nsegs / nH;
    const int c0 = blockIdx.y * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gy0 = 2 * th - 1, lo = max(gy0, 0), hi = min(gy0 + 4, H);
    const int tw0 = seg * S_, ns = min(S_, nW - tw0);
    const int x0 = max(2 * tw0 - 1, 0), SW = min(2 * (tw0 + ns) + 1, W) - x0;     // staged columns: the tiles' and their neighbours
    stage_channels(X + (((long long)b * C + c0) * H + lo) * W + x0, (long long)H * W, C - c0, (hi - lo) * SW, S + (lo - gy0) * SW, pitch,
                   [&](int i) { return i + (i / SW) * (W - SW); });
    __syncthreads();
    if (c0 + lane >= C) return;
    const long long plane = (long long)B * nH * nW * C;
    const float *Sc = S + lane * pitch;
    const float sc = AFFINE ? __ldg(scale + c0 + lane) : 1.f, sh = AFFINE ? __ldg(shift + c0 + lane) : 0.f;
    for (int tl = warp; tl < ns; tl += 8) {
        float d[4][4], v[4][4];
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const bool row_ok = gy0 + y >= 0 && gy0 + y < H;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int gx = 2 * (tw0 + tl) - 1 + x;
                const bool in = row_ok && gx >= 0 && gx < W;
                d[y][x] = in ? (AFFINE ? fmaf(Sc[y * SW + gx - x0], sc, sh) : Sc[y * SW + gx - x0]) : 0.f;
            }
        }
        bt_d_b(d, v);
        const long long off = (((long long)b * nH + th) * nW + tw0 + tl) * C + c0 + lane;
        if (SIGNS) signs[off] = signs_of(v);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) V[(long long)(4 * i + j) * plane + off] = relu ? fmaxf(v[i][j], 0.f) : v[i][j];
    }
}

// ------------------------------------------------------------------------------------------
// Forward, NCHW, short rows and enough tiles to fill the GPU: two channels per lane (64 per CTA), image kept in shared memory as
// [pixel][channel] with its zero padding, so that a warp reads it without predicates, and walks consecutive tiles of a row, of
// which it loads only the two new columns and keeps the row-transformed two old ones.  Per tile of 64 channels 8 eight-byte
// loads, 16 + 32 additions, 16 stores of 256 bytes off uniform plane addresses, against 32 loads, 128 additions and predicates
// and 32 stores with one channel per lane.
// ------------------------------------------------------------------------------------------
template <bool AFFINE, bool RELU, bool SIGNS>
__global__ void __launch_bounds__(256, 4) imtrans_fwd_nchw_pair_kernel(const float *__restrict__ X, float *__restrict__ V,
                                                                         signs_t *__restrict__ signs, int H, int W, int C,
                                                                         int nH, int nW, int R, int nbands, unsigned inv, unsigned plane_bytes,
                                                                         const float *__restrict__ scale, const float *__restrict__ shift)
{
    after_previous_kernel(X, V, signs, scale, shift);
    extern __shared__ __align__(16) float S[];
    const int band = blockIdx.x % nbands, b = blockIdx.x / nbands, c0 = blockIdx.y * kPairCB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int th0 = band * R, rows_tile = min(R, nH - th0), PW = 2 * nW + 2, gy0 = 2 * th0 - 1;
    stage_pairs(X, S, b, c0, C, H, W, gy0, 1, 2 * rows_tile + 2, PW, inv);
    __syncthreads();
    if (c0 + 2 * lane >= C) return;
    // the warp's share of the band's tiles, in row order
    const int ntiles = rows_tile * nW, each = cdiv(ntiles, 8);
    const int q0 = warp * each, q1 = min(q0 + each, ntiles);
    if (q0 >= q1) return;
    int tr = q0 / nW, tw = q0 - tr * nW;
    unsigned off = (unsigned)((((long long)b * nH + th0) * nW + q0) * C + c0 + 2 * lane) * 4u;
    const float2 *P = reinterpret_cast<const float2 *>(S + (2 * tr * PW + 2 * tw) * kPairPitch) + lane;
    char *const Vb = reinterpret_cast<char *>(V);
    float2 sc = make_float2(1.f, 1.f), sh = make_float2(0.f, 0.f);
    if (AFFINE) { sc = __ldg(reinterpret_cast<const float2 *>(scale + c0) + lane); sh = __ldg(reinterpret_cast<const float2 *>(shift + c0) + lane); }
    float2 r[4][4];
    auto column = [&](int x) {            // column x of the window, transformed along the rows
        float2 d[4];
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            d[y] = P[(y * PW + x) * (kPairPitch / 2)];
            if (AFFINE && gy0 + 2 * tr + y >= 0 && gy0 + 2 * tr + y < H && 2 * tw + x >= 1 && 2 * tw + x <= W)
                d[y] = make_float2(fmaf(d[y].x, sc.x, sh.x), fmaf(d[y].y, sc.y, sh.y));
        }
        r[0][x] = make_float2(d[0].x - d[2].x, d[0].y - d[2].y);
        r[1][x] = make_float2(d[1].x + d[2].x, d[1].y + d[2].y);
        r[2][x] = make_float2(d[2].x - d[1].x, d[2].y - d[1].y);
        r[3][x] = make_float2(d[1].x - d[3].x, d[1].y - d[3].y);
    };
    column(0);
    column(1);
#pragma unroll 1
    for (int q = q0;;) {
        column(2);
        column(3);
        unsigned m = 0, m2 = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int a = j == 0 ? 0 : j == 2 ? 2 : 1, c = j == 2 ? 1 : j == 3 ? 3 : 2;      // r0 - r2, r1 + r2, r2 - r1, r1 - r3
                float2 v = j == 1 ? make_float2(r[i][a].x + r[i][c].x, r[i][a].y + r[i][c].y) : make_float2(r[i][a].x - r[i][c].x, r[i][a].y - r[i][c].y);
                if (RELU) v = make_float2(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f));
                if (SIGNS) { m |= v.x > 0.f ? 1u << (4 * i + j) : 0u; m2 |= v.y > 0.f ? 1u << (4 * i + j) : 0u; }
                *reinterpret_cast<float2 *>(Vb + (size_t)plane_bytes * (4 * i + j) + off) = v;
            }
        if (SIGNS) *reinterpret_cast<unsigned *>(reinterpret_cast<char *>(signs) + (off >> 1)) = m | (m2 << 16);
        if (++q >= q1) break;
        off += (unsigned)C * 4u;
        P += kPairPitch;                  // two slots, in units of two floats
        if (++tw == nW) {                 // a new row: over the last two slots of this one and one more row
            tw = 0;
            ++tr;
            P += (PW + 2) * (kPairPitch / 2);
            column(0);
            column(1);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) { r[i][0] = r[i][2]; r[i][1] = r[i][3]; }
        }
    }
}


// ------------------------------------------------------------------------------------------
// Backward gather for one 2x2 output block (bh,bw) and VEC channels.
// dX[2bh+a][2bw+e] = sum over the 3x3 neighbourhood of tiles of G[y][x], y = a+1-2*dth,
// x = e+1-2*dtw, G = B g B^T, i.e. G[y][x] = sum_ij BT[i][y] BT[j][x] g[i][j].
// Everything below is unrolled with compile-time coefficients: the centre tile contributes
// its 16 values, the 4 edge neighbours 4 each, the 4 corner neighbours one each.
// ------------------------------------------------------------------------------------------
__host__ __device__ constexpr bool row_needed(int dt, int i)
{
    // dt=0 touches y in {1,2} (all i); dt=-1 touches y=3 (i=3 only); dt=+1 touches y=0 (i=0 only)
    return dt == 0 ? true : (dt < 0 ? i == 3 : i == 0);
}

// MASK: the ReLU mask of a gradient, none, V > 0, or bits (signs_t)
enum { kNoMask = 0, kMaskV = 1, kMaskBits = 2 };
__device__ __forceinline__ float keep_bits(float g, unsigned m, int t) { return (m >> t) & 1u ? g : 0.f; }
__device__ __forceinline__ float2 keep_bits(float2 g, unsigned m, int t)
{
    return make_float2((m >> t) & 1u ? g.x : 0.f, (m >> (16 + t)) & 1u ? g.y : 0.f);
}
__device__ __forceinline__ float4 keep_bits(float4 g, uint2 m, int t)
{
    return make_float4((m.x >> t) & 1u ? g.x : 0.f, (m.x >> (16 + t)) & 1u ? g.y : 0.f, (m.y >> t) & 1u ? g.z : 0.f, (m.y >> (16 + t)) & 1u ? g.w : 0.f);
}
__device__ __forceinline__ float2 ldg(const float2 *p) { return __ldg(p); }
__device__ __forceinline__ float2 zero_of(float2) { return make_float2(0.f, 0.f); }
__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
template <> struct Vec<2> { using type = float2; };
// the bits of the channels a lane holds at element `at` of [P][C / VEC]
template <typename T> struct SignBits;
template <> struct SignBits<float>  { unsigned m; __device__ __forceinline__ void load(const void *s, long long at) { m = __ldg(static_cast<const signs_t *>(s) + at); } };
template <> struct SignBits<float2> { unsigned m; __device__ __forceinline__ void load(const void *s, long long at) { m = __ldg(static_cast<const unsigned *>(s) + at); } };
template <> struct SignBits<float4> { uint2 m;    __device__ __forceinline__ void load(const void *s, long long at) { m = __ldg(static_cast<const uint2 *>(s) + at); } };

// ------------------------------------------------------------------------------------------
// Backward gather along a row of tiles (without a mask or with bits).  The sums over the tile rows come first, per tile column
// and Winograd column j
//   h0[j] = g1j - g2j + g3j - g3j(tile above),  h1[j] = g1j + g2j - g0j + g0j(tile below)
// and the two pixels of a tile in output row a are  h[1] - h[2] + h[3] - h[3](tile left)  and  h[1] + h[2] - h[0] + h[0](tile
// right), so that a walk along the row loads 24 values per tile (16, 4 above, 4 below) where a gather on its own loads 36,
// and keeps the neighbours' sums in registers.  put(a, x, value): pixel x of output row a.  (For NHWC the gather per tile
// stays: 54 against 59 us at 64 x 64 x 56 x 56, its 36 independent loads hide more latency.)
// ------------------------------------------------------------------------------------------
template <typename T, int MASK, typename Put>
__device__ __forceinline__ void imtrans_bwd_walk(const T *__restrict__ dV, const void *__restrict__ Vm, long long plane, int b, int th, int tw0,
                                                 int tw1, int nH, int nW, int CV, int cv, Put put)
{
    const long long row = (((long long)b * nH + th) * nW) * CV + cv, up = (long long)nW * CV;
    const bool above = th > 0, below = th + 1 < nH;
    auto get = [&](int t, long long at, const SignBits<T> &bits) {
        const T g = ldg(dV + (long long)t * plane + at);
        return MASK == kMaskBits ? keep_bits(g, bits.m, t) : g;
    };
    auto sums = [&](int tw, int j0, int j1, T (&h0)[4], T (&h1)[4]) {
        const long long at = row + (long long)tw * CV;
        SignBits<T> bc = {}, ba = {}, bb = {};
        if (MASK == kMaskBits) {
            bc.load(Vm, at);
            if (above) ba.load(Vm, at - up);
            if (below) bb.load(Vm, at + up);
        }
        T ga[4], gb[4], g[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j < j0 || j >= j1) continue;
#pragma unroll
            for (int i = 0; i < 4; ++i) g[i][j] = get(4 * i + j, at, bc);
            ga[j] = above ? get(12 + j, at - up, ba) : zero_of(T());
            gb[j] = below ? get(j, at + up, bb) : zero_of(T());
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j < j0 || j >= j1) continue;
            h0[j] = g[1][j] - g[2][j] + g[3][j] - ga[j];
            h1[j] = g[1][j] + g[2][j] - g[0][j] + gb[j];
        }
    };
    T h[2][4], left[2] = {zero_of(T()), zero_of(T())}, odd[2];
    if (tw0 > 0) {
        sums(tw0 - 1, 3, 4, h[0], h[1]);
        left[0] = h[0][3]; left[1] = h[1][3];
    }
#pragma unroll 1
    for (int tw = tw0; tw < tw1; ++tw) {
        sums(tw, 0, 4, h[0], h[1]);
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            if (tw > tw0) put(a, 2 * tw - 1, odd[a] + h[a][0]);
            put(a, 2 * tw, h[a][1] - h[a][2] + h[a][3] - left[a]);
            odd[a] = h[a][1] + h[a][2] - h[a][0];
            left[a] = h[a][3];
        }
    }
    if (tw1 < nW) {
        sums(tw1, 0, 1, h[0], h[1]);
        put(0, 2 * tw1 - 1, odd[0] + h[0][0]);
        put(1, 2 * tw1 - 1, odd[1] + h[1][0]);
    } else {
        put(0, 2 * tw1 - 1, odd[0]);
        put(1, 2 * tw1 - 1, odd[1]);
    }
}

template <typename T, int MASK>
__device__ __forceinline__ void imtrans_bwd_block(const T *__restrict__ dV, const void *__restrict__ Vm, long long plane,
                                                  int b, int bh, int bw, int nH, int nW, int CV, int cv, T (&out)[2][2])
{
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < 2; ++e) out[a][e] = zero_of(T());
#pragma unroll
    for (int dth = -1; dth <= 1; ++dth) {
        const int th = bh + dth;
        if (th < 0 || th >= nH) continue;
#pragma unroll
        for (int dtw = -1; dtw <= 1; ++dtw) {
            const int tw = bw + dtw;
            if (tw < 0 || tw >= nW) continue;
            const long long base = (((long long)b * nH + th) * nW + tw) * CV + cv;
            SignBits<T> bits = {};
            if (MASK == kMaskBits) bits.load(Vm, base);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (!row_needed(dth, i) || !row_needed(dtw, j)) continue;
                    T g = ldg(dV + (long long)(4 * i + j) * plane + base);
                    if (MASK == kMaskV) g = keep_where_pos(g, ldg(static_cast<const T *>(Vm) + (long long)(4 * i + j) * plane + base));
                    if (MASK == kMaskBits) g = keep_bits(g, bits.m, 4 * i + j);
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int y = a + 1 - 2 * dth, x = e + 1 - 2 * dtw;
                            if (y < 0 || y > 3 || x < 0 || x > 3) continue;
                            const int cf = bt_coef(i, y) * bt_coef(j, x);
                            if (cf > 0) out[a][e] = out[a][e] + g;
                            if (cf < 0) out[a][e] = out[a][e] - g;
                        }
                    }
                }
            }
        }
    }
}

template <int VEC, int MASK>
__global__ void __launch_bounds__(256) imtrans_bwd_nhwc_kernel(const float *__restrict__ dV, const void *__restrict__ Vm,
                                                                 float *__restrict__ dX, int B, int H, int W, int C, int nH, int nW)
{
    after_previous_kernel(dV, Vm, dX);
    using T = typename Vec<VEC>::type;
    const int CV = C / VEC;
    const long long total = (long long)B * nH * nW * CV;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const int cv = (int)(idx % CV);
    const long long p = idx / CV;
    const int bw = (int)(p % nW);
    const int bh = (int)((p / nW) % nH);
    const int b = (int)(p / ((long long)nW * nH));
    T out[2][2];
    imtrans_bwd_block<T, MASK>(reinterpret_cast<const T *>(dV), Vm,
                               (long long)B * nH * nW * CV, b, bh, bw, nH, nW, CV, cv, out);
    T *dXv = reinterpret_cast<T *>(dX);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int h = 2 * bh + a, w = 2 * bw + e;
            if (h < H && w < W) dXv[(((long long)b * H + h) * W + w) * CV + cv] = out[a][e];
        }
}

// NCHW, enough tiles to fill the GPU: the walk with lane = VEC channels over a band of R tile rows, each cut into segments of S
// tiles for the eight warps; the pixels collect in shared memory as [pixel][channel] and leave as one contiguous run per channel.
// 64 x 64 x 56 x 56 without a mask 84 us as gathers, 62 so (257 MB: 40 at the copy rate); 128 x 96 x 20 x 22 51 -> 30; with the ReLU
// mask 108 (V) -> 74 (bits).
template <int VEC, int MASK>
__global__ void __launch_bounds__(256, 3) imtrans_bwd_nchw_walk_kernel(const float *__restrict__ dV, const void *__restrict__ Vm,
                                                                         float *__restrict__ dX, int B, int H, int W, int C, int nH, int nW,
                                                                         int R, int nbands, int S, int nseg)
{
    after_previous_kernel(dV, Vm, dX);
    using T = typename Vec<VEC>::type;
    constexpr int CB = 32 * VEC, CBP = CB + (VEC == 1 ? 1 : 2);
    extern __shared__ __align__(16) float O[];          // [2R rows x W pixels][CBP]
    const int c0 = blockIdx.y * CB;
    const int band = blockIdx.x % nbands, b = blockIdx.x / nbands;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int th0 = band * R, rows = min(R, nH - th0);
    const int CV = C / VEC;
    if (c0 + VEC * lane < C) {
#pragma unroll 1
        for (int q = warp; q < rows * nseg; q += 8) {
            const int tr = q / nseg, seg = q - tr * nseg, tw0 = seg * S;
            if (tw0 >= nW) continue;
            float *const o = O + 2 * tr * W * CBP + VEC * lane;
            imtrans_bwd_walk<T, MASK>(reinterpret_cast<const T *>(dV), Vm, (long long)B * nH * nW * CV, b, th0 + tr, tw0, min(tw0 + S, nW), nH, nW,
                                      CV, c0 / VEC + lane, [&](int a, int x, T v) {
                                          if (x < W) *reinterpret_cast<T *>(o + (a * W + x) * CBP) = v;
                                      });
        }
    }
    __syncthreads();
    const int n = (min(2 * (th0 + rows), H) - 2 * th0) * W, nch = min(CB, C - c0);
    for (int c = warp; c < nch; c += 8) {
        float *d = dX + (((long long)b * C + c0 + c) * H + 2 * th0) * W;
        for (int i = lane; i < n; i += 32) d[i] = O[i * CBP + c];
    }
}

// NCHW: the same gather with the channel index fastest across a warp (coalesced dV reads), then a
// shared-memory turn so that dX rows are written contiguously along W.
template <int MASK>
__global__ void __launch_bounds__(256) imtrans_bwd_nchw_kernel(const float *__restrict__ dV, const void *__restrict__ Vm,
                                                                 float *__restrict__ dX, int B, int H, int W, int C, int nH, int nW)
{
    after_previous_kernel(dV, Vm, dX);
    constexpr int OP = 2 * kTSEG + 1;  // 65: odd pitch per (c,a) row
    __shared__ float O[kCCH * 2 * OP];
    const int nseg = cdiv(nW, kTSEG);
    int bx = blockIdx.x;
    const int seg = bx % nseg; bx /= nseg;
    const int bh = bx % nH;
    const int b = bx / nH;
    const int c0 = blockIdx.y * kCCH;
    const int bw0 = seg * kTSEG;
    const int tid = threadIdx.x;
    const int c = tid & 31;
    const long long plane = (long long)B * nH * nW * C;
#pragma unroll 1
    for (int it = 0; it < kTSEG / 8; ++it) {
        const int bwl = (tid >> 5) + 8 * it;
        const int bw = bw0 + bwl;
        float out[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
        if (bw < nW && c0 + c < C)
            imtrans_bwd_block<float, MASK>(dV, Vm, plane, b, bh, bw, nH, nW, C, c0 + c, out);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int e = 0; e < 2; ++e) O[(c * 2 + a) * OP + 2 * bwl + e] = out[a][e];
    }
    __syncthreads();
    for (int idx = tid; idx < kCCH * 2 * 2 * kTSEG; idx += 256) {
        const int x = idx % (2 * kTSEG);
        const int a = (idx / (2 * kTSEG)) & 1;
        const int cc = idx / (4 * kTSEG);
        const int h = 2 * bh + a, w = 2 * bw0 + x;
        if (c0 + cc < C && h < H && w < W)
            dX[(((long long)b * C + c0 + cc) * H + h) * W + w] = O[(cc * 2 + a) * OP + x];
    }
}

// NCHW, image rows up to 192 pixels, with V as the mask or too few tiles for the walk above to fill the GPU: the same gather with
// lane = VEC consecutive channels over a band of R tile rows; the 2R x W output pixels of each channel collect in shared memory (odd
// pitch between channels) and leave as one contiguous run per channel -- or, where the band is the whole image, as one contiguous run
// for all the block's channels.  VEC = 4 reads dV (and the ReLU mask) with 16-byte loads: LC = 32 lanes along the channels (128 per
// block, 512 bytes per request) where such a band fits four blocks per SM, else LC = 16 (64 channels per block, the two halves of a
// warp on two tiles at once).
template <int VEC, int LC, int MASK, bool SEG>
__global__ void __launch_bounds__(256, 4) imtrans_bwd_nchw_band_kernel(const float *__restrict__ dV, const void *__restrict__ Vm,
                                                                         float *__restrict__ dX, int B, int H, int W, int C, int nH,
                                                                         int nW, int R, int nbands, int S, int nsegs, int pitch)
{
    after_previous_kernel(dV, Vm, dX);
    using T = typename Vec<VEC>::type;
    constexpr int CB = LC * VEC;             // channels per block
    constexpr int QW = 32 / LC;              // tiles a warp works on at once
    extern __shared__ float O[];             // [CB channels][pitch]
    // Block order.  One input stream: a one-dimensional grid with the channel blocks fastest, so that neighbouring
    // blocks read neighbouring segments of every dV row.  With V as the mask (32 streams of rows open at once) that
    // order measured slower than images fastest, which is the two-dimensional grid (66 vs 78 us on
    // 256 x 512 x 7 x 7; without the mask 50 vs 58 us the other way).
    int c0, bb;
    if (MASK == kMaskV) {
        c0 = blockIdx.y * CB;
        bb = blockIdx.x;
    } else {
        const int ncb = (C + CB - 1) / CB;
        c0 = (int)(blockIdx.x % ncb) * CB;
        bb = blockIdx.x / ncb;
    }
    const int seg = SEG ? bb % nsegs : 0;
    if (SEG) bb /= nsegs;
    const int band = bb % nbands;
    const int b = bb / nbands;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lc = lane % LC, lq = lane / LC;
    const int th0 = band * R;
    const int rows_blk = min(R, nH - th0);
    const int tw0 = SEG ? seg * S : 0, ns = SEG ? min(S, nW - tw0) : nW;   // tile columns of the block
    const int OW = SEG ? min(2 * ns, W - 2 * tw0) : W;                     // pixels of an output row
    const int CV = C / VEC;
    const long long plane = (long long)B * nH * nW * CV;
    const bool c_ok = c0 + VEC * lc < C;
#pragma unroll 1
    for (int q = warp * QW + lq; q < rows_blk * ns; q += 8 * QW) {
        const int br = q / ns, bl = q - br * ns, bw = tw0 + bl;
        T out[2][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int e = 0; e < 2; ++e) out[a][e] = zero_of(T());
        if (c_ok)
            imtrans_bwd_block<T, MASK>(reinterpret_cast<const T *>(dV), Vm, plane, b, th0 + br, bw, nH,
                                       nW, CV, c0 / VEC + lc, out);
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (2 * bw + e < W) {
                    float *o = O + VEC * lc * pitch + (2 * br + a) * OW + 2 * bl + e;
                    put_lanes(o, pitch, out[a][e]);
                }
    }
    __syncthreads();
    const int lo = 2 * th0, hi = min(2 * th0 + 2 * rows_blk, H);
    const int n = (hi - lo) * OW;
    const int nch = min(CB, C - c0);
    if (n == H * W) {
        // the block's channels are one run of nch * H * W floats
        float *dst = dX + ((long long)b * C + c0) * n;
        for (int k = threadIdx.x; k < nch * n; k += 256) {
            const int cc = k / n;
            dst[k] = O[cc * pitch + (k - cc * n)];
        }
    } else {
        for (int cc = warp; cc < nch; cc += 8) {
            float *dst = dX + (((long long)b * C + c0 + cc) * H + lo) * W;
            const float *src = O + cc * pitch;
            if (!SEG) {
                for (int i = lane; i < n; i += 32) dst[i] = src[i];
            } else {                                         // two rows of a segment
                for (int i = lane; i < n; i += 32) dst[(i >= OW ? W : 0) + 2 * tw0 + (i >= OW ? i - OW : i)] = src[i];
            }
        }
    }
}


// NCHW, small images (a whole image of 128 or 64 channels fits shared memory): every value of dV is read from memory
// exactly once.  A block takes one image x CB channels; a warp takes one tile x 32 channels at a time (lane = channel:
// sixteen coalesced 128-byte loads), turns its sixteen gradients into the 4 x 4 window B g B^T and adds the window
// into the block's image in shared memory.  Windows of tiles two apart do not overlap, so the tiles are walked in four
// passes by the parity of (tile row, tile column) with a barrier between passes, and plain read-modify-writes suffice
// (no atomics: the result does not depend on the order of the warps).  The image is kept as [channel][pixel] with an
// odd pitch (lanes hit distinct banks) and leaves as one contiguous run: CB channels x H*W pixels are adjacent in dX.
template <int MASK>
__global__ void __launch_bounds__(256) imtrans_bwd_nchw_image_kernel(const float *__restrict__ dV, const void *__restrict__ Vm,
                                                                       float *__restrict__ dX, int B, int H, int W, int C, int nH, int nW,
                                                                       int CB, int pitch)
{
    after_previous_kernel(dV, Vm, dX);
    extern __shared__ float O[];                   // [CB][pitch]
    const int b = blockIdx.x, c0 = blockIdx.y * CB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int HW = H * W;
    const int nch = min(CB, C - c0);
    const int ngr = (nch + 31) >> 5;               // groups of 32 channels
    const long long plane = (long long)B * nH * nW * C;
    for (int k = threadIdx.x; k < CB * pitch; k += 256) O[k] = 0.f;
    __syncthreads();
#pragma unroll 1
    for (int pc = 0; pc < 4; ++pc) {
        const int pr = pc >> 1, pq = pc & 1;
        const int ntr = (nH - pr + 1) >> 1, ntc = (nW - pq + 1) >> 1;
        const int ntiles = ntr * ntc;
        // (tile, channel group) pairs go round the eight warps; with 1, 2, 4 or 8 groups a warp keeps its group and
        // walks the tiles with a fixed stride, which keeps divisions out of the loop
        const bool fixed = (8 % ngr) == 0;
        const int step = fixed ? 8 / ngr : 8;
        int gr = fixed ? warp % ngr : 0, tt = fixed ? warp / ngr : warp;
        int tr = tt / ntc, tc = tt - tr * ntc;
        const int items = fixed ? ntiles : ntiles * ngr;
#pragma unroll 1
        for (; tt < items; tt += step) {
            int th, tw;
            if (fixed) {
                th = 2 * tr + pr; tw = 2 * tc + pq;
                tc += step;
                while (tc >= ntc) { tc -= ntc; ++tr; }
            } else {
                gr = tt % ngr;
                const int t2 = tt / ngr;
                th = 2 * (t2 / ntc) + pr; tw = 2 * (t2 % ntc) + pq;
            }
            const int cl = gr * 32 + lane;
            if (cl < nch) {
                const float *gp = dV + ((((long long)b * nH + th) * nW + tw) * C + c0 + cl);
                const long long at = (((long long)b * nH + th) * nW + tw) * C + c0 + cl;
                float g[4][4];
#pragma unroll
                for (int t = 0; t < 16; ++t) g[t >> 2][t & 3] = __ldg(gp + (long long)t * plane);
                if (MASK == kMaskBits) {
                    SignBits<float> bits;
                    bits.load(Vm, at);
#pragma unroll
                    for (int t = 0; t < 16; ++t) g[t >> 2][t & 3] = keep_bits(g[t >> 2][t & 3], bits.m, t);
                }
                if (MASK == kMaskV) {
                    float v[16];
#pragma unroll
                    for (int t = 0; t < 16; ++t) v[t] = __ldg(static_cast<const float *>(Vm) + at + (long long)t * plane);
#pragma unroll
                    for (int t = 0; t < 16; ++t)
                        if (!(v[t] > 0.f)) g[t >> 2][t & 3] = 0.f;
                }
                // d = B g B^T, B[y][i] = Bt[i][y]: along one axis (u0..u3) -> (u0, u1 - u2 + u3, -u0 + u1 + u2, -u3)
                float r[4][4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    r[0][j] = g[0][j];
                    r[1][j] = g[1][j] - g[2][j] + g[3][j];
                    r[2][j] = g[1][j] + g[2][j] - g[0][j];
                    r[3][j] = -g[3][j];
                }
                float *o = O + cl * pitch;
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const int h = 2 * th - 1 + y;
                    if (h < 0 || h >= H) continue;
                    const float d0 = r[y][0], d1 = r[y][1] - r[y][2] + r[y][3], d2 = r[y][1] + r[y][2] - r[y][0], d3 = -r[y][3];
                    const int w0 = 2 * tw - 1;
                    float *row = o + h * W;
                    if (w0 >= 0) row[w0] += d0;
                    row[w0 + 1] += d1;
                    if (w0 + 2 < W) row[w0 + 2] += d2;
                    if (w0 + 3 < W) row[w0 + 3] += d3;
                }
            }
        }
        __syncthreads();
    }
    float *dst = dX + ((long long)b * C + c0) * HW;
    if (pitch == HW) {
        for (int k = threadIdx.x; k < nch * HW; k += 256) dst[k] = O[k];
    } else {   // a warp per channel: no division per element, and the channels' runs are adjacent in dX
        for (int c = warp; c < nch; c += 8) {
            const float *src = O + c * pitch;
            float *d = dst + c * HW;
            for (int i = lane; i < HW; i += 32) d[i] = src[i];
        }
    }
}

// The same with two channels per lane (8-byte loads, a warp covers a tile x 64 channels): half the instructions per byte,
// which is what this kernel is short of.  The image is kept as [pixel][channel] (channels innermost, so that the lanes'
// 8-byte read-modify-writes are conflict-free) with a pitch of CB + 2 floats, and leaves per channel through strided
// reads (two-way bank conflicts on the smaller side of the traffic).  Needs an even C and 8-byte aligned tensors.
template <int MASK>
__global__ void __launch_bounds__(256, 4) imtrans_bwd_nchw_image2_kernel(const float *__restrict__ dV, const void *__restrict__ Vm,
                                                                           float *__restrict__ dX, int B, int H, int W, int C, int nH,
                                                                           int nW, int CB)
{
    after_previous_kernel(dV, Vm, dX);
    extern __shared__ __align__(16) float O[];     // [H*W][CB + 2]
    const int b = blockIdx.x, c0 = blockIdx.y * CB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int HW = H * W, CBP = CB + 2;
    const int nch = min(CB, C - c0);
    const int ngr = (nch + 63) >> 6;               // groups of 64 channels
    const long long plane = (long long)B * nH * nW * C;
    for (int k = threadIdx.x; k < HW * CBP / 2; k += 256) reinterpret_cast<float2 *>(O)[k] = make_float2(0.f, 0.f);
    __syncthreads();
#pragma unroll 1
    for (int pc = 0; pc < 4; ++pc) {
        const int pr = pc >> 1, pq = pc & 1;
        const int ntr = (nH - pr + 1) >> 1, ntc = (nW - pq + 1) >> 1;
        const int items = ntr * ntc * ngr;
#pragma unroll 1
        for (int tt = warp; tt < items; tt += 8) {
            const int gr = tt % ngr, t2 = tt / ngr;
            const int th = 2 * (t2 / ntc) + pr, tw = 2 * (t2 % ntc) + pq;
            const int cl = gr * 64 + 2 * lane;
            if (cl < nch) {
                const long long base = (((long long)b * nH + th) * nW + tw) * C + c0 + cl;
                float2 g[4][4];
#pragma unroll
                for (int t = 0; t < 16; ++t) g[t >> 2][t & 3] = __ldg(reinterpret_cast<const float2 *>(dV + base + (long long)t * plane));
                if (MASK == kMaskBits) {
                    SignBits<float2> bits;
                    bits.load(Vm, base >> 1);
#pragma unroll
                    for (int t = 0; t < 16; ++t) g[t >> 2][t & 3] = keep_bits(g[t >> 2][t & 3], bits.m, t);
                }
                if (MASK == kMaskV) {
#pragma unroll
                    for (int t = 0; t < 16; ++t) {
                        const float2 v = __ldg(reinterpret_cast<const float2 *>(static_cast<const float *>(Vm) + base + (long long)t * plane));
                        if (!(v.x > 0.f)) g[t >> 2][t & 3].x = 0.f;
                        if (!(v.y > 0.f)) g[t >> 2][t & 3].y = 0.f;
                    }
                }
                // d = B g B^T: along one axis (u0..u3) -> (u0, u1 - u2 + u3, -u0 + u1 + u2, -u3); rows in place
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 u1 = g[1][j], u2 = g[2][j];
                    g[1][j] = u1 - u2 + g[3][j];
                    g[2][j] = u1 + u2 - g[0][j];
                    g[3][j] = make_float2(-g[3][j].x, -g[3][j].y);
                }
                float *o = O + cl;
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const int h = 2 * th - 1 + y;
                    if (h < 0 || h >= H) continue;
                    const float2 d0 = g[y][0], d1 = g[y][1] - g[y][2] + g[y][3], d2 = g[y][1] + g[y][2] - g[y][0],
                                 d3 = make_float2(-g[y][3].x, -g[y][3].y);
                    const int w0 = 2 * tw - 1;
                    float *row = o + (h * W + w0) * CBP;
                    if (w0 >= 0) { float2 *q = reinterpret_cast<float2 *>(row); *q = *q + d0; }
                    { float2 *q = reinterpret_cast<float2 *>(row + CBP); *q = *q + d1; }
                    if (w0 + 2 < W) { float2 *q = reinterpret_cast<float2 *>(row + 2 * CBP); *q = *q + d2; }
                    if (w0 + 3 < W) { float2 *q = reinterpret_cast<float2 *>(row + 3 * CBP); *q = *q + d3; }
                }
            }
        }
        __syncthreads();
    }
    // a warp per channel: its H*W pixels are one contiguous run of dX, and the channels' runs are adjacent
    float *dst = dX + ((long long)b * C + c0) * HW;
    for (int c = warp; c < nch; c += 8) {
        float *d = dst + c * HW;
        for (int i = lane; i < HW; i += 32) d[i] = O[i * CBP + c];
    }
}

// ------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------
static bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int imtrans_fwd(const float *X, float *V, void *signs_out, int B, int H, int W, int C, int layout, int relu, const float *scale,
                const float *shift, cudaStream_t st)
{
    if (!X || !V || B <= 0 || H <= 0 || W <= 0 || C <= 0) return WG2X2_ERR_BAD_ARG;
    if ((scale == nullptr) != (shift == nullptr)) return WG2X2_ERR_BAD_ARG;
    signs_t *signs = static_cast<signs_t *>(signs_out);
    if (signs && (scale || !relu || !aligned16(signs))) return WG2X2_ERR_BAD_ARG;      // the ReLU's mask of a layer without an affine map
    if (layout != WG2X2_NHWC && layout != WG2X2_NCHW) return WG2X2_ERR_BAD_ARG;
    const int nH = (H + 1) / 2, nW = (W + 1) / 2;
    if (layout == WG2X2_NHWC) {
        if ((C % 4 == 0) && aligned16(X) && aligned16(V) && (!scale || (aligned16(scale) && aligned16(shift)))) {
            const long long total = (long long)B * nH * nW * (C / 4);
            const unsigned g = (unsigned)cdivll(total, 256);
            launch(scale ? imtrans_fwd_nhwc_kernel<4, true, false> : signs ? imtrans_fwd_nhwc_kernel<4, false, true> : imtrans_fwd_nhwc_kernel<4, false, false>,
                   dim3(g), 256, 0, st, X, V, signs, B, H, W, C, nH, nW, relu, scale, shift);
        } else {
            const long long total = (long long)B * nH * nW * C;
            const unsigned g = (unsigned)cdivll(total, 256);
            launch(scale ? imtrans_fwd_nhwc_kernel<1, true, false> : signs ? imtrans_fwd_nhwc_kernel<1, false, true> : imtrans_fwd_nhwc_kernel<1, false, false>,
                   dim3(g), 256, 0, st, X, V, signs, B, H, W, C, nH, nW, relu, scale, shift);
        }
    } else {
        const long long gx = (long long)B * nH * cdiv(nW, kTSEG);
        if (gx > 0x7fffffffLL || cdiv(C, kCCH) > 65535) return WG2X2_ERR_UNSUPPORTED;
        dim3 grid((unsigned)gx, cdiv(C, kCCH));
        // Two channels per lane where a row of tiles is short (the one-channel kernel's predicates and divisions weigh more there:
        // 256 x 512 x 7 x 7 39 -> 34 us, 256 x 256 x 14 x 14 59 -> 53, 32 x 256 x 28 x 28 32 -> 31, but 54 -> 58 at 56 x 56),
        // blocks of 64 channels are full, the bands fill the GPU, and a plane is within 32-bit reach.
        const bool pair_ok = C % kPairCB == 0 && W <= 28 && ((reinterpret_cast<uintptr_t>(V) | reinterpret_cast<uintptr_t>(scale) |
                             reinterpret_cast<uintptr_t>(shift)) & 7u) == 0 && (long long)B * nH * nW * C < (1LL << 30) && C / kPairCB <= 65535;
        const int R = pair_ok ? pair_rows(B, C, nH, nW, W, 2) : 0;
        if (R) {
            const int nbands = cdiv(nH, R), smem = (2 * R + 2) * (2 * nW + 2) * kPairPitch * (int)sizeof(float);
            if ((long long)B * nbands > 0x7fffffffLL) return WG2X2_ERR_UNSUPPORTED;
            auto *kernel = scale ? (relu ? imtrans_fwd_nchw_pair_kernel<true, true, false> : imtrans_fwd_nchw_pair_kernel<true, false, false>)
                         : signs ? imtrans_fwd_nchw_pair_kernel<false, true, true>
                                 : (relu ? imtrans_fwd_nchw_pair_kernel<false, true, false> : imtrans_fwd_nchw_pair_kernel<false, false, false>);
            launch(kernel, dim3((unsigned)(B * nbands), C / kPairCB), 256, smem, st, X, V, signs, H, W, C, nH, nW, R, nbands,
                   (unsigned)cdiv(1 << 20, 2 * nW + 2), (unsigned)((long long)B * nH * nW * C * 4), scale, shift);
        } else if (W <= 128) {
            const BandCut cut = cut_bands(nH, nW, (long long)B * cdiv(C, 32), (kBandFloats / W - 2) / 2);
            const int pitch = ((2 * cut.R + 2) * (cut.nsegs == 1 ? W : 2 * cut.S + 2)) | 1;
            const int smem = 32 * pitch * (int)sizeof(float);
            const long long gxb = (long long)B * cut.nbands * cut.nsegs;
            if (gxb > 0x7fffffffLL) return WG2X2_ERR_UNSUPPORTED;
            const dim3 gb((unsigned)gxb, cdiv(C, 32));
            if (cut.nsegs == 1)
                launch(scale ? imtrans_fwd_nchw_band_kernel<true, false> : signs ? imtrans_fwd_nchw_band_kernel<false, true> : imtrans_fwd_nchw_band_kernel<false, false>,
                       gb, 256, smem, st, X, V, signs, B, H, W, C, nH,
                       nW, relu, cut.R, cut.nbands, pitch, scale, shift);
            else
                launch(scale ? imtrans_fwd_nchw_row_kernel<true, false> : signs ? imtrans_fwd_nchw_row_kernel<false, true> : imtrans_fwd_nchw_row_kernel<false, false>,
                       gb, 256, smem, st, X, V, signs, B, H, W, C, nH, nW,
                       relu, cut.S, cut.nsegs, pitch, scale, shift);
        } else {
            launch(imtrans_fwd_nchw_kernel, grid, 256, 0, st, X, V, signs, B, H, W, C, nH, nW, relu, scale, shift);
        }
    }
    return launch_status();
}

// The kernel of a family for the kind of mask
#define WG_BY_MASK(...) (mask == kNoMask ? WG_INST(kNoMask, __VA_ARGS__) : mask == kMaskV ? WG_INST(kMaskV, __VA_ARGS__) : WG_INST(kMaskBits, __VA_ARGS__))

// Vm: the mask, V itself (mask_bits == 0) or its bits as imtrans_fwd wrote them; NULL: none
int imtrans_bwd(const float *dV, const void *Vm, int mask_bits, float *dX, int B, int H, int W, int C, int layout, cudaStream_t st)
{
    if (!dV || !dX || B <= 0 || H <= 0 || W <= 0 || C <= 0) return WG2X2_ERR_BAD_ARG;
    if (layout != WG2X2_NHWC && layout != WG2X2_NCHW) return WG2X2_ERR_BAD_ARG;
    const int nH = (H + 1) / 2, nW = (W + 1) / 2;
    const int mask = !Vm ? kNoMask : mask_bits ? kMaskBits : kMaskV;
    // n-byte accesses to dV and to the mask (`n` bytes of V are n / 2 bytes of bits)
    const auto on = [&](uintptr_t n) {
        return (reinterpret_cast<uintptr_t>(dV) & (n - 1)) == 0 && (reinterpret_cast<uintptr_t>(Vm) & ((mask == kMaskBits ? n / 2 : n) - 1)) == 0;
    };
    if (layout == WG2X2_NHWC) {
        const bool vec = C % 4 == 0 && on(16) && aligned16(dX);
        const long long grid = cdivll((long long)B * nH * nW * (vec ? C / 4 : C), 256);
        if (grid > 0x7fffffffLL) return WG2X2_ERR_UNSUPPORTED;
#define WG_INST(M, V) imtrans_bwd_nhwc_kernel<V, M>
        launch(vec ? WG_BY_MASK(4) : WG_BY_MASK(1), dim3((unsigned)grid), 256, 0, st, dV, Vm, dX, B, H, W, C, nH, nW);
#undef WG_INST
        return launch_status();
    }
    // small images: one block per image and channel block, every value of dV read once (above 64 pixels the walk below is faster
    // unless it would have V for a mask: 256 x 256 x 14 x 14 68 against 59 us, 256 x 512 x 7 x 7 37 against 39)
    const int HW = H * W;
    if (HW <= (mask == kMaskV ? 200 : 64) && (long long)B * cdiv(C, HW <= 64 ? 128 : 64) >= 2LL * kNumSMs && cdiv(C, HW <= 64 ? 128 : 64) <= 65535) {
        const int CB = HW <= 64 ? 128 : 64;
        const dim3 grid((unsigned)B, cdiv(C, CB));
        if ((C & 1) == 0 && on(8)) {      // two channels per lane
#define WG_INST(M, V) imtrans_bwd_nchw_image2_kernel<M>
            launch(WG_BY_MASK(0), grid, 256, HW * (CB + 2) * sizeof(float), st, dV, Vm, dX, B, H, W, C, nH, nW, CB);
#undef WG_INST
        } else {
            const int pitch = HW | 1;
#define WG_INST(M, V) imtrans_bwd_nchw_image_kernel<M>
            launch(WG_BY_MASK(0), grid, 256, CB * pitch * sizeof(float), st, dV, Vm, dX, B, H, W, C, nH, nW, CB, pitch);
#undef WG_INST
        }
        return launch_status();
    }
    if (W <= 192) {
        // The walk, except with V as the mask (it holds too much then: 141 against 108 us at 64 x 64 x 56 x 56).  Two channels per lane
        // where the last block of 64 is more than half full and there is no mask (with bits 81 against 74 us); bands as high as
        // leave the busiest SM least to do, below 64 KB of shared memory.
        const bool two = mask == kNoMask && (C & 1) == 0 && on(8) && (C % 64 == 0 || C % 64 > 32);
        const int cb = two ? 64 : 32, px = (two ? cb + 2 : cb + 1) * (int)sizeof(float);
        int R = 0;
        double t = 1e300;
        for (int r = 1; mask != kMaskV && r <= nH && (r == 1 || 2 * r * W * px <= 64 * 1024); ++r) {
            const long long ctas = (long long)B * cdiv(nH, r) * cdiv(C, cb);
            if (ctas < 3LL * kNumSMs) break;
            const double u = (double)cdivll(ctas, 3 * kNumSMs) * (r * nW + 8.0);
            if (u < t) { t = u; R = r; }
        }
        if (R && cdiv(C, cb) <= 65535 && (long long)B * cdiv(nH, R) <= 0x7fffffffLL) {
            R = cdiv(nH, cdiv(nH, R));
            const int nbands = cdiv(nH, R), S = cdiv(nW, R >= 8 ? 1 : cdiv(8, R)), nseg = cdiv(nW, S);
            launch(two ? imtrans_bwd_nchw_walk_kernel<2, kNoMask> : mask == kNoMask ? imtrans_bwd_nchw_walk_kernel<1, kNoMask>
                                                                 : imtrans_bwd_nchw_walk_kernel<1, kMaskBits>,
                   dim3((unsigned)(B * nbands), cdiv(C, cb)), 256, 2 * R * W * px, st, dV, Vm, dX, B, H, W, C, nH, nW, R, nbands, S, nseg);
            return launch_status();
        }
        // four channels per lane (16-byte loads) where the channels allow it; 128 channels per block where a band of
        // them stays below 50 KB (four blocks per SM), else 64
        // -- and where that still leaves four CTAs for every SM (a small batch keeps the narrower blocks)
        auto ctas = [&](int cbk, int band_floats) { return (long long)B * cdiv(nH, max(1, min(nH, band_floats / (2 * W)))) * cdiv(C, cbk); };
        const long long fill = 4LL * kNumSMs;
        const bool vec_ok = mask == kMaskV && (C % 4 == 0) && C >= 64 && on(16) && 2 * W <= kBandFloats / 2;
        const bool wide = vec_ok && C >= 128 && 2 * W <= kBandFloats / 4 && ctas(128, kBandFloats / 4) >= fill;
        const bool vec = wide || (vec_ok && ctas(64, kBandFloats / 2) >= fill);
        const int bcb = wide ? 128 : (vec ? 64 : 32);
        const int max_rows = (wide ? kBandFloats / 4 : (vec ? kBandFloats / 2 : kBandFloats)) / (2 * W);
        const BandCut cut = cut_bands(nH, nW, (long long)B * cdiv(C, bcb), max_rows);
        const int pitch = (2 * cut.R * (cut.nsegs == 1 ? W : 2 * cut.S)) | 1;
        const long long blocks = (long long)B * cut.nbands * cut.nsegs;
        if (blocks * cdiv(C, bcb) > 0x7fffffffLL || cdiv(C, bcb) > 65535) return WG2X2_ERR_UNSUPPORTED;
        const dim3 grid = mask == kMaskV ? dim3((unsigned)blocks, cdiv(C, bcb)) : dim3((unsigned)(blocks * cdiv(C, bcb)));
        // (the kernels with wider blocks are only taken where those already fill the GPU: they have no segments)
#define WG_INST(M, S) imtrans_bwd_nchw_band_kernel<1, 32, M, S>
        launch(wide ? imtrans_bwd_nchw_band_kernel<4, 32, kMaskV, false> : vec ? imtrans_bwd_nchw_band_kernel<4, 16, kMaskV, false>
                    : cut.nsegs == 1 ? WG_BY_MASK(false) : WG_BY_MASK(true),
               grid, 256, bcb * pitch * sizeof(float), st, dV, Vm, dX, B, H, W, C, nH, nW, cut.R, cut.nbands, cut.S, cut.nsegs, pitch);
#undef WG_INST
        return launch_status();
    }
    const long long gx = (long long)B * nH * cdiv(nW, kTSEG);
    if (gx > 0x7fffffffLL || cdiv(C, kCCH) > 65535) return WG2X2_ERR_UNSUPPORTED;
#define WG_INST(M, V) imtrans_bwd_nchw_kernel<M>
    launch(WG_BY_MASK(0), dim3((unsigned)gx, cdiv(C, kCCH)), 256, 0, st, dV, Vm, dX, B, H, W, C, nH, nW);
#undef WG_INST
    return launch_status();
}

}  // namespace wg
