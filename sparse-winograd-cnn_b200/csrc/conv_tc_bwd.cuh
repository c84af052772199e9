// Tensor-core gradient products.  Included by conv_tc.cu (same translation unit: the kernels share the
// PTX wrappers, the status word and the plane-mode instantiation of the tcgen05 kernel).
//
//   dM  = A dY A^T           conv_dm_*_kernel: one HBM-bound pass, 16 planes [t][P][K], rounded to TF32
//   dV_t = dM_t . W_t^T      conv_grad_gemm_tc_kernel<1> (A = dM, B = W as stored: (16,C,K) is already
//                            contraction-contiguous for this product), ReLU mask in the epilogue
//   dW_t = V_t^T . dM_t      conv_grad_gemm_tc_kernel<0> (both operands MN-major), split over P
#pragma once

static inline bool misaligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; }   // NULL passes

// ---------------------------------------------------------------------------------------
// dM producer
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ float round_tf32(float x)
{
    uint32_t u;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(x));
    return __uint_as_float(u);
}
// The bits of x for an operand that only the tensor core reads, which keeps the upper 19: half a unit of the last kept place added
// rounds to nearest as the conversion does, for an integer add.  NaN is set apart: CUDA's own, 0x7fffffff, would wrap to -0.
__device__ __forceinline__ uint32_t tf32_operand(float x) { return x == x ? __float_as_uint(x) + 0x1000u : 0x7fffffffu; }

// NHWC: one thread = one tile x 4 output channels
__global__ void __launch_bounds__(256) conv_dm_nhwc_kernel(const float *__restrict__ dY, float *__restrict__ dM, long long P, int nH,
                                                             int nW, int H, int W, int K)
{
    after_previous_kernel(dY, dM);
    const int KV = K >> 2;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= P * KV) return;
    const int kv = (int)(idx % KV);
    const long long p = idx / KV;
    const int tw = (int)(p % nW), th = (int)((p / nW) % nH), b = (int)(p / ((long long)nW * nH));
    float4 g[2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int h = 2 * th + a, w = 2 * tw + e;
            g[a][e] = (h < H && w < W) ? __ldg(reinterpret_cast<const float4 *>(dY + (((long long)b * H + h) * W + w) * K) + kv)
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    float m0[4][4], m1[4][4], m2[4][4], m3[4][4];
    a_g_at(g[0][0].x, g[0][1].x, g[1][0].x, g[1][1].x, m0);
    a_g_at(g[0][0].y, g[0][1].y, g[1][0].y, g[1][1].y, m1);
    a_g_at(g[0][0].z, g[0][1].z, g[1][0].z, g[1][1].z, m2);
    a_g_at(g[0][0].w, g[0][1].w, g[1][0].w, g[1][1].w, m3);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            reinterpret_cast<float4 *>(dM + ((long long)(4 * i + j) * P + p) * K)[kv] =
                make_float4(round_tf32(m0[i][j]), round_tf32(m1[i][j]), round_tf32(m2[i][j]), round_tf32(m3[i][j]));
}

// NCHW: a CTA stages a band of 2R rows of dY (or two rows of a segment of S tiles) for 32 channels, then walks tiles with
// lane = channel so that the plane stores are contiguous along K.  Any layout/width: R >= 1.
template <bool SEG>
__global__ void __launch_bounds__(256) conv_dm_nchw_kernel(const float *__restrict__ dY, float *__restrict__ dM, long long P, int nH,
                                                             int nW, int H, int W, int K, int R, int nbands, int S_, int nsegs, int pitch)
{
    after_previous_kernel(dY, dM);
    extern __shared__ float S[];
    int bb = blockIdx.x;
    const int seg = SEG ? bb % nsegs : 0;
    if (SEG) bb /= nsegs;
    const int band = bb % nbands;
    const int b = bb / nbands;
    const int k0 = blockIdx.y * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int th0 = band * R;
    const int rows_tile = min(R, nH - th0);
    const int tw0 = SEG ? seg * S_ : 0, ns = SEG ? min(S_, nW - tw0) : nW;
    const int w0 = 2 * tw0, SW = SEG ? min(2 * ns, W - w0) : W;      // pixels of a staged row
    const int lo = 2 * th0, hi = min(2 * th0 + 2 * rows_tile, H);
    const int nfill = (hi - lo) * SW;
    if (SEG) {       // two rows of a segment
        stage_channels(dY + (((long long)b * K + k0) * H + lo) * W + w0, (long long)H * W, K - k0, nfill, S, pitch,
                       [&](int i) { return i >= SW ? W + i - SW : i; });
    } else {
        for (int kk = warp; kk < 32; kk += 8) {
            if (k0 + kk >= K) break;
            const float *src = dY + (((long long)b * K + k0 + kk) * H + lo) * W;
            float *dst = S + kk * pitch;
            for (int i = lane; i < nfill; i += 32) dst[i] = __ldg(src + i);
        }
    }
    __syncthreads();
    if (k0 + lane >= K) return;
    const float *Sk = S + lane * pitch;
#pragma unroll 1
    for (int q = warp; q < rows_tile * ns; q += 8) {
        const int tr = q / ns, tl = q - tr * ns;
        float g[2][2];
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int h = lo + 2 * tr + a, w = 2 * tl + e;
                g[a][e] = (h < H && w < SW) ? Sk[(2 * tr + a) * SW + w] : 0.f;
            }
        float m[4][4];
        a_g_at(g[0][0], g[0][1], g[1][0], g[1][1], m);
        const long long p = ((long long)b * nH + th0 + tr) * nW + tw0 + tl;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dM[((long long)(4 * i + j) * P + p) * K + k0 + lane] = round_tf32(m[i][j]);
    }
}

// The same for whole blocks of 64 channels and enough tiles to fill the GPU: two channels per lane off an asynchronously staged
// image, 256 bytes per store off uniform plane addresses.  dM is only ever read by the tensor core: tf32_operand.  256 x 512 x 7 x 7
// 36 -> 28 us (160 MB: 25 at the copy rate), dM and dW of 256 x 256 x 14 x 14 136 -> 128, of 64 x 64 x 56 x 56 128 -> 120.
__global__ void __launch_bounds__(256, 4) conv_dm_nchw_pair_kernel(const float *__restrict__ dY, float *__restrict__ dM, int nH, int nW, int H,
                                                                     int W, int K, int R, int nbands, unsigned inv, unsigned plane_bytes)
{
    after_previous_kernel(dY, dM);
    extern __shared__ __align__(16) float S[];
    const int band = blockIdx.x % nbands, b = blockIdx.x / nbands, k0 = blockIdx.y * kPairCB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int th0 = band * R, rows = min(R, nH - th0), PW = 2 * nW;
    stage_pairs(dY, S, b, k0, K, H, W, 2 * th0, 0, 2 * rows, PW, inv);
    __syncthreads();
    char *const Mb = reinterpret_cast<char *>(dM);
    const int n = rows * nW;
#pragma unroll 2
    for (int q = warp; q < n; q += 8) {
        const int tr = q / nW, tw = q - tr * nW;
        const float2 *p = reinterpret_cast<const float2 *>(S + (2 * tr * PW + 2 * tw) * kPairPitch) + lane;
        const float2 g00 = p[0], g01 = p[kPairPitch / 2], g10 = p[PW * (kPairPitch / 2)], g11 = p[(PW + 1) * (kPairPitch / 2)];
        float m0[4][4], m1[4][4];
        a_g_at(g00.x, g01.x, g10.x, g11.x, m0);
        a_g_at(g00.y, g01.y, g10.y, g11.y, m1);
        const unsigned off = (unsigned)((((long long)b * nH + th0) * nW + q) * K + k0 + 2 * lane) * 4u;
#pragma unroll
        for (int t = 0; t < 16; ++t)
            *reinterpret_cast<uint2 *>(Mb + (size_t)plane_bytes * t + off) =
                make_uint2(tf32_operand(m0[t >> 2][t & 3]), tf32_operand(m1[t >> 2][t & 3]));
    }
}

// W (16, C, K) -> W rounded to TF32, plus the zero-block map of the forward's prepared weights: bit cc of
// map[t][kb] is set when the block (input channels cc*32.., output channels kb*64..) holds a non-zero.
// One CTA per eight blocks along the input channels: one byte of the map, 256 threads per block (see pack_weights_kernel).
__global__ void __launch_bounds__(kPackThreads) round_and_map_kernel(const float *__restrict__ Wt, float *__restrict__ Wr,
                                                                       unsigned long long *__restrict__ map, int C, int K, int nKB, int nCC)
{
    after_previous_kernel(Wt, Wr, map);
    __shared__ int live;
    if (threadIdx.x == 0) live = 0;
    __syncthreads();
    const int kb = blockIdx.x, t = blockIdx.z, tid = threadIdx.x & 255;
    const bool vec = (K & 3) == 0 && ((reinterpret_cast<uintptr_t>(Wt) | reinterpret_cast<uintptr_t>(Wr)) & 15u) == 0;
    for (int r = threadIdx.x >> 8; r < 8; r += kPackThreads / 256) {
        const int c0 = (blockIdx.y * 8 + r) * 32;
        if (c0 >= C) break;
        int nz = 0;
        if (vec) {
            // 16 bytes per access: 32 rows of 16 float4, two per thread
            float4 w[2];
            long long o[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int e = tid + 256 * q, c = c0 + (e >> 4), k = kb * 64 + 4 * (e & 15);
                o[q] = (c < C && k < K) ? ((long long)t * C + c) * K + k : -1;
                if (o[q] >= 0) w[q] = __ldg(reinterpret_cast<const float4 *>(Wt + o[q]));
            }
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (o[q] >= 0) {
                    w[q].x = round_tf32(w[q].x); w[q].y = round_tf32(w[q].y); w[q].z = round_tf32(w[q].z); w[q].w = round_tf32(w[q].w);
                    *reinterpret_cast<float4 *>(Wr + o[q]) = w[q];
                    nz |= (w[q].x != 0.f) | (w[q].y != 0.f) | (w[q].z != 0.f) | (w[q].w != 0.f);
                }
        } else {
            for (int e = tid; e < 32 * 64; e += 256) {
                const int c = c0 + (e >> 6), k = kb * 64 + (e & 63);
                if (c < C && k < K) {
                    const long long o = ((long long)t * C + c) * K + k;
                    const float w = round_tf32(__ldg(Wt + o));
                    Wr[o] = w;
                    nz |= (w != 0.f);
                }
            }
        }
        if (__any_sync(0xffffffffu, nz) && (threadIdx.x & 31) == 0) atomicOr(&live, 1 << r);
    }
    __syncthreads();
    if (threadIdx.x == 0) store_map_byte(map + (long long)t * nKB + kb, blockIdx.y, gridDim.y, nCC, (unsigned)live);
}

static int launch_dm(const float *dY, float *dM, int B, int H, int W, int K, int layout, cudaStream_t st)
{
    const int nH = (H + 1) / 2, nW = (W + 1) / 2;
    const long long P = (long long)B * nH * nW;
    if (layout == WG2X2_NHWC) {
        launch(conv_dm_nhwc_kernel, dim3((unsigned)cdivll(P * (K / 4), 256)), 256, 0, st, dY, dM, P, nH, nW, H, W, K);
    } else if (const int R = K % kPairCB == 0 && K / kPairCB <= 65535 && 2 * nW * 2 * kPairPitch * 4 <= 72 * 1024 && P * K < (1LL << 30) &&
                                     (reinterpret_cast<uintptr_t>(dM) & 7u) == 0 ? pair_rows(B, K, nH, nW, W, 0) : 0) {
        const int nbands = cdiv(nH, R);
        if ((long long)B * nbands > 0x7fffffffLL) return WG2X2_ERR_UNSUPPORTED;
        launch(conv_dm_nchw_pair_kernel, dim3((unsigned)(B * nbands), K / kPairCB), 256, 2 * R * 2 * nW * kPairPitch * sizeof(float), st, dY, dM, nH, nW, H, W,
               K, R, nbands, (unsigned)cdiv(1 << 20, 2 * nW), (unsigned)(P * K * 4));
    } else {
        const BandCut cut = cut_bands(nH, nW, (long long)B * cdiv(K, 32), 384 / (2 * W));
        const int pitch = (2 * cut.R * (cut.nsegs == 1 ? W : 2 * cut.S)) | 1;
        const int smem = 32 * pitch * (int)sizeof(float);
        const long long blocks = (long long)B * cut.nbands * cut.nsegs;
        if (blocks > 0x7fffffffLL || smem > 200 * 1024) return WG2X2_ERR_UNSUPPORTED;
        launch(cut.nsegs == 1 ? conv_dm_nchw_kernel<false> : conv_dm_nchw_kernel<true>, dim3((unsigned)blocks, cdiv(K, 32)), 256, smem, st, dY, dM,
               P, nH, nW, H, W, K, cut.R, cut.nbands, cut.S, cut.nsegs, pitch);
    }
    return launch_status();
}

// ---------------------------------------------------------------------------------------
// Workspace of the tensor-core backward pass: [dM | W rounded to TF32 | dW partials]
// ---------------------------------------------------------------------------------------
struct BwdWs {
    size_t dm, wr, map, partial, total;
};
static BwdWs bwd_ws_layout(long long P, int C, int K, int dw_splits)
{
    BwdWs w;
    w.dm = 0;
    size_t off = align_up((size_t)16 * P * K * sizeof(float), 256);
    w.wr = off;      off += align_up((size_t)16 * C * K * sizeof(float), 256);
    w.map = off;     off += align_up((size_t)16 * cdiv(K, 64) * sizeof(unsigned long long), 256);
    w.partial = off; off += dw_splits > 1 ? align_up((size_t)dw_splits * 16 * C * K * sizeof(float), 256) : 0;
    w.total = off;
    return w;
}

bool tc_bwd_shape_supported(int C, int K) { return C % 4 == 0 && K % 4 == 0 && C >= 4 && K >= 4; }

// ---------------------------------------------------------------------------------------
// The two gradient products as plain batched GEMMs on the tensor cores (16 independent positions):
//
//   KIND 0   dW_t[c][k] = sum_p V_t[p][c] dM_t[p][k]    rows = C, columns = K, contraction over P (split)
//   KIND 1   dV_t[p][c] = sum_k dM_t[p][k] W_t[c][k]    rows = P, columns = C, contraction over K
//
// Unit = (position t, block of 128 rows, block of N = 64/128/256 columns[, split of the contraction]);
// one fp32 accumulator of N TMEM columns, double-buffered, so the epilogue of a unit overlaps the MMAs of
// the next.  A wide N is what makes these run well: the A tile is read from shared memory and from L2 once
// per 128 x N x 32 products.
//
// KIND 0 operands are stored with the contraction index p as the slow axis, i.e. "MN-major" for UMMA: a
// [32 p x 32 channel] box lands in shared memory as 32 rows of 128 bytes (128B swizzle, 32B atoms), which
// is one MN block of 32 channels x eight K groups of 4 tiles.  A (V_t^T, 128 input channels) is four such
// boxes 4 KB apart (the descriptor's leading-dimension offset), B (dM_t) is N/32 of them.  One MMA (K = 8)
// reads 8 rows: start address + 1024 B per step.
// KIND 1 operands are contraction-contiguous ("K-major"): A = a [128 p x 32 k] box of dM, B = an [N x 32 k]
// box of W exactly as the reference stores it, both with the plain 128B swizzle; + 32 B per MMA step.
//
// The epilogue turns each 32 x 32 block through shared memory so that stores are whole 128-byte lines, and
// applies the pruning mask (KIND 0, one split) or the ReLU mask V > 0 (KIND 1) on the way out.
// ---------------------------------------------------------------------------------------
constexpr int kGgMaxStages = 8;                          // 4 / 6 / 8 stages of 48 / 32 / 24 KB for 256 / 128 / 64 columns
constexpr int kGgBoxBytes = 32 * 32 * 4;                 // [32 rows][32 fp32]
constexpr int kGgABytes = 4 * kGgBoxBytes;               // 128 rows x 32 contraction steps
constexpr int kGgBBytesMax = 8 * kGgBoxBytes;            // up to 256 columns
constexpr int kGgRingBytes = 4 * (kGgABytes + kGgBBytesMax);   // 192 KB
constexpr int kGgSmemBytes = kGgRingBytes + 1024 + kCtrlBytes + kEpiWarps * kEpiStageBytes;

struct GgParams {
    float *out;              // [split][16][rows][cols] (split dimension only when !direct)
    const float *mask;       // KIND 0: multiplies the result (direct only); KIND 1: result zeroed where mask <= 0
    long long rows;          // C (KIND 0) or P (KIND 1)
    long long contr;         // P (KIND 0) or K (KIND 1)
    int cols, N;
    int nRB, nCB;
    int splits, chunks_per_split;
    int units;
    int direct;
    // Zero-block skipping (KIND 1 only).  block_map[t][kb] has bit cc set when the 64 x 32 weight block (output
    // channels kb*64.., input channels cc*32..) of position t holds a non-zero (pack_weights_kernel / block_map_kernel).
    //   map_mode 1: columns = output channels, contraction over input channels (forward products)
    //   map_mode 2: columns = input channels, contraction over output channels (dV)
    //   map_mode 0: every chunk runs
    const unsigned long long *block_map;
    int map_mode, map_nkb;
    int tma_out;             // results that need no mask leave by TMA store (mapOut) straight from the staging block
    int mn4;                 // KIND 0: the operand maps are 4-D (channel blocks of 32 as a dimension of their own): one TMA load per operand and chunk
};

// Bit n of the result is set when contraction chunk n (32 elements) of this unit has to run: the first chunk always
// (it zero-initialises the accumulator), a later one unless every weight block it would multiply is all zero.
// Contractions of more than 64 chunks run in full.
__device__ __forceinline__ unsigned long long gg_live_chunks(const GgParams &prm, int t, int cb)
{
    if (prm.map_mode == 0 || prm.contr > 64 * 32) return ~0ull;
    const unsigned long long *row = prm.block_map + (long long)t * prm.map_nkb;
    unsigned long long live = 1ull;
    if (prm.map_mode == 1) {
        const int kb0 = cb * (prm.N >> 6), kb1 = min(prm.map_nkb, kb0 + max(prm.N >> 6, 1));
        for (int kb = kb0; kb < kb1; ++kb) live |= __ldg(row + kb);
    } else {
        const int c0 = cb * (prm.N >> 5), nc = prm.N >> 5;                 // 32-channel chunks covered by this unit's columns
        if (c0 + nc > 64) return ~0ull;
        const unsigned long long sel = (nc >= 64 ? ~0ull : ((1ull << nc) - 1ull)) << c0;
        const int nkb = (int)((prm.contr + 63) >> 6);
        for (int kb = 0; kb < nkb && kb < prm.map_nkb; ++kb)
            if (__ldg(row + kb) & sel) live |= 3ull << (2 * kb);          // both 32-wide halves of the 64-wide block
    }
    return live;
}

// MN-major TF32 operand.  The only shared-memory layout UMMA accepts for it is the 128-byte swizzle with a
// 32-byte base (layout type 1; TMA writes it with CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B): rows of 128 bytes,
// the 32-byte chunk index XORed with (row & 3), pattern repeating every 4 rows.  MN blocks of 32 elements
// are 4 KB apart (leading-dimension offset), K groups of 4 rows 512 B apart (stride offset).
__device__ __forceinline__ uint64_t make_desc_mn_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(kGgBoxBytes >> 4) << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)1 << 61;
    return d;
}

__device__ __forceinline__ void tma_load_4d_gg(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2, int c3)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}

// shared memory -> global, clipped to the tensor; completion is tracked by the thread's bulk async-groups
__device__ __forceinline__ void tma_store_3d(uint32_t src, const CUtensorMap *map, int c0, int c1, int c2)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%1, {%2, %3, %4}], [%0];"
        ::"r"(src), "l"(map), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

template <int KIND>
__global__ void __launch_bounds__(kTcThreads, 1)
conv_grad_gemm_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                         const __grid_constant__ CUtensorMap mapOut, const GgParams prm)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gen_base = smem_raw + (base - raw);
    const uint32_t bars = base + kGgRingBytes;
    uint64_t *bars_gen = reinterpret_cast<uint64_t *>(gen_base + kGgRingBytes);
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kGgMaxStages + s); };
    auto accf_bar = [&](int b) { return bars + 8u * (2 * kGgMaxStages + b); };
    auto acce_bar = [&](int b) { return bars + 8u * (2 * kGgMaxStages + 2 + b); };
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(bars_gen + 2 * kGgMaxStages + 4);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bars_gen + 2 * kGgMaxStages + 5);
    float *epi_stage_all = reinterpret_cast<float *>(gen_base + kGgRingBytes + kCtrlBytes);
    const int nstages = prm.N > 128 ? 4 : (prm.N > 64 ? 6 : 8);
    const uint32_t stage_bytes = (uint32_t)(kGgABytes + prm.N * 128);

    // (broadcast from lane 0: the compiler then treats the warp index, and all that is derived from it, as warp-uniform)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kGgMaxStages; ++s) { mbar_init(full_bar(s), 1); mbar_init(empty_bar(s), 1); }
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

    const int N = prm.N;
    // unit -> (split, t, row block, column block); column block fastest so that neighbouring CTAs share the A tile in L2
    auto decode = [&](int u, int &split, int &t, int &rb, int &cb) {
        cb = u % prm.nCB; u /= prm.nCB;
        rb = u % prm.nRB; u /= prm.nRB;
        t = u % 16;
        split = u / 16;
    };

    if (warp == 0) {
        if (lane == 0) {
            int s = 0; uint32_t ph = 0;
            bool ok = true;
            const uint32_t stage_tx = (uint32_t)(kGgABytes + N * 128);
            for (int u = blockIdx.x; u < prm.units && ok; u += gridDim.x) {
                int split, t, rb, cb;
                decode(u, split, t, rb, cb);
                const long long kbeg = (long long)split * prm.chunks_per_split * 32;
                const long long kend = min(prm.contr, kbeg + (long long)prm.chunks_per_split * 32);
                const unsigned long long live = KIND == 1 ? gg_live_chunks(prm, t, cb) : ~0ull;
                for (long long kc = kbeg; kc < kend; kc += 32) {
                    if (KIND == 1 && kc < 64 * 32 && !((live >> (kc >> 5)) & 1ull)) continue;   // all-zero weight blocks: nothing to add
                    if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, 0x500u | s)) { ok = false; break; }
                    mbar_expect_tx(full_bar(s), stage_tx);
                    const uint32_t a_dst = base + s * stage_bytes;
                    const uint32_t b_dst = a_dst + kGgABytes;
                    if (KIND == 0 && prm.mn4) {      // all 32-channel blocks of an operand in one box each
                        tma_load_4d_gg(a_dst, &mapA, full_bar(s), 0, (int)kc, rb * 4, t);
                        tma_load_4d_gg(b_dst, &mapB, full_bar(s), 0, (int)kc, cb * (N / 32), t);
                    } else if (KIND == 0) {
#pragma unroll
                        for (int mb = 0; mb < 4; ++mb)
                            tma_load_3d(a_dst + mb * kGgBoxBytes, &mapA, full_bar(s), rb * 128 + mb * 32, (int)kc, t);
                        for (int nb = 0; nb < N / 32; ++nb)
                            tma_load_3d(b_dst + nb * kGgBoxBytes, &mapB, full_bar(s), cb * N + nb * 32, (int)kc, t);
                    } else {
                        tma_load_3d(a_dst, &mapA, full_bar(s), (int)kc, rb * 128, t);
                        tma_load_3d(b_dst, &mapB, full_bar(s), (int)kc, cb * N, t);
                    }
                    if (++s == nstages) { s = 0; ph ^= 1u; }
                }
            }
            if (!ok)
                for (int it = 0; it < 1000; ++it) __nanosleep(1000);
        }
    } else if (warp == 1) {
        // The whole warp walks the loop with warp-uniform values (descriptors and addresses in uniform registers); one
        // elected lane issues the MMAs and the commits.  Issued by a lone lane from per-thread registers, an MMA costs
        // several times as many issue slots, for which the eight epilogue warps compete.
        {
            const bool leader = elect_one();
            const uint32_t idesc = make_idesc_tf32(128, N) | (KIND == 0 ? ((1u << 15) | (1u << 16)) : 0u);
            int s = 0; uint32_t ph = 0;
            uint32_t acc_use[2] = {0, 0};
            int buf = 0;
            bool ok = true;
            for (int u = blockIdx.x; u < prm.units && ok; u += gridDim.x) {
                int split, t, rb, cb;
                decode(u, split, t, rb, cb);
                const long long kbeg = (long long)split * prm.chunks_per_split * 32;
                const long long kend = min(prm.contr, kbeg + (long long)prm.chunks_per_split * 32);
                if (!mbar_wait_warp(acce_bar(buf), (acc_use[buf] & 1u) ^ 1u, abort_flag, 0x600u | buf)) { ok = false; break; }
                acc_use[buf]++;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(buf * 256);
                uint32_t first = 1;
                const unsigned long long live = KIND == 1 ? gg_live_chunks(prm, t, cb) : ~0ull;
                for (long long kc = kbeg; kc < kend; kc += 32) {
                    if (KIND == 1 && kc < 64 * 32 && !((live >> (kc >> 5)) & 1ull)) continue;
                    if (!mbar_wait_warp(full_bar(s), ph, abort_flag, 0x700u | s)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = base + s * stage_bytes;
                    const uint64_t adesc = KIND == 0 ? make_desc_mn_sw128(a_addr) : make_desc_k_sw128(a_addr);
                    const uint64_t bdesc = KIND == 0 ? make_desc_mn_sw128(a_addr + kGgABytes) : make_desc_k_sw128(a_addr + kGgABytes);
                    const uint32_t step = KIND == 0 ? 64u : 2u;   // 1024 B / 32 B per 8 contraction steps
                    if (leader) {
#pragma unroll
                        for (int kg = 0; kg < 4; ++kg)
                            umma_tf32(d_tmem, adesc + step * kg, bdesc + step * kg, idesc, (first && kg == 0) ? 0u : 1u);
                        umma_commit(empty_bar(s));
                    }
                    __syncwarp();
                    first = 0;
                    if (++s == nstages) { s = 0; ph ^= 1u; }
                }
                if (ok && leader) umma_commit(accf_bar(buf));
                __syncwarp();
                buf ^= 1;
            }
        }
    } else {
        const int ew = warp - 2;
        const int q = warp & 3;
        const int half = ew >> 2;
        float *stg = epi_stage_all + ew * (kEpiStageBytes / 4);
        uint32_t acc_use[2] = {0, 0};
        int buf = 0;
        bool ok = true;
        const long long plane_elems = 16 * prm.rows * prm.cols;
        for (int u = blockIdx.x; u < prm.units && ok; u += gridDim.x) {
            int split, t, rb, cb;
            decode(u, split, t, rb, cb);
            const bool use_mask = prm.mask && (KIND == 1 || prm.direct);
            const long long row = (long long)rb * 128 + q * 32 + lane;
            const long long row_off = (prm.direct ? 0 : (long long)split * plane_elems) + ((long long)t * prm.rows + row) * prm.cols;
            const int ncol_half = N / 2;
            // offsets of the 8 lines this lane will store in a 32-column block, and their mask values.  They are fetched one
            // block ahead (the first block of a unit before the accumulator is even waited for), so that the memory latency
            // of the mask hides behind the previous block's TMEM load, turn and stores instead of stalling every block.
            long long off[8], off_nx[8];
            float4 mk[8], mk_nx[8];
            auto fetch = [&](int cc_f, long long (&o)[8], float4 (&m)[8]) {
                const int col_f = cb * N + half * ncol_half + cc_f;
                const long long my_f = (row < prm.rows && col_f < prm.cols) ? row_off + col_f : -1;
                const bool vec_f = (col_f + 32 <= prm.cols) && ((prm.cols & 3) == 0);
#pragma unroll
                for (int rr = 0; rr < 8; ++rr) {
                    o[rr] = __shfl_sync(0xffffffffu, my_f, 4 * rr + (lane >> 3));
                    m[rr] = make_float4(1.f, 1.f, 1.f, 1.f);
                    if (vec_f && use_mask && o[rr] >= 0) m[rr] = __ldg(reinterpret_cast<const float4 *>(prm.mask + o[rr] + 4 * (lane & 7)));
                }
            };
            fetch(0, off, mk);
            for (int cc = 0; cc < ncol_half; cc += 32) {
                const int col0 = half * ncol_half + cc;
                const int col = cb * N + col0;
                const long long my_off = (row < prm.rows && col < prm.cols) ? row_off + col : -1;
                const bool vec = (col + 32 <= prm.cols) && ((prm.cols & 3) == 0);
                const bool more = cc + 32 < ncol_half;
                if (more) fetch(cc + 32, off_nx, mk_nx);
                if (cc == 0) {   // first chunk of the unit: only now wait for the accumulator
                    if (!mbar_wait_warp(accf_bar(buf), acc_use[buf] & 1u, abort_flag, 0x800u | (ew << 4) | buf)) { ok = false; break; }
                    acc_use[buf]++;
                    tc_fence_after();
                }
                float r[32];
                const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 256 + col0);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) tmem_ld8(taddr + (uint32_t)(ch * 8), &r[ch * 8]);
                tmem_ld_wait();
                if (vec && prm.tma_out && !use_mask) {
                    // The staging block (32 rows of 128 bytes, 16-byte chunk index XORed with row & 7) is exactly TMA's
                    // 128-byte swizzle: one lane hands it to a TMA store, which also clips the rows beyond the tensor; the
                    // block is not read back through the load/store unit, whose shared-memory traffic competes with the
                    // tensor core's operand reads.  The store that last used the block must have read it first.
                    if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    __syncwarp();
#pragma unroll
                    for (int c8 = 0; c8 < 8; ++c8)
                        *reinterpret_cast<float4 *>(stg + lane * 32 + ((c8 ^ (lane & 7)) << 2)) =
                            make_float4(r[4 * c8], r[4 * c8 + 1], r[4 * c8 + 2], r[4 * c8 + 3]);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) {
                        tma_store_3d(smem_u32(stg), &mapOut, col, rb * 128 + q * 32, (prm.direct ? 0 : split * 16) + t);
                        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    }
                } else if (vec) {
                    if (prm.tma_out) {      // a TMA store of an earlier block may still be reading the staging block
                        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
                    }
                    __syncwarp();
#pragma unroll
                    for (int c8 = 0; c8 < 8; ++c8)
                        *reinterpret_cast<float4 *>(stg + lane * 32 + ((c8 ^ (lane & 7)) << 2)) =
                            make_float4(r[4 * c8], r[4 * c8 + 1], r[4 * c8 + 2], r[4 * c8 + 3]);
                    __syncwarp();
#pragma unroll
                    for (int rr = 0; rr < 8; ++rr) {
                        const int srow = 4 * rr + (lane >> 3), ch = lane & 7;
                        float4 v = *reinterpret_cast<const float4 *>(stg + srow * 32 + ((ch ^ (srow & 7)) << 2));
                        if (off[rr] >= 0) {
                            if (KIND == 0) { v.x *= mk[rr].x; v.y *= mk[rr].y; v.z *= mk[rr].z; v.w *= mk[rr].w; }
                            else { v.x = mk[rr].x > 0.f ? v.x : 0.f; v.y = mk[rr].y > 0.f ? v.y : 0.f;
                                   v.z = mk[rr].z > 0.f ? v.z : 0.f; v.w = mk[rr].w > 0.f ? v.w : 0.f; }
                            *reinterpret_cast<float4 *>(prm.out + off[rr] + 4 * ch) = v;
                        }
                    }
                } else if (my_off >= 0) {
#pragma unroll
                    for (int x = 0; x < 32; ++x) {
                        if (col + x >= prm.cols) continue;
                        float v = r[x];
                        if (use_mask) {
                            const float m1 = __ldg(prm.mask + my_off + x);
                            v = KIND == 0 ? v * m1 : (m1 > 0.f ? v : 0.f);
                        }
                        prm.out[my_off + x] = v;
                    }
                }
                if (more) {
#pragma unroll
                    for (int rr = 0; rr < 8; ++rr) { off[rr] = off_nx[rr]; mk[rr] = mk_nx[rr]; }
                }
            }
            if (!ok) break;
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acce_bar(buf));
            buf ^= 1;
        }
        // the last stores must have reached memory before the CTA ends
        if (prm.tma_out && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// 3-D map over a (16, rows, ch) fp32 tensor, ch contiguous.  mn_major: box = 32 channels x 32 rows with the
// 32-B-atom 128-B swizzle; otherwise box = 32 channels x box_rows with the plain 128-B swizzle.
static bool make_map_gg(CUtensorMap *map, const float *ptr, long long ch, long long rows, bool mn_major, int box_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    cuuint64_t dims[3] = {(cuuint64_t)ch, (cuuint64_t)rows, 16};
    cuuint64_t strides[2] = {(cuuint64_t)ch * 4, (cuuint64_t)rows * ch * 4};
    cuuint32_t box[3] = {32, (cuuint32_t)(mn_major ? 32 : box_rows), 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, mn_major ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// MN-major operand with the 32-channel blocks as a dimension of their own: (32, rows, ch / 32, 16), box = 32 x 32 rows x
// nblk blocks, which lands in shared memory as nblk consecutive 4 KB blocks -- the layout the MN-major descriptor reads --
// from ONE load instead of nblk.  Needs ch % 32 == 0.
static bool make_map_gg4(CUtensorMap *map, const float *ptr, long long ch, long long rows, int nblk)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn || (ch & 31) || nblk < 1 || nblk > 8) return false;
    cuuint64_t dims[4] = {32, (cuuint64_t)rows, (cuuint64_t)(ch / 32), 16};
    cuuint64_t strides[3] = {(cuuint64_t)ch * 4, 128, (cuuint64_t)rows * ch * 4};
    cuuint32_t box[4] = {32, 32, (cuuint32_t)nblk, 1};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(ptr), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int gg_cols(int n) { return n > 128 ? 256 : (n > 64 ? 128 : 64); }

// Columns per unit of a product with `rows` x n results and a contraction of `contr`: the width whose rounds over the SMs
// take least.  A unit takes about (chunks of 32) x c + e microseconds, measured with c = 0.37 / 0.45 / 0.60 and e = 0.3 / 0.5 / 0.9
// for 64 / 128 / 256 columns: wide units share the A tile among more columns, narrow ones put more SMs to work (one 14 x 14
// image of 512 channels: 13.9 us with 256 columns, 10.4 with 64).
static int gg_pick_cols(long long rows, int n, int contr, double *us = nullptr)
{
    const int widest = gg_cols(n);
    const double ch = cdiv(contr, 32);
    int best = widest;
    double t = 1e30;
    for (int N = widest; N >= 64; N >>= 1) {
        const long long units = 16 * cdivll(rows, 128) * cdiv(n, N);
        const double per = N == 64 ? 0.37 * ch + 0.3 : N == 128 ? 0.45 * ch + 0.5 : 0.60 * ch + 0.9;
        const double u = (double)cdivll(units, kNumSMs) * per;
        if (u < t) { t = u; best = N; }
    }
    if (us) *us = t;
    return best;
}

// Splits of the P range for dW: the count that takes least, rounds over the SMs x chunks of 32 tiles per split (at least 8)
// at 0.37 us each, plus the reduction pass over the partial sums.  (Just covering the SMs is not enough: 16 blocks x 10
// splits are two rounds where 16 x 9 are one -- 109 against 64 us at 64 x 64 x 56 x 56.)
int conv_dw_tc_splits(long long P, int C, int K)
{
    const long long base_units = (long long)16 * cdiv(C, 128) * cdiv(K, gg_cols(K));
    const long long chunks = cdivll(P, 32);
    const long long max_s = chunks / 8 > 0 ? chunks / 8 : 1;
    const double pass = 16.0 * C * K * 4 / 4e6;         // microseconds to move dW once
    long long best = 1;
    double t = 1e30;
    for (long long s = 1; s <= max_s && s <= kNumSMs; ++s) {
        const double u = (double)cdivll(base_units * s, kNumSMs) * cdivll(chunks, s) * 0.37 + (s > 1 ? 2.5 + (2 * s + 1) * pass : 0.0);
        if (u < t) { t = u; best = s; }
    }
    const long long cps = cdivll(chunks, best);
    return (int)cdivll(chunks, cps);
}

// 3-D map over the result (planes, rows, cols) fp32, cols contiguous, for the epilogue's TMA stores: box = 32 columns x 32
// rows with the 128-byte swizzle.  Usable when the base is 16-byte aligned and the rows are multiples of 16 bytes.
static bool make_map_out(CUtensorMap *map, float *ptr, long long cols, long long rows, long long planes)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn || (reinterpret_cast<uintptr_t>(ptr) & 15u) || (cols & 3)) return false;
    cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)planes};
    cuuint64_t strides[2] = {(cuuint64_t)cols * 4, (cuuint64_t)rows * cols * 4};
    cuuint32_t box[3] = {32, 32, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, ptr, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

#include "conv_tc_gemm2.cuh"

// How many pairs of SMs can hold a pair of CTAs of the cta_group::2 kernel at once (0: this device cannot, or
// WG2X2_GEMM_PAIR=0 in the environment); asked once per device and kernel.
template <int KIND>
static int gg_pair_clusters()
{
    static std::atomic<int> cached[64];
    static std::atomic<int> init{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    if (!init.load()) {
        for (auto &c : cached) c.store(-1);
        init.store(1);
    }
    int n = cached[dev].load();
    if (n >= 0) return n;
    const char *env = getenv("WG2X2_GEMM_PAIR");
    n = 0;
    if (!(env && env[0] == '0') &&
        cudaFuncSetAttribute(conv_grad_gemm_tc2_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGg2SmemBytes) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * kNumSMs);
        cfg.blockDim = dim3(kTcThreads);
        cfg.dynamicSmemBytes = kGg2SmemBytes;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int got = 0;
        if (cudaOccupancyMaxActiveClusters(&got, conv_grad_gemm_tc2_kernel<KIND>, &cfg) == cudaSuccess && got > 0) n = got;
        else (void)cudaGetLastError();
    }
    cached[dev].store(n);
    return n;
}

// mapB_half: the B operand with boxes of N/2 rows (KIND 1) or N/64 channel blocks (KIND 0, 4-D maps) for the kernel on pairs
// of SMs; NULL: KIND 1 stays on one CTA, KIND 0 loads its 32 x 32 boxes one by one in either kernel.
template <int KIND>
static int gg_launch(const CUtensorMap &mapA, const CUtensorMap &mapB, GgParams &prm, cudaStream_t st, const CUtensorMap *mapB_half = nullptr)
{
    // results without a mask leave by TMA store where the output can be described to TMA (else: the load/store path)
    CUtensorMap mapOut = mapA;
    const bool needs_mask = prm.mask && (KIND == 1 || prm.direct);
    prm.tma_out = (!needs_mask && prm.cols >= 32 &&
                   make_map_out(&mapOut, prm.out, prm.cols, prm.rows, 16LL * (prm.direct ? 1 : prm.splits))) ? 1 : 0;
    // Two SMs per 256 x N tile where that measured faster: long contractions (dW always contracts over all tiles; the
    // products with 512 or more channels), whose pipeline outlasts the pair's extra hand-shakes, and no mask to fetch in
    // the epilogue.  Short contractions (256 channels) and dV with its ReLU mask are HBM-bound and stay on one CTA.
    const bool pair_pays = KIND == 0 ? prm.contr >= 1024 : (mapB_half && prm.contr >= 512 && !needs_mask);
    const int nclusters = (prm.nRB >= 2 && prm.N >= 128 && pair_pays) ? gg_pair_clusters<KIND>() : 0;
    if (nclusters > 0) {
        GgParams p2 = prm;
        p2.nRB = cdiv(prm.nRB, 2);
        p2.units = prm.units / prm.nRB * p2.nRB;
        const int pairs = p2.units < nclusters ? p2.units : nclusters;
        launch(conv_grad_gemm_tc2_kernel<KIND>, dim3(2 * pairs), kTcThreads, kGg2SmemBytes, st, mapA, mapB_half ? *mapB_half : mapB, mapOut, p2);
        return launch_status();
    }
    const int grid = prm.units < kNumSMs ? prm.units : kNumSMs;
    launch(conv_grad_gemm_tc_kernel<KIND>, dim3((unsigned)grid), kTcThreads, kGgSmemBytes, st, mapA, mapB, mapOut, prm);
    return launch_status();
}

int conv_dw_tc(const float *V, const float *dM, const float *mask, float *dW, float *partial, long long P, int C, int K,
               cudaStream_t st)
{
    GgParams prm;
    prm.rows = C; prm.cols = K; prm.contr = P;
    prm.N = gg_cols(K);
    prm.nRB = cdiv(C, 128);
    prm.nCB = cdiv(K, prm.N);
    prm.splits = conv_dw_tc_splits(P, C, K);
    prm.chunks_per_split = (int)cdivll(cdivll(P, 32), prm.splits);
    prm.units = 16 * prm.nRB * prm.nCB * prm.splits;
    prm.direct = prm.splits == 1;
    prm.out = prm.direct ? dW : partial;
    prm.mask = mask;
    prm.block_map = nullptr; prm.map_mode = 0; prm.map_nkb = 0;
    CUtensorMap mapV, mapM, mapMh;
    prm.mn4 = (C % 32 == 0 && K % 32 == 0) ? 1 : 0;
    if (prm.mn4) {
        if (!make_map_gg4(&mapV, V, C, P, 4) || !make_map_gg4(&mapM, dM, K, P, prm.N / 32) ||
            (prm.N >= 64 && !make_map_gg4(&mapMh, dM, K, P, prm.N / 64)))
            return WG2X2_ERR_LAUNCH;
    } else if (!make_map_gg(&mapV, V, C, P, true, 32) || !make_map_gg(&mapM, dM, K, P, true, 32)) {
        return WG2X2_ERR_LAUNCH;
    }
    const int s = gg_launch<0>(mapV, mapM, prm, st, (prm.mn4 && prm.N >= 64) ? &mapMh : nullptr);
    if (s != WG2X2_OK) return s;
    if (!prm.direct) dw_reduce_launch(partial, mask, dW, (long long)16 * C * K, prm.splits, st);
    return launch_status();
}

int conv_dv_tc(const float *V, const float *Wt, const float *dM, float *Wr, unsigned long long *map, float *dV, long long P, int C,
               int K, int relu, cudaStream_t st)
{
    if (P > 0x7fffffffLL - 128) return WG2X2_ERR_UNSUPPORTED;
    const int nKB = cdiv(K, 64), nCC = cdiv(C, 32);
    if (nCC > 65535) return WG2X2_ERR_UNSUPPORTED;
    if (launch(round_and_map_kernel, dim3(nKB, cdiv(nCC, 8), 16), kPackThreads, 0, st, Wt, Wr, map, C, K, nKB, nCC) != WG2X2_OK) return WG2X2_ERR_LAUNCH;
    GgParams prm;
    prm.rows = P; prm.cols = C; prm.contr = K;
    prm.N = gg_pick_cols(P, C, K);
    prm.nRB = (int)cdivll(P, 128);
    prm.nCB = cdiv(C, prm.N);
    prm.splits = 1;
    prm.chunks_per_split = cdiv(K, 32);
    prm.units = 16 * prm.nRB * prm.nCB;
    prm.direct = 1;
    prm.out = dV;
    prm.mask = relu ? V : nullptr;
    prm.block_map = map; prm.map_mode = 2; prm.map_nkb = nKB; prm.mn4 = 0;
    CUtensorMap mapA, mapB, mapBh;
    if (!make_map_gg(&mapA, dM, K, P, false, 128) || !make_map_gg(&mapB, Wr, K, C, false, prm.N) ||
        !make_map_gg(&mapBh, Wr, K, C, false, prm.N / 2))
        return WG2X2_ERR_LAUNCH;
    return gg_launch<1>(mapA, mapB, prm, st, &mapBh);
}

size_t conv_bwd_tc_workspace_bytes(long long P, int C, int K, int want_dW)
{
    return bwd_ws_layout(P, C, K, want_dW ? conv_dw_tc_splits(P, C, K) : 1).total;
}

// dV and/or dW of the product op on the tensor cores.  V is only needed for dW and for the ReLU mask.
int conv_bwd_tc(const float *V, const float *Wt, const float *dY, const float *mask, float *dV, float *dW, int B, int H, int W,
                int C, int K, int layout, int relu, void *ws, size_t ws_bytes, cudaStream_t st)
{
    if (!tc_bwd_shape_supported(C, K)) return WG2X2_ERR_UNSUPPORTED;
    // TMA bases and the 16-byte loads/stores of the producer and the epilogues: every operand that is given
    // must sit on a 16-byte boundary (checked before anything is enqueued)
    if (misaligned16(V) || misaligned16(Wt) || misaligned16(dY) || misaligned16(mask) || misaligned16(dV) || misaligned16(dW))
        return WG2X2_ERR_BAD_ARG;
    const int nH = (H + 1) / 2, nW = (W + 1) / 2;
    const long long P = (long long)B * nH * nW;
    const int splits = dW ? conv_dw_tc_splits(P, C, K) : 1;
    const BwdWs lay = bwd_ws_layout(P, C, K, splits);
    if (!ws || ws_bytes < lay.total || (reinterpret_cast<uintptr_t>(ws) & 255u)) return WG2X2_ERR_WORKSPACE;
    char *wsb = static_cast<char *>(ws);
    float *dM = reinterpret_cast<float *>(wsb + lay.dm);
    int s = launch_dm(dY, dM, B, H, W, K, layout, st);
    if (s != WG2X2_OK) return s;
    if (dV) {
        s = conv_dv_tc(V, Wt, dM, reinterpret_cast<float *>(wsb + lay.wr), reinterpret_cast<unsigned long long *>(wsb + lay.map), dV,
                       P, C, K, relu, st);
        if (s != WG2X2_OK) return s;
    }
    if (dW) {
        s = conv_dw_tc(V, dM, mask, dW, reinterpret_cast<float *>(wsb + lay.partial), P, C, K, st);
        if (s != WG2X2_OK) return s;
    }
    return WG2X2_OK;
}

// ---------------------------------------------------------------------------------------
// Wide forward path, for layers with many channels (C, K >= 256) and wherever conv_fwd_wide_preferred says: the 16 products as plain
// GEMMs with up to N = 256 output channels per unit (conv_grad_gemm_tc_kernel<1>: same operands' major-ness as dV), the
// products M (16, P, K) written once to scratch memory, then one HBM-bound pass for A^T m A.  With N = 64
// (the row-walk kernel, which needs four accumulators live per unit) every A tile is re-read from L2 and
// from shared memory four times as often, and that, not HBM, is what bounds these shapes.
// ---------------------------------------------------------------------------------------
struct OutExtras {
    const float *scale, *shift, *residual;
    int res_relu;            // the residual passes through a ReLU first
    __device__ __forceinline__ float shortcut(long long o) const { const float r = __ldg(residual + o); return res_relu ? relu_nan(r) : r; }
};

// NHWC: one thread = one tile x 4 output channels
__global__ void __launch_bounds__(256) out_transform_nhwc_kernel(const float *__restrict__ M, float *__restrict__ Y, long long P,
                                                                   int nH, int nW, int K, int outH, int outW, OutExtras ex)
{
    after_previous_kernel(M, Y, ex.scale, ex.shift, ex.residual);
    const int KV = K >> 2;
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= P * KV) return;
    const int kv = (int)(idx % KV);
    const long long p = idx / KV;
    const int tw = (int)(p % nW), th = (int)((p / nW) % nH), b = (int)(p / ((long long)nW * nH));
    float4 y[2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < 2; ++e) y[a][e] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float4 m[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) m[j] = __ldg(reinterpret_cast<const float4 *>(M + ((long long)(4 * i + j) * P + p) * K) + kv);
        const float4 z0 = make_float4(m[0].x + m[1].x + m[2].x, m[0].y + m[1].y + m[2].y, m[0].z + m[1].z + m[2].z, m[0].w + m[1].w + m[2].w);
        const float4 z1 = make_float4(m[1].x - m[2].x - m[3].x, m[1].y - m[2].y - m[3].y, m[1].z - m[2].z - m[3].z, m[1].w - m[2].w - m[3].w);
        if (i <= 2) { y[0][0] = y[0][0] + z0; y[0][1] = y[0][1] + z1; }
        if (i == 1) { y[1][0] = y[1][0] + z0; y[1][1] = y[1][1] + z1; }
        if (i >= 2) { y[1][0] = y[1][0] - z0; y[1][1] = y[1][1] - z1; }
    }
    float4 sc = make_float4(1.f, 1.f, 1.f, 1.f), sh = make_float4(0.f, 0.f, 0.f, 0.f);
    if (ex.scale) { sc = __ldg(reinterpret_cast<const float4 *>(ex.scale) + kv); sh = __ldg(reinterpret_cast<const float4 *>(ex.shift) + kv); }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int h = 2 * th + a, w = 2 * tw + e;
            if (h >= outH || w >= outW) continue;
            const long long o = ((((long long)b * outH + h) * outW + w) * K) / 4 + kv;
            float4 v = y[a][e];
            if (ex.scale) { v.x = fmaf(v.x, sc.x, sh.x); v.y = fmaf(v.y, sc.y, sh.y); v.z = fmaf(v.z, sc.z, sh.z); v.w = fmaf(v.w, sc.w, sh.w); }
            if (ex.residual) { float4 r = __ldg(reinterpret_cast<const float4 *>(ex.residual) + o);
                               if (ex.res_relu) r = relu_nan(r);
                               v = v + r; }
            reinterpret_cast<float4 *>(Y)[o] = v;
        }
}

// NCHW: lane = output channel over a band of R tile rows (or, SEG, a segment of one row); the output pixels of each channel
// collect in shared memory and leave as one contiguous run per channel.
template <bool SEG>
__global__ void __launch_bounds__(256) out_transform_nchw_kernel(const float *__restrict__ M, float *__restrict__ Y, long long P,
                                                                   int nH, int nW, int K, int outH, int outW, int R, int nbands, int S,
                                                                   int nsegs, int pitch, OutExtras ex)
{
    after_previous_kernel(M, Y, ex.scale, ex.shift, ex.residual);
    extern __shared__ float O[];
    int bb = blockIdx.x;
    const int seg = SEG ? bb % nsegs : 0;
    if (SEG) bb /= nsegs;
    const int band = bb % nbands;
    const int b = bb / nbands;
    const int k0 = blockIdx.y * 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int th0 = band * R;
    const int rows_blk = min(R, nH - th0);
    const int tw0 = SEG ? seg * S : 0, ns = SEG ? min(S, nW - tw0) : nW;
    const int OW = SEG ? min(2 * ns, outW - 2 * tw0) : outW;        // pixels of an output row of the block
    const bool k_ok = k0 + lane < K;
    const float sc = (ex.scale && k_ok) ? __ldg(ex.scale + k0 + lane) : 1.f;
    const float sh = (ex.scale && k_ok) ? __ldg(ex.shift + k0 + lane) : 0.f;
    for (int q = warp; q < rows_blk * ns; q += 8) {
        const int br = q / ns, tl = q - br * ns;
        const long long p = ((long long)b * nH + th0 + br) * nW + tw0 + tl;
        float y[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
        if (k_ok) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float m[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) m[j] = __ldg(M + ((long long)(4 * i + j) * P + p) * K + k0 + lane);
                float z0, z1;
                at_cols(m[0], m[1], m[2], m[3], z0, z1);
                at_rows_accum(i, z0, z1, y);
            }
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (2 * tl + e < OW) O[lane * pitch + (2 * br + a) * OW + 2 * tl + e] = fmaf(y[a][e], sc, sh);
    }
    __syncthreads();
    const int lo = 2 * th0, hi = min(2 * th0 + 2 * rows_blk, outH);
    const int n = (hi - lo) * OW;
    for (int kk = warp; kk < 32; kk += 8) {
        if (k0 + kk >= K) break;
        const long long o = (((long long)b * K + k0 + kk) * outH + lo) * outW + 2 * tw0;
        const float *src = O + kk * pitch;
        if (!SEG) {
            if (ex.residual) { for (int i = lane; i < n; i += 32) Y[o + i] = src[i] + ex.shortcut(o + i); }
            else             { for (int i = lane; i < n; i += 32) Y[o + i] = src[i]; }
        } else {                                                    // two rows of a segment
            for (int i = lane; i < n; i += 32) {
                const long long d = o + (i >= OW ? outW + i - OW : i);
                Y[d] = ex.residual ? src[i] + ex.shortcut(d) : src[i];
            }
        }
    }
}

// NCHW, enough tiles to fill the GPU and whole blocks of 64 channels: two channels per lane, a tile's sixteen 8-byte loads all in
// flight before the first is used (the kernel above, short of registers, has four), pixels in shared memory as [pixel][channel].
// The shortcut arrives there first, by asynchronous copies beside the other CTAs' work; loaded in the copy-out it cost 20 us more.
// Products + output transform: 128 x 256 x 14 x 14 68.5 -> 64 us, 256 x 256 x 14 x 14 with a shortcut 147 -> 130, 12 x 256 x 56 x 56 with
// one 141 -> 98.
constexpr int kOutCB = 64, kOutPitch = kOutCB + 2;
__global__ void __launch_bounds__(256, 3) out_transform_nchw_pair_kernel(const float *__restrict__ M, float *__restrict__ Y, long long P, int nH,
                                                                           int nW, int K, int outH, int outW, int R, int nbands, OutExtras ex)
{
    after_previous_kernel(M, Y, ex.scale, ex.shift, ex.residual);
    extern __shared__ __align__(16) float O[];          // [2R rows x outW pixels][kOutPitch]
    const int band = blockIdx.x % nbands, b = blockIdx.x / nbands, k0 = blockIdx.y * kOutCB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int th0 = band * R, rows = min(R, nH - th0);
    const int KV = K >> 1;
    const long long plane = P * KV;
    const float2 *const Mv = reinterpret_cast<const float2 *>(M) + (k0 >> 1) + lane;
    float2 sc = make_float2(1.f, 1.f), sh = make_float2(0.f, 0.f);
    if (ex.scale) { sc = __ldg(reinterpret_cast<const float2 *>(ex.scale + k0) + lane); sh = __ldg(reinterpret_cast<const float2 *>(ex.shift + k0) + lane); }
    const int n = (min(2 * (th0 + rows), outH) - 2 * th0) * outW;
    const long long o0 = (((long long)b * K + k0 + warp) * outH + 2 * th0) * outW, hw8 = 8LL * outH * outW;     // channels warp, warp + 8, ...
    if (ex.residual) {
        for (int i = lane; i < n; i += 32) {
            const uint32_t dst = smem_u32(O + i * kOutPitch + warp);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 32u * c), "l"(ex.residual + o0 + c * hw8 + i) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
    }
#pragma unroll 1
    for (int q = warp; q < rows * nW; q += 8) {
        const int br = q / nW, tw = q - br * nW;
        const float2 *p = Mv + (((long long)b * nH + th0 + br) * nW + tw) * KV;
        float2 m[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) m[t] = __ldg(p + t * plane);
        float y0[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, y1[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float z0, z1;
            at_cols(m[4 * i].x, m[4 * i + 1].x, m[4 * i + 2].x, m[4 * i + 3].x, z0, z1);
            at_rows_accum(i, z0, z1, y0);
            at_cols(m[4 * i].y, m[4 * i + 1].y, m[4 * i + 2].y, m[4 * i + 3].y, z0, z1);
            at_rows_accum(i, z0, z1, y1);
        }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int e = 0; e < 2; ++e)
                if (2 * tw + e < outW && 2 * (th0 + br) + a < outH) {
                    float2 *o = reinterpret_cast<float2 *>(O + ((2 * br + a) * outW + 2 * tw + e) * kOutPitch) + lane;
                    float2 v = make_float2(fmaf(y0[a][e], sc.x, sh.x), fmaf(y1[a][e], sc.y, sh.y));
                    if (ex.residual) {
                        const float2 r = *o;
                        v = ex.res_relu ? make_float2(v.x + relu_nan(r.x), v.y + relu_nan(r.y)) : make_float2(v.x + r.x, v.y + r.y);
                    }
                    *o = v;
                }
    }
    __syncthreads();
    for (int c = 0; c < 8; ++c) {
        float *dst = Y + o0 + c * hw8;
        const float *src = O + warp + 8 * c;
        for (int i = lane; i < n; i += 32) dst[i] = src[i * kOutPitch];
    }
}
// its band height: least rounds of three CTAs per SM x tiles, 72 KB of shared memory at most; 0: too few CTAs to fill the GPU
static int out_pair_rows(int B, int K, int nH, int nW, int outW)
{
    int best = 0;
    double t = 1e300;
    for (int R = 1; R <= nH && (R == 1 || 2 * R * outW * kOutPitch * 4 <= 72 * 1024); ++R) {
        const long long ctas = (long long)B * cdiv(nH, R) * (K / kOutCB);
        if (ctas < 3LL * kNumSMs) break;
        const double u = (double)cdivll(ctas, 3 * kNumSMs) * (R * nW + 8.0);
        if (u < t) { t = u; best = R; }
    }
    return best ? cdiv(nH, cdiv(nH, best)) : 0;
}

// Row-walk kernel or wide path for P tiles?  Microseconds, from timing both over 16 .. 25088 tiles and 32 .. 512 channels: a
// row-walk unit (128 tiles x 64 channels) is a serial chain of 16 x C / 32 chunks of 0.27 us and few tiles are few units, while
// the GEMM spreads the 16 positions over the SMs; the wide path in turn moves the products through memory.  3 x 11 x 11 tiles
// of a 512 -> 96 channel layer: 71 us on two SMs against 11.
bool conv_fwd_wide_preferred(long long P, int C, int K)
{
    if (C % 4 || K % 4) return false;
    if (C >= 256 && K >= 256) return true;
    const double rounds = (double)cdivll(cdivll(P, kBlockM) * cdiv(K, kBlockN), kNumSMs);
    const double row_walk = fmax(7.5 + rounds * 4.3 * cdiv(C, kBlockK), 5.0 + (64.0 * P * C + 16.0 * P * K) / 6e6);
    const double wide = 6.8 + (64.0 * P * (C + 2.0 * K) + 16.0 * P * K) / 5.5e6;
    return wide < row_walk;
}
size_t conv_fwd_wide_workspace_bytes(long long P, int K) { return align_up((size_t)16 * P * K * sizeof(float), 256); }

int conv_fwd_tc_wide(const float *V, const void *prepared, float *Y, int B, int nH, int nW, int C, int K, int outH, int outW,
                     int layout, const float *out_scale, const float *out_shift, const float *residual, int res_relu, void *ws,
                     size_t ws_bytes, cudaStream_t st)
{
    const long long P = (long long)B * nH * nW;
    if (P > 0x7fffffffLL - 128) return WG2X2_ERR_UNSUPPORTED;
    if (!V || !prepared || !Y) return WG2X2_ERR_BAD_ARG;
    if (misaligned16(V) || misaligned16(prepared) || misaligned16(Y) || misaligned16(out_scale) || misaligned16(out_shift) ||
        misaligned16(residual))
        return WG2X2_ERR_BAD_ARG;
    if (!ws || ws_bytes < conv_fwd_wide_workspace_bytes(P, K) || (reinterpret_cast<uintptr_t>(ws) & 255u)) return WG2X2_ERR_WORKSPACE;
    float *M = static_cast<float *>(ws);
    GgParams prm;
    prm.rows = P; prm.cols = K; prm.contr = C;
    prm.N = gg_pick_cols(P, K, C);
    prm.nRB = (int)cdivll(P, 128);
    prm.nCB = cdiv(K, prm.N);
    prm.splits = 1;
    prm.chunks_per_split = cdiv(C, 32);
    prm.units = 16 * prm.nRB * prm.nCB;
    prm.direct = 1;
    prm.out = M;
    prm.mask = nullptr;
    // the zero-block map that weights_prepare built behind the packed weights
    prm.block_map = reinterpret_cast<const unsigned long long *>(static_cast<const unsigned char *>(prepared) +
                                                                 align_up((size_t)16 * K * C * sizeof(float), 256));
    prm.map_mode = 1; prm.map_nkb = cdiv(K, kBlockN); prm.mn4 = 0;
    CUtensorMap mapA, mapB, mapBh;
    if (!make_map_gg(&mapA, V, C, P, false, 128) || !make_map_gg(&mapB, static_cast<const float *>(prepared), C, K, false, prm.N) ||
        !make_map_gg(&mapBh, static_cast<const float *>(prepared), C, K, false, prm.N / 2))
        return WG2X2_ERR_LAUNCH;
    int s = gg_launch<1>(mapA, mapB, prm, st, &mapBh);
    if (s != WG2X2_OK) return s;
    OutExtras ex{out_scale, out_shift, residual, res_relu};
    if (layout == WG2X2_NHWC) {
        launch(out_transform_nhwc_kernel, dim3((unsigned)cdivll(P * (K / 4), 256)), 256, 0, st, M, Y, P, nH, nW, K, outH, outW, ex);
    } else if (const int R = K % kOutCB == 0 && K / kOutCB <= 65535 && outW <= 128 ? out_pair_rows(B, K, nH, nW, outW) : 0) {
        const int nbands = cdiv(nH, R);
        if ((long long)B * nbands > 0x7fffffffLL) return WG2X2_ERR_UNSUPPORTED;
        launch(out_transform_nchw_pair_kernel, dim3((unsigned)(B * nbands), K / kOutCB), 256, 2 * R * outW * kOutPitch * sizeof(float), st, M, Y, P, nH, nW,
               K, outH, outW, R, nbands, ex);
    } else {
        const BandCut cut = cut_bands(nH, nW, (long long)B * cdiv(K, 32), 384 / (2 * outW));
        const int pitch = (2 * cut.R * (cut.nsegs == 1 ? outW : 2 * cut.S)) | 1;
        const int smem = 32 * pitch * (int)sizeof(float);
        const long long blocks = (long long)B * cut.nbands * cut.nsegs;
        if (blocks > 0x7fffffffLL || smem > 200 * 1024) return WG2X2_ERR_UNSUPPORTED;
        launch(cut.nsegs == 1 ? out_transform_nchw_kernel<false> : out_transform_nchw_kernel<true>, dim3((unsigned)blocks, cdiv(K, 32)), 256, smem, st,
               M, Y, P, nH, nW, K, outH, outW, cut.R, cut.nbands, cut.S, cut.nsegs, pitch, ex);
    }
    return launch_status();
}
