// The dense head of the reference's ResNet-18-var graph in one kernel: the 7x7 / stride 2 convolution of the
// 3-channel image into 64 channels (Conv2D('conv1', image, 64, 7, stride=2), no bias, no activation) followed by
// the 3x3 / stride 2 max-pool ('pool1'), both with TensorFlow's SAME padding
// (ResNet-18-var/imagenet-resnet-transWino-prune.py:112-114), and optionally relu(scale * pooled + shift), the
// BNReLU the first stage's shortcut starts from (:126-127).  The reference leaves this layer dense; it is here
// because a stock convolution of a 3-channel image costs more than all sixteen Winograd layers together, and
// because fusing the pool keeps the (B,64,H/2,W/2) convolution result, the largest tensor of the network, out of
// memory altogether.  Included by conv_tc.cu.
//
// Method: implicit GEMM on tcgen05 with the A operand in tensor memory, where the im2col view costs nothing to share: the 24
// columns (channel, tap) that image row y contributes for output column px -- pixels 2 px - 2 .. 2 px + 5 of three channels -- do
// not depend on which convolution row reads them.  So every image row is written to tensor memory once (lane = output column), a
// ring of 16 of them, and convolution row r is 7 x 3 MMAs (M = 128 columns, N = 64 channels, K = 8) over rows 2r - 2 .. 2r + 4 of
// the ring with the weights of ky = 0 .. 6 in shared memory.  Warp w covers output columns 28 w .. 28 w + 28, one more than its
// own: a pool window then never leaves a warp's lanes.
//   warps 0-3   image rows: global -> shared memory (cp.async, eight rows ahead) -> TF32 (nearest) -> tensor memory
//   warp 4      MMAs
//   warps 5-12  two per lane quarter, 32 channels each: vertical maximum of the pool window in registers from convolution row to
//               convolution row, horizontal maximum through shared memory, both outputs stored
// Bound: 21 MMAs of 32 clocks per convolution row would be 68 us for 256 images of 224 x 224 on 148 SMs, the image and both outputs
// (257 MB) 40 us; measured 234 us, with the tensor pipe at 0.31, issue slots at 0.40 and shared memory at 0.45 of active
// cycles: 7000 instructions per pooled row over thirteen warps, each a chain of barrier, shared memory, tensor memory and barrier.  (A
// second set of image-row warps, at 96 registers a thread, took 572 us.)  The warp-level tensor path (mma.sync), whose fragments
// re-read the staged image for every convolution row, took 490 us.  (6 of the 234 us are the comparisons that set NaN apart.)
#pragma once

constexpr int kStThreads = 32 * 13;
constexpr int kStMaxW = 224;
constexpr int kStRing = 16;                     // image rows in tensor memory
constexpr int kStCols = 24;                     // columns of one
constexpr int kStAccCol = kStRing * kStCols;    // two accumulators behind the ring: all 512 columns
constexpr int kStAhead = 8, kStStages = kStAhead + 2;   // image rows on their way to shared memory, and slots there
constexpr int kStPitch = 240;                   // a staged row of one channel: 4 zeros, up to 224 pixels, zeros
constexpr int kStWtBytes = 7 * 64 * 128;        // per ky 64 output channels x 32 (24 of them taps), 128-byte swizzle
constexpr int kStWtFloats = 7 * 64 * kStCols;   // as prepared: [ky][out channel][8 c + kx]
constexpr int kStImgBytes = kStStages * 3 * kStPitch * 4;
constexpr int kStEPitch = 120;                  // pixels of a channel in a pool buffer: up to 112, then NaN
constexpr int kStSmemBytes = 1024 + kStWtBytes + kStImgBytes + 1024 + 2 * 64 * kStEPitch * 4;   // one CTA per SM, it takes all of tensor memory
static_assert(kStSmemBytes > 116 * 1024 && kStSmemBytes <= 232448 && kStAccCol + 128 <= 512, "carve-up");

struct StParams {
    const float *X, *Wp;
    float *Y, *Yr;
    const float *rs, *rb;
    int H, W, bands, band_rows, units;
    uint32_t spin_limit;
};

// (64,3,7,7) weights -> [ky][out channel][8 c + kx], TF32 (nearest), zeros at kx = 7
__global__ void stem_prepare_kernel(const float *__restrict__ W, float *__restrict__ Wp)
{
    after_previous_kernel(W, Wp);
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= kStWtFloats) return;
    const int k = idx % kStCols, n = (idx / kStCols) & 63, ky = idx / (64 * kStCols), c = k >> 3, kx = k & 7;
    Wp[idx] = kx < 7 ? round_tf32(W[((n * 3 + c) * 7 + ky) * 7 + kx]) : 0.f;
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&u)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]) : "memory");
}

// A unit: pooled rows pr0 .. pr0 + rows - 1 of an image, convolution rows 2 pr0 .. (one more than 2 rows of them, where it exists)
struct StUnit {
    int b, pr0, rows, convs;
    __device__ __forceinline__ StUnit(const StParams &p, int u)
    {
        b = u / p.bands;
        pr0 = (u - b * p.bands) * p.band_rows;
        rows = min(p.band_rows, (p.H >> 2) - pr0);
        convs = min(2 * rows + 1, (p.H >> 1) - 2 * pr0);
    }
    __device__ __forceinline__ int image_rows() const { return 2 * convs + 5; }      // from image row 4 pr0 - 2 on
};

__global__ void __launch_bounds__(kStThreads, 1) stem_pool_kernel(const StParams prm)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gen_base = smem_raw + (base - raw);
    float *img_s = reinterpret_cast<float *>(gen_base + kStWtBytes);
    float *pool_s = reinterpret_cast<float *>(gen_base + kStWtBytes + kStImgBytes + 1024);
    float2 *affine = reinterpret_cast<float2 *>(gen_base + kStWtBytes + kStImgBytes + 512);     // scale and shift of the ReLU output
    const uint32_t bars = base + kStWtBytes + kStImgBytes;
    static_assert((kStWtBytes + kStImgBytes) % 8 == 0, "barriers");
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kStRing + s); };
    auto accf_bar = [&](int b) { return bars + 8u * (2 * kStRing + b); };
    auto acce_bar = [&](int b) { return bars + 8u * (2 * kStRing + 2 + b); };
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(gen_base + kStWtBytes + kStImgBytes + 8 * (2 * kStRing + 4));
    volatile int *abort_flag = reinterpret_cast<volatile int *>(gen_base + kStWtBytes + kStImgBytes + 8 * (2 * kStRing + 5));

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, tid = threadIdx.x;
    if (tid == 0) {
        for (int s = 0; s < kStRing; ++s) { mbar_init(full_bar(s), 4); mbar_init(empty_bar(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(accf_bar(b), 1); mbar_init(acce_bar(b), 8); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 4) {
        tmem_alloc(smem_u32((const void *)tmem_ptr_slot), kTmemCols);
        tmem_relinquish();
    }
    for (int i = tid; i < kStImgBytes / 4; i += kStThreads) img_s[i] = 0.f;       // (the padding columns stay zero)
    for (int i = tid; i < 2 * 64 * kStEPitch; i += kStThreads) pool_s[i] = __int_as_float(0x7fffffff);   // (columns beyond the row: fmaxf takes the other value)
    wait_for_previous_kernel(kNumSMs);
    for (int i = tid; i < kStWtFloats / 4; i += kStThreads) {       // a row is six 16-byte pieces (the last two of its 128 bytes are not read)
        const int row = i / 6, piece = i - 6 * row;
        *reinterpret_cast<float4 *>(gen_base + row * 128 + ((piece ^ (row & 7)) << 4)) = __ldg(reinterpret_cast<const float4 *>(prm.Wp) + i);
    }
    if (tid < 64) affine[tid] = prm.rs ? make_float2(__ldg(prm.rs + tid), __ldg(prm.rb + tid)) : make_float2(1.f, 0.f);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_slot, 0);
    const int OW = prm.W >> 1, PH = prm.H >> 2, PW = prm.W >> 2;

    if (warp < 4) {
        // ---------------- image rows ----------------
        // The copies run kStAhead rows in front of the conversion, over the same sequence of (unit, row).  A row is up to 168 pieces
        // of 16 bytes: piece tid, and tid + 128 for the first threads.
        const int W4 = prm.W >> 2;
        long long at[2];                                   // of the thread's pieces: within a row of the image, and in a slot
        uint32_t to[2];
        bool has[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int e = tid + 128 * j, c = e / W4, x = e - c * W4;
            has[j] = c < 3;
            at[j] = (long long)c * prm.H * prm.W + 4 * x;
            to[j] = smem_u32(img_s + (c < 3 ? c : 0) * kStPitch + 4 + 4 * x);
        }
        int fu = blockIdx.x, fy = 0, fend = 0, fslot = 0;  // what is fetched next: image row fy of unit fu, up to fend
        const float *frow = prm.X;
        auto fetch = [&]() {
            if (fu < prm.units) {
                if (fy == fend) {                          // a new unit
                    const StUnit t(prm, fu);
                    fy = 4 * t.pr0 - 2;
                    fend = fy + t.image_rows();
                    frow = prm.X + ((long long)t.b * 3 * prm.H + fy) * prm.W;
                }
                if (fy >= 0 && fy < prm.H) {
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        if (has[j])
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                         ::"r"(to[j] + (uint32_t)fslot * (3 * kStPitch * 4)), "l"(frow + at[j]) : "memory");
                }
                frow += prm.W;
                if (++fslot == kStStages) fslot = 0;
                if (++fy == fend) fu += gridDim.x;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int i = 0; i < kStAhead; ++i) fetch();
        bool ok = true;
        int q = 0, slot = 0;
        const uint32_t lanes = tmem_base + ((uint32_t)(warp * 32) << 16);
        for (int u = blockIdx.x; u < prm.units; u += gridDim.x) {
            const StUnit t(prm, u);
            const int n = t.image_rows();
            // Two rows at a time (a unit has an odd number: the last one alone): a row by itself is a chain of waits and latencies of
            // 1100 clocks, more than the MMAs of half a convolution row take.
#pragma unroll 1
            for (int iy = 0; iy < n; iy += 2) {
                const int both = min(2, n - iy);
                asm volatile("cp.async.wait_group %0;" ::"n"(kStAhead - 2) : "memory");
                asm volatile("bar.sync 1, 128;" ::: "memory");     // these rows have landed for all, those before have been read by all
                uint32_t v[2][3][8];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (e == both) break;
                    fetch();
                    const int y = 4 * t.pr0 - 2 + iy + e;
                    const bool in = y >= 0 && y < prm.H;
                    const float *p = img_s + slot * 3 * kStPitch + 2 * (28 * warp + lane) + 2;
                    if (++slot == kStStages) slot = 0;
#pragma unroll
                    for (int c = 0; c < 3; ++c)
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            const float2 f = in ? *reinterpret_cast<const float2 *>(p + c * kStPitch + 2 * h) : make_float2(0.f, 0.f);
                            v[e][c][2 * h] = tf32_operand(f.x);
                            v[e][c][2 * h + 1] = tf32_operand(f.y);
                        }
                }
                // (a warp that gave up keeps walking: the others count on it at the barrier)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (e == both) break;
                    const int s = (q + e) % kStRing;
                    if (ok) ok = mbar_wait_warp(empty_bar(s), (((q + e) / kStRing) & 1) ^ 1u, abort_flag, 0x1600u | s, prm.spin_limit);
                    if (!ok) continue;
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < 3; ++c) tmem_st8(lanes + (uint32_t)(s * kStCols + 8 * c), v[e][c]);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (ok && lane == 0)
                    for (int e = 0; e < both; ++e) mbar_arrive(full_bar((q + e) % kStRing));
                q += both;
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == 4) {
        // ---------------- MMAs ----------------
        const bool leader = elect_one();
        const uint32_t idesc = make_idesc_tf32(128, 64);
        bool ok = true;
        int q0 = 0, r = 0;                     // first image row of the unit, convolution rows so far
        for (int u = blockIdx.x; u < prm.units && ok; u += gridDim.x) {
            const StUnit t(prm, u);
            int ready = 0;                     // image rows of the unit known to be there
            for (int k = 0; k < t.convs && ok; ++k, ++r) {
                const int buf = r & 1;
                if (!mbar_wait_warp(acce_bar(buf), ((r >> 1) & 1) ^ 1u, abort_flag, 0x1700u | buf, prm.spin_limit)) { ok = false; break; }
                for (; ready < 2 * k + 7 && ok; ++ready) {
                    const int q = q0 + ready;
                    ok = mbar_wait_warp(full_bar(q % kStRing), (q / kStRing) & 1, abort_flag, 0x1800u | (q % kStRing), prm.spin_limit);
                }
                if (!ok) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(kStAccCol + 64 * buf);
                if (leader) {
                    for (int ky = 0; ky < 7; ++ky) {
                        const uint32_t a = tmem_base + (uint32_t)(((q0 + 2 * k + ky) % kStRing) * kStCols);
                        const uint64_t bdesc = make_desc_k_sw128(base + ky * (64 * 128));
#pragma unroll
                        for (int c = 0; c < 3; ++c) umma_tf32_ts(d_tmem, a + 8u * c, bdesc + 2u * c, idesc, (ky > 0 || c > 0) ? 1u : 0u);
                    }
                    umma_commit(accf_bar(buf));
                    const int done = k + 1 == t.convs ? 7 : 2;         // image rows that nothing reads any more
                    for (int e = 0; e < done; ++e) umma_commit(empty_bar((q0 + 2 * k + e) % kStRing));
                }
                __syncwarp();
            }
            q0 += t.image_rows();
        }
    } else {
        // ---------------- pool and store ----------------
        // The vertical maxima of a pooled row meet in shared memory (two buffers); there every thread takes the horizontal maxima of
        // four outputs and stores them as 16 bytes of both results.  (Shuffles and stores straight from the lanes, 56 bytes
        // each, kept the load/store unit busy for 2500 clocks a pooled row: 235 us at 256 images.)
        const int quarter = warp & 3, half = (warp - 5) >> 2, et = tid - 160;
        const int px = 28 * quarter + lane;
        const bool mine = lane < 28 && px < OW;
        const int nq = (PW + 3) >> 2, items = 64 * nq;
        const bool vec = (PW & 3) == 0 && ((reinterpret_cast<uintptr_t>(prm.Y) | reinterpret_cast<uintptr_t>(prm.Yr)) & 15u) == 0;
        const int ch0 = et / nq, xq0 = et - ch0 * nq, dch = 256 / nq, dxq = 256 - dch * nq;     // item et, and the step to item et + 256
        const long long plane = (long long)PH * PW;
        bool ok = true;
        int r = 0, eb = 0;
        for (int u = blockIdx.x; u < prm.units; u += gridDim.x) {
            const StUnit t(prm, u);
            float m[32];
            for (int k = 0; k < t.convs; ++k, ++r) {
                const int buf = r & 1;
                // (a warp that gave up keeps walking: the others count on it at the barrier)
                if (ok) ok = mbar_wait_warp(accf_bar(buf), (r >> 1) & 1, abort_flag, 0x1900u | buf, prm.spin_limit);
                tc_fence_after();
                float v[32];
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(kStAccCol + 64 * buf + 32 * half);
#pragma unroll
                for (int e = 0; e < 4; ++e) tmem_ld8(taddr + 8 * e, v + 8 * e);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(acce_bar(buf));
                // convolution row 2 i + 2 ends pooled row i = pr0 + k / 2 - 1 and begins the next; where it does not exist, row
                // 2 i + 1 ends it
                const bool last = k + 1 == t.convs && (k & 1);
                if (k > 0) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) m[c] = fmaxf(m[c], v[c]);
                }
                if (k > 0 && (!(k & 1) || last)) {
                    const int i = t.pr0 + (last ? k >> 1 : (k >> 1) - 1);
                    float *E = pool_s + eb * (64 * kStEPitch);
                    eb ^= 1;
                    if (mine) {
#pragma unroll
                        for (int c = 0; c < 32; ++c) E[(32 * half + c) * kStEPitch + px] = m[c];
                    }
                    asm volatile("bar.sync 2, 256;" ::: "memory");
                    int ch = ch0, xq = xq0;
#pragma unroll 1
                    for (int e = et; e < items; e += 256) {
                        const float *p = E + ch * kStEPitch + 8 * xq;
                        const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
                        const float z = p[8];
                        const float4 o = make_float4(fmaxf(fmaxf(a.x, a.y), a.z), fmaxf(fmaxf(a.z, a.w), b.x), fmaxf(fmaxf(b.x, b.y), b.z),
                                                     fmaxf(fmaxf(b.z, b.w), z));
                        const long long at = ((long long)t.b * 64 + ch) * plane + (long long)i * PW + 4 * xq;
                        const float2 af = affine[ch];
                        const float4 q = make_float4(fmaxf(fmaf(o.x, af.x, af.y), 0.f), fmaxf(fmaf(o.y, af.x, af.y), 0.f),
                                                     fmaxf(fmaf(o.z, af.x, af.y), 0.f), fmaxf(fmaf(o.w, af.x, af.y), 0.f));
                        if (vec) {
                            *reinterpret_cast<float4 *>(prm.Y + at) = o;
                            if (prm.Yr) *reinterpret_cast<float4 *>(prm.Yr + at) = q;
                        } else {
                            const int nx = PW - 4 * xq;
                            const float ov[4] = {o.x, o.y, o.z, o.w}, qv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                            for (int x = 0; x < 4; ++x)
                                if (x < nx) {
                                    prm.Y[at + x] = ov[x];
                                    if (prm.Yr) prm.Yr[at + x] = qv[x];
                                }
                        }
                        ch += dch;
                        xq += dxq;
                        if (xq >= nq) { xq -= nq; ++ch; }
                    }
                }
                if (!(k & 1)) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) m[c] = v[c];
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 4) {
        if (*abort_flag) let_them_land();
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

int stem_prepare(const float *W, float *Wp, cudaStream_t st)
{
    if (!W || !Wp) return WG2X2_ERR_BAD_ARG;
    return launch(stem_prepare_kernel, dim3(cdiv(kStWtFloats, 256)), 256, 0, st, W, Wp);
}

int stem_pool(const float *X, const float *Wp, float *Y, float *Yrelu, const float *rs, const float *rb, int B, int H, int W,
              cudaStream_t st)
{
    if (!X || !Wp || !Y || B <= 0) return WG2X2_ERR_BAD_ARG;
    if ((rs == nullptr) != (rb == nullptr) || (rs && !Yrelu)) return WG2X2_ERR_BAD_ARG;
    if (H < 4 || W < 4 || (H & 3) || (W & 3)) return WG2X2_ERR_UNSUPPORTED;   // even convolution and pool sizes only
    if (W > kStMaxW) return WG2X2_ERR_UNSUPPORTED;
    if (misaligned16(X) || misaligned16(Wp)) return WG2X2_ERR_BAD_ARG;
    StParams p;
    p.X = X; p.Wp = Wp; p.Y = Y; p.Yr = Yrelu; p.rs = rs; p.rb = rb;
    p.H = H; p.W = W;
    // Pooled rows per unit: a unit computes one convolution row twice and fills the pipeline again (about one pooled row's time in
    // all); the height with the least rows on the busiest SM.
    const int PH = H / 4;
    double best = 1e30;
    p.band_rows = PH;
    for (int r = 1; r <= PH; ++r) {
        const double cost = (double)cdivll((long long)B * cdiv(PH, r), kNumSMs) * (r + 1.0);
        if (cost < best) { best = cost; p.band_rows = r; }
    }
    p.bands = cdiv(PH, p.band_rows);
    const long long units = (long long)B * p.bands;
    if (units > 0x7fffffffLL) return WG2X2_ERR_UNSUPPORTED;
    p.units = (int)units;
    p.spin_limit = wait_limit();
    return launch(stem_pool_kernel, dim3((unsigned)(units < kNumSMs ? units : kNumSMs)), kStThreads, kStSmemBytes, st, p);
}
