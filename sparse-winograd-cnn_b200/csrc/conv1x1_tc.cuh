// 1 x 1 convolution of an NCHW image for few pixels, the shortcut branch of a residual block that changes the channel count
// (ResNet-18-var/imagenet-resnet-transWino-prune.py:127-128): Y[b][k][p] = sum_c W[k][c] X[b][c][p].  Included by conv_tc.cu.
//
// A CTA owns 128 pixels (of any images) x 64 output channels.  All its operands fit shared memory at once (C <= 256: eight chunks of
// 32 channels), so nothing is recycled: TMA brings every weight tile at the start, eight warps turn the pixels (lane = pixel,
// 4 channels at a time) into K-major operand tiles, one warp issues the MMAs chunk by chunk, and the eight warps store the
// accumulator, 32 consecutive pixels per instruction.  Image values and weights are rounded to TF32 (nearest; the weights by
// the caller).  Why: the library's call costs 10 us of host time, this one 4, and the network makes four of them; on the GPU this one
// takes 4.4 us for 64 channels and 9 for 256 against 3.1 and 7.7 as long as a CTA per SM holds all pixels.  (Four chunks of pixels in
// flight per thread instead of one measured slower.)
#pragma once

constexpr int kC1MaxChunks = 8;
constexpr int kC1Threads = 288;                          // eight pixel warps, MMA issuer
constexpr int kC1StageBytes = kABytes + kBBytes;         // 24 KB a chunk

struct C1Params {
    const float *X;
    float *Y;
    long long pixels;        // B * HW
    int C, K, HW, chunks;
    uint32_t spin_limit;
    int drop_load;           // test hook: CTA 0 stops in front of this weight load, so that the wait for it runs out
};

__global__ void __launch_bounds__(kC1Threads) conv1x1_tc_kernel(const __grid_constant__ CUtensorMap mapW, const C1Params prm)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    __shared__ uint64_t bars[kC1MaxChunks + 1];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    volatile int *abort_flag = &abort_word;
    const uint32_t full0 = smem_u32(bars), done_bar = full0 + 8u * kC1MaxChunks;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int c = 0; c < kC1MaxChunks; ++c) mbar_init(full0 + 8u * c, 9);
        mbar_init(done_bar, 1);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) {
        tmem_alloc(smem_u32(&tmem_slot), 64);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *reinterpret_cast<volatile uint32_t *>(&tmem_slot), 0);
    wait_for_previous_kernel(kNumSMs);

    const int row = (warp & 3) * 32 + lane;                         // the thread's pixel of the block, as producer and at the end
    const long long p = (long long)blockIdx.x * kBlockM + row;
    const bool live = p < prm.pixels;
    const long long b = live ? p / prm.HW : 0;
    const int px = live ? (int)(p - b * prm.HW) : 0, k0 = blockIdx.y * kBlockN;
    if (warp < 8) {
        // groups of 4 channels: half = warp / 4 takes the even or the odd ones of a chunk's eight
        const int half = warp >> 2;
        const float *src = prm.X + b * prm.C * (long long)prm.HW + px;
        for (int cc = 0; cc < prm.chunks; ++cc) {
            float v[4][4];
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const int c = cc * kBlockK + 4 * (2 * g + half);
                const bool ok = live && c < prm.C;
#pragma unroll
                for (int q = 0; q < 4; ++q) v[g][q] = ok ? __ldg(src + (long long)(c + q) * prm.HW) : 0.f;
            }
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const uint32_t dst = base + cc * kC1StageBytes + row * 128 + (((2 * g + half) ^ (row & 7)) << 4);
                asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(tf32_operand(v[g][0])), "r"(tf32_operand(v[g][1])),
                             "r"(tf32_operand(v[g][2])), "r"(tf32_operand(v[g][3])) : "memory");
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8u * cc);
        }
    } else {
        const bool leader = elect_one();
        if (leader)
            for (int cc = 0; cc < prm.chunks; ++cc) {
                if (cc == prm.drop_load && blockIdx.x == 0 && blockIdx.y == 0) break;
                mbar_expect_tx(full0 + 8u * cc, kBBytes);
                tma_load_3d(base + cc * kC1StageBytes + kABytes, &mapW, full0 + 8u * cc, cc * kBlockK, k0, 0);
            }
        __syncwarp();
        const uint32_t idesc = make_idesc_tf32(kBlockM, kBlockN);
        for (int cc = 0; cc < prm.chunks; ++cc) {
            if (!mbar_wait_warp(full0 + 8u * cc, 0, abort_flag, 0x1A00u | cc, prm.spin_limit)) break;
            tc_fence_after();
            if (leader) {
                const uint64_t ad = make_desc_k_sw128(base + cc * kC1StageBytes), bd = make_desc_k_sw128(base + cc * kC1StageBytes + kABytes);
#pragma unroll
                for (int kk = 0; kk < kBlockK / 8; ++kk) umma_tf32(tmem_base, ad + 2u * kk, bd + 2u * kk, idesc, (cc > 0 || kk > 0) ? 1u : 0u);
                if (cc + 1 == prm.chunks) umma_commit(done_bar);
            }
            __syncwarp();
        }
    }
    const bool done = mbar_wait_warp(done_bar, 0, abort_flag, 0x1B00u, prm.spin_limit);
    tc_fence_after();
    if (warp < 8 && done) {
        const int half = warp >> 2;
        float r[32];
#pragma unroll
        for (int e = 0; e < 4; ++e) tmem_ld8(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(32 * half + 8 * e), r + 8 * e);
        tmem_ld_wait();
        const int k = k0 + 32 * half;
        float *dst = prm.Y + (b * prm.K + k) * (long long)prm.HW + px;
        if (live) {
#pragma unroll
            for (int c = 0; c < 32; ++c, dst += prm.HW)
                if (k + c < prm.K) *dst = r[c];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        if (!done) let_them_land();
        tc_fence_after();
        tmem_dealloc(tmem_base, 64);
    }
}

// Where the network is faster with this kernel than with the library's call: up to two rounds of CTAs, each of which transforms its
// pixels for 64 output channels only and starts from nothing.  ResNet-18-var, microseconds with every call in these bounds here / with
// none: 1 image 194 / 215, 2 images 216 / 219, 4: 260 / 263, 8: 352 / 360, 16: 457 / 460, 32: 616 / 625, 48: 878 / 884.  Beyond, the
// library's kernel is the faster one by more than host time can hide (256 channels of 48 x 14 x 14 in two rounds 8.7 against 7.2 us, in
// four 15.4 against 10.0).
bool conv1x1_preferred(int B, int C, int K, int HW)
{
    return C % 4 == 0 && C <= kC1MaxChunks * kBlockK && cdivll((long long)B * HW, kBlockM) * cdiv(K, kBlockN) <= 2 * kNumSMs;
}

int conv1x1(const float *X, const float *W, float *Y, int B, int C, int K, int HW, cudaStream_t st)
{
    if (!X || !W || !Y || B <= 0 || C <= 0 || K <= 0 || HW <= 0) return WG2X2_ERR_BAD_ARG;
    if (C % 4 || C > kC1MaxChunks * kBlockK) return WG2X2_ERR_UNSUPPORTED;
    if (misaligned16(W)) return WG2X2_ERR_BAD_ARG;
    C1Params p;
    p.X = X; p.Y = Y; p.pixels = (long long)B * HW; p.C = C; p.K = K; p.HW = HW; p.chunks = cdiv(C, kBlockK);
    p.spin_limit = wait_limit();
    p.drop_load = take_drop_load();
    const long long blocks = cdivll(p.pixels, kBlockM);
    if (blocks > 0x7fffffffLL || cdiv(K, kBlockN) > 65535) return WG2X2_ERR_UNSUPPORTED;
    EncodeTiledFn fn = encode_fn();
    if (!fn) return WG2X2_ERR_LAUNCH;
    CUtensorMap mapW;
    cuuint64_t dims[3] = {(cuuint64_t)C, (cuuint64_t)K, 1};
    cuuint64_t strides[2] = {(cuuint64_t)C * 4, (cuuint64_t)K * C * 4};
    cuuint32_t box[3] = {(cuuint32_t)kBlockK, (cuuint32_t)kBlockN, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    if (fn(&mapW, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float *>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return WG2X2_ERR_LAUNCH;
    return launch(conv1x1_tc_kernel, dim3((unsigned)blocks, cdiv(K, kBlockN)), kC1Threads, 1024 + (size_t)p.chunks * kC1StageBytes, st, mapW, p);
}
