// One-kernel layer for problems of few tiles: X -> Y in one launch, for either layout and any image size.  Included by
// conv_tc.cu.
//
// A cluster of four CTAs owns `tpu` tiles x N output channels.  CTA i computes Winograd row i of the products, positions
// (i, 0..3): its sixteen producer warps form row i of B^T d B from the two image rows it needs, straight from global memory into
// the tensor core's operand tiles (four [tpu tiles x 32 channels] tiles a stage), TMA brings the weights, and four 128 x N
// accumulators stay in tensor memory.  At the end every CTA applies A^T along the columns, hands each of the four a quarter of
// the channels through distributed shared memory, and the four rows meet there: y0 = z0 + z1 + z2, y1 = z1 - z2 - z3, with
// the optional affine map and shortcut.  Neither V nor the products touch memory.
//
// Why: such a layer is bound by launches and by the latency chains inside its kernels, not by bytes.  As three kernels (transform,
// sixteen GEMMs, output transform) it takes 10 us of GPU time however small it is, and as much host time; this kernel takes 3.9 us
// with one chunk of 32 input channels (2 x 9 x 13 x 32), 5.6 us for one image of 64 x 64 x 56 x 56 (11.9 before).  Per CTA, in
// clocks: first pixels 2000, a chunk 1200 - 2000, exchange 2500, stores 500 - 1500.  What it pays is that every block of N
// channels transforms its tiles again and that a second round of CTAs costs as much as the first, so it is left to few tiles
// (cl_cut, layer_cluster_preferred).
#pragma once

constexpr int kClWarps = 16;                             // producers, then epilogue
constexpr int kClThreads = 32 * (kClWarps + 2);          // + MMA issuer and TMEM owner, + weight producer
constexpr int kClMaxStages = 6;
constexpr int kClRingBytes = 192 * 1024;                 // operand stages: 2 of 128 tiles x 64 channels .. 6 of 32 x 32
// The exchange buffer: [Winograd row][output column][channel][tile], 8 N (tpu + 2) bytes (the 2: channels 4 apart on different
// banks).  All but the largest cut (128 tiles x 64 channels) have it beside the stages, the largest one over them.
constexpr int kClZBytes = 8 * 64 * (64 + 2);
constexpr int kClMaxN = 64;
constexpr int kClSmemBytes = 1024 + kClRingBytes + kClZBytes + kCtrlBytes;
static_assert(kClSmemBytes <= 232448, "shared memory per CTA");

struct ClParams {
    const float *X;
    float *Y;
    const float *in_scale, *in_shift, *out_scale, *out_shift, *residual;
    long long P;
    int H, W, C, K, nH, nW;
    int N, tpu;              // output channels (32 or 64) and tiles (32, 64 or 128) per cluster
    int nKB, nCC, stages;
    int relu, res_relu;
    uint32_t spin_limit;
};

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float *r)
{
    uint32_t u[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "r"(taddr));
#pragma unroll
    for (int q = 0; q < 4; ++q) r[q] = __uint_as_float(u[q]);
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) { asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
// started: every CTA of the cluster is running, so that its shared memory may be written (arrive once, early; wait once)
__device__ __forceinline__ void cluster_arrive_started() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait_started() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }

enum { kClNhwc = 0, kClNchwEven = 1, kClNchwOdd = 2 };   // MODE: the image's layout, NCHW by the parity of W

template <int MODE>
__global__ void __cluster_dims__(4, 1, 1) __launch_bounds__(kClThreads, 1)
layer_fwd_cluster_kernel(const __grid_constant__ CUtensorMap mapW, const ClParams prm)
{
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gen_base = smem_raw + (base - raw);
    const uint32_t b_bytes = (uint32_t)prm.N * 4 * kBlockK * 4;
    // A tile of a position: `tpu` rows of 128 bytes.  The MMA reads 128 rows; those beyond the tile are other tiles' bytes and
    // end in accumulator rows that nobody reads.
    const uint32_t a_bytes = (uint32_t)prm.tpu * 4 * kBlockK * 4, a_pos = (uint32_t)prm.tpu * kBlockK * 4;
    const uint32_t stage_bytes = a_bytes + b_bytes;
    const int stages = prm.stages;
    constexpr int kCtrlAt = kClRingBytes + kClZBytes;
    const uint32_t bars = base + kCtrlAt;
    auto full_bar = [&](int s) { return bars + 8u * s; };
    auto empty_bar = [&](int s) { return bars + 8u * (kClMaxStages + s); };
    const uint32_t done_bar = bars + 16u * kClMaxStages;
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(gen_base + kCtrlAt + 16 * kClMaxStages + 8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(gen_base + kCtrlAt + 16 * kClMaxStages + 16);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31, tid = threadIdx.x;
    const uint32_t wrow = cluster_ctarank();                 // the Winograd row of this CTA
    const int unit = blockIdx.x >> 2, kb = unit % prm.nKB;
    const long long p0 = (long long)(unit / prm.nKB) * prm.tpu;
    if (tid == 0) {
        // 32 tiles are work for eight warps: the two halves of the producers take chunks in turn
        for (int s = 0; s < kClMaxStages; ++s) { mbar_init(full_bar(s), (prm.tpu == 32 ? kClWarps / 2 : kClWarps) + 1); mbar_init(empty_bar(s), 1); }
        mbar_init(done_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kClWarps) {
        tmem_alloc(smem_u32((const void *)tmem_ptr_slot), 4 * kClMaxN);
        tmem_relinquish();
    }

    // ---- which pixels are this thread's: worked out in front of the wait for the kernel before ----
    // the tile (NHWC: and the group of 4 channels) whose outputs it will store
    const int NQ = prm.N >> 2;                               // channels per CTA after the exchange
    const int tpu_log2 = prm.tpu == 128 ? 7 : prm.tpu == 64 ? 6 : 5;
    const int ng_log2 = prm.N == 64 ? 2 : 1;                 // groups of 4 among them
    const int kq = kb * prm.N + (int)wrow * NQ;              // the first of them
    const int t_out = MODE == kClNhwc ? tid >> ng_log2 : tid & (prm.tpu - 1);
    auto decode = [&](long long p, int &b, int &th, int &tw) {
        const unsigned q = (unsigned)p, r = q / (unsigned)prm.nW;
        tw = (int)(q - r * (unsigned)prm.nW);
        b = (int)(r / (unsigned)prm.nH);
        th = (int)(r - (unsigned)b * (unsigned)prm.nH);
    };
    int b_out, th_out, tw_out;
    const bool out_ok = t_out < prm.tpu && p0 + t_out < prm.P;
    decode(out_ok ? p0 + t_out : 0, b_out, th_out, tw_out);
    // producers: rows of the 4 x 4 window and the sign of the second: d0 - d2, d1 + d2, d2 - d1, d1 - d3
    const int ya = wrow == 0 ? 0 : wrow == 2 ? 2 : 1, yb = wrow == 2 ? 1 : wrow == 3 ? 3 : 2;
    const float sb = wrow == 1 ? 1.f : -1.f;
    const int teams = prm.tpu == 32 ? 2 : 1, team = teams == 2 ? warp >> 3 : 0;
    const int id = teams == 2 ? tid & 255 : tid;
    const int per = prm.tpu == 128 ? 2 : 1;                  // items (tile x 4 channels) of a thread in a chunk
    const int C = prm.C, W = prm.W;
    const long long cstride = MODE == kClNhwc ? 1 : (long long)prm.H * W;   // between channels
    // NHWC: eight lanes along the channels, tiles id / 8 and 64 further on.  NCHW: lanes along the tiles; one tile per
    // thread, groups id / tpu and 4 further on.
    const float *pa[2], *pb[2];
    int tile[2], cols[2], tws[2];
    bool ra[2], rb[2];
#pragma unroll
    for (int it = 0; it < (MODE == kClNhwc ? 2 : 1); ++it) {
        tile[it] = MODE == kClNhwc ? (id >> 3) + 64 * it : id & (prm.tpu - 1);
        const long long p = p0 + tile[it];
        const bool ok = p < prm.P;
        int tw = tw_out, b = b_out, th = th_out;             // (NCHW: the same tile)
        if (MODE == kClNhwc) decode(ok ? p : 0, b, th, tw);
        const int fa = 2 * th - 1 + ya, fb = 2 * th - 1 + yb, fx = 2 * tw - 1;
        ra[it] = ok && fa >= 0 && fa < prm.H;
        rb[it] = ok && fb >= 0 && fb < prm.H;
        cols[it] = (fx >= 0 ? 1 : 0) | 2 | (fx + 2 < W ? 4 : 0) | (fx + 3 < W ? 8 : 0);
        tws[it] = tw;
        if (MODE == kClNhwc) {
            pa[it] = prm.X + (((long long)b * prm.H + fa) * W + fx) * C;
            pb[it] = prm.X + (((long long)b * prm.H + fb) * W + fx) * C;
        } else {
            pa[it] = prm.X + ((long long)b * C * prm.H + fa) * W + fx;
            pb[it] = prm.X + ((long long)b * C * prm.H + fb) * W + fx;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_slot, 0);
    cluster_arrive_started();
    wait_for_previous_kernel(kNumSMs);

    if (warp < kClWarps) {
        // ---------------- producers: row `wrow` of B^T d B, straight into the operand tiles ----------------
        // v[4 x + q] / v[16 + 4 x + q]: column x, channel q of the two rows; NCHW with even W: the two middle pixels come as
        // one pair (x = 1, 2), x = 0 is the one outer pixel that no neighbouring lane holds
        auto group = [&](int it) { return MODE == kClNhwc ? id & 7 : (id >> tpu_log2) + 4 * it; };
        auto load = [&](float (&v)[32], int cc, int it) {
            const int k = MODE == kClNhwc ? it : 0;
            const int c = cc * kBlockK + 4 * group(it);
            const bool live = c < C;
            const long long off = MODE == kClNhwc ? (long long)c : c * cstride;
            const float *qa = (k ? pa[1] : pa[0]) + off, *qb = (k ? pb[1] : pb[0]) + off;
            const bool la = live && (k ? ra[1] : ra[0]), lb = live && (k ? rb[1] : rb[0]);
            const int cm = k ? cols[1] : cols[0];
            if (MODE == kClNhwc) {
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const bool cx = (cm >> x) & 1;
                    const float4 a = la && cx ? __ldg(reinterpret_cast<const float4 *>(qa + (long long)x * C)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float4 b = lb && cx ? __ldg(reinterpret_cast<const float4 *>(qb + (long long)x * C)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[4 * x] = a.x; v[4 * x + 1] = a.y; v[4 * x + 2] = a.z; v[4 * x + 3] = a.w;
                    v[16 + 4 * x] = b.x; v[16 + 4 * x + 1] = b.y; v[16 + 4 * x + 2] = b.z; v[16 + 4 * x + 3] = b.w;
                }
            } else if (MODE == kClNchwEven) {
                const bool outer = (lane == 0 && tws[0] > 0) || (lane == 31 && tws[0] < prm.nW - 1);
                const int ox = lane == 0 ? 0 : 3;
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float2 a = la ? __ldg(reinterpret_cast<const float2 *>(qa + q * cstride + 1)) : make_float2(0.f, 0.f);
                    const float2 b = lb ? __ldg(reinterpret_cast<const float2 *>(qb + q * cstride + 1)) : make_float2(0.f, 0.f);
                    v[4 + q] = a.x; v[8 + q] = a.y; v[20 + q] = b.x; v[24 + q] = b.y;
                    v[q] = la && outer ? __ldg(qa + q * cstride + ox) : 0.f;
                    v[16 + q] = lb && outer ? __ldg(qb + q * cstride + ox) : 0.f;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const bool cx = (cm >> x) & 1;
                        v[4 * x + q] = la && cx ? __ldg(qa + q * cstride + x) : 0.f;
                        v[16 + 4 * x + q] = lb && cx ? __ldg(qb + q * cstride + x) : 0.f;
                    }
            }
        };
        auto emit = [&](float (&v)[32], int cc, int it, uint32_t a_addr) {
            const int k = MODE == kClNhwc ? it : 0;
            const int g = group(it), c = cc * kBlockK + 4 * g;
            const int cm = k ? cols[1] : cols[0];
            if (prm.in_scale && c < C) {
                const float4 s = __ldg(reinterpret_cast<const float4 *>(prm.in_scale + c)), t = __ldg(reinterpret_cast<const float4 *>(prm.in_shift + c));
                const float s4[4] = {s.x, s.y, s.z, s.w}, t4[4] = {t.x, t.y, t.z, t.w};
                const bool la = k ? ra[1] : ra[0], lb = k ? rb[1] : rb[0];
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const bool cx = MODE == kClNchwEven || ((cm >> x) & 1);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (la && cx) v[4 * x + q] = fmaf(v[4 * x + q], s4[q], t4[q]);
                        if (lb && cx) v[16 + 4 * x + q] = fmaf(v[16 + 4 * x + q], s4[q], t4[q]);
                    }
                }
            }
            float out[4][4];             // [position][channel]
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float r[4];
                if (MODE == kClNchwEven) {
                    const float m1 = fmaf(sb, v[20 + q], v[4 + q]), m2 = fmaf(sb, v[24 + q], v[8 + q]), o = fmaf(sb, v[16 + q], v[q]);
                    const float l = __shfl_up_sync(0xffffffffu, m2, 1), h = __shfl_down_sync(0xffffffffu, m1, 1);
                    r[0] = tws[0] == 0 ? 0.f : lane == 0 ? o : l;
                    r[1] = m1;
                    r[2] = m2;
                    r[3] = tws[0] == prm.nW - 1 ? 0.f : lane == 31 ? o : h;
                } else {
#pragma unroll
                    for (int x = 0; x < 4; ++x) r[x] = fmaf(sb, v[16 + 4 * x + q], v[4 * x + q]);
                }
                out[0][q] = r[0] - r[2];
                out[1][q] = r[1] + r[2];
                out[2][q] = r[2] - r[1];
                out[3][q] = r[1] - r[3];
            }
            const int row = k ? tile[1] : tile[0];
            const uint32_t dst = a_addr + (uint32_t)(row * 128 + ((g ^ (row & 7)) << 4));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (prm.relu) {
#pragma unroll
                    for (int q = 0; q < 4; ++q) out[j][q] = fmaxf(out[j][q], 0.f);
                }
                asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + j * a_pos), "f"(out[j][0]), "f"(out[j][1]), "f"(out[j][2]), "f"(out[j][3]) : "memory");
            }
        };
        // items in turn, (chunk, it); the loads of the next one are in flight while one is turned
        float cur[32], nxt[32];
        int cc = team, it = 0, s = team;
        uint32_t ph = 0;
        if (cc < prm.nCC) load(cur, cc, 0);
        while (cc < prm.nCC) {
            const int it1 = it + 1 < per ? it + 1 : 0, cc1 = it1 ? cc : cc + teams;
            if (cc1 < prm.nCC) load(nxt, cc1, it1);
            if (it == 0 && !mbar_wait_warp(empty_bar(s), ph ^ 1u, abort_flag, 0x1200u | s, prm.spin_limit)) break;
            emit(cur, cc, it, base + s * stage_bytes);
            if (it1 == 0) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(full_bar(s));
                s += teams;
                if (s >= stages) { s -= stages; ph ^= 1u; }
            }
            cc = cc1; it = it1;
#pragma unroll
            for (int e = 0; e < 32; ++e) cur[e] = nxt[e];
        }
    } else if (warp == kClWarps) {
        // ---------------- MMA issuer ----------------
        const bool leader = elect_one();
        const uint32_t idesc = make_idesc_tf32(kBlockM, prm.N);
        int s = 0;
        uint32_t ph = 0;
        for (int cc = 0; cc < prm.nCC; ++cc) {
            if (!mbar_wait_warp(full_bar(s), ph, abort_flag, 0x1300u | s, prm.spin_limit)) break;
            tc_fence_after();
            const uint32_t a_addr = base + s * stage_bytes, b_addr = a_addr + a_bytes;
            if (leader) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint64_t adesc = make_desc_k_sw128(a_addr + j * a_pos), bdesc = make_desc_k_sw128(b_addr + j * prm.N * 128);
#pragma unroll
                    for (int kk = 0; kk < kBlockK / 8; ++kk)
                        umma_tf32(tmem_base + (uint32_t)(j * prm.N), adesc + 2u * kk, bdesc + 2u * kk, idesc, (cc > 0 || kk > 0) ? 1u : 0u);
                }
                umma_commit(cc == prm.nCC - 1 ? done_bar : empty_bar(s));
            }
            __syncwarp();
            if (++s == stages) { s = 0; ph ^= 1u; }
        }
    } else if (lane == 0) {
        // ---------------- weights: positions 4 wrow .. + 3 of a chunk in one box ----------------
        bool ok = true;
        int s = 0;
        uint32_t ph = 0;
        for (int cc = 0; cc < prm.nCC; ++cc) {
            if (!mbar_wait(empty_bar(s), ph ^ 1u, abort_flag, 0x1400u | s, prm.spin_limit)) { ok = false; break; }
            mbar_expect_tx(full_bar(s), b_bytes);
            tma_load_3d(base + s * stage_bytes + a_bytes, &mapW, full_bar(s), cc * kBlockK, kb * prm.N, (int)wrow * 4);
            if (++s == stages) { s = 0; ph ^= 1u; }
        }
        if (!ok)
            for (int it = 0; it < 1000; ++it) __nanosleep(1000);
    }

    // ---------------- exchange: column transform, then quarter r of the channels to CTA r ----------------
    __syncwarp();
    const bool done = mbar_wait_warp(done_bar, 0, abort_flag, 0x1500u, prm.spin_limit);
    tc_fence_after();
    const bool z_apart = 8 * prm.N * (prm.tpu + 2) <= kClZBytes;
    const uint32_t z_at = z_apart ? kClRingBytes : 0;
    cluster_wait_started();
    if (!z_apart) cluster_sync_all();              // every CTA's MMAs have read their operands: the stages may be overwritten
    const int pitch = prm.tpu + 2;
    const int q = warp & 3, r = (warp >> 2) & 3;
    if (warp < kClWarps && done && q * 32 < prm.tpu) {
        const uint32_t dst = mapa_rank(base + z_at, (uint32_t)r) + 4u * (wrow * 2 * NQ * pitch + q * 32 + lane);
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(r * NQ);
        for (int c = 0; c < NQ; c += 4) {
            float m[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) tmem_ld4(taddr + (uint32_t)(j * prm.N + c), m[j]);
            tmem_ld_wait();
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                float z0, z1;
                at_cols(m[0][x], m[1][x], m[2][x], m[3][x], z0, z1);
                st_cluster(dst + 4u * (uint32_t)((c + x) * pitch), z0);
                st_cluster(dst + 4u * (uint32_t)((NQ + c + x) * pitch), z1);
            }
        }
    }
    tc_fence_before();
    cluster_sync_all();              // all four rows have arrived; nobody writes here any more
    if (warp == kClWarps) {
        if (!done) let_them_land();
        tc_fence_after();
        tmem_dealloc(tmem_base, 4 * kClMaxN);
    }
    if (warp >= kClWarps || !out_ok) return;

    // ---------------- rows meet; store ----------------
    const float *Z = reinterpret_cast<const float *>(gen_base + z_at) + t_out;
    auto outputs = [&](int c, float (&y)[2][2]) {
        y[0][0] = y[0][1] = y[1][0] = y[1][1] = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) at_rows_accum(i, Z[(i * 2 * NQ + c) * pitch], Z[(i * 2 * NQ + NQ + c) * pitch], y);
    };
    if (MODE == kClNhwc) {
        const int g = tid & ((1 << ng_log2) - 1), k = kq + 4 * g, nk = prm.K - k;
        if (nk <= 0) return;
        float y[4][2][2];
#pragma unroll
        for (int x = 0; x < 4; ++x) outputs(4 * g + x, y[x]);
        float s[4] = {1.f, 1.f, 1.f, 1.f}, h[4] = {0.f, 0.f, 0.f, 0.f};
        if (prm.out_scale) {
#pragma unroll
            for (int x = 0; x < 4; ++x)
                if (x < nk) { s[x] = __ldg(prm.out_scale + k + x); h[x] = __ldg(prm.out_shift + k + x); }
        }
        const bool vec = (prm.K & 3) == 0;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int f = 0; f < 2; ++f) {
                const int oy = 2 * th_out + a, ox = 2 * tw_out + f;
                if (oy >= prm.H || ox >= prm.W) continue;
                const long long o = (((long long)b_out * prm.H + oy) * prm.W + ox) * prm.K + k;
                float w[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) w[x] = fmaf(y[x][a][f], s[x], h[x]);
                if (prm.residual) {
                    float rs[4] = {0.f, 0.f, 0.f, 0.f};
                    if (vec) {
                        const float4 v = __ldg(reinterpret_cast<const float4 *>(prm.residual + o));
                        rs[0] = v.x; rs[1] = v.y; rs[2] = v.z; rs[3] = v.w;
                    } else {
#pragma unroll
                        for (int x = 0; x < 4; ++x) if (x < nk) rs[x] = __ldg(prm.residual + o + x);
                    }
#pragma unroll
                    for (int x = 0; x < 4; ++x) w[x] += prm.res_relu ? relu_nan(rs[x]) : rs[x];
                }
                if (vec) {
                    *reinterpret_cast<float4 *>(prm.Y + o) = make_float4(w[0], w[1], w[2], w[3]);
                } else {
#pragma unroll
                    for (int x = 0; x < 4; ++x) if (x < nk) prm.Y[o + x] = w[x];
                }
            }
    } else {
        const bool two = 2 * tw_out + 1 < prm.W;
        for (int c = tid >> tpu_log2; c < NQ; c += (32 * kClWarps) >> tpu_log2) {
            const int k = kq + c;
            if (k >= prm.K) break;
            float y[2][2];
            outputs(c, y);
            const float s = prm.out_scale ? __ldg(prm.out_scale + k) : 1.f, h = prm.out_scale ? __ldg(prm.out_shift + k) : 0.f;
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                if (2 * th_out + a >= prm.H) continue;
                const long long o = (((long long)b_out * prm.K + k) * prm.H + 2 * th_out + a) * prm.W + 2 * tw_out;
                float w0 = fmaf(y[a][0], s, h), w1 = fmaf(y[a][1], s, h);
                if (prm.residual) {
                    float2 rs = make_float2(0.f, 0.f);
                    if (MODE == kClNchwEven) rs = __ldg(reinterpret_cast<const float2 *>(prm.residual + o));
                    else { rs.x = __ldg(prm.residual + o); if (two) rs.y = __ldg(prm.residual + o + 1); }
                    w0 += prm.res_relu ? relu_nan(rs.x) : rs.x;
                    w1 += prm.res_relu ? relu_nan(rs.y) : rs.y;
                }
                if (MODE == kClNchwEven) *reinterpret_cast<float2 *>(prm.Y + o) = make_float2(w0, w1);
                else { prm.Y[o] = w0; if (two) prm.Y[o + 1] = w1; }
            }
        }
    }
}

// How many clusters the device holds at once (0: none); asked once per device.
static int cl_clusters()
{
    static std::atomic<int> cached[64];          // 0: not asked yet, else the count + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    int n = cached[dev].load();
    if (n > 0) return n - 1;
    n = 0;
    const void *kernel = reinterpret_cast<const void *>(layer_fwd_cluster_kernel<kClNhwc>);
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSmemBytes) == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(4 * kNumSMs);
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = kClSmemBytes;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 4; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int got = 0;
        if (cudaOccupancyMaxActiveClusters(&got, layer_fwd_cluster_kernel<kClNhwc>, &cfg) == cudaSuccess && got > 0) n = got;
        else (void)cudaGetLastError();
    }
    cached[dev].store(n + 1);
    return n;
}

// Tiles and channels per cluster, and what the layer then takes in microseconds: rounds of clusters x (a + b x chunks of 32 input
// channels), fitted to within 8 % over 110 shapes of 16 .. 42300 tiles and 16 .. 512 channels in both layouts.  Narrow cuts put
// more SMs to work on a chunk, wide ones transform a tile for fewer blocks of channels.
struct ClCut { int N, tpu; double us; };
static ClCut cl_cut(long long P, int C, int K)
{
    static const struct { int N, tpu; double a, b; } cuts[] = {{32, 32, 4.0, 0.73}, {64, 32, 4.3, 0.80},  {32, 64, 4.1, 1.15},
                                                               {64, 64, 4.5, 1.25}, {32, 128, 4.7, 2.03}, {64, 128, 6.6, 2.12}};
    ClCut best{64, 128, 1e30};
    const int at_once = cl_clusters();
    if (at_once <= 0) return best;
    for (const auto &c : cuts) {
        const double us = (double)cdivll(cdivll(P, c.tpu) * cdiv(K, c.N), at_once) * (c.a + c.b * cdiv(C, kBlockK));
        if (us < best.us) best = ClCut{c.N, c.tpu, us};
    }
    return best;
}

int layer_fwd_cluster(const float *X, const void *prepared, float *Y, int B, int H, int W, int C, int K, int layout, int relu,
                      const float *in_scale, const float *in_shift, const float *out_scale, const float *out_shift, const float *residual,
                      int res_relu, cudaStream_t st)
{
    if (!X || !prepared || !Y) return WG2X2_ERR_BAD_ARG;
    if ((out_scale == nullptr) != (out_shift == nullptr) || (in_scale == nullptr) != (in_shift == nullptr)) return WG2X2_ERR_BAD_ARG;
    if (!tc_shape_supported(C, K)) return WG2X2_ERR_UNSUPPORTED;
    if (misaligned16(X) || misaligned16(prepared) || misaligned16(Y) || misaligned16(in_scale) || misaligned16(in_shift) ||
        misaligned16(residual))
        return WG2X2_ERR_BAD_ARG;
    ClParams p;
    p.X = X; p.Y = Y; p.in_scale = in_scale; p.in_shift = in_shift; p.out_scale = out_scale; p.out_shift = out_shift; p.residual = residual;
    p.H = H; p.W = W; p.C = C; p.K = K; p.nH = (H + 1) / 2; p.nW = (W + 1) / 2;
    p.P = (long long)B * p.nH * p.nW;
    p.relu = relu; p.res_relu = res_relu;
    const ClCut cut = cl_cut(p.P, C, K);
    p.N = cut.N; p.tpu = cut.tpu;
    p.nKB = cdiv(K, p.N); p.nCC = cdiv(C, kBlockK);
    p.stages = kClRingBytes / (4 * kBlockK * 4 * (p.tpu + p.N));
    if (p.stages > kClMaxStages) p.stages = kClMaxStages;
    if (p.tpu == 32) p.stages &= ~1;          // the two halves of the producers keep to their own stages
    p.spin_limit = wait_limit();
    const long long ctas = 4 * cdivll(p.P, p.tpu) * p.nKB;
    if (p.P > 0x7fffffffLL || ctas > 0x7fffffffLL) return WG2X2_ERR_UNSUPPORTED;
    EncodeTiledFn fn = encode_fn();
    if (!fn) return WG2X2_ERR_LAUNCH;
    CUtensorMap mapW;
    cuuint64_t dims[3] = {(cuuint64_t)C, (cuuint64_t)K, 16};
    cuuint64_t strides[2] = {(cuuint64_t)C * 4, (cuuint64_t)K * C * 4};
    cuuint32_t box[3] = {(cuuint32_t)kBlockK, (cuuint32_t)p.N, 4};
    cuuint32_t estr[3] = {1, 1, 1};
    if (fn(&mapW, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void *>(prepared), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return WG2X2_ERR_LAUNCH;
    auto *kernel = layout == WG2X2_NHWC ? layer_fwd_cluster_kernel<kClNhwc>
                                        : (W & 1) ? layer_fwd_cluster_kernel<kClNchwOdd> : layer_fwd_cluster_kernel<kClNchwEven>;
    return launch(kernel, dim3((unsigned)ctas), kClThreads, kClSmemBytes, st, mapW, p);
}
