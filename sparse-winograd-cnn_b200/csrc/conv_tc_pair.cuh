// Winograd-ReLU layer forward, X -> Y in one kernel, on pairs of SMs (NCHW, any image size, and channels last where a
// row of quads is whole, W % 4 == 0 and K % 4 == 0): neither the transformed input V nor the
// sixteen Winograd-domain products ever exist outside an SM.  Included by conv_tc.cu.
//
// As in conv_tc_fused.cuh both transforms ride on the tensor core's operands: the A operand of every MMA (position (i, j) of B^T d B,
// after the ReLU) is written into tensor memory by transform warps, and position (i, j) is accumulated with the sign
// At[a][i] At[e][j] straight into the output accumulators (a, e) it contributes to, 36 MMAs per 8 input channels.  What differs:
//   * tcgen05 cta_group::2: two CTAs share an M = 256, N = 64 unit, each holding half of every weight tile, so that the weight
//     tiles' reads from shared memory, half of that kernel's shared-memory time, are halved; with up to 64 outputs all weights stay in
//     shared memory for the whole launch where they fit beside the pixels: up to 64 input channels (channels last not in every
//     width), up to 80 in two image sizes of five;
//   * tiles go to tensor-memory lanes densely, in quads of 2 x 2 (4 x 4 output pixels), whatever image and row they lie in: 64 images
//     of 56 x 56 are 196 units of 256 tiles in three rounds on 66 pairs, where whole rows of tiles need four;
//   * a thread forms all sixteen positions of a quad's four tiles from one 6 x 6 window: 36 loads for 64 values, and one
//     tcgen05.st of 16 lanes x 32 columns per Winograd row and row of tiles;
//   * pixels come as plain bulk copies of the rows' contiguous memory, so that an NCHW image needs no row length of 16-byte pieces; channels
//     last as one TMA box of 8 channels per row of quads, read by thread pairs as two channels at a time;
//   * Y leaves from registers, 16 bytes a thread where rows allow; the shortcut is added in front of the stores, or behind them in L2 where
//     rows are of 16-byte pieces and a pair has more than one unit.
// A unit walks the input channels in slots of 8: transform team n % 2 fills A group n % 2 (16 positions x 8 columns), four issuers,
// one per accumulator, take it from there.
//
// What it measured (us, this against the fastest of the other paths): 64 x 64 x 56 x 56 45 -> 34, 256 images of it 137 -> 105,
// 256 x 128 x 28 x 28 138 -> 97, 128 x 256 x 14 x 14 93 -> 68, 64 x 256 x 40 x 40 341 -> 170;
// channels last 32 x 128 x 28 x 28 37 -> 22.  What bounds it: a slot's MMAs take 1152
// clocks, a slot takes about 1600.  With the MMAs at full rate tensor memory takes one store of 1 KB per subpartition and MMA (16 of 36
// such gaps are needed, so that stores are slow and the warps behind them wait), a transform warp's own chain of loads, shuffles, 288
// arithmetic instructions and eight stores is 2700 clocks for its two slots, and issue slots are 57 % busy.  At the end of a unit the
// stores of one output row hold the other's accumulators: 4000 - 5000 clocks, when all SMs store at once.
// Tried, at 256 x 128 x 28 x 28 with 97 .. 100 us as it is: pixels by loads into registers (latency: 111), sixteen transform warps of one
// channel each (stores of 256 bytes: 106), three teams (101 .. 105), issuers that look ahead for the next slot's barrier (104, with three
// teams 113), one issuer per output row (two in all: 141), a full barrier per half group (126); at 256 x 64 x 56 x 56, 108 as it is, an
// epilogue that takes three of the four quarter rows into registers before its first store (111).
#pragma once

constexpr int kPrThreads = 768;                    // 4 issuing, 4 loading, 8 epilogue, 8 transform warps
constexpr int kPrQuads = 32;                       // quads (2 x 2 tiles, 4 x 4 output pixels) per CTA and unit: 128 lanes
constexpr int kPrACol0 = 256, kPrGroupCols = 128;  // tensor memory: four accumulators, then two A groups (16 positions x 8 channels)
constexpr int kPrRegsMma = 32, kPrRegsLoad = 24, kPrRegsEpi = 96, kPrRegsXf = 112, kPrRegsLaunch = 80;
static_assert(128 * kPrRegsMma + 128 * kPrRegsLoad + 256 * kPrRegsEpi + 256 * kPrRegsXf <= kPrRegsLaunch * kPrThreads,
              "setmaxnreg shares exceed the registers the CTA was launched with");
constexpr int kPrN = kBlockN;                      // output channels per unit
constexpr int kPrStageBytes = 16 * (kPrN / 2) * 64;   // weights: 16 positions x half of N x 16 channels
constexpr int kPrMaxW = 6, kPrMaxX = 3;            // stages of weights and of pixels at most
constexpr int kPrSmemMax = 232448 - 1024 - kCtrlBytes;

struct PrParams {
    const float *X;
    float *Y;
    const float *in_scale, *in_shift, *out_scale, *out_shift, *residual;
    const unsigned long long *masks;       // zero-block map of the prepared weights: bit cc of masks[t][k / 64]
    int B, H, W, C, K;
    int nQH, nQW, quads;                   // quads down, across, in all
    int nW, nX, xbytes;                    // stages of weights and pixels, bytes of a pixel stage
    int xpitch, xpart, whole;              // floats of a channel and of a whole image in a pixel stage; whole images are copied (pr_geometry)
    int nKB, nS, units;                    // blocks of N output channels, slots of 8 channels, units of 64 quads x N channels
    int relu, res_relu, front;             // front: the shortcut is added in front of the stores
    int in_place;                          // in_place: Y holds the shortcut, its ReLU applied, and 16-byte pieces are added to it
    uint32_t zero;                         // 0, which the compiler does not know
    uint32_t spin_limit;                   // polls before a wait gives up (wg2x2_set_wait_limit)
    int drop_load;                         // >= 0: the W producer of CTA 0 leaves out its drop_load-th stage (wg2x2_test_drop_load), else -1
};

// An arrival on a barrier of the pair's leader by a role whose tensor-memory accesses are complete (tcgen05.wait) and which wrote
// nothing else: no fence over the loads that it has in flight
__device__ __forceinline__ void mbar_arrive_peer(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// D[tmem of both CTAs] (+)= A[tmem] * B[smem], M = 256, K = 8 (tf32).  Executed by a whole converged warp, issued by the lane with
// `leader`: a predicate, no branch, so that the operands stay in uniform registers.
__device__ __forceinline__ void umma_tf32_ts_pair(uint32_t leader, uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p, l;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "setp.ne.b32 l, %6, 0;\n\t"
        "mov.b64 b, {%2, %3};\n\t"
        "@l tcgen05.mma.cta_group::2.kind::tf32 [%0], [%1], b, %4, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(leader) : "memory");
}
// the barrier at this offset in both CTAs of the pair gets one arrival once all MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_both(uint32_t leader, uint32_t bar)
{
    asm volatile("{\n\t.reg .pred l;\n\tsetp.ne.b32 l, %2, 0;\n\t"
                 "@l tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
                 ::"r"(bar), "h"((unsigned short)3), "r"(leader) : "memory");
}
// two sums / differences in one instruction
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
    float2 o;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(o.x), "=f"(o.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return o;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b)
{
    float2 o;
    asm("{\n\t.reg .b64 x, y;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tsub.rn.f32x2 x, x, y;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(o.x), "=f"(o.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return o;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
    float2 o;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\tfma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(o.x), "=f"(o.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return o;
}
// 16 lanes x 32 columns: r[2 q], r[2 q + 1] = lanes l / 4 and l / 4 + 8 of column 4 q + l % 4
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, float *r)
{
    uint32_t u[16];
    asm volatile("tcgen05.ld.sync.aligned.16x128b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]),
                   "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(taddr));
#pragma unroll
    for (int q = 0; q < 16; ++q) r[q] = __uint_as_float(u[q]);
}
// 16 lanes x 32 columns, as tmem_ld_16x32
__device__ __forceinline__ void tmem_st_16x32(uint32_t taddr, const float *r)
{
    asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(__float_as_uint(r[0])), "r"(__float_as_uint(r[1])), "r"(__float_as_uint(r[2])), "r"(__float_as_uint(r[3])), "r"(__float_as_uint(r[4])), "r"(__float_as_uint(r[5])),
                   "r"(__float_as_uint(r[6])), "r"(__float_as_uint(r[7])), "r"(__float_as_uint(r[8])), "r"(__float_as_uint(r[9])), "r"(__float_as_uint(r[10])), "r"(__float_as_uint(r[11])),
                   "r"(__float_as_uint(r[12])), "r"(__float_as_uint(r[13])), "r"(__float_as_uint(r[14])), "r"(__float_as_uint(r[15])) : "memory");
}

// The same with pairs of columns: r[4 q + 2 d + p] = lane l / 4 + 8 d of column 8 q + 2 (l % 4) + p
__device__ __forceinline__ void tmem_ld_16x32_pairs(uint32_t taddr, float *r)
{
    uint32_t u[16];
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]),
                   "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
                 : "r"(taddr));
#pragma unroll
    for (int q = 0; q < 16; ++q) r[q] = __uint_as_float(u[q]);
}
__device__ __forceinline__ void tmem_st_16x32_pairs(uint32_t taddr, const float *r)
{
    asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "f"(r[0]), "f"(r[1]), "f"(r[2]), "f"(r[3]), "f"(r[4]), "f"(r[5]), "f"(r[6]), "f"(r[7]), "f"(r[8]), "f"(r[9]), "f"(r[10]), "f"(r[11]),
                   "f"(r[12]), "f"(r[13]), "f"(r[14]), "f"(r[15]) : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap *map, uint32_t bar, int c0, int c1, int c2, int c3, int c4)
{
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4) : "memory");
}

// Where a thread's quad lies, as bits: rows 0 .. 5 of the window inside the image; the quad's left / right neighbour does not exist;
// an outer pixel has to be loaded (the neighbouring quad is another warp's)
constexpr uint32_t kPrNoLeft = 1u << 6, kPrNoRight = 1u << 7, kPrEdge = 1u << 8;

// Shared-memory loads of up to four floats, zero where `ok` is not set.  Not volatile: the compiler schedules them freely; they are kept
// behind the barrier waits by the "memory" clobber of those.
__device__ __forceinline__ void pr_lds4(float (&d)[4], uint32_t at, uint32_t ok)
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
        "@p ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];\n\t}" : "=&f"(d[0]), "=&f"(d[1]), "=&f"(d[2]), "=&f"(d[3]) : "r"(at), "r"(ok) : "memory");
}
__device__ __forceinline__ void pr_lds2(float &x, float &y, uint32_t at, uint32_t ok)
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t@p ld.shared.v2.f32 {%0,%1}, [%2];\n\t}"
        : "=&f"(x), "=&f"(y) : "r"(at), "r"(ok) : "memory");
}
__device__ __forceinline__ void pr_lds1(float &x, uint32_t at, uint32_t ok)
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.shared.f32 %0, [%1];\n\t}" : "=&f"(x) : "r"(at), "r"(ok) : "memory");
}
__device__ __forceinline__ float2 pr_lds2(uint32_t at)
{
    float2 v;
    asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
    return v;
}
// Two channels of a pixel from and to memory
__device__ __forceinline__ void pr_ldg2(float &x, float &y, const float *p, bool ok)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t@p ld.global.v2.f32 {%0,%1}, [%2];\n\t}"
                 : "=&f"(x), "=&f"(y) : "l"(p), "r"((int)ok));
}
__device__ __forceinline__ void pr_stg2(float *p, float x, float y, bool ok)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t@p st.global.v2.f32 [%0], {%1,%2};\n\t}" ::"l"(p), "f"(x), "f"(y), "r"((int)ok) : "memory");
}
// Four pixels of a row from and to memory, `cols` of them inside the image, none where `ok` is not set: predicates, no branches, so that a
// row's eight accesses go out together
template <int VEC>
__device__ __forceinline__ void pr_ldg(float (&d)[4], const float *p, int cols, bool ok)
{
    if (VEC == 4) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
                     "@p ld.global.v4.f32 {%0,%1,%2,%3}, [%4];\n\t}" : "=&f"(d[0]), "=&f"(d[1]), "=&f"(d[2]), "=&f"(d[3]) : "l"(p), "r"((int)ok));
    } else if (VEC == 2) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\tmov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t@p ld.global.v2.f32 {%0,%1}, [%2];\n\t}"
                         : "=&f"(d[2 * h]), "=&f"(d[2 * h + 1]) : "l"(p + 2 * h), "r"((int)(ok && 2 * h < cols)));
    } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\tmov.b32 %0, 0;\n\t@p ld.global.f32 %0, [%1];\n\t}" : "=&f"(d[x]) : "l"(p + x), "r"((int)(ok && x < cols)));
    }
}
template <int VEC>
__device__ __forceinline__ void pr_stg(float *p, float o0, float o1, float o2, float o3, int cols, bool ok)
{
    if (VEC == 4) {
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p st.global.v4.f32 [%0], {%1,%2,%3,%4};\n\t}" ::"l"(p), "f"(o0), "f"(o1), "f"(o2), "f"(o3), "r"((int)ok) : "memory");
    } else if (VEC == 2) {
        asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t@p st.global.v2.f32 [%0], {%1,%2};\n\t@q st.global.v2.f32 [%0+8], {%3,%4};\n\t}"
                     ::"l"(p), "f"(o0), "f"(o1), "f"(o2), "f"(o3), "r"((int)ok), "r"((int)(ok && cols > 2)) : "memory");
    } else {
        const float o[4] = {o0, o1, o2, o3};
#pragma unroll
        for (int x = 0; x < 4; ++x)
            asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(p + x), "f"(o[x]), "r"((int)(ok && x < cols)) : "memory");
    }
}
// 16 bytes added to what is there
__device__ __forceinline__ void pr_red4(float *p, float o0, float o1, float o2, float o3, bool ok)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p red.global.add.v4.f32 [%0], {%1,%2,%3,%4};\n\t}" ::"l"(p), "f"(o0), "f"(o1), "f"(o2), "f"(o3), "r"((int)ok) : "memory");
}
// One channel of a quad's window: the own columns of its six rows, and in lanes at a warp's end the pixel beyond
template <int VEC>
__device__ __forceinline__ void pr_window(float (&d)[6][4], float (&e)[6], uint32_t at, int W, int eoff, uint32_t flags, int cols)
{
#pragma unroll
    for (int r = 0; r < 6; ++r) {
        const uint32_t in = flags & (1u << r), q = at + 4u * (uint32_t)(r * W);
        if (VEC == 4) {
            pr_lds4(d[r], q, in);
        } else if (VEC == 2) {
            pr_lds2(d[r][0], d[r][1], q, in);
            pr_lds2(d[r][2], d[r][3], q + 8u, cols > 2 ? in : 0u);
        } else {
#pragma unroll
            for (int x = 0; x < 4; ++x) pr_lds1(d[r][x], q + 4u * x, x < cols ? in : 0u);
        }
    }
#pragma unroll
    for (int r = 0; r < 6; ++r) pr_lds1(e[r], at + 4u * (uint32_t)(r * W) + (uint32_t)eoff, flags & kPrEdge ? flags & (1u << r) : 0u);
}

// The pixels of a unit's 32 quads: of each image that they touch the rows of their windows, contiguous in memory.
struct PrSpan {
    int b0, n, y0, y1;       // first image, images; rows [y0, H) of the first (to y1 where it is the only one), [0, y1) of the last, all of those between
};
__device__ __forceinline__ PrSpan pr_span(const PrParams &prm, int q0)
{
    PrSpan s;
    const int q1 = min(q0 + kPrQuads, prm.quads) - 1;
    if (q1 < q0) { s.b0 = 0; s.n = 0; s.y0 = 0; s.y1 = 0; return s; }
    const int t0 = q0 / prm.nQW, t1 = q1 / prm.nQW;
    s.b0 = t0 / prm.nQH;
    const int b1 = t1 / prm.nQH;
    s.n = b1 - s.b0 + 1;
    s.y0 = prm.whole ? 0 : max(4 * (t0 - s.b0 * prm.nQH) - 1, 0);
    s.y1 = prm.whole ? prm.H : min(4 * (t1 - b1 * prm.nQH) + 5, prm.H);
    return s;
}
// floats that `n` floats from any 4-byte boundary may take when copied in 16-byte pieces
__host__ __device__ __forceinline__ int pr_room(int n) { return (n + 6) & ~3; }

// where in a stage channel ch of the span's image `part` begins
__device__ __forceinline__ int pr_offset(const PrParams &prm, const PrSpan &sp, int part, int ch)
{
    return ch * prm.xpitch + (part == 0 ? 0 : prm.whole ? part * prm.xpart : pr_room((prm.H - sp.y0) * prm.W) + (part - 1) * prm.xpart);
}

// VEC: 4, 2, 1 = NCHW, floats that can be accessed at once by the row length; kPrNhwc = channels last
constexpr int kPrNhwc = 0;

template <int VEC, bool AFFINE, bool EXTRAS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPrThreads, 1)
layer_fwd_pair_kernel(const __grid_constant__ CUtensorMap mapW, const __grid_constant__ CUtensorMap mapX, PrParams prm)
{
    constexpr bool NHWC = VEC == kPrNhwc;
    constexpr int N = kPrN, kStageBytes = kPrStageBytes;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t *gen_base = smem_raw + (base - raw);
    const uint32_t xbase = base + prm.nW * kStageBytes;
    const uint32_t bars = xbase + prm.nX * prm.xbytes;
    uint64_t *bars_gen = reinterpret_cast<uint64_t *>(gen_base + prm.nW * kStageBytes + prm.nX * prm.xbytes);
    // Slot n fills pixel stage n % nX but signals xfull[n % (2 nX)]: the two teams may take turns on a stage, and a parity wait can only
    // tell a barrier's current phase from the one before it, so a waiter has to see every phase of the barrier it waits on.
    constexpr int kB0 = 0, kB1 = 4, kB2 = 8, kB3 = 10, kB4 = 12, kB5 = kB4 + kPrMaxW, kB6 = kB5 + kPrMaxW, kB7 = kB6 + 2 * kPrMaxX, kB8 = kB7 + kPrMaxX;
    static_assert((kB8 + 2) * 8 <= kCtrlBytes, "control block");
    auto full_bar = [&](int h) { return bars + 8u * (kB0 + h); };
    auto free_bar = [&](int h) { return bars + 8u * (kB1 + h); };
    auto accf_bar = [&](int a) { return bars + 8u * (kB2 + a); };
    auto acce_bar = [&](int a) { return bars + 8u * (kB3 + a); };
    auto wfull_bar = [&](int s) { return bars + 8u * (kB4 + s); };
    auto wempty_bar = [&](int s) { return bars + 8u * (kB5 + s); };
    auto xfull_bar = [&](int s) { return bars + 8u * (kB6 + s); };
    auto xempty_bar = [&](int s) { return bars + 8u * (kB7 + s); };
    volatile uint32_t *tmem_ptr_slot = reinterpret_cast<volatile uint32_t *>(bars_gen + kB8);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(bars_gen + kB8 + 1);

    // (broadcast from lane 0: the compiler then treats the warp index, and all that is derived from it, as warp-uniform)
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    if (threadIdx.x == 0) {
        for (int g = 0; g < 2; ++g) mbar_init(full_bar(g), 8);
        for (int h = 0; h < 4; ++h) mbar_init(free_bar(h), 4);
        for (int a = 0; a < 2; ++a) { mbar_init(accf_bar(a), 2); mbar_init(acce_bar(a), 2 * kEpiWarps); }
        for (int s = 0; s < kPrMaxW; ++s) { mbar_init(wfull_bar(s), 1); mbar_init(wempty_bar(s), 4); }
        for (int s = 0; s < 2 * kPrMaxX; ++s) mbar_init(xfull_bar(s), 3);
        for (int s = 0; s < kPrMaxX; ++s) mbar_init(xempty_bar(s), 4);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32((const void *)tmem_ptr_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();    // the partner's barriers exist before anything is signalled into them
    tc_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_ptr_slot, 0);
    // (set-up touched no global memory; from here on the kernel reads and writes it, through pointers that pass through the wait)
    after_previous_kernel(prm.X, prm.Y, prm.in_scale, prm.in_shift, prm.out_scale, prm.out_shift, prm.residual, prm.masks);

    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int nS = prm.nS, nW2 = (nS + 1) >> 1;    // slots of 8 channels and weight stages of 16 in a unit
    const int my_units = (prm.units - pair + npairs - 1) / npairs;
    const bool resident = prm.nKB == 1 && nW2 <= prm.nW;      // a unit's weights stay in shared memory for all units

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPrRegsMma));
        if (rank == 0) {
            // ------------------------------ MMA issuers -----------------------------------
            constexpr uint32_t idesc = make_idesc_tf32(256, N);
            // Issuer (a, e) = warp 2 a + e owns that accumulator, to which the positions (i, j) of three Winograd rows and columns contribute
            // with sign At[a][i] At[e][j]: At = [[1,1,1,0],[0,1,-1,-1]].
            const uint32_t leader = elect_one() ? 1u : 0u;
            const int a = warp >> 1, e = warp & 1;
            const uint32_t d0 = tmem_base + (uint32_t)(warp * N);
            const uint32_t idesc_a = idesc ^ ((uint32_t)a << 14), idesc_e = idesc ^ ((uint32_t)e << 14), idesc_ae = idesc ^ ((uint32_t)(a ^ e) << 14);   // bit 14: negate B
            const uint64_t bdesc0 = make_desc_k_sw64(base);
            const uint32_t b_hi = (uint32_t)(bdesc0 >> 32), b_lo0 = (uint32_t)bdesc0;
            int stage = 0; uint32_t wph = 0;
            uint32_t n = 0;                                               // slots so far
            bool ok = true;
            for (int iu = 0; iu < my_units && ok; ++iu) {
                // zero-block word of position `lane` (bit cc: the weights of input channels cc*32.. have a non-zero)
                const unsigned long long mask = lane < 16 ? __ldg(prm.masks + (long long)lane * prm.nKB + (pair + iu * npairs) % prm.nKB) : ~0ull;
                if (resident) stage = 0;
                uint32_t live = 0xffffu;
                for (int sl = 0; sl < nS; ++sl, ++n) {
                    // all-zero weight blocks add nothing (the unit's first chunk always runs: it zero-initialises)
                    if (!(sl & 3)) live = sl == 0 || sl >= 256 ? 0xffffu : __ballot_sync(0xffffffffu, (mask >> (sl >> 2)) & 1ull);
                    if (!(sl & 1) && !(resident && iu > 0) && !mbar_wait_warp(wfull_bar(stage), wph, abort_flag, 0x1000u | (warp << 8) | stage, prm.spin_limit)) { ok = false; break; }
                    const uint32_t g = n & 1u, gph = (n >> 1) & 1u;
                    const uint32_t a_tmem = tmem_base + (uint32_t)kPrACol0 + g * kPrGroupCols + 8u * (4 * a + e);
                    const uint32_t b_lo = b_lo0 + (uint32_t)(stage * (kStageBytes >> 4)) + (sl & 1) * 2u + (uint32_t)((4 * a + e) * (N / 2 * 64 >> 4));
                    if (!mbar_wait_warp(full_bar(g), gph, abort_flag, 0x1040u | (warp << 8) | g, prm.spin_limit)) { ok = false; break; }
                    // the unit's first MMA overwrites the accumulator: the epilogues must have read the previous unit's
                    if (sl == 0 && !mbar_wait_warp(acce_bar(a), ((uint32_t)iu & 1u) ^ 1u, abort_flag, 0x1080u | (warp << 8), prm.spin_limit)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t live_ae = (live >> (4 * a + e)) & (0u - leader);
#pragma unroll
                    for (int ii = 0; ii < 3; ++ii) {                       // position (a + ii, e + jj)
#pragma unroll
                        for (int jj = 0; jj < 3; ++jj)
                            umma_tf32_ts_pair(live_ae & (1u << (4 * ii + jj)), d0, a_tmem + 8u * (4 * ii + jj), b_lo + (uint32_t)((4 * ii + jj) * (N / 2 * 64 >> 4)), b_hi,
                                              ii == 0 ? (jj == 0 ? idesc : idesc_e) : (jj == 0 ? idesc_a : idesc_ae), ii == 0 && jj == 0 && sl == 0 ? 0u : 1u);
                        if (ii == 1 - a) umma_commit_both(leader, free_bar(2 * g));
                    }
                    umma_commit_both(leader, free_bar(2 * g + 1));
                    if ((sl & 1) || sl == nS - 1) {
                        if (!resident) umma_commit_both(leader, wempty_bar(stage));
                        if (sl == nS - 1) umma_commit_both(leader, accf_bar(a));
                        if (++stage == prm.nW) { stage = 0; if (!resident) wph ^= 1u; }
                    }
                }
            }
        }
    } else if (warp < 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kPrRegsLoad));
        if (warp == 4 && lane == 0) {
            // ------------------------------ W producer -----------------------------------
            int s = 0; uint32_t ph = 0;
            bool ok = true;
            int nload = 0;
            const int loads = resident ? (my_units > 0 ? nW2 : 0) : my_units * nW2;
            int iu = 0, c16 = 0;
            for (int n = 0; n < loads; ++n) {
                const int kb = (pair + iu * npairs) % prm.nKB;
                if (!mbar_wait_sleepy(wempty_bar(s), ph ^ 1u, abort_flag, 0xA00u | s, 100, prm.spin_limit)) { ok = false; break; }
                // test hook: these weights never arrive (nothing is put in flight), so the issuers' wait on them runs out
                if (blockIdx.x == 0 && nload++ == prm.drop_load) { ok = false; break; }
                if (rank == 0) mbar_expect_tx(wfull_bar(s), 2u * kStageBytes);
                tma_load_3d_pair(base + s * kStageBytes, &mapW, mapa_rank0(wfull_bar(s)), c16 * 16, kb * N + (int)rank * (N / 2), 0);
                if (++s == prm.nW) { s = 0; ph ^= 1u; }
                if (++c16 == nW2) { c16 = 0; ++iu; }
            }
            if (!ok) let_them_land();
        } else if (warp > 4) {
            // ------------------------------ X producers -----------------------------------
            if constexpr (NHWC) {
                // Eight channels of the windows of every row of quads that the unit touches, one box each: [row of the window][column of a
                // quad][quad, with one more on either side][channel], zeros outside the image
                int xs = 0, xf = 0;
                uint32_t ph = 1;
                bool ok = true;
                for (int iu = 0; iu < my_units && ok; ++iu) {
                    const int q0 = ((pair + iu * npairs) / prm.nKB) * (2 * kPrQuads) + (int)rank * kPrQuads, q1 = min(q0 + kPrQuads, prm.quads) - 1;
                    const int t = q0 / prm.nQW + lane, b = t / prm.nQH, y = 4 * (t - b * prm.nQH) - 1;
                    const bool mine = q1 >= q0 && t <= q1 / prm.nQW && lane % 3 == warp - 5;
                    const uint32_t bytes = (uint32_t)__popc(__ballot_sync(0xffffffffu, mine)) * (uint32_t)prm.xpitch, dst = xbase + (uint32_t)(lane * prm.xpitch);
                    for (int sl = 0; sl < nS; ++sl) {
                        ok = mbar_wait_warp(xempty_bar(xs), ph, abort_flag, 0x900u | xs, prm.spin_limit);
                        if (!ok) break;
                        if (lane == 0) mbar_expect_tx(xfull_bar(xf), bytes);
                        __syncwarp();
                        if (mine) tma_load_5d(dst + xs * prm.xbytes, &mapX, xfull_bar(xf), 8 * sl, -1, 0, y, b);
                        if (++xs == prm.nX) { xs = 0; ph ^= 1u; }
                        if (++xf == 2 * prm.nX) xf = 0;
                    }
                }
                if (!ok) let_them_land();
            } else {
                // Eight channels of the unit's pixels per slot, as plain copies of contiguous memory: one per channel and image, or per image
                // where whole images are taken.  Copies go by 16 bytes: they start up to three floats early and end up to three late, inside
                // the tensor all the same (its size is a multiple of 16 bytes, as C is one of 4).
                // A lane has the same copy to make in every slot of a unit, 8 channels further on (8 H W floats: no other remainder).
                const int per = prm.whole ? 1 : 8;
                const long long step = 8LL * prm.H * prm.W;
                int xs = 0, xf = 0;
                uint32_t ph = 1;
                bool ok = true;
                for (int iu = 0; iu < my_units && ok; ++iu) {
                    const PrSpan sp = pr_span(prm, ((pair + iu * npairs) / prm.nKB) * (2 * kPrQuads) + (int)rank * kPrQuads);
                    const int part = lane / per, ch = lane - part * per;
                    const bool mine = part < sp.n && lane % 3 == warp - 5;
                    const int y0 = part == 0 ? sp.y0 : 0, floats = ((part == sp.n - 1 ? sp.y1 : prm.H) - y0) * prm.W;
                    const long long at = ((long long)(sp.b0 + part) * prm.C + ch) * prm.H * prm.W + (long long)y0 * prm.W;
                    const int rem = (int)(at & 3);
                    const float *src = prm.X + (at - rem);
                    const uint32_t dst = xbase + 4u * (uint32_t)pr_offset(prm, sp, part, ch);
                    for (int sl = 0; sl < nS; ++sl) {
                        ok = mbar_wait_warp(xempty_bar(xs), ph, abort_flag, 0x900u | xs, prm.spin_limit);
                        if (!ok) break;
                        const int chans = min(8, prm.C - 8 * sl);
                        const uint32_t bytes = mine && ch < chans ? 4u * (uint32_t)((rem + floats * (prm.whole ? chans : 1) + 3) & ~3) : 0u;
                        const uint32_t all = __reduce_add_sync(0xffffffffu, bytes);
                        if (lane == 0) mbar_expect_tx(xfull_bar(xf), all);
                        __syncwarp();
                        if (bytes)
                            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                         ::"r"(dst + xs * prm.xbytes), "l"(src), "r"(bytes), "r"(xfull_bar(xf)) : "memory");
                        src += step;
                        if (++xs == prm.nX) { xs = 0; ph ^= 1u; }
                        if (++xf == 2 * prm.nX) xf = 0;
                    }
                }
                if (!ok) let_them_land();
            }
        }
    } else {
        // the quad of this thread in a unit, by lane: eight quads per warp, four lanes (channels) per quad
        const int sub = warp & 3, qg = lane >> 2, cl = lane & 3;
        auto locate = [&](int iu, int &b, int &qr, int &qc) {
            const int q = ((pair + iu * npairs) / prm.nKB) * (2 * kPrQuads) + (int)rank * kPrQuads + sub * 8 + qg;
            qc = q % prm.nQW;
            const int t = q / prm.nQW;
            qr = t % prm.nQH;
            b = t / prm.nQH;
            return q < prm.quads;
        };
        if (warp >= 16) {
            // ------------------------------ transform teams ----------------------------------
            // Team t fills the slots n with n % 2 = t, always into A group t.  A thread walks its quad's channels, two a slot (cl and cl + 4).
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPrRegsXf));
            const int team = (warp - 16) >> 2;
            const float lo = prm.relu ? 0.f : __int_as_float(0x7fffffff);      // the larger of a number and NaN is the number: without a ReLU all stay
            const long long plane = (long long)prm.H * prm.W;
            const int total = my_units * nS;
            const uint32_t a_tmem = tmem_base + ((uint32_t)(sub * 32) << 16) + (uint32_t)(kPrACol0 + team * kPrGroupCols);
            const uint32_t full0 = mapa_rank0(full_bar(team));
            int iu = 0, sl = team, cols = 0;
            uint32_t flags = 0, quad = 0;                       // quad: byte offset of this thread's window in a stage
            long long at0 = 0;
            auto enter = [&]() {
                int b, qr, qc;
                const bool valid = locate(iu, b, qr, qc);
                const int q0 = ((pair + iu * npairs) / prm.nKB) * (2 * kPrQuads) + (int)rank * kPrQuads;
                if constexpr (NHWC) {
                    quad = (valid ? (uint32_t)((b * prm.nQH + qr - q0 / prm.nQW) * prm.xpitch + 32 * qc) : 0u) + 8u * cl;
                } else {
                    const PrSpan sp = pr_span(prm, q0);
                    const int part = b - sp.b0, y0 = part == 0 ? sp.y0 : 0;
                    at0 = ((long long)b * prm.C + cl) * plane + (long long)y0 * prm.W;
                    quad = valid ? 4u * (uint32_t)(pr_offset(prm, sp, part, cl) + (4 * qr - 1 - y0) * prm.W + 4 * qc) : 0u;
                }
                flags = 0;
#pragma unroll
                for (int r = 0; r < 6; ++r) {
                    const int y = 4 * qr - 1 + r;
                    if (valid && y >= 0 && y < prm.H) flags |= 1u << r;
                }
                cols = prm.W - 4 * qc;
                const bool no_l = qc == 0, no_r = cols <= 4;
                if (no_l) flags |= kPrNoLeft;
                if (no_r) flags |= kPrNoRight;
                if ((qg == 0 && !no_l) || (qg == 7 && !no_r)) flags |= kPrEdge;
            };
            while (sl >= nS) { sl -= nS; ++iu; }
            if (iu < my_units) enter();
            uint32_t fph = 1;                                   // parity of the free barriers' phase to wait for
            int xs = team % prm.nX, xf = team % (2 * prm.nX);
            uint32_t xph = 0;
            for (int n = team; n < total; n += 2) {
                bool ok = mbar_wait_warp(xfull_bar(xf), xph, abort_flag, 0xB00u | xf, prm.spin_limit);
                if (!ok) break;
                // [channel][row]: columns 0 1 | 2 3, and the outer two; channels last: [row][column], both channels
                float2 m[2][6][2], lr[2][6], win[6][6];
                uint32_t loaded = 0;                                 // a register of every load
                if constexpr (NHWC) {
                    const uint32_t at = xbase + xs * prm.xbytes + quad, px = 32u * (uint32_t)(prm.nQW + 2);
#pragma unroll
                    for (int r = 0; r < 6; ++r) {
                        const uint32_t ar = at + 4u * r * px;
                        win[r][0] = pr_lds2(ar + 3u * px);
#pragma unroll
                        for (int x = 0; x < 4; ++x) win[r][1 + x] = pr_lds2(ar + (uint32_t)x * px + 32u);
                        win[r][5] = pr_lds2(ar + 64u);
#pragma unroll
                        for (int x = 0; x < 6; ++x) loaded ^= __float_as_uint(win[r][x].x);
                    }
                    if (AFFINE) {
                        const int c = 8 * sl + 2 * cl;
                        const float2 sc = c < prm.C ? make_float2(__ldg(prm.in_scale + c), __ldg(prm.in_scale + c + 1)) : make_float2(1.f, 1.f);
                        const float2 tc = c < prm.C ? make_float2(__ldg(prm.in_shift + c), __ldg(prm.in_shift + c + 1)) : make_float2(0.f, 0.f);
                        // pixels outside the image stay zero, whatever the scale
#pragma unroll
                        for (int r = 0; r < 6; ++r) {
                            const bool row = (flags >> r) & 1u;
                            const float2 sr = make_float2(row ? sc.x : 0.f, row ? sc.y : 0.f), tr = make_float2(row ? tc.x : 0.f, row ? tc.y : 0.f);
#pragma unroll
                            for (int x = 0; x < 6; ++x) win[r][x] = fma2(sr, win[r][x], tr);
                            if (flags & kPrNoLeft) win[r][0] = make_float2(0.f, 0.f);
                            if (flags & kPrNoRight) win[r][5] = make_float2(0.f, 0.f);
                        }
                    }
                } else {
                    float d[2][6][4], ed[2][6];                          // [channel][row]
                    float sc[2], tc[2];
#pragma unroll
                    for (int p = 0; p < 2; ++p) {
                        const int c = 8 * sl + 4 * p;
                        const bool chan = c < prm.C;                     // C is a multiple of 4: the same for the four lanes of a quad
                        uint32_t at = xbase + xs * prm.xbytes + quad + p * (uint32_t)(16 * prm.xpitch);
                        if (VEC < 4 && !prm.whole) at += 4u * (uint32_t)((at0 + (long long)c * plane) & 3);   // where the copy's first 16 bytes begin
                        pr_window<VEC>(d[p], ed[p], at, prm.W, qg == 0 ? -4 : 16, chan ? flags : 0u, cols);
#pragma unroll
                        for (int r = 0; r < 6; ++r) {
                            loaded ^= __float_as_uint(ed[p][r]);
#pragma unroll
                            for (int x = 0; x < 4; x += VEC) loaded ^= __float_as_uint(d[p][r][x]);
                        }
                        if (AFFINE) { sc[p] = chan ? __ldg(prm.in_scale + c + cl) : 1.f; tc[p] = chan ? __ldg(prm.in_shift + c + cl) : 0.f; }
                    }
                    // the windows with their outer columns, from the neighbouring quads' lanes where those are in this warp
#pragma unroll
                    for (int p = 0; p < 2; ++p)
#pragma unroll
                        for (int r = 0; r < 6; ++r) {
                            if (AFFINE) {
                                // pixels outside the image stay zero, whatever the scale (an outer pixel that was not loaded is not looked at)
                                const bool row = (flags >> r) & 1u;
                                const float sr = row ? sc[p] : 0.f, tr = row ? tc[p] : 0.f;
#pragma unroll
                                for (int x = 0; x < 4; ++x)
                                    if (VEC == 4 || x < cols) d[p][r][x] = fmaf(sr, d[p][r][x], tr);
                                ed[p][r] = fmaf(sr, ed[p][r], tr);
                            }
                            lr[p][r].x = __shfl_up_sync(0xffffffffu, d[p][r][3], 4);
                            lr[p][r].y = __shfl_down_sync(0xffffffffu, d[p][r][0], 4);
                            m[p][r][0] = make_float2(d[p][r][0], d[p][r][1]);
                            m[p][r][1] = make_float2(d[p][r][2], d[p][r][3]);
                        }
#pragma unroll
                    for (int p = 0; p < 2; ++p)
#pragma unroll
                        for (int r = 0; r < 6; ++r) {
                            lr[p][r].x = flags & kPrNoLeft ? 0.f : (qg == 0 ? ed[p][r] : lr[p][r].x);
                            lr[p][r].y = flags & kPrNoRight ? 0.f : (qg == 7 ? ed[p][r] : lr[p][r].y);
                        }
                }
                // The stage is handed back once every load of every lane has delivered.  An arrival does not wait for loads that have only been
                // issued, and behind tensor-memory stores those may be hundreds of clocks away from shared memory: the arrival's address
                // depends on a vote over all that they brought (which is always 0).
                const uint32_t none = __any_sync(0xffffffffu, (loaded & prm.zero) != 0u) ? 8u : 0u;
                if (lane == 0) mbar_arrive(xempty_bar(xs) + none);
                xs += 2; if (xs >= prm.nX) xs -= prm.nX;
                xf += 2; if (xf >= 2 * prm.nX) { xf -= 2 * prm.nX; xph ^= 1u; }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    ok = mbar_wait_warp(free_bar(2 * team + h), fph, abort_flag, 0xC00u | (2 * team + h), prm.spin_limit);
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int i = 2 * h; i < 2 * h + 2; ++i) {
#pragma unroll
                        for (int dy = 0; dy < 2; ++dy) {
                            const int y = 2 * dy;
                            float o[16];                             // [j][channel][dx], channels last [j][dx][channel]
                            auto rows = [&](float2 d0, float2 d1, float2 d2, float2 d3) {
                                return i == 0 ? sub2(d0, d2) : i == 1 ? add2(d1, d2) : i == 2 ? sub2(d2, d1) : sub2(d1, d3);
                            };
                            if constexpr (NHWC) {
                                float2 r[6];                         // Winograd row i of the two tiles
#pragma unroll
                                for (int x = 0; x < 6; ++x) r[x] = rows(win[y][x], win[y + 1][x], win[y + 2][x], win[y + 3][x]);
#pragma unroll
                                for (int dx = 0; dx < 2; ++dx) {
                                    const float2 v[4] = {sub2(r[2 * dx], r[2 * dx + 2]), add2(r[2 * dx + 1], r[2 * dx + 2]), sub2(r[2 * dx + 2], r[2 * dx + 1]),
                                                         sub2(r[2 * dx + 1], r[2 * dx + 3])};
#pragma unroll
                                    for (int j = 0; j < 4; ++j) { o[4 * j + 2 * dx] = fmaxf(v[j].x, lo); o[4 * j + 2 * dx + 1] = fmaxf(v[j].y, lo); }
                                }
                            } else {
                                // columns 1 2 | 3 4 | 0 5 of the window
#pragma unroll
                                for (int p = 0; p < 2; ++p) {
                                    const float2 r12 = rows(m[p][y][0], m[p][y + 1][0], m[p][y + 2][0], m[p][y + 3][0]),
                                                 r34 = rows(m[p][y][1], m[p][y + 1][1], m[p][y + 2][1], m[p][y + 3][1]),
                                                 r05 = rows(lr[p][y], lr[p][y + 1], lr[p][y + 2], lr[p][y + 3]);
                                    const float2 d = sub2(r12, r34);
                                    o[2 * p] = fmaxf(r05.x - r12.y, lo); o[2 * p + 1] = fmaxf(d.y, lo);
                                    o[4 + 2 * p] = fmaxf(r12.x + r12.y, lo); o[5 + 2 * p] = fmaxf(r34.x + r34.y, lo);
                                    o[8 + 2 * p] = fmaxf(r12.y - r12.x, lo); o[9 + 2 * p] = fmaxf(r34.y - r34.x, lo);
                                    o[12 + 2 * p] = fmaxf(d.x, lo); o[13 + 2 * p] = fmaxf(r34.x - r05.y, lo);
                                }
                            }
                            if (i == 1) {
                                // Position (1, 1), of non-negative pixels the largest, is rounded to TF32 (half a unit of the last kept
                                // place, then the tensor core's cut), the others are cut: the accumulators take 36 MMAs per 8 channels
                                // instead of 16, whose longer sums cost up to 1.3 % of the error against 64 bits; with this one it is below the former
                                // paths' (64 x 512 x 14 x 14: 4.63e-4 -> 4.52e-4, relative).  All rounded: 2.96e-4, 3 to 18 % slower.
#pragma unroll
                                for (int x = 4; x < 8; ++x)
                                    if (fabsf(o[x]) < __int_as_float(0x7f800000)) o[x] = __uint_as_float(__float_as_uint(o[x]) + 0x1000u);     // (infinities and NaN stay)
                            }
                            const uint32_t to = a_tmem + ((uint32_t)(16 * dy) << 16) + (uint32_t)(32 * i);
                            if (NHWC) tmem_st_16x32_pairs(to, o); else tmem_st_16x32(to, o);
                        }
                    }
                }
                if (!ok) break;
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_peer(full0);
                fph ^= 1u;
                sl += 2;
                if (sl >= nS && n + 2 < total) {
                    do { sl -= nS; ++iu; } while (sl >= nS);
                    enter();
                }
            }
        } else {
            // ------------------------------ epilogue ------------------------------------------
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kPrRegsEpi));
            const int half = (warp - 8) >> 2;                    // which half of the block's output channels
            const uint32_t acce0 = mapa_rank0(acce_bar(0)), acce1 = mapa_rank0(acce_bar(1));
            const long long plane = (long long)prm.H * prm.W;
            // this thread's part of unit iu: rows 4 qr .. of its quad in channels k0, k0 + 4, ... (channels last: k0, k0 + 1, k0 + 8, ...)
            struct Where { long long off; int k0, rows, cols; };
            auto place = [&](int iu) {
                int b, qr, qc;
                const bool valid = locate(iu, b, qr, qc);
                Where w;
                w.k0 = ((pair + iu * npairs) % prm.nKB) * N + half * (N / 2) + (NHWC ? 2 * cl : cl);
                w.cols = prm.W - 4 * qc;
                w.rows = valid ? prm.H - 4 * qr : 0;
                w.off = NHWC ? (((long long)b * prm.H + 4 * qr) * prm.W + 4 * qc) * prm.K + w.k0
                             : ((long long)b * prm.K + w.k0) * plane + (long long)(4 * qr) * prm.W + 4 * qc;
                return w;
            };
            auto store = [&](const Where &w, int y, const float (&v)[2][N / 4]) {       // row y of the quad, v as [e][channel, dx]
                if constexpr (NHWC) {
                    float *yp = prm.Y + w.off + (long long)y * prm.W * prm.K;
#pragma unroll
                    for (int x = 0; x < 4; ++x, yp += prm.K)
#pragma unroll
                        for (int j = 0; j < N / 16; ++j)
                            pr_stg2(yp + 8 * j, v[x & 1][4 * j + (x & 2)], v[x & 1][4 * j + (x & 2) + 1], y < w.rows && w.k0 + 8 * j < prm.K);
                    return;
                }
                float *yp = prm.Y + w.off + (long long)y * prm.W;
#pragma unroll
                for (int c = 0; c < N / 8; ++c, yp += 4 * plane)
                    pr_stg<NHWC ? 1 : VEC>(yp, v[0][2 * c], v[1][2 * c], v[0][2 * c + 1], v[1][2 * c + 1], w.cols, y < w.rows && w.k0 + 4 * c < prm.K);
            };
            auto add = [&](const Where &w, int y, const float (&v)[2][N / 4]) {         // the same, added to what is there
                float *yp = prm.Y + w.off + (long long)y * prm.W;
#pragma unroll
                for (int c = 0; c < N / 8; ++c, yp += 4 * plane)
                    pr_red4(yp, v[0][2 * c], v[1][2 * c], v[0][2 * c + 1], v[1][2 * c + 1], y < w.rows && w.k0 + 4 * c < prm.K);
            };
            const uint32_t t_half = tmem_base + ((uint32_t)(sub * 32) << 16) + (uint32_t)(half * (N / 2));
            // v[e] of rows dy of output row a
            auto fetch = [&](int a, int dy, float (&v)[2][N / 4]) {
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint32_t from = t_half + ((uint32_t)(16 * dy) << 16) + (uint32_t)((2 * a + e) * N);
                    if (NHWC) tmem_ld_16x32_pairs(from, v[e]); else tmem_ld_16x32(from, v[e]);
                }
            };
            auto hand_back = [&](int a) {                        // the accumulators of output row a are in registers
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_peer(a == 0 ? acce0 : acce1);
            };
            // the shortcut's row y, as v
            auto shortcut = [&](const Where &w, int y, float (&r)[2][N / 4]) {
                if constexpr (NHWC) {
                    const float *rp = prm.residual + w.off + (long long)y * prm.W * prm.K;
#pragma unroll
                    for (int x = 0; x < 4; ++x, rp += prm.K)
#pragma unroll
                        for (int j = 0; j < N / 16; ++j)
                            pr_ldg2(r[x & 1][4 * j + (x & 2)], r[x & 1][4 * j + (x & 2) + 1], rp + 8 * j, y < w.rows && w.k0 + 8 * j < prm.K);
                    return;
                }
                const float *rp = prm.residual + w.off + (long long)y * prm.W;
#pragma unroll
                for (int c = 0; c < N / 8; ++c, rp += 4 * plane) {
                    float t[4];
                    pr_ldg<NHWC ? 1 : VEC>(t, rp, w.cols, y < w.rows && w.k0 + 4 * c < prm.K);
                    r[0][2 * c] = t[0]; r[1][2 * c] = t[1]; r[0][2 * c + 1] = t[2]; r[1][2 * c + 1] = t[3];
                }
            };
            bool ok = true;
            if (EXTRAS && (VEC < 4 || prm.front)) {
                // The shortcut in narrow pieces, or with one unit per pair: added in front of the stores (8- and 4-byte reductions behind them
                // take longer than its latency, 103 against 90 us for 128 x 256 x 14 x 14, and with no unit to follow nothing hides them,
                // 29.2 against 26.0 for 16 x 96 x 40 x 36), also where Y lies over it.  A row's loads go out when the row before has
                // been added, the first row's of a unit while that unit is still being multiplied, and the others into L2 by then.
                float r[2][N / 4], scale = 1.f, shift = 0.f;
                Where w = my_units > 0 ? place(0) : Where{};
                // lane l: the affine map of the half's channel l (N / 2 of them)
                auto maps = [&]() {
                    const int k = w.k0 - (NHWC ? 2 * cl : cl) + lane;
                    if (prm.out_scale && lane < N / 2 && k < prm.K) { scale = __ldg(prm.out_scale + k); shift = __ldg(prm.out_shift + k); }
                };
                auto ahead = [&]() {
                    shortcut(w, 0, r);
#pragma unroll 1
                    for (int y = 1; y < 4; ++y) {
                        const float *rp = prm.residual + w.off + (long long)y * prm.W * (NHWC ? prm.K : 1);
#pragma unroll
                        for (int c = 0; c < (NHWC ? 4 : N / 8); ++c, rp += NHWC ? prm.K : 4 * plane)       // (channels last: a pixel's half is one line)
                            if (y < w.rows && w.k0 + (NHWC ? 0 : 4 * c) < prm.K) asm volatile("prefetch.global.L2 [%0];" ::"l"(rp));
                    }
                };
                if (my_units > 0) maps();
                if (prm.residual && my_units > 0) ahead();
                for (int iu = 0; iu < my_units && ok; ++iu) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int a = i >> 1, dy = i & 1;
                        if (dy == 0) {
                            if (!mbar_wait_warp(accf_bar(a), (uint32_t)iu & 1u, abort_flag, 0x400u | (warp << 4) | a, prm.spin_limit)) { ok = false; break; }
                            tc_fence_after();
                        }
                        float v[2][N / 4];
                        fetch(a, dy, v);
                        tmem_ld_wait();
                        if (dy == 1) hand_back(a);
#pragma unroll
                        for (int c = 0; c < N / 8; ++c) {            // the c-th channel of this thread: two values per e
                            const int at = NHWC ? 4 * (c >> 1) + (c & 1) : 2 * c, step = NHWC ? 2 : 1, ch = NHWC ? 8 * (c >> 1) + 2 * cl + (c & 1) : 4 * c + cl;
                            if (prm.out_scale) {
                                const float s1 = __shfl_sync(0xffffffffu, scale, ch), b1 = __shfl_sync(0xffffffffu, shift, ch);
#pragma unroll
                                for (int x = 0; x < 4; ++x) v[x & 1][at + step * (x >> 1)] = fmaf(v[x & 1][at + step * (x >> 1)], s1, b1);
                            }
                            if (prm.residual) {
#pragma unroll
                                for (int x = 0; x < 4; ++x)
                                    v[x & 1][at + step * (x >> 1)] += prm.res_relu ? relu_nan(r[x & 1][at + step * (x >> 1)]) : r[x & 1][at + step * (x >> 1)];
                            }
                        }
                        const Where here = w;
                        if (i == 3 && iu + 1 < my_units) { w = place(iu + 1); maps(); }
                        if (prm.residual) {
                            if (i < 3) shortcut(w, 2 * ((i + 1) & 1) + ((i + 1) >> 1), r);
                            else if (iu + 1 < my_units) ahead();
                        }
                        store(here, 2 * dy + a, v);
                    }
                }
            } else {
                for (int iu = 0; iu < my_units && ok; ++iu) {
                    const Where w = place(iu);
                    float scale = 1.f, shift = 0.f;                  // lane l: the affine map of the half's channel l (N / 2 of them)
                    if (EXTRAS) {
                        const int k = w.k0 - cl + lane;
                        if (prm.out_scale && lane < N / 2 && k < prm.K) { scale = __ldg(prm.out_scale + k); shift = __ldg(prm.out_shift + k); }
                        if (prm.residual) {                          // into L2 while the unit is being multiplied
#pragma unroll 1
                            for (int y = 0; y < 4; ++y) {
                                const float *rp = prm.residual + w.off + (long long)y * prm.W;
#pragma unroll
                                for (int c = 0; c < N / 8; ++c, rp += 4 * plane)
                                    if (y < w.rows && w.k0 + 4 * c < prm.K) asm volatile("prefetch.global.L2 [%0];" ::"l"(rp));
                            }
                        }
                    }
#pragma unroll
                    for (int a = 0; a < 2; ++a) {
                        if (!mbar_wait_warp(accf_bar(a), (uint32_t)iu & 1u, abort_flag, 0x400u | (warp << 4) | a, prm.spin_limit)) { ok = false; break; }
                        tc_fence_after();
                        float v[2][2][N / 4];                        // [dy][e][channel, dx]
                        fetch(a, 0, v[0]); fetch(a, 1, v[1]);
                        tmem_ld_wait();
                        hand_back(a);
                        if (EXTRAS && prm.out_scale) {
#pragma unroll
                            for (int c = 0; c < N / 8; ++c) {
                                const float s1 = __shfl_sync(0xffffffffu, scale, 4 * c + cl), b1 = __shfl_sync(0xffffffffu, shift, 4 * c + cl);
#pragma unroll
                                for (int x = 0; x < 8; ++x) v[x >> 2][(x >> 1) & 1][2 * c + (x & 1)] = fmaf(v[x >> 2][(x >> 1) & 1][2 * c + (x & 1)], s1, b1);
                            }
                        }
                        if (EXTRAS && prm.in_place) { add(w, a, v[0]); add(w, 2 + a, v[1]); }
                        else { store(w, a, v[0]); store(w, 2 + a, v[1]); }
                    }
                    // The shortcut is added to what was just stored, in L2, while the next unit is being multiplied: its latency, in front of
                    // the stores, would hold the accumulators back.
                    if (EXTRAS && prm.residual && ok) {
                        float r[2][2][N / 4];
                        shortcut(w, 0, r[0]);
#pragma unroll
                        for (int y = 0; y < 4; ++y) {
                            if (y < 3) shortcut(w, y + 1, r[(y + 1) & 1]);
                            if (prm.res_relu) {
#pragma unroll
                                for (int x = 0; x < N / 2; ++x) r[y & 1][x & 1][x >> 1] = relu_nan(r[y & 1][x & 1][x >> 1]);
                            }
                            add(w, y, r[y & 1]);
                        }
                    }
                }
            }
        }
    }

    // Neither CTA may leave (or free its tensor memory) while the other can still read its memories through an MMA or
    // signal one of its barriers
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 5) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// Shared memory: the pixels of eight channels of 32 quads, wherever these begin, per stage; three stages if a unit's weights then
// still stay resident (or the ring of those has four), else two; the rest for weights.
static bool pr_geometry(PrParams &p, int layout)
{
    constexpr int wstage = kPrStageBytes;
    // quad rows that 32 quads can touch
    const int qrows = kPrQuads % p.nQW == 0 ? kPrQuads / p.nQW : (kPrQuads - 2) / p.nQW + 2;
    const long long per_image = (long long)p.nQH * p.nQW, HW = (long long)p.H * p.W;
    if (HW * 32 > 0x7fffffffLL) return false;
    const int images = per_image >= kPrQuads ? (per_image % kPrQuads ? 2 : 1) : kPrQuads % per_image == 0 ? (int)(kPrQuads / per_image) : (int)((kPrQuads - 2) / per_image) + 2;
    long long floats;
    p.whole = images * 8 > 32;
    if (layout == WG2X2_NHWC) {                                   // a box per quad row
        if (p.W % 4 || p.K % 4 || p.nQW + 2 > 256) return false;
        p.xpitch = 6 * 4 * (p.nQW + 2) * 32;
        p.xpart = p.whole = 0;
        floats = (long long)qrows * (p.xpitch / 4);
    } else if (p.whole) {
        p.xpitch = (int)HW; p.xpart = (int)(8 * HW);
        floats = (long long)images * p.xpart + 4;
    } else {
        // four rows of pixels per quad row, and one above and one below (none where an image ends)
        p.xpart = pr_room((int)HW);
        const long long rows = std::min<long long>(4LL * qrows + 2, (long long)images * p.H);
        long long pitch = rows * p.W + 8LL * images;
        pitch = (pitch + 23) / 32 * 32 + 8;                       // eight banks apart: four channels of a quad side by side
        p.xpitch = (int)pitch;
        floats = 8 * pitch;
    }
    const long long bytes = (floats * 4 + 127) / 128 * 128;
    if (bytes > (kPrSmemMax - 2 * wstage) / 2) return false;
    p.xbytes = (int)bytes;
    const int nW2 = (p.nS + 1) / 2;
    p.nX = 3;
    p.nW = (int)((kPrSmemMax - 3 * bytes) / wstage);
    if (p.nW < 4 && p.nW < nW2) { p.nX = 2; p.nW = (int)((kPrSmemMax - 2 * bytes) / wstage); }
    if (p.nW > kPrMaxW) p.nW = kPrMaxW;
    if (p.nW > nW2 && p.nKB == 1) p.nW = nW2;
    return p.nW >= 2 || p.nW == nW2;
}

// Sizes of the kernel for a layer; false: not one that it takes
static bool pr_sizes(PrParams &p, int B, int H, int W, int C, int K, int layout)
{
    if (!tc_shape_supported(C, K)) return false;
    p.B = B; p.H = H; p.W = W; p.C = C; p.K = K;
    p.nQH = cdiv(H, 4); p.nQW = cdiv(W, 4);
    const long long quads = (long long)B * p.nQH * p.nQW;
    p.nKB = cdiv(K, kPrN); p.nS = cdiv(C, 8);
    const long long units = cdivll(quads, 2 * kPrQuads) * p.nKB;
    if (quads > 0x7fffffffLL - 2 * kPrQuads || units * p.nS > 0x7fffffffLL) return false;
    p.quads = (int)quads; p.units = (int)units;
    return pr_geometry(p, layout);
}
int layer_fwd_pair(const float *X, const void *prepared, float *Y, int B, int H, int W, int C, int K, int layout, int relu,
                   const float *in_scale, const float *in_shift, const float *out_scale, const float *out_shift,
                   const float *residual, int res_relu, cudaStream_t st)
{
    if (!X || !prepared || !Y) return WG2X2_ERR_BAD_ARG;
    if ((in_scale == nullptr) != (in_shift == nullptr) || (out_scale == nullptr) != (out_shift == nullptr)) return WG2X2_ERR_BAD_ARG;
    if (misaligned16(X) || misaligned16(prepared) || misaligned16(Y) || misaligned16(residual)) return WG2X2_ERR_BAD_ARG;
    PrParams p;
    if (!pr_sizes(p, B, H, W, C, K, layout)) return WG2X2_ERR_UNSUPPORTED;
    p.X = X; p.Y = Y;
    p.in_scale = in_scale; p.in_shift = in_shift; p.out_scale = out_scale; p.out_shift = out_shift; p.residual = residual;
    p.masks = reinterpret_cast<const unsigned long long *>(static_cast<const unsigned char *>(prepared) + align_up((size_t)16 * K * C * sizeof(float), 256));
    p.relu = relu; p.res_relu = res_relu;
    // Y over the shortcut: a thread adds its elements to those there
    p.front = p.units <= kNumSMs / 2;
    p.in_place = layout == WG2X2_NCHW && W % 4 == 0 && !p.front && residual == Y;      // (a NULL Y was refused)
    if (p.in_place) {
        if (res_relu) {
            const long long n4 = (long long)B * K * H * W / 4;
            const int s = launch(relu_copy_kernel, dim3((unsigned)std::min(cdivll(n4, 256), 32LL * kNumSMs)), 256, 0, st, residual, Y, n4);
            if (s != WG2X2_OK) return s;
        }
        p.residual = nullptr;
    }
    p.zero = 0;
    p.spin_limit = wait_limit();
    p.drop_load = take_drop_load();
    CUtensorMap mapW;
    {
        const cuuint64_t dims[3] = {(cuuint64_t)C, (cuuint64_t)K, 16};
        const cuuint64_t strides[2] = {(cuuint64_t)C * 4, (cuuint64_t)K * C * 4};
        const cuuint32_t box[3] = {16, kPrN / 2, 16};
        if (!tensor_map_f32(&mapW, 3, static_cast<const float *>(prepared), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B)) return WG2X2_ERR_LAUNCH;
    }
    CUtensorMap mapX = mapW;                                      // (NCHW: not looked at)
    if (layout == WG2X2_NHWC) {
        // a row of the image as [column of a quad][quad][channel]
        const cuuint64_t px = (cuuint64_t)C * 4;
        const cuuint64_t dims[5] = {(cuuint64_t)C, (cuuint64_t)p.nQW, 4, (cuuint64_t)H, (cuuint64_t)B};
        const cuuint64_t strides[4] = {4 * px, px, px * W, px * W * H};
        const cuuint32_t box[5] = {8, (cuuint32_t)(p.nQW + 2), 4, 6, 1};
        if (!tensor_map_f32(&mapX, 5, X, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE)) return WG2X2_ERR_LAUNCH;
    }
    // a grid that divides the units evenly: every pair runs the same number of them, or one fewer
    const int pairs = cdiv(p.units, cdiv(p.units, kNumSMs / 2));
    const bool extras = out_scale || residual, affine = in_scale != nullptr;
    auto pick = [&](auto v) {
        constexpr int V = decltype(v)::value;
        return extras ? (affine ? layer_fwd_pair_kernel<V, true, true> : layer_fwd_pair_kernel<V, false, true>)
                      : (affine ? layer_fwd_pair_kernel<V, true, false> : layer_fwd_pair_kernel<V, false, false>);
    };
    auto *kernel = layout == WG2X2_NHWC ? pick(std::integral_constant<int, kPrNhwc>{}) : W % 4 == 0 ? pick(std::integral_constant<int, 4>{}) : W % 2 == 0 ? pick(std::integral_constant<int, 2>{}) : pick(std::integral_constant<int, 1>{});
    return launch(kernel, dim3((unsigned)(2 * pairs)), kPrThreads, (size_t)p.nW * kPrStageBytes + (size_t)p.nX * p.xbytes + kCtrlBytes + 1024, st, mapW, mapX, p);
}

// Microseconds of the layer on pairs of SMs (plain, both layouts, 1 .. 256 images of 7 .. 64 pixels, 16 .. 512 channels: within a fifth of
// the measured): rounds of units, each a walk over the input channels and the change of accumulators at its end, which takes
// long where rows are stored pixel by pixel.  (Images that lie whole in shared memory have their channels on the same banks.)
static double pair_us(const PrParams &p, int layout)
{
    const double rounds = cdiv(p.units, kNumSMs / 2);
    return layout == WG2X2_NHWC ? 6.5 + rounds * (1.5 + 0.98 * p.nS) : 6.3 + rounds * ((p.W % 2 ? 9.5 : 3.2) + (p.whole ? 1.05 : 0.82) * p.nS);
}

// The same layer with an affine map in front or a shortcut (0: none, 1: of its own, 2: under Y), against the wide path and the layer on
// clusters with the same.  There the margins of the plain rule are too narrow: a shortcut costs a pair 5 .. 7 us a round and a map 0.04 ..
// 0.16 us a slot, the others 5 .. 12 % (the estimates are within 5 .. 12 % of the measured, one standard deviation).  Of 1272 drawn layers
// that the plain rule takes, 25 were more than 3 % slower than before with map and shortcut, the worst 0.80 of the speed (in another draw 111 x 128 x
// 10 x 10 24.8 -> 34.5 us); with this test 4 of 1206 are, the worst 0.89, and the 66 it turns away are on the mean as fast either way.
static bool options_lose(const PrParams &p, int layout, double clusters, bool wide, bool affine, int shortcut)
{
    const bool nhwc = layout == WG2X2_NHWC, w4 = p.W % 4 == 0, w2 = p.W % 2 == 0;
    const double rounds = cdiv(p.units, kNumSMs / 2);
    const double slot = nhwc ? 0.93 + (affine ? 0.08 : 0.) : w4 ? 0.83 + (affine ? 0.08 : 0.) : w2 ? 0.86 + (affine ? 0.18 : 0.) : 0.97 + (affine ? 0.15 : 0.);
    const double last = !shortcut ? 0. : nhwc ? 4.9 : w4 ? (shortcut == 2 && rounds > 1. ? 1.2 : 6.8) : w2 ? 6.3 : 4.8;
    const double us = (nhwc ? 6.4 : w2 ? 6.8 : 9.0) + rounds * ((nhwc ? 2.5 : w4 ? 2.4 : w2 ? 3.0 : 5.0) + last + slot * p.nS);
    double other = clusters * (affine ? 1.07 : 1.02) * (shortcut == 2 ? 1.12 : shortcut ? 1.08 : 1.);
    if (wide) {
        const long long P = (long long)p.B * ((p.H + 1) / 2) * ((p.W + 1) / 2);
        double products = 0.;
        gg_pick_cols(P, p.K, p.C, &products);
        const double mb = (4e-6 * p.B * p.H * p.W + 128e-6 * P) * ((double)p.C + p.K);
        other = (nhwc ? 7.1 + 0.108 * mb + 0.68 * products : 9.0 + 0.130 * mb + 0.63 * products) * (p.C % 32 || p.K % 32 ? 1.12 : 1.) *
                (affine && nhwc ? 1.08 : 1.) * (shortcut ? 1.07 : 1.);
    }
    return us >= other;
}

// Against all other paths.  It wins where its units fill the SMs at least once: over 172 NCHW layers of 1 .. 128 images it takes 0.50 ..
// 0.95 of the time in 75 (64 x 256 x 40 x 40 341 -> 170 us, 128 x 256 x 14 x 14 93 -> 68, 64 x 64 x 56 x 56 45 -> 34), with fewer units up
// to four times as long.  Over 3030 layers of both layouts that this rule picks plain the geometric mean is 1.65 times as fast.  The factors
// are the margins that the estimates need: channels last, 0.95 takes 46 x 96 x 192 x 12 x 12 too, 19.9 us (24.9 with a
// shortcut) against 18.7 (19.7), and nothing else that 0.85 leaves.  A layer of fewer than 16 units is a call of a few microseconds, for
// which the estimates themselves (60 ns, asked twice) would count.  shortcut: as above; -1: whatever options the call has.
bool layer_pair_preferred(int B, int H, int W, int C, int K, int layout, bool affine, int shortcut)
{
    PrParams p;
    if (cdivll((long long)B * cdiv(H, 4) * cdiv(W, 4), 2 * kPrQuads) * cdiv(K, 64) < 16 || !pr_sizes(p, B, H, W, C, K, layout)) return false;
    const long long P = (long long)B * ((H + 1) / 2) * ((W + 1) / 2);
    if (P > 0x7fffffffLL - kBlockM) return false;
    const double unpaired = unpaired_us(B, H, W, C, K, layout), clusters = cl_cut(P, C, K).us;
    if (pair_us(p, layout) >= (layout == WG2X2_NHWC ? 0.85 : 0.95) * fmin(unpaired, clusters)) return false;
    double us = 0.;
    const bool few = clusters < 0.97 * unpaired;                  // (layer_cluster_preferred)
    const bool wide = !few && !fused_beats_wide(B, H, W, C, K, layout, &us) && conv_fwd_wide_preferred(P, C, K);
    if (!few && !wide) return true;
    for (int a = 0; a < 2; ++a)
        for (int s = 0; s < 3; ++s)
            if ((a || s) && (shortcut < 0 || (affine == (a != 0) && shortcut == s)) && options_lose(p, layout, clusters, wide, a != 0, s)) return false;
    return true;
}
