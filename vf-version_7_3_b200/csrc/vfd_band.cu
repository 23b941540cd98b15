// vfd_band.cu -- axis pass as a banded matrix product on the 5th-generation
// tensor cores, and the set-up of the operators it applies (vfd_band.h).
//
// A tile is 128 lines over their whole length.  A line is cut into blocks of
// 64 outputs; block b of B^m needs the K = 64 + 2H positions from 64 b - H on:
//     D[128 lines x 64 outputs] = U[128 x K] * W_b[K x 64].
// Input block k holds positions 64 k - H .. 64 k + 63 - H, so block b's window
// starts with input block b.  U stays in tensor memory, where line = lane: a
// position is read from HBM once, split into three bf16 parts (8 + 8 + 8
// bits: the whole FP32 significand) and stored in a ring of four input
// blocks; the parts w0, w1, w2 of W_b come from shared memory.  Six
// tensor-core products of FP32 accumulation a k-step -- x_i w_j for i + j <= 2,
// the five small ones of every k-step first -- give the FP32 product.  The
// tensor cores truncate when they accumulate, so values are taken relative to
// an offset, whose own product (offset times a row sum of B^m) is added in
// FP32: what is truncated is then small and of either sign.  The offset of a
// line is that of its input block, the block's mean: the mean is the value
// that leaves least (its sum of squares is never above that of the values
// themselves), and what a block holds cannot cost bits in blocks that do not
// see it.  One offset for the whole line did: a voxel of 1 in the middle of a
// line of zeros left 2e-5 of the result's L2 and 8e-5 of its sum (ten substeps,
// sigma 2.6), a plume residues over all of its lines.  Relative L2 against
// FP64, one substep of positive values: 1.1e-7 without offsets, 3.7e-8 with
// them, the FFT passes 1e-7; ten substeps, sigma 2.6: 3.6e-8 and 1.2e-6; the
// voxel of 1: 9.7e-8 and 1.3e-6.  The third part of a value below 2^-110 (8e-34)
// underflows: such values are rounded to 2^-133 (1e-40) instead of 2^-149.
//
// In place: outputs of block b are stored once its product is complete; all
// input blocks that hold those positions are in tensor memory by then, and
// blocks still to be read start at 64 (b + 2) - H or later.
//
// Roles (one CTA per SM, persistent): warps 0..7 read the accumulators back
// and store the outputs, warps 8..15 convert input blocks and store them to
// tensor memory, warps 16..19 copy input blocks to shared memory (bulk tensor
// copies, or cp.async where the layout does not allow them; nstage blocks
// deep), warps 20 and 21 issue the products of even and of odd blocks, warp 22
// fetches weight images (bulk copies).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#include "vfd_band.h"
#include "vfd_internal.h"
#include "vfd_tma.h"

namespace vfd {

namespace {

constexpr int BD_EPI_WARPS = 8, BD_CONV_WARPS = 8, BD_COPY_WARPS = 4;
constexpr int BD_CONV0 = BD_EPI_WARPS, BD_COPY0 = BD_CONV0 + BD_CONV_WARPS, BD_ISSUE = BD_COPY0 + BD_COPY_WARPS,
              BD_FETCH = BD_ISSUE + 2, BD_WARPS = 24;  // one warp idle: whole warpgroups
constexpr int BD_THREADS = 32 * BD_WARPS;
constexpr int BD_RING = 4;           // input blocks in tensor memory
constexpr int BD_PART_COLS = 32;     // 64 positions of one bf16 part
constexpr int BD_PART_RING = BD_RING * BD_PART_COLS;  // a part's ring: 16 k-steps of 8 columns
constexpr int BD_ACC_COL = 3 * BD_PART_RING;          // two accumulators of 64 columns, used in turn
constexpr int BD_HALF_BYTES = BD_STEP_BYTES / 2;      // 8 positions of a k-step: 64 outputs of each part
constexpr int BD_STAGE_BYTES = BD_LINES * BD_BLK * 4;
constexpr int BD_XOUT_BYTES = BD_EPI_WARPS * 32 * 16 * 4;
constexpr int BD_OFFS = 8;           // input blocks' offsets kept: the loaders are ahead of the epilogue by 7 at most
constexpr int BD_MAXSTAGE = 4, BD_MAXSLOT = 4;
constexpr size_t BD_SMEM_MAX = 213 * 1024;  // beside BandShared
constexpr size_t BD_SMEM_MIN = 120 * 1024;  // one CTA per SM: each takes all of tensor memory

// D FP32, A and B bf16, both K-major, M 128, N 64
constexpr uint32_t BD_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((BD_BLK / 8u) << 17) | ((BD_LINES / 16u) << 24);

struct BandShared {
    BandJob job[BD_WARPS];        // each warp's current job: most of L1 is shared memory here, global reads miss it
    uint64_t sfull[BD_MAXSTAGE];  // input block copied to its stage
    uint64_t sempty[BD_MAXSTAGE]; // its values read from there
    uint64_t afull[BD_RING];      // input block in tensor memory
    uint64_t aempty[BD_RING];     // its last products complete (an arrival of each issuer)
    uint64_t dfull[2], dempty[2]; // accumulator complete / read back
    uint64_t wfull[2];            // weight image of the next even / odd block landed
    int wslot[2];                 // its slot
    alignas(16) float off[BD_OFFS][BD_LINES];   // each line's offset in an input block
    float half[2][2][BD_LINES];   // sums of a block's halves, in turn
    alignas(16) float fn[BD_CONV_WARPS][2][32];  // a block's functional weights, alpha and lambda
    uint32_t tmem;
    int dead;                     // a wait gave up: nothing waits or stores any more
};

// One try of up to 20 us: the hardware suspends the thread, so that waiting
// warps do not take issue slots from working ones.
__device__ __forceinline__ bool band_try(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}
// Waits for phase `parity`, about 1 s at most; after a wait gave up every
// wait returns at once, so all roles run out their loops (in bounds, storing
// nothing) and the CTA ends.
__device__ __forceinline__ bool band_wait(uint64_t *bar, uint32_t parity, volatile int *dead,
                                          long long limit = kTmaWaitCycles)
{
    if (band_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!band_try(bar, parity)) {
        if (*dead) return false;
        if (clock64() - t0 > limit) {
            *dead = 1;
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp_arrive_noinc(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void cp16(uint32_t dst, const float *src, bool ok)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const float *src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint64_t *bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar))
                 : "memory");
}
// D[tmem d] (+)= A[tmem a] * B[shared descriptor]
__device__ __forceinline__ void tc_mma(uint32_t d, uint32_t a, uint64_t bdesc, uint32_t acc)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.u32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" ::"r"(d),
        "r"(a), "l"(bdesc), "r"(BD_IDESC), "r"(acc)
        : "memory");
}
// 16 columns of this warp's 32 lanes
__device__ __forceinline__ void tc_st16(uint32_t addr, const uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16};\n" ::"r"(addr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory"); }
// t = 32 columns of this warp's 32 lanes, in pairs
__device__ __forceinline__ void tc_ld32(uint32_t addr, float2 (&t)[16])
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr)
        : "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
}

// Shared-memory matrix descriptor of a k-step of an image: outputs x 16
// positions, K-major core matrices (8 outputs x 16 bytes) without swizzle, 128
// bytes between groups of 8 outputs (part 1 follows part 0, part 2 part 1),
// BD_HALF_BYTES between the two halves of the positions.
__device__ __forceinline__ uint64_t band_desc(uint32_t addr)
{
    return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)(BD_HALF_BYTES >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
           (1ull << 46);
}

// Two values as the upper and lower halves of a bf16 pair (b above a).
__device__ __forceinline__ uint32_t pack_bf16(float a, float b)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;\n" : "=r"(r) : "f"(b), "f"(a));
    return r;
}

__device__ __forceinline__ double band_warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// A launch's tiles: tile t belongs to job jobs[tjob[t]].
struct BandTiles {
    const BandJob *jobs;
    const int *tjob;
    int begin, end;
    __device__ __forceinline__ int first() const { return begin + (int)blockIdx.x; }
    // tile t's job, or -1
    __device__ __forceinline__ int job(int t) const { return t < end ? __ldg(tjob + t) : -1; }
    // copies a job to the warp's place in shared memory
    __device__ __forceinline__ void load(int j, BandJob *to, int lane) const
    {
        __syncwarp();
        const int4 *src = reinterpret_cast<const int4 *>(jobs + j);
        if (lane < (int)(sizeof(BandJob) / 16)) reinterpret_cast<int4 *>(to)[lane] = __ldg(src + lane);
        __syncwarp();
    }
};
static_assert(sizeof(BandJob) / 16 <= 32, "one piece a lane");
static_assert(sizeof(BandShared) + BD_SMEM_MAX <= 227 * 1024, "shared memory of a block");

// Byte offset of (line, position) in a stage, as the bulk copies leave it.  x
// pass: two boxes of 32 positions, a row of 128 bytes per line, its 16-byte
// chunks permuted by the line; y / z pass: four boxes of 32 lines, a row of
// 128 bytes per position.  Threads of a warp that read one position of 32
// lines meet no bank conflict.
template <bool XP>
__device__ __forceinline__ int band_at(int line, int pos)
{
    return XP ? (pos >> 5) * (BD_STAGE_BYTES / 2) + line * 128 + ((((pos >> 2) & 7) ^ (line & 7)) << 4) + ((pos & 3) << 2)
              : (line >> 5) * (BD_STAGE_BYTES / 4) + pos * 128 + (line & 31) * 4;
}

// ---------------------------------------------------------------------------
// The pass.  Measured on B200, 512x256x384 x 8 fields: 0.70-0.72 ms a pass for
// ten folded substeps (4.5 TB/s of the 8 bytes a voxel it moves; without its
// products 0.60), so a tick of ten substeps and its deposit takes 2.64 ms back to
// back against 19.0 ms on 30 register-FFT passes of 0.58-0.66 ms.  768x384x576:
// 9.4 against 60 ms.  An accumulator is free for the next block as soon as its
// eight warps have read it (each a quarter of the lines, half of the outputs);
// four warps that worked through the halves in turn held it for 0.71-0.75 ms a
// pass (97x61x45 x 3, ten substeps: 52 -> 47 us a tick).
// What bounds it: HBM, with the products (48 cycles each, two issuing threads
// together), the read-back of the accumulators and the ring of four input
// blocks limiting how far its stages overlap.
// ---------------------------------------------------------------------------
// Copies input blocks to the stages.
template <bool XP>
__device__ __forceinline__ void band_copy(const BandTiles &T, int nstage, unsigned char *stages, BandShared &S)
{
    const int lt = threadIdx.x - 32 * BD_COPY0;  // 0..127
    int st = 0, job = -1, jn = T.job(T.first());
    uint32_t phase = 1;  // a stage's first use waits for nothing
    BandJob &J = S.job[threadIdx.x >> 5];
    for (int t = T.first(); t < T.end; t += gridDim.x) {
        const int j = jn;
        jn = T.job(t + gridDim.x);
        if (j != job) {
            job = j;
            T.load(j, &J, threadIdx.x & 31);
        }
        const int n = J.n, nin = J.nin;
        const bool vec = J.vec;
        const int64_t ps = J.pos_stride;
        const int l0 = (t - J.tile0) * BD_LINES;
        const int rows = J.nlines - l0;  // lines left from this tile on
        const float *src = J.data + (XP ? (int64_t)l0 * n : 0);
        bool lok = false;
        if (!XP && !J.map) {
            const int l = l0 + (vec ? (lt & 31) * 4 : lt);
            lok = l < J.nlines;
            const int o = lok ? l / J.n0 : 0;
            src += lok ? (int64_t)o * J.outer_stride + (l - o * J.n0) : 0;
        }
        constexpr int boxes = XP ? 2 : 4;
        int bx = 0, by = 0;  // y / z pass: the line a lane's box starts at
        if (!XP && J.map) {
            by = (l0 + 32 * (lt & 3)) / J.n0;
            bx = l0 + 32 * (lt & 3) - by * J.n0;
        }
        int p0 = -J.H;
        for (int k = 0; k < nin; ++k, p0 += BD_BLK) {
            // parity 1 of a barrier in its first phase counts as complete
            band_wait(&S.sempty[st], phase, &S.dead);
            const uint32_t dst = smem_u32(stages) + (uint32_t)st * BD_STAGE_BYTES;
            if (J.map) {
                // bulk tensor copies, a box a lane; positions outside the line are
                // filled with zeros
                if (lt < 32 && !S.dead) {
                    if (lt == 0) mbar_arrive_expect_tx(&S.sfull[st], BD_STAGE_BYTES);
                    __syncwarp();
                    if (lt < boxes) {
                        fence_proxy_async_smem();
                        tma_load_3d(stages + (size_t)st * BD_STAGE_BYTES + lt * (BD_STAGE_BYTES / boxes), J.map,
                                    XP ? p0 + 32 * lt : bx, XP ? l0 : p0, XP ? 0 : by, &S.sfull[st]);
                    }
                }
                if (lt > 0) mbar_arrive(&S.sfull[st]);
            } else if (XP) {
                const int c = lt & 63, r0 = lt >> 6, p = p0 + c;
                const int rmax = (p >= 0 && p < n) ? rows : 0;
                const float *q = src + (int64_t)r0 * n + p;
#pragma unroll 4
                for (int i = 0; i < 64; ++i, q += 2 * n) {
                    const int r = r0 + 2 * i;
                    const bool ok = r < rmax;
                    cp4(dst + band_at<true>(r, c), ok ? q : src, ok);
                }
                cp_arrive_noinc(&S.sfull[st]);
            } else {
                const int q0 = vec ? lt >> 5 : 0, p1 = p0 + q0, step = vec ? 4 : 1;
                const int64_t dq = step * ps;
                const float *q = src + p1 * ps;
                const int a = lok ? max(0, -p1) : 1 << 20, z = n - p1;  // positions p1 + i in [0, n)
                if (vec) {
                    const uint32_t d = dst + band_at<false>((lt & 31) * 4, q0);
#pragma unroll 4
                    for (int i = 0; i < 16; ++i, q += dq) {
                        const bool ok = 4 * i >= a && 4 * i < z;
                        cp16(d + i * 512, ok ? q : src, ok);
                    }
                } else {
                    const uint32_t d = dst + band_at<false>(lt, 0);
#pragma unroll 4
                    for (int i = 0; i < BD_BLK; ++i, q += dq) {
                        const bool ok = i >= a && i < z;
                        cp4(d + i * 128, ok ? q : src, ok);
                    }
                }
                cp_arrive_noinc(&S.sfull[st]);
            }
            if (++st == nstage) {
                st = 0;
                phase ^= 1;
            }
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    if (S.dead) {
        // after a wait gave up: time for the bulk copies in flight to land
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000) {}
    }
}

__device__ __forceinline__ float sum32(const float2 (&v)[16])
{
    float2 a[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = __fadd2_rn(v[i], v[i + 8]);
#pragma unroll
    for (int s = 4; s > 0; s >>= 1)
#pragma unroll
        for (int i = 0; i < s; ++i) a[i] = __fadd2_rn(a[i], a[i + s]);
    return a[0].x + a[0].y;
}
// sum of v[i] w[i], FP32 within groups of 8, FP64 across
__device__ __forceinline__ double dot32(const float2 (&v)[16], const float *w)
{
    double q = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 w0 = reinterpret_cast<const float4 *>(w)[2 * i], w1 = reinterpret_cast<const float4 *>(w)[2 * i + 1];
        const float2 *x = v + 4 * i;
        float2 s = __fmul2_rn(x[0], make_float2(w0.x, w0.y));
        float2 r = __fmul2_rn(x[2], make_float2(w1.x, w1.y));
        s = __ffma2_rn(x[1], make_float2(w0.z, w0.w), s);
        r = __ffma2_rn(x[3], make_float2(w1.z, w1.w), r);
        s = __fadd2_rn(s, r);
        q += (double)(s.x + s.y);
    }
    return q;
}

// Converts input blocks: the padding rule, the accounting's input terms, the
// three bf16 parts of value minus the block's offset, into tensor memory.
template <int AXIS>
__device__ __forceinline__ void band_convert(const BandTiles &T, int sums, int nstage, unsigned char *stages,
                                             BandShared &S, uint32_t tmem)
{
    constexpr bool XP = AXIS == PASS_X;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int quad = warp & 3, half = (warp - BD_CONV0) >> 2;
    const int ln = quad * 32 + lane;  // line of the tile = lane of tensor memory
    int done = 0, st = 0, sphase = 0, job = -1;
    double accP = 0.0, accL = 0.0;
    const BandJob &J = S.job[warp];
    auto flush = [&]() {
        if (!sums || job < 0 || !J.sums) return;
        const double sl = band_warp_sum(accL);
        const double sp = XP ? band_warp_sum(accP) : 0.0;
        if (lane == 0 && !S.dead) {
            if (XP) atomicAdd(J.mass + MS_INPUT, sp);
            if (sl != 0.0) atomicAdd(J.mass + (XP ? MS_LEAK_X : AXIS == PASS_Y ? MS_LEAK_Y : MS_LEAK_Z), sl);
        }
        accP = accL = 0.0;
    };
    int jn = T.job(T.first());
    for (int t = T.first(); t < T.end; t += gridDim.x) {
        const int j = jn;
        jn = T.job(t + gridDim.x);
        if (j != job) {
            flush();
            job = j;
            T.load(j, &S.job[warp], lane);
        }
        const int n = J.n, H = J.H, nin = J.nin;
        const bool mask = XP && J.mask;
        const float b = J.b;
        const int l = (t - J.tile0) * BD_LINES + ln;
        float lw1 = 1.0f, lw2 = 1.0f;  // the line's weights, read long before they are used
        int lo = 0, hi = mask ? 0 : n;  // the positions that count
        const bool acc = sums && J.sums;
        if (l < J.nlines && (mask || acc)) {
            if (XP) {
                const int z = l / J.ny, y = l - z * J.ny;
                if (acc) {
                    lw1 = __ldg(J.lw1 + y);
                    lw2 = __ldg(J.lw2 + z);
                }
                if (mask && y >= J.box_lo[1] && y < J.box_hi[1] && z >= J.box_lo[2] && z < J.box_hi[2]) {
                    lo = J.box_lo[0];
                    hi = J.box_hi[0];
                }
            } else if (AXIS == PASS_Y) {
                lw2 = __ldg(J.lw2 + l / J.n0);
            }
        }
        double tP = 0.0, tL = 0.0;  // the line's sums
        // a block's functional weights, one position a lane, read a block ahead
        const float *fn = J.fn + 32 * half + lane;
        float fa = 0.0f, fl = 0.0f;
        if (acc && !(J.plain & 1ull)) {
            fa = XP ? __ldg(fn) : 0.0f;
            fl = __ldg(fn + BD_BLK * nin);
        }
        for (int k = 0; k < nin; ++k, ++done) {
            const int slot = done % BD_RING;
            band_wait(&S.sfull[st], sphase, &S.dead);
            float2 v[16];  // positions 2 i, 2 i + 1 of this half
            const unsigned char *sp = stages + (size_t)st * BD_STAGE_BYTES;
            if (XP) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 q = *reinterpret_cast<const float4 *>(sp + band_at<true>(ln, 4 * (half * 8 + c)));
                    v[2 * c] = make_float2(q.x, q.y);
                    v[2 * c + 1] = make_float2(q.z, q.w);
                }
            } else {
                const float *f = reinterpret_cast<const float *>(sp + band_at<false>(ln, half * 32));  // 32 floats apart
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = make_float2(f[2 * i * 32], f[(2 * i + 1) * 32]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.sempty[st]);
            if (++st == nstage) {
                st = 0;
                sphase ^= 1;
            }
            if (mask) {
                const int p0 = BD_BLK * k - H + 32 * half;
                const float2 nb = make_float2(-b, -b);
                if (p0 >= lo && p0 + 32 <= hi) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] = __fadd2_rn(v[i], nb);
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int p = p0 + 2 * i;
                        v[i].x = (p >= lo && p < hi) ? v[i].x - b : 0.0f;
                        v[i].y = (p + 1 >= lo && p + 1 < hi) ? v[i].y - b : 0.0f;
                    }
                }
            }
            const float vs = sum32(v);
            S.half[done & 1][half][ln] = vs;
            if (acc) {
                if ((J.plain >> k) & 1ull) {
                    if (XP) tP += (double)(vs * J.fscale);
                } else {
                    float(*f)[32] = S.fn[warp - BD_CONV0];
                    __syncwarp();
                    if (XP) f[0][lane] = fa;
                    f[1][lane] = fl;
                    __syncwarp();
                    if (XP) tP += dot32(v, f[0]);
                    tL += dot32(v, f[1]);
                }
                if (k + 1 < nin && !((J.plain >> (k + 1)) & 1ull)) {
                    fa = XP ? __ldg(fn + BD_BLK * (k + 1)) : 0.0f;
                    fl = __ldg(fn + BD_BLK * (nin + k + 1));
                }
            }
            if (done >= BD_RING) band_wait(&S.aempty[slot], ((done / BD_RING) - 1) & 1, &S.dead);
            tc_fence_after();
            // the block's offset: the mean of its positions that count (those in
            // the line and inside the padding box; the others have weight 0)
            __syncwarp();
            asm volatile("bar.sync %0, 64;\n" ::"r"(1 + quad) : "memory");
            const int count = min(BD_BLK * (k + 1) - H, hi) - max(BD_BLK * k - H, lo);
            float off = count > 0 ? __fdividef(vs + S.half[done & 1][half ^ 1][ln], (float)count) : 0.0f;
            if (!(fabsf(off) < 1e37f)) off = 0.0f;
            if (half == 0) S.off[done % BD_OFFS][ln] = off;
            __syncwarp();
            const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(slot * BD_PART_COLS + half * 16);
            const float2 noff = make_float2(-off, -off), neg = make_float2(-1.0f, -1.0f);
            uint32_t w[16];
#pragma unroll
            for (int part = 0; part < 3; ++part) {
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if (part == 0) v[i] = __fadd2_rn(v[i], noff);
                    w[i] = pack_bf16(v[i].x, v[i].y);
                    if (part < 2)
                        v[i] = __ffma2_rn(make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u)),
                                          neg, v[i]);
                }
                tc_st16(ta + part * BD_PART_RING, w);
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.afull[slot]);
        }
        const double lw = (double)lw1 * (double)lw2;
        if (XP) accP += tP * lw;
        accL += tL * lw;
    }
    flush();
}

// Keeps the weight images in a few slots of shared memory: for each block in
// turn finds its image or fetches it (one thread).
__device__ __forceinline__ void band_fetch(const BandTiles &T, int nslots, int slot_bytes, unsigned char *wsm,
                                           BandShared &S)
{
    const unsigned char *held[BD_MAXSLOT];  // the image in each slot
#pragma unroll
    for (int q = 0; q < BD_MAXSLOT; ++q) held[q] = nullptr;
    const uint32_t w0 = smem_u32(wsm);
    int i = 0, next = 0, last = -1, job = -1, pending = -1;
    BandJob &J = S.job[BD_FETCH];
    int jn = T.job(T.first());
    for (int t = T.first(); t < T.end; t += gridDim.x) {
        const int j = jn;
        jn = T.job(t + gridDim.x);
        if (j != job) {
            job = j;
            J = T.jobs[j];
        }
        const int bytes = J.ksteps * BD_STEP_BYTES;
        for (int b = 0; b < J.nb; ++b, ++i) {
            // block i - 2's products are complete (and so all earlier ones):
            // every slot but block i - 1's is free, and so is wslot[i & 1]
            if (i >= 2) band_wait(&S.dfull[i & 1], ((i >> 1) - 1) & 1, &S.dead);
            const unsigned char *img = J.img + (size_t)J.image(b) * bytes;
            int s = -1;
#pragma unroll
            for (int q = 0; q < BD_MAXSLOT; ++q)
                if (held[q] == img) s = q;
            const bool load = s < 0;
            if (load) {
                s = next == last ? (next + 1 == nslots ? 0 : next + 1) : next;
                next = s + 1 == nslots ? 0 : s + 1;
#pragma unroll
                for (int q = 0; q < BD_MAXSLOT; ++q)
                    if (q == s) held[q] = img;
            }
            last = s;
            S.wslot[i & 1] = s;
            if (load && !S.dead) {
                // landed before the next block is looked at: it may use the
                // same image, and has a barrier of its own
                pending = i;
                mbar_arrive_expect_tx(&S.wfull[i & 1], (uint32_t)bytes);
                bulk_load(w0 + (uint32_t)s * (uint32_t)slot_bytes, img, (uint32_t)bytes, &S.wfull[i & 1]);
                band_wait(&S.wfull[i & 1], (i >> 1) & 1, &S.dead);
            } else {
                mbar_arrive(&S.wfull[i & 1]);
            }
        }
    }
    // if a wait gave up, the last fetch may still be in flight
    if (S.dead && pending >= 0) {
        const long long t0 = clock64();
        while (!mbar_try_wait(&S.wfull[pending & 1], (pending >> 1) & 1))
            if (clock64() - t0 > kTmaWaitCycles) break;
    }
}

// Issues the products of every other block (par: even or odd) into
// accumulator par (one thread).
__device__ __forceinline__ void band_issuer(const BandTiles &T, int par, int slot_bytes, unsigned char *wsm,
                                            BandShared &S, uint32_t tmem)
{
    const uint32_t w0 = smem_u32(wsm), d = tmem + BD_ACC_COL + par * BD_BLK;
    int i = 0, mine = 0, abase = 0, awaited = 0, job = -1;
    BandJob &J = S.job[BD_ISSUE + par];
    int jn = T.job(T.first());
    for (int t = T.first(); t < T.end; t += gridDim.x) {
        const int j = jn;
        jn = T.job(t + gridDim.x);
        if (j != job) {
            job = j;
            J = T.jobs[j];
        }
        const int n = J.n, H = J.H, ks = J.ksteps, nb = J.nb, nin = J.nin;
        const int nwb = (ks + 3) >> 2;  // input blocks of a window
        int freed = 0;                  // input blocks of the tile this thread has let go
        for (int b = (i ^ par) & 1; b < nb; b += 2, ++mine) {
            band_wait(&S.wfull[par], mine & 1, &S.dead);
            const int need = abase + min(b + nwb, nin);
            for (; awaited < need; ++awaited)
                band_wait(&S.afull[awaited % BD_RING], (awaited / BD_RING) & 1, &S.dead);
            if (mine >= 1) band_wait(&S.dempty[par], (mine - 1) & 1, &S.dead);
            tc_fence_after();
            // k-steps that hold positions of the line
            const int p0 = BD_BLK * b - H;
            const int s0 = p0 < 0 ? (-p0) >> 4 : 0;
            const int s1 = min(ks, (n - p0 + 15) >> 4);
            const uint32_t col0 = (uint32_t)((abase + b) % BD_RING) * BD_PART_COLS + s0 * 8;
            const uint64_t desc0 =
                band_desc(w0 + (uint32_t)S.wslot[par] * (uint32_t)slot_bytes + (uint32_t)s0 * BD_STEP_BYTES);
            constexpr int WP = BD_HALF_BYTES / 3 / 16;  // from one part of an image to the next
            // The five small products first, then the large one, so that each of
            // the latter's sums is truncated once a k-step.  A product takes 45
            // cycles; this loop issues one in 58, a loop of one in 90, and
            // unrolled over the k-steps the code outgrows the instruction cache
            // (130): hence two issuing threads (one product in 48 cycles together).
            uint32_t col = col0;
            uint64_t desc = desc0;
#pragma unroll 1
            for (int q = s0; q < s1; ++q) {
                const uint32_t a = tmem + col % BD_PART_RING;
                tc_mma(d, a + BD_PART_RING, desc + WP, q > s0);
                tc_mma(d, a, desc + 2 * WP, 1);
                tc_mma(d, a + 2 * BD_PART_RING, desc, 1);
                tc_mma(d, a, desc + WP, 1);
                tc_mma(d, a + BD_PART_RING, desc, 1);
                desc += BD_STEP_BYTES / 16;
                col += 8;
            }
            col = col0;
            desc = desc0;
            int q = s0;
#pragma unroll 1
            for (; q + 3 <= s1; q += 3) {
                tc_mma(d, tmem + col % BD_PART_RING, desc, 1);
                tc_mma(d, tmem + (col + 8) % BD_PART_RING, desc + BD_STEP_BYTES / 16, 1);
                tc_mma(d, tmem + (col + 16) % BD_PART_RING, desc + 2 * (BD_STEP_BYTES / 16), 1);
                desc += 3 * (BD_STEP_BYTES / 16);
                col += 24;
            }
            if (q < s1) tc_mma(d, tmem + col % BD_PART_RING, desc, 1);
            if (q + 1 < s1) tc_mma(d, tmem + (col + 8) % BD_PART_RING, desc + BD_STEP_BYTES / 16, 1);
            tc_commit(&S.dfull[par]);
            // Input blocks this thread needs no more (its next block of the tile
            // starts at input block b + 2).  An arrival for an input block
            // follows the wait for it, so that it cannot fall into the phase of
            // the block that had its place before.
            for (const int k1 = b + 2 < nb ? b + 2 : nin; freed < k1; ++freed) {
                for (; awaited <= abase + freed; ++awaited)
                    band_wait(&S.afull[awaited % BD_RING], (awaited / BD_RING) & 1, &S.dead);
                tc_commit(&S.aempty[(abase + freed) % BD_RING]);
            }
        }
        // a tile without a block of this thread
        for (; freed < nin; ++freed) {
            for (; awaited <= abase + freed; ++awaited)
                band_wait(&S.afull[awaited % BD_RING], (awaited / BD_RING) & 1, &S.dead);
            mbar_arrive(&S.aempty[(abase + freed) % BD_RING]);
        }
        i += nb;
        abase += nin;
    }
    // what is in flight lands before the CTA ends
    if (mine >= 1) band_wait(&S.dfull[par], (mine - 1) & 1, &S.dead);
}

// Stores the outputs: 32 positions of a block, of the warp's 32 lines.
template <int AXIS>
__device__ __forceinline__ void band_epilogue(const BandTiles &T, int sums, unsigned char *xout, BandShared &S,
                                              uint32_t tmem)
{
    constexpr bool XP = AXIS == PASS_X, zl = AXIS == PASS_Z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the lines and the half of every block's outputs this warp reads: all warps
    // have read an accumulator before they work on its values
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t ta = tmem + ((uint32_t)(quad * 32) << 16) + BD_ACC_COL + 32 * half;
    int i = 0, job = -1;
    double acc_ot = 0.0, acc_ct = 0.0;  // of the values stored, and (where there is a baseline) before it is added
    const BandJob &J = S.job[warp];
    auto flush = [&]() {
        if (!zl || !sums || job < 0 || !J.sums) return;
        const double so = band_warp_sum(acc_ot), sc = J.b != 0.0f ? band_warp_sum(acc_ct) : so;
        if (lane == 0 && !S.dead) {
            atomicAdd(J.mass + MS_CONV, sc / (double)J.keep);
            atomicAdd(J.mass + MS_OUT, so);
        }
        acc_ot = acc_ct = 0.0;
    };
    int ein = 0;  // input blocks of the tiles before
    int jn = T.job(T.first());
    for (int t_ = T.first(); t_ < T.end; t_ += gridDim.x) {
        const int j = jn;
        jn = T.job(t_ + gridDim.x);
        if (j != job) {
            flush();
            job = j;
            T.load(j, &S.job[warp], lane);
        }
        // (what is read from the job where it is used need not stay in a register)
        const int n = J.n;
        const int l0 = (t_ - J.tile0) * BD_LINES + quad * 32, l = l0 + lane;
        const bool lok = l < J.nlines;
        float *dst = J.data;
        if (!XP) {
            const int o = lok ? l / J.n0 : 0;
            dst += lok ? (int64_t)o * J.outer_stride + (l - o * J.n0) : 0;
        }
        for (int b = 0; b < J.nb; ++b, ++i) {
            const int par = i & 1;
            band_wait(&S.dfull[par], (i >> 1) & 1, &S.dead);
            tc_fence_after();
            const bool live = !*(volatile int *)&S.dead;
            // the offsets of the window's blocks (two, or three where it spans as
            // many): the last one's, the steps to it from the first (d0) and from
            // the second (d1)
            const bool three = J.ksteps > 2 * BD_BLK / 16;
            auto offset = [&](int k) { return S.off[(ein + min(k, J.nin - 1)) % BD_OFFS][quad * 32 + lane]; };
            float off = offset(b + 1), d1 = 0.0f;
            const float d0 = offset(b) - off;
            if (three) {
                const float last = offset(b + 2);
                d1 = off - last;
                off = last;
            }
            float2 t[16];  // positions 2 c, 2 c + 1 of this half
            __syncwarp();
            tc_ld32(ta + par * BD_BLK, t);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.dempty[par]);
            // the offsets' share: the weights' sums over the window's first
            // block, its first two and all of it
            const float4 *rho = reinterpret_cast<const float4 *>(J.rho + J.image(b) * (3 * BD_BLK) + 32 * half);
            auto add = [&](float d, const float4 *r) {
                const float2 d2 = make_float2(d, d);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 q = __ldg(r + c);
                    t[2 * c] = __ffma2_rn(d2, make_float2(q.x, q.y), t[2 * c]);
                    t[2 * c + 1] = __ffma2_rn(d2, make_float2(q.z, q.w), t[2 * c + 1]);
                }
            };
            add(d0, rho);
            if (three) add(d1, rho + BD_BLK / 4);
            const bool inner = b >= J.b0 && b < J.b1;  // the sums over all of a window are all the same
            if (!inner) add(off, rho + 2 * (BD_BLK / 4));
            auto shift = [&](float o) {
                const float2 o2 = make_float2(o, o);
#pragma unroll
                for (int c = 0; c < 16; ++c) t[c] = __fadd2_rn(t[c], o2);
            };
            if (inner) shift(off * J.fscale);
            const int p0 = BD_BLK * b + 32 * half;
            if (XP) {
                // 32 rows x 16 positions at a time through shared memory,
                // 64-byte row segments out
                unsigned char *o = xout + warp * 2048;
                const int rmax = live ? J.nlines - l0 : 0;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    __syncwarp();
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<float4 *>(o + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) =
                            make_float4(t[8 * g + 2 * c].x, t[8 * g + 2 * c].y, t[8 * g + 2 * c + 1].x,
                                        t[8 * g + 2 * c + 1].y);
                    __syncwarp();
                    if (J.vec) {
                        const int c = lane & 3, r0 = lane >> 2, p = p0 + 16 * g + 4 * c;
                        const int rm = p < n ? rmax : 0;
                        float *q = dst + (int64_t)(l0 + r0) * n + p;
#pragma unroll
                        for (int e = 0; e < 4; ++e, q += 8 * n) {
                            const int r = 8 * e + r0;
                            const float4 x =
                                *reinterpret_cast<const float4 *>(o + r * 64 + ((c ^ ((r >> 1) & 3)) << 4));
                            if (r < rm) *reinterpret_cast<float4 *>(q) = x;
                        }
                    } else {
                        const int c = lane & 15, r0 = lane >> 4, p = p0 + 16 * g + c;
                        const int rm = p < n ? rmax : 0;
                        float *q = dst + (int64_t)(l0 + r0) * n + p;
#pragma unroll 8
                        for (int e = 0; e < 16; ++e, q += 2 * n) {
                            const int r = 2 * e + r0;
                            const float x = *reinterpret_cast<const float *>(
                                o + r * 64 + (((c >> 2) ^ ((r >> 1) & 3)) << 4) + ((c & 3) << 2));
                            if (r < rm) *q = x;
                        }
                    }
                }
            } else {
                const int naff = zl ? J.naff : 0, ly = naff ? l / J.nx : 0, lx = l - ly * J.nx;
                for (int g = 0; g < naff; ++g) {
                    // the affine rows, decayed like the rest
                    const float q = lok ? J.keep * J.affc[g] * J.aff[0][(int64_t)g * J.affs[0] + lx] *
                                              J.aff[1][(int64_t)g * J.affs[1] + ly]
                                        : 0.0f;
                    const float2 q2 = make_float2(q, q);
                    const float4 *z = reinterpret_cast<const float4 *>(J.aff[2] + (int64_t)g * J.affs[2] + p0);
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float4 zz = __ldg(z + c);
                        t[2 * c] = __ffma2_rn(q2, make_float2(zz.x, zz.y), t[2 * c]);
                        t[2 * c + 1] = __ffma2_rn(q2, make_float2(zz.z, zz.w), t[2 * c + 1]);
                    }
                }
                const int m = lok ? min(32, n - p0) : 0;
                auto sum = [&]() {  // over the line's positions
                    if (m < 32) {
#pragma unroll
                        for (int x = 0; x < 16; ++x) {
                            if (2 * x >= m) t[x].x = 0.0f;
                            if (2 * x + 1 >= m) t[x].y = 0.0f;
                        }
                    }
                    return (double)sum32(t);
                };
                const bool acc = zl && sums && J.sums && m > 0;
                if (zl && J.b != 0.0f) {
                    // out = keep (t + baseline), keep being part of the operator
                    if (acc) acc_ct += sum();
                    shift(J.keep * J.b);
                }
                if (acc) acc_ot += sum();
                const int64_t ps = J.pos_stride;
                float *q = dst + (int64_t)p0 * ps;
                if (m == 32 && live) {
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        q[0] = t[x].x;
                        q[ps] = t[x].y;
                        q += 2 * ps;
                    }
                } else if (live) {
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        if (2 * x < m) q[0] = t[x].x;
                        if (2 * x + 1 < m) q[ps] = t[x].y;
                        q += 2 * ps;
                    }
                }
            }
        }
        ein += J.nin;
    }
    flush();
}

template <int AXIS>
__global__ void __launch_bounds__(BD_THREADS, 1)
    band_kernel(const BandJob *__restrict__ jobs, const int *__restrict__ tjob, int tile_begin, int tile_end,
                int sums, int nstage, int nslots, int slot_bytes)
{
    extern __shared__ unsigned char dyn_[];
    __shared__ __align__(16) BandShared S;
    // the stages at a multiple of 1024 bytes (the copies' permutation)
    unsigned char *wsm = dyn_ + ((1024u - (smem_u32(dyn_) & 1023u)) & 1023u);
    unsigned char *stages = wsm + (size_t)nslots * slot_bytes;
    unsigned char *xout = stages + (size_t)nstage * BD_STAGE_BYTES;
    const int warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        S.dead = 0;
        for (int s = 0; s < BD_MAXSTAGE; ++s) {
            mbar_init(&S.sfull[s], 32 * BD_COPY_WARPS);
            mbar_init(&S.sempty[s], BD_CONV_WARPS);
        }
        for (int s = 0; s < BD_RING; ++s) {
            mbar_init(&S.afull[s], BD_CONV_WARPS);
            mbar_init(&S.aempty[s], 2);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&S.dfull[s], 1);
            mbar_init(&S.dempty[s], BD_EPI_WARPS);
            mbar_init(&S.wfull[s], 1);
        }
        mbar_fence_init();
    }
    if (warp == BD_ISSUE) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(smem_u32(&S.tmem))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem;
    grid_dep_launch();
    // the weights do not depend on the kernel before; the fields do
    if (warp != BD_FETCH) grid_dep_wait();
    const BandTiles T{jobs, tjob, tile_begin, tile_end};
    // registers: 80 a thread at launch; 256 x (104 + 88 + 48) = 768 x 80
    if (warp < BD_CONV0) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;\n");
    } else if (warp < BD_COPY0) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 88;\n");
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 48;\n");
    }
    if (warp < BD_CONV0) {
        band_epilogue<AXIS>(T, sums, xout, S, tmem);
    } else if (warp < BD_COPY0) {
        band_convert<AXIS>(T, sums, nstage, stages, S, tmem);
    } else if (warp < BD_ISSUE) {
        band_copy<AXIS == PASS_X>(T, nstage, stages, S);
    } else if ((threadIdx.x & 31) == 0) {
        if (warp < BD_FETCH) band_issuer(T, warp - BD_ISSUE, slot_bytes, wsm, S, tmem);
        else if (warp == BD_FETCH) band_fetch(T, nslots, slot_bytes, wsm, S);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // every world this CTA had a tile of learns that a wait gave up
    if (S.dead && threadIdx.x == 0)
        for (int t = T.first(); t < T.end; t += gridDim.x) atomicExch(jobs[tjob[t]].gave_up, 1);
    if (warp == BD_ISSUE)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem) : "memory");
}

__global__ void band_wait_probe_kernel(long long limit, int *gave_up)
{
    __shared__ __align__(8) uint64_t bar;
    __shared__ int dead;
    if (threadIdx.x == 0) {
        dead = 0;
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncwarp();
    band_wait(&bar, 0, &dead, limit);
    __syncwarp();
    if (dead && threadIdx.x == 0) atomicExch(gave_up, 1);
}

// ---------------------------------------------------------------------------
// Set-up of the operators.
// ---------------------------------------------------------------------------
constexpr int BD_ROWHW = 160;  // half-width a row of B^m is computed with (what lies beyond is far below 1e-8)

// One warp per row of an image: row i of B^m = (A M)^m in FP64, A the cropped
// convolution, M the interior mask, then its three bf16 parts.
__global__ void __launch_bounds__(128) band_image_kernel(const BandAxis *axes)
{
    __shared__ double buf[4][2][2 * BD_ROWHW + 1];
    const BandAxis &X = axes[blockIdx.y];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * 4 + warp;
    const int im = row / BD_BLK, o = row % BD_BLK;
    if (im >= X.nimg) return;
    const int b = X.blk[im], i = BD_BLK * b + o, n = X.n, r = X.r;
    const int hw = min(X.m * r, BD_ROWHW), wd = 2 * hw + 1;
    double *cur = buf[warp][0], *nxt = buf[warp][1];
    for (int q = lane; q < wd; q += 32) cur[q] = (q == hw && i < n) ? 1.0 : 0.0;
    __syncwarp();
    for (int s = 0; s < X.m; ++s) {
        for (int q = lane; q < wd; q += 32) {
            const int j = i - hw + q;
            double a = 0.0;
            if (j >= X.lo && j < X.hi)
                for (int d = max(-r, q - wd + 1); d <= min(r, q); ++d) a += X.taps[d + r] * cur[q - d];
            nxt[q] = a;
        }
        __syncwarp();
        double *t = cur;
        cur = nxt;
        nxt = t;
    }
    // A weight w at distance j beyond H becomes w j^2 / H^2 at H and its excess
    // over w is taken off the centre: the row keeps its sum and its variance
    // (dropped, the tails of 1e-8 would cost 3e-7 of the variance a step).
    // Half-widths for tails of 1e-8 are 8 % below those for 1e-10: ten substeps
    // of radius 5.1 on average 2.66 -> 2.60 ms, the error against FP64 as before.
    double at_lo = 0.0, at_hi = 0.0, centre = 0.0;
    const double h2 = (double)X.H * X.H;
    for (int q = lane; q < wd; q += 32) {
        const int j = q - hw;
        if (abs(j) <= X.H) continue;
        const double f = cur[q] * ((double)j * j / h2);
        (j < 0 ? at_lo : at_hi) += f;
        centre += cur[q] - f;
    }
    at_lo = band_warp_sum(at_lo);
    at_hi = band_warp_sum(at_hi);
    centre = band_warp_sum(centre);
    if (lane == 0 && hw > X.H) {
        cur[hw - X.H] += at_lo;
        cur[hw + X.H] += at_hi;
        cur[hw] += centre;
    }
    __syncwarp();
    unsigned char *img = X.img + (size_t)im * X.ksteps * BD_STEP_BYTES;
    double sum[3] = {0.0, 0.0, 0.0};  // over the window's first input block, its first two, all of it
    for (int kk = lane; kk < X.ksteps * 16; kk += 32) {
        const int j = BD_BLK * b - X.H + kk, q = j - i + hw;
        double w = 0.0;
        if (j >= 0 && j < n && abs(i - j) <= X.H && q >= 0 && q < wd) w = cur[q] * X.scale;
        for (int k = kk / BD_BLK; k < 3; ++k) sum[k] += w;
        const size_t at = (size_t)(kk >> 4) * BD_STEP_BYTES + ((kk >> 3) & 1) * BD_HALF_BYTES + (o >> 3) * 128 +
                          (o & 7) * 16 + (kk & 7) * 2;
#pragma unroll
        for (int part = 0; part < 3; ++part) {
            const __nv_bfloat16 h = __float2bfloat16_rn((float)w);
            w -= (double)__bfloat162float(h);
            *reinterpret_cast<__nv_bfloat16 *>(img + at + part * (BD_HALF_BYTES / 3)) = h;
        }
    }
    for (int k = 0; k < 3; ++k) {
        const double r = band_warp_sum(sum[k]);
        if (lane == 0) X.rho[(im * 3 + k) * BD_BLK + o] = (float)r;
    }
}

// y(j) = sum_i x(i) g(i - j) over [0, n): A is symmetric
__device__ __forceinline__ double band_conv(const double *x, const double *taps, int r, int n, int j)
{
    double a = 0.0;
    for (int d = max(-r, -j); d <= min(r, n - 1 - j); ++d) a += taps[d + r] * x[j + d];
    return a;
}

// One block per operator: the functional weights alpha = M B^(m-1) and
// lambda = (M (1 - colsum A)) B^(m-1), the affine rows X_j = B^j 1 and their
// sums.
__global__ void __launch_bounds__(256) band_vector_kernel(const BandAxis *axes)
{
    __shared__ double x[2][2048];
    __shared__ double red[8];
    const BandAxis &X = axes[blockIdx.x];
    const int n = X.n, r = X.r, tid = threadIdx.x;
    auto masked = [&](int j) { return j >= X.lo && j < X.hi; };
    auto leak0 = [&](int j) {  // mass of position j's kernel outside [0, n)
        double a = 0.0;
        for (int d = -r; d <= r; ++d)
            if (j + d < 0 || j + d >= n) a += X.taps[d + r];
        return masked(j) ? a : 0.0;
    };
    for (int which = 0; which < 2; ++which) {
        for (int j = tid; j < n; j += 256) x[0][j] = which == 0 ? (masked(j) ? 1.0 : 0.0) : leak0(j);
        __syncthreads();
        int c = 0;
        for (int s = 1; s < X.m; ++s) {
            for (int j = tid; j < n; j += 256) x[c ^ 1][j] = masked(j) ? band_conv(x[c], X.taps, r, n, j) : 0.0;
            __syncthreads();
            c ^= 1;
        }
        float *out = X.fn + (size_t)which * X.nin * BD_BLK;
        for (int q = tid; q < X.nin * BD_BLK; q += 256) {
            const int j = q - X.H;
            out[q] = (j >= 0 && j < n) ? (float)(x[c][j] * X.fscale) : 0.0f;
        }
        __syncthreads();
    }
    if (X.naff <= 0) return;
    auto block_sum = [&](double v) {
        v = band_warp_sum(v);
        __syncthreads();
        if ((tid & 31) == 0) red[tid >> 5] = v;
        __syncthreads();
        double t = 0.0;
        for (int i = 0; i < 8; ++i) t += red[i];
        return t;
    };
    for (int j = tid; j < n; j += 256) x[0][j] = 1.0;
    __syncthreads();
    int c = 0;
    for (int s = 0; s <= X.naff; ++s) {
        double a = 0.0, l = 0.0, o = 0.0;
        for (int j = tid; j < n; j += 256) {
            const double v = x[c][j];
            a += masked(j) ? v : 0.0;
            l += leak0(j) * v;
            o += v;
            if (s > 0) X.aff[(size_t)(s - 1) * X.affs + j] = (float)v;
        }
        if (s > 0)
            for (int j = n + tid; j < X.affs; j += 256) X.aff[(size_t)(s - 1) * X.affs + j] = 0.0f;
        a = block_sum(a);
        l = block_sum(l);
        o = block_sum(o);
        if (tid == 0) {
            X.dots[s] = a;
            X.dots[(BD_MMAX) + s] = l;
            X.dots[2 * BD_MMAX + s] = o;
        }
        // x_{s+1} = A (M x_s)
        for (int j = tid; j < n; j += 256) {
            double v = 0.0;
            for (int d = max(-r, -j); d <= min(r, n - 1 - j); ++d)
                if (masked(j + d)) v += X.taps[d + r] * x[c][j + d];
            x[c ^ 1][j] = v;
        }
        __syncthreads();
        c ^= 1;
    }
}

// The affine part's share of the accounting: the last substep's input is
// keep^(m-1) B^(m-1) v_0 + c sum_{j=0}^{m-2} keep^j B^j 1, naff = m - 1.
__global__ void band_init_kernel(const BandInit *init, int nfields)
{
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= nfields) return;
    const BandInit &I = init[f];
    for (int i = 0; i < MS_COUNT; ++i) I.out[i] = 0.0;
    double k = I.c;
    for (int j = 0; j < I.naff; ++j, k *= I.keep) {
        const double *x = I.dots[0], *y = I.dots[1], *z = I.dots[2];
        I.out[MS_INPUT] += k * x[j] * y[j] * z[j];
        I.out[MS_LEAK_X] += k * x[BD_MMAX + j] * y[j] * z[j];
        I.out[MS_LEAK_Y] += k * x[2 * BD_MMAX + j + 1] * y[BD_MMAX + j] * z[j];
        I.out[MS_LEAK_Z] += k * x[2 * BD_MMAX + j + 1] * y[2 * BD_MMAX + j + 1] * z[BD_MMAX + j];
        I.affc[j] = (float)k;
    }
}

template <int AXIS>
cudaError_t launch_band_t(const BandJob *jobs, const int *tjob, int tile_begin, int ntiles, BandGeom geo,
                          bool sums, cudaStream_t st)
{
    static thread_local unsigned long long ctx_done = 0;
    static thread_local int sms = 148;
    const unsigned long long ctx = current_context_id();
    if (ctx == 0 || ctx != ctx_done) {
        cudaError_t e = cudaFuncSetAttribute(band_kernel<AXIS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)BD_SMEM_MAX);
        if (e != cudaSuccess) return e;
        int dev = 0;
        if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
        if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
        ctx_done = ctx;
    }
    const int slot = geo.ksteps * BD_STEP_BYTES;
    const size_t xo = AXIS == PASS_X ? BD_XOUT_BYTES : 0;
    // two images, then stages up to three, then more images, then a fourth stage
    int nstage = 2, nslots = 2;
    auto bytes = [&]() { return (size_t)nslots * slot + (size_t)nstage * BD_STAGE_BYTES + xo + 1024; };
    auto grow = [&](int &v, int top) {
        if (v >= top) return;
        ++v;
        if (bytes() > BD_SMEM_MAX) --v;
    };
    if (bytes() > BD_SMEM_MAX) return cudaErrorInvalidConfiguration;
    grow(nstage, 3);
    grow(nslots, 3);
    grow(nstage, BD_MAXSTAGE);
    grow(nslots, BD_MAXSLOT);
    const size_t sm = std::max(bytes(), BD_SMEM_MIN);
    const cudaError_t e = launch_overlapped(ntiles <= 8 * sms, band_kernel<AXIS>, dim3((unsigned)std::min(ntiles, sms)), BD_THREADS, sm, st, jobs,
                                            tjob, tile_begin, tile_begin + ntiles, sums ? 1 : 0, nstage, nslots, slot);
    note_launch();
    return e == cudaSuccess ? cudaGetLastError() : e;
}

}  // namespace

bool band_encode_map(const BandJob &j, int nz, CUtensorMap *m)
{
    if (!j.vec) return false;
    const uint64_t nx = j.nx, ny = j.ny, row = nx * 4, plane = nx * ny * 4;
    if (j.kind == PASS_X)
        return tma_encode_3d(m, j.data, nx, ny * nz, 1, row, plane * nz, 32, BD_LINES, 1, true);
    if (j.kind == PASS_Z) return tma_encode_3d(m, j.data, nx * ny, nz, 1, plane, plane * nz, 32, BD_BLK, 1);
    return nx % 32 == 0 && tma_encode_3d(m, j.data, nx, ny, nz, row, plane, 32, BD_BLK, 1);
}

int band_half_widths(const double *taps, int r, int mmax, int hmax, int *out)
{
    std::vector<double> a(1, 1.0), b;
    for (int m = 1; m <= mmax; ++m) {
        b.assign(a.size() + 2 * r, 0.0);
        for (size_t i = 0; i < a.size(); ++i)
            for (int d = 0; d <= 2 * r; ++d) b[i + d] += a[i] * taps[d];
        a.swap(b);
        const int R = m * r;
        double tail = 0.0;
        int h = R;
        while (h > 0 && tail + 2.0 * a[R + h] < 1e-8) {
            tail += 2.0 * a[R + h];
            --h;
        }
        out[m - 1] = (std::max(h, 1) + 3) / 4 * 4;
        if (out[m - 1] > hmax) return m - 1;
    }
    return mmax;
}

cudaError_t launch_band_setup(const BandAxis *axes, int naxes, int max_rows, const BandInit *init, int nfields,
                              cudaStream_t st)
{
    if (naxes > 0 && max_rows > 0) {
        band_image_kernel<<<dim3((unsigned)((max_rows + 3) / 4), (unsigned)naxes), 128, 0, st>>>(axes);
        note_launch();
        band_vector_kernel<<<naxes, 256, 0, st>>>(axes);
        note_launch();
    }
    if (nfields > 0) {
        band_init_kernel<<<(nfields + 31) / 32, 32, 0, st>>>(init, nfields);
        note_launch();
    }
    return cudaGetLastError();
}

cudaError_t launch_band(const BandJob *jobs, const int *tjob, int tile_begin, int ntiles, int axis,
                        BandGeom geo, bool sums, cudaStream_t st)
{
    if (ntiles <= 0) return cudaSuccess;
    return axis == PASS_X   ? launch_band_t<PASS_X>(jobs, tjob, tile_begin, ntiles, geo, sums, st)
           : axis == PASS_Y ? launch_band_t<PASS_Y>(jobs, tjob, tile_begin, ntiles, geo, sums, st)
                            : launch_band_t<PASS_Z>(jobs, tjob, tile_begin, ntiles, geo, sums, st);
}

cudaError_t band_wait_probe(long long limit, int *gave_up, cudaStream_t st)
{
    band_wait_probe_kernel<<<1, 32, 0, st>>>(limit, gave_up);
    note_launch();
    return cudaGetLastError();
}

}  // namespace vfd
