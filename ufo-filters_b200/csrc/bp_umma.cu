// Parallel-beam backprojection of a stack on the 5th-gen tensor cores: FP16 filtered sinograms,
// fixed-point interpolation weights, FP32 accumulation (the FP16 form of the FBP for stacks, and
// stacked-backproject's half mode).  Same image as backproject.cu's kernels (src/kernels/
// backproject.cl:50-94): slice[y][x] = pi / P * sum_p lerp(sino[p], h_p), zero outside the detector.
//
// For one angle, the interpolation of a few pixels that share a short detector window is a matrix
// product: D[pixel][slice] += A[pixel][tap] * B[tap][slice], where a row of A holds 1 - f and f at
// the pixel's two taps and zeros elsewhere, and B is the staged window.  11 x 10 pixels reach at
// most 16 bins at any angle (projected diagonal sqrt(10^2 + 9^2) = 13.5), so the product has
// K = 16, one tcgen05.mma of M = 128 (110 rows used) and N = all slices of the CTA.  7 of 8
// products are with zeros, but the slice-quad kernel (backproject.cu) is bound by shared-memory
// gathers and FP32 issue at 22.7 updates per clock and SM, where a product of 128 slices makes
// 110 * 128 updates in 64 tensor-core clocks.
//
//   Sinograms: slice octets [ceil(nz/8)][P][W] of 16-byte cells, cell j = bin j of eight slices.
//     A window is one TMA box of KW cells x 1 angle x ns/8 groups, which lies in shared memory as
//     an N-major operand without swizzle (core matrix = 8 bins x 8 slices), readable from any
//     first bin: the accumulators of a CTA take their own 16 bins of one staged window.
//     (FP16 rows as a K-major operand: 64-byte TMA rows, 6.4 clocks each, 11.7 against 19.8 TGUPS
//     for 128 slices with the first version of this kernel.)
//   Weights: built by CUDA cores, a row of two accumulators per thread, and stored to tensor memory
//     (tcgen05.st), where the product reads A.  (Scattered 4-byte stores to shared memory and A
//     read from there bound the SM's shared memory: 440 of 481 clocks per angle.)  A row is
//     hat(u - k) = max(min(1 + u - k, 1 + k - u), 0) for the taps k = 0..15 in fixed point with 11
//     fractional bits, two taps per 32-bit word (a packed add-min-relu each).  The integers
//     0..2048 read as FP16 are n * 2^-24 exactly (subnormals and the first normals), so the
//     accumulators count in 2^-13 of the sum.  Errors of the weights are at most 2^-12 (the
//     slice-quad kernel: 10 fractional bits).
//   Accumulators: FP32 in tensor memory, MT * ns columns, over blocks of 64 angles whose sums the
//     builders add to totals in registers and shared memory.  The tensor cores cut an addition off at the
//     accumulator's last bit: one sum over 1500 angles of rows in [1, 2) is 3.9e-5 too small, 6000 angles
//     1.6e-4, with blocks 1.1e-6 for any number (the slice-quad kernel's error, rounding of the rows
//     included, 4.6e-6 and 2.3e-6; this one's 4.3e-6 and 2.4e-6).  Up to 32 slices the blocks
//     use two sets of accumulators in turn, so nobody waits for the adding (one set: 16.0 against
//     15.7 ms).  Costs 0.6 of 15.1 ms for 32 slices, 0.7 of 16.8 for 64; blocks of 32 angles 0.5 to 1 ms
//     more, of 128 a bias of 2.2e-6.
//
// Roles of a CTA: four builder warps, a producer warp (one TMA per angle), an MMA warp per
// accumulator (the issuing lane's instructions, not the tensor pipe, limit one warp for both: 29
// against 24 ms).  Stages of KA angles; SA stages of weights, SB of windows; a stage's products
// arrive on one barrier that frees its weights and its windows.  What bounds it is the fixed cost
// of a stage (barriers, issue latencies), so up to 64 slices two CTAs share an SM (KA = 4); above,
// tensor memory holds one CTA, whose stages are longer (KA = 8) and whose totals are mostly registers.
// 2048^2 x 1500 angles, ms per pass: ns <= 32 15.7, 64 17.5, 96 23.7, 128 28.4 (12.8, 23.0, 25.5,
// 28.4 TGUPS; slice quads 6.6).  Four CTAs per SM with KA = 2 up to 32 slices: 16.2 (2% faster without the
// totals, which then are all in shared memory); two with KA = 2 for 96: 26.4.
//
// A non-finite value of a window would reach every pixel of its tile (0 * inf).  The filter flags
// the slices and angles that have one; k_octs_finite puts -0 in the place of such values in these rows
// (and +0 for any -0), notes which class they were and their range, and the epilogue looks up which pixels
// interpolate them: a pixel with a non-finite sample is infinite or NaN whatever its other samples are.
// (Zeroing them in the staged windows cost clean stacks 2 to 9%; leaving the flagged angles out of the
// products and sampling them in the epilogue took 724 ms for 64 x 1500 x 2048 with one dead slice.)
#include <cuda.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <climits>

#include "tcgen05.cuh"
#include "ufob_internal.h"

namespace ufob {

namespace {

constexpr int MX = 11, MY = 10;  // pixels of one accumulator
constexpr int MT = 2;            // accumulators of a CTA, one above the other
static_assert(MT * MY == kUmmaTileRows, "tile height");
constexpr int KT = 16;           // taps of one product
constexpr int KW = 28;           // staged bins: KT + 10 |sin| + 1, rounded up
constexpr int SA = 2;            // stages of weights
constexpr int kBlock = 64;       // angles per sum in tensor memory
constexpr int kBuildWarps = 4;
constexpr int kThreads = 32 * (kBuildWarps + 1 + MT);
enum { CLASS_NAN = 1, CLASS_POS = 2, CLASS_NEG = 4 };  // flag bytes: what the -0 of a row stand for
constexpr int kErrUmmaTimeout = 0x1003;

// KA angles per stage, SB stages of windows, CTAs per SM, and how many 16-column chunks of a builder
// thread's totals are in registers (the others in shared memory; the CTA's slices fill at least RC chunks).
template <int KA_, int SB_, int CTAS_, int RC_>
struct UmmaShape {
    static constexpr int KA = KA_, SB = SB_, CTAS = CTAS_, RC = RC_;
    static constexpr uint32_t kACols = SA * KA * MT * (KT / 2);  // tensor-memory columns of the weights
    static constexpr uint32_t window_bytes(uint32_t ns) { return ns * KW * 2; }  // one angle, all slices
    static constexpr uint32_t totals_bytes(uint32_t ns)
    {
        return MT * ns > 16u * RC ? (MT * ns - 16 * RC) * MX * MY * 4 : 0;
    }
    static constexpr uint32_t smem(uint32_t ns) { return SB * KA * window_bytes(ns) + totals_bytes(ns) + 128; }
};

// Sixteen columns of a warp's lanes; the registers hold them after tmem_wait16.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait16(uint32_t (&r)[16])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                   "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
                 "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

struct UmmaArgs {
    uint32_t P, nz, ns;  // angles, slices, slices per CTA (multiple of 16)
    uint32_t roi_x, roi_y, roi_w, roi_h;
    float axis, norm;
    const float2 *sincos;
    const uint4 *sino;     // slice octets, for the flagged ones
    uint32_t W, pitch;     // bins, cells per row
    uint64_t group_pitch;  // cells per octet
    const uint2 *flags;    // [octets][P] classes of the octet's slices
    const int2 *ranges;    // [octets][P] first and last bin with a non-finite value (none: INT_MAX, -1)
    const uint32_t *any;   // [octets] slices with one at some angle
    float *out;
    uint64_t plane;  // output floats between slices
    int *err;
    uint32_t tiles_x, tiles_y, tmem_cols;
    uint32_t sets;  // of accumulators, used in turn by the blocks of angles
    uint32_t one;  // 1, not known to the compiler: keeps the weights' sums off the busier ALU pipe
};

// Tile of a CTA.  Tiles go in bands about 200 pixels wide, walked top to bottom: the CTAs resident at
// one time cover a compact region, whose windows the L2 serves to all of them.
__device__ __forceinline__ void tile_origin(const UmmaArgs &args, int &x0, int &y0)
{
    constexpr uint32_t GW = 18;
    const uint32_t id = blockIdx.x, band_tiles = GW * args.tiles_y;
    const uint32_t band = id / band_tiles, rr = id - band * band_tiles;
    const uint32_t bw = min(GW, args.tiles_x - band * GW);
    x0 = (int)(band * GW + rr % bw) * MX;
    y0 = (int)(rr / bw) * (MT * MY);
}

// Centre of the tile's upper accumulator along one axis
__device__ __forceinline__ float tile_centre(uint32_t roi0, int first, int pixels, float axis)
{
    return (float)(roi0 + first) - axis + 0.5f + 0.5f * (pixels - 1);
}

// First detector bin reached by the accumulator centred at (cx, cy).  Every role computes it with
// the same operations, so they agree to the bit.
__device__ __forceinline__ int window_start(float cx, float cy, float2 sc, float axis)
{
    const float hc = fmaf(cy, sc.x, fmaf(cx, sc.y, axis));
    const float ext = fmaf(0.5f * (MX - 1), fabsf(sc.y), __fmul_rn(0.5f * (MY - 1), fabsf(sc.x)));
    float e = floorf(__fsub_rn(__fsub_rn(hc, ext), 0.51f));
    e = fminf(fmaxf(e, -16777216.f), 16777216.f);
    return (int)e;
}

// Value that bin `h` (16 bits) of a row of class `cls` stands for.
__device__ __forceinline__ float octet_value(uint32_t h, uint32_t cls)
{
    if (h == 0x8000u && cls) return cls == CLASS_NAN ? NAN : cls == CLASS_POS ? INFINITY : -INFINITY;
    return __half2float(__ushort_as_half((unsigned short)h));
}

// Slices of octet g (of those in `bad`) whose samples at this lane's pixel sum to NaN (bits 0..7), to
// +infinity (8..15) or to -infinity (16..23), by a whole warp: a lane per angle finds those whose
// window at the tile centred at (cx, cy) has a non-finite value, and all lanes sample these.  Done once
// all of `bad` are NaN at every pixel, as after the first angles of slices whose rows the filter's FFT has
// filled with NaN.
__device__ __forceinline__ uint32_t nonfinite_slices(const UmmaArgs &a, float cx, float cy, float bx, float by, bool in,
                                                     uint32_t g, uint32_t bad)
{
    const uint32_t lane = threadIdx.x & 31;
    const size_t row0 = (size_t)g * a.P;
    uint32_t nan = 0, pos = 0, neg = 0;
    constexpr int N = 4;  // groups of 32 angles tested together: one latency for their tables
    for (uint32_t p0 = 0; p0 < a.P; p0 += 32 * N) {
        int2 r[N];
        float2 sl[N];
#pragma unroll
        for (int k = 0; k < N; k++) {
            const uint32_t p = p0 + 32 * k + lane;
            r[k] = p < a.P ? __ldg(a.ranges + row0 + p) : make_int2(INT_MAX, -1);
            sl[k] = __ldg(&a.sincos[min(p, a.P - 1)]);
        }
#pragma unroll
        for (int k = 0; k < N; k++) {
            const int w0 = min(window_start(cx, cy, sl[k], a.axis), window_start(cx, cy + MY, sl[k], a.axis));
            uint32_t hits = __ballot_sync(0xffffffffu, r[k].x <= w0 + KW && r[k].y >= w0 - 1);
            for (; hits && __any_sync(0xffffffffu, in && (bad & ~nan)); hits &= hits - 1) {
                const uint32_t q = __ffs(hits) - 1, p = p0 + 32 * k + q;
                const float s = __shfl_sync(0xffffffffu, sl[k].x, q), c = __shfl_sync(0xffffffffu, sl[k].y, q);
                const int first = __shfl_sync(0xffffffffu, r[k].x, q), last = __shfl_sync(0xffffffffu, r[k].y, q);
                const float h = fmaf(by, s, fmaf(bx, c, a.axis)) - 0.5f;
                const float e = floorf(h), f = h - e;
                if (!in || !(e >= -1.0f && e < (float)a.W)) continue;
                const int j = (int)e;
                if (j + 1 < first || j > last) continue;
                const uint2 cls = __ldg(a.flags + row0 + p);
                const uint4 *row = a.sino + (size_t)g * a.group_pitch + (size_t)p * a.pitch;
                const uint4 zero = make_uint4(0, 0, 0, 0);
                const uint4 lo = j >= 0 ? __ldg(row + j) : zero, hi = j + 1 < (int)a.W ? __ldg(row + j + 1) : zero;
                const uint32_t l[4] = {lo.x, lo.y, lo.z, lo.w}, u[4] = {hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint32_t b = ((i < 4 ? cls.x : cls.y) >> (8 * (i & 3))) & 0xffu;
                    const float s0 = octet_value((l[i / 2] >> (16 * (i & 1))) & 0xffffu, b);
                    const float s1 = octet_value((u[i / 2] >> (16 * (i & 1))) & 0xffffu, b);
                    const float v = (1.0f - f) * s0 + f * s1;
                    if (v != v) nan |= 1u << i;
                    if (v == INFINITY) pos |= 1u << i;
                    if (v == -INFINITY) neg |= 1u << i;
                }
                nan |= pos & neg;
            }
        }
        if (!__any_sync(0xffffffffu, in && (bad & ~nan))) break;
    }
    return nan | (pos & ~nan) << 8 | (neg & ~nan) << 16;
}

// Writes the infinities and NaNs of a CTA's tile over its stored results.  Everything is found anew from
// the block's and thread's indices, so that it keeps no register of the kernel's loops; and it is inlined:
// a call anywhere in the kernel made clean stacks 3 to 8% slower.
__device__ __forceinline__ void store_nonfinite(const UmmaArgs &args)
{
    int x0, y0;
    tile_origin(args, x0, y0);
    const uint32_t lane = threadIdx.x & 31, z0 = blockIdx.y * args.ns, nz = min(args.ns, args.nz - z0);
    const float cx = tile_centre(args.roi_x, x0, MX, args.axis), cy = tile_centre(args.roi_y, y0, MY, args.axis);
    constexpr uint32_t R = (MX * MT * MY + 31) / 32;  // warps' shares of the tile's pixels
    for (uint32_t item = threadIdx.x >> 5; item < R * ((nz + 7) / 8); item += kThreads / 32) {
        const uint32_t q = item / R, pix = (item - q * R) * 32 + lane, bad = __ldg(args.any + z0 / 8 + q);
        if (!bad) continue;
        const int px = x0 + (int)(pix % MX), py = y0 + (int)(pix / MX);
        const bool in = pix < MX * MT * MY && px < (int)args.roi_w && py < (int)args.roi_h;
        const float bx = (float)(args.roi_x + px) - args.axis + 0.5f, by = (float)(args.roi_y + py) - args.axis + 0.5f;
        const uint32_t k = nonfinite_slices(args, cx, cy, bx, by, in, z0 / 8 + q, bad);
        float *o = args.out + (size_t)(z0 + 8 * q) * args.plane + (size_t)py * args.roi_w + px;
        for (uint32_t bits = in ? (k | k >> 8 | k >> 16) & 0xffu : 0; bits; bits &= bits - 1) {
            const uint32_t i = __ffs(bits) - 1;
            o[(size_t)i * args.plane] = (k >> i) & 1u ? NAN : (k >> (8 + i)) & 1u ? INFINITY : -INFINITY;
        }
    }
}

// Flagged rows of a slice octet (blockIdx.x): -0 for the non-finite values of the flagged slices, whose
// bytes then hold the class (a row with several classes counts as NaN), and +0 for any -0 they had.
// Without flags, one read of their words (2 us in all).
__global__ void __launch_bounds__(1024) k_octs_finite(uint4 *__restrict__ cells, uint32_t W, uint32_t pitch,
                                                      uint64_t group_pitch, uint32_t P, uint2 *__restrict__ flags,
                                                      int2 *__restrict__ ranges, uint32_t *__restrict__ any)
{
    __shared__ uint32_t s_any;
    const uint32_t g = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    flags += (size_t)g * P;
    ranges += (size_t)g * P;
    uint32_t some = 0;
    for (uint32_t p = threadIdx.x; p < P; p += 1024) some |= flags[p].x | flags[p].y;
    if (threadIdx.x == 0) any[g] = s_any = 0;
    if (!__syncthreads_or((int)some)) return;
    for (uint32_t base = 0; base < P; base += 1024) {
        const uint32_t p = base + lane * 32 + warp;  // neighbouring angles go to different warps
        const uint2 mine = p < P ? flags[p] : make_uint2(0, 0);
        const bool found = (mine.x | mine.y) != 0;
        if (p < P && !found) ranges[p] = make_int2(INT_MAX, -1);
        for (uint32_t rows = __ballot_sync(0xffffffffu, found); rows; rows &= rows - 1) {
            const int from = __ffs(rows) - 1;
            const uint32_t r = base + from * 32 + warp;
            const uint32_t fx = __shfl_sync(0xffffffffu, mine.x, from), fy = __shfl_sync(0xffffffffu, mine.y, from);
            uint4 *row = cells + (size_t)g * group_pitch + (size_t)r * pitch;
            uint32_t nan = 0, pos = 0, neg = 0;
            int lo = INT_MAX, hi = -1;
#pragma unroll 4
            for (uint32_t j = lane; j < W; j += 32) {
                const uint4 v = row[j];
                uint32_t w[4] = {v.x, v.y, v.z, v.w};
                uint32_t bad = 0;
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const uint32_t sh = 16 * (k & 1), h = (w[k / 2] >> sh) & 0xffffu;
                    if (!((k < 4 ? fx : fy) >> (8 * (k & 3)) & 1u)) continue;
                    if ((h & 0x7C00u) == 0x7C00u) {
                        ((h & 0x3ffu) ? nan : h >> 15 ? neg : pos) |= 1u << k;
                        w[k / 2] = (w[k / 2] & ~(0xffffu << sh)) | 0x8000u << sh;
                        bad = 1;
                    } else if (h == 0x8000u) {
                        w[k / 2] &= ~(0xffffu << sh);
                    }
                }
                if (bad) {
                    lo = min(lo, (int)j);
                    hi = (int)j;
                }
                if (w[0] != v.x || w[1] != v.y || w[2] != v.z || w[3] != v.w)
                    row[j] = make_uint4(w[0], w[1], w[2], w[3]);
            }
            nan = __reduce_or_sync(0xffffffffu, nan);
            pos = __reduce_or_sync(0xffffffffu, pos);
            neg = __reduce_or_sync(0xffffffffu, neg);
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (lane == 0) {
                uint2 f = make_uint2(0, 0);
                for (int k = 0; k < 8; k++) {
                    const uint32_t n = (nan >> k) & 1u, a = (pos >> k) & 1u, b = (neg >> k) & 1u;
                    const uint32_t cls = n || (a && b) ? CLASS_NAN : a ? CLASS_POS : b ? CLASS_NEG : 0;
                    (k < 4 ? f.x : f.y) |= cls << (8 * (k & 3));
                }
                flags[r] = f;
                ranges[r] = make_int2(lo, hi);
                atomicOr(&s_any, nan | pos | neg);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) any[g] = s_any;
}

template <typename Sh>
__global__ void __launch_bounds__(kThreads, Sh::CTAS)
    k_bp_umma(const __grid_constant__ CUtensorMap map, const __grid_constant__ UmmaArgs args)
{
    constexpr int KA = Sh::KA, SB = Sh::SB, RC = Sh::RC;
    static_assert(32 % KA == 0 && kBlock % 32 == 0 && SB >= SA,
                  "whole stages per 32 angles; one barrier ring serves both slots");
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint64_t full_a[SA], full_b[SB], empty[SB], added, done;
    __shared__ float4 s_tab[kBuildWarps][32];
    __shared__ int s_win[32];
    __shared__ uint32_t s_off[MT][32];
    __shared__ uint32_t tslot;
    __shared__ uint32_t s_any;  // an octet has a non-finite value
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bbytes = Sh::window_bytes(args.ns);
    const uint32_t base = (smem_u32(smem_dyn) + 127u) & ~127u;
    unsigned char *gbase = smem_dyn + (base - smem_u32(smem_dyn));

    int x0, y0;
    tile_origin(args, x0, y0);
    const uint32_t z0 = blockIdx.y * args.ns;

    if (warp == kBuildWarps) tmem_alloc(&tslot, args.tmem_cols);
    if (warp == 0) {
        const uint32_t o = z0 / 8 + lane;
        const bool any = 8u * lane < args.ns && o < (args.nz + 7) / 8 && __ldg(args.any + o) != 0;
        if (lane == 0) s_any = 0;
        __syncwarp();
        if (any) s_any = 1;
    }
    if (tid == 0) {
        for (int s = 0; s < SA; s++) mbar_init(&full_a[s], kBuildWarps);
        for (int s = 0; s < SB; s++) {
            mbar_init(&full_b[s], 1);
            mbar_init(&empty[s], MT);
        }
        mbar_init(&added, kBuildWarps);
        mbar_init(&done, MT);
        s_abort = 0;
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tslot;
    volatile int *abort_flag = &s_abort;

    const uint32_t P = args.P;
    const float axis = args.axis;
    const float cx = tile_centre(args.roi_x, x0, MX, axis), cy = tile_centre(args.roi_y, y0, MY, axis);
    // row of both accumulators of a builder thread and its pixel in the upper one (rows past
    // MX * MY repeat pixel 0 and are not stored)
    const int row = (warp & 3) * 32 + lane;
    const int pix = row < MX * MY ? row : 0;
    const int px = x0 + pix % MX, py = y0 + pix / MX;
    const float bx = (float)(args.roi_x + px) - axis + 0.5f;
    const float by = (float)(args.roi_y + py) - axis + 0.5f;

    // Totals of a builder thread's pixels over the blocks added so far, as 16-column chunks of the
    // accumulators' columns: registers, then shared memory.
    const uint32_t chunks = MT * args.ns / 16;
    float4 *totals = reinterpret_cast<float4 *>(gbase + SB * KA * bbytes) + row;
    float tot[RC > 0 ? 16 * RC : 1];
    const uint32_t tlane = tmem + ((uint32_t)(warp & 3) << 21);
    // (one CTA's tensor memory has no room for two sets)
    const uint32_t sets = Sh::CTAS > 1 ? args.sets : 1, set_cols = MT * args.ns;
    // adds the sums of block b, whose products are done, and lets a later block's begin in their place
    auto add_block = [&](uint32_t b) {
        const bool first = b == 0;
        const uint32_t tcol = tlane + (b % sets) * set_cols;
        tc_fence_after();
        uint32_t r[16];
#pragma unroll
        for (int q = 0; q < RC; q++) {
            tmem_ld16(tcol + 16 * q, r);
            tmem_wait16(r);
#pragma unroll
            for (int i = 0; i < 16; i++) tot[16 * q + i] = __uint_as_float(r[i]) + (first ? 0.0f : tot[16 * q + i]);
        }
#pragma unroll 1
        for (uint32_t q = RC; q < chunks; q++) {
            float4 *t = totals + (q - RC) * 4 * (MX * MY), v[4];
            tmem_ld16(tcol + 16 * q, r);
#pragma unroll
            for (int i = 0; i < 4; i++)
                v[i] = first || row >= MX * MY ? make_float4(0.f, 0.f, 0.f, 0.f) : t[i * (MX * MY)];
            tmem_wait16(r);
            if (row < MX * MY)
#pragma unroll
                for (int i = 0; i < 4; i++)
                    t[i * (MX * MY)] =
                        make_float4(v[i].x + __uint_as_float(r[4 * i]), v[i].y + __uint_as_float(r[4 * i + 1]),
                                    v[i].z + __uint_as_float(r[4 * i + 2]), v[i].w + __uint_as_float(r[4 * i + 3]));
            __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&added);
    };

    if (warp < kBuildWarps) {
        const float kFix = 6144.0f;  // 1.5 * 2^12: 11 fractional bits left in the mantissa
        const uint32_t ta = tmem + sets * set_cols + ((uint32_t)warp << 21);
        uint32_t added_blocks = 0;
        const uint32_t one = args.one;
        float4 *tab = s_tab[warp];
        bool ok = true;
        for (uint32_t p0 = 0; p0 < P && ok; p0 += 32) {
            // the sums of a block once its products are done: with one set of accumulators at its end, with
            // two half a block later, when there is nothing to wait for
            const uint32_t late = (sets - 1) * (kBlock / 2);
            if (p0 >= kBlock && p0 % kBlock == late) {
                const uint32_t prev = (p0 - late) / KA - 1;  // its last stage
                ok = late != 0 || wait_or_abort(&empty[prev % SB], (prev / SB) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                add_block(added_blocks++);
            }
            {
                const float2 sc = __ldg(&args.sincos[min(p0 + lane, P - 1)]);
                __syncwarp();
                tab[lane] = make_float4(sc.x, sc.y, axis - 0.5f - (float)window_start(cx, cy, sc, axis),
                                        axis - 0.5f - (float)window_start(cx, cy + MY, sc, axis));
                __syncwarp();
            }
            const uint32_t n = min(32u, P - p0);
            for (uint32_t j = 0; j < n; j += KA) {
                const uint32_t it = (p0 + j) / KA, s = it % SA;
                // slot s is free when the products of stage it - SA are done
                ok = it < SA || wait_or_abort(&empty[(it - SA) % SB], ((it - SA) / SB) & 1u, abort_flag);
                if (!__all_sync(0xffffffffu, ok)) {
                    ok = false;
                    break;
                }
                tc_fence_after();
#pragma unroll
                for (int a = 0; a < KA; a++) {
                    const float4 t = tab[(j + a) & 31];
#pragma unroll
                    for (int h = 0; h < MT; h++) {
                        // tap coordinate, then +-u in units of 2^-11 in both 16-bit halves
                        const float u = fmaf(by + (float)(h * MY), t.x, fmaf(bx, t.y, h ? t.w : t.z));
                        const uint32_t up = __float_as_uint(kFix + u), un = __float_as_uint(kFix - u);
                        const uint32_t up2 = __byte_perm(up, up, 0x1010), un2 = __byte_perm(un, un, 0x1010);
                        uint32_t w[KT / 2];
#pragma unroll
                        for (int k = 0; k < KT / 2; k++) {
                            // taps 2k and 2k + 1.  The second operand is one 32-bit sum: its lower
                            // half carries into the upper one only where it is not negative
                            // (u <= 2k + 1), where the upper half is not the smaller operand
                            constexpr uint32_t c1 = 2048u;
                            const uint32_t lo = ((c1 - (2 * k) * c1) & 0xffffu) | ((c1 - (2 * k + 1) * c1) << 16);
                            const uint32_t hi = (c1 + (2 * k) * c1) + ((c1 + (2 * k + 1) * c1) << 16);
                            w[k] = __viaddmin_s16x2_relu(up2, lo, un2 * one + hi);
                        }
                        tmem_st8(ta + ((s * KA + a) * MT + h) * (KT / 2), w);
                    }
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_a[s]);
            }
        }
        // a block before a last one too short for that: with all products done
        if (ok && (added_blocks + 1) * kBlock < P) {
            ok = wait_or_abort(&done, 0, abort_flag);
            if (__all_sync(0xffffffffu, ok)) add_block(added_blocks);
        }
    } else {
        const bool produce = warp == kBuildWarps;
        const int m = warp - kBuildWarps - 1;  // accumulator of an MMA warp
        // D = F32, A = B = F16, B N-major
        const uint32_t idesc = (1u << 4) | (1u << 16) | ((args.ns >> 3) << 17) | ((128u >> 4) << 24);
        const uint64_t desc0 = plain_desc(base, 128, KW * 16);
        uint32_t dcol = tmem + (uint32_t)m * args.ns;
        const uint32_t acol = tmem + sets * set_cols + (uint32_t)m * (KT / 2);
        uint32_t acc = 0;
        bool ok = true;
        for (uint32_t p0 = 0; p0 < P; p0 += 32) {
            {
                // windows of the next 32 angles, and where in them the accumulators' taps start
                const uint32_t p = min(p0 + lane, P - 1);
                const float2 sc = __ldg(&args.sincos[p]);
                const int w0 = window_start(cx, cy, sc, axis), w1 = window_start(cx, cy + MY, sc, axis);
                const int wm = min(w0, w1);
                __syncwarp();
                if (produce)
                    s_win[lane] = wm;
                else
                    s_off[m][lane] = (uint32_t)min((m ? w1 : w0) - wm, KW - KT);
                __syncwarp();  // the issuing lane reads the other lanes' entries
            }
            const uint32_t n = min(32u, P - p0);
            if (!produce && p0 % kBlock == 0) {
                // a block's first products overwrite the sums of an earlier one, once these are added
                const uint32_t b = p0 / kBlock;
                acc = 0;
                dcol = tmem + (b % sets) * set_cols + (uint32_t)m * args.ns;
                if (b >= sets && lane == 0) ok = wait_or_abort(&added, (b - sets) & 1u, abort_flag);
            }
            if (lane == 0 && ok) {
                for (uint32_t j = 0; j < n; j += KA) {
                    const uint32_t it = (p0 + j) / KA, sb = it % SB, sa = it % SA;
                    const uint32_t nval = min((uint32_t)KA, n - j);
                    if (produce) {
                        ok = it < SB || wait_or_abort(&empty[sb], ((it / SB) - 1) & 1u, abort_flag);
                        if (!ok) break;
                        mbar_arrive_expect_tx(&full_b[sb], nval * bbytes);
#pragma unroll
                        for (uint32_t a = 0; a < KA; a++)
                            if (a < nval)
                                tma_load_3d(gbase + (sb * KA + a) * bbytes, &map, &full_b[sb], s_win[j + a] * 8,
                                            (int)(p0 + j + a), (int)(z0 / 8));
                    } else {
                        uint32_t off[KA];
#pragma unroll
                        for (int a = 0; a < KA; a++) off[a] = s_off[m][j + a];
                        ok = wait_or_abort(&full_b[sb], (it / SB) & 1u, abort_flag) &&
                             wait_or_abort(&full_a[sa], (it / SA) & 1u, abort_flag);
                        if (!ok) break;
                        tc_fence_after();
                        if (nval == KA) {
#pragma unroll
                            for (int a = 0; a < KA; a++)
                                mma_ts(dcol, acol + (sa * KA + a) * (MT * (KT / 2)),
                                        desc0 + (uint64_t)((sb * KA + a) * (bbytes >> 4) + off[a]), idesc,
                                        a > 0 ? 1u : acc);
                        } else {
#pragma unroll 1
                            for (uint32_t a = 0; a < nval; a++)
                                mma_ts(dcol, acol + (sa * KA + a) * (MT * (KT / 2)),
                                        desc0 + (uint64_t)((sb * KA + a) * (bbytes >> 4) + s_off[m][j + a]), idesc,
                                        a > 0 ? 1u : acc);
                        }
                        acc = 1;
                        mma_commit(&empty[sb]);
                    }
                }
            }
            ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            if (!ok) break;
        }
        if (!produce && lane == 0) mma_commit(&done);
    }
    __syncwarp();
    bool ok = true;
    if (warp < kBuildWarps) ok = wait_or_abort(&done, 0, abort_flag);
    __syncthreads();
    if (warp < kBuildWarps) {
        // results: a pixel of each accumulator per thread, slices along its columns
        tc_fence_after();
        if (__all_sync(0xffffffffu, ok)) {
            const size_t plane = args.plane;
            const uint32_t nz = min(args.ns, args.nz - z0);
            const bool added_some = P > kBlock;
            const uint32_t tlast = tlane + ((P - 1) / kBlock % sets) * set_cols;
            // chunk q, with the totals so far in v
            auto store = [&](uint32_t q, float (&v)[16]) {
                const uint32_t h = 16 * q >= args.ns, c = 16 * q - h * args.ns;
                const int y = py + (int)h * MY;
                if (c >= nz) return;
                uint32_t r[16];
                tmem_ld16(tlast + 16 * q, r);
                tmem_wait16(r);
                if (row < MX * MY && px < (int)args.roi_w && y < (int)args.roi_h) {
                    float *o = args.out + (size_t)(z0 + c) * plane + (size_t)y * args.roi_w + px;
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const float sum = (__uint_as_float(r[i]) + (added_some ? v[i] : 0.0f)) * 8192.0f;
                        if (c + i < nz) o[(size_t)i * plane] = sum * args.norm;
                    }
                }
                __syncwarp();
            };
#pragma unroll
            for (int q = 0; q < RC; q++) {
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; i++) v[i] = tot[16 * q + i];
                store(q, v);
            }
#pragma unroll 1
            for (uint32_t q = RC; q < chunks; q++) {
                float v[16] = {};
                if (added_some && row < MX * MY) {
                    const float4 *t = totals + (q - RC) * 4 * (MX * MY);
#pragma unroll
                    for (int i = 0; i < 4; i++) *reinterpret_cast<float4 *>(v + 4 * i) = t[i * (MX * MY)];
                }
                store(q, v);
            }
        }
        tc_fence_before();
    }
    __syncthreads();
    if (s_abort && tid == 0) {
        atomicExch(args.err, kErrUmmaTimeout);
        // copies and products in flight end before the CTA's shared memory and accumulators go
        for (int s = 0; s < SB; s++)
            for (int k = 0; k < 2; k++) mbar_wait_bounded(&full_b[s], (uint32_t)k, kWaitLimitNs / 8);
        mbar_wait_bounded(&done, 0, kWaitLimitNs / 8);
    }
    __syncthreads();
    if (warp == kBuildWarps) tmem_dealloc(tmem, args.tmem_cols);
    if (s_any && !s_abort) store_nonfinite(args);
}

// Map over the slice octets [groups][P][W] of 16-byte cells; box = KW cells x 1 angle x box_groups.
ufob_status make_octet_map(CUtensorMap *map, const void *base, uint32_t W, uint32_t P, uint32_t groups,
                           uint32_t pitch, uint64_t group_pitch, uint32_t box_groups)
{
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
        return fail(UFOB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    auto fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    cuuint64_t dims[3] = {(cuuint64_t)W * 8, P, groups};
    cuuint64_t strides[2] = {(cuuint64_t)pitch * 16, (cuuint64_t)group_pitch * 16};
    cuuint32_t box[3] = {KW * 8, 1, box_groups};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return fail(UFOB_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d): cells=%u P=%u groups=%u pitch=%u box=%u",
                    (int)r, W, P, groups, pitch, box_groups);
    return UFOB_OK;
}

template <typename Sh>
ufob_status launch(const CUtensorMap &map, UmmaArgs a, uint32_t most_slices, cudaStream_t stream)
{
    // two sets of accumulators where that does not cost tensor memory for another CTA
    const uint32_t cols = MT * a.ns + Sh::kACols;
    a.tmem_cols = 32;
    while (a.tmem_cols < cols) a.tmem_cols *= 2;
    a.sets = Sh::CTAS > 1 && cols + MT * a.ns <= a.tmem_cols ? 2 : 1;
    static std::atomic<uint64_t> attr_devs{0};
    UFOB_CUDA_TRY(smem_limit_per_device(k_bp_umma<Sh>, (int)Sh::smem(most_slices), attr_devs));
    dim3 grid(a.tiles_x * a.tiles_y, (a.nz + a.ns - 1) / a.ns);
    k_bp_umma<Sh><<<grid, kThreads, Sh::smem(a.ns), stream>>>(map, a);
    UFOB_CUDA_TRY(cudaGetLastError());
    note_launch();
    return UFOB_OK;
}

}  // namespace

uint32_t bp_umma_slices(uint32_t nz)
{
    // Time of one pass over a tile by slices per CTA (ms at 2048^2 x 1500 angles, as above): equal
    // shares of the stack that take the least in all.
    static const struct {
        uint32_t ns;
        float ms;
    } kPass[] = {{32, 15.7f}, {64, 17.5f}, {96, 23.7f}, {128, 28.4f}};
    uint32_t best = 128;
    float best_t = 1e30f;
    for (uint32_t chunks = (nz + 127) / 128; chunks <= (nz + 31) / 32; chunks++) {
        uint32_t ns = std::max(32u, round_up((nz + chunks - 1) / chunks, 16));
        if (ns > 64) ns = std::max(ns, 96u);  // as many columns as the shape's totals in registers
        float ms = kPass[3].ms;
        for (int i = 3; i >= 0; i--)
            if (ns <= kPass[i].ns) ms = kPass[i].ms;
        if (chunks * ms < best_t) {
            best_t = chunks * ms;
            best = ns;
        }
    }
    return best;
}

size_t umma_flag_bytes(uint32_t P, uint32_t nz)
{
    const size_t octs = (nz + 7) / 8;
    return octs * P * (sizeof(uint2) + sizeof(int2)) + octs * 4;
}

ufob_status umma_finite_launch(const BPGeometry &g, void *d_sino, uint32_t pitch, uint64_t group_pitch,
                               uint8_t *d_flags, cudaStream_t stream)
{
    const uint32_t octs = (g.nz + 7) / 8;
    if (!octs || !g.P) return UFOB_OK;
    const size_t words = (size_t)octs * g.P;
    uint2 *flags = reinterpret_cast<uint2 *>(d_flags);
    int2 *ranges = reinterpret_cast<int2 *>(flags + words);
    k_octs_finite<<<octs, 1024, 0, stream>>>(reinterpret_cast<uint4 *>(d_sino), g.W, pitch, group_pitch, g.P, flags,
                                             ranges, reinterpret_cast<uint32_t *>(ranges + words));
    UFOB_CUDA_TRY(cudaGetLastError());
    note_launch();
    return UFOB_OK;
}

ufob_status bp_umma_launch(const BPGeometry &g, const void *d_sino, uint32_t pitch, uint64_t group_pitch,
                           const uint8_t *d_flags, float *d_out, uint64_t plane, cudaStream_t stream)
{
    if (!g.roi_w || !g.roi_h || !g.nz || !g.P) return UFOB_OK;
    if ((uintptr_t)d_sino & 15) return fail(UFOB_ERR_INVALID, "backproject: slice-octet base must be 16-byte aligned");
    UmmaArgs a;
    a.P = g.P;
    a.nz = g.nz;
    a.ns = bp_umma_slices(g.nz);
    a.roi_x = g.roi_x;
    a.roi_y = g.roi_y;
    a.roi_w = g.roi_w;
    a.roi_h = g.roi_h;
    a.axis = g.axis;
    a.norm = g.norm;
    a.sincos = g.d_sincos;
    a.sino = reinterpret_cast<const uint4 *>(d_sino);
    a.W = g.W;
    a.pitch = pitch;
    a.group_pitch = group_pitch;
    const size_t words = (size_t)((g.nz + 7) / 8) * g.P;
    a.flags = reinterpret_cast<const uint2 *>(d_flags);
    a.ranges = reinterpret_cast<const int2 *>(a.flags + words);
    a.any = reinterpret_cast<const uint32_t *>(a.ranges + words);
    a.out = d_out;
    a.plane = plane;
    a.err = device_error_word();
    a.one = 1;
    a.tiles_x = (g.roi_w + MX - 1) / MX;
    a.tiles_y = (g.roi_h + MT * MY - 1) / (MT * MY);
    CUtensorMap map;
    UFOB_TRY(make_octet_map(&map, d_sino, g.W, g.P, (g.nz + 7) / 8, pitch, group_pitch, a.ns / 8));
    // two CTAs per SM while the accumulators and four angles' weights of both fit in tensor memory
    using Small = UmmaShape<4, 4, 2, 4>;
    using Large = UmmaShape<8, 3, 1, 12>;
    static_assert(MT * 32 >= 16 * Small::RC && MT * 96 >= 16 * Large::RC, "see bp_umma_slices");
    if (a.ns <= 64) return launch<Small>(map, a, 64, stream);
    return launch<Large>(map, a, 128, stream);
}

}  // namespace ufob
