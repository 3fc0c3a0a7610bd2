// Parallel-beam backprojection of an FP32 stack from slice cells (the plain form of the FBP for
// stacks): the image of backproject.cu's 32 x 32 tiles, bit for bit (src/kernels/backproject.cl:50-94).
//
// The row kernel (k_bp_linear) loads both taps of every update as 4-byte words and is bound by
// shared memory: 8 bytes per update, 3.7 TGUPS of the 4.6 that its loads allow.  Two changes:
//   * slice-quad cells [ceil(nz/4)][P][W] of four floats (bin j of four slices): one 16-byte load is
//     a tap of four updates, a quarter of the load instructions;
//   * a thread walks eight rows of one pixel column.  From one row to the next the detector
//     coordinate moves by sin(theta), at most one bin, so the lower tap of a row is the lower or the
//     upper tap of the row before, which is in registers: one new tap per update, 4.5 bytes.  Rows
//     are walked in the direction in which the coordinate grows; near sin = +-1 rounding can make
//     it pass two bins, there both taps are loaded.
// 32 slices of 2048^2 x 1500 angles: 54.1 -> 38.3 ms (3.72 -> 5.25 TGUPS), shared-memory wavefronts at
// 78% of their rate; with the lower tap's step checked per row 43.3 ms, with both taps of every row
// loaded the rate of the loads themselves would be 4.6 TGUPS.
// Same operations in the same order as the row kernel: coordinates relative to the 32 x 32 tile's
// 16-byte aligned window origin, the two FMAs of an update, sums over blocks of 16 angles added to
// the total.  The totals live in shared memory (one read and write per 16 angles), the block sums in
// registers.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

#include "f32x2.cuh"
#include "tma.cuh"
#include "ufob_internal.h"

namespace ufob {

namespace {

constexpr int TX = 32, TY = 64, RY = 8;  // tile, rows per thread
constexpr int ZT = 8, NG = ZT / 4;       // slices per CTA, cells of a tap
constexpr int A = 8, S = 2;              // angles per stage, stages
constexpr int FOLD = 2;                  // stages per block sum
constexpr int kWarps = TY / RY;
constexpr int kThreads = 32 * kWarps;
// bins a tile reaches: its diagonal (71), floor, upper tap, and up to 4 of the window origin
constexpr int NW = 80;
constexpr int kOldWin = 52;  // window of the row kernel's 32 x 32 tile, to which it clamps
constexpr uint32_t kAngleBytes = NW * 16 * NG;
constexpr uint32_t kAccBytes = TX * TY * ZT * 4;
constexpr uint32_t kSmem = S * A * kAngleBytes + kAccBytes + 128;

__device__ __forceinline__ void tma_load_cells(void *dst, const CUtensorMap *map, uint64_t *bar, int c1, int c2, int c3)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
        : "memory");
}

// Window origin of the 32 x 32 tile at (x, y), as the row kernel computes it.
__device__ __forceinline__ int window_origin(const BPArgs &args, int x, int y, float2 sc)
{
    const float axis = args.axis;
    const float cx0 = (float)(args.roi_x + x) - axis + 0.5f, cx1 = cx0 + 31.0f;
    const float cy0 = (float)(args.roi_y + y) - axis + 0.5f, cy1 = cy0 + 31.0f;
    const float h0 = fmaf(cy0, sc.x, fmaf(cx0, sc.y, axis)), h1 = fmaf(cy0, sc.x, fmaf(cx1, sc.y, axis));
    const float h2 = fmaf(cy1, sc.x, fmaf(cx0, sc.y, axis)), h3 = fmaf(cy1, sc.x, fmaf(cx1, sc.y, axis));
    int e = (int)floorf(fminf(fminf(h0, h1), fminf(h2, h3)) - 0.5f) - 1;
    e = max(min(e, 1 << 24), -(1 << 24));
    return e & ~3;
}

struct Tap {
    float4 v[NG];
};

__device__ __forceinline__ Tap load_tap(const float4 *cells, uint32_t e)
{
    Tap t;
#pragma unroll
    for (int g = 0; g < NG; g++) t.v[g] = cells[g * NW + e];
    return t;
}

// part += (1 - w) lo + w hi of one pixel, slices as packed FP32 pairs
__device__ __forceinline__ void add_sample(uint64_t (&part)[ZT / 2], const Tap &lo, const Tap &hi, float omw, float w)
{
    const uint64_t o2 = f2pack(omw, omw), w2 = f2pack(w, w);
#pragma unroll
    for (int g = 0; g < NG; g++) {
        part[2 * g] = f2fma(o2, f2pack(lo.v[g].x, lo.v[g].y), part[2 * g]);
        part[2 * g] = f2fma(w2, f2pack(hi.v[g].x, hi.v[g].y), part[2 * g]);
        part[2 * g + 1] = f2fma(o2, f2pack(lo.v[g].z, lo.v[g].w), part[2 * g + 1]);
        part[2 * g + 1] = f2fma(w2, f2pack(hi.v[g].z, hi.v[g].w), part[2 * g + 1]);
    }
}

// How a thread's eight rows are walked: in the order in which the coordinate grows, each lower tap
// taken from the row before, or (where rounding can pass two bins) every tap loaded.
enum Walk { WALK_UP, WALK_DOWN, WALK_LOAD };

template <Walk WALK>
__device__ __forceinline__ void add_rows(uint64_t (&part)[RY][ZT / 2], const float4 *cells, const float *by, float s,
                                         float t, uint32_t shift)
{
    const float kMagic = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer in the mantissa
    const int kMagicBits = 0x4B400000;
    Tap lo, hi;
    uint32_t last = 0;
#pragma unroll
    for (int i = 0; i < RY; i++) {
        const int j = WALK == WALK_DOWN ? RY - 1 - i : i;
        const float vv = fmaf(by[j], s, t);
        const float r = vv + kMagic;
        const float d = vv - (r - kMagic);
        const float w = d + 0.5f, omw = 0.5f - d;
        const uint32_t e = min(min((uint32_t)(__float_as_int(r) - kMagicBits), (uint32_t)(kOldWin - 2)) + shift,
                               (uint32_t)(NW - 2));
        if (WALK == WALK_LOAD || i == 0) {
            lo = load_tap(cells, e);
        } else {
            const bool step = e != last;
#pragma unroll
            for (int g = 0; g < NG; g++) {
                lo.v[g].x = step ? hi.v[g].x : lo.v[g].x;
                lo.v[g].y = step ? hi.v[g].y : lo.v[g].y;
                lo.v[g].z = step ? hi.v[g].z : lo.v[g].z;
                lo.v[g].w = step ? hi.v[g].w : lo.v[g].w;
            }
        }
        hi = load_tap(cells, e + 1);
        last = e;
        add_sample(part[j], lo, hi, omw, w);
    }
}

__global__ void __launch_bounds__(kThreads, 2) k_bp_cells(const __grid_constant__ CUtensorMap map, const BPArgs args)
{
    extern __shared__ unsigned char smem_dyn[];
    __shared__ uint64_t full[S], empty[S];
    __shared__ float4 s_tab[S][A];   // sin, cos, window origin offsets of the two 32-row halves
    __shared__ uint2 s_shift[S][A];  // their origins relative to the staged window
    __shared__ float s_by[kWarps][RY];
    __shared__ int s_abort;
    unsigned char *raw =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~(uintptr_t)127);
    float4 *acc = reinterpret_cast<float4 *>(raw + S * A * kAngleBytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kWarps);
        }
        s_abort = 0;
        fence_barrier_init();
    }
    __syncthreads();
    // tiles in bands of 8 tile columns walked top to bottom: resident CTAs cover a compact region
    constexpr int GW = 8;
    const int id = blockIdx.y * gridDim.x + blockIdx.x, band_tiles = GW * gridDim.y;
    const int band = id / band_tiles, rr = id - band * band_tiles;
    const int bw = min(GW, (int)gridDim.x - band * GW);
    const int x0 = (band * GW + rr % bw) * TX, y0 = rr / bw * TY, z0 = blockIdx.z * ZT;
    const uint32_t P = args.P;
    const int nblk = (int)((P + A - 1) / A);
    const float eoff = args.axis - 1.0f;  // h - 0.5 - 0.5
    bool ok = true;

    // Windows of stage b: a lane per angle, then one TMA each.  The warps take turns, so none falls
    // behind (a ninth warp would cost a quarter of the registers).
    auto issue = [&](int b) {
        const int slot = b % S, p0 = b * A, nval = min(A, (int)P - p0);
        int ws = 0;
        if (lane < nval) {
            const float2 sc = __ldg(&args.sincos[p0 + lane]);
            const int w0 = window_origin(args, x0, y0, sc), w1 = window_origin(args, x0, y0 + 32, sc);
            ws = min(w0, w1);
            s_tab[slot][lane] = make_float4(sc.x, sc.y, eoff - (float)w0, eoff - (float)w1);
            s_shift[slot][lane] = make_uint2((uint32_t)(w0 - ws), (uint32_t)(w1 - ws));
        }
        __syncwarp();
        if (lane == 0) mbar_arrive_expect_tx(&full[slot], (uint32_t)nval * kAngleBytes);
        for (int a = 0; a < nval; a++) {
            const int w = __shfl_sync(0xffffffffu, ws, a);
            if (lane == 0)
                tma_load_cells(raw + (size_t)(slot * A + a) * kAngleBytes, &map, &full[slot], w, p0 + a, z0 / 4);
        }
    };
    if (warp < S && warp < nblk) issue(warp);

    {
        const int x = x0 + lane, yb = y0 + warp * RY;
        const float bx = (float)(args.roi_x + x) - args.axis + 0.5f;
        // the rows' coordinates, read back per angle: as registers they would spill
        const float *by = s_by[warp];
        if (lane < RY) s_by[warp][lane] = (float)(args.roi_y + yb + lane) - args.axis + 0.5f;
        __syncwarp();
        const bool near = fabsf(by[0]) < 32000.0f && fabsf(by[RY - 1]) < 32000.0f;
        const bool lower = warp >= kWarps / 2;
        uint64_t part[RY][ZT / 2];
#pragma unroll
        for (int i = 0; i < RY; i++)
#pragma unroll
            for (int z = 0; z < ZT / 2; z++) part[i][z] = 0ull;
#pragma unroll
        for (int k = 0; k < RY * NG; k++) acc[k * (32 * kWarps) + tid] = make_float4(0.f, 0.f, 0.f, 0.f);

        for (int b = 0; b < nblk; b++) {
            const int slot = b % S, nval = min(A, (int)P - b * A);
            if (b >= 1 && b - 1 + S < nblk && warp == (b - 1) % kWarps) {
                // stage b - 1 is done everywhere: its slot takes stage b - 1 + S
                ok = mbar_wait_bounded(&empty[(b - 1) % S], (uint32_t)((b - 1) / S) & 1u, kWaitLimitNs);
                if (__all_sync(0xffffffffu, ok)) issue(b - 1 + S);
            }
            ok = ok && mbar_wait_bounded(&full[slot], (uint32_t)(b / S) & 1u, kWaitLimitNs);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
#pragma unroll 1
            for (int a = 0; a < nval; a++) {
                const float4 tab = s_tab[slot][a];
                const uint2 sh = s_shift[slot][a];
                const float4 *cells = reinterpret_cast<const float4 *>(raw + (size_t)(slot * A + a) * kAngleBytes);
                const float t = fmaf(bx, tab.y, lower ? tab.w : tab.z);
                const uint32_t shift = lower ? sh.y : sh.x;
                // a row's step is sin(theta) to within 2^-9 (rounding of rows below 2^15)
                if (!(fabsf(tab.x) < 0.995f) || !near)
                    add_rows<WALK_LOAD>(part, cells, by, tab.x, t, shift);
                else if (tab.x >= 0.0f)
                    add_rows<WALK_UP>(part, cells, by, tab.x, t, shift);
                else
                    add_rows<WALK_DOWN>(part, cells, by, tab.x, t, shift);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);
            if ((b + 1) % FOLD == 0 || b + 1 == nblk) {
#pragma unroll
                for (int i = 0; i < RY; i++)
#pragma unroll
                    for (int g = 0; g < NG; g++) {
                        float4 v = acc[(i * NG + g) * (32 * kWarps) + tid];
                        float p0, p1, p2, p3;
                        f2unpack(part[i][2 * g], p0, p1);
                        f2unpack(part[i][2 * g + 1], p2, p3);
                        v.x += p0;
                        v.y += p1;
                        v.z += p2;
                        v.w += p3;
                        acc[(i * NG + g) * (32 * kWarps) + tid] = v;
                        part[i][2 * g] = part[i][2 * g + 1] = 0ull;
                    }
            }
        }
        if (!ok) s_abort = 1;
        if (ok && x < (int)args.roi_w) {
            const size_t plane = (size_t)args.roi_w * args.roi_h;
#pragma unroll
            for (int i = 0; i < RY; i++) {
                if (yb + i >= (int)args.roi_h) break;
                float *o = args.out + (size_t)z0 * plane + (size_t)(yb + i) * args.roi_w + x;
#pragma unroll
                for (int g = 0; g < NG; g++) {
                    const float4 v = acc[(i * NG + g) * (32 * kWarps) + tid];
                    const float r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (z0 + 4 * g + q < (int)args.nz) o[(size_t)(4 * g + q) * plane] = r[q] * args.norm;
                }
            }
        }
    }
    __syncthreads();
    if (s_abort && tid == 0) {
        atomicExch(args.err, kErrTmaTimeout);
        // let every copy that may still be in flight land before the CTA exits
        for (int s = 0; s < S; s++)
            for (int k = 0; k < 2; k++) mbar_wait_bounded(&full[s], (uint32_t)k, kWaitLimitNs / 8);
    }
    __syncthreads();
}

// FP32 stack [Z][P][pitch] -> cells [ceil(Z/4)][P][W] of four slices
__global__ void k_pack_cells(const float *__restrict__ in, uint32_t pitch, uint64_t slice_pitch, uint32_t W, uint32_t P,
                             uint32_t Z, float4 *__restrict__ out)
{
    const uint32_t g = blockIdx.y;
    for (uint32_t p = blockIdx.x; p < P; p += gridDim.x)
        for (uint32_t j = threadIdx.x; j < W; j += blockDim.x) {
            float v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const uint32_t z = 4 * g + k;
                v[k] = z < Z ? __ldg(in + z * slice_pitch + (uint64_t)p * pitch + j) : 0.f;
            }
            out[((uint64_t)g * P + p) * W + j] = make_float4(v[0], v[1], v[2], v[3]);
        }
}

}  // namespace

bool bp_cells_applies(const BPGeometry &g)
{
    // two CTAs on every SM; below that the row kernel's smaller tiles spread better.  One to four
    // slices would leave half of the CTA's slices empty.
    const uint64_t sms = (uint64_t)num_sms(), tx = (g.roi_w + TX - 1) / TX;
    const uint64_t tiles = tx * ((g.roi_h + TY - 1) / TY);
    if (g.nz <= 4 || tiles * ((g.nz + ZT - 1) / ZT) < 2 * sms) return false;
    // Every launch of up to kCellsGroup slices ends in a partly filled wave of two CTAs per SM, which takes
    // 0.55 of a full one with a CTA per SM; the row kernel's 32 x 32 x 4 tiles (padded to whole ones, too)
    // take 1.45 times as long per tile volume and even out.  us of rows / cells (waves, volume): 64 x 201
    // x 288^2 326 / 409 (2, 1.10), 64 x 224 x 320^2 431 / 450 (2, 1.35), 40 x 291 x 416^2 605 / 631 (2.1, 1.43),
    // 24 x 336 x 480^2 582 / 514 (1.55, 1.14), 12 x 700 x 1001^2 2462 / 2313 (3.55, 2.60).
    auto waves = [&](uint32_t nz) {
        const uint64_t ctas = tiles * ((nz + ZT - 1) / ZT), rest = ctas % (2 * sms);
        return (double)(ctas / (2 * sms)) + (rest == 0 ? 0.0 : rest <= sms ? 0.55 : 1.0);
    };
    const double cells = g.nz / kCellsGroup * waves(kCellsGroup) + waves(g.nz % kCellsGroup);
    const double volume = (double)(tx * ((g.roi_h + 31) / 32) * ((g.nz + 3) / 4)) * (32 * 32 * 4) /
                          (2.0 * (double)sms * TX * TY * ZT);
    return cells <= 1.45 * volume;
}

ufob_status pack_cells_launch(const float *d_in, uint32_t pitch, uint64_t slice_pitch, uint32_t W, uint32_t P,
                              uint32_t Z, void *d_out, cudaStream_t s)
{
    const uint32_t groups = (Z + 3) / 4;
    if (!groups || !P || !W) return UFOB_OK;
    dim3 grid(std::min<uint32_t>(P, std::max<uint32_t>(1, (uint32_t)num_sms() * 16 / groups)), groups);
    k_pack_cells<<<grid, 256, 0, s>>>(d_in, pitch, slice_pitch, W, P, Z, reinterpret_cast<float4 *>(d_out));
    UFOB_CUDA_TRY(cudaGetLastError());
    note_launch();
    return UFOB_OK;
}

ufob_status bp_cells_launch(const BPGeometry &g, const void *d_cells, float *d_out, cudaStream_t stream)
{
    if (!g.roi_w || !g.roi_h || !g.nz || !g.P) return UFOB_OK;
    static std::atomic<uint64_t> attr_devs{0};
    UFOB_CUDA_TRY(smem_limit_per_device(k_bp_cells, (int)kSmem, attr_devs));
    CUtensorMap map;
    UFOB_TRY(make_quad_map(&map, d_cells, g.W, g.P, (g.nz + 3) / 4, g.W, (uint64_t)g.W * g.P, NW, NG));
    BPArgs a;
    a.P = g.P;
    a.nz = g.nz;
    a.roi_x = g.roi_x;
    a.roi_y = g.roi_y;
    a.roi_w = g.roi_w;
    a.roi_h = g.roi_h;
    a.axis = g.axis;
    a.norm = g.norm;
    a.sincos = g.d_sincos;
    a.out = d_out;
    a.err = device_error_word();
    dim3 grid((g.roi_w + TX - 1) / TX, (g.roi_h + TY - 1) / TY, (g.nz + ZT - 1) / ZT);
    k_bp_cells<<<grid, kThreads, kSmem, stream>>>(map, a);
    UFOB_CUDA_TRY(cudaGetLastError());
    note_launch();
    return UFOB_OK;
}

}  // namespace ufob
