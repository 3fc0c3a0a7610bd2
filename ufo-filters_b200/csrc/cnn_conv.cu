// 3x3 convolutions for the sparse-view correction network on the 5th-gen
// tensor cores (tcgen05): BF16 operands, FP32 accumulation in tensor memory.
//
// Layouts: activations NHWC bf16 with C a multiple of 16; forward weights
// [Cout][9][Cin] bf16 (tap t = 3*(dy+1) + (dx+1)).
//
// Forward (and data-gradient) convolution as an implicit GEMM:
//   D[p][co] = sum_{t, ci} A[p][(t, ci)] * B[co][(t, ci)]
//   A[p][(t, ci)] = in[p shifted by tap t][ci] (zero outside the image),
// M = 128 consecutive pixels per CTA, N = Cout (the whole output width,
// <= 256 TMEM columns), K walked tap by tap in chunks of <= 64 channels.  The
// data gradient is the same GEMM on the output gradient with the weights
// transposed and tap-flipped ([Cin][9][Cout], t -> 8 - t).
// Weight gradient: dW[co][t][ci] = sum_p dZ[p][co] * in[p + off(t)][ci], a GEMM
// with M = 128 output channels (zero-padded), N = Cin, K = pixels, fed from the
// NHWC tensors as MN-major operands; each CTA reduces a pixel range and adds
// its tile to the FP32 gradient with atomics.
//
// Operand tiles are staged by the CTA's threads into the canonical
// no-swizzle core-matrix layout (8 rows x 16 bytes per core matrix) and made
// visible to the tensor core with fence.proxy.async; one thread issues
// tcgen05.mma (M=128, N=Cout, K=16 per instruction) and tcgen05.commit arrives
// on an mbarrier per shared-memory stage (two stages), so loads of the next K
// chunk overlap the running MMAs.  The epilogue reads the accumulators with
// tcgen05.ld (32 lanes x 32 bit, 8 columns at a time), one pixel per thread.
// Descriptor encodings follow the SM100 UMMA shared-memory and instruction
// descriptor formats (start address>>4, leading/stride byte offsets>>4,
// version 1, no swizzle; c=F32, a=b=BF16, N>>3, M>>4, K- or MN-major bits).
#include <cuda_bf16.h>

#include "tcgen05.cuh"
#include "ufob_internal.h"

namespace ufob {

// Instruction descriptor of kind::f16: D = F32, A = B = BF16, M x N, majorness bits.
__host__ __device__ constexpr uint32_t idesc_bf16(uint32_t M, uint32_t N, uint32_t a_mn_major, uint32_t b_mn_major)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_mn_major << 15) | (b_mn_major << 16) | ((N >> 3) << 17) |
           ((M >> 4) << 24);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8])
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

static constexpr int kErrConvTimeout = 0x2001;

// ------------------------------------------------------------------ forward / data-gradient conv

struct ConvArgs {
    const __nv_bfloat16 *in;  // [NB][H][W][Cin]
    const __nv_bfloat16 *w;   // [Cout][9][Cin]
    const float *bias;        // [Cout] or null
    const __nv_bfloat16 *residual;  // [NB][H][W][Cout] added after the activation, or null
    __nv_bfloat16 *out;       // [NB][H][W][Cout] or null
    float *out_f32;           // [NB][H][W][Cout] or null
    int NB, H, W, Cin, Cout, relu;
    int cols;  // output columns per CTA
    int *err;
};

// Core-matrix (8 rows x 16 B) no-swizzle K-major layout of a rows x BK tile:
// chunk k (8 bf16 along K) of row r at  k*LBO + (r/8)*128 + (r%8)*16.
//
// What bounds it is the latency of a K chunk (loads, store to shared memory, barrier, products), so
// the next chunk's loads are in registers while the current one is multiplied, chunks run across
// taps (16 channels: three chunks of 64 for nine taps), shared memory is what the CTA's columns need
// (96 KB for any layer allowed two CTAs per SM), and layers with few pixel tiles split their output
// columns over blockIdx.y.
// Training step of 16 x 512^2 (us per launch, before -> after): the three layers at 128^2 99 -> 57, at
// 64^2 50 -> 38, at 32^2 54 -> 44, 128<->256 channels at 16^2 160 -> 45..62.
constexpr int kConvBK = 64;     // K chunk: (tap, channel) pairs
constexpr int kConvCols = 128;  // output columns per CTA at most

__host__ __device__ constexpr uint32_t conv_smem_bytes(int cols) { return 2u * (128 + cols) * kConvBK * 2; }

__global__ void __launch_bounds__(128) k_conv3x3(const ConvArgs a)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int Cin = a.Cin, Cout = a.Cout;
    const int n0 = blockIdx.y * a.cols, cols = min(a.cols, Cout - n0);  // output columns of this CTA
    constexpr int kchunks = kConvBK / 8;
    const uint32_t A_BYTES = 128 * kConvBK * 2, B_BYTES = a.cols * kConvBK * 2;
    unsigned char *sA[2] = {smem, smem + A_BYTES + B_BYTES};
    unsigned char *sB[2] = {smem + A_BYTES, smem + 2 * A_BYTES + B_BYTES};
    const uint32_t lboA = 16 * 128, lboB = (uint32_t)(cols / 8) * 128;
    const uint32_t ncols = cols <= 32 ? 32 : (cols <= 64 ? 64 : 128);

    if (warp == 0) tmem_alloc(&tslot, ncols);
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tslot;

    const long long npix = (long long)a.NB * a.H * a.W;
    const long long p = (long long)blockIdx.x * 128 + tid;  // this thread's pixel for loading and output
    int pb = 0, py = 0, px = 0;
    const bool pvalid = p < npix;
    if (pvalid) {
        px = (int)(p % a.W);
        py = (int)((p / a.W) % a.H);
        pb = (int)(p / ((long long)a.W * a.H));
    }
    const uint32_t idesc = idesc_bf16(128, (uint32_t)cols, 0, 0);
    const int K = 9 * Cin, kc = Cin / 8;  // K index (tap, channel), as the weights lie
    const int nk = (K + kConvBK - 1) / kConvBK;
    constexpr int brows = 128 / kchunks;  // weight rows a sweep of the CTA loads
    const int bk_ = tid % kchunks, br = tid / kchunks;
    uint32_t taps = 0;  // taps of this thread's pixel that lie in the image
#pragma unroll
    for (int t = 0; t < 9; t++) {
        const int yy = py + t / 3 - 1, xx = px + t % 3 - 1;
        if (pvalid && yy >= 0 && yy < a.H && xx >= 0 && xx < a.W) taps |= 1u << t;
    }
    const __nv_bfloat16 *pix = a.in + (((size_t)pb * a.H + py) * a.W + px) * Cin;
    const __nv_bfloat16 *wrow = a.w + (size_t)(n0 + br) * K + bk_ * 8;
    uint4 ra[kchunks], rb[kConvCols / brows];
    // chunk i of this thread's pixel (eight channels at a time, shifted by their tap) and of its share
    // of the weight rows
    auto load = [&](int i) {
        const int k0 = i * kchunks;
        int t = k0 / kc, c = k0 - t * kc;
#pragma unroll
        for (int k = 0; k < kchunks; k++) {
            ra[k] = (taps >> t) & 1u
                        ? __ldg(reinterpret_cast<const uint4 *>(pix + ((t / 3 - 1) * a.W + t % 3 - 1) * Cin) + c)
                        : make_uint4(0, 0, 0, 0);
            if (++c == kc) {
                c = 0;
                t++;
            }
        }
        if ((k0 + bk_) * 8 < K) {
#pragma unroll
            for (int q = 0; q < kConvCols / brows; q++)
                if (br + q * brows < cols)
                    rb[q] = __ldg(reinterpret_cast<const uint4 *>(wrow + (size_t)q * brows * K + k0 * 8));
        }
    };
    bool ok = true;
    load(0);
    for (int i = 0; i < nk && ok; i++) {
        const int st = i & 1;
        // MMAs of chunk i-2 done
        if (i >= 2) ok = mbar_wait_bounded(&bars[st], (uint32_t)(((i - 2) >> 1) & 1), kWaitLimitNs);
#pragma unroll
        for (int k = 0; k < kchunks; k++)
            *reinterpret_cast<uint4 *>(sA[st] + k * lboA + (tid >> 3) * 128 + (tid & 7) * 16) = ra[k];
#pragma unroll
        for (int q = 0; q < kConvCols / brows; q++) {
            const int row = br + q * brows;
            if (row < cols)
                *reinterpret_cast<uint4 *>(sB[st] + bk_ * lboB + (row >> 3) * 128 + (row & 7) * 16) = rb[q];
        }
        if (i + 1 < nk) load(i + 1);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA[st]), b0 = smem_u32(sB[st]);
            const int steps = min(kConvBK, K - i * kConvBK) / 16;
            for (int s = 0; s < steps; s++)
                mma_ss(tmem, plain_desc(a0 + s * 2 * lboA, lboA, 128), plain_desc(b0 + s * 2 * lboB, lboB, 128),
                          idesc, (i > 0 || s > 0) ? 1u : 0u);
            mma_commit(&bars[st]);
        }
    }
    // the last chunk's commit covers every earlier MMA of this thread
    if (ok) ok = mbar_wait_bounded(&bars[(nk - 1) & 1], (uint32_t)(((nk - 1) >> 1) & 1), kWaitLimitNs);
    tc_fence_after();
    if (!ok) {
        if (tid == 0) atomicExch(a.err, kErrConvTimeout);
    } else {
        // epilogue: warp w owns TMEM lanes (pixels) 32w .. 32w+31
        const long long q = (long long)blockIdx.x * 128 + warp * 32 + lane;
        for (int cl = 0; cl < cols; cl += 8) {
            const int c = n0 + cl;
            float v[8];
            tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)cl, v);
            if (q < npix) {
                if (a.bias)
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] += a.bias[c + j];
                if (a.relu)
#pragma unroll
                    for (int j = 0; j < 8; j++) v[j] = fmaxf(v[j], 0.f);
                if (a.residual) {
                    const uint4 r = *reinterpret_cast<const uint4 *>(a.residual + q * Cout + c);
                    const __nv_bfloat162 *rh = reinterpret_cast<const __nv_bfloat162 *>(&r);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float2 f = __bfloat1622float2(rh[j]);
                        v[2 * j] += f.x;
                        v[2 * j + 1] += f.y;
                    }
                }
                if (a.out) {
                    uint4 o;
                    __nv_bfloat162 *oh = reinterpret_cast<__nv_bfloat162 *>(&o);
#pragma unroll
                    for (int j = 0; j < 4; j++) oh[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                    *reinterpret_cast<uint4 *>(a.out + q * Cout + c) = o;
                }
                if (a.out_f32)
#pragma unroll
                    for (int j = 0; j < 8; j++) a.out_f32[q * Cout + c + j] = v[j];
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// ------------------------------------------------------------------ weight gradient

struct WgradArgs {
    const __nv_bfloat16 *in;  // [NB][H][W][Cin]   (layer input)
    const __nv_bfloat16 *dz;  // [NB][H][W][Cout]  (gradient at the pre-activation)
    float *dw;                // [Cout][9][Cin] FP32, accumulated with atomics
    int NB, H, W, Cin, Cout;
    long long pix_per_cta;    // K range of one CTA (multiple of 64)
    int taps;                 // taps per CTA
    int *err;
};

__device__ __forceinline__ void red_add4(float *dst, float x, float y, float z, float w)
{
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(x), "f"(y), "f"(z), "f"(w) : "memory");
}

// MN-major no-swizzle layout of an R x 64 (rows x K) tile fed from NHWC data:
// the 16-byte chunk of rows 8g..8g+7 at K index k sits at g*128 + (k/8)*LBO + (k%8)*16.
// A holds only the layer's channels: the rows of the M = 128 product past them read whatever lies
// behind (inside the CTA's shared memory) and are not used.
//
// As the forward kernel, bound by the latency of a chunk: next chunk's loads in registers, several
// taps of a small layer along N (nine CTAs per pixel range before), shared memory by the channels, 32-bit
// pixel arithmetic in the loads (64-bit divisions per 16 bytes had been most of a chunk's instructions),
// at least 512 pixels per CTA and 16-byte reductions into the gradient.  Training step of 16 x 512^2 (us, before -> after): 165 -> 38..89 for the layers up to 128
// channels, 107..165 -> 36 for 128<->256.
constexpr int kWgradCols = 128;  // channels of either operand per CTA at most

__host__ __device__ constexpr uint32_t wgrad_smem_bytes(int co, int ci) { return 2u * (co + ci) * 64 * 2 + 16 * 1024; }

__global__ void __launch_bounds__(128) k_conv3x3_wgrad(const WgradArgs a)
{
    constexpr int BK = 64;  // pixels per K chunk
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ uint64_t bars[2];
    __shared__ uint32_t tslot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int Cin = a.Cin, Cout = a.Cout;
    const int t0 = blockIdx.y * a.taps, taps = min(a.taps, 9 - t0);  // taps of this CTA, along N
    const int mtiles = (Cout + kWgradCols - 1) / kWgradCols;
    const int co0 = (int)(blockIdx.z % mtiles) * kWgradCols, ci0 = (int)(blockIdx.z / mtiles) * kWgradCols;
    const int mrows = min(kWgradCols, Cout - co0), chans = min(kWgradCols, Cin - ci0), nrows = taps * chans;
    const uint32_t A_BYTES = (uint32_t)mrows * BK * 2, B_BYTES = (uint32_t)(a.taps * chans) * BK * 2;
    unsigned char *sA[2] = {smem, smem + A_BYTES + B_BYTES};
    unsigned char *sB[2] = {smem + A_BYTES, smem + 2 * A_BYTES + B_BYTES};
    const uint32_t lboA = (uint32_t)(mrows / 8) * 128, lboB = (uint32_t)(nrows / 8) * 128;  // K-group strides
    const uint32_t ncols = nrows <= 32 ? 32 : (nrows <= 64 ? 64 : 128);

    if (warp == 0) tmem_alloc(&tslot, ncols);
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_barrier_init();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tslot;

    const long long npix = (long long)a.NB * a.H * a.W;
    const long long p_begin = (long long)blockIdx.x * a.pix_per_cta;
    const long long p_end = min(npix, p_begin + a.pix_per_cta);
    const int nk = p_end > p_begin ? (int)((p_end - p_begin + BK - 1) / BK) : 0;
    const uint32_t idesc = idesc_bf16(128, (uint32_t)nrows, 1, 1);
    const uint32_t ca = (uint32_t)mrows / 8, cb = (uint32_t)nrows / 8;  // 16-byte chunks per pixel for A and B
    const uint32_t cc = (uint32_t)chans / 8;  // of them per tap
    const uint32_t W = (uint32_t)a.W, H = (uint32_t)a.H;
    // column and row of the CTA's first pixel
    const uint32_t x_begin = (uint32_t)(p_begin % a.W), y_begin = (uint32_t)((p_begin / a.W) % a.H);
    constexpr int NR = BK * kWgradCols / 8 / 128;  // 16-byte loads of either operand per thread at most
    uint4 ra[NR], rb[NR];
    auto load = [&](int i) {
        const long long pk0 = p_begin + (long long)i * BK;
        const uint32_t left = (uint32_t)min((long long)BK, p_end - pk0);
        // dz[p][co0 .. co0+mrows) and in[p + off(t)][ci0 .. ci0+nrows) for the 64 pixels of the chunk
#pragma unroll
        for (int q = 0; q < NR; q++) {
            const uint32_t idx = tid + 128 * q, k = idx / ca, g = idx - k * ca;
            if (k >= BK) break;
            ra[q] = k < left ? __ldg(reinterpret_cast<const uint4 *>(a.dz + (pk0 + k) * Cout + co0) + g)
                             : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int q = 0; q < NR; q++) {
            const uint32_t idx = tid + 128 * q, k = idx / cb, g = idx - k * cb;
            if (k >= BK) break;
            const uint32_t xl = x_begin + (uint32_t)i * BK + k, yl = xl / W;
            const int tl = (int)(g / cc), dy = (t0 + tl) / 3 - 1, dx = (t0 + tl) % 3 - 1;
            const int x = (int)(xl - yl * W), y = (int)((y_begin + yl) % H);
            const bool in = k < left && y + dy >= 0 && y + dy < a.H && x + dx >= 0 && x + dx < a.W;
            rb[q] = in ? __ldg(reinterpret_cast<const uint4 *>(a.in + (pk0 + k + (long long)dy * a.W + dx) * Cin + ci0) +
                               (g - tl * cc))
                       : make_uint4(0, 0, 0, 0);
        }
    };
    bool ok = true;
    if (nk > 0) load(0);
    for (int i = 0; i < nk && ok; i++) {
        const int st = i & 1;
        if (i >= 2) ok = mbar_wait_bounded(&bars[st], (uint32_t)(((i - 2) >> 1) & 1), kWaitLimitNs);
#pragma unroll
        for (int q = 0; q < NR; q++) {
            const uint32_t idx = tid + 128 * q, k = idx / ca, g = idx - k * ca;
            if (k >= BK) break;
            *reinterpret_cast<uint4 *>(sA[st] + g * 128 + (k >> 3) * lboA + (k & 7) * 16) = ra[q];
        }
#pragma unroll
        for (int q = 0; q < NR; q++) {
            const uint32_t idx = tid + 128 * q, k = idx / cb, g = idx - k * cb;
            if (k >= BK) break;
            *reinterpret_cast<uint4 *>(sB[st] + g * 128 + (k >> 3) * lboB + (k & 7) * 16) = rb[q];
        }
        if (i + 1 < nk) load(i + 1);
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA[st]), b0 = smem_u32(sB[st]);
            // MN-major: leading offset = K-group stride, stride offset = 8-row group stride
            for (int s = 0; s < BK / 16; s++)
                mma_ss(tmem, plain_desc(a0 + s * 2 * lboA, lboA, 128), plain_desc(b0 + s * 2 * lboB, lboB, 128),
                          idesc, (i > 0 || s > 0) ? 1u : 0u);
            mma_commit(&bars[st]);
        }
    }
    if (nk > 0 && ok) ok = mbar_wait_bounded(&bars[(nk - 1) & 1], (uint32_t)(((nk - 1) >> 1) & 1), kWaitLimitNs);
    tc_fence_after();
    if (!ok) {
        if (tid == 0) atomicExch(a.err, kErrConvTimeout);
    } else if (nk > 0) {
        const int row = warp * 32 + lane;  // TMEM lane = output channel
        const bool vec = ((uintptr_t)a.dw & 15u) == 0;
        for (int c = 0; c < nrows; c += 8) {
            float v[8];
            tmem_ld8(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
            if (row < mrows) {
                const int tl = c / chans;
                float *dst = a.dw + ((size_t)(co0 + row) * 9 + t0 + tl) * Cin + ci0 + (c - tl * chans);
                if (vec) {
                    red_add4(dst, v[0], v[1], v[2], v[3]);
                    red_add4(dst + 4, v[4], v[5], v[6], v[7]);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; j++) atomicAdd(dst + j, v[j]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, ncols);
}

// ------------------------------------------------------------------ host launchers

ufob_status conv3x3_launch(const __nv_bfloat16 *in, const __nv_bfloat16 *w, const float *bias,
                           const __nv_bfloat16 *residual, __nv_bfloat16 *out, float *out_f32, int NB, int H, int W,
                           int Cin, int Cout, int relu, cudaStream_t s)
{
    if (Cin % 16 || Cout % 16 || Cin < 16 || Cout < 16 || Cin > 256 || Cout > 256 || (Cin > 64 && Cin % 64))
        return fail(UFOB_ERR_INVALID, "conv3x3: channels must be multiples of 16 in [16, 256] (Cin > 64: of 64)");
    static std::atomic<uint64_t> attr_devs{0};
    UFOB_CUDA_TRY(smem_limit_per_device(k_conv3x3, (int)conv_smem_bytes(kConvCols), attr_devs));
    ConvArgs a;
    a.in = in;
    a.w = w;
    a.bias = bias;
    a.residual = residual;
    a.out = out;
    a.out_f32 = out_f32;
    a.NB = NB;
    a.H = H;
    a.W = W;
    a.Cin = Cin;
    a.Cout = Cout;
    a.relu = relu;
    a.err = device_error_word();
    const long long npix = (long long)NB * H * W;
    const unsigned grid = (unsigned)((npix + 127) / 128);
    // few pixel tiles: split the output columns until every SM has two CTAs or a CTA 32 columns
    a.cols = std::min(Cout, kConvCols);
    while (a.cols > 32 && a.cols % 32 == 0 && (long long)grid * ((Cout + a.cols - 1) / a.cols) < 2 * num_sms())
        a.cols /= 2;
    k_conv3x3<<<dim3(grid, (Cout + a.cols - 1) / a.cols), 128, conv_smem_bytes(a.cols), s>>>(a);
    UFOB_CUDA_TRY(cudaGetLastError());
    note_launch();
    return UFOB_OK;
}

ufob_status conv3x3_wgrad_launch(const __nv_bfloat16 *in, const __nv_bfloat16 *dz, float *dw, int NB, int H, int W,
                                 int Cin, int Cout, cudaStream_t s)
{
    if (Cin % 16 || Cout % 16 || Cin < 16 || Cout < 16 || Cin > 256 || Cout > 256)
        return fail(UFOB_ERR_INVALID, "conv3x3 wgrad: channels must be multiples of 16 in [16, 256]");
    static std::atomic<uint64_t> attr_devs{0};
    UFOB_CUDA_TRY(smem_limit_per_device(k_conv3x3_wgrad, (int)wgrad_smem_bytes(kWgradCols, kWgradCols), attr_devs));
    const long long npix = (long long)NB * H * W;
    // as many taps as fill the columns, in equal shares; about eight CTAs per SM over (pixel ranges x
    // tap groups x channel tiles), 512 pixels each at least
    const int tiles = ((Cout + kWgradCols - 1) / kWgradCols) * ((Cin + kWgradCols - 1) / kWgradCols);
    const int most = std::max(1, kWgradCols / std::min(Cin, kWgradCols));
    const int groups = (9 + most - 1) / most, taps = (9 + groups - 1) / groups;
    long long ranges =
        std::max<long long>(1, std::min<long long>((long long)num_sms() * 8 / (groups * tiles), npix / 512));
    long long per = (npix + ranges - 1) / ranges;
    per = (per + 63) / 64 * 64;
    ranges = (npix + per - 1) / per;
    WgradArgs a;
    a.in = in;
    a.dz = dz;
    a.dw = dw;
    a.NB = NB;
    a.H = H;
    a.W = W;
    a.Cin = Cin;
    a.Cout = Cout;
    a.pix_per_cta = per;
    a.taps = taps;
    a.err = device_error_word();
    k_conv3x3_wgrad<<<dim3((unsigned)ranges, (9 + taps - 1) / taps, tiles), 128,
                      wgrad_smem_bytes(std::min(Cout, kWgradCols), taps * std::min(Cin, kWgradCols)), s>>>(a);
    UFOB_CUDA_TRY(cudaGetLastError());
    note_launch();
    return UFOB_OK;
}

}  // namespace ufob

using namespace ufob;

// Low-level entry points (used by the network and by the gradient tests).
extern "C" ufob_status ufob_conv3x3_forward(const void *d_in, const void *d_w, const float *d_bias,
                                            const void *d_residual, void *d_out, float *d_out_f32, int nb, int h,
                                            int w, int cin, int cout, int relu, void *stream)
{
    UFOB_TRY(ensure_device());
    return conv3x3_launch((const __nv_bfloat16 *)d_in, (const __nv_bfloat16 *)d_w, d_bias,
                          (const __nv_bfloat16 *)d_residual, (__nv_bfloat16 *)d_out, d_out_f32, nb, h, w, cin, cout,
                          relu, (cudaStream_t)stream);
}

extern "C" ufob_status ufob_conv3x3_wgrad(const void *d_in, const void *d_dz, float *d_dw, int nb, int h, int w,
                                          int cin, int cout, void *stream)
{
    UFOB_TRY(ensure_device());
    return conv3x3_wgrad_launch((const __nv_bfloat16 *)d_in, (const __nv_bfloat16 *)d_dz, d_dw, nb, h, w, cin, cout,
                                (cudaStream_t)stream);
}
