// 3x3 convolutions for the learned pressure warm start (BF16 operands, FP32
// accumulation), NHWC activations with 32 channels.
//
// conv3x3_tc_kernel is an implicit GEMM on the tcgen05 tensor cores: one CTA computes
// 128 output slots x 32 output channels, D[128x32] = A[128x288] * B[32x288]^T with
// K = 9 taps x 32 input channels, as 18 K = 16 MMAs of one thread into a 32-column FP32
// accumulator in tensor memory, committed to an mbarrier; each warp then reads its 32 rows
// back with tcgen05.ld and applies bias, the optional skip input, ReLU and the stores.
//
// No im2col copy is made. The pixels are numbered with one border column on either side
// (rows of W + 2 slots), and a tap one column over is the same operand one slot on. A CTA
// stages three bands, rows y - 1, y and y + 1 of its 128 slots and one on either side,
// zero-filled outside the image, with 16-byte cp.async copies: 25 KB instead of the 74 KB
// of all nine taps, five CTAs an SM instead of two. Slot k of band dy, channels 8g .. 8g+7,
// lives at byte (4*dy + g)*kPlane + 16*k, so that the A operand of tap (dy, dx) and 16
// channels is a no-swizzle K-major operand from slot dx on: core matrices of 8 slots x 8
// channels are 128 contiguous bytes, the next along K one plane on (LBO), the next 8 rows
// 128 bytes on (SBO). The two border slots of a row are computed and dropped (2 in W + 2).
// kPlane is 32 modulo 128 bytes: a warp's copies, 8 slots x 4 channel groups, then fall
// into different banks. What bounds it is the latency of one CTA's copies and epilogue, so
// CTAs an SM count: 65,536 pixels take 10.5 us, 30 with the im2col copy (ncu, cold caches).
//
// The B operand, packed by pack_weights_kernel: element (row r, k) of [32 x 288] lives at
// byte ((r/8)*36 + k/8)*128 + (r%8)*16 + (k%8)*2, core matrices adjacent along K +128 B
// (LBO), along rows +36*128 B (SBO).
//
// conv3x3_ref_kernel computes the same thing on CUDA cores, one output value per
// thread; it is the checked reference for the tensor-core kernel and a fallback for
// debugging only.
//
// No counterpart in the reference (it has no learned component).

#include <cuda_bf16.h>
#include <algorithm>
#include <cuda_runtime.h>

#include "../../include/fluid2d_gb300.h"
#include "fs_internal.cuh"
#include "tc.cuh"

namespace fs {
namespace {

constexpr int kC = 32;             // channels
constexpr int kK = 9 * kC;         // GEMM K = 288
constexpr int kKC = kK / 8;        // core matrices along K = 36
constexpr int kTileM = 128;        // slots per CTA
constexpr int kBand = kTileM + 2;  // slots of a band
constexpr int kPlane = 16 * kBand;        // bytes of a band's channel group: 32 modulo 128
constexpr int kAbytes = 12 * kPlane;      // 24960
constexpr int kBbytes = kC * kK * 2;      // 18432
static_assert(kPlane % 128 == 32, "8 slots x 4 channel groups in different banks");
constexpr int kConvSmem = kAbytes + kBbytes + 64;
constexpr uint32_t kWaitLimit = 1u << 22;

struct ConvArgs {
    const __nv_bfloat16* x;    // input NHWC, 32 channels: (H x W), or (H/2 x W/2) when up
    const __nv_bfloat16* wpk;  // packed weights, 32 x 288 in the core-matrix layout
    const float* bias;         // 32 (nullable)
    const __nv_bfloat16* skip; // NHWC H x W x 32 added before the activation (nullable)
    __nv_bfloat16* y;          // output NHWC H x W x 32 (nullable)
    float* yf;                 // output FP32 H x W x 32 (nullable)
    int H, W;                  // output size (H = images x img_h rows)
    int img_h;                 // rows per image: zero padding applies at image borders
    int up;                    // 1: the input is nearest-upsampled by 2 on the fly
    int relu;
    int* err;                  // set to 1 if an mbarrier wait gave up
    const int* skip_if;        // nullable: when *skip_if != 0 the launch does nothing
    const __nv_bfloat16* mask; // nullable: outputs are zero where it (NHWC H x W x 32) is not positive
};

// Slots s (rows of W + 2) near slot `first`: row y and border column xp (pixel xp - 1) of
// slot first + k for k >= -1, without a 64-bit division per slot.
struct SlotRow {
    long y;   // row (-1 or >= H outside)
    int ly;   // row within its image
    int xp;
};
struct SlotBase {
    long y0;
    int ly0, xp0, W2, img_h;
    __device__ __forceinline__ SlotBase(long first, int W, int img_h_) {
        W2 = W + 2;
        img_h = img_h_;
        y0 = first / W2;
        xp0 = (int)(first - y0 * W2);
        ly0 = (int)(y0 % img_h);
    }
    __device__ __forceinline__ SlotRow at(int k) const {
        const unsigned t = (unsigned)(xp0 + k + W2), d = t / (unsigned)W2;  // one row up, to stay positive
        SlotRow r;
        r.xp = (int)(t - d * (unsigned)W2);
        r.y = y0 + (long)d - 1;
        r.ly = (int)((unsigned)(ly0 + (int)d + img_h - 1) % (unsigned)img_h);
        return r;
    }
};

// Copies the 16 bytes of channel group g of the pixels above, at and below slot r (dy = 0,
// 1, 2) to dst + dy*4*kPlane; zeros outside the image. Images of img_h rows are stacked
// along y; with `up` the input has img_h/2 rows per image and W/2 columns.
__device__ __forceinline__ void stage_taps(uint8_t* dst, const __nv_bfloat16* x, const SlotRow& r, int H, int W,
                                           int img_h, int up, int g) {
    const int ix = r.xp - 1;
    const bool col = ix >= 0 && ix < W && r.y >= 0 && r.y < H;
#pragma unroll
    for (int dy = 0; dy < 3; ++dy) {
        const int ly = r.ly + dy - 1;
        const bool in = col && ly >= 0 && ly < img_h;
        const long iy = r.y + dy - 1;
        const long src = up ? (iy >> 1) * (W >> 1) + (ix >> 1) : iy * W + ix;
        tc::cp_async16(dst + dy * 4 * kPlane, x + (in ? src * kC + g * 8 : 0), in ? 16u : 0u);
    }
}

// Source pixel of tap (dy, dx) for output pixel (y, x), or -1 outside its image.
// Images of img_h rows are stacked along y; with `up` the input has img_h/2 rows per
// image and W/2 columns, so the source row (y+dy)/2 stays inside the same image.
__device__ __forceinline__ long tap_source(const ConvArgs& P, int y, int x, int dy, int dx) {
    const int ly = y % P.img_h + dy, ix = x + dx;
    if (ly < 0 || ly >= P.img_h || ix < 0 || ix >= P.W) return -1;
    const int iy = y + dy;
    if (P.up) return (long)(iy >> 1) * (P.W >> 1) + (ix >> 1);
    return (long)iy * P.W + ix;
}

__device__ __forceinline__ void epilogue_store(const ConvArgs& P, long p, float (&v)[32]) {
    if (P.bias) {
#pragma unroll
        for (int c = 0; c < kC; ++c) v[c] += __ldg(P.bias + c);
    }
    if (P.skip) {
        const uint4* s = reinterpret_cast<const uint4*>(P.skip + p * kC);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint4 w = __ldg(s + q);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float2 f = __bfloat1622float2(h[e]);
                v[q * 8 + 2 * e] += f.x;
                v[q * 8 + 2 * e + 1] += f.y;
            }
        }
    }
    if (P.relu) {
#pragma unroll
        for (int c = 0; c < kC; ++c) v[c] = fmaxf(v[c], 0.f);
    }
    if (P.mask) {
        const uint4* s = reinterpret_cast<const uint4*>(P.mask + p * kC);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint4 w = __ldg(s + q);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h[e]);
                if (!(f.x > 0.f)) v[q * 8 + 2 * e] = 0.f;
                if (!(f.y > 0.f)) v[q * 8 + 2 * e + 1] = 0.f;
            }
        }
    }
    if (P.y) {
        uint4* o = reinterpret_cast<uint4*>(P.y + p * kC);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            uint4 w;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&w);
#pragma unroll
            for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(v[q * 8 + 2 * e], v[q * 8 + 2 * e + 1]);
            o[q] = w;
        }
    }
    if (P.yf) {
        float4* o = reinterpret_cast<float4*>(P.yf + p * kC);
#pragma unroll
        for (int q = 0; q < 8; ++q) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
}

__global__ void __launch_bounds__(128) conv3x3_tc_kernel(const ConvArgs P) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t* As = sm;
    uint8_t* Bs = sm + kAbytes;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kAbytes + kBbytes);
    uint32_t* s_taddr = reinterpret_cast<uint32_t*>(sm + kAbytes + kBbytes + 16);
    if (P.skip_if && __ldcg(P.skip_if)) return;  // uniform across the CTA, before any TMEM use
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long p0 = (long)blockIdx.x * kTileM;
    const SlotBase base(p0, P.W, P.img_h);

    if (warp == 0) {
        tc::tmem_alloc(s_taddr, 32);
        tc::tmem_relinquish();
    }
    if (tid == 0) tc::mbar_init(bar, 1);

    // B: 32 rows x 36 core-matrix columns, already packed in this layout
    for (int c = tid; c < kC * kKC; c += 128) tc::cp_async16(Bs + c * 16, P.wpk + c * 8, 16);
    // A: a row below the last image starts the next one or lies outside; a row of the band
    // above or below is the slot's own row -1 or +1, so that one slot gives three copies
    for (int q = tid; q < 4 * kBand; q += 128)
        stage_taps(As + (q & 3) * kPlane + (q >> 2) * 16, P.x, base.at((q >> 2) - 1), P.H, P.W, P.img_h, P.up, q & 3);
    tc::cp_async_wait_all();
    tc::fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t taddr = *s_taddr;

    if (tid == 0) {
        const uint32_t a0 = tc::smem_u32(As), b0 = tc::smem_u32(Bs);
        constexpr uint32_t idesc = tc::idesc_bf16_f32(128, 32);
#pragma unroll
        for (int kk = 0; kk < kK / 16; ++kk) {
            const int t = kk >> 1, dy = t / 3, dx = t - 3 * dy;
            const uint64_t ad = tc::smem_desc(a0 + (4 * dy + 2 * (kk & 1)) * kPlane + dx * 16, kPlane, 128);
            const uint64_t bd = tc::smem_desc(b0 + kk * 256, 128, kKC * 128);
            tc::mma_bf16(taddr, ad, bd, idesc, kk > 0);
        }
        tc::commit_to(bar);
    }
    // Bounded wait for the MMAs. Tensor memory is read and freed only after the commit
    // has arrived, since an MMA still in flight writes it (and reads the shared-memory
    // operands). If the first bound runs out the CTA flags the error, skips the
    // epilogue, and waits once more with the same bound before freeing; a CTA whose
    // warp 0 never sees the arrival leaves the allocation in place rather than free
    // columns an MMA may still write (the host treats the flagged error as fatal for
    // the network).
    auto wait_commit = [&]() {
        uint32_t spins = 0;
        while (!tc::mbar_try_wait(bar, 0))
            if (++spins > kWaitLimit) return false;
        return true;
    };
    bool arrived = wait_commit();
    if (!arrived && P.err) atomicOr(P.err, 1);
    tc::fence_after_sync();
    if (__all_sync(0xffffffffu, arrived)) {
        float v[32];
        tc::tmem_ld_32x32(taddr + ((uint32_t)(warp * 32) << 16), v);
        const SlotRow r = base.at(warp * 32 + lane);
        if (r.y < P.H && r.xp >= 1 && r.xp <= P.W) epilogue_store(P, r.y * P.W + (r.xp - 1), v);
    } else {
        arrived = wait_commit();
    }
    const bool free_ok = __all_sync(0xffffffffu, arrived);

    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0 && free_ok) tc::tmem_dealloc(taddr, 32);
}

// Reference: one thread per (pixel, output channel), FP32 accumulation of BF16 values.
__global__ void __launch_bounds__(256) conv3x3_ref_kernel(const ConvArgs P, const float* __restrict__ w32) {
    if (P.skip_if && __ldcg(P.skip_if)) return;
    const long npix = (long)P.H * P.W;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npix) return;
    const int y = (int)(i / P.W), x = (int)(i - (long)y * P.W);
    float v[32];
    for (int co = 0; co < kC; ++co) {
        float acc = 0.f;
        for (int t = 0; t < 9; ++t) {
            const long src = tap_source(P, y, x, t / 3 - 1, t % 3 - 1);
            if (src < 0) continue;
            for (int ci = 0; ci < kC; ++ci) {
                const float a = __bfloat162float(P.x[src * kC + ci]);
                const float b = __bfloat162float(__float2bfloat16_rn(w32[(co * 9 + t) * kC + ci]));
                acc = fmaf(a, b, acc);
            }
        }
        v[co] = acc;
    }
    epilogue_store(P, i, v);
}

// ------------------------------------------------------------- weight gradient
// wgrad_tc_kernel: dW[co][t][ci] = sum_p dz[p][co] * x(p, tap t)[ci] and db[co] =
// sum_p dz[p][co] as an implicit GEMM on the tensor cores with the pixels as the reduction
// dimension, in the slot numbering of conv3x3_tc_kernel (dz is zero in a border slot). Both
// operands are used as they lie in memory, channels contiguous, that is MN-major: for the
// tap column dx the rows of A are three bands x 32 channels of slots dx onward (rows 32*dy +
// ci), row 96 is all ones (its product is db) and rows 97..127 are zero; B is the 32
// channels of dz. So one M = 128 tile per dx, three 32-column FP32 accumulators in tensor
// memory. A core matrix of 8 channels x 8 slots is 128 contiguous bytes, the next 8 slots
// 128 bytes on (LBO), the next 8 channels one plane on (SBO). Each CTA reduces a contiguous
// range of slots in chunks of 128 (eight K = 16 MMAs per tile), double-buffered: the copies
// of chunk s + 1 run while chunk s is multiplied. The CTA writes its 289 x 32 partial sums
// to a workspace and wgrad_reduce_kernel adds the CTAs' partials in a fixed order, so the
// gradient is deterministic. The product of a border slot's zero gradient with the pixel next
// to it is zero unless that pixel is not finite; NaN in a row that has such products (dx = 0
// and 2) is therefore summed again over the pixels alone (wgrad_row_again).
// 65,536 pixels: 13.3 us (ncu, cold caches; 25 us where the threads loaded the nine taps of 64 pixels at a
// time and transposed them), bound by the latency of a CTA's two to four chunks.
constexpr int kWgK = kTileM;               // slots per chunk
constexpr int kWgAbytes = 16 * kPlane;     // three bands, the ones, zeros
constexpr int kWgStage = kWgAbytes + 4 * kPlane;
constexpr int kWgSmem = 2 * kWgStage + 64;
constexpr int kWgOut = 289;                // rows of the partial result (288 weights + bias)
constexpr int kWgThreads = 256;            // 8 warps; two CTAs per SM (shared memory and TMEM allow it)

struct WgradArgs {
    const __nv_bfloat16* x;   // layer input NHWC (as in ConvArgs, `up` for nearest-upsampled)
    const __nv_bfloat16* dz;  // BF16 gradient at the layer output, NHWC H x W x 32
    float* work;              // [gridDim.x][289][32] partial sums
    int H, W, img_h, up;
    int per;                  // slots per CTA (a multiple of kWgK)
    int* err;
};

// The NaN of one row (tap dy, dx and channel ci) of a CTA's partial result, summed once more
// over the pixels of slots [pbeg, pend) in order, until the sum is NaN for good.
__device__ __noinline__ void wgrad_row_again(const WgradArgs& P, float* out, int dy, int dx, int ci, long pbeg,
                                             long pend) {
    for (int c = 0; c < kC; ++c) {
        if (!isnan(out[c])) continue;
        float acc = 0.f;
        for (long s = pbeg; s < pend && !isnan(acc); ++s) {
            const long y = s / (P.W + 2);
            const int xx = (int)(s - y * (P.W + 2)) - 1;
            if (xx < 0 || xx >= P.W) continue;
            const int ly = (int)(y % P.img_h) + dy - 1, ix = xx + dx - 1;
            const long iy = y + dy - 1, src = P.up ? (iy >> 1) * (P.W >> 1) + (ix >> 1) : iy * P.W + ix;
            const bool in = ly >= 0 && ly < P.img_h && ix >= 0 && ix < P.W;
            const float x = in ? __bfloat162float(P.x[src * kC + ci]) : 0.f;
            acc = fmaf(x, __bfloat162float(P.dz[(y * P.W + xx) * kC + c]), acc);
        }
        out[c] = acc;
    }
}

__global__ void __launch_bounds__(kWgThreads) wgrad_tc_kernel(const WgradArgs P) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + 2 * kWgStage);  // one per buffer
    uint32_t* s_taddr = reinterpret_cast<uint32_t*>(sm + 2 * kWgStage + 32);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const long nslots = (long)P.H * (P.W + 2);
    const long pbeg = (long)blockIdx.x * P.per;
    const long pend = min(nslots, pbeg + (long)P.per);
    const int nchunks = pbeg < pend ? (int)((pend - pbeg + kWgK - 1) / kWgK) : 0;

    if (warp == 0) {
        tc::tmem_alloc(s_taddr, 128);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        tc::mbar_init(bar, 1);
        tc::mbar_init(bar + 1, 1);
    }
    // planes 12..15 of both A buffers: channel 0 of plane 12 all ones, the rest zero; the
    // staging below never writes them
    for (int e = tid; e < 2 * 4 * kBand; e += kWgThreads) {
        const int b = e / (4 * kBand), k = e - b * (4 * kBand);
        *reinterpret_cast<uint4*>(sm + b * kWgStage + 12 * kPlane + 16 * k) =
            make_uint4(k < kBand ? 0x00003F80u : 0u, 0, 0, 0);
    }

    // Chunk s: the three bands of its slots and one on either side, and dz of its slots,
    // zero at the border columns and from pend on (whose slots belong to the next CTA).
    auto stage = [&](int s) {
        uint8_t* const As = sm + (s & 1) * kWgStage;
        const long c0 = pbeg + (long)s * kWgK;
        const SlotBase base(c0, P.W, P.img_h);
        const int g = tid & 3, left = (int)min((long)kWgK, pend - c0);
        for (int k = tid >> 2; k < kBand; k += kWgThreads / 4) {
            const SlotRow r = base.at(k - 1);
            stage_taps(As + g * kPlane + k * 16, P.x, r, P.H, P.W, P.img_h, P.up, g);
            if (k >= 1 && k <= kWgK) {
                const bool in = r.xp >= 1 && r.xp <= P.W && k <= left;
                tc::cp_async16(As + kWgAbytes + g * kPlane + (k - 1) * 16,
                               P.dz + (in ? (r.y * P.W + (r.xp - 1)) * kC + g * 8 : 0), in ? 16u : 0u);
            }
        }
        tc::cp_async_commit();
    };
    auto wait_bar = [&](uint64_t* b, uint32_t parity) {
        uint32_t spins = 0;
        while (!tc::mbar_try_wait(b, parity))
            if (++spins > kWaitLimit) return false;
        return true;
    };
    bool ok = true;
    int last_issued = -1;  // last chunk whose MMAs were committed
    uint32_t taddr = 0;
    if (nchunks > 0) stage(0);
    for (int s = 0; s < nchunks; ++s) {
        if (s + 1 < nchunks) {
            if (s >= 1) {  // the MMAs of chunk s - 1 read the buffer of chunk s + 1
                const bool got = wait_bar(bar + ((s - 1) & 1), (uint32_t)((s - 1) >> 1) & 1u);
                ok = __syncthreads_and(got) != 0;
                if (!ok) break;
            }
            stage(s + 1);
            tc::cp_async_wait<1>();
        } else {
            tc::cp_async_wait<0>();
        }
        tc::fence_proxy_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        taddr = *s_taddr;
        if (tid == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16_f32_mn(128, 32);
            const uint32_t a0 = tc::smem_u32(sm + (s & 1) * kWgStage), b0 = a0 + kWgAbytes;
#pragma unroll
            for (int dx = 0; dx < 3; ++dx)
#pragma unroll
                for (int kk = 0; kk < kWgK / 16; ++kk) {
                    const uint64_t ad = tc::smem_desc(a0 + dx * 16 + kk * 256, 128, kPlane);
                    const uint64_t bd = tc::smem_desc(b0 + kk * 256, 128, kPlane);
                    tc::mma_bf16(taddr + dx * 32, ad, bd, idesc, s > 0 || kk > 0);
                }
            tc::commit_to(bar + (s & 1));
        }
        last_issued = s;
    }
    tc::cp_async_wait<0>();
    // The last commit covers every MMA this CTA issued. Tensor memory is read and freed
    // only after it has arrived; a CTA that gives up waiting (here, or for a buffer in
    // the loop) flags the error, skips the epilogue, and keeps its allocation unless
    // the last commit arrives after all, rather than free columns an MMA may still write.
    bool arrived = true;
    if (last_issued >= 0) arrived = wait_bar(bar + (last_issued & 1), (uint32_t)(last_issued >> 1) & 1u);
    tc::fence_before_sync();
    const bool all_arrived = __syncthreads_and(arrived) != 0;
    if ((!ok || !all_arrived) && tid == 0 && P.err) atomicOr(P.err, 1);
    tc::fence_after_sync();
    taddr = *s_taddr;
    if (ok && all_arrived) {
        float* out = P.work + (size_t)blockIdx.x * kWgOut * kC;
        // warp w reads tensor-memory lanes 32*(w%4).. of the tiles dx = w/4, w/4 + 2: lane
        // quarter dy is band dy (weights of tap 3*dy + dx), quarter 3's first lane the bias
        const int dy = warp & 3;
#pragma unroll 1
        for (int dx = warp >> 2; dx < 3; dx += kWgThreads / 128) {
            float v[32];
            if (nchunks > 0) {
                tc::tmem_ld_32x32(taddr + ((uint32_t)(dy * 32) << 16) + dx * 32, v);
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) v[c] = 0.f;
            }
            const int f = dy < 3 ? (3 * dy + dx) * kC + lane : dx == 0 && lane == 0 ? kK : kWgOut;
            if (f < kWgOut) {
                float4* o = reinterpret_cast<float4*>(out + (size_t)f * kC);
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
            bool nan = false;
#pragma unroll
            for (int c = 0; c < 32; ++c) nan |= isnan(v[c]);
            if (nan && dx != 1 && f < kK) wgrad_row_again(P, out + (size_t)f * kC, dy, dx, lane, pbeg, pend);
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0 && all_arrived) tc::tmem_dealloc(taddr, 128);
}

// dw[co][f] += sum over CTAs of work[cta][f][co] (f < 288); db[co] += the f = 288 row. A
// block per f: its warps sum every sixteenth partial each, and their sums are added in
// order (5.2 us for 272 partials; 12.4 us for 256 where one thread added all of them).
constexpr int kRedWarps = 16;
__global__ void __launch_bounds__(32 * kRedWarps) wgrad_reduce_kernel(const float* __restrict__ work, int nblocks,
                                                                      float* __restrict__ dw, float* __restrict__ db) {
    __shared__ float part[kRedWarps][kC];
    const int f = blockIdx.x, co = threadIdx.x & 31, w = threadIdx.x >> 5;
    float s = 0.f;
#pragma unroll 8
    for (int b = w; b < nblocks; b += kRedWarps) s += __ldcg(work + ((size_t)b * kWgOut + f) * kC + co);
    part[w][co] = s;
    __syncthreads();
    if (w != 0) return;
#pragma unroll
    for (int k = 1; k < kRedWarps; ++k) s += part[k][co];
    if (f < kK)
        dw[co * kK + f] += s;
    else if (db)
        db[co] += s;
}

// ------------------------------------------------------------- fused inference
// net_infer32_kernel: the whole 8-layer network on one 32 x 32 grid in one CTA (one CTA
// per image of a batch): e1 = conv(x0) -> pool -> e2, e3 (16 x 16) -> pool -> b1, b2
// (8 x 8) -> d1 = conv(up b2) + e3 -> d2 = conv(up d1) + e1 -> out = conv(d2), the same
// layer sequence and arithmetic as the per-layer launches of conv3x3_tc_kernel.
//
// Activations stay in shared memory, one buffer per level, in a zero-padded layout
// that makes every 3x3 tap a plain shifted operand, so no im2col copy is made: the
// (g+2) x (g+2) padded pixels of a level are numbered m = py*(g+2) + px, preceded by
// g+3 and followed by enough zero slots that every shifted read stays inside, and
// channel group c/8 of slot k lives at plane (c/8) * PL + k*16 bytes (PL = plane
// stride). Rows m..m+127 of the A operand for tap (dy, dx) are then slots m + dy*(g+2)
// + dx onward: one K-major no-swizzle descriptor with 16-byte rows (SBO = 128 B between
// 8-row groups, LBO = PL between channel groups). The GEMM runs over all padded pixels
// (border outputs are computed and dropped), 18 MMAs (9 taps x K = 32) per 128-pixel
// tile, every tile of a layer in its own 32 columns of tensor memory (10 tiles = 320
// columns at 32 x 32). All MMAs of a layer complete before its epilogue writes, so each
// layer writes its output over its input; the skip of layer 5 (e3) is kept in a
// separate shared buffer and that of layer 6 (e1) in global memory. Pooling and
// upsampling move data between the level buffers; only interior pixels are written,
// so the borders stay zero.
// Bound by the latency of eight dependent layers in one CTA: 57 us (67 with each layer's
// weights fetched when its turn came, 8 warps and pooling one channel at a time).
constexpr int kInfG = 32;
constexpr int kInfThreads = 512;
struct InfLevel {
    int g, P, npad, tiles, guard, slots, PL, bytes;
};
__host__ __device__ constexpr InfLevel inf_level(int g) {
    return InfLevel{g,
                    g + 2,
                    (g + 2) * (g + 2),
                    ((g + 2) * (g + 2) + 127) / 128,
                    g + 3,
                    (g + 3) + ((g + 2) * (g + 2) + 127) / 128 * 128 + (g + 3),
                    16 * ((g + 3) + ((g + 2) * (g + 2) + 127) / 128 * 128 + (g + 3)),
                    4 * 16 * ((g + 3) + ((g + 2) * (g + 2) + 127) / 128 * 128 + (g + 3))};
}
constexpr InfLevel kL0 = inf_level(kInfG), kL1 = inf_level(kInfG / 2), kL2 = inf_level(kInfG / 4);
constexpr int kInfWOff = 0;                           // packed weights of the current and the next layer
constexpr int kInfB0 = kInfWOff + 2 * kBbytes;        // level buffers
constexpr int kInfB1 = kInfB0 + kL0.bytes;
constexpr int kInfB2 = kInfB1 + kL1.bytes;
constexpr int kInfE3 = kInfB2 + kL2.bytes;            // e3, NHWC 16 x 16 x 32
constexpr int kInfBar = kInfE3 + (kInfG / 2) * (kInfG / 2) * kC * 2;
constexpr int kInfSmem = kInfBar + 64;
static_assert(kL0.tiles * 32 <= 512, "tensor memory holds every tile of a layer");
static_assert(kInfSmem <= 227 * 1024, "fits one CTA's shared memory");
static_assert(kL0.PL % 16 == 0 && kL1.PL % 16 == 0 && kL2.PL % 16 == 0, "16-byte planes");

struct InferArgs {
    const __nv_bfloat16* x0;  // network input, B images of 32 x 32 x 32 (NHWC)
    const __nv_bfloat16* wpk; // 8 layers x 9216 packed weights
    const float* params;      // FP32 parameters, layer li's bias at li*9248 + 9216
    __nv_bfloat16* e1;        // scratch, B x 32 x 32 x 32: the skip of layer 6
    float* y;                 // output, B x 32 x 32 x 32 FP32
    int* err;
    const int* skip_if;
};

// 16 bytes (8 channels) of slot k, channel group cg, in a level buffer
__device__ __forceinline__ uint4* inf_slot(uint8_t* buf, const InfLevel L, int k, int cg) {
    return reinterpret_cast<uint4*>(buf + cg * L.PL + k * 16);
}
__device__ __forceinline__ int inf_interior(const InfLevel L, int y, int x) {
    return L.guard + (y + 1) * L.P + (x + 1);
}

__global__ void __launch_bounds__(kInfThreads) net_infer32_kernel(const InferArgs A) {
    extern __shared__ __align__(1024) uint8_t sm[];
    if (A.skip_if && __ldcg(A.skip_if)) return;  // uniform, before any tensor-memory use
    uint8_t* Ws = sm + kInfWOff;
    uint8_t* B0 = sm + kInfB0;
    uint8_t* B1 = sm + kInfB1;
    uint8_t* B2 = sm + kInfB2;
    uint8_t* E3 = sm + kInfE3;
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kInfBar);
    uint32_t* s_taddr = reinterpret_cast<uint32_t*>(sm + kInfBar + 16);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int img = blockIdx.x;
    constexpr int G = kInfG;
    const __nv_bfloat16* x0 = A.x0 + (size_t)img * G * G * kC;
    __nv_bfloat16* e1g = A.e1 + (size_t)img * G * G * kC;
    float* yout = A.y + (size_t)img * G * G * kC;

    // a layer's weights to its buffer, one copy group (an empty one after the last layer)
    auto load_weights = [&](int li) {
        const __nv_bfloat16* src = A.wpk + (size_t)li * (kC * kK);
        if (li < 8)
            for (int c = tid; c < kC * kKC; c += kInfThreads) tc::cp_async16(Ws + (li & 1) * kBbytes + c * 16, src + c * 8, 16);
        tc::cp_async_commit();
    };
    load_weights(0);
    if (warp == 0) {
        tc::tmem_alloc(s_taddr, 512);
        tc::tmem_relinquish();
    }
    if (tid == 0) tc::mbar_init(bar, 1);
    // zero the level buffers (borders and guards stay zero), then the input's interior
    for (int e = tid; e < (kL0.bytes + kL1.bytes + kL2.bytes) / 16; e += kInfThreads)
        reinterpret_cast<uint4*>(B0)[e] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    for (int e = tid; e < G * G * 4; e += kInfThreads) {
        const int p = e >> 2, cg = e & 3;
        *inf_slot(B0, kL0, inf_interior(kL0, p / G, p % G), cg) =
            __ldg(reinterpret_cast<const uint4*>(x0 + (size_t)p * kC + cg * 8));
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t taddr = *s_taddr;

    auto pool = [&](uint8_t* src, const InfLevel Ls, uint8_t* dst, const InfLevel Ld) {
        // 2x2 average (avgpool2_kernel's order and rounding) into the next level, eight
        // channels at a time
        for (int e = tid; e < Ld.g * Ld.g * 4; e += kInfThreads) {
            const int p = e >> 2, cg = e & 3, Y = p / Ld.g, X = p % Ld.g;
            uint4 q[4], w;
#pragma unroll
            for (int k = 0; k < 4; ++k) q[k] = *inf_slot(src, Ls, inf_interior(Ls, 2 * Y + (k >> 1), 2 * X + (k & 1)), cg);
            const __nv_bfloat162(*h)[4] = reinterpret_cast<const __nv_bfloat162(*)[4]>(q);
            __nv_bfloat162* o = reinterpret_cast<__nv_bfloat162*>(&w);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                float2 s = __bfloat1622float2(h[0][c]);
#pragma unroll
                for (int k = 1; k < 4; ++k) {
                    const float2 f = __bfloat1622float2(h[k][c]);
                    s = make_float2(__fadd_rn(s.x, f.x), __fadd_rn(s.y, f.y));
                }
                o[c] = __floats2bfloat162_rn(__fmul_rn(0.25f, s.x), __fmul_rn(0.25f, s.y));
            }
            *inf_slot(dst, Ld, inf_interior(Ld, Y, X), cg) = w;
        }
    };
    auto upsample = [&](uint8_t* src, const InfLevel Ls, uint8_t* dst, const InfLevel Ld) {
        // nearest x2 into the interior of the finer level
        for (int e = tid; e < Ld.g * Ld.g * 4; e += kInfThreads) {
            const int p = e >> 2, cg = e & 3, y = p / Ld.g, x = p % Ld.g;
            *inf_slot(dst, Ld, inf_interior(Ld, y, x), cg) = *inf_slot(src, Ls, inf_interior(Ls, y >> 1, x >> 1), cg);
        }
    };

    bool ok = true;
    // layer li on the level buffer `buf` (input, overwritten by the output), with the
    // given skip source; out_kind 0: BF16 in place, 1: also e1 to global, 2: also e3 to
    // the skip buffer, 3: FP32 to the output (no ReLU)
    auto layer = [&](int li, uint8_t* buf, const InfLevel L, int skip_kind, int out_kind) {
        if (!ok) return;
        // the next layer's weights into the other buffer (the MMAs of the layer before, which
        // read it, are complete); this layer's are on their way since then
        load_weights(li + 1);
        tc::cp_async_wait<1>();
        tc::fence_proxy_async_smem();  // weights and the activations written by this CTA
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        if (tid == 0) {
            constexpr uint32_t idesc = tc::idesc_bf16_f32(128, 32);
            const uint32_t a0 = tc::smem_u32(buf), w0 = tc::smem_u32(Ws + (li & 1) * kBbytes);
            for (int T = 0; T < L.tiles; ++T) {
#pragma unroll
                for (int t = 0; t < 9; ++t) {
                    const int shift = (t / 3 - 1) * L.P + (t % 3 - 1);
                    const uint32_t row0 = (uint32_t)(L.guard + T * 128 + shift) * 16u;
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk) {
                        const uint64_t ad = tc::smem_desc(a0 + (uint32_t)(2 * kk * L.PL) + row0, L.PL, 128);
                        const uint64_t bd = tc::smem_desc(w0 + (uint32_t)(t * 2 + kk) * 256, 128, kKC * 128);
                        tc::mma_bf16(taddr + T * 32, ad, bd, idesc, t > 0 || kk > 0);
                    }
                }
            }
            tc::commit_to(bar);
        }
        uint32_t spins = 0;
        bool got = true;
        while (!tc::mbar_try_wait(bar, (uint32_t)(li & 1)))
            if (++spins > kWaitLimit) {
                got = false;
                break;
            }
        ok = __syncthreads_and(got) != 0;
        tc::fence_after_sync();
        if (!ok) return;
        const float* bias = A.params + (size_t)li * (kC * kK + kC) + kC * kK;
        // warp w reads tensor-memory lanes 32*(w%4).. of the tiles T = w/4, w/4 + 4, ...
        for (int T = warp >> 2; T < L.tiles; T += kInfThreads / 128) {
            float v[32];
            tc::tmem_ld_32x32(taddr + ((uint32_t)((warp & 3) * 32) << 16) + T * 32, v);
            const int m = T * 128 + (warp & 3) * 32 + lane;
            const int py = m / L.P, px = m - py * L.P;
            if (m >= L.npad || py < 1 || py > L.g || px < 1 || px > L.g) continue;
            const int y = py - 1, x = px - 1, k = L.guard + m;
#pragma unroll
            for (int c = 0; c < kC; ++c) v[c] += __ldg(bias + c);
            if (skip_kind) {
                const uint4* sp = skip_kind == 1 ? reinterpret_cast<const uint4*>(e1g + (size_t)(y * G + x) * kC)
                                                 : reinterpret_cast<const uint4*>(E3 + (y * (G / 2) + x) * kC * 2);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint4 w = skip_kind == 1 ? __ldcg(sp + q) : sp[q];
                    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __bfloat1622float2(h[e]);
                        v[q * 8 + 2 * e] += f.x;
                        v[q * 8 + 2 * e + 1] += f.y;
                    }
                }
            }
            if (out_kind == 3) {
                float4* o = reinterpret_cast<float4*>(yout + (size_t)(y * G + x) * kC);
#pragma unroll
                for (int q = 0; q < 8; ++q) o[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                continue;
            }
#pragma unroll
            for (int c = 0; c < kC; ++c) v[c] = fmaxf(v[c], 0.f);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint4 w;
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&w);
#pragma unroll
                for (int e = 0; e < 4; ++e) h[e] = __floats2bfloat162_rn(v[q * 8 + 2 * e], v[q * 8 + 2 * e + 1]);
                *inf_slot(buf, L, k, q) = w;
                if (out_kind == 1) reinterpret_cast<uint4*>(e1g + (size_t)(y * G + x) * kC)[q] = w;
                if (out_kind == 2) reinterpret_cast<uint4*>(E3 + (y * (G / 2) + x) * kC * 2)[q] = w;
            }
        }
        tc::fence_before_sync();
        __syncthreads();
    };

    layer(0, B0, kL0, 0, 1);  // e1
    if (ok) {
        pool(B0, kL0, B1, kL1);  // pool1
        __syncthreads();
    }
    layer(1, B1, kL1, 0, 0);  // e2
    layer(2, B1, kL1, 0, 2);  // e3 (+ skip copy)
    if (ok) {
        pool(B1, kL1, B2, kL2);  // pool2
        __syncthreads();
    }
    layer(3, B2, kL2, 0, 0);  // b1
    layer(4, B2, kL2, 0, 0);  // b2
    if (ok) {
        upsample(B2, kL2, B1, kL1);
        __syncthreads();
    }
    layer(5, B1, kL1, 2, 0);  // d1 = relu(conv(up b2) + b + e3)
    if (ok) {
        __threadfence_block();  // e1 stores to global by this CTA, read back in layer 6
        upsample(B1, kL1, B0, kL0);
        __syncthreads();
    }
    layer(6, B0, kL0, 1, 0);  // d2 = relu(conv(up d1) + b + e1)
    layer(7, B0, kL0, 0, 3);  // out
    tc::cp_async_wait<0>();
    if (!ok && tid == 0 && A.err) atomicOr(A.err, 1);
    // every MMA was waited for, unless a wait gave up: then keep the allocation rather
    // than free columns an MMA may still write
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0 && ok) tc::tmem_dealloc(taddr, 512);
}

// FP32 weights [co][tap][ci] (32 x 9 x 32) -> BF16 B operand in the core-matrix layout.
__global__ void pack_weights_kernel(const float* __restrict__ w32, __nv_bfloat16* __restrict__ wpk) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;  // one element
    if (e >= kC * kK) return;
    const int n = e / kK, k = e - n * kK;
    const int off = ((n >> 3) * kKC + (k >> 3)) * 64 + (n & 7) * 8 + (k & 7);  // in BF16 elements
    wpk[off] = __float2bfloat16_rn(w32[e]);
}

// The three forms of every layer's weights that a training step needs, one launch for all
// layers (blockIdx.y) of the parameters: packed, flipped for the backward-data convolution
// (w'[ci][8 - t][co] = w[co][t][ci]) and the flipped ones packed.
__global__ void pack_layers_kernel(const float* __restrict__ params, int stride, __nv_bfloat16* __restrict__ wpk,
                                   float* __restrict__ wflip, __nv_bfloat16* __restrict__ wflip_pk) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= kC * kK) return;
    const size_t l = blockIdx.y, lo = l * (kC * kK);
    const float w = params[l * stride + e];
    auto off = [](int n, int k) { return ((n >> 3) * kKC + (k >> 3)) * 64 + (n & 7) * 8 + (k & 7); };
    const int n = e / kK, k = e - n * kK, ci = k & (kC - 1), kf = (8 - k / kC) * kC + n;
    wpk[lo + off(n, k)] = __float2bfloat16_rn(w);
    wflip[lo + ci * kK + kf] = w;
    wflip_pk[lo + off(ci, kf)] = __float2bfloat16_rn(w);
}

}  // namespace
}  // namespace fs

using namespace fs;

// Opt the tensor-core kernels into their dynamic shared memory on the current device.
cudaError_t fs::conv_prepare() {
    cudaError_t e = cudaFuncSetAttribute(conv3x3_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kConvSmem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(net_infer32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kInfSmem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem);
}

int fs::net_infer32_launch(const void* x0, const void* wpk, const float* params, void* e1, float* y, int images,
                           int* err, const int* skip_if, void* stream) {
    if (!x0 || !wpk || !params || !e1 || !y || images < 1)
        return record_error(FS_ERR_ARG, "fs_net_infer32: bad argument");
    int dev = 0;
    cudaGetDevice(&dev);
    static unsigned long long configured = 0;
    if (!(configured & (1ull << (dev & 63)))) {
        if (cudaFuncSetAttribute(net_infer32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kInfSmem) !=
            cudaSuccess)
            return record_error(FS_ERR_CUDA, "fs_net_infer32: smem attribute");
        configured |= 1ull << (dev & 63);
    }
    InferArgs A;
    A.x0 = static_cast<const __nv_bfloat16*>(x0);
    A.wpk = static_cast<const __nv_bfloat16*>(wpk);
    A.params = params;
    A.e1 = static_cast<__nv_bfloat16*>(e1);
    A.y = y;
    A.err = err;
    A.skip_if = skip_if;
    net_infer32_kernel<<<images, kInfThreads, kInfSmem, (cudaStream_t)stream>>>(A);
    return cudaGetLastError() == cudaSuccess ? FS_OK : record_error(FS_ERR_CUDA, "fs_net_infer32: launch failed");
}

extern "C" int fs_net_infer32(const void* x0, const void* wpk, const float* params, void* e1, float* y, int images,
                              int* err, void* stream) {
    return fs::net_infer32_launch(x0, wpk, params, e1, y, images, err, nullptr, stream);
}

extern "C" long long fs_net_weight_grad_tc_work_floats(int H, int W) {
    (void)H;
    (void)W;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 1;
    return 2LL * sms * kWgOut * kC;
}

extern "C" int fs_net_weight_grad_tc(const void* dzb, const void* x, float* dw, float* db, float* work,
                                     long long work_floats, int H, int W, int img_h, int up, int* err, void* stream) {
    if (!dzb || !x || !dw || !work || H < 1 || W < 1) return record_error(FS_ERR_ARG, "fs_net_weight_grad_tc: bad argument");
    if (img_h <= 0) img_h = H;
    if (H % img_h != 0) return record_error(FS_ERR_ARG, "fs_net_weight_grad_tc: H must be a multiple of img_h");
    if (up && ((img_h & 1) || (W & 1)))
        return record_error(FS_ERR_ARG, "fs_net_weight_grad_tc: upsampled output must be even");
    const long long per_block = (long long)kWgOut * kC;
    const long long max_blocks = work_floats / per_block;
    // two CTAs per SM
    if (max_blocks < 1) return record_error(FS_ERR_ARG, "fs_net_weight_grad_tc: workspace too small");
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1) sms = 1;
    static unsigned long long configured = 0;
    if (!(configured & (1ull << (dev & 63)))) {
        if (cudaFuncSetAttribute(wgrad_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem) != cudaSuccess)
            return record_error(FS_ERR_CUDA, "fs_net_weight_grad_tc: smem attribute");
        configured |= 1ull << (dev & 63);
    }
    // two CTAs per SM at most, each over a whole number of chunks
    const long nslots = (long)H * (W + 2);
    const long chunks = (nslots + kWgK - 1) / kWgK;
    long nb = std::min<long>({2L * sms, chunks, (long)max_blocks});
    const long per = ((chunks + nb - 1) / nb) * kWgK;
    nb = (nslots + per - 1) / per;
    WgradArgs P;
    P.x = static_cast<const __nv_bfloat16*>(x);
    P.dz = static_cast<const __nv_bfloat16*>(dzb);
    P.work = work;
    P.H = H;
    P.W = W;
    P.img_h = img_h;
    P.up = up;
    P.per = (int)per;
    P.err = err;
    cudaStream_t st = (cudaStream_t)stream;
    wgrad_tc_kernel<<<(unsigned)nb, kWgThreads, kWgSmem, st>>>(P);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return record_error(FS_ERR_CUDA, "fs_net_weight_grad_tc: launch failed");
    wgrad_reduce_kernel<<<kWgOut, 32 * kRedWarps, 0, st>>>(work, (int)nb, dw, db);
    e = cudaGetLastError();
    return e == cudaSuccess ? FS_OK : record_error(FS_ERR_CUDA, "fs_net_weight_grad_tc: reduce launch failed");
}

extern "C" int fs_conv_pack_weights(const float* w32, void* wpk, void* stream) {
    if (!w32 || !wpk) return record_error(FS_ERR_ARG, "fs_conv_pack_weights: null pointer");
    pack_weights_kernel<<<(kC * kK + 255) / 256, 256, 0, (cudaStream_t)stream>>>(
        w32, static_cast<__nv_bfloat16*>(wpk));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FS_OK : record_error(FS_ERR_CUDA, "fs_conv_pack_weights: launch failed");
}

extern "C" int fs_net_pack_layers(const float* params, int layers, int stride, void* wpk, float* wflip,
                                  void* wflip_pk, void* stream) {
    if (!params || !wpk || !wflip || !wflip_pk || layers < 1 || layers > 65535 || stride < kC * kK)
        return record_error(FS_ERR_ARG, "fs_net_pack_layers: bad argument");
    pack_layers_kernel<<<dim3((kC * kK + 255) / 256, layers), 256, 0, (cudaStream_t)stream>>>(
        params, stride, static_cast<__nv_bfloat16*>(wpk), wflip, static_cast<__nv_bfloat16*>(wflip_pk));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FS_OK : record_error(FS_ERR_CUDA, "fs_net_pack_layers: launch failed");
}

extern "C" int fs_conv3x3(const void* x, const void* wpk, const float* w32, const float* bias, const void* skip,
                          void* y, float* yf, int H, int W, int img_h, int up, int relu, int use_tensor_cores,
                          int* err, void* stream) {
    return fs::conv3x3_launch(x, wpk, w32, bias, skip, y, yf, H, W, img_h, up, relu, use_tensor_cores, err, nullptr,
                              stream);
}

extern "C" int fs_conv3x3_relu_bwd(const void* dzb, const void* wpk_flip, const void* a, void* dzb_in, float* dz_in,
                                   int H, int W, int img_h, int* err, void* stream) {
    if (!dzb || !wpk_flip || !a || !dzb_in) return record_error(FS_ERR_ARG, "fs_conv3x3_relu_bwd: null pointer");
    return fs::conv3x3_launch(dzb, wpk_flip, nullptr, nullptr, nullptr, dzb_in, dz_in, H, W, img_h, 0, 0, 1, err,
                              nullptr, stream, a);
}

int fs::conv3x3_launch(const void* x, const void* wpk, const float* w32, const float* bias, const void* skip, void* y,
                       float* yf, int H, int W, int img_h, int up, int relu, int use_tensor_cores, int* err,
                       const int* skip_if, void* stream, const void* mask) {
    if (!x || H < 1 || W < 1 || (!y && !yf)) return record_error(FS_ERR_ARG, "fs_conv3x3: bad argument");
    if (img_h <= 0) img_h = H;
    if (H % img_h != 0) return record_error(FS_ERR_ARG, "fs_conv3x3: H must be a multiple of img_h");
    if (up && ((img_h & 1) || (W & 1))) return record_error(FS_ERR_ARG, "fs_conv3x3: upsampled output must be even");
    ConvArgs P;
    P.x = static_cast<const __nv_bfloat16*>(x);
    P.wpk = static_cast<const __nv_bfloat16*>(wpk);
    P.bias = bias;
    P.skip = static_cast<const __nv_bfloat16*>(skip);
    P.y = static_cast<__nv_bfloat16*>(y);
    P.yf = yf;
    P.H = H;
    P.W = W;
    P.img_h = img_h;
    P.up = up;
    P.relu = relu;
    P.err = err;
    P.skip_if = skip_if;
    P.mask = static_cast<const __nv_bfloat16*>(mask);
    cudaStream_t st = (cudaStream_t)stream;
    const long npix = (long)H * W;
    if (use_tensor_cores) {
        if (!wpk) return record_error(FS_ERR_ARG, "fs_conv3x3: packed weights required");
        static unsigned long long configured = 0;
        int dev = 0;
        cudaGetDevice(&dev);
        if (!(configured & (1ull << (dev & 63)))) {
            cudaError_t e = cudaFuncSetAttribute(conv3x3_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 kConvSmem);
            if (e != cudaSuccess) return record_error(FS_ERR_CUDA, "fs_conv3x3: smem attribute");
            configured |= 1ull << (dev & 63);
        }
        conv3x3_tc_kernel<<<(unsigned)(((long)H * (W + 2) + kTileM - 1) / kTileM), 128, kConvSmem, st>>>(P);
    } else {
        if (!w32) return record_error(FS_ERR_ARG, "fs_conv3x3: FP32 weights required");
        conv3x3_ref_kernel<<<(unsigned)((npix + 255) / 256), 256, 0, st>>>(P, w32);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FS_OK : record_error(FS_ERR_CUDA, "fs_conv3x3: launch failed");
}
