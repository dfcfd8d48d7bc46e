// Exact reproduction of the reference's host solver (fluid_solver_cpu, src/
// fluid_solver_cpu.cpp:6-215) on the GPU, for square grids up to gs_tiled_max_size().
//
// The host solver differs from the CUDA one in method, not just rounding: its
// diffusion and pressure sweeps update in place in row-major order (lexicographic
// Gauss-Seidel), every boundary fill also averages the four corners, the diffusion
// divisor is float, there is no smoothing, and the forward splat adds in raster order.
//
// Solves (gs_solve_kernel). Cell (i, j) of sweep s needs the new values above and to its
// left and the previous sweep's to its right and below, so a sweep is a chain of
// dependences through the grid, but sweeps can follow one another closely. The grid is cut
// into bands of 32 rows, one CTA per band and one warp per sweep: a lane owns a row and
// walks along the columns, lane l one column behind lane l - 1, so that
//   left:  the lane's value of the step before (a register);
//   above: the previous lane's value of the step before (a shuffle);
//   right, below: the previous sweep's values, from the band's array, which every sweep
//          updates in place; the value below comes from the next lane's load (a shuffle).
// Sweep s runs `lag` columns behind sweep s - 1 on the next warp, all warps in step: chunks
// of kChunk columns, a block barrier between them, a chunk's loads one chunk ahead of their
// use. The row above a band and the row below it come from the neighbouring bands' CTAs
// through global memory: each exported value is an 8-byte word {value, tag of the sweep},
// read until the tag is the expected one, so that no fence and no separate flag is needed; a
// word is overwritten only by a sweep that depends on its reader. Words are loaded two
// chunks before their use (a load of another SM's store takes longer than a chunk).
// Waits are bounded: a warp that gives up sets ctrl->error and the solve ends
// (FS_ERR_TIMEOUT on the host). All CTAs are co-resident (cooperative launch); a CTA with
// several bands takes every gridDim.x-th in turn, which cannot deadlock: a band's last sweep
// needs one sweep less of the band below, two less of the next, so at most as many bands as a
// launch has sweeps, and the lowest unfinished band and the gridDim.x - 1 after it are all
// under way (solve() keeps a launch's sweeps at or below the SMs, and so the CTAs).
//
// Grids whose bands all fit one SM's shared memory (up to 141 x 141) run in one CTA per
// field instead, bands side by side, so that nothing leaves the SM.
//
// What bounds it: the chain of bands, columns and sweeps, a chunk of eight columns after another,
// each as long as its slowest warp's instructions (ncu: the largest stall is the barrier behind
// a chunk, then waits for the own instructions before; schedulers issue in 51 % of the cycles
// with 24 warps in one CTA, in 27 % with 20), and from band to band the 32 columns of skew and
// a trip between SMs, 7 us in all. At 20/20 sweeps a step takes 0.41 ms at 130 x 130 (1.12 ms
// with a block barrier per anti-diagonal of one CTA) and 1.58 ms at 800 x 800 (21.0 ms with a
// grid barrier per diagonal of 64 x 64 tiles).
//
// The splat keeps the host solver's order of additions to every cell: a cell receives
// its contributions in the raster order of their source cells. Source cells are linked
// into one list per target, and a thread sorts the few that its cell receives; a cell that
// receives more gets a warp, or a CTA.
//
// Every operation uses explicitly rounded single-precision intrinsics so that no
// contraction changes a result; the outputs are bit-identical to the host solver's.

#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/fluid2d_gb300.h"
#include "fs_internal.cuh"

namespace fs {
namespace {

constexpr int kMaxWarps = 24;    // warps of a CTA; sweeps of one launch with a CTA per band
constexpr int kLine = 33;        // floats per line of a band's array: 32 lanes and a pad
constexpr int kChunk = 8;        // columns a warp advances between barriers
constexpr unsigned kGsPolls = 1u << 21;  // default bound of a wait, about 2 s

// One field of a solve. Diffusion: x + dt*src is both the start and the constant term;
// pressure: the constant term is the divergence of (u, v), the start zero. A later launch
// of the same solve (more than kMaxWarps sweeps) starts from `start`.
struct GsField {
    const float* x;
    const float* src;
    const float* u;
    const float* v;
    const float* start;  // null: the first launch
    float* out;
    float* big;  // global memory for the band arrays that shared memory does not hold
    int mode;
    float a, den, rden;
};

struct GsSolve {
    GsField f[3];
    int nf;
    int n, P, sweeps;
    int lag, band_lag;
    int bands;
    float dt, cdiv;
    unsigned epoch;                // distinguishes the tags of a step's launches
    unsigned long long* words;     // exported rows: [field][band][top, bottom][column]
    SolveCtrl* ctrl;
    const unsigned* poll_limit;
};

__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, float v, unsigned tag) {
    const unsigned long long w = ((unsigned long long)tag << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}

// x / b correctly rounded, y = RN(1/b): Markstein's correction step (P. Markstein, IBM J.
// Res. Dev. 34(1), 1990), exact for normal quotients and remainders; other x, and divisors
// outside (2^-20, 2^20) (y passed as zero), take the IEEE division.
__device__ __forceinline__ float gs_div(float x, float b, float y) {
    const float ax = fabsf(x);
    const float q0 = __fmul_rn(x, y);
    const float r = __fmaf_rn(-q0, b, x);
    const float q = ax == 0.f ? x : __fmaf_rn(r, y, q0);
    if (((ax <= 0x1p-100f || !(ax < 0x1p100f)) && ax != 0.f) || y == 0.f) return __fdiv_rn(x, b);
    return q;
}

// x + dt*s on an interior cell (fluid_solver_cpu.cpp:85-92).
__device__ __forceinline__ float gs_source(float x, float s, float dt) { return __fadd_rn(x, __fmul_rn(dt, s)); }

// Lines of a band's arrays: the columns, the lanes' skew, whole chunks.
__host__ __device__ inline int gs_lines(int m) { return (m + 31 + kChunk - 1) / kChunk * kChunk; }

// Where a band's arrays are: both in shared memory, the constant terms in global memory,
// both there. Value of row (lane) l in column j of either: line j + l, place l.
enum GsPlace { GS_SHARED = 0, GS_CONST_GLOBAL = 1, GS_GLOBAL = 2 };

template <bool DIFF, int PLACE>
struct GsBand {
    const GsSolve& S;
    const GsField& F;
    int xo, co;          // offsets of the arrays in shared memory
    float *xg, *cg;      // the arrays in global memory
    int band, m, lane, lm;  // lm: lane of the grid's last interior row (the last band), else 32
    bool top, bot;
    float s_lr, s_tb;

    __device__ __forceinline__ float& x(int line, int l) const {
        extern __shared__ float4 gs_smem[];
        const int k = line * kLine + l;
        return PLACE == GS_GLOBAL ? xg[k] : reinterpret_cast<float*>(gs_smem)[xo + k];
    }
    __device__ __forceinline__ float& c(int line, int l) const {
        extern __shared__ float4 gs_smem[];
        const int k = line * kLine + l;
        return PLACE == GS_SHARED ? reinterpret_cast<float*>(gs_smem)[co + k] : cg[k];
    }

    // The value a sweep 0 finds in grid cell (i, j).
    __device__ __forceinline__ float initial(int i, int j) const {
        const size_t o = (size_t)i * S.P + j;
        if (F.start) return __ldcg(F.start + o);
        if (!DIFF) return 0.f;
        const float v = __ldg(F.x + o);
        const bool in = i > 0 && i < S.n - 1 && j > 0 && j < S.n - 1;
        return in ? gs_source(v, __ldg(F.src + o), S.dt) : v;
    }

    // a value of the neighbouring band's last or first row (arrays of one CTA)
    __device__ __forceinline__ float x_above(int line) const { return x(line - (gs_lines(m) + 1), 31); }
    __device__ __forceinline__ float x_below(int line) const { return x(line + (gs_lines(m) + 1), 0); }

    // Load and store of the band by `parts` warps, this one the part-th.
    __device__ void load(int part, int parts) const {
        const int rows = min(32, m - band * 32);
        // one more row than the band's own: the edge row, where it has a lane to live in
        const int extra = bot && rows < 32 ? 1 : 0;
        for (int l = part; l < rows + extra; l += parts) {
            const int i = 1 + band * 32 + l;
            const size_t row = (size_t)i * S.P + 1;
#pragma unroll 4
            for (int j = lane; j < m; j += 32) {
                const float v = initial(i, 1 + j);
                x(j + l, l) = v;
                if (l >= rows) continue;
                const size_t o = row + j;
                if (DIFF) {
                    c(j + l, l) = F.start ? gs_source(__ldg(F.x + o), __ldg(F.src + o), S.dt) : v;
                } else {
                    // (-0.5*h) * (uR - uL + vD - vU), fluid_solver_cpu.cpp:186-191
                    float d = __fsub_rn(__ldg(F.u + o + 1), __ldg(F.u + o - 1));
                    d = __fadd_rn(d, __ldg(F.v + o + S.P));
                    d = __fsub_rn(d, __ldg(F.v + o - S.P));
                    c(j + l, l) = __fmul_rn(S.cdiv, d);
                }
            }
        }
    }

    // The band's final values with the host solver's fill (fluid_solver_cpu.cpp:33-83):
    // edges from their inner neighbours, corners the mean of their two edge neighbours.
    __device__ void store(int part, int parts) const {
        const int rows = min(32, m - band * 32), P = S.P, n = S.n;
        float* __restrict__ g = F.out;
        for (int l = part; l < rows; l += parts) {
            const int i = 1 + band * 32 + l;
            const bool it = i == 1, ib = i == n - 2;
#pragma unroll 4
            for (int j = lane; j < m; j += 32) {
                const float v = x(j + l, l);
                const size_t o = (size_t)i * P + 1 + j;
                g[o] = v;
                const float ex = __fmul_rn(s_lr, v), ey = __fmul_rn(s_tb, v);
                const bool jl = j == 0, jr = j == m - 1;
                if (jl) g[o - 1] = ex;
                if (jr) g[o + 1] = ex;
                if (it) g[o - P] = ey;
                if (ib) g[o + P] = ey;
                if ((it || ib) && (jl || jr)) {
                    const float q = __fmul_rn(0.5f, __fadd_rn(ey, ex));
                    if (it && jl) g[o - P - 1] = q;
                    if (it && jr) g[o - P + 1] = q;
                    if (ib && jl) g[o + P - 1] = q;
                    if (ib && jr) g[o + P + 1] = q;
                }
            }
        }
    }

    // The previous sweep's values one column to the right, and the constant terms, of lines
    // t0 .. t0 + kChunk - 1.
    __device__ __forceinline__ void lines_of(int t0, float (&xr)[kChunk], float (&cc)[kChunk]) const {
#pragma unroll
        for (int k = 0; k < kChunk; ++k) {
            xr[k] = x(t0 + k + 1, lane);
            cc[k] = c(t0 + k, lane);
        }
    }
};

// One chunk of one sweep: lines t0 .. t0 + kChunk - 1. xr: the previous sweep's values one
// column to the right; old: the one in line t0 before this sweep. inj: for lane 0 the values
// above its row, for lane 31 those below its row. RAMP: some lane is outside the columns or
// at an edge column. The fills of the domain's edges are known before the sweep's chain
// starts (sign x a value of the previous sweep), so they go into its inputs.
template <bool DIFF, int PLACE, bool RAMP>
__device__ __forceinline__ void gs_chunk(const GsBand<DIFF, PLACE>& B, bool first, int t0, float (&xr)[kChunk],
                                         const float (&cc)[kChunk], float (&inj)[kChunk], float& val, float& old,
                                         float l_edge, float r_edge, float a, float den, float rden) {
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = B.lane, m = B.m;
    const float next_old = xr[kChunk - 1];
    float below[kChunk], left[kChunk];
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
        below[k] = __shfl_down_sync(FULL, xr[k], 1);
        if (lane == 31) below[k] = inj[k];
    }
    if (!first) {
        if (B.top && lane == 0) {
#pragma unroll
            for (int k = 0; k < kChunk; ++k) inj[k] = __fmul_rn(B.s_tb, k > 0 ? xr[k > 0 ? k - 1 : 0] : old);
        }
        if (B.bot && lane == B.lm) {
#pragma unroll
            for (int k = 0; k < kChunk; ++k) below[k] = __fmul_rn(B.s_tb, k > 0 ? xr[k > 0 ? k - 1 : 0] : old);
        }
    }
    if (RAMP) {
#pragma unroll
        for (int k = kChunk - 1; k >= 0; --k) {
            const float e = __fmul_rn(B.s_lr, k > 0 ? xr[k > 0 ? k - 1 : 0] : old);
            left[k] = first ? l_edge : e;
            if (t0 + k - lane == m - 1) xr[k] = first ? r_edge : e;
        }
    }
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
        const int j = t0 + k - lane;
        float U = __shfl_up_sync(FULL, val, 1);
        if (lane == 0) U = inj[k];
        float L = val;
        if (RAMP && j == 0) L = left[k];
        float v;
        if (DIFF) {  // (x0 + a*(U + D + L + R)) / (1 + 4a), fluid_solver_cpu.cpp:107-108
            float sum = __fadd_rn(U, below[k]);
            sum = __fadd_rn(sum, L);
            sum = __fadd_rn(sum, xr[k]);
            v = gs_div(__fadd_rn(cc[k], __fmul_rn(a, sum)), den, rden);
            // cells outside the columns write places no valid cell reads; zero keeps them
            // from decaying into the slow division
            if (RAMP && (unsigned)j >= (unsigned)m) v = 0.f;
        } else {  // (div + R + L + D + U) / 4, fluid_solver_cpu.cpp:199-200
            float sum = __fadd_rn(cc[k], xr[k]);
            sum = __fadd_rn(sum, L);
            sum = __fadd_rn(sum, below[k]);
            sum = __fadd_rn(sum, U);
            v = __fmul_rn(sum, 0.25f);
        }
        val = v;
        B.x(t0 + k, lane) = v;
    }
    old = next_old;
}

// ONE: a CTA holds all bands of a field, blockDim / 32 / bands sweeps of each in flight (a
// warp takes every such sweep in turn), and neighbouring bands read each other's arrays.
// Otherwise a CTA holds one band and a warp per sweep. Lags: columns between sweeps, and
// (ONE) between bands.
template <bool DIFF, int PLACE, bool ONE>
__global__ void __launch_bounds__(32 * kMaxWarps) gs_solve_kernel(const __grid_constant__ GsSolve S) {
    __shared__ int s_stop[2];  // a warp gave up in an even, an odd chunk
    __shared__ __align__(16) float s_mail[kMaxWarps][2 * kChunk];
    const int m = S.n - 2, lines = gs_lines(m);
    const int array = (lines + 1) * kLine;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int in_flight = ONE ? (int)(blockDim.x >> 5) / S.bands : S.sweeps;
    const unsigned lim_set = S.poll_limit ? __ldcg(S.poll_limit) : 0u;
    const unsigned limit = lim_set ? lim_set : kGsPolls;
    if (threadIdx.x == 0) s_stop[0] = s_stop[1] = 0;
    for (int item = blockIdx.x; item < (ONE ? S.nf : S.nf * S.bands); item += gridDim.x) {
        const int fi = ONE ? item : item / S.bands;
        const GsField& F = S.f[fi];
        const int band = ONE ? w % S.bands : item - fi * S.bands;
        int s = ONE ? w / S.bands : w;
        GsBand<DIFF, PLACE> B{S, F};
        B.xo = ONE ? band * array : 0;
        B.co = ONE ? (S.bands + band) * array : array;
        B.xg = F.big + (size_t)band * array * (PLACE == GS_GLOBAL ? 2 : 1);
        B.cg = B.xg + (PLACE == GS_GLOBAL ? array : 0);
        B.band = band;
        B.m = m;
        B.lane = lane;
        B.top = band == 0;
        B.bot = band == S.bands - 1;
        B.lm = B.bot ? m - 1 - band * 32 : 32;
        B.s_lr = F.mode == BND_OPP_H ? -1.f : 1.f;
        B.s_tb = F.mode == BND_OPP_V ? -1.f : 1.f;
        // lanes behind the grid's last row stay zero (their constant terms are)
        const float a = lane > B.lm ? 0.f : F.a, den = F.den, rden = F.rden;
        // the warps that load and store a band: all of the CTA, or (ONE) the band's own
        const int part = ONE ? s : w, parts = ONE ? in_flight : (int)(blockDim.x >> 5);
        __syncthreads();  // the previous band's store has read the arrays
        // places outside the columns and rows stay finite: nothing reads them, but a NaN
        // would send its lane through the slow division
        for (int k = part * 32 + lane; k < array; k += parts * 32) B.x(0, k) = B.c(0, k) = 0.f;
        __syncthreads();
        B.load(part, parts);
        __syncthreads();
        // edge values a first sweep reads
        float l_edge = 0.f, r_edge = 0.f;
        if (s == 0 && 1 + band * 32 + lane < S.n - 1) {
            l_edge = B.initial(1 + band * 32 + lane, 0);
            r_edge = B.initial(1 + band * 32 + lane, S.n - 1);
        }
        // Imported rows, one value per lane and chunk: lanes 0 .. kChunk-1 the last row of the
        // band above, this sweep's values; lanes 16 .. 16+kChunk-1 the first row of the band
        // below, the sweep before. Exported rows: the same lanes the band's first and last row.
        unsigned long long* const W = S.words + ((size_t)fi * S.bands + band) * 2 * m;
        const unsigned tag = S.epoch * 64u + s + 1u;
        const bool role_u = lane < kChunk, role_d = lane >= 16 && lane < 16 + kChunk;
        const int k_role = lane & 15, shift = role_d ? k_role - 31 : k_role;  // column = t0 + shift
        const unsigned long long* imp = nullptr;
        unsigned want = tag;
        if (!ONE && role_u && !B.top) imp = W - m;
        if (!ONE && role_d && !B.bot && s > 0) {
            imp = W + 2 * m;
            want = tag - 1u;
        }
        unsigned long long* exp = nullptr;
        if (!ONE && role_u && !B.top) exp = W;
        if (!ONE && role_d && !B.bot) exp = W + m;
        const int direct_row = role_u ? 0 : 1 + (band + 1) * 32;
        float* const mail = s_mail[w] + (role_d ? kChunk : 0) + k_role;
        const float4* const box = reinterpret_cast<const float4*>(s_mail[w] + (lane == 31 ? kChunk : 0));
        auto fetch = [&](int t0) {
            const int j = t0 + shift;
            return imp != nullptr && (unsigned)j < (unsigned)m ? ld_word(imp + j) : 0ull;
        };
        float val = 0.f, old = 0.f;
        float xa[kChunk], ca[kChunk], xb[kChunk], cb[kChunk];
#pragma unroll
        for (int k = 0; k < kChunk; ++k) xa[k] = ca[k] = xb[k] = cb[k] = 0.f;
        const int start = ONE ? band * S.band_lag : 0;
        const int total = lines + S.lag * (S.sweeps - 1) + (ONE ? S.band_lag * (S.bands - 1) : 0);
        // chunk q; word, xr, cc: its import, loaded two chunks before, and its lines, loaded one
        // before; next, xn, cn: the next chunk's
        auto chunk = [&](int q, int& stop, unsigned long long& word, unsigned long long& next, float (&xr)[kChunk],
                         float (&cc)[kChunk], float (&xn)[kChunk], float (&cn)[kChunk]) {
            if (ONE && q * kChunk - s * S.lag - start >= lines) s += in_flight;
            const int t0 = q * kChunk - s * S.lag - start;
            const bool first = s == 0;
            if (t0 >= 0 && t0 < lines && s < S.sweeps) {  // t0 is a multiple of kChunk
                if (t0 == 0) {
                    word = fetch(t0);
                    next = fetch(t0 + kChunk);
                    old = B.x(0, lane);
                    val = 0.f;
                    B.lines_of(t0, xr, cc);
                }
                const int jr = t0 + shift;
                const bool in_row = (unsigned)jr < (unsigned)m;
                float in = 0.f;
                if (ONE) {
                    // completed by the barrier: the band above is 31 columns and a chunk ahead
                    if (in_row && role_u && !B.top) in = B.x_above(t0 + k_role + 31);
                    if (in_row && role_d && !B.bot && !first) in = B.x_below(jr);
                } else {
                    const bool needs = imp != nullptr && in_row;
                    unsigned polls = 0;
                    while (!__all_sync(0xffffffffu, !needs || (unsigned)(word >> 32) == want)) {
                        if (++polls > limit || ((polls & 63u) == 0 && *(volatile int*)&S.ctrl->error != 0)) {
                            if (lane == 0) {
                                atomicExch(&S.ctrl->error, 1);
                                *(volatile int*)&stop = 1;
                            }
                            break;
                        }
                        word = fetch(t0);
                    }
                    in = __uint_as_float((unsigned)word);
                }
                // a first sweep's values of rows outside the band that no import carries
                if (first && ((role_u && B.top) || role_d))
                    in = in_row && direct_row < S.n ? B.initial(direct_row, 1 + jr) : 0.f;
                if (role_u || role_d) *mail = in;
                __syncwarp();
                float inj[kChunk];
#pragma unroll
                for (int k = 0; k < kChunk; k += 4) {
                    const float4 v = box[k / 4];
                    inj[k] = v.x;
                    inj[k + 1] = v.y;
                    inj[k + 2] = v.z;
                    inj[k + 3] = v.w;
                }
                if (!ONE) word = fetch(t0 + 2 * kChunk);
                // the next chunk's lines: the previous sweep is past them (lag > 2 chunks)
                if (t0 + kChunk < lines) B.lines_of(t0 + kChunk, xn, cn);
                if (t0 < 32 || t0 + kChunk >= m)
                    gs_chunk<DIFF, PLACE, true>(B, first, t0, xr, cc, inj, val, old, l_edge, r_edge, a, den, rden);
                else
                    gs_chunk<DIFF, PLACE, false>(B, first, t0, xr, cc, inj, val, old, l_edge, r_edge, a, den, rden);
                if (!ONE) {
                    __syncwarp();
                    if (exp != nullptr && in_row) st_word(exp + jr, B.x(t0 + k_role, role_d ? 31 : 0), tag);
                }
            }
            __syncthreads();
            // the same for every thread: a faster warp may write the next chunk's word already,
            // but this one not before the next barrier
            return ONE || *(volatile int*)&stop == 0;
        };
        unsigned long long wa = 0, wb = 0;
#pragma unroll 1
        for (int q = 0; q * kChunk < total; q += 2) {
            if (!chunk(q, s_stop[0], wa, wb, xa, ca, xb, cb)) return;
            if (!chunk(q + 1, s_stop[1], wb, wa, xb, cb, xa, ca)) return;
        }
        B.store(part, parts);
    }
}

// The fields a solve of no sweeps leaves: x + dt*s, edges as given.
__global__ void gs_add_kernel(const GsSolve S) {
    const GsField& F = S.f[blockIdx.y];
    for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < (long)S.n * S.n; e += (long)gridDim.x * blockDim.x) {
        const int i = (int)(e / S.n), j = (int)(e % S.n);
        const size_t o = (size_t)i * S.P + j;
        const bool in = i > 0 && i < S.n - 1 && j > 0 && j < S.n - 1;
        F.out[o] = in ? gs_source(F.x[o], F.src[o], S.dt) : F.x[o];
    }
}

struct GsVel {
    const float *u, *v;  // in
    const float* p;      // remove_p only
    float *uo, *vo;
    int n, P;
    float h, dt0;
};

// Writes (un, vn) of inner cell (i, j) to cell (gi, gj) = itself or an edge or corner cell
// next to it, with the host solver's reflecting fills.
__device__ __forceinline__ void gs_put(const GsVel& A, int gi, int gj, int i, int j, float un, float vn) {
    const size_t o = (size_t)gi * A.P + gj;
    const bool ei = gi != i, ej = gj != j;
    float a = un, b = vn;
    if (ei && ej) {  // the mean of the corner's two edge neighbours
        a = __fmul_rn(0.5f, __fadd_rn(un, -un));
        b = __fmul_rn(0.5f, __fadd_rn(-vn, vn));
    } else if (ej) {
        a = -un;
    } else if (ei) {
        b = -vn;
    }
    A.uo[o] = a;
    A.vo[o] = b;
}

// remove_p (fluid_solver_cpu.cpp:205-210) and the reflecting fills, one thread per cell.
__global__ void __launch_bounds__(256) gs_remove_p_kernel(const GsVel A) {
    const int gj = blockIdx.x * 32 + threadIdx.x, gi = blockIdx.y * 8 + threadIdx.y;
    if (gi >= A.n || gj >= A.n) return;
    const int i = min(max(gi, 1), A.n - 2), j = min(max(gj, 1), A.n - 2);
    const size_t o = (size_t)i * A.P + j;
    const float* __restrict__ p = A.p;
    const float un = __fsub_rn(A.u[o], __fdiv_rn(__fmul_rn(0.5f, __fsub_rn(p[o + 1], p[o - 1])), A.h));
    const float vn = __fsub_rn(A.v[o], __fdiv_rn(__fmul_rn(0.5f, __fsub_rn(p[o + A.P], p[o - A.P])), A.h));
    gs_put(A, gi, gj, i, j, un, vn);
}

// advect(trace=false) (fluid_solver_cpu.cpp:154-173) of u and v by themselves and the
// reflecting fills, one thread per cell.
__global__ void __launch_bounds__(256) gs_gather_kernel(const GsVel A) {
    const int gj = blockIdx.x * 32 + threadIdx.x, gi = blockIdx.y * 8 + threadIdx.y;
    if (gi >= A.n || gj >= A.n) return;
    const int i = min(max(gi, 1), A.n - 2), j = min(max(gj, 1), A.n - 2), P = A.P;
    const size_t o = (size_t)i * P + j;
    const float hi = (float)A.n - 1.5f;
    float x = __fsub_rn((float)j, __fmul_rn(A.dt0, A.u[o]));
    float y = __fsub_rn((float)i, __fmul_rn(A.dt0, A.v[o]));
    x = (x < hi) ? x : hi;
    x = (1.5f < x) ? x : 1.5f;
    y = (y < hi) ? y : hi;
    y = (1.5f < y) ? y : 1.5f;
    const int j0 = (int)x, i0 = (int)y;
    const float s0 = __fsub_rn(x, (float)j0), s1 = __fsub_rn(1.f, s0);
    const float s2 = __fsub_rn(y, (float)i0), s3 = __fsub_rn(1.f, s2);
    const size_t a = (size_t)i0 * P + j0;
    auto mix = [&](const float* __restrict__ g) {
        const float t = __fadd_rn(__fmul_rn(s1, g[a]), __fmul_rn(s0, g[a + 1]));
        const float b = __fadd_rn(__fmul_rn(s1, g[a + P]), __fmul_rn(s0, g[a + P + 1]));
        return __fadd_rn(__fmul_rn(s3, t), __fmul_rn(s2, b));
    };
    gs_put(A, gi, gj, i, j, mix(A.u), mix(A.v));
}

// ------------------------------------------------------------------- splat
struct GsSplat {
    const float *d, *u, *v;  // diffused density, the step's initial velocity
    float* out;
    int* head;   // per target cell: the last source linked to it (-1: none)
    int* next;   // per source cell: the source linked before it
    int* crowd;    // [0], [1]: cells on the lists below so far, [2]: the farthest a source moves
    int* cells;    // the cells that receive more than kGsSorted sources
    int* crowded;  // those of them that receive more than kGsBunch
    int n, P;
    float dt0;
};
constexpr int kGsSorted = 24;  // sources that a thread sorts in its own array
constexpr int kGsBunch = 128;  // sources that a warp sorts in shared memory
constexpr int kGsCrowdThreads = 1024, kGsListed = kGsCrowdThreads;  // sources that a CTA sorts

// Target cell and offsets of source (i, j) (fluid_solver_cpu.cpp:132-139); false when the
// source leaves the grid (a NaN position too).
__device__ __forceinline__ bool gs_target(const GsSplat& A, int i, int j, int& i0, int& j0, float& s0, float& s2) {
    const size_t o = (size_t)i * A.P + j;
    const float hi = (float)A.n - 1.5f;
    const float x = __fadd_rn((float)j, __fmul_rn(A.dt0, __ldg(A.u + o)));
    const float y = __fadd_rn((float)i, __fmul_rn(A.dt0, __ldg(A.v + o)));
    if (!(x >= 0.5f && x <= hi && y >= 0.5f && y <= hi)) return false;
    j0 = (int)x;
    i0 = (int)y;
    s0 = __fsub_rn(x, (float)j0);
    s2 = __fsub_rn(y, (float)i0);
    return true;
}

__global__ void __launch_bounds__(256) gs_link_kernel(const GsSplat A) {
    const int j = 1 + blockIdx.x * 32 + threadIdx.x, i = 1 + blockIdx.y * 8 + threadIdx.y;
    int i0, j0, far = 0;
    float s0, s2;
    if (i <= A.n - 2 && j <= A.n - 2 && gs_target(A, i, j, i0, j0, s0, s2)) {
        const int o = i * A.P + j;
        A.next[o] = atomicExch(A.head + (i0 * A.P + j0), o);
        far = max(abs(i0 - i), abs(j0 - j));
    }
    far = __reduce_max_sync(0xffffffffu, far);
    if (threadIdx.x == 0 && far > __ldcg(A.crowd + 2)) atomicMax(A.crowd + 2, far);
}

// What a source adds to the cell at offset (di, dj) from its target.
__device__ __forceinline__ float gs_weighted(float s0, float s2, int di, int dj, float d) {
    const float wx = dj ? s0 : __fsub_rn(1.f, s0), wy = di ? s2 : __fsub_rn(1.f, s2);
    return __fmul_rn(__fmul_rn(wx, wy), d);
}
// The same of source o (source * 4 + corner).
__device__ __forceinline__ float gs_share(const GsSplat& A, int source) {
    const int o = source >> 2, i = o / A.P, j = o - i * A.P;
    int i0, j0;
    float s0, s2;
    gs_target(A, i, j, i0, j0, s0, s2);
    return gs_weighted(s0, s2, (source >> 1) & 1, source & 1, __ldg(A.d + o));
}

// Sum of the contributions to interior cell (i, j) in the raster order of their sources
// (advect(trace=true), fluid_solver_cpu.cpp:127-152); false when there are too many.
__device__ bool gs_collect(const GsSplat& A, int i, int j, float& acc) {
    int src[kGsSorted];  // source * 4 + corner; a source reaches a cell through one corner
    int cnt = 0;
    for (int c = 0; c < 4; ++c) {
        const int di = c >> 1, dj = c & 1;
        for (int o = __ldcg(A.head + ((i - di) * A.P + j - dj)); o >= 0; o = __ldcg(A.next + o)) {
            if (cnt == kGsSorted) return false;
            int k = cnt++;
            for (; k > 0 && (src[k - 1] >> 2) > o; --k) src[k] = src[k - 1];
            src[k] = o * 4 + c;
        }
    }
    acc = 0.f;
    for (int k = 0; k < cnt; ++k) acc = __fadd_rn(acc, gs_share(A, src[k]));
    return true;
}

// One thread per cell; edges and corners repeat or average (their two edge neighbours hold
// the same value) the inner cell's sum. Cells with more sources than a thread sorts are left
// to the kernels below.
__device__ __forceinline__ float gs_edge(float x, bool corner) { return corner ? __fmul_rn(0.5f, __fadd_rn(x, x)) : x; }
__global__ void __launch_bounds__(256) gs_splat_kernel(const GsSplat A) {
    const int gj = blockIdx.x * 32 + threadIdx.x, gi = blockIdx.y * 8 + threadIdx.y;
    if (gi >= A.n || gj >= A.n) return;
    const int i = min(max(gi, 1), A.n - 2), j = min(max(gj, 1), A.n - 2);
    float x;
    if (gs_collect(A, i, j, x))
        A.out[(size_t)gi * A.P + gj] = gs_edge(x, gi != i && gj != j);
    else if (gi == i && gj == j)
        A.cells[atomicAdd(A.crowd, 1)] = i * A.P + j;
}

// acc and the first cnt of v (16-byte aligned) one after another, by one thread.
__device__ float gs_add_up(float acc, const float* v, int cnt) {
    int k = 0;
#pragma unroll 1
    for (; k + 8 <= cnt; k += 8) {
        const float4 a = *reinterpret_cast<const float4*>(v + k), b = *reinterpret_cast<const float4*>(v + k + 4);
        const float t[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) acc = __fadd_rn(acc, t[e]);
    }
    for (; k < cnt; ++k) acc = __fadd_rn(acc, v[k]);
    return acc;
}
// A cell's sum to the cell, and to the edges and the corner that repeat it, by one thread.
__device__ void gs_put_sum(const GsSplat& A, int i, int j, float x) {
    for (int gi : {i, i == 1 ? 0 : -1, i == A.n - 2 ? A.n - 1 : -1})
        for (int gj : {j, j == 1 ? 0 : -1, j == A.n - 2 ? A.n - 1 : -1})
            if (gi >= 0 && gj >= 0) A.out[(size_t)gi * A.P + gj] = gs_edge(x, gi != i && gj != j);
}

// Cells of up to kGsBunch sources, a warp each in turn: four lanes walk the four lists (0.35 us
// a link), the warp sorts what they find by rank and one lane adds. Others go on to
// gs_crowd_kernel.
constexpr int kGsBunchWarps = 8;
__global__ void __launch_bounds__(32 * kGsBunchWarps) gs_bunch_kernel(const GsSplat A) {
    __shared__ int lists[kGsBunchWarps][kGsBunch];
    __shared__ __align__(16) float shares[kGsBunchWarps][kGsBunch];
    constexpr unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, cells = __ldcg(A.crowd);
    int* const list = lists[w];
    float* const share = shares[w];
    for (int q = blockIdx.x * kGsBunchWarps + w; q < cells; q += gridDim.x * kGsBunchWarps) {
        const int cell = __ldcg(A.cells + q), i = cell / A.P, j = cell - i * A.P;
        int o = lane < 4 ? __ldcg(A.head + ((i - (lane >> 1)) * A.P + j - (lane & 1))) : -1, cnt = 0;
        for (unsigned m; cnt <= kGsBunch && (m = __ballot_sync(FULL, o >= 0)) != 0;) {
            const int k = cnt + __popc(m & ((1u << lane) - 1));
            cnt += __popc(m);
            if (o >= 0) {
                if (k < kGsBunch) list[k] = o * 4 + lane;
                o = __ldcg(A.next + o);
            }
        }
        __syncwarp();
        if (cnt > kGsBunch) {
            if (lane == 0) A.crowded[atomicAdd(A.crowd + 1, 1)] = cell;
            continue;
        }
        for (int e = lane; e < cnt; e += 32) {
            const int mine = list[e];
            int place = 0;  // the sources before it
#pragma unroll 8
            for (int k = 0; k < cnt; ++k) place += list[k] < mine;
            share[place] = gs_share(A, mine);
        }
        __syncwarp();
        if (lane == 0) gs_put_sum(A, i, j, gs_add_up(0.f, share, cnt));
        __syncwarp();
    }
}

// Cells of more sources, a CTA each in turn. Every source that could reach the cell, those
// within the farthest move of any source, is looked at in raster order, a thousand at a time
// (about 1 us); those that do reach it are packed, and one thread adds them while the others
// look on. Where the cell's lists are shorter than that takes (0.35 us a link), they are walked
// and sorted instead. A step at 800 x 800 (1.6 ms, 1.8 with the flow that makes the crowd), ms
// with n sources in a cell, and where a thread walked its cell's lists once per source up to
// 256 and one thread applied all sources beyond: 149 1.84 and 7.7, 253 1.85 and 20.7, 11289
// 1.91 and 144, all 640,000 4.7 and 130.
__global__ void __launch_bounds__(kGsCrowdThreads) gs_crowd_kernel(const GsSplat A) {
    constexpr int T = kGsCrowdThreads;
    __shared__ int list[kGsListed];
    __shared__ __align__(16) float share[T];
    __shared__ int hits[T / 32];
    __shared__ int s_count;
    static_assert(T / 32 == 32, "a warp's lanes hold the warps' counts");
    const int crowded = __ldcg(A.crowd + 1), reach = __ldcg(A.crowd + 2) + 1;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, n = A.n, P = A.P;
    for (int q = blockIdx.x; q < crowded; q += gridDim.x) {
        const int cell = __ldcg(A.crowded + q), i = cell / P, j = cell - i * P;
        const int top = max(1, i - reach), left = max(1, j - reach);
        const int cols = min(n - 2, j + reach) - left + 1, box = (min(n - 2, i + reach) - top + 1) * cols;
        const int most = min(kGsListed, 3 * (box / T));  // links worth walking
        float acc = 0.f;
        int cnt = kGsListed + 1;
        if (most > kGsBunch) {
            if (tid == 0) s_count = 0;
            __syncthreads();
            if (lane == 0 && w < 4)
                for (int o = __ldcg(A.head + ((i - (w >> 1)) * P + j - (w & 1))); o >= 0; o = __ldcg(A.next + o)) {
                    const int k = atomicAdd(&s_count, 1);
                    if (k >= most) break;
                    list[k] = o * 4 + w;
                }
            __syncthreads();
            cnt = s_count;
        }
        if (cnt <= most) {
            if (tid < cnt) {
                const int mine = list[tid];
                int place = 0;
#pragma unroll 8
                for (int k = 0; k < cnt; ++k) place += list[k] < mine;
                share[place] = gs_share(A, mine);
            }
            __syncthreads();
            if (tid == 0) acc = gs_add_up(acc, share, cnt);
        } else {
            for (int e0 = 0; e0 < box; e0 += T) {
                const int e = e0 + tid, r = e / cols, si = top + r, sj = left + e - r * cols;
                int i0, j0;
                float s0, s2, mine = 0.f;
                bool hit = e < box && gs_target(A, si, sj, i0, j0, s0, s2);
                if (hit) {
                    const int di = i - i0, dj = j - j0;
                    hit = (unsigned)(di | dj) <= 1u;
                    if (hit) mine = gs_weighted(s0, s2, di, dj, __ldg(A.d + (size_t)si * P + sj));
                }
                const unsigned m = __ballot_sync(0xffffffffu, hit);
                if (lane == 0) hits[w] = __popc(m);
                __syncthreads();
                const int h = hits[lane];
                const int before = __reduce_add_sync(0xffffffffu, lane < w ? h : 0);
                cnt = __reduce_add_sync(0xffffffffu, h);
                if (hit) share[before + __popc(m & ((1u << lane) - 1))] = mine;
                __syncthreads();
                if (tid == 0) acc = gs_add_up(acc, share, cnt);
            }
        }
        if (tid == 0) gs_put_sum(A, i, j, acc);
        __syncthreads();
    }
}

// ------------------------------------------------------------------- host
size_t array_bytes(int n) { return (size_t)(gs_lines(n - 2) + 1) * kLine * sizeof(float); }

int smem_limit() {
    int dev = 0, smem = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    if (cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) return 0;
    return smem - 2048;  // the kernel's static shared memory
}

// Columns between a sweep and the next, in whole chunks: the next chunk's loads need two
// chunks and one column.
// With a CTA per band the previous sweep must also have come back from the band below, two
// trips between SMs away. Between bands of one CTA: the band above must be a chunk past the
// column above.
constexpr int kLagOne = 3 * kChunk;
constexpr int kLagMany = 5 * kChunk;
constexpr int kBandLag = 32 + kChunk;

// Bands of one CTA: the grids whose arrays all fit its shared memory.
bool one_cta(int n) {
    const int bands = (n - 2 + 31) / 32;
    return bands <= 6 && 2 * bands * array_bytes(n) <= (size_t)smem_limit();
}

template <bool DIFF, int PLACE, bool ONE>
cudaError_t launch_solve(GsSolve& S, cudaStream_t st) {
    S.bands = (S.n - 2 + 31) / 32;
    S.band_lag = kBandLag;
    const int in_flight = std::min(S.sweeps, kMaxWarps / S.bands);
    const int warps = ONE ? S.bands * in_flight : S.sweeps;
    // ONE: a warp's next sweep begins when its last one is done
    const int per_warp = (gs_lines(S.n - 2) / kChunk + in_flight - 1) / in_flight * kChunk;
    S.lag = ONE ? std::max(kLagOne, per_warp) : kLagMany;
    const size_t smem = (PLACE == GS_GLOBAL ? 0 : (PLACE == GS_SHARED ? 2 : 1) * array_bytes(S.n)) * (ONE ? S.bands : 1);
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, gs_solve_kernel<DIFF, PLACE, ONE>, 32 * warps, smem);
    if (e != cudaSuccess) return e;
    if (per * sms <= 0) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::min(per * sms, ONE ? S.nf : S.nf * S.bands));
    cfg.blockDim = dim3(32 * warps);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ONE ? 0 : 1;  // only CTAs that wait for one another must be co-resident
    return cudaLaunchKernelEx(&cfg, gs_solve_kernel<DIFF, PLACE, ONE>, S);
}

template <bool DIFF>
cudaError_t launch_placed(GsSolve& S, cudaStream_t st) {
    const size_t limit = (size_t)smem_limit(), one = array_bytes(S.n);
    if (one_cta(S.n)) return launch_solve<DIFF, GS_SHARED, true>(S, st);
    if (2 * one <= limit) return launch_solve<DIFF, GS_SHARED, false>(S, st);
    if (one <= limit) return launch_solve<DIFF, GS_CONST_GLOBAL, false>(S, st);
    return launch_solve<DIFF, GS_GLOBAL, false>(S, st);
}

// All sweeps of a solve, kMaxWarps to a launch where a warp runs one sweep.
cudaError_t solve(GsSolve S, bool diff, int sweeps, unsigned& epoch, cudaStream_t st, int* launches) {
    int dev = 0, sms = 0;
    cudaError_t q = cudaGetDevice(&dev);
    if (q == cudaSuccess) q = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (q != cudaSuccess) return q;
    const int most = one_cta(S.n) ? sweeps : std::min(kMaxWarps, sms);
    for (int done = 0; done < sweeps;) {
        S.sweeps = std::min(most, sweeps - done);
        S.epoch = ++epoch;
        for (int k = 0; k < S.nf; ++k) S.f[k].start = done > 0 ? S.f[k].out : nullptr;
        const cudaError_t e = diff ? launch_placed<true>(S, st) : launch_placed<false>(S, st);
        if (e != cudaSuccess) return e;
        ++*launches;
        done += S.sweeps;
    }
    return cudaSuccess;
}

}  // namespace

bool gs_one_cta(int n) { return one_cta(n); }

int gs_tiled_max_size() { return smem_limit() > 0 ? 16384 : 0; }

cudaError_t gs_prepare() {
    const int bytes = smem_limit();
    if (bytes <= 0) return cudaErrorNoDevice;
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(gs_solve_kernel<true, GS_SHARED, false>, attr, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gs_solve_kernel<false, GS_SHARED, false>, attr, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gs_solve_kernel<true, GS_SHARED, true>, attr, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gs_solve_kernel<false, GS_SHARED, true>, attr, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gs_solve_kernel<true, GS_CONST_GLOBAL, false>, attr, bytes);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(gs_solve_kernel<false, GS_CONST_GLOBAL, false>, attr, bytes);
    return e;
}

// A step in the host solver's order (fluid_solver_cpu.cpp:6-31). The state keeps the step's
// initial velocity until the last launch, so the density's splat runs on the side stream
// beside the projections.
cudaError_t gs_step(const GsFields& G, int n, int pitch, int kd, int kp, float diff, float visc, float dt,
                    cudaStream_t st, int* launches) {
    *launches = 0;
    // constants as the host solver computes them, in float (fluid_solver_cpu.cpp:97-98,
    // 119, 181): a = dt * (rows*cols) * rate, den = 1 + 4a, dt0 = sqrt(rows*cols) * dt
    const float cells = (float)((size_t)n * (size_t)n);
    const float h = 1.0f / sqrtf(cells), dt0 = sqrtf(cells) * dt;
    cudaError_t e;
#define GS_CK(call) \
    if ((e = (call)) != cudaSuccess) return e
    GsSolve S{};
    S.n = n;
    S.P = pitch;
    S.dt = dt;
    S.cdiv = -0.5f * h;
    S.ctrl = G.ctrl;
    S.poll_limit = G.poll_limit;
    // the words' tags and the splat's counts start at zero, the lists empty
    int* crowd = reinterpret_cast<int*>(G.words);
    S.words = reinterpret_cast<unsigned long long*>(G.words) + 32;
    const int max_bands = (n - 2 + 31) / 32;
    GS_CK(cudaMemsetAsync(G.words, 0, 256 + (size_t)3 * max_bands * 2 * (n - 2) * 8, st));
    GS_CK(cudaMemsetAsync(G.ctrl, 0, sizeof(SolveCtrl), st));
    const int modes[3] = {BND_CONT, BND_OPP_H, BND_OPP_V};
    const float rates[3] = {diff, visc, visc};
    for (int k = 0; k < 3; ++k) {
        GsField& F = S.f[k];
        F.x = G.state[k];
        F.src = G.src[k];
        F.out = G.dif[k];
        F.big = G.big[k];
        F.mode = modes[k];
        F.a = dt * cells * rates[k];
        F.den = 1.f + 4.f * F.a;  // 4a is exact, so a fused form rounds the same
        F.rden = F.den > 0x1p-20f && F.den < 0x1p20f ? 1.f / F.den : 0.f;
    }
    unsigned epoch = 0;
    S.nf = 3;
    if (kd == 0) {
        gs_add_kernel<<<dim3(std::min(4096, (n * n + 255) / 256), 3), 256, 0, st>>>(S);
        GS_CK(cudaGetLastError());
        ++*launches;
    } else if (array_bytes(n) <= (size_t)smem_limit()) {
        GS_CK(solve(S, true, kd, epoch, st, launches));
    } else {
        // both band arrays in global memory: one field at a time in all of the scratch
        for (int k = 0; k < 3; ++k) {
            GsSolve one = S;
            one.nf = 1;
            one.f[0] = S.f[k];
            one.f[0].big = G.big[0];
            GS_CK(solve(one, true, kd, epoch, st, launches));
        }
    }
    const dim3 cells2((n + 31) / 32, (n + 7) / 8), threads(32, 8);
    // density on the side stream
    GS_CK(cudaEventRecord(G.fork, st));
    GS_CK(cudaStreamWaitEvent(G.side, G.fork, 0));
    const GsSplat A{G.dif[0], G.state[1], G.state[2], G.state[0], G.head, G.next, crowd, G.cells,
                    G.cells + (size_t)n * pitch / 2, n, pitch, dt0};
    GS_CK(cudaMemsetAsync(G.head, 0xff, (size_t)n * pitch * sizeof(int), G.side));
    gs_link_kernel<<<cells2, threads, 0, G.side>>>(A);
    gs_splat_kernel<<<cells2, threads, 0, G.side>>>(A);
    int dev = 0, sms = 0;
    GS_CK(cudaGetDevice(&dev));
    GS_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    gs_bunch_kernel<<<4 * sms, 32 * kGsBunchWarps, 0, G.side>>>(A);
    gs_crowd_kernel<<<sms, kGsCrowdThreads, 0, G.side>>>(A);
    GS_CK(cudaGetLastError());
    *launches += 4;
    GS_CK(cudaEventRecord(G.join, G.side));
    // velocity
    auto project = [&](const float* u, const float* v, float* uo, float* vo) -> cudaError_t {
        GsSolve Q = S;
        Q.nf = 1;
        Q.f[0] = GsField{};
        Q.f[0].u = u;
        Q.f[0].v = v;
        Q.f[0].out = G.p;
        Q.f[0].big = G.big[0];
        Q.f[0].mode = BND_CONT;
        if (kp == 0) {
            GS_CK(cudaMemsetAsync(G.p, 0, (size_t)n * pitch * sizeof(float), st));
        } else {
            GS_CK(solve(Q, false, kp, epoch, st, launches));
        }
        if (uo == G.state[1]) GS_CK(cudaStreamWaitEvent(st, G.join, 0));
        gs_remove_p_kernel<<<cells2, threads, 0, st>>>(GsVel{u, v, G.p, uo, vo, n, pitch, h, dt0});
        ++*launches;
        return cudaGetLastError();
    };
    GS_CK(project(G.dif[1], G.dif[2], G.vel[0], G.vel[1]));
    gs_gather_kernel<<<cells2, threads, 0, st>>>(GsVel{G.vel[0], G.vel[1], nullptr, G.dif[1], G.dif[2], n, pitch, h, dt0});
    ++*launches;
    return project(G.dif[1], G.dif[2], G.state[1], G.state[2]);
#undef GS_CK
}

}  // namespace fs
