// Semi-Lagrangian advection kernels.
//
// Reference behaviour (mworchel/fluid-2d src/fluid_solver_gpu.cu):
//   density  advect(trace=true) 325-356: D2D copy, memset, advect_trace_kernel
//            131-162 (forward bilinear splat with fp32 atomicAdd), Neumann fill,
//            then smooth 314-323 (D2D copy + smooth_kernel 87-97, no fill);
//   velocity two advect(trace=false) calls 248-251 on copies u0, v0 with
//            advect_kernel 99-129 (backtrace, clamp, bilinear gather), each followed
//            by its reflecting fill.
// Here the density path is three launches with no copies: a memset of the
// accumulator, the splat, and one "finish" kernel that applies the Neumann fill and
// the smoothing together. The velocity path is one kernel that backtraces once per
// cell and gathers u and v together, writing the reflecting edges directly.
//
// Operand order and rounding follow the reference expressions as its compiled kernels
// evaluate them: explicit _rn intrinsics, with a fused multiply-add exactly where nvcc
// fuses the reference source (the positions j +- dt0*u and, in the gather, the bilinear
// sum as s3*fma(s0, B, s1*A) + s2*fma(s0, D, s1*C), fused at the first product). These
// fusions were found by comparing the reference's compiled kernels with candidate
// restatements bit for bit. The splat order of the atomics is unspecified, as in the
// reference.
//
// All three are bound by memory at large grids (8194 x 8194, ncu: splat 242 us, of which
// 1.08 GB read and 0.27 GB written take 198 us at 6.8 TB/s, 300 us with four atomics a cell;
// finish 107 us for 0.54 GB, 264 us one cell per thread; velocity 260 us, where eight
// unaligned gathers a cell keep the L1 busy beyond the 158 us that its 1.07 GB take, 304 us
// one row per thread) and by latency at small ones (4.5-5 us each at 130 x 130).

#include <algorithm>

#include "fs_internal.cuh"

namespace fs {
namespace {

// Forward splat of the interior source cells of column j, rows i .. i + R - 1,
// advect_trace_kernel (fluid_solver_gpu.cu:141-159). The whole warp calls it, on 32
// consecutive columns. The reference adds four weighted values per cell with one atomic
// each; here the values that neighbouring cells of a warp add to the same target are summed
// first, since the L2 takes a float atomic at a time: where the cell to the right lands one
// column on (what a smooth flow does), it takes over this cell's two right-hand values, and
// where the cell below lands one row on, the two lower ones, so that a cell costs little
// more than one atomic. Any other landing place keeps its own atomics. The order in which a
// target's values are added is as unspecified as before.
template <int R>
__device__ __forceinline__ void splat_rows(const float* __restrict__ d0, const float* __restrict__ u,
                                           const float* __restrict__ v, float* __restrict__ acc, const AdvectArgs& A,
                                           int i, int j) {
    constexpr unsigned FULL = 0xffffffffu;
    const size_t P = (size_t)A.pitch;
    const int lane = threadIdx.x & 31;
    float ur[R], vr[R], dr[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const bool in = i + r >= 1 && i + r < A.rows - 1 && j >= 1 && j < A.cols - 1;
        const size_t o = (size_t)(i + r) * P + j;
        ur[r] = in ? __ldg(u + o) : __int_as_float(0x7fffffff);  // NaN lands nowhere
        vr[r] = in ? __ldg(v + o) : 0.f;
        dr[r] = in ? __ldg(d0 + o) : 0.f;
    }
    int ci = -2, cj = -2;  // where the value carried from the row above goes (ci < 0: none)
    float carry = 0.f;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float x = __fmaf_rn(A.dt0, ur[r], (float)j);
        const float y = __fmaf_rn(A.dt0, vr[r], (float)(i + r));
        // skipped unless inside [0.5, n-1.5] (fluid_solver_gpu.cu:144); NaN is skipped too
        const bool lands = x >= 0.5f && x <= A.xmax && y >= 0.5f && y <= A.ymax;
        const int j0 = lands ? (int)x : -2, i0 = lands ? (int)y : -2;
        const float s0 = __fsub_rn(x, (float)j0), s1 = __fsub_rn(1.f, s0);
        const float s2 = __fsub_rn(y, (float)i0), s3 = __fsub_rn(1.f, s2);
        float tl = __fmul_rn(__fmul_rn(s1, s3), dr[r]), bl = __fmul_rn(__fmul_rn(s1, s2), dr[r]);
        const float tr = __fmul_rn(__fmul_rn(s0, s3), dr[r]), br = __fmul_rn(__fmul_rn(s0, s2), dr[r]);
        // the right-hand values go to the next lane where it lands one column on
        const float ptr = __shfl_up_sync(FULL, tr, 1), pbr = __shfl_up_sync(FULL, br, 1);
        const int pi = __shfl_up_sync(FULL, i0, 1), pj = __shfl_up_sync(FULL, j0, 1);
        const bool joins = lands && lane > 0 && pi == i0 && pj + 1 == j0;
        const bool taken = (__ballot_sync(FULL, joins) >> 1 >> lane) & 1u;
        if (joins) {
            tl = __fadd_rn(tl, ptr);
            bl = __fadd_rn(bl, pbr);
        }
        if (ci >= 0) {
            if (lands && ci == i0 && cj == j0)
                tl = __fadd_rn(tl, carry);
            else
                atomicAdd(acc + (size_t)ci * P + cj, carry);
            ci = -2;
        }
        if (lands) {
            float* t = acc + (size_t)i0 * P + j0;
            atomicAdd(t, tl);
            if (!taken) {
                atomicAdd(t + 1, tr);
                atomicAdd(t + P + 1, br);
            }
            ci = i0 + 1;
            cj = j0;
            carry = bl;
        }
    }
    if (ci >= 0) atomicAdd(acc + (size_t)ci * P + cj, carry);
}

// Value of the accumulator after set_boundary_continuous (fluid_solver_gpu.cu:11-24):
// edges read their inner neighbour, corners and the interior read themselves.
__device__ __forceinline__ float filled(const float* __restrict__ acc, int r, int c, const AdvectArgs& A) {
    const bool ri = r >= 1 && r <= A.rows - 2, ci = c >= 1 && c <= A.cols - 2;
    if (ri && !ci) c = (c == 0) ? 1 : A.cols - 2;
    else if (ci && !ri) r = (r == 0) ? 1 : A.rows - 2;
    return __ldg(acc + (size_t)r * A.pitch + c);
}

// Neumann fill of the splat result plus smooth_kernel (fluid_solver_gpu.cu:94) for
// cell (i, j); returns 1 if the value is not finite.
__device__ __forceinline__ int finish_cell(const float* __restrict__ acc, float* __restrict__ d, int smooth,
                                           const AdvectArgs& A, int i, int j) {
    float out = filled(acc, i, j, A);
    if (smooth && i >= 1 && i <= A.rows - 2 && j >= 1 && j <= A.cols - 2) {
        // 0.2f * (c + l + r + u + d)
        float s = __fadd_rn(out, filled(acc, i, j - 1, A));
        s = __fadd_rn(s, filled(acc, i, j + 1, A));
        s = __fadd_rn(s, filled(acc, i - 1, j, A));
        s = __fadd_rn(s, filled(acc, i + 1, j, A));
        out = __fmul_rn(0.2f, s);
    }
    d[(size_t)i * A.pitch + j] = out;
    return !isfinite(out);
}

// Four consecutive cells (i, j0 .. j0 + 3): 16-byte loads and stores where all of them and
// their neighbours are interior cells, cell by cell otherwise. Rows are 16-byte aligned
// (pitch a multiple of four, buffers of the solver).
__device__ __forceinline__ int finish_group(const float* __restrict__ acc, float* __restrict__ d, int smooth,
                                            const AdvectArgs& A, int i, int j0) {
    const size_t P = (size_t)A.pitch, o = (size_t)i * P + j0;
    int bad = 0;
    if (i >= 2 && i <= A.rows - 3 && j0 >= 2 && j0 + 3 <= A.cols - 3) {
        const float4 c4 = __ldg(reinterpret_cast<const float4*>(acc + o));
        float c[6] = {0.f, c4.x, c4.y, c4.z, c4.w, 0.f};
        float out[4] = {c4.x, c4.y, c4.z, c4.w};
        if (smooth) {
            const float4 u4 = __ldg(reinterpret_cast<const float4*>(acc + o - P));
            const float4 d4 = __ldg(reinterpret_cast<const float4*>(acc + o + P));
            c[0] = __ldg(acc + o - 1);
            c[5] = __ldg(acc + o + 4);
            const float up[4] = {u4.x, u4.y, u4.z, u4.w}, dn[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // finish_cell's sum
                float s = __fadd_rn(c[k + 1], c[k]);
                s = __fadd_rn(s, c[k + 2]);
                s = __fadd_rn(s, up[k]);
                s = __fadd_rn(s, dn[k]);
                out[k] = __fmul_rn(0.2f, s);
            }
        }
        *reinterpret_cast<float4*>(d + o) = make_float4(out[0], out[1], out[2], out[3]);
#pragma unroll
        for (int k = 0; k < 4; ++k) bad |= !isfinite(out[k]);
    } else {
        for (int j = j0; j < min(A.cols, j0 + 4); ++j) bad |= finish_cell(acc, d, smooth, A, i, j);
    }
    return bad;
}

// Backtrace advection of u and v for the cells of column j, rows i .. i + R - 1,
// advect_kernel (fluid_solver_gpu.cu:111-126), with the reflecting fills for edge cells.
// The rows' backtraced positions come first and their gathers follow together: a cell is
// two dependent reads deep, and one at a time a warp waits for both.
template <int R>
__device__ __forceinline__ void advect_rows(const float* __restrict__ u0, const float* __restrict__ v0,
                                            float* __restrict__ u, float* __restrict__ v, const AdvectArgs& A, int i,
                                            int j) {
    if (j >= A.cols) return;
    const size_t P = (size_t)A.pitch;
    const bool ci = j >= 1 && j <= A.cols - 2;
    // Edge cells copy the advected inner neighbour: u is negated on the left/right
    // edges, v on the top/bottom edges (fluid_solver_gpu.cu:26-54).
    const int sj = ci ? j : (j == 0) ? 1 : A.cols - 2;
    auto row = [&](int r) { return min(i + r, A.rows - 1); };  // rows past the grid repeat the last
    auto source_row = [&](int r) { return ci ? min(max(i + r, 1), A.rows - 2) : row(r); };
    float x[R], y[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const size_t o = (size_t)source_row(r) * P + sj;
        x[r] = __ldg(u0 + o);
        y[r] = __ldg(v0 + o);
    }
    float s0[R], s2[R], g[R][8];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        x[r] = __fmaf_rn(-A.dt0, x[r], (float)sj);
        y[r] = __fmaf_rn(-A.dt0, y[r], (float)source_row(r));
        x[r] = fmaxf(1.5f, fminf(A.xmax, x[r]));
        y[r] = fmaxf(1.5f, fminf(A.ymax, y[r]));
        const int j0 = (int)x[r], i0 = (int)y[r];
        s0[r] = __fsub_rn(x[r], (float)j0);
        s2[r] = __fsub_rn(y[r], (float)i0);
        const size_t q = (size_t)i0 * P + j0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            g[r][k] = __ldg(u0 + q + (k & 1) + (k >> 1) * P);
            g[r][4 + k] = __ldg(v0 + q + (k & 1) + (k >> 1) * P);
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (i + r >= A.rows) break;
        const bool ri = i + r >= 1 && i + r <= A.rows - 2;
        const size_t o = (size_t)(i + r) * P + j;
        if (!ri && !ci) {  // corners are never written by the reference
            u[o] = __ldg(u0 + o);
            v[o] = __ldg(v0 + o);
            continue;
        }
        const float s1 = __fsub_rn(1.f, s0[r]), s3 = __fsub_rn(1.f, s2[r]);
        float w[2];
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            const float* a = g[r] + 4 * f;
            const float top = __fmaf_rn(s0[r], a[1], __fmul_rn(s1, a[0]));
            const float bot = __fmaf_rn(s0[r], a[3], __fmul_rn(s1, a[2]));
            w[f] = __fmaf_rn(s3, top, __fmul_rn(s2[r], bot));
        }
        u[o] = (ci ? 1.f : -1.f) * w[0];
        v[o] = (ri || !ci ? 1.f : -1.f) * w[1];
    }
}

template <int R>
__global__ void __launch_bounds__(256) splat_kernel(const float* __restrict__ d0, const float* __restrict__ u,
                                                    const float* __restrict__ v, float* __restrict__ acc,
                                                    const AdvectArgs A) {
    for (int i = (blockIdx.y * 8 + threadIdx.y) * R; i < A.rows - 1; i += 8 * R * gridDim.y)
        splat_rows<R>(d0, u, v, acc, A, i, blockIdx.x * 32 + threadIdx.x);
}

__global__ void __launch_bounds__(256) density_finish_kernel(const float* __restrict__ acc, float* __restrict__ d,
                                                             int smooth, const AdvectArgs A, int* nonfinite) {
    const int j0 = 4 * (blockIdx.x * 32 + threadIdx.x);
    int bad = 0;
    if (j0 < A.cols)
        for (int i = blockIdx.y * 8 + threadIdx.y; i < A.rows; i += 8 * gridDim.y)
            bad |= finish_group(acc, d, smooth, A, i, j0);
    if (bad && nonfinite) report_nonfinite(nonfinite);
}

template <int R>
__global__ void __launch_bounds__(256) advect_velocity_kernel(const float* __restrict__ u0,
                                                              const float* __restrict__ v0, float* __restrict__ u,
                                                              float* __restrict__ v, const AdvectArgs A) {
    for (int i = (blockIdx.y * 8 + threadIdx.y) * R; i < A.rows; i += 8 * R * gridDim.y)
        advect_rows<R>(u0, v0, u, v, A, i, blockIdx.x * 32 + threadIdx.x);
}

// ----------------------------------------------------------------- batched
// One launch covers every grid of a batch: blocks of 32 x 8 threads each cover 32 x 32
// cells (128 x 32 for the finish, four cells of a row per thread), numbered grid by grid
// (prefix[g] = first block of grid g, block_job[b] = grid of block b).
constexpr int kBatchRows = 32;

template <int OP>
__global__ void __launch_bounds__(256) advect_batch_kernel(const AdvectJob* __restrict__ jobs,
                                                           const int* __restrict__ prefix,
                                                           const int* __restrict__ block_job, int* nonfinite) {
    const int b = blockIdx.x;
    const int g = __ldg(block_job + b);
    const AdvectJob& J = jobs[g];
    const int lb = b - __ldg(prefix + g);
    const int bx = (J.A.cols + (OP == 1 ? 127 : 31)) / (OP == 1 ? 128 : 32);
    const int j = (lb % bx) * 32 + threadIdx.x, i0 = (lb / bx) * kBatchRows;
    if (OP == 0) {
        splat_rows<4>(J.in0, J.in1, J.in2, J.out0, J.A, i0 + 4 * threadIdx.y, j);
    } else if (OP == 1) {
        int bad = 0;
#pragma unroll
        for (int r = 0; r < kBatchRows; r += 8)
            if (i0 + r + threadIdx.y < J.A.rows && 4 * j < J.A.cols)
                bad |= finish_group(J.in0, J.out0, J.smooth, J.A, i0 + r + threadIdx.y, 4 * j);
        if (bad && nonfinite) report_nonfinite(nonfinite);
    } else {
        advect_rows<4>(J.in0, J.in1, J.out0, J.out1, J.A, i0 + 4 * threadIdx.y, j);
    }
}

// Blocks of 32 x 8 threads over the grid, per_x columns and per_y rows a block.
dim3 grid_for(int rows, int cols, int per_x, int per_y) {
    return dim3((cols + per_x - 1) / per_x, std::min((rows + per_y - 1) / per_y, 65535));
}

// Cells of a column per thread: four give a warp the reads to keep in flight and the splat
// its sums along the column; small grids then have too few warps to hide a read's latency.
// Whole steps (15 diffusion, 20 pressure sweeps), us with 1 and with 4: 130 x 130 41.0 and
// 43.1, 771 x 1283 87.1 and 88.1, 1154 x 1154 100.7 and 100.2, 1400 x 1400 144.5 and 143.5,
// 1540 x 1540 160.2 and 159.3, 1700 x 1700 186.4 and 183.7, 2050 x 2050 259 and 252,
// 8194 x 8194 3569 and 3436.
bool four_rows(int rows, int cols) { return (long)rows * cols >= 2L << 20; }

}  // namespace

cudaError_t launch_splat(const float* d0, const float* u, const float* v, float* acc, const AdvectArgs& A,
                         cudaStream_t st) {
    if (four_rows(A.rows, A.cols))
        splat_kernel<4><<<grid_for(A.rows, A.cols, 32, 32), dim3(32, 8), 0, st>>>(d0, u, v, acc, A);
    else
        splat_kernel<1><<<grid_for(A.rows, A.cols, 32, 8), dim3(32, 8), 0, st>>>(d0, u, v, acc, A);
    return cudaGetLastError();
}

cudaError_t launch_density_finish(const float* acc, float* d, int smooth, const AdvectArgs& A, int* nonfinite,
                                  cudaStream_t st) {
    density_finish_kernel<<<grid_for(A.rows, A.cols, 128, 8), dim3(32, 8), 0, st>>>(acc, d, smooth, A, nonfinite);
    return cudaGetLastError();
}

cudaError_t launch_advect_velocity(const float* u0, const float* v0, float* u, float* v, const AdvectArgs& A,
                                   cudaStream_t st) {
    if (four_rows(A.rows, A.cols))
        advect_velocity_kernel<4><<<grid_for(A.rows, A.cols, 32, 32), dim3(32, 8), 0, st>>>(u0, v0, u, v, A);
    else
        advect_velocity_kernel<1><<<grid_for(A.rows, A.cols, 32, 8), dim3(32, 8), 0, st>>>(u0, v0, u, v, A);
    return cudaGetLastError();
}

int advect_batch_blocks(int op, int rows, int cols) {
    const int per = op == 1 ? 128 : 32;
    return ((cols + per - 1) / per) * ((rows + kBatchRows - 1) / kBatchRows);
}

cudaError_t launch_advect_batch(int op, const AdvectJob* jobs, const int* prefix, const int* block_job, int nblocks,
                                int* nonfinite, cudaStream_t st) {
    if (nblocks <= 0) return cudaSuccess;
    if (op == 0)
        advect_batch_kernel<0><<<nblocks, dim3(32, 8), 0, st>>>(jobs, prefix, block_job, nonfinite);
    else if (op == 1)
        advect_batch_kernel<1><<<nblocks, dim3(32, 8), 0, st>>>(jobs, prefix, block_job, nonfinite);
    else
        advect_batch_kernel<2><<<nblocks, dim3(32, 8), 0, st>>>(jobs, prefix, block_job, nonfinite);
    return cudaGetLastError();
}

}  // namespace fs
