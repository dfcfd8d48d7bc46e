// Temporally blocked 5-point Jacobi passes for diffusion and pressure.
//
// Reference behaviour (mworchel/fluid-2d src/fluid_solver_gpu.cu):
//   diffuse 290-312 + diffuse_iteration_kernel 69-85: per sweep, a D2D copy of the
//     field, one Jacobi kernel, a device sync, one boundary kernel, a device sync;
//   project 358-404 + kernels 164-206: clear div and p, divergence, Neumann fill,
//     Kp x (copy, Jacobi, fill), gradient subtract, two reflecting fills.
// That is ~20 B/cell of HBM traffic and two launches per sweep. Here one launch runs
// `sweeps` sweeps of one or more fields: each CTA holds a region of 128 columns x RH rows
// (its output tile grown by a halo of at least `sweeps` cells) in registers, sweeps it
// with the boundary fill's effect reproduced exactly after every sweep, and writes only
// its output tile back. The first pass of a solve fuses what precedes it (add_sources for
// diffusion, the divergence for pressure); the gradient subtract and the two reflecting
// fills follow a projection's passes as a launch of their own (gradient_kernel).
//
// Arithmetic follows the reference's operand order with explicit round-to-nearest
// intrinsics and a fused multiply-add exactly where the reference's compiled kernels fuse
// one (add_sources x + dt*s and the diffusion numerator x0 + a*sum). The reference divides
// by D = 1.0 + 4.0*a in double; FP64 is slow on GB300, so the quotient is formed as
//   q = fma(num, rh, num*rl),   rh + rl = 1/D split into two floats:
// the error before the last rounding is below 2^-47 of the quotient (the split's and the small
// product's) while num*rl is a normal number, and at most 2^-150 more below, so q is the
// correctly rounded quotient or, where that lies so close to a rounding boundary, the float
// next to it. 0 of 2^28 random quotients of numerators near one (a from 1e-4 to 1e4) differed
// from (float)((double)num / D), against 1 for the Newton-corrected quotient of two more
// operations that this replaced. Of 2^24 at each smaller magnitude, this and Newton: none down
// to 2^-92; 133 and 0 at 2^-100, 3 % and 0.3 % at 2^-120, 0.6 % and 4.6 % at 2^-130, none by
// more than one unit in the last place.

#include <algorithm>

#include "fs_internal.cuh"
#include "tc.cuh"

namespace fs {
namespace {

// ---------------------------------------------------------------------------
// A region in registers.
//
// The CTA's NW warps own R rows each and a lane owns four consecutive columns, so a thread
// holds an R x 4 block of the field and of its constant term (x0 or div) for the whole
// pass: global memory is read and written once, 16 bytes per access and 512 contiguous
// bytes per warp and row. The block is kept as rows of two float2, X[i][0] = columns 0-1 and
// X[i][1] = columns 2-3, the register order of the 16-byte accesses, so that one packed FP32
// instruction (FADD2 / FMUL2 / FFMA2, each lane rounding exactly as the scalar form) updates
// two cells and no register is moved to form a pair. Per sweep and row:
//   left / right neighbours: the thread's own columns and one shuffle per side; their sums
//     are scalar adds, since a pair shifted by one column is not a register pair;
//   up / down neighbours: the rows above and below, packed; above the first and below the
//     last row of the block a double-buffered exchange area in shared memory (each warp
//     publishes its first and last rows as float4, one barrier per sweep; the rows that need
//     no published row are updated before the barrier, which hides most of its wait).
// What bounds it: the FP32 pipe and instruction issue. A pressure sweep is 5 operations per
// cell, a diffusion sweep 6. (Pairs of rows (i, i + 4) instead would be packed throughout,
// but every 16-byte access and every published or received row then needs its registers
// moved: 2435 against 1743 warp instructions per tile and warp of 8 diffusion sweeps.)
// At 2050 x 2050 a pass of 8 sweeps takes 37.3 us for two diffused fields and 21.2 us for
// the pressure (ncu, cold caches; 51-53 and 28-29 us with the field in registers but the
// constant term in shared memory and edge tiles staged there), the FP32 pipe 57 % busy. At
// 8194 x 8194 a pressure pass takes 143 us up to 4 sweeps, the rate of HBM (5.6 TB/s), 220 us
// with 8 and 0.35 us more per sweep and tile beyond, 88 % of the FP32 pipe's rate.
//
// Regions and tiles (field_tiling). Every region lies inside the grid where the grid is
// large enough: the first one starts at row (column) 0 and the last one ends at the last
// row (column group), so only grids smaller than a region mask rows or lanes, and an edge
// row or column sits at a fixed place of its warp or lane: row 0 in warp 0's first row,
// row rows-1 in the last warp's last row, column 0 in lane 0, column cols-1 in lane 31.
// Region columns start at multiples of four and output tiles begin and end at multiples
// of four columns, so that loads and stores are whole 16-byte groups. A group may reach
// past the last column into the row's padding: the padding holds values nothing reads.
// Cells at the border of a region read clamped neighbours and compute values that nothing
// stored depends on (the halo is at least the number of sweeps).
//
// Domain edges. The reference fills the edge cells after every sweep with their inner
// neighbour's new value times a sign (set_boundary_*, fluid_solver_gpu.cu:11-54), corners
// excepted. Here every cell of the block is updated by the stencil, and from the second
// sweep on the edge cells are filled just before a sweep reads them: in the thread itself
// where edge and inner cell share a thread, and otherwise in the value received from the
// neighbour (the shuffled column or the exchanged row is replaced by sign x the inner
// cell's own value, the float the fill would have stored). Only interior cells' values
// ever depend on an edge cell, and never on a corner. The fill is applied once more before
// the stores; corners get their input value back.

struct Coef2 {
    float2 a, rh, rl;  // diffusion: a, and 1/(1 + 4a) as rh + rl (head of this file)
};

// Four cells of a row from its neighbours: l, r the columns left and right of the row's
// four, U and D the rows above and below.
template <bool DIFF>
__device__ __forceinline__ void update4(float2 (&y)[2], const float2 (&x)[2], const float2 (&k)[2], float l, float r,
                                        const float2 (&U)[2], const float2 (&D)[2], const Coef2& c) {
    if (DIFF) {
        // (x0 + a*(L + R + U + D)) / (1 + 4a), fluid_solver_gpu.cu:81-82
        float2 s[2] = {make_float2(__fadd_rn(l, x[0].y), __fadd_rn(x[0].x, x[1].x)),
                       make_float2(__fadd_rn(x[0].y, x[1].y), __fadd_rn(x[1].x, r))};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            s[h] = __fadd2_rn(s[h], U[h]);
            s[h] = __fadd2_rn(s[h], D[h]);
            const float2 num = __ffma2_rn(c.a, s[h], k[h]);
            y[h] = __ffma2_rn(num, c.rh, __fmul2_rn(num, c.rl));
        }
    } else {
        // (div + R + L + D + U) / 4, fluid_solver_gpu.cu:187-188
        float2 s[2] = {make_float2(__fadd_rn(__fadd_rn(k[0].x, x[0].y), l), __fadd_rn(__fadd_rn(k[0].y, x[1].x), x[0].x)),
                       make_float2(__fadd_rn(__fadd_rn(k[1].x, x[1].y), x[0].y), __fadd_rn(__fadd_rn(k[1].y, r), x[1].x))};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            s[h] = __fadd2_rn(s[h], D[h]);
            s[h] = __fadd2_rn(s[h], U[h]);
            y[h] = __fmul2_rn(s[h], make_float2(0.25f, 0.25f));
        }
    }
}

// x / b correctly rounded, for b > 0 with y = RN(1/b): Markstein's correction step
// (P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34(1), 1990): q0 = RN(x*y), r = x - q0*b (exact with one
// FMA), RN(q0 + r*y) = RN(x/b) while x, the quotient and r stay in the normal range.
// Zero (x / b = x for b > 0), very small or large and non-finite x take the IEEE
// division. Used for the gradient subtract's division by h.
__device__ __noinline__ float ieee_div(float x, float b) { return __fdiv_rn(x, b); }

__device__ __forceinline__ float div_by(float x, float b, float y) {
    const float ax = fabsf(x);
    if (ax > 0x1p-100f && ax < 0x1p100f) {
        const float q0 = __fmul_rn(x, y);
        const float r = __fmaf_rn(-q0, b, x);
        return __fmaf_rn(r, y, q0);
    }
    return ax == 0.f ? x : ieee_div(x, b);  // out of line: rare, and keeps the kernel small
}

// Where a thread's block meets the domain edge.
constexpr int kELeft = 1;    // its column 0 is grid column 0
constexpr int kERight = 2;   // its column qe > 0 is grid column cols - 1
constexpr int kERightN = 4;  // grid column cols - 1 is the next lane's column 0
constexpr int kETop = 8;     // its row 0 is grid row 0
constexpr int kEBot = 16;    // its row ib > 0 is grid row rows - 1
constexpr int kEBotN = 32;   // grid row rows - 1 is the next warp's row 0
constexpr int kEOnly = 64;   // its column 0 is column cols - 1, or its row 0 row rows - 1
// Edge::tile, the same in every thread of the CTA: some lane has the column flag. A branch on
// these is one the whole warp takes or not, and the lane's own flag then only selects (a
// branch on the lane's flag took both sides one after the other: 41.0 against 39.5 us for a
// step of 130 x 130).
constexpr int kTLeft = 128, kTRight = 256, kTRightN = 512;
struct Edge {
    int flags, tile;
    int qe, ib;
    float s_lr, s_tb;
};

template <int I> __device__ __forceinline__ float& colref(float2 (&x)[2]) {
    return (I & 1) ? x[I >> 1].y : x[I >> 1].x;
}
__device__ __forceinline__ float colval(const float2 (&x)[2], int q) { return (q & 1) ? x[q >> 1].y : x[q >> 1].x; }
__device__ __forceinline__ float2 scale2(float sg, float2 v) { return make_float2(__fmul_rn(sg, v.x), __fmul_rn(sg, v.y)); }
template <int R, int DST, int SRC> __device__ __forceinline__ void fill_row(float2 (&X)[R][2], float sg) {
    if (DST < R) {
        X[DST % R][0] = scale2(sg, X[SRC % R][0]);
        X[DST % R][1] = scale2(sg, X[SRC % R][1]);
    }
}
template <int R, int DST, int SRC> __device__ __forceinline__ void fill_col(float2 (&X)[R][2], bool mine, float sg) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const float v = __fmul_rn(sg, colref<SRC>(X[i]));
        colref<DST>(X[i]) = mine ? v : colref<DST>(X[i]);
    }
}

// The reference's edge fill where edge and inner cell share this thread's block. Corner
// cells this also writes are never read by interior cells.
template <int R> __device__ __forceinline__ void fill_in_thread(float2 (&X)[R][2], const Edge& e, float s_lr, float s_tb) {
    if (e.tile & kTLeft) fill_col<R, 0, 1>(X, e.flags & kELeft, s_lr);
    if (e.tile & kTRight) {
        const bool mine = e.flags & kERight;
        if (e.qe == 1) fill_col<R, 1, 0>(X, mine, s_lr);
        else if (e.qe == 2) fill_col<R, 2, 1>(X, mine, s_lr);
        else fill_col<R, 3, 2>(X, mine, s_lr);
    }
    if (e.flags & kETop) fill_row<R, 0, 1>(X, s_tb);
    if (e.flags & kEBot) {
        if (e.ib == R - 1) {  // the last row of a region that ends at the grid's last row
            fill_row<R, R - 1, R - 2>(X, s_tb);
        } else {
            switch (e.ib) {  // grids of fewer rows than a region
                case 1: fill_row<R, 1, 0>(X, s_tb); break;
                case 2: fill_row<R, 2, 1>(X, s_tb); break;
                case 3: fill_row<R, 3, 2>(X, s_tb); break;
                case 4: fill_row<R, 4, 3>(X, s_tb); break;
                case 5: fill_row<R, 5, 4>(X, s_tb); break;
                case 6: fill_row<R, 6, 5>(X, s_tb); break;
                default: break;
            }
        }
    }
}

// One pass over the block X: body(i, l, r, U, D) for every row i with its neighbours (the
// columns left and right of the row's four, the rows above and below), in tiles that touch
// the domain edge (EDGE) with the edge fill folded in when `fold`. E: the exchange buffer
// of this pass (2 rows of 128 floats per warp). X is filled in place where edge and inner
// cell share a thread.
template <int R, int NW, bool EDGE, class Body>
__device__ __forceinline__ void for_neighbours(float2 (&X)[R][2], float* __restrict__ E, int w, int lane, bool fold,
                                               const Edge& e, Body&& body) {
    constexpr int RW = kRegionW;
    constexpr unsigned FULL = 0xffffffffu;
    if (EDGE && fold) fill_in_thread<R>(X, e, e.s_lr, e.s_tb);
    const int my_top = 2 * w * RW + 4 * lane, my_bot = my_top + RW;
    *reinterpret_cast<float2*>(E + my_top) = X[0][0];
    *reinterpret_cast<float2*>(E + my_top + 2) = X[0][1];
    *reinterpret_cast<float2*>(E + my_bot) = X[R - 1][0];
    *reinterpret_cast<float2*>(E + my_bot + 2) = X[R - 1][1];
    const bool over_r = e.flags & kERightN;
    auto row = [&](int i, const float2 (&U)[2], const float2 (&D)[2]) {
        const float l = __shfl_up_sync(FULL, X[i][1].y, 1);
        float r = __shfl_down_sync(FULL, X[i][0].x, 1);
        if (EDGE && fold && (e.tile & kTRightN)) r = over_r ? __fmul_rn(e.s_lr, X[i][1].y) : r;
        body(i, l, r, U, D);
    };
    // rows that need no published row
#pragma unroll
    for (int i = 1; i < R - 1; ++i) row(i, X[i - 1], X[i + 1]);
    __syncthreads();
    // bottom row of warp w - 1 and top row of warp w + 1; the first and last warps read
    // their own rows instead (the region border, whose values nothing stored uses)
    const float4 u4 = *reinterpret_cast<const float4*>(E + (w > 0 ? my_top - RW : my_top));
    const float4 d4 = *reinterpret_cast<const float4*>(E + (w < NW - 1 ? my_top + 2 * RW : my_bot));
    const float2 up[2] = {make_float2(u4.x, u4.y), make_float2(u4.z, u4.w)};
    float2 dn[2] = {make_float2(d4.x, d4.y), make_float2(d4.z, d4.w)};
    if (EDGE && fold && (e.flags & kEBotN)) {
        dn[0] = scale2(e.s_tb, X[R - 1][0]);
        dn[1] = scale2(e.s_tb, X[R - 1][1]);
    }
    row(0, up, X[1]);
    row(R - 1, X[R - 2], dn);
}

// 16-byte (VEC) or per-column access to columns c0 .. c0+3 of a row. VEC needs 16-byte
// aligned rows (pitch a multiple of four, aligned buffers); otherwise only columns below
// cols are touched.
template <bool VEC> __device__ __forceinline__ float4 load4(const float* p, int n) {
    if (VEC) return __ldcg(reinterpret_cast<const float4*>(p));
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (n > 0) v.x = __ldcg(p);
    if (n > 1) v.y = __ldcg(p + 1);
    if (n > 2) v.z = __ldcg(p + 2);
    if (n > 3) v.w = __ldcg(p + 3);
    return v;
}
template <bool VEC> __device__ __forceinline__ void store4(float* p, float4 v, int n) {
    if (VEC) {
        *reinterpret_cast<float4*>(p) = v;
        return;
    }
    if (n > 0) p[0] = v.x;
    if (n > 1) p[1] = v.y;
    if (n > 2) p[2] = v.z;
    if (n > 3) p[3] = v.w;
}
__device__ __forceinline__ float4 row4(const float2 (&x)[2]) { return make_float4(x[0].x, x[0].y, x[1].x, x[1].y); }
__device__ __forceinline__ void set4(float4& v, int q, float x) {
    if (q == 0) v.x = x;
    else if (q == 1) v.y = x;
    else if (q == 2) v.z = x;
    else v.w = x;
}

// A thread's place in its tile.
struct Place {
    int w, lane;
    int gyb, c0;     // grid row and column of the block's first cell
    int nrow;        // block rows inside the grid (may exceed the block or be <= 0)
    int ncol;        // columns c0 .. of the grid (may exceed four or be <= 0)
    int r_lo, r_hi;  // output rows of the block
    bool ocol;       // the block's columns are output columns
};

// Stores the block's output rows of a field whose sweeps are done: the edge fill (signs
// s_lr, s_tb), the rows, the edge row below the block where the next warp owns it, and the
// corners' input values from src (null: zero).
template <int R, bool VEC>
__device__ __forceinline__ void store_filled(float2 (&X)[R][2], float* __restrict__ y, const float* __restrict__ src,
                                             const Place& t, const Edge& e, float s_lr, float s_tb, size_t o,
                                             size_t pitch, bool edge_tile) {
    constexpr unsigned FULL = 0xffffffffu;
    if (!edge_tile) {
        if (!t.ocol) return;
        float* p = y + o;
#pragma unroll
        for (int i = 0; i < R; ++i, p += pitch)
            if (i >= t.r_lo && i < t.r_hi) store4<VEC>(p, row4(X[i]), t.ncol);
        return;
    }
    fill_in_thread<R>(X, e, s_lr, s_tb);
    // column cols - 1 in a lane's column 0: its inner neighbour is the previous lane's
    if (__any_sync(FULL, e.flags & kERightN)) {
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float inner = __shfl_up_sync(FULL, X[i][1].y, 1);
            if (t.ncol == 1) X[i][0].x = __fmul_rn(s_lr, inner);
        }
    }
    if (!t.ocol) return;
    // the corners of an edge row keep their input
    auto corners = [&](float4& v, size_t off) {
        if (t.c0 == 0) v.x = src ? __ldcg(src + off) : 0.f;
        if (t.ncol >= 1 && t.ncol <= 4) set4(v, t.ncol - 1, src ? __ldcg(src + off + (t.ncol - 1)) : 0.f);
    };
    const int hi = min(t.r_hi, t.nrow);
    // a last row that the previous warp's inner row fills is stored by that warp
    const bool skip0 = t.nrow == 1 && t.w > 0;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        if (i < t.r_lo || i >= hi || (i == 0 && skip0)) continue;
        float4 v = row4(X[i]);
        const size_t off = o + (size_t)i * pitch;
        if ((i == 0 && (e.flags & kETop)) || (i == e.ib && (e.flags & kEBot))) corners(v, off);
        store4<VEC>(y + off, v, t.ncol);
    }
    if ((e.flags & kEBotN) && t.r_hi > R) {
        float4 v = row4(X[R - 1]);
        v = make_float4(__fmul_rn(s_tb, v.x), __fmul_rn(s_tb, v.y), __fmul_rn(s_tb, v.z), __fmul_rn(s_tb, v.w));
        const size_t off = o + (size_t)R * pitch;
        corners(v, off);
        store4<VEC>(y + off, v, t.ncol);
    }
}

// The sweeps of one tile on its block X with constant terms K.
template <int R, int NW, bool DIFF, bool EDGE>
__device__ __forceinline__ void run_sweeps(float2 (&X)[R][2], const float2 (&K)[R][2], float* E0, float* E1, int n,
                                           const Place& t, const Edge& e, const Coef2& c) {
    float2 Y[R][2];
    auto sweep = [&](float2 (&A)[R][2], float2 (&B)[R][2], float* E, bool fold) {
        for_neighbours<R, NW, EDGE>(A, E, t.w, t.lane, fold, e,
                                    [&](int i, float l, float r, const float2 (&U)[2], const float2 (&D)[2]) {
                                        update4<DIFF>(B[i], A[i], K[i], l, r, U, D, c);
                                    });
    };
    int s = 0;
#pragma unroll 1
    for (; s + 1 < n; s += 2) {
        sweep(X, Y, E0, s > 0);
        sweep(Y, X, E1, true);
    }
    if (s < n) {
        sweep(X, Y, E0, s > 0);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            X[i][0] = Y[i][0];
            X[i][1] = Y[i][1];
        }
    }
}

// A CTA's walk over the tiles of a field, every `stride`-th from tile t on, without a
// division per tile. The columns rotate by one tile per tile row: a CTA would otherwise stay
// in one column (the slower edge column) where its stride is a multiple of the tiles per row.
struct TileWalk {
    int ty, tx;         // tile row and (unrotated) column
    int rot;            // ty mod n
    int n, dy, dx, dr;  // tiles per row; the stride in rows and columns, dy mod n
    __device__ __forceinline__ void start(const StencilField& F, int t, int stride) {
        n = F.tiles_x;
        ty = t / n;
        tx = t - ty * n;
        rot = ty % n;
        dy = stride / n;
        dx = stride - dy * n;
        dr = dy % n;
    }
    __device__ __forceinline__ void next() {
        tx += dx;
        const int carry = tx >= n ? 1 : 0;
        tx -= carry ? n : 0;
        ty += dy + carry;
        rot += dr + carry;
        rot -= rot >= n ? n : 0;
    }
    __device__ __forceinline__ int col() const { return tx + rot >= n ? tx + rot - n : tx + rot; }
};

// First row and column of this thread's block in tile (ty, tx).
template <int R>
__device__ __forceinline__ void tile_origin(const StencilField& F, int ty, int tx, int w, int lane, int& gyb, int& c0) {
    gyb = min(ty * F.tile_h, F.gy_last) + w * R;
    c0 = min(tx * F.tile_w, F.gx_last) + 4 * lane;
}

// Prefetch of a tile's block into shared memory by the TMA engine: each warp copies its own
// rows on its own mbarrier (no CTA barrier is needed to read them back), R rows of the field
// and R rows of the second array (constant term or sources; of v in a first pressure pass
// R + 2, from the row above the block on), 512 bytes a row. What lies outside the grid is
// zero-filled. A CTA prefetches its next tile while it sweeps the current one: loading each
// tile only when its turn came left the warps waiting on global loads for 37 % of their time,
// and one 16-byte cp.async per thread and row held up the shuffles and exchange rows behind
// it in the load/store unit's queue (two diffused fields at 2050^2, 8 sweeps: 39.6 us a pass
// against 37.3).
template <int R> constexpr int stage_rows() { return 2 * R + 2; }
template <int R, int NW> __device__ __forceinline__ float4* stage_ptr() {
    extern __shared__ __align__(128) float4 smem4[];
    return smem4 + (4 * NW + (threadIdx.x >> 5) * stage_rows<R>()) * (kRegionW / 4);
}
template <int R, int NW> __device__ __forceinline__ uint64_t* stage_bar() {
    extern __shared__ __align__(128) float4 smem4[];
    return reinterpret_cast<uint64_t*>(smem4 + (4 + stage_rows<R>()) * NW * (kRegionW / 4)) + (threadIdx.x >> 5);
}
// Once per kernel, by every warp.
template <int R, int NW> __device__ __forceinline__ void stage_init() {
    if ((threadIdx.x & 31) == 0) {
        tc::mbar_init(stage_bar<R, NW>(), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc::fence_proxy_async_smem();
    }
    __syncwarp();
}
__device__ __forceinline__ void tma_load(unsigned dst, const CUtensorMap* map, int x, int y, unsigned bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
// mx, mk: the tensor maps of the field and of the second array (boxes of 128 columns x R, for
// v R + 2, rows). Column coordinates are multiples of four (16 bytes).
template <int R, int NW, bool DIFF>
__device__ __forceinline__ void prefetch_tile(const StencilField& F, int ty, int tx, const CUtensorMap* mx,
                                              const CUtensorMap* mk) {
    int gyb, gx;
    tile_origin<R>(F, ty, tx, threadIdx.x >> 5, 0, gyb, gx);
    if ((threadIdx.x & 31) == 0) {
        const bool border = !DIFF && F.kind == PASS_PRESSURE_FIRST;
        const unsigned bar = tc::smem_u32(stage_bar<R, NW>()), dst = tc::smem_u32(stage_ptr<R, NW>());
        constexpr unsigned row = 4 * kRegionW;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"((border ? 2 * R + 2 : 2 * R) * row)
                     : "memory");
        tma_load(dst, mx, gx, gyb, bar);
        tma_load(dst + R * row, mk, gx, border ? gyb - 1 : gyb, bar);
    }
}
// Waits for the warp's prefetch, the same answer in every lane; false when the wait gave up:
// after `polls` polls of about 120 ns, or without such a bound after 2^20 suspending tries
// (1.3 us each).
constexpr unsigned kStageWait = 1u << 20;
__device__ __forceinline__ bool stage_wait(uint64_t* bar, unsigned parity, unsigned polls) {
    unsigned left = polls != 0 ? polls : kStageWait;
    bool there;
    while (!(there = polls != 0 ? tc::mbar_test_wait(bar, parity) : tc::mbar_try_wait(bar, parity)) && --left != 0)
        if (polls != 0) __nanosleep(100);
    return __all_sync(0xffffffffu, there);
}
// After a wait that gave up: the copy may still be on its way into the warp's rows, so one more
// bounded wait, that it does not outlive the CTA, and NaN in the lane's columns of the rows.
// Out of line: inlined, its registers cost the residual-driven solve 1 %.
template <int ROWS>
__device__ __noinline__ void stage_give_up(uint64_t* bar, unsigned parity, float4* rows) {
    for (unsigned left = kStageWait; !tc::mbar_try_wait(bar, parity) && --left != 0;) {
    }
    const float nan = __int_as_float(0x7fffffff);
    for (int k = 0; k < ROWS; ++k) rows[k * 32] = make_float4(nan, nan, nan, nan);
}

// The same wait without a result to carry: it reports a wait that gave up by itself (*error = 1)
// and waits once more as long, so that the barrier is armed again behind its copy. For kernels
// whose every result is void once the word is set, batches and solves on 64-row regions. One
// statement, since the compiler's registers and schedule around the loop above cost those
// kernels 1 to 2 % (batch of 24 grids of 64 to 512 a side 278 against 275 us a step; steps of
// two solves of 512 sweeps, 514 x 514 and 2050 x 2050, 938 and 3310 against 926 and 3270;
// 128-row regions, 1026 x 1026, are the other way round: 1308 against 1319).
__device__ __forceinline__ void stage_wait_or_report(uint64_t* bar, unsigned parity, int* error) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .u32 left;\n mov.u32 left, %3;\n"
        "W%=:\n mbarrier.try_wait.parity.shared::cta.b64 p, [%0], %1;\n @p bra D%=;\n"
        " sub.u32 left, left, 1;\n setp.ne.u32 p, left, %4;\n @p bra N%=;\n st.volatile.global.u32 [%2], 1;\n"
        "N%=:\n setp.ne.u32 p, left, 0;\n @p bra W%=;\n"
        "D%=:\n}\n" ::"r"(tc::smem_u32(bar)),
        "r"(parity), "l"(error), "n"(2 * kStageWait), "n"(kStageWait)
        : "memory");
}

// What a warp carries from tile to tile: the parity of its prefetch and whether a wait for one
// gave up, and the exchange buffer that the next sweep uses (so that no barrier is needed
// between tiles).
constexpr unsigned kPhase = 1, kGaveUp = 2;
struct Carry {
    unsigned stage = 0;
    int buf = 0;
    __device__ __forceinline__ unsigned phase() const { return stage & kPhase; }
    __device__ __forceinline__ bool gave_up() const { return stage >= kGaveUp; }
};

// Tile (ty, tx) of one pass: load the region (fusing add_sources or the divergence into the
// first pass), run n sweeps, store the output tile, then the optional residual partial sums (for
// residual-driven pressure solves). xin/yout stand in for F.x/F.y so a persistent caller can
// ping-pong buffers across passes. VEC: the block comes from the prefetch (polls: the bound of the wait
// for it), and `next` starts the next tile's once it has been read. A warp whose wait gave up
// fills its staged rows with NaN and prefetches nothing more (its barrier's parity would no
// longer tell one copy from another), so that this block and all that follow are NaN; the
// kernel reports it at its end. SELF: the wait reports to `error` by itself instead.
template <int R, int NW, bool DIFF, bool VEC, bool RESID, bool SELF, class Next>
__device__ __forceinline__ void process_tile(const StencilField& F, int n, int ty, int tx, const float* __restrict__ xin,
                                             float* __restrict__ yout, bool resid, float& rnum, float& rden,
                                             Carry& carry, unsigned polls, int* error, Next&& next) {
    constexpr int RW = kRegionW;
    constexpr unsigned FULL = 0xffffffffu;
    extern __shared__ float4 smem4[];
    // the two exchange buffers, the next sweep's first
    float* const E0 = reinterpret_cast<float*>(smem4) + carry.buf * (2 * NW * RW);
    float* const E1 = reinterpret_cast<float*>(smem4) + (carry.buf ^ 1) * (2 * NW * RW);
    Place t;
    t.w = threadIdx.x >> 5;
    t.lane = threadIdx.x & 31;
    tile_origin<R>(F, ty, tx, t.w, t.lane, t.gyb, t.c0);
    const int rows = F.rows, cols = F.cols;
    const size_t pitch = (size_t)F.pitch;
    t.nrow = rows - t.gyb;
    t.ncol = cols - t.c0;
    const int hx = (F.halo + 3) & ~3;
    t.r_lo = (ty == 0 ? 0 : ty * F.tile_h + F.halo) - t.gyb;
    t.r_hi = (ty == F.tiles_y - 1 ? rows : (ty + 1) * F.tile_h + F.halo) - t.gyb;
    t.ocol = t.c0 >= (tx == 0 ? 0 : tx * F.tile_w + hx) && t.c0 < (tx == F.tiles_x - 1 ? cols : (tx + 1) * F.tile_w + hx);
    const bool edge_tile = ty == 0 || tx == 0 || ty == F.tiles_y - 1 || tx == F.tiles_x - 1;
    Edge e{};
    e.s_lr = DIFF ? F.s_lr : 1.f;  // the pressure's fill is a copy
    e.s_tb = DIFF ? F.s_tb : 1.f;
    if (edge_tile) {
        e.qe = (cols - 1) & 3;
        e.ib = t.nrow - 1;
        e.flags = (t.c0 == 0 ? kELeft : 0) | (t.ncol >= 2 && t.ncol <= 4 ? kERight : 0) | (t.ncol == 5 ? kERightN : 0) |
                  (t.gyb == 0 ? kETop : 0) | (t.nrow >= 2 && t.nrow <= R ? kEBot : 0) | (t.nrow == R + 1 ? kEBotN : 0) |
                  (t.ncol == 1 || t.nrow == 1 ? kEOnly : 0);
        e.tile = (tx == 0 ? kTLeft : 0) | (tx == F.tiles_x - 1 ? (e.qe == 0 ? kTRightN : kTRight) : 0);
        // the residual-driven solve has no register left for it: one word with the lane's flags
        // (256 sweeps at 1026 x 1026 310 us, 316 with its own)
        if (RESID) e.tile = e.flags |= e.tile;
    }
    const size_t o = (size_t)t.gyb * pitch + t.c0;
    const bool lane_in = t.ncol > 0;
    float4* const S = stage_ptr<R, NW>() + t.lane;

    float2 X[R][2], K[R][2];
    auto put = [](float2 (&x)[2], float4 v) {
        x[0] = make_float2(v.x, v.y);
        x[1] = make_float2(v.z, v.w);
    };
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load = [&](const float* base, int i) {
        return lane_in && i < t.nrow ? load4<VEC>(base + o + (size_t)i * pitch, t.ncol) : zero4;
    };
    // row i of the field and of the second array (rows -1 and R of a first pressure pass too)
    auto load_x = [&](int i) { return VEC ? S[i * 32] : load(xin, i); };
    const int k0 = !DIFF && F.kind == PASS_PRESSURE_FIRST ? R + 1 : R;
    auto load_k = [&](const float* base, int i) {
        if (VEC) return S[(k0 + i) * 32];
        if (i < 0) return lane_in && t.gyb > 0 && t.nrow > 0 ? load4<VEC>(base + o - pitch, t.ncol) : zero4;
        return load(base, i);
    };
    // columns q of this block and rows i that are interior cells of the grid
    auto int_col = [&](int q) { return t.c0 + q >= 1 && q <= t.ncol - 2; };
    auto int_row = [&](int i) { return t.gyb + i >= 1 && i <= t.nrow - 2; };
    if (SELF) {
        stage_wait_or_report(stage_bar<R, NW>(), carry.phase(), error);
        carry.stage ^= kPhase;
    } else if (VEC && !carry.gave_up()) {
        if (stage_wait(stage_bar<R, NW>(), carry.phase(), polls)) {
            carry.stage ^= kPhase;
        } else {
            carry.stage |= kGaveUp;
            stage_give_up<stage_rows<R>()>(stage_bar<R, NW>(), carry.phase(), S);
        }
    }

    // ------------------------------------------------------------------ load
    if (!DIFF && F.kind == PASS_PRESSURE_FIRST) {
        // divergence_kernel (fluid_solver_gpu.cu:173-174): div = cdiv*(((uR - uL) + vD) - vU)
        // on interior cells, zero on the edge; the starting pressure (zero without one).
        const float cdiv = F.cdiv;
        const float* __restrict__ vp = F.x2;
        float4 vu = load_k(vp, -1), vc = load_k(vp, 0);
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const float4 vd = load_k(vp, i + 1);
            const float4 u = load_x(i);
            const float uL = __shfl_up_sync(FULL, u.w, 1), uR = __shfl_down_sync(FULL, u.x, 1);
            const float ul[4] = {uL, u.x, u.y, u.z}, ur[4] = {u.y, u.z, u.w, uR};
            const float dn[4] = {vd.x, vd.y, vd.z, vd.w}, upv[4] = {vu.x, vu.y, vu.z, vu.w};
            float dv[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float sd = __fsub_rn(ur[q], ul[q]);
                sd = __fadd_rn(sd, dn[q]);
                sd = __fsub_rn(sd, upv[q]);
                dv[q] = !edge_tile || (int_col(q) && int_row(i)) ? __fmul_rn(cdiv, sd) : 0.f;
            }
            put(K[i], make_float4(dv[0], dv[1], dv[2], dv[3]));
            vu = vc;
            vc = vd;
        }
        const float* __restrict__ start = F.cst;
#pragma unroll
        for (int i = 0; i < R; ++i) put(X[i], start ? load(start, i) : zero4);
    } else {
        float4 x4[R], k4[R];
        const bool first = DIFF && F.kind == PASS_DIFFUSE_FIRST;
        const float* __restrict__ kin = first ? F.x2 : F.cst;
#pragma unroll
        for (int i = 0; i < R; ++i) x4[i] = load_x(i);
#pragma unroll
        for (int i = 0; i < R; ++i) k4[i] = load_k(kin, i);
        if (first) {
            // add_sources_kernel (fluid_solver_gpu.cu:64), fused as compiled: x0 = x + dt*s
            // on interior cells
            const float dt = F.dt;
#pragma unroll
            for (int i = 0; i < R; ++i) {
                float4 f = make_float4(__fmaf_rn(dt, k4[i].x, x4[i].x), __fmaf_rn(dt, k4[i].y, x4[i].y),
                                       __fmaf_rn(dt, k4[i].z, x4[i].z), __fmaf_rn(dt, k4[i].w, x4[i].w));
                if (edge_tile && e.flags) {
                    if (!(int_row(i) && int_col(0))) f.x = x4[i].x;
                    if (!(int_row(i) && int_col(1))) f.y = x4[i].y;
                    if (!(int_row(i) && int_col(2))) f.z = x4[i].z;
                    if (!(int_row(i) && int_col(3))) f.w = x4[i].w;
                }
                x4[i] = k4[i] = f;
            }
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            put(X[i], x4[i]);
            put(K[i], k4[i]);
        }
    }
    if (VEC) {
        __syncwarp();  // the block has been read
        if (!carry.gave_up()) next();
    }
    if ((DIFF ? F.kind == PASS_DIFFUSE_FIRST : F.kind == PASS_PRESSURE_FIRST) && F.cst_out != nullptr && t.ocol) {
        const int hi = min(t.r_hi, t.nrow);
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (i >= t.r_lo && i < hi) store4<VEC>(F.cst_out + o + (size_t)i * pitch, row4(K[i]), t.ncol);
    }

    // ------------------------------------------------------------------ sweeps
    if (n > 0) {
        const Coef2 c = {make_float2(F.a, F.a), make_float2(F.rh, F.rh), make_float2(F.rl, F.rl)};
        if (edge_tile)
            run_sweeps<R, NW, DIFF, true>(X, K, E0, E1, n, t, e, c);
        else
            run_sweeps<R, NW, DIFF, false>(X, K, E0, E1, n, t, e, c);
    }

    // ------------------------------------------------------------------ store
    const float* src = !DIFF && F.kind == PASS_PRESSURE_FIRST ? F.cst : xin;
    if (yout != nullptr) {
        if (n > 0) {
            store_filled<R, VEC>(X, yout, src, t, e, e.s_lr, e.s_tb, o, pitch, edge_tile);
        } else if (t.ocol) {
            const int hi = min(t.r_hi, t.nrow);
#pragma unroll
            for (int i = 0; i < R; ++i)
                if (i >= t.r_lo && i < hi) store4<VEC>(yout + o + (size_t)i * pitch, row4(X[i]), t.ncol);
        }
    }

    // ------------------------------------------------ residual partial sums
    // ||div + sum(nbrs) - 4p||^2 and ||div||^2 over this tile's interior output cells,
    // from the final p (valid one ring beyond the tile: halo = sweeps + 1).
    carry.buf ^= n & 1;
    if (RESID && resid) {
        float* const E = (n & 1) ? E1 : E0;
        carry.buf ^= 1;
        for_neighbours<R, NW, true>(X, E, t.w, t.lane, n > 0, e,
                                    [&](int i, float l, float r, const float2 (&U)[2], const float2 (&D)[2]) {
            const bool row = t.ocol && i >= t.r_lo && i < t.r_hi && int_row(i);
            const float ls[4] = {l, X[i][0].x, X[i][0].y, X[i][1].x}, rs[4] = {X[i][0].y, X[i][1].x, X[i][1].y, r};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if (!(row && int_col(q))) continue;
                const float k = colval(K[i], q);
                float sres = __fadd_rn(k, rs[q]);
                sres = __fadd_rn(sres, ls[q]);
                sres = __fadd_rn(sres, colval(D, q));
                sres = __fadd_rn(sres, colval(U, q));
                const float res = __fsub_rn(sres, __fmul_rn(4.f, colval(X[i], q)));
                rnum = fmaf(res, res, rnum);
                rden = fmaf(k, k, rden);
            }
        });
    }
}

// Gradient subtract and reflecting fills as a separate pass, from a final pressure p whose
// edge cells are already filled: remove_p_kernel (fluid_solver_gpu.cu:202-203) on interior
// cells, then set_boundary_opposite_horizontal(u) / _vertical(v) (fluid_solver_gpu.cu:
// 402-403): an edge cell takes its inner neighbour's new value, negated for the normal
// component; corners keep their input value. Bound by memory (p, u, v read, u, v written:
// 209 us at 8194 x 8194, 198 at HBM's measured rate).
__device__ __forceinline__ void gradient_cell(const float* __restrict__ p, const float* __restrict__ u_in,
                                              const float* __restrict__ v_in, int i, int j, int rows, int cols,
                                              size_t pitch, float h, float rh, float& un, float& vn) {
    const bool ri = i >= 1 && i <= rows - 2, ci = j >= 1 && j <= cols - 2;
    const size_t o = (size_t)i * pitch + j;
    if (!ri && !ci) {
        un = __ldg(u_in + o);
        vn = __ldg(v_in + o);
        return;
    }
    int ii = i, jj = j;
    float su = 1.f, sv = 1.f;
    if (!ci) {  // left / right edge
        jj = (j == 0) ? 1 : cols - 2;
        su = -1.f;
    } else if (!ri) {  // top / bottom edge
        ii = (i == 0) ? 1 : rows - 2;
        sv = -1.f;
    }
    const size_t q = (size_t)ii * pitch + jj;
    const float gu = div_by(__fmul_rn(0.5f, __fsub_rn(__ldg(p + q + 1), __ldg(p + q - 1))), h, rh);
    const float gv = div_by(__fmul_rn(0.5f, __fsub_rn(__ldg(p + q + pitch), __ldg(p + q - pitch))), h, rh);
    un = su * __fsub_rn(__ldg(u_in + q), gu);
    vn = sv * __fsub_rn(__ldg(v_in + q), gv);
}

// Four consecutive cells (i, j0 .. j0 + 3) of the gradient subtract: an interior group
// with 16-byte loads and stores (p's row and its rows above and below, two more p values
// at the group's ends), a group touching an edge cell per cell. Requires the rows 16-byte
// aligned (pitch a multiple of four, buffers 16-byte aligned). Returns true when an
// output is NaN or Inf.
__device__ __forceinline__ bool gradient_group(const float* __restrict__ p, const float* __restrict__ u_in,
                                               const float* __restrict__ v_in, float* __restrict__ u_out,
                                               float* __restrict__ v_out, int i, int j0, int rows, int cols,
                                               size_t P, float h, float rh) {
    const size_t o = (size_t)i * P + j0;
    float un[4], vn[4];
    int n = 4;
    if (i >= 1 && i <= rows - 2 && j0 >= 1 && j0 + 3 <= cols - 2) {
        const float4 pc = __ldg(reinterpret_cast<const float4*>(p + o));
        const float4 pu = __ldg(reinterpret_cast<const float4*>(p + o - P));
        const float4 pd = __ldg(reinterpret_cast<const float4*>(p + o + P));
        const float4 u4 = __ldg(reinterpret_cast<const float4*>(u_in + o));
        const float4 v4 = __ldg(reinterpret_cast<const float4*>(v_in + o));
        const float pl0 = __ldg(p + o - 1), pr3 = __ldg(p + o + 4);
        const float pcv[6] = {pl0, pc.x, pc.y, pc.z, pc.w, pr3};
        const float puv[4] = {pu.x, pu.y, pu.z, pu.w}, pdv[4] = {pd.x, pd.y, pd.z, pd.w};
        const float uv[4] = {u4.x, u4.y, u4.z, u4.w}, vv[4] = {v4.x, v4.y, v4.z, v4.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float gu = div_by(__fmul_rn(0.5f, __fsub_rn(pcv[k + 2], pcv[k])), h, rh);
            const float gv = div_by(__fmul_rn(0.5f, __fsub_rn(pdv[k], puv[k])), h, rh);
            un[k] = __fsub_rn(uv[k], gu);
            vn[k] = __fsub_rn(vv[k], gv);
        }
        *reinterpret_cast<float4*>(u_out + o) = make_float4(un[0], un[1], un[2], un[3]);
        *reinterpret_cast<float4*>(v_out + o) = make_float4(vn[0], vn[1], vn[2], vn[3]);
    } else {
        n = min(4, cols - j0);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k >= n) break;
            gradient_cell(p, u_in, v_in, i, j0 + k, rows, cols, P, h, rh, un[k], vn[k]);
            u_out[o + k] = un[k];
            v_out[o + k] = vn[k];
        }
    }
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k < n) bad |= !(isfinite(un[k]) && isfinite(vn[k]));
    return bad;
}

// One thread per four consecutive cells of a row: gradient_group, or for rows without
// 16-byte alignment (VEC false) and a caller's rows cell by cell.
template <bool VEC>
__global__ void __launch_bounds__(256) gradient_kernel(const float* p0, const float* __restrict__ u_in,
                                                       const float* __restrict__ v_in, float* __restrict__ u_out,
                                                       float* __restrict__ v_out, int rows, int cols, int pitch,
                                                       float h, int* nonfinite, const float* p_alt, const int* sel) {
    const int j0 = 4 * (blockIdx.x * 32 + threadIdx.x);
    if (j0 >= cols) return;
    const float* __restrict__ p = (sel != nullptr && __ldcg(sel) != 0) ? p_alt : p0;
    const float rh = __frcp_rn(h);
    bool bad = false;
    for (int i = blockIdx.y * 8 + threadIdx.y; i < rows; i += 8 * gridDim.y) {
        if (VEC) {
            bad |= gradient_group(p, u_in, v_in, u_out, v_out, i, j0, rows, cols, (size_t)pitch, h, rh);
        } else {
            for (int j = j0; j < min(cols, j0 + 4); ++j) {
                float un, vn;
                gradient_cell(p, u_in, v_in, i, j, rows, cols, (size_t)pitch, h, rh, un, vn);
                u_out[(size_t)i * pitch + j] = un;
                v_out[(size_t)i * pitch + j] = vn;
                bad |= !(isfinite(un) && isfinite(vn));
            }
        }
    }
    if (bad && nonfinite) report_nonfinite(nonfinite);
}

// Batched form: blocks of 32 x 8 threads over 128 columns x kGradBatchRows rows of one
// grid (gradient_batch_blocks per grid), numbered grid by grid (prefix[g] = first block of
// grid g, block_job[b] = grid of block b); each thread takes four cells of a row, as
// gradient_kernel, in kGradBatchRows / 8 rows.
constexpr int kGradBatchRows = 32;
__global__ void __launch_bounds__(256) gradient_batch_kernel(const AdvectJob* __restrict__ jobs,
                                                             const int* __restrict__ prefix,
                                                             const int* __restrict__ block_job, int* nonfinite) {
    const int b = blockIdx.x;
    const int g = __ldg(block_job + b);
    const AdvectJob& J = jobs[g];
    const int lb = b - __ldg(prefix + g);
    const int rows = J.A.rows, cols = J.A.cols;
    const int bx = ((cols + 3) / 4 + 31) / 32;
    const int j0 = 4 * ((lb % bx) * 32 + threadIdx.x);
    const float h = J.A.h, rh = __frcp_rn(h);
    bool bad = false;
#pragma unroll
    for (int r = 0; r < kGradBatchRows; r += 8) {
        const int i = (lb / bx) * kGradBatchRows + r + threadIdx.y;
        if (i >= rows || j0 >= cols) continue;
        bad |= gradient_group(J.in0, J.in1, J.in2, J.out0, J.out1, i, j0, rows, cols, (size_t)J.A.pitch, h, rh);
    }
    if (bad && nonfinite) report_nonfinite(nonfinite);
}

// Rows a warp owns and warps of a CTA: 8 x 8 rows (64-row regions, two CTAs per SM) or
// 8 x 16 (128-row regions, one).
constexpr int kR = 8;

// One launch = one pass over the tiles of up to kMaxStencilFields fields: persistent CTAs,
// as many as are resident at once, each taking every gridDim.x-th tile and prefetching the
// next one while it sweeps. VEC: 16-byte rows (see load4).
template <int NW, bool DIFF, bool VEC>
__global__ void __launch_bounds__(32 * NW, (NW <= 8 ? 2 : 1))
    stencil_kernel(const __grid_constant__ StencilLaunch L, int total) {
    auto field_of = [&](int b) {
        int f = 0;
#pragma unroll 1
        while (f + 1 < L.nfields && b >= L.f[f + 1].tile_begin) ++f;
        return f;
    };
    int b = blockIdx.x, f = field_of(b);
    TileWalk walk;
    walk.start(L.f[f], b - L.f[f].tile_begin, gridDim.x);
    Carry carry;
    if (VEC) {
        stage_init<kR, NW>();
        prefetch_tile<kR, NW, DIFF>(L.f[f], walk.ty, walk.col(), &L.f[f].mx, &L.f[f].mk);
    }
    float rn = 0.f, rd = 0.f;
#pragma unroll 1
    while (b < total) {
        const int ty = walk.ty, tx = walk.col(), nb = b + gridDim.x;
        const int nf = nb < total ? field_of(nb) : f;
        if (nf == f)
            walk.next();
        else
            walk.start(L.f[nf], nb - L.f[nf].tile_begin, gridDim.x);
        const StencilField& F = L.f[f];
        process_tile<kR, NW, DIFF, VEC, false, false>(F, F.sweeps, ty, tx, F.x, F.y, false, rn, rd, carry, L.polls, nullptr, [&] {
            if (nb < total) prefetch_tile<kR, NW, DIFF>(L.f[nf], walk.ty, walk.col(), &L.f[nf].mx, &L.f[nf].mk);
        });
        b = nb;
        f = nf;
    }
    if (carry.gave_up()) report_timeout(L.flags);
}

// One pass over the fields of a batch of grids of uneven size, up to kMaxWideFields
// of them, with their descriptors in the launch's parameters like the single-grid
// kernel's, a tile's field found by a binary search of the fields' first tiles.
template <int NW, bool DIFF>
__global__ void __launch_bounds__(32 * NW, (NW <= 8 ? 2 : 1)) stencil_wide_kernel(const __grid_constant__ WideLaunch L) {
    auto field_of = [&](int b) {
        int lo = 0, hi = L.nfields - 1;
#pragma unroll 1
        while (lo < hi) {  // the last field whose first tile is <= b
            const int mid = (lo + hi + 1) >> 1;
            if (L.begin[mid] <= b)
                lo = mid;
            else
                hi = mid - 1;
        }
        return lo;
    };
    const int total = L.begin[L.nfields];
    int b = blockIdx.x, f = field_of(b);
    TileWalk walk;
    walk.start(L.f[f], b - L.begin[f], gridDim.x);
    Carry carry;
    stage_init<kR, NW>();
    prefetch_tile<kR, NW, DIFF>(L.f[f], walk.ty, walk.col(), &L.f[f].mx, &L.f[f].mk);
    float rn = 0.f, rd = 0.f;
#pragma unroll 1
    while (b < total) {
        const int ty = walk.ty, tx = walk.col(), nb = b + gridDim.x;
        const int nf = nb < total ? field_of(nb) : f;
        if (nf == f)
            walk.next();
        else
            walk.start(L.f[nf], nb - L.begin[nf], gridDim.x);
        const StencilField& F = L.f[f];
        process_tile<kR, NW, DIFF, true, false, true>(F, F.sweeps, ty, tx, F.x, F.y, false, rn, rd, carry, 0, L.timed_out, [&] {
            if (nb < total) prefetch_tile<kR, NW, DIFF>(L.f[nf], walk.ty, walk.col(), &L.f[nf].mx, &L.f[nf].mk);
        });
        b = nb;
        f = nf;
    }
}

// ---------------------------------------------------------------------------
// Residual-driven pressure solve in one persistent cooperative launch. What bounds it on
// small and middle grids is what a round costs beside its sweeps. Cycles of a 16-sweep round
// at 514 x 514 before the sums, the outcome and the barrier took their present form: sweeps
// 8,900 (13,900 in an edge tile), load 1,000, store 600-2,400, residual sums 3,300, barrier
// 6,200, outcome 6,300. 256 sweeps there: 385 us in single passes, 289 in pairs, 230 with
// short sums and the one-word barrier (1026 x 1026: 472 and 319 us, 2050 x 2050: 874 and 790).
// What is left there (ncu): the barriers of the sweeps (3.1 of 7.9 cycles a warp spends per
// instruction at 514 x 514, 4.4 of 11.5 at 1026 x 1026) with issue 25 and 35 % busy.

constexpr unsigned kBarrierSpinLimit = 1u << 24;  // default: ~2 s of polling, then give up

// Grid-wide barrier for a cooperative launch (all CTAs co-resident): a CTA adds its arrival
// and waits until `target` arrivals are there, one word and one trip to the L2 each way. The
// wait is bounded: after `limit` polls the CTA sets ctrl->error and the word's top bit, which
// ends every wait, so the kernel always terminates. Returns false once that has happened.
constexpr unsigned long long kBarrierGaveUp = 1ull << 63;
__device__ __forceinline__ unsigned long long poll_arrivals(const unsigned long long* bar) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(bar) : "memory");
    return v;
}
__device__ __forceinline__ bool grid_barrier(SolveCtrl* ctrl, unsigned long long target, unsigned limit) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(&ctrl->bar) : "memory");
        unsigned spins = 0;
        unsigned long long v;
        while ((v = poll_arrivals(&ctrl->bar)) < target) {
            if (++spins > limit) {
                atomicExch(&ctrl->error, 1);
                atomicOr(&ctrl->bar, kBarrierGaveUp);
                v = kBarrierGaveUp;
                break;
            }
            __nanosleep(32);
        }
        s_ok = v < kBarrierGaveUp;
    }
    __syncthreads();
    return s_ok != 0;
}

template <int NW>
__global__ void __launch_bounds__(32 * NW, (NW <= 8 ? 2 : 1))
    pressure_solve_kernel(const __grid_constant__ PressureSolve P) {
    const unsigned G = gridDim.x;
    const int tid = threadIdx.x, nt = blockDim.x;
    const unsigned ntiles = P.mid.tiles_x * P.mid.tiles_y;
    int passes = 0;
    double ratio = 0.0;
    bool ok = true, done = false;
    int cur = -1;  // index in P.p of the latest pressure; -1 before the first pass
    // segment mode, converged in an earlier segment: the flag was written by an earlier
    // launch, so every CTA reads the same value and none waits at a barrier
    if (P.segment && __ldcg(&P.ctrl->converged)) return;
    const unsigned lim_set = P.poll_limit ? __ldcg(P.poll_limit) : 0u;
    const unsigned limit = lim_set ? lim_set : kBarrierSpinLimit;
    Carry carry;
    stage_init<kR, NW>();
    __shared__ float s_sum[2][32 * NW];
    __shared__ double s_ratio;
    // the next barrier's arrivals: earlier segments left a multiple of G, and none of this
    // launch's barriers completes before this CTA's arrival
    unsigned long long target = poll_arrivals(&P.ctrl->bar);
    target = target - target % G;
#pragma unroll 1
    for (int round = 0; ok && !done && passes < P.max_passes; ++round) {
        const StencilField& F = cur < 0 ? P.first : P.mid;
        const float* x = cur < 0 ? F.x : P.p[cur];
        const CUtensorMap* const mx = cur < 0 ? &F.mx : &P.mp[cur];
        const int dst = cur < 0 ? 0 : cur ^ 1;
        // the residual is formed and tested after every second pass (and the last one
        // allowed): a pass without it skips the residual sums and the reduction, and a solve
        // runs at most one pass beyond the one that met the target. In pairs a round is two
        // passes, or a last one by itself.
        const int take = P.pair ? min(2, P.max_passes - passes) : 1;
        const bool check = P.pair || (passes & 1) || passes + 1 >= P.max_passes;
        float rn = 0.f, rd = 0.f;
        TileWalk walk;
        walk.start(F, blockIdx.x, G);
        // the previous pass's stores, ordered by the grid barrier, before the TMA engine reads
        asm volatile("fence.proxy.async;" ::: "memory");
        if (blockIdx.x < ntiles && !carry.gave_up())
            prefetch_tile<kR, NW, false>(F, walk.ty, walk.col(), mx, &F.mk);
#pragma unroll 1
        for (unsigned t = blockIdx.x; t < ntiles; t += G) {
            const int ty = walk.ty, tx = walk.col();
            walk.next();
            process_tile<kR, NW, false, true, true, NW <= 8>(F, take * F.sweeps, ty, tx, x, P.p[dst], check, rn, rd, carry, 0,
                                                    &P.ctrl->error, [&] {
                if (t + G < ntiles) prefetch_tile<kR, NW, false>(F, walk.ty, walk.col(), mx, &F.mk);
            });
        }
        double* part = P.partials + (size_t)(round & 1) * 2 * G;
        if (check) {
            s_sum[0][tid] = rn;
            s_sum[1][tid] = rd;
            __syncthreads();
            if (tid < 32) {
                const float* v = s_sum[tid >> 4];
                const double t = half_warp_sum(32 * NW, [&](int i) { return v[i]; });
                if ((tid & 15) == 0) part[2 * blockIdx.x + (tid >> 4)] = t;
            }
        }
        target += G;
        ok = grid_barrier(P.ctrl, target, limit);
        passes += take;
        cur = dst;
        if (!ok) break;
        if (!check) continue;
        // every CTA sums all partials in the same order, so all agree on the outcome
        if (tid < 32) {
            const double* v = part + (tid >> 4);
            const double t = half_warp_sum((int)G, [&](int i) { return __ldcg(v + 2 * i); });
            const double a = __shfl_sync(0xffffffffu, t, 0), b = __shfl_sync(0xffffffffu, t, 16);
            if (tid == 0) s_ratio = b > 0.0 ? sqrt(a / b) : sqrt(a);
        }
        __syncthreads();
        ratio = s_ratio;
        done = ratio <= (double)P.tol;
    }
    if (ok && cur >= 0) {
        if (P.segment) {
            // every CTA passed the last pass's barrier: the final pressure is complete
            const float4* src = reinterpret_cast<const float4*>(P.p[cur]);
            float4* dst = reinterpret_cast<float4*>(P.p_cur);
            const long n4 = (long)P.mid.rows * P.mid.pitch / 4;
            for (long e = (long)blockIdx.x * nt + tid; e < n4; e += (long)G * nt) dst[e] = __ldcg(src + e);
        } else {
            // the final pressure: which buffer holds it (the gradient pass that follows
            // reads it there), and a copy for the next step's warm start
            if (blockIdx.x == 0 && tid == 0) P.ctrl->cur = cur;
            if (P.p_out) {
                const float4* src = reinterpret_cast<const float4*>(P.p[cur]);
                float4* dst = reinterpret_cast<float4*>(P.p_out);
                const long n4 = (long)P.mid.rows * P.mid.pitch / 4;
                for (long e = (long)blockIdx.x * nt + tid; e < n4; e += (long)G * nt) dst[e] = __ldcg(src + e);
            }
        }
    }
    if (carry.gave_up()) atomicExch(&P.ctrl->error, 1);
    if (blockIdx.x == 0 && tid == 0) {
        P.ctrl->passes = (P.segment ? P.ctrl->passes : 0) + passes;
        P.ctrl->residual = ratio;
        P.ctrl->converged = ok && ratio <= (double)P.tol;
    }
}

// Exchange rows (two per warp, double-buffered), the prefetched block of each warp and its
// barrier.
constexpr size_t smem_bytes(int nw) { return (size_t)nw * ((4 + stage_rows<kR>()) * kRegionW * sizeof(float) + 8); }

// CTAs of a pass that are resident at once on the current device.
cudaError_t resident_ctas(int nw, int* n) {
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    *n = sms * (nw <= 8 ? 2 : 1);
    return e;
}

template <class K> cudaError_t opt_in(K* kernel, int nw) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(nw));
}
template <int NW> cudaError_t prepare_variant() {
    cudaError_t e = opt_in(stencil_kernel<NW, true, true>, NW);
    if (e == cudaSuccess) e = opt_in(stencil_kernel<NW, false, true>, NW);
    if (e == cudaSuccess) e = opt_in(stencil_kernel<NW, false, false>, NW);
    if (e == cudaSuccess) e = opt_in(pressure_solve_kernel<NW>, NW);
    if (e == cudaSuccess) e = opt_in(stencil_wide_kernel<NW, true>, NW);
    if (e == cudaSuccess) e = opt_in(stencil_wide_kernel<NW, false>, NW);
    return e;
}

// Whether the two arrays that a pass reads are there: a launch without one is refused, since the
// kernels read both whatever they are.
const float* second_array(const StencilField& f) {
    return f.kind == PASS_DIFFUSE_FIRST || f.kind == PASS_PRESSURE_FIRST ? f.x2 : f.cst;
}
bool complete(const StencilField& f) { return f.x != nullptr && second_array(f) != nullptr; }

// Tensor map of a field's rows in boxes of `box` rows x 128 columns (base and pitch 16-byte
// aligned).
cudaError_t encode_map(CUtensorMap* map, const float* base, int rows, int cols, int pitch, int box) {
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess)
            fn = nullptr;
        return reinterpret_cast<Encode>(fn);
    }();
    if (!encode) return cudaErrorNotSupported;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch * sizeof(float)};
    const cuuint32_t boxes[2] = {(cuuint32_t)kRegionW, (cuuint32_t)box}, steps[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(base), dims, strides, boxes, steps,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t encode_second(StencilField& f) {
    return encode_map(&f.mk, second_array(f), f.rows, f.cols, f.pitch, f.kind == PASS_PRESSURE_FIRST ? kR + 2 : kR);
}
cudaError_t encode_field(StencilField& f) {
    const cudaError_t e = encode_map(&f.mx, f.x, f.rows, f.cols, f.pitch, kR);
    return e == cudaSuccess ? encode_second(f) : e;
}

template <int NW>
cudaError_t launch_wide_variant(const WideLaunch& L, bool diffuse, cudaStream_t st) {
    if (L.nfields <= 0 || L.nfields > kMaxWideFields) return cudaErrorInvalidValue;
    const int total = L.begin[L.nfields];
    if (total <= 0) return cudaSuccess;
    int ctas = 0;
    cudaError_t e = resident_ctas(NW, &ctas);
    if (e != cudaSuccess) return e;
    ctas = std::min(ctas, total);
    if (diffuse)
        stencil_wide_kernel<NW, true><<<ctas, 32 * NW, smem_bytes(NW), st>>>(L);
    else
        stencil_wide_kernel<NW, false><<<ctas, 32 * NW, smem_bytes(NW), st>>>(L);
    return cudaGetLastError();
}

template <int NW>
cudaError_t solve_blocks(int* blocks) {
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, pressure_solve_kernel<NW>, 32 * NW, smem_bytes(NW));
    *blocks = per * sms;
    return e;
}

template <int NW>
cudaError_t launch_solve_variant(const PressureSolve& P, int blocks, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(32 * NW);
    cfg.dynamicSmemBytes = smem_bytes(NW);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, pressure_solve_kernel<NW>, P);
}

// 16-byte rows: every buffer of the field aligned, and the pitch.
bool vector_rows(const StencilField& f) {
    const void* ptrs[] = {f.x, f.x2, f.cst, f.y, f.cst_out};
    uintptr_t bits = (uintptr_t)f.pitch * sizeof(float);
    for (const void* p : ptrs) bits |= reinterpret_cast<uintptr_t>(p);
    return (bits & 15) == 0;
}

template <int NW>
cudaError_t launch_variant(StencilLaunch& L, cudaStream_t st) {
    const size_t smem = smem_bytes(NW);
    int blocks = 0;
    bool vec = true;
    for (int i = 0; i < L.nfields; ++i) {
        if (!complete(L.f[i])) return cudaErrorInvalidValue;
        blocks += L.f[i].tiles_x * L.f[i].tiles_y;
        vec = vec && vector_rows(L.f[i]);
    }
    if (blocks == 0) return cudaSuccess;
    int ctas = 0;
    cudaError_t e = resident_ctas(NW, &ctas);
    if (e != cudaSuccess) return e;
    ctas = std::min(ctas, blocks);
    for (int i = 0; vec && i < L.nfields; ++i)
        if ((e = encode_field(L.f[i])) != cudaSuccess) return e;
    // all fields of one launch are of the same class (diffusion or pressure); a handle's and
    // a batch's fields have 128-byte rows, only a caller's velocity may not
    const bool diff = L.f[0].kind == PASS_DIFFUSE_FIRST || L.f[0].kind == PASS_DIFFUSE;
    if (diff && !vec) return cudaErrorInvalidValue;
    if (diff)
        stencil_kernel<NW, true, true><<<ctas, 32 * NW, smem, st>>>(L, blocks);
    else if (vec)
        stencil_kernel<NW, false, true><<<ctas, 32 * NW, smem, st>>>(L, blocks);
    else
        stencil_kernel<NW, false, false><<<ctas, 32 * NW, smem, st>>>(L, blocks);
    return cudaGetLastError();
}

}  // namespace

// The halo is bounded by the region's rows and by its columns (whole groups of four on
// each side, and one group of output).
int stencil_max_halo(int tile_rows) { return std::min(tile_rows / 2 - 2, kRegionW / 2 - 4); }

// Opt the kernels into more than 48 KB of dynamic shared memory on the current
// device. Called once per handle at creation, outside any stream capture.
cudaError_t stencil_prepare() {
    cudaError_t e = prepare_variant<8>();
    if (e == cudaSuccess) e = prepare_variant<16>();
    return e;
}

cudaError_t launch_gradient(const float* p, const float* u_in, const float* v_in, float* u_out, float* v_out, int rows,
                            int cols, int pitch, float h, int* nonfinite, cudaStream_t st, const float* p_alt,
                            const int* sel) {
    const bool vec = pitch % 4 == 0 &&
                     ((reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(p_alt) |
                       reinterpret_cast<uintptr_t>(u_in) | reinterpret_cast<uintptr_t>(v_in) |
                       reinterpret_cast<uintptr_t>(u_out) | reinterpret_cast<uintptr_t>(v_out)) & 15) == 0;
    const dim3 grid(((cols + 3) / 4 + 31) / 32, std::min((rows + 7) / 8, 65535));
    if (vec)
        gradient_kernel<true><<<grid, dim3(32, 8), 0, st>>>(p, u_in, v_in, u_out, v_out, rows, cols, pitch, h, nonfinite,
                                                            p_alt, sel);
    else
        gradient_kernel<false><<<grid, dim3(32, 8), 0, st>>>(p, u_in, v_in, u_out, v_out, rows, cols, pitch, h,
                                                             nonfinite, p_alt, sel);
    return cudaGetLastError();
}

int gradient_batch_blocks(int rows, int cols) {
    return (((cols + 3) / 4 + 31) / 32) * ((rows + kGradBatchRows - 1) / kGradBatchRows);
}

cudaError_t launch_gradient_batch(const AdvectJob* jobs, const int* prefix, const int* block_job, int nblocks,
                                  int* nonfinite, cudaStream_t st) {
    if (nblocks <= 0) return cudaSuccess;
    gradient_batch_kernel<<<nblocks, dim3(32, 8), 0, st>>>(jobs, prefix, block_job, nonfinite);
    return cudaGetLastError();
}

cudaError_t launch_stencil(StencilLaunch& L, int tile_rows, cudaStream_t st) {
    if (tile_rows == 128) return launch_variant<16>(L, st);
    return launch_variant<8>(L, st);
}

cudaError_t pressure_solve_max_blocks(int tile_rows, int* blocks) {
    if (tile_rows == 128) return solve_blocks<16>(blocks);
    return solve_blocks<8>(blocks);
}

cudaError_t launch_pressure_solve(PressureSolve& P, int tile_rows, int blocks, cudaStream_t st) {
    if (blocks <= 0 || !complete(P.first) || !P.mid.cst || !P.p[0] || !P.p[1]) return cudaErrorInvalidValue;
    cudaError_t e = encode_field(P.first);
    if (e == cudaSuccess) e = encode_second(P.mid);  // its field is p[0] or p[1]
    for (int k = 0; k < 2 && e == cudaSuccess; ++k)
        e = encode_map(&P.mp[k], P.p[k], P.mid.rows, P.mid.cols, P.mid.pitch, kR);
    if (e != cudaSuccess) return e;
    if (tile_rows == 128) return launch_solve_variant<16>(P, blocks, st);
    return launch_solve_variant<8>(P, blocks, st);
}

cudaError_t prepare_stencil_wide(WideLaunch& L) {
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < L.nfields && e == cudaSuccess; ++i)
        e = complete(L.f[i]) ? encode_field(L.f[i]) : cudaErrorInvalidValue;
    return e;
}

cudaError_t launch_stencil_wide(const WideLaunch& L, bool diffuse, int tile_rows, cudaStream_t st) {

    if (tile_rows == 128) return launch_wide_variant<16>(L, diffuse, st);
    return launch_wide_variant<8>(L, diffuse, st);
}

}  // namespace fs
