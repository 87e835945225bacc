// ytgb_offaxis.cu -- octree off-axis projection by cell splatting.
//
// add_cells_to_image_offaxis (image_utilities.pyx:167-289) projects every
// cell of an octree dataset along the camera's normal: the cell's projected
// square is cut into jmax x kmax sub-squares ("subcells", jmax = kmax =
// 2^depth, capped by the stamp extent), each weighted by the precomputed
// stamp of that depth (the projected thickness of a unit cube) and spread
// bilinearly over the pixels it overlaps (_add_cell_to_image_offaxis,
// :46-165).
//
// The per-subcell weights are separable: subcell (j, k) gives pixel (P, Q)
//     stamp[j][k] * fx_j(P) * fy_k(Q) * dx^3 Nx Ny * q,
// with fx_j(P) = dvx_j where P is the subcell's left pixel jj1 and
// 1 - dvx_j where P is its right pixel jj2 (likewise in y).  The reference
// evaluates the boundaries ((j - jmax/2) dx_loc + x) Nx, their truncations
// and dvx per subcell; here they are evaluated once per row and column of
// subcells, with the same float64 operations in the same order, into a
// per-warp table, so every subcell lands on exactly the reference's pixels
// with the reference's dvx, dvy.  One warp then handles one cell: each lane
// owns one pixel column Q (and a share of the rows j), sums
// stamp[j][k] * fy_k(Q) over the few k that touch Q, spreads the row sum
// over P with fx_j, and adds each finished pixel to the image with one
// float64 atomic per buffer, scaled by dx^3 Nx Ny q (resp. w).  Only the
// association of the products differs from the reference: the sums are
// float64 fused multiply-adds, a few roundings per contribution.  Cells whose rows exceed the table take the
// reference's per-subcell loop (with atomics) instead.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <string>

#include "ytgb.h"
#include "ytgb_internal.h"
#include "ytgb_ray.cuh"

namespace {

using namespace ytgb;

constexpr int OA_BLOCK = 128;
constexpr int OA_WARPS = OA_BLOCK / 32;
constexpr int OA_KT = 256;  // subcells per row or column held in the table

constexpr int OA_MAXK = 10;  // subcells of a row meeting one pixel column, held in registers

struct AxisTable {
    int edge[OA_KT + 1];  // (int) of the subcell boundaries, in pixels
    double dv[OA_KT];     // fclip((edge[i+1] - b_i) / (b_{i+1} - b_i), 0, 1)
    double uv[OA_KT];     // 1 - dv
};

// fp_utils.pxd:17-40 (fmax, fmin, fclip)
__device__ __forceinline__ double fpmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double fpmin(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ double fclip(double f, double a, double b) { return fpmin(fpmax(f, a), b); }

// Subcell boundary i of an axis in pixels: ((i - m / 2.) * d_loc + x) * N
// (image_utilities.pyx:110-111, 124-125)
__device__ __forceinline__ double boundary(int i, int m, double d_loc, double x, int N) {
    return ytgb::dmul(ytgb::dadd(ytgb::dmul(ytgb::dsub((double)i, (double)m * 0.5), d_loc), x), (double)N);
}

// Entry i of an axis table: boundaries i and i + 1, their truncations and
// dv (image_utilities.pyx:110-120 and 124-138); entry m - 1 also stores the
// last edge.
__device__ __forceinline__ void fill_entry(AxisTable &t, int i, int m, double d_loc, double x, int N) {
    const double b0 = boundary(i, m, d_loc, x, N), b1 = boundary(i + 1, m, d_loc, x, N);
    const int e1 = __double2int_rz(b1);
    t.edge[i] = __double2int_rz(b0);
    if (i == m - 1) t.edge[m] = e1;
    const double dv = fclip(ytgb::ddiv(ytgb::dsub((double)e1, b0), ytgb::dsub(b1, b0)), 0.0, 1.0);
    t.dv[i] = dv;
    t.uv[i] = ytgb::dsub(1.0, dv);
}

// ceil(log2(v)) for finite v > 1 as the C library's log2 gives it: E for
// v = 2^E exactly, E + 1 when v lies more than 2^12 ulps above 2^E (log2(v)
// then exceeds E by over ten of its own ulps), and the library log2 in the
// narrow band between.
__device__ __forceinline__ int ceil_log2_above1(double v) {
    const long long b = dbits(v);
    const int E = (int)(b >> 52) - 1023;
    const long long f = b & MANT52;
    if (f == 0) return E;
    if (f >= 4096) return E + 1;
    return __double2int_rz(ceil(log2(v)));
}

// smallest k in [0, m) with edge[k + 1] >= Q (m if none)
__device__ __forceinline__ int first_reaching(const AxisTable &t, int m, int Q) {
    int lo = 0, hi = m;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (t.edge[mid + 1] >= Q) hi = mid;
        else lo = mid + 1;
    }
    return lo;
}

// largest k in [0, m) with edge[k] <= Q (-1 if none)
__device__ __forceinline__ int last_starting(const AxisTable &t, int m, int Q) {
    int lo = 0, hi = m;  // first k with edge[k] > Q, minus one
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (t.edge[mid] > Q) hi = mid;
        else lo = mid + 1;
    }
    return lo - 1;
}

struct PixelRun {
    int P = -1;
    double acc = 0.0;
};

__device__ __forceinline__ void flush(PixelRun &r, double *buf, double *bufw, long long Q, int nx, long long npix,
                                      double cq, double cw) {
    if (r.P >= 0) {
        const long long idx = (long long)r.P * nx + Q;
        if (idx < npix) {
            atomicAdd(buf + idx, ytgb::dmul(r.acc, cq));
            atomicAdd(bufw + idx, ytgb::dmul(r.acc, cw));
        }
    }
}

// acc += t * f for pixel P, flushing the previous pixel when P moves on
// (the pixels of a column arrive in nondecreasing order)
__device__ __forceinline__ void add_to(PixelRun &r, int P, double t, double f, double *buf, double *bufw, long long Q,
                                       int nx, long long npix, double cq, double cw) {
    if (P != r.P) {
        flush(r, buf, bufw, Q, nx, npix, cq, cw);
        r.P = P;
        r.acc = 0.0;
    }
    r.acc = __fma_rn(t, f, r.acc);
}

struct Column {
    const double *stamp;  // this depth's stamp
    long long nsy;
    int klo, kcap, Q, nx;  // kcap: the last subcell of a row
    long long npix;
    double cq, cw;
    double *buf, *bufw;
};

// One pixel column Q over the subcell rows [j0, j1): the row's sum of
// stamp[j][k] * fy_k(Q) over the N subcells k = klo .. klo + N - 1 that
// meet Q (weights w), spread over the row's two pixels with dvx, 1 - dvx.
template <int N>
__device__ __forceinline__ void column_rows(const AxisTable &tx, const Column &c, const double (&wk)[OA_MAXK], int j0,
                                            int j1) {
    PixelRun run;
    for (int j = j0; j < j1; j++) {
        const int e0 = tx.edge[j], e1 = tx.edge[j + 1];
        if (e1 < 0 || e0 >= c.nx) continue;  // image_utilities.pyx:116
        const double *srow = c.stamp + (long long)j * c.nsy;
        double t = 0.0;
#pragma unroll
        for (int u = 0; u < N; u++) t = __fma_rn(__ldg(srow + min(c.klo + u, c.kcap)), wk[u], t);
        if (e0 >= 0) add_to(run, e0, t, tx.dv[j], c.buf, c.bufw, c.Q, c.nx, c.npix, c.cq, c.cw);
        if (e1 < c.nx) add_to(run, e1, t, tx.uv[j], c.buf, c.bufw, c.Q, c.nx, c.npix, c.cq, c.cw);
    }
    flush(run, c.buf, c.bufw, c.Q, c.nx, c.npix, c.cq, c.cw);
}

// the same with the weights read from the table (more than OA_MAXK subcells
// of a row in one pixel: a very wide image against its height)
__device__ void column_rows_wide(const AxisTable &tx, const AxisTable &ty, const Column &c, int khi, int j0, int j1) {
    PixelRun run;
    for (int j = j0; j < j1; j++) {
        const int e0 = tx.edge[j], e1 = tx.edge[j + 1];
        if (e1 < 0 || e0 >= c.nx) continue;
        const double *srow = c.stamp + (long long)j * c.nsy;
        double t = 0.0;
        for (int k = c.klo; k <= khi; k++) {
            const double st = __ldg(srow + k);
            if (ty.edge[k] == c.Q) t = __fma_rn(st, ty.dv[k], t);
            if (ty.edge[k + 1] == c.Q) t = __fma_rn(st, ty.uv[k], t);
        }
        if (e0 >= 0) add_to(run, e0, t, tx.dv[j], c.buf, c.bufw, c.Q, c.nx, c.npix, c.cq, c.cw);
        if (e1 < c.nx) add_to(run, e1, t, tx.uv[j], c.buf, c.bufw, c.Q, c.nx, c.npix, c.cq, c.cw);
    }
    flush(run, c.buf, c.bufw, c.Q, c.nx, c.npix, c.cq, c.cw);
}

// The reference's own per-subcell loop (image_utilities.pyx:105-165) for a
// cell whose subcell rows do not fit the table: lanes over the subcells.
__device__ void cell_direct(const ytgb_offaxis_args &a, int lane, int depth, int jm, int km, double dx_loc,
                            double dy_loc, double x, double y, double dx3, double w, double q) {
    const int nx = a.nx, ny = a.ny;
    const long long npix = (long long)nx * ny;
    const long long n_sub = (long long)jm * km;
    for (long long s = lane; s < n_sub; s += 32) {
        const int j = (int)(s / km), k = (int)(s % km);
        const double xx1 = boundary(j, jm, dx_loc, x, nx), xx2 = boundary(j + 1, jm, dx_loc, x, nx);
        const int jj1 = __double2int_rz(xx1), jj2 = __double2int_rz(xx2);
        if (jj2 < 0 || jj1 >= nx) continue;
        const double dvx = fclip(ytgb::ddiv(ytgb::dsub((double)jj2, xx1), ytgb::dsub(xx2, xx1)), 0.0, 1.0);
        const double st = __ldg(a.stamp + ((long long)depth * a.nsx + j) * a.nsy + k);
        if (st == 0.0) continue;  // outside the stamp's mask
        const double yy1 = boundary(k, km, dy_loc, y, ny), yy2 = boundary(k + 1, km, dy_loc, y, ny);
        const int kk1 = __double2int_rz(yy1), kk2 = __double2int_rz(yy2);
        if (kk2 < 0 || kk1 >= ny) continue;
        const double tmp = ytgb::dmul(st, dx3);
        const double sw = ytgb::dmul(tmp, w), sq = ytgb::dmul(tmp, q);
        const double dvy = fclip(ytgb::ddiv(ytgb::dsub((double)kk2, yy1), ytgb::dsub(yy2, yy1)), 0.0, 1.0);
        const double ux = ytgb::dsub(1.0, dvx), uy = ytgb::dsub(1.0, dvy);
        long long idx;
        double f;
        if (jj1 >= 0 && kk1 >= 0 && (idx = (long long)jj1 * nx + kk1) < npix) {
            f = ytgb::dmul(dvx, dvy);
            atomicAdd(a.buffer + idx, ytgb::dmul(sq, f));
            atomicAdd(a.buffer_weight + idx, ytgb::dmul(sw, f));
        }
        if (jj1 >= 0 && kk2 < ny && (idx = (long long)jj1 * nx + kk2) < npix) {
            f = ytgb::dmul(dvx, uy);
            atomicAdd(a.buffer + idx, ytgb::dmul(sq, f));
            atomicAdd(a.buffer_weight + idx, ytgb::dmul(sw, f));
        }
        if (jj2 < nx && kk1 >= 0 && (idx = (long long)jj2 * nx + kk1) < npix) {
            f = ytgb::dmul(ux, dvy);
            atomicAdd(a.buffer + idx, ytgb::dmul(sq, f));
            atomicAdd(a.buffer_weight + idx, ytgb::dmul(sw, f));
        }
        if (jj2 < nx && kk2 < ny && (idx = (long long)jj2 * nx + kk2) < npix) {
            f = ytgb::dmul(ux, uy);
            atomicAdd(a.buffer + idx, ytgb::dmul(sq, f));
            atomicAdd(a.buffer_weight + idx, ytgb::dmul(sw, f));
        }
    }
}

__global__ void __launch_bounds__(OA_BLOCK) offaxis_kernel(const ytgb_offaxis_args a, int32_t *error) {
    __shared__ AxisTable s_x[OA_WARPS], s_y[OA_WARPS];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    AxisTable &tx = s_x[wib], &ty = s_y[wib];
    const int nx = a.nx, ny = a.ny;
    const long long npix = (long long)nx * ny;
    const double sq3 = ytgb::dsqrt(3.0);
    const double sq3x4 = ytgb::dmul(4.0, sq3);
    const double nmax = nx > ny ? (double)nx : (double)ny;  // fmax(Nx, Ny)
    const long long n_warps = (long long)gridDim.x * OA_WARPS;
    for (long long c = (long long)blockIdx.x * OA_WARPS + wib; c < a.n; c += n_warps) {
        const double dx = __ldg(a.dxp + c), w = __ldg(a.weight + c), q = __ldg(a.qty + c);
        const double X0 = __ldg(a.xp + 3 * c), X1 = __ldg(a.xp + 3 * c + 1), X2 = __ldg(a.xp + 3 * c + 2);
        if (!(dx > 0.0) || !isfinite(dx)) {
            if (lane == 0 && error) atomicCAS(error, 0, YTGB_DEVERR_BAD_CELL);
            continue;
        }
        // image_utilities.pyx:264-276 and :66-80
        const double cmw = ytgb::dmul(dx, sq3);
        const double x = ytgb::dadd(ytgb::dadd(ytgb::dadd(ytgb::dmul(a.rot[0], X0), ytgb::dmul(a.rot[1], X1)), ytgb::dmul(a.rot[2], X2)), 0.5);
        const double y = ytgb::dadd(ytgb::dadd(ytgb::dadd(ytgb::dmul(a.rot[3], X0), ytgb::dmul(a.rot[4], X1)), ytgb::dmul(a.rot[5], X2)), 0.5);
        const double half = ytgb::dmul(cmw, 0.5);  // cmw / 2, exactly
        const double dx3 = ytgb::dmul(ytgb::dmul(ytgb::dmul(ytgb::dmul(dx, dx), dx), (double)nx), (double)ny);
        const double lx = ytgb::dsub(x, half), rx = ytgb::dadd(x, half), ly = ytgb::dsub(y, half), ry = ytgb::dadd(y, half);
        const int jmin = max(__double2int_rz(floor(ytgb::dmul(lx, (double)nx))), 0);
        const int jmax = max(__double2int_rz(ceil(ytgb::dmul(rx, (double)nx))), nx - 1);
        const int kmin = min(__double2int_rz(floor(ytgb::dmul(ly, (double)ny))), 0);
        const int kmax = max(__double2int_rz(ceil(ytgb::dmul(ry, (double)ny))), ny - 1);
        if (jmax == jmin + 1 && kmax == kmin + 1) {  // :83-87, the cell inside one pixel
            const long long idx = (long long)jmin * nx + kmin;
            if (lane == 0 && idx >= 0 && idx < npix) {
                atomicAdd(a.buffer + idx, ytgb::dmul(q, dx3));
                atomicAdd(a.buffer_weight + idx, ytgb::dmul(w, dx3));
            }
            continue;
        }
        // :92-99: the stamp level with at least 4 subcells per pixel diagonal
        const double v = ytgb::dmul(ytgb::dmul(sq3x4, dx), nmax);
        int depth = v > 1.0 ? ceil_log2_above1(v) : 1;
        depth = depth < 1 ? 1 : (depth > a.max_depth - 1 ? a.max_depth - 1 : depth);
        const int jm = min(a.nsx, 1 << depth), km = min(a.nsy, 1 << depth);
        // cmw / 2^depth is an exact scaling
        const double pw = dfrom((long long)(1023 - depth) << 52);
        const double dx_loc = jm == (1 << depth) ? ytgb::dmul(cmw, pw) : ytgb::ddiv(cmw, (double)jm);
        const double dy_loc = km == (1 << depth) ? ytgb::dmul(cmw, pw) : ytgb::ddiv(cmw, (double)km);
        const double cq = ytgb::dmul(dx3, q), cw = ytgb::dmul(dx3, w);
        if (jm > OA_KT || km > OA_KT) {
            cell_direct(a, lane, depth, jm, km, dx_loc, dy_loc, x, y, dx3, w, q);
            continue;
        }
        __syncwarp();
        for (int e = lane; e < jm + km; e += 32) {
            if (e < jm) fill_entry(tx, e, jm, dx_loc, x, nx);
            else fill_entry(ty, e - jm, km, dy_loc, y, ny);
        }
        __syncwarp();
        // pixels the cell can reach (the edges are nondecreasing)
        const int Plo = max(tx.edge[0], 0), Phi = min(tx.edge[jm], nx - 1);
        const int Qlo = max(ty.edge[0], 0), Qhi = min(ty.edge[km], ny - 1);
        if (Plo > Phi || Qlo > Qhi) continue;
        // lanes: pixel columns Q (wp of them), times groups sharing out the rows
        const int wy = Qhi - Qlo + 1;
        const int wp = wy < 32 ? wy : 32;
        const int groups = 32 / wp;
        const int g = lane / wp;
        const int j0 = g * jm / groups, j1 = (g + 1) * jm / groups;
        Column col;
        col.stamp = a.stamp + (long long)depth * a.nsx * a.nsy;
        col.nsy = a.nsy;
        col.kcap = km - 1;
        col.nx = nx;
        col.npix = npix;
        col.cq = cq;
        col.cw = cw;
        col.buf = a.buffer;
        col.bufw = a.buffer_weight;
        const int passes = (wy + wp - 1) / wp;
        for (int pass = 0; pass < passes; pass++) {
            const int Q = Qlo + pass * wp + lane - g * wp;
            const bool act = g < groups && Q <= Qhi;
            int klo = 0, nk = 0;
            if (act) {
                klo = first_reaching(ty, km, Q);
                nk = last_starting(ty, km, Q) - klo + 1;
            }
            col.klo = klo;
            col.Q = Q;
            // one unrolled length for the whole warp: lanes of different
            // lengths would otherwise run their loops one after another
            const int N = __reduce_max_sync(0xffffffffu, nk > 0 ? nk : 0);
            if (!act || nk < 1) continue;
            if (N > OA_MAXK) {
                column_rows_wide(tx, ty, col, klo + nk - 1, j0, j1);
                continue;
            }
            // fy_k(Q) of the subcells meeting Q (image_utilities.pyx:141-159),
            // 0 past this lane's own nk
            double w[OA_MAXK];
#pragma unroll
            for (int u = 0; u < OA_MAXK; u++) {
                const int k = klo + u;
                double wv = 0.0;
                if (u < nk) {
                    if (ty.edge[k] == Q) wv = ty.dv[k];
                    if (ty.edge[k + 1] == Q) wv = ytgb::dadd(wv, ty.uv[k]);
                }
                w[u] = wv;
            }
            switch (N) {
            case 1: column_rows<1>(tx, col, w, j0, j1); break;
            case 2: column_rows<2>(tx, col, w, j0, j1); break;
            case 3: column_rows<3>(tx, col, w, j0, j1); break;
            case 4: column_rows<4>(tx, col, w, j0, j1); break;
            case 5: column_rows<5>(tx, col, w, j0, j1); break;
            case 6: column_rows<6>(tx, col, w, j0, j1); break;
            case 7: column_rows<7>(tx, col, w, j0, j1); break;
            case 8: column_rows<8>(tx, col, w, j0, j1); break;
            case 9: column_rows<9>(tx, col, w, j0, j1); break;
            default: column_rows<10>(tx, col, w, j0, j1); break;
            }
        }
    }
}


// ---- splatting by summed stamps --------------------------------------------
//
// A subcell's mass goes to its left pixel with dv and to its right pixel with
// 1 - dv, so the mass of a cell in the pixels (<= P, <= Q) is the stamp's sum
// over the subcells whose right pixels are within, plus the dv of the one
// column and the one row that P and Q cut: a bilinear look-up in the stamp's
// summed-area table.  A pixel's mass is the difference of four such corners.
// The subcell kernel above spends some 30 to 90 float64 operations on a pixel,
// at 2 per SM and cycle its bound (float64 pipe 90 % busy); a corner takes
// three products of integers, on the integer pipe.
//
// The table is in fixed point of 128 bits, modulo 2^128, in units of
// 2^-(126 + s) of the stamp's unit sum (level_shift): only differences are
// used, and those that occur (one subcell column's or row's sum, a pixel's
// mass) fit, so that they are exact.  An entry keeps its 53 bits down to 2^-73
// of the sum, a cut subcell's dv its own 53 bits at any size, and a product is
// rounded down by less than a unit: a pixel of n subcells is within n / 2 + 12
// units.  So a pixel that a cell only grazes is as exact as a whole one down to
// 1e-20 of the stamp's sum (64 bits lost 1e-12 of pixels of 1e-5 of the largest).
//
// The subcell boundaries, their pixels and dv are formed by the reference's
// float64 operations, once per pixel boundary and axis.  A warp takes a few cells,
// strided over the list so that each batch has cells of all sizes (one where there
// are no more cells than warps): first one lane per cell for what depends on the
// cell alone, then one lane per pixel boundary of as many cells as the table in
// shared memory holds, then the pixels cell by cell, lanes over the columns and
// groups of lanes over the rows.
// 217,000 cells of levels 5-9 at 1024^2 (38 pixels to 2): 5.17 ms by the subcell
// kernel, 1.02 here (0.69 with 64 bits, see above).  Issue is 62 % busy, the integer
// pipe 60 % (the corners' products), the float64 pipe 39 % (boundaries and their
// divisions).  7 blocks per SM and 8 cells a batch lie within 2 % of the best of 5
// to 7 and 4 to 16.
constexpr int OS_CAP = 520;   // pixel boundaries held per warp: a cell of 258 pixels each way
constexpr int OS_CELLS = 8;   // cells of a warp's batch
constexpr int OS_WARPS = 4;
constexpr int OS_BLOCKS = 7;  // resident blocks per SM: 72 registers

typedef unsigned __int128 u128;

// s of a level of jm x km subcells.  A row or column of subcells holds at
// most sqrt(6) / min(jm, km) of the sum (the largest plane section of a cube
// is sqrt(2) of a face, across a cube 1 / sqrt(3) of the stamp's width) and a
// subcell 3 sqrt(3) / (jm km) (the cube's diagonal); the level is chosen with
// fewer than 8 subcells per pixel along the longer image axis
// (image_utilities.pyx:92-99).  So the former stay below 2^128 units and a
// pixel, which may hold the whole sum, at most 2^126 (with a margin of 1.3 for
// the stamp's own discretisation).
__device__ __forceinline__ int level_shift(int jm, int km, int nx, int ny) {
    const int lg = 31 - __clz(min(jm, km));
    const float n = (float)max(nx, ny), px = 8.0f * n / (float)nx, py = 8.0f * n / (float)ny;
    const float mass = 1.3f * 5.2f * px * py / ((float)jm * (float)km);
    int s = 0;
    while (s < lg && mass * (float)(1ll << (s + 1)) <= 1.0f) s++;
    return s;
}

// The table of level d holds (jm + 1) x (km + 1) sums, rows of km + 1, behind
// those of the levels before it.
__host__ __device__ __forceinline__ int level_extent(int ns, int depth) { return depth < 31 && (1 << depth) < ns ? 1 << depth : ns; }
__host__ __device__ __forceinline__ long long level_offset(int nsx, int nsy, int depth) {
    long long o = 0;
    for (int d = 0; d < depth; d++) o += (long long)(level_extent(nsx, d) + 1) * (level_extent(nsy, d) + 1);
    return o;
}

struct SplatCell {
    double x, y, dlx, dly, cq, cw;
    float bx, by, sx, sy;  // estimate of the subcell at a pixel boundary: ceil(s * P + b) - 1
    int depth, jm, km, unit;  // unit: 2^-unit is the table's
    long long base;           // the level's first sum
    int P0, Pn, Q0, Qn;    // first pixel and number of pixels, per axis (0: nothing to do)
};

struct SplatSmem {
    SplatCell cell[OS_CELLS];
    unsigned long long w[OS_CAP];  // dv of the cut subcell (split_share)
    int at[OS_CAP];                // its index
    int off[OS_CELLS], who[OS_CELLS];          // the packed cells' first entries, and which cells they are
};

// A dv in (0, 1) as its mantissa (1 at bit 63) and, in the low bits that its 53
// leave free, the power of two it stands below 1; 0 for what is not above 0
// (and below 2^-64, which no dv is: it is a difference of numbers of pixels).
__device__ __forceinline__ unsigned long long split_share(double x) {
    const long long b = dbits(x);
    const int sh = 1022 - (int)(b >> 52);
    if (b <= 0 || sh > 63) return 0ull;
    return ((unsigned long long)((b & MANT52) | (1LL << 52)) << 11) | (unsigned)sh;
}

// floor(a w) of a split_share w
__device__ __forceinline__ u128 scale_share(u128 a, unsigned long long w) {
    const unsigned long long m = w & ~2047ull, hi = (unsigned long long)(a >> 64);
    const u128 p = (u128)hi * m + __umul64hi((unsigned long long)a, m);
    return p >> (int)(w & 63);
}

__device__ __forceinline__ u128 load_sum(const ulonglong2 *__restrict__ S, long long i) {
    const ulonglong2 v = __ldg(S + i);
    return ((u128)v.y << 64) | v.x;
}

// (double)v for 0 <= v < 2^31 and the truncation of |x| < 2^31 (others by the
// conversion), on the integer pipe: the conversions take the float64 pipe
__device__ __forceinline__ double to_double(int v) {
    const int lead = 31 - __clz(v);
    const unsigned m = (unsigned)v << (31 - lead);  // 1 at bit 31
    return v == 0 ? 0.0 : __hiloint2double((int)(((unsigned)(lead + 1023) << 20) | ((m >> 11) & 0xfffffu)), (int)(m << 21));
}
__device__ __forceinline__ int truncate(double x) {
    const int e = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
    if (e < 0) return 0;
    if (e > 30) return __double2int_rz(x);
    const unsigned long long m = ((unsigned long long)dbits(x) & MANT52) | (1ull << 52);
    const int v = (int)(m >> (52 - e));
    return __double2hiint(x) < 0 ? -v : v;
}

// Subcell boundary i as `boundary` forms it: i - m / 2 is exact, so its
// product with d is that of 2 i - m with d / 2 (dh, exact)
__device__ __forceinline__ double boundary_half(int i, int m, double dh, double x, double N) {
    const int k = 2 * i - m;
    const double a = to_double(k < 0 ? -k : k);
    return ytgb::dmul(ytgb::dadd(ytgb::dmul(k < 0 ? -a : a, dh), x), N);
}

// The subcell that pixel boundary P (the right edge of pixel P; -1: of what
// lies left of pixel 0) cuts: the first whose right boundary truncates past
// P, with its dv where its left boundary does not (image_utilities.pyx:
// 110-120 and 124-138); m and 0 past the last.
__device__ __forceinline__ void cut_subcell(int P, int m, double d, double x, int n, float s, float b, int &at,
                                            unsigned long long &w) {
    const double dh = ytgb::dmul(d, 0.5), N = to_double(n);
    const float est = ceilf(ffma(s, (float)(P < 0 ? -1 : P + 1), b));
    int j = (int)fminf(fmaxf(est - 1.0f, 0.0f), (float)(m - 1));
    double b0 = boundary_half(j, m, dh, x, N), b1 = boundary_half(j + 1, m, dh, x, N);
    int e0 = truncate(b0), e1 = truncate(b1);
    // (the estimate is within a subcell or two: float32 of P * subcells per pixel)
    while (j > 0 && e0 > P) {
        j--;
        b1 = b0;
        e1 = e0;
        b0 = boundary_half(j, m, dh, x, N);
        e0 = truncate(b0);
    }
    while (j < m && !(e1 > P)) {
        j++;
        b0 = b1;
        e0 = e1;
        b1 = boundary_half(j + 1, m, dh, x, N);
        e1 = truncate(b1);
    }
    at = j;
    w = 0ull;
    if (j < m && e0 <= P) {
        const double dv = ytgb::ddiv(ytgb::dsub(to_double(e1), b0), ytgb::dsub(b1, b0));
        if (dv >= 1.0) at = j + 1;  // the whole subcell is left of the boundary
        else w = split_share(dv);
    }
}

// A float64 factor as a 64-bit mantissa (1 at bit 63), exponent and sign, for
// scaled_mass; ok false (subnormal, zero, infinite, NaN) where the product is
// left to float64.
struct Factor {
    unsigned long long m;
    long long eb;  // sign and biased exponent field, shifted into place
    bool ok;
};
__device__ __forceinline__ Factor factor_of(double x) {
    const long long b = dbits(x);
    const int e = (int)(b >> 52) & 0x7ff;
    Factor f;
    f.m = ((unsigned long long)(b & MANT52) | (1ull << 52)) << 11;
    f.eb = b & ~MANT52;
    f.ok = e > 200 && e < 1800;  // (the product's exponent stays inside the field)
    return f;
}

// x times mass 2^-unit, where m is mass shifted to have 1 at bit 63 and `down`
// = unit - 63 + the shift: the 128-bit product's upper half, rounded to 53 bits
// (ties away from zero; the part dropped before is below 2^-63 of the value),
// on the integer pipe where a float64 product takes the float64 pipe 64 cycles.
__device__ __forceinline__ double scaled_mass(unsigned long long m, int down, const Factor &f) {
    unsigned long long p = __umul64hi(m, f.m);  // in [2^62, 2^64)
    const int up = (int)(p >> 63);
    p = up ? p : p << 1;
    const unsigned long long r = ((p & 0x7fffffffffffffffull) + 0x400ull) >> 11;  // a carry adds to the exponent
    return dfrom(f.eb + (long long)r + ((long long)(up - down) << 52));
}

// the table's value at a corner: rows at, at + 1 and columns b0, b1 (two
// neighbours, or twice the last)
__device__ __forceinline__ u128 corner(const ulonglong2 *__restrict__ S, int stride, int m, int at,
                                       unsigned long long wa, int b0, int b1, unsigned long long wb) {
    const ulonglong2 *r0 = S + (long long)at * stride, *r1 = S + (long long)min(at + 1, m) * stride;
    const u128 u0 = load_sum(r0, b0), u1 = load_sum(r0, b1), v0 = load_sum(r1, b0), v1 = load_sum(r1, b1);
    const u128 u = u0 + scale_share(u1 - u0, wb), v = v0 + scale_share(v1 - v0, wb);
    return u + scale_share(v - u, wa);
}

__device__ __forceinline__ u128 shuffle_up(u128 v, int d) {
    const unsigned long long lo = __shfl_up_sync(0xffffffffu, (unsigned long long)v, d);
    const unsigned long long hi = __shfl_up_sync(0xffffffffu, (unsigned long long)(v >> 64), d);
    return ((u128)hi << 64) | lo;
}

__global__ void __launch_bounds__(OS_WARPS * 32, OS_BLOCKS)
splat_kernel(const ytgb_offaxis_args a, const ulonglong2 *__restrict__ sums, long long batches, int32_t *error) {
    __shared__ SplatSmem s_all[OS_WARPS];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    SplatSmem &sm = s_all[wib];
    const int nx = a.nx, ny = a.ny;
    const long long npix = (long long)nx * ny;
    const double sq3 = ytgb::dsqrt(3.0);
    const double sq3x4 = ytgb::dmul(4.0, sq3);
    const double nmax = nx > ny ? (double)nx : (double)ny;  // fmax(Nx, Ny)
    for (long long bt = (long long)blockIdx.x * OS_WARPS + wib; bt < batches; bt += (long long)gridDim.x * OS_WARPS) {
        // ---- one lane per cell
        const long long c = bt + (long long)lane * batches;
        int Pn = 0, Qn = 0;
        bool wide = false;
        if (lane < OS_CELLS && c < a.n) {
            const double dx = __ldg(a.dxp + c), w = __ldg(a.weight + c), q = __ldg(a.qty + c);
            const double X0 = __ldg(a.xp + 3 * c), X1 = __ldg(a.xp + 3 * c + 1), X2 = __ldg(a.xp + 3 * c + 2);
            if (!(dx > 0.0) || !isfinite(dx)) {
                if (error) atomicCAS(error, 0, YTGB_DEVERR_BAD_CELL);
            } else {
                SplatCell &sc = sm.cell[lane];
                const double cmw = ytgb::dmul(dx, sq3);
                const double x = ytgb::dadd(ytgb::dadd(ytgb::dadd(ytgb::dmul(a.rot[0], X0), ytgb::dmul(a.rot[1], X1)), ytgb::dmul(a.rot[2], X2)), 0.5);
                const double y = ytgb::dadd(ytgb::dadd(ytgb::dadd(ytgb::dmul(a.rot[3], X0), ytgb::dmul(a.rot[4], X1)), ytgb::dmul(a.rot[5], X2)), 0.5);
                const double half = ytgb::dmul(cmw, 0.5);  // cmw / 2, exactly
                const double dx3 = ytgb::dmul(ytgb::dmul(ytgb::dmul(ytgb::dmul(dx, dx), dx), (double)nx), (double)ny);
                const double lx = ytgb::dsub(x, half), rx = ytgb::dadd(x, half), ly = ytgb::dsub(y, half), ry = ytgb::dadd(y, half);
                const int jmin = max(__double2int_rz(floor(ytgb::dmul(lx, (double)nx))), 0);
                const int jmax = max(__double2int_rz(ceil(ytgb::dmul(rx, (double)nx))), nx - 1);
                const int kmin = min(__double2int_rz(floor(ytgb::dmul(ly, (double)ny))), 0);
                const int kmax = max(__double2int_rz(ceil(ytgb::dmul(ry, (double)ny))), ny - 1);
                if (jmax == jmin + 1 && kmax == kmin + 1) {  // image_utilities.pyx:83-87, the cell inside one pixel
                    const long long idx = (long long)jmin * nx + kmin;
                    if (idx >= 0 && idx < npix) {
                        atomicAdd(a.buffer + idx, ytgb::dmul(q, dx3));
                        atomicAdd(a.buffer_weight + idx, ytgb::dmul(w, dx3));
                    }
                } else {
                    // :92-99: the stamp level with at least 4 subcells per pixel diagonal
                    const double v = ytgb::dmul(ytgb::dmul(sq3x4, dx), nmax);
                    int depth = v > 1.0 ? ceil_log2_above1(v) : 1;
                    depth = depth < 1 ? 1 : (depth > a.max_depth - 1 ? a.max_depth - 1 : depth);
                    const int jm = min(a.nsx, 1 << depth), km = min(a.nsy, 1 << depth);
                    // cmw / 2^depth is an exact scaling
                    const double pw = dfrom((long long)(1023 - depth) << 52);
                    sc.dlx = jm == (1 << depth) ? ytgb::dmul(cmw, pw) : ytgb::ddiv(cmw, (double)jm);
                    sc.dly = km == (1 << depth) ? ytgb::dmul(cmw, pw) : ytgb::ddiv(cmw, (double)km);
                    sc.x = x;
                    sc.y = y;
                    sc.cq = ytgb::dmul(dx3, q);
                    sc.cw = ytgb::dmul(dx3, w);
                    sc.depth = depth;
                    sc.jm = jm;
                    sc.km = km;
                    sc.unit = 126 + level_shift(jm, km, nx, ny);
                    sc.base = level_offset(a.nsx, a.nsy, depth);
                    // pixels the cell can reach (the boundaries are nondecreasing)
                    const int P0 = max(__double2int_rz(boundary(0, jm, sc.dlx, x, nx)), 0);
                    const int P1 = min(__double2int_rz(boundary(jm, jm, sc.dlx, x, nx)), nx - 1);
                    const int Q0 = max(__double2int_rz(boundary(0, km, sc.dly, y, ny)), 0);
                    const int Q1 = min(__double2int_rz(boundary(km, km, sc.dly, y, ny)), ny - 1);
                    sc.P0 = P0;
                    sc.Q0 = Q0;
                    const float fdx = (float)sc.dlx, fdy = (float)sc.dly;
                    sc.sx = 1.0f / ((float)nx * fdx);
                    sc.sy = 1.0f / ((float)ny * fdy);
                    sc.bx = 0.5f * (float)jm - (float)x / fdx;
                    sc.by = 0.5f * (float)km - (float)y / fdy;
                    if (P0 <= P1 && Q0 <= Q1 && isfinite(x) && isfinite(y)) {
                        Pn = P1 - P0 + 1;
                        Qn = Q1 - Q0 + 1;
                        wide = (long long)Pn + Qn + 2 > OS_CAP;
                    }
                    sc.Pn = Pn;
                    sc.Qn = Qn;
                }
            }
        }
        __syncwarp();
        // ---- cells wider than the table holds: the reference's own loop
        for (unsigned m = __ballot_sync(0xffffffffu, wide); m; m &= m - 1) {
            const SplatCell &sc = sm.cell[__ffs(m) - 1];
            const long long cc = bt + (long long)(__ffs(m) - 1) * batches;
            const double dx = __ldg(a.dxp + cc);
            cell_direct(a, lane, sc.depth, sc.jm, sc.km, sc.dlx, sc.dly, sc.x, sc.y,
                        ytgb::dmul(ytgb::dmul(ytgb::dmul(ytgb::dmul(dx, dx), dx), (double)nx), (double)ny),
                        __ldg(a.weight + cc), __ldg(a.qty + cc));
        }
        const int need = Pn > 0 && !wide ? Pn + Qn + 2 : 0;  // this lane's cell's pixel boundaries
        unsigned left = __ballot_sync(0xffffffffu, need > 0);
        while (left) {
            // ---- the first cells whose boundaries fit the table
            int incl = (left >> lane) & 1u ? need : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += v;
            }
            const bool in = ((left >> lane) & 1u) && incl <= OS_CAP;
            const unsigned take = __ballot_sync(0xffffffffu, in);
            const int total = __reduce_max_sync(0xffffffffu, in ? incl : 0);
            const int rank = __popc(take & ((1u << lane) - 1u)), n_take = __popc(take);
            if (in) {
                sm.off[rank] = incl - need;
                sm.who[rank] = lane;
            }
            __syncwarp();
            // ---- one lane per pixel boundary
            for (int t = lane; t < total; t += 32) {
                int lo = 0, hi = n_take - 1;
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (sm.off[mid] <= t) lo = mid;
                    else hi = mid - 1;
                }
                const SplatCell &sc = sm.cell[sm.who[lo]];
                const int k = t - sm.off[lo];
                const bool col = k > sc.Pn;  // rows' boundaries first, then the columns'
                const int P = col ? sc.Q0 - 1 + (k - sc.Pn - 1) : sc.P0 - 1 + k;
                int at;
                unsigned long long w;
                cut_subcell(P, col ? sc.km : sc.jm, col ? sc.dly : sc.dlx, col ? sc.y : sc.x, col ? ny : nx,
                            col ? sc.sy : sc.sx, col ? sc.by : sc.bx, at, w);
                sm.at[t] = at;
                sm.w[t] = w;
            }
            __syncwarp();
            // ---- the pixels, cell by cell
            for (int i = 0; i < n_take; i++) {
                const SplatCell &sc = sm.cell[sm.who[i]];
                const int o = sm.off[i], rows = sc.Pn, jm = sc.jm, km = sc.km, stride = km + 1;
                const ulonglong2 *S = sums + sc.base;
                const Factor fq = factor_of(sc.cq), fw = factor_of(sc.cw);
                const bool plain = fq.ok && fw.ok;
                const int *ra = sm.at + o, *ca = ra + rows + 1;
                const unsigned long long *rw = sm.w + o, *cw = rw + rows + 1;
                for (int q0 = 0; q0 < sc.Qn; q0 += 31) {
                    // lanes over the column boundaries q0 .. q0 + nb - 1, groups of
                    // them over the rows
                    const int nb = min(32, sc.Qn + 1 - q0);
                    const int groups = 32 / nb, g = lane / nb, q = q0 + lane - g * nb;
                    const bool on = g < groups;
                    const int b = on ? ca[q] : 0;
                    const int b1 = min(b + 1, km);
                    const unsigned long long wb = on ? cw[q] : 0ull;
                    const int r0 = on ? g * rows / groups : 0, r1 = on ? (g + 1) * rows / groups : 0;
                    const int steps = (rows + groups - 1) / groups;
                    const int Q = sc.Q0 + q - 1;  // the pixel left of this boundary
                    const bool px = on && lane > g * nb;
                    u128 prev = on ? corner(S, stride, jm, ra[r0], rw[r0], b, b1, wb) : (u128)0;
                    for (int k = 0; k < steps; k++) {
                        const int r = min(r0 + k + 1, r1);
                        const u128 G = on ? corner(S, stride, jm, ra[r], rw[r], b, b1, wb) : (u128)0;
                        const u128 d = G - prev;
                        prev = G;
                        const __int128 mass = (__int128)(d - shuffle_up(d, 1));  // (rounding may leave a few units below 0)
                        if (px && r0 + k < r1 && mass > 0) {
                            const long long idx = (long long)(sc.P0 + r0 + k) * nx + Q;
                            if (idx < npix) {
                                // the mass' upper 64 bits from its first 1
                                const unsigned long long mh = (unsigned long long)(mass >> 64);
                                const int sh = mh ? __clzll((long long)mh) : 64 + __clzll((long long)mass);
                                const unsigned long long m = (unsigned long long)(((u128)mass << sh) >> 64);
                                const int down = sc.unit - 127 + sh;
                                double vq, vw;
                                if (plain) {
                                    vq = scaled_mass(m, down, fq);
                                    vw = scaled_mass(m, down, fw);
                                } else {
                                    const double f = dfrom(dbits((double)m) - ((long long)(down + 63) << 52));
                                    vq = ytgb::dmul(f, sc.cq);
                                    vw = ytgb::dmul(f, sc.cw);
                                }
                                atomicAdd(a.buffer + idx, vq);
                                atomicAdd(a.buffer_weight + idx, vw);
                            }
                        }
                    }
                }
            }
            // a quantity or weight that is not finite reaches every pixel of its cell's
            // rectangle, also those of no mass, as in the subcell kernel
            for (int i = 0; i < n_take; i++) {
                const SplatCell &sc = sm.cell[sm.who[i]];
                if (isfinite(sc.cq) && isfinite(sc.cw)) continue;
                for (long long t = lane; t < (long long)sc.Pn * sc.Qn; t += 32) {
                    const long long idx = (sc.P0 + t / sc.Qn) * nx + sc.Q0 + t % sc.Qn;
                    if (idx < npix) {
                        atomicAdd(a.buffer + idx, ytgb::dmul(0.0, sc.cq));
                        atomicAdd(a.buffer_weight + idx, ytgb::dmul(0.0, sc.cw));
                    }
                }
            }
            __syncwarp();  // the tables are rewritten
            left &= ~take;
        }
        __syncwarp();  // the cells are rewritten
    }
}

// ---- the summed-area tables: rows, then columns ------------------------------
// One warp per row of a level, lanes along it; then one block per level and 32
// columns, each warp adding up a run of rows: every access is a warp's 512
// contiguous bytes.  A view's tables for cells of 0.15 and 0.3 of a 1024^2 image:
// 644 and 2139 us with one block per level and a thread per row, now 56 and 78
// (36 of them the launches, the allocation and the wait).
constexpr int SR_WARPS = 4, SC_WARPS = 16;

// a stamp entry in units of 2^-unit (to nearest; 0 where it is not above 0)
__device__ __forceinline__ u128 stamp_units(double x, int unit) {
    const long long b = dbits(x);
    const int e = (int)(b >> 52);
    if (b <= 0 || e >= 0x7ff) return 0;
    const u128 m = (u128)(unsigned long long)((b & MANT52) | (e > 0 ? 1LL << 52 : 0LL));
    const int sh = (e > 0 ? e : 1) - 1075 + unit;
    if (sh >= 0) return sh < 128 ? m << sh : (u128)0;
    return sh > -64 ? (m + ((u128)1 << (-sh - 1))) >> -sh : (u128)0;
}

__device__ __forceinline__ void store_sum(ulonglong2 *S, long long i, u128 v) {
    S[i] = make_ulonglong2((unsigned long long)v, (unsigned long long)(v >> 64));
}

__global__ void __launch_bounds__(SR_WARPS * 32)
sum_rows_kernel(const double *stamp, int nsx, int nsy, int nx, int ny, ulonglong2 *sums) {
    const int depth = blockIdx.y, lane = threadIdx.x & 31;
    const int jm = level_extent(nsx, depth), km = level_extent(nsy, depth);
    const int j = blockIdx.x * SR_WARPS + (threadIdx.x >> 5);  // the sums' row: 0 is empty
    if (j > jm) return;
    ulonglong2 *row = sums + level_offset(nsx, nsy, depth) + (long long)j * (km + 1);
    const double *st = stamp + ((long long)depth * nsx + (j - 1)) * nsy;
    const int unit = 126 + level_shift(jm, km, nx, ny);
    u128 before = 0;
    if (lane == 0) store_sum(row, 0, 0);
    for (int k0 = 0; k0 < km; k0 += 32) {
        const int k = k0 + lane;
        u128 v = j > 0 && k < km ? stamp_units(__ldg(st + k), unit) : (u128)0;
        for (int d = 1; d < 32; d <<= 1) {
            const u128 u = shuffle_up(v, d);
            if (lane >= d) v += u;
        }
        v += before;
        if (k < km) store_sum(row, k + 1, v);
        const unsigned long long lo = __shfl_sync(0xffffffffu, (unsigned long long)v, 31);
        const unsigned long long hi = __shfl_sync(0xffffffffu, (unsigned long long)(v >> 64), 31);
        before = ((u128)hi << 64) | lo;
    }
}

__global__ void __launch_bounds__(SC_WARPS * 32) sum_columns_kernel(int nsx, int nsy, ulonglong2 *sums) {
    __shared__ ulonglong2 part[SC_WARPS][32];
    const int depth = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int jm = level_extent(nsx, depth), stride = level_extent(nsy, depth) + 1;
    const int k = blockIdx.x * 32 + lane;
    if ((int)blockIdx.x * 32 >= stride) return;  // (the whole block)
    ulonglong2 *col = sums + level_offset(nsx, nsy, depth) + k;
    const int per = (jm + SC_WARPS) / SC_WARPS;  // of jm + 1 rows
    const int j0 = min(warp * per, jm + 1), j1 = min(j0 + per, jm + 1);
    u128 acc = 0;
    if (k < stride)
#pragma unroll 4
        for (int j = j0; j < j1; j++) {
            const ulonglong2 v = col[(long long)j * stride];
            acc += ((u128)v.y << 64) | v.x;
        }
    part[warp][lane] = make_ulonglong2((unsigned long long)acc, (unsigned long long)(acc >> 64));
    __syncthreads();
    acc = 0;
    for (int w = 0; w < warp; w++) acc += ((u128)part[w][lane].y << 64) | part[w][lane].x;
    if (k < stride)
#pragma unroll 4
        for (int j = j0; j < j1; j++) {
            const ulonglong2 v = col[(long long)j * stride];
            acc += ((u128)v.y << 64) | v.x;
            store_sum(col, (long long)j * stride, acc);
        }
}

}  // namespace

static int offaxis_checks(const ytgb_offaxis_args *args, const int32_t *d_error) {
    if (!args) {
        ytgb_set_error("ytgb_offaxis_cells: null args");
        return YTGB_ERR_INVALID;
    }
    const ytgb_offaxis_args &a = *args;
    if (a.n < 0 || a.nx < 1 || a.ny < 1 || a.nx > a.ny || a.nsx < 1 || a.nsy < 1 || a.max_depth < 2 ||
        a.max_depth > 30) {
        ytgb_set_error("ytgb_offaxis_cells: bad sizes (nx must not exceed ny; 2 <= max_depth <= 30)");
        return YTGB_ERR_INVALID;
    }
    if (a.n > 0 && (!a.xp || !a.dxp || !a.qty || !a.weight || !a.stamp || !a.buffer || !a.buffer_weight ||
        ((uintptr_t)a.xp & 7) || ((uintptr_t)a.dxp & 7) || ((uintptr_t)a.qty & 7) || ((uintptr_t)a.weight & 7) ||
        ((uintptr_t)a.stamp & 7) || ((uintptr_t)a.buffer & 7) || ((uintptr_t)a.buffer_weight & 7) ||
        ((uintptr_t)d_error & 3))) {
        ytgb_set_error("ytgb_offaxis_cells: null or misaligned device array");
        return YTGB_ERR_INVALID;
    }
    return YTGB_OK;
}

// Blocks for `want` warps' work, at most `per_sm` resident blocks on every SM.
static int offaxis_blocks(long long want, int per_sm) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long cap = (long long)(sms > 0 ? sms : 152) * per_sm;
    return (int)(want < cap ? want : cap);
}

extern "C" int ytgb_offaxis_cells(const ytgb_offaxis_args *args, int32_t *d_error, void *stream) {
    if (int st = offaxis_checks(args, d_error)) return st;
    const ytgb_offaxis_args &a = *args;
    if (a.n == 0) return YTGB_OK;
    const int blocks = offaxis_blocks((a.n + OA_WARPS - 1) / OA_WARPS, 8);
    offaxis_kernel<<<blocks, OA_BLOCK, 0, (cudaStream_t)stream>>>(a, d_error);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        ytgb_set_error(std::string("ytgb_offaxis_cells: ") + cudaGetErrorString(e));
        return YTGB_ERR_CUDA;
    }
    return YTGB_OK;
}

extern "C" int ytgb_offaxis_sums_bytes(int32_t nsx, int32_t nsy, int32_t max_depth, int64_t *bytes) {
    if (!bytes || nsx < 1 || nsy < 1 || max_depth < 2 || max_depth > 30) {
        ytgb_set_error("ytgb_offaxis_sums_bytes: null argument or bad sizes");
        return YTGB_ERR_INVALID;
    }
    *bytes = (int64_t)sizeof(ulonglong2) * level_offset(nsx, nsy, max_depth);
    return YTGB_OK;
}

extern "C" int ytgb_offaxis_sums(const double *d_stamp, int32_t nsx, int32_t nsy, int32_t max_depth, int32_t nx,
                                 int32_t ny, void *d_sums, void *stream) {
    if (!d_stamp || !d_sums || ((uintptr_t)d_stamp & 7) || ((uintptr_t)d_sums & 15) || nsx < 1 || nsy < 1 ||
        max_depth < 2 || max_depth > 30 || nx < 1 || ny < 1) {
        ytgb_set_error("ytgb_offaxis_sums: null or misaligned array, or bad sizes");
        return YTGB_ERR_INVALID;
    }
    const int jm = level_extent(nsx, max_depth - 1), km = level_extent(nsy, max_depth - 1);  // the largest level
    sum_rows_kernel<<<dim3(jm / SR_WARPS + 1, max_depth), SR_WARPS * 32, 0, (cudaStream_t)stream>>>(
        d_stamp, nsx, nsy, nx, ny, reinterpret_cast<ulonglong2 *>(d_sums));
    sum_columns_kernel<<<dim3(km / 32 + 1, max_depth), SC_WARPS * 32, 0, (cudaStream_t)stream>>>(
        nsx, nsy, reinterpret_cast<ulonglong2 *>(d_sums));
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        ytgb_set_error(std::string("ytgb_offaxis_sums: ") + cudaGetErrorString(e));
        return YTGB_ERR_CUDA;
    }
    return YTGB_OK;
}

extern "C" int ytgb_offaxis_cells_sums(const ytgb_offaxis_args *args, const void *d_sums, int32_t *d_error,
                                       void *stream) {
    if (int st = offaxis_checks(args, d_error)) return st;
    const ytgb_offaxis_args &a = *args;
    if (!d_sums || ((uintptr_t)d_sums & 15)) {
        ytgb_set_error("ytgb_offaxis_cells_sums: null or misaligned table of sums");
        return YTGB_ERR_INVALID;
    }
    if (a.n == 0) return YTGB_OK;
    // a warp takes a second cell only where there are more cells than resident warps:
    // in batches of OS_CELLS fewer cells left most of the chip idle (1,000 cells of
    // 111 pixels 1.92 ms, now 0.29)
    const long long resident = (long long)offaxis_blocks(1ll << 40, OS_BLOCKS) * OS_WARPS;
    const long long batches = std::max<long long>((a.n + OS_CELLS - 1) / OS_CELLS, std::min<long long>(a.n, resident));
    const int blocks = (int)std::min<long long>((batches + OS_WARPS - 1) / OS_WARPS, 1 << 20);
    splat_kernel<<<blocks, OS_WARPS * 32, 0, (cudaStream_t)stream>>>(
        a, reinterpret_cast<const ulonglong2 *>(d_sums), batches, d_error);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        ytgb_set_error(std::string("ytgb_offaxis_cells_sums: ") + cudaGetErrorString(e));
        return YTGB_ERR_CUDA;
    }
    return YTGB_OK;
}
