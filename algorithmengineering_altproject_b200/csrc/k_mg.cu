// Geometric-multigrid kernels: BC masks per level, Jacobi diagonals, restriction, prolongation
// fused with the additive smoother, the coarsest dense Galerkin matrix, its Cholesky factor and
// the coarsest triangular solves.  Every kernel mirrors the reference's arithmetic order
// (transfers.cpp, diagonal.cpp, coarsest.cpp, preconditioner.cpp) operation for operation.
#include "kernels.hpp"
#include "red.cuh"

#include <algorithm>

namespace t3d {

namespace {

struct LevelIdx {
    int nnx, nny, nnz;
    __device__ LevelIdx(const MgLevel& L) : nnx(L.nx + 1), nny(L.ny + 1), nnz(L.nz + 1) {}
    __device__ int node(int x, int y, int z) const { return (z * nny + y) * nnx + x; }
};

__device__ __forceinline__ double hat(int i, int s) {   // 1 - |i-(s-1)|/s  (transfers.cpp:123-126)
    return 1.0 - fabs((double)(i - (s - 1))) * (1.0 / s);
}

// trilinear weight of coarse corner a at sub-node (ix,iy,iz) of a span-s element (hierarchy.cpp:13-42)
__device__ __forceinline__ double corner_weight(int s, int ix, int iy, int iz, int a) {
    const double xi = -1.0 + 2.0 * ((double)ix / (double)s);
    const double eta = -1.0 + 2.0 * ((double)iy / (double)s);
    const double zeta = -1.0 + 2.0 * ((double)iz / (double)s);
    const double sx = (a == 1 || a == 2 || a == 5 || a == 6) ? 1.0 : -1.0;
    const double sy = (a == 2 || a == 3 || a == 6 || a == 7) ? 1.0 : -1.0;
    const double sz = a >= 4 ? 1.0 : -1.0;
    return 0.125 * (1.0 + sx * xi) * (1.0 + sy * eta) * (1.0 + sz * zeta);
}

// ------------------------------------------------------------------ masks (masks.cpp:11-37)
// coarse bit c = normalised restriction (valSum/wSum form) of the fine 0/1 field > 0.5
__global__ void k_mask_restrict(MgLevel Lc, MgLevel Lf) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= Lc.nn) return;
    const LevelIdx C(Lc), F(Lf);
    const int cx = n % C.nnx, cy = (n / C.nnx) % C.nny, cz = n / (C.nnx * C.nny);
    const int s = Lc.span, ws = 2 * s - 1;
    double v[3] = {0, 0, 0}, wsum = 0.0;
    for (int iz = 0; iz < ws; ++iz) {
        const int fz = cz * s + iz - (s - 1);
        if (fz < 0 || fz >= F.nnz) continue;
        for (int iy = 0; iy < ws; ++iy) {
            const int fy = cy * s + iy - (s - 1);
            if (fy < 0 || fy >= F.nny) continue;
            const double wzy = hat(iz, s) * hat(iy, s);
            for (int ix = 0; ix < ws; ++ix) {
                const int fx = cx * s + ix - (s - 1);
                if (fx < 0 || fx >= F.nnx) continue;
                const double w = wzy * hat(ix, s);
                const int m = Lf.mask[F.node(fx, fy, fz)];
                for (int c = 0; c < 3; ++c) v[c] = v[c] + ((m >> c) & 1 ? 1.0 : 0.0) * w;
                wsum = wsum + w;
            }
        }
    }
    int out = 0;
    for (int c = 0; c < 3; ++c) {
        const double r = wsum > 1e-12 ? v[c] / wsum : 0.0;
        if (r > 0.5) out |= 1 << c;
    }
    Lc.mask[n] = (uint8_t)out;
}

// ------------------------------------------------------------------ coarse diagonal (diagonal.cpp:66-138)
// Gather per coarse DOF: incident coarse elements in colour order, their (s+1)^3 sub-nodes in
// (iz,iy,ix) order, weight W_a^2, skipping fixed coarse or fine DOFs.
// COMPS components of a node per thread (3 / COMPS blocks in y).  The order is a chain of 8 (s+1)^3 additions; a row of
// sub-nodes is loaded ahead of it, and a skipped sub-node (fixed, or in no element) adds +0, which changes no sum.
template <int COMPS>
__global__ void __launch_bounds__(64) k_diag_coarsen(MgLevel Lc, MgLevel Lf) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x, c0 = COMPS * blockIdx.y;
    if (n >= Lc.nn) return;
    const LevelIdx C(Lc), F(Lf);
    const int X = n % C.nnx, Y = (n / C.nnx) % C.nny, Z = n / (C.nnx * C.nny);
    const int s = Lc.span;
    const int fixed = Lc.mask[n] >> c0;   // bit k: component c0 + k
    const double* __restrict__ fd = Lf.diag + c0 * Lf.nn;
    double dc[COMPS], ws[COMPS];
#pragma unroll
    for (int k = 0; k < COMPS; ++k) dc[k] = ws[k] = 0.0;
    const bool skip = (fixed & ((1 << COMPS) - 1)) == (1 << COMPS) - 1;
    for (int col = 0; col < 8 && !skip; ++col) {
        const int ccx = (((X - 1) & 1) == (col & 1)) ? X - 1 : X;
        const int ccy = (((Lc.ny - Y) & 1) == ((col >> 1) & 1)) ? Y - 1 : Y;
        const int ccz = (((Z - 1) & 1) == ((col >> 2) & 1)) ? Z - 1 : Z;
        if (ccx < 0 || ccy < 0 || ccz < 0 || ccx >= Lc.nx || ccy >= Lc.ny || ccz >= Lc.nz) continue;
        const int a = corner_of(X - ccx, Y - ccy, Z - ccz);
        const int fx0 = ccx * s, fy0 = (ccy + 1) * s, fz0 = ccz * s;
        for (int iz = 0; iz <= s; ++iz)
#pragma unroll (COMPS == 1 ? 5 : 1)
            for (int iy = 0; iy <= s; ++iy) {
                double d[COMPS][5];
                int off[5];
#pragma unroll
                for (int ix = 0; ix < 5; ++ix) {
                    const int fn = F.node(fx0 + ix, fy0 - iy, fz0 + iz);
                    off[ix] = ix <= s ? Lf.mask[fn] >> c0 : 7;
#pragma unroll
                    for (int k = 0; k < COMPS; ++k) d[k][ix] = ix <= s ? fd[k * Lf.nn + fn] : 0.0;
                }
#pragma unroll
                for (int ix = 0; ix < 5; ++ix) {
                    const double w = corner_weight(s, ix, iy, iz, a), w2 = w * w;
#pragma unroll
                    for (int k = 0; k < COMPS; ++k) {
                        const bool on = !((off[ix] >> k) & 1);
                        const double v = on ? w2 : 0.0;
                        dc[k] = dc[k] + v * (on ? d[k][ix] : 0.0);
                        ws[k] = ws[k] + v;
                    }
                }
            }
    }
#pragma unroll
    for (int k = 0; k < COMPS; ++k) {
        double v = 1.0;
        if (!((fixed >> k) & 1) && ws[k] > 0) {
            v = dc[k] / ws[k];
            if (!(v > 0.0)) v = 1.0;
        }
        Lc.diag[(c0 + k) * Lc.nn + n] = v;
    }
}

// ------------------------------------------------------------------ restriction (transfers.cpp:449-533)
// The normalised hat-weighted window average, evaluated separably in three passes (x sums for each
// fine (z,y) row, then y, then z; each sum in increasing index order from 0; weight sum = product
// of the exact 1D sums), then scaled by 1/wSum and masked (preconditioner.cpp:183-191).  The CPU
// oracle's canonical mode evaluates the same order.
__global__ void k_restrict_x(MgLevel Lc, MgLevel Lf, const double* __restrict__ rf, double* __restrict__ a1,
                             const PcgScalars* S) {
    if (S != nullptr && S->done) return;
    const int cnx = Lc.nx + 1, fnx = Lf.nx + 1, fny = Lf.ny + 1, fnz = Lf.nz + 1;
    const int64_t total = (int64_t)fnz * fny * cnx;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int cx = (int)(t % cnx);
    const int64_t row = t / cnx;   // fz*fny + fy
    const int s = Lc.span, ws = 2 * s - 1;
    const int64_t fNN = Lf.nn;
    const double* __restrict__ src = rf + row * fnx;
    double v0 = 0.0, v1 = 0.0, v2 = 0.0;
    for (int ix = 0; ix < ws; ++ix) {
        const int fx = cx * s + ix - (s - 1);
        if (fx < 0 || fx >= fnx) continue;
        const double w = hat(ix, s);
        v0 = v0 + w * src[fx];
        v1 = v1 + w * src[fNN + fx];
        v2 = v2 + w * src[2 * fNN + fx];
    }
    a1[t] = v0;
    a1[total + t] = v1;
    a1[2 * total + t] = v2;
}

// sum of the in-range hat weights of coarse index c's window over n fine points
__device__ __forceinline__ double hat_sum(int c, int s, int n) {
    double sw = 0.0;
    for (int i = 0; i < 2 * s - 1; ++i) {
        const int f = c * s + i - (s - 1);
        if (f >= 0 && f < n) sw = sw + hat(i, s);
    }
    return sw;
}

// component c of a coarse node from its window sum: scaled by 1/wSum and masked.  normalize = 0: the plain
// hat-weighted sum, i.e. the transpose of the trilinear prolongation (the 'Standard' V-cycle option).
__device__ __forceinline__ double restrict_scale(const MgLevel& Lc, const MgLevel& Lf, int n, int cx, int cy, int cz,
                                                 int c, double v, int normalize) {
    const int s = Lc.span;
    double o = 0.0;
    if (!normalize) {
        o = v;
    } else {
        const double wsum = hat_sum(cz, s, Lf.nz + 1) * hat_sum(cy, s, Lf.ny + 1) * hat_sum(cx, s, Lf.nx + 1);
        if (wsum > 1e-12) o = v * (1.0 / wsum);
    }
    return ((Lc.mask[n] >> c) & 1) ? 0.0 : o;
}
__device__ __forceinline__ void restrict_store(const MgLevel& Lc, int n, int c, double o, double* __restrict__ rc,
                                               double* __restrict__ x0, double w0) {
    const int64_t i = c * Lc.nn + n;
    rc[i] = o;
    if (x0) {   // the Standard cycle's Jacobi start x0 = w0 rc / D
        const double d = Lc.diag[i];
        x0[i] = ((Lc.mask[n] >> c) & 1) ? 0.0 : (w0 * o) * (1.0 / (1.0e-30 < d ? d : 1.0e-30));
    }
}

// The y and z sums of a span-SP transition from the x pass, one thread per coarse node and component (blockIdx.y):
// the y sum of each fine z first, then the z sum, as three separate passes would add them.
template <int SP>
__global__ void __launch_bounds__(128) k_restrict_yz(MgLevel Lc, MgLevel Lf, const double* __restrict__ a1,
                                                     double* __restrict__ rc, const PcgScalars* S, int normalize,
                                                     double* __restrict__ x0, double w0) {
    if (S != nullptr && S->done) return;
    constexpr int WS = 2 * SP - 1;
    const int n = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (n >= Lc.nn) return;
    const int cnx = Lc.nx + 1, cny = Lc.ny + 1, fny = Lf.ny + 1, fnz = Lf.nz + 1;
    const int cx = n % cnx, cy = (n / cnx) % cny, cz = n / (cnx * cny);
    const double* __restrict__ a = a1 + c * ((int64_t)fnz * fny * cnx) + cx;
    double q[WS * WS];   // the whole window in flight; points outside the grid load nothing and add +0 (no change)
#pragma unroll
    for (int k = 0; k < WS * WS; ++k) {
        const int fy = cy * SP + k % WS - (SP - 1), fz = cz * SP + k / WS - (SP - 1);
        q[k] = fz >= 0 && fz < fnz && fy >= 0 && fy < fny ? a[(fz * fny + fy) * cnx] : 0.0;
    }
    double v = 0.0;
#pragma unroll
    for (int iz = 0; iz < WS; ++iz) {
        double t = 0.0;
#pragma unroll
        for (int iy = 0; iy < WS; ++iy) t = t + hat(iy, SP) * q[iz * WS + iy];
        v = v + hat(iz, SP) * t;
    }
    restrict_store(Lc, n, c, restrict_scale(Lc, Lf, n, cx, cy, cz, c, v, normalize), rc, x0, w0);
}

// The same two sums as separate passes, for large coarse grids: the y sum of every fine z once (a2: fine z x coarse y x
// coarse x), instead of once for each of the two coarse z whose windows hold it.  a, a2: one component (blockIdx.y).
template <int SP>
__global__ void __launch_bounds__(256) k_restrict_y(MgLevel Lc, MgLevel Lf, const double* __restrict__ a1,
                                                    double* __restrict__ a2, const PcgScalars* S) {
    if (S != nullptr && S->done) return;
    constexpr int WS = 2 * SP - 1;
    const int cnx = Lc.nx + 1, cny = Lc.ny + 1, fny = Lf.ny + 1, fnz = Lf.nz + 1, n2 = fnz * cny * cnx;
    const int i = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (i >= n2) return;
    const int cx = i % cnx, cy = (i / cnx) % cny, fz = i / (cnx * cny);
    const double* __restrict__ a = a1 + c * ((int64_t)fnz * fny * cnx) + cx;
    double q[WS];
#pragma unroll
    for (int iy = 0; iy < WS; ++iy) {
        const int fy = cy * SP + iy - (SP - 1);
        q[iy] = fy >= 0 && fy < fny ? a[(fz * fny + fy) * cnx] : 0.0;
    }
    double t = 0.0;
#pragma unroll
    for (int iy = 0; iy < WS; ++iy) t = t + hat(iy, SP) * q[iy];
    a2[(int64_t)c * n2 + i] = t;
}
template <int SP>
__global__ void __launch_bounds__(128) k_restrict_z(MgLevel Lc, MgLevel Lf, const double* __restrict__ a2,
                                                    double* __restrict__ rc, const PcgScalars* S, int normalize,
                                                    double* __restrict__ x0, double w0) {
    if (S != nullptr && S->done) return;
    constexpr int WS = 2 * SP - 1;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= Lc.nn) return;
    const int cnx = Lc.nx + 1, cny = Lc.ny + 1, fnz = Lf.nz + 1;
    const int cx = n % cnx, cy = (n / cnx) % cny, cz = n / (cnx * cny);
    const int64_t n2 = (int64_t)fnz * cny * cnx;
    const double* __restrict__ a = a2 + cy * cnx + cx;
    double v[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int iz = 0; iz < WS; ++iz) {
        const int fz = cz * SP + iz - (SP - 1);
        const bool in = fz >= 0 && fz < fnz;
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = v[c] + hat(iz, SP) * (in ? a[c * n2 + fz * cny * cnx] : 0.0);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
        restrict_store(Lc, n, c, restrict_scale(Lc, Lf, n, cx, cy, cz, c, v[c], normalize), rc, x0, w0);
}

// The 27-point window of a span-2 transition in the same nested order, from one component's residual
__device__ __forceinline__ double window2(const MgLevel& Lc, const MgLevel& Lf, int cx, int cy, int cz,
                                          const double* rf) {
    const int fnx = Lf.nx + 1, fny = Lf.ny + 1, fnz = Lf.nz + 1;
    double q[27];
#pragma unroll
    for (int k = 0; k < 27; ++k) {
        const int fx = cx * 2 + k % 3 - 1, fy = cy * 2 + (k / 3) % 3 - 1, fz = cz * 2 + k / 9 - 1;
        const bool in = fx >= 0 && fx < fnx && fy >= 0 && fy < fny && fz >= 0 && fz < fnz;
        q[k] = in ? rf[(fz * fny + fy) * fnx + fx] : 0.0;
    }
    double v = 0.0;
#pragma unroll
    for (int iz = 0; iz < 3; ++iz) {
        double t = 0.0;
#pragma unroll
        for (int iy = 0; iy < 3; ++iy) {
            double p = 0.0;
#pragma unroll
            for (int ix = 0; ix < 3; ++ix) p = p + hat(ix, 2) * q[9 * iz + 3 * iy + ix];
            t = t + hat(iy, 2) * p;
        }
        v = v + hat(iz, 2) * t;
    }
    return v;
}
__global__ void __launch_bounds__(128) k_restrict_xyz2(MgLevel Lc, MgLevel Lf, const double* __restrict__ rf,
                                                       double* __restrict__ rc, const PcgScalars* S, int normalize,
                                                       double* __restrict__ x0, double w0) {
    if (S != nullptr && S->done) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y;
    if (n >= Lc.nn) return;
    const int cnx = Lc.nx + 1, cny = Lc.ny + 1;
    const int cx = n % cnx, cy = (n / cnx) % cny, cz = n / (cnx * cny);
    const double v = window2(Lc, Lf, cx, cy, cz, rf + c * Lf.nn);
    restrict_store(Lc, n, c, restrict_scale(Lc, Lf, n, cx, cy, cz, c, v, normalize), rc, x0, w0);
}

// trilinear prolongation from the coarse cell floor(f/s), clamped to the last cell
// (transfers.cpp:378-445), then x = ((w r/D) + P x_c) + (w r/D), 0 on fixed DOFs
// (preconditioner.cpp:163-173, 230-253).
struct ProlongAt {   // a fine node's coarse cell and weights
    int b, py, pz;   // lowest corner, y and z strides
    double wx0, wx1, wy0, wy1, wz0, wz1;
    __device__ __forceinline__ ProlongAt(const MgLevel& Lc, int s, int fx, int fy, int fz) {
        const int cnx = Lc.nx + 1, cny = Lc.ny + 1;
        int cx = fx / s, cy = fy / s, cz = fz / s;
        int rx = fx % s, ry = fy % s, rz = fz % s;
        if (cx >= Lc.nx) { cx = Lc.nx - 1; rx = s; }
        if (cy >= Lc.ny) { cy = Lc.ny - 1; ry = s; }
        if (cz >= Lc.nz) { cz = Lc.nz - 1; rz = s; }
        const double inv = 1.0 / s;
        wx1 = rx * inv; wx0 = 1.0 - wx1;
        wy1 = ry * inv; wy0 = 1.0 - wy1;
        wz1 = rz * inv; wz0 = 1.0 - wz1;
        b = (cz * cny + cy) * cnx + cx;
        py = cnx;
        pz = cnx * cny;
    }
    __device__ __forceinline__ double operator()(const double* X) const {
        const int n000 = b, n100 = b + 1, n010 = b + py, n110 = b + py + 1;
        return X[n000] * wx0 * wy0 * wz0 + X[n100] * wx1 * wy0 * wz0 + X[n010] * wx0 * wy1 * wz0 +
               X[n110] * wx1 * wy1 * wz0 + X[n000 + pz] * wx0 * wy0 * wz1 + X[n100 + pz] * wx1 * wy0 * wz1 +
               X[n010 + pz] * wx0 * wy1 * wz1 + X[n110 + pz] * wx1 * wy1 * wz1;
    }
};
// x = ((w r/D) + P) + (w r/D), 0 on a fixed DOF
__device__ __forceinline__ double smooth(double w, double r, double d, double P, bool fixed) {
    const double t = w * r / (1.0e-30 < d ? d : 1.0e-30);
    return fixed ? 0.0 : (t + P) + t;
}

// COMPS components of a node per thread (3 / COMPS blocks in y)
template <int COMPS>
__global__ void __launch_bounds__(COMPS == 1 ? 128 : 256) k_prolong_smooth(MgLevel Lc, MgLevel Lf,
                                                                           const double* __restrict__ xc,
                                                                           const double* __restrict__ rf,
                                                                           double* __restrict__ xf, double w,
                                                                           const PcgScalars* S) {
    if (S != nullptr && S->done) return;
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= Lf.nn) return;
    const int fnx = Lf.nx + 1, fny = Lf.ny + 1;
    const ProlongAt P(Lc, Lc.span, n % fnx, (n / fnx) % fny, n / (fnx * fny));
#pragma unroll
    for (int k = 0; k < COMPS; ++k) {
        const int c = COMPS * blockIdx.y + k;
        const int64_t i = c * Lf.nn + n;
        xf[i] = smooth(w, rf[i], Lf.diag[i], P(xc + c * Lc.nn), (Lf.mask[n] >> c) & 1);
    }
}

// level 0: writes z and forms r.z in the canonical order; the last block sets rz (first use) or
// beta = rz_new/max(1e-30,rz), rz = rz_new (solver.cpp:186-198)
// CORNERS_FIRST: the coarse corners of all three components ahead of the fine node's values, in 60 registers instead of 80
// (more blocks per SM); else each component's together.
template <bool CORNERS_FIRST>
__global__ void __launch_bounds__(RED_THREADS) k_prolong_smooth0(MgLevel Lc, MgLevel Lf, const double* __restrict__ xc,
                                                                 const double* __restrict__ r, double* __restrict__ z,
                                                                 double w, RedSlot dot, PcgScalars* S) {
    __shared__ double sh[32];
    if (S->done) return;
    const int NN = (int)Lf.nn;
    const int fnx = Lf.nx + 1, fny = Lf.ny + 1;
    double part = 0.0;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < NN; n += gridDim.x * blockDim.x) {
        const ProlongAt at(Lc, Lc.span, n % fnx, (n / fnx) % fny, n / (fnx * fny));
        double P[3];
        if (CORNERS_FIRST)
            for (int c = 0; c < 3; ++c) P[c] = at(xc + c * Lc.nn);
        const int m = Lf.mask[n];
        for (int c = 0; c < 3; ++c) {
            const double rv = r[c * (int64_t)NN + n];
            const double p = CORNERS_FIRST ? P[c] : at(xc + c * Lc.nn);
            const double zv = smooth(w, rv, Lf.diag[c * (int64_t)NN + n], p, (m >> c) & 1);
            z[c * (int64_t)NN + n] = zv;
            part = part + rv * zv;
        }
    }
    double tot;
    if (grid_fold(part, dot, sh, &tot) && threadIdx.x == 0) {
        if (S->first) {
            S->rz = tot;
            S->first = 0;
        } else {
            const double rz = S->rz;
            S->beta = tot / (1.0e-30 < rz ? rz : 1.0e-30);
            S->rz = tot;
        }
    }
}

// ------------------------------------------------------------------ coarsest Galerkin (coarsest.cpp:138-323)
// One CTA (576 threads, thread = entry (i,j)) per coarse element.  The s^3 finest-grid sub-elements
// at the corner-sampled positions contribute T'(Kf T); Kf = Ke with modulus max(Emin,E) of the
// y-mirrored cell, with fixed DOFs' rows/cols replaced by identity when the sub-element touches any.
__global__ void __launch_bounds__(576) k_coarse_element(Grid g0, MgLevel Lc, int s, const uint8_t* __restrict__ mask0,
                                                        const double* __restrict__ E, const double* __restrict__ Keg,
                                                        double emin, double* __restrict__ Kce) {
    __shared__ double T[576], Kf[576], M[576];
    __shared__ int fmask[8];
    const int cel = blockIdx.x;   // (cez*nxc + cex)*nyc + cey
    const int nyc = Lc.ny, nxc = Lc.nx;
    const int cey = cel % nyc, cex = (cel / nyc) % nxc, cez = cel / (nyc * nxc);
    const int i = threadIdx.x / 24, j = threadIdx.x % 24;
    double acc_e = 0.0;
    for (int iz = 0; iz < s; ++iz)
        for (int iy = 0; iy < s; ++iy)
            for (int ix = 0; ix < s; ++ix) {
                const int fex = cex * s + ix, fey = (nyc - cey) * s - iy - 1, fez = cez * s + iz;
                double Ee = E[g0.cell(fex, g0.ny - 1 - fey, fez)];
                Ee = emin < Ee ? Ee : emin;
                if (threadIdx.x < 8) {
                    const int v = threadIdx.x;
                    fmask[v] = mask0[g0.node(fex + corner_dx(v), fey + corner_dy(v), fez + corner_dz(v))];
                }
                __syncthreads();
                int masked = 0;
                for (int v = 0; v < 8; ++v) masked |= fmask[v];
                {
                    // T[(3v+d), (3a+d)] = W_a at sub-node (ix+vx, iy+vy, iz+vz)
                    const int v = i / 3, d = i % 3, a = j / 3, e = j % 3;
                    const int vx = corner_dx(v), vy = 1 - corner_dy(v), vz = corner_dz(v);
                    T[threadIdx.x] = (d == e) ? corner_weight(s, ix + vx, iy + vy, iz + vz, a) : 0.0;
                    double k = masked ? Ee * Keg[threadIdx.x] : Keg[threadIdx.x];
                    if (masked) {
                        const int vi = i / 3, di = i % 3, vj = j / 3, dj = j % 3;
                        const int fi = (fmask[vi] >> di) & 1, fj = (fmask[vj] >> dj) & 1;
                        if (fi || fj) k = (i == j) ? 1.0 : 0.0;
                    }
                    Kf[threadIdx.x] = k;
                }
                __syncthreads();
                double m = 0.0;
                for (int k = 0; k < 24; ++k) m = m + Kf[i * 24 + k] * T[k * 24 + j];
                M[threadIdx.x] = m;
                __syncthreads();
                double acc = 0.0;
                for (int k = 0; k < 24; ++k) acc = acc + T[k * 24 + i] * M[k * 24 + j];
                acc_e = acc_e + (masked ? acc : Ee * acc);
                __syncthreads();
            }
    Kce[(int64_t)cel * 576 + threadIdx.x] = acc_e;
}

// Kc (row-major N x N, N = 3*coarse nodes, DOF 3n+c): lower-triangle sums over coarse elements in
// (cez, cex, cey) order, upper triangle 0, coarsest BC rows/cols -> identity (preconditioner.cpp:65-73)
__global__ void k_coarse_assemble(MgLevel Lc, const double* __restrict__ Kce, double* __restrict__ Kc) {
    const int N = 3 * (int)Lc.nn;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * N) return;
    const int gi = (int)(t / N), gj = (int)(t % N);
    const int nnx = Lc.nx + 1, nny = Lc.ny + 1;
    const int ni = gi / 3, ci = gi % 3, nj = gj / 3, cj = gj % 3;
    double v = 0.0;
    if (gi >= gj) {
        const int Xi = ni % nnx, Yi = (ni / nnx) % nny, Zi = ni / (nnx * nny);
        const int Xj = nj % nnx, Yj = (nj / nnx) % nny, Zj = nj / (nnx * nny);
        for (int ccz = Zi - 1; ccz <= Zi; ++ccz)
            for (int ccx = Xi - 1; ccx <= Xi; ++ccx)
                for (int ccy = Yi; ccy >= Yi - 1; --ccy) {   // cey = nyc-1-ccy ascending
                    if (ccx < 0 || ccx >= Lc.nx || ccy < 0 || ccy >= Lc.ny || ccz < 0 || ccz >= Lc.nz) continue;
                    const int dxj = Xj - ccx, dyj = Yj - ccy, dzj = Zj - ccz;
                    if (dxj < 0 || dxj > 1 || dyj < 0 || dyj > 1 || dzj < 0 || dzj > 1) continue;
                    const int ai = corner_of(Xi - ccx, Yi - ccy, Zi - ccz), aj = corner_of(dxj, dyj, dzj);
                    const int cel = (ccz * Lc.nx + ccx) * Lc.ny + (Lc.ny - 1 - ccy);
                    v = v + Kce[(int64_t)cel * 576 + (3 * ai + ci) * 24 + (3 * aj + cj)];
                }
    }
    const int mi = (Lc.mask[ni] >> ci) & 1, mj = (Lc.mask[nj] >> cj) & 1;
    if (mi || mj) v = (gi == gj) ? 1.0 : 0.0;
    Kc[t] = v;
}

// Cholesky of the lower triangle with the row-oriented sums of coarsest.cpp:13-35:
// L_ij = (A_ij - sum_{k<j} L_ik L_jk) / L_jj, L_jj = sqrt(A_jj - sum_{k<j} L_jk^2), sums in k order.
// Factor column j is LT[j*N + i] = L_ij.  Blocked right-looking: when column j is reached, LT holds in its rows
// i >= j the entry A_ij minus the products L_ik L_jk of the earlier columns, subtracted one at a time in
// increasing k -- the very sequence of the left-looking sum s = A_ij - L_i0 L_j0 - L_i1 L_j1 - ...
// (coarsest.cpp:24-58), so the factor is the same bit for bit.  Panels of CHOL_NB columns are factored by one
// CTA in shared memory; the panel's products are then subtracted from all later columns, in increasing k, by
// a grid of 32x32 tiles.  *status = 1 on success, 0 if not SPD (a non-positive pivot).
constexpr int CHOL_NB = 32;                  // panel width
constexpr int CHOL_SMEM_DOUBLES = 25600;     // panel bound: CHOL_NB x N doubles for N <= 800 (200 KB)
constexpr int CHOL_TILE = 32;

// LT = the lower triangle of A, transposed (column j contiguous); *status = 1
__global__ void k_chol_init(const double* __restrict__ A, double* __restrict__ LT, int N, int* status) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) *status = 1;
    if (t >= (int64_t)N * N) return;
    const int jj = (int)(t / N), ii = (int)(t % N);   // LT[jj][ii] = A[ii][jj] (lower)
    LT[t] = ii >= jj ? A[(int64_t)ii * N + jj] : 0.0;
}

// columns [k0, k1) of the factor, rows [k0, N): pan[c * R + o] = LT[(k0 + c) * N + k0 + o], R = N - k0
__global__ void __launch_bounds__(1024) k_chol_panel(double* __restrict__ LT, int N, int k0, int k1, int* status) {
    extern __shared__ double pan[];
    __shared__ int fail;
    if (*status == 0) return;   // an earlier panel failed (the same value for every thread)
    const int R = N - k0, W = k1 - k0;
    for (int t = threadIdx.x; t < W * R; t += blockDim.x) {
        const int c = t / R, o = t - c * R;
        pan[t] = LT[(int64_t)(k0 + c) * N + k0 + o];
    }
    if (threadIdx.x == 0) fail = 0;
    __syncthreads();
    for (int c = 0; c < W; ++c) {
        double* col = pan + c * R;   // column j = k0 + c; its row i at col[i - k0]
        if (threadIdx.x == 0) {
            const double s = col[c];
            if (s <= 0.0) fail = 1;
            else col[c] = sqrt(s);
        }
        __syncthreads();
        if (fail) break;
        const double ljj = col[c];
        for (int o = c + 1 + threadIdx.x; o < R; o += blockDim.x) col[o] = col[o] / ljj;
        __syncthreads();
        // the panel's later columns m = k0 + d, rows i >= m: subtract L_ij L_mj
        const int rest = W - c - 1;
        for (int t = threadIdx.x; t < rest * R; t += blockDim.x) {
            const int d = c + 1 + t / R, o = t % R;
            if (o >= d) pan[d * R + o] = pan[d * R + o] - col[o] * col[d];
        }
        __syncthreads();
    }
    if (fail) {
        if (threadIdx.x == 0) *status = 0;
        return;
    }
    for (int t = threadIdx.x; t < W * R; t += blockDim.x) {
        const int c = t / R, o = t - c * R;
        LT[(int64_t)(k0 + c) * N + k0 + o] = pan[t];
    }
}

// columns m >= k1, rows i >= m: subtract L_ij L_mj for the panel's columns j = k0..k1-1 in increasing j.
// Block t is the lower-triangular tile (bm <= bi) of 32 columns m and 32 rows i.
__global__ void __launch_bounds__(256) k_chol_trailing(double* __restrict__ LT, int N, int k0, int k1,
                                                       const int* status) {
    __shared__ double Pm[CHOL_NB][CHOL_TILE], Pi[CHOL_NB][CHOL_TILE];
    if (*status == 0) return;
    const int t = blockIdx.x;
    int bi = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
    while (bi * (bi + 1) / 2 > t) --bi;
    const int bm = t - bi * (bi + 1) / 2;
    const int m0 = k1 + bm * CHOL_TILE, i0 = k1 + bi * CHOL_TILE, W = k1 - k0;
    for (int q = threadIdx.x; q < W * CHOL_TILE; q += blockDim.x) {
        const int c = q / CHOL_TILE, x = q % CHOL_TILE;
        const double* Lj = LT + (int64_t)(k0 + c) * N;
        Pm[c][x] = m0 + x < N ? Lj[m0 + x] : 0.0;
        Pi[c][x] = i0 + x < N ? Lj[i0 + x] : 0.0;
    }
    __syncthreads();
    const int x = threadIdx.x % CHOL_TILE, y = threadIdx.x / CHOL_TILE;
    const int i = i0 + x;
    for (int u = y; u < CHOL_TILE; u += blockDim.x / CHOL_TILE) {
        const int m = m0 + u;
        if (m >= N || i >= N || i < m) continue;
        double* w = LT + (int64_t)m * N + i;
        double v = *w;
        for (int c = 0; c < W; ++c) v = v - Pi[c][x] * Pm[c][u];
        *w = v;
    }
}

// Lrow = the factor by rows (Lrow[i*N + j] = L_ij, 0 above the diagonal), written only on success
__global__ void k_chol_rows(const double* __restrict__ LT, double* __restrict__ Lrow, int N, const int* status) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)N * N || *status == 0) return;
    const int ii = (int)(t / N), jj = (int)(t % N);
    Lrow[t] = jj <= ii ? LT[(int64_t)jj * N + ii] : 0.0;
}

// Coarsest inverse for the canonical coarsest solve: column j of X = L'^-1 L^-1 e_j (coarsest.cpp:92-122),
// stored contiguously (X[j*N + i]).  A warp per column, both substitutions column-oriented: when x_k is final
// every row below takes its term L_ik x_k, so each row's running value receives its terms in increasing k
// (forward) and decreasing i (backward) and is divided last -- the order of the row-oriented sums, bit for bit.
// Rows above j are skipped in the forward pass: their values stay +0 and leave the others unchanged (each
// running value there is +0 or 1, never -0).  The warp's lanes split the rows, NV = N/32 (rounded up) running values
// in each lane's registers; the factor is read by columns (LT) in the forward pass and by rows (Lrow) in the backward
// one, both coalesced and a step ahead of their use.  What bounds it is the chain of divisions, one per step; with the
// running values in shared memory and the factor's loads in the chain it took 0.20, 0.53 and 1.39 ms for 135, 336 and
// 675 unknowns, now 0.12, 0.22 and 0.51.
constexpr int INV_WARPS = 4;   // columns per block
constexpr int INV_MAX_N = 1000;   // the largest dense coarsest system (NlimitDofs)
template <int NV>
__global__ void __launch_bounds__(INV_WARPS * 32) k_coarse_inverse(const double* __restrict__ LT,
                                                                   const double* __restrict__ Lrow, int N,
                                                                   const int* __restrict__ status,
                                                                   double* __restrict__ X) {
    if (*status != 1) return;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int j = blockIdx.x * INV_WARPS + w;
    if (j >= N) return;   // the whole warp (no block barrier below)
    double x[NV], a[NV], d;
#pragma unroll
    for (int v = 0; v < NV; ++v) x[v] = v * 32 + lane == j ? 1.0 : 0.0;
    // factor entries of step k's rows below (forward) or above (backward) it; others 0, which changes no value
    auto below = [&](int k) {
        d = k < N ? LT[(int64_t)k * N + k] : 1.0;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int i = v * 32 + lane;
            a[v] = k < N && i > k && i < N ? LT[(int64_t)k * N + i] : 0.0;
        }
    };
    auto above = [&](int i) {
        d = i >= 0 ? Lrow[(int64_t)i * N + i] : 1.0;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
            const int k = v * 32 + lane;
            a[v] = k < i ? Lrow[(int64_t)i * N + k] : 0.0;
        }
    };
    below(j);
#pragma unroll
    for (int vb = 0; vb < NV; ++vb) {
        if (vb * 32 + 31 < j) continue;
        for (int kk = 0; kk < 32; ++kk) {
            const int k = vb * 32 + kk;
            if (k < j || k >= N) continue;
            const double xk = __shfl_sync(0xffffffffu, x[vb], kk) / d;
            double q[NV];
#pragma unroll
            for (int v = vb; v < NV; ++v) q[v] = a[v] * xk;
            below(k + 1);
            if (lane == kk) x[vb] = xk;
#pragma unroll
            for (int v = vb; v < NV; ++v)
                if (v * 32 + lane > k) x[v] = x[v] - q[v];
        }
    }
    above(N - 1);
#pragma unroll
    for (int vb = NV - 1; vb >= 0; --vb) {
        for (int kk = 31; kk >= 0; --kk) {
            const int i = vb * 32 + kk;
            if (i >= N) continue;
            const double xi = __shfl_sync(0xffffffffu, x[vb], kk) / d;
            double q[NV];
#pragma unroll
            for (int v = 0; v <= vb; ++v) q[v] = a[v] * xi;
            above(i - 1);
            if (lane == kk) x[vb] = xi;
#pragma unroll
            for (int v = 0; v <= vb; ++v)
                if (v * 32 + lane < i) x[v] = x[v] - q[v];
        }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v)
        if (v * 32 + lane < N) X[(int64_t)j * N + v * 32 + lane] = x[v];
}

// Coarsest solve x_i = sum_j X[i][j] r_j (sequential in j) when the factorisation succeeded, else
// the Jacobi fallback x = r/max(1e-30,D) (preconditioner.cpp:195-215); masked (:217-227).
// The sum over j is one chain of additions per output, but its products are independent: a block of 32 outputs forms
// the products of CS_ROWS values of j at a time in shared memory with all its threads (eight loads of a thread in
// flight instead of one load per addition), then one thread per output adds them in order.
__device__ __forceinline__ double coarse_jacobi(double r, double d, bool fixed) {
    return fixed ? 0.0 : r / (1.0e-30 < d ? d : 1.0e-30);
}
constexpr int CS_THREADS = 512, CS_ROWS = 128;   // 32 outputs a block: 16 rows at a time, 32 KB of products
__global__ void __launch_bounds__(CS_THREADS) k_coarse_solve(MgLevel L, const double* __restrict__ X, int N,
                                                             const int* __restrict__ status, const PcgScalars* S) {
    extern __shared__ double rs[];
    if (S != nullptr && S->done) return;
    const int64_t nn = L.nn;
    if (*status != 1) {
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < 3 * nn; i += (int64_t)gridDim.x * blockDim.x)
            L.x[i] = coarse_jacobi(L.r[i], L.diag[i], (L.mask[i % nn] >> (i / nn)) & 1);
        return;
    }
    for (int j = threadIdx.x; j < N; j += blockDim.x) rs[j] = L.r[(j % 3) * nn + j / 3];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    double* prod = rs + N;
    double acc = 0.0;
    for (int j0 = 0; j0 < N; j0 += CS_ROWS) {
        double q[CS_ROWS / (CS_THREADS / 32)];
#pragma unroll
        for (int k = 0; k < CS_ROWS / (CS_THREADS / 32); ++k) {
            const int j = j0 + k * (CS_THREADS / 32) + warp;
            q[k] = j < N && i < N ? X[(int64_t)j * N + i] * rs[j] : 0.0;
        }
#pragma unroll
        for (int k = 0; k < CS_ROWS / (CS_THREADS / 32); ++k) prod[(k * (CS_THREADS / 32) + warp) * 32 + lane] = q[k];
        __syncthreads();
        if (warp == 0) {
            const int nr = min(CS_ROWS, N - j0);
#pragma unroll 8
            for (int j = 0; j < nr; ++j) acc = acc + prod[j * 32 + lane];
        }
        __syncthreads();
    }
    if (warp != 0 || i >= N) return;
    const int ni = i / 3, ci = i % 3;
    L.x[ci * nn + ni] = ((L.mask[ni] >> ci) & 1) ? 0.0 : acc;
}

// The Adapted cycle below a small level in one block: residuals restricted level by level, the coarsest solve, and
// prolongation with smoothing back up, all in shared memory, with the separate kernels' operations and order; the
// coarsest inverse is copied in while the residuals are restricted.  Replaces 2 (T - 1) + 1 launches for T levels.
// Levels of at most TAIL_NODES nodes and a coarsest system of at most TAIL_N, as long as all of it fits: above that
// one SM needs longer for the data than the launches take.  With it, two transfer kernels per level fewer and the
// predicated windows, a V-cycle takes 73 -> 41 us at 30x60x30 and 105 -> 68 us at 64x128x64.
constexpr int TAIL_NODES = 1536, TAIL_N = 160, TAIL_THREADS = 1024, TAIL_SMEM = 227 * 1024;
struct TailLevels {
    MgLevel lv[8];
    int n;
};
__global__ void __launch_bounds__(TAIL_THREADS, 1) k_adapted_tail(TailLevels T, const double* __restrict__ X, int N,
                                                                  const int* __restrict__ status, double w,
                                                                  const PcgScalars* S) {
    extern __shared__ __align__(16) double sm[];
    if (S != nullptr && S->done) return;
    double* Xs = sm;                           // the coarsest inverse (N x N, rounded up to whole 16 bytes)
    double* r = sm + (((int64_t)N * N + 1) & ~1ll);   // level residuals, level solutions; rs in the latter
    for (int i = threadIdx.x; i < (N * N) / 2; i += TAIL_THREADS)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(Xs + 2 * i)),
                     "l"(X + 2 * i)
                     : "memory");
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (((N * N) & 1) && threadIdx.x == 0) Xs[N * N - 1] = X[N * N - 1];
    const MgLevel& L0 = T.lv[0];
    for (int i = threadIdx.x; i < 3 * (int)L0.nn; i += TAIL_THREADS) r[i] = L0.r[i];
    __syncthreads();
    int off = 0;      // of level l's residual
    for (int l = 0; l + 1 < T.n; ++l) {
        const MgLevel &Lf = T.lv[l], &Lc = T.lv[l + 1];
        const int cnx = Lc.nx + 1, cny = Lc.ny + 1, nn = (int)Lc.nn, next = off + 3 * (int)Lf.nn;
        for (int i = threadIdx.x; i < 3 * nn; i += TAIL_THREADS) {
            const int c = i / nn, n = i - c * nn;
            const int cx = n % cnx, cy = (n / cnx) % cny, cz = n / (cnx * cny);
            const double v = window2(Lc, Lf, cx, cy, cz, r + off + c * Lf.nn);
            r[next + i] = restrict_scale(Lc, Lf, n, cx, cy, cz, c, v, 1);
        }
        __syncthreads();
        off = next;
    }
    const MgLevel& LL = T.lv[T.n - 1];
    const int nL = (int)LL.nn;
    double* x = r + off + 3 * nL;   // level l's solution; moves on as the cycle goes up
    if (*status != 1) {
        for (int i = threadIdx.x; i < 3 * nL; i += TAIL_THREADS)
            x[i] = coarse_jacobi(r[off + i], LL.diag[i], (LL.mask[i % nL] >> (i / nL)) & 1);
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");   // no copy of the inverse outlives the block
    } else {
        double* rs = x + 3 * nL;
        for (int j = threadIdx.x; j < N; j += TAIL_THREADS) rs[j] = r[off + (j % 3) * nL + j / 3];
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        const int i = threadIdx.x;
        if (i < N) {
            double acc = 0.0;
#pragma unroll 9
            for (int j = 0; j < N; ++j) acc = acc + Xs[j * N + i] * rs[j];
            x[(i % 3) * nL + i / 3] = ((LL.mask[i / 3] >> (i % 3)) & 1) ? 0.0 : acc;
        }
    }
    __syncthreads();
    for (int l = T.n - 2; l >= 0; --l) {
        const MgLevel &Lf = T.lv[l], &Lc = T.lv[l + 1];
        const int fnx = Lf.nx + 1, fny = Lf.ny + 1, nn = (int)Lf.nn;
        off -= 3 * nn;
        double* y = x + 3 * Lc.nn;
        for (int i = threadIdx.x; i < 3 * nn; i += TAIL_THREADS) {
            const int c = i / nn, n = i - c * nn;
            const ProlongAt P(Lc, 2, n % fnx, (n / fnx) % fny, n / (fnx * fny));
            const double v = smooth(w, r[off + i], Lf.diag[i], P(x + c * Lc.nn), (Lf.mask[n] >> c) & 1);
            if (l > 0) y[i] = v;
            else L0.x[i] = v;
        }
        __syncthreads();
        x = y;
    }
    if (T.n == 1)
        for (int i = threadIdx.x; i < 3 * nL; i += TAIL_THREADS) L0.x[i] = x[i];
}

inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void launch_mask_restrict(const MgLevel& Lc, const MgLevel& Lf, cudaStream_t s) {
    k_mask_restrict<<<blocks_for(Lc.nn, 128), 128, 0, s>>>(Lc, Lf);
}
// A thread per component ends a small level sooner, a thread per node shares the masks and weights: 37-40 and 41-43 us up
// to 4,000 nodes, 45 and 45 at 9,537, 0.191 and 0.164 ms at 30,625, 2.73 and 1.77 at 545,025.
constexpr int64_t DIAG_LARGE = 10000;
void launch_diag_coarsen(const MgLevel& Lc, const MgLevel& Lf, cudaStream_t s) {
    if (Lc.nn <= DIAG_LARGE) k_diag_coarsen<1><<<dim3(blocks_for(Lc.nn, 64), 3), 64, 0, s>>>(Lc, Lf);
    else k_diag_coarsen<3><<<blocks_for(Lc.nn, 64), 64, 0, s>>>(Lc, Lf);
}
// Levels of more nodes take fewer operations a node: separate y and z passes, and one thread for a node's three
// components.  Below, more threads with less work each finish sooner.  An Adapted V-cycle with all levels in the first
// and in the second form, ms: 0.264 and 0.261 at 70,785 level-1 nodes, 0.419 and 0.428 at 136,161, 0.662 and 0.682 at
// 232,897, 1.467 and 1.525 at 545,025.
constexpr int64_t LARGE_LEVEL = 100000;

// span 4 (the first transition): x pass, then the y-z pass or separate y and z passes; span 2: the whole window.
void launch_restrict(const MgLevel& Lc, const MgLevel& Lf, const double* rf, double* rc, double* a1, double* a2,
                     const PcgScalars* S, cudaStream_t s, bool normalize, double* x0, double w) {
    const dim3 b(blocks_for(Lc.nn, 128), 3);
    if (Lc.span == 2) {
        k_restrict_xyz2<<<b, 128, 0, s>>>(Lc, Lf, rf, rc, S, normalize ? 1 : 0, x0, w);
        return;
    }
    const int64_t n1 = (int64_t)(Lf.nz + 1) * (Lf.ny + 1) * (Lc.nx + 1);
    k_restrict_x<<<blocks_for(n1, 256), 256, 0, s>>>(Lc, Lf, rf, a1, S);
    if (!restrict_by_axes(Lc)) {
        k_restrict_yz<4><<<b, 128, 0, s>>>(Lc, Lf, a1, rc, S, normalize ? 1 : 0, x0, w);
        return;
    }
    const int64_t n2 = (int64_t)(Lf.nz + 1) * (Lc.ny + 1) * (Lc.nx + 1);
    k_restrict_y<4><<<dim3(blocks_for(n2, 256), 3), 256, 0, s>>>(Lc, Lf, a1, a2, S);
    k_restrict_z<4><<<b.x, 128, 0, s>>>(Lc, Lf, a2, rc, S, normalize ? 1 : 0, x0, w);
}
bool restrict_by_axes(const MgLevel& Lc) { return Lc.span == 4 && Lc.nn > LARGE_LEVEL; }
int restrict_launches(const MgLevel& Lc) { return Lc.span == 2 ? 1 : restrict_by_axes(Lc) ? 3 : 2; }
void launch_prolong_smooth(const MgLevel& Lc, const MgLevel& Lf, const double* xc, const double* rf, double* xf,
                           double weight, const PcgScalars* S, cudaStream_t s) {
    if (Lf.nn <= LARGE_LEVEL)
        k_prolong_smooth<1><<<dim3(blocks_for(Lf.nn, 128), 3), 128, 0, s>>>(Lc, Lf, xc, rf, xf, weight, S);
    else
        k_prolong_smooth<3><<<blocks_for(Lf.nn, 256), 256, 0, s>>>(Lc, Lf, xc, rf, xf, weight, S);
}
// Finest nodes from which the corners come first.  A PCG iteration with each component's together and with the corners
// first, us: 35.8 and 36.6 at 1,377 nodes, 61.4 and 62.2 at 70,785, 75.0 and 75.6 at 210,945, 88.7 and 88.2 at 232,897, 147.5
// and 146.6 at 545,025, 338 and 331 at 1.8 M; the kernel 1.17 and 1.12 ms at 33.9 M.
constexpr int64_t CORNERS_FIRST_MIN = 220000;
void launch_prolong_smooth0(const MgLevel& Lc, const MgLevel& Lf, const double* xc, const double* r, double* z,
                            double weight, RedSlot dot, PcgScalars* S, cudaStream_t s) {
    if (Lf.nn <= CORNERS_FIRST_MIN)
        k_prolong_smooth0<false><<<red_blocks(Lf.nn), RED_THREADS, 0, s>>>(Lc, Lf, xc, r, z, weight, dot, S);
    else
        k_prolong_smooth0<true><<<red_blocks(Lf.nn), RED_THREADS, 0, s>>>(Lc, Lf, xc, r, z, weight, dot, S);
}
void launch_coarse_element_matrices(const Grid& g0, const MgLevel& Lc, int span, const uint8_t* mask0, const double* E,
                                    const double* Ke, double emin, double* Kce, cudaStream_t s) {
    const int ncel = Lc.nx * Lc.ny * Lc.nz;
    k_coarse_element<<<ncel, 576, 0, s>>>(g0, Lc, span, mask0, E, Ke, emin, Kce);
}
void launch_coarse_assemble(const MgLevel& Lc, const double* Kce, double* Kc, cudaStream_t s) {
    const int64_t N = 3 * Lc.nn;
    k_coarse_assemble<<<blocks_for(N * N, 256), 256, 0, s>>>(Lc, Kce, Kc);
}
int launch_cholesky(const double* A, double* LT, double* Lrow, int N, int* status, cudaStream_t s) {
    const int64_t NN = (int64_t)N * N;
    k_chol_init<<<std::max(1u, blocks_for(NN, 256)), 256, 0, s>>>(A, LT, N, status);
    int launches = 1;
    if (N <= 0) return launches;
    const int nb = std::max(1, std::min(CHOL_NB, CHOL_SMEM_DOUBLES / N));
    // the attribute is per function, not per launch: always the bound, so that contexts set up concurrently
    // from several host threads never lower it under another thread's launch
    cudaFuncSetAttribute(k_chol_panel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(CHOL_SMEM_DOUBLES * sizeof(double)));
    for (int k0 = 0; k0 < N; k0 += nb) {
        const int k1 = std::min(k0 + nb, N);
        k_chol_panel<<<1, 1024, (size_t)(k1 - k0) * (N - k0) * sizeof(double), s>>>(LT, N, k0, k1, status);
        const int T = (N - k1 + CHOL_TILE - 1) / CHOL_TILE;
        if (T > 0) k_chol_trailing<<<T * (T + 1) / 2, 256, 0, s>>>(LT, N, k0, k1, status);
        launches += T > 0 ? 2 : 1;
    }
    k_chol_rows<<<blocks_for(NN, 256), 256, 0, s>>>(LT, Lrow, N, status);
    return launches + 1;
}
void launch_coarse_inverse(const double* LT, const double* Lrow, int N, const int* status, double* X,
                           cudaStream_t s) {
    const unsigned b = blocks_for(N, INV_WARPS);
    if (N <= 160) k_coarse_inverse<5><<<b, INV_WARPS * 32, 0, s>>>(LT, Lrow, N, status, X);
    else if (N <= 352) k_coarse_inverse<11><<<b, INV_WARPS * 32, 0, s>>>(LT, Lrow, N, status, X);
    else if (N <= 704) k_coarse_inverse<22><<<b, INV_WARPS * 32, 0, s>>>(LT, Lrow, N, status, X);
    else k_coarse_inverse<32><<<b, INV_WARPS * 32, 0, s>>>(LT, Lrow, N, status, X);
}
void launch_coarse_solve(const MgLevel& L, const double* X, int N, const int* status, const PcgScalars* S,
                         cudaStream_t s) {
    const unsigned blocks = N > 0 ? blocks_for(N, 32) : blocks_for(3 * L.nn, CS_THREADS);
    const size_t smem = (size_t)(std::max(N, 0) + 32 * CS_ROWS) * sizeof(double);   // N <= 1000: at most 41 KB
    k_coarse_solve<<<blocks, CS_THREADS, smem, s>>>(L, X, N, status, S);
}
cudaError_t mg_kernel_attributes() {
    const cudaError_t e = cudaFuncSetAttribute(k_coarse_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)((INV_MAX_N + 32 * CS_ROWS) * sizeof(double)));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_adapted_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, TAIL_SMEM);
}
static size_t tail_smem(const MgLevel* lv, int nlev, int first, int N) {
    int64_t doubles = (((int64_t)N * N + 1) & ~1ll) + N;
    for (int l = first; l < nlev; ++l) doubles += 6 * lv[l].nn;
    return (size_t)doubles * sizeof(double);
}
int adapted_tail_first(const MgLevel* lv, int nlev, int N) {
    if (N > TAIL_N) return nlev;
    int first = nlev;
    for (int l = nlev - 1; l >= 1 && lv[l].nn <= TAIL_NODES && (l == nlev - 1 || lv[l + 1].span == 2) &&
                           tail_smem(lv, nlev, l, N) <= TAIL_SMEM;
         --l)
        first = l;
    // a Jacobi coarsest level alone is better spread
    return first < nlev - 1 || (first == nlev - 1 && N > 0) ? first : nlev;
}
void launch_adapted_tail(const MgLevel* lv, int nlev, int first, const double* X, int N, const int* status, double w,
                         const PcgScalars* S, cudaStream_t s) {
    TailLevels T{};
    T.n = nlev - first;
    for (int l = first; l < nlev; ++l) T.lv[l - first] = lv[l];
    k_adapted_tail<<<1, TAIL_THREADS, tail_smem(lv, nlev, first, N), s>>>(T, X, N, status, w, S);
}

}  // namespace t3d
