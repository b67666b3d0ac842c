// K(E) u in FP64, element-streaming, bit-identical to the node-centric k_matvec64 (and so to the oracle).
//
// k_matvec64 gathers, for every node, the 24 values of each of its 8 elements (192 loads per node) and
// runs the 24-term FMA chain of the node's 3 rows of Ke; that form is L1-bound.  Here each element's 24
// values are gathered once and all 8 x 3 chains of the element are run in the same operation order
// (f = fma(Ke[row][j], u_e[j], f), j = 0..23); each node then adds its 8 element contributions in the
// reference's colour order (colour = ex&1 | (ey&1)<<1 | (ez&1)<<2, fea.cpp:300), y = fma(f, E, y),
// skipping E <= 1e-16, exactly as k_matvec64 does.  Only the place where each chain runs changes.
//
// Streaming: a CTA of BX x BY threads (one element column each) owns a (BX-1) x (BY-1) tile of node
// columns and marches up a slab of node planes; node planes come through a 3-slot cp.async ring in
// shared memory (the plane below stays in the ring while the plane above arrives).  Per element layer
// the chains' results go to shared memory, the top corners' in one of two slots by the layer's parity, so that
// when the layer above is done each owned node of the plane between folds its 8 elements in colour order (the
// four of the even layer first).
// Coefficients: a DFMA whose coefficient is a constant-bank operand issues at about half the rate of
// one with register operands only, and a shared-memory broadcast of FP64 coefficients costs more than
// the DFMAs it feeds.  The built-in Ke has only KE_ND distinct magnitudes (ke_pattern.inc), so for it
// (PAT) they sit in registers and each coefficient is +-D[ke_idx(i)] (negation is an exact operand
// modifier); the 24 rows of a column run in ke_row_order so that consecutive DFMAs share a coefficient
// register.  Any other Ke (t3d_set_ke) is passed by value and read from the constant bank.
// p.Ap is not fused: the caller folds it in the canonical order.
// What bounds it: the chains are 576 DFMAs a thread and layer, 1.3 ms at 256x512x256 with the tile halo, and the rest of a
// layer does not overlap them.  Hence the loads' places fixed per thread and the fold's order reduced to three parity
// bits: with index divisions in the loads and corner and side arithmetic in the fold, which were as many instructions as
// the chains, the launch took 2.81 ms, now 2.33 (96x192x96 with its dot 0.183, 0.155; 48x96x48 44 us, 36).
// One source file per MODE instantiates the kernel (k_matvec64_stream.cu, k_matvec64_residual.cu, k_matvec64_correct.cu):
// the pattern's unrolled chains take the compiler two minutes each, and the files build side by side.
#pragma once
#include "kernels.hpp"
#include "ke_pattern.inc"
#include "t3d_b200.h"

namespace t3d {

namespace {

__device__ __forceinline__ void cp_async8(unsigned s, const double* gsrc, bool valid) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(s), "l"(gsrc), "r"(valid ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }


static_assert(KE_ND <= KE_MAX_DISTINCT, "distinct-magnitude buffer too small");

constexpr int S64_BX = 32;
constexpr int S64_BY = 8;
constexpr int S64_ITEM_LAYERS = 2;   // a work item's overhead in element layers: its first one is computed twice, and
                                     // nothing overlaps its first loads

// Shared-memory layout of one CTA, in doubles.
struct S64 {
    static constexpr int BX = S64_BX, BY = S64_BY, PX = BX + 1, PY = BY + 1, NT = BX * BY;
    static constexpr int PLANE = 0;                     // [3 ring slots][3 components][PY][PX]
    static constexpr int PLANE_SZ = 3 * PY * PX;
    static constexpr int EMOD = PLANE + 3 * PLANE_SZ;   // [3 ring slots][BY][BX]: E of one element layer
    static constexpr int FB = EMOD + 3 * NT;            // [12][BY][BX]: rows 3a+r, corners a = 0..3
    static constexpr int FT = FB + 12 * NT;             // [2 layer parity][12][BY][BX]: rows 3(a-4)+r, a = 4..7
    static constexpr int TOTAL = FT + 24 * NT;
    static constexpr size_t BYTES = TOTAL * sizeof(double);
};

__device__ __forceinline__ unsigned smem_addr(const double* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

// One thread's share of a tile's loads: its own node of the (PX x PY) footprint from (X0-1, Y0-1), one node of the
// last row (warp 0) or column (the first PY threads of warp 1), and the modulus of its element column from cell
// (X0-1, Y0-1).  Places outside the grid load zero; cells beyond the ghost ring too (they are skipped like ghosts).
// The offsets in a plane are fixed for the item, so a step costs an address and a copy per value.
struct S64Loads {
    int off, off2;        // node offsets within a plane of u; the second for warps 0 and 1
    int dst2;             // the second node's place in the footprint
    bool ok, ok2, have2;  // inside the grid; a second node at all
    int eoff;             // cell offset within a layer (ghost ring included)
    bool eok;
    __device__ __forceinline__ S64Loads(const Grid& g, int X0, int Y0) {
        const int tx = threadIdx.x % S64::BX, ty = threadIdx.x / S64::BX;
        const int ix = X0 - 1 + tx, iy = Y0 - 1 + ty;
        ok = ix >= 0 && ix < g.nnx && iy >= 0 && iy < g.nny;
        off = ok ? iy * g.nnx + ix : 0;
        const int px = ty == 0 ? tx : S64::BX, py = ty == 0 ? S64::BY : tx;
        have2 = ty == 0 || (ty == 1 && tx < S64::PY);
        const int jx = X0 - 1 + px, jy = Y0 - 1 + py;
        ok2 = jx >= 0 && jx < g.nnx && jy >= 0 && jy < g.nny;
        off2 = ok2 ? jy * g.nnx + jx : 0;
        dst2 = py * S64::PX + px;
        eok = ix <= g.nx && iy <= g.ny;
        eoff = eok ? (iy + 1) * g.ex + ix + 1 : 0;
    }
    __device__ __forceinline__ void plane(const Grid& g, const double* __restrict__ u, int iz, double* dst) const {
        constexpr int AREA = S64::PY * S64::PX;
        const bool zok = iz >= 0 && iz < g.nnz;
        const double* src = u + (zok ? (int64_t)iz * g.nnx * g.nny : 0);
        const int tx = threadIdx.x % S64::BX, ty = threadIdx.x / S64::BX;
        const unsigned d = smem_addr(dst + ty * S64::PX + tx);
#pragma unroll
        for (int c = 0; c < 3; ++c) cp_async8(d + c * AREA * 8, src + c * g.NN + off, zok && ok);
        if (have2) {
            const unsigned d2 = smem_addr(dst + dst2);
#pragma unroll
            for (int c = 0; c < 3; ++c) cp_async8(d2 + c * AREA * 8, src + c * g.NN + off2, zok && ok2);
        }
    }
    __device__ __forceinline__ void emod(const Grid& g, const double* __restrict__ E, int cz, double* dst) const {
        cp_async8(smem_addr(dst + threadIdx.x), E + (eok ? (int64_t)(cz + 1) * g.ex * g.ey : 0) + eoff, eok);
    }
};
static_assert(S64_BX == 32 && S64_BY >= 2 && S64::PY <= 32, "S64Loads: warps 0 and 1 take the last row and column");

// MODE 0: y = K u;  1: the Standard V-cycle's residual y = r - K u;  2: its correction y = u + w (r - K u) / D, y other
// than u.  Fixed DOFs 0.  As one pass each, modes 1 and 2 save the two that read K u again.
template <bool PAT, int MODE>
__global__ void __launch_bounds__(S64::NT, 2) k_matvec64_stream(Grid g, Stream64Tiling t, const Ke64 ke,
                                                                const double* __restrict__ Kd,
                                                                const double* __restrict__ E,
                                                                const uint8_t* __restrict__ mask,
                                                                const double* __restrict__ u,
                                                                double* __restrict__ y, const PcgScalars* S,
                                                                const double* __restrict__ r,
                                                                const double* __restrict__ diag, double w_jac) {
    extern __shared__ __align__(16) double sm[];
    if (S != nullptr && S->done) return;
    constexpr int BX = S64::BX, BY = S64::BY, NT = S64::NT, PX = S64::PX, AREA = S64::PY * S64::PX;
    double* Fb = sm + S64::FB;
    const int tx = threadIdx.x % BX, ty = threadIdx.x / BX;
    const int64_t NN = g.NN;
    double D[PAT ? KE_ND : 1];   // PAT: the distinct magnitudes of Ke, loaded once into registers
#pragma unroll
    for (int d = 0; d < (PAT ? KE_ND : 1); ++d) D[d] = PAT ? __ldg(Kd + d) : 0.0;

    for (int w = blockIdx.x; w < t.items; w += gridDim.x) {
        const int tix = w % t.tiles_x, rest = w / t.tiles_x;
        const int tiy = rest % t.tiles_y, sl = rest / t.tiles_y;
        const int X0 = tix * (BX - 1), Y0 = tiy * (BY - 1);
        const int Z0 = sl * t.slab, Z1 = min(Z0 + t.slab, g.nnz);
        const int nlay = Z1 - Z0 + 1;   // element layers Z0-1 .. Z1-1
        const S64Loads ld(g, X0, Y0);
        __syncthreads();                // the previous item's owners are done with the rings
        ld.plane(g, u, Z0 - 1, sm + S64::PLANE);
        ld.plane(g, u, Z0, sm + S64::PLANE + S64::PLANE_SZ);
        ld.emod(g, E, Z0 - 1, sm + S64::EMOD);
        cp_commit();
#pragma unroll 1
        for (int k = 0; k < nlay; ++k) {
            const int cz = Z0 - 1 + k;   // element layer between node planes cz and cz+1
            cp_wait0();
            __syncthreads();
            if (k + 1 < nlay) {          // node plane cz+2 and the E of layer cz+1 for the next step
                ld.plane(g, u, cz + 2, sm + S64::PLANE + ((k + 2) % 3) * S64::PLANE_SZ);
                ld.emod(g, E, cz + 1, sm + S64::EMOD + ((k + 1) % 3) * NT);
            }
            cp_commit();
            // ---- element (tx, ty) of layer cz: the 24 FMA chains f_row = fma(Ke[row][j], u_e[j], f_row), j = 0..23
            double* Ft = sm + S64::FT + (k & 1) * 12 * NT;
            const double Ee = sm[S64::EMOD + (k % 3) * NT + threadIdx.x];
            if (PAT && !(Ee <= 1.0e-16)) {   // the owners skip exactly the elements skipped here
                const double* Pb = sm + S64::PLANE + (k % 3) * S64::PLANE_SZ;
                const double* Pt = sm + S64::PLANE + ((k + 1) % 3) * S64::PLANE_SZ;
                double f[24];
#pragma unroll
                for (int q = 0; q < 24; ++q) f[q] = 0.0;
#pragma unroll
                for (int j = 0; j < 24; ++j) {
                    const int a = j / 3, c = j % 3;
                    const double uj = (a < 4 ? Pb : Pt)[c * AREA + (ty + corner_dy(a)) * PX + tx + corner_dx(a)];
#pragma unroll
                    for (int r = 0; r < 24; ++r) {
                        const int q = ke_row_order(24 * j + r), i = 24 * q + j;
                        f[q] = fma(ke_neg(i) ? -D[ke_idx(i)] : D[ke_idx(i)], uj, f[q]);
                    }
                }
#pragma unroll
                for (int q = 0; q < 12; ++q) Fb[q * NT + threadIdx.x] = f[q];
#pragma unroll
                for (int q = 0; q < 12; ++q) Ft[q * NT + threadIdx.x] = f[12 + q];
            } else if (!PAT && !(Ee <= 1.0e-16)) {
                // any Ke: two halves of 12 rows, coefficients from the constant bank.  This form spills about 30 values a
                // thread and is the faster one: 24 rows in one pass, or u_e read again for each half, spill nothing and
                // take 45 us instead of 35 at 30x60x30, 1.14 ms instead of 0.97 at 160x320x160.
                const double* Pb = sm + S64::PLANE + (k % 3) * S64::PLANE_SZ;
                const double* Pt = sm + S64::PLANE + ((k + 1) % 3) * S64::PLANE_SZ;
                double ue[24];
#pragma unroll
                for (int a = 0; a < 8; ++a) {
                    const double* P = a < 4 ? Pb : Pt;
                    const int o = (ty + corner_dy(a)) * PX + tx + corner_dx(a);
#pragma unroll
                    for (int c = 0; c < 3; ++c) ue[3 * a + c] = P[c * AREA + o];
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    double f[12];
#pragma unroll
                    for (int q = 0; q < 12; ++q) f[q] = 0.0;
#pragma unroll
                    for (int j = 0; j < 24; ++j)
#pragma unroll
                        for (int q = 0; q < 12; ++q) f[q] = fma(ke.v[(12 * h + q) * 24 + j], ue[j], f[q]);
                    double* F = h == 0 ? Fb : Ft;
#pragma unroll
                    for (int q = 0; q < 12; ++q) F[q * NT + threadIdx.x] = f[q];
                }
            }
            __syncthreads();
            // ---- owners finish node plane iz = cz: 8 elements in colour order, even element layer first
            if (k >= 1 && tx < BX - 1 && ty < BY - 1) {
                const int ix = X0 + tx, iy = Y0 + ty, iz = cz;
                if (ix < g.nnx && iy < g.nny) {
                    const int64_t n = g.node(ix, iy, iz);
                    const int mk = mask[n];
                    double r0 = 0.0, r1 = 0.0, r2 = 0.0, d0 = 1.0, d1 = 1.0, d2 = 1.0;
                    if (MODE != 0) {
                        r0 = r[n];
                        r1 = r[NN + n];
                        r2 = r[2 * NN + n];
                    }
                    if (MODE == 2) {
                        d0 = diag[n];
                        d1 = diag[NN + n];
                        d2 = diag[2 * NN + n];
                    }
                    const double* Ebelow = sm + S64::EMOD + ((k - 1) % 3) * NT;
                    const double* Eabove = sm + S64::EMOD + (k % 3) * NT;
                    const double* Fbelow = sm + S64::FT + ((k - 1) & 1) * 12 * NT;
                    double y0 = 0.0, y1 = 0.0, y2 = 0.0;
                    // the node's colour order: bit 0, 1, 2 of the colour choose the element's side in x, y, z, the even
                    // one first; element column tx + sx (cx = ix-1+sx), row ty + sy, layer iz-1 (sz = 0) or iz
                    const int fx = (ix - 1) & 1, fy = (g.ny - iy) & 1, fz = (iz - 1) & 1;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int sz = h ^ fz;   // the same for the whole block
                        const double* Em = sz ? Eabove : Ebelow;
                        const double* Fm = sz ? Fb : Fbelow;
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const int sx = (q & 1) ^ fx, sy = (q >> 1) ^ fy;
                            const int e = threadIdx.x + sy * BX + sx;
                            const double Ec = Em[e];
                            if (Ec <= 1.0e-16) continue;
                            // corner of the element in its layer's plane: 1 - sx, 1 - sy -> 0 (0,1), 1 (1,1), 2 (1,0), 3 (0,0)
                            const int a = sy ? 3 - (1 - sx) : 1 - sx;
                            const double* F = Fm + 3 * a * NT + e;
                            y0 = fma(F[0], Ec, y0);
                            y1 = fma(F[NT], Ec, y1);
                            y2 = fma(F[2 * NT], Ec, y2);
                        }
                    }
                    if (MODE != 0) {
                        y0 = r0 - y0;
                        y1 = r1 - y1;
                        y2 = r2 - y2;
                    }
                    if (MODE == 2) {
                        const double* U = sm + S64::PLANE + (k % 3) * S64::PLANE_SZ + (ty + 1) * PX + tx + 1;
                        y0 = U[0] + (w_jac * y0) * (1.0 / (1.0e-30 < d0 ? d0 : 1.0e-30));
                        y1 = U[AREA] + (w_jac * y1) * (1.0 / (1.0e-30 < d1 ? d1 : 1.0e-30));
                        y2 = U[2 * AREA] + (w_jac * y2) * (1.0 / (1.0e-30 < d2 ? d2 : 1.0e-30));
                    }
                    if (mk & 1) y0 = 0.0;
                    if (mk & 2) y1 = 0.0;
                    if (mk & 4) y2 = 0.0;
                    y[n] = y0;
                    y[NN + n] = y1;
                    y[2 * NN + n] = y2;
                }
            }
        }
    }
    cp_wait0();
}

// the dynamic shared memory of MODE's two kernels, and the fewest of their CTAs that fit an SM
template <int MODE>
int occupancy(int* per_sm) {
    *per_sm = 1 << 30;
    for (auto fn : {k_matvec64_stream<true, MODE>, k_matvec64_stream<false, MODE>}) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S64::BYTES);
        if (e != cudaSuccess) return set_cuda_error(e, "cudaFuncSetAttribute", __FILE__, __LINE__);
        int n = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, S64::NT, S64::BYTES);
        if (e != cudaSuccess) return set_cuda_error(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor", __FILE__, __LINE__);
        if (n < *per_sm) *per_sm = n;
    }
    return T3D_OK;
}

template <int MODE>
void launch_stream(const Grid& g, const Stream64Tiling& t, const double* Ke_host, const double* Kd, const double* E,
                   const uint8_t* mask, const double* u, double* y, const PcgScalars* S, const double* r,
                   const double* diag, double w, cudaStream_t s) {
    if (Kd) {   // the by-value Ke is not read in this form
        static const Ke64 unused{};
        k_matvec64_stream<true, MODE><<<t.grid, S64::NT, S64::BYTES, s>>>(g, t, unused, Kd, E, mask, u, y, S, r, diag, w);
        return;
    }
    Ke64 ke;
    for (int i = 0; i < 576; ++i) ke.v[i] = Ke_host[i];
    k_matvec64_stream<false, MODE><<<t.grid, S64::NT, S64::BYTES, s>>>(g, t, ke, nullptr, E, mask, u, y, S, r, diag, w);
}

}  // namespace
}  // namespace t3d
