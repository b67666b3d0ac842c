// Products with a coarse level's Galerkin element matrices, shared by the FP64 and FP32 Standard V-cycles
// (k_mg_standard.cu, k_mg_standard32.cu).
//
// A node's row is one chain of 192 multiply-adds in the order elements (dz, dy, dx), columns.  Absent elements
// (outside the grid) contribute K = x = 0 instead of branching, which leaves the chain's value as it is (it starts
// at +0 and never becomes -0).  Consecutive lanes work on consecutive nodes and read consecutive addresses of the
// entry-major matrices.
//   level_split  small levels, latency-bound: a block is 32 nodes x 3 rows x 8 elements (a warp per row and
//                element), so all 192 loads of a row are in flight at once; the eight warps of a row then add
//                their 24 columns one after the other, handing the running sum on through shared memory.
//   level_nodes  larger levels, bound by the matrices' L2 and DRAM traffic: a thread per node with ROWS of its rows
//                (3 in FP32; 1 in FP64, the other rows in the block's other warps), a rolled loop over the elements.
//                (Unrolled over all elements the code, 50 KB, runs at the rate of instruction-cache misses at 30,625
//                nodes: 6 of 8 stall cycles per instruction.  The FP32 product is unrolled all the same on the largest
//                levels, k_mg_standard32.cu.)
// All add in the same order: identical bits.  Against a thread per node, fully unrolled, and separate residual and
// correction passes (ncu, cold caches): FP32 25 + 4 -> 7 us at 4,225 nodes, 31 + 6 -> 22 us at 30,625; FP64 57 + 6
// -> 9 us at 4,225, 433 + 9 -> 409 us at 545,025.  A V-cycle: FP32 0.386 -> 0.277 ms at 96x192x96, FP64 0.338 -> 0.251
// ms at 48x96x48.
#pragma once
#include "t3d_common.cuh"

namespace t3d {
namespace {

constexpr int LS_NODES = 32, LS_THREADS = 24 * LS_NODES;   // level_split
constexpr int LN_NODES = 128;                               // level_nodes, FP32; FP64: 32 x 3 rows

// what the kernels do with K x at a node: t = r - K x, or x + w (r - K x) / D
enum class LevelOp { Residual, Correct };

__device__ __forceinline__ float lp_add(float acc, float k, float x) { return fmaf(k, x, acc); }
__device__ __forceinline__ double lp_add(double acc, double k, double x) { return acc + k * x; }

// OFF(i, take): take(j, position of entry (i, j) of the 24 x 24 element matrix times the number of elements), j = 0..23
struct LpElement {   // element q of node (X, Y, Z): q = dx + 2 dy + 4 dz, at (X - dx, Y - dy, Z - dz)
    bool in;
    int e, m, a;     // element and its lowest node (0 when outside), the corner the node is of it
    __device__ LpElement(int nx, int ny, int nz, int X, int Y, int Z, int q) {
        const int dx = q & 1, dy = (q >> 1) & 1, dz = q >> 2;
        const int ex = X - dx, ey = Y - dy, ez = Z - dz;
        in = ex >= 0 && ey >= 0 && ez >= 0 && ex < nx && ey < ny && ez < nz;
        e = in ? (ez * ny + ey) * nx + ex : 0;
        m = in ? (ez * (ny + 1) + ey) * (nx + 1) + ex : 0;
        a = corner_of(dx, dy, dz);
    }
};
template <class T>
__device__ __forceinline__ void lp_load_x(const LpElement& q, int nnx, int nny, const T* __restrict__ x, int64_t cs,
                                          T (&xv)[24]) {
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const T* __restrict__ p = x + q.m + (corner_dz(b) * nny + corner_dy(b)) * nnx + corner_dx(b);
        xv[3 * b] = q.in ? p[0] : T(0);
        xv[3 * b + 1] = q.in ? p[cs] : T(0);
        xv[3 * b + 2] = q.in ? p[2 * cs] : T(0);
    }
}

// nodes n0 .. n0 + 31 of the level; store(n, row, K x) in the warps that end the chains.  Call from all threads of
// an LS_THREADS block; sums: 96 values of shared memory.
template <class T, class LEVEL, class OFF, class STORE>
__device__ __forceinline__ void level_split(const LEVEL& L, int64_t cs, int64_t n0, const T* __restrict__ Kel,
                                            const T* __restrict__ x, T* sums, OFF off, STORE store) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, row = wp % 3, q = wp / 3;
    const int nnx = L.nx + 1, nny = L.ny + 1;
    const bool live = n0 + lane < L.nn;
    const int n = (int)(live ? n0 + lane : 0);
    const int X = n % nnx, Y = (n / nnx) % nny, Z = n / (nnx * nny);
    const LpElement el(L.nx, L.ny, L.nz, X, Y, Z, q);
    T kv[24], xv[24];
    const T* __restrict__ K = Kel + el.e;
    off(3 * el.a + row, [&](int j, int64_t o) { kv[j] = el.in ? __ldg(K + o) : T(0); });
    lp_load_x(el, nnx, nny, x, cs, xv);
    T* sum = sums + row * LS_NODES + lane;
#pragma unroll 1
    for (int s = 0; s < 8; ++s) {
        if (q == s) {
            T acc = s == 0 ? T(0) : *sum;
#pragma unroll
            for (int j = 0; j < 24; ++j) acc = lp_add(acc, kv[j], xv[j]);
            if (s < 7) *sum = acc;
            else if (live) store(n, row, acc);
        }
        __syncthreads();
    }
}

// K x at node n: its rows row0 .. row0 + ROWS - 1
template <int ROWS, class T, class LEVEL, class OFF>
__device__ __forceinline__ void level_nodes(const LEVEL& L, int64_t cs, int n, int row0, const T* __restrict__ Kel,
                                            const T* __restrict__ x, OFF off, T (&acc)[ROWS]) {
    const int nnx = L.nx + 1, nny = L.ny + 1;
    const int X = n % nnx, Y = (n / nnx) % nny, Z = n / (nnx * nny);
#pragma unroll
    for (int r = 0; r < ROWS; ++r) acc[r] = T(0);
#pragma unroll 1
    for (int q = 0; q < 8; ++q) {
        const LpElement el(L.nx, L.ny, L.nz, X, Y, Z, q);
        const T* __restrict__ K = Kel + el.e;
        T kv[ROWS][24], xv[24];
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
            off(3 * el.a + row0 + r, [&](int j, int64_t o) { kv[r][j] = el.in ? __ldg(K + o) : T(0); });
        lp_load_x(el, nnx, nny, x, cs, xv);
#pragma unroll
        for (int j = 0; j < 24; ++j)
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r] = lp_add(acc[r], kv[r][j], xv[j]);
    }
}

}  // namespace
}  // namespace t3d
