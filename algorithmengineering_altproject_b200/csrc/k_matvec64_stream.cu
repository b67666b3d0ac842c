// The FP64 streaming product's tiling, its plain form and p.Ap (matvec64_stream.cuh has the kernel).
#include <algorithm>
#include <cmath>

#include "matvec64_stream.cuh"
#include "red.cuh"

namespace t3d {

namespace {

// p.Ap in the canonical order of k_dot (the fused dot of the node-centric kernel), skipped once S->done
__global__ void __launch_bounds__(RED_THREADS) k_dot_pcg(Grid g, const double* __restrict__ a,
                                                         const double* __restrict__ b, RedSlot red, PcgScalars* S) {
    __shared__ double sh[32];
    if (S->done) return;
    const int NN = (int)g.NN;
    double part = 0.0;
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < NN; n += gridDim.x * blockDim.x)
        for (int c = 0; c < 3; ++c) part = part + a[c * (int64_t)NN + n] * b[c * (int64_t)NN + n];
    double tot;
    if (grid_fold(part, red, sh, &tot) && threadIdx.x == 0) S->denom = tot;
}

}  // namespace

bool ke_pattern_magnitudes(const double* Ke, double* D) {
    for (int d = 0; d < KE_ND; ++d) D[d] = std::fabs(Ke[ke_first(d)]);
    for (int i = 0; i < 576; ++i)
        if (Ke[i] != (ke_neg(i) ? -D[ke_idx(i)] : D[ke_idx(i)])) return false;
    return true;
}

int stream64_tiling(const Grid& g, int dev, Stream64Tiling* t) {
    int per_sm = 1 << 30, sms = 0;
    for (auto mode : {occupancy<0>, stream64_occupancy_residual, stream64_occupancy_correct}) {
        int n = 0;
        const int rc = mode(&n);
        if (rc != T3D_OK) return rc;
        per_sm = std::min(per_sm, n);
    }
    cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return set_cuda_error(e, "cudaDeviceGetAttribute", __FILE__, __LINE__);
    if (per_sm < 1) return set_error(T3D_ERR_CUDA, "FP64 streaming K(E)u does not fit on an SM");
    const int resident = per_sm * sms;
    t->tiles_x = (g.nnx + S64::BX - 2) / (S64::BX - 1);
    t->tiles_y = (g.nny + S64::BY - 2) / (S64::BY - 1);
    const int tiles = t->tiles_x * t->tiles_y;
    // Planes per slab: a layer of a tile costs an SM about the same time whether one or two CTAs are resident (2.5 us,
    // half of it the FP64 pipe), so the launch takes as long as the SM with the most layers.  The smallest such maximum
    // wins: one plane per slab on toy grids (33 -> 15 us at 6x12x6), whole waves of long slabs on large ones.
    long best = 0;
    for (int slabs = 1; slabs <= g.nnz; ++slabs) {
        const int slab = (g.nnz + slabs - 1) / slabs;
        if (slabs != (g.nnz + slab - 1) / slab) continue;   // the same split as a smaller count
        const long cost = (long)((tiles * (long)slabs + sms - 1) / sms) * (slab + S64_ITEM_LAYERS);
        if (best == 0 || cost < best) {
            best = cost;
            t->slab = slab;
        }
    }
    t->slabs = (g.nnz + t->slab - 1) / t->slab;
    t->items = tiles * t->slabs;
    t->grid = std::min(resident, t->items);
    return T3D_OK;
}

void launch_matvec64_stream(const Grid& g, const Stream64Tiling& t, const double* Ke_host, const double* Kd,
                            const double* E, const uint8_t* mask, const double* u, double* y, const PcgScalars* S,
                            cudaStream_t s) {
    launch_stream<0>(g, t, Ke_host, Kd, E, mask, u, y, S, nullptr, nullptr, 0.0, s);
}
void launch_dot_pcg(const Grid& g, const double* p, const double* Ap, RedSlot red, PcgScalars* S, cudaStream_t s) {
    k_dot_pcg<<<red_blocks(g.NN), RED_THREADS, 0, s>>>(g, p, Ap, red, S);
}

}  // namespace t3d
