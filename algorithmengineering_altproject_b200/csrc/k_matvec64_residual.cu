// The FP64 streaming product with the Standard V-cycle's residual (matvec64_stream.cuh).
#include "matvec64_stream.cuh"

namespace t3d {

int stream64_occupancy_residual(int* per_sm) { return occupancy<1>(per_sm); }
void launch_residual64_stream(const Grid& g, const Stream64Tiling& t, const double* Ke_host, const double* Kd,
                              const double* E, const uint8_t* mask, const double* u, const double* r, double* y,
                              const PcgScalars* S, cudaStream_t s) {
    launch_stream<1>(g, t, Ke_host, Kd, E, mask, u, y, S, r, nullptr, 0.0, s);
}

}  // namespace t3d
