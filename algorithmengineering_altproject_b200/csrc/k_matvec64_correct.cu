// The FP64 streaming product with the Standard V-cycle's correction (matvec64_stream.cuh).
#include "matvec64_stream.cuh"

namespace t3d {

int stream64_occupancy_correct(int* per_sm) { return occupancy<2>(per_sm); }
void launch_correct64_stream(const Grid& g, const Stream64Tiling& t, const double* Ke_host, const double* Kd,
                             const double* E, const uint8_t* mask, const double* u, const double* r, const double* diag,
                             double w, double* y, const PcgScalars* S, cudaStream_t s) {
    launch_stream<2>(g, t, Ke_host, Kd, E, mask, u, y, S, r, diag, w, s);
}

}  // namespace t3d
