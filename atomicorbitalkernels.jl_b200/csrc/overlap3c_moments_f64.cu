// overlap3c_moments_f64.cu -- double instantiation of the 3-center kernels of bases with f
// shells.
#include "overlap3c_moments.cuh"

namespace aok {
namespace m3 {

int reserve_moments3_f64(aok_plan* p, cudaError_t* e) { return reserve_moments3<double>(p, e); }

int launch_moments3_f64(aok_plan* p, void* out, const void* posA, const void* posB, const void* posC, int64_t B,
                        double lengthscale, cudaStream_t s) {
    return launch_moments3<double>(p, out, posA, posB, posC, B, lengthscale, s);
}

}  // namespace m3
}  // namespace aok
