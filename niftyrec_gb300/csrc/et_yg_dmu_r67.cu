// d/dmu kernels for PSF radii 6 and 7.
#include "et_yg_dmu_kernels.cuh"

namespace nrgb {

template int launch_dmu_R<6>(const YgArgs& a, int n, int* slabs, cudaStream_t st);
template int launch_dmu_R<7>(const YgArgs& a, int n, int* slabs, cudaStream_t st);

}  // namespace nrgb
