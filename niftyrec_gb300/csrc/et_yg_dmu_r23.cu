// d/dmu kernels for PSF radii 2 and 3.
#include "et_yg_dmu_kernels.cuh"

namespace nrgb {

template int launch_dmu_R<2>(const YgArgs& a, int n, int* slabs, cudaStream_t st);
template int launch_dmu_R<3>(const YgArgs& a, int n, int* slabs, cudaStream_t st);

}  // namespace nrgb
