// d/dmu kernels for PSF radii 0 and 1.
#include "et_yg_dmu_kernels.cuh"

namespace nrgb {

template int launch_dmu_R<0>(const YgArgs& a, int n, int* slabs, cudaStream_t st);
template int launch_dmu_R<1>(const YgArgs& a, int n, int* slabs, cudaStream_t st);

}  // namespace nrgb
