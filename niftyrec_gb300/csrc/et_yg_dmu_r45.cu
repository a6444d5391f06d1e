// d/dmu kernels for PSF radii 4 and 5.
#include "et_yg_dmu_kernels.cuh"

namespace nrgb {

template int launch_dmu_R<4>(const YgArgs& a, int n, int* slabs, cudaStream_t st);
template int launch_dmu_R<5>(const YgArgs& a, int n, int* slabs, cudaStream_t st);

}  // namespace nrgb
