// Exact-transpose spread kernels for PSF radii 6 and 7.
#include "et_yg_spread_kernels.cuh"

namespace nrgb {

template int launch_spread_R<6, true>(const YgArgs& a, int c0, int gcount, cudaStream_t st);
template int launch_spread_pair_R<6, true>(const YgArgs& a, int u0, int gcount, cudaStream_t st);
template int launch_spread_R<7, true>(const YgArgs& a, int c0, int gcount, cudaStream_t st);
template int launch_spread_pair_R<7, true>(const YgArgs& a, int u0, int gcount, cudaStream_t st);

}  // namespace nrgb
