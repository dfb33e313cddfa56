// k_hii_zr at 256 (one translation unit per size: they compile in parallel).
#include "rg_hii_z.cuh"

namespace rg {
template int launch_hii_zr<256>(rg_context*, const cf*, int, const HiiZUnits&, cudaStream_t);
}  // namespace rg
