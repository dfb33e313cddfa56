// k_hii_zr at 512 (one translation unit per size: they compile in parallel).
#include "rg_hii_z.cuh"

namespace rg {
template int launch_hii_zr<512>(rg_context*, const cf*, int, const HiiZUnits&, cudaStream_t);
}  // namespace rg
