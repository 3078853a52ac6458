// mlp_nt64.cu -- FP32 MLP kernels of nets whose weight chunks are 64 columns wide.
#include "mlp_impl.cuh"

namespace tmd {
template void mlp_plan_nt<64>(int, const int *, int, MlpPlan &);
template void launch_mlp_tr<64>(const MlpArgs &, cudaStream_t);
}  // namespace tmd
