// mlp_nt32.cu -- FP32 MLP kernels of nets whose weight chunks are 32 columns wide.
#include "mlp_impl.cuh"

namespace tmd {
template void mlp_plan_nt<32>(int, const int *, int, MlpPlan &);
template void launch_mlp_tr<32>(const MlpArgs &, cudaStream_t);
}  // namespace tmd
