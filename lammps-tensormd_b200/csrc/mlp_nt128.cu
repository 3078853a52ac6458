// mlp_nt128.cu -- FP32 MLP kernels of nets whose weight chunks are 128 columns wide.
#include "mlp_impl.cuh"

namespace tmd {
template void mlp_plan_nt<128>(int, const int *, int, MlpPlan &);
template void launch_mlp_tr<128>(const MlpArgs &, cudaStream_t);
}  // namespace tmd
