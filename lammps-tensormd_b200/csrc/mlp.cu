// mlp.cu -- FP32 MLP: shape limits, forms, weight packing and dispatch
// (kernel and semantics in mlp_impl.cuh).
#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "mlp_impl.cuh"
#include "tmd_b200.h"

namespace tmd {

void set_last_error(const std::string &m);  // abi.cpp

// one object per column-block width (mlp_nt32.cu, mlp_nt64.cu, mlp_nt128.cu)
extern template void mlp_plan_nt<32>(int, const int *, int, MlpPlan &);
extern template void mlp_plan_nt<64>(int, const int *, int, MlpPlan &);
extern template void mlp_plan_nt<128>(int, const int *, int, MlpPlan &);
extern template void launch_mlp_tr<32>(const MlpArgs &, cudaStream_t);
extern template void launch_mlp_tr<64>(const MlpArgs &, cudaStream_t);
extern template void launch_mlp_tr<128>(const MlpArgs &, cudaStream_t);

namespace {

__global__ void k_mlp_activation(int actfn, int n, const float *__restrict__ z,
                                 float *__restrict__ y, float *__restrict__ d) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float di;
  y[i] = mlp_act(actfn, z[i], di);
  d[i] = di;
}

// Column-block width of a net: the narrowest of 32, 64, 128 that holds its
// widest hidden layer in one block (wider layers take several blocks of 128).
// Widths between the blocks run padded, against the kernels this one replaced at
// 128,000 atoms: 80-80-80 878 -> 458 us, 96-96 568 -> 324, 160-160 1131 -> 987,
// 40-40 173 -> 109.
int mlp_nt(int nl, const int *sizes) {
  int maxh = 1;
  for (int l = 1; l < nl; l++) maxh = std::max(maxh, sizes[l]);
  return maxh <= 32 ? 32 : (maxh <= 64 ? 64 : 128);
}

}  // namespace

bool mlp_fp32_accepts(int nl, const int *sizes, int resnet) {
  // The widths this library takes: G, two activations and act' of 32 atoms
  // in 220 KB, or, for widths in multiples of 32, two activations, act' and
  // the residual gradient of 64 atoms beside two 128-column weight chunks.
  int maxh = 1, sum = 0, chunks = 0;
  bool all32 = true;
  for (int l = 0; l < nl - 1; l++) {
    maxh = std::max(maxh, sizes[l + 1]);
    sum += sizes[l + 1];
    all32 = all32 && sizes[l] % 32 == 0 && sizes[l + 1] % 32 == 0;
    chunks += mlp_cdiv(sizes[l + 1], 128) * (sizes[l] / 32) + mlp_cdiv(sizes[l], 128) * (sizes[l + 1] / 32);
  }
  const size_t f32 = ((size_t)std::max(sizes[0], maxh) + maxh + sum) * 36 + 32 * 68;
  const size_t f64 = ((size_t)(resnet ? 3 : 2) * maxh + sum - sizes[nl - 1]) * 68 +
                     2 * 32 * (128 + 68) + sum + 2 * sizes[nl - 1];
  return f32 * 4 <= 220 * 1024 || (all32 && chunks <= 256 && f64 * 4 <= 224 * 1024);
}

MlpPlan mlp_fp32_plan(int nl, const int *sizes, int actfn, int resnet, int nsm) {
  MlpPlan p{};
  p.nt = mlp_nt(nl, sizes);
  p.actfn = actfn;
  p.nsm = nsm;
  for (int l = 0; l < nl - 1; l++)
    p.nchunk += mlp_cdiv(sizes[l + 1], p.nt) * mlp_cdiv(sizes[l], kMlpPad) +
                mlp_cdiv(sizes[l], p.nt) * mlp_cdiv(sizes[l + 1], kMlpPad);
  switch (p.nt) {
    case 32: mlp_plan_nt<32>(nl, sizes, resnet, p); break;
    case 64: mlp_plan_nt<64>(nl, sizes, resnet, p); break;
    default: mlp_plan_nt<128>(nl, sizes, resnet, p); break;
  }
  return p;
}

int mlp_fp32_form(const MlpPlan &p, const int *count, int nelt) {
  // Time of the busiest SM, in units of one tile of 4 row registers on an SM
  // full of them, from timings of all forms inside a step on the B200 (five
  // nets of the three block widths, 108 to 400,000 atoms).  With every CTA slot
  // taken a tile costs thr (1 and 2 row registers are bound by shared memory, 4
  // and 8 by the FMA pipe).  The last, partial wave takes lat for its first
  // tile on an SM (bound by latency) and 0.75 thr for each further one beside
  // it.  In a grid of several waves the first 148 CTAs do not lie on 148 SMs:
  // from about 108 tiles (0.73 of the SMs) on, the last wave has two on one SM
  // (128,000 atoms in 1,000 tiles 162 us, 126,976 in 992 tiles 140).  Small
  // tiles spread few atoms over more SMs, large ones read the weights less
  // often: 8 row registers lose at 32 columns, where a tile has too few
  // weights to fill the pipe, and win at 64 and 128 once their waves are
  // nearly full.
  // Over that sweep the choice is within 0.2 / 0.2 / 0.6% of the best form on
  // average at 32 / 64 / 128 columns, within 3 / 6 / 9% at worst (one table for
  // all widths: 7.6 / 1.1 / 2.2%, 50 / 14 / 14%).  Times with 1 / 2 / 4 / 8 row
  // registers: 64-64-64 net, 4,000 atoms 19.6 / 18.7 / 27.5 / 37.4 us, 128,000
  // atoms - / 202 / 150 / 162; 32-wide net, 97,556 atoms 140 / 112 / 107 / 150;
  // 128-128x3 net, 23,328 atoms 316 / 235 / 155 / 146.
  static const double kLat[3][4] = {{0.84, 1.17, 2.22, 3.18}, {1.16, 1.20, 2.10, 3.04}, {0.97, 1.34, 1.71, 2.57}};
  static const double kThr[3][4] = {{0.41, 0.57, 1.0, 3.08}, {0.48, 0.66, 1.0, 1.77}, {0.57, 0.81, 1.0, 1.64}};
  const int w = p.nt == 32 ? 0 : (p.nt == 64 ? 1 : 2);
  int best = -1;
  double best_c = 0.0;
  for (int v = 0; v < 4; v++) {
    const int ctas = p.form[v].ctas;
    if (ctas == 0) continue;
    long tiles = 0;
    for (int e = 0; e < nelt; e++) tiles += mlp_cdiv(count[e], p.form[v].rows);
    const long waves = tiles / ((long)p.nsm * ctas), rest = tiles - waves * p.nsm * ctas;
    double c = (double)waves * ctas * kThr[w][v];
    if (rest > 0) {  // with `deep` tiles of the last wave on the busiest SM
      const double deep = std::ceil((double)rest / p.nsm + (waves > 0 ? 0.27 : 0.0));
      c += kLat[w][v] + 0.75 * (std::min(deep, (double)ctas) - 1.0) * kThr[w][v];
    }
    if (best < 0 || c < best_c) { best = v; best_c = c; }
  }
  return best;
}

void mlp_fp32_pack(int nl, const int *sizes, int nt, const std::vector<float> *W,
                   std::vector<float> &out) {
  out.clear();
  auto chunks = [&](int K, int N, auto at) {
    for (int n0 = 0; n0 < N; n0 += nt)
      for (int k0 = 0; k0 < K; k0 += kMlpPad)
        for (int k = k0; k < k0 + kMlpPad; k++)
          for (int n = n0; n < n0 + nt; n++) out.push_back(k < K && n < N ? at(k, n) : 0.f);
  };
  for (int l = 0; l < nl - 1; l++) {
    const int N = sizes[l + 1];
    chunks(sizes[l], N, [&](int k, int n) { return W[l][(size_t)k * N + n]; });
  }
  for (int l = nl - 2; l >= 0; l--) {
    const int N = sizes[l + 1];
    chunks(N, sizes[l], [&](int k, int n) { return W[l][(size_t)n * N + k]; });
  }
}

void launch_mlp_fp32(const MlpArgs &args, cudaStream_t st, long &launches) {
  if (args.ntiles <= 0) return;
  launches += 1;
  MlpArgs a = args;
  if (a.wait_cycles <= 0) a.wait_cycles = tc::kWaitCycles;
  switch (a.nt) {
    case 32: launch_mlp_tr<32>(a, st); break;
    case 64: launch_mlp_tr<64>(a, st); break;
    default: launch_mlp_tr<128>(a, st); break;
  }
}

}  // namespace tmd

extern "C" int tmd_mlp_activation(int device, int actfn, int n, const float *z, float *y,
                                  float *d) {
  if (actfn < 0 || actfn > 3 || n < 1 || !z || !y || !d) {
    tmd::set_last_error("tmd_mlp_activation: bad argument");
    return TMD_ERR_ARG;
  }
  int prev = 0;
  cudaGetDevice(&prev);
  float *buf = nullptr;
  const size_t bytes = (size_t)n * sizeof(float);
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaMalloc(&buf, 3 * bytes);
  if (e == cudaSuccess) e = cudaMemcpy(buf, z, bytes, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    tmd::k_mlp_activation<<<(n + 255) / 256, 256>>>(actfn, n, buf, buf + n, buf + 2 * (size_t)n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(y, buf + n, bytes, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(d, buf + 2 * (size_t)n, bytes, cudaMemcpyDeviceToHost);
  if (buf) cudaFree(buf);
  cudaSetDevice(prev);
  if (e == cudaSuccess) return TMD_OK;
  tmd::set_last_error(std::string("tmd_mlp_activation: ") + cudaGetErrorString(e));
  return TMD_ERR_CUDA;
}
