// mlp_impl.cuh -- per-element atomic MLP E_i = NN_e(G_i) and dE/dG, FP32 plain form.
//
// Semantics (src/ML-TENSORMD/gpu/cuda/nnp.cu:9-57,149-281, nnp.cpp:246-365):
//   hidden layer l:  z = x W_l + b_l,  y = act(z) (+ x if use_resnet_dt,
//                    l > 0 and the layer keeps its width)
//   output layer:    E = x W_L (+ b_L if apply_output_bias)
//   backward:        g_{L-1} = W_L (sum over outputs), g_{l-1} = (g_l * act'(z_l))
//                    W_l^T (+ g_l on residual layers); dE/dG = g_{-1}
// Activations: 0 ReLU, 1 softplus, 2 tanh, 3 squareplus.
//
// One kernel for every net.  A CTA of 128 consumer threads walks tiles of R atoms of
// one element (R = TR row registers x 128 / (NT / 8) row groups) and runs each
// tile forward and backward.  Every GEMM of a tile is a sequence of weight
// chunks, KC (16 or 32) reduction rows x NT output columns (NT = 32, 64 or 128
// by the widest hidden layer).  The host packs an element's chunks in the order the
// tile consumes them (forward W, backward W^T, zero padded), and a producer
// warp streams them through a ring of S shared-memory stages with one cp.async.bulk each;
// layer 0's chunks carry the matching KC columns of the tile's G rows, copied
// row by row into a slot of their own on the same mbarrier.  The stream runs ahead across layers and
// tiles.  Thread (rg, cg) owns TR rows x 8 columns: per 4 reduction rows TR
// float4 of A and 8 of W feed 16 TR FFMA2.  A warp spans 4 row groups x 8
// column groups, so a half warp reads 128 distinct bytes of W and two rows of
// A: no bank conflicts, and at TR = 8 shared memory is half as busy as the FMA
// pipe.  act' stays in a per-CTA scratch (each thread reads back what it
// wrote, L2 resident), so a CTA needs ~110 KB of shared memory at most for
// the shipped nets and two or more share an SM: one's epilogue and barriers
// overlap the other's FMAs.
//
// Measured on the B200 against the kernels it replaced (a warp-tile form, a
// resident-weight form and a streamed form with 64- to 512-atom tiles), same
// sums bit for bit and before the activations below: 16 atoms of a 512-64x4 residual net 111 -> 40 us, 4,000
// atoms 64-64-64 49 -> 14, 23,040 atoms 128-128x3 residual 270 -> 169, 128,000
// atoms 64-64-64 180 -> 160, 432,000 atoms 512-128x3 5.86 -> 4.50 ms (56% of
// the FP32 peak).  (8 row registers at 128 columns spill 12 bytes, outside the
// GEMM.)  The producer needs a warp of its own: in a consumer warp
// its waits and copies hold up that warp's FMAs (5.1 ms).
//
// Sums per output run over the reduction index in ascending order whatever R
// is, so an atom's energy and gradient do not depend on the tile it is in.
#pragma once

#include <float.h>

#include <algorithm>
#include <vector>

#include "rcp.cuh"
#include "tc_util.cuh"
#include "tmd_kernels.h"

namespace tmd {

constexpr int kMlpThreads = 128;  // consumers: the threads of the GEMMs and epilogues
constexpr int kMlpBlock = kMlpThreads + 32;  // and one producer warp
constexpr int kMlpPad = 32;  // reduction rows of the packed weights are padded to this

// x < lim ? a : b as one select.  Left to the compiler, the cheaper side's
// operands go behind a branch that diverges lane by lane.
__device__ __forceinline__ float mlp_select(float x, float lim, float a, float b) {
  float y;
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %3, %4;\n\tselp.f32 %0, %1, %2, p;\n\t}"
      : "=f"(y)
      : "f"(a), "f"(b), "f"(x), "f"(lim));
  return y;
}

// Activation and its derivative (nnp.cu:9-57).  With one or two full-range
// divisions per value the epilogues were a sixth to a third of the kernel;
// these take one exponential (or square root) and reciprocals of sums in a
// known range, three quarters of the time per value (432,000-atom alloy,
// softplus: 4.50 -> 3.98 ms).  What a sum u = a + b with a >= b loses to
// rounding is b - (u - a) exactly (Dekker's fast two-sum), so the reciprocals
// hold the unrounded sum to about half an ulp.  Errors against FP64 over
// |z| < 12, rms (before, with divisions and tanhf): softplus 3.8e-8 (3.9e-8),
// its derivative 3.7e-8 (4.6e-8); tanh 1.7e-8 (2.2e-8), 5.4e-8 (7.5e-8);
// squareplus 3.3e-8 (3.9e-8), 4.8e-8 (5.4e-8).
__device__ __forceinline__ float mlp_act(int actfn, float z, float &d) {
  switch (actfn) {
    case 0:
      d = z > 0.f ? 1.f : 0.f;
      return z > 0.f ? z : 0.f;
    case 1: {
      // softplus = max(z, 0) + log1p(a), a = exp(-|z|); its derivative is
      // 1 / (1 + a) or a / (1 + a)
      const float a = expf(-fabsf(z));
      const float u = 1.f + a, r = rcp_sum(u, a - (u - 1.f));
      d = mlp_select(z, 0.f, a * r, r);
      return (z < 0.f ? 0.f : z) + log1pf(a);
    }
    case 2: {
      // with e = exp(-2|z|): tanh|z| = 1 - 2 e / (1 + e), whose term loses
      // (1 - T) / T of an ulp of T = tanh|z| per ulp of its own: half an ulp
      // and less from T = 2/3, |z| = 0.8.  Below, z + z^3 p(z^2) with p fitted
      // to that range (3.7e-9 of tanh).  tanh' = 1 - T^2 below and
      // sech^2 z = 4 e / (1 + e)^2 above, where 1 - T^2 cancels (at |z| = 3
      // one ulp of T is 1e-5 of it, an error that does not cancel in the
      // virial).
      const float t = fabsf(z);
      const float e = expf(-2.f * t);
      const float u = 1.f + e, r = rcp_sum(u, e - (u - 1.f));
      const float s = z * z;
      float p = fmaf(0.00158704445f, s, -0.00741417659f);
      p = fmaf(p, s, 0.0213065278f);
      p = fmaf(p, s, -0.0538535975f);
      p = fmaf(p, s, 0.133322418f);
      p = fmaf(p, s, -0.333332986f);
      const float y = mlp_select(t, 0.8f, fmaf(t * s, p, t), fmaf(-2.f * e, r, 1.f));
      d = mlp_select(t, 0.8f, fmaf(-y, y, 1.f), 4.f * e * (r * r));
      return copysignf(y, z);
    }
    default: {
      // squareplus = (z + q) / 2 with q = sqrt(z^2 + 4); for z < 0 the same
      // value is 2 / (|z| + q), which avoids the cancellation that costs FP32
      // most of its digits when z << 0.  Derivative: (1 + z / q) / 2, for
      // z < 0 the value over q.  q and 1/q come from the approximate reciprocal
      // square root i of w = z^2 + 4 by Karp and Markstein's arrangement of
      // Newton's step, q = w i + (w - (w i)^2) i / 2 (ACM TOMS 23, 1997), and
      // a Newton step of 1/q from i.  z is held at -1e18, where the value is
      // 1e-18 and z^2 does not overflow yet (not-a-number passes); z above
      // 1.8e19, whose square does, gives not-a-number.
      asm("max.NaN.f32 %0, %0, 0fDD5E0B6B;" : "+f"(z));
      const float t = fabsf(z);
      const float w = fmaf(z, z, 4.f);
      float i;
      asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(i) : "f"(w));
      const float q0 = w * i;
      const float q = fmaf(fmaf(-q0, q0, w), 0.5f * i, q0);
      const float iq = fmaf(i, fmaf(-q, i, 1.f), i);
      const float v = q + t, n = 2.f * rcp_sum(v, t - (v - q));
      d = mlp_select(z, 0.f, n * iq, fmaf(0.5f * z, iq, 0.5f));
      return mlp_select(z, 0.f, n, 0.5f * v);
    }
  }
}

__host__ __device__ inline int mlp_cdiv(int a, int b) { return (a + b - 1) / b; }

template <int NT, int TR>
struct MlpCfg {
  static constexpr int CG = NT / 8;                // column groups of 8 columns
  static constexpr int RG = kMlpThreads / CG;      // row groups
  static constexpr int R = RG * TR;                // atoms per tile
  static constexpr int CGW = CG < 8 ? CG : 8;      // column groups of a warp
  static constexpr int WC = CG / CGW;              // warps side by side in columns
  // small tiles run few CTAs and want the stream far ahead; large ones want
  // two or three CTAs on an SM
  static constexpr int KC = TR == 4 ? 16 : 32;     // reduction rows of a chunk
  static constexpr int S = TR <= 2 ? 6 : 3;        // stages
  static constexpr int GS = TR <= 2 ? S : 2;       // slots of G columns
  static constexpr int CTAS = TR == 8 ? 2 : 3;
  static constexpr int LDG = KC + 4;               // row stride of a G slot (floats)
  static constexpr int kW = KC * NT, kG = R * LDG; // floats of a stage, a slot
};

// Shared-memory layout behind the stages (floats); widths padded to NT.
struct MlpLay {
  int ldh, nbuf, h, bias, wout, ered, total;
};
__host__ __device__ inline MlpLay mlp_lay(int nl, const int *sizes, int nt, int r, int wc,
                                          int ring) {
  MlpLay f{};
  int maxh = 1, nb = 0;
  for (int l = 1; l < nl; l++) {
    const int np = mlp_cdiv(sizes[l], nt) * nt;
    maxh = maxh > np ? maxh : np;
    nb += np;
  }
  f.ldh = maxh + 4;
  f.nbuf = maxh > nt ? 2 : 1;  // one block of columns is rewritten in place
  int o = ring;
  f.h = o; o += f.nbuf * r * f.ldh;
  f.bias = o; o += nb;
  f.wout = o; o += 2 * mlp_cdiv(sizes[nl - 1], nt) * nt;  // doubles
  f.ered = o; o += 2 * wc * r;                         // doubles
  f.total = o;
  return f;
}

// acc += A[rows][k0..k0+4 k4) W chunk, the reduction index ascending.
template <int NT, int TR, int UN>
__device__ __forceinline__ void mlp_chunk(const float *A, int lda, const float *W, int k4,
                                          float2 (&acc)[TR][4]) {
  constexpr int RG = MlpCfg<NT, TR>::RG;
#pragma unroll UN
  for (int q = 0; q < k4; q++) {
    float4 av[TR];
#pragma unroll
    for (int i = 0; i < TR; i++)
      av[i] = *reinterpret_cast<const float4 *>(A + i * RG * lda + 4 * q);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const float4 b0 = *reinterpret_cast<const float4 *>(W + (4 * q + u) * NT);
      const float4 b1 = *reinterpret_cast<const float4 *>(W + (4 * q + u) * NT + NT / 2);
      const float2 bb[4] = {make_float2(b0.x, b0.y), make_float2(b0.z, b0.w),
                            make_float2(b1.x, b1.y), make_float2(b1.z, b1.w)};
#pragma unroll
      for (int i = 0; i < TR; i++) {
        const float x = u == 0 ? av[i].x : (u == 1 ? av[i].y : (u == 2 ? av[i].z : av[i].w));
        const float2 x2 = make_float2(x, x);
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = __ffma2_rn(x2, bb[j], acc[i][j]);
      }
    }
  }
}

template <int NT, int TR, int ACT>
__global__ void __launch_bounds__(kMlpBlock, MlpCfg<NT, TR>::CTAS)
k_mlp_fp32(MlpArgs a) {
  using C = MlpCfg<NT, TR>;
  constexpr int RG = C::RG, R = C::R, S = C::S, KC = C::KC, LDG = C::LDG;
  extern __shared__ float4 mlp_dyn[];
  float *sm = reinterpret_cast<float *>(mlp_dyn);
  __shared__ __align__(8) uint64_t fullb[S], emptyb[S];
  __shared__ int rows_s[R];
  const int L = a.nl, nin = a.nin;
  const int *sizes = a.sizes;
  const MlpLay lay = mlp_lay(L, sizes, NT, R, C::WC, S * C::kW + C::GS * C::kG);
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  const int wc = w % C::WC;
  const int cg = wc * C::CGW + lane % C::CGW;
  const int rg = (w / C::WC) * (32 / C::CGW) + lane / C::CGW;
  float *hin = sm + lay.h, *hout = lay.nbuf == 2 ? hin + R * lay.ldh : hin;
  const int ldh = lay.ldh;
  float *bias_s = sm + lay.bias;
  double *wout_s = reinterpret_cast<double *>(sm + lay.wout);
  double *ered = reinterpret_cast<double *>(sm + lay.ered);
  const int woutp = mlp_cdiv(sizes[L - 1], NT) * NT;
  // this thread's act' (and residual gradient) slots, 2 float4 per row and
  // column block of the hidden layers below the last
  float4 *dzs = a.scratch + (size_t)blockIdx.x * a.scratch_f4 + tid;
  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      tc::mbar_init(&fullb[s], 1);
      tc::mbar_init(&emptyb[s], kMlpThreads / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();

  const int Q = a.nchunk * (kMlpPad / KC);
  const int gq = mlp_cdiv(nin, kMlpPad) * (kMlpPad / KC);
  const int q0 = mlp_cdiv(sizes[1], NT) * gq;  // chunks that carry G columns
  bool bad = false;
  auto wait = [&](uint64_t *b, uint32_t parity) {
    if (tc::mbar_test(b, parity)) return;
    if (!tc::mbar_wait(b, parity, bad ? 1 : a.wait_cycles)) bad = true;
  };
  auto sync = [] { asm volatile("bar.sync 1, %0;" ::"n"(kMlpThreads) : "memory"); };
  if (w == kMlpThreads / 32) {
    // ---- producer: every chunk of this CTA's tiles into the ring, a stage
    // as soon as the four consumer warps have released it
    if (a.probe == kMlpProbeConsumer) return;
    int st = 0, round = 0, slot = 0;
    for (int tile = blockIdx.x; tile < a.ntiles && !bad; tile += gridDim.x) {
      const int elt = __ldg(a.tiles + 3 * tile), start = __ldg(a.tiles + 3 * tile + 1),
                count = __ldg(a.tiles + 3 * tile + 2);
      constexpr int kRows = (R + 31) / 32;
      int at[kRows];
#pragma unroll
      for (int u = 0; u < kRows; u++) {
        const int r = lane + 32 * u;
        at[u] = r < count && r < R ? __ldg(a.perm + start + r) : -1;
      }
      const float *src = a.stream + (size_t)elt * Q * (KC * NT);
      int kg = 0;
      for (int q = 0; q < Q; q++) {
        if (round > 0) wait(&emptyb[st], (uint32_t)(round - 1) & 1u);
        int wid = 0;  // G columns of the chunk
        if (q < q0) {
          wid = max(min(KC, nin - KC * kg), 0);
          // its G slot is that of the chunk GS before it at the latest: chunks
          // are consumed in order, so that chunk's stage must be released
          if (C::GS < S) {
            const int ps = st >= C::GS ? st - C::GS : st - C::GS + S;
            const int pr = st >= C::GS ? round : round - 1;
            if (pr >= 0) wait(&emptyb[ps], (uint32_t)pr & 1u);
          }
        }
        bad = __any_sync(0xffffffffu, bad);  // the warp issues or stops together
        if (bad) break;
        const uint32_t bar = tc::smem_u32(&fullb[st]);
        if (lane == 0) {
          tc::mbar_expect_tx(bar, (uint32_t)(KC * NT * 4 + count * wid * 4));
          tc::bulk_g2s(tc::smem_u32(sm + st * C::kW), src + (size_t)q * (KC * NT), KC * NT * 4,
                       bar);
        }
        if (q < q0) {
          __syncwarp();
          if (wid > 0) {
            float *gst = sm + S * C::kW + slot * C::kG;
#pragma unroll
            for (int u = 0; u < kRows; u++)
              if (at[u] >= 0)
                tc::bulk_g2s(tc::smem_u32(gst + (lane + 32 * u) * LDG),
                             a.G + (size_t)at[u] * nin + KC * kg, (uint32_t)wid * 4u, bar);
          }
          kg = kg + 1 == gq ? 0 : kg + 1;
          slot = slot + 1 == C::GS ? 0 : slot + 1;
        }
        if (++st == S) { st = 0; round++; }
      }
    }
    if (bad) {
      // a wait gave up: report it, and give the copies still in flight a
      // bounded time to land before the CTA's shared memory is released
      if (a.status && lane == 0) atomicOr(a.status, kStatusTimeout);
      for (int s = 0; s < S; s++) {
        const int issued = round + (s < st ? 1 : 0);
        if (issued > 0) tc::mbar_wait(&fullb[s], (uint32_t)(issued - 1) & 1u);
      }
    }
    return;
  }
  // ---- consumer
  if (a.probe == kMlpProbeProducer) return;
  int c_st = 0, c_g = 0;
  uint32_t c_ph = 0;
  float2 acc[TR][4];
  // acc = A W over K reduction rows (one column block), A from the chunk's G
  // columns (from_g) or the hidden buffer
  auto gemm = [&](bool from_g, int K) {
#pragma unroll
    for (int i = 0; i < TR; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) acc[i][j] = make_float2(0.f, 0.f);
    for (int k0 = 0; k0 < mlp_cdiv(K, kMlpPad) * kMlpPad; k0 += KC) {
      wait(&fullb[c_st], c_ph);
      const float *W = sm + c_st * C::kW + 4 * cg;
      const int k4 = max(min(KC / 4, (K - k0 + 3) / 4), 0);
      constexpr int UN = TR == 8 ? 1 : (TR == 4 ? 2 : 4);
      if (from_g) {
        const float *A = sm + S * C::kW + c_g * C::kG + rg * LDG;
        c_g = c_g + 1 == C::GS ? 0 : c_g + 1;
        if (k4 == KC / 4) mlp_chunk<NT, TR, UN>(A, LDG, W, KC / 4, acc);
        else mlp_chunk<NT, TR, 1>(A, LDG, W, k4, acc);
      } else if (ldh == NT + 4 && k4 == KC / 4) {
        mlp_chunk<NT, TR, UN>(hin + rg * (NT + 4) + k0, NT + 4, W, KC / 4, acc);
      } else {
        mlp_chunk<NT, TR, 1>(hin + rg * ldh + k0, ldh, W, k4, acc);
      }
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&emptyb[c_st]);
      if (++c_st == S) { c_st = 0; c_ph ^= 1u; }
    }
  };
  auto col_of = [&](int nb, int h) { return nb * NT + h * (NT / 2) + 4 * cg; };
  auto is_res = [&](int l) { return a.resnet && l > 0 && sizes[l] == sizes[l + 1]; };

  int cur_elt = -1;
  for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
    const int elt = __ldg(a.tiles + 3 * tile), start = __ldg(a.tiles + 3 * tile + 1),
              count = __ldg(a.tiles + 3 * tile + 2);
    sync();  // the previous tile's readers of rows_s, bias_s and ered are done
    for (int r = tid; r < R; r += kMlpThreads)
      rows_s[r] = r < count ? __ldg(a.perm + start + r) : -1;
    const MlpLayer *Ls = a.layers + (size_t)elt * L;
    if (elt != cur_elt) {
      cur_elt = elt;
      int ob = 0;
      for (int l = 0; l < L - 1; l++) {
        const int N = sizes[l + 1], np = mlp_cdiv(N, NT) * NT;
        const float *b = Ls[l].b;
        for (int c = tid; c < np; c += kMlpThreads)
          bias_s[ob + c] = (b != nullptr && c < N) ? __ldg(b + c) : 0.f;
        ob += np;
      }
      for (int c = tid; c < woutp; c += kMlpThreads)
        wout_s[c] = c < sizes[L - 1] ? __ldg(Ls[L - 1].Wd + c) : 0.0;
    }
    sync();

    // ---------------- forward ----------------
    int ob = 0, slot = 0;
    for (int l = 0; l < L - 1; l++) {
      const int K = sizes[l], nbn = mlp_cdiv(sizes[l + 1], NT);
      const bool last = l == L - 2, res = is_res(l);
      for (int nb = 0; nb < nbn; nb++) {
        gemm(l == 0, K);
        sync();  // every warp has read the layer's input block
        // z into the hidden buffer, then the activation as a loop over the
        // thread's own groups of four columns: inlined for the whole register
        // tile it is 100 KB of code and stalls on instruction fetch
#pragma unroll
        for (int i = 0; i < TR; i++) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int c = col_of(nb, h);
            float4 *p = reinterpret_cast<float4 *>(hout + (i * RG + rg) * ldh + c);
            const float4 b4 = *reinterpret_cast<const float4 *>(bias_s + ob + c);
            if (res)  // the layer's input, out of the way of z
              dzs[(size_t)(slot + (nb * TR + i) * 2 + h) * kMlpThreads] =
                  *reinterpret_cast<const float4 *>(hin + (i * RG + rg) * ldh + c);
            *p = make_float4(acc[i][2 * h].x + b4.x, acc[i][2 * h].y + b4.y,
                             acc[i][2 * h + 1].x + b4.z, acc[i][2 * h + 1].y + b4.w);
          }
        }
        constexpr int GU = TR < 2 ? TR : 2;  // rows per trip
#pragma unroll 1
        for (int i0 = 0; i0 < TR; i0 += GU) {
#pragma unroll
          for (int iu = 0; iu < GU; iu++) {
            const int i = i0 + iu;
            double e = 0.0;
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int c = col_of(nb, h);
              float4 *p = reinterpret_cast<float4 *>(hout + (i * RG + rg) * ldh + c);
              float4 *dp = dzs + (size_t)(slot + (nb * TR + i) * 2 + h) * kMlpThreads;
              const float4 z4 = *p;
              float4 x4 = make_float4(0.f, 0.f, 0.f, 0.f);
              if (res) x4 = *dp;
              float y[4], d[4];
              y[0] = mlp_act(ACT, z4.x, d[0]) + x4.x;
              y[1] = mlp_act(ACT, z4.y, d[1]) + x4.y;
              y[2] = mlp_act(ACT, z4.z, d[2]) + x4.z;
              y[3] = mlp_act(ACT, z4.w, d[3]) + x4.w;
              if (!last) {
                *dp = make_float4(d[0], d[1], d[2], d[3]);
              } else {
                // output layer in FP64; gradient seed g = w_out, g act' kept
#pragma unroll
                for (int j = 0; j < 4; j++) {
                  const double wo = wout_s[c + j];
                  e = fma((double)y[j], wo, e);
                  y[j] = (float)wo * d[j];
                }
              }
              *p = make_float4(y[0], y[1], y[2], y[3]);
            }
            if (last) {
              // the row's column groups in this warp, block by block
#pragma unroll
              for (int o = C::CGW / 2; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
              if (lane % C::CGW == 0) {
                double *q = ered + wc * R + i * RG + rg;
                *q = nb == 0 ? e : *q + e;
              }
            }
          }
        }
      }
      sync();
      if (lay.nbuf == 2) { float *t = hin; hin = hout; hout = t; }
      ob += nbn * NT;
      if (!last) slot += nbn * TR * 2;
    }
    for (int r = tid; r < R; r += kMlpThreads)
      if (rows_s[r] >= 0) {
        double e = ered[r];
#pragma unroll
        for (int p = 1; p < C::WC; p++) e += ered[p * R + r];
        if (Ls[L - 1].bd) e += __ldg(Ls[L - 1].bd);
        a.E[rows_s[r]] = e;
      }

    // ---------------- backward ----------------
    for (int l = L - 2; l >= 1; l--) {
      // g_{l-1} = (g_l act'_l) W_l^T, plus g_l through a residual layer
      const int kbn = mlp_cdiv(sizes[l], NT);
      const bool res = is_res(l), keep = is_res(l - 1);
      const int below = slot - kbn * TR * 2;  // layer l - 1's slots; layer l's follow
      for (int kb = 0; kb < kbn; kb++) {
        gemm(false, sizes[l + 1]);
        sync();
#pragma unroll
        for (int i = 0; i < TR; i++) {
          const int r = i * RG + rg;
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int c = col_of(kb, h), u = (kb * TR + i) * 2 + h;
            float g[4] = {acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x,
                          acc[i][2 * h + 1].y};
            if (res) {
              // layer l's own gradient: w_out for the last hidden layer, else
              // kept in its slots (their act' is spent)
              if (l == L - 2) {
#pragma unroll
                for (int j = 0; j < 4; j++) g[j] += (float)wout_s[c + j];
              } else {
                const float4 gl = dzs[(size_t)(slot + u) * kMlpThreads];
                g[0] += gl.x; g[1] += gl.y; g[2] += gl.z; g[3] += gl.w;
              }
            }
            const float4 d = dzs[(size_t)(below + u) * kMlpThreads];
            if (keep) dzs[(size_t)(below + u) * kMlpThreads] = make_float4(g[0], g[1], g[2], g[3]);
            *reinterpret_cast<float4 *>(hout + r * ldh + c) =
                make_float4(g[0] * d.x, g[1] * d.y, g[2] * d.z, g[3] * d.w);
          }
        }
      }
      sync();
      if (lay.nbuf == 2) { float *t = hin; hin = hout; hout = t; }
      slot = below;
    }
    for (int kb = 0; kb * NT < nin; kb++) {
      gemm(false, sizes[1]);
#pragma unroll
      for (int i = 0; i < TR; i++) {
        const int at = rows_s[i * RG + rg];
        if (at >= 0) {
          float *dst = a.dEdG + (size_t)at * nin;
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int c = col_of(kb, h);
            if (c < nin)  // nin is a multiple of 4
              *reinterpret_cast<float4 *>(dst + c) = make_float4(
                  acc[i][2 * h].x, acc[i][2 * h].y, acc[i][2 * h + 1].x, acc[i][2 * h + 1].y);
          }
        }
      }
    }
  }
  if (bad && a.status && lane == 0) atomicOr(a.status, kStatusTimeout);
}

template <int NT, int TR>
void mlp_plan_one(int nl, const int *sizes, int resnet, MlpPlan &p, int v) {
  using C = MlpCfg<NT, TR>;
  MlpPlan::Form &f = p.form[v];
  f.rows = C::R;
  f.smem = sizeof(float) * (size_t)mlp_lay(nl, sizes, NT, C::R, C::WC, C::S * C::kW + C::GS * C::kG).total;
  f.scratch_f4 = 0;
  for (int l = 0; l + (resnet ? 1 : 2) < nl; l++)  // the last hidden layer's input only
    f.scratch_f4 += (size_t)mlp_cdiv(sizes[l + 1], NT) * TR * 2 * kMlpThreads;
  f.ctas = 0;
  auto set = [&](auto kern) {
    cudaFuncAttributes fa{};
    if (cudaFuncGetAttributes(&fa, kern) != cudaSuccess) return;
    if (f.smem + fa.sharedSizeBytes > 227 * 1024) return;
    if (allow_dynamic_smem(kern) != cudaSuccess) return;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kMlpBlock, f.smem) ==
        cudaSuccess)
      f.ctas = occ;
  };
  switch (p.actfn) {
    case 0: set(k_mlp_fp32<NT, TR, 0>); break;
    case 1: set(k_mlp_fp32<NT, TR, 1>); break;
    case 2: set(k_mlp_fp32<NT, TR, 2>); break;
    default: set(k_mlp_fp32<NT, TR, 3>); break;
  }
}

template <int NT>
void mlp_plan_nt(int nl, const int *sizes, int resnet, MlpPlan &p) {
  mlp_plan_one<NT, 1>(nl, sizes, resnet, p, 0);
  mlp_plan_one<NT, 2>(nl, sizes, resnet, p, 1);
  mlp_plan_one<NT, 4>(nl, sizes, resnet, p, 2);
  mlp_plan_one<NT, 8>(nl, sizes, resnet, p, 3);
}

template <int NT, int TR>
void launch_mlp_act(const MlpArgs &a, cudaStream_t st) {
  switch (a.actfn) {
    case 0: k_mlp_fp32<NT, TR, 0><<<a.grid, kMlpBlock, a.smem, st>>>(a); break;
    case 1: k_mlp_fp32<NT, TR, 1><<<a.grid, kMlpBlock, a.smem, st>>>(a); break;
    case 2: k_mlp_fp32<NT, TR, 2><<<a.grid, kMlpBlock, a.smem, st>>>(a); break;
    default: k_mlp_fp32<NT, TR, 3><<<a.grid, kMlpBlock, a.smem, st>>>(a); break;
  }
}

template <int NT>
void launch_mlp_tr(const MlpArgs &a, cudaStream_t st) {
  switch (a.form) {
    case 0: launch_mlp_act<NT, 1>(a, st); break;
    case 1: launch_mlp_act<NT, 2>(a, st); break;
    case 2: launch_mlp_act<NT, 4>(a, st); break;
    default: launch_mlp_act<NT, 8>(a, st); break;
  }
}

}  // namespace tmd
