// Transforms along a strided axis by 256 threads: W = 256 / T adjacent columns per CTA, a warp's lanes
// on adjacent columns (fsm_plane_reg.cuh's column pass, fsm_volume.cu).
#pragma once

#include "fsm_internal.cuh"
#include "fsm_regfft.cuh"

namespace fsm {

template <int NX>
struct ColCfg {
  using RS = RegShape<NX>;
  static constexpr int T = RS::T;
  static constexpr int E = RS::E;
  static constexpr int W = 256 / T;  // columns of a CTA
  // words of an exchange buffer (512 points: one row of padding per 16)
  static constexpr int XB = (NX == 512 ? 512 + 32 : E * T) * W;
  // shared memory (float2): twiddles, kx, two exchange buffers
  static constexpr int WORDS = NX + NX / 2 + 2 * XB;
};

// x transform of a CTA's W columns: thread (t, g) = threadIdx / W, threadIdx % W holds rows t + T j of
// column g in registers on entry and exit (fsm_regfft.cuh's passes). The lanes of a warp are adjacent
// columns, so that global loads and stores of those registers are coalesced as they are, and so are
// the exchange's accesses to shared memory; the price is a CTA barrier per exchange, one each with
// two buffers in turn (par selects the next).
template <int NX, bool INV>
__device__ __forceinline__ void col_fft(float2 (&v)[RegShape<NX>::E], float2* buf, int& par,
                                        const float2* __restrict__ twt, int t, int g) {
  using Cfg = ColCfg<NX>;
  constexpr int T = Cfg::T, E = Cfg::E, W = Cfg::W;
  auto tw = [&](float2 a, float2 w) {
    if (INV) w.y = -w.y;
    return cmul(a, w);
  };
  float2* x = buf + par * Cfg::XB + g;
  par ^= 1;
  if constexpr (NX == 512) {
    auto pad = [](int i) { return (i + (i >> 4)) * W; };
    float2* y = buf + par * Cfg::XB + g;
    par ^= 1;
    dft16<INV>(v);
#pragma unroll
    for (int j = 0; j < 16; ++j) x[(17 * t + j) * W] = v[j];
    __syncthreads();
    const int k2 = t & 15;
    const float2 w2 = twt[k2];
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      v[2 * b] = x[pad(t + 32 * b)];
      v[2 * b + 1] = tw(x[pad(t + 32 * b + 256)], w2);
      dft2<INV>(v + 2 * b);
    }
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const int base = (t + 32 * b - k2) * 2 + k2;
      y[pad(base)] = v[2 * b];
      y[pad(base + 16)] = v[2 * b + 1];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v[j] = y[pad(t + 32 * j)];
      if (j > 0) v[j] = tw(v[j], twt[16 + 32 * (j - 1) + t]);
    }
    dft16<INV>(v);
  } else {
    constexpr int PER = E / T;
    dft_reg<E, INV>(v);
#pragma unroll
    for (int m = 1; m < E; ++m) v[m] = tw(v[m], twt[m * T + t]);
#pragma unroll
    for (int m = 0; m < E; ++m) x[(m * T + t) * W] = v[m];
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int m = t + p * T;
      float2 w[T];
#pragma unroll
      for (int tt = 0; tt < T; ++tt) w[tt] = x[(m * T + tt) * W];
      dft_reg<T, INV>(w);
#pragma unroll
      for (int k = 0; k < T; ++k) v[p + PER * k] = w[k];
    }
  }
}

}  // namespace fsm
