// Transforms of one line by T = N / E threads, the elements t + T j of thread t in registers on entry
// and exit: register passes (radix E first and last) with exchanges through two shared buffers in
// turn. Used by the 1D line kernel and by the last-axis transforms above 512 points.
#pragma once

#include "fsm_internal.cuh"
#include "fsm_regfft.cuh"

namespace fsm {

// E elements per thread: enough threads for four schedulers where the passes allow it, with first
// and last radix E (N / E^2 is what the passes between them combine). 128 points take 4 (a full
// warp: 0.57 us a stage) rather than 8 (half a warp: 0.88). 4096 points take 16 (three passes, 256
// threads) rather than 8 (four passes, 512 threads): fewer exchanges, fewer instructions.
template <int N>
struct LineCfg {
  static constexpr int E = N <= 128 ? 4 : (N <= 2048 ? 8 : 16);
  static constexpr int T = N / E;
  static constexpr int G = T < 32 ? 32 : T;  // threads of a sample (lanes beyond T only keep the barriers)
  static constexpr int H = N / 2 + 1;
  static constexpr int NB = N + N / 16;  // exchange buffer: one word of padding per 16
  // radix of the pass that follows span P (1: the first one)
  static constexpr int radix(int P) {
    const int rem = N / P;
    if (P == 1 || rem == E) return E;
    const int mid = rem / E;  // left for the passes before the last
    return mid >= E ? E : (mid == 16 ? 4 : (mid > 8 ? 8 : mid));
  }
  // twiddles of all passes: R x P entries of each pass with span P > 1
  static constexpr int tw_words() {
    int w = 0;
    for (int P = radix(1); P < N; P *= radix(P)) w += radix(P) * P;
    return w;
  }
  static constexpr int TW = tw_words();
  // a sample's region (float2): two exchange buffers, state and the scheme's running sums
  __host__ __device__ static constexpr size_t region(int n_aux) {
    return (size_t)2 * NB + (size_t)(1 + (n_aux > 2 ? n_aux : 2)) * H;
  }
};

__device__ __forceinline__ int line_pad(int i) { return i + (i >> 4); }

// Twiddles of every pass, [j][k] = W_{R P}^{j k} (consecutive threads read consecutive words).
template <int N, int P = LineCfg<N>::radix(1)>
__device__ __forceinline__ void line_twiddles(float2* __restrict__ dst, const float2* __restrict__ master, int tid,
                                              int nthreads) {
  if constexpr (P < N) {
    constexpr int R = LineCfg<N>::radix(P);
    for (int i = tid; i < R * P; i += nthreads) dst[i] = master[(i / P) * (i % P) * (kTwiddleMax / (R * P))];
    line_twiddles<N, P * R>(dst + R * P, master, tid, nthreads);
  }
}

// Barrier of the sample's T threads (id: the sample's sub-group in the CTA).
template <int N>
__device__ __forceinline__ void line_sync(int id) {
  if constexpr (LineCfg<N>::T <= 32) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(LineCfg<N>::T) : "memory");
}

// The passes of a transform from span P on; v holds the pass's inputs (butterfly b in v[b R ..]).
template <int N, bool INV, int P>
__device__ __forceinline__ void line_passes(float2 (&v)[LineCfg<N>::E], float2* cur,
                                            float2* nxt, const float2* __restrict__ tw, int t, int id,
                                            bool on) {
  using Cfg = LineCfg<N>;
  constexpr int E = Cfg::E, T = Cfg::T, R = Cfg::radix(P), PER = E / R;
  if (on) {
#pragma unroll
    for (int b = 0; b < PER; ++b) {
      if constexpr (P > 1) {
        const int k = (t + b * T) & (P - 1);
#pragma unroll
        for (int j = 1; j < R; ++j) {
          float2 w = tw[j * P + k];
          if (INV) w.y = -w.y;
          v[b * R + j] = cmul(v[b * R + j], w);
        }
      }
      dft_reg<R, INV>(v + b * R);
    }
  }
  if constexpr (P * R < N) {
    constexpr int RN = Cfg::radix(P * R), NBN = N / RN;
    if (on) {
#pragma unroll
      for (int b = 0; b < PER; ++b) {
        const int i = t + b * T, k = i & (P - 1);
#pragma unroll
        for (int j = 0; j < R; ++j) cur[line_pad((i - k) * R + k + j * P)] = v[b * R + j];
      }
    }
    line_sync<N>(id);
    if (on) {
#pragma unroll
      for (int b = 0; b < E / RN; ++b)
#pragma unroll
        for (int j = 0; j < RN; ++j) v[b * RN + j] = cur[line_pad(t + b * T + j * NBN)];
    }
    line_passes<N, INV, P * R>(v, nxt, cur, tw + (P > 1 ? R * P : 0), t, id, on);
  }
}

// Exchanges of one transform (which buffer the next exchange takes).
template <int N>
constexpr int line_exchanges() {
  int n = 0;
  for (int P = LineCfg<N>::radix(1); P < N; P *= LineCfg<N>::radix(P)) ++n;
  return n;
}

}  // namespace fsm
