// Complex arithmetic and small DFTs in registers, for every transform of the spectral ETD kernels (sm_103a).
//
// The transforms themselves keep their points in registers: fsm_regfft.cuh (rows of up to 512 points),
// fsm_linefft.cuh (longer lines), fsm_colfft.cuh (strided columns).
//
// Sign convention: forward = exp(-2 pi i k n / N), inverse = exp(+...), both
// unnormalised (the caller folds the 1/N of torch's "backward" norm into the
// spectral arithmetic). Twiddles come from a table W_N^k = exp(-2 pi i k/N),
// k < N, computed in FP64 on the host and rounded to FP32.
#pragma once

#include <cuda_runtime.h>

namespace fsm {

// Complex sums as one packed instruction (add / sub.rn.f32x2): the transforms are mostly complex
// sums, and the kernels are bound by instruction issue or by the latency of one warp's chain. Each
// component rounds as a scalar sum does. Measured: resident 2D kernel 128^2 x 16 (convection)
// 35.2 -> 33.3 us per step, 128 x 256 (Leray) 91 -> 81; 3D Burgers 256^3 19.9 -> 19.3 ms per 4 steps.
// nvcc 13.0.88 was seen to compile packed sums wrong: a vorticity row pass with its two rows in a rolled
// loop, at the 128-register cap, gave wrong products, the same at every run, with a CTA barrier in place of the
// warp's and with the compiler's own packed intrinsics alike, and right ones with scalar sums or without the cap.
// Every kernel at the cap is therefore held against the oracle (tests/test_gpu_long_axes.py); the
// library's results with scalar sums in place of these are the same bit for bit (2264 calls over all sizes and terms).
__device__ __forceinline__ unsigned long long pack2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(r);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(r);
}
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
// i * a
__device__ __forceinline__ float2 cmuli(float2 a) { return make_float2(-a.y, a.x); }
// -i * a
__device__ __forceinline__ float2 cmulmi(float2 a) { return make_float2(a.y, -a.x); }
// a + c * b (complex)
__device__ __forceinline__ float2 cfma(float2 c, float2 b, float2 a) {
  return make_float2(fmaf(c.x, b.x, fmaf(-c.y, b.y, a.x)), fmaf(c.x, b.y, fmaf(c.y, b.x, a.y)));
}

// Programmatic dependent launch (launch_pdl): wait for the grid before this one; let the next grid in
// the stream be placed. Both do nothing in a plain launch.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// A kernel's `__restrict__` pointer parameter after pdl_wait(): loads through the parameter itself may be
// moved ahead of the wait (nothing else is taken to write that memory while the kernel runs); loads
// through the returned pointer may not. Pointers that come in a struct need no such care.
template <class T>
__device__ __forceinline__ T* pdl_ptr(T* p) {
  asm volatile("" : "+l"(p)::"memory");
  return p;
}
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <bool INV>
__device__ __forceinline__ void dft2(float2* v) {
  float2 a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2* v) {
  float2 t0 = cadd(v[0], v[2]);
  float2 t1 = csub(v[0], v[2]);
  float2 t2 = cadd(v[1], v[3]);
  float2 d = csub(v[1], v[3]);
  float2 t3 = INV ? cmuli(d) : cmulmi(d);  // W4^1 = -i (forward), +i (inverse)
  v[0] = cadd(t0, t2);
  v[2] = csub(t0, t2);
  v[1] = cadd(t1, t3);
  v[3] = csub(t1, t3);
}

template <bool INV>
__device__ __forceinline__ void dft8(float2* v) {
  const float h = 0.70710678118654752440f;
  float2 a[4], b[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    a[j] = cadd(v[j], v[j + 4]);
    b[j] = csub(v[j], v[j + 4]);
  }
  // b_j *= W8^j
  if (!INV) {
    b[1] = make_float2(h * (b[1].x + b[1].y), h * (b[1].y - b[1].x));   // (1 - i)/sqrt2
    b[2] = cmulmi(b[2]);                                                   // -i
    b[3] = make_float2(h * (b[3].y - b[3].x), -h * (b[3].x + b[3].y));   // (-1 - i)/sqrt2
  } else {
    b[1] = make_float2(h * (b[1].x - b[1].y), h * (b[1].y + b[1].x));   // (1 + i)/sqrt2
    b[2] = cmuli(b[2]);                                                    // +i
    b[3] = make_float2(-h * (b[3].x + b[3].y), h * (b[3].x - b[3].y));   // (-1 + i)/sqrt2
  }
  dft4<INV>(a);
  dft4<INV>(b);
#pragma unroll
  for (int m = 0; m < 4; ++m) {
    v[2 * m] = a[m];
    v[2 * m + 1] = b[m];
  }
}

}  // namespace fsm
