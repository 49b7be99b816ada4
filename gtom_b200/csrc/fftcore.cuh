// Complex arithmetic and small in-register DFTs shared by the gridding
// reconstructor's own FFT kernels (gridfft.cu, gridsym.cu, gridgen.cu).
#pragma once

#include <cuda_runtime.h>

namespace gtomrln {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
}
// Complex sums as one packed f32x2 instruction each (two IEEE round-to-
// nearest operations, one per component, as the scalar forms).
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  unsigned long long av, bv, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(av) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(bv) : "f"(b.x), "f"(b.y));
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(av), "l"(bv));
  float2 o;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  unsigned long long av, bv, r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(av) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(bv) : "f"(b.x), "f"(b.y));
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(av), "l"(bv));
  float2 o;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
  return o;
}
// times -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 mul_mi(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

// In-register DFT of length R, forward (exp(-2 pi i nk/R)) or inverse.
template <int R, bool INV>
__device__ __forceinline__ void dft(float2* v) {
  if (R == 2) {
    const float2 t = v[0];
    v[0] = cadd(t, v[1]);
    v[1] = csub(t, v[1]);
  } else if (R == 4) {
    const float2 a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]);
    const float2 a2 = cadd(v[1], v[3]), a3 = mul_mi<INV>(csub(v[1], v[3]));
    v[0] = cadd(a0, a2);
    v[2] = csub(a0, a2);
    v[1] = cadd(a1, a3);
    v[3] = csub(a1, a3);
  } else {  // R == 8: two DFT-4 of the even and odd elements, then W8^k
    float2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
    dft<4, INV>(e);
    dft<4, INV>(o);
    const float h = 0.70710678118654752440f;
    // W8^1, W8^2, W8^3 (forward: (1-i)/sqrt2, -i, (-1-i)/sqrt2; inverse: conjugates)
    const float2 o1 = INV ? make_float2((o[1].x - o[1].y) * h, (o[1].x + o[1].y) * h)
                          : make_float2((o[1].x + o[1].y) * h, (o[1].y - o[1].x) * h);
    const float2 o2 = mul_mi<INV>(o[2]);
    const float2 o3 = INV ? make_float2(-(o[3].x + o[3].y) * h, (o[3].x - o[3].y) * h)
                          : make_float2((o[3].y - o[3].x) * h, -(o[3].x + o[3].y) * h);
    v[0] = cadd(e[0], o[0]);
    v[4] = csub(e[0], o[0]);
    v[1] = cadd(e[1], o1);
    v[5] = csub(e[1], o1);
    v[2] = cadd(e[2], o2);
    v[6] = csub(e[2], o2);
    v[3] = cadd(e[3], o3);
    v[7] = csub(e[3], o3);
  }
}

// ---------------------------------------------- compile-time twiddles --
constexpr double kPiD = 3.14159265358979323846264338327950288;

// sin and cos by their Taylor series after reduction to [-pi, pi] (the
// remaining error is far below FP32 rounding); compile-time only.
constexpr double ce_sin(double x) {
  while (x > kPiD) x -= 2 * kPiD;
  while (x < -kPiD) x += 2 * kPiD;
  double term = x, sum = x;
  for (int k = 1; k < 20; k++) {
    term *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
    sum += term;
  }
  return sum;
}
constexpr double ce_cos(double x) { return ce_sin(x + kPiD / 2); }

// Odd prime DFT of length R in registers (R = 3 .. 13), unnormalised, forward
// (exp(-)) or inverse (exp(+)): X(k) and X(R-k) are
//   a(0) + sum over n = 1 .. (R-1)/2 of (a(n) + a(R-n)) cos(2 pi k n / R)
//   -+ i (a(n) - a(R-n)) sin(2 pi k n / R).
template <int R, bool INV>
__device__ __forceinline__ void dft_odd(float2* v) {
  float2 sp[(R - 1) / 2], sm[(R - 1) / 2];
#pragma unroll
  for (int n = 1; n <= (R - 1) / 2; n++) {
    sp[n - 1] = cadd(v[n], v[R - n]);
    sm[n - 1] = csub(v[n], v[R - n]);
  }
  const float2 v0 = v[0];
#pragma unroll
  for (int n = 0; n < (R - 1) / 2; n++) v[0] = cadd(v[0], sp[n]);
#pragma unroll
  for (int k = 1; k <= (R - 1) / 2; k++) {
    float2 re = v0, im = make_float2(0.f, 0.f);  // re: cosine part, im: sine part (before the factor -+i)
#pragma unroll
    for (int n = 1; n <= (R - 1) / 2; n++) {
      const float cs = (float)ce_cos(2 * kPiD * ((k * n) % R) / R);
      const float sn = (float)ce_sin(2 * kPiD * ((k * n) % R) / R);
      re = make_float2(fmaf(cs, sp[n - 1].x, re.x), fmaf(cs, sp[n - 1].y, re.y));
      im = make_float2(fmaf(sn, sm[n - 1].x, im.x), fmaf(sn, sm[n - 1].y, im.y));
    }
    const float2 minus = make_float2(re.x + im.y, re.y - im.x);  // re - i im
    const float2 plus = make_float2(re.x - im.y, re.y + im.x);
    v[k] = INV ? plus : minus;
    v[R - k] = INV ? minus : plus;
  }
}

// In-register DFT of length N (factors 2, 3, 5, or N = 7, 11, 13), unnormalised,
// forward (exp(-)) or inverse (exp(+)), natural order in and out: decimation
// in time by the smallest factor (2, then 3, then 5) down to the radix-8/4/2
// kernels and the odd prime kernels above, with the combining twiddles as
// constants.
template <int N, bool INV>
__device__ __forceinline__ void dftr(float2* v) {
  if constexpr (N == 1) {
    return;
  } else if constexpr (N == 2 || N == 4 || N == 8) {
    dft<N, INV>(v);
  } else if constexpr (N == 3 || N == 5 || N == 7 || N == 11 || N == 13) {
    dft_odd<N, INV>(v);
  } else {
    constexpr int R = N % 2 == 0 ? 2 : (N % 3 == 0 ? 3 : 5);
    constexpr int M = N / R;
    static_assert(M * R == N, "dftr: lengths with factors 2, 3 and 5 only");
    float2 sub[R][M];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int i = 0; i < M; i++) sub[r][i] = v[R * i + r];
#pragma unroll
    for (int r = 0; r < R; r++) dftr<M, INV>(sub[r]);
#pragma unroll
    for (int k = 0; k < M; k++) {
      float2 u[R];
#pragma unroll
      for (int r = 0; r < R; r++) {
        if (r * k == 0) {
          u[r] = sub[r][k];
        } else if (4 * r * k == N) {
          u[r] = mul_mi<INV>(sub[r][k]);  // e(-+1/4) = -+i
        } else if (8 * r * k == N || 8 * r * k == 3 * N) {
          // e(-+1/8), e(-+3/8): (1 -+ i)/sqrt2, (-1 -+ i)/sqrt2, four operations
          const float h = 0.70710678118654752440f;
          const float2 a = sub[r][k];
          const float2 p = 8 * r * k == N ? a : mul_mi<INV>(a);  // e(-+3/8) = -+i e(-+1/8)
          u[r] = INV ? make_float2((p.x - p.y) * h, (p.x + p.y) * h) : make_float2((p.x + p.y) * h, (p.y - p.x) * h);
        } else {
          const float wr = (float)ce_cos(2 * kPiD * r * k / N);
          const float wi = (float)(INV ? ce_sin(2 * kPiD * r * k / N) : -ce_sin(2 * kPiD * r * k / N));
          u[r] = cmul(sub[r][k], make_float2(wr, wi));
        }
      }
      if constexpr (R == 2) {
        dft<2, INV>(u);
      } else {
        dft_odd<R, INV>(u);
      }
#pragma unroll
      for (int q = 0; q < R; q++) v[k + M * q] = u[q];
    }
  }
}

// The pre-twiddle of a Hermitian-to-real transform of length P = 2H as an
// H-point complex transform: Z(k) = (X(k) + conj X(H-k)) + i e(sg k/P)
// (X(k) - conj X(H-k)) (sg = +1: the inverse C2R; -1: the forward sum); the
// H-point transform of the same sign then gives x(2n) = Re z(n),
// x(2n+1) = Im z(n).
template <bool PLUS>
__device__ __forceinline__ float2 c2r_pre(float2 xk, float2 xm, float2 w) {
  if (PLUS) w.y = -w.y;  // the table holds e(-k/P)
  const float2 a = make_float2(xk.x + xm.x, xk.y - xm.y);  // X(k) + conj X(H-k)
  const float2 b = make_float2(xk.x - xm.x, xk.y + xm.y);  // X(k) - conj X(H-k)
  const float2 wb = cmul(w, b);
  return make_float2(a.x - wb.y, a.y + wb.x);  // a + i wb
}

// The post-twiddle of a real-to-Hermitian transform of length P computed as
// an H-point complex transform of the packed pairs: Y(k) = (Z(k) + conj
// Z(H-k)) / 2 - (i/2) e(sg k/P) (Z(k) - conj Z(H-k)) (Z indices mod H;
// sg = -1: the forward R2C; +1: exp(+)).  Y(H) = Re Z(0) - Im Z(0).
template <bool PLUS>
__device__ __forceinline__ float2 r2c_post(float2 zk, float2 zm, float2 w) {
  if (PLUS) w.y = -w.y;
  const float2 a = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
  const float2 b = make_float2(0.5f * (zk.x - zm.x), 0.5f * (zk.y + zm.y));
  const float2 wb = cmul(w, b);
  return make_float2(a.x + wb.y, a.y - wb.x);  // a - i wb
}

}  // namespace gtomrln
