// Complex transforms of run-time lengths in shared memory, for the kernels
// whose lengths are not compiled in (gridgen.cu).
//
// A CTA holds 16 columns (or rows) in shared memory and transforms them by
// Stockham passes of the radices 2 .. 13 and 16 (in-register DFTs); G threads
// per column, the factors and G chosen per length on the host (gen_plan).
// Each pass reads one buffer and writes the other, a half-warp's 16 columns
// one 128-byte row of shared memory.
#pragma once

#include <algorithm>
#include <vector>

#include "fftcore.cuh"

namespace gtomrln {

constexpr int kGenCols = 16;
constexpr int kGenMaxFactors = 8;

struct GenFft {
  int N, G, nf;  // length, threads per column, factors
  int f[kGenMaxFactors];
};

constexpr int kGenRowPitch = kGenCols + 1;  // rows are written along x and read along rows

// One Stockham pass of radix R over the CTA's columns (pitch CP between
// element indices): with s the product of the earlier radices,
//   out[q s R + k s + k0] = sum_j in[q s + k0 + j N/R] e(-+ j k0/(s R)) e(-+ j k/R).
template <int R, bool INV, int CP>
__device__ __forceinline__ void gen_pass(const float2* in, float2* out, int N, int s, float inv_s, const float2* tw,
                                         int tscale, int g, int G, int c) {
  const int nb = N / R;
  for (int b = g; b < nb; b += G) {
    const int q = (int)(((float)b + 0.5f) * inv_s);
    const int k0 = b - q * s;
    const int step = k0 * (nb / s) * tscale;
    float2 v[R];
    v[0] = in[b * CP + c];
#pragma unroll
    for (int j = 1; j < R; j++) {
      float2 w = tw[j * step];
      if (INV) w.y = -w.y;
      v[j] = cmul(in[(b + j * nb) * CP + c], w);
    }
    dftr<R, INV>(v);
    float2* o = out + (q * s * R + k0) * CP + c;
#pragma unroll
    for (int k = 0; k < R; k++) o[k * s * CP] = v[k];
  }
}

// The transform of every column in a; b is the other buffer.  Returns the
// buffer that holds the result.  Begins and ends with a barrier.
template <bool INV, int CP>
__device__ __forceinline__ float2* gen_fft(float2* a, float2* b, const GenFft& p, const float2* tw, int tscale, int g,
                                           int c) {
  int s = 1;
  __syncthreads();
  for (int i = 0; i < p.nf; i++) {
    const int R = p.f[i];
    const float inv_s = 1.f / (float)s;
    switch (R) {
      case 2: gen_pass<2, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 3: gen_pass<3, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 4: gen_pass<4, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 5: gen_pass<5, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 6: gen_pass<6, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 7: gen_pass<7, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 8: gen_pass<8, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 9: gen_pass<9, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 10: gen_pass<10, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 11: gen_pass<11, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 12: gen_pass<12, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      case 13: gen_pass<13, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
      default: gen_pass<16, INV, CP>(a, b, p.N, s, inv_s, tw, tscale, g, p.G, c); break;
    }
    __syncthreads();
    float2* t = a;
    a = b;
    b = t;
    s *= R;
  }
  return a;
}

// Asynchronous 8-byte copy global -> shared (zeros when !in).
__device__ __forceinline__ void gen_copy8(float2* dst, const float2* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(in ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void gen_copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void gen_twiddles(float2* tw, const float2* __restrict__ twg, int P) {
  for (int m = threadIdx.x; m < P; m += blockDim.x) tw[m] = __ldg(twg + m);
}

inline size_t gen_smem(int P, int n, int pitch) { return sizeof(float2) * ((size_t)P + 2 * (size_t)n * pitch); }

// --------------------------------------------------------------- plans --
constexpr int kGenRadices[] = {16, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
constexpr int kGenMaxPrime = 13;

// The factors and threads per column of length N with the least estimated
// work: per pass, the rounds of its butterflies over G threads times what a
// round costs (two shared accesses and a twiddle per element, the DFT's
// arithmetic, the pass's barrier).  Fewer than 24 warps per SM, at `ctas`
// CTAs each, leave latency uncovered.
inline void gen_search(int rest, int maxr, std::vector<int>& cur, int N, int ctas, GenFft* best, double* best_cost) {
  if (rest == 1) {
    if ((int)cur.size() > kGenMaxFactors) return;
    for (int G = 8; G <= 32; G += 2) {
      double cost = 0;
      for (int r : cur) cost += (N / r + G - 1) / G * ((r == 11 || r == 13 ? 6.0 : 4.0) * r + 6.0) + 12.0;
      cost *= G;  // a CTA's thread-rounds: its share of the SM
      cost *= std::max(1.0, 24.0 / (ctas * G * kGenCols / 32.0));
      if (cost < *best_cost) {
        *best_cost = cost;
        best->N = N;
        best->G = G;
        best->nf = (int)cur.size();
        std::copy(cur.begin(), cur.end(), best->f);
      }
    }
    return;
  }
  for (int r : kGenRadices)
    if (r <= maxr && rest % r == 0) {
      cur.push_back(r);
      gen_search(rest / r, r, cur, N, ctas, best, best_cost);
      cur.pop_back();
    }
}

// False if N has a prime factor above kGenMaxPrime.
inline bool gen_plan(int N, size_t smem, GenFft* out) {
  std::vector<int> cur;
  double cost = 1e30;
  const int ctas = (int)std::max<size_t>(1, (227 << 10) / (smem + 1024));
  gen_search(N, 16, cur, N, ctas, out, &cost);
  return cost < 1e30;
}

inline bool gen_smooth(int n) {
  for (int p = 2; p <= kGenMaxPrime; p++)
    while (n % p == 0) n /= p;
  return n == 1;
}

}  // namespace gtomrln
