// The symmetric gridding iteration and final map (gridsym.cu) on any even
// grid whose transforms gridsym.cu has no compiled lengths for: the same
// four passes over the Hermitian half along z of the real iterated spectrum
// and the same three cropping passes of the final map, with the transform
// length a run-time value.
//
// A CTA holds 16 columns (y and z passes: 16 consecutive x) or rows (x
// passes) in shared memory and transforms them there (genfft.cuh).
//
// What bounds it: shared memory (two to four round trips per transform) and
// HBM or L2, instead of the six strided passes per 3D transform pair, the
// real grid and the separate blob and update kernels of the cuFFT path.  Ten
// iterations and the map (cuFFT against here): P = 40 393 -> 209 us, P = 88
// 522 -> 283, P = 200 2.18 -> 0.93 ms, P = 286 10.9 -> 2.28, P = 480 26.9 ->
// 11.1, P = 720 90.5 -> 36.9.  The compiled lengths of gridsym.cu, one round
// trip per transform, are faster where they exist: P = 160 515 -> 385 us,
// P = 320 2.89 -> 2.16 ms, P = 768 45.7 -> 31.3.
#include <algorithm>
#include <cstdint>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "genfft.cuh"
#include "gridfft.cuh"

namespace gtomrln {

namespace {

// Everything a launch needs of grid P.
struct GenGrid {
  int P, H, RW;    // grid, P/2, pitch of W's rows (a multiple of four: 32 bytes)
  int r2;          // squared radius of the gridding sphere (of the mask in the final map)
  GenFft y, x;     // lengths P and H
  const float2* tw;  // e(-m/P), m < P
};

__host__ __device__ inline int gen_tiles(int H) { return (H + kGenCols - 1) / kGenCols; }

// ------------------------------------------------------------ y pass --
// Grid: (ceil(H/16) (H+1), volumes): 16 consecutive x < H at one z.  Rows
// outside the sphere are zero on the spectrum's side, as in gridsym.cu.
template <bool INV>
__global__ void __launch_bounds__(512)
gridgen_y_kernel(float2* __restrict__ W, const __grid_constant__ GenGrid gr) {
  extern __shared__ float2 smem[];
  const int P = gr.P, XT = gen_tiles(gr.H);
  float2* tw = smem;
  float2* a = smem + P;
  float2* b = a + P * kGenCols;
  const int c = threadIdx.x & (kGenCols - 1), g = threadIdx.x / kGenCols, G = gr.y.G;
  const int z = blockIdx.x / XT, x = (blockIdx.x - z * XT) * kGenCols + c;
  const bool in = x < gr.H;
  const int ylim2 = in ? gr.r2 - x * x : 0;
  auto inside = [&](int y) {
    const int yp = y < gr.H ? y : P - y;
    return yp * yp < ylim2;
  };
  float2* col = W + ((int64_t)blockIdx.y * (gr.H + 1) + z) * P * gr.RW + (in ? x : 0);
  gen_twiddles(tw, gr.tw, P);
  grid_dependency_wait();
  for (int i = g; i < P; i += G)
    gen_copy8(a + i * kGenCols + c, col + (int64_t)i * gr.RW, INV ? inside(i) : in);
  gen_copy_wait();
  const float2* r = gen_fft<INV, kGenCols>(a, b, gr.y, tw, 1, g, c);
  for (int i = g; i < P; i += G)
    if (INV ? in : inside(i)) col[(int64_t)i * gr.RW] = r[i * kGenCols + c];
}

// ------------------------------------------------------------ x pass --
// 16 consecutive rows per CTA (grid ((H+1) P / 16 rounded up, volumes)):
// C2R along x, times blob(r) / P^3, R2C along x.
__global__ void __launch_bounds__(512)
gridgen_x_kernel(float2* __restrict__ W, const __grid_constant__ GenGrid gr, const float* __restrict__ table, float inv_n,
                 float funcsampling) {
  extern __shared__ float2 smem[];
  constexpr int CP = kGenRowPitch;
  const int P = gr.P, H = gr.H, G = gr.x.G;
  float2* tw = smem;
  float2* a = smem + P;
  float2* b = a + (H + 1) * CP;
  const int c = threadIdx.x & (kGenCols - 1), g = threadIdx.x / kGenCols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int rows = (H + 1) * P, row0 = blockIdx.x * kGenCols;
  float2* base = W + ((int64_t)blockIdx.y * rows + row0) * gr.RW;
  gen_twiddles(tw, gr.tw, P);
  grid_dependency_wait();
  for (int r = warp; r < kGenCols; r += nwarps) {
    const bool in = row0 + r < rows;
    for (int x = lane; x <= H; x += 32)  // x = P/2 lies outside the sphere
      gen_copy8(a + x * CP + r, base + (in ? (int64_t)r * gr.RW + x : 0), in && x < H);
  }
  gen_copy_wait();
  __syncthreads();
  for (int k = g; k < H; k += G) {
    float2 xk = a[k * CP + c], xm = a[(H - k) * CP + c];
    if (k == 0) xk.y = 0.f;  // the x = 0 term of a C2R is real
    b[k * CP + c] = c2r_pre<true>(xk, xm, tw[k]);
  }
  float2* v = gen_fft<true, CP>(b, a, gr.x, tw, 2, g, c);
  {
    const int rg = row0 + c, z = rg / P, y = rg - z * P;
    const int zp = z < H ? z : z - P, yp = y < H ? y : y - P;
    const float cyz = (float)(yp * yp + zp * zp);
    // element n of the packed pairs is (x = 2n, x = 2n + 1); x and P - x have
    // the same radius, bit for bit: one blob value for 2n and P - 2n (element
    // H - n), one for 2n + 1 and P - 2n - 1 (element H - 1 - n)
    auto blob = [&](int x) {
      const float xp = (float)(x < H ? x : x - P);
      return __ldg(table + grid_blob_index_sq(xp * xp + cyz, (float)P, funcsampling));
    };
    for (int n = g; 2 * n <= H; n += G) {
      const float b0 = blob(2 * n), b1 = blob(2 * n + 1);
      const int m0 = H - n, m1 = H - 1 - n;
      v[n * CP + c].x = v[n * CP + c].x * inv_n * b0;
      if (n > 0 && m0 != n) v[m0 * CP + c].x = v[m0 * CP + c].x * inv_n * b0;
      if (n <= m1) v[n * CP + c].y = v[n * CP + c].y * inv_n * b1;
      if (n < m1) v[m1 * CP + c].y = v[m1 * CP + c].y * inv_n * b1;
    }
  }
  float2* o = v == a ? b : a;
  const float2* r = gen_fft<false, CP>(v, o, gr.x, tw, 2, g, c);
  o = r == a ? b : a;
  for (int k = g; k < H; k += G)
    o[k * CP + c] = r2c_post<false>(r[k * CP + c], r[(k == 0 ? 0 : H - k) * CP + c], tw[k]);
  __syncthreads();
  for (int rr = warp; rr < kGenCols; rr += nwarps) {
    if (row0 + rr >= rows) break;
    for (int x = lane; x < H; x += 32) base[(int64_t)rr * gr.RW + x] = o[x * CP + rr];
  }
}

// ------------------------------------------------------------ z pass --
// gridsym_z_kernel's steps.  Grid: (ceil(H/16) P, volumes): 16 consecutive
// x < H at one y.
template <bool ITER, bool MOM>
__global__ void __launch_bounds__(512)
gridgen_z_kernel(float2* __restrict__ W, const float* __restrict__ Fw, float* __restrict__ Fnw, float* __restrict__ V,
                 const __grid_constant__ GenGrid gr, float beta, int write_next, double* __restrict__ change,
                 const float* __restrict__ ref) {
  extern __shared__ float2 smem[];
  constexpr int CP = kGenCols;
  const int P = gr.P, H = gr.H, R = H + 1, G = gr.x.G, XT = gen_tiles(H);
  float2* tw = smem;
  float2* a = smem + P;
  float2* b = a + (H + 1) * CP;
  const int c = threadIdx.x & (kGenCols - 1), g = threadIdx.x / kGenCols;
  const int y = blockIdx.x / XT, x0 = (blockIdx.x - y * XT) * kGenCols;
  const int yp = y < H ? y : P - y;
  if (x0 * x0 + yp * yp >= gr.r2) return;  // the whole tile is outside the circle
  const int zlim2 = gr.r2 - (x0 + c) * (x0 + c) - yp * yp;
  const bool in = x0 + c < H && zlim2 > 0;
  const int x = in ? x0 + c : 0;
  const int64_t EW = (int64_t)P * gr.RW, ES = (int64_t)P * R;
  float2* wc = W + (int64_t)blockIdx.y * (H + 1) * EW + (int64_t)y * gr.RW + x;
  const int64_t wo = (int64_t)blockIdx.y * P * ES + (int64_t)y * R + x;
  float2* v = a;
  gen_twiddles(tw, gr.tw, P);
  grid_dependency_wait();
  if (ITER) {
    for (int k = g; k <= H; k += G) gen_copy8(a + k * CP + c, wc + k * EW, in);
    // the tile's weights are asked for now and read after the first transform
    const int zlim0 = gr.r2 - x0 * x0 - yp * yp, last = min(kGenCols, H - x0) - 1;
    for (int z = threadIdx.x; z < P; z += blockDim.x) {
      const int zp = z < H ? z : P - z;
      if (zp * zp < zlim0) {
        const int64_t gi = (int64_t)blockIdx.y * P * ES + (int64_t)y * R + x0 + (int64_t)z * ES;
        grid_prefetch(Fw + gi);
        grid_prefetch(Fw + gi + last);
        grid_prefetch(Fnw + gi);
        grid_prefetch(Fnw + gi + last);
      }
    }
    gen_copy_wait();
    __syncthreads();
    for (int k = g; k < H; k += G) {
      float2 xk = a[k * CP + c], xm = a[(H - k) * CP + c];
      if (k == 0) xk.y = xm.y = 0.f;  // the z = 0 and z = P/2 terms of a Hermitian column are real
      b[k * CP + c] = c2r_pre<false>(xk, xm, tw[k]);
    }
    v = gen_fft<false, CP>(b, a, gr.x, tw, 2, g, c);
  }
  double d2 = 0, o2 = 0, r2 = 0, q2 = 0;
  const bool dist = ITER && change && ref;
  auto inside = [&](int z) {
    const int zp = z < H ? z : P - z;
    return in && zp * zp < zlim2;
  };
#pragma unroll 4
  for (int n = g; n < H; n += G) {
    float2 e = ITER ? v[n * CP + c] : make_float2(0.f, 0.f);
    float fw[2], old[2], vv[2], sv[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t gi = wo + (int64_t)(2 * n + h) * ES;
      const bool on = inside(2 * n + h);
      fw[h] = on ? __ldg(Fw + gi) : 0.f;
      old[h] = on && (ITER || !MOM) ? Fnw[gi] : 0.f;
      vv[h] = on && MOM ? V[gi] : 0.f;
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int64_t gi = wo + (int64_t)(2 * n + h) * ES;
      const bool on = inside(2 * n + h);
      float next;
      if (ITER) {
        const float cval = h ? e.y : e.x;
        float nw;
        if (MOM) {
          grid_update_momentum_value(cval, old[h], vv[h], beta, nw, next);
          if (on) V[gi] = next;
        } else {
          nw = grid_update_value(cval, old[h]);
          next = nw;
        }
        if (on) Fnw[gi] = nw;
        if (change && on) {
          const double d = (double)fw[h] * ((double)nw - (double)old[h]), q = (double)fw[h] * (double)old[h];
          d2 += d * d;
          o2 += q * q;
          if (dist) {
            const double rf = (double)__ldg(ref + gi);
            const double dr = (double)fw[h] * ((double)nw - rf), qr = (double)fw[h] * rf;
            r2 += dr * dr;
            q2 += qr * qr;
          }
        }
      } else {
        next = MOM ? vv[h] : old[h];
      }
      sv[h] = fw[h] * next;
    }
    v[n * CP + c] = make_float2(sv[0], sv[1]);
  }
  if (ITER && change) {
    grid_change_reduce(d2, o2, change);
    if (ref) {
      __syncthreads();  // grid_change_reduce's shared scratch is reused
      grid_change_reduce(r2, q2, change + 2);
    }
  }
  if (ITER && !write_next) return;  // uniform
  float2* o = v == a ? b : a;
  const float2* r = gen_fft<true, CP>(v, o, gr.x, tw, 2, g, c);
  if (in)
    for (int k = g; k <= H; k += G) {
      const float2 zk = r[(k < H ? k : 0) * CP + c], zm = r[(k == 0 || k == H ? 0 : H - k) * CP + c];
      wc[k * EW] = k < H ? r2c_post<true>(zk, zm, tw[k]) : make_float2(zk.x - zk.y, 0.f);
    }
}

// -------------------------------------------------------- final map --
// The three cropping passes of gridsym.cu: T is (P/2+1) x P x ori, [zc][y][x].
__global__ void __launch_bounds__(512)
gridgen_final_z_kernel(float2* __restrict__ T, const __grid_constant__ GridFinalArgs f,
                       const __grid_constant__ GenGrid gr) {
  extern __shared__ float2 smem[];
  constexpr int CP = kGenCols;
  const int P = gr.P, H = gr.H, R = H + 1, G = gr.y.G, XT = gen_tiles(H);
  float2* tw = smem;
  float2* a = smem + P;
  float2* b = a + P * CP;
  const int c = threadIdx.x & (kGenCols - 1), g = threadIdx.x / kGenCols;
  const int y = blockIdx.x / XT, x0 = (blockIdx.x - y * XT) * kGenCols;
  const int yp = y < H ? y : P - y;
  const int zlim2 = gr.r2 - (x0 + c) * (x0 + c) - yp * yp;
  const bool in = x0 + c < H && zlim2 > 0;
  const int x = in ? x0 + c : 0;
  const int64_t vol = blockIdx.y, NC = (int64_t)R * P * P;
  // data outside the sphere must be finite, as in gridsym_final_z_kernel
  // (columns x <= P/2; where the column is inside the circle they are part of
  // it; x = P/2 is the thread's after the last one's)
  grid_dependency_wait();  // the flag's zero is the predecessor's where no iteration ran
  const GridColumn col(f, vol, P, x0 + c, y), rim(f, vol, P, H, y);
  const bool out = x0 + c <= H && !in, last = H % kGenCols == 0 && x0 + kGenCols == H && c == 0;
  if (out || last) {
    float p = 0.f;
#pragma unroll 4
    for (int z = g; z < P; z += G) {
      if (out) p += col.zero(z);
      if (last) p += rim.zero(z);
    }
    if (p != 0.f) f.Fnw[vol * NC + H] = p;
  }
  if (x0 * x0 + yp * yp >= gr.r2) return;  // outside the mask's circle: read as zero by the y pass
  const float* wcol = (f.divide ? f.Fw : f.Fnw) + vol * NC + (int64_t)y * R + x;
  gen_twiddles(tw, gr.tw, P);
#pragma unroll 8
  for (int z = g; z < P; z += G) {
    const int zp = z < H ? z : P - z;
    const bool on = in && zp * zp < zlim2;
    const float2 v = in ? col.value(z) : make_float2(0.f, 0.f);
    const float w = on ? __ldg(wcol + (int64_t)z * (P * R)) : 0.f;
    a[z * CP + c] = grid_final_apply(v, w, P, x, y, z, f.divide != 0);
  }
  const float2* r = gen_fft<true, CP>(a, b, gr.y, tw, 1, g, c);
  float2* tv = T + vol * ((int64_t)R * P * f.ori);
  if (in)
    for (int zc = g; zc < f.ori; zc += G) tv[((int64_t)zc * P + y) * R + x] = r[(zc + f.off) * CP + c];
}

__global__ void __launch_bounds__(512)
gridgen_final_y_kernel(float2* __restrict__ T, int ori, int off, const __grid_constant__ GenGrid gr) {
  extern __shared__ float2 smem[];
  constexpr int CP = kGenCols;
  const int P = gr.P, R = gr.H + 1, G = gr.y.G, XT = gen_tiles(gr.H);
  float2* tw = smem;
  float2* a = smem + P;
  float2* b = a + P * CP;
  const int c = threadIdx.x & (kGenCols - 1), g = threadIdx.x / kGenCols;
  const int zc = blockIdx.x / XT, x = (blockIdx.x - zc * XT) * kGenCols + c;
  const bool in = x < gr.H;
  const int ylim2 = in ? gr.r2 - x * x : 0;
  float2* col = T + ((int64_t)blockIdx.y * ori + zc) * P * R + (in ? x : 0);
  gen_twiddles(tw, gr.tw, P);
  grid_dependency_wait();
  for (int i = g; i < P; i += G) {
    const int yp = i < gr.H ? i : P - i;
    gen_copy8(a + i * CP + c, col + (int64_t)i * R, yp * yp < ylim2);
  }
  gen_copy_wait();
  const float2* r = gen_fft<true, CP>(a, b, gr.y, tw, 1, g, c);
  if (in)
    for (int yc = g; yc < ori; yc += G) col[(int64_t)yc * R] = r[(yc + off) * CP + c];
}

__global__ void __launch_bounds__(512)
gridgen_final_x_kernel(const float2* __restrict__ T, const __grid_constant__ GridFinalArgs f,
                       const __grid_constant__ GenGrid gr) {
  extern __shared__ float2 smem[];
  constexpr int CP = kGenRowPitch;
  const int P = gr.P, H = gr.H, R = H + 1, G = gr.x.G, ori = f.ori;
  float2* tw = smem;
  float2* a = smem + P;
  float2* b = a + (H + 1) * CP;
  const int c = threadIdx.x & (kGenCols - 1), g = threadIdx.x / kGenCols;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int64_t vol = blockIdx.y, rows = (int64_t)ori * ori, row0 = (int64_t)blockIdx.x * kGenCols;
  const float2* tv = T + vol * ((int64_t)R * P * ori);
  gen_twiddles(tw, gr.tw, P);
  grid_dependency_wait();
  for (int r = warp; r < kGenCols; r += nwarps) {
    const bool in = row0 + r < rows;
    const int zc = in ? (int)((row0 + r) / ori) : 0, yc = in ? (int)(row0 + r - (int64_t)zc * ori) : 0;
    const float2* src = tv + ((int64_t)zc * P + yc) * R;
    for (int x = lane; x <= H; x += 32) gen_copy8(a + x * CP + r, src + x, in && x < H);
  }
  gen_copy_wait();
  __syncthreads();
  for (int k = g; k < H; k += G) {
    float2 xk = a[k * CP + c], xm = a[(H - k) * CP + c];
    if (k == 0) xk.y = 0.f;
    b[k * CP + c] = c2r_pre<true>(xk, xm, tw[k]);
  }
  const float2* v = gen_fft<true, CP>(b, a, gr.x, tw, 2, g, c);
  float* out = f.outs ? f.outs[vol] : f.out;
  const bool bad = f.Fnw[vol * ((int64_t)R * P * P) + H] != 0.f;  // data outside the sphere are not finite
  for (int r = warp; r < kGenCols; r += nwarps) {
    if (row0 + r >= rows) break;
    const int zc = (int)((row0 + r) / ori), yc = (int)(row0 + r - (int64_t)zc * ori);
    for (int xc = lane; xc < ori; xc += 32) {
      const int x = xc + f.off;
      const float2 e = v[(x >> 1) * CP + r];
      out[(row0 + r) * ori + xc] = bad ? __int_as_float(0x7fc00000)
                                       : grid_crop_value((x & 1) ? e.y : e.x, xc, yc, zc, ori, P, f.scale);
    }
  }
}

constexpr int kGenMinP = 16, kGenMaxP = 768;

int gen_grid(int P, int r2, GenGrid* gr) {
  gr->P = P;
  gr->r2 = r2;
  gr->H = P / 2;
  gr->RW = (P / 2 + 1 + 3) & ~3;
  if (!gen_plan(P, gen_smem(P, P, kGenCols), &gr->y) ||
      !gen_plan(P / 2, gen_smem(P, P / 2 + 1, kGenRowPitch), &gr->x))
    return set_error(GTOMRLN_ERR_INVALID, "gridgen: unsupported grid %d", P);
  return fft_twiddles(P, &gr->tw);
}

// Shared-memory limits of the kernels, per (device, context): set once, to
// the device's opt-in maximum.
std::mutex g_gen_mutex;
std::map<std::pair<int, unsigned long long>, bool> g_gen_done;

int gen_attributes() {
  int dev = 0;
  GTOMRLN_CUDA_TRY(cudaGetDevice(&dev));
  const auto key = std::make_pair(dev, context_id());
  std::lock_guard<std::mutex> lock(g_gen_mutex);
  if (g_gen_done.count(key)) return GTOMRLN_OK;
  const int most = (int)gen_smem(kGenMaxP, kGenMaxP, kGenCols);
  const void* kernels[] = {(const void*)gridgen_y_kernel<true>,          (const void*)gridgen_y_kernel<false>,
                           (const void*)gridgen_x_kernel,                (const void*)gridgen_z_kernel<true, true>,
                           (const void*)gridgen_z_kernel<true, false>,   (const void*)gridgen_z_kernel<false, true>,
                           (const void*)gridgen_z_kernel<false, false>,  (const void*)gridgen_final_z_kernel,
                           (const void*)gridgen_final_y_kernel,          (const void*)gridgen_final_x_kernel};
  for (const void* k : kernels)
    GTOMRLN_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
  g_gen_done[key] = true;
  return GTOMRLN_OK;
}

}  // namespace

// Even grids within shared memory of prime factors that run in registers.
// (Larger primes as direct sums lost to cuFFT below P = 132, 0.59 to 0.93 of
// its speed, and ran about level with it above.)
bool gridgen_available(int P) {
  return P >= kGenMinP && P <= kGenMaxP && P % 2 == 0 && gen_smooth(P);
}

int gridgen_prepare(int P) {
  int st = gen_attributes();
  if (st) return st;
  GenGrid gr;
  return gen_grid(P, 0, &gr);
}

int gridgen_first(float2* W, const GridGeom& geom, int count, const float* Fw, float* Fnw, float* V,
                  cudaStream_t stream) {
  const int P = geom.P;
  GenGrid gr;
  int st = gen_attributes();
  if (!st) st = gen_grid(P, geom.maskr2, &gr);
  if (st) return st;
  const dim3 grid((unsigned)(gen_tiles(gr.H) * P), count);
  const size_t smem = gen_smem(P, gr.H + 1, kGenCols);
  if (V)
    launch_dependent(gridgen_z_kernel<false, true>, grid, kGenCols * gr.x.G, smem, stream,
                   W, Fw, Fnw, V, gr, 0.f, 1, nullptr, nullptr);
  else
    launch_dependent(gridgen_z_kernel<false, false>, grid, kGenCols * gr.x.G, smem, stream,
                   W, Fw, Fnw, V, gr, 0.f, 1, nullptr, nullptr);
  GTOMRLN_LAUNCH_CHECK("gridgen_z_kernel (first)");
  return GTOMRLN_OK;
}

int gridgen_iteration(float2* W, const GridGeom& geom, int count, const float* table, const float* Fw, float* Fnw,
                      float* V, float beta, bool write_next, double* change, const float* ref, cudaStream_t stream) {
  const int P = geom.P;
  GenGrid gr;
  int st = gen_attributes();
  if (!st) st = gen_grid(P, geom.maskr2, &gr);
  if (st) return st;
  const unsigned xt = gen_tiles(gr.H);
  const dim3 gy(xt * (gr.H + 1), count), gz(xt * P, count);
  const dim3 gx((unsigned)(((gr.H + 1) * P + kGenCols - 1) / kGenCols), count);
  const size_t sy = gen_smem(P, P, kGenCols), sx = gen_smem(P, gr.H + 1, kGenRowPitch),
               sz = gen_smem(P, gr.H + 1, kGenCols);
  const int ty = kGenCols * gr.y.G, tx = kGenCols * gr.x.G;
  launch_dependent(gridgen_y_kernel<true>, gy, ty, sy, stream,
                   W, gr);
  launch_dependent(gridgen_x_kernel, gx, tx, sx, stream,
                   W, gr, table, 1.0f / ((float)P * (float)P * (float)P), (float)(0.5 / kBlobSamples));
  launch_dependent(gridgen_y_kernel<false>, gy, ty, sy, stream,
                   W, gr);
  if (V)
    launch_dependent(gridgen_z_kernel<true, true>, gz, tx, sz, stream,
                   W, Fw, Fnw, V, gr, beta, write_next, change, ref);
  else
    launch_dependent(gridgen_z_kernel<true, false>, gz, tx, sz, stream,
                   W, Fw, Fnw, V, gr, beta, write_next, change, ref);
  GTOMRLN_LAUNCH_CHECK("the gridgen iteration");
  return GTOMRLN_OK;
}

int gridgen_final(float2* T, int P, int count, const GridFinalArgs& f, cudaStream_t stream) {
  GenGrid gr;
  int st = gen_attributes();
  if (!st) st = gen_grid(P, P / 2 * (P / 2), &gr);
  if (st) return st;
  const unsigned xt = gen_tiles(gr.H);
  const size_t sy = gen_smem(P, P, kGenCols), sx = gen_smem(P, gr.H + 1, kGenRowPitch);
  const int ty = kGenCols * gr.y.G, tx = kGenCols * gr.x.G;
  launch_dependent(gridgen_final_z_kernel, dim3(xt * P, count), ty, sy, stream,
                   T, f, gr);
  launch_dependent(gridgen_final_y_kernel, dim3(xt * f.ori, count), ty, sy, stream,
                   T, f.ori, f.off, gr);
  launch_dependent(gridgen_final_x_kernel, dim3((unsigned)(((int64_t)f.ori * f.ori + kGenCols - 1) / kGenCols), count), tx, sx, stream,
                   T, f, gr);
  GTOMRLN_LAUNCH_CHECK("the gridgen final map");
  return GTOMRLN_OK;
}

// Forgets the launch attributes set on device dev.
int release_gridgen_caches(int dev, unsigned long long /*ctx*/) {
  std::lock_guard<std::mutex> lock(g_gen_mutex);
  for (auto it = g_gen_done.begin(); it != g_gen_done.end();) {
    if (it->first.first == dev) it = g_gen_done.erase(it);
    else ++it;
  }
  return GTOMRLN_OK;
}

}  // namespace gtomrln
