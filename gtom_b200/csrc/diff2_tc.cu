// Dense squared differences and cross-correlations on the tensor cores.
//
//   diff2[p][r][s] = 0.5 sum_i w_i |c_pi ref_ri - part_pi shift_si|^2
//                  = 0.5 (A_pr + B_ps) - C_prs,
// with a = sqrt(w) c ref, b = sqrt(w) part shift, A = sum |a|^2, B = sum |b|^2
// and C = sum Re(a conj b): per particle a real matrix product over 2 x
// elements terms (real and imaginary parts), which runs as tcgen05.mma
// (kind::tf32, FP32 accumulators in tensor memory).
//
// Precision.  Every operand is split exactly into hi (rounded to 11 bits) and
// lo (the rest, of either sign, of which the instruction keeps 11 bits), and
// hi hi + hi lo + lo hi is accumulated: 22 bits of each product.  The tensor
// core's own additions truncate, so hi hi is added to FP32 sums in registers
// with round-to-nearest every 32 elements (8 steps); the cross terms, 2^-11 of
// it, have one accumulator for the whole range.  A and B are FP32 sums of a
// thread's terms of the range, then of its eight lanes; ranges and the final
// combination are summed in double.
//
// The expansion cancels where a and b are close, so a tile of outputs with
// any diff2 below half of (A + B) / 2 (or not finite) is computed again by
// the direct kernel (estep.cu), whose FP32 sums of |a - b|^2 do not cancel.
// Relative error (rms) against 64 bits by diff2 / ((A + B) / 2), direct and
// here, at 544 elements, the shortest sums but the least favourable (at 8 320
// the direct kernel's are 1.1e-6 throughout, at 33 024 4e-6):
//   0.97: 2.5e-7, 0.4e-7   0.67: 2.3e-7, 1.0e-7   0.50: 2.6e-7, 1.7e-7
//   0.33: 2.4e-7, 4.3e-7 (and so redone); cross-correlations of the operands'
//   power: 0.73 of the largest: 2.4e-7, 1.4e-7.
// (Parts by truncation, drained every 64 elements: 0.50: 6.0e-7.  Drained
// every 16 elements: 1.0e-7, but 349 instead of 300 us below.)  In
// single-particle data the noise alone keeps diff2 near (A + B) / 2; data
// whose matches explain more than half of the power pay for both kernels.
//
// One CTA: 128 references x 64 shifts of one particle over a range of
// elements (split so that every SM has two CTAs' work).  Its 256 threads
// form the operands of 16 elements at a time in shared memory (128-byte
// swizzled rows, hi and lo, 48 KB a stage, two stages), one thread issues
// the 12 matrix instructions of a stage, and a commit on the stage's
// mbarrier frees it.  Two hi hi accumulators in tensor memory alternate, so
// one is drained while the other is filled.
//
// 16 particles x 600 references x 49 shifts at 128^2: 1.54 ms by the direct
// kernel (bound by its FP32 instructions), 0.30 ms here (bound by the
// instructions that form and split the operands).
#include <algorithm>
#include <cstdint>

#include "common.cuh"
#include "diff2_tc.cuh"

namespace gtomrln {

namespace {

constexpr int kM = 128, kN = 64, kE = 16;  // references, shifts, elements per stage
constexpr int kThreads = 256;
constexpr int kGroup = 2;  // stages per hi hi accumulator
constexpr unsigned kABytes = kM * kE * 8, kBBytes = kN * kE * 8;  // one of hi, lo
constexpr unsigned kStageBytes = 2 * (kABytes + kBBytes);
constexpr unsigned kCross = 2 * kN;     // column of the cross terms, after the two hi hi accumulators
constexpr unsigned kTmemCols = 4 * kN;  // (a power of two)
constexpr size_t kSmem = 1024 + 2 * kStageBytes;
constexpr unsigned long long kWaitNs = 1000000000ull;  // 1 s
constexpr float kCloseFraction = 0.5f;

// kind::tf32, FP32 accumulators, both operands K-major, 128 x 64.
constexpr unsigned kIdesc = (1u << 4) | (2u << 7) | (2u << 10) | ((kN / 8) << 17) | ((kM / 16) << 24);

// The last of `issued` chunks (more than s) in stage s; chunk t is in stage
// t & 1, as that stage's phase t >> 1.
__host__ __device__ constexpr int last_chunk(int issued, int s) { return issued - 1 - ((issued - 1 - s) & 1); }
static_assert(last_chunk(1, 0) == 0 && last_chunk(2, 0) == 0 && last_chunk(2, 1) == 1 && last_chunk(5, 0) == 4 &&
                  last_chunk(5, 1) == 3 && last_chunk(6, 0) == 4 && last_chunk(6, 1) == 5,
              "last_chunk: the latest chunk of the stage");

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory descriptor of a K-major tile of 128-byte swizzled rows
// (eight rows per 1024 bytes).
__device__ __forceinline__ unsigned long long tile_desc(unsigned addr) {
  return (unsigned long long)((addr >> 4) & 0x3fffu) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mma_tf32(unsigned d, unsigned long long a, unsigned long long b, unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(kIdesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// False if the phase has not completed after kWaitNs.
__device__ __forceinline__ bool bar_wait(unsigned bar, unsigned parity) {
  if (bar_try(bar, parity)) return true;
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
  for (;;) {
    if (bar_try(bar, parity)) return true;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    if (t - t0 > kWaitNs) return false;
  }
}
__device__ __forceinline__ void tmem_load32(unsigned addr, float* v) {
  unsigned r[32];
  // one statement: nothing may read the registers before the wait
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 32; i++) v[i] += __uint_as_float(r[i]);
}

// Splits v into its value rounded to 11 bits and the exact rest (NaN where the
// rounding overflows).
__device__ __forceinline__ void split4(float4 v, float4& hi, float4& lo) {
  auto top = [](float x) { return __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u); };
  hi = make_float4(top(v.x), top(v.y), top(v.z), top(v.w));
  lo = make_float4(v.x - hi.x, v.y - hi.y, v.z - hi.z, v.w - hi.w);
}

// Two consecutive complex elements, of which `left` exist.
__device__ __forceinline__ float4 load2(const float2* __restrict__ p, int64_t left) {
  const float2 a = left > 0 ? __ldg(p) : make_float2(0.f, 0.f);
  const float2 b = left > 1 ? __ldg(p + 1) : make_float2(0.f, 0.f);
  return make_float4(a.x, a.y, b.x, b.y);
}

struct TcArgs {
  const float2* particle;
  const float* minvsigma2;
  const float* ctf;
  int64_t elements;
  const float2* shifts;
  const float2* refs;
  unsigned nparticles, nrefs, nshifts;
  int mtiles, ntiles, splits, cc, vec;
  float2* ps;   // sqrt(w) particle, as particle
  float* cs;    // sqrt(w) ctf: [particle][element]
  float* part;  // C: [split][particle][ref][shift]
  float* sa;    // A: [split][particle][ref]
  float* sb;    // B: [split][particle][shift]
};

// The per-particle factors of the operands (sqrt(w) = 1 for the
// cross-correlation).
__global__ void __launch_bounds__(256) diff2_tc_scale_kernel(const TcArgs a) {
  const int64_t n = a.elements * a.nparticles;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float w = a.cc || !a.minvsigma2 ? 1.f : sqrtf(__ldg(a.minvsigma2 + i % a.elements));
    const float2 v = __ldg(a.particle + i);
    a.ps[i] = make_float2(v.x * w, v.y * w);
    a.cs[i] = (a.ctf ? __ldg(a.ctf + i) : 1.f) * w;
  }
}

__global__ void __launch_bounds__(kThreads, 2) diff2_tc_kernel(const TcArgs a) {
  extern __shared__ unsigned char raw[];
  __shared__ unsigned long long bars[2];
  __shared__ unsigned tmem_s;
  const unsigned base = (smem_u32(raw) + 1023u) & ~1023u;
  unsigned char* stage0 = raw + (base - smem_u32(raw));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  unsigned b = blockIdx.x;
  const int split = b % a.splits;
  b /= a.splits;
  const int nt = b % a.ntiles;
  b /= a.ntiles;
  const int mt = b % a.mtiles;
  const unsigned p = b / a.mtiles;
  const unsigned r0 = mt * kM, s0 = nt * kN;
  const int64_t chunks = (a.elements + kE - 1) / kE;
  const int64_t c0 = chunks * split / a.splits, c1 = chunks * (split + 1) / a.splits;
  const int nch = (int)(c1 - c0);
  const int64_t end = a.elements;

  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[0])) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[1])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_s)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem = tmem_s;
  grid_dependency_wait();

  // thread -> 16-byte unit j (two elements) of rows row0 + 32 k
  const int j = tid & 7, row0 = tid >> 3;
  const unsigned swz = (unsigned)((j ^ (row0 & 7)) << 4) + (unsigned)(row0 & 7) * 128 + (unsigned)(row0 >> 3) * 1024;
  const float2* pp = a.ps + a.elements * p;
  const float* cp = a.cs + a.elements * p;
  float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[2] = {0.f, 0.f};
  float acc[32];
#pragma unroll
  for (int i = 0; i < 32; i++) acc[i] = 0.f;

  struct Raw {  // the raw operands of a chunk
    float4 rv[4], sv[2], pv;
    float cs[2];
  };
  // the thread's places in its first rows, and which of its rows exist
  const int64_t at0 = c0 * kE + 2 * j, pitch = 32 * a.elements;
  const float2* rrow = a.refs + a.elements * (r0 + row0) + at0;
  const float2* srow = a.shifts + a.elements * (s0 + row0) + at0;
  const float2* prow = pp + at0;
  const float* crow = cp + at0;
  const int nr = r0 + row0 < a.nrefs ? min(4u, (a.nrefs - r0 - row0 + 31) / 32) : 0;
  const int ns = s0 + row0 < a.nshifts ? min(2u, (a.nshifts - s0 - row0 + 31) / 32) : 0;
  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  auto fetch = [&](Raw& q, int t) {
    const int i = t * kE;
    if (a.vec && (c0 + t + 1) * kE <= end) {  // a whole chunk of 16-byte aligned rows
      auto load = [&](const float2* p4) { return __ldg(reinterpret_cast<const float4*>(p4 + i)); };
#pragma unroll
      for (int k = 0; k < 4; k++) q.rv[k] = k < nr ? load(rrow + k * pitch) : zero4;
#pragma unroll
      for (int k = 0; k < 2; k++) q.sv[k] = k < ns ? load(srow + k * pitch) : zero4;
      q.pv = load(prow);
      const float2 cv = __ldg(reinterpret_cast<const float2*>(crow + i));
      q.cs[0] = cv.x;
      q.cs[1] = cv.y;
    } else {
      const int64_t left = end - at0 - i;  // elements from this thread's first on
#pragma unroll
      for (int k = 0; k < 4; k++) q.rv[k] = k < nr ? load2(rrow + k * pitch + i, left) : zero4;
#pragma unroll
      for (int k = 0; k < 2; k++) q.sv[k] = k < ns ? load2(srow + k * pitch + i, left) : zero4;
      q.pv = load2(prow + i, left);
#pragma unroll
      for (int h = 0; h < 2; h++) q.cs[h] = h < left ? __ldg(crow + i + h) : 0.f;
    }
  };
  // warps 0-3 drain columns 0-31 of their lanes' rows, warps 4-7 the others
  const unsigned lane_tmem = tmem + (unsigned)((warp >> 2) * 32) + ((unsigned)(warp & 3) << 21);
  auto drain = [&](int group) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    tmem_load32(lane_tmem + (unsigned)((group & 1) * kN), acc);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  };

  bool ok = true;
  int drained = 0, issued = 0;  // accumulators read back; chunks whose matrix instructions were issued
  // chunk t from its raw operands, which are then those of chunk t + 2 (two
  // chunks ahead: one does not cover the loads' latency)
  auto step = [&](Raw& q, int t) {
    const int s = t & 1;
    if (t >= 2) {  // the stage's earlier matrix instructions are done
      const bool w = bar_wait(smem_u32(&bars[s]), (unsigned)((t >> 1) - 1) & 1u);
      if (!__syncthreads_and(w)) {
        ok = false;
        return;
      }
      if ((t - 1) % kGroup == 0) drain(drained++);  // and with chunk t - 2 its accumulator
    }
    unsigned char* st = stage0 + s * kStageBytes;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 v = make_float4(q.rv[k].x * q.cs[0], q.rv[k].y * q.cs[0], q.rv[k].z * q.cs[1], q.rv[k].w * q.cs[1]);
      sa[k] = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sa[k]))));
      float4 hi, lo;
      split4(v, hi, lo);
      *reinterpret_cast<float4*>(st + swz + k * 4096) = hi;
      *reinterpret_cast<float4*>(st + kABytes + swz + k * 4096) = lo;
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const float4 v = make_float4(q.pv.x * q.sv[k].x - q.pv.y * q.sv[k].y, q.pv.x * q.sv[k].y + q.pv.y * q.sv[k].x,
                                   q.pv.z * q.sv[k].z - q.pv.w * q.sv[k].w, q.pv.z * q.sv[k].w + q.pv.w * q.sv[k].z);
      sb[k] = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, fmaf(v.w, v.w, sb[k]))));
      float4 hi, lo;
      split4(v, hi, lo);
      *reinterpret_cast<float4*>(st + 2 * kABytes + swz + k * 4096) = hi;
      *reinterpret_cast<float4*>(st + 2 * kABytes + kBBytes + swz + k * 4096) = lo;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const unsigned sb0 = base + s * kStageBytes;
      const unsigned long long ah = tile_desc(sb0), al = tile_desc(sb0 + kABytes), bh = tile_desc(sb0 + 2 * kABytes),
                               bl = tile_desc(sb0 + 2 * kABytes + kBBytes);
      const unsigned d = tmem + (unsigned)(((t / kGroup) & 1) * kN), dc = tmem + kCross;
      const unsigned first = t % kGroup == 0;
#pragma unroll
      for (int k = 0; k < 4; k++) {  // 8 values (32 bytes) a step
        mma_tf32(d, ah + 2 * k, bh + 2 * k, !(first && k == 0));
        mma_tf32(dc, ah + 2 * k, bl + 2 * k, t > 0 || k > 0);
        mma_tf32(dc, al + 2 * k, bh + 2 * k, 1);
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&bars[s]))
                   : "memory");
    }
    issued = t + 1;
    if (t + 2 < nch) fetch(q, t + 2);
  };
  Raw q0, q1;
  if (nch > 0) fetch(q0, 0);
  if (nch > 1) fetch(q1, 1);
  for (int t = 0; t < nch && ok; t += 2) {
    step(q0, t);
    if (t + 1 < nch && ok) step(q1, t + 1);
  }
  // the last commit covers everything issued before it
  if (nch > 0 && ok) {
    const int t = nch - 1;
    ok = bar_wait(smem_u32(&bars[t & 1]), (unsigned)(t >> 1) & 1u);
    ok = __syncthreads_and(ok);
    if (ok) {
      while (drained <= t / kGroup) drain(drained++);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tmem_load32(lane_tmem + kCross, acc);
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
  }
  // a wait that ran out (nothing of this kernel's own can cause it): NaN, after
  // one more wait for the last matrix instructions of either stage, which must
  // not be in flight when the tensor memory is given back
  if (!ok)
    for (int s = 0; s < 2; s++)
      if (issued > s) bar_wait(smem_u32(&bars[s]), (unsigned)(last_chunk(issued, s) >> 1) & 1u);
  const float bad = ok ? 0.f : __int_as_float(0x7fc00000);
  {
    const unsigned r = r0 + (warp & 3) * 32 + lane;
    if (r < a.nrefs) {
      float* out = a.part + (((int64_t)split * a.nparticles + p) * a.nrefs + r) * a.nshifts;
#pragma unroll
      for (int i = 0; i < 32; i++) {
        const unsigned s = s0 + (warp >> 2) * 32 + i;
        if (s < a.nshifts) out[s] = acc[i] + bad;
      }
    }
  }
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
#pragma unroll
    for (int k = 0; k < 4; k++) sa[k] += __shfl_xor_sync(0xffffffffu, sa[k], o);
#pragma unroll
    for (int k = 0; k < 2; k++) sb[k] += __shfl_xor_sync(0xffffffffu, sb[k], o);
  }
  if (j == 0) {
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const unsigned r = r0 + row0 + 32 * k;
      if (nt == 0 && r < a.nrefs) a.sa[((int64_t)split * a.nparticles + p) * a.nrefs + r] = sa[k];
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const unsigned s = s0 + row0 + 32 * k;
      if (mt == 0 && s < a.nshifts) a.sb[((int64_t)split * a.nparticles + p) * a.nshifts + s] = sb[k];
    }
  }
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// Combines the splits, writes the outputs and marks the 64 x 64 tiles (of the
// direct kernel) that hold a close match or a value that is not finite.
__global__ void __launch_bounds__(256)
diff2_tc_combine_kernel(const TcArgs a, float* __restrict__ diff2, int* __restrict__ flags) {
  const int64_t n = (int64_t)a.nparticles * a.nrefs * a.nshifts;
  grid_dependency_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t pr = i / a.nshifts;
    const unsigned s = (unsigned)(i - pr * a.nshifts);
    const int64_t p = pr / a.nrefs;
    const unsigned r = (unsigned)(pr - p * a.nrefs);
    double c = 0, sa = 0, sb = 0;
    for (int k = 0; k < a.splits; k++) {
      c += (double)a.part[k * n + i];
      sa += (double)a.sa[((int64_t)k * a.nparticles) * a.nrefs + pr];
      if (!a.cc) sb += (double)a.sb[((int64_t)k * a.nparticles + p) * a.nshifts + s];
    }
    const double half = 0.5 * (sa + sb);
    const float v = a.cc ? (float)(-c / sqrt(sa)) : (float)(half - c);
    diff2[i] = v;
    if (a.cc ? !isfinite(v) : !(v >= kCloseFraction * (float)half) || !isfinite(v)) {
      const unsigned rt = (a.nrefs + kDiffTile - 1) / kDiffTile, st = (a.nshifts + kDiffTile - 1) / kDiffTile;
      flags[(p * rt + r / kDiffTile) * st + s / kDiffTile] = 1;
    }
  }
}

}  // namespace

int diff2_tensor(const float2* particle, const float* minvsigma2, const float* ctf, int64_t elements,
                 const float2* shifts, const float2* refs, float* diff2, unsigned nparticles, unsigned nrefs,
                 unsigned nshifts, bool cc, cudaStream_t stream) {
  TcArgs a;
  a.particle = particle;
  a.minvsigma2 = minvsigma2;
  a.ctf = ctf;
  a.elements = elements;
  a.shifts = shifts;
  a.refs = refs;
  a.nparticles = nparticles;
  a.nrefs = nrefs;
  a.nshifts = nshifts;
  a.mtiles = (int)((nrefs + kM - 1) / kM);
  a.ntiles = (int)((nshifts + kN - 1) / kN);
  a.cc = cc ? 1 : 0;
  a.vec = elements % 2 == 0 && ((uintptr_t)shifts | (uintptr_t)refs) % 16 == 0;
  int dev = 0, sms = 148;
  GTOMRLN_CUDA_TRY(cudaGetDevice(&dev));
  GTOMRLN_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int64_t units = (int64_t)nparticles * a.mtiles * a.ntiles, slots = 2 * sms;
  const int64_t chunks = (elements + kE - 1) / kE;
  // the split of the elements that fills whole waves of two CTAs per SM
  // best, each part 16 stages at least and a set-up of about four
  double best = 1e30;
  a.splits = 1;
  for (int k = 1; k <= 32 && (k == 1 || chunks / k >= 16); k++) {
    const double waves = (double)((units * k + slots - 1) / slots);
    const double cost = waves * ((double)chunks / k + 4.0);
    if (cost < best * 0.97) {
      best = cost;
      a.splits = k;
    }
  }
  const int64_t n = (int64_t)nparticles * nrefs * nshifts;
  const size_t tiles = (size_t)nparticles * ((nrefs + kDiffTile - 1) / kDiffTile) * ((nshifts + kDiffTile - 1) / kDiffTile);
  if (units * a.splits > 0x7fffffffLL) return set_error(GTOMRLN_ERR_INVALID, "squared differences: too many tiles");
  const size_t nsa = (size_t)nparticles * nrefs * a.splits, nsb = (size_t)nparticles * nshifts * a.splits;
  const size_t npe = (size_t)nparticles * (size_t)elements;
  float* scratch = nullptr;
  if (pool_alloc((void**)&scratch, sizeof(float) * (3 * npe + (size_t)n * a.splits + nsa + nsb + tiles), stream)) {
    clear_error();  // no room for the partial products: the direct kernel needs none
    return diff2_direct(particle, minvsigma2, ctf, elements, shifts, refs, diff2, nparticles, nrefs, nshifts, cc,
                        nullptr, stream);
  }
  a.ps = reinterpret_cast<float2*>(scratch);  // (pool allocations are 256-byte aligned)
  a.cs = scratch + 2 * npe;
  a.part = a.cs + npe;
  a.sa = a.part + (size_t)n * a.splits;
  a.sb = a.sa + nsa;
  int* flags = reinterpret_cast<int*>(a.sb + nsb);
  cudaError_t e = cudaMemsetAsync(flags, 0, tiles * sizeof(int), stream);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(diff2_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  if (e == cudaSuccess) {
    diff2_tc_scale_kernel<<<(unsigned)std::min<size_t>((npe + 255) / 256, 8 * (size_t)sms), 256, 0, stream>>>(a);
    launch_dependent(diff2_tc_kernel, (unsigned)(units * a.splits), kThreads, kSmem, stream, a);
    launch_dependent(diff2_tc_combine_kernel, (unsigned)std::min<int64_t>((n + 255) / 256, 16 * sms), 256, 0, stream, a,
                     diff2, flags);
    e = cudaGetLastError();
  }
  int st = GTOMRLN_OK;
  if (e == cudaSuccess)
    st = diff2_direct(particle, minvsigma2, ctf, elements, shifts, refs, diff2, nparticles, nrefs, nshifts, cc, flags,
                      stream);
  const int st2 = pool_free(scratch, stream);
  if (e != cudaSuccess)
    return set_error(GTOMRLN_ERR_CUDA, "launch of diff2_tc_kernel failed: %s", cudaGetErrorString(e));
  return st ? st : st2;
}

}  // namespace gtomrln
