// Device-side building blocks shared by the QMIV kernels (sm_100a).
//
// Data layout in HBM: frames stay in their native planar layout (Y, Cb, Cr; 1 byte per sample up
// to 8 bits, else 2 bytes). Chroma of 4:2:0/4:2:2 is never upsampled into a buffer: every consumer
// reads sample (x >> sx, y >> sy) of the chroma plane, which is exactly the 2x2 (or 2x1) nearest
// replication of the reference loader (libs/pmbb-core/src/xPixelOpsSTD.cpp:30-49, :68-87).
// Out-of-picture reads clamp the coordinate, which equals the reference's edge-replicated margin
// (margin = roundUp(R,2) >= R, apps/QMIV/src/xAppQMIV.cpp:353, extend(Nearest) at :899).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace qmiv {

// A planar picture as the kernels see it. Pitches are in elements of the sample type.
struct Img
{
  const void* p[3];
  int32_t     pitch[3];
  int8_t      sx[3], sy[3];   // chroma subsampling shifts per component (0 for luma / 4:4:4)
};

struct MutImg
{
  void*   p[3];
  int32_t pitch[3];
};

template <typename T>
__device__ __forceinline__ int32_t fetch(const Img& im, int c, int32_t x, int32_t y)
{
  const T* base = static_cast<const T*>(im.p[c]);
  return (int32_t)__ldg(base + (size_t)(y >> im.sy[c]) * im.pitch[c] + (x >> im.sx[c]));
}

__device__ __forceinline__ int32_t clampi(int32_t v, int32_t lo, int32_t hi) { return min(max(v, lo), hi); }
// The int32 product of the reference's integer code where it may wrap (two's complement), formed in
// unsigned arithmetic: a signed overflow is undefined in C++ and lets the compiler widen the product.
__device__ __forceinline__ int32_t mul_wrap(int32_t a, int32_t b) { return (int32_t)((uint32_t)a * (uint32_t)b); }

// Exact conversions between integers in [0, 2^23) and floats without the (quarter-rate) conversion
// pipe: a float in [2^23, 2^24) has a unit ulp, so its low mantissa bits are the integer.
__device__ __forceinline__ float u2f_exact(uint32_t v) { return __uint_as_float(v | 0x4B000000u) - 8388608.0f; }
__device__ __forceinline__ int32_t f2i_exact(float f) { return (int32_t)(__float_as_uint(f + 8388608.0f) - 0x4B000000u); }

// Exact IEEE double operations, never contracted into FMA, so device results equal the host
// reference's separately rounded operations bit for bit.
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// Kahan-Babuska-Neumaier compensated sum (libs/pmbb-core/src/xKBNS.h:36-43).
// The reference adds to c the rounding error of s + v, computed by Fast2Sum with the larger of the
// two operands first: (big - t) + small. Here the operands are chosen by a compare and two selects
// instead of a branch, four FP64 additions and one FP64 compare per term (Knuth's branch-free TwoSum,
// which yields the same exactly representable error, takes six additions).
struct Kbns
{
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double v)
  {
    const double t = dadd(s, v);
    const bool   sb = fabs(s) >= fabs(v);
    const double big = sb ? s : v, small = sb ? v : s;
    c = dadd(c, dadd(dsub(big, t), small));
    s = t;
  }
  // N terms in order where |s| >= |v| is known for each: the larger operand is s, so the compare and the
  // selects go away. The four additions of a term depend on one another, and a lone warp issues in order,
  // so they are written a term apart: the next sum, the difference of the last one, the error of the one
  // before, the compensation of the one before that. WS-PSNR of a 4096x2048 pair whose row errors span more than
  // ExactSum takes: 63 us a call term by term, 56 like this.
  template <int N>
  __device__ __forceinline__ void add_small(const double (&v)[N])
  {
    static_assert(N >= 3, "three terms in flight");
    double t0 = s, t1 = dadd(s, v[0]);                       // the sums before and after the last term
    double d = 0.0, e = 0.0;                                 // t0 - t1 of the term before, error of the one before that
    #pragma unroll
    for(int k = 1; k < N; k++)
    {
      const double t2 = dadd(t1, v[k]);
      const double d1 = dsub(t0, t1);
      if(k >= 2)
      {
        const double e1 = dadd(d, v[k - 2]);
        if(k >= 3) { c = dadd(c, e); }
        e = e1;
      }
      asm volatile("" ::: "memory");                         // keeps the order
      d = d1; t0 = t1; t1 = t2;
    }
    const double d1 = dsub(t0, t1), e1 = dadd(d, v[N - 2]);
    c = dadd(c, e);
    c = dadd(c, e1);
    c = dadd(c, dadd(d1, v[N - 1]));
    s = t1;
  }
  __device__ __forceinline__ double result() const { return dadd(s, c); }
};

// The result of a Kbns chain, from its terms in any order, where order cannot matter.
//
// Every addition to s leaves an error that is a multiple of q, the last bit of the smallest term other than
// zero, and is at most half a last bit of a sum below n times the largest term. When all n such errors together
// stay below 2^53 q, each addition to c is exact, so that s + c is exactly the sum of the terms and
// result() is that sum rounded once. With |v| < 2^(emax + 1), q = 2^(emin - 52) and n < 2^L the errors are at most
// 2^(emax + L - 53) each, and emax - emin <= 53 - 2 L is enough (L >= 1 more is kept below). The same
// bound holds for any other tree of the same additions (n terms have n - 1 that are not exact by
// themselves), so the terms are summed by as many threads as there are, with the branch-free TwoSum, and their
// sums combined. A chain that fails the test (terms more than about 2^30 apart, infinite, NaN or subnormal ones)
// is summed in order.
//
// What bounded the ordered chains: the latency of their additions, 8 cycles a term with one thread at work. A
// chain of 2048 rows took 14 us of a 26 us launch, one of 1023 windows 25 us with its loads.
struct ExactSum
{
  double s = 0.0, c = 0.0;
  uint32_t top = 0u, low = 0xffffffffu, sign = 0u;            // of the terms' high words: largest, smallest non-zero - 1, sign bits
  __device__ __forceinline__ void two_sum(double v)
  {
    const double t = dadd(s, v), z = dsub(t, s);
    c = dadd(c, dadd(dsub(s, dsub(t, z)), dsub(v, z)));
    s = t;
  }
  __device__ __forceinline__ void add(double v)
  {
    const uint32_t h = (uint32_t)__double2hiint(v);
    const uint32_t u = (h & 0x7fffffffu) | min((uint32_t)__double2loint(v), 1u);   // 0 for zeros alone
    top = max(top, u);
    low = min(low, u - 1u);
    sign |= h;
    two_sum(v);
  }
  __device__ __forceinline__ void join(const ExactSum& o)
  {
    two_sum(o.s);
    c = dadd(c, o.c);
    top = max(top, o.top); low = min(low, o.low); sign |= o.sign;
  }
  __device__ __forceinline__ void join_warp()
  {
    #pragma unroll
    for(int d = 16; d > 0; d >>= 1)
    {
      const double os = __shfl_xor_sync(0xffffffffu, s, d), oc = __shfl_xor_sync(0xffffffffu, c, d);
      two_sum(os);
      c = dadd(c, oc);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    low = __reduce_min_sync(0xffffffffu, low);
    sign = __reduce_or_sync(0xffffffffu, sign);
  }
  // n: the number of terms, or more
  __device__ __forceinline__ bool exact(int n) const
  {
    if(top == 0u) { return true; }                           // zeros only
    const int L = 32 - __clz(n), emax = (int)(top >> 20), emin = (int)(low >> 20);
    return emin > 0 && emax + L + 2 < 0x7ff && emax - emin <= 51 - 2 * L;
  }
  __device__ __forceinline__ double result() const { return dadd(s, c); }
};

// Ordered compensated sum of vals[0, n) after `k`, by one thread. all: the terms of the whole chain, for their
// largest and their signs. While all terms are non-negative the sum never falls, so from the first
// prefix that reaches the largest term on every addition has |s| >= |v|. Reached only by chains that ExactSum
// cannot take.
__device__ __forceinline__ void chain_sum(Kbns& k, const double* vals, int n, const ExactSum& all)
{
  int y = 0;
  const double vmax = __hiloint2double((int)(all.top + 1u), 0);
  const bool ordered = (int32_t)all.sign >= 0 && all.top < 0x7fe00000u;   // finite and non-negative
  for(; y + 8 <= n && !(ordered && k.s >= vmax); y += 8)     // eight at a time: a call whose largest term comes late took 77 us one by one, 60 so
  {
    double v[8];
    #pragma unroll
    for(int u = 0; u < 8; u++) { v[u] = vals[y + u]; }
    #pragma unroll
    for(int u = 0; u < 8; u++) { k.add(v[u]); }
  }
  for(; y + 32 <= n; y += 32)
  {
    double v[32];
    #pragma unroll
    for(int u = 0; u < 32; u++) { v[u] = vals[y + u]; }
    k.add_small(v);
  }
  for(; y < n; y++) { k.add(vals[y]); }
}

// SSIM of one window (xStructSimSTD.cpp:420-461, same operation order; AVX-512 CalcBlckAvg8 /
// CalcMultiBlckAvg8S4 give the same per-window value) from its moments divided by the window area:
// ar = SumR / 64, at = SumT / 64, qr = SumR2 / 64, qt = SumT2 / 64, qrt = SumRT / 64 (all exact).
// 2 x is formed as x + x, which is the same double.
__device__ __forceinline__ double ssim_window_avg(double ar, double at, double qr, double qt, double qrt, double C1,
                                                  double C2, bool calc_l)
{
  const double ar2 = dmul(ar, ar), at2 = dmul(at, at);
  const double var_r = dsub(qr, ar2);
  const double var_t = dsub(qt, at2);
  const double cov   = dsub(qrt, dmul(ar, at));
  const double cs    = ddiv(dadd(dadd(cov, cov), C2), dadd(dadd(var_r, var_t), C2));
  if(!calc_l) { return cs; }
  const double l = ddiv(dadd(dmul(dadd(ar, ar), at), C1), dadd(dadd(ar2, at2), C1));
  return dmul(l, cs);
}

// 4x4 sub-block moments of an SSIM picture pair, five uint32 planes per component:
// [c][m][nby][pitch], m = 0: sum a, 1: sum b, 2: sum a^2, 3: sum b^2, 4: sum a*b
// (a = the "Tst" picture, b = the "Ref" picture of xSSIM::xCalcPicSSIM). Every 8x8/stride-4 window is
// the sum of 2x2 sub-blocks, so window moments are exact integers.
struct Moments
{
  uint32_t* p;      // base of component 0, moment 0
  int32_t   nbx, nby, pitch;
  __host__ __device__ size_t plane() const { return (size_t)nby * pitch; }
};

// Round half away from zero by adding +-0.5 in double and truncating (xHelpersFLT.h:33).
__device__ __forceinline__ int32_t round_half_away(double v)
{
  const double t = dadd(v, copysign(0.5, v));
  return (int32_t)t;  // truncation toward zero, as cvttsd2si
}

// Per-pair device outputs consumed by the host finishing step.
constexpr int kMaxSsimSlots = 18;   // SSIM 1 + IV-SSIM 2 + MS-SSIM 5 + IV-MS-SSIM 2x5

struct PairOut
{
  int32_t  gcd[4];
  int32_t  flags;            // bit0: frame0 invalid, bit1: frame1 invalid, bit2: integer CPS path,
                             // bit3: a CPS tile load did not complete (bounded wait ran out)
  uint32_t or_sample[2];     // OR of every sample per frame: above maxv (2^bd - 1) iff some sample is
  uint32_t done;             // CTAs of the prepass that have added their rows; then chains finished
  int64_t  sd[3];            // 4:4:4 totals of In1 - In0 (raw sums while the prepass runs)
  uint64_t ssd[3];           // 4:4:4 totals
  double   ws_ssd[3];        // KBNS over rows of rowSSD*w[y] (WS-PSNR, before correction)
  uint64_t cps_sum[2][3];    // sum over rows of sign-extended 32-bit row sums, [R2T, T2R]
  double   cps_ws[2][3];     // KBNS over rows of rowSSE*w[y]
  double   ssim[kMaxSsimSlots][3];
};

// ---- dependent launches ------------------------------------------------------------------------
// A kernel launched by launch_next may be scheduled while its predecessor in the stream still runs, from
// when every CTA of that one has called next_may_start. It begins with wait_for_previous, which returns
// when the predecessor, and so all work before it, is complete and its writes are visible. In an ordinary
// launch both do nothing.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ---- mbarriers and bulk copies ----------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_barrier_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
  uint32_t ok;
  asm volatile(
    "{\n\t.reg .pred p;\n\t"
    "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
    "selp.u32 %0, 1, 0, p;\n\t}"
    : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok != 0;
}
// Waits for the phase with the given parity; gives up (false) after about `limit` cycles.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long long limit)
{
  if(mbar_try_wait(bar, parity)) { return true; }
  const long long t0 = clock64();
  do
  {
    if(mbar_try_wait(bar, parity)) { return true; }
  } while(clock64() - t0 <= limit);
  return false;
}
}  // namespace qmiv
