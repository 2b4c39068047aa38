// QMIV metric kernels for B200 (sm_100a).
//
// Pipeline of one frame pair (the reference runs the same steps per frame on the CPU,
// apps/QMIV/src/xAppQMIV.cpp:761-827):
//   k_prepass   SD(In1-In0), SSD per raw row, OR of the samples (reads both frames once); its last
//               CTA: totals, GCD, exactness of the key search path
//   k_cps       (qmiv_cps.cu, qmiv_cps420.cuh) corresponding-pixel-shift search, both directions in one pass;
//               per-row SSE into 32-bit lanes, the IV-SSIM sub-block moments of (test, SCP) and,
//               when IV-MS-SSIM or the caller needs them, the shift-compensated pictures
//   k_ssim_*    (qmiv_ssim.cu) block SSIM from exact integer moments, FP64 windows, row sums
//   k_finalize  every FP64 pooling chain of the pair (one CTA per chain)
#include "qmiv_kernels.cuh"

#include <cstdio>
#include <mutex>

namespace qmiv {

constexpr unsigned kFull = 0xffffffffu;

// =============================================================================================
// prepass
// =============================================================================================
// A warp takes one raw row. Its sums join the picture's by way of the CTA (eight rows, six additions to the
// result block), and the CTA that adds last turns the totals into the GCD (xGlobClrDiff.cpp:70-103) and the
// path flags: a launch of its own for that took 7 us of a one-pair call, most of it latency.
// Bound by the loads' latency for one pair and near the memory's rate for many: with one 16-byte load of each row in
// flight, 64-bit sums per sample and only rows that start on 16 bytes, 4096x2048 10 bits took 25.6 us (eight
// pairs, 400 MB, 79); like this 21.4 (71). A 1998x1080 12-bit call, whose rows start anywhere: 227 -> 218 us.
// Sum and sum of squares of B - A over the samples of one 16-byte vector of either row (8-bit samples: Gram
// sums by byte dot products; 16-bit samples below 2^14: both differences of a word from one subtraction).
template <typename T>
__device__ __forceinline__ void prepass_vector(const uint32_t (&A)[4], const uint32_t (&B)[4], int32_t& d, uint32_t& dd)
{
  uint32_t sa = 0, sb = 0, qq = 0, ab = 0;
  d = 0; dd = 0;
  #pragma unroll
  for(int k = 0; k < 4; k++)
  {
    if constexpr(sizeof(T) == 1)
    {
      sa = __dp4a(A[k], 0x01010101u, sa);
      sb = __dp4a(B[k], 0x01010101u, sb);
      qq = __dp4a(A[k], A[k], __dp4a(B[k], B[k], qq));
      ab = __dp4a(A[k], B[k], ab);
    }
    else
    {
      const int32_t w = (int32_t)(B[k] - A[k]), lo = (int16_t)w, hi = (w + 0x8000) >> 16;   // |lo| < 2^14 borrows nothing from the rounding
      d += lo + hi;
      dd += (uint32_t)(lo * lo);
      dd += (uint32_t)(hi * hi);                             // eight squares below 2^28
    }
  }
  if constexpr(sizeof(T) == 1) { d = (int32_t)(sb - sa); dd = qq - 2u * ab; }
}

template <typename T>
__device__ __forceinline__ void prepass_row(const PrepassArgs& a, int warp, int lane, int& c, int64_t& sd_out, uint64_t& ssd_out, uint32_t& m0_out,
                                            uint32_t& m1_out)
{
  int r = warp;
  c = 0;
  if(r >= a.rows[0]) { r -= a.rows[0]; c = 1; if(r >= a.rows[1]) { r -= a.rows[1]; c = 2; } }
  const T* p0 = static_cast<const T*>(a.in0.p[c]) + (size_t)r * a.in0.pitch[c];
  const T* p1 = static_cast<const T*>(a.in1.p[c]) + (size_t)r * a.in1.pitch[c];
  const int n = a.cols[c];

  int64_t  sd  = 0;
  uint64_t ssd = 0;
  uint32_t m0 = 0, m1 = 0;                                 // OR of the samples
  auto sample = [&](uint32_t v0, uint32_t v1) {
    v0 = min(v0, a.clip); v1 = min(v1, a.clip);
    const int32_t d = (int32_t)v1 - (int32_t)v0;
    sd  += d;
    ssd += (uint32_t)d * (uint32_t)d;                    // d^2 < 2^32 for 16-bit samples
  };
  // 16-byte loads, four of each row in flight per lane, where both rows lie alike to 16 bytes; what is before the first
  // boundary and behind the last sample by sample
  int head = 0, x0 = 0;
  if((((uintptr_t)p0 ^ (uintptr_t)p1) & 15) == 0)
  {
    constexpr int V = 16 / (int)sizeof(T), U = 4;
    head = min(n, (int)((0u - (uint32_t)(uintptr_t)p0) & 15u) / (int)sizeof(T));
    const int nv = (n - head) / V;
    const uint4* q0 = reinterpret_cast<const uint4*>(p0 + head);
    const uint4* q1 = reinterpret_cast<const uint4*>(p1 + head);
    const bool clips = a.clip < (sizeof(T) == 1 ? 0xffu : 0xffffu);
    for(int v0 = lane; v0 < nv; v0 += 32 * U)
    {
      uint4 A[U], B[U];
      #pragma unroll
      for(int u = 0; u < U; u++)
      {
        const int v = v0 + 32 * u;
        A[u] = B[u] = make_uint4(0u, 0u, 0u, 0u);          // equal samples add nothing
        if(v < nv) { A[u] = __ldg(q0 + v); B[u] = __ldg(q1 + v); }
      }
      #pragma unroll
      for(int u = 0; u < U; u++)
      {
        const uint32_t wa[4] = { A[u].x, A[u].y, A[u].z, A[u].w }, wb[4] = { B[u].x, B[u].y, B[u].z, B[u].w };
        const uint32_t oa = wa[0] | wa[1] | wa[2] | wa[3], ob = wb[0] | wb[1] | wb[2] | wb[3];
        m0 |= oa; m1 |= ob;
        if(!clips && (sizeof(T) == 1 || ((oa | ob) & 0xc000c000u) == 0u))
        {
          int32_t d;
          uint32_t dd;
          prepass_vector<T>(wa, wb, d, dd);
          sd += d; ssd += dd;
        }
        else
        {
          #pragma unroll 1
          for(int k = 0; k < V; k++)
          {
            constexpr int BITS = 8 * (int)sizeof(T);
            const uint32_t w0 = k * BITS < 64 ? (k * BITS < 32 ? wa[0] : wa[1]) : (k * BITS < 96 ? wa[2] : wa[3]);
            const uint32_t w1 = k * BITS < 64 ? (k * BITS < 32 ? wb[0] : wb[1]) : (k * BITS < 96 ? wb[2] : wb[3]);
            const int sh = (k * BITS) & 31;
            sample((w0 >> sh) & ((1u << BITS) - 1u), (w1 >> sh) & ((1u << BITS) - 1u));
          }
        }
      }
    }
    constexpr uint32_t low = sizeof(T) == 1 ? 0xffu : 0xffffu;
    m0 = sizeof(T) == 1 ? (m0 | (m0 >> 8) | (m0 >> 16) | (m0 >> 24)) & low : (m0 | (m0 >> 16)) & low;
    m1 = sizeof(T) == 1 ? (m1 | (m1 >> 8) | (m1 >> 16) | (m1 >> 24)) & low : (m1 | (m1 >> 16)) & low;
    x0 = head + nv * V;
  }
  auto at = [&](int x) {
    const uint32_t v0 = __ldg(p0 + x), v1 = __ldg(p1 + x);
    m0 |= v0; m1 |= v1;
    sample(v0, v1);
  };
  if(lane < head) { at(lane); }
  for(int x = x0 + lane; x < n; x += 32) { at(x); }
  #pragma unroll
  for(int o = 16; o > 0; o >>= 1)
  {
    sd  += __shfl_xor_sync(kFull, sd, o);
    ssd += __shfl_xor_sync(kFull, ssd, o);
  }
  m0_out = __reduce_or_sync(kFull, m0);
  m1_out = __reduce_or_sync(kFull, m1);
  sd_out = sd;
  ssd_out = ssd;
  if(lane == 0) { a.row_ssd[warp] = ssd; }
}

__device__ __forceinline__ void prepass_totals(const PrepassArgs& a);

template <typename T>
__device__ __forceinline__ void prepass_body(const PrepassArgs& a, int block)
{
  __shared__ int64_t  s_sd[8];
  __shared__ uint64_t s_ssd[8];
  __shared__ uint32_t s_m[2][8];
  __shared__ int32_t  s_c[8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warp = block * 8 + wid;
  const int total = a.rows[0] + a.rows[1] + a.rows[2];
  if(block * 8 >= total) { return; }                       // uniform: not a CTA of this pair
  int c = -1;
  int64_t sd = 0;
  uint64_t ssd = 0;
  uint32_t m0 = 0, m1 = 0;
  if(warp < total) { prepass_row<T>(a, warp, lane, c, sd, ssd, m0, m1); }
  if(lane == 0) { s_sd[wid] = sd; s_ssd[wid] = ssd; s_m[0][wid] = m0; s_m[1][wid] = m1; s_c[wid] = c; }
  __syncthreads();
  if(threadIdx.x >= 32) { return; }
  PairOut* o = a.out;
  if(lane < 6)
  {
    const int k = lane % 3;
    unsigned long long v = 0;
    bool any = false;
    #pragma unroll
    for(int w = 0; w < 8; w++)
    {
      if(s_c[w] == k) { v += lane < 3 ? (unsigned long long)s_sd[w] : (unsigned long long)s_ssd[w]; any = true; }
    }
    if(any) { atomicAdd(lane < 3 ? reinterpret_cast<unsigned long long*>(&o->sd[k]) : reinterpret_cast<unsigned long long*>(&o->ssd[k]), v); }
  }
  else if(lane < 8)
  {
    uint32_t m = 0;
    #pragma unroll
    for(int w = 0; w < 8; w++) { m |= s_m[lane - 6][w]; }
    atomicOr(&o->or_sample[lane - 6], m);
  }
  __threadfence();                                          // the additions before the count
  __syncwarp();
  if(lane == 0 && atomicAdd(&o->done, 1u) == (uint32_t)((total + 7) / 8) - 1u)
  {
    __threadfence();
    prepass_totals(a);
  }
}

template <typename T>
__global__ void __launch_bounds__(256) k_prepass(const __grid_constant__ PrepassArgs a)
{
  prepass_body<T>(a, (int)blockIdx.x);
}

// one job (frame pair) per blockIdx.y
template <typename T>
__global__ void __launch_bounds__(256) k_prepass_multi(const PrepassArgs* __restrict__ jobs)
{
  prepass_body<T>(jobs[blockIdx.y], (int)blockIdx.x);
}

template <typename T>
cudaError_t launch_prepass(const PrepassArgs& a, cudaStream_t s)
{
  const int total  = a.rows[0] + a.rows[1] + a.rows[2];
  const int blocks = (total + 7) / 8;
  k_prepass<T><<<blocks, 256, 0, s>>>(a);
  return cudaGetLastError();
}
template cudaError_t launch_prepass<uint8_t>(const PrepassArgs&, cudaStream_t);
template cudaError_t launch_prepass<uint16_t>(const PrepassArgs&, cudaStream_t);

template <typename T>
cudaError_t launch_prepass_multi(const PrepassArgs* d_jobs, int njobs, int max_rows, cudaStream_t s)
{
  if(njobs <= 0) { return cudaSuccess; }
  k_prepass_multi<T><<<dim3((max_rows + 7) / 8, njobs), 256, 0, s>>>(d_jobs);
  return cudaGetLastError();
}
template cudaError_t launch_prepass_multi<uint8_t>(const PrepassArgs*, int, int, cudaStream_t);
template cudaError_t launch_prepass_multi<uint16_t>(const PrepassArgs*, int, int, cudaStream_t);

// Totals, GCD and path flags, by one thread of the last CTA (libs/pmbb-ivqm/src/xGlobClrDiff.cpp:70-103).
__device__ __forceinline__ void prepass_totals(const PrepassArgs& a)
{
  PairOut* o = a.out;
  const double area = (double)a.area;
  int64_t sd[4] = { 0, 0, 0, 0 };
  for(int c = 0; c < 3; c++)
  {
    sd[c] = (int64_t)__ldcg(reinterpret_cast<const unsigned long long*>(&o->sd[c])) * a.mult[c];
    o->sd[c]  = sd[c];
    o->ssd[c] = (uint64_t)__ldcg(reinterpret_cast<const unsigned long long*>(&o->ssd[c])) * (uint64_t)a.mult[c];
  }
  #pragma unroll
  for(int c = 0; c < 4; c++)
  {
    int32_t g = 0;
    if(a.gcd_override_on) { g = a.gcd_override[c]; }
    else if(a.need_gcd) { g = clampi(round_half_away(ddiv((double)sd[c], area)), -a.maxdiff[c], a.maxdiff[c]); }
    o->gcd[c] = g;
  }
  const int inv0 = __ldcg(&o->or_sample[0]) > (uint32_t)a.maxv;
  const int inv1 = __ldcg(&o->or_sample[1]) > (uint32_t)a.maxv;
  const int int_path = !a.fp32_ok || ((inv0 || inv1) && !a.clip_on);
  o->flags = inv0 | (inv1 << 1) | (int_path << 2);
  o->done = 0u;
}

// (CPS search: qmiv_cps.cu)

// =============================================================================================
// finalize: the FP64 pooling chains of one pair.
// Inputs are staged into shared memory and summed by all threads (ExactSum); a chain whose order matters
// is summed again by one. 4096x2048, all chains: 26 us with one thread per chain, 12.6 like this (latency
// of the launch, the loads and the reduction).
//   WS-PSNR   KBNS over rows of rowSSD * w[y]            (xWSPSNR.cpp:123-132)
//   IV-PSNR   KBNS over rows of rowSSE * w[y] (ERP)       (xIVPSNR.cpp:171-175) + exact uint64 sums
//   SSIM      KBNS over window rows (ERP: row * w[base + step j], weights KBNS) (xSSIM.cpp:348-351,
//             xIVSSIM.cpp:148-172)
// =============================================================================================
// One CTA per chain, so that the chains of one pair run on different SMs.
__device__ __forceinline__ double chain_value(const FinalizeArgs& a, const FinChain& ch, int y)
{
  if(ch.kind == kChainWsPsnr)
  {
    int off = 0;
    for(int q = 0; q < ch.a; q++) { off += a.rows[q]; }
    const uint64_t r = a.row_ssd[off + (y >> a.sy[ch.a])] * (uint64_t)a.mult_row[ch.a];
    return dmul((double)r, a.ws[y]);
  }
  if(ch.kind == kChainIvPsnr)
  {
    const uint64_t r = (uint64_t)(int64_t)(int32_t)a.cps_rows[((size_t)ch.a * a.H + y) * 3 + ch.b];
    return dmul((double)r, a.ws[y]);
  }
  const SsimSlot& sl = a.slot[ch.a];
  const double v = sl.row_sum[(size_t)ch.b * sl.ny + y];
  return sl.use_ws ? dmul(v, a.ws[sl.ws_base + sl.ws_step * y]) : v;
}

__device__ __forceinline__ void finalize_body(const FinalizeArgs& a, int chain, double* stage)
{
  PairOut* o = a.out;
  if(chain == a.nchains)
  {
    // exact uint64 totals of the sign-extended 32-bit CPS row sums (order independent)
    __shared__ unsigned long long acc[6];
    if(threadIdx.x < 6) { acc[threadIdx.x] = 0ull; }
    __syncthreads();
    unsigned long long loc[6] = { 0, 0, 0, 0, 0, 0 };
    for(int y = threadIdx.x; y < a.H; y += blockDim.x)
    {
      #pragma unroll
      for(int k = 0; k < 6; k++)
      {
        loc[k] += (unsigned long long)(long long)(int32_t)a.cps_rows[((size_t)(k / 3) * a.H + y) * 3 + (k % 3)];
      }
    }
    #pragma unroll
    for(int k = 0; k < 6; k++)
    {
      #pragma unroll
      for(int o2 = 16; o2 > 0; o2 >>= 1) { loc[k] += __shfl_down_sync(0xffffffffu, loc[k], o2); }
      if((threadIdx.x & 31) == 0) { atomicAdd(&acc[k], loc[k]); }
    }
    __syncthreads();
    if(threadIdx.x < 6) { o->cps_sum[threadIdx.x / 3][threadIdx.x % 3] = acc[threadIdx.x]; }
    return;
  }
  const FinChain ch = a.chain[chain];
  const bool wsum = ch.kind == kChainSsim && a.slot[ch.a].use_ws;
  const int len = ch.kind == kChainSsim ? a.slot[ch.a].ny : a.H;
  double* vals = stage;
  double* wts = stage + len;
  __shared__ ExactSum part[2][8];                            // per warp: of the values and of the weights
  __shared__ double wtotal;
  // eight rows per thread and pass with their loads issued together (one round trip per pass)
  constexpr int U = 8;
  ExactSum sv, sw;
  for(int y0 = threadIdx.x; y0 < len; y0 += 256 * U)
  {
    double v[U], w[U];
    #pragma unroll
    for(int u = 0; u < U; u++)
    {
      const int y = y0 + u * 256;
      v[u] = y < len ? chain_value(a, ch, y) : 0.0;
      w[u] = (wsum && y < len) ? a.ws[a.slot[ch.a].ws_base + a.slot[ch.a].ws_step * y] : 0.0;
    }
    #pragma unroll
    for(int u = 0; u < U; u++)
    {
      const int y = y0 + u * 256;
      if(y < len) { vals[y] = v[u]; if(wsum) { wts[y] = w[u]; } }
      sv.add(v[u]);
      if(wsum) { sw.add(w[u]); }
    }
  }
  sv.join_warp();
  if(wsum) { sw.join_warp(); }
  if((threadIdx.x & 31) == 0) { part[0][threadIdx.x >> 5] = sv; part[1][threadIdx.x >> 5] = sw; }
  __syncthreads();
  // thread 0 adds up the warps' sums of the values, the second warp's first thread those of the weights; a
  // chain whose order matters is summed again from the staged terms
  double total = 0.0;
  if(threadIdx.x == 0 || (threadIdx.x == 32 && wsum))
  {
    const int k = threadIdx.x >> 5;
    ExactSum all = part[k][0];
    for(int q = 1; q < 8; q++) { all.join(part[k][q]); }
    total = all.result();
    if(!all.exact(len))
    {
      Kbns sum;
      chain_sum(sum, k ? wts : vals, len, all);
      total = sum.result();
    }
    if(k) { wtotal = total; }
  }
  __syncthreads();
  if(threadIdx.x != 0) { return; }
  if(ch.kind == kChainWsPsnr) { o->ws_ssd[ch.a] = total; }
  else if(ch.kind == kChainIvPsnr) { o->cps_ws[ch.a][ch.b] = total; }
  else
  {
    const SsimSlot& sl = a.slot[ch.a];
    const double active = (double)((int64_t)sl.nx * sl.ny);
    double r;
    if(wsum)
    {
      const double corr = ddiv(wtotal, (double)sl.ny);
      r = ddiv(total, dmul(active, corr));
    }
    else { r = ddiv(total, active); }
    o->ssim[ch.a][ch.b] = r;
  }
}

__global__ void __launch_bounds__(256) k_finalize(const __grid_constant__ FinalizeArgs a)
{
  extern __shared__ double stage[];  // [len] values, then [len] ERP weights for weighted SSIM chains
  wait_for_previous();
  finalize_body(a, blockIdx.x, stage);
  if(a.host == nullptr) { return; }
  // The CTA that finishes last writes the results to the host: a copy behind the kernel took 5 us more.
  __shared__ bool last;
  __syncthreads();
  if(threadIdx.x == 0) { __threadfence(); last = atomicAdd(&a.out->done, 1u) == gridDim.x - 1u; }
  __syncthreads();
  if(!last) { return; }
  __threadfence();
  static_assert(sizeof(PairOut) % 4 == 0, "word copies");
  for(int w = threadIdx.x; w < (int)(sizeof(PairOut) / 4); w += blockDim.x)
  {
    reinterpret_cast<volatile uint32_t*>(a.host)[w] = __ldcg(reinterpret_cast<const uint32_t*>(a.out) + w);
  }
}

// one (pair, chain) job per CTA
__global__ void __launch_bounds__(256) k_finalize_multi(const FinalizeArgs* __restrict__ pairs, const FinJob* __restrict__ jobs)
{
  extern __shared__ double stage[];
  const FinJob j = jobs[blockIdx.x];
  finalize_body(pairs[j.pair], j.chain, stage);
}

int finalize_plan(FinalizeArgs& a)
{
  a.nchains = 0;
  if(a.do_wspsnr && a.ws) { for(int c = 0; c < 3; c++) { a.chain[a.nchains++] = { kChainWsPsnr, c, 0 }; } }
  if(a.cps_rows && a.ws) { for(int d = 0; d < 2; d++) { for(int c = 0; c < 3; c++) { a.chain[a.nchains++] = { kChainIvPsnr, d, c }; } } }
  for(int sl = 0; sl < a.nslots; sl++)
  {
    if(a.slot[sl].row_sum == nullptr || a.slot[sl].ny <= 0) { continue; }
    for(int c = 0; c < 3; c++) { a.chain[a.nchains++] = { kChainSsim, sl, c }; }
  }
  return a.nchains + (a.cps_rows ? 1 : 0);
}

size_t finalize_smem(const FinalizeArgs& a) { return (size_t)2 * max(a.H, 1) * sizeof(double); }

static cudaError_t finalize_configure()
{
  static std::mutex mu;
  static uint64_t done = 0;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if(e != cudaSuccess) { return e; }
  const uint64_t bit = 1ULL << (dev & 63);
  std::lock_guard<std::mutex> lk(mu);
  if(done & bit) { return cudaSuccess; }
  e = cudaFuncSetAttribute(k_finalize, cudaFuncAttributeMaxDynamicSharedMemorySize, kFinalizeMaxSmem);
  if(e == cudaSuccess) { e = cudaFuncSetAttribute(k_finalize_multi, cudaFuncAttributeMaxDynamicSharedMemorySize, kFinalizeMaxSmem); }
  if(e == cudaSuccess) { done |= bit; }
  return e;
}

cudaError_t launch_finalize(const FinalizeArgs& a_in, cudaStream_t s)
{
  FinalizeArgs a = a_in;
  const int blocks = finalize_plan(a);
  if(blocks == 0) { return cudaSuccess; }
  const size_t smem = finalize_smem(a);
  if(smem > kFinalizeMaxSmem) { return cudaErrorInvalidValue; }
  cudaError_t e = finalize_configure();
  if(e != cudaSuccess) { return e; }
  return launch_next(k_finalize, blocks, 256, smem, s, a);
}

cudaError_t launch_finalize_multi(const FinalizeArgs* d_pairs, const FinJob* d_jobs, int njobs, size_t smem, cudaStream_t s)
{
  if(njobs <= 0) { return cudaSuccess; }
  if(smem > kFinalizeMaxSmem) { return cudaErrorInvalidValue; }
  cudaError_t e = finalize_configure();
  if(e != cudaSuccess) { return e; }
  k_finalize_multi<<<njobs, 256, smem, s>>>(d_pairs, d_jobs);
  return cudaGetLastError();
}

}  // namespace qmiv
