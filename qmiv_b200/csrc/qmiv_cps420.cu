// Host side of the 4:2:0 search (qmiv_cps420.cuh) and its unmasked forms. The masked forms are a translation unit,
// and so a device module, of their own: a process loads only the forms that it uses.
#include "qmiv_cps420.cuh"

namespace qmiv {

bool cps420_fits(int R, int esz)
{
  int dev = 0;
  if(cudaGetDevice(&dev) != cudaSuccess) { return false; }
  bool fits = false;
  with_geo<false>(R, esz, 0, [&](auto g) { using G = decltype(g); fits = (size_t)G::SMEM + 4096 <= (size_t)dev_info(dev).smem_optin; });
  return fits;
}

int cps420_tiles(int W, int H) { return ((W + 127) / 128) * ((H + 15) / 16); }

// Tile counts, tensor maps and key constants of a pair whose k.a is filled.
cudaError_t cps420_describe(CpsKernelArgs& k, int R, int esz, CpsPairPlan* plan)
{
  k.g.ntx = (k.a.W + 127) / 128;
  k.g.ntiles = cps420_tiles(k.a.W, k.a.H);
  if(k.a.mask) { cps_masked_key(R, k.a.maxv, k.a.wi, k.a.gmax, &k.a.key_masked); }
  cps_shared_key(R, k.a.maxv, k.a.wi, k.a.gmax, &k.a.key_bias, &k.a.key_mid);
  auto describe = [&](auto g) {
    using G = decltype(g);
    bool tma = true;
    for(int f = 0; f < 2; f++)
    {
      const Img& im = f ? k.a.in1 : k.a.in0;
      tma = tma && cps_encode_plane(&k.map[f][0], im.p[0], k.a.W, k.a.H, im.pitch[0], esz, G::BWL, G::BHL) &&
            cps_encode_plane(&k.map[f][1], im.p[1], k.a.W >> 1, k.a.H >> 1, im.pitch[1], esz, G::BWC, G::BHC) &&
            cps_encode_plane(&k.map[f][2], im.p[2], k.a.W >> 1, k.a.H >> 1, im.pitch[2], esz, G::BWC, G::BHC);
    }
    if(G::MASK) { tma = tma && cps_encode_plane(&k.mask_map, k.a.mask, k.a.W, k.a.H, k.a.mask_pitch, k.a.mask_esz, G::BWM, G::BHL); }
    k.g.use_tma = tma ? 1 : 0;
    if(plan) { plan->ntiles = k.g.ntiles; plan->raw_bytes = 0; plan->smem = G::SMEM; }
  };
  const bool known = k.a.mask ? with_geo<true>(R, esz, k.a.mask_esz, describe) : with_geo<false>(R, esz, 0, describe);
  return known ? cudaSuccess : cudaErrorInvalidConfiguration;
}

cudaError_t cps420_launch(const CpsKernelArgs& k, int R, int esz, cudaStream_t s) { return launch420_any<false>(k, R, esz, s); }

cudaError_t cps420_launch_multi(const CpsKernelArgs* d, const int32_t* prefix, int ntiles, int R, int esz, cudaStream_t s)
{
  return launch420_list_any<false>(d, prefix, ntiles, R, esz, 0, s);
}

// Integer keys: with |s'| <= mid + |GCD|, |r'| <= mid, the subtracted terms are at most
// lo = sum w (mid + g)^2 and e less them at most hi = sum w (mid^2 + 2 (mid + g) mid).
bool cps_shared_key(int R, int32_t maxv, const int32_t w[3], const int32_t gmax[3], uint32_t* bias, int32_t* mid)
{
  const int64_t m = ((int64_t)maxv + 1) / 2;
  const int D = 2 * R + 1;
  const int64_t K = (int64_t)1 << cps_key_bits(R);
  long double lo = 0, hi = 0;
  for(int c = 0; c < 3; c++)
  {
    const long double g = gmax[c] < 0 ? -(long double)gmax[c] : (long double)gmax[c];
    lo += (long double)w[c] * (m + g) * (m + g);
    hi += (long double)w[c] * (m * (long double)m + 2 * (m + g) * m);
  }
  const long double top = (long double)K * (lo + hi) + (long double)((3 + 2 * R) * D + 3 + 2 * R);
  const bool ok = w[0] >= 0 && w[1] >= 0 && w[2] >= 0 && top < 4294967295.0L;
  if(bias) { *bias = ok ? (uint32_t)lo : 0u; }
  if(mid) { *mid = (int32_t)m; }
  return ok;
}

// Masked search: a masked sample's keys, masked + P + code, must lie above every real key and below 2^32.
// P lies between K w_0 (mid + g_0)^2 and K (lo + hi_1 + hi_2), with lo and hi as above; the row sums' split
// (kMaskSumSplit) needs differences below 2^13.
bool cps_masked_key(int R, int32_t maxv, const int32_t w[3], const int32_t gmax[3], uint32_t* masked)
{
  if(!cps_shared_key(R, maxv, w, gmax, nullptr, nullptr)) { return false; }
  const int64_t m = ((int64_t)maxv + 1) / 2, D = 2 * R + 1, K = (int64_t)1 << cps_key_bits(R), code = (3 + 2 * R) * D + 3 + 2 * R;
  int64_t lo = 0, hi = 0, hic = 0;   // bounded by cps_shared_key
  bool small = true;
  for(int c = 0; c < 3; c++)
  {
    const int64_t g = gmax[c] < 0 ? -(int64_t)gmax[c] : gmax[c], h = (int64_t)w[c] * (m * m + 2 * (m + g) * m);
    lo += (int64_t)w[c] * (m + g) * (m + g);
    hi += h;
    if(c) { hic += h; }
    small = small && maxv + g < (1 << 13);
  }
  const int64_t g0 = gmax[0] < 0 ? -(int64_t)gmax[0] : gmax[0];
  const int64_t big = K * (lo + hi) + code + 1 - K * (int64_t)w[0] * (m + g0) * (m + g0);
  if(masked) { *masked = (uint32_t)big; }
  return small && big + K * (lo + hic) + code < ((int64_t)1 << 32);
}

}  // namespace qmiv
