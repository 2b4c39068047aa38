// The masked forms of the 4:2:0 search (qmiv_cps420.cuh).
#include "qmiv_cps420.cuh"

namespace qmiv {

cudaError_t launch_cps_masked420(const CpsArgs& a, int R, int esz, cudaStream_t s)
{
  CpsKernelArgs k;
  std::memset(&k, 0, sizeof(k));
  k.a = a;
  k.g.status = const_cast<int32_t*>(&a.gcd_src->flags);
  const cudaError_t e = cps420_describe(k, R, esz, nullptr);
  return e != cudaSuccess ? e : launch420_any<true>(k, R, esz, s);
}

cudaError_t launch_cps_masked420_multi(const void* d_descs, const int32_t* d_prefix, int ntiles, int R, int esz, int mesz, cudaStream_t s)
{
  return launch420_list_any<true>(static_cast<const CpsKernelArgs*>(d_descs), d_prefix, ntiles, R, esz, mesz, s);
}

}  // namespace qmiv
