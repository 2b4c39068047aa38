// Pieces shared by the two forms of the corresponding-pixel-shift search: the work-list descriptor,
// TMA tile loads with bounded waits, tensor-map encoding and launch helpers (qmiv_cps.cu: any chroma
// format; qmiv_cps420.cuh: 4:2:0).
#pragma once
#include "qmiv_kernels.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <map>
#include <mutex>

namespace qmiv {

constexpr long long kWaitCycles = 1LL << 31; // bound of one tile-load wait (about a second)

struct CpsGeomArgs
{
  int32_t  ntx, ntiles;
  int32_t  use_tma;
  int32_t  ax;                 // 16 bytes in samples: TMA boxes start this far left of the tile
  int32_t  bwl, bhl, bwc, bhc; // raw box sizes in samples (luma, chroma)
  int32_t  sx, sy;             // chroma subsampling shifts
  uint32_t off[2][3];          // byte offsets of the raw boxes in shared memory
  uint32_t raw_bytes;          // raw region, multiple of 128
  uint32_t tx_bytes;           // bytes the six copies of one tile deliver
  int32_t* status;             // PairOut::flags: bit 3 = a tile load did not complete
};

struct alignas(64) CpsKernelArgs
{
  CUtensorMap map[2][3];       // [picture][plane]
  CUtensorMap mask_map;        // masked 4:2:0 search
  CpsArgs     a;
  CpsGeomArgs g;
};

// ---- TMA / mbarrier ---------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar)
{
  asm volatile(
    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
    ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)) : "memory");
}

// Tensor maps written to global memory by a host copy are made visible to the TMA unit
__device__ __forceinline__ void fence_tensormap_acquire(const CUtensorMap* map)
{
  asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map) : "memory");
}

// ---- host -------------------------------------------------------------------------------------
inline PFN_cuTensorMapEncodeTiled_v12000 cps_encode_fn()
{
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
       q == cudaDriverEntryPointSuccess)
    {
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    }
  });
  return fn;
}

// One 2D tensor map per plane. Returns false when TMA cannot take the plane (alignment, pitch).
inline bool cps_encode_plane(CUtensorMap* m, const void* p, int32_t w, int32_t h, int64_t pitch_elems, int esz, int bw, int bh)
{
  const uint64_t pitch = (uint64_t)pitch_elems * (uint64_t)esz;
  if(((uintptr_t)p & 15) != 0 || (pitch & 15) != 0 || pitch >= (1ULL << 40) || w <= 0 || h <= 0) { return false; }
  PFN_cuTensorMapEncodeTiled_v12000 fn = cps_encode_fn();
  if(fn == nullptr) { return false; }
  const cuuint64_t dims[2] = { (cuuint64_t)w, (cuuint64_t)h };
  const cuuint64_t strides[1] = { (cuuint64_t)pitch };
  const cuuint32_t box[2] = { (cuuint32_t)bw, (cuuint32_t)bh };
  const cuuint32_t estr[2] = { 1, 1 };
  const CUresult r = fn(m, esz == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(p),
                        dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

struct DevInfo
{
  int sms = 0, smem_optin = 0;
};
inline DevInfo dev_info(int dev)
{
  static std::mutex mu;
  static DevInfo cache[64];
  std::lock_guard<std::mutex> lk(mu);
  if(dev < 0 || dev >= 64) { return DevInfo{ 1, 48 * 1024 }; }
  if(cache[dev].sms == 0)
  {
    cudaDeviceGetAttribute(&cache[dev].sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&cache[dev].smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if(cache[dev].sms <= 0) { cache[dev].sms = 1; }
  }
  return cache[dev];
}

// Raises the kernel's dynamic shared memory limit once per (kernel, device). The opt-in limit
// covers the kernel's static shared memory (the argument copy) and the dynamic part together.
template <typename F>
cudaError_t configure_once(F* fn, int dev)
{
  static std::mutex mu;
  static std::map<const void*, uint64_t> done;
  const uint64_t bit = 1ULL << (dev & 63);
  std::lock_guard<std::mutex> lk(mu);
  uint64_t& m = done[reinterpret_cast<const void*>(fn)];
  if(m & bit) { return cudaSuccess; }
  cudaFuncAttributes fa{};
  cudaError_t e = cudaFuncGetAttributes(&fa, fn);
  if(e != cudaSuccess) { return e; }
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, dev_info(dev).smem_optin - (int)fa.sharedSizeBytes);
  if(e == cudaSuccess) { m |= bit; }
  return e;
}

template <typename F>
int grid_for(F* fn, int threads, size_t smem, int ntiles, int dev)
{
  int occ = 1;
  if(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, smem) != cudaSuccess || occ < 1) { occ = 1; }
  return std::max(1, std::min(ntiles, dev_info(dev).sms * occ));
}

constexpr int kAlign = 128;
__host__ __device__ constexpr uint32_t align_up(uint32_t v, uint32_t a) { return (v + a - 1) / a * a; }

// ---- the 4:2:0 form (qmiv_cps420.cuh) ----------------------------------------------------------
bool        cps420_fits(int R, int esz);
int         cps420_tiles(int W, int H);
cudaError_t cps420_describe(CpsKernelArgs& k, int R, int esz, CpsPairPlan* plan);
cudaError_t cps420_launch(const CpsKernelArgs& k, int R, int esz, cudaStream_t s);
cudaError_t cps420_launch_multi(const CpsKernelArgs* d, const int32_t* prefix, int ntiles, int R, int esz, cudaStream_t s);

}  // namespace qmiv
