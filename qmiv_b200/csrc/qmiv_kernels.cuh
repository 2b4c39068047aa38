// Kernel argument blocks and host-side launch wrappers of the QMIV metric kernels.
#pragma once
#include "qmiv_device.cuh"

#include <utility>

namespace qmiv {

// Launches a kernel that begins with wait_for_previous, so that its launch overlaps the end of the kernel
// before it in the stream. Used in calls of one pair where it paid: the finalisers (1920x1080 88 -> 86 us,
// masked 4096x2048 with the mask's totals 190 -> 185) and the moment windows (4096x2048 246 -> 243). It
// cost time before the search (four searches of a mixed batch 1464 -> 1490 us) and before the picture
// windows and their rows (4:4:4 1920x1080 123 -> 130, eight MS-SSIM pairs 1118 -> 1185): those kernels
// are launched plainly, and so are all of a batch, where it gave nothing that could be measured and the launches
// are captured into graphs by several threads.
template <typename... P, typename... A>
cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args)
{
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s; cfg.attrs = &at; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// ---------------------------------------------------------------------------------------------
// prepass: per raw row of every plane SSD, over the planes SD (In1 - In0), SSD and the OR of the samples
// per frame; the last CTA forms the totals, the GCD and the path flags
// ---------------------------------------------------------------------------------------------
struct PrepassArgs
{
  Img       in0, in1;
  int32_t   rows[3];       // raw rows per plane
  int32_t   cols[3];       // raw samples per row per plane
  uint32_t  clip;          // conceal: samples above are clipped (65535 = no clipping)
  uint64_t* row_ssd;       // [rows[0] + rows[1] + rows[2]]
  PairOut*  out;           // zeroed
  int32_t   mult[3];       // 4:4:4 multiplicity of a raw chroma sample (1 << (sx + sy))
  int64_t   area;
  int32_t   maxv;
  int32_t   maxdiff[4];    // round(unc * Max) per component, computed on the host in float
  int32_t   need_gcd;
  int32_t   gcd_override_on;  // use gcd_override instead of the computed GCD
  int32_t   gcd_override[4];
  int32_t   fp32_ok;       // the exact-key CPS path is valid for in-range samples
  int32_t   clip_on;       // conceal active
};

// ---------------------------------------------------------------------------------------------
// CPS search, both directions in one pass
// ---------------------------------------------------------------------------------------------
struct CpsArgs
{
  Img            in0, in1;
  int32_t        W, H;
  int32_t        maxv;
  uint32_t       clip;
  int32_t        wi[3];        // search weights
  float          wf[3];
  int32_t        gmax[3];      // bound of |GCD| per component
  int32_t        key_mid;      // 4:2:0 form: mid value and key bias (set when the pair is described)
  uint32_t       key_bias;
  // masked 4:2:0 search: luma plane of the mask (null = none), its pitch in samples and bytes per
  // sample, the staged value of a masked sample, 64-bit row sums [2][H][3]
  const void*    mask;
  int32_t        mask_pitch, mask_esz;
  uint32_t       key_masked;
  unsigned long long* rows64;
  const PairOut* gcd_src;      // gcd + flags
  uint32_t*      rows;         // [2][H][3], zeroed, 32-bit wrap-around sums
  void*          scp0;         // In0 resampled (T2R search result), planar 3 x W*H, may be null
  void*          scp1;         // In1 resampled (R2T search result)
  // SSIM moments of (test picture, its SCP) per direction, for IV-SSIM without storing the SCP:
  // mom[0] = (In0, SCP1) (T2R), mom[1] = (In1, SCP0) (R2T); null to skip
  Moments        mom[2];
};

// ---------------------------------------------------------------------------------------------
// block SSIM
// ---------------------------------------------------------------------------------------------
// windows of one component of a picture pair, straight from the pictures, and the 2x2 means of both
// for the next MS-SSIM scale
enum { kLoadAny = 0, kLoadRow = 1, kLoadSub = 2 };   // any plane / full-size plane / 4:2:0 chroma
struct SsimImgJob
{
  double      C1, C2;          // (0.01 Max)^2, (0.03 Max)^2 of the pair's bit depth
  const void* a;               // plane of the "Tst" picture of xSSIM::xCalcPicSSIM
  const void* b;               // ... of the "Ref" picture
  double*     win;             // window values [ceil(ny / 32)][nx][32] (pool_win_elems)
  void*       down_a;          // (W >> 1) x (H >> 1), pitch W >> 1, or null
  void*       down_b;
  int32_t     pitch_a, pitch_b;
  int32_t     W, H;            // 4:4:4 size
  int32_t     nx, ny;          // windows per row / column
  uint32_t    clip;
  int8_t      sxa, sya, sxb, syb, load_a, load_b, vec_a, vec_b;
  int8_t      esz, calc_l, wide, down_vec;
};

// MS-SSIM scales 2 .. 4 of one plane from scale 1, each the 2x2 means of the one before (xPixelOpsSTD.cpp:50-67)
struct SsimPyrJob
{
  const void* src;             // scale 1, pitch W
  void*       dst[3];          // scales 2, 3, 4, null where not needed
  int32_t     W, H;            // of scale 1
  int32_t     esz, pad_;
};

// windows from moments, ordered row sums (xSSIM.cpp:353-369), for up to 6 (pair, component) jobs
struct SsimPoolJob
{
  double          C1, C2;      // (0.01 Max)^2, (0.03 Max)^2 of the pair's bit depth
  const uint32_t* mom;         // the five moment planes of one component
  size_t          plane;       // elements between moment planes
  int32_t         pitch;
  int32_t         nx, ny;      // windows per row / column
  int32_t         calc_l;
  int32_t         wide;        // window sums can exceed 32 bits (bit depth > 12)
  int32_t         pad_;
  double*         win;         // window values [ceil(ny / 32)][nx][32] (pool_win_elems)
};

// The launches of one pair's block SSIM family (add_ssim_jobs): windows from the search's moments, windows
// from the pictures at scale 0 and at the smaller scales, the scales between, row sums of all windows.
constexpr int kMaxPoolJobs = 6, kMaxImgJobs0 = 12, kMaxImgJobsN = 36, kMaxPyrJobs = 12, kMaxRowJobs = kMaxPoolJobs + kMaxImgJobs0 + kMaxImgJobsN;
struct SsimRowJob
{
  const double* win;           // [ceil(ny / 32)][nx][32]
  double*       row_sum;       // [ny]
  int32_t       nx, ny;
};
template <typename J, int N> struct JobArgs { J job[N]; };   // by-value form of a launch's jobs
struct SsimJobs
{
  int32_t npool = 0, nimg0 = 0, nimgn = 0, npyr = 0, nrows = 0;
  JobArgs<SsimPoolJob, kMaxPoolJobs> pool;
  JobArgs<SsimImgJob, kMaxImgJobs0>  img0;
  JobArgs<SsimImgJob, kMaxImgJobsN>  imgn;
  JobArgs<SsimPyrJob, kMaxPyrJobs>   pyr;
  JobArgs<SsimRowJob, kMaxRowJobs>   rows;
};
// Largest window grid / plane of the jobs of each launch, over every pair that shares it
struct SsimDims
{
  int pool_nx = 0, pool_ny = 0, img0_nx = 0, img0_ny = 0, imgn_nx = 0, imgn_ny = 0, pyr_w = 0, pyr_h = 0, rows_ny = 0;
  void add(const SsimJobs& q);
};

// ---------------------------------------------------------------------------------------------
// SSIM under any structural similarity option (qmiv_ssim_gen.cu): window values of up to 9
// (picture pair, component) jobs into their band-transposed scratch, then k_ssim_rows
// ---------------------------------------------------------------------------------------------
struct SsimGenJob
{
  Img      a, b;       // a = "Tst", b = "Ref" (xSSIM::xCalcPicSSIM argument order)
  int32_t  comp;
  int32_t  W, H;       // picture size in 4:4:4 samples
  int32_t  x0, y0;     // input position of the first window's top-left sample
  int32_t  nx, ny;     // windows per row / column
  int32_t  calc_l;
  uint32_t clip;       // conceal: samples above are clipped (65535 = no clipping)
  int32_t  esz;        // bytes per sample of a and b
  int32_t  small_range;   // the bit depth's maximum is below 2^14
  const int32_t* flags;   // PairOut::flags: bits 0 and 1 = samples above the maximum
  double   C1, C2;
  double*  win;        // [ceil(ny / 32)][nx][32] (pool_win_elems)
};

constexpr int kGenMaxJobs = 9;
struct SsimGenArgs
{
  int32_t    njobs;
  int32_t    S, border, coef;   // stride, QMIV_BRD_*, offset of the window's coefficients (set by the launcher)
  double     inv;               // scale of the integer sums: 2^-18, 1 / 121 or 1 / N^2 (set by the launcher)
  int32_t    tw, th, cw;        // tile width / height in samples, columns per phase (set by the launcher)
  int32_t    wr;                // window rows per CTA of the row-walking form (set by the launcher)
  SsimGenJob job[kGenMaxJobs];
};

// ---------------------------------------------------------------------------------------------
// finalize: every serial KBNS chain of one frame pair, one thread per chain
// ---------------------------------------------------------------------------------------------
struct SsimSlot
{
  const double* row_sum;       // [3][ny]
  int32_t       nx, ny;
  int32_t       use_ws;        // ERP row weights w[ws_base + ws_step j] (xIVSSIM.cpp:148-165)
  int32_t       ws_base, ws_step;
};

enum { kChainWsPsnr = 0, kChainIvPsnr = 1, kChainSsim = 2 };
struct FinChain
{
  int32_t kind;  // kChain*
  int32_t a, b;  // component / direction / slot
};

struct FinalizeArgs
{
  int32_t         H;
  int32_t         rows[3];
  int32_t         sy[3], mult_row[3];   // 4:4:4 row y of plane c = raw row (y >> sy) times mult_row
  const uint64_t* row_ssd;              // prepass rows
  const double*   ws;                   // [H] equirectangular weights or null
  int32_t         do_wspsnr;
  const uint32_t* cps_rows;             // [2][H][3] or null
  int32_t         nslots;
  SsimSlot        slot[kMaxSsimSlots];
  int32_t         nchains;              // filled by launch_finalize
  FinChain        chain[3 + 6 + 3 * kMaxSsimSlots];
  PairOut*        out;
  PairOut*        host;                 // one pair: pinned host memory the finished results are written to, or null
};

// The pictures, buffers and sizes of one pair's block SSIM family
struct SsimPairArgs
{
  Img      in0, in1, scp0, scp1;   // scp: 4:4:4, where IV-MS-SSIM needs them
  uint32_t mask;
  int32_t  W, H, esz, bitdepth;
  uint32_t clip;
  int32_t  ns;                     // MS-SSIM scales
  int32_t  nx[5], ny[5];
  double   C1, C2;
  int32_t  use_ws;                 // ERP row weights of IV-SSIM
  Moments  mom[2];                 // of the search: (In0, SCP1), (In1, SCP0)
  double*  rowsum;                 // [kMaxSsimSlots][3][ny[0]]
  double*  win;                    // ssim_win_elems doubles
  char*    pyr;                    // scales 1 .. ns - 1 of In0, In1, SCP0, SCP1
};
size_t ssim_win_elems(uint32_t mask, int ns, const int32_t nx[5], const int32_t ny[5]);
void   add_ssim_jobs(const SsimPairArgs& p, SsimJobs& q, FinalizeArgs& fa);

// one (pair, chain) CTA of the multi-pair finalize; chain == nchains of the pair is its exact CPS sums
struct FinJob
{
  int32_t pair, chain;
};
constexpr size_t kFinalizeMaxSmem = 200 * 1024;

// launch wrappers (return cudaError_t of the launch)
template <typename T> cudaError_t launch_prepass(const PrepassArgs& a, cudaStream_t s);
template <typename T> cudaError_t launch_cps(const CpsArgs& a, int R, cudaStream_t s);
// Block SSIM launches of one pair (jobs by value) or of many (job tables in device memory, one after the
// other: pool, img0, imgn, pyr, rows with n entries each)
cudaError_t launch_ssim_jobs(const SsimJobs& q, cudaStream_t s, bool rows_only);
struct SsimTables
{
  const SsimPoolJob* pool = nullptr;
  const SsimImgJob*  img0 = nullptr;
  const SsimImgJob*  imgn = nullptr;
  const SsimPyrJob*  pyr = nullptr;
  const SsimRowJob*  rows = nullptr;
  int npool = 0, nimg0 = 0, nimgn = 0, npyr = 0, nrows = 0;
  SsimDims dims;
};
cudaError_t launch_ssim_tables(const SsimTables& t, cudaStream_t s, bool rows_only);
cudaError_t launch_ssim_rows(const JobArgs<SsimRowJob, kMaxRowJobs>& a, int njobs, cudaStream_t s);   // row sums of ready window values
// SSIM windows of one option set for up to kGenMaxJobs jobs: mode QMIV_SSM_*, window N, stride S,
// border QMIV_BRD_* (regular modes)
cudaError_t launch_ssim_gen(SsimGenArgs& a, int mode, int N, int S, int border, cudaStream_t s);
template <typename T>
cudaError_t launch_downsample2(const Img& a, const Img& b, const MutImg& da, const MutImg& db, int dw, int dh, uint32_t clip,
                               cudaStream_t s);
cudaError_t launch_finalize(const FinalizeArgs& a, cudaStream_t s);
int         finalize_plan(FinalizeArgs& a);          // fills a.chain / a.nchains, returns the CTA count
size_t      finalize_smem(const FinalizeArgs& a);

// multi-pair forms: argument blocks in device memory, one launch for every pair of a batch
template <typename T> cudaError_t launch_prepass_multi(const PrepassArgs* d_jobs, int njobs, int max_rows, cudaStream_t s);
size_t      pool_win_elems(int nx, int ny);   // doubles of the windows of nx x ny
// 16-byte alignment of the moment rows and the scratch, which the pooling kernels copy with cp.async
bool        pool_job_aligned(const SsimPoolJob& J);
cudaError_t launch_finalize_multi(const FinalizeArgs* d_pairs, const FinJob* d_jobs, int njobs, size_t smem, cudaStream_t s);

// CPS work-list form: one 64-byte aligned descriptor (tensor maps + tile geometry) per frame pair,
// pairs grouped by (search range, sample size, tile height); pair p owns work-list tiles
// [prefix[p], prefix[p + 1]).
struct CpsPairPlan
{
  int32_t  ntiles;
  uint32_t raw_bytes;   // raw-box region of the pair
  size_t   smem;        // dynamic shared memory of the pair alone
};
size_t      cps_desc_bytes();
// tile form: kCpsForm420 for 4:2:0, else warps per tile column: 8 (128x32) or 4 (128x16); 0 = none
int         cps_pick_wy(int R, int esz, int sx, int sy);
bool        cps_tile_fits(int R, int wy, int esz, int sx, int sy);
cudaError_t cps_describe(void* desc, const CpsArgs& a, int R, int esz, int wy, CpsPairPlan* plan);
cudaError_t launch_cps_multi(const void* d_descs, const int32_t* d_prefix, int npairs, int ntiles, int R, int wy,
                             int esz, uint32_t raw_cap, size_t smem, cudaStream_t s);

// The masked search of 4:2:0 pictures (CpsArgs::mask set) for one pair, and for a work list of described pairs
cudaError_t launch_cps_masked420(const CpsArgs& a, int R, int esz, cudaStream_t s);
cudaError_t launch_cps_masked420_multi(const void* d_descs, const int32_t* d_prefix, int ntiles, int R, int esz, int mesz, cudaStream_t s);

// Exactness check of the fp32 key path for a given bit depth, weights and GCD clip range.
bool cps_fp32_exact(int32_t maxv, const int32_t w[3], const int32_t maxdiff[3]);
// The same for the integer keys of the 4:2:0 form (qmiv_cps420.cu), with the constants its keys use.
bool cps_shared_key(int R, int32_t maxv, const int32_t w[3], const int32_t gmax[3], uint32_t* bias, int32_t* mid);
// ... and for its masked search.
bool cps_masked_key(int R, int32_t maxv, const int32_t w[3], const int32_t gmax[3], uint32_t* masked);
// Bits of a key below the error: 2^bits lies above the largest raster index.
__host__ __device__ constexpr int cps_key_bits(int R) { return R <= 2 ? 5 : (R == 3 ? 6 : 7); }
// Masked row sums: a lane's four terms d^2 M of a row are below 2^44 (cps_masked_key: |d| < 2^13; any 16-bit M);
// over a warp their parts below and from this bit up, below 2^22 each, are summed apart in 32 bits.
constexpr int kMaskSumSplit = 22;
// ... for the form a picture of these chroma shifts is searched with.
bool cps_key_exact(int R, int sx, int sy, int32_t maxv, const int32_t w[3], const int32_t maxdiff[3]);
// Tile form 1 is the 4:2:0 form; the others are the warps of a tile column.
constexpr int kCpsForm420 = 1;
inline int cps_tile_height(int wy) { return wy == kCpsForm420 ? 16 : 4 * wy; }

}  // namespace qmiv
