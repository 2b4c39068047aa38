// Block SSIM (8x8 windows at stride 4, xSSIM.cpp:276-369, xStructSimSTD.cpp:420-461) on B200.
//
// Window moments are sums of 2x2 exact integer 4x4 sub-block moments. For IV-SSIM they come from the CPS
// search's epilogue (test picture vs its shift-compensated picture, so the SCP never needs to be stored;
// k_ssim_win); for plain SSIM and the MS-SSIM scales k_ssim_img forms them in shared memory from the
// pictures themselves, evaluates the windows there and writes the next scale's 2x2 means
// (xPixelOpsSTD.cpp:50-67) on the way: no moment planes in device memory. k_ssim_pyr makes the scales
// below from the first of them, so that one launch takes the windows of all smaller scales. Windows are
// evaluated in FP64 with the reference's operation order; k_ssim_rows forms the compensated sum of each
// window row, all scales and pairs in one launch.
// Measured against moment planes in device memory and three launches per scale: 8 pairs of 2048x2048 10-bit,
// MS-SSIM and IV-MS-SSIM, 827 -> 523 us of device time; one 1998x1080 12-bit pair, every metric, 33 -> 9
// launches and 262 -> 98 us. What bounds k_ssim_img: load latency and issue (58 % at 32 warps per SM; 4 CTAs
// of 8 warps measured 478 us for the windows above, 3 and 5 CTAs 525 and 539, 5 CTAs of 4 warps 765).
#include "qmiv_host.h"

#include <type_traits>

namespace qmiv {

// =============================================================================================
// windows + row sums (xSSIM.cpp:353-369), two kernels:
//   k_ssim_win   a CTA (eight warps) evaluates the windows [x0, x0 + 64) of one band of 32 window rows.
//                The 33 block rows x 68 columns of the five moment planes it needs (45 KB) are staged
//                in shared memory by cp.async, all in flight at once. Lane l then takes columns
//                x0 + l and x0 + 32 + l and walks its warp's 4 window rows: block row r gives the
//                horizontal pair sums h(r) = m(r, x) + m(r, x + 1), window (x, r - 1) is h(r - 1) + h(r).
//                Each window is evaluated in FP64 with the reference's operation order; the 64 x 32
//                values reuse the staging space and leave as 16 contiguous KB of the job's scratch
//                [band][x][32].
//   k_ssim_rows  a CTA per band of 32 window rows forms their sums (ExactSum).
// =============================================================================================
constexpr int kWinX = 64;                                  // windows per CTA in x
constexpr int kWinNT = 256;                                // threads per CTA
constexpr int kWinRows = 32 / (kWinNT / 32);               // window rows per warp
constexpr int kWinOcc = 5, kImgOcc = 4;                    // CTAs per SM of k_ssim_win and k_ssim_img
constexpr int kStRows = 33;                                // block rows of a band
constexpr int kStCols = 68;                                // block columns staged (65 used), 16-byte pieces
constexpr int kStPieces = kStCols / 4;
constexpr int kRowWarps = 8;                               // of k_ssim_rows
static_assert(kWinX * 33 * sizeof(double) <= 5 * kStRows * kStCols * sizeof(uint32_t), "values fit the staging space");

size_t pool_win_elems(int nx, int ny) { return (size_t)((ny + 31) / 32) * 32 * (size_t)nx; }

bool pool_job_aligned(const SsimPoolJob& J)
{
  return ((uintptr_t)J.mom & 15) == 0 && (J.pitch & 3) == 0 && (J.plane & 3) == 0 && ((uintptr_t)J.win & 15) == 0;
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// v / 64 for an integer v < 2^52, exactly: 2^46 + v 2^-6 is the double whose mantissa field is v
// and whose exponent is 46, and removing 2^46 is exact. Equals (double)v * (1.0 / 64).
template <typename S>
__device__ __forceinline__ double div64_exact(S v)
{
  const uint32_t hi = 0x42D00000u | (uint32_t)((uint64_t)v >> 32);
  return dsub(__hiloint2double((int)hi, (int)(uint32_t)v), 70368744177664.0);
}

// The windows of one thread: columns x0 + l and x0 + 32 + l, the warp's rows.
// The fields of a pool job one CTA of k_ssim_win uses, read once into registers.
struct WinJob
{
  double C1, C2;
  int    nx, ny, calc_l;
};

template <bool WIDE>
__device__ __forceinline__ void ssim_win_eval(const WinJob& J, const uint32_t (*st)[kStRows][kStCols], int x0, int band,
                                              double v[2][kWinRows])
{
  using S = typename std::conditional<WIDE, uint64_t, uint32_t>::type;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int r0 = warp * kWinRows;                           // the warp's first block row in the band
  const int nrow = min(kWinRows, J.ny - band * 32 - r0);    // window rows of this warp (may be <= 0)
  #pragma unroll
  for(int h = 0; h < 2; h++)
  {
    const int xl = 32 * h + lane;
    const bool xin = x0 + xl < J.nx;
    S hp[5] = { 0, 0, 0, 0, 0 };
    #pragma unroll
    for(int k = 0; k <= kWinRows; k++)
    {
      const bool live = xin && k <= nrow;                   // block row r0 + k was staged
      S hc[5];
      #pragma unroll
      for(int m = 0; m < 5; m++) { hc[m] = live ? (S)st[m][r0 + k][xl] + (S)st[m][r0 + k][xl + 1] : (S)0; }
      if(k > 0)
      {
        double r = 0.0;
        if(live)
        {
          // moment 0/2 = "Tst" picture, 1/3 = "Ref" picture (xStructSimSTD.cpp:420-461)
          const double at = div64_exact<S>(hp[0] + hc[0]), ar = div64_exact<S>(hp[1] + hc[1]);
          const double qt = div64_exact<S>(hp[2] + hc[2]), qr = div64_exact<S>(hp[3] + hc[3]);
          const double qrt = div64_exact<S>(hp[4] + hc[4]);
          r = ssim_window_avg(ar, at, qr, qt, qrt, J.C1, J.C2, J.calc_l != 0);
        }
        v[h][k - 1] = r;
      }
      #pragma unroll
      for(int m = 0; m < 5; m++) { hp[m] = hc[m]; }
    }
  }
}

// The CTA's windows from the staged sub-block moments, which all threads have written.
__device__ __forceinline__ void ssim_win_finish(const WinJob& J, uint32_t (*st)[kStRows][kStCols], bool wide, double* win, int x0, int band)
{
  __syncthreads();
  double v[2][kWinRows];
  if(wide) { ssim_win_eval<true>(J, st, x0, band, v); }
  else { ssim_win_eval<false>(J, st, x0, band, v); }
  __syncthreads();                                          // the staging space becomes the values
  double (*vals)[33] = reinterpret_cast<double (*)[33]>(&st[0][0][0]);   // [x][row in band]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  #pragma unroll
  for(int h = 0; h < 2; h++)
  {
    #pragma unroll
    for(int k = 0; k < kWinRows; k++) { vals[32 * h + lane][warp * kWinRows + k] = v[h][k]; }
  }
  __syncthreads();
  const int n = min(kWinX, J.nx - x0) * 32;
  double* out = win + ((size_t)band * J.nx + x0) * 32;      // this tile's columns are contiguous
  for(int e = threadIdx.x; e < n; e += kWinNT) { out[e] = vals[e >> 5][e & 31]; }
}

__device__ __forceinline__ void ssim_win_body(const SsimPoolJob& Jg, uint32_t (*st)[kStRows][kStCols], int tile_x, int band)
{
  const WinJob J{ Jg.C1, Jg.C2, Jg.nx, Jg.ny, Jg.calc_l };
  const int x0 = tile_x * kWinX, j0 = band * 32;
  if(x0 >= J.nx || j0 >= J.ny) { return; }                 // uniform over the CTA
  const uint32_t* mom = Jg.mom;
  const size_t plane = Jg.plane;
  const int pitch = Jg.pitch;
  // block rows j0 .. min(j0 + 32, ny) exist (ny + 1 block rows); 16-byte pieces that start inside
  // the padded row (pitch, a multiple of 4 columns) end inside it. Piece q = (m, r, c) walks in steps
  // of kWinNT.
  static_assert(kStRows * kStPieces > kWinNT, "a step stays within two planes");
  const int nrows = min(kStRows, J.ny + 1 - j0);
  int m = 0, r = threadIdx.x / kStPieces, c = threadIdx.x - r * kStPieces;
  for(int q = threadIdx.x; q < 5 * kStRows * kStPieces; q += kWinNT)
  {
    if(r < nrows && x0 + 4 * c < pitch)
    {
      cp_async16(&st[m][r][4 * c], mom + (size_t)m * plane + (size_t)(j0 + r) * pitch + x0 + 4 * c);
    }
    r += kWinNT / kStPieces; c += kWinNT % kStPieces;
    if(c >= kStPieces) { c -= kStPieces; r++; }
    if(r >= kStRows) { r -= kStRows; m++; }
  }
  cp_async_commit();
  cp_async_wait<0>();
  ssim_win_finish(J, st, Jg.wide != 0, Jg.win, x0, band);
}

// The samples of one 4x4 block of a plane: 16, or the 4 samples of 4:2:0 chroma that stand for 2x2 pixels
// each. All accesses resolve at compile time.
template <int MODE>
struct Block
{
  static constexpr bool SUB = MODE == kLoadSub;
  static constexpr int N = SUB ? 4 : 16;
  uint32_t v[N];
  // sum of the pixels of 2x2 quad q = 2 (y / 2) + x / 2
  __device__ __forceinline__ uint32_t quad(int q) const
  {
    const int k = 8 * (q >> 1) + 2 * (q & 1);
    return SUB ? 4u * v[q] : (v[k] + v[k + 1]) + (v[k + 4] + v[k + 5]);
  }
};

// VEC: rows of the plane start on 4-sample (kLoadRow) or 2-sample (kLoadSub) boundaries
template <typename T, int MODE, bool VEC>
__device__ __forceinline__ Block<MODE> load_block(const void* plane, int pitch, int sx, int sy, int bx, int by, int W, int H, uint32_t clip)
{
  Block<MODE> B;
  const T* p = static_cast<const T*>(plane);
  if constexpr(MODE == kLoadRow)
  {
    const T* q = p + (size_t)(4 * by) * pitch + 4 * bx;
    #pragma unroll
    for(int y = 0; y < 4; y++, q += pitch)
    {
      if constexpr(!VEC)
      {
        #pragma unroll
        for(int x = 0; x < 4; x++) { B.v[4 * y + x] = __ldg(q + x); }
      }
      else if constexpr(sizeof(T) == 2)
      {
        const uint2 w = __ldg(reinterpret_cast<const uint2*>(q));
        B.v[4 * y] = w.x & 0xffffu; B.v[4 * y + 1] = w.x >> 16; B.v[4 * y + 2] = w.y & 0xffffu; B.v[4 * y + 3] = w.y >> 16;
      }
      else
      {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(q));
        B.v[4 * y] = w & 0xffu; B.v[4 * y + 1] = (w >> 8) & 0xffu; B.v[4 * y + 2] = (w >> 16) & 0xffu; B.v[4 * y + 3] = w >> 24;
      }
    }
  }
  else if constexpr(MODE == kLoadSub)
  {
    const T* q = p + (size_t)(2 * by) * pitch + 2 * bx;
    #pragma unroll
    for(int h = 0; h < 2; h++, q += pitch)
    {
      if constexpr(!VEC) { B.v[2 * h] = __ldg(q); B.v[2 * h + 1] = __ldg(q + 1); }
      else if constexpr(sizeof(T) == 2) { const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(q)); B.v[2 * h] = w & 0xffffu; B.v[2 * h + 1] = w >> 16; }
      else { const uint32_t w = __ldg(reinterpret_cast<const uint16_t*>(q)); B.v[2 * h] = w & 0xffu; B.v[2 * h + 1] = w >> 8; }
    }
  }
  else
  {
    #pragma unroll
    for(int y = 0; y < 4; y++)
    {
      const T* q = p + (size_t)(min(4 * by + y, H - 1) >> sy) * pitch;
      #pragma unroll
      for(int x = 0; x < 4; x++) { B.v[4 * y + x] = min((uint32_t)__ldg(q + (min(4 * bx + x, W - 1) >> sx)), clip); }
    }
  }
  return B;
}

template <int MODE>
__device__ __forceinline__ uint32_t sum_of_squares(const Block<MODE>& B)
{
  uint32_t s = 0;
  #pragma unroll
  for(int k = 0; k < Block<MODE>::N; k++) { s += B.v[k] * B.v[k]; }
  return Block<MODE>::SUB ? 4u * s : s;
}

// 2x2 means of a 4x4 block from its quad sums, pairs packed where the rows allow it
template <typename T>
__device__ __forceinline__ void store_down(void* down, const uint32_t q[4], int bx, int by, int dw, int dh, bool vec)
{
  #pragma unroll
  for(int y = 0; y < 2; y++)
  {
    const uint32_t m0 = (q[2 * y] + 2) >> 2, m1 = (q[2 * y + 1] + 2) >> 2;
    T* d = static_cast<T*>(down) + (size_t)(2 * by + y) * dw + 2 * bx;
    if(vec)
    {
      if constexpr(sizeof(T) == 2) { *reinterpret_cast<uint32_t*>(d) = m0 | (m1 << 16); }
      else { *reinterpret_cast<uint16_t*>(d) = (uint16_t)(m0 | (m1 << 8)); }
    }
    else if(2 * by + y < dh)
    {
      if(2 * bx < dw) { d[0] = (T)m0; }
      if(2 * bx + 1 < dw) { d[1] = (T)m1; }
    }
  }
}

// Sub-block moments (and 2x2 means) of the CTA's tile of windows: a thread per 4x4 block of its 65 x 33, all
// inside the picture. The blocks shared with the neighbouring tiles, 5 %, are read by both.
template <typename T, int MA, int MB, bool VEC>
__device__ __forceinline__ void ssim_img_stage(const SsimImgJob& Jg, uint32_t (*st)[kStRows][kStCols], int x0, int j0, int ncol, int nrow)
{
  const SsimImgJob J = Jg;                                  // in registers: the stores below could alias a table
  const int dr = kWinNT / ncol, dc = kWinNT - dr * ncol;
  int r = (int)threadIdx.x / ncol, c = (int)threadIdx.x - r * ncol;
  #pragma unroll 1
  while(r < nrow)
  {
    const int bx = x0 + c, by = j0 + r;
    const Block<MA> A = load_block<T, MA, VEC>(J.a, J.pitch_a, J.sxa, J.sya, bx, by, J.W, J.H, J.clip);
    const Block<MB> B = load_block<T, MB, VEC>(J.b, J.pitch_b, J.sxb, J.syb, bx, by, J.W, J.H, J.clip);
    uint32_t qa[4], qb[4], ab = 0;
    #pragma unroll
    for(int q = 0; q < 4; q++) { qa[q] = A.quad(q); qb[q] = B.quad(q); }
    if constexpr(Block<MA>::SUB || Block<MB>::SUB)
    {
      // a sample that stands for a quad multiplies the other picture's quad sum
      #pragma unroll
      for(int q = 0; q < 4; q++) { ab += Block<MA>::SUB ? A.v[q] * qb[q] : qa[q] * B.v[q]; }
    }
    else
    {
      #pragma unroll
      for(int k = 0; k < 16; k++) { ab += A.v[k] * B.v[k]; }
    }
    st[0][r][c] = (qa[0] + qa[1]) + (qa[2] + qa[3]);
    st[1][r][c] = (qb[0] + qb[1]) + (qb[2] + qb[3]);
    st[2][r][c] = sum_of_squares(A);
    st[3][r][c] = sum_of_squares(B);
    st[4][r][c] = ab;
    // the tile's own blocks (in the last tile of a row or column there is no neighbour to write the rest)
    if((c < kWinX || x0 + kWinX >= J.nx) && (r < 32 || j0 + 32 >= J.ny))
    {
      if(J.down_a) { store_down<T>(J.down_a, qa, bx, by, J.W >> 1, J.H >> 1, J.down_vec != 0); }
      if(J.down_b) { store_down<T>(J.down_b, qb, bx, by, J.W >> 1, J.H >> 1, J.down_vec != 0); }
    }
    r += dr; c += dc;
    if(c >= ncol) { c -= ncol; r++; }
  }
}

// 2x2 means of the blocks that reach past the picture, in the last tiles: block columns [ncol, ncol_all) and
// block rows [nrow, nrow_all).
template <typename T>
__device__ __forceinline__ void ssim_img_rest(const SsimImgJob& J, int x0, int j0, int ncol, int nrow, int ncol_all, int nrow_all)
{
  for(int q = threadIdx.x; q < ncol_all * nrow_all; q += kWinNT)
  {
    const int r = q / ncol_all, c = q - r * ncol_all;
    if(r < nrow && c < ncol) { continue; }
    uint32_t s[4];
    #pragma unroll 1
    for(int k = 0; k < 2; k++)
    {
      void* down = k ? J.down_b : J.down_a;
      if(!down) { continue; }
      const Block<kLoadAny> B = load_block<T, kLoadAny, false>(k ? J.b : J.a, k ? J.pitch_b : J.pitch_a, k ? J.sxb : J.sxa, k ? J.syb : J.sya,
                                                        x0 + c, j0 + r, J.W, J.H, J.clip);
      #pragma unroll
      for(int i = 0; i < 4; i++) { s[i] = B.quad(i); }
      store_down<T>(down, s, x0 + c, j0 + r, J.W >> 1, J.H >> 1, false);
    }
  }
}

// Windows [64 tile_x, + 64) of band 32 band from the pictures.
template <typename T>
__device__ __forceinline__ void ssim_img_body(const SsimImgJob& J, uint32_t (*st)[kStRows][kStCols], int tile_x, int band)
{
  const int x0 = tile_x * kWinX, j0 = band * 32;
  const bool last_x = x0 + kWinX >= J.nx, last_y = j0 + 32 >= J.ny;
  const int ncol = last_x ? J.W / 4 - x0 : kWinX + 1, nrow = last_y ? J.H / 4 - j0 : 33;   // whole blocks, nx + 1 and ny + 1 at most
  const bool clip = J.clip < (sizeof(T) == 1 ? 0xffu : 0xffffu);                            // conceal: the general loads clip
  const int form = clip ? 0 : J.load_a == kLoadRow && J.load_b == kLoadRow ? 1 : J.load_a == kLoadSub && J.load_b == kLoadSub ? 2
                 : J.load_a == kLoadSub && J.load_b == kLoadRow ? 3 : 0;
  switch(2 * form + (J.vec_a && J.vec_b ? 1 : 0))
  {
  case 2: ssim_img_stage<T, kLoadRow, kLoadRow, false>(J, st, x0, j0, ncol, nrow); break;
  case 3: ssim_img_stage<T, kLoadRow, kLoadRow, true>(J, st, x0, j0, ncol, nrow); break;
  case 4: ssim_img_stage<T, kLoadSub, kLoadSub, false>(J, st, x0, j0, ncol, nrow); break;
  case 5: ssim_img_stage<T, kLoadSub, kLoadSub, true>(J, st, x0, j0, ncol, nrow); break;
  case 6: ssim_img_stage<T, kLoadSub, kLoadRow, false>(J, st, x0, j0, ncol, nrow); break;
  case 7: ssim_img_stage<T, kLoadSub, kLoadRow, true>(J, st, x0, j0, ncol, nrow); break;
  default: ssim_img_stage<T, kLoadAny, kLoadAny, false>(J, st, x0, j0, ncol, nrow); break;
  }
  if((last_x || last_y) && (J.down_a || J.down_b) && (J.W % 4 != 0 || J.H % 4 != 0))
  {
    ssim_img_rest<T>(J, x0, j0, ncol, nrow, last_x ? (J.W + 3) / 4 - x0 : kWinX, last_y ? (J.H + 3) / 4 - j0 : 32);
  }
  const WinJob Jw{ J.C1, J.C2, J.nx, J.ny, J.calc_l };
  ssim_win_finish(Jw, st, J.wide != 0, J.win, x0, band);
}

// Scales 2, 3, 4 of one plane: a CTA takes 128 x 64 samples of scale 1 (with 32 x 32 the launch of the 8-pair
// 2048x2048 workload took 132 us for its 200 MB, bound by the number of CTAs).
constexpr int kPyrW = 64, kPyrH = 32;                       // samples of scale 2 per CTA
template <typename T>
__device__ __forceinline__ void ssim_pyr_body(const SsimPyrJob& J, uint16_t (*l2)[kPyrW], uint16_t (*l3)[kPyrW / 2], int bx, int by)
{
  const T* src = static_cast<const T*>(J.src);
  const int W = J.W;
  if(J.dst[0] == nullptr) { return; }
  {
    const int w = W >> 1, h = J.H >> 1;
    const int lx = threadIdx.x % kPyrW, x = bx * kPyrW + lx;
    const bool pairs = (W & 1) == 0 && (reinterpret_cast<uintptr_t>(src) & (2 * sizeof(T) - 1)) == 0;   // two samples per load
    uint32_t v[kPyrH / 4];
    #pragma unroll
    for(int i = 0; i < kPyrH / 4; i++)
    {
      const int y = by * kPyrH + threadIdx.x / kPyrW + 4 * i;
      v[i] = 0;
      if(x < w && y < h)
      {
        const T* p = src + (size_t)(2 * y) * W + 2 * x;
        if(!pairs) { v[i] = (uint32_t)__ldg(p) + __ldg(p + 1) + __ldg(p + W) + __ldg(p + W + 1); }
        else if constexpr(sizeof(T) == 2)
        {
          const uint32_t a = __ldg(reinterpret_cast<const uint32_t*>(p)), b = __ldg(reinterpret_cast<const uint32_t*>(p + W));
          v[i] = (a & 0xffffu) + (a >> 16) + (b & 0xffffu) + (b >> 16);
        }
        else
        {
          const uint32_t a = __ldg(reinterpret_cast<const uint16_t*>(p)), b = __ldg(reinterpret_cast<const uint16_t*>(p + W));
          v[i] = (a & 0xffu) + (a >> 8) + (b & 0xffu) + (b >> 8);
        }
      }
    }
    #pragma unroll
    for(int i = 0; i < kPyrH / 4; i++)
    {
      const int ly = threadIdx.x / kPyrW + 4 * i, y = by * kPyrH + ly;
      const uint32_t m = (v[i] + 2) >> 2;
      l2[ly][lx] = (uint16_t)m;
      if(x < w && y < h) { static_cast<T*>(J.dst[0])[(size_t)y * w + x] = (T)m; }
    }
  }
  if(J.dst[1] == nullptr) { return; }                       // uniform
  __syncthreads();
  const int w3 = W >> 2, h3 = J.H >> 2;
  for(int q = threadIdx.x; q < kPyrW * kPyrH / 4; q += 256)
  {
    const int ly = q / (kPyrW / 2), lx = q % (kPyrW / 2);
    const int x = bx * (kPyrW / 2) + lx, y = by * (kPyrH / 2) + ly;
    const uint32_t m = ((uint32_t)l2[2 * ly][2 * lx] + l2[2 * ly][2 * lx + 1] + l2[2 * ly + 1][2 * lx] + l2[2 * ly + 1][2 * lx + 1] + 2) >> 2;
    l3[ly][lx] = (uint16_t)m;
    if(x < w3 && y < h3) { static_cast<T*>(J.dst[1])[(size_t)y * w3 + x] = (T)m; }
  }
  if(J.dst[2] == nullptr) { return; }
  __syncthreads();
  const int w4 = W >> 3, h4 = J.H >> 3;
  if(threadIdx.x < kPyrW * kPyrH / 16)
  {
    const int ly = threadIdx.x / (kPyrW / 4), lx = threadIdx.x % (kPyrW / 4);
    const int x = bx * (kPyrW / 4) + lx, y = by * (kPyrH / 4) + ly;
    const uint32_t m = ((uint32_t)l3[2 * ly][2 * lx] + l3[2 * ly][2 * lx + 1] + l3[2 * ly + 1][2 * lx] + l3[2 * ly + 1][2 * lx + 1] + 2) >> 2;
    if(x < w4 && y < h4) { static_cast<T*>(J.dst[2])[(size_t)y * w4 + x] = (T)m; }
  }
}

__device__ __forceinline__ void ssim_img_any(const SsimImgJob& J, int tile_x, int band)
{
  __shared__ __align__(16) uint32_t st[5][kStRows][kStCols];
  if(tile_x * kWinX >= J.nx || band * 32 >= J.ny) { return; }   // uniform over the CTA
  if(J.esz == 1) { ssim_img_body<uint8_t>(J, st, tile_x, band); }
  else { ssim_img_body<uint16_t>(J, st, tile_x, band); }
}

__device__ __forceinline__ void ssim_pyr_any(const SsimPyrJob& J, int bx, int by)
{
  __shared__ uint16_t l2[kPyrH][kPyrW], l3[kPyrH / 2][kPyrW / 2];
  if(bx * 2 * kPyrW >= J.W || by * 2 * kPyrH >= J.H) { return; }
  if(J.esz == 1) { ssim_pyr_body<uint8_t>(J, l2, l3, bx, by); }
  else { ssim_pyr_body<uint16_t>(J, l2, l3, bx, by); }
}

// Sums of the window values along the rows: a CTA per band of 32 rows, a lane per row, the columns dealt to
// the warps. A column of a band is 256 contiguous bytes. Bound by the latency of the loads with few bands and
// by reading the values from memory with many: with one warp per band, summing in order behind copies
// into shared memory, 25 us for the six evaluations of a 4096x2048 pair and 40 for eight pairs (200 MB); now
// 12.6 and 42.6. With 16 warps 12.7 and 45.4, with 4 21 and 43, with eight loads in flight 14.7 and 49.9.
__device__ __forceinline__ void ssim_rows_body(const SsimRowJob& J, int band)
{
  __shared__ ExactSum part[kRowWarps / 2][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if(band * 32 >= J.ny) { return; }                         // uniform over the CTA
  const double* src = J.win + (size_t)band * J.nx * 32 + lane;
  constexpr int U = 16;                                     // loads in flight per thread
  ExactSum sum;
  for(int x0 = warp; x0 < J.nx; x0 += U * kRowWarps)
  {
    double v[U];
    #pragma unroll
    for(int u = 0; u < U; u++) { const int x = x0 + u * kRowWarps; v[u] = x < J.nx ? src[(size_t)x * 32] : 0.0; }
    #pragma unroll
    for(int u = 0; u < U; u++) { sum.add(v[u]); }
  }
  #pragma unroll
  for(int half = kRowWarps / 2; half > 0; half >>= 1)        // warps in [half, 2 half) hand theirs over
  {
    if(warp >= half) { if(warp < 2 * half) { part[warp - half][lane] = sum; } }
    __syncthreads();
    if(warp < half) { sum.join(part[warp][lane]); }
    if(half > 1) { __syncthreads(); }
  }
  if(warp != 0) { return; }
  const int j = band * 32 + lane;
  const bool valid = j < J.ny;                              // rows past the last one hold zeros or nothing
  double r = sum.result();
  if(__any_sync(0xffffffffu, valid && !sum.exact(J.nx)))
  {
    Kbns row;                                               // the chain in order, loads ahead of it
    for(int x0 = 0; x0 < J.nx; x0 += 16)
    {
      double v[16];
      #pragma unroll
      for(int u = 0; u < 16; u++) { v[u] = x0 + u < J.nx ? src[(size_t)(x0 + u) * 32] : 0.0; }
      #pragma unroll
      for(int u = 0; u < 16; u++) { if(x0 + u < J.nx) { row.add(v[u]); } }
    }
    r = row.result();
  }
  if(valid) { J.row_sum[j] = r; }
}

// Every kernel takes its jobs by value (one pair) or from a table in device memory. The job is the fastest
// grid dimension of the picture kernels, so that the evaluations that share a picture read its tiles close
// together in time, and of every table kernel: a pair has up to 54 jobs, and only the first grid dimension goes
// past 65535.
__device__ __forceinline__ void ssim_win_any(const SsimPoolJob& J, int tile_x, int band)
{
  __shared__ __align__(16) uint32_t st[5][kStRows][kStCols];
  ssim_win_body(J, st, tile_x, band);
}
__global__ void __launch_bounds__(kWinNT, kWinOcc) k_ssim_win(const __grid_constant__ JobArgs<SsimPoolJob, kMaxPoolJobs> a) { wait_for_previous(); ssim_win_any(a.job[blockIdx.z], blockIdx.x, blockIdx.y); }
__global__ void __launch_bounds__(kWinNT, kWinOcc) k_ssim_win_multi(const SsimPoolJob* __restrict__ jobs) { ssim_win_any(jobs[blockIdx.x], blockIdx.y, blockIdx.z); }
template <int N>
__global__ void __launch_bounds__(kWinNT, kImgOcc) k_ssim_img(const __grid_constant__ JobArgs<SsimImgJob, N> a) { ssim_img_any(a.job[blockIdx.x], blockIdx.y, blockIdx.z); }
__global__ void __launch_bounds__(kWinNT, kImgOcc) k_ssim_img_multi(const SsimImgJob* __restrict__ jobs) { ssim_img_any(jobs[blockIdx.x], blockIdx.y, blockIdx.z); }
__global__ void __launch_bounds__(256) k_ssim_pyr(const __grid_constant__ JobArgs<SsimPyrJob, kMaxPyrJobs> a) { ssim_pyr_any(a.job[blockIdx.z], blockIdx.x, blockIdx.y); }
__global__ void __launch_bounds__(256) k_ssim_pyr_multi(const SsimPyrJob* __restrict__ jobs) { ssim_pyr_any(jobs[blockIdx.x], blockIdx.y, blockIdx.z); }
__global__ void __launch_bounds__(32 * kRowWarps, 3) k_ssim_rows(const __grid_constant__ JobArgs<SsimRowJob, kMaxRowJobs> a) { next_may_start(); ssim_rows_body(a.job[blockIdx.y], blockIdx.x); }
__global__ void __launch_bounds__(32 * kRowWarps, 3) k_ssim_rows_multi(const SsimRowJob* __restrict__ jobs) { ssim_rows_body(jobs[blockIdx.x], blockIdx.y); }

// ---- host ---------------------------------------------------------------------------------------
static int tiles_of(int nx) { return (nx + kWinX - 1) / kWinX; }
static int bands_of(int ny) { return (ny + 31) / 32; }

void SsimDims::add(const SsimJobs& q)
{
  for(int k = 0; k < q.npool; k++) { pool_nx = max(pool_nx, q.pool.job[k].nx); pool_ny = max(pool_ny, q.pool.job[k].ny); }
  for(int k = 0; k < q.nimg0; k++) { img0_nx = max(img0_nx, q.img0.job[k].nx); img0_ny = max(img0_ny, q.img0.job[k].ny); }
  for(int k = 0; k < q.nimgn; k++) { imgn_nx = max(imgn_nx, q.imgn.job[k].nx); imgn_ny = max(imgn_ny, q.imgn.job[k].ny); }
  for(int k = 0; k < q.npyr; k++) { pyr_w = max(pyr_w, q.pyr.job[k].W); pyr_h = max(pyr_h, q.pyr.job[k].H); }
  for(int k = 0; k < q.nrows; k++) { rows_ny = max(rows_ny, q.rows.job[k].ny); }
}

size_t ssim_win_elems(uint32_t mask, int ns, const int32_t nx[5], const int32_t ny[5])
{
  const int at0 = ((mask & QMIV_IVSSIM) ? 2 : 0) + ((mask & QMIV_SSIM) ? 1 : 0);
  const int per_scale = ((mask & QMIV_MSSSIM) ? 1 : 0) + ((mask & QMIV_IVMSSSIM) ? 2 : 0);
  size_t n = (size_t)3 * at0 * pool_win_elems(nx[0], ny[0]);
  for(int s = 0; per_scale && s < ns; s++) { n += (size_t)3 * per_scale * pool_win_elems(nx[s], ny[s]); }
  return n;
}

// How the 4x4 blocks of a plane are loaded, and whether its rows allow the vector loads of that form.
static void load_mode(const Img& im, int c, int esz, int8_t& mode, int8_t& vec)
{
  mode = im.sx[c] == 0 && im.sy[c] == 0 ? kLoadRow : im.sx[c] == 1 && im.sy[c] == 1 ? kLoadSub : kLoadAny;
  const int n = mode == kLoadRow ? 4 : 2;
  vec = reinterpret_cast<uintptr_t>(im.p[c]) % (size_t)(n * esz) == 0 && im.pitch[c] % n == 0 ? 1 : 0;
}

// Jobs of one pair: IV-SSIM windows from the search's moments, plain SSIM at scale 0, MS-SSIM and IV-MS-SSIM
// at every scale (xSSIM.cpp:199-256, xIVSSIM.cpp:31-92), each picture's next scale written by the first
// evaluation that reads it.
void add_ssim_jobs(const SsimPairArgs& p, SsimJobs& q, FinalizeArgs& fa)
{
  double* win = p.win;
  auto out = [&](int scale, int slot, int c) -> double* {
    double* w = win;
    win += pool_win_elems(p.nx[scale], p.ny[scale]);
    SsimRowJob& R = q.rows.job[q.nrows++];
    R.win = w; R.nx = p.nx[scale]; R.ny = p.ny[scale];
    R.row_sum = p.rowsum + (size_t)slot * 3 * p.ny[0] + (size_t)c * p.ny[scale];   // finalize reads [c][ny of the scale]
    return w;
  };
  auto slot_of = [&](int scale, int slot, int use_ws) {
    SsimSlot& s = fa.slot[slot];
    s.row_sum = p.rowsum + (size_t)slot * 3 * p.ny[0];
    s.nx = p.nx[scale]; s.ny = p.ny[scale]; s.use_ws = use_ws;
    s.ws_base = 4; s.ws_step = 4;                           // window row j covers rows 4j .. 4j + 7 (xIVSSIM.cpp:153)
  };
  auto add_moments = [&](const Moments& m, int slot) {
    for(int c = 0; c < 3; c++)
    {
      SsimPoolJob& J = q.pool.job[q.npool++];
      J.C1 = p.C1; J.C2 = p.C2; J.mom = m.p + (size_t)c * 5 * m.plane(); J.plane = m.plane(); J.pitch = m.pitch;
      J.nx = p.nx[0]; J.ny = p.ny[0]; J.calc_l = 1; J.wide = p.bitdepth > 12 ? 1 : 0; J.pad_ = 0;
      J.win = out(0, slot, c);
    }
    slot_of(0, slot, p.use_ws);
  };
  size_t lv = 0;
  for(int s = 1; s < p.ns; s++) { lv += (size_t)(p.W >> s) * (p.H >> s) * 3; }
  auto level = [&](int img, int scale, int c) -> char* {    // plane c of picture img at a scale >= 1
    size_t o = (size_t)img * lv;
    for(int s = 1; s < scale; s++) { o += (size_t)(p.W >> s) * (p.H >> s) * 3; }
    return p.pyr + (o + (size_t)c * (p.W >> scale) * (p.H >> scale)) * p.esz;
  };
  const Img* pics[4] = { &p.in0, &p.in1, &p.scp0, &p.scp1 };
  bool written[4] = { false, false, false, false };
  auto add_pictures = [&](int ia, int ib, int scale, int slot, int calc_l, bool down) {
    const bool da = down && !written[ia], db = down && !written[ib];
    for(int c = 0; c < 3; c++)
    {
      SsimImgJob& J = scale == 0 ? q.img0.job[q.nimg0++] : q.imgn.job[q.nimgn++];
      J = SsimImgJob{};
      J.C1 = p.C1; J.C2 = p.C2; J.W = p.W >> scale; J.H = p.H >> scale; J.nx = p.nx[scale]; J.ny = p.ny[scale];
      J.clip = p.clip; J.esz = (int8_t)p.esz; J.calc_l = (int8_t)calc_l; J.wide = p.bitdepth > 12 ? 1 : 0;
      Img small[2];
      const Img* im[2] = { pics[ia], pics[ib] };
      if(scale > 0)
      {
        for(int k = 0; k < 2; k++)
        {
          small[k] = Img{};
          small[k].p[c] = level(k ? ib : ia, scale, c); small[k].pitch[c] = J.W;
          im[k] = &small[k];
        }
      }
      J.a = im[0]->p[c]; J.pitch_a = im[0]->pitch[c]; J.sxa = im[0]->sx[c]; J.sya = im[0]->sy[c]; load_mode(*im[0], c, p.esz, J.load_a, J.vec_a);
      J.b = im[1]->p[c]; J.pitch_b = im[1]->pitch[c]; J.sxb = im[1]->sx[c]; J.syb = im[1]->sy[c]; load_mode(*im[1], c, p.esz, J.load_b, J.vec_b);
      J.down_a = da ? level(ia, 1, c) : nullptr;
      J.down_b = db ? level(ib, 1, c) : nullptr;
      J.down_vec = ((J.W >> 1) & 1) == 0 && (!da || (uintptr_t)J.down_a % (2 * p.esz) == 0) && (!db || (uintptr_t)J.down_b % (2 * p.esz) == 0) ? 1 : 0;
      J.win = out(scale, slot, c);
    }
    if(down) { written[ia] = written[ib] = true; }
    slot_of(scale, slot, 0);
  };
  if(p.mask & QMIV_IVSSIM) { add_moments(p.mom[0], kSlotIvT2R); add_moments(p.mom[1], kSlotIvR2T); }   // xIVSSIM.cpp:46-47
  if(p.mask & QMIV_SSIM) { add_pictures(0, 1, 0, kSlotSsim, 1, false); }                                 // xSSIM.h:83
  const bool ms = p.mask & (QMIV_MSSSIM | QMIV_IVMSSSIM);
  for(int s = 0; ms && s < p.ns; s++)
  {
    const int last = s == p.ns - 1 ? 1 : 0;
    const bool down = s == 0 && !last;
    if(p.mask & QMIV_MSSSIM) { add_pictures(0, 1, s, kSlotMs + s, last, down); }
    if(p.mask & QMIV_IVMSSSIM)                              // xIVSSIM.cpp:77-78, no ERP weighting
    {
      add_pictures(0, 3, s, kSlotIvmsT2R + s, last, down);
      add_pictures(1, 2, s, kSlotIvmsR2T + s, last, down);
    }
  }
  for(int img = 0; ms && p.ns > 2 && img < ((p.mask & QMIV_IVMSSSIM) ? 4 : 2); img++)
  {
    for(int c = 0; c < 3; c++)
    {
      SsimPyrJob& J = q.pyr.job[q.npyr++];
      J = SsimPyrJob{};
      J.src = level(img, 1, c); J.W = p.W >> 1; J.H = p.H >> 1; J.esz = p.esz;
      for(int s = 2; s < p.ns; s++) { J.dst[s - 2] = level(img, s, c); }
    }
  }
}

static cudaError_t last_or(cudaError_t e) { return e != cudaSuccess ? e : cudaGetLastError(); }

cudaError_t launch_ssim_rows(const JobArgs<SsimRowJob, kMaxRowJobs>& a, int njobs, cudaStream_t s)
{
  if(njobs <= 0) { return cudaSuccess; }
  int maxny = 0;
  for(int k = 0; k < njobs; k++) { maxny = max(maxny, a.job[k].ny); }
  k_ssim_rows<<<dim3(bands_of(maxny), njobs), 32 * kRowWarps, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_ssim_jobs(const SsimJobs& q, cudaStream_t s, bool rows_only)
{
  if(rows_only) { return launch_ssim_rows(q.rows, q.nrows, s); }
  SsimDims d;
  d.add(q);
  cudaError_t e = cudaSuccess;
  for(int k = 0; k < q.npool; k++) { if(!pool_job_aligned(q.pool.job[k])) { return cudaErrorMisalignedAddress; } }
  if(e == cudaSuccess && q.npool) { e = launch_next(k_ssim_win, dim3(tiles_of(d.pool_nx), bands_of(d.pool_ny), q.npool), kWinNT, 0, s, q.pool); }
  if(q.nimg0) { k_ssim_img<kMaxImgJobs0><<<dim3(q.nimg0, tiles_of(d.img0_nx), bands_of(d.img0_ny)), kWinNT, 0, s>>>(q.img0); e = last_or(e); }
  if(q.npyr) { k_ssim_pyr<<<dim3((d.pyr_w + 2 * kPyrW - 1) / (2 * kPyrW), (d.pyr_h + 2 * kPyrH - 1) / (2 * kPyrH), q.npyr), 256, 0, s>>>(q.pyr); e = last_or(e); }
  if(q.nimgn) { k_ssim_img<kMaxImgJobsN><<<dim3(q.nimgn, tiles_of(d.imgn_nx), bands_of(d.imgn_ny)), kWinNT, 0, s>>>(q.imgn); e = last_or(e); }
  return e;
}

cudaError_t launch_ssim_tables(const SsimTables& t, cudaStream_t s, bool rows_only)
{
  const SsimDims& d = t.dims;
  cudaError_t e = cudaSuccess;
  if(rows_only)
  {
    if(t.nrows) { k_ssim_rows_multi<<<dim3(t.nrows, bands_of(d.rows_ny)), 32 * kRowWarps, 0, s>>>(t.rows); e = last_or(e); }
    return e;
  }
  if(t.npool) { k_ssim_win_multi<<<dim3(t.npool, tiles_of(d.pool_nx), bands_of(d.pool_ny)), kWinNT, 0, s>>>(t.pool); e = last_or(e); }
  if(t.nimg0) { k_ssim_img_multi<<<dim3(t.nimg0, tiles_of(d.img0_nx), bands_of(d.img0_ny)), kWinNT, 0, s>>>(t.img0); e = last_or(e); }
  if(t.npyr) { k_ssim_pyr_multi<<<dim3(t.npyr, (d.pyr_w + 2 * kPyrW - 1) / (2 * kPyrW), (d.pyr_h + 2 * kPyrH - 1) / (2 * kPyrH)), 256, 0, s>>>(t.pyr); e = last_or(e); }
  if(t.nimgn) { k_ssim_img_multi<<<dim3(t.nimgn, tiles_of(d.imgn_nx), bands_of(d.imgn_ny)), kWinNT, 0, s>>>(t.imgn); e = last_or(e); }
  return e;
}

}  // namespace qmiv
