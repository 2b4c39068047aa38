// Corresponding-pixel-shift search (libs/pmbb-ivqm/src/xCorrespPixelShiftSSE.cpp:18-127) of 4:2:0
// pictures: integer keys, the chroma part of the error shared by the pixels that share a chroma sample.
//
// For a test pixel s (test + GCD, unclipped) and a candidate r the reference minimises
// e = sum_c w_c (s_c - r_c)^2 and keeps the first strict minimum in raster order. With every sample
// taken relative to the mid value m (s' = s - m, r' = r - m), K a power of two above the largest
// raster index and k = (dy+R)(2R+1) + (dx+R),
//     key = K (e - w_0 s'_0^2 - w_1 s'_1^2 - w_2 s'_2^2 + B) + k
// orders a pixel's candidates exactly as (e, raster index) does, in 32-bit unsigned arithmetic, when
// B bounds the subtracted terms and the largest key stays below 2^32 (cps_shared_key checks it on the
// host: up to 11 bits with the default weights, 12 bits up to R = 2). It splits into
//     P(2x2 test block, chroma sample)  = K (w_1 u'^2 + w_2 v'^2 + B) - 2 K (w_1 s'_1 u' + w_2 s'_2 v')
//     t(2x2 test block, reference pixel) = K w_0 y'^2 + P + raster code of the reference pixel
//     key(test pixel, reference pixel)   = -2 K w_0 s'_0 y' + t
// In a 4:2:0 picture P serves the four pixels of a 2x2 block against the (up to) four reference pixels
// of a chroma sample and t serves the block's four pixels, so a candidate costs one integer
// multiply-add and half a three-input minimum; per candidate at R = 2 the shared parts add 0.36
// additions and 0.18 multiply-adds. The per-candidate form before it (three FFMAs, a multiply-add for
// the key, half a minimum) needs about 6 dispatch cycles per 32 candidates; this mix measured 2.3 in a
// loop of its own (integer multiply-add, add and minimum: two cycles each, on two pipes).
//
// Per tile of 128 x 16 pixels a CTA of 8 warps
//   1. receives both pictures' raw samples of the tile and an R-pixel halo by TMA;
//   2. completes the halo outside the picture in place (edge replication, tiles at the picture's
//      border only) and stages both pictures as (y', K w_0 y'^2) per luma sample and
//      (u', v', K (w_1 u'^2 + w_2 v'^2 + B)) per chroma sample;
//   3. each thread searches one 4x4 block in one direction (warps 0-3: In0 in In1, warps 4-7 the
//      other; lane L the block of columns 4 L): a reference pixel is read once for up to 16 test pixels,
//   4. and goes on with the block's epilogue in registers: it gathers its 16 winners from the raw
//      boxes, adds their squared differences to the 32-bit row sums, and writes the shift-compensated
//      samples or the IV-SSIM sub-block moments. No barrier separates search and epilogue.
// A staged luma row keeps its pixel pairs (16 bytes) split by parity of the pair, so the 16-byte loads
// of a warp (lane stride two pairs) are contiguous; a chroma row's pairs are contiguous as they are.
//
// What bounds it: the integer pipes. A warp's tile takes about 2290 instructions at R = 2 with IV-SSIM
// moments (search 960, epilogue 760, staging 260), of which the multiply-adds keep their pipe busy 63 %
// of the time at two cycles each and the additions and minima theirs 41 %; issue is at 64 % with 24 warps
// per SM. 4096x2048, 10 bits, R = 2, moments: 1239 -> 838 us per 8 pairs (one pair 154 -> 111), 897 of it while
// one kernel served one pair and the work list alike; without moments and with the compensated pictures stored,
// 2048x2048: 723 -> 447 us per 8 pairs; 12 bits, 1998x1080 (the literal search before): 262 -> 84 us. Against that
// kernel of 897 and 470 us, gathering the winners from the staged rows instead,
// which frees the raw boxes for the next tile's copies, measured 918-930 us (bank conflicts); two CTAs
// with double-buffered boxes measure 883 us with moments but 485 with stored pictures, so the raw boxes
// are double-buffered only where three CTAs do not fit.
//
// With a mask (mask mode) the same tiles also bring the mask's samples; masked reference samples are staged
// above every real key and the winners' squared differences are weighted by the test pixels' mask values. A strip of
// 128 x 4 pixels without a kept one is not searched, a tile without one not staged. Calls of 4096x2048, 10 bits,
// 8-bit mask, R = 2: full mask 290 us by the fp32-key kernel (one pixel column per thread, tiles staged sample by sample, no
// copies in flight) -> 162, a disc (32 % of the picture) 214 -> 113, a rectangle of 5 % 184 -> 89; R = 4 452 -> 296,
// 270 -> 163, 197 -> 100. Where single 16x16 blocks are strewn over the picture, 20 % of them kept, the strips of
// 32 x 4 pixels of that kernel left out more: 219 -> 156 at R = 2, 280 -> 287 at R = 4, 367 -> 405 at R = 5. Dealing the
// kept 4x4 blocks to as few warps as hold them took longer still (424 at R = 4): a tile lasts as long as one warp.
// 8 pairs of 1920x1080, 8 bits, 60 % of the 16x16 blocks kept: 729 -> 402.
//
// Pictures with samples above the maximum (SKIP and WARN actions) and parameters whose keys do not fit
// take the literal int32 search below (the SSE path's wrap-around arithmetic) in the same frame.
#pragma once
#include "qmiv_cps.cuh"

#include <cstring>
#include <type_traits>

namespace qmiv {

namespace {

constexpr unsigned kFull = 0xffffffffu;

// Sample type of the mask of a search without one
struct NoMask { };

// Geometry of one search range, sample type and mask sample type; every size is known at compile time.
template <int R, typename T, typename TM = NoMask>
struct Geo420
{
  static constexpr bool MASK = !std::is_same<TM, NoMask>::value;
  static constexpr int D = 2 * R + 1;
  static constexpr int KB = cps_key_bits(R);                           // key bits of the raster code
  static constexpr uint32_t K = 1u << KB;
  static_assert(D * D <= (1 << KB), "raster codes fit");
  static constexpr int TW = 128, TH = 16, NT = 256;
  static constexpr int ODD = R & 1;
  static constexpr int SW = TW + 2 * R, SH = TH + 2 * R;           // staged luma samples
  static constexpr int CR0 = (R + 1) / 2;                          // chroma samples left of / above the tile
  static constexpr int CW = ((TW - 1 + R) >> 1) + CR0 + 1, CH = ((TH - 1 + R) >> 1) + CR0 + 1;
  static constexpr int ESZ = (int)sizeof(T);
  static constexpr int AX = 16 / ESZ;                              // TMA boxes start 16 bytes left of the tile
  static constexpr int BWL = (int)align_up(AX + TW + R, AX), BHL = SH;
  static constexpr int BWC = (int)align_up(AX + ((TW - 1 + R) >> 1) + 1, AX), BHC = CH;
  static constexpr int PLB = BWL * ESZ, PCB = BWC * ESZ;           // raw row pitches in bytes
  // raw boxes of one picture: luma, Cb, Cr
  static constexpr uint32_t OFFU = align_up(BHL * PLB, kAlign), OFFV = OFFU + align_up(BHC * PCB, kAlign);
  static constexpr uint32_t PIC = OFFV + align_up(BHC * PCB, kAlign);
  // the mask's box behind both pictures'
  static constexpr int MESZ = (int)sizeof(TM), AXM = 16 / MESZ, BWM = (int)align_up(AXM + TW + R, AXM);
  static constexpr uint32_t OFFM = 2 * PIC;
  static constexpr uint32_t STAGE = OFFM + (MASK ? align_up(BHL * BWM * MESZ, kAlign) : 0u);
  static constexpr uint32_t TX = 2u * (uint32_t)(BHL * PLB + 2 * BHC * PCB) + (MASK ? (uint32_t)(BHL * BWM * MESZ) : 0u);
  // staged rows, in 16-byte pairs of samples
  static constexpr int HALF = (SW / 2 + 1) / 2, LPP = 2 * HALF;    // luma: even pairs, then odd pairs
  static constexpr int CPP = CW / 2;                               // chroma
  static_assert(CW % 2 == 0, "whole chroma pairs");
  static constexpr uint32_t LUMA = (uint32_t)SH * LPP * 16u, CHROMA = (uint32_t)CH * CPP * 16u;   // per picture
  // Three CTAs per SM where they fit with one raw stage each (R <= 2, R = 3 with bytes), else two (unmasked one at
  // R = 5), with the raw boxes double-buffered where as many CTAs still fit. With a mask, full, 4096x2048 10 bits: one
  // CTA was resident with two stages, 372 us a call at R = 4 and 536 at R = 5; two with one stage take 296 and 408.
  static constexpr uint32_t TILES = 2 * LUMA + 2 * CHROMA + kAlign + 32, PER_SM = 227u * 1024u, FIXED = 3584u;   // static and reserved
  static constexpr int CTAS = 3 * (TILES + STAGE + FIXED) <= PER_SM ? 3 : (R <= 4 || MASK ? 2 : 1);
  static constexpr uint32_t STAGES = CTAS < 3 && CTAS * (TILES + 2 * STAGE + FIXED) <= PER_SM ? 2 : 1;
  static constexpr uint32_t SMEM = TILES + STAGES * STAGE;
  static_assert(CTAS * (SMEM + FIXED) <= PER_SM, "the CTAs that the registers are shared out for are resident");
  // a thread's window: luma samples and chroma samples across / down
  static constexpr int WL = 4 + 2 * R, WC = ((3 + 2 * R + ODD) >> 1) + 1;
  static_assert(WL % 2 == 0 && WC % 2 == 0, "windows of whole pairs");
};

// Code of window sample (ry, rx); candidate (dy + R, dx + R) of block pixel (i, j) is window sample
// (dy + R + i, dx + R + j), whose code less code(i, j) is the candidate's raster index.
template <int D> __host__ __device__ constexpr uint32_t code_of(int ry, int rx) { return (uint32_t)(ry * D + rx); }

struct Pair420
{
  const CpsKernelArgs* k;
  int                  tile;
};

template <int R, typename T, typename TM>
__device__ __forceinline__ void issue_tile420(const CpsKernelArgs& k, bool new_maps, unsigned char* raw, uint64_t* bar, int t)
{
  using G = Geo420<R, T, TM>;
  const int x0 = (t % k.g.ntx) * G::TW, y0 = (t / k.g.ntx) * G::TH;
  if(new_maps)   // the first use of a pair's tensor maps, which the host copied to global memory
  {
    #pragma unroll
    for(int f = 0; f < 2; f++)
    {
      #pragma unroll
      for(int c = 0; c < 3; c++) { fence_tensormap_acquire(&k.map[f][c]); }
    }
    if(G::MASK) { fence_tensormap_acquire(&k.mask_map); }
  }
  mbar_expect_tx(bar, G::TX);
  #pragma unroll
  for(int f = 0; f < 2; f++)
  {
    unsigned char* p = raw + f * G::PIC;
    tma_load_2d(p, &k.map[f][0], x0 - G::AX, y0 - R, bar);
    tma_load_2d(p + G::OFFU, &k.map[f][1], (x0 >> 1) - G::AX, (y0 - R) >> 1, bar);
    tma_load_2d(p + G::OFFV, &k.map[f][2], (x0 >> 1) - G::AX, (y0 - R) >> 1, bar);
  }
  if(G::MASK) { tma_load_2d(raw + G::OFFM, &k.mask_map, x0 - G::AXM, y0 - R, bar); }
}

// One box by plain loads, for planes whose address or pitch TMA cannot take (samples outside the picture
// stay unwritten: complete_halo fills them). xs, ys: picture position of the box; pw, ph: plane size.
template <typename S, int NT>
__device__ __forceinline__ void load_box(const S* src, int pitch, S* dst, int bw, int bh, int xs, int ys, int pw, int ph)
{
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for(int r = warp; r < bh; r += NT / 32)
  {
    const int gy = ys + r;
    if(gy < 0 || gy >= ph) { continue; }
    for(int col = lane; col < bw; col += 32)
    {
      const int gx = xs + col;
      if(gx >= 0 && gx < pw) { dst[r * bw + col] = __ldg(src + (size_t)gy * pitch + gx); }
    }
  }
}

template <int R, typename T, typename TM>
__device__ __noinline__ void load_plain420(const CpsArgs& a, unsigned char* raw, int x0, int y0)
{
  using G = Geo420<R, T, TM>;
  #pragma unroll 1
  for(int fc = 0; fc < 6; fc++)
  {
    const int f = fc / 3, c = fc - 3 * f;
    const Img& im = f ? a.in1 : a.in0;
    load_box<T, G::NT>(static_cast<const T*>(im.p[c]), im.pitch[c],
                       reinterpret_cast<T*>(raw + f * G::PIC + (c == 0 ? 0u : c == 1 ? G::OFFU : G::OFFV)), c ? G::BWC : G::BWL,
                       c ? G::BHC : G::BHL, (c ? x0 >> 1 : x0) - G::AX, c ? (y0 - R) >> 1 : y0 - R, c ? a.W >> 1 : a.W, c ? a.H >> 1 : a.H);
  }
  if constexpr(G::MASK)
  {
    load_box<TM, G::NT>(static_cast<const TM*>(a.mask), a.mask_pitch, reinterpret_cast<TM*>(raw + G::OFFM), G::BWM, G::BHL, x0 - G::AXM, y0 - R, a.W, a.H);
  }
}

// Edge replication, in place, of a box's samples outside the picture that a candidate of a pixel inside can
// reach. left: first column used; m: reach past the picture; inx0 .. inx1, iny0 .. iny1: the part inside.
// Sources lie inside the picture and the box (a tile starts inside the picture) and are not written.
template <typename S, int NT>
__device__ __forceinline__ void replicate_box(S* p, int bw, int bh, int left, int m, int inx0, int inx1, int iny0, int iny1)
{
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int right = min(bw, inx1 + m), rows = min(bh, iny1 + m);
  for(int r = warp; r < rows; r += NT / 32)
  {
    const int sr = clampi(r, iny0, iny1 - 1);
    const S* src = p + sr * bw;
    S* dst = p + r * bw;
    if(sr != r)
    {
      for(int x = left + lane; x < right; x += 32) { dst[x] = src[clampi(x, inx0, inx1 - 1)]; }
    }
    else
    {
      for(int x = left + lane; x < inx0; x += 32) { dst[x] = src[inx0]; }
      for(int x = inx1 + lane; x < right; x += 32) { dst[x] = src[inx1 - 1]; }
    }
  }
}

// Conceal clipping of the whole boxes, then the halo outside the picture.
template <int R, typename T, typename TM>
__device__ __noinline__ void complete_halo(const CpsArgs& a, unsigned char* raw, int x0, int y0, bool clip, bool border)
{
  using G = Geo420<R, T, TM>;
  #pragma unroll 1
  for(int pass = clip ? 0 : 1; pass < (border ? 2 : 1); pass++)
  {
    #pragma unroll 1
    for(int fc = 0; fc < 6; fc++)
    {
      const int f = fc / 3, c = fc - 3 * f;
      const int bw = c ? G::BWC : G::BWL, bh = c ? G::BHC : G::BHL, m = c ? G::CR0 : R;
      T* p = reinterpret_cast<T*>(raw + f * G::PIC + (c == 0 ? 0u : c == 1 ? G::OFFU : G::OFFV));
      if(pass == 0)
      {
        for(int e = threadIdx.x; e < bw * bh; e += G::NT) { p[e] = (T)min((uint32_t)p[e], a.clip); }
        continue;
      }
      const int xs = (c ? x0 >> 1 : x0) - G::AX, ys = c ? (y0 - R) >> 1 : y0 - R;
      replicate_box<T, G::NT>(p, bw, bh, G::AX - m, m, max(0, -xs), (c ? a.W >> 1 : a.W) - xs, max(0, -ys), (c ? a.H >> 1 : a.H) - ys);
    }
    if constexpr(G::MASK)
    {
      if(pass == 1)
      {
        replicate_box<TM, G::NT>(reinterpret_cast<TM*>(raw + G::OFFM), G::BWM, G::BHL, G::AXM - R, R, max(0, G::AXM - x0), a.W - x0 + G::AXM,
                                 max(0, R - y0), a.H - y0 + R);
      }
    }
    __syncthreads();
  }
}

// Four neighbouring samples from an address aligned to ALIGN samples
template <typename T, int ALIGN>
__device__ __forceinline__ void load4(const T* p, uint32_t v[4])
{
  if constexpr(sizeof(T) == 2 && ALIGN >= 4)
  {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    v[0] = w.x & 0xffffu; v[1] = w.x >> 16; v[2] = w.y & 0xffffu; v[3] = w.y >> 16;
  }
  else if constexpr(sizeof(T) == 1 && ALIGN >= 4)
  {
    const uint32_t w = *reinterpret_cast<const uint32_t*>(p);
    v[0] = w & 0xffu; v[1] = (w >> 8) & 0xffu; v[2] = (w >> 16) & 0xffu; v[3] = w >> 24;
  }
  else if constexpr(ALIGN >= 2)
  {
    if constexpr(sizeof(T) == 2)
    {
      const uint32_t w = reinterpret_cast<const uint32_t*>(p)[0], x = reinterpret_cast<const uint32_t*>(p)[1];
      v[0] = w & 0xffffu; v[1] = w >> 16; v[2] = x & 0xffffu; v[3] = x >> 16;
    }
    else
    {
      const uint32_t w = reinterpret_cast<const uint16_t*>(p)[0], x = reinterpret_cast<const uint16_t*>(p)[1];
      v[0] = w & 0xffu; v[1] = w >> 8; v[2] = x & 0xffu; v[3] = x >> 8;
    }
  }
  else
  {
    #pragma unroll
    for(int k = 0; k < 4; k++) { v[k] = p[k]; }
  }
}

// Bit q: the mask keeps a sample in the tile's rows 4 q .. 4 q + 3 (128 columns; past the picture the box holds anything,
// so a bit too many there). The same for every warp, which reads the whole tile: 16 bytes a lane and load.
template <int R, typename T, typename TM>
__device__ __forceinline__ uint32_t kept_strips(const unsigned char* raw, int lane)
{
  using G = Geo420<R, T, TM>;
  constexpr int PER_ROW = G::TW * G::MESZ / 16, ROWS = 32 / PER_ROW;   // lanes of a row, rows of a load
  static_assert(4 % ROWS == 0 && G::AXM * G::MESZ == 16 && G::BWM * G::MESZ % 16 == 0 && G::OFFM % 16 == 0, "aligned loads");
  const unsigned char* p = raw + G::OFFM + (R + lane / PER_ROW) * (G::BWM * G::MESZ) + 16 + 16 * (lane % PER_ROW);
  uint32_t bits = 0;
  #pragma unroll
  for(int q = 0; q < 4; q++)
  {
    uint32_t any = 0;
    #pragma unroll
    for(int r = 4 * q; r < 4 * q + 4; r += ROWS)
    {
      const uint4 v = *reinterpret_cast<const uint4*>(p + r * (G::BWM * G::MESZ));
      any |= v.x | v.y | v.z | v.w;
    }
    bits |= __any_sync(kFull, any != 0u) ? 1u << q : 0u;
  }
  return bits;
}

// Test samples of the 4x4 block at (block row by, block column lane): 16 luma, 2x2 of either chroma.
template <int R, typename T>
__device__ __forceinline__ void load_test420(const unsigned char* tst, int by, int lane, int shift, uint32_t ty[16],
                                             uint32_t tu[4], uint32_t tv[4])
{
  using G = Geo420<R, T>;
  const T* p = reinterpret_cast<const T*>(tst) + shift + (4 * by + R) * G::BWL + G::AX + 4 * lane;
  const T* pu = reinterpret_cast<const T*>(tst + G::OFFU) + shift + (2 * by + G::CR0) * G::BWC + G::AX + 2 * lane;
  const T* pv = reinterpret_cast<const T*>(tst + G::OFFV) + shift + (2 * by + G::CR0) * G::BWC + G::AX + 2 * lane;
  #pragma unroll
  for(int i = 0; i < 4; i++) { load4<T, 4>(p + i * G::BWL, ty + 4 * i); }
  #pragma unroll
  for(int b = 0; b < 4; b++) { tu[b] = pu[(b >> 1) * G::BWC + (b & 1)]; tv[b] = pv[(b >> 1) * G::BWC + (b & 1)]; }
}

// raw boxes -> staged luma and chroma of both pictures. Under a mask a masked luma sample is staged as
// (0, masked): its keys are masked + P + code whatever the test pixel, above every key of an unmasked one.
template <int R, typename T, typename TM>
__device__ __forceinline__ void stage420(const unsigned char* raw, uint4* luma, uint4* chroma, uint32_t kw0, uint32_t kw1,
                                         uint32_t kw2, uint32_t bias, int32_t mid, uint32_t masked)
{
  using G = Geo420<R, T, TM>;
  constexpr int MA = (G::AXM - R) % 4 == 0 ? 4 : (G::AXM - R) % 2 == 0 ? 2 : 1;
  static_assert(!G::MASK || G::AXM - R + 4 * ((G::SW + 3) / 4) <= G::BWM, "mask units read inside the box");
  constexpr int NU = (G::SW + 3) / 4;                       // four-sample units per row; the last may hold two
  static_assert(G::AX - R + 4 * NU <= G::BWL, "units read inside the box");
  constexpr int LA = (G::AX - R) % 4 == 0 ? 4 : (G::AX - R) % 2 == 0 ? 2 : 1;
  {
    // unit u = row * NU + c walks in steps of NT
    constexpr int DR = G::NT / NU, DC = G::NT % NU;
    int row = threadIdx.x / NU, c = threadIdx.x - row * NU;
    #pragma unroll 1
    while(row < 2 * G::SH)
    {
      const int rowofs = row * G::PLB + (row >= G::SH ? (int)G::PIC - G::SH * G::PLB : 0);
      uint32_t v[4], q[4];
      load4<T, LA>(reinterpret_cast<const T*>(raw + rowofs) + (G::AX - R) + 4 * c, v);
      #pragma unroll
      for(int k = 0; k < 4; k++) { v[k] -= (uint32_t)mid; q[k] = v[k] * v[k] * kw0; }
      if constexpr(G::MASK)
      {
        uint32_t m[4];
        load4<TM, MA>(reinterpret_cast<const TM*>(raw + G::OFFM) + (row >= G::SH ? row - G::SH : row) * G::BWM + (G::AXM - R) + 4 * c, m);
        #pragma unroll
        for(int k = 0; k < 4; k++) { if(m[k] == 0u) { v[k] = 0u; q[k] = masked; } }
      }
      uint4* d = luma + row * G::LPP + c;
      d[0] = make_uint4(v[0], q[0], v[1], q[1]);
      d[G::HALF] = make_uint4(v[2], q[2], v[3], q[3]);
      row += DR; c += DC;
      if(c >= NU) { c -= NU; row++; }
    }
  }
  {
    constexpr int DR = G::NT / G::CPP, DC = G::NT % G::CPP;
    int row = threadIdx.x / G::CPP, c = threadIdx.x - row * G::CPP;
    #pragma unroll 1
    while(row < 2 * G::CH)
    {
      const int rowofs = row * G::PCB + (row >= G::CH ? (int)G::PIC - G::CH * G::PCB : 0);
      const T* pu = reinterpret_cast<const T*>(raw + G::OFFU + rowofs) + (G::AX - G::CR0) + 2 * c;
      const T* pv = reinterpret_cast<const T*>(raw + G::OFFV + rowofs) + (G::AX - G::CR0) + 2 * c;
      uint32_t w[2], q[2];
      #pragma unroll
      for(int k = 0; k < 2; k++)
      {
        const uint32_t cu = (uint32_t)pu[k] - (uint32_t)mid, cv = (uint32_t)pv[k] - (uint32_t)mid;
        w[k] = (cu & 0xffffu) | (cv << 16);
        q[k] = cu * cu * kw1 + (cv * cv * kw2 + bias);
      }
      chroma[row * G::CPP + c] = make_uint4(w[0], q[0], w[1], q[1]);
      row += DR; c += DC;
      if(c >= G::CPP) { c -= G::CPP; row++; }
    }
  }
}

// Raster indices of the 16 winners of a block. luma / chroma: the thread's window in the reference
// picture's staged rows; c0: -2 K w_0 s'_0 of the 16 pixels, c1 / c2: of the four 2x2 blocks' chroma.
template <int R, typename T>
__device__ __forceinline__ void search420(const uint4* luma, const uint4* chroma, const uint32_t c0[16], const uint32_t c1[4],
                                          const uint32_t c2[4], uint32_t idx[16])
{
  using G = Geo420<R, T>;
  constexpr int D = G::D;
  uint32_t best[16], pend[16];
  #pragma unroll
  for(int p = 0; p < 16; p++) { best[p] = 0xffffffffu; }
  uint32_t P[4][G::WC];                                     // [2x2 block][chroma column]
  #pragma unroll
  for(int ry = 0; ry < G::WL; ry++)
  {
    const int cy = (ry + G::ODD) >> 1;
    if(ry == 0 || cy != ((ry - 1 + G::ODD) >> 1))
    {
      // a new chroma row: its terms for every 2x2 block whose candidates use it
      #pragma unroll
      for(int cp = 0; cp < G::WC / 2; cp++)
      {
        const uint4 s = chroma[cy * G::CPP + cp];
        #pragma unroll
        for(int h = 0; h < 2; h++)
        {
          const int cx = 2 * cp + h;
          const uint32_t w = h ? s.z : s.x, q = h ? s.w : s.y;
          const uint32_t cu = (uint32_t)((int32_t)(w << 16) >> 16), cv = (uint32_t)((int32_t)w >> 16);
          #pragma unroll
          for(int b = 0; b < 4; b++)
          {
            const int bi = b >> 1, bj = b & 1;
            if(cy >= bi && cy <= bi + R + G::ODD && cx >= bj && cx <= bj + R + G::ODD) { P[b][cx] = c2[b] * cv + (c1[b] * cu + q); }
          }
        }
      }
    }
    #pragma unroll
    for(int rx = 0; rx < G::WL; rx += 2)
    {
      const uint4 s = luma[ry * G::LPP + ((rx >> 1) & 1) * G::HALF + (rx >> 2)];
      #pragma unroll
      for(int b = 0; b < 4; b++)
      {
        const int bi = b >> 1, bj = b & 1;
        if(ry < 2 * bi || ry > 2 * bi + 1 + 2 * R) { continue; }
        const bool va = rx >= 2 * bj && rx <= 2 * bj + 1 + 2 * R, vc = rx + 1 >= 2 * bj && rx + 1 <= 2 * bj + 1 + 2 * R;
        if(!va && !vc) { continue; }
        uint32_t ta = va ? s.y + P[b][(rx + G::ODD) >> 1] + code_of<D>(ry, rx) : 0u;
        uint32_t tc = vc ? s.w + P[b][(rx + 1 + G::ODD) >> 1] + code_of<D>(ry, rx + 1) : 0u;
        // formed once: reassociated into the four pixels' sums they would cost each an addition
        asm("" : "+r"(ta));
        asm("" : "+r"(tc));
        #pragma unroll
        for(int ii = 0; ii < 2; ii++)
        {
          const int i = 2 * bi + ii, dy = ry - i;
          if(dy < 0 || dy >= D) { continue; }
          #pragma unroll
          for(int jj = 0; jj < 2; jj++)
          {
            const int j = 2 * bj + jj, p = 4 * i + j;
            const bool ka = rx - j >= 0 && rx - j < D, kc = rx + 1 - j >= 0 && rx + 1 - j < D;
            if(ka && kc) { best[p] = __vimin3_u32(best[p], c0[p] * s.x + ta, c0[p] * s.z + tc); }
            else if(ka || kc)
            {
              // the one leftover candidate of a search row: two rows share a three-input minimum
              const uint32_t ks = ka ? c0[p] * s.x + ta : c0[p] * s.z + tc;
              if(dy == D - 1) { best[p] = min(best[p], ks); }
              else if((dy & 1) == 0) { pend[p] = ks; }
              else { best[p] = __vimin3_u32(best[p], pend[p], ks); }
            }
          }
        }
      }
    }
  }
  #pragma unroll
  for(int p = 0; p < 16; p++) { idx[p] = (best[p] - code_of<D>(p >> 2, p & 3)) & (G::K - 1u); }
}

// The same winners by the SSE path's arithmetic taken literally (wrapping int32 errors, first strict
// minimum in raster order), from the raw boxes of any 16-bit samples. Bound by its shared-memory loads, three a
// candidate; a call of 1920x1080, 12 bits, R = 3 / 4 / 5 took 395 / 571 / 1119 us when the literal search ran on
// float4 tiles, 279 / 410 / 686 like this; 14 bits, R = 2: 247 -> 163.
template <int R, typename T>
__device__ __noinline__ void search420_literal(const unsigned char* tst, const unsigned char* ref, int lofs, int cofs,
                                               uint32_t w0, uint32_t w1, uint32_t w2, int g0, int g1, int g2, uint32_t idx[16])
{
  using G = Geo420<R, T>;
  constexpr int D = G::D;
  const T* ty = reinterpret_cast<const T*>(tst) + lofs + R * G::BWL + R;
  const T* tu = reinterpret_cast<const T*>(tst + G::OFFU) + cofs + G::CR0 * G::BWC + G::CR0;
  const T* tv = reinterpret_cast<const T*>(tst + G::OFFV) + cofs + G::CR0 * G::BWC + G::CR0;
  const T* ry = reinterpret_cast<const T*>(ref) + lofs;
  const T* ru = reinterpret_cast<const T*>(ref + G::OFFU) + cofs;
  const T* rv = reinterpret_cast<const T*>(ref + G::OFFV) + cofs;
  #pragma unroll 1
  for(int p = 0; p < 16; p++)
  {
    const int i = p >> 2, j = p & 3;
    const uint32_t s0 = (uint32_t)((int)ty[i * G::BWL + j] + g0);
    const uint32_t s1 = (uint32_t)((int)tu[(i >> 1) * G::BWC + (j >> 1)] + g1);
    const uint32_t s2 = (uint32_t)((int)tv[(i >> 1) * G::BWC + (j >> 1)] + g2);
    int32_t best = 0x7fffffff;
    uint32_t bi = 0;
    #pragma unroll 1
    for(int dy = 0; dy < D; dy++)
    {
      #pragma unroll 1
      for(int dx = 0; dx < D; dx++)
      {
        const int co = ((i + dy + G::ODD) >> 1) * G::BWC + ((j + dx + G::ODD) >> 1);
        const uint32_t d0 = s0 - ry[(i + dy) * G::BWL + j + dx], d1 = s1 - ru[co], d2 = s2 - rv[co];
        const int32_t err = (int32_t)(d0 * d0 * w0 + d1 * d1 * w1 + d2 * d2 * w2);
        if(err < best) { best = err; bi = code_of<D>(dy, dx); }
      }
    }
    idx[p] = bi;
  }
}

// Raw-box offsets of candidate k of a pixel of parity (pi, pj) relative to the block's first candidate
// (luma in the low 16 bits, chroma in the high), in bytes; entry [2 pi + pj][k].
template <int R, typename T>
__device__ __forceinline__ void build_offsets420(uint32_t* off)
{
  using G = Geo420<R, T>;
  static_assert(G::PIC < 65536u, "offsets fit 16 bits");
  for(int e = threadIdx.x; e < 4 * 128; e += G::NT)
  {
    const int pi = e >> 8, pj = (e >> 7) & 1, k = e & 127;
    const int dy = k / G::D, dx = k - dy * G::D;
    const uint32_t lo = (uint32_t)(dy * G::PLB + dx * G::ESZ);
    const uint32_t ch = (uint32_t)(((pi + dy + G::ODD) >> 1) * G::PCB + ((pj + dx + G::ODD) >> 1) * G::ESZ);
    off[e] = k < G::D * G::D ? lo | (ch << 16) : 0u;
  }
}

__device__ __forceinline__ void red_add_global(uint32_t* p, uint32_t v)
{
  asm volatile("red.global.add.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void st_global(uint32_t* p, uint32_t v)
{
  asm volatile("st.global.u32 [%0], %1;" ::"l"(__cvta_generic_to_global(p)), "r"(v) : "memory");
}

// Squared differences to the row sums, SCP samples, sub-block moments of one 4x4 block. All sums wrap
// at 32 bits as the reference's lanes do. EDGE: the tile reaches past the picture (2x2 blocks of an
// even-sized picture lie wholly inside or outside). ty / tu / tv: the block's test samples.
template <int R, typename T, bool EDGE, bool MOM, bool SCP>
__device__ __forceinline__ void epilogue420(const CpsArgs& a, const unsigned char* ref, const uint32_t* off, uint32_t base,
                                            const uint32_t ty[16], const uint32_t tu[4], const uint32_t tv[4],
                                            const uint32_t idx[16], int dir, int xb, int yb, int g0, int g1, int g2)
{
  using G = Geo420<R, T>;
  const int lane = threadIdx.x & 31;
  uint32_t* rows = a.rows + (size_t)dir * a.H * 3;
  T* scp = static_cast<T*>(dir ? a.scp0 : a.scp1);
  const size_t plane = (size_t)a.W * a.H;
  int maxv = a.maxv, ng[3] = { -g0, -g1, -g2 };
  // in plain registers: as warp-uniform values every clip would first copy them
  asm volatile("" : "+r"(maxv), "+r"(ng[0]), "+r"(ng[1]), "+r"(ng[2]));
  bool in[4];
  #pragma unroll
  for(int b = 0; b < 4; b++) { in[b] = !EDGE || (xb + 2 * (b & 1) < a.W && yb + 2 * (b >> 1) < a.H); }
  uint32_t sb[3] = { 0, 0, 0 }, sbb[3] = { 0, 0, 0 }, stb[3] = { 0, 0, 0 };
  uint32_t st[3] = { 0, 0, 0 }, stt[3] = { 0, 0, 0 }, mine = 0;
  #pragma unroll
  for(int i = 0; i < 4; i++)
  {
    uint32_t rs[3] = { 0, 0, 0 };
    uint32_t o[3][4];
    #pragma unroll
    for(int j = 0; j < 4; j++)
    {
      const int p = 4 * i + j, b = (i >> 1) * 2 + (j >> 1);
      const uint32_t w = off[(2 * (i & 1) + (j & 1)) * 128 + idx[p]] + base;
      const unsigned char* pl = ref + (w & 0xffffu);
      const unsigned char* pc = ref + (w >> 16);
      const int co = (i >> 1) * G::PCB + (j >> 1) * G::ESZ;
      const int r[3] = { *reinterpret_cast<const T*>(pl + i * G::PLB + j * G::ESZ), *reinterpret_cast<const T*>(pc + G::OFFU + co),
                         *reinterpret_cast<const T*>(pc + G::OFFV + co) };
      const uint32_t t[3] = { ty[p], tu[b], tv[b] };
      #pragma unroll
      for(int c = 0; c < 3; c++)
      {
        uint32_t d = t[c] - (uint32_t)ng[c] - (uint32_t)r[c];
        if(EDGE && !in[b]) { d = 0u; }
        rs[c] += d * d;
        if(MOM || SCP)
        {
          uint32_t v = (uint32_t)__viaddmin_s32_relu(r[c], ng[c], maxv);   // clip(r - g)
          if(EDGE && !in[b]) { v = 0u; }
          o[c][j] = v;
          if(MOM)
          {
            sb[c] += v;
            sbb[c] += v * v;
            stb[c] += t[c] * v;
          }
        }
      }
      if(MOM && (!EDGE || in[b])) { st[0] += ty[p]; stt[0] += ty[p] * ty[p]; }
    }
    if(SCP && (!EDGE || yb + i < a.H))
    {
      #pragma unroll
      for(int c = 0; c < 3; c++)
      {
        T* q = scp + (size_t)c * plane + (size_t)(yb + i) * a.W + xb;
        const bool whole = !EDGE || xb + 4 <= a.W;
        if((a.W & 3) == 0 && whole)
        {
          if constexpr(sizeof(T) == 2) { *reinterpret_cast<uint2*>(q) = make_uint2(o[c][0] | (o[c][1] << 16), o[c][2] | (o[c][3] << 16)); }
          else { *reinterpret_cast<uint32_t*>(q) = o[c][0] | (o[c][1] << 8) | (o[c][2] << 16) | (o[c][3] << 24); }
        }
        else
        {
          #pragma unroll
          for(int j = 0; j < 4; j++) { if(!EDGE || xb + j < a.W) { q[j] = (T)o[c][j]; } }
        }
      }
    }
    #pragma unroll
    for(int c = 0; c < 3; c++)
    {
      const uint32_t sum = __reduce_add_sync(kFull, rs[c]);
      if(lane == 3 * i + c) { mine = sum; }
    }
  }
  // lane 3 i + c holds component c of row yb + i: twelve neighbouring words
  if(lane < 12 && (!EDGE || yb + lane / 3 < a.H)) { red_add_global(rows + (size_t)yb * 3 + lane, mine); }
  if(MOM)
  {
    #pragma unroll
    for(int b = 0; b < 4; b++)
    {
      if(!EDGE || in[b])
      {
        st[1] += 4u * tu[b]; stt[1] += 4u * tu[b] * tu[b];
        st[2] += 4u * tv[b]; stt[2] += 4u * tv[b] * tv[b];
      }
    }
    const Moments mom = a.mom[dir];
    const int bx = xb >> 2, by = yb >> 2;
    if(bx < mom.nbx && by < mom.nby)
    {
      uint32_t* q = mom.p + (size_t)by * mom.pitch + bx;
      const size_t mplane = mom.plane();
      #pragma unroll
      for(int c = 0; c < 3; c++)
      {
        const uint32_t v[5] = { st[c], sb[c], stt[c], sbb[c], stb[c] };
        #pragma unroll
        for(int m = 0; m < 5; m++) { st_global(q, v[m]); q += mplane; }
      }
    }
  }
}

// Epilogue of a masked search: squared differences weighted by the test pixels' mask values, summed per row in
// 64 bits, over the warp as two 32-bit parts (kMaskSumSplit).
template <int R, typename T, typename TM>
__device__ __forceinline__ void epilogue420_masked(const CpsArgs& a, const unsigned char* ref, const TM* mask, const uint32_t* off, uint32_t base,
                                                   const uint32_t ty[16], const uint32_t tu[4], const uint32_t tv[4],
                                                   const uint32_t idx[16], int dir, int xb, int yb, int g0, int g1, int g2)
{
  using G = Geo420<R, T, TM>;
  const int lane = threadIdx.x & 31;
  // the mask mode's labels: rows 0 hold the search of In1 in In0
  unsigned long long* rows = a.rows64 + (size_t)(dir ^ 1) * a.H * 3;
  uint32_t hi = 0, lo = 0;
  #pragma unroll
  for(int i = 0; i < 4; i++)
  {
    uint64_t rs[3] = { 0, 0, 0 };
    uint32_t m[4];
    load4<TM, 4>(mask + i * G::BWM, m);
    #pragma unroll
    for(int j = 0; j < 4; j++)
    {
      const int p = 4 * i + j, b = (i >> 1) * 2 + (j >> 1);
      const uint32_t w = off[(2 * (i & 1) + (j & 1)) * 128 + idx[p]] + base;
      const unsigned char* pl = ref + (w & 0xffffu);
      const unsigned char* pc = ref + (w >> 16);
      const int co = (i >> 1) * G::PCB + (j >> 1) * G::ESZ;
      const uint32_t d0 = ty[p] + (uint32_t)g0 - *reinterpret_cast<const T*>(pl + i * G::PLB + j * G::ESZ);
      const uint32_t d1 = tu[b] + (uint32_t)g1 - *reinterpret_cast<const T*>(pc + G::OFFU + co);
      const uint32_t d2 = tv[b] + (uint32_t)g2 - *reinterpret_cast<const T*>(pc + G::OFFV + co);
      const uint32_t mv = xb + j < a.W ? m[j] : 0u;
      rs[0] += (uint64_t)(d0 * d0) * mv;
      rs[1] += (uint64_t)(d1 * d1) * mv;
      rs[2] += (uint64_t)(d2 * d2) * mv;
    }
    #pragma unroll
    for(int c = 0; c < 3; c++)
    {
      const uint32_t h = __reduce_add_sync(kFull, (uint32_t)(rs[c] >> kMaskSumSplit));
      const uint32_t l = __reduce_add_sync(kFull, (uint32_t)rs[c] & ((1u << kMaskSumSplit) - 1u));
      if(lane == 3 * i + c) { hi = h; lo = l; }
    }
  }
  const uint64_t sum = ((uint64_t)hi << kMaskSumSplit) + lo;
  if(lane < 12 && yb + lane / 3 < a.H && sum != 0) { atomicAdd(rows + (size_t)yb * 3 + lane, (unsigned long long)sum); }
}

// Persistent tile loop over a work list (LIST: pair p owns tiles [prefix[p], prefix[p + 1]) of descs) or over
// the tiles of the one pair in descs[0].
template <int R, typename T, typename TM, bool LIST>
__device__ __forceinline__ void cps420_body(const CpsKernelArgs* descs, const int32_t* prefix, int ntiles)
{
  using G = Geo420<R, T, TM>;
  extern __shared__ __align__(16) unsigned char smem_dyn[];
  unsigned char* raw = smem_dyn + ((128u - (smem_u32(smem_dyn) & 127u)) & 127u);   // TMA boxes: 128-byte aligned
  uint4* luma = reinterpret_cast<uint4*>(raw + G::STAGES * G::STAGE);
  uint4* chroma = reinterpret_cast<uint4*>(raw + G::STAGES * G::STAGE + 2 * G::LUMA);
  uint64_t* bar = reinterpret_cast<uint64_t*>(raw + G::STAGES * G::STAGE + 2 * G::LUMA + 2 * G::CHROMA);
  __shared__ __align__(16) CpsArgs s_a;       // the current pair's arguments
  __shared__ int32_t s_gcd[4];                // its GCD and path flags
  __shared__ uint32_t s_off[4 * 128];
  static_assert(sizeof(CpsArgs) % 4 == 0, "word copies");

  // The pair of a work-list tile. The list is walked forwards, so each caller keeps the current pair
  // and its tile range and moves on only when the range ends.
  struct Cursor { int p, begin, end; };
  auto locate = [&](Cursor& c, int t) -> Pair420 {
    if(!LIST) { return Pair420{ descs, t }; }
    while(t >= c.end) { c.p++; c.begin = c.end; c.end = prefix[c.p + 1]; }
    return Pair420{ &descs[c.p], t - c.begin };
  };
  Cursor here{ -1, 0, 0 }, next{ -1, 0, 0 };

  const int warp = __shfl_sync(kFull, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int dir = warp >> 2, by = warp & 3;   // direction and block row of the thread's 4x4 block (column block: lane)
  next_may_start();
  if(threadIdx.x == 0) { mbar_init(bar, 1); mbar_init(bar + 1, 1); fence_barrier_init(); }
  build_offsets420<R, T>(s_off);
  __syncthreads();
  int t = blockIdx.x;
  if(t < ntiles && threadIdx.x == 0)
  {
    const Pair420 L = locate(next, t);
    if(L.k->g.use_tma) { issue_tile420<R, T, TM>(*L.k, LIST, raw, bar, L.tile); }
  }
  // the next tile's copies, once every warp is done with the raw stage they go to
  auto issue_next = [&](int tn, uint32_t to) {
    if(tn < ntiles && threadIdx.x == 0)
    {
      const int last = next.p;
      const Pair420 N = locate(next, tn);
      if(N.k->g.use_tma)
      {
        fence_proxy_async();
        issue_tile420<R, T, TM>(*N.k, next.p != last, raw + to * G::STAGE, bar + to, N.tile);
      }
    }
  };
  uint32_t stage = 0, parity = 0;             // bit s of parity: phase of stage s's next copies
  const CpsKernelArgs* cur = nullptr;
  for(; t < ntiles; t += gridDim.x, stage = G::STAGES == 2 ? stage ^ 1u : 0u)
  {
    const Pair420 L = locate(here, t);
    unsigned char* box = raw + stage * G::STAGE;
    const bool tma = L.k->g.use_tma != 0;
    bool ok = true;
    if(tma)
    {
      ok = mbar_wait(bar + stage, (parity >> stage) & 1u, kWaitCycles);
      parity ^= 1u << stage;
    }
    // every warp is past the previous tile: the staged rows and the other raw stage are free
    if(__syncthreads_or(!ok))
    {
      // the copies did not complete: report, give them one more bounded wait, stop
      if(threadIdx.x == 0) { atomicOr(L.k->g.status, 8); mbar_wait(bar + stage, ((parity >> stage) & 1u) ^ 1u, kWaitCycles); }
      return;
    }
    if(L.k != cur)
    {
      const uint32_t* sa = reinterpret_cast<const uint32_t*>(&L.k->a);
      for(int w = threadIdx.x; w < (int)(sizeof(CpsArgs) / 4); w += G::NT) { reinterpret_cast<uint32_t*>(&s_a)[w] = sa[w]; }
      if(threadIdx.x < 4)
      {
        const PairOut* src = L.k->a.gcd_src;
        s_gcd[threadIdx.x] = threadIdx.x < 3 ? src->gcd[threadIdx.x] : src->flags;
      }
      __syncthreads();
      cur = L.k;
    }
    const CpsArgs& a = s_a;
    const int ntx = L.k->g.ntx;
    const int tyi = L.tile / ntx, txi = L.tile - tyi * ntx;
    const int x0 = txi * G::TW, y0 = tyi * G::TH;
    if(!tma) { load_plain420<R, T, TM>(a, box, x0, y0); __syncthreads(); }
    const bool clip = a.clip < (sizeof(T) == 1 ? 0xffu : 0xffffu);
    const bool border = x0 < R || y0 < R || x0 + G::TW + R > a.W || y0 + G::TH + R > a.H;
    if(clip || border) { complete_halo<R, T, TM>(a, box, x0, y0, clip, border); }
    const int xb = x0 + 4 * lane, yb = y0 + 4 * by;
    bool kept = true;
    if constexpr(G::MASK)
    {
      // A pixel with M = 0 adds nothing: a warp without another in its strip skips search and epilogue, a tile
      // without another is done.
      const uint32_t strips = kept_strips<R, T, TM>(box, lane);
      kept = (strips >> by) & 1u;
      if(strips == 0u)                                      // the same for every warp
      {
        if(G::STAGES == 1) { __syncthreads(); }             // the one raw stage has been read
        issue_next(t + (int)gridDim.x, G::STAGES == 2 ? stage ^ 1u : 0u);
        continue;
      }
    }
    const uint32_t kw0 = G::K * (uint32_t)a.wi[0], kw1 = G::K * (uint32_t)a.wi[1], kw2 = G::K * (uint32_t)a.wi[2];
    const int32_t mid = a.key_mid;
    stage420<R, T, TM>(box, luma, chroma, kw0, kw1, kw2, G::K * a.key_bias, mid, a.key_masked);
    __syncthreads();
    if(G::STAGES == 2) { issue_next(t + (int)gridDim.x, stage ^ 1u); }
    if(!G::MASK || kept)
    {
      // dir 0 (R2T): test = In0 + GCD searched in In1 -> rows[0], SCP1 = clip(In1[best] - GCD)
      // dir 1 (T2R): test = In1 - GCD searched in In0 -> rows[1], SCP0 = clip(In0[best] + GCD)
      const int sg = dir ? -1 : 1;
      const int g0 = sg * s_gcd[0], g1 = sg * s_gcd[1], g2 = sg * s_gcd[2];
      const unsigned char* tst = box + dir * G::PIC;
      const unsigned char* ref = box + (dir ^ 1) * G::PIC;
      uint32_t idx[16];
      const int lofs = 4 * by * G::BWL + (G::AX - R) + 4 * lane, cofs = 2 * by * G::BWC + (G::AX - G::CR0) + 2 * lane;
      if(G::MASK || (s_gcd[3] & 4) == 0)
      {
        uint32_t c0[16], c1[4], c2[4], ty[16], tu[4], tv[4];
        load_test420<R, T>(tst, by, lane, 0, ty, tu, tv);
        const uint32_t m0 = 0u - 2u * kw0, m1 = 0u - 2u * kw1, m2 = 0u - 2u * kw2;
        const uint32_t o0 = m0 * (uint32_t)(g0 - mid), o1 = m1 * (uint32_t)(g1 - mid), o2 = m2 * (uint32_t)(g2 - mid);
        #pragma unroll
        for(int p = 0; p < 16; p++) { c0[p] = m0 * ty[p] + o0; }
        #pragma unroll
        for(int b = 0; b < 4; b++) { c1[b] = m1 * tu[b] + o1; c2[b] = m2 * tv[b] + o2; }
        // held in registers from here on: recomputed from the test samples at every use they would
        // cost the search as many multiply-adds again
        #pragma unroll
        for(int p = 0; p < 16; p++) { asm volatile("" : "+r"(c0[p])); }
        #pragma unroll
        for(int b = 0; b < 4; b++) { asm volatile("" : "+r"(c1[b]), "+r"(c2[b])); }
        search420<R, T>(luma + (dir ^ 1) * (G::SH * G::LPP) + 4 * by * G::LPP + lane,
                        chroma + (dir ^ 1) * (G::CH * G::CPP) + 2 * by * G::CPP + lane, c0, c1, c2, idx);
      }
      else
      {
        uint32_t found[16];
        search420_literal<R, T>(tst, ref, lofs, cofs, (uint32_t)a.wi[0], (uint32_t)a.wi[1], (uint32_t)a.wi[2], g0, g1, g2, found);
        #pragma unroll
        for(int p = 0; p < 16; p++) { idx[p] = found[p]; }
      }
      // the test samples are read again: kept through the search they would take 24 registers from it
      uint32_t ty[16], tu[4], tv[4];
      int zero = 0;
      asm volatile("" : "+r"(zero));
      load_test420<R, T>(tst, by, lane, zero, ty, tu, tv);
      const uint32_t base = (uint32_t)(lofs * G::ESZ) | ((uint32_t)(cofs * G::ESZ) << 16);
      if constexpr(G::MASK)
      {
        epilogue420_masked<R, T, TM>(a, ref, reinterpret_cast<const TM*>(box + G::OFFM) + (4 * by + R) * G::BWM + G::AXM + 4 * lane, s_off, base, ty, tu,
                                     tv, idx, dir, xb, yb, g0, g1, g2);
      }
      else
      {
      const int sel = ((x0 + G::TW > a.W || y0 + G::TH > a.H) ? 4 : 0) | (a.mom[dir].p != nullptr ? 2 : 0) |
                      ((dir ? a.scp0 : a.scp1) != nullptr ? 1 : 0);
      switch(sel)
      {
      case 0: epilogue420<R, T, false, false, false>(a, ref, s_off, base, ty, tu, tv, idx, dir, xb, yb, g0, g1, g2); break;
      case 1: epilogue420<R, T, false, false, true>(a, ref, s_off, base, ty, tu, tv, idx, dir, xb, yb, g0, g1, g2); break;
      case 2: epilogue420<R, T, false, true, false>(a, ref, s_off, base, ty, tu, tv, idx, dir, xb, yb, g0, g1, g2); break;
      case 4: epilogue420<R, T, true, false, false>(a, ref, s_off, base, ty, tu, tv, idx, dir, xb, yb, g0, g1, g2); break;
      case 6: epilogue420<R, T, true, true, false>(a, ref, s_off, base, ty, tu, tv, idx, dir, xb, yb, g0, g1, g2); break;
      case 5: epilogue420<R, T, true, false, true>(a, ref, s_off, base, ty, tu, tv, idx, dir, xb, yb, g0, g1, g2); break;
      default: epilogue420<R, T, true, true, true>(a, ref, s_off, base, ty, tu, tv, idx, dir, xb, yb, g0, g1, g2); break;   // 3, 7
      }
      }
    }
    if(G::STAGES == 1)
    {
      __syncthreads();
      issue_next(t + (int)gridDim.x, 0u);
    }
  }
}

template <int R, typename T, typename TM>
__global__ void __launch_bounds__(256, Geo420<R, T, TM>::CTAS) k_cps420(const __grid_constant__ CpsKernelArgs one, int ntiles)
{
  cps420_body<R, T, TM, false>(&one, nullptr, ntiles);
}
// The work list's kernel takes pointers alone: it is what a batch captures into a graph.
template <int R, typename T, typename TM>
__global__ void __launch_bounds__(256, Geo420<R, T, TM>::CTAS) k_cps420_multi(const CpsKernelArgs* __restrict__ descs,
                                                                              const int32_t* __restrict__ prefix, int ntiles)
{
  cps420_body<R, T, TM, true>(descs, prefix, ntiles);
}

// ---- host -------------------------------------------------------------------------------------
// Calls f(Geo420<R, T, TM>) for the runtime (R, sample size, mask sample size; 0 = no mask) of the masked or the
// unmasked forms; false when there is no such form.
template <typename T, typename TM, typename F>
bool with_geo_r(int R, F&& f)
{
  switch(R)
  {
  case 1: f(Geo420<1, T, TM>{}); return true;
  case 2: f(Geo420<2, T, TM>{}); return true;
  case 3: f(Geo420<3, T, TM>{}); return true;
  case 4: f(Geo420<4, T, TM>{}); return true;
  case 5: f(Geo420<5, T, TM>{}); return true;
  default: return false;
  }
}
template <bool MASKED, typename F>
bool with_geo(int R, int esz, int mesz, F&& f)
{
  if constexpr(MASKED)
  {
    switch(esz * 4 + mesz)
    {
    case 1 * 4 + 1: return with_geo_r<uint8_t, uint8_t>(R, f);
    case 1 * 4 + 2: return with_geo_r<uint8_t, uint16_t>(R, f);
    case 2 * 4 + 1: return with_geo_r<uint16_t, uint8_t>(R, f);
    case 2 * 4 + 2: return with_geo_r<uint16_t, uint16_t>(R, f);
    default: return false;
    }
  }
  else
  {
    return mesz != 0 ? false : esz == 1 ? with_geo_r<uint8_t, NoMask>(R, f) : esz == 2 ? with_geo_r<uint16_t, NoMask>(R, f) : false;
  }
}

template <typename G, typename F, typename... A>
cudaError_t launch420(G, F* kernel, int ntiles, cudaStream_t s, A... args)
{
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if(e == cudaSuccess) { e = configure_once(kernel, dev); }
  if(e != cudaSuccess) { return e; }
  kernel<<<grid_for(kernel, G::NT, G::SMEM, ntiles, dev), G::NT, G::SMEM, s>>>(args..., ntiles);
  return cudaGetLastError();
}
template <int R, typename T, typename TM>
cudaError_t launch420_one(Geo420<R, T, TM> g, const CpsKernelArgs& k, cudaStream_t s) { return launch420(g, k_cps420<R, T, TM>, k.g.ntiles, s, k); }
template <int R, typename T, typename TM>
cudaError_t launch420_list(Geo420<R, T, TM> g, const CpsKernelArgs* d, const int32_t* prefix, int ntiles, cudaStream_t s)
{
  return launch420(g, k_cps420_multi<R, T, TM>, ntiles, s, d, prefix);
}

template <bool MASKED>
cudaError_t launch420_any(const CpsKernelArgs& k, int R, int esz, cudaStream_t s)
{
  cudaError_t e = cudaErrorInvalidValue;
  with_geo<MASKED>(R, esz, MASKED ? k.a.mask_esz : 0, [&](auto g) { e = launch420_one(g, k, s); });
  return e;
}
template <bool MASKED>
cudaError_t launch420_list_any(const CpsKernelArgs* d, const int32_t* prefix, int ntiles, int R, int esz, int mesz, cudaStream_t s)
{
  cudaError_t e = cudaErrorInvalidValue;
  with_geo<MASKED>(R, esz, mesz, [&](auto g) { e = launch420_list(g, d, prefix, ntiles, s); });
  return e;
}

}  // namespace

}  // namespace qmiv
