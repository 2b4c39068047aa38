/*
  qmiv_probe.h — measurement utilities of the QMIV B200 library (no counterpart in the reference).

  The corresponding-pixel-shift search is bound by the SM's integer/FP32 issue rate, not by HBM or
  tensor cores. These probes measure, on the device they run on, the sustained rate of the simple
  32-bit integer operations (add, min) and of FP32 FMAs, so that the search kernel's roofline is a
  fraction of a measured number; the FP64 probe does the same for the regular-window SSIM kernel.
  qmiv_probe_cps_keys reports the constants of the 4:2:0 search's integer keys; it needs no GPU.
*/
#ifndef QMIV_PROBE_H
#define QMIV_PROBE_H
#include <stdint.h>
#include "qmiv_gpu.h"

#ifdef __cplusplus
extern "C" {
#endif

/* Sustained 32-bit integer add/min throughput in tera-operations per second (each add and each min
   counts as one operation), measured with CUDA events over `iters` iterations per thread. */
QMIV_API qmiv_status qmiv_probe_int32_peak(int32_t device, int32_t iters, double* tops);

/* Sustained FP32 FMA throughput in TFLOP/s (2 flops per FMA). */
QMIV_API qmiv_status qmiv_probe_fp32_peak(int32_t device, int32_t iters, double* tflops);

/* Sustained FP64 multiply and add throughput in tera-operations per second (each separately rounded
   DMUL and DADD counts as one operation), the instruction mix of the SSIM window sums. */
QMIV_API qmiv_status qmiv_probe_fp64_peak(int32_t device, int32_t iters, double* tops);

/* The 4:2:0 search's integer keys for samples 0..max_sample, the first three search weights and bounds of
   |GCD| per component: whether they order every candidate as the reference does (else the search is done
   by literal int32 errors), without and with a mask, and the constants they use. */
typedef struct qmiv_cps_keys
{
  int32_t  shared, masked;   /* 1: the unmasked / masked search takes the keys */
  int32_t  key_bits;         /* a key is (biased error << key_bits) + raster code */
  int32_t  mid;              /* samples are taken relative to this value */
  uint32_t bias;             /* added to the error before the shift */
  uint32_t masked_value;     /* staged square term of a masked sample */
  int32_t  sum_split;        /* masked row sums: a lane's terms are summed below and from this bit up */
} qmiv_cps_keys;
QMIV_API qmiv_status qmiv_probe_cps_keys(int32_t search_range, int32_t max_sample, const int32_t weights[3],
                                         const int32_t gcd_bound[3], qmiv_cps_keys* out);

#ifdef __cplusplus
}
#endif
#endif
