// qsf_tuning.h -- pass kernel shapes per line length: the points per thread of the row
// passes, and the radix plan of the one-CTA 1D line kernel.
//
// Written by the autotuner (qsf_gb300/autotune.py) from step times measured on a GB300:
//   python -m qsf_gb300.autotune --write
// Row passes: points x threads, whose ratio is the points per thread and selects the
// line plan (16: radix-16 plans, 128 registers; 8: radix-8 plans); lengths not listed
// take 4096x256.
// Measured (one call of graph-replayed steps per workload, ms per step):
//   2d64    ms/step  4096x256: 0.0341  4096x512: 0.0272
//   2d128   ms/step  4096x256: 0.0386  4096x512: 0.0337
//   2d192   ms/step  4096x256: 0.0336  4096x512: 0.0311
//   2d256   ms/step  4096x256: 0.0399  4096x512: 0.0336
//   2d320   ms/step  4096x256: 0.0514  4096x512: 0.0367
//   2d384   ms/step  4096x256: 0.0437  4096x512: 0.0363
//   2d512   ms/step  4096x256: 0.0374  4096x512: 0.0313
//   2d640   ms/step  4096x256: 0.0628  4096x512: 0.0527
//   2d768   ms/step  4096x256: 0.0571  4096x512: 0.0573
//   2d1024  ms/step  4096x256: 0.0821  4096x512: 0.0742
//   2d1280  ms/step  4096x256: 0.1663  4096x512: 0.1486
//   2d1536  ms/step  4096x256: 0.2175  4096x512: 0.2085
//   2d2048  ms/step  4096x256: 0.2927  4096x512: 0.3003
//   2d4096  ms/step  4096x256: 1.1692  4096x512: 1.3821
//   3d128   ms/step  4096x256: 0.2212  4096x512: 0.2097
//   3d256   ms/step  4096x256: 1.3053  4096x512: 1.1908
#pragma once

namespace qsf {

__host__ __device__ constexpr int tuned_row_threads(int n) {
  return n == 64 ? 512 : n == 128 ? 512 : n == 192 ? 512 : n == 256 ? 512 : n == 320 ? 512 : n == 384 ? 512 : n == 512 ? 512 : n == 640 ? 512 : n == 1024 ? 512 : n == 1280 ? 512 : n == 1536 ? 512 : 256;
}

__host__ __device__ constexpr int tuned_tile(int n) {
  return 4096;
}

// Points per thread of 1D lines held by one CTA as one line (up to 320 points; 8: radix-8
// plans, 16: radix 16); a length between measured ones takes the plan of the next longer
// measured length.  Measured (one call of graph-replayed steps, points per
// thread: ms per step):
//   1d64    ms/step  8: 0.0114  16: 0.0316
//   1d128   ms/step  8: 0.0120  16: 0.0330
//   1d320   ms/step  8: 0.0171  16: 0.0425
__host__ __device__ constexpr int tuned_line_ppt(int n) {
  return n <= 320 ? 8 : 16;
}

}  // namespace qsf
