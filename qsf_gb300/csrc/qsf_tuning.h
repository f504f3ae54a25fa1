// qsf_tuning.h -- pass kernel shapes per line length: the points per thread of the row
// passes, and the radix plan of the one-CTA 1D line kernel.
//
// Written by the autotuner (qsf_gb300/autotune.py) from step times measured on a GB300:
//   python -m qsf_gb300.autotune --write
// Row passes: points x threads, whose ratio is the points per thread and selects the
// line plan (16: radix-16 plans, 128 registers; 8: radix-8 plans); lengths not listed
// take 4096x256.
// Measured (one call of graph-replayed steps per workload, ms per step):
//   2d64    ms/step  4096x256: 0.0356  4096x512: 0.0308
//   2d128   ms/step  4096x256: 0.0382  4096x512: 0.0343
//   2d192   ms/step  4096x256: 0.0355  4096x512: 0.0339
//   2d256   ms/step  4096x256: 0.0397  4096x512: 0.0339
//   2d320   ms/step  4096x256: 0.0527  4096x512: 0.0403
//   2d384   ms/step  4096x256: 0.0443  4096x512: 0.0380
//   2d512   ms/step  4096x256: 0.0400  4096x512: 0.0342
//   2d640   ms/step  4096x256: 0.0674  4096x512: 0.0603
//   2d768   ms/step  4096x256: 0.0630  4096x512: 0.0629
//   2d1024  ms/step  4096x256: 0.0853  4096x512: 0.0793
//   2d1280  ms/step  4096x256: 0.1569  4096x512: 0.1661
//   2d1536  ms/step  4096x256: 0.2077  4096x512: 0.2000
//   2d2048  ms/step  4096x256: 0.2871  4096x512: 0.2873
//   2d4096  ms/step  4096x256: 1.1613  4096x512: 1.3885
//   3d128   ms/step  4096x256: 0.1928  4096x512: 0.1854
//   3d256   ms/step  4096x256: 1.3193  4096x512: 1.2235
#pragma once

namespace qsf {

__host__ __device__ constexpr int tuned_row_threads(int n) {
  return n == 64 ? 512 : n == 128 ? 512 : n == 192 ? 512 : n == 256 ? 512 : n == 320 ? 512 : n == 384 ? 512 : n == 512 ? 512 : n == 640 ? 512 : n == 768 ? 512 : n == 1024 ? 512 : n == 1536 ? 512 : 256;
}

__host__ __device__ constexpr int tuned_tile(int n) {
  return 4096;
}

// Points per thread of 1D lines held by one CTA as one line (up to 640 points; 8: radix-8
// plans, 16: radix 16); a length between measured ones takes the plan of the next longer
// measured length.  Measured (one call of graph-replayed steps, points per
// thread: ms per step):
//   1d64    ms/step  8: 0.0113  16: 0.0314
//   1d128   ms/step  8: 0.0120  16: 0.0329
//   1d256   ms/step  8: 0.0129  16: 0.0338
//   1d384   ms/step  8: 0.0161  16: 0.0394
//   1d640   ms/step  8: 0.0199  16: 0.0434
__host__ __device__ constexpr int tuned_line_ppt(int n) {
  return n <= 640 ? 8 : 16;
}

}  // namespace qsf
