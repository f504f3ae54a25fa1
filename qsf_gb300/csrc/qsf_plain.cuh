// qsf_plain.cuh -- the plain transforms of the member operations (qsf_fourier, region
// transfers): whole tiles staged in shared memory, one exponent per tile.
//
// These keep their tiles, radix plans and block exponents although the register-resident
// lines (qsf_lines.cuh) are a little faster here (4 regions of 1024^2: 24.3 -> 23.1 ms a
// run): the small outer regions of a multi-region grid are sums of margins in which the
// rounding of every earlier transform survives (relative differences of 1e-9 in the
// doubly-free region between two equally accurate roundings), so a change of grouping
// changes results that programs compare between versions.
#pragma once
#include "qsf_fxfft.cuh"

namespace qsf {

constexpr int kPlainThreads = 512;
// Threads of a strided-axis tile: the shapes that steps on such tiles ran fastest with (2D
// steps, ms with 256 / 512 threads: 320 0.090 / 0.074, 384 0.086 / 0.080, 512 0.089 / 0.073,
// 640 0.092 / 0.086, 2048 0.445 / 0.433; 768 0.105 / 0.121, 1024 0.107 / 0.128, 256 alike).
// They stay, because the shape sets the radix plan and with it the rounding (above).
__host__ __device__ constexpr int plain_threads(int n) {
  return n == 320 || n == 384 || n == 512 || n == 640 || n == 2048 ? 512 : 256;
}
// points of a strided-axis tile (one whole line when lines are longer) and its columns
__host__ __device__ constexpr int plain_tile(int n) { return n > 4096 ? n : 4096; }
__host__ __device__ constexpr int plain_ppt(int n) { return plain_tile(n) / plain_threads(n); }

// Lines in shared memory: element e of line l sits at buf[l * ls + e * es].
struct LineSet {
  int nlines;
  int ls;
  int es;
  bool line_fastest;  // work-item order: consecutive threads take consecutive lines
};

// the same from the high words alone (32-bit operations): 32 + the high words' bit
// length, or 0 when every component is below 2^32 in magnitude
__device__ __forceinline__ unsigned fmag_hi(longlong2 x) {
  const int hx = (int)(x.x >> 32), hy = (int)(x.y >> 32);
  return (unsigned)(hx ^ (hx >> 31)) | (unsigned)(hy ^ (hy >> 31));
}
__device__ __forceinline__ int bitlen_hi(unsigned v) { return v ? 64 - __clz((int)v) : 0; }
// guard bits a radix-R pass needs above the block maximum (growth <= R * sqrt(2))
__host__ __device__ constexpr int fguard(int r) { return r == 16 ? 5 : r == 8 ? 4 : r == 5 ? 4 : r == 4 ? 3 : r == 3 ? 3 : 2; }

// Block-wide max of per-thread values over one barrier: every warp's maximum goes to
// slot[warp], then all threads read the slots.  The slots are reused only after at
// least one further barrier (the FFT passes alternate between two slot arrays).
__device__ __forceinline__ int block_max_once(int v, int* slot) {
  v = __reduce_max_sync(0xffffffffu, (unsigned)v);
  if ((threadIdx.x & 31) == 0) slot[threadIdx.x >> 5] = v;
  __syncthreads();
  const int nw = (blockDim.x + 31) >> 5;
  int m = 0;
  for (int w = 0; w < nw; ++w) m = max(m, slot[w]);
  return m;
}

// Block-wide max of per-thread values (red[0..31]); result returned to all.  The
// shared arrays named red in the kernels hold kRedInts ints: [0, 32) for this function,
// [32, 96) for the alternating slots of the FFT passes.
constexpr int kRedInts = 96;
__device__ __forceinline__ int block_max_int(int v, int* red) {
  v = __reduce_max_sync(0xffffffffu, (unsigned)v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  if (lane == 0) red[wid] = v;
  __syncthreads();
  int m = 0;
  for (int w = 0; w < nw; ++w) m = max(m, red[w]);
  __syncthreads();
  return m;
}

// One in-place forward Stockham pass in fixed point (an inverse transform is the
// forward one between two conjugations) with stride NS (the product of the earlier
// radices; a runtime value, so that passes of equal radix share one code body).
// Inputs are scaled by 2^shift_in on load; returns, valid in every thread after the
// call, the bit length of the block's largest output component (see fmag).
template <int R, int MAXB, int N>
__device__ __forceinline__ int fx_stockham(longlong2* __restrict__ buf, const LineSet& L, const int4* __restrict__ tw,
                                           int tid, int nth, int shift_in, int* red, int parity, int NS) {
  constexpr int nr = N / R;
  constexpr bool kSplit = R > 2;
  const int twstep = N / (NS * R);
  const int total = nr * L.nlines;
  // the load-time scaling 2^shift_in without branches: (x << sl + half) >> sr; with
  // pre-split twiddles the elements that get one (q >= 1 of a pass after the first)
  // are loaded 2 bits higher (sl2 / sr2), since their product is a * w / 2^64
  const int sl = shift_in > 0 ? shift_in : 0, sr = shift_in < 0 ? min(-shift_in, 63) : 0;
  const i64 half = sr ? (i64)1 << (sr - 1) : 0;
  const int shift_q = (kSplit && NS > 1) ? shift_in + 2 : shift_in;
  const int sl2 = shift_q > 0 ? shift_q : 0, sr2 = shift_q < 0 ? min(-shift_q, 63) : 0;
  const i64 half2 = sr2 ? (i64)1 << (sr2 - 1) : 0;
  // index maps without divisions where the counts are powers of two
  const bool ns_pow2 = (NS & (NS - 1)) == 0;
  const bool nl_pow2 = (L.nlines & (L.nlines - 1)) == 0;
  const int nl_sh = __ffs(L.nlines) - 1;
  longlong2 v[MAXB][R];
  int dsto[MAXB];
#pragma unroll
  for (int b = 0; b < MAXB; ++b) {
    const int w = tid + b * nth;
    dsto[b] = -1;
    if (w < total) {
      int line, j;
      if (L.line_fastest) {
        line = nl_pow2 ? (w & (L.nlines - 1)) : w % L.nlines;
        j = nl_pow2 ? (w >> nl_sh) : w / L.nlines;
      } else {
        j = w % nr;
        line = w / nr;
      }
      const longlong2* src = buf + line * L.ls;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        const longlong2 x = src[(j + q * nr) * L.es];
        if (q == 0)
          v[b][q] = make_longlong2(((i64)((u64)x.x << sl) + half) >> sr, ((i64)((u64)x.y << sl) + half) >> sr);
        else
          v[b][q] = make_longlong2(((i64)((u64)x.x << sl2) + half2) >> sr2, ((i64)((u64)x.y << sl2) + half2) >> sr2);
      }
      const int jm = ns_pow2 ? (j & (NS - 1)) : j % NS;
      if (NS > 1) {
#pragma unroll
        for (int q = 1; q < R; ++q) {
          if constexpr (kSplit) v[b][q] = fmul_tw(v[b][q], tw[jm * q * twstep]);
          else v[b][q] = fmul62(v[b][q], tw_join(tw[jm * q * twstep]));
        }
      }
      dsto[b] = line * L.ls + ((j - jm) * R + jm) * L.es;
    }
  }
  __syncthreads();
  unsigned mag = 0;
#pragma unroll
  for (int b = 0; b < MAXB; ++b) {
    if (dsto[b] >= 0) {
      fbfly<R, true>(v[b]);
      longlong2* dst = buf + dsto[b];
      const int st = NS * L.es;
#pragma unroll
      for (int q = 0; q < R; ++q) {
        dst[q * st] = v[b][q];
        mag |= fmag_hi(v[b][q]);
      }
    }
  }
  int bits = block_max_once(bitlen_hi(mag), red + 32 + 32 * parity);  // its barrier ends the pass
  if (bits == 0) {  // every component below 2^32 (rare): bit length from the full words
    u64 m64 = 0;
#pragma unroll
    for (int b = 0; b < MAXB; ++b)
      if (dsto[b] >= 0)
#pragma unroll
        for (int q = 0; q < R; ++q) m64 |= fmag(v[b][q]);
    bits = block_max_int(bitlen(m64), red);
  }
  return bits;
}

// Full forward fixed-point transform of every line of the set, in place.  On entry
// the data have block exponent `scale` (value = int * 2^-scale) and, after the shift
// 2^shift_in applied on load, fit the first pass's guard; on return `scale` is the
// exponent of the output and its largest component has bit length `bits`.
// Requires nlines * N <= 16 * nth.  The passes run as a loop over the stages with one
// inlined pass body per distinct radix of N (instruction-cache footprint).
// radix_at(N, s, L2) for a runtime stage index, from compile-time stage counts
template <int N, int L2>
__device__ __forceinline__ int radix_rt(int s) {
  constexpr int a = count_factor(N, 2), q = a / L2, rem = a % L2;
  constexpr int c3 = count_factor(N, 3);
  if (s < q) return 1 << L2;
  int k = s - q;
  if (rem) {
    if (k == 0) return 1 << rem;
    k -= 1;
  }
  return k < c3 ? 3 : 5;
}
// butterflies per thread of radix R when every thread holds PPT points of the tile
__host__ __device__ constexpr int maxb_ppt(int r, int ppt) { return (ppt + r - 1) / r; }

// main radix of the plan for PPT points per thread: radix 16 needs 16 per thread,
// radix 8 needs 8, radix 4 four
__host__ __device__ constexpr int plan_l2(int ppt) { return ppt >= 16 ? QSF_RADIX_LOG2 : ppt >= 8 ? 3 : 2; }

// the compile-time stages S.. of fft_fx
template <int N, int S, int PPT>
__device__ __forceinline__ void fft_fx_tail(longlong2* buf, const LineSet& L, const int4* __restrict__ tw,
                                            int tid, int nth, int& scale, int& bits, int* red, int shift_in) {
  constexpr int L2 = plan_l2(PPT);
  if constexpr (S < nstages(N, L2)) {
    constexpr int R = radix_at(N, S, L2);
    bits = fx_stockham<R, maxb_ppt(R, PPT), N>(buf, L, tw, tid, nth, shift_in, red, S & 1, ns_at(N, S, L2));
    if constexpr (S + 1 < nstages(N, L2)) {
      // renormalise for the next pass: largest component below 2^(62 - guard(next))
      const int target = 62 - fguard(radix_at(N, S + 1, L2));
      const int sh = bits == 0 ? 0 : target - bits;
      scale += sh;
      fft_fx_tail<N, S + 1, PPT>(buf, L, tw, tid, nth, scale, bits, red, sh);
    }
  }
}
// PPT: points of the tile per thread (tile points / threads), which sets the butterflies
// each thread carries per pass.
template <int N, int PPT = 16>
__device__ __forceinline__ void fft_fx(longlong2* buf, const LineSet& L, const int4* __restrict__ tw, int tid,
                                       int nth, int& scale, int& bits, int* red, int shift_in = 0) {
  // the leading passes of the plan's main radix share one code body (a loop); the rest
  // are unrolled
  constexpr int L2 = plan_l2(PPT);
  constexpr int R0 = 1 << L2;
  constexpr int q = count_factor(N, 2) / L2;
  if constexpr (q >= 2) {
    int sh = shift_in, ns = 1;
#pragma unroll 1
    for (int s = 0; s < q; ++s) {
      bits = fx_stockham<R0, maxb_ppt(R0, PPT), N>(buf, L, tw, tid, nth, sh, red, s & 1, ns);
      ns *= R0;
      if (s + 1 < nstages(N, L2)) {
        const int target = 62 - fguard(radix_rt<N, L2>(s + 1));
        sh = bits == 0 ? 0 : target - bits;
        scale += sh;
      }
    }
    fft_fx_tail<N, q, PPT>(buf, L, tw, tid, nth, scale, bits, red, sh);
  } else {
    fft_fx_tail<N, 0, PPT>(buf, L, tw, tid, nth, scale, bits, red, shift_in);
  }
}

// fourier<R>() without phases, in block fixed point: each block takes its exponent from
// the largest double it loads (one global read, staged in smem), converts with integer
// operations, runs the fixed-point passes (an inverse is the forward transform between two
// conjugations) and converts back (times post_scale).
template <int N, bool FWD>
__global__ void __launch_bounds__(kPlainThreads, 1) k_row_fft(GridDev g, int L, double post_scale) {
  extern __shared__ __align__(128) longlong2 smx[];
  __shared__ int red[kRedInts];
  const AxisDev& a = g.ax[g.dim - 1];
  const long long row0 = (long long)blockIdx.x * L;
  const long long nrows = g.m / N;
  const int Lh = (int)min((long long)L, nrows - row0);
  const long long base = row0 * N;
  const int cnt = Lh * N;
  double2* sd = reinterpret_cast<double2*>(smx);
  int em = 0;
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    const double2 v = g.psi[base + e];
    sd[e] = v;
    em = max(em, max(dexp(v.x), dexp(v.y)));
  }
  em = block_max_int(em, red);
  int scale = (62 - fguard(radix_at(N, 0))) - (em - 1022);
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    const double2 v = sd[e];
    const longlong2 x = make_longlong2(d2fx(v.x, scale), d2fx(v.y, scale));
    smx[e] = FWD ? x : fconj(x);
  }
  __syncthreads();
  const LineSet ls{Lh, N, 1, false};
  int bits = 0;
  fft_fx<N>(smx, ls, a.tw, threadIdx.x, blockDim.x, scale, bits, red);
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    const longlong2 x = FWD ? smx[e] : fconj(smx[e]);
    double2 v = make_double2(fx2d(x.x, scale), fx2d(x.y, scale));
    if (post_scale != 1.0) v = cscale(v, post_scale);
    g.psi[base + e] = v;
  }
}

template <int N, bool FWD>
__global__ void __launch_bounds__(plain_threads(N), 2) k_axis_fft(GridDev g, int ax, int C, double post_scale) {
  extern __shared__ __align__(128) longlong2 smx[];
  __shared__ int red[kRedInts];
  const AxisDev& a = g.ax[ax];
  const long long inner = a.stride;
  const long long tiles_per_outer = (inner + C - 1) / C;
  const long long o = blockIdx.x / tiles_per_outer;
  const long long c0 = (blockIdx.x % tiles_per_outer) * C;
  const int Ch = (int)min((long long)C, inner - c0);
  const long long obase = o * (long long)N * inner + c0;
  const int cnt = N * Ch;
  double2* sd = reinterpret_cast<double2*>(smx);
  int em = 0;
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    const int i = e / Ch, c = e % Ch;
    const double2 v = g.psi[obase + (long long)i * inner + c];
    sd[i * C + c] = v;
    em = max(em, max(dexp(v.x), dexp(v.y)));
  }
  em = block_max_int(em, red);
  int scale = (62 - fguard(radix_at(N, 0))) - (em - 1022);
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    const int i = e / Ch, c = e % Ch;
    const double2 v = sd[i * C + c];
    const longlong2 x = make_longlong2(d2fx(v.x, scale), d2fx(v.y, scale));
    smx[i * C + c] = FWD ? x : fconj(x);
  }
  __syncthreads();
  const LineSet ls{Ch, 1, C, true};
  int bits = 0;
  fft_fx<N, plain_ppt(N)>(smx, ls, a.tw, threadIdx.x, blockDim.x, scale, bits, red);
  for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
    const int i = e / Ch, c = e % Ch;
    const longlong2 x = FWD ? smx[i * C + c] : fconj(smx[i * C + c]);
    double2 v = make_double2(fx2d(x.x, scale), fx2d(x.y, scale));
    if (post_scale != 1.0) v = cscale(v, post_scale);
    g.psi[obase + (long long)i * inner + c] = v;
  }
}

}  // namespace qsf
