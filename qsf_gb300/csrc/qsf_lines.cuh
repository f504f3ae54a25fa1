// qsf_lines.cuh -- register-resident block-fixed-point line transforms.
//
// A line of N points is held by T = N / E threads, E points each: thread t owns the
// points t + s T (s < E) on entry and on return.  Every radix pass works on registers;
// between two passes the line is exchanged once through shared memory.  Because the
// first pass of a transform reads, and the last pass writes, the same E points of a
// thread, whatever happens between two transforms of one line (the P phase between the
// forward and the inverse transform, the closing and the next opening X half between
// the inverse and the next forward one) is a loop over registers: a pass kernel loads
// each point from global memory once, exchanges it twice per transform (three-pass
// plans) and stores it once.
//
// What bounds it: the issue of integer instructions (the arithmetic of qsf_fxfft.cuh).
// What the layout saves over staging every pass and every sweep in shared memory: at
// 2048 points a pass kernel makes 4 exchanges where it made 17 reads and writes of the
// tile, and the renormalising shift between passes costs nothing (below).
//
// Scaling.  Each group of threads that synchronises together (sync kinds below) keeps
// one power-of-two exponent.  After a pass the group's largest component has `bits`
// bits; the next pass needs it below 2^(62 - guard), i.e. the data shifted right by
// s = bits - (62 - guard).  A twiddle product returns x w / 4 per 2^62 twiddle, so s = 2
// is free, s = 2 + r reads the twiddles from a copy of the table scaled by 2^-r (r <=
// 4), and s < 2 shifts x left by 2 - s first: no element is shifted right and rounded on
// its own except the untwiddled one of each butterfly.
#pragma once
#include "qsf_fxfft.cuh"
#include "qsf_tuning.h"

namespace qsf {

// Shape of the pass kernels per line length, as the autotuner measured it (qsf_tuning.h):
// points per block over threads per block is the points per thread, which selects the
// line plan below (16 or more: radix 16; 8: radix 8).  The autotuner's candidate builds
// define QSF_TILE and QSF_ROW_THREADS to force one shape everywhere.
#ifdef QSF_ROW_THREADS
__host__ __device__ constexpr int row_threads(int) { return QSF_ROW_THREADS; }
#else
__host__ __device__ constexpr int row_threads(int n) { return tuned_row_threads(n); }
#endif
#ifdef QSF_TILE
__host__ __device__ constexpr int tile_size(int) { return QSF_TILE; }
#else
__host__ __device__ constexpr int tile_size(int n) { return tuned_tile(n); }
#endif
__host__ __device__ constexpr int tuned_ppt(int n) { return tile_size(n) / row_threads(n); }
// Points per thread of the strided-axis passes (candidate builds force one with QSF_COL_PPT):
// 16 from 1024 points on, where the lines fill the SMs, and at 256, where cubes gain what
// planes run alone lose; 128 goes with 256.  ms a step with 8 / 16 points, 2D: 64 0.0275 /
// 0.0300, 128 0.0289 / 0.0333, 256 0.0282 / 0.0336, 512 0.0312 / 0.0411, 768 0.0570 / 0.0634,
// 1024 0.0810 / 0.0742, 1280 0.173 / 0.164, 2048 0.329 / 0.294, 4096 1.333 / 1.164; 3D: 64
// 0.0489 / 0.0579, 128 0.206 / 0.210, 256 1.386 / 1.189.
#ifdef QSF_COL_PPT
__host__ __device__ constexpr int axis_ppt(int) { return QSF_COL_PPT; }
#else
__host__ __device__ constexpr int axis_ppt(int n) { return n == 128 || n == 256 || n >= 1024 ? 16 : 8; }
#endif

// ------------------------------------------------------------ plans
// E points per thread, S passes of radix r[0..S-1].  The first and the last radix divide
// E (register ownership); a middle radix need not.  Two plans per length where both make
// sense, selected by the tuned points per thread (16 or 8): more points per thread save
// passes and twiddles, fewer give more warps.
struct LinePlan {
  int E, S, r[4];
};
constexpr int kEight = 1, kFour = 2;  // plan selectors: the factors of 1D lines (qsf_line1d.cuh), 8 or 4 points per thread
__host__ __device__ constexpr LinePlan line_plan(int n, int ppt) {
  if (ppt == kFour) {
    switch (n) {
      case 16: return {4, 2, {4, 4, 1, 1}};
      case 24: return {4, 3, {4, 3, 2, 1}};
      case 32: return {4, 3, {4, 2, 4, 1}};
      case 40: return {4, 3, {4, 5, 2, 1}};
      case 48: return {4, 3, {4, 3, 4, 1}};
      case 64: return {4, 3, {4, 4, 4, 1}};
      case 80: return {4, 3, {4, 5, 4, 1}};
      case 96: return {4, 4, {4, 3, 2, 4}};
      case 128: return {4, 4, {4, 2, 4, 4}};
      case 160: return {4, 4, {4, 5, 2, 4}};
      case 192: return {4, 4, {4, 3, 4, 4}};
      default: return {0, 0, {1, 1, 1, 1}};
    }
  }
  if (ppt == kEight) {
    switch (n) {
      case 128: return {8, 3, {8, 2, 8, 1}};
      case 160: return {8, 3, {8, 5, 4, 1}};
      case 192: return {8, 3, {8, 3, 8, 1}};
      case 256: return {8, 3, {8, 4, 8, 1}};
      default: return {0, 0, {1, 1, 1, 1}};
    }
  }
  const bool w = ppt >= 16;
  switch (n) {
    case 8: return {8, 1, {8, 1, 1, 1}};
    case 12: return {12, 1, {12, 1, 1, 1}};
    case 16: return {16, 1, {16, 1, 1, 1}};
    case 20: return {20, 1, {20, 1, 1, 1}};
    case 24: return {12, 2, {12, 2, 1, 1}};
    case 32: return {8, 2, {8, 4, 1, 1}};
    case 40: return {20, 2, {20, 2, 1, 1}};
    case 48: return {12, 2, {12, 4, 1, 1}};
    case 64: return w ? LinePlan{16, 2, {16, 4, 1, 1}} : LinePlan{8, 2, {8, 8, 1, 1}};
    case 80: return {20, 2, {20, 4, 1, 1}};
    case 96: return {12, 3, {12, 2, 4, 1}};
    case 128: return w ? LinePlan{16, 2, {16, 8, 1, 1}} : LinePlan{8, 3, {8, 2, 8, 1}};
    case 160: return w ? LinePlan{20, 3, {20, 2, 4, 1}} : LinePlan{8, 3, {8, 5, 4, 1}};
    case 192: return w ? LinePlan{12, 3, {12, 4, 4, 1}} : LinePlan{8, 3, {8, 3, 8, 1}};
    case 256: return w ? LinePlan{16, 2, {16, 16, 1, 1}} : LinePlan{8, 3, {8, 4, 8, 1}};
    case 320: return w ? LinePlan{16, 3, {16, 5, 4, 1}} : LinePlan{8, 3, {8, 5, 8, 1}};
    case 384: return w ? LinePlan{16, 3, {16, 3, 8, 1}} : LinePlan{8, 3, {8, 6, 8, 1}};
    case 512: return w ? LinePlan{16, 3, {16, 2, 16, 1}} : LinePlan{8, 3, {8, 8, 8, 1}};
    case 640: return w ? LinePlan{16, 3, {16, 5, 8, 1}} : LinePlan{8, 3, {8, 10, 8, 1}};
    case 768: return w ? LinePlan{16, 3, {16, 3, 16, 1}} : LinePlan{8, 3, {8, 12, 8, 1}};
    case 1024: return w ? LinePlan{16, 3, {16, 4, 16, 1}} : LinePlan{8, 4, {8, 2, 8, 8}};
    case 1280: return w ? LinePlan{16, 3, {16, 5, 16, 1}} : LinePlan{8, 4, {8, 5, 4, 8}};
    case 1536: return w ? LinePlan{16, 3, {16, 6, 16, 1}} : LinePlan{8, 4, {8, 3, 8, 8}};
    case 2048: return w ? LinePlan{16, 3, {16, 8, 16, 1}} : LinePlan{8, 4, {8, 4, 8, 8}};
    case 2560: return w ? LinePlan{16, 3, {16, 10, 16, 1}} : LinePlan{8, 4, {8, 5, 8, 8}};
    case 3072: return w ? LinePlan{16, 4, {16, 3, 4, 16}} : LinePlan{8, 4, {8, 6, 8, 8}};
    case 4096: return w ? LinePlan{16, 3, {16, 16, 16, 1}} : LinePlan{8, 4, {8, 8, 8, 8}};
    default: return {0, 0, {1, 1, 1, 1}};
  }
}
__host__ __device__ constexpr bool plan_ok(int n, int ppt) {
  const LinePlan p = line_plan(n, ppt);
  if (p.S == 0) return false;
  int m = 1;
  for (int i = 0; i < p.S; ++i) m *= p.r[i];
  return m == n && p.E % p.r[0] == 0 && p.E % p.r[p.S - 1] == 0 && n % p.E == 0;
}
// Guard bits of a radix-R butterfly: R sqrt(2) times the largest component stays below
// 2^62 (the radix-2 and -3 guards are one bit wider than that needs, so that products
// with the twiddles keep the 2^61 bound on their operand)
__host__ __device__ constexpr int line_guard(int r) { return r <= 4 ? 3 : r <= 10 ? 4 : 5; }

constexpr int kTwVar = 5;  // twiddle copies scaled by 2^-0 .. 2^-4

// twiddle entries of pass p (p >= 1): [(q - 1) * ns + jm] = exp(-2 pi i jm q / (ns R)),
// q = 1 .. R - 1, jm < ns, at line_tw_off; one copy is line_tw_len entries
__host__ __device__ constexpr int line_ns(int n, int ppt, int p) {
  const LinePlan L = line_plan(n, ppt);
  int m = 1;
  for (int i = 0; i < p; ++i) m *= L.r[i];
  return m;
}
__host__ __device__ constexpr int line_tw_off(int n, int ppt, int p) {
  const LinePlan L = line_plan(n, ppt);
  int o = 0;
  for (int i = 1; i < p; ++i) o += (L.r[i] - 1) * line_ns(n, ppt, i);
  return o;
}
__host__ __device__ constexpr int line_tw_len(int n, int ppt) { return line_tw_off(n, ppt, line_plan(n, ppt).S); }

// Compile-time layout of the line kernels of one length and plan.
template <int N_, int PPT>
struct Ln {
  static constexpr int N = N_, ppt = PPT;
  static constexpr LinePlan P = line_plan(N, ppt);
  static constexpr int E = P.E, S = P.S, T = N / P.E;
  static_assert(plan_ok(N, ppt), "no line plan for this length");
  __host__ __device__ static constexpr int R(int p) { return P.r[p]; }
  __host__ __device__ static constexpr int NS(int p) { return line_ns(N, ppt, p); }
  // which threads share an exponent and synchronise: 0 a warp (whole lines inside it),
  // 1 the warps of one line, 2 the whole block (line boundaries inside warps)
  static constexpr int kSync = T % 32 == 0 && T > 32 ? 1 : 32 % T == 0 ? 0 : 2;
  // one padding chunk per PD points keeps the first pass's stride-R stores off each
  // other's banks (PD divides the first radix and T, so every address stays base +
  // constant)
  __host__ __device__ static constexpr int pd(int c) { return T % c == 0 && P.r[0] % c == 0; }
  static constexpr int PD = S == 1 ? 0 : pd(16) ? 16 : pd(8) ? 8 : pd(4) ? 4 : 0;
  __host__ __device__ static constexpr int pad(int i) { return PD ? i + i / PD : i; }
  static constexpr int LS = pad(N);  // points of a line in the exchange buffer
  // lines per block.  Rows: about two warps (one line when it has as many threads), so
  // that small grids give as many blocks as they can; a multiple that ends on a warp
  // where lines do not.  Columns: 128-byte row segments where lines are short, 32-byte
  // sectors at 2048 points.
  static constexpr int L = kSync == 1 ? 1 : kSync == 0 ? (64 / T < 1 ? 1 : 64 / T > 32 ? 32 : 64 / T)
                           : T % 16 == 0 ? 2 : T % 8 == 0 ? 4 : 8;
  static constexpr int C = 8 * T <= 256 ? 8 : 4 * T <= 256 ? 4 : T <= 256 ? 2 : 1;
  __host__ __device__ static constexpr int threads(int lines) { return (lines * T + 31) / 32 * 32; }
  static constexpr int kRowThreads = threads(L), kColThreads = threads(C);
  // dynamic shared memory: the exchange buffer (for every whole or idle line of the
  // block's threads), then the group slots; the column tile as the tensor map's box
  // leaves it (N rows of C columns) shares the exchange buffer's space
  __host__ __device__ static constexpr int buf_bytes(int nth) { return S == 1 ? 0 : (nth / T * LS * 16 + 127) / 128 * 128; }
  static constexpr int kColBytes = C * N * 16 > buf_bytes(kColThreads) ? C * N * 16 : buf_bytes(kColThreads);
  static constexpr int kRowSmem = buf_bytes(kRowThreads) + 256;
  static constexpr int kColSmem = (kColBytes + 127) / 128 * 128 + 256 + 128;
  // resident blocks per SM the kernels are compiled for: those of 128 registers a thread for
  // 12 and more points, of 112 for 8 (rows of 256^3: 597, 568, 550, 545 us with bounds of 64,
  // 80, 96, 112 registers, the wider ones without spills; the compiler needs 96 of the 112.
  // 144 and more with 16 points lose a quarter of the warps and 29 % at 2048^2)
  __host__ __device__ static constexpr int blocks(int nth) {
    constexpr int regs = E > 8 ? 128 : 112;
    return 65536 / (regs * nth) > 32 ? 32 : 65536 / (regs * nth) < 1 ? 1 : 65536 / (regs * nth);
  }
  // slots of register arrays: a middle radix that does not divide E takes whole rounds
  __host__ __device__ static constexpr int rounds(int p) { return E % R(p) == 0 ? E / R(p) : (N / R(p) + T - 1) / T; }
  __host__ __device__ static constexpr int slots() {
    int k = E;
    for (int p = 0; p < S; ++p) k = rounds(p) * R(p) > k ? rounds(p) * R(p) : k;
    return k;
  }
  static constexpr int K = slots();
};

// ------------------------------------------------------------ butterflies 6, 10, 12, 20
// Coprime factors (Good-Thomas): input index n = (B n1 + A n2) mod AB, output index k with
// k = k1 mod A, k = k2 mod B; no twiddles between the two stages.
__host__ __device__ constexpr int pfa_unit(int a, int b) {  // the k < ab with k = 1 mod a, 0 mod b
  int k = 0;
  while (k % a != 1 % a || k % b != 0) ++k;
  return k;
}
template <int A, int B>
__device__ __forceinline__ void fbfly_pfa(longlong2* v) {
  longlong2 w[A][B];
#pragma unroll
  for (int i = 0; i < A; ++i) {
#pragma unroll
    for (int j = 0; j < B; ++j) w[i][j] = v[(B * i + A * j) % (A * B)];
    fbfly<B, true>(w[i]);
  }
#pragma unroll
  for (int j = 0; j < B; ++j) {
    longlong2 u[A];
#pragma unroll
    for (int i = 0; i < A; ++i) u[i] = w[i][j];
    fbfly<A, true>(u);
#pragma unroll
    for (int i = 0; i < A; ++i) {
      constexpr int ea = pfa_unit(A, B), eb = pfa_unit(B, A);
      v[(i * ea + j * eb) % (A * B)] = u[i];
    }
  }
}
template <int R>
__device__ __forceinline__ void line_bfly(longlong2* v) {
  if constexpr (R == 6) fbfly_pfa<2, 3>(v);
  else if constexpr (R == 10) fbfly_pfa<2, 5>(v);
  else if constexpr (R == 12) fbfly_pfa<4, 3>(v);
  else if constexpr (R == 20) fbfly_pfa<4, 5>(v);
  else fbfly<R, true>(v);
}

// ------------------------------------------------------------ shifts and maxima
// x 2^s, rounded half up when s < 0
struct Shift {
  int sl, sr;
  i64 half;
  __device__ __forceinline__ explicit Shift(int s) {
    sl = s > 0 ? s : 0;
    sr = s < 0 ? (s < -63 ? 63 : -s) : 0;
    half = sr ? (i64)1 << (sr - 1) : 0;
  }
  __device__ __forceinline__ i64 operator()(i64 x) const { return ((i64)((u64)x << sl) + half) >> sr; }
  __device__ __forceinline__ longlong2 operator()(longlong2 x) const { return make_longlong2((*this)(x.x), (*this)(x.y)); }
};
__device__ __forceinline__ longlong2 shl_by(longlong2 x, int s) {
  return make_longlong2((i64)((u64)x.x << s), (i64)((u64)x.y << s));
}
// running extremes of the high words; mag() < 2^k bounds every component by 2^(32 + k)
struct HiMax {
  int mx = 0, mn = 0;
  __device__ __forceinline__ void add(longlong2 x) {
    const int a = (int)(x.x >> 32), b = (int)(x.y >> 32);
    mx = max(mx, max(a, b));
    mn = min(mn, min(a, b));
  }
  __device__ __forceinline__ void add_hi(int a, int b) {
    mx = max(mx, max(a, b));
    mn = min(mn, min(a, b));
  }
  __device__ __forceinline__ unsigned mag() const { return (unsigned)max(mx, ~mn); }
};

// A thread's place: line `l` of the block, thread `t` of the line, the line's exchange
// buffer, and the slots of the group maxima ([2][32] ints of shared memory).
template <class G>
struct LineCtx {
  int l, t;
  longlong2* buf;
  unsigned (*slot)[32];
  int nth;  // threads that take part in the block's barriers
  bool on = true;  // false: a thread that only fills a warp (its values count for nothing)
  int par = 0;
  __device__ __forceinline__ LineCtx(longlong2* smem, unsigned (*sl)[32], int n = blockDim.x) : slot(sl), nth(n) {
    l = threadIdx.x / G::T;
    t = threadIdx.x % G::T;
    buf = smem + (size_t)l * G::LS;
  }
  // this thread's exchange slot of point s (regular passes read it from there)
  __device__ __forceinline__ longlong2* own(int s) const { return buf + G::pad(t) + s * G::pad(G::T); }
  // barrier of the group
  __device__ __forceinline__ void sync() const {
    if constexpr (G::kSync == 0) __syncwarp();
    else if constexpr (G::kSync == 1) asm volatile("bar.sync %0, %1;" ::"r"(l + 1), "n"(G::T) : "memory");
    else asm volatile("bar.sync 15, %0;" ::"r"(nth) : "memory");
  }
  // the group's maximum in two halves around one of its barriers: put before, get after.
  // Slots alternate, so a slot is written again only after another barrier.
  __device__ __forceinline__ void put(unsigned& m) {
    m = __reduce_max_sync(0xffffffffu, on ? m : 0u);
    if constexpr (G::kSync != 0) {
      if ((threadIdx.x & 31) == 0) slot[par][threadIdx.x >> 5] = m;
    }
  }
  __device__ __forceinline__ void get(unsigned& m) {
    if constexpr (G::kSync != 0) {
      constexpr int nw = G::kSync == 1 ? G::T / 32 : 0;
      const int w0 = G::kSync == 1 ? l * nw : 0;
      const int n = G::kSync == 1 ? nw : nth >> 5;
      m = slot[par][w0];
      for (int w = 1; w < n; ++w) m = max(m, slot[par][w0 + w]);
      par ^= 1;
    }
  }
  __device__ __forceinline__ unsigned group_max(unsigned m) {
    put(m);
    sync();
    get(m);
    return m;
  }
  // bit length from the group's largest high word (0: every component below 2^32)
  __device__ __forceinline__ static int bits_of(unsigned m) { return m ? 64 - __clz((int)m) : 0; }
};

// ------------------------------------------------------------ the transform
// outputs of pass P into the exchange buffer
template <class G, int P>
__device__ __forceinline__ void line_store(const longlong2* v, const LineCtx<G>& c) {
  constexpr int R = G::R(P), ns = G::NS(P), NB = G::rounds(P);
  constexpr bool reg = G::E % R == 0;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j = c.t + b * G::T;
    if (!reg && j >= G::N / R) continue;
    int ph;
    if constexpr (P == 0) {
      ph = j * G::pad(R);
    } else {
      const int jm = j % ns, base = (j - jm) * R + jm;
      ph = G::pad(base);
    }
#pragma unroll
    for (int q = 0; q < R; ++q)
      c.buf[ph + (P == 0 ? G::pad(q) : q * G::pad(ns))] = v[reg ? b + q * NB : b * R + q];
  }
}
// inputs of pass P from the exchange buffer, twiddled and scaled by 2^-s, and its
// butterflies; `taken` is called with each point's slot once its value is in registers
template <class G, int P, class F>
__device__ __forceinline__ void line_load(longlong2* v, const LineCtx<G>& c, const int4* __restrict__ tw, int s,
                                          const F& taken) {
  constexpr int R = G::R(P), ns = G::NS(P), NB = G::rounds(P);
  constexpr bool reg = G::E % R == 0;
  const Shift sh0(-s);
  const int lsh = s < 2 ? 2 - s : 0;
  const int4* w = tw + (s > 2 ? s - 2 : 0) * line_tw_len(G::N, G::ppt) + line_tw_off(G::N, G::ppt, P);
  const longlong2* src = c.buf + G::pad(c.t);
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    const int j = c.t + b * G::T;
    if (!reg && j >= G::N / R) continue;
    const int4* wj = w + j % ns;
    longlong2 x[R];
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = src[b * G::pad(G::T) + q * G::pad(G::N / R)];
    x[0] = sh0(x[0]);
    if (lsh) {
#pragma unroll
      for (int q = 1; q < R; ++q) x[q] = shl_by(x[q], lsh);
    }
#pragma unroll
    for (int q = 1; q < R; ++q) x[q] = fmul_tw(x[q], __ldg(wj + (q - 1) * ns));
    if constexpr (reg && P + 1 == G::S) {
#pragma unroll
      for (int q = 0; q < R; ++q) taken(b + q * NB);
    }
    line_bfly<R>(x);
#pragma unroll
    for (int q = 0; q < R; ++q) v[reg ? b + q * NB : b * R + q] = x[q];
  }
}
template <class G, int P>
__device__ __forceinline__ unsigned line_mag(const longlong2* v, const LineCtx<G>& c) {
  constexpr int R = G::R(P), NB = G::rounds(P);
  constexpr bool reg = G::E % R == 0;
  HiMax h;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    if (!reg && c.t + b * G::T >= G::N / R) continue;
#pragma unroll
    for (int q = 0; q < R; ++q) h.add(v[reg ? b + q * NB : b * R + q]);
  }
  return h.mag();
}
// passes P .. S - 1, the outputs of pass P - 1 in v
template <class G, int P, class F>
__device__ __forceinline__ void line_passes(longlong2* v, LineCtx<G>& c, const int4* __restrict__ tw, int& scale,
                                            const F& taken) {
  if constexpr (P < G::S) {
    unsigned m = line_mag<G, P - 1>(v, c);
    c.put(m);
    c.sync();  // the group's reads of the exchange buffer are done
    line_store<G, P - 1>(v, c);
    c.sync();
    c.get(m);
    // the last pass leaves one bit more room, so that what follows only shifts left
    constexpr int target = (P + 1 == G::S ? 61 : 62) - line_guard(G::R(P));
    const int bits = LineCtx<G>::bits_of(m);
    const int s = bits ? bits - target : 0;
    scale -= s;
    line_load<G, P>(v, c, tw, s, taken);
    line_passes<G, P + 1>(v, c, tw, scale, taken);
  }
}
// Forward transform of the line in v (thread t: points t + s T in v[s]) whose moduli
// are below 2^57.5; afterwards every component is below 2^61 (2^62 for one-pass plans).
// `taken(s)`: the thread's own exchange slot of point s has been read for the last time.
struct NoHook {
  __device__ __forceinline__ void operator()(int) const {}
};
template <class G, class F = NoHook>
__device__ __forceinline__ void line_fft(longlong2* v, LineCtx<G>& c, const int4* __restrict__ tw, int& scale,
                                         const F& taken = F()) {
  constexpr int R = G::R(0), NB = G::E / R;
#pragma unroll
  for (int b = 0; b < NB; ++b) {
    longlong2 x[R];
#pragma unroll
    for (int q = 0; q < R; ++q) x[q] = v[b + q * NB];
    line_bfly<R>(x);
#pragma unroll
    for (int q = 0; q < R; ++q) v[b + q * NB] = x[q];
  }
  line_passes<G, 1>(v, c, tw, scale, taken);
}
constexpr int kLineIn = 57;  // components a transform takes are below 2^57 (moduli 2^57.5)

// bit length of the line outputs over the group (0: all zero or below 2^32)
template <class G>
__device__ __forceinline__ int line_bits(const longlong2* v, LineCtx<G>& c) {
  HiMax h;
#pragma unroll
  for (int s = 0; s < G::E; ++s) h.add(v[s]);
  return LineCtx<G>::bits_of(c.group_max(h.mag()));
}

// the line outputs brought to TOP bits (products keep 2^-(TOP - 2) of the largest
// component); returns the shift
template <class G, int TOP = 61>
__device__ __forceinline__ int line_up(longlong2* v, LineCtx<G>& c) {
  const int bits = line_bits<G>(v, c);
  const int sh = bits ? TOP - bits : 0;
#pragma unroll
  for (int s = 0; s < G::E; ++s) {
    if constexpr (G::S == 1 || TOP < 61) v[s] = Shift(sh)(v[s]);
    else v[s] = shl_by(v[s], sh);
  }
  return sh;
}

// Raw fixed-point points v[s] of exponents gm - d[s] (d <= 0: gm is the pass minimum)
// aligned to one exponent and normalised for a transform; returns that exponent.
template <class G>
__device__ __forceinline__ int line_align(longlong2* v, const int* d, int gm, LineCtx<G>& c) {
  constexpr int E = G::E;
  HiMax h;
#pragma unroll
  for (int s = 0; s < E; ++s) {
    const int r = min(-d[s], 31);
    h.add_hi((int)(v[s].x >> 32) >> r, (int)(v[s].y >> 32) >> r);
  }
  int bits = LineCtx<G>::bits_of(c.group_max(h.mag()));
  if (bits == 0) {  // the whole group below 2^32 of the pass exponent: the full words' length
    u64 m = 0;
#pragma unroll
    for (int s = 0; s < E; ++s) m |= fmag(Shift(d[s])(v[s]));
    bits = (int)c.group_max((unsigned)bitlen(m));
    if (bits == 0) bits = kLineIn;
  }
  const int sh = kLineIn - bits;
#pragma unroll
  for (int s = 0; s < E; ++s) v[s] = Shift(d[s] + sh)(v[s]);
  return gm + sh;
}

// psi as doubles (v[s] holds the two words) -> fixed point below 2^top, returns the
// exponent; em: the largest biased exponent of the group (0x7ff: an Inf or NaN)
template <class G>
__device__ __forceinline__ int line_from_double(longlong2* v, LineCtx<G>& c, unsigned& em, int top = kLineIn) {
  constexpr int E = G::E;
  unsigned m = 0;
#pragma unroll
  for (int s = 0; s < E; ++s)
    m = max(m, max((unsigned)(v[s].x >> 52) & 0x7ffu, (unsigned)(v[s].y >> 52) & 0x7ffu));
  em = c.group_max(m);
  const int sc = top - ((int)em - 1022);
#pragma unroll
  for (int s = 0; s < E; ++s)
    v[s] = make_longlong2(d2fx(__longlong_as_double(v[s].x), sc), d2fx(__longlong_as_double(v[s].y), sc));
  return sc;
}

}  // namespace qsf
