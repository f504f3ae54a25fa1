// qsf_bluestein.cu -- fourier<R>() of 2D and 3D grids whose axis length is outside the
// built kernel list, and what their step kernels need.
//
// The reference's FFTW plans take any n (wf/grid.h:251-274); the fused step kernels of
// this library are compiled for a list of lengths 2^a, 3*2^a and 5*2^a (8 ... 16384,
// the add_sizes_* tables).  For any other n one axis of the transform runs as Bluestein's
// chirp-z convolution: with c[j] = exp(-i pi j^2 / n),
//     X[k] = c[k] * sum_j (x[j] c[j]) conj(c[k - j]),
// a linear convolution evaluated as a cyclic one of length M >= 2n - 1 (a length with
// built kernels) through the library's own M-point transforms:
//     a = pad_M(x * c);  A = FFT_M(a);  A *= B = FFT_M(conj(c), wrapped);  a = IFFT_M(A) / M;
//     X[k] = c[k] a[k], k < n.
// The inverse transform is the forward one between two conjugations.  The chirp comes
// from exact integer angle reduction (j^2 mod 2n) and sincospi on the device; B is
// transformed once per grid.  The steps of such grids are the convolution form of the pass
// kernels (qsf_passes.cuh), which take the same chirp and B; what is here serves the member
// operations.  Batches take built lengths only, the server runs such solves beside its
// batch.  1D lines of such lengths have step kernels of their own (qsf_line1d.cuh).
#include <algorithm>
#include <string>
#include <vector>

#include "qsf_internal.h"

namespace qsf {
namespace {

// psi index (o, j, c) of axis ax with length nj: o * nj * inner + j * inner + c
__global__ void k_bs_pre(const double2* __restrict__ psi, double2* __restrict__ scr, const double2* __restrict__ chirp,
                         long long outer, int n, int M, long long inner, int conj_in) {
  const long long total = outer * M * inner;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < total; p += stride) {
    const long long c = p % inner, t = p / inner;
    const int j = (int)(t % M);
    const long long o = t / M;
    double2 v = make_double2(0.0, 0.0);
    if (j < n) {
      double2 x = psi[(o * n + j) * inner + c];
      if (conj_in) x.y = -x.y;
      v = cmul(x, chirp[j]);
    }
    scr[p] = v;
  }
}

__global__ void k_bs_mul(double2* __restrict__ scr, const double2* __restrict__ bhat, long long outer, int M,
                         long long inner) {
  const long long total = outer * M * inner;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < total; p += stride) {
    const int j = (int)((p / inner) % M);
    scr[p] = cmul(scr[p], bhat[j]);
  }
}

__global__ void k_bs_post(double2* __restrict__ psi, const double2* __restrict__ scr, const double2* __restrict__ chirp,
                          long long outer, int n, int M, long long inner, int conj_out, double post) {
  const long long total = outer * n * inner;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < total; p += stride) {
    const long long c = p % inner, t = p / inner;
    const int k = (int)(t % n);
    const long long o = t / n;
    double2 y = cmul(scr[(o * M + k) * inner + c], chirp[k]);
    if (conj_out) y.y = -y.y;
    psi[p] = make_double2(y.x * post, y.y * post);
  }
}

// chirp[j] = exp(-i pi (j^2 mod 2n) / n) (exact integer angle reduction) and the
// convolution kernel w = conj(chirp) wrapped onto M points (w[j] = w[M - j]), zero
// between
__global__ void k_bs_chirp(double2* __restrict__ chirp, double2* __restrict__ w, int n, int M) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < M; j += gridDim.x * blockDim.x) {
    const int k = j < n ? j : M - j;  // the chirp index w[j] holds, or >= n (zero)
    double2 v = make_double2(0.0, 0.0);
    if (k < n) {
      const long long r = ((long long)k * k) % (2LL * n);
      double sn, cs;
      sincospi((double)r / (double)n, &sn, &cs);
      v = make_double2(cs, sn);  // conj(chirp[k])
      if (j < n) chirp[j] = make_double2(cs, -sn);
    }
    w[j] = v;
  }
}

// bhat / M times 2^-e, e such that its largest modulus lies in [1/2, 1), in split form; one
// block
__global__ void __launch_bounds__(1024) k_bs_split(const double2* __restrict__ b, int4* __restrict__ out, int* bexp, int M) {
  __shared__ double red[32];
  double mx = 0.0;
  for (int j = threadIdx.x; j < M; j += blockDim.x) mx = fmax(mx, fma(b[j].x, b[j].x, b[j].y * b[j].y));
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  mx = 0.0;
  for (int w = 0; w < 32; ++w) mx = fmax(mx, red[w]);
  const double one = 1.0 / (double)M;
  int e;
  frexp(sqrt(mx) * one, &e);
  if (threadIdx.x == 0) *bexp = e;
  // 1 / M in two parts: the rounding of one would be the same at every step
  const double hi = ldexp(one, -e), lo = ldexp(fma(-one, (double)M, 1.0) / (double)M, -e);
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    const double2 v = b[j];
    out[j] = split62(make_double2(fma(v.x, hi, v.x * lo), fma(v.y, hi, v.y * lo)));
  }
}

int blocks_for(long long count) {
  const long long b = (count + 255) / 256;
  return (int)std::min<long long>(std::max<long long>(b, 1), (long long)device_sm_count() * 16);
}

// geometry of the scratch: psi's with axis ax of length M
GridDev scratch_view(const qsf_grid* g, int ax) {
  GridDev S = g->G;
  S.psi = g->bs.scratch;
  S.ax[ax].n = g->bs.M;
  S.ax[ax].n2 = g->bs.M / 2;
  S.ax[ax].shift = (g->bs.M & (g->bs.M - 1)) == 0 ? __builtin_ctz((unsigned)g->bs.M) : -1;
  S.ax[ax].tw = g->bs.ax.tw;
  long long st = 1;
  for (int k = S.dim - 1; k >= 0; --k) {
    S.ax[k].stride = st;
    st *= S.ax[k].n;
  }
  S.m = st;
  return S;
}

// the convolution length of an n-point axis: the smallest built length M >= 2n - 1 up to
// 4096 (0: none)
int bs_plan(int n) {
  for (int c = 2 * n - 1; c <= 4096; ++c)
    if (kernels_for(c)) return c;
  return 0;
}

}  // namespace

int bs_size(int n, int dim) { return dim == 1 ? line_conv_length(n) : bs_plan(n); }

int bs_setup(qsf_grid* g) {
  GridDev& G = g->G;
  const int n = G.ax[0].n, M = bs_plan(n);
  if (!M)
    return fail(QSF_EINVAL, "grid size " + std::to_string(n) + " has no kernels and no Bluestein length in this build " +
                                "(1D lines up to 16384 points, other grids up to 2048 points per axis)");
  qsf_grid::Bluestein& b = g->bs;
  b.n = n;
  b.M = M;
  b.ks = kernels_for(M);
  int rc;
  if ((rc = axis_twiddles(M, true, &b.ax))) return rc;
  const size_t scr = (size_t)(G.m / n) * (size_t)M;
  if ((rc = dev_alloc(b.chirp, (size_t)n)) || (rc = dev_alloc(b.bhat, (size_t)M)) ||
      (rc = dev_alloc(b.scratch, std::max(scr, (size_t)M))))
    return rc;
  k_bs_chirp<<<blocks_for(M), 256, 0, g->stream>>>(b.chirp, b.bhat, n, M);
  QSF_CU(cudaGetLastError());
  // B = FFT_M(w): the kernel array as a one-line grid of M points
  GridDev L = G;
  L.dim = 1;
  L.psi = b.bhat;
  L.ax[0].n = M;
  L.ax[0].stride = 1;
  L.ax[0].tw = b.ax.tw;
  L.m = M;
  launch_axis_fft(*b.ks, L, 0, true, 1.0, g->stream);
  if ((rc = dev_alloc(b.bsplit, (size_t)M + 1))) return rc;
  int* bexp = reinterpret_cast<int*>(b.bsplit + M);
  k_bs_split<<<1, 1024, 0, g->stream>>>(b.bhat, b.bsplit, bexp, M);
  QSF_CU(cudaGetLastError());
  G.chirp = b.chirp;
  G.bhat = b.bsplit;
  G.bexp = bexp;
  for (int k = 0; k < G.dim; ++k)
    for (int p = 0; p < 2; ++p) G.ax[k].twl[p] = b.ax.twl[p];
  return QSF_OK;
}

void bs_release(qsf_grid* g) {
  qsf_grid::Bluestein& b = g->bs;
  for (void* p : {(void*)b.chirp, (void*)b.bhat, (void*)b.bsplit, (void*)b.scratch})  // the twiddles are shared
    if (p) cudaFree(p);
  b = qsf_grid::Bluestein();
}

int bs_axis(qsf_grid* g, double2* arr, int ax, bool fwd, double post) {
  const GridDev& G = g->G;
  const qsf_grid::Bluestein& b = g->bs;
  const int n = b.n, M = b.M;
  const long long inner = G.ax[ax].stride, outer = G.m / ((long long)n * inner);
  const GridDev S = scratch_view(g, ax);
  cudaStream_t st = g->stream;
  const int inv = fwd ? 0 : 1;
  k_bs_pre<<<blocks_for(outer * M * inner), 256, 0, st>>>(arr, b.scratch, b.chirp, outer, n, M, inner, inv);
  QSF_CU(cudaGetLastError());
  launch_axis_fft(*b.ks, S, ax, true, 1.0, st);
  k_bs_mul<<<blocks_for(outer * M * inner), 256, 0, st>>>(b.scratch, b.bhat, outer, M, inner);
  QSF_CU(cudaGetLastError());
  launch_axis_fft(*b.ks, S, ax, false, 1.0 / (double)M, st);
  k_bs_post<<<blocks_for(outer * n * inner), 256, 0, st>>>(arr, b.scratch, b.chirp, outer, n, M, inner, inv, post);
  QSF_CU(cudaGetLastError());
  return QSF_OK;
}

}  // namespace qsf
