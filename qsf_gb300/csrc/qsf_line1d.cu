// qsf_line1d.cu -- host side of the 1D step kernels (qsf_line1d.cuh): the tables of a
// line's geometry, the tables of a run of sub-steps, and the launches.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <vector>

#include "qsf_internal.h"

namespace qsf {

void add_lines_one(std::vector<LineKernels>& out);
void add_lines_p2a(std::vector<LineKernels>& out);
void add_lines_p2b(std::vector<LineKernels>& out);
void add_lines_r3(std::vector<LineKernels>& out);
void add_lines_r5(std::vector<LineKernels>& out);

namespace {

std::vector<LineKernels>& line_table() {
  static std::vector<LineKernels> t;
  return t;
}

// entry `pos` of a slot-order table: the index in the X or the K layout, -1: none
__device__ __forceinline__ int slot_index(const LineDev& D, long long pos, bool kspace) {
  const long long str = (long long)D.ctas * D.nth;
  const int s = (int)(pos / str), r = (int)(pos % str) / D.nth, tid = (int)(pos % D.nth);
  if (D.n2 == 0) return tid < D.t1 ? tid + s * D.t1 : -1;
  if (tid >= D.n1 * D.n2 / (D.ctas * D.epp)) return -1;
  if (kspace) return r * (D.n1 / D.ctas) + tid / D.t2 + D.n1 * (tid % D.t2 + s * D.t2);
  return D.n2 * (tid % D.t1 + s * D.t1) + r * (D.n2 / D.ctas) + tid / D.t1;
}

// The tables of the next `most` sub-steps: gridDim.x = 3 tb (P phases, length-gauge opening
// and closing factors), y = most + 1, z = solves.  Imaginary-time tables whose values
// exceed 1 are stored times 2^-e (texp; every block of a table evaluates its maximum, so
// the slices agree).  What bounds it: FP64 sincos, N per table and sub-step, which is why
// the tables of many sub-steps are one launch over the whole GPU and not part of the
// line's own CTAs (a step's tables on the line's SM alone made a step 2.4x slower).
__global__ void __launch_bounds__(256) k_line_tables(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss,
                                                     int most, int tb) {
  const GridDev& g = Gs[blockIdx.z];
  const StepDev& S = Ss[blockIdx.z];
  const LineDev& D = S.line;
  const long long sub0 = S.ctl[0];
  if (!(sub0 <= S.ctl[1] && sub0 < S.nsteps)) return;
  const int kind = blockIdx.x / tb, piece = blockIdx.x % tb, i = blockIdx.y;
  if (kind == 0 && i == 0 && piece == 0 && threadIdx.x == 0) *D.sub0 = sub0;
  const bool lg = g.gauge == 1 && g.n_fields && S.coupling;
  const long long sub = sub0 + i;
  if (kind == 0 && (D.pstride ? (i >= most || sub >= S.nsteps) : i > 0)) return;
  if (kind == 1 && (!lg || sub >= S.nsteps)) return;
  if (kind == 2 && (!lg || i >= most || sub >= S.nsteps)) return;
  const double* cp = S.coupling ? S.coupling + sub * S.coup_stride : nullptr;
  const int n = g.ax[0].n;
  const long long slots = (long long)D.ctas * D.nth * D.epp;
  const double mant = kind == 0 ? S.m_mant : 1.0;
  __shared__ double red[32];
  __shared__ int e_sh;
  double mx = mant;
  if (S.mode == 1) {
    mx = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) mx = fmax(mx, table_entry(g, S, cp, nullptr, kind, 0, j).x * mant);
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_down_sync(0xffffffffu, mx, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 1; w < (int)(blockDim.x >> 5); ++w) mx = fmax(mx, red[w]);
  }
  if (threadIdx.x == 0) {
    int e = 0;
    if (mx > 1.0) frexp(mx, &e);  // mx < 2^e
    e_sh = e;
    if (piece == 0) const_cast<int*>(D.texp)[i * 3 + kind] = e;
  }
  __syncthreads();
  const double sc = ldexp(mant, -e_sh);
  int4* out = kind == 0   ? const_cast<int4*>(D.ptab) + i * D.pstride
              : kind == 1 ? const_cast<int4*>(D.ctab) + i * slots
                          : const_cast<int4*>(D.ctab) + (D.csteps + 1 + i) * slots;
  const bool kspace = kind == 0 && !D.bs;
  for (long long pos = (long long)piece * blockDim.x + threadIdx.x; pos < slots; pos += (long long)tb * blockDim.x) {
    const int j = slot_index(D, pos, kspace);
    int4 w = make_int4(0, 0, 0, 0);
    if (j >= 0 && j < n) {
      double2 f = table_entry(g, S, cp, nullptr, kind, 0, j);
      if (kind == 0 && D.bs) f.y = -f.y;  // Bluestein's P phase meets conjugated data
      w = split62(make_double2(fmin(fmax(f.x * sc, -1.0), 1.0), fmin(fmax(f.y * sc, -1.0), 1.0)));
    }
    out[pos] = w;
  }
}

// chirp[j] = exp(-i pi (j^2 mod 2n) / n) (exact integer angle reduction) in split form, and
// the convolution kernel w = conj(chirp) wrapped onto M points (w[j] = w[M - j]), zero between
__global__ void k_line_chirp(int4* __restrict__ chirp, double2* __restrict__ w, int n, int M) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < M; j += gridDim.x * blockDim.x) {
    const int k = j < n ? j : M - j;
    double2 v = make_double2(0.0, 0.0);
    if (k < n) {
      const long long r = ((long long)k * k) % (2LL * n);
      double sn, cs;
      sincospi((double)r / (double)n, &sn, &cs);
      v = make_double2(cs, sn);  // conj(chirp[k])
      if (j < n) chirp[j] = split62(make_double2(cs, -sn));
    }
    w[j] = v;
  }
}
// transformed kernel / M, scaled by 2^-e so that its largest modulus lies in [1/2, 1),
// as [k1][k2]; one block
__global__ void __launch_bounds__(1024) k_line_bhat(const double2* __restrict__ b, int4* __restrict__ out, int* bexp, int M,
                                                    int n1, int n2) {
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
  // 1 / M in two parts: the rounding of one would be the same at every step (5003 points, M =
  // 10240: the norm grew by 1.9e-16 a step)
  const double hi = ldexp(one, -e), lo = ldexp(fma(-one, (double)M, 1.0) / (double)M, -e);
  for (int j = threadIdx.x; j < M; j += blockDim.x) {
    const double2 v = b[j];
    out[(j % n1) * n2 + j / n1] = split62(make_double2(fma(v.x, hi, v.x * lo), fma(v.y, hi, v.y * lo)));
  }
}
// Bluestein's static factors: the X factor times the chirp, conjugated for the closing half
__global__ void k_line_static(const int4* __restrict__ xs, const int4* __restrict__ chirp, int n, int4* xa, int4* xb) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const longlong2 x = tw_join(xs[j]), c = tw_join(chirp[j]);
    xa[j] = split_fx(fmul62(x, fconj(c)));
    xb[j] = split_fx(fmul62(x, c));
  }
}

// exp(-2 pi i k1 n2 / N) as [n2][k1] and [k1][n2], once per length, process and device
int shared_turns(const LineKernels& L, const int4** w1, const int4** w2) {
  static std::mutex mu;
  static std::map<std::pair<int, int>, int4*> cache;
  int dev = 0;
  QSF_CU(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find({dev, L.n});
  if (it == cache.end()) {
    const int N = L.n;
    std::vector<int4> h((size_t)2 * N), turn((size_t)N);
    const Roots root(N);
    for (int t = 0; t < N; ++t) turn[(size_t)t] = root.split(t);
    for (int a = 0; a < L.n1; ++a)
      for (int b = 0; b < L.n2; ++b) {
        const int4 w = turn[(size_t)((long long)a * b % N)];
        h[(size_t)b * L.n1 + a] = w;
        h[(size_t)N + (size_t)a * L.n2 + b] = w;
      }
    int4* d = nullptr;
    if (int rc = dev_alloc(d, h.size())) return rc;
    cudaError_t ce = cudaMemcpy(d, h.data(), h.size() * sizeof(int4), cudaMemcpyHostToDevice);
    if (ce == cudaSuccess) ce = cudaDeviceSynchronize();  // a pageable copy may still be on its way
    if (ce != cudaSuccess) {
      cudaFree(d);
      return fail(QSF_ECUDA, std::string("line tables: ") + cudaGetErrorString(ce));
    }
    it = cache.emplace(std::make_pair(dev, N), d).first;
  }
  *w1 = it->second;
  *w2 = it->second + L.n;
  return QSF_OK;
}

constexpr int kLineSteps = 256;              // sub-steps of one launch at most
constexpr size_t kLineTableBytes = 48 << 20;  // bytes of their tables at most (at least 16 sub-steps)

// the tables of a run made `chunk` sub-steps at a time: sub-steps they hold, entries (vg, lg:
// a velocity- or a length-gauge field couples)
struct LineTables {
  int64_t steps;
  size_t ptab, ctab, texp;
};
LineTables line_tables(const LineKernels& L, bool vg, bool lg, int64_t chunk) {
  const size_t slots = (size_t)L.ctas * L.nth * L.epp, per = slots * sizeof(int4) * (lg ? 2 : 1);
  const int64_t fit = std::min<int64_t>(std::max<int64_t>(16, (int64_t)(kLineTableBytes / per)), kLineSteps);
  const int64_t steps = std::max<int64_t>(1, std::min(fit, chunk));
  return {steps, slots * (vg ? (size_t)steps : 1), lg ? slots * (size_t)(2 * steps + 1) : 0, (size_t)(steps + 1) * 3};
}

}  // namespace

const LineKernels* line_kernels(int n) {
  for (const LineKernels& k : line_table())
    if (k.n == n) return &k;
  return nullptr;
}

int init_line_table() {
  std::vector<LineKernels>& t = line_table();
  t.clear();
  add_lines_one(t);
  add_lines_p2a(t);
  add_lines_p2b(t);
  add_lines_r3(t);
  add_lines_r5(t);
  for (const LineKernels& k : t) {
    const std::pair<const void*, int> f[4] = {{(const void*)k.run, k.smem}, {(const void*)k.run_bs, k.smem_bs},
                                              {(const void*)k.fft, k.smem}, {(const void*)k.fft_bs, k.smem}};
    for (const auto& [fn, bytes] : f)
      if (fn) QSF_CU(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  }
  return QSF_OK;
}

int line_conv_length(int n) {
  int best = 0;
  for (const LineKernels& k : line_table())
    if (k.run_bs && k.n >= 2 * n - 1 && (!best || k.n < best)) best = k.n;
  return best;
}

// the geometry tables of a 1D grid
int line_setup(qsf_grid* g) {
  const int n = g->G.ax[0].n;
  const LineKernels* L = line_kernels(n);
  const bool bs = !g->ks;
  if (bs) L = line_kernels(line_conv_length(n));
  if (!L) return fail(QSF_EINVAL, "grid size " + std::to_string(n) + " has no 1D kernels in this build");
  g->lk = L;
  LineDev& D = g->line;
  D.n1 = L->n1;
  D.n2 = L->n2;
  D.ctas = L->ctas;
  D.nth = L->nth;
  D.epp = L->epp;
  D.t1 = L->t1;
  D.t2 = L->t2;
  D.bs = bs;
  int rc;
  if ((rc = shared_line_twiddles(L->n1, L->ppt, &D.tw1))) return rc;
  if (L->n2 && ((rc = shared_line_twiddles(L->n2, L->ppt, &D.tw2)) || (rc = shared_turns(*L, &D.w1, &D.w2)))) return rc;
  if ((rc = dev_alloc(g->l_sub0, 1))) return rc;
  D.sub0 = g->l_sub0;
  if (!bs) return QSF_OK;
  const int M = L->n;
  double2* w = nullptr;
  if ((rc = dev_alloc(g->l_chirp, (size_t)n)) || (rc = dev_alloc(g->l_bhat, (size_t)M + 1)) ||
      (rc = dev_alloc(g->l_xab, (size_t)2 * n)) || (rc = dev_alloc(w, (size_t)M)))
    return rc;
  const int blocks = std::min((M + 255) / 256, device_sm_count());
  k_line_chirp<<<blocks, 256, 0, g->stream>>>(g->l_chirp, w, n, M);
  GridDev V{};
  V.dim = 1;
  V.m = M;
  V.psi = w;
  V.ax[0].n = M;
  L->fft<<<L->ctas, L->nth, L->smem, g->stream>>>(V, D, 1, 1.0);
  int* bexp = reinterpret_cast<int*>(g->l_bhat + M);
  k_line_bhat<<<1, 1024, 0, g->stream>>>(w, g->l_bhat, bexp, M, L->n1, L->n2);
  cudaError_t ce = cudaGetLastError();
  if (ce == cudaSuccess) ce = cudaStreamSynchronize(g->stream);
  cudaFree(w);
  if (ce != cudaSuccess) return fail(QSF_ECUDA, std::string("line set-up: ") + cudaGetErrorString(ce));
  D.chirp = g->l_chirp;
  D.bhat = g->l_bhat;
  D.bexp = bexp;
  return QSF_OK;
}

void line_release(qsf_grid* g) {
  for (void* p : {(void*)g->l_sub0, (void*)g->l_chirp, (void*)g->l_bhat, (void*)g->l_xab,
                  (void*)g->l_ptab, (void*)g->l_ctab, (void*)g->l_texp})
    if (p) cudaFree(p);
}

// device bytes of the tables of n-point lines whose runs are made `chunk` sub-steps at a time
size_t line_table_bytes(int n, bool field, bool lg, int64_t chunk) {
  const LineKernels* L = fused_length(n) ? line_kernels(n) : line_kernels(line_conv_length(n));
  if (!L) return 0;
  const LineTables t = line_tables(*L, field && !lg, field && lg, chunk);
  return (t.ptab + t.ctab) * sizeof(int4) + t.texp * sizeof(int);
}

// the tables a program runs on, `chunk` sub-steps at a time, into S.line
int line_prepare(qsf_grid* g, StepDev& S, int64_t chunk) {
  const LineKernels& L = *g->lk;
  LineDev D = g->line;
  const size_t slots = (size_t)L.ctas * L.nth * L.epp;
  const bool field = g->G.n_fields && S.coupling, lg = field && g->G.gauge == QSF_GAUGE_LENGTH, vg = field && !lg;
  // (BOX, the one border of a line, needs six)
  if (S.row_ptr && S.nsnap > kLineSnap) return fail(QSF_EINVAL, "too many border points on a 1D line");
  const LineTables t = line_tables(L, vg, lg, chunk);
  const int64_t steps = t.steps;
  g->l_steps = (int)steps;
  int rc;
  if ((rc = dev_reserve(g->l_ptab, g->l_ptab_cap, t.ptab)) || (rc = dev_reserve(g->l_texp, g->l_texp_cap, t.texp)))
    return rc;
  if (lg && (rc = dev_reserve(g->l_ctab, g->l_ctab_cap, t.ctab))) return rc;
  D.ptab = g->l_ptab;
  D.pstride = vg ? (long long)slots : 0;
  D.ctab = g->l_ctab;
  D.csteps = (int)steps;
  D.texp = g->l_texp;
  D.xa = D.xb = S.xs;
  if (D.bs) {
    const int n = g->G.ax[0].n;
    if (g->lx_mode != g->xs_mode || g->lx_delta != g->xs_delta) {
      k_line_static<<<std::min((n + 255) / 256, device_sm_count()), 256, 0, g->stream>>>(S.xs, g->l_chirp, n, g->l_xab,
                                                                                       g->l_xab + n);
      QSF_CU(cudaGetLastError());
      g->lx_mode = g->xs_mode;
      g->lx_delta = g->xs_delta;
    }
    D.xa = g->l_xab;
    D.xb = g->l_xab + n;
  }
  S.line = D;
  return QSF_OK;
}

// the next `steps` sub-steps of `count` solves of the same line kernels (tables, then steps)
int line_launch_tables(const LineKernels& L, const GridDev* dG, const StepDev* dS, int count, int steps, bool lg, cudaStream_t st) {
  // about 1024 entries per block: FP64 sincos want many SMs
  const int tb = std::max(1, std::min(16, L.ctas * L.nth * L.epp / 1024));
  k_line_tables<<<dim3((lg ? 3 : 1) * tb, steps + 1, count), 256, 0, st>>>(dG, dS, steps, tb);
  QSF_CU(cudaGetLastError());
  return QSF_OK;
}
int line_launch_steps(const LineKernels& L, bool bs, const GridDev* dG, const StepDev* dS, int count, int steps,
                      cudaStream_t st) {
  (bs ? L.run_bs : L.run)<<<dim3(L.ctas, count), L.nth + 32, bs ? L.smem_bs : L.smem, st>>>(dG, dS, steps);
  QSF_CU(cudaGetLastError());
  return QSF_OK;
}

// fourier<R>() of the line G.psi in one launch
int line_fourier(qsf_grid* g, const GridDev& G, bool fwd, double sc) {
  const LineKernels& L = *g->lk;
  (g->line.bs ? L.fft_bs : L.fft)<<<L.ctas, L.nth, L.smem, g->stream>>>(G, g->line, fwd, sc);
  QSF_CU(cudaGetLastError());
  return QSF_OK;
}

}  // namespace qsf
