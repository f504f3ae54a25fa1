// qsf_internal.h -- library-internal declarations shared by the host translation units
// of libqsfgpu.so (not part of the C ABI): the grid handle's device state, error
// reporting and allocation helpers.
#pragma once
#include <algorithm>
#include <string>
#include <utility>
#include <vector>

#include <cuda_runtime.h>

#include "qsf_gpu.h"
#include "qsf_borders.h"
#include "qsf_kernels.cuh"

namespace qsf {

// records msg as the text qsf_last_error() returns on this thread and returns code
int fail(int code, const std::string& msg);

// multiprocessor count of the current device (queried once per device); grid-stride
// kernels size their grids as a multiple of it
int device_sm_count();

template <class T>
int dev_alloc(T*& p, size_t count) {
  if (p) cudaFree(p);
  p = nullptr;
  if (count == 0) return QSF_OK;
  if (cudaMalloc((void**)&p, count * sizeof(T)) != cudaSuccess) {
    cudaGetLastError();
    p = nullptr;
    return fail(QSF_ENOMEM, "cudaMalloc of " + std::to_string(count * sizeof(T)) + " bytes failed");
  }
  return QSF_OK;
}
template <class T>
int dev_reserve(T*& p, size_t& cap, size_t count) {
  if (count <= cap && p) return QSF_OK;
  size_t c = std::max(count, cap * 2);
  int rc = dev_alloc(p, c);
  cap = rc == QSF_OK ? c : 0;
  return rc;
}

}  // namespace qsf

#define QSF_CU(call)                                                                                   \
  do {                                                                                                 \
    cudaError_t e_ = (call);                                                                           \
    if (e_ != cudaSuccess) return qsf::fail(QSF_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

using qsf::AxisDev;
using qsf::GridDev;
using qsf::KernelSet;
using qsf::LineDev;
using qsf::LineKernels;
using qsf::StepDev;
using qsf::FluxPoint;
using qsf::FluxTerm;
using qsf::BorderNodes;

// What a call sends to the device and brings back, in one copy each way: control words,
// convergence and Normalize state, the observables rows and the coupling rows of a short
// call, the step descriptor.  (Five copies down and two back took half of a one-step
// call on a 1024-point line.)
struct CallBlock {
  static constexpr int kRows = 256, kCoup = 256;  // doubles of rows and of coupling kept here
  long long ctl[8];
  double energy[2], scale[4];
  double rows[kRows];
  // the pass minima change by atomics while every block reads the words around them: lines
  // of their own
  alignas(128) int gmin[32];
  alignas(128) StepDev S;
  double coupling[kCoup];
};

struct qsf_grid {
  qsf_grid_desc desc{};
  GridDev G{};
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  BorderNodes bn;
  const KernelSet* ks = nullptr;  // kernels for this grid's line length (nullptr: none are built)
  qsf::KernelSet pass{};          // 2D and 3D: the kernels of its steps
  GridDev* dG = nullptr;          // device copy of G (step kernels read descriptors from device arrays)
  CallBlock* blk = nullptr;       // device memory of the words below and of short calls' rows
  StepDev* dS = nullptr;          // device copy of the current step descriptor
  // the batch this grid is a member of (qsf_batch_add) and its slot there: destroying
  // the grid removes it from that batch first (the batch's graph reads its memory)
  qsf_batch* batch = nullptr;
  int64_t batch_slot = -1;
  // static tables
  longlong2* xs = nullptr;
  long long* Vx = nullptr;
  int xs_mode = 0;
  double xs_delta = 0.0;
  int xs_exp = 0;
  int vshift = 0;
  double vmax = 0.0, vneg = 0.0;  // max V and max -V over the grid
  bool V_ready = false;
  // per-step tables
  longlong2* ptab = nullptr;
  longlong2* xdyn = nullptr;
  int nmax = 0;
  int l2m = 0;
  double m_mant = 1.0;
  size_t xdyn_cap = 0;
  // fixed-point pass bookkeeping: [kTableSteps][kTexp] table exponents, [4][scmax] line exponents
  int* ibuf = nullptr;
  int scmax = 1;
  // reductions
  double* partials = nullptr;
  int pmax = 0;
  double* fpartials = nullptr;
  long long* ctl = nullptr;
  double* energy = nullptr;
  double* scale = nullptr;
  double* rows_dev = nullptr;
  size_t rows_cap = 0;
  double* coup_dev = nullptr;
  size_t coup_cap = 0;
  // flux structures
  std::vector<int> fl_borders;
  int64_t fl_box = -1;
  bool fl_ready = false;
  double2* snap = nullptr;
  long long* snap_idx = nullptr;
  int* row_ptr = nullptr;
  FluxPoint* fpts = nullptr;
  FluxTerm* fterms = nullptr;
  int nsnap = 0, nfterms = 0, nfpts = 0, nfblk = 1;
  // launch geometry
  int nrowblk = 1;
  int ax_blocks[3] = {0, 0, 0};
  // multi-region transfer: slice buffer (m points) and the event that orders streams
  double2* mg_slice = nullptr;
  // member evolve: cached X-phase factors for (mode, delta) and per-axis P factors
  double2* etab = nullptr;
  int etab_mode = 0;
  double etab_delta = 0.0;
  double2* eptab = nullptr;
  // observables log of qsf_average_log (device, grow-only)
  double* obs_log = nullptr;
  size_t obs_cap = 0;
  double* vtab = nullptr;  // potential per point for member E_pot averages (built on first use)
  double* mtab = nullptr;  // per-axis one-node absorber masks [dim][nmax] (built on first use)
  cudaEvent_t mg_event = nullptr;
  // k_finalize of graph-replayed steps on a second stream, beside the next sub-step's
  // first passes: the stream and its fork / join events (created on first use)
  cudaStream_t fin_stream = nullptr;
  cudaEvent_t fin_fork = nullptr, fin_done = nullptr;
  // executable step graphs of qsf_step, kept per launch shape and replayed by later
  // calls (the kernels read every per-call value from the device descriptors)
  struct StepGraph {
    int64_t per, shape;  // sub-steps, and which passes they launch (run_passes)
    int overlap, nfblk;
    cudaGraphExec_t exec;
  };
  std::vector<StepGraph> step_graphs;
  StepDev solo{};  // the program of a solve that runs beside a batch (solo_begin)
  // TMA tensor maps of psi for the strided-axis passes (GridDev::tmap), 128 bytes each
  unsigned char* tmaps = nullptr;
  // Bluestein transforms of a 2D / 3D grid whose axis length has a prime factor above 5 (no
  // fused kernels, ks == nullptr): chirp c[j] = exp(-i pi j^2 / n), the transform of
  // the convolution kernel conj(c) padded to M (a length >= 2n - 1 with built
  // kernels), the M-point kernels and twiddles, and a scratch of (m / n) * M points.
  struct Bluestein {
    int n = 0, M = 0;
    const KernelSet* ks = nullptr;  // M-point kernels
    double2* chirp = nullptr;
    double2* bhat = nullptr;
    double2* scratch = nullptr;
    int4* bsplit = nullptr;  // bhat as the step kernels read it
    AxisDev ax{};  // twiddles of M (shared)
  } bs;
  // 1D grids (qsf_line1d.cu): the step kernels, their geometry tables, the tables of a run of sub-steps and the current program
  const LineKernels* lk = nullptr;
  LineDev line{};
  long long* l_sub0 = nullptr;
  int4 *l_chirp = nullptr, *l_bhat = nullptr, *l_xab = nullptr;
  int lx_mode = 0;
  double lx_delta = 0.0;
  int4 *l_ptab = nullptr, *l_ctab = nullptr;
  int* l_texp = nullptr;
  size_t l_ptab_cap = 0, l_ctab_cap = 0, l_texp_cap = 0;
  int l_steps = 1;  // sub-steps the tables hold
};

namespace qsf {
// whether n is a line length with fused step kernels in this build
bool fused_length(int n);
// whether the grid's solves run in batches (the others run on their own streams)
bool grid_batched(const qsf_grid* g);
// psi = 0 on the grid's stream
int grid_clear(qsf_grid* g);
// Steps of a grid that is not batched (2D and 3D lines run as convolutions, 1D lines), in
// parts for the server: begin checks the program and zeroes its device rows and
// NaN flag; enqueue queues steps [first, first + count) on the grid's stream without
// waiting (no convergence test); wait waits for the stream and reads the NaN flag;
// rows copies the first nsteps rows to the host.  round: steps queued at a time at most.
int solo_begin(qsf_grid* g, const qsf_step_desc* d, int64_t round);
int solo_enqueue(qsf_grid* g, const qsf_step_desc* d, int64_t first, int64_t count);
int solo_wait(qsf_grid* g, bool* bad);
int solo_rows(qsf_grid* g, const qsf_step_desc* d, double* rows, int64_t nsteps);
// qsf_batch_add without waiting for the batch's stream, for a grid that no queued work
// of the batch touches (a solve the server prepares while a round runs); it joins at
// the next batch_launch
int batch_add_nowait(qsf_batch* b, qsf_grid* g, const qsf_step_desc* d, int64_t* slot);
// qsf_batch_run in two halves: launch (rebuild after membership changes, queue the
// steps' graph launches) and finish (wait, read every member's counters)
int batch_launch(qsf_batch* b, int64_t steps);
int batch_finish(qsf_batch* b, int64_t* active);
// exp(-2 pi i t / n), n a multiple of 4, from the angles of one octant, evaluated once
class Roots {
  long long n;
  std::vector<std::pair<long double, long double>> cs;

 public:
  explicit Roots(long long n);
  // times 2^-r, in the split form of the kernels: 2^62 fixed point, the signed 32-bit halves
  // of each component; a component whose low half would be -2^31 moves one unit, 2^-62, so
  // that the kernels can negate the halves
  int4 split(long long t, int r = 0) const;
};
// device twiddles of the line plan (n, ppt), and all of a built length; shared
// by all grids of the process (not to be freed by the caller)
int shared_line_twiddles(int n, int ppt, const int4** out);
constexpr int kPlain = 0;  // selects the plain transforms' twiddles
int axis_twiddles(int n, bool passes, AxisDev* a);
void launch_axis_fft(const KernelSet& K, const GridDev& G, int ax, bool fwd, double sc, cudaStream_t st);
// 1D grids (qsf_line1d.cu)
int init_line_table();
int line_conv_length(int n);  // convolution length of an n-point line (0: none)
int line_setup(qsf_grid* g);
void line_release(qsf_grid* g);
int line_prepare(qsf_grid* g, StepDev& S, int64_t chunk);
size_t line_table_bytes(int n, bool field, bool lg, int64_t chunk);
int line_launch_tables(const LineKernels& L, const GridDev* dG, const StepDev* dS, int count, int steps, bool lg,
                       cudaStream_t st);
int line_launch_steps(const LineKernels& L, bool bs, const GridDev* dG, const StepDev* dS, int count, int steps,
                      cudaStream_t st);
int line_fourier(qsf_grid* g, const GridDev& G, bool fwd, double sc);
// Bluestein plan of a grid whose length has no kernels (qsf_bluestein.cu)
int bs_setup(qsf_grid* g);
void bs_release(qsf_grid* g);
// one axis of fourier<R>() by Bluestein's chirp-z convolution, in place on the array
// arr (psi's geometry: psi itself, or a region-transfer slice), scaled by post
int bs_axis(qsf_grid* g, double2* arr, int ax, bool fwd, double post);
// the convolution length M >= 2n - 1 of an n-point axis of a dim-D grid (0: none)
int bs_size(int n, int dim);
}  // namespace qsf
