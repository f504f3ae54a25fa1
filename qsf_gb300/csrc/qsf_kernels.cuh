// qsf_kernels.cuh -- sm_103a kernels of the fused split-operator step.
//
// One Strang step  X(dt/2) . P(dt) . X(dt/2)  (propagator.h:311-346 with Split3Base
// mults {0.5, 1, 0.5}, splitting.h:18-27) runs as a short fixed sequence of passes
// over the wavefunction, ending with psi back in X space:
//
//   k_tables      per-step per-axis phase tables (A(t) / E(t) change every step)
//   k_row_open    X half-phase . forward FFT (last axis)
//   k_axis  (3D)  forward FFT axis 1
//   k_axis        forward FFT axis 0 . P phase (with 1/m and Normalize's power of two) .
//                 inverse FFT axis 0
//   k_axis  (3D)  inverse FFT axis 1
//   k_row_close   inverse FFT (last axis) . X half-phase . norm / E_pot partials,
//                 flux snapshot . [next step's X half-phase . forward FFT (last axis)]
//   k_row_ekin, k_axis (E_kin only) forward FFT of psi_n along each axis, sum k^2 |.|^2
//   k_finalize    deterministic reductions, border fluxes, Normalize scale,
//                 imaginary-time convergence, step counter
//
// For dim == 1 a run of whole steps is one kernel (k_line_run, qsf_line1d.cuh).  A
// device step counter lets one captured CUDA graph replay any step.
// Step kernels read their grid and step descriptors from device arrays indexed by
// blockIdx.y, so one launch per stage advances every solve of a batch that shares
// the line length (a single grid is a batch of one).
// FFT kernels are templates on the line length N (compile-time radix plan); the host
// picks the instantiation for the grid's size.
//
// Arithmetic: psi is stored as complex128 between steps; inside a step every pass
// works in block fixed point (int64 components sharing one power-of-two exponent per
// line, or per group of lines that one warp or block holds, qsf_lines.cuh), because
// GB300's integer pipes issue ~64x more instructions per clock than its FP64 pipe.
// Intermediate passes write int64 pairs into psi's own buffer together with their line
// exponents; the next pass aligns every element to the smallest exponent of the
// producing pass.  Phase tables are stored in 2^62 fixed point with magnitude <= 1.
// Norm and E_pot sums of a thread's points are integers.
#pragma once
#include "qsf_fft.cuh"
#include "qsf_fxfft.cuh"
#include "qsf_lines.cuh"
#include "qsf_tuning.h"

namespace qsf {

constexpr int kMaxDim = 3;
constexpr int kMaxFluxBorders = 16;
constexpr int kFinCols = kMaxFluxBorders + 5;  // sums of a k_finalize block: borders, norm, E_pot, E_kin per axis
struct AxisDev {
  int n, n2;
  int shift;  // log2(n) when n is a power of two, else -1
  long long stride;
  double dx, xmin, dp, inv_2dx;
  const int4* tw;      // exp(-2 pi i t / n), t < n, in split form, read by the plain transforms
  const int4* twl[2];  // per-pass twiddle tables of the 8- and the 16-point line plan (qsf_lines.cuh), kTwVar copies
};

struct GridDev {
  int dim;
  long long m;
  AxisDev ax[kMaxDim];
  double dV, dVm, inv_m, eta;
  long long nCAP;
  int pot;
  double NEcharge, EEcharge, Nsoft, Esoft;
  int gauge, n_fields, p_swap;
  int free_mask;  // region of a multi-region grid: axes kept in momentum space (bit d)
  int multi;      // multi-region grid: partial potentials, no absorber in evolve
  int abs_kind;     // QSF_ABS_CAP or QSF_ABS_COS8
  double abs_rate;  // cos^(1/8) mask: applications per unit time (1 / mask_dt)
  double2* psi;
  // TMA tensor maps (CUtensorMap, 128 bytes, 64-byte aligned, in device memory) of psi
  // for the strided-axis passes of axis d < dim - 1: psi as 64-bit words, dims
  // {2 * stride_d, n_d, outer}, box {2 * tile columns, tma_box_rows(n_d), 1}, swizzled
  // over the row of a box; null when the driver offers no encoder (plain copies then)
  const void* tmap[kMaxDim];
  // lines run as convolutions (qsf_bluestein.cu): exp(-i pi j^2 / n), and the transformed
  // kernel over the plan's M points divided by M, times 2^-bexp[0]
  const double2* chirp;
  const int4* bhat;
  const int* bexp;
};

// flux evaluation point: slots into the snapshot of psi_n
struct FluxPoint {
  int c;           // slot of the point itself
  int p[kMaxDim];  // slot of psi[c + stride_d], -1 when the reference's bounds test fails
  int q[kMaxDim];  // slot of psi[c - stride_d]
};
// one (point, border) contribution with the normalised border vector
struct FluxTerm {
  int point;
  int border;
  double w[kMaxDim];
};

struct LineDev {
  int n1, n2, ctas, nth, epp;  // factors (n2 == 0: one line), CTAs, worker threads per CTA, points per thread
  int t1, t2;                  // threads per line of either layout
  int bs;                      // Bluestein: M-point convolution
  const int4 *tw1, *tw2;       // pass twiddles of the lines of either layout
  const int4 *w1, *w2;         // exp(-2 pi i k1 n2 / N) as [n2][k1] and [k1][n2]
  const int4 *xa, *xb;         // static factors of the closing / the opening X half, natural order (Bluestein: times
                               // the chirp, conjugated in xa)
  const int4* bhat;            // Bluestein: transformed chirp times 2^-*bexp / M, [k1][k2]
  const int* bexp;
  const int4* chirp;           // Bluestein: exp(-i pi j^2 / n)
  const int4* ptab;            // [sub-step][slot order] P phases (pstride 0: the same for every sub-step)
  long long pstride;
  const int4* ctab;            // length gauge: [steps + 1] opening, then [steps] closing x.E factors, slot order
  int csteps;                  // steps of ctab
  const int* texp;             // [sub-step][3] exponents of the P, opening and closing tables
  long long* sub0;             // first sub-step the tables hold
};

struct StepDev {
  int mode;  // 1 IM, 2 RE
  double dt;
  long long nsteps;
  const double* coupling;  // device copy of the per-step coupling rows (may be null)
  int coup_stride;         // 3 (velocity gauge) or 6 (length gauge)
  // phase tables in the split form (split62: 2^62 fixed point as signed 32-bit halves)
  const int4* xs;          // static X half-step factor per point (dt/2, incl. absorber), * 2^-xs_exp
  const long long* Vx;     // potential per point in 2^vshift fixed point
  // tables of the sub-steps from ctl[7] on (k_tables), one after another
  int4* ptab;              // [sub-step][dim][nmax] P-phase tables (|.| <= 1)
  int4* xdyn;              // [sub-step][3][dim][nmax] length-gauge factors: open half, close half, close . next open half
  int lg;                  // 2D / 3D: the X halves carry length-gauge factors (a field couples x.E)
  int xs_exp;              // exponent taken out of xs (factors above 1: imaginary time, absorbers backwards in time)
  int vshift;              // Vx = round(V * 2^vshift)
  int l2m;                 // 1/m = m_mant * 2^-l2m, m_mant in (0.5, 1] (folded into axis 0's P table)
  double m_mant;
  int* texp;               // [sub-step][kTexp] exponents taken out of the per-step tables (set by k_tables)
  int* gmin;               // [kGmin] minimum line exponent of each fixed-point pass (gmin_slot)
  int* sc;                 // [4][scmax] line exponents of each fixed-point pass (qsf_passes.cuh)
  int scmax;
  // fused: a sub-step's closing row pass also applies the next sub-step's opening X half
  // and forward transform (ψ stays in fixed point between the steps of a call)
  int fused;
  // E_kin (QSF_OBS_EKIN) at the end of every ekin_every-th step of the call and of its
  // last step; such a step ends with psi_n stored as complex128 (its other transforms
  // need it) and the next one opens from there, the steps between stay fused
  int ekin_every;
  int nmax;
  // reductions
  double* partials;  // [5][pmax]: norm, epot, ekin axis 0..2
  int pmax;
  int nrowblk;          // row blocks of the close pass
  int naxblk[kMaxDim];  // blocks of the E_kin axis passes
  // observables
  unsigned obs;
  int normalize;
  int energy_after_normalize;
  double state_accuracy;
  int nborders;
  double2* snap;              // snapshot slots (1D: two sets, by the parity of the step)
  int nsnap;
  const int* row_ptr;         // CSR over rows: snapshot entries of row r are [row_ptr[r], row_ptr[r+1])
  const long long* snap_idx;  // flat index per snapshot entry (sorted)
  const FluxPoint* fpts;
  const FluxTerm* fterms;
  int nfterms;
  int nfin;           // blocks of k_finalize
  double* fpartials;  // [blocks][kFinCols] sums of k_finalize's blocks
  // control (device): ctl[0] sub-step within call (k_finalize's), ctl[1] stop after
  // this sub-step (or nsteps), ctl[2] steps done, ctl[3] finalize block counter,
  // ctl[4] NaN flag, ctl[6] sub-step of the pass kernels up to axis 0's, which copies it to
  // ctl[5] for those after it (the closing pass advances ctl[6]: no kernel reads the word
  // that it or a kernel beside it writes), ctl[7] first sub-step the tables hold.  The
  // pass kernels' own counter lets k_finalize of one sub-step run beside the next one's
  // first passes.
  // nsteps counts sub-steps: steps * substeps (MultiProductSplit order).
  int substeps;
  long long* ctl;
  double* energy_state;  // [0] last E
  double* rows;          // [nsteps][3 + nborders]
  // Normalize only scales psi: psi stays unscaled in a call and the sums are scaled.
  // [0] the pending factor of psi in memory, [2] its square for psi as the passes hold it,
  // [scale_slot(s)] the power of two (exact) that sub-step s + 2 takes out of it: the step
  // end of s may still run beside the passes of s + 1 (1024^2: 101 us a step when those
  // waited for it)
  double* scale;
  LineDev line;          // 1D grids (qsf_line1d.cuh)
};

__device__ __forceinline__ int scale_slot(long long sub) { return 1 + 2 * (int)(sub & 1); }
// whether sub-step `sub` ends a step whose observables include E_kin
__device__ __forceinline__ bool ekin_at(const StepDev& S, long long sub) {
  if (!(S.obs & 4u) || (sub + 1) % S.substeps) return false;
  const long long step = sub / S.substeps;
  return (step + 1) % S.ekin_every == 0 || sub + 1 >= S.nsteps || sub >= S.ctl[1];
}
// hint: move the 128-byte line holding p from DRAM into L2 (p must be in an allocation)
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ bool pass_active(const StepDev& S, long long sub) { return sub <= S.ctl[1] && sub < S.nsteps; }

// ------------------------------------------------------------ reductions
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
// block-wide sum of NV values; result valid in thread 0.  red needs 32 * NV doubles.
template <int NV>
__device__ __forceinline__ void block_sum(double* v, double* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
  for (int k = 0; k < NV; ++k) v[k] = warp_sum(v[k]);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < NV; ++k) red[k * 32 + wid] = v[k];
  __syncthreads();
  if (wid == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) {
      double t = lane < nw ? red[k * 32 + lane] : 0.0;
      v[k] = warp_sum(t);
    }
  }
  __syncthreads();
}

// ------------------------------------------------------------ geometry
__device__ __forceinline__ double xpos(const AxisDev& a, int i) { return a.xmin + (double)i * a.dx; }
__device__ __forceinline__ double kpos(const AxisDev& a, int i) { return a.dp * (double)(i < a.n2 ? i : i - a.n); }

// ReducedDimInteraction::partial (potential.h:144-178): the interactions of the bounded
// coordinates of region fc (free-axis mask), same operation order
__device__ __forceinline__ double partial_potential(const GridDev& g, int fc, const double* c) {
  auto ne = [&](double x) { return g.NEcharge / sqrt(x * x + g.Nsoft); };
  auto ee = [&](double x, double y) {
    return g.pot == 1 ? g.EEcharge / sqrt((x - y) * (x - y) + x * y + g.Esoft)
                      : g.EEcharge / sqrt((x - y) * (x - y) + g.Esoft);
  };
  if (g.dim == 1) return fc == 0 ? ne(c[0]) : 0.0;
  if (g.dim == 2) {
    if (fc == 0) return ee(c[0], c[1]) + ne(c[0]) + ne(c[1]);
    if (fc == 2) return ne(c[0]);
    if (fc == 1) return ne(c[1]);
    return 0.0;
  }
  switch (fc) {
    case 0: return ee(c[0], c[1]) + ee(c[1], c[2]) + ee(c[2], c[0]) + ne(c[0]) + ne(c[1]) + ne(c[2]);
    case 4: return ee(c[0], c[1]) + ne(c[0]) + ne(c[1]);
    case 2: return ee(c[0], c[2]) + ne(c[0]) + ne(c[2]);
    case 1: return ee(c[1], c[2]) + ne(c[1]) + ne(c[2]);
    case 6: return ne(c[0]);
    case 5: return ne(c[1]);
    case 3: return ne(c[2]);
    default: return 0.0;
  }
}

// potential at a point (potential.h:130-143 and 40-44), same operation order
__device__ __forceinline__ double potential_at(const GridDev& g, const double* c) {
  if (g.pot == 3) return 0.0;
  if (g.multi) return partial_potential(g, g.free_mask, c);
  if (g.pot == 2) {
    double s;
    if (g.dim == 1) s = c[0] * c[0];
    else if (g.dim == 2) s = c[0] * c[0] + c[1] * c[1];
    else s = c[0] * c[0] + (c[1] * c[1] + c[2] * c[2]);
    return g.NEcharge / sqrt(s + g.Nsoft);
  }
  auto ne = [&](double x) { return g.NEcharge / sqrt(x * x + g.Nsoft); };
  auto ee = [&](double x, double y) {
    return g.pot == 1 ? g.EEcharge / sqrt((x - y) * (x - y) + x * y + g.Esoft)
                      : g.EEcharge / sqrt((x - y) * (x - y) + g.Esoft);
  };
  if (g.dim == 1) return ne(c[0]);
  if (g.dim == 2) return ee(c[0], c[1]) + ne(c[0]) + ne(c[1]);
  return ee(c[0], c[1]) + ee(c[1], c[2]) + ee(c[2], c[0]) + ne(c[0]) + ne(c[1]) + ne(c[2]);
}

__device__ __forceinline__ void unflatten(const GridDev& g, long long p, int* idx) {
  if (g.m <= 0x7fffffffLL) {  // 32-bit index arithmetic; shifts for power-of-two axes
    unsigned q = (unsigned)p;
    for (int d = g.dim - 1; d >= 0; --d) {
      const AxisDev& a = g.ax[d];
      if (a.shift >= 0) {
        idx[d] = (int)(q & ((1u << a.shift) - 1u));
        q >>= a.shift;
      } else {
        idx[d] = (int)(q % (unsigned)a.n);
        q /= (unsigned)a.n;
      }
    }
    return;
  }
  for (int d = g.dim - 1; d >= 0; --d) {
    idx[d] = (int)(p % g.ax[d].n);
    p /= g.ax[d].n;
  }
}

// absorbers.h:40-46 with neg_dist_from_edge (grid.h:181-185)
__device__ __forceinline__ double absorb_at(const GridDev& g, double delta, const int* idx) {
  if (g.nCAP <= 0) return 1.0;
  long long nodes[kMaxDim];
  bool all_neg = true;
  for (int d = 0; d < g.dim; ++d) {
    const int i = idx[d];
    const long long nd = i < g.ax[d].n2 ? -(long long)i : (long long)i - g.ax[d].n + 1;
    nodes[d] = g.nCAP + nd;
    if (!(nodes[d] < 0)) all_neg = false;
  }
  if (all_neg) return 1.0;
  if (g.abs_kind == 1) {  // cos^(1/8) mask M = prod_d cos(pi/2 nodes_d / nCAP)^(1/8), to the power delta / mask_dt
    double lsum = 0.0;
    for (int d = 0; d < g.dim; ++d)
      if (nodes[d] > 0) lsum += log(cos(1.5707963267948966 * ((double)nodes[d] / (double)g.nCAP)));
    return exp(delta * g.abs_rate * 0.125 * lsum);
  }
  long long s = 0;
  for (int d = g.dim - 1; d >= 0; --d) {
    const long long v = nodes[d] > 0 ? nodes[d] * (nodes[d] * (nodes[d] * nodes[d])) : 0;
    s = v + s;
  }
  return exp(-delta * (double)s * g.eta);
}

__device__ __forceinline__ double2 expop(int mode, double val) {
  if (mode == 1) return make_double2(exp(-val), 0.0);
  double sn, cs;
  sincos(-val, &sn, &cs);
  return make_double2(cs, sn);
}

// ------------------------------------------------------------ fixed-point helpers
// Tile copies on the TMA engine complete on an mbarrier: one thread issues the copies of
// a whole tile, the others wait on the barrier.
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned phase) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(phase)
      : "memory");
  return ok != 0;
}
// one box of a 3D tensor map into shared memory, completing on the barrier; the first
// coordinate (64-bit words) is a multiple of 2, so every copy starts on 16 bytes
__device__ __forceinline__ void tma_load3(void* dst, const void* tmap, int x, int y, int z, unsigned long long* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          smem_u32(dst)),
      "l"(tmap), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
// bounded wait for phase `phase` of the barrier: false when the limit ran out (the
// caller records the failure; nothing spins without end)
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned phase) {
  for (int it = 0; it < (1 << 20); ++it)
    if (mbar_try_wait(bar, phase)) return true;
  return false;
}

// rows of one TMA box of a strided-axis tile: the largest divisor of n up to 256 (the
// box limit), so that the boxes cover the n rows exactly and none writes past the tile
__host__ __device__ constexpr int tma_box_rows(int n) {
  int b = n < 256 ? n : 256;
  while (n % b) --b;
  return b;
}
// rows of a box when a line of n >= 64 points runs on a tile of M >= 2n - 1 rows: rounded up
// to whole boxes the n rows still fit into the tile
constexpr int kConvBoxRows = 64;
// Passes that leave the wavefunction in fixed point inside a step; each line of a pass
// records its exponent in sc[pass] and the pass minimum in gmin[pass]: 0 last-axis rows
// (open), 1 axis-1 lines forward (3D), 2 axis-0 lines, 3 axis-1 lines inverse (3D).  The
// next pass aligns every element to gmin of its producer.
// Exponent bookkeeping of the step's fixed-point tables: every table is stored with
// magnitude <= 1 in 2^62 fixed point; a table whose exact values exceed 1 (imaginary
// time) is stored times 2^-e and e is added back to the block exponent.
//   texp[0][d]: P table of axis d, texp[1][d] / texp[2][d]: length-gauge X tables of
//   axis d (open / close half), texp[3][d]: opening half of the next sub-step (fused).
//   The static X table's exponent is StepDev::xs_exp.
constexpr int kTexp = 12;
// Pass minima alternate with the parity of the sub-step: the closing pass of sub-step k
// produces pass 0 of k + 1 while pass 0 of k may still be read.  Axis 0's pass resets the
// next sub-step's slot of pass 0, the closing pass those of passes 1 - 3.
constexpr int kGmin = 8;
__device__ __forceinline__ int gmin_slot(int pass, long long sub) { return pass * 2 + (int)(sub & 1); }

// Phase factors (|components| <= 1) are stored in 2^62 fixed point as the signed
// 32-bit halves of each component (int4 {re lo, re hi, im lo, im hi}, as the FFT's
// twiddles), with every low half kept away from -2^31 so that it can be negated.  A
// product x * f returns x * f / 4 from twelve 32 x 32 -> 64-bit multiply-adds (fmul_tw)
// and needs |x| < 2^61.
__device__ __forceinline__ int4 split62(double2 f) {
  long long a = __double2ll_rn(f.x * 4611686018427387904.0), b = __double2ll_rn(f.y * 4611686018427387904.0);
  if ((a & 0xffffffffLL) == 0x80000000LL) ++a;
  if ((b & 0xffffffffLL) == 0x80000000LL) ++b;
  return make_int4((int)a, split_hi(a), (int)b, split_hi(b));
}
__device__ __forceinline__ int4 split_fx(longlong2 v) {
  if ((v.x & 0xffffffffLL) == 0x80000000LL) ++v.x;
  if ((v.y & 0xffffffffLL) == 0x80000000LL) ++v.y;
  return make_int4((int)v.x, split_hi(v.x), (int)v.y, split_hi(v.y));
}
// value of one per-step table entry: kind 0 P phase (hamiltonian.h:52-58: kinetic and,
// in the velocity gauge, A.k), kind 1 / 2 length-gauge x.E factor of the open / close
// X half (hamiltonian.h:60-66 via DipoleCoupling), kind 3 the close half times the open
// half of the next sub-step (coupling row `cn`)
__device__ __forceinline__ double2 table_entry(const GridDev& g, const StepDev& S, const double* cp, const double* cn,
                                               int kind, int d, int i) {
  const AxisDev& a = g.ax[d];
  if (kind == 0) {
    double A = 0.0;
    if (g.gauge != 1 && cp && g.n_fields) {
      int dd = d;
      if (g.p_swap && g.dim >= 2 && d < 2) dd = 1 - d;
      A = cp[dd];
    }
    const double k = kpos(a, i);
    return expop(S.mode, S.dt * (0.5 * k * k + k * A));
  }
  double E = 0.0;
  if (g.n_fields) {
    if (cp) E = cp[(kind == 1 ? 0 : 3) + d];
    if (kind == 3 && cn) E += cn[d];
  }
  return expop(S.mode, (S.dt * 0.5) * (xpos(a, i) * E));
}

__device__ __forceinline__ void flux_block(const GridDev& g, const FluxPoint* __restrict__ fpts, const FluxTerm* __restrict__ fterms,
                           int t0, int t1, const double2* __restrict__ snap, const double* A, int nb, double* red,
                           double* out) {
  double fl[kMaxFluxBorders];
#pragma unroll
  for (int b = 0; b < kMaxFluxBorders; ++b) fl[b] = 0.0;
  for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x) {
    const FluxTerm ft = fterms[t];
    const FluxPoint fp = fpts[ft.point];
    const double2 c = snap[fp.c];
    double dot = 0.0;
    for (int d = 0; d < g.dim; ++d) {
      if (ft.w[d] == 0.0) continue;
      double j = 0.0;
      if (fp.p[d] >= 0) {
        const double2 tt = csub(snap[fp.p[d]], snap[fp.q[d]]);
        j = g.ax[d].inv_2dx * (c.x * tt.y + (-c.y) * tt.x);
      }
      if (A) j += A[d] * (c.x * c.x + c.y * c.y);
      dot += j * ft.w[d];
    }
#pragma unroll
    for (int b = 0; b < kMaxFluxBorders; ++b)
      if (b == ft.border) fl[b] += dot;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int b = 0; b < kMaxFluxBorders; ++b) {
    if (b < nb) {
      const double v = warp_sum(fl[b]);
      if (lane == 0) red[b * 32 + wid] = v;
    }
  }
  __syncthreads();
  if (threadIdx.x < nb) {
    double v = 0.0;
    for (int w = 0; w < nw; ++w) v += red[threadIdx.x * 32 + w];
    out[threadIdx.x] = v;
  }
  __syncthreads();
}

#ifdef QSF_DEFINE_KERNELS
// ------------------------------------------------------------ tables
// Range of the potential (for its fixed-point scale and the imaginary-time X factor
// bound): out[0] = max over points of V (ordered-integer encoding), out[1] = max of -V.
__device__ __forceinline__ long long ordered_bits(double x) {
  long long i = __double_as_longlong(x);
  return i < 0 ? i ^ 0x7fffffffffffffffLL : i;
}
__global__ void k_vrange(GridDev g, long long* out) {
  __shared__ long long r0[32], r1[32];
  long long a = LLONG_MIN, b = LLONG_MIN;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    double c[kMaxDim];
    unflatten(g, p, idx);
    for (int d = 0; d < g.dim; ++d) c[d] = xpos(g.ax[d], idx[d]);
    const double v = potential_at(g, c);
    a = max(a, ordered_bits(v));
    b = max(b, ordered_bits(-v));
  }
  for (int o = 16; o > 0; o >>= 1) {
    a = max(a, __shfl_down_sync(0xffffffffu, a, o));
    b = max(b, __shfl_down_sync(0xffffffffu, b, o));
  }
  if ((threadIdx.x & 31) == 0) {
    r0[threadIdx.x >> 5] = a;
    r1[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      a = max(a, r0[w]);
      b = max(b, r1[w]);
    }
    atomicMax(&out[0], a);
    atomicMax(&out[1], b);
  }
}

// Static tables for X(delta): expOp(delta V) * absorb(delta) per point in 2^62 fixed
// point times 2^-xs_exp, and the potential in 2^vshift fixed point.
__global__ void k_build_static(GridDev g, int mode, double delta, int xs_exp, int4* xsx, long long* Vx,
                               int vshift) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  const double vs = ldexp(1.0, vshift), xsc = ldexp(1.0, -xs_exp);
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    double c[kMaxDim];
    unflatten(g, p, idx);
    for (int d = 0; d < g.dim; ++d) c[d] = xpos(g.ax[d], idx[d]);
    const double v = potential_at(g, c);
    Vx[p] = __double2ll_rn(v * vs);
    const double2 f = expop(mode, delta * v);
    const double a = (g.multi ? 1.0 : absorb_at(g, delta, idx)) * xsc;
    const double2 fa = make_double2(f.x * a, f.y * a);
    xsx[p] = split62(make_double2(fmin(fmax(fa.x, -1.0), 1.0), fmin(fmax(fa.y, -1.0), 1.0)));
  }
}

// The tables of the next `steps` sub-steps, so that no step waits for its own: `tb` blocks
// per (kind, axis) table, each storing a contiguous slice; gridDim.y sub-steps, z solves.  A
// table whose values exceed 1 in magnitude (imaginary time) is stored times 2^-e, e from
// its maximum (every block of the table evaluates that maximum, so the slices agree), and
// e is recorded in texp.  Axis 0's P table carries the mantissa of 1/m (its power of two
// goes into the exponent).
__global__ void __launch_bounds__(256) k_tables(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss,
                                                int tb) {
  const GridDev& g = Gs[blockIdx.z];
  const StepDev& S = Ss[blockIdx.z];
  const long long first = S.ctl[6], sub = first + blockIdx.y;
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) S.ctl[7] = first;
  if (!pass_active(S, sub)) return;
  __shared__ double red[32];
  __shared__ int e_sh;
  const int D = g.dim;
  const int table = blockIdx.x / tb, part = blockIdx.x % tb;
  const int kind = table / D, d = table % D;
  if (kind > 0 && !S.lg) return;
  if (kind == 3 && (!S.fused || sub + 1 >= S.nsteps)) return;
  const double* cp = S.coupling ? S.coupling + sub * S.coup_stride : nullptr;
  const double* cn = (S.coupling && sub + 1 < S.nsteps) ? S.coupling + (sub + 1) * S.coup_stride : nullptr;
  const int n = g.ax[d].n;
  const double mant = kind == 0 && d == 0 ? S.m_mant : 1.0;
  double mx = mant;  // real time: phases of modulus 1 times the mantissa
  if (S.mode == 1) {  // imaginary time: real factors, maximum over the table
    mx = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) mx = fmax(mx, table_entry(g, S, cp, cn, kind, d, i).x * mant);
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
    if (part == 0) S.texp[blockIdx.y * kTexp + kind * 3 + d] = e;
  }
  __syncthreads();
  const double sc = ldexp(mant, -e_sh);
  int4* out = kind == 0 ? S.ptab + ((size_t)blockIdx.y * D + d) * S.nmax
                        : S.xdyn + (((size_t)blockIdx.y * 3 + kind - 1) * D + d) * S.nmax;
  const int chunk = (n + tb - 1) / tb;
  const int i1 = min(n, (part + 1) * chunk);
  for (int i = part * chunk + threadIdx.x; i < i1; i += blockDim.x) {
    const double2 f = table_entry(g, S, cp, cn, kind, d, i);
    out[i] = split62(make_double2(fmin(fmax(f.x * sc, -1.0), 1.0), fmin(fmax(f.y * sc, -1.0), 1.0)));
  }
}

#endif  // QSF_DEFINE_KERNELS

#ifdef QSF_DEFINE_KERNELS
// ------------------------------------------------------------ flux + finalize
// Block-partial border fluxes over flux terms [t0, t1): each term is one grid point
// and one border type; j_d = inv_2dx Im(conj(psi) (psi_+ - psi_-)) (0 where the
// reference's flat-index bounds test fails, grid.h:470-472) + A_d |psi|^2 (velocity
// gauge), dotted with the normalised border vector.  out[b] written by thread b.
__global__ void __launch_bounds__(256) k_flux(GridDev g, const FluxPoint* fpts, const FluxTerm* fterms, int nfterms,
                                              const double2* snap, double A0, double A1, double A2, int useA, int nb,
                                              double* out_partials) {
  __shared__ double red[32 * kMaxFluxBorders];
  double Av[3] = {A0, A1, A2};
  const int chunk = (nfterms + gridDim.x - 1) / gridDim.x;
  const int t0 = blockIdx.x * chunk, t1 = min(nfterms, t0 + chunk);
  flux_block(g, fpts, fterms, t0, t1, snap, useA ? Av : nullptr, nb, red, out_partials + blockIdx.x * kFinCols);
}

// End of a sub-step: border fluxes (grid.h:519-573, propagator.h:249-265) from the psi_n
// snapshot, the sums of all partials in a fixed order, the observables row, the Normalize
// factor, the imaginary-time convergence test and the counters.  Block b sums its share of
// the flux terms and of the row and E_kin partials; the last block to finish adds the
// blocks' sums and writes the row.  What bounds it: chains of dependent loads, so the words
// of the last part are loaded before the sums they wait for.
__global__ void __launch_bounds__(256) k_finalize(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss) {
  const GridDev& g = Gs[blockIdx.y];
  const StepDev& S = Ss[blockIdx.y];
  const long long sub = S.ctl[0], stop = S.ctl[1], nsteps = S.nsteps;
  const int nblk = S.nfin;  // its own count, whatever the launch's: the sums do not depend on the batch
  if (!(sub <= stop && sub < nsteps) || (int)blockIdx.x >= nblk) return;
  __shared__ double red[32 * kMaxFluxBorders];
  __shared__ int is_last;
  const int K = S.substeps, nb = S.nborders, tid = threadIdx.x;
  // observables, Normalize and the convergence test once per step (its last sub-step)
  const bool step_end = K == 1 || (sub + 1) % K == 0;
  const long long step = K == 1 ? sub : sub / K;
  if (!step_end) {
    // only the counters move, and only when every block has read them: a block that starts
    // late would take the next sub-step for its own
    __syncthreads();  // this block's threads have
    if (nblk > 1) __threadfence();
    if (tid == 0 && (nblk == 1 || atomicAdd((unsigned long long*)&S.ctl[3], 1ull) == (unsigned long long)nblk - 1)) {
      S.scale[scale_slot(sub)] = 0.0;
      S.ctl[3] = 0;
      S.ctl[0] = sub + 1;
    }
    return;
  }
  const bool ek = ekin_at(S, sub);
  const double cf0 = S.scale[2], e0 = S.energy_state[0], e1 = S.scale[scale_slot(sub + 1)];
  const int nrow = S.nrowblk, nft = S.nfterms, D = g.dim;
  double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  double* mine = S.fpartials + (size_t)blockIdx.x * kFinCols;
  {
    const int chunk = (nrow + nblk - 1) / nblk, i1 = min(nrow, ((int)blockIdx.x + 1) * chunk);
    for (int i = blockIdx.x * chunk + tid; i < i1; i += blockDim.x) {
      acc[0] += S.partials[i];
      acc[1] += S.partials[S.pmax + i];
    }
    if (ek)
      for (int d = 0; d < D; ++d) {
        const int n = d == D - 1 ? nrow : S.naxblk[d], c = (n + nblk - 1) / nblk, j1 = min(n, ((int)blockIdx.x + 1) * c);
        for (int i = blockIdx.x * c + tid; i < j1; i += blockDim.x) acc[2 + d] += S.partials[(size_t)(2 + d) * S.pmax + i];
      }
  }
  if (nft > 0) {
    const double* A = (g.gauge == 0 && S.coupling && g.n_fields) ? S.coupling + sub * S.coup_stride : nullptr;
    const int chunk = (nft + nblk - 1) / nblk;
    const int t0 = blockIdx.x * chunk, t1 = min(nft, t0 + chunk);
    flux_block(g, S.fpts, S.fterms, t0, t1, S.snap, A, nb, red, mine);
  }
  if (ek) block_sum<5>(acc, red);
  else block_sum<2>(acc, red);
  if (nblk > 1) {
    if (tid == 0) {
      for (int k = 0; k < 5; ++k) mine[kMaxFluxBorders + k] = acc[k];
      __threadfence();
      const unsigned long long done = atomicAdd((unsigned long long*)&S.ctl[3], 1ull);
      is_last = done == (unsigned long long)nblk - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
  } else {
    __syncthreads();  // this block's fluxes
  }
  // the blocks' sums: one warp per column, blocks in order of lanes and strides
  __shared__ double tot[kFinCols];
  const int lane = tid & 31;
  for (int c = tid >> 5; c < kFinCols; c += (int)(blockDim.x >> 5)) {
    if (c < kMaxFluxBorders ? c >= nb || nft == 0 : nblk == 1) continue;
    double v = 0.0;
    for (int k = lane; k < nblk; k += 32) v += S.fpartials[(size_t)k * kFinCols + c];
    v = warp_sum(v);
    if (lane == 0) tot[c] = v;
  }
  __syncthreads();
  double* row = S.rows + step * (3 + nb);
  if (tid < nb) row[3 + tid] = nft > 0 ? tot[tid] * cf0 * g.dV / g.ax[0].dx : 0.0;
  if (tid == 0) {
    if (nblk > 1)
      for (int k = 0; k < 5; ++k) acc[k] = tot[kMaxFluxBorders + k];
    double cfac = cf0;
    const double norm = acc[0] * g.dV * cfac;
    const double epot = acc[1] * g.dV * cfac;
    double ekin = 0.0;
    if (ek) {
      for (int d = 0; d < D; ++d) ekin += (double)(g.m / g.ax[d].n) * acc[2 + d];
      ekin = 0.5 * g.dVm * ekin * cfac;
    }
    row[0] = norm;
    row[1] = epot;
    row[2] = ekin;
    if (!(norm > 0.0) || isnan(epot) || isnan(ekin)) S.ctl[4] = 1;
    if (S.normalize && norm > 0.0) {
      cfac = cfac / norm;
      *S.scale = sqrt(cfac);
      // the next sub-step takes e1, the one after it the power chosen here
      if (K == 1) cfac = ldexp(cfac, -2 * (int)e1);
      int e;
      frexp(cfac, &e);
      e >>= 1;
      S.scale[scale_slot(sub)] = (double)e;
      S.scale[2] = K == 1 ? cfac : ldexp(cfac, -2 * e);
    }
    // the convergence test needs E = E_pot + E_kin: with E_kin on every k-th step only,
    // it runs on those steps (comparing with the previous one that had it)
    if (S.mode == 1 && S.state_accuracy > 0.0 && (ek || !(S.obs & 4u))) {
      const double se = (S.energy_after_normalize & 1) ? 1.0 / norm : 1.0;
      const double sk = (S.energy_after_normalize & 2) ? 1.0 / norm : 1.0;
      const double E = epot * se + ekin * sk;
      S.energy_state[0] = E;
      // converged: one more step runs (its last sub-step is sub + substeps)
      if (stop >= nsteps && fabs(E - e0) <= S.state_accuracy) S.ctl[1] = sub + K;
    }
    S.ctl[2] = step + 1;
    S.ctl[3] = 0;
    S.ctl[0] = sub + 1;
  }
}

// apply a pending Normalize factor (end of a qsf_step call / qsf_normalize)
__global__ void k_scale(double2* psi, long long m, const double* scale) {
  const double s = *scale;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < m; p += stride) psi[p] = cscale(psi[p], s);
}

// ------------------------------------------------------------ granular members
// evolve<M,R>(delta) with the reference's per-point formula (grid.h:394-418)
// X-phase factor per point of evolve<M, X>(delta) without an X-space coupling term:
// expOp(delta V) times the absorber (grid.h:394-418), as one complex factor
__global__ void k_evolve_xtab(GridDev g, int mode, double delta, double2* __restrict__ tab) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    double c[kMaxDim];
    unflatten(g, p, idx);
    for (int d = 0; d < g.dim; ++d) c[d] = xpos(g.ax[d], idx[d]);
    double2 f = expop(mode, delta * potential_at(g, c));
    if (g.nCAP > 0 && !g.multi) f = cscale(f, absorb_at(g, delta, idx));
    tab[p] = f;
  }
}
// per-axis factors of evolve<M, P>(delta): expOp(delta (k^2 / 2 + A_d k)) for axis d
// (the P Hamiltonian is a sum over axes, so its exponential is their product)
__global__ void k_evolve_ptab(GridDev g, int mode, double delta, double c0, double c1, double c2, int nmax,
                              double2* __restrict__ tab) {
  double cv[3] = {c0, c1, c2};
  if (g.p_swap && g.dim >= 2) {
    const double t = cv[0];
    cv[0] = cv[1];
    cv[1] = t;
  }
  const bool coupled = g.gauge == 0 && g.n_fields;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.dim * nmax; e += gridDim.x * blockDim.x) {
    const int d = e / nmax, i = e % nmax;
    if (i >= g.ax[d].n) continue;
    const double k = kpos(g.ax[d], i);
    tab[e] = expop(mode, delta * (0.5 * k * k + (coupled ? k * cv[d] : 0.0)));
  }
}
// psi *= tab[p] (X) or psi *= prod_d tab[d][idx_d] (P)
__global__ void k_apply_xtab(double2* __restrict__ psi, const double2* __restrict__ tab, long long m) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < m; p += stride) {
    const double2 a = psi[p], f = tab[p];
    psi[p] = make_double2(a.x * f.x - a.y * f.y, a.x * f.y + a.y * f.x);
  }
}
__global__ void k_apply_ptab(GridDev g, const double2* __restrict__ tab, int nmax) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    unflatten(g, p, idx);
    double2 f = tab[idx[0]];
    for (int d = 1; d < g.dim; ++d) {
      const double2 t = tab[d * nmax + idx[d]];
      f = make_double2(f.x * t.x - f.y * t.y, f.x * t.y + f.y * t.x);
    }
    const double2 a = g.psi[p];
    g.psi[p] = make_double2(a.x * f.x - a.y * f.y, a.x * f.y + a.y * f.x);
  }
}

__global__ void k_evolve(GridDev g, int mode, int rep, double delta, double c0, double c1, double c2) {
  double cv[3] = {c0, c1, c2};
  if (rep == 2 && g.p_swap && g.dim >= 2) {
    const double t = cv[0];
    cv[0] = cv[1];
    cv[1] = t;
  }
  const int couples = g.gauge == 0 ? 2 : 1;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    double c[kMaxDim];
    unflatten(g, p, idx);
    double H;
    if (rep == 2) {
      for (int d = 0; d < g.dim; ++d) c[d] = kpos(g.ax[d], idx[d]);
      if (g.dim == 1) H = 0.5 * c[0] * c[0];
      else if (g.dim == 2) H = 0.5 * c[0] * c[0] + 0.5 * c[1] * c[1];
      else H = 0.5 * c[0] * c[0] + (0.5 * c[1] * c[1] + 0.5 * c[2] * c[2]);
    } else {
      for (int d = 0; d < g.dim; ++d) c[d] = xpos(g.ax[d], idx[d]);
      H = potential_at(g, c);
    }
    double ct = 0.0;
    if (couples == rep && g.n_fields) {
      if (g.dim == 1) ct = c[0] * cv[0];
      else if (g.dim == 2) ct = c[0] * cv[0] + c[1] * cv[1];
      else ct = c[0] * cv[0] + (c[1] * cv[1] + c[2] * cv[2]);
    }
    const double val = delta * (H + ct);
    double2 v = g.psi[p];
    if (mode == 1) v = cscale(v, exp(-val));
    else {
      double sn, cs;
      sincos(-val, &sn, &cs);
      v = make_double2(v.x * cs - v.y * sn, v.x * sn + v.y * cs);
    }
    if (rep == 1 && g.nCAP > 0 && !g.multi) v = cscale(v, absorb_at(g, delta, idx));
    g.psi[p] = v;
  }
}

// sum |psi|^2 w(p) per block (average_, grid.h:425-441); op 0 identity, 1 potential, 2 kinetic
__global__ void __launch_bounds__(256) k_average(GridDev g, int rep, int op, double* out_partials) {
  __shared__ double red[32];
  double acc = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    const double2 v = g.psi[p];
    double w = 1.0;
    if (op != 0) {
      int idx[kMaxDim];
      double c[kMaxDim];
      unflatten(g, p, idx);
      if (op == 2) {
        for (int d = 0; d < g.dim; ++d) c[d] = kpos(g.ax[d], idx[d]);
        if (g.dim == 1) w = 0.5 * c[0] * c[0];
        else if (g.dim == 2) w = 0.5 * c[0] * c[0] + 0.5 * c[1] * c[1];
        else w = 0.5 * c[0] * c[0] + (0.5 * c[1] * c[1] + 0.5 * c[2] * c[2]);
      } else {
        for (int d = 0; d < g.dim; ++d) c[d] = xpos(g.ax[d], idx[d]);
        w = potential_at(g, c);
      }
    }
    acc = fma(fma(v.x, v.x, v.y * v.y), w, acc);
  }
  block_sum<1>(&acc, red);
  if (threadIdx.x == 0) out_partials[blockIdx.x] = acc;
}

// potential per point (X representation), for the member averages of E_pot
__global__ void k_build_vtab(GridDev g, double* __restrict__ vtab) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    double c[kMaxDim];
    unflatten(g, p, idx);
    for (int d = 0; d < g.dim; ++d) c[d] = xpos(g.ax[d], idx[d]);
    vtab[p] = potential_at(g, c);
  }
}
// sum |psi|^2 w(p) per block with the weights from a table (E_pot from the potential table)
__global__ void __launch_bounds__(256) k_average_tab(GridDev g, const double* __restrict__ w, double* out_partials) {
  __shared__ double red[32];
  double acc = 0.0;
  const long long stride = (long long)gridDim.x * blockDim.x;
#pragma unroll 4
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    const double2 v = g.psi[p];
    acc = fma(fma(v.x, v.x, v.y * v.y), w[p], acc);
  }
  block_sum<1>(&acc, red);
  if (threadIdx.x == 0) out_partials[blockIdx.x] = acc;
}

__global__ void k_reduce_partials(const double* part, int n, double scale, double* out) {
  __shared__ double red[32];
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) acc += part[i];
  block_sum<1>(&acc, red);
  if (threadIdx.x == 0) *out = acc * scale;
}

// gather psi at the snapshot indices (granular flux)
__global__ void k_gather(const double2* psi, const long long* idx, int n, double2* out) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = psi[idx[i]];
}

// maskRegion (grid.h:582-597) with CAP::mask (absorbers.h:48-54)
// CAP::mask of one node (absorbers.h:48-54): 1 outside the margin
__device__ __forceinline__ double mask1(const GridDev& g, long long nd) {
  const long long nodes = g.nCAP + nd;
  if (nodes < 0) return 1.0;
  const double v = nodes > 0 ? (double)(nodes * (nodes * (nodes * nodes))) : 0.0;
  return exp(-(v + 0) * g.eta);
}
__device__ __forceinline__ long long neg_dist(const GridDev& g, int d, int i) {
  return i < g.ax[d].n2 ? -(long long)i : (long long)i - g.ax[d].n + 1;
}

// Per-axis values of the one-node absorber mask, mtab[d * nmax + i] = CAP::mask of axis
// d's node i (absorbers.h:48-54).  The mask of several nodes, exp(-eta sum_d n_d^4), is
// the product of these (to rounding), so the region masks and transfers below need no exp.
__global__ void k_mask_tab(GridDev g, int nmax, double* __restrict__ mtab) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < g.dim * nmax; e += gridDim.x * blockDim.x) {
    const int d = e / nmax, i = e % nmax;
    mtab[e] = i < g.ax[d].n ? mask1(g, neg_dist(g, d, i)) : 1.0;
  }
}

// Slice of a region transfer (getBox + maskSlice, multigrid.h:454-569): src in the
// margins along fc times 1 - mask(fc) and, for a destination in group 1, the corner
// correction (mask_correction, multigrid.h:519-530); zero elsewhere, except in 1D,
// where the whole line is copied and only its margins are masked.  In 3D the sliding
// axis is limited to the n / nCAP boxes (slide_lim planes).
__global__ void k_mg_slice(GridDev g, const double2* __restrict__ src, double2* __restrict__ slice, int fc, int group,
                           long long slide_lim, const double* __restrict__ mtab, int nmax) {
  const int D = g.dim;
  const int slide = D == 3 ? (fc == 1 ? 2 : 1) : -1;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    unflatten(g, p, idx);
    const int i = idx[fc];
    const bool band = i < g.nCAP || i >= g.ax[fc].n - g.nCAP;
    if (!band || (slide >= 0 && idx[slide] >= slide_lim)) {
      slice[p] = (D == 1 && !band) ? src[p] : make_double2(0.0, 0.0);
      continue;
    }
    const double mv = 1.0 - mtab[fc * nmax + i];
    double f = mv;
    if (group == 1) {
      double corr = 1.0;
      if (D == 2) {
        const int o = 1 - fc;
        const double b0 = fc == 0 ? 1.0 : 1.0 - mtab[o * nmax + idx[o]];
        const double b1 = fc == 1 ? 1.0 : 1.0 - mtab[o * nmax + idx[o]];
        corr = 1 - 0.5 * (b0 * b1);
      } else if (D == 3) {
        double a[3], b[3];
        for (int d = 0; d < 3; ++d) {
          const double mk = mtab[d * nmax + idx[d]];
          a[d] = d == fc ? 0 : mk;
          b[d] = d == fc ? 1.0 : mk;
        }
        corr = 0.5 * (a[0] + (a[1] + (a[2] + 0))) + (1.0 / 6.0) * (1 - (b[0] * (b[1] * b[2])));
      }
      f = mv * corr;
    }
    const double2 v = src[p];
    slice[p] = make_double2(v.x * f, v.y * f);
  }
}

// coherent addition (add, multigrid.h:571-586): dst += slice
__global__ void k_add_slice(double2* __restrict__ dst, const double2* __restrict__ slice, long long m) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < m; p += stride) {
    const double2 a = dst[p], b = slice[p];
    dst[p] = make_double2(a.x + b.x, a.y + b.y);
  }
}

// maskRegion_ (grid.h:582-597): psi *= the mask of the bounded axes' nodes, as the
// product of the per-axis one-node masks (a free axis contributes 1)
__global__ void k_mask(GridDev g, int b0, int b1, int b2, const double* __restrict__ mtab, int nmax) {
  const int bounded[3] = {b0, b1, b2};
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    unflatten(g, p, idx);
    double mk = 1.0;
    for (int d = 0; d < g.dim; ++d)
      if (bounded[d]) mk *= mtab[d * nmax + idx[d]];
    if (mk != 1.0) g.psi[p] = cscale(g.psi[p], mk);
  }
}

// psi += gaussian(at, delta, x...) (wf/preset.h:5-10)
__global__ void k_add_gaussian(GridDev g, double at, double delta) {
  const double delta_inv = 1.0 / delta;
  const double base = sqrt(delta_inv * sqrt(1.0 / 3.14159265358979323846));
  const double nrm = g.dim == 1 ? base : (g.dim == 2 ? base * base : base * (base * base));
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < g.m; p += stride) {
    int idx[kMaxDim];
    unflatten(g, p, idx);
    double t[kMaxDim];
    for (int d = 0; d < g.dim; ++d) {
      const double x = xpos(g.ax[d], idx[d]);
      t[d] = (x - at) * (x - at) * delta_inv * delta_inv;
    }
    const double s = g.dim == 1 ? t[0] : (g.dim == 2 ? t[0] + t[1] : t[0] + (t[1] + t[2]));
    g.psi[p].x += exp(-0.5 * s) * nrm;
  }
}

#endif  // QSF_DEFINE_KERNELS

// ------------------------------------------------------------ per-size kernel table
struct KernelSet {
  int n;
  void (*row_open)(const GridDev*, const StepDev*);
  void (*row_close)(const GridDev*, const StepDev*);
  void (*row_ekin)(const GridDev*, const StepDev*);
  void (*axis_one)(const GridDev*, const StepDev*, int, int);  // one transform: forward or inverse (last argument)
  void (*axis_fpi)(const GridDev*, const StepDev*, int, int);
  void (*axis_ekin)(const GridDev*, const StepDev*, int, int);
  // the same six for shorter lines as convolutions over the n points
  void (*conv_open)(const GridDev*, const StepDev*);
  void (*conv_close)(const GridDev*, const StepDev*);
  void (*conv_rekin)(const GridDev*, const StepDev*);
  void (*conv_one)(const GridDev*, const StepDev*, int, int);
  void (*conv_fpi)(const GridDev*, const StepDev*, int, int);
  void (*conv_aekin)(const GridDev*, const StepDev*, int, int);
  // plain transforms, [0] inverse, [1] forward: lines (axis: ax, columns) of a block, scale on the way out
  void (*row_fft[2])(GridDev, int, double);
  void (*axis_fft[2])(GridDev, int, int, double);
  int axis_cols, axis_threads;
  int row_lines, row_threads, row_smem;  // last-axis passes: lines, threads, dynamic shared memory of a block
  int col_lines, col_threads, col_smem;  // strided-axis passes: columns, threads, dynamic shared memory
};

// the passes of grids whose lines are convolutions over k.n points
inline KernelSet conv_kernels(const KernelSet& k) {
  KernelSet c = k;
  c.row_open = k.conv_open;
  c.row_close = k.conv_close;
  c.row_ekin = k.conv_rekin;
  c.axis_one = k.conv_one;
  c.axis_fpi = k.conv_fpi;
  c.axis_ekin = k.conv_aekin;
  return c;
}

// kernel table of the supported sizes (qsf_sizes_*.cu); nullptr when n is not built
const KernelSet* kernels_for(int n);

}  // namespace qsf
#include "qsf_passes.cuh"
#include "qsf_plain.cuh"
#include "qsf_line1d.cuh"
namespace qsf {

// sizes up to 4096 get the multi-dimensional passes, up to 8192 the plain row transform;
// longer lines are 1D and only have their place in the list of built lengths here: the 1D
// steps, and the transforms of the longer lines, have kernels of their own (LineKernels)
template <int N>
KernelSet make_kernel_set() {
  static_assert(is_smooth(N), "grid sizes must be 2^a 3^b 5^c");
  static_assert(N <= 16384, "1D lines longer than 16384 points are not built");
  KernelSet k{};
  k.n = N;
  if constexpr (N <= 8192) {
    using G = Ln<N, tuned_ppt(N)>;
    using A = Ln<N, axis_ppt(N)>;
    if constexpr (N <= 4096) {
      k.row_open = k_row_open<G>;
      k.row_close = k_row_close<G>;
      k.row_ekin = k_row_ekin<G>;
      k.axis_one = k_axis<0, A>;
      k.axis_fpi = k_axis<2, A>;
      k.axis_ekin = k_axis<3, A>;
      k.conv_open = k_row_open<G, true>;
      k.conv_close = k_row_close<G, true>;
      k.conv_rekin = k_row_ekin<G, true>;
      k.conv_one = k_axis<0, A, true>;
      k.conv_fpi = k_axis<2, A, true>;
      k.conv_aekin = k_axis<3, A, true>;
      k.axis_fft[0] = k_axis_fft<N, false>;
      k.axis_fft[1] = k_axis_fft<N, true>;
      k.axis_threads = plain_threads(N);
      k.axis_cols = plain_tile(N) / N < 64 ? plain_tile(N) / N : 64;
      k.row_lines = G::L;
      k.row_threads = G::kRowThreads;
      k.row_smem = G::kRowSmem;
      k.col_lines = A::C;
      k.col_threads = A::kColThreads;
      k.col_smem = A::kColSmem;
    }
    k.row_fft[0] = k_row_fft<N, false>;
    k.row_fft[1] = k_row_fft<N, true>;
  }
  return k;
}

}  // namespace qsf
