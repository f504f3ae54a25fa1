// qsf_line1d.cuh -- whole 1D steps on register-resident lines, many steps per launch.
//
// A 1D line is one small transform after another, so what bounds a step is latency: the
// chain of passes, exchanges and launches, not any pipe.  k_line_run therefore keeps psi
// in registers over all the sub-steps of a launch and spreads a line over the CTAs of a
// cluster, one warp per scheduler or so.  Short lines (below 256 points, and 320) sit in one
// CTA as one line of qsf_lines.cuh.  Longer ones are N = N1 x N2 with 4 points per thread,
// 8 above 12288:
//   X layout  thread (column n2, t1) holds x[N2 (t1 + s T1) + n2]
//   K layout  thread (row k1, t2) holds X[k1 + N1 (t2 + s T2)]
// The transform is N1-point lines along the columns, twiddles exp(-2 pi i k1 n2 / N), one
// all-to-all through distributed shared memory, N2-point lines along the rows; the way
// back is the same in the opposite order on conjugated data.  So a step costs two
// cluster barriers; all other exchanges stay inside a warp or a CTA.  Each group of lines
// keeps its own exponent, which travels with the all-to-all.
//
// An n-point line with a prime factor above 5 runs Bluestein's convolution on the same
// engine (M >= 2n - 1 points): forward, times the transformed chirp, inverse, twice per
// step; the chirps before and after the P phase cancel, those around the X halves are
// part of the static factors.
//
// psi is rounded to complex128 at the end of every step, in registers, as it would be in
// memory: a run does not depend on how it is cut into launches, and without Normalize not
// on how it is cut into calls or by backups either (each call's end applies its factor).
//
// One extra warp of CTA 0 ends the steps (sums, fluxes, the observables row, the
// Normalize factor, the convergence test) while the others work on the next one.  The
// Normalize factor only scales psi: psi takes its power of two, which is exact, at the
// start of a launch and one step after it is known (psi left unscaled over the 256
// sub-steps of a launch would leave the range of a double), and the sums take the rest.
#pragma once
#include "qsf_lines.cuh"

namespace qsf {

// ------------------------------------------------------------ geometry
// N1 x N2 over C CTAs, E points per thread.  4 points where a CTA then has about four warps
// (one per scheduler): a warp's instruction stream is the step's latency, and half the
// points per thread is half the stream and half the code (4096 points: 8 points over 4
// CTAs 25 us a step, with 40 % of the issue slots lost to instruction fetch; 4 points over
// 8 CTAs 12.4 us).  8 points above 12288, where 4 would need more threads than registers
// allow.
template <int N1_, int N2_, int C_, int E_ = 4>
struct Four {
  static constexpr int N1 = N1_, N2 = N2_, N = N1 * N2, C = C_, E = E_;
  using A = Ln<N1, E == 8 ? kEight : kFour>;
  using B = Ln<N2, E == 8 ? kEight : kFour>;
  static_assert(A::E == E && B::E == E && N1 % C == 0 && N2 % C == 0, "layouts");
  static constexpr int real = N / (C * E), nth = (real + 31) / 32 * 32;
  static constexpr int K = A::K > B::K ? A::K : B::K;
  static constexpr int L1 = N2 / C, L2 = N1 / C;  // lines of a CTA in the X and the K layout
  static constexpr int bytes1 = L1 * (N1 + 1) * 16, bytes2 = L2 * (N2 + 1) * 16;
  static constexpr int bytesx = (nth / A::T + 1) * A::LS * 16 > (nth / B::T + 1) * B::LS * 16
                                    ? (nth / A::T + 1) * A::LS * 16
                                    : (nth / B::T + 1) * B::LS * 16;
};
// One line in one CTA.  Its plan per length comes from the autotuner (tuned_line_ppt,
// qsf_tuning.h: 16 points per thread or 8); candidate builds force one with QSF_LINE_PPT.
#ifdef QSF_LINE_PPT
__host__ __device__ constexpr int line_ppt(int) { return QSF_LINE_PPT >= 16 ? 16 : 8; }
#else
__host__ __device__ constexpr int line_ppt(int n) { return tuned_line_ppt(n) >= 16 ? 16 : 8; }
#endif
template <int N_>
struct One {
  static constexpr int N = N_, N1 = N, N2 = 0, C = 1;
  using A = Ln<N, line_ppt(N)>;
  using B = A;
  static constexpr int E = A::E, real = A::T, nth = (real + 31) / 32 * 32, K = A::K;
  static constexpr int L1 = 1, L2 = 1, bytes1 = 0, bytes2 = 0, bytesx = (nth / A::T + 1) * A::LS * 16;
};
// static factors and the potential in shared memory in slot order, where they fit
template <class F, bool BS>
struct LineSmem {
  static constexpr int W = F::nth / 32;
  static constexpr int tab = F::nth * F::E * (BS ? 40 : 24);
  static constexpr int fixed = F::bytes1 + F::bytes2 + F::bytesx + (F::N1 + F::N2) * 4 + 256 + 2 * F::C * W * 48 + 4096;
  static constexpr bool in_smem = fixed + tab <= 220 * 1024;
  static constexpr int bytes = fixed + (in_smem ? tab : 0);
};

// ------------------------------------------------------------ cluster primitives
template <int C>
__device__ __forceinline__ void cl_sync() {
  __syncwarp();
  if constexpr (C == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
__device__ __forceinline__ unsigned peer_addr(const void* p, int rank) {
  unsigned a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
template <int C>
__device__ __forceinline__ void put16(longlong2* p, int rank, longlong2 v) {
  if constexpr (C == 1) *p = v;
  else
    asm volatile("st.shared::cluster.v2.b64 [%0], {%1, %2};" ::"r"(peer_addr(p, rank)), "l"(v.x), "l"(v.y) : "memory");
}
template <int C>
__device__ __forceinline__ void put4(int* p, int rank, int v) {
  if constexpr (C == 1) *p = v;
  else asm volatile("st.shared::cluster.b32 [%0], %1;" ::"r"(peer_addr(p, rank)), "r"(v) : "memory");
}

// one warp's sums of a step: norm and E_pot as three 22-bit limbs each (sums of the lanes'
// words), the exponents they count in, and E_kin
struct WarpSum {
  int n[4], v[4];
  double ek;
  double pad;
};

// ------------------------------------------------------------ the engine
template <class F>
struct LineEngine {
  using A = typename F::A;
  using B = typename F::B;
  LineCtx<A> a;
  LineCtx<B> b;
  longlong2 *buf1, *buf2;
  int *sc1, *sc2;
  // the descriptor's words the steps need, read once (memory barriers would read them again)
  const int4 *tw1, *tw2, *w1, *w2, *bhat;
  int bexp;
  int rank;
  bool real;
  __device__ __forceinline__ LineEngine(unsigned char* sm, const LineDev& d, int r, unsigned (*slot)[32], int* sc)
      : a(reinterpret_cast<longlong2*>(sm + F::bytes1 + F::bytes2), slot, F::nth),
        b(reinterpret_cast<longlong2*>(sm + F::bytes1 + F::bytes2), slot, F::nth), tw1(d.tw1), tw2(d.tw2), w1(d.w1),
        w2(d.w2), bhat(d.bhat), bexp(d.bexp ? *d.bexp : 0), rank(r) {
    buf1 = reinterpret_cast<longlong2*>(sm);
    buf2 = reinterpret_cast<longlong2*>(sm + F::bytes1);
    sc1 = sc;
    sc2 = sc + F::N1;
    real = threadIdx.x < F::real;
    a.on = b.on = real;
  }
  // natural index of slot s in the X and the K layout
  __device__ __forceinline__ int xi(int s) const {
    if constexpr (F::N2 == 0) return a.t + s * A::T;
    else return F::N2 * (a.t + s * A::T) + rank * F::L1 + a.l;
  }
  __device__ __forceinline__ int ki(int s) const {
    if constexpr (F::N2 == 0) return b.t + s * B::T;
    else return rank * F::L2 + b.l + F::N1 * (b.t + s * B::T);
  }
  // lines of layout G to lines of layout H: twiddles, all-to-all, alignment
  template <class G, class H, int LG, int LH>
  __device__ __forceinline__ void turn(longlong2* v, LineCtx<G>& g, LineCtx<H>& h, const int4* w, longlong2* buf, int* sc,
                                       int& scale) {
    constexpr int NG = G::N, NH = H::N;
    scale += line_up<G>(v, g) - 2;
    const int line = rank * LG + g.l;  // this line's index, the position in the lines it goes to
    if (real) {
      const int4* wl = w + line * NG + g.t;
#pragma unroll
      for (int s = 0; s < F::E; ++s) v[s] = fmul_tw(v[s], __ldg(wl + s * G::T));
#pragma unroll
      for (int s = 0; s < F::E; ++s) {
        const int p = g.t + s * G::T;  // the line it goes to
        put16<F::C>(buf + (p % LH) * (NH + 1) + line, p / LH, v[s]);
      }
      for (int r = g.t; r < F::C; r += G::T) put4<F::C>(sc + line, r, scale);
    }
    cl_sync<F::C>();
    int d[F::E], m = 0x7fffffff;
    const longlong2* src = buf + (real ? h.l : 0) * (NH + 1) + h.t;
#pragma unroll
    for (int s = 0; s < F::E; ++s) {
      d[s] = sc[h.t + s * H::T];
      m = min(m, d[s]);
      v[s] = real ? src[s * H::T] : make_longlong2(0, 0);
    }
    m = 0x40000000 - (int)h.group_max((unsigned)(0x40000000 - m));
#pragma unroll
    for (int s = 0; s < F::E; ++s) d[s] = m - d[s];
    scale = line_align<H>(v, d, m, h);
  }
  // X layout -> K layout (the forward transform)
  __device__ __forceinline__ void fwd(longlong2* v, int& scale) {
    line_fft<A>(v, a, tw1, scale);
    if constexpr (F::N2 == 0) cl_sync<F::C>();
    else {
      turn<A, B, F::L1, F::L2>(v, a, b, w1, buf2, sc2, scale);
      line_fft<B>(v, b, tw2, scale);
    }
  }
  // K layout -> X layout (a forward transform too: the inverse takes conjugated data)
  __device__ __forceinline__ void inv(longlong2* v, int& scale) {
    if constexpr (F::N2 == 0) {
      line_fft<A>(v, a, tw1, scale);
      cl_sync<F::C>();
    } else {
      line_fft<B>(v, b, tw2, scale);
      turn<B, A, F::L2, F::L1>(v, b, a, w2, buf1, sc1, scale);
      line_fft<A>(v, a, tw1, scale);
    }
  }
  // Bluestein: times the transformed chirp, in the K layout, conjugated for the way back
  __device__ __forceinline__ void convolve(longlong2* v, int& scale) {
    fwd(v, scale);
    scale += line_up<B, 59>(v, b) - 2 - bexp;
    const int4* w = bhat + (real ? (rank * F::L2 + b.l) * F::N2 + b.t : 0);
#pragma unroll
    for (int s = 0; s < F::E; ++s) v[s] = fconj(fmul_tw(v[s], __ldg(w + s * B::T)));
    inv(v, scale);
  }
};

// ------------------------------------------------------------ the end of a step
// The observables row of step `step` from the warps' sums, by one warp of CTA 0 (lane:
// 0..31).  cfac: the factor of the raw sums (the Normalize factors so far, squared).
// Returns true when the imaginary-time convergence test stops the run.
__device__ __forceinline__ bool line_row(const GridDev& g, const StepDev& S, const WarpSum* part, int nparts, long long sub,
                                         long long step, const double2* snap, bool ek, double& cfac, double& energy, int lane) {
  double a[3] = {0.0, 0.0, 0.0};
  for (int i = lane; i < nparts; i += 32) {
    const WarpSum& p = part[i];
    a[0] += pow2(p.n[3]) * ((double)p.n[2] * 17592186044416.0 + ((double)p.n[1] * 4194304.0 + (double)p.n[0]));
    a[1] += pow2(p.v[3]) * ((double)p.v[2] * 17592186044416.0 + ((double)p.v[1] * 4194304.0 + (double)p.v[0]));
    a[2] += p.ek;
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) a[k] = __shfl_sync(0xffffffffu, warp_sum(a[k]), 0);
  const double norm = a[0] * g.dV * cfac, epot = (S.obs & 2u) ? a[1] * g.dV * cfac : 0.0;
  const double ekin = ek ? 0.5 * g.dVm * ((double)(g.m / g.ax[0].n) * a[2]) * cfac : 0.0;
  const int nb = S.nborders;
  double* row = S.rows + step * (3 + nb);
  if (lane == 0) {
    row[0] = norm;
    row[1] = epot;
    row[2] = ekin;
    if (!(norm > 0.0) || isnan(epot) || isnan(ekin)) S.ctl[4] = 1;
  }
  const double* cA = (g.gauge == 0 && S.coupling && g.n_fields) ? S.coupling + sub * S.coup_stride : nullptr;
  for (int b = 0; b < nb; ++b) {
    double v = 0.0;
    for (int t = lane; t < S.nfterms; t += 32) {
      const FluxTerm ft = S.fterms[t];
      if (ft.border != b) continue;
      const FluxPoint fp = S.fpts[ft.point];
      const double2 c = snap[fp.c];
      double j = 0.0;
      if (ft.w[0] != 0.0) {
        if (fp.p[0] >= 0) {
          const double2 tt = csub(snap[fp.p[0]], snap[fp.q[0]]);
          j = g.ax[0].inv_2dx * (c.x * tt.y + (-c.y) * tt.x);
        }
        if (cA) j += cA[0] * (c.x * c.x + c.y * c.y);
      }
      v += j * ft.w[0];
    }
    v = warp_sum(v);
    if (lane == 0) row[3 + b] = v * cfac * g.dV / g.ax[0].dx;
  }
  if (S.normalize && norm > 0.0) cfac = cfac / norm;
  bool stop = false;
  if (S.mode == 1 && S.state_accuracy > 0.0 && (ek || !(S.obs & 4u))) {
    const double se = (S.energy_after_normalize & 1) ? 1.0 / norm : 1.0;
    const double sk = (S.energy_after_normalize & 2) ? 1.0 / norm : 1.0;
    const double E = epot * se + ekin * sk;
    stop = fabs(E - energy) <= S.state_accuracy;
    energy = E;
  }
  return stop;
}

// sums of a warp's points: lane words to three 22-bit limb sums in lane 0's registers
__device__ __forceinline__ void limb_sum(i64 n, int* out) {
  out[0] = (int)__reduce_add_sync(0xffffffffu, (unsigned)n & 0x3fffffu);
  out[1] = (int)__reduce_add_sync(0xffffffffu, (unsigned)(n >> 22) & 0x3fffffu);
  out[2] = __reduce_add_sync(0xffffffffu, (int)(n >> 44));
}

// the power of two psi takes out of a pending Normalize factor of square cfac: psi goes on
// as psi 2^two, the square as cfac 2^(-2 two)
__device__ __forceinline__ int line_two(double cfac) {
  if (!(cfac > 0.0) || isinf(cfac)) return 0;
  int e;
  frexp(cfac, &e);
  return e >> 1;
}
__device__ __forceinline__ int line_two(const StepDev& S) { return S.normalize ? line_two(S.scale[2]) : 0; }
// whether sub-step `sub` ends a step with E_kin when the run stops after sub-step `stop`
// (ekin_at with a stop that every thread of the cluster agrees on)
__device__ __forceinline__ bool line_ekin_at(const StepDev& S, long long sub, long long stop) {
  if (!(S.obs & 4u) || (sub + 1) % S.substeps) return false;
  return (sub / S.substeps + 1) % S.ekin_every == 0 || sub + 1 >= S.nsteps || sub >= stop;
}

constexpr int kLineSnap = 256;  // snapshot entries a 1D program may have (their lists are in shared memory)

template <class F, bool BS>
__global__ void __cluster_dims__(F::C, 1, 1) __launch_bounds__(F::nth + 32, 1)
    k_line_run(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss, int most) {
  using M = LineSmem<F, BS>;
  constexpr int E = F::E;
  const GridDev& g = Gs[blockIdx.y];
  const StepDev& S = Ss[blockIdx.y];
  const LineDev& D = S.line;
  const long long sub0 = S.ctl[0];
  const long long stop_at = S.ctl[1];  // last sub-step to run (uniform over the cluster)
  if (!(sub0 <= stop_at && sub0 < S.nsteps)) return;
  const long long sub1 = min(S.nsteps, sub0 + most);
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* rest = sm + F::bytes1 + F::bytes2 + F::bytesx;
  unsigned(*slot)[32] = reinterpret_cast<unsigned(*)[32]>(rest);
  WarpSum* part = reinterpret_cast<WarpSum*>(rest + 256);  // [2][C W], CTA 0's are written
  int* sc = reinterpret_cast<int*>(part + 2 * F::C * M::W);
  short* next = reinterpret_cast<short*>(sc + F::N1 + F::N2);      // next snapshot entry of the same thread
  // [1] last sub-step of a converged run, counted from the launch's first; [2] the power of
  // two psi takes at the end of the first sub-step after a step
  int* flags = reinterpret_cast<int*>(next + kLineSnap + 16);
  int4* xat = reinterpret_cast<int4*>((reinterpret_cast<unsigned long long>(flags + 4) + 15) & ~15ull);
  int4* xbt = xat + (BS ? F::nth * E : 0);
  long long* vt = reinterpret_cast<long long*>(xbt + F::nth * E);
  const int rank = F::C == 1 ? 0 : (int)(blockIdx.x % F::C), tid = threadIdx.x;
  const bool worker = tid < F::nth;
  const int n = g.ax[0].n;
  const int K = S.substeps;
  const int kb = BS ? 4 : 2;  // cluster barriers of a sub-step
  if (tid == 0) {
    flags[1] = 0x7fffffff;
  }
  if (!worker) {
    // ------------------------------------------------ the warp that ends the steps
    const int lane = tid & 31;
    const int two = line_two(S);
    double cfac = S.scale[2] * pow2(-2 * two), energy = S.energy_state[0];
    long long step = sub0 / K;
    int k = (int)(sub0 % K), par = 0, due = 0;  // due: the power of two psi takes in this sub-step
    bool pending = false, pek = false, stopped = false;
    long long psub = 0;
    cl_sync<F::C>();
    auto finish = [&]() {
      if (rank == 0) {
        const bool st = line_row(g, S, part + (par ^ 1) * F::C * M::W, F::C * M::W, psub, step, S.snap + (par ^ 1) * S.nsnap,
                                 pek, cfac, energy, lane);
        if (st && !stopped && S.ctl[1] >= S.nsteps) {
          stopped = true;
          const int left = (int)(psub + K - sub0);  // one more step runs
          for (int r = lane; r < F::C; r += 32) put4<F::C>(flags + 1, r, left);
          __syncwarp();
          if (lane == 0) S.ctl[1] = psub + K;
        }
        if (S.normalize) {
          due = line_two(cfac);
          for (int r = lane; r < F::C; r += 32) put4<F::C>(flags + 2, r, due);
        }
      }
      ++step;
      pending = false;
    };
    long long sub = sub0;
    for (; sub < sub1; ++sub) {
      cl_sync<F::C>();
      if (pending) finish();
      for (int i = 1; i < kb; ++i) cl_sync<F::C>();
      cfac *= pow2(-2 * due);
      due = 0;
      const long long stop = min(stop_at, sub0 + (long long)*(volatile int*)(flags + 1));
      const bool end = ++k == K;
      const bool ek = end && line_ekin_at(S, sub, stop);
      if (ek)
        for (int i = 0; i < (BS ? 3 : 2); ++i) cl_sync<F::C>();
      if (end) {
        k = 0;
        pending = true;
        pek = ek;
        psub = sub;
        par ^= 1;
      }
      if (sub >= stop) {
        ++sub;
        break;
      }
    }
    cl_sync<F::C>();
    if (pending) finish();
    if (rank == 0 && lane == 0) {
      S.scale[2] = cfac;
      if (S.normalize) *S.scale = sqrt(cfac);
      S.energy_state[0] = energy;
      S.ctl[2] = step;
      S.ctl[0] = sub;
    }
    cl_sync<F::C>();  // no CTA leaves while its shared memory may still be written
    return;
  }
  // -------------------------------------------------- workers
  LineEngine<F> en(sm, D, rank, slot, sc);
  const long long sid = rank * F::nth + tid, sstr = (long long)F::C * F::nth;  // slot order: sid + s sstr
  const bool lg = g.gauge == 1 && g.n_fields && S.coupling;
  longlong2* psi = reinterpret_cast<longlong2*>(g.psi);
  unsigned valid = 0;
#pragma unroll
  for (int s = 0; s < E; ++s)
    if (en.real && en.xi(s) < n) valid |= 1u << s;
  // static factors and potential of this thread's points
  if constexpr (M::in_smem) {
#pragma unroll
    for (int s = 0; s < E; ++s) {
      const bool ok = valid >> s & 1;
      const int i = en.xi(s);
      xat[s * F::nth + tid] = ok ? D.xa[i] : make_int4(0, 0, 0, 0);
      if (BS) xbt[s * F::nth + tid] = ok ? D.xb[i] : make_int4(0, 0, 0, 0);
      vt[s * F::nth + tid] = ok ? S.Vx[i] : 0;
    }
  }
  auto fa = [&](int s) -> int4 {
    if constexpr (M::in_smem) return xat[s * F::nth + tid];
    else return valid >> s & 1 ? __ldg(D.xa + en.xi(s)) : make_int4(0, 0, 0, 0);
  };
  auto fb = [&](int s) -> int4 {
    if constexpr (M::in_smem) return xbt[s * F::nth + tid];
    else return valid >> s & 1 ? __ldg(D.xb + en.xi(s)) : make_int4(0, 0, 0, 0);
  };
  auto fv = [&](int s) -> long long {
    if constexpr (M::in_smem) return vt[s * F::nth + tid];
    else return valid >> s & 1 ? __ldg(S.Vx + en.xi(s)) : 0;
  };
  // snapshot entries of this thread, as a list
  const int nsnap = S.row_ptr ? S.nsnap : 0;
  int mine = -1;
  for (int e = nsnap - 1; e >= 0; --e) {
    const int i = (int)S.snap_idx[e];
#pragma unroll
    for (int s = 0; s < E; ++s)
      if ((valid >> s & 1) && en.xi(s) == i) {
        next[e] = (short)mine;
        mine = e;
      }
  }
  cl_sync<F::C>();  // every CTA of the cluster runs and has its flags set
  longlong2 v[F::K];
#pragma unroll
  for (int s = 0; s < E; ++s) v[s] = valid >> s & 1 ? psi[en.xi(s)] : make_longlong2(0, 0);
  const long long t0 = *D.sub0;  // first sub-step of the tables
  const int4* copen = D.ctab;
  const int4* cclose = D.ctab + (long long)(D.csteps + 1) * (sstr * E);
  const int xs_exp = S.xs_exp;
  // opening half of sub-step t0 + t: v from doubles (times 2^two) to the transform's input
  auto open = [&](long long t, int two) -> int {
    unsigned em;
    int sc = line_from_double<typename F::A>(v, en.a, em, kLineIn + 2) - two;
    if (em >= 0x7ff) S.ctl[4] = 1;  // Inf or NaN in psi: QSF_ENUMERIC
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = fmul_tw(v[s], fb(s));
    sc -= 2 + xs_exp;
    if (lg) {
      const int4* c = copen + t * (sstr * E) + sid;
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = fmul_tw(shl_by(v[s], 2), __ldg(c + s * sstr));
      sc -= __ldg(D.texp + t * 3 + 1);
    }
    return sc;
  };
  int scale = open(sub0 - t0, line_two(S));
  const int l2m = S.l2m, vexp = 111 - S.vshift;
  const bool any_ek = S.obs & 4u, normalize = S.normalize;
  double2* const snap = S.snap;
  const int* const texp = D.texp;
  const int4* const ptab = D.ptab;
  const long long pstride = D.pstride;
  int k = (int)(sub0 % K), par = 0;
  for (long long sub = sub0;; ++sub) {
    const long long tt = sub - t0;
    const int4* pt = ptab + (pstride ? tt * pstride : 0) + sid;
    const int pe = __ldg(texp + (pstride ? tt : 0) * 3), ce = lg ? __ldg(texp + tt * 3 + 2) : 0;
    if constexpr (BS) {
#pragma unroll 1
      for (int h = 0;; ++h) {
        en.convolve(v, scale);
        if (h) break;
        // P phase of the n transformed points (the chirps around it cancel), conjugated
        scale += line_up<typename F::A, 59>(v, en.a) - 2 - pe;
#pragma unroll
        for (int s = 0; s < E; ++s) v[s] = valid >> s & 1 ? fmul_tw(v[s], __ldg(pt + s * sstr)) : make_longlong2(0, 0);
      }
    } else {
      en.fwd(v, scale);
      scale += line_up<typename F::B, 59>(v, en.b) - 2 - pe;
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = fconj(fmul_tw(v[s], __ldg(pt + s * sstr)));
      en.inv(v, scale);
    }
    // closing half: psi_n, its sums and snapshot
    scale += line_up<typename F::A>(v, en.a) + l2m - 2 - xs_exp;
#pragma unroll
    for (int s = 0; s < E; ++s) v[s] = fmul_tw(BS ? v[s] : fconj(v[s]), fa(s));
    if (lg) {
      const int4* c = cclose + tt * (sstr * E) + sid;
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = shl_by(fmul_tw(v[s], __ldg(c + s * sstr)), 2);
      scale -= ce;
    }
    // the step-ending warp has set this and the stop, if any, before the sub-step's last barrier
    if (normalize && k == 0 && sub > sub0) scale -= *(volatile int*)(flags + 2);
    const bool end = ++k == K;
    const long long stop = min(stop_at, sub0 + (long long)*(volatile int*)(flags + 1));
    const bool ek = any_ek && end && line_ekin_at(S, sub, stop);
    const bool last = sub + 1 >= sub1 || sub >= stop;
    if (end) {
      k = 0;
      ObsSum ob;
#pragma unroll
      for (int s = 0; s < E; ++s) ob.add(v[s], fv(s));
      WarpSum* w = part + par * F::C * M::W + rank * M::W + (tid >> 5);
      int ln[3], lv[3];
      limb_sum((i64)(ob.norm_word() >> 1), ln);
      limb_sum(ob.epot_word(), lv);
      if ((tid & 31) == 0) {
        put16<F::C>(reinterpret_cast<longlong2*>(w->n), 0,
                    make_longlong2((i64)((u64)(unsigned)ln[0] | (u64)(unsigned)ln[1] << 32),
                                   (i64)((u64)(unsigned)ln[2] | (u64)(unsigned)(61 - 2 * scale) << 32)));
        put16<F::C>(reinterpret_cast<longlong2*>(w->v), 0,
                    make_longlong2((i64)((u64)(unsigned)lv[0] | (u64)(unsigned)lv[1] << 32),
                                   (i64)((u64)(unsigned)lv[2] | (u64)(unsigned)(vexp - 2 * scale) << 32)));
      }
      for (int e = mine; e >= 0; e = next[e]) {
        const int i = (int)S.snap_idx[e];
        longlong2 x = make_longlong2(0, 0);
#pragma unroll
        for (int s = 0; s < E; ++s)
          if (en.xi(s) == i) x = v[s];
        snap[par * nsnap + e] = make_double2(fx2d(x.x, scale), fx2d(x.y, scale));
      }
    }
    // psi_n as complex128
#pragma unroll
    for (int s = 0; s < E; ++s)
      v[s] = valid >> s & 1 ? make_longlong2(__double_as_longlong(fx2d(v[s].x, scale)), __double_as_longlong(fx2d(v[s].y, scale)))
                            : make_longlong2(0, 0);
    if (last || ek) {
#pragma unroll
      for (int s = 0; s < E; ++s)
        if (valid >> s & 1) psi[en.xi(s)] = v[s];
    }
    if (ek) {  // transform of psi_n
      unsigned em;
      int se = line_from_double<typename F::A>(v, en.a, em, BS ? kLineIn + 2 : kLineIn);
      if constexpr (BS) {
#pragma unroll
        for (int s = 0; s < E; ++s)
          if (valid >> s & 1) v[s] = fmul_tw(v[s], __ldg(D.chirp + en.xi(s)));
        se -= 2;
        en.convolve(v, se);
      } else {
        en.fwd(v, se);
      }
      double ekv = 0.0;
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const bool ok = BS ? valid >> s & 1 : en.real;
        const double kk = kpos(g.ax[0], BS ? en.xi(s) : en.ki(s));
        const double xr = ok ? fx2d(v[s].x, se) : 0.0, xim = ok ? fx2d(v[s].y, se) : 0.0;
        ekv = fma(kk * kk, fma(xr, xr, xim * xim), ekv);
      }
      ekv = warp_sum(ekv);
      if ((tid & 31) == 0) {
        WarpSum* w = part + par * F::C * M::W + rank * M::W + (tid >> 5);
        put16<F::C>(reinterpret_cast<longlong2*>(&w->ek), 0, make_longlong2(__double_as_longlong(ekv), 0));
      }
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = valid >> s & 1 ? psi[en.xi(s)] : make_longlong2(0, 0);
      cl_sync<F::C>();  // the buffers of this transform are free again
    }
    if (end) par ^= 1;
    if (last) break;
    scale = open(tt + 1, 0);
  }
  cl_sync<F::C>();
  cl_sync<F::C>();
}

// fourier<R>() of a line spread over a cluster: X layout in, K layout out, both natural
// order in memory
template <class F>
__global__ void __cluster_dims__(F::C, 1, 1) __launch_bounds__(F::nth, 1)
    k_line_fft(GridDev g, LineDev D, int fwd, double post_scale) {
  constexpr int E = F::E;
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* rest = sm + F::bytes1 + F::bytes2 + F::bytesx;
  LineEngine<F> en(sm, D, F::C == 1 ? 0 : (int)(blockIdx.x % F::C), reinterpret_cast<unsigned(*)[32]>(rest),
                   reinterpret_cast<int*>(rest + 256));
  longlong2* psi = reinterpret_cast<longlong2*>(g.psi) + (long long)(blockIdx.x / F::C) * F::N;
  longlong2 v[F::K];
#pragma unroll
  for (int s = 0; s < E; ++s) v[s] = en.real ? dconj(psi[en.xi(s)], !fwd) : make_longlong2(0, 0);
  unsigned em;
  int scale = line_from_double<typename F::A>(v, en.a, em);
  cl_sync<F::C>();  // every CTA of the cluster runs, and every point is read
  en.fwd(v, scale);
  line_to_double<typename F::A>(v, scale, !fwd, post_scale);
  if (en.real) {
#pragma unroll
    for (int s = 0; s < E; ++s) psi[en.ki(s)] = v[s];
  }
  cl_sync<F::C>();
}

// the same of an n-point line by Bluestein's convolution
template <class F>
__global__ void __cluster_dims__(F::C, 1, 1) __launch_bounds__(F::nth, 1)
    k_line_bs_fft(GridDev g, LineDev D, int fwd, double post_scale) {
  constexpr int E = F::E;
  extern __shared__ __align__(1024) unsigned char sm[];
  unsigned char* rest = sm + F::bytes1 + F::bytes2 + F::bytesx;
  LineEngine<F> en(sm, D, F::C == 1 ? 0 : (int)(blockIdx.x % F::C), reinterpret_cast<unsigned(*)[32]>(rest),
                   reinterpret_cast<int*>(rest + 256));
  longlong2* psi = reinterpret_cast<longlong2*>(g.psi);
  const int n = g.ax[0].n;
  longlong2 v[F::K];
#pragma unroll
  for (int s = 0; s < E; ++s) v[s] = en.real && en.xi(s) < n ? dconj(psi[en.xi(s)], !fwd) : make_longlong2(0, 0);
  unsigned em;
  int scale = line_from_double<typename F::A>(v, en.a, em, kLineIn + 2) - 2;
#pragma unroll
  for (int s = 0; s < E; ++s)
    if (en.real && en.xi(s) < n) v[s] = fmul_tw(v[s], __ldg(D.chirp + en.xi(s)));
  cl_sync<F::C>();  // every CTA of the cluster runs
  en.convolve(v, scale);
  scale += line_up<typename F::A>(v, en.a) - 2;
#pragma unroll
  for (int s = 0; s < E; ++s)
    if (en.real && en.xi(s) < n) v[s] = fmul_tw(fconj(v[s]), __ldg(D.chirp + en.xi(s)));
  line_to_double<typename F::A>(v, scale, !fwd, post_scale);
#pragma unroll
  for (int s = 0; s < E; ++s)
    if (en.real && en.xi(s) < n) psi[en.xi(s)] = v[s];
  cl_sync<F::C>();
}

// kernels of one transform length
struct LineKernels {
  int n, n1, n2, ctas, nth, epp, t1, t2, ppt;
  int smem, smem_bs;
  void (*run)(const GridDev*, const StepDev*, int);
  void (*run_bs)(const GridDev*, const StepDev*, int);  // this length as a convolution length
  void (*fft)(GridDev, LineDev, int, double);
  void (*fft_bs)(GridDev, LineDev, int, double);
};
template <class F, bool RUN = true>
LineKernels make_line() {
  LineKernels k{};
  k.n = F::N;
  k.n1 = F::N1;
  k.n2 = F::N2;
  k.ctas = F::C;
  k.nth = F::nth;
  k.epp = F::E;
  k.t1 = F::A::T;
  k.t2 = F::B::T;
  k.ppt = F::A::ppt;
  k.smem = LineSmem<F, false>::bytes;
  k.smem_bs = LineSmem<F, true>::bytes;
  if constexpr (RUN) k.run = k_line_run<F, false>;
  if constexpr (F::N2 != 0) {
    k.run_bs = k_line_run<F, true>;
    k.fft = k_line_fft<F>;
    k.fft_bs = k_line_bs_fft<F>;
  }
  return k;
}
const LineKernels* line_kernels(int n);

}  // namespace qsf
