// qsf_passes.cuh -- the pass kernels of 2D and 3D grids over register-resident lines
// (qsf_lines.cuh).
//
// Passes leave psi in fixed point between them (int64 pairs in psi's buffer) with one
// exponent per line of the producing pass:
//   pass 0  rows            sc[0][row]                   (row = i0 n + i1 in 3D)
//   pass 1  axis 1 forward  sc[1][i2 n + i0]             (3D)
//   pass 2  axis 0          sc[2][i1] (2D), [i2 n + i1] (3D)
//   pass 3  axis 1 inverse  sc[3][i0 n + i2]             (3D)
// in the order the consumer's points run, so that a thread reads its points' exponents
// as coalesced words.  The next pass aligns every point to the smallest exponent of its
// producer (gmin).  Inverse transforms are forward ones on conjugated data; passes 2 and
// 3 store the conjugated form, which the next inverse pass takes as it is.
#pragma once

namespace qsf {

// ------------------------------------------------------------ column tiles
// The C columns of a strided-axis block as the tensor map's box leaves them: row i holds
// C 16-byte points, column l at position l ^ column_swz(i) (the hardware's 128-, 64- and
// 32-byte swizzles), so that a warp reading one column's consecutive rows meets every
// bank once.
template <int C>
__host__ __device__ constexpr int column_swz(int i) {
  return C == 8 ? (i & 7) : C == 4 ? ((i >> 1) & 3) : C == 2 ? ((i >> 2) & 1) : 0;
}

// One box (rows [y, y + box), columns [x / 2, x / 2 + C)) between shared memory and psi
__device__ __forceinline__ void tma_store3(const void* tmap, int x, int y, int z, const void* src) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(tmap), "r"(x),
               "r"(y), "r"(z), "r"(smem_u32(src))
               : "memory");
}

// Points of a line of axis d: the plan's, or in a convolution plan (BS) the axis' own.
template <class G, bool BS>
__device__ __forceinline__ int line_len(const AxisDev& a) {
  return BS ? a.n : G::N;
}

// Geometry of a strided-axis block and its shared memory.
template <class G, bool BS>
struct ColBlock {
  const int N;  // rows of the tile that psi has
  longlong2* tile;
  unsigned long long* bar;
  const void* tmap;
  longlong2* psi;
  long long inner, o, c0, obase;
  int Ch;
  bool boxes;
  __device__ __forceinline__ ColBlock(const GridDev& g, int ax, unsigned char* sm) : N(line_len<G, BS>(g.ax[ax])) {
    tile = reinterpret_cast<longlong2*>(sm);
    bar = reinterpret_cast<unsigned long long*>(sm + (G::kColBytes + 127) / 128 * 128 + 256);
    psi = reinterpret_cast<longlong2*>(g.psi);
    inner = g.ax[ax].stride;
    const long long tiles = (inner + G::C - 1) / G::C;
    o = blockIdx.x / tiles;
    c0 = (blockIdx.x % tiles) * G::C;
    Ch = (int)min((long long)G::C, inner - c0);
    obase = o * (long long)N * inner + c0;
    tmap = g.tmap[ax];
    // the swizzle pattern is relative to the shared address: the tile must start on it
    boxes = tmap && (smem_u32(tile) & 1023u) == 0;
  }
  // starts the tile's copy (boxes on the TMA engine: one thread, one barrier)
  __device__ __forceinline__ void load_begin() const {
    if (boxes) {
      if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // (a convolution plan's last box ends beyond psi: its rows there arrive as zeros)
        constexpr int br = BS ? kConvBoxRows : tma_box_rows(G::N);
        mbar_expect_tx(bar, (unsigned)((N + br - 1) / br * br * G::C * 16));
        for (int r0 = 0; r0 < N; r0 += br) tma_load3(tile + (size_t)r0 * G::C, tmap, (int)(2 * c0), r0, (int)o, bar);
      }
    } else {
      for (int e = threadIdx.x; e < N * G::C; e += blockDim.x) {
        const int i = e / G::C, l = e % G::C;
        tile[i * G::C + (l ^ column_swz<G::C>(i))] =
            l < Ch ? psi[obase + (long long)i * inner + l] : make_longlong2(0, 0);
      }
    }
    __syncthreads();
  }
  // waits for the copy; false: it did not arrive within the bounded polls
  __device__ __forceinline__ bool load_wait() const {
    if (!boxes) return true;
    if (mbar_wait(bar, 0)) return true;
    mbar_wait(bar, 0);
    return false;
  }
  // this thread's points of line l, after load_wait
  __device__ __forceinline__ void read(longlong2* v, const LineCtx<G>& c) const {
    const int l = c.l < G::C ? c.l : 0;
#pragma unroll
    for (int s = 0; s < G::E; ++s) {
      const int i = c.t + s * G::T;
      const int sw = column_swz<G::C>(G::T % 8 == 0 ? c.t : i);
      v[s] = !BS || i < N ? tile[i * G::C + (l ^ sw)] : make_longlong2(0, 0);
    }
    __syncthreads();  // the tile becomes the lines' exchange buffer
  }
  // the lines back into the tile and from there to psi (every thread of the block)
  __device__ __forceinline__ void write(const longlong2* v, const LineCtx<G>& c) const {
    __syncthreads();  // every line's exchanges are over
    if (c.l < G::C) {
#pragma unroll
      for (int s = 0; s < G::E; ++s) {
        const int i = c.t + s * G::T;
        const int sw = column_swz<G::C>(G::T % 8 == 0 ? c.t : i);
        tile[i * G::C + (c.l ^ sw)] = v[s];
      }
    }
    if (boxes) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (threadIdx.x == 0) {
        constexpr int br = BS ? kConvBoxRows : tma_box_rows(G::N);
        for (int r0 = 0; r0 < N; r0 += br) tma_store3(tmap, (int)(2 * c0), r0, (int)o, tile + (size_t)r0 * G::C);
        asm volatile("cp.async.bulk.commit_group;\ncp.async.bulk.wait_group 0;" ::: "memory");
      }
    } else {
      __syncthreads();
      for (int e = threadIdx.x; e < N * G::C; e += blockDim.x) {
        const int i = e / G::C, l = e % G::C;
        if (l < Ch) psi[obase + (long long)i * inner + l] = tile[i * G::C + (l ^ column_swz<G::C>(i))];
      }
    }
  }
  __device__ __forceinline__ unsigned (*slots(unsigned char* sm) const)[32] {
    return reinterpret_cast<unsigned(*)[32]>(sm + (G::kColBytes + 127) / 128 * 128);
  }
};

// 16-byte global -> shared copy of a thread's own data (cp.async), visible to the thread
// after own_wait
__device__ __forceinline__ void own_copy(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void own_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// 2^e as a double (0 below the normal range, the largest power of two above it)
__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double((i64)(e < -1022 ? 0 : e > 1023 ? 2046 : e + 1023) << 52);
}

// ------------------------------------------------------------ observables
// Norm and E_pot sums of a thread's points, exact in integers: a component u (below
// 2^59.5 in modulus) is taken as uh 2^28 + ul in units of 2^4, |u|^2 in three words, and
// V |u|^2 from the top 62 bits of |u|^2 and V in 2^vshift fixed point (|V| 2^vshift < 2^50).
struct ObsSum {
  u64 hh = 0, ll = 0;
  i64 hl = 0, a1 = 0, a2 = 0, a3 = 0, a4 = 0;
  __device__ __forceinline__ void add(longlong2 u, i64 v) {
    const int xh = (int)(u.x >> 32), yh = (int)(u.y >> 32);
    const int xl = (int)((unsigned)u.x >> 4), yl = (int)((unsigned)u.y >> 4);
    const u64 phh = (u64)((i64)xh * xh + (i64)yh * yh);
    const i64 phl = (i64)xh * xl + (i64)yh * yl;
    const u64 pll = (u64)((i64)xl * xl + (i64)yl * yl);
    hh += phh;
    hl += phl;
    ll += pll;
    const i64 n2 = (i64)(phh << 7) + ((phl + (i64)(pll >> 29)) >> 20);
    const int nl = (int)(n2 & 0x7fffffffLL), nh = (int)(n2 >> 31);
    const int vl = (int)v & 0x1ffffff, vh = (int)(v >> 25);
    a1 += (i64)nh * vh;
    a2 += (i64)nh * vl;
    a3 += (i64)nl * vh;
    a4 += (i64)nl * vl;
  }
  // the sums as one word each, in units of the largest point's 2^-59 (2^-58 for E_pot):
  // norm = norm_word 2^(60 - 2 s), E_pot = epot_word 2^(111 - vshift - 2 s) for points of
  // exponent s (value = u 2^-s)
  __device__ __forceinline__ u64 norm_word() const {
    return (hh << 4) + (u64)((hl + (i64)(ll >> 29) + (1 << 22)) >> 23);
  }
  __device__ __forceinline__ i64 epot_word() const {
    return (a1 << 2) + ((a2 + (a3 >> 6) + (a4 >> 31) + (1 << 22)) >> 23);
  }
  __device__ __forceinline__ double norm(int s) const { return pow2(60 - 2 * s) * (double)norm_word(); }
  __device__ __forceinline__ double epot(int s, int vshift) const {
    return pow2(111 - vshift - 2 * s) * (double)epot_word();
  }
};

// Length-gauge factors of half `kind` (0 open, 1 close, 2 close of this sub-step times
// open of the next): the last axis' table and the factor of the other axes at `row` of
// lines of N points.
__device__ __forceinline__ int4 lg_row(const GridDev& g, const StepDev& S, long long sub, int kind, long long row, int N) {
  const int4* t = S.xdyn + ((size_t)(sub - S.ctl[7]) * 3 + kind) * g.dim * S.nmax;
  if (g.dim == 2) return t[(int)row];
  return split_fx(fmul62(tw_join(t[(int)(row / N)]), tw_join(t[S.nmax + (int)(row % N)])));
}
__device__ __forceinline__ const int4* lg_col(const GridDev& g, const StepDev& S, long long sub, int kind) {
  return S.xdyn + (((size_t)(sub - S.ctl[7]) * 3 + kind) * g.dim + g.dim - 1) * S.nmax;
}
__device__ __forceinline__ int lg_exp(const GridDev& g, const StepDev& S, long long sub, int kind) {
  int e = 0;
  for (int d = 0; d < g.dim; ++d) e += S.texp[(int)(sub - S.ctl[7]) * kTexp + (1 + kind) * 3 + d];
  return e;
}

// ------------------------------------------------------------ convolution plans
// Lines of n points without a plan of their own (BS below) run Bluestein's convolution on
// a plan of M >= 2n - 1 points (qsf_bluestein.cu).  With c[j] = exp(-i pi j^2 / n), B the
// transform of the wrapped conj(c) over M, and
//     D(w) = FFT_M(conj(FFT_M(w) B)),
// a transform is X = c conj(D(c x)) and an inverse one x = conj(c) D(c conj(X)) / n, and
// D(a w) = conj(a) D(w) for a factor a constant along the line.  So every pass is a
// conjugation of what it loads and a D, with zeros beyond n: the chirps of the transforms
// cancel against those of the inverses at the P phase, and what is left is the factor
// C = prod_d c[j_d] of psi, which the opening half puts on (conv_row, g.chirp), which the
// middle of a run (X half . X half) carries along, and which the last step's psi and the
// flux snapshot lose again.  Bound by integer issue as the plain plans are, with four
// M-point transforms in place of two n-point ones per pass.  1000^2 points: 262 us a step,
// 780 through the member operations (pre, transform, product, transform and post kernels
// per axis, in doubles).

// C without the last axis' part
__device__ __forceinline__ double2 conv_row(const GridDev& g, long long row) {
  if (g.dim == 2) return g.chirp[row];
  const int n = g.ax[2].n;
  return cmul(g.chirp[row / n], g.chirp[row % n]);
}
// psi (double, in v) times `c`
__device__ __forceinline__ longlong2 conv_chirp(longlong2 v, double2 c) {
  const double2 z = cmul(make_double2(__longlong_as_double(v.x), __longlong_as_double(v.y)), c);
  return make_longlong2(__double_as_longlong(z.x), __double_as_longlong(z.y));
}
// the line's transform, or D of it.  taken: see line_fft, of the last transform
template <class G, bool BS, class F = NoHook>
__device__ __forceinline__ void line_pass(longlong2* v, LineCtx<G>& c, const GridDev& g, const int4* tw, int& scale,
                                          const F& taken = F()) {
  if constexpr (!BS) {
    line_fft<G>(v, c, tw, scale, taken);
  } else {
#pragma unroll 1
    for (int q = 0;; ++q) {
      line_fft<G>(v, c, tw, scale, [&](int s) {
        if (q) taken(s);
      });
      if (q) break;
      scale += line_up<G, 59>(v, c) - 2 - __ldg(g.bexp);
      const int4* b = g.bhat + c.t;
#pragma unroll
      for (int s = 0; s < G::E; ++s) v[s] = fconj(fmul_tw(v[s], __ldg(b + s * G::T)));
    }
  }
}

// the flux snapshot of psi_n for the rows of this thread's group: v holds the conjugated
// points of exponent s before the closing half; the group's lines pass through the
// exchange buffer because an entry's point lies in any of its threads (true when it was
// used)
template <class G, bool BS>
__device__ __forceinline__ bool row_snapshot(const GridDev& g, const StepDev& S, const longlong2* v, LineCtx<G>& c,
                                             longlong2* smx, long long row0, long long nrows, int s, long long sub) {
  const int N = line_len<G, BS>(g.ax[g.dim - 1]);
  constexpr int gl = G::kSync == 1 ? 1 : G::kSync == 0 ? 32 / G::T : G::L;  // lines of a group
  const int l0 = c.l / gl * gl;
  const long long r0 = row0 + l0;
  if (r0 >= nrows) return false;
  const long long r1 = min(r0 + gl, min(row0 + G::L, nrows));
  const int e0 = S.row_ptr[r0], e1 = S.row_ptr[r1];
  if (e0 == e1) return false;
  const bool lg = S.lg != 0;
  const int sy = s - 2 - S.xs_exp + S.l2m - (lg ? 2 + lg_exp(g, S, sub, 1) : 0);
  constexpr int gt = G::kSync == 1 ? G::T : G::kSync == 0 ? 32 : G::kRowThreads;
  const int ti = G::kSync == 1 ? c.t : G::kSync == 0 ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  if constexpr (G::S == 1) {  // lines of one thread each: an entry is found by its owner
    const long long r = row0 + c.l;
    if (c.l < G::L && r < nrows)
      for (int e = S.row_ptr[r]; e < S.row_ptr[r + 1]; ++e) {
        const int j = (int)(S.snap_idx[e] - r * N);
        longlong2 x = make_longlong2(0, 0);
#pragma unroll
        for (int k = 0; k < G::E; ++k)
          if (k == j) x = v[k];
        x = fmul_tw(BS ? x : fconj(x), S.xs[r * N + j]);
        if (lg) x = fmul_tw(shl_by(fmul_tw(x, lg_col(g, S, sub, 1)[j]), 2), lg_row(g, S, sub, 1, r, N));
        const double2 z = make_double2(fx2d(x.x, sy), fx2d(x.y, sy));
        S.snap[e] = BS ? cmulc(z, cmul(conv_row(g, r), g.chirp[j])) : z;
      }
    return true;
  }
  own_wait();  // nothing may still be on its way into the slots
  c.sync();
#pragma unroll
  for (int k = 0; k < G::E; ++k) c.buf[G::pad(c.t) + k * G::pad(G::T)] = v[k];
  c.sync();
  for (int e = e0 + ti; e < e1; e += gt) {
    const long long p = S.snap_idx[e], r = p / N;
    const int j = (int)(p % N);
    longlong2 x = smx[(r - row0) * G::LS + G::pad(j)];
    x = fmul_tw(BS ? x : fconj(x), S.xs[p]);
    if (lg) x = fmul_tw(shl_by(fmul_tw(x, lg_col(g, S, sub, 1)[j]), 2), lg_row(g, S, sub, 1, r, N));
    const double2 z = make_double2(fx2d(x.x, sy), fx2d(x.y, sy));
    S.snap[e] = BS ? cmulc(z, cmul(conv_row(g, r), g.chirp[j])) : z;
  }
  c.sync();
  return true;
}

// ------------------------------------------------------------ row passes
// Open: psi (double) . X half . forward transform of the last axis -> fixed point (pass 0).
template <class G, bool BS = false>
__global__ void __launch_bounds__(G::kRowThreads, G::blocks(G::kRowThreads))
    k_row_open(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss) {
  const GridDev& g = Gs[blockIdx.y];
  const StepDev& S = Ss[blockIdx.y];
  const int N = line_len<G, BS>(g.ax[g.dim - 1]);
  const long long sub = S.ctl[6];
  if (!pass_active(S, sub)) return;
  // the previous sub-step's closing pass produced pass 0, unless it ended with psi_n in
  // memory for E_kin
  if (S.fused && sub > 0 && !ekin_at(S, sub - 1)) return;
  extern __shared__ __align__(1024) unsigned char sm[];
  LineCtx<G> c(reinterpret_cast<longlong2*>(sm), reinterpret_cast<unsigned(*)[32]>(sm + G::buf_bytes(G::kRowThreads)));
  const long long nrows = g.m / N, row = (long long)blockIdx.x * G::L + c.l;
  const bool on = c.l < G::L && row < nrows;
  longlong2* psi = reinterpret_cast<longlong2*>(g.psi) + (on ? row * N : 0) + c.t;
  auto has = [&](int s) { return !BS || c.t + s * G::T < N; };  // points beyond a convolution's line are zero
  longlong2 v[G::K];
#pragma unroll
  for (int s = 0; s < G::E; ++s) v[s] = on && has(s) ? psi[s * G::T] : make_longlong2(0, 0);
  if constexpr (BS) {
    const double2 cr = conv_row(g, on ? row : 0);
#pragma unroll
    for (int s = 0; s < G::E; ++s)
      if (has(s)) v[s] = conv_chirp(v[s], cmul(cr, g.chirp[c.t + s * G::T]));
  }
  unsigned em;
  int scale = line_from_double<G>(v, c, em, kLineIn + 2);
  // an Inf or NaN component (exponent field all ones) has no fixed-point image: flag
  // the solve (QSF_ENUMERIC) instead of converting garbage
  if (em >= 0x7ff) S.ctl[4] = 1;
  const int4* xs = S.xs + (on ? row * N : 0) + c.t;
#pragma unroll
  for (int s = 0; s < G::E; ++s)
    if (has(s)) v[s] = fmul_tw(v[s], xs[s * G::T]);
  scale -= 2 + S.xs_exp;
  if (S.lg) {
    const int4* cf = lg_col(g, S, sub, 0) + c.t;
    const int4 rf = lg_row(g, S, sub, 0, on ? row : 0, N);
#pragma unroll
    for (int s = 0; s < G::E; ++s)
      if (has(s)) v[s] = fmul_tw(shl_by(fmul_tw(shl_by(v[s], 2), cf[s * G::T]), 2), rf);
    scale -= lg_exp(g, S, sub, 0);
  }
  line_pass<G, BS>(v, c, g, g.ax[g.dim - 1].twl[G::ppt >= 16], scale);
  if (!on) return;
#pragma unroll
  for (int s = 0; s < G::E; ++s)
    if (has(s)) psi[s * G::T] = v[s];
  if (c.t == 0) {
    S.sc[row] = scale;
    atomicMin(&S.gmin[gmin_slot(0, sub)], scale);
  }
}

// Close: (fixed point, from the last strided-axis pass) inverse transform of the last
// axis . X half -> psi_n: norm / E_pot partials and the flux snapshot.  At the last
// sub-step of a call (or always when not fused, or when E_kin follows) psi_n is stored as
// double; otherwise the pass goes on into the next sub-step in the same registers: its
// opening X half and forward transform, leaving pass 0 of that sub-step.  In the length
// gauge the closing half's x.E phases do not change |psi_n|, so going on they merge with
// the next opening half's into one factor per axis (kind 2).
template <class G, bool BS = false>
__global__ void __launch_bounds__(G::kRowThreads, G::blocks(G::kRowThreads))
    k_row_close(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss) {
  const GridDev& g = Gs[blockIdx.y];
  const StepDev& S = Ss[blockIdx.y];
  const int N = line_len<G, BS>(g.ax[g.dim - 1]);
  const long long sub = S.ctl[5];
  if (!pass_active(S, sub)) return;
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ double dred[32 * 2];
  longlong2* smx = reinterpret_cast<longlong2*>(sm);
  LineCtx<G> c(smx, reinterpret_cast<unsigned(*)[32]>(sm + G::buf_bytes(G::kRowThreads)));
  const long long row0 = (long long)blockIdx.x * G::L, nrows = g.m / N, row = row0 + c.l;
  const bool on = c.l < G::L && row < nrows;
  const long long base = on ? row * N : 0;
  longlong2* psi = reinterpret_cast<longlong2*>(g.psi) + base + c.t;
  const int in_pass = g.dim == 3 ? 3 : 2;
  // the potential is read in the middle of the pass: start moving it into L2 now
  for (int i = c.t * 16; i < N; i += G::T * 16) prefetch_l2(S.Vx + base + i);
  auto has = [&](int s) { return !BS || c.t + s * G::T < N; };  // points beyond a convolution's line are zero
  longlong2 v[G::K];
  int scale;
  {
    int d[G::E];
#pragma unroll
    for (int s = 0; s < G::E; ++s) v[s] = on && has(s) ? psi[s * G::T] : make_longlong2(0, 0);
    const int gm = S.gmin[gmin_slot(in_pass, sub)];
    const int* sc = S.sc + (size_t)in_pass * S.scmax + (g.dim == 3 && on ? row / N * N : 0) + c.t;
#pragma unroll
    for (int s = 0; s < G::E; ++s) d[s] = has(s) ? gm - sc[s * G::T] : 0;
    scale = line_align<G>(v, d, gm, c);
    if constexpr (BS) {
#pragma unroll
      for (int s = 0; s < G::E; ++s) v[s] = fconj(v[s]);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    S.ctl[6] = sub + 1;  // the sub-step's last pass
    for (int p = 1; p < 4; ++p) S.gmin[gmin_slot(p, sub + 1)] = 0x7fffffff;
  }
  const bool last = !S.fused || sub >= S.ctl[1] || sub + 1 >= S.nsteps || ekin_at(S, sub);
  const int4* tw = g.ax[g.dim - 1].twl[G::ppt >= 16];
  const int4* xs = S.xs + base + c.t;
  const long long* Vx = S.Vx + base + c.t;
  // the static factors of this thread's points travel into its own exchange slots while
  // the last pass of the inverse transform works on what it read from them
  int h = 0;
  auto fetch = [&](int s) {
    if (h == 0 && has(s)) own_copy(c.own(s), xs + s * G::T);
  };
#pragma unroll 1  // one code body for both transforms
  for (;; ++h) {
    line_pass<G, BS>(v, c, g, tw, scale, fetch);
    if (h) break;
    scale += line_up<G>(v, c);
    if (S.row_ptr && row_snapshot<G, BS>(g, S, v, c, smx, row0, nrows, scale, sub) && G::S > 1) {
#pragma unroll
      for (int s = 0; s < G::E; ++s) fetch(s);  // the snapshot took the slots
    }
    scale += S.l2m - 2 - S.xs_exp;
    int su = scale;  // exponent of u = f psi, |u| = |psi_n|
    own_wait();
    ObsSum ob;
    if (__builtin_expect(!last, 1)) {
#pragma unroll
      for (int s = 0; s < G::E; ++s) {
        if (!has(s)) {
          v[s] = make_longlong2(0, 0);
          continue;
        }
        int4 f;
        if constexpr (G::S > 1) f = *reinterpret_cast<const int4*>(c.own(s));
        else f = xs[s * G::T];
        const longlong2 u = fmul_tw(BS ? v[s] : fconj(v[s]), f);
        ob.add(u, __ldg(Vx + s * G::T));
        v[s] = fmul_tw(u, f);
      }
      scale -= 2 + S.xs_exp;
    } else {
#pragma unroll
      for (int s = 0; s < G::E; ++s)
        v[s] = has(s) ? fmul_tw(BS ? v[s] : fconj(v[s]), xs[s * G::T]) : make_longlong2(0, 0);
    }
    if (S.lg) {
      const int kind = last ? 1 : 2, pre = last ? 0 : 2;
      const int4* cf = lg_col(g, S, sub, kind) + c.t;
      const int4 rf = lg_row(g, S, sub, kind, on ? row : 0, N);
#pragma unroll
      for (int s = 0; s < G::E; ++s)
        if (has(s)) v[s] = fmul_tw(shl_by(fmul_tw(shl_by(v[s], pre), cf[s * G::T]), 2), rf);
      scale += pre - 2 - lg_exp(g, S, sub, kind);
    }
    if (__builtin_expect(last, 0)) {
      su = scale;  // (in imaginary time the x.E factors are real and count)
#pragma unroll
      for (int s = 0; s < G::E; ++s)
        if (has(s)) ob.add(v[s], Vx[s * G::T]);
    }
    double acc[2] = {ob.norm(su), S.obs & 2u ? ob.epot(su, S.vshift) : 0.0};
    block_sum<2>(acc, dred);
    if (threadIdx.x == 0) {
      S.partials[0 * S.pmax + blockIdx.x] = acc[0];
      S.partials[1 * S.pmax + blockIdx.x] = acc[1];
    }
    if (__builtin_expect(last, 0)) {
      if (on) {
        const double2 cr = BS ? conv_row(g, row) : make_double2(1.0, 0.0);
#pragma unroll
        for (int s = 0; s < G::E; ++s) {
          if (!has(s)) continue;
          double2 z = make_double2(fx2d(v[s].x, scale), fx2d(v[s].y, scale));
          if constexpr (BS) z = cmulc(z, cmul(cr, g.chirp[c.t + s * G::T]));
          psi[s * G::T] = make_longlong2(__double_as_longlong(z.x), __double_as_longlong(z.y));
        }
      }
      return;
    }
  }
  if (!on) return;
#pragma unroll
  for (int s = 0; s < G::E; ++s)
    if (has(s)) psi[s * G::T] = v[s];
  if (c.t == 0) {
    S.sc[row] = scale;
    atomicMin(&S.gmin[gmin_slot(0, sub + 1)], scale);
  }
}

// sum k^2 |X|^2 over this thread's points of a transformed line
template <class G, bool BS>
__device__ __forceinline__ double line_ekin(const AxisDev& a, const longlong2* v, int t, int scale) {
  double ek = 0.0;
#pragma unroll
  for (int s = 0; s < G::E; ++s) {
    if (BS && t + s * G::T >= a.n) continue;
    const double k = kpos(a, t + s * G::T);
    const double xr = fx2d(v[s].x, scale), xi = fx2d(v[s].y, scale);
    ek = fma(k * k, fma(xr, xr, xi * xi), ek);
  }
  return ek;
}

// E_kin part of the last axis: forward transform of psi_n (double, left as it is)
template <class G, bool BS = false>
__global__ void __launch_bounds__(G::kRowThreads, G::blocks(G::kRowThreads))
    k_row_ekin(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss) {
  const GridDev& g = Gs[blockIdx.y];
  const StepDev& S = Ss[blockIdx.y];
  const int N = line_len<G, BS>(g.ax[g.dim - 1]);
  if (!pass_active(S, S.ctl[5]) || !ekin_at(S, S.ctl[5])) return;
  extern __shared__ __align__(1024) unsigned char sm[];
  __shared__ double dred[32];
  LineCtx<G> c(reinterpret_cast<longlong2*>(sm), reinterpret_cast<unsigned(*)[32]>(sm + G::buf_bytes(G::kRowThreads)));
  const long long row = (long long)blockIdx.x * G::L + c.l;
  const bool on = c.l < G::L && row < g.m / N;
  const AxisDev& a = g.ax[g.dim - 1];
  const longlong2* psi = reinterpret_cast<const longlong2*>(g.psi) + (on ? row * N : 0) + c.t;
  auto has = [&](int s) { return !BS || c.t + s * G::T < N; };  // points beyond a convolution's line are zero
  longlong2 v[G::K];
#pragma unroll
  for (int s = 0; s < G::E; ++s) v[s] = on && has(s) ? psi[s * G::T] : make_longlong2(0, 0);
  if constexpr (BS) {
#pragma unroll
    for (int s = 0; s < G::E; ++s)
      if (has(s)) v[s] = conv_chirp(v[s], g.chirp[c.t + s * G::T]);
  }
  unsigned em;
  int scale = line_from_double<G>(v, c, em);
  line_pass<G, BS>(v, c, g, a.twl[G::ppt >= 16], scale);
  double ek = on ? line_ekin<G, BS>(a, v, c.t, scale) : 0.0;
  block_sum<1>(&ek, dred);
  if (threadIdx.x == 0) S.partials[(size_t)(2 + g.dim - 1) * S.pmax + blockIdx.x] = ek;
}

// ------------------------------------------------------------ strided axes
// Axis `ax` (not the last): C adjacent columns per block.  Modes:
//   0 forward (3D axis 1: pass 0 -> 1) or, with inv, inverse (pass 2 -> 3)
//   2 forward . P phase . inverse (axis 0: pass 0 (2D) or 1 (3D) -> 2)
//   3 forward of psi_n (double) + E_kin partial
template <int MODE, class G, bool BS = false>
__global__ void __launch_bounds__(G::kColThreads, G::blocks(G::kColThreads))
    k_axis(const GridDev* __restrict__ Gs, const StepDev* __restrict__ Ss, int ax, int inv) {
  const GridDev& g = Gs[blockIdx.y];
  const StepDev& S = Ss[blockIdx.y];
  const int N = line_len<G, BS>(g.ax[g.dim - 1]);
  const long long sub = MODE == 3 ? S.ctl[5] : S.ctl[6];
  if (MODE == 2 && blockIdx.x == 0 && threadIdx.x == 0) S.ctl[5] = sub;  // also when there is nothing left to do
  if (!pass_active(S, sub)) return;
  if (MODE == 3 && !ekin_at(S, sub)) return;
  extern __shared__ __align__(1024) unsigned char sm[];
  const ColBlock<G, BS> cb(g, ax, sm);
  cb.load_begin();
  LineCtx<G> c(cb.tile, cb.slots(sm));
  const bool on = c.l < cb.Ch;
  const long long col = cb.c0 + (on ? c.l : 0);
  const AxisDev& a = g.ax[ax];
  auto has = [&](int s) { return !BS || c.t + s * G::T < N; };  // points beyond a convolution's line are zero
  longlong2 v[G::K];
  if constexpr (MODE == 3) {
    __shared__ double dred[32];
    if (!cb.load_wait()) S.ctl[4] = 2;
    cb.read(v, c);
    if constexpr (BS) {
#pragma unroll
      for (int s = 0; s < G::E; ++s)
        if (has(s)) v[s] = conv_chirp(v[s], g.chirp[c.t + s * G::T]);
    }
    unsigned em;
    int scale = line_from_double<G>(v, c, em);
    line_pass<G, BS>(v, c, g, a.twl[G::ppt >= 16], scale);
    double ek = on ? line_ekin<G, BS>(a, v, c.t, scale) : 0.0;
    block_sum<1>(&ek, dred);
    if (threadIdx.x == 0) S.partials[(size_t)(2 + ax) * S.pmax + blockIdx.x] = ek;
    return;
  } else {
    const int in_pass = MODE == 2 ? (g.dim == 3 ? 1 : 0) : inv ? 2 : 0;
    const int out_pass = MODE == 2 ? 2 : inv ? 3 : 1;
    // the exponents of the producing lines along this one, and this line's own slot
    const long long i2 = g.dim == 3 ? col % N : 0;
    const long long in_at = MODE == 2 ? i2 * N : inv ? i2 * N : cb.o * N;
    const long long out_at = MODE == 2 ? (g.dim == 3 ? i2 * N + col / N : col) : inv ? cb.o * N + col : col * N + cb.o;
    int scale;
    {
      int d[G::E];
      const int gm = S.gmin[gmin_slot(in_pass, sub)];
      const int* sc = S.sc + (size_t)in_pass * S.scmax + in_at + c.t;
#pragma unroll
      for (int s = 0; s < G::E; ++s) d[s] = has(s) ? gm - sc[s * G::T] : 0;
      if (!cb.load_wait()) S.ctl[4] = 2;  // the copy did not complete in time: QSF_ETIMEDOUT
      cb.read(v, c);
      scale = line_align<G>(v, d, gm, c);
      if constexpr (BS) {
#pragma unroll
        for (int s = 0; s < G::E; ++s) v[s] = fconj(v[s]);
      }
    }
    if constexpr (MODE == 2) {
      const int at = (int)(sub - S.ctl[7]);
      if (blockIdx.x == 0 && threadIdx.x == 0) S.gmin[gmin_slot(0, sub + 1)] = 0x7fffffff;
      // per-column factor: product of the P tables of the other axes
      const int4* tab = S.ptab + (size_t)at * g.dim * S.nmax;
      longlong2 f = tw_join(tab[(size_t)(g.dim - 1) * S.nmax + (g.dim == 3 ? i2 : col)]);
      if (g.dim == 3) f = fmul62(f, tw_join(tab[S.nmax + col / N]));
      const int4 pc = split_fx(f);
      const int4* pt = tab + c.t;
      // the exponents of the P phase's two products and tables, and of the pending Normalize factor
      scale -= 4 + (S.normalize ? (int)S.scale[scale_slot(sub)] : 0);
      for (int d = 0; d < g.dim; ++d) scale -= S.texp[at * kTexp + d];
#pragma unroll 1  // one code body for both transforms
      for (int h = 0;; ++h) {
        line_pass<G, BS>(v, c, g, a.twl[G::ppt >= 16], scale);
        if (h) break;
        scale += line_up<G>(v, c);
        // (the table is the same for every line: it stays in L1, where a copy through
        // the exchange slots as in k_row_close came from L2, 315 -> 364 us at 256^3)
#pragma unroll
        for (int s = 0; s < G::E; ++s)
          v[s] = has(s) ? fconj(fmul_tw(fmul_tw(BS ? fconj(v[s]) : v[s], __ldg(pt + s * G::T)), pc)) : make_longlong2(0, 0);
      }
    } else {
      line_pass<G, BS>(v, c, g, a.twl[G::ppt >= 16], scale);
    }
    cb.write(v, c);
    if (on && c.t == 0) {
      S.sc[(size_t)out_pass * S.scmax + out_at] = scale;
      atomicMin(&S.gmin[gmin_slot(out_pass, sub)], scale);
    }
  }
}

// ------------------------------------------------------------ from and to doubles
// conjugation of a double pair (the sign bit of the imaginary part)
__device__ __forceinline__ longlong2 dconj(longlong2 x, bool on) {
  return on ? make_longlong2(x.x, x.y ^ (i64)0x8000000000000000ull) : x;
}
template <class G>
__device__ __forceinline__ void line_to_double(longlong2* v, int scale, bool conj, double post) {
#pragma unroll
  for (int s = 0; s < G::E; ++s) {
    double2 z = make_double2(fx2d(v[s].x, scale), fx2d(v[s].y, scale));
    if (post != 1.0) z = cscale(z, post);
    v[s] = dconj(make_longlong2(__double_as_longlong(z.x), __double_as_longlong(z.y)), conj);
  }
}
}  // namespace qsf
