// swdk_coop.cuh -- the root search with several lanes per chain, for calls
// with too few (chain, column) items to fill the GPU with one lane each.  The
// retries' single evaluations use it too (k_retry).  Included by swdk.cu.
//
// A secular evaluation is a recurrence over the layers of one column, but
// only its product e <- e * M(layer) is sequential: the entries of M (square
// roots, exponentials or sines and cosines, about 200 of the 250
// instructions of a layer) depend on the layer and the trial velocity alone.
// A group of W lanes therefore forms the entries of W layers at once, one
// per lane, leaves them in shared memory, and runs the W products from
// there.  The entries and products are the functions that the one-lane
// evaluation runs (layer_coef, dunkin_entries, dunkin_product; love_coef,
// love_product; for layered models the _ref ones), every rounding written
// out, in the same order, so the values are the same bits.
//
// What bounds it: the dependent FP64 chain.  With W = 32 and a warp or two per
// scheduler an evaluation of 161 layers takes 57 000 cycles (entries 19 000,
// products 27 000, 170 a layer) against 210 000 by one lane; a round of the
// state machine between evaluations 4000 to 8000.
#pragma once

namespace {

// One group's chain, in shared memory.  cc / cf: trial velocities evaluated
// ahead of the chain's requests and their values, valid for cw = omega; a
// request whose velocity is one of them, bit for bit, is answered from here.
struct CoopGroup {
  ChainState s;
  ChainParams P;
  ChainIO io;
  LayerView V;
  double cc[32], cf[32];
  double cw;
  int npts;    // velocities to evaluate now
  int cn, ch;  // valid entries, the one expected next
  int have, exhausted, asked, item;  // a chain is running; the queue is empty; cc[0] is the chain's request; its item
  unsigned ev[NPHASE_EV];  // evaluations by phase of the current chain
};

constexpr int COOP_ROW = 22;  // doubles per layer row: 19 entries, padded so that 16-byte stores of 8 rows hit 32 banks
constexpr size_t COOP_BUF = (size_t)32 * COOP_ROW * sizeof(double);  // one warp's rows

constexpr int COOP_MIN_G = 4;  // lanes of the smallest group
inline size_t coop_smem(int G) { return 4 * COOP_BUF + (128 / G) * sizeof(CoopGroup); }

// Every lane of the warp calls this; lanes with on = true evaluate, in
// subgroups of W lanes with the same V, wvno and omega.  l: lane in the
// subgroup; rows: the subgroup's first row.  The trip counts are the same in
// every lane so that the warp stays converged.
__device__ __forceinline__ Dunkin load_dunkin(const double* row) {
  const double2* q = reinterpret_cast<const double2*>(row);
  Dunkin d;
  double2 t;
  t = q[0]; d.c11 = t.x; d.c12 = t.y;
  t = q[1]; d.c13 = t.x; d.c14 = t.y;
  t = q[2]; d.c15 = t.x; d.c21 = t.y;
  t = q[3]; d.c22 = t.x; d.c23 = t.y;
  t = q[4]; d.c24 = t.x; d.c31 = t.y;
  t = q[5]; d.c32 = t.x; d.c33 = t.y;
  t = q[6]; d.c34 = t.x; d.c35 = t.y;
  t = q[7]; d.c41 = t.x; d.c42 = t.y;
  t = q[8]; d.c43 = t.x; d.c51 = t.y;
  d.c53 = row[18];
  return d;
}

// NORM 0: dltar4 as written (normalised at every layer by the reciprocal)
template <int NORM>
__device__ double coop_rayleigh(bool on, const LayerView& V, double wvno, double omga, int W, int l, double* rows) {
  double omega = omga;
  if (omega < 1.0e-4) omega = 1.0e-4;
  const double wvno2 = wvno * wvno;
  const double iom = 1.0 / omega;
  const int hs = on ? V.L - 1 : 0, mlo = on ? V.llw - 1 : 0;
  double e0 = 0.0, e1 = 0.0, e2 = 0.0, e3 = 0.0, e4 = 0.0;
  if (on) {
    const RayVec st = NORM == 0 ? rayleigh_start_ref(V.get(hs), wvno, wvno2, omega, iom)
                                : rayleigh_start(V.layer(hs), wvno, wvno2, omega, iom);
    e0 = st.e0; e1 = st.e1; e2 = st.e2; e3 = st.e3; e4 = st.e4;
  }
  const int n = hs - mlo;  // layers to propagate
  const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
  int since = 0;
  for (int a = 0; a < nmax; a += W) {
    const int m = hs - 1 - a - l;
    if (m >= mlo && on) {
      const LayerCoef k = NORM == 0 ? layer_coef_ref(V.get(m), wvno, wvno2, omega, iom)
                                    : layer_coef(V.layer(m), wvno, wvno2, omega, iom);
      const Dunkin d = dunkin_entries(k, wvno2);
      double2* q = reinterpret_cast<double2*>(rows + (size_t)l * COOP_ROW);
      q[0] = make_double2(d.c11, d.c12);
      q[1] = make_double2(d.c13, d.c14);
      q[2] = make_double2(d.c15, d.c21);
      q[3] = make_double2(d.c22, d.c23);
      q[4] = make_double2(d.c24, d.c31);
      q[5] = make_double2(d.c32, d.c33);
      q[6] = make_double2(d.c34, d.c35);
      q[7] = make_double2(d.c41, d.c42);
      q[8] = make_double2(d.c43, d.c51);
      q[9] = make_double2(d.c53, 0.0);
    }
    __syncwarp();
    // the normalisation falls on every NORM-th layer of the whole recurrence
    // and on its last; four layers between two of them run unrolled (the
    // loads of a layer's row then overlap the products before it)
    const int steps = min(W, n - a);  // <= 0 once this subgroup's layers are done
    int i = 0;
    if (NORM == 4 && since == 0) {
      for (; i + 4 <= steps; i += 4) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
          dunkin_product(load_dunkin(rows + (size_t)(i + r) * COOP_ROW), e0, e1, e2, e3, e4);
        rayleigh_norm<NORM>(e0, e1, e2, e3, e4);
      }
    }
#pragma unroll 1
    for (; i < steps; ++i) {
      dunkin_product(load_dunkin(rows + (size_t)i * COOP_ROW), e0, e1, e2, e3, e4);
      if (++since >= NORM || a + i == n - 1) {
        since = 0;
        rayleigh_norm<NORM == 0 ? 4 : NORM>(e0, e1, e2, e3, e4);
      }
    }
    __syncwarp();
  }
  if (on && V.llw != 1) {
    if (NORM == 0) return rayleigh_fluid_top_ref(V.get(0), wvno, omega, e0, e1);
    return rayleigh_fluid_top(V.layer(0), wvno, omega, e0, e1);
  }
  return e0;
}

template <int NORM>
__device__ double coop_love(bool on, const LayerView& V, double wvno, double omega, int W, int l, double* rows) {
  const int hs = on ? V.L - 1 : 0, mlo = on ? V.llw - 1 : 0;
  double e1 = 0.0, e2 = 0.0;
  if (on && NORM == 0) {
    love_start_ref(V.get(hs), wvno, omega, e1, e2);
  } else if (on) {
    love_start(V.layer(hs), wvno, omega, e1, e2);
  }
  const int n = hs - mlo;
  const int nmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)n);
  int since = 0;
  for (int a = 0; a < nmax; a += W) {
    const int m = hs - 1 - a - l;
    if (m >= mlo && on) {
      const LoveCoef k = NORM == 0 ? love_coef_ref(V.get(m), wvno, omega) : love_coef(V.layer(m), wvno, omega);
      double2* q = reinterpret_cast<double2*>(rows + (size_t)l * COOP_ROW);
      q[0] = make_double2(k.cosq, k.y);
      q[1] = make_double2(k.z, k.xmu);
      q[2] = make_double2(k.ixmu, 0.0);
    }
    __syncwarp();
    const int steps = min(W, n - a);
#pragma unroll 2
    for (int i = 0; i < steps; ++i) {
      const double2* q = reinterpret_cast<const double2*>(rows + (size_t)i * COOP_ROW);
      LoveCoef k;
      double2 t;
      t = q[0]; k.cosq = t.x; k.y = t.y;
      t = q[1]; k.z = t.x; k.xmu = t.y;
      t = q[2]; k.ixmu = t.x;
      const bool norm = ++since >= NORM || a + i == n - 1;
      if (norm) since = 0;
      love_product<NORM>(k, norm, e1, e2);
    }
    __syncwarp();
  }
  return e1;
}

// Brent's steps below this (km/s) are taken for the last interpolation of a
// root.  A second velocity costs a group the layers' entries once more, half of
// a round's products and control if it is the next request.  ms of the search
// without / 1e-6 / 1e-5 / 1e-4 / 1e-3: 1188 chains of 161 layers 4.20 / 4.13 /
// 4.04 / 4.03 / 4.05, 3564 chains 9.90 / 9.68 / 9.55 / 9.63 / 9.75.  (Both sides
// of the root, four velocities: 4.15 and 9.97.)
constexpr double BRENT_NEAR = 1e-5;

// Trial velocities worth evaluating together with the chain's request
// (s.creq, s.next), in cc[0..n): the request itself, then the ones that the
// search asks for next unless a sign change ends its walk before.  G: lanes
// of the group; n is a power of two and at most G.  Only the values' reuse depends on this guess, never a root.
__device__ int coop_plan(ChainState& s, const ChainParams& P, const ChainIO& io, int G, double* cc) {
  cc[0] = s.creq;
  int n = 1;
  switch (s.next) {
    case PH_SCAN_GOT: {  // the scan's next points; the first period's scan is the long one
      const double step = s.idir > 0 ? DC : -DC;
      n = s.k == 1 ? G : G / 4;
      for (int i = 1; i < n; ++i) cc[i] = cc[i - 1] + step;
      break;
    }
    case PH_GS_FIRST: {  // c1 and the upward scan (or the checked jump) from it
      const double d1 = s.del1st;
      int m;
      s.del1st = 1.0;  // known only with f(c1)
      const bool jump = s.pj == -1 && first_cell(s, P, io, m);
      s.del1st = d1;
      if (jump) {
        n = min(G, 1 + m / FIRST_STRIDE);
        int g = 1;
        while (g < n) g <<= 1;
        n = g;
        for (int i = 1; i < n; ++i) {
          double c = cc[i - 1];
          for (int j = 0; j < FIRST_STRIDE; ++j) c = c + DC;
          cc[i] = c;
        }
        break;
      }
      n = s.k == 1 ? G : G / 4;
      for (int i = 1; i < n; ++i) cc[i] = cc[i - 1] + DC;
      break;
    }
    case PH_FIRST_GOT: {  // coarse points up to the learned cell
      int left = 1 + (s.pm - s.pj) / FIRST_STRIDE;
      n = 1;
      while (n < left && n < G) n <<= 1;
      for (int i = 1; i < n; ++i) {
        double c = cc[i - 1];
        for (int j = 0; j < FIRST_STRIDE; ++j) c = c + DC;
        cc[i] = c;
      }
      break;
    }
    case PH_PROP_HI: {  // the learned cell's two ends
      if (G >= 16) {
        n = 2;
        cc[1] = s.phi;
      }
      break;
    }
    case PH_BRENT_GOT: {
      // an interpolation that lands within the tolerance of the root is
      // followed by a step of the tolerance; half of them go back to the side
      // it came from
      const double eps = 2.220446049250313e-16, c = s.creq;
      const double tol1 = 2.0 * eps * fabs(c) + 0.5 * P.rtol * fabs(c);
      if (G >= 16 && fabs(s.rd) > tol1 && fabs(s.rd) < BRENT_NEAR) {
        n = 2;
        cc[1] = c + copysign(tol1, s.ra_ - c);
      }
      break;
    }
    default: break;
  }
  return n;
}

// What every group of a launch shares.
struct CoopArgs {
  int ncol, nitems, G;
  const int* order;
  const ChainDesc* chains;
  const double* periods;
  const float4 *layR, *layL;
  const ColInfo* info;
  int refine;
  double rtol;
  int sngl, retry;
  double* croot;
  int32_t* cstat;
  unsigned int* queue;
  const float2* prop;
  int2* retry_list;
  unsigned int* retry_count;
  unsigned int retry_cap;
  unsigned long long* nevals;
  RaggedMap rg;
  const float4* nodes;
  const DepthLayer* dl;
  int32_t* ierr_out;  // REF: the chains' ierr
  const unsigned long long* gate;  // if given, the launch is for calls where (*gate != 0) == gate_on
  int gate_on;
};

// The group's first lane: gives the chain its value, runs its state machine
// through all that needs no new evaluation (taking the next item when the
// chain ends) and plans the next evaluations.  Returns their number, 0 when
// there is no work left.  Not inlined.
template <bool REF>
__device__ __noinline__ int coop_step(CoopGroup& g, const CoopArgs& A, unsigned long long* phase_ev,
                                      unsigned long long* blk_ev) {
  ChainState& s = g.s;
  ChainParams& P = g.P;
  ChainIO& io = g.io;
  // the chain takes its value
  auto answer = [&](int i) {
    g.ev[eval_phase(s)] += 1u;
    s.last = g.cf[i];
    s.nevals++;
    s.phase = s.next;
    g.ch = i + 1 < g.cn ? i + 1 : 0;
  };
  if (g.asked) answer(0);
  g.asked = 0;
  for (;;) {
    if (!g.have) {
      if (g.exhausted) return 0;
      const unsigned int r = atomicAdd(A.queue, 1u);
      if (r >= (unsigned int)A.nitems) { g.exhausted = 1; return 0; }
      const int item_of = (int)r;
      g.item = item_of;
      int mcol = A.ncol, lstride = A.rg.lstride, col;
      ChainDesc cd;
      long long o_col = 0, o_lay = 0, o_root = 0, o_node = 0, o_dl = 0;
      if (A.rg.blocks) {
        const RBlock B = A.rg.blocks[ragged_find(A.rg.blocks, A.rg.nblocks, (long long)item_of, &RBlock::item0)];
        const RModel& M = A.rg.models[B.model];
        cd = A.chains[B.chain];
        col = (int)((long long)item_of - B.item0);
        mcol = M.ncol;
        lstride = M.Lmax;
        o_col = M.col0; o_lay = M.lay0; o_root = M.root0; o_node = M.node0; o_dl = M.dl0;
      } else {
        cd = A.chains[REF ? 0 : A.order[item_of / A.ncol]];
        col = item_of % A.ncol;
      }
      const ColInfo ci = A.info[o_col + col];
      double* outp = A.croot + o_root + (size_t)cd.out_off * mcol + col;
      int32_t* stp = A.cstat + o_root + (size_t)cd.out_off * mcol + col;
      if (!ci.valid) {
        for (int i = 0; i < cd.nmode * cd.np; ++i) {
          outp[(size_t)i * mcol] = 0.0;
          stp[(size_t)i * mcol] = ST_NAN_INPUT;
        }
        if (REF) A.ierr_out[col] = 1;
        continue;
      }
      LayerView& V = g.V;
      V.lay = ((cd.iwave == 2) ? A.layR : A.layL) + o_lay;
      V.fast = REF ? 0 : 1;
      V.ncol = mcol;
      V.col = col;
      V.lstride = lstride;
      V.L = ci.L;
      V.llw = ci.llw;
      V.nodes = (A.nodes && ci.nw == 0) ? A.nodes + o_node + (size_t)col * ((lstride + 3) / 4) : nullptr;
      V.dl = A.dl + o_dl;
      V.wave = cd.iwave;
      P.t = A.periods + cd.t_off;
      P.kmax = cd.np;
      P.nmode = cd.nmode;
      P.igr = cd.igr;
      P.iwave = cd.iwave;
      P.refine = A.refine;
      P.rtol = A.rtol;
      P.sngl = A.sngl;
      P.cc = ci.cc;
      P.betmx = ci.betmx;
      P.retry = A.retry;
      io.out = outp;
      io.st = stp;
      io.stride = cd.np * mcol;
      io.ostride = mcol;
      io.prop = A.prop ? A.prop + o_root + (size_t)cd.out_off * mcol + col : nullptr;
      chain_init(s);
      g.cn = 0;
      for (int i = 0; i < NPHASE_EV; ++i) g.ev[i] = 0u;
      g.have = 1;
    }
    if (!chain_advance(s, P, io)) {  // chain finished
      if (REF) A.ierr_out[g.V.col] = s.ierr;
      if (s.iterlim)
        for (int i = 0; i < P.nmode * P.kmax; ++i)
          if (io.st[(size_t)i * io.ostride] == ST_OK) io.st[(size_t)i * io.ostride] = ST_ITER_LIMIT;
      if (A.retry == RETRY_DEFERRED && s.ierr != 0) {  // failed slots: single-period work items for k_retry
        for (int m = 1; m <= P.nmode; ++m)
          for (int k = 1; k <= P.kmax; ++k) {
            const double v = out_at(io, m, k);
            if (v == 0.0 || !(v == v)) {
              const unsigned int q = atomicAdd(A.retry_count, 1u);
              if (q < A.retry_cap) A.retry_list[q] = make_int2(g.item, (m << 16) | k);
            }
          }
      }
      for (int i = 0; i < NPHASE_EV; ++i)
        if (g.ev[i]) atomicAdd(&phase_ev[i], (unsigned long long)g.ev[i]);
      atomicAdd(&blk_ev[0], (unsigned long long)s.nevals);
      atomicAdd(&blk_ev[P.iwave == 2 ? 1 : 2], (unsigned long long)s.nevals * g.V.L);
      if (s.nprop_ok) atomicAdd(&blk_ev[3], (unsigned long long)s.nprop_ok);
      if (s.nprop_fail) atomicAdd(&blk_ev[4], (unsigned long long)s.nprop_fail);
      g.have = 0;
      continue;
    }
    // a value evaluated ahead?
    int hit = -1;
    if (g.cw == s.omega) {
      const int cn = g.cn, ch = g.ch;
      for (int t = 0; t < cn && hit < 0; ++t) {
        const int i = ch + t < cn ? ch + t : ch + t - cn;
        if (g.cc[i] == s.creq) hit = i;
      }
    }
    if (hit < 0) {
      g.cn = coop_plan(s, P, io, A.G, g.cc);
      g.cw = s.omega;
      g.asked = 1;
      return g.cn;
    }
    answer(hit);
  }
}

// k_roots_coop: G lanes (4, 8, 16 or 32) per work item of k_roots_queue; an
// evaluation takes all of the group's lanes, for one trial velocity or for
// several planned together (W = G / number lanes each).  NORM 4 and 1: the
// tight and the reference refinement's secular functions; 0: layered models,
// one chain each, the functions as dltar1 / dltar4 write them.
template <int NORM>
__global__ void __launch_bounds__(128, 3) k_roots_coop(const __grid_constant__ CoopArgs A) {
  const unsigned FULL = 0xffffffffu;
  if (A.gate && (*A.gate != 0ull) != (A.gate_on != 0)) return;
  extern __shared__ __align__(16) unsigned char coop_sm[];
  __shared__ unsigned long long phase_ev[NPHASE_EV];
  __shared__ unsigned long long blk_ev[5];
  if (threadIdx.x < NPHASE_EV) phase_ev[threadIdx.x] = 0ull;
  if (threadIdx.x < 5) blk_ev[threadIdx.x] = 0ull;
  __syncthreads();
  const int G = A.G, lane = threadIdx.x & 31, gl = lane & (G - 1);
  double* wbuf = reinterpret_cast<double*>(coop_sm + (threadIdx.x >> 5) * COOP_BUF);
  CoopGroup& g = reinterpret_cast<CoopGroup*>(coop_sm + 4 * COOP_BUF)[threadIdx.x / G];
  double cbuf[KMAX_CHAIN];
  double cbbuf[KMAX_CHAIN + 24];
  if (gl == 0) {
    g.cn = 0;
    g.have = g.exhausted = g.asked = 0;
    g.io.c = cbuf;
    g.io.cb = cbbuf;
  }
  for (;;) {
    // the number goes through shared memory: with it in a register the
    // compiler left the first lane apart from the others, and the evaluation
    // ran twice (16 active lanes an instruction instead of 30)
    if (gl == 0) {
      const int np = coop_step<NORM == 0>(g, A, phase_ev, blk_ev);
      g.npts = np;
    }
    __syncwarp();
    const int npts = g.npts;
    unsigned todo = __ballot_sync(FULL, npts > 0);
    if (todo == 0u) break;
    // the groups that evaluate the same number of velocities together
    while (todo) {
      const int n = __shfl_sync(FULL, npts, __ffs(todo) - 1);
      const bool mine = npts == n;
      todo &= ~__ballot_sync(FULL, mine);
      const int W = G / n;            // lanes per velocity
      const int j = gl / W, l = gl & (W - 1);
      const double om = mine ? g.s.omega : 1.0;
      const double wv = mine ? om / g.cc[j] : 1.0;
      const bool ray = mine && g.P.iwave == 2, lov = mine && g.P.iwave != 2;
      double f = 0.0;
      if (W == 1) {  // a velocity per lane: nothing to share
        const LayerView V = g.V;
        if (mine)
          f = NORM == 0 ? secular(V, g.P.iwave, wv, om) : secular_fast(V, g.P.iwave, NORM == 1 ? 0 : 1, wv, om);
      } else {
        double* rows = wbuf + (size_t)(lane - l) * COOP_ROW;
        if (__ballot_sync(FULL, ray)) {
          const double v = coop_rayleigh<NORM>(ray, g.V, wv, om, W, l, rows);
          if (ray) f = v;
        }
        if (__ballot_sync(FULL, lov)) {
          const double v = coop_love<NORM>(lov, g.V, wv, om, W, l, rows);
          if (lov) f = v;
        }
      }
      if (mine && l == 0) g.cf[j] = f;
      __syncwarp();
    }
  }
  __syncthreads();
  if (threadIdx.x < NPHASE_EV && A.nevals && phase_ev[threadIdx.x])
    atomicAdd(A.nevals + EV_BASE + threadIdx.x, phase_ev[threadIdx.x]);
  if (threadIdx.x < 5 && A.nevals && blk_ev[threadIdx.x]) atomicAdd(A.nevals + threadIdx.x, blk_ev[threadIdx.x]);
}

}  // namespace
