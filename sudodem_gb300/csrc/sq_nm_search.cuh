// Pass 2 of the Hertz-Mindlin model: the Nelder-Mead searches of
// Ig2_Superquadrics_Superquadrics_SuperquadricsGeom2::go (Superquadrics_Ig2.cpp:2391-2430), started at
// the stored contactAngle with a simplex of 0.1 rad for a new geometry and 0.001 rad for an existing
// one.  Included by sqdem_engine.cu after sq_wave_search.cuh and sq_warp_search.cuh.
//
// What bounds it: FP64 instructions, whose cost does not depend on the lanes that take part, and for the
// longest searches the chain of evaluations.  In a packed lattice two thirds of the searches
// converge on their first simplex (three evaluations), a fifth takes 4-9, and 0.8% take 30 to 85, the
// same ones step after step.  So:
//   k_nm_round   one launch advances a list of searches, a pair of lanes per point (the even one
//                evaluates body A, the odd one body B); one, two or four points a search (those nmPlan
//                says it may ask for next), as many as the FP64 pipes have room for; the first launch
//                evaluates the whole first simplex
//   k_nm_warp    one search per warp (six points, five lanes each): what the rounds leave; two warps
//                (twelve points) for those that ran long at the last step, from the start and beside
//                the rounds
//   k_nm_finish  the contact ellipse, Ip2 and the law, one thread per contact
// A packed lattice of 20,000 (17,000 searches, 148,000 evaluations a step): 4.3 -> 2.1 ms a step, of 977
// 1.76 -> 0.85.  (Before: one persistent kernel, a search per lane, spare lanes evaluating planned points
// once its queue was empty.)
// The states live in the collider's merge buffer (table B), unused between collider passes.  A
// search's results do not depend on the schedule: speculative points it does not ask for are dropped.

__device__ __forceinline__ void nmLoad(const Dev& d, int i, NMState& M, unsigned& rounds) {
  const Table& B = d.B;
  const int4 c = B.cd[i];
  M.st = c.x & 7; M.touching = true;   // a search that finds the particles apart ends there
  M.ilo = (c.x >> 4) & 3; M.ihi = (c.x >> 6) & 3; M.inhi = (c.x >> 8) & 3; M.si = ((c.x >> 10) & 3) - 1;
  M.nfunc = c.y; rounds = (unsigned)c.z;
  const double4 n = B.normal[i], s = B.shear[i], g = B.nforce[i], h = B.phys[i];
  M.p[0][0] = n.x; M.p[0][1] = n.y; M.p[1][0] = n.z; M.p[1][1] = n.w;
  M.p[2][0] = s.x; M.p[2][1] = s.y; M.y[0] = s.z; M.y[1] = s.w;
  M.y[2] = g.x; M.psum[0] = g.y; M.psum[1] = g.z; M.ysave = g.w;
  M.ptry[0] = h.x; M.ptry[1] = h.y; M.q0 = h.z; M.q1 = h.w;
}
__device__ __forceinline__ void nmStore(const Dev& d, int i, const NMState& M, unsigned rounds) {
  const Table& B = d.B;
  B.cd[i] = make_int4(M.st | (M.ilo << 4) | (M.ihi << 6) | (M.inhi << 8) | ((M.si + 1) << 10), M.nfunc, (int)rounds, 0);
  B.normal[i] = make_double4(M.p[0][0], M.p[0][1], M.p[1][0], M.p[1][1]);
  B.shear[i] = make_double4(M.p[2][0], M.p[2][1], M.y[0], M.y[1]);
  B.nforce[i] = make_double4(M.y[2], M.psum[0], M.psum[1], M.ysave);
  B.phys[i] = make_double4(M.ptry[0], M.ptry[1], M.q0, M.q1);
}
// a search's result, for k_nm_finish
__device__ __forceinline__ void nmFinal(const Dev& d, int i, int e, const NMState& M, D3 P1, D3 P2) {
  const Table& B = d.B;
  B.owner[i] = e;
  B.cd[i] = make_int4(M.nfunc, M.touching ? 1 : 0, 0, 0);
  B.angle[i] = make_double2(M.r0, M.r1); B.depth[i] = M.dist;
  B.p1[i] = dd4(P1, 0); B.p2[i] = dd4(P2, 0);
}

template <bool FIRST>
__global__ void __launch_bounds__(LM_BS, 3) k_nm_round(Dev d, int round) {
  const unsigned FULL = 0xffffffffu;
  const SceneState& S = *d.S;
  const int nFront = S.lmCount;
  const int n = FIRST ? S.lmCount + S.nmShort : d.Q->nT[round];
  const int* in = (round & 1) ? d.waveT1 : d.waveT0;
  int* next = (round & 1) ? d.waveT0 : d.waveT1;
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (LM_BS / 32);
  int pts = 1;   // points per search: doubled while a warp per scheduler (half the grid's) holds them
  if (d.prm->lmSpread) while (pts < 4 && (long long)n * (4 * pts) <= 16ll * warps) pts *= 2;
  const int width = 2 * pts, per = 32 / width;
  const int g0 = lane & ~(width - 1), pt = (lane - g0) >> 1;
  unsigned long long ev64 = 0;
  unsigned roundsMax = 0;
  for (int t = blockIdx.x * (LM_BS / 32) + (threadIdx.x >> 5); t * per < n; t += warps) {
    const int idx = t * per + lane / width;
    const bool valid = idx < n;
    const int j = valid ? idx : n - 1;
    const int i = FIRST ? j : in[j];
    const int e = FIRST ? (j < nFront ? d.lmQueue[j] : d.lmQueue[d.qCap - 1 - (j - nFront)]) : d.B.owner[i];
    NMState M;
    unsigned rounds = 0;
    if (FIRST) {
      const bool isNew = !(d.A.flags[e] & F_GEOM);
      const double2 an = isNew ? make_double2(0, 0) : d.A.angle[e];
      nmStart(M, an.x, an.y, isNew ? 0.1 : 0.001);
    } else nmLoad(d, i, M, rounds);
    PairLane l;
    pairLoad(d, e, lane & 1, l, false);
    const D3 other = swapD3(l.s.pos);
    const Rot G = cRotationMat(l.isB ? other : l.s.pos, l.isB ? l.s.pos : other);
    bool done = false;
    D3 R1 = d3(0, 0, 0), R2 = d3(0, 0, 0);   // support points of the last evaluation asked for
    do {
      double2 q;
      const bool has = nmPlanned(M, pt, q) && !done;
      D3 c, P1, P2, f;
      double sep;
      pairEval(l, q.x, q.y, c, P1, P2, f, sep, &G);
      const double dist = nrm(f);
      if (!done) rounds++;
      if (valid && has && !(lane & 1)) ev64++;
      int last = lane;
      bool ends = false;
      for (;;) {   // as long as some search asks for a point that it has
        const unsigned m = __ballot_sync(FULL, has && !done && sameBits(q, M.q0, M.q1));
        if (!m) break;
        const unsigned mine = (m >> g0) & (width == 32 ? FULL : (1u << width) - 1u);
        const int src = mine ? g0 + __ffs(mine) - 1 : lane;
        const double fs = __shfl_sync(FULL, dist, src);
        const bool apart = __shfl_sync(FULL, sep, src) > 0;
        if (mine) {
          last = src;
          if (!nmConsume(M, fs, apart)) done = ends = true;
        }
      }
      const D3 L1 = d3(__shfl_sync(FULL, P1.x, last), __shfl_sync(FULL, P1.y, last), __shfl_sync(FULL, P1.z, last));
      const D3 L2 = d3(__shfl_sync(FULL, P2.x, last), __shfl_sync(FULL, P2.y, last), __shfl_sync(FULL, P2.z, last));
      if (ends) { R1 = L1; R2 = L2; }
    } while (__any_sync(FULL, !done && M.st <= NM_V2));
    const bool own = valid && lane == g0;
    if (own) {
      if (done) { nmFinal(d, i, e, M, R1, R2); roundsMax = max(roundsMax, rounds); }
      else {
        if (FIRST) d.B.owner[i] = e;
        nmStore(d, i, M, rounds);
      }
    }
    waveAppend(own && !done, i, next, &d.Q->nT[round + 1]);
    waveAppend(own && done, i, d.waveF, &d.Q->nF);
  }
  for (int o = 16; o > 0; o >>= 1) {
    ev64 += __shfl_down_sync(FULL, ev64, o);
    roundsMax = max(roundsMax, __shfl_down_sync(FULL, roundsMax, o));
  }
  if (lane == 0 && ev64) {
    atomicAdd(&d.S->err[E_EVAL64], ev64);
    atomicMax(&d.S->err[E_ROUNDS_MAX], (unsigned long long)roundsMax);
  }
}

// A point's evaluation, for both warps of a search.
struct NMSlot {
  double q0, q1, dist, sep, a[3], b[3];
};

// mode: WS_LONG, WS_MAIN, or WS_TAIL after `nRounds` launches of k_nm_round.  Blocks of W warps, one
// search at a time; W = 2 (twelve points a round) for the longest searches, which bound the stage.
template <int W>
__global__ void __launch_bounds__(32 * W, 12 / W) k_nm_warp(Dev d, int mode, int nRounds) {
  const unsigned FULL = 0xffffffffu;
  __shared__ NMSlot slots[2][WS_POINTS * W];
  __shared__ int taken;
  const SceneState& S = *d.S;
  const int lane = threadIdx.x & 31;
  const bool real = lane < WS_LANES * WS_POINTS;
  const int g0 = real ? lane / WS_LANES * WS_LANES : 0;
  const int r = real ? lane - g0 : lane - WS_LANES * WS_POINTS;
  const int grp = (threadIdx.x >> 5) * WS_POINTS + g0 / WS_LANES;
  const int nFront = S.lmCount, nMain = S.lmCount + S.nmShort;
  const int nLong1 = S.vlCount;
  const int total = mode == WS_LONG ? S.vlCount + d.Q->vl2Count : mode == WS_TAIL ? d.Q->nT[nRounds] : nMain;
  int* head = mode == WS_LONG ? &d.S->vlHead : mode == WS_TAIL ? &d.Q->tailHead : &d.S->lmHead;
  if ((int)blockIdx.x >= total) return;
  const int points = d.prm->lmSpread ? WS_POINTS * W : 1;
  unsigned long long ev64 = 0;
  unsigned roundsMax = 0;
  int flip = 0;
  auto join = [&]() { if (W == 1) __syncwarp(); else __syncthreads(); };
  for (;;) {
    if (threadIdx.x == 0) taken = atomicAdd(head, 1);
    join();
    const int idx = taken;
    join();
    if (idx >= total) break;
    int i, e;   // long searches take the slots after the main queue's
    if (mode == WS_TAIL) { i = ((nRounds & 1) ? d.waveT1 : d.waveT0)[idx]; e = d.B.owner[i]; }
    else if (mode == WS_LONG) { i = nMain + idx; e = idx < nLong1 ? d.fbQueue[idx] : d.fbQueue[d.Pcap - 1 - (idx - nLong1)]; }
    else { i = idx; e = idx < nFront ? d.lmQueue[idx] : d.lmQueue[d.qCap - 1 - (idx - nFront)]; }
    const unsigned fl = d.A.flags[e];
    int id1, id2;
    entryIds(d, e, fl, id1, id2);
    NMState M;
    unsigned rounds = 0;
    if (mode == WS_TAIL) nmLoad(d, i, M, rounds);
    else {
      const bool isNew = !(fl & F_GEOM);
      const double2 an = isNew ? make_double2(0, 0) : d.A.angle[e];
      nmStart(M, an.x, an.y, isNew ? 0.1 : 0.001);
    }
    WShape s;
    warpShape(d, r == 2 || r == 3 ? id2 : id1, s);
    const double e1B = d.shpB[id2].x;
    const Rot G = cRotationMat(xyz(d.pos[id1]), xyz(d.pos[id2]));
    bool done = false;
    while (!done) {
      double2 p;
      const bool has = grp < points && nmPlanned(M, grp, p);
      if (!has) p = make_double2(M.q0, M.q1);
      WEval v;
      warpEval(s, e1B, g0, r, p.x, p.y, v, &G);
      rounds++;
      if (has && real && r == 0) ev64++;
      flip ^= 1;
      NMSlot* q = slots[flip];
      if (real) {
        NMSlot& o = q[grp];
        if (r == 0) { o.q0 = p.x; o.q1 = p.y; o.dist = v.nrm; o.sep = v.sep; o.a[0] = v.pxy; o.a[2] = v.pz; }
        if (r == 1) o.a[1] = v.pxy;
        if (r == 2) { o.b[0] = v.pxy; o.b[2] = v.pz; }
        if (r == 3) o.b[1] = v.pxy;
      }
      join();
      const NMSlot& mine = q[lane < WS_POINTS * W ? lane : 0];
      const double2 pt = make_double2(mine.q0, mine.q1);
      unsigned m;
      int last = 0;
      while (!done && (m = __ballot_sync(FULL, lane < WS_POINTS * W && sameBits(pt, M.q0, M.q1)))) {
        last = __ffs(m) - 1;
        done = !nmConsume(M, q[last].dist, q[last].sep > 0);
      }
      if (done && threadIdx.x == 0) {
        const NMSlot& o = q[last];
        nmFinal(d, i, e, M, d3(o.a[0], o.a[1], o.a[2]), d3(o.b[0], o.b[1], o.b[2]));
        d.waveF[atomicAdd(&d.Q->nF, 1)] = i;
      }
    }
    roundsMax = max(roundsMax, rounds);
  }
  if (ev64) atomicAdd(&d.S->err[E_EVAL64], ev64);
  if (threadIdx.x == 0) atomicMax(&d.S->err[E_ROUNDS_MAX], (unsigned long long)roundsMax);
}

