// The main queue's searches of the FP64 form in rounds over compact lists.
// Included by sqdem_engine.cu after sq_warp_search.cuh.
//
// What bounds it: the FP64 pipe, whose instruction costs the same whether 1 or 32 lanes take part.  In a
// dense cell a third of the searches end at their first evaluation, another third after one
// iteration (trial and two probes), 3% after more than seven: lanes that run a whole search each
// stand at different places of it, so that every round of a warp pays for the start, the
// Jacobian, the trial's tests and the contact law of a few lanes each (a third of the pipe's time), and
// the warps end unevenly.  Here a launch does one thing for a list of searches, 16 per warp:
//   k_wave_trial   the evaluation at the start point or the pending trial and what follows from it:
//                  the search ends, its probes are wanted (list P), or a rejected trial's successor
//                  is (next list T)
//   k_wave_probe   two probes, Jacobian, damped step: the pending trial (next list T)
// so that all lanes of a warp do the same FP64 work.  A pair of lanes shares a search: the even one
// evaluates body A, the odd one body B, and each holds only its own body's shape.  The states
// live in the collider's merge buffer (table B), unused between collider passes.  After a number of
// rounds (waveRounds) the few searches left are finished one per warp (k_search_warp), as are, from
// the start and beside these launches, those that ran long at the last step.  The rounds run at the
// FP64 evaluation peak (200,000 particles: 2.6M evaluations in 9.7 ms; 0.27 G/s alone in a loop).
// Search time of a jammed cell of 200,000: 24.4 -> 18 ms, of 43,011: 11.4 -> 5.8.  Values, decisions
// and results per search are those of k_search_warp, bit for bit.

// flag word of a slot: phase in bits 0-2, these, calls from bit 8, maxit from 12, rounds so far from 16
static const unsigned WF_FROMCENTER = 8u, WF_NEW = 16u, WF_STOPFLAG = 32u, WF_INIT = 64u;

// A search's state between launches, slot i of table B.
struct WaveState {
  double p0, p1, mu, D0, D1, pfL2, diag0, diag1, j01, jt0, jt1;
  D3 pf, contact;
  int e, k, nu;
  unsigned phase, calls, iters, maxit, rounds;   // rounds: evaluations one after another, for the report
  bool fromCenter, isNew, stopFlag, init;
};
__device__ __forceinline__ void waveLoad(const Dev& d, int i, WaveState& w) {
  const Table& B = d.B;
  w.e = B.owner[i];
  const int4 c = B.cd[i];
  const unsigned f = (unsigned)c.z;
  w.k = c.x; w.nu = c.y; w.iters = (unsigned)c.w;
  w.phase = f & 7u; w.fromCenter = f & WF_FROMCENTER; w.isNew = f & WF_NEW; w.stopFlag = f & WF_STOPFLAG; w.init = f & WF_INIT;
  w.calls = (f >> 8) & 15u; w.maxit = (f >> 12) & 15u; w.rounds = f >> 16;
  const double2 p = B.angle[i];
  const double4 n = B.normal[i], s = B.shear[i], g = B.nforce[i], h = B.phys[i];
  w.p0 = p.x; w.p1 = p.y;
  w.pf = xyz(n); w.pfL2 = n.w;
  w.jt0 = s.x; w.jt1 = s.y; w.j01 = s.z; w.mu = s.w;
  w.diag0 = g.x; w.diag1 = g.y; w.D0 = g.z; w.D1 = g.w;
  w.contact = xyz(h);
}
__device__ __forceinline__ void waveStore(const Dev& d, int i, const WaveState& w) {
  const Table& B = d.B;
  const unsigned f = w.phase | (w.fromCenter ? WF_FROMCENTER : 0u) | (w.isNew ? WF_NEW : 0u) | (w.stopFlag ? WF_STOPFLAG : 0u) |
                     (w.init ? WF_INIT : 0u) | (w.calls << 8) | (w.maxit << 12) | (w.rounds << 16);
  B.owner[i] = w.e;
  B.cd[i] = make_int4(w.k, w.nu, (int)f, (int)w.iters);
  B.angle[i] = make_double2(w.p0, w.p1);
  B.normal[i] = dd4(w.pf, w.pfL2);
  B.shear[i] = make_double4(w.jt0, w.jt1, w.j01, w.mu);
  B.nforce[i] = make_double4(w.diag0, w.diag1, w.D0, w.D1);
  B.phys[i] = dd4(w.contact, 0);
}
// a search's contact, for k_wave_finish
__device__ __forceinline__ void waveFinal(const Dev& d, int i, const WaveState& w, bool touching, D3 P1, D3 P2) {
  const Table& B = d.B;
  B.owner[i] = w.e;
  B.cd[i] = make_int4((int)w.calls, (int)w.iters, (int)w.maxit, (int)(w.rounds << 1) | (touching ? 1 : 0));
  B.angle[i] = make_double2(w.p0, w.p1);
  B.phys[i] = dd4(w.contact, 0);
  B.p1[i] = dd4(P1, 0); B.p2[i] = dd4(P2, 0);
}

// Own body's shape of a pair of lanes, and what the pair shares.
struct PairLane {
  SqShape s;
  bool isB;
};
// shift: body B's nearest image (the Hertz-Mindlin search takes the positions as they are)
__device__ __forceinline__ void pairLoad(const Dev& d, int e, bool isB, PairLane& l, bool shift = true) {
  const unsigned fl = d.A.flags[e];
  int id1, id2;
  entryIds(d, e, fl, id1, id2);
  const int b = isB ? id2 : id1;
  const double4 a = d.shpA[b], x = d.shpB[b], q = d.ori[b];
  shapeInit(l.s, a.x, a.y, a.z, x.x, x.y, a.w);
  l.s.R = quatToRot(q.x, q.y, q.z, q.w);
  l.s.pos = xyz(d.pos[b]);
  if (isB && shift) l.s.pos = l.s.pos + cellShift(*d.S, d.A.cd[e]);
  l.isB = isB;
}
__device__ __forceinline__ D3 swapD3(D3 a) {
  const unsigned FULL = 0xffffffffu;
  return d3(__shfl_xor_sync(FULL, a.x, 1), __shfl_xor_sync(FULL, a.y, 1), __shfl_xor_sync(FULL, a.z, 1));
}
// Disfunction at (q0, q1), in the frame G if given (Disfun): support points, their difference and
// c . (p2 - p1)
__device__ __forceinline__ void pairEval(const PairLane& l, double q0, double q1, D3& c, D3& P1, D3& P2, D3& f, double& sep,
                                         const Rot* G = nullptr) {
  const unsigned FULL = 0xffffffffu;
  double sv, cv;
  sincos(l.isB ? q1 : q0, &sv, &cv);
  const double so = __shfl_xor_sync(FULL, sv, 1), co = __shfl_xor_sync(FULL, cv, 1);
  const double sa0 = l.isB ? so : sv, ca0 = l.isB ? co : cv, sa1 = l.isB ? sv : so, ca1 = l.isB ? cv : co;
  c = d3(ca0 * ca1, sa0 * ca1, sa1);
  if (G) c = mulG(*G, c);
  D3 n = mulL(l.s.R, c);
  if (l.isB) n = -n;
  const D3 own = mulG(l.s.R, supportLocal(l.s, n)) + l.s.pos;
  const D3 oth = swapD3(own);
  P1 = l.isB ? oth : own;
  P2 = l.isB ? own : oth;
  f = P2 - P1;
  sep = dot(c, f);
}

// top of lmder2's loop at an accepted point (lmOuter); true while the call goes on
__device__ __forceinline__ bool waveOuter(WaveState& w, int& stop, bool& touching, D3 c, double sep) {
  if (!(w.k < 50 && !stop)) { if (w.k >= 50) stop = 3; return false; }
  if (w.pfL2 <= 1e-20) { stop = 6; return false; }
  if (w.stopFlag) { stop = 9; touching = false; return false; }
  w.contact = c;
  if (angleTest(sep, w.pfL2, c)) { stop = 8; return false; }
  return true;
}
// the damped step for w.mu (lmInner): each lane of the pair one component; false when the call ends
__device__ __forceinline__ bool waveSolve(WaveState& w, int& stop, bool odd) {
  const double bo = (odd ? w.diag0 : w.diag1) + w.mu, bx = (odd ? w.diag1 : w.diag0) + w.mu;
  const double n_a = bo * bx - w.j01 * w.j01;
  const double D = ((odd ? w.jt1 : w.jt0) * bo - (odd ? w.jt0 : w.jt1) * w.j01) / n_a;
  const double Do = __shfl_xor_sync(0xffffffffu, D, 1);
  w.D0 = odd ? Do : D; w.D1 = odd ? D : Do;
  const double DL2 = sqrt(w.D0 * w.D0 + w.D1 * w.D1);
  if (DL2 < 1e-5) { stop = 2; w.k++; if (w.k >= 50) stop = 3; return false; }
  if (!(DL2 < 1e20) && DL2 >= (sqrt(w.p0 * w.p0 + w.p1 * w.p1) + 1e-3) / (1e-12 * 1e-12)) {
    stop = 4; w.k++;
    if (w.k >= 50) stop = 3;
    return false;
  }
  return true;
}
// End of an lmder2 call: the restart rules of Superquadrics_Ig2.cpp:2013-2053 (as lmCallEnd).
// True when a call from the centre line follows.  Called by all lanes of the warp (`ended`: this
// pair's call ended); the isInside tests run only in warps where a pair needs them.
__device__ __forceinline__ bool waveCallEnd(WaveState& w, const PairLane& l, int stop, bool touching, D3 P1, D3 P2, bool ended) {
  const unsigned FULL = 0xffffffffu;
  const double rmaxA = __shfl_sync(FULL, l.s.rmax, threadIdx.x & 30);
  const bool far = ended && touching && 10.0 * nrm(P2 - P1) > rmaxA;
  bool inside = true;
  if (__any_sync(FULL, far)) {
    const D3 p = (l.isB ? P1 : P2) - l.s.pos;
    const int fast = insideFast(l.s, p);
    bool mine = fast == 1;
    if (__any_sync(FULL, far && fast < 0)) mine = fast < 0 ? isInside(l.s, p) : mine;
    const bool other = __shfl_xor_sync(FULL, (int)mine, 1) != 0;
    inside = mine && other;
  }
  bool restart = false;
  if (ended)
    for (;;) {
      w.calls++; w.iters += w.k; w.maxit += (stop == 3);
      restart = false;
      if (w.phase == 0) {
        w.phase = 1;
        if ((isnan(w.p0) || isnan(w.p1) || 7 == stop) && touching) restart = true;
      }
      if (!restart) {
        if (w.phase == 1) {
          w.phase = 3;
          if (far && !inside) { w.phase = 2; restart = true; }
        } else w.phase = 3;
      }
      if (!restart || !w.fromCenter) break;
      // a restart from the centre line the call itself started from: the same outcome, counted
    }
  const D3 mine = l.s.pos, other = swapD3(mine);
  if (restart) {
    double para[2];
    centerLine(l.isB ? other : mine, l.isB ? mine : other, para);
    w.p0 = para[0]; w.p1 = para[1];
    w.fromCenter = true; w.stopFlag = false; w.init = true;
  }
  return restart;
}
// warp-aggregated append of `i` by the even lanes where `want` holds
__device__ __forceinline__ void waveAppend(bool want, int i, int* list, int* count) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __ballot_sync(0xffffffffu, want && !(lane & 1));
  if (!m) return;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(count, __popc(m));
  base = __shfl_sync(0xffffffffu, base, leader);
  if ((m >> lane) & 1u) list[base + __popc(m & ((1u << lane) - 1))] = i;
}

template <bool FIRST>
__global__ void __launch_bounds__(LM_BS, 3) k_wave_trial(Dev d, int round, int few) {
  const SceneState& S = *d.S;
  const int nFront = S.lmCount;
  const int n = FIRST ? S.lmCount + S.nmShort : d.Q->nT[round];
  if (FIRST && n <= few) return;   // k_search_warp takes them all
  const int* in = (round & 1) ? d.waveT1 : d.waveT0;
  int* next = (round & 1) ? d.waveT0 : d.waveT1;
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (LM_BS / 32);
  unsigned long long ev64 = 0;
  for (int t = blockIdx.x * (LM_BS / 32) + (threadIdx.x >> 5); t * 16 < n; t += warps) {
    const int idx = t * 16 + (lane >> 1);
    const bool valid = idx < n;
    const int j = valid ? idx : n - 1;
    const int i = FIRST ? j : in[j];
    WaveState w;
    PairLane l;
    if (FIRST) {
      w.e = j < nFront ? d.lmQueue[j] : d.lmQueue[d.qCap - 1 - (j - nFront)];
      w.isNew = !(d.A.flags[w.e] & F_GEOM);
      w.fromCenter = w.isNew; w.init = true; w.stopFlag = false;
      w.phase = 0; w.calls = 0; w.iters = 0; w.maxit = 0; w.rounds = 0;
      w.jt0 = w.jt1 = w.j01 = w.diag0 = w.diag1 = 0;
      w.contact = d3(0, 0, 0);
    } else waveLoad(d, i, w);
    pairLoad(d, w.e, lane & 1, l);
    if (FIRST) {
      const D3 other = swapD3(l.s.pos);
      if (w.isNew) {
        double para[2];
        centerLine(l.isB ? other : l.s.pos, l.isB ? l.s.pos : other, para);
        w.p0 = para[0]; w.p1 = para[1];
      } else { const double2 an = d.A.angle[w.e]; w.p0 = an.x; w.p1 = an.y; }
    }
    const bool init = FIRST || w.init;
    const double q0 = init ? w.p0 : w.p0 + w.D0, q1 = init ? w.p1 : w.p1 + w.D1;
    D3 c, P1, P2, f;
    double sep;
    pairEval(l, q0, q1, c, P1, P2, f, sep);
    if (valid && !(lane & 1)) ev64++;
    w.rounds++;
    const double fl2 = nrm(f);
    if (sep > 0) w.stopFlag = true;
    int stop = 0;
    bool touching = true, more = false, rejected = false;
    if (init) {
      w.pf = f; w.pfL2 = fl2;
      stop = isfinite(fl2) ? 0 : 7;
      w.k = 0; w.mu = 0; w.nu = 2; w.D0 = 1e-7; w.D1 = 1e-7;
      w.init = false;
      more = waveOuter(w, stop, touching, c, sep);
    }
    if (!FIRST) {
      const double dm0 = w.D0 * (w.mu * w.D0 + w.jt0), dm1 = w.D1 * (w.mu * w.D1 + w.jt1);
      const double dL = dm0 + dm1, dF = w.pfL2 - fl2;
      double tmp = dF / dL;
      if (!init) {
        if (!isfinite(fl2)) { stop = 7; w.k++; if (w.k >= 50) stop = 3; }
        else if (tmp > 0.0) {
          tmp = 1.0 - cube(2 * tmp - 1.);
          w.mu = w.mu * ((tmp >= 0.3333333333333334) ? tmp : 0.3333333333333334);
          w.nu = 2;
          w.p0 = q0; w.p1 = q1;
          w.pf = f; w.pfL2 = fl2;
          w.k++;
          more = waveOuter(w, stop, touching, c, sep);
        } else {
          w.mu *= w.nu;
          const int nu2 = (int)((unsigned)w.nu << 1);
          if (nu2 <= w.nu) { stop = 5; w.k++; if (w.k >= 50) stop = 3; }
          else { w.nu = nu2; rejected = true; }
        }
      }
      if (__any_sync(0xffffffffu, rejected)) {
        WaveState x = w;
        int st = 0;
        const bool go = waveSolve(x, st, lane & 1);
        if (rejected) { w = x; if (!go) { stop = st; rejected = false; } }
      }
    }
    const bool ended = !more && !rejected;
    const bool restart = waveCallEnd(w, l, stop, touching, P1, P2, ended);
    if (valid && !(lane & 1)) {
      if (ended && !restart) waveFinal(d, i, w, touching, P1, P2);
      else waveStore(d, i, w);
    }
    waveAppend(valid && more, i, d.waveP, &d.Q->nP[round]);
    waveAppend(valid && (rejected || restart), i, next, &d.Q->nT[round + 1]);
    waveAppend(valid && ended && !restart, i, d.waveF, &d.Q->nF);
  }
  for (int o = 16; o > 0; o >>= 1) ev64 += __shfl_down_sync(0xffffffffu, ev64, o);
  if (lane == 0 && ev64) atomicAdd(&d.S->err[E_EVAL64], ev64);
}

__global__ void __launch_bounds__(LM_BS, 3) k_wave_probe(Dev d, int round) {
  const unsigned FULL = 0xffffffffu;
  const int n = d.Q->nP[round];
  int* next = (round & 1) ? d.waveT0 : d.waveT1;
  const int lane = threadIdx.x & 31;
  const bool odd = lane & 1;
  const int warps = gridDim.x * (LM_BS / 32);
  unsigned long long ev64 = 0;
  for (int t = blockIdx.x * (LM_BS / 32) + (threadIdx.x >> 5); t * 16 < n; t += warps) {
    const int idx = t * 16 + (lane >> 1);
    const bool valid = idx < n;
    const int i = d.waveP[valid ? idx : n - 1];
    WaveState w;
    PairLane l;
    waveLoad(d, i, w);
    pairLoad(d, w.e, odd, l);
    D3 c, P1, P2, f1, f2;
    double sep;
    pairEval(l, w.p0 + w.D0, w.p1, c, P1, P2, f1, sep);
    if (sep > 0) w.stopFlag = true;
    pairEval(l, w.p0, w.p1 + w.D1, c, P1, P2, f2, sep);
    if (sep > 0) w.stopFlag = true;
    if (valid && !odd) ev64 += 2;
    w.rounds += 2;
    // even lane: column 0 of the Jacobian, odd lane: column 1
    const D3 g = odd ? f2 : f1;
    const double D = odd ? w.D1 : w.D0;
    const D3 J = d3((g.x - w.pf.x) / D, (g.y - w.pf.y) / D, (g.z - w.pf.z) / D);
    const D3 Jo = swapD3(J);
    const double jj = J.x * J.x + (J.y * J.y + J.z * J.z);
    const double jt = J.x * (-1.0 * w.pf.x) + (J.y * (-1.0 * w.pf.y) + J.z * (-1.0 * w.pf.z));
    w.j01 = J.x * Jo.x + (J.y * Jo.y + J.z * Jo.z);
    const double jjo = __shfl_xor_sync(FULL, jj, 1), jto = __shfl_xor_sync(FULL, jt, 1);
    w.diag0 = odd ? jjo : jj; w.diag1 = odd ? jj : jjo;
    w.jt0 = odd ? jto : jt; w.jt1 = odd ? jt : jto;
    const double jinf = (fabs(w.jt0) > fabs(w.jt1) ? fabs(w.jt0) : fabs(w.jt1));
    int stop = 0;
    bool more = true;
    if (w.k == 0) w.mu = 1.0 * (w.diag0 > w.diag1 ? w.diag0 : w.diag1);
    const bool flat = jinf <= 1e-15;
    {
      WaveState x = w;
      int st = 0;
      more = waveSolve(x, st, odd);
      if (flat) { stop = 1; more = false; }
      else { w = x; stop = st; }
    }
    const bool restart = waveCallEnd(w, l, stop, true, P1, P2, !more);
    if (valid && !odd) {
      if (!more && !restart) waveFinal(d, i, w, true, P1, P2);
      else waveStore(d, i, w);
    }
    waveAppend(valid && (more || restart), i, next, &d.Q->nT[round + 1]);
    waveAppend(valid && !more && !restart, i, d.waveF, &d.Q->nF);
  }
  for (int o = 16; o > 0; o >>= 1) ev64 += __shfl_down_sync(FULL, ev64, o);
  if (lane == 0 && ev64) atomicAdd(&d.S->err[E_EVAL64], ev64);
}

// Geometry, Ip2 and the law of the searches that ended in the rounds, one thread per search.
__global__ void __launch_bounds__(128) k_wave_finish(Dev d) {
  const int n = d.Q->nF;
  Counters cnt = {0, 0, 0, 0, 0};
  unsigned roundsMax = 0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    const int i = d.waveF[j], e = d.B.owner[i];
    const int4 c = d.B.cd[i];
    const double2 p = d.B.angle[i];
    const unsigned fl = d.A.flags[e];
    int id1, id2;
    entryIds(d, e, fl, id1, id2);
    roundsMax = max(roundsMax, (unsigned)c.w >> 1);
    finishSearch(d, e, fl, id1, id2, !(fl & F_GEOM), p.x, p.y, (c.w & 1) != 0, xyz(d.B.p1[i]), xyz(d.B.p2[i]), xyz(d.B.phys[i]),
                 (unsigned)c.x, (unsigned)c.y, (unsigned)c.z, cnt);
  }
  flushCounters(d, cnt);
  flushRounds(d, E_ROUNDS_MAX, roundsMax);
}
