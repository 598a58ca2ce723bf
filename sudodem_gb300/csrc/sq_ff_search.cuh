// The double-float searches of the mixed form: rounds over compact lists, then one warp per search.
// Included by sqdem_engine.cu after sq_wave_search.cuh, whose lists and table-B slots it uses.
//
// What bounds it: instruction issue and instruction fetch.  A double-float evaluation of both
// support points is some 4,700 FP32 operations in 25 KB of called functions; run by one lane per
// search, with the state machine of lmder2 around it, warps stood at different places of more code
// than the instruction caches hold, and the evaluations ran at an eighth of the rate a kernel of
// nothing else reaches (0.6 against 4.8 G/s).  Here a launch does one thing for a list of searches
// (the trial evaluations with their tests, or the two probes with the damped step), so that the
// warps of an SM run through the same code together, and a pair of lanes shares a search: the even
// one evaluates body A, the odd one body B, which halves the chain of dependent operations; the
// state machine runs on the even lane, its state in shared memory.  After some rounds the searches
// left are finished one per warp, sixteen points a round: five trials, each the successor of the one
// before should that be rejected, with their probes.  200,000 particles (2.9M evaluations): 5.2 -> 4.0
// ms alone (6.2 beside the long FP64 searches, which take 5.8 meanwhile); 12,800: 1.9 -> 1.0; 2,197:
// 1.15 -> 0.48.  Values, decisions and results per search are those of the state machine in
// sq_lmff.cuh, bit for bit.

__device__ __forceinline__ ff ffXor(ff a, int m) {
  const unsigned FULL = 0xffffffffu;
  return mkff(__shfl_xor_sync(FULL, a.hi, m), __shfl_xor_sync(FULL, a.lo, m));
}
__device__ __forceinline__ ff ffFrom(ff a, int lane) {
  const unsigned FULL = 0xffffffffu;
  return mkff(__shfl_sync(FULL, a.hi, lane), __shfl_sync(FULL, a.lo, lane));
}
// ffDisfunction by a pair of lanes: s the lane's own body, pB the centre of B relative to A's
__device__ __forceinline__ void ffPairEval(const FFShape& s, bool isB, const ff pB[3], ff q0, ff q1, FFEval& v) {
  const unsigned FULL = 0xffffffffu;
  ff sv, cv;
  const bool ok = ffSinCos(isB ? q1 : q0, sv, cv);
  const ff so = ffXor(sv, 1), co = ffXor(cv, 1);
  const ff s0 = isB ? so : sv, c0 = isB ? co : cv, s1 = isB ? sv : so, c1 = isB ? cv : co;
  v.c[0] = ffMul(c0, c1); v.c[1] = ffMul(s0, c1); v.c[2] = s1;
  ff n[3], q[3];
  for (int k = 0; k < 3; k++) {
    n[k] = ffDot3(s.R[k], s.R[3 + k], s.R[6 + k], v.c[0], v.c[1], v.c[2]);
    if (isB) n[k] = ffNeg(n[k]);
  }
  bool ill = !ok;
  ffSupport(s, n[0], n[1], n[2], q, ill);
  for (int i = 0; i < 3; i++) {
    ff p = ffDot3(s.R[3 * i], s.R[3 * i + 1], s.R[3 * i + 2], q[0], q[1], q[2]);
    if (isB) p = ffAdd(p, pB[i]);
    const ff o = ffXor(p, 1);
    v.p1[i] = isB ? o : p;
    v.p2[i] = isB ? p : o;
    v.d[i] = ffSub(v.p2[i], v.p1[i]);
  }
  v.sep = ffDot3(v.c[0], v.c[1], v.c[2], v.d[0], v.d[1], v.d[2]);
  v.ill = ill || __shfl_xor_sync(FULL, (int)ill, 1) != 0 || !(fabsf(v.sep.hi) < INFINITY);
}

// A double slot of table B holds a double-float's two parts.
__device__ __forceinline__ double ffPack(ff a) { return __hiloint2double(__float_as_int(a.hi), __float_as_int(a.lo)); }
__device__ __forceinline__ ff ffUnpack(double x) { return mkff(__int_as_float(__double2hiint(x)), __int_as_float(__double2loint(x))); }
__device__ __forceinline__ void ffLoad(const Dev& d, int i, LMF& L) {
  const Table& B = d.B;
  L.e = B.owner[i];
  const int4 c = B.cd[i];
  const unsigned f = (unsigned)c.z;
  L.k = c.x; L.nu = c.y; L.iters = (unsigned)c.w; L.stop = 0; L.touching = true;
  L.phase = (int)(f & 7u); L.fromCenter = f & WF_FROMCENTER; L.isNew = f & WF_NEW; L.stopFlag = f & WF_STOPFLAG;
  L.calls = (f >> 8) & 15u; L.maxit = (f >> 12) & 15u; L.rounds = f >> 16;
  const double2 p = B.angle[i];
  const double4 n = B.normal[i], s = B.shear[i], g = B.nforce[i], h = B.phys[i];
  L.p0 = ffUnpack(p.x); L.p1 = ffUnpack(p.y);
  L.pf[0] = ffUnpack(n.x); L.pf[1] = ffUnpack(n.y); L.pf[2] = ffUnpack(n.z); L.pfL2 = ffUnpack(n.w);
  L.jt0 = ffUnpack(s.x); L.jt1 = ffUnpack(s.y); L.j01 = ffUnpack(s.z); L.mu = ffUnpack(s.w);
  L.diag0 = ffUnpack(g.x); L.diag1 = ffUnpack(g.y); L.Dp0 = ffUnpack(g.z); L.Dp1 = ffUnpack(g.w);
  L.c[0] = ffUnpack(h.x); L.c[1] = ffUnpack(h.y); L.c[2] = ffUnpack(h.z);
  if (f & WF_INIT) { L.st = LMF_ST_INIT; L.q0 = L.p0; L.q1 = L.p1; }
  else { L.st = LMF_ST_TRIAL; L.q0 = ffAdd(L.p0, L.Dp0); L.q1 = ffAdd(L.p1, L.Dp1); }
}
__device__ __forceinline__ void ffStore(const Dev& d, int i, const LMF& L) {
  const Table& B = d.B;
  const unsigned f = (unsigned)L.phase | (L.fromCenter ? WF_FROMCENTER : 0u) | (L.isNew ? WF_NEW : 0u) |
                     (L.stopFlag ? WF_STOPFLAG : 0u) | (L.st == LMF_ST_INIT ? WF_INIT : 0u) | (L.calls << 8) | (L.maxit << 12) |
                     (L.rounds << 16);
  B.owner[i] = L.e;
  B.cd[i] = make_int4(L.k, L.nu, (int)f, (int)L.iters);
  B.angle[i] = make_double2(ffPack(L.p0), ffPack(L.p1));
  B.normal[i] = make_double4(ffPack(L.pf[0]), ffPack(L.pf[1]), ffPack(L.pf[2]), ffPack(L.pfL2));
  B.shear[i] = make_double4(ffPack(L.jt0), ffPack(L.jt1), ffPack(L.j01), ffPack(L.mu));
  B.nforce[i] = make_double4(ffPack(L.diag0), ffPack(L.diag1), ffPack(L.Dp0), ffPack(L.Dp1));
  B.phys[i] = make_double4(ffPack(L.c[0]), ffPack(L.c[1]), ffPack(L.c[2]), 0);
}
// the search's geometry, still in double-float: k_ff_finish converts and completes it in FP64
__device__ __forceinline__ void ffFinal(const Dev& d, int i, const LMF& L) {
  const Table& B = d.B;
  B.owner[i] = L.e;
  B.angle[i] = make_double2(ffPack(L.p0), ffPack(L.p1));
  B.p1[i] = make_double4(ffPack(L.P1[0]), ffPack(L.P1[1]), ffPack(L.P1[2]), 0);
  B.p2[i] = make_double4(ffPack(L.P2[0]), ffPack(L.P2[1]), ffPack(L.P2[2]), 0);
  B.phys[i] = make_double4(ffPack(L.c[0]), ffPack(L.c[1]), ffPack(L.c[2]), 0);
  B.cd[i] = make_int4((int)L.calls, (int)L.iters, (int)L.maxit, (int)(L.rounds << 1) | (L.touching ? 1 : 0));
}
__device__ __forceinline__ int mainEntry(const Dev& d, int j) {
  const int nFront = d.S->lmCount;
  return j < nFront ? d.lmQueue[j] : d.lmQueue[d.qCap - 1 - (j - nFront)];
}
// The bodies of entry e, and the centre of B relative to A's: from the positions in a search's first
// launch, which leaves it in the slot for the next ones (some 40 FP64 instructions of 19 cycles each
// per SM, a third of a double-float evaluation's time).
__device__ __forceinline__ void ffCentre(const Dev& d, int e, int id1, int id2, D3& pa, D3& pb, ff pB[3]) {
  pa = xyz(d.pos[id1]);
  pb = xyz(d.pos[id2]) + cellShift(*d.S, d.A.cd[e]);
  pB[0] = ffFromD(pb.x - pa.x); pB[1] = ffFromD(pb.y - pa.y); pB[2] = ffFromD(pb.z - pa.z);
}
__device__ __forceinline__ void ffCentreLoad(const Dev& d, int i, ff pB[3]) {
  const double4 f = d.B.F[i];
  pB[0] = ffUnpack(f.x); pB[1] = ffUnpack(f.y); pB[2] = ffUnpack(f.z);
}
__device__ __forceinline__ void ffFresh(const Dev& d, int e, D3 pa, D3 pb, LMF& L) {
  L.e = e;
  L.isNew = !(d.A.flags[e] & F_GEOM);
  if (L.isNew) { double para[2]; centerLine(pa, pb, para); L.p0 = ffFromD(para[0]); L.p1 = ffFromD(para[1]); }
  else { const double2 an = d.A.angle[e]; L.p0 = ffFromD(an.x); L.p1 = ffFromD(an.y); }
  L.fromCenter = L.isNew;
  L.phase = 0; L.calls = 0; L.iters = 0; L.maxit = 0; L.rounds = 0;
  L.k = 0; L.nu = 2;
  L.mu = L.Dp0 = L.Dp1 = L.pfL2 = L.diag0 = L.diag1 = L.j01 = L.jt0 = L.jt1 = mkff(0.f, 0.f);
  for (int i = 0; i < 3; i++) L.pf[i] = L.c[i] = mkff(0.f, 0.f);
  lmfStartSolve(L);
}
// what became of a search after a launch's consumed evaluations: lists and queues (even lanes)
__device__ __forceinline__ void ffRoute(const Dev& d, int i, bool mine, int r, const LMF& L, int* next, int round, unsigned long long& deferred) {
  if (mine) {
    if (r == LMF_END) ffFinal(d, i, L);
    else if (r == LMF_MORE) ffStore(d, i, L);
    else {
      d.deferQueue[atomicAdd(&d.S->fbCount, 1)] = L.e;
      deferred++;
      atomicMax(&d.S->err[E_ROUNDS_MAX_FF], (unsigned long long)L.rounds);
    }
  }
  const bool more = mine && r == LMF_MORE;
  waveAppend(more && L.st == LMF_ST_PROBE0, i, d.waveP, &d.Q->nP[round]);
  waveAppend(more && L.st != LMF_ST_PROBE0, i, next, &d.Q->nT[round + 1]);
  waveAppend(mine && r == LMF_END, i, d.waveF, &d.Q->nF);
}
__device__ __forceinline__ void ffCount(const Dev& d, unsigned long long ev, unsigned long long deferred) {
  for (int o = 16; o > 0; o >>= 1) {
    ev += __shfl_down_sync(0xffffffffu, ev, o);
    deferred += __shfl_down_sync(0xffffffffu, deferred, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (ev) atomicAdd(&d.S->err[E_EVAL32], ev);
    if (deferred) atomicAdd(&d.S->err[E_FALLBACK], deferred);
  }
}

template <bool FIRST>
__global__ void __launch_bounds__(LM_BS, 4) k_ff_trial(Dev d, int round, int few) {
  __shared__ LMF sL[LM_BS / 2];
  const int n = FIRST ? d.S->lmCount + d.S->nmShort : d.Q->nT[round];
  if (FIRST && n <= few) return;   // k_ff_warp takes them all
  const int* in = (round & 1) ? d.waveT1 : d.waveT0;
  int* next = (round & 1) ? d.waveT0 : d.waveT1;
  const int lane = threadIdx.x & 31;
  const bool isB = lane & 1;
  const int warps = gridDim.x * (LM_BS / 32);
  LMF& L = sL[threadIdx.x >> 1];
  unsigned long long ev = 0, deferred = 0;
  for (int t = blockIdx.x * (LM_BS / 32) + (threadIdx.x >> 5); t * 16 < n; t += warps) {
    const int idx = t * 16 + (lane >> 1);
    const bool mine = idx < n && !isB;
    const int j = min(idx, n - 1);
    const int i = FIRST ? j : in[j];
    const int e = FIRST ? mainEntry(d, j) : d.B.owner[i];
    int id1, id2;
    entryIds(d, e, d.A.flags[e], id1, id2);
    D3 pa, pb;
    ff pB[3];
    if (FIRST) {
      ffCentre(d, e, id1, id2, pa, pb, pB);
      if (mine) d.B.F[i] = make_double4(ffPack(pB[0]), ffPack(pB[1]), ffPack(pB[2]), 0);
    } else ffCentreLoad(d, i, pB);
    if (!isB) {
      if (FIRST) ffFresh(d, e, pa, pb, L);
      else ffLoad(d, i, L);
      L.E = 4e-13f * (d.bodyFF[id1].rmax + d.bodyFF[id2].rmax);
    }
    __syncwarp();
    FFEval v;
    ffPairEval(d.bodyFF[isB ? id2 : id1], isB, pB, L.q0, L.q1, v);
    int r = LMF_DEFER;
    if (mine) {
      ev++;
      L.rounds++;
      r = lmfConsume(L, v);
      if (r == LMF_END) r = lmfCallEnd(d, L, id1, id2, pB);
    }
    __syncwarp();
    ffRoute(d, i, mine, r, L, next, round, deferred);
    __syncwarp();
  }
  ffCount(d, ev, deferred);
}

__global__ void __launch_bounds__(LM_BS, 4) k_ff_probe(Dev d, int round) {
  __shared__ LMF sL[LM_BS / 2];
  const int n = d.Q->nP[round];
  int* next = (round & 1) ? d.waveT0 : d.waveT1;
  const int lane = threadIdx.x & 31;
  const bool isB = lane & 1;
  const int warps = gridDim.x * (LM_BS / 32);
  LMF& L = sL[threadIdx.x >> 1];
  unsigned long long ev = 0, deferred = 0;
  for (int t = blockIdx.x * (LM_BS / 32) + (threadIdx.x >> 5); t * 16 < n; t += warps) {
    const int idx = t * 16 + (lane >> 1);
    const bool mine = idx < n && !isB;
    const int i = d.waveP[min(idx, n - 1)];
    const int e = d.B.owner[i];
    int id1, id2;
    entryIds(d, e, d.A.flags[e], id1, id2);
    ff pB[3];
    ffCentreLoad(d, i, pB);
    const FFShape& s = d.bodyFF[isB ? id2 : id1];
    if (!isB) {
      ffLoad(d, i, L);
      L.E = 4e-13f * (d.bodyFF[id1].rmax + d.bodyFF[id2].rmax);
      L.st = LMF_ST_PROBE0; L.q0 = ffAdd(L.p0, L.Dp0); L.q1 = L.p1;
    }
    __syncwarp();
    FFEval v;
    ffPairEval(s, isB, pB, L.q0, L.q1, v);
    int r = LMF_DEFER;
    __syncwarp();
    if (!isB) {
      r = lmfConsume(L, v);
      if (r == LMF_DEFER) { L.q0 = L.p0; L.q1 = L.p1; }   // the second probe is not wanted: any point
    }
    __syncwarp();
    ffPairEval(s, isB, pB, L.q0, L.q1, v);
    if (mine) {
      ev += 2;
      L.rounds += 2;
      if (r == LMF_MORE) r = lmfConsume(L, v);
      if (r == LMF_END) r = lmfCallEnd(d, L, id1, id2, pB);
    }
    __syncwarp();
    ffRoute(d, i, mine, r, L, next, round, deferred);
    __syncwarp();
  }
  ffCount(d, ev, deferred);
}

// One search per warp, sixteen points a round.  tail: the searches left after `rounds` rounds, unless
// the main queue is no longer than `few`; else the main queue.
__global__ void __launch_bounds__(LM_BS, 4) k_ff_warp(Dev d, int tail, int rounds, int few) {
  const unsigned FULL = 0xffffffffu;
  if (tail && d.S->lmCount + d.S->nmShort <= few) tail = 0;
  const int lane = threadIdx.x & 31, grp = lane >> 1;
  const bool isB = lane & 1;
  const int trial = grp < 15 ? grp / 3 : 0, role = grp < 15 ? grp % 3 : 0;   // group 15 mirrors group 0
  const int total = tail ? d.Q->nT[rounds] : d.S->lmCount + d.S->nmShort;
  int* head = tail ? &d.Q->tailHead : &d.S->lmHead;
  if ((int)(threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x >= total) return;
  unsigned long long ev = 0, deferred = 0;
  unsigned roundsMax = 0;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(head, 1);
    idx = __shfl_sync(FULL, idx, 0);
    if (idx >= total) break;
    const int i = tail ? ((rounds & 1) ? d.waveT1 : d.waveT0)[idx] : idx;
    const int e = tail ? d.B.owner[i] : mainEntry(d, idx);
    int id1, id2;
    entryIds(d, e, d.A.flags[e], id1, id2);
    D3 pa, pb;
    ff pB[3];
    if (tail) ffCentreLoad(d, i, pB);
    else ffCentre(d, e, id1, id2, pa, pb, pB);
    const FFShape& s = d.bodyFF[isB ? id2 : id1];
    LMF L;
    if (tail) ffLoad(d, i, L);
    else ffFresh(d, e, pa, pb, L);
    const float E = 4e-13f * (d.bodyFF[id1].rmax + d.bodyFF[id2].rmax);
    L.E = E;
    bool resume = tail && L.st != LMF_ST_INIT;   // the call goes on at the pending trial
    int r = LMF_MORE;
    unsigned nr = L.rounds;
    // every lane carries the whole state; L holds it between calls
    do {   // one lmder2 call
      ff p0 = L.p0, p1 = L.p1, mu = L.mu, Dp0 = L.Dp0, Dp1 = L.Dp1, pfL2 = L.pfL2;
      ff diag0 = L.diag0, diag1 = L.diag1, j01 = L.j01, jt0 = L.jt0, jt1 = L.jt1;
      ff pf[3] = {L.pf[0], L.pf[1], L.pf[2]};
      int k = L.k, nu = L.nu, stop = 0;
      bool stopFlag = L.stopFlag, touching = true;
      int base = 0, last = 0;
      FFEval v = {};
      // each group's verdicts on its own point, for the one that is accepted: bits of its first lane
      unsigned badB = 0, posB = 0, smallB = 0, nearB = 0, onB = 0;
      ff nrmv = mkff(0.f, 0.f);
      auto verdicts = [&]() {
        const ff f2 = ffDot3(v.d[0], v.d[1], v.d[2], v.d[0], v.d[1], v.d[2]);
        nrmv = ffSqrt(f2);
        const ff fc = ffDot3(v.d[0], v.d[1], v.d[2], v.c[0], v.c[1], v.c[2]);
        const ff c2 = ffDot3(v.c[0], v.c[1], v.c[2], v.c[0], v.c[1], v.c[2]);
        const ff th = ffFromD(0.95);
        const ff diff = ffSub(ffMul(fc, fc), ffMul(ffMul(th, th), ffMul(f2, c2)));
        const float band = 1.9f * (1e-12f * f2.hi + 4.f * E * sqrtf(f2.hi)) * c2.hi;
        badB = __ballot_sync(FULL, v.ill || !(fabsf(v.sep.hi) >= E));
        posB = __ballot_sync(FULL, v.sep.hi > 0.f);
        smallB = __ballot_sync(FULL, nrmv.hi < E);
        nearB = __ballot_sync(FULL, !(fabsf(diff.hi) >= band));
        onB = __ballot_sync(FULL, diff.hi > 0.f);
      };
      // consume the evaluation of group g: false when the search is deferred
      auto consume = [&](int g) {
        if ((badB >> (2 * g)) & 1u) return false;
        if ((posB >> (2 * g)) & 1u) stopFlag = true;
        last = g;
        return true;
      };
      // group `base`'s point is the current one: lmder2's tests there (lmfOuter)
      auto outer = [&]() {
        const int l = 2 * base;
        for (int c = 0; c < 3; c++) { pf[c] = ffFrom(v.d[c], l); L.c[c] = ffFrom(v.c[c], l); }
        pfL2 = ffFrom(nrmv, l);
        if (k >= 50) return (int)LMF_DEFER;
        if (stop) return (int)LMF_END;
        if ((smallB >> l) & 1u) return (int)LMF_DEFER;
        if (stopFlag) { stop = 9; touching = false; return (int)LMF_END; }
        if ((nearB >> l) & 1u) return (int)LMF_DEFER;
        if ((onB >> l) & 1u) { stop = 8; return (int)LMF_END; }
        return (int)LMF_MORE;
      };
      r = LMF_MORE;
      if (!resume) {
        mu = mkff(0.f, 0.f); nu = 2; k = 0;
        Dp0 = ffInitStep(); Dp1 = ffInitStep();
        ffPairEval(s, isB, pB, grp == 1 ? ffAdd(p0, Dp0) : p0, grp == 2 ? ffAdd(p1, Dp1) : p1, v);
        nr++;
        ev += 3;
        verdicts();
        r = consume(0) ? outer() : (int)LMF_DEFER;
      }
      while (r == LMF_MORE) {
        if (!resume) {
          if (!consume(base + 1) || !consume(base + 2)) { r = LMF_DEFER; break; }
          // even lanes: column 0 of the Jacobian, odd lanes: column 1 (lanes differ in nothing else)
          const int src = 2 * (base + 1 + (isB ? 1 : 0));
          const ff inv = ffDiv(mkff(1.f, 0.f), isB ? Dp1 : Dp0);
          ff J[3], O[3];
          for (int c = 0; c < 3; c++) { J[c] = ffMul(ffSub(ffFrom(v.d[c], src), pf[c]), inv); O[c] = ffXor(J[c], 1); }
          const ff jj = ffDot3(J[0], J[1], J[2], J[0], J[1], J[2]);
          const ff jt = ffNeg(ffDot3(J[0], J[1], J[2], pf[0], pf[1], pf[2]));
          ff a[3], b[3];   // columns 0 and 1
          for (int c = 0; c < 3; c++) { a[c] = isB ? O[c] : J[c]; b[c] = isB ? J[c] : O[c]; }
          j01 = ffDot3(a[0], a[1], a[2], b[0], b[1], b[2]);
          const ff jjo = ffXor(jj, 1), jto = ffXor(jt, 1);
          diag0 = isB ? jjo : jj; diag1 = isB ? jj : jjo;
          jt0 = isB ? jto : jt; jt1 = isB ? jt : jto;
          const float jinf = fmaxf(fabsf(jt0.hi), fabsf(jt1.hi));
          if (!(fabsf(jinf * 1e15f - 1.f) >= 1e-5f)) { r = LMF_DEFER; break; }
          if (jinf <= 1e-15f) { stop = 1; r = LMF_END; break; }
          if (k == 0) mu = ffGt(diag0, diag1) ? diag0 : diag1;
        }
        resume = false;
        for (;;) {   // damping loop: the step for mu and those of the next four rejections
          ff myMu = mu;
          for (int j = 0, m = nu; j < trial; j++, m = (int)((unsigned)m << 1)) myMu = ffMulF(myMu, (float)m);
          ff D0, D1, dp2;
          lmfSolve(ffAdd(diag0, myMu), j01, ffAdd(diag1, myMu), jt0, jt1, D0, D1, dp2);
          const unsigned edgeB = __ballot_sync(FULL, !(fabsf(dp2.hi * 1e10f - 1.f) >= 2e-5f));
          const unsigned tinyB = __ballot_sync(FULL, dp2.hi < 1e-10f);
          const float pL2 = sqrtf(p0.hi * p0.hi + p1.hi * p1.hi);
          const unsigned hugeB = __ballot_sync(FULL, sqrtf(dp2.hi) >= (pL2 + 1e-3f) * 1e24f);
          // the step of trial a ends the call (lmfInner's stops): its outcome, LMF_MORE if it does not
          auto step = [&](int l) {
            if ((edgeB >> l) & 1u) return (int)LMF_DEFER;
            if (((tinyB >> l) | (hugeB >> l)) & 1u) { stop = ((tinyB >> l) & 1u) ? 2 : 4; k++; return k >= 50 ? (int)LMF_DEFER : (int)LMF_END; }
            return (int)LMF_MORE;
          };
          r = step(0);
          if (r != LMF_MORE) break;
          const ff t0 = ffAdd(p0, D0), t1 = ffAdd(p1, D1);
          ffPairEval(s, isB, pB, role == 1 ? ffAdd(t0, D0) : t0, role == 2 ? ffAdd(t1, D1) : t1, v);
          nr++;
          ev += 15;
          verdicts();
          const ff dF = ffSub(pfL2, nrmv);
          const unsigned fuzzB = __ballot_sync(FULL, !(fabsf(dF.hi) >= E)), gainB = __ballot_sync(FULL, dF.hi > 0.f);
          const ff dL = ffAdd(ffMul(D0, ffAdd(ffMul(myMu, D0), jt0)), ffMul(D1, ffAdd(ffMul(myMu, D1), jt1)));
          const ff t = ffAddF(ffMulF(ffDiv(dF, dL), 2.f), -1.f);
          const ff tmp = ffAddF(ffNeg(ffMul(ffMul(t, t), t)), 1.f);
          const ff third = ffFromD(0.3333333333333334);
          const ff muNext = ffMul(myMu, ffGt(third, tmp) ? third : tmp);
          bool taken = false;
          for (int a = 0; a < 5; a++) {
            const int l = 6 * a;
            if (a > 0 && (r = step(l)) != LMF_MORE) break;
            if (!consume(3 * a) || ((fuzzB >> l) & 1u)) { r = LMF_DEFER; break; }
            if ((gainB >> l) & 1u) {
              base = 3 * a;
              mu = ffFrom(muNext, l);
              nu = 2;
              Dp0 = ffFrom(D0, l); Dp1 = ffFrom(D1, l);
              p0 = ffFrom(t0, l); p1 = ffFrom(t1, l);
              k++;
              r = outer();
              taken = true;
              break;
            }
            mu = ffMulF(mu, (float)nu);
            const int nn = (int)((unsigned)nu << 1);
            if (nn <= nu) { stop = 5; k++; r = k >= 50 ? (int)LMF_DEFER : (int)LMF_END; break; }
            nu = nn;
          }
          if (taken || r != LMF_MORE) break;
        }
      }
      L.p0 = p0; L.p1 = p1;
      L.k = k; L.stop = stop; L.touching = touching;
      if (r == LMF_END) {
        for (int c = 0; c < 3; c++) { L.P1[c] = ffFrom(v.p1[c], 2 * last); L.P2[c] = ffFrom(v.p2[c], 2 * last); }
        r = lmfCallEnd(d, L, id1, id2, pB);
        resume = false;
      }
    } while (r == LMF_MORE);
    L.rounds = nr;
    if (lane == 0) {
      if (r == LMF_END) { ffFinal(d, i, L); d.waveF[atomicAdd(&d.Q->nF, 1)] = i; }
      else { d.deferQueue[atomicAdd(&d.S->fbCount, 1)] = e; deferred++; }
    }
    roundsMax = max(roundsMax, nr);
  }
  ffCount(d, lane == 0 ? ev : 0ull, deferred);
  if (lane == 0 && roundsMax) atomicMax(&d.S->err[E_ROUNDS_MAX_FF], (unsigned long long)roundsMax);
}
