// One Levenberg-Marquardt search (lmder2, Superquadrics_Ig2.cpp:1057-1354) by one warp, FP64.
// Included by sqdem_engine.cu after the per-entry functions it finishes a contact with.
//
// What bounds it: GB300 issues one FP64 warp instruction per 64 cycles and scheduler, whether 1 or
// 32 lanes take part (a chain of dependent DFMAs: 64.6 cycles each at any lane count, and no
// fewer with four independent chains; pow 6,040 cycles, atan2 2,760, sincos 1,610, a division 580),
// and an evaluation of the pair's two support points needs 18 pow, 4 atan2, 6 sincos one after
// another if one lane does it (146,000 cycles).  The searches that bound a step run 50-100
// iterations, each a trial evaluation, 0.9 rejected trials on average, and two
// finite-difference probes, all dependent on one another.  So the 32 lanes of a warp serve one
// search: six points per round, five lanes a point (two lanes per body, the fifth takes the ninth
// pow of both), which makes a round's evaluation 4 pow + 2 atan2 + 3 sincos long: the pending trial,
// those that follow if it is rejected, and the probes of the one likely to be accepted (1.3 rounds
// an iteration; 1.4 with always two trials).  The state machine's own arithmetic (the Jacobian's six divisions, the normal equations, the
// steps, gain ratios and damping of all trials) is spread over the lanes as well; it took a third
// of a round when the owning lane did it alone.  A round takes 21-23 us (26-29 before, of one third
// of an iteration while four searches shared a warp).  Longest searches of a jammed cell of 12,800
// particles: FP64 pass 5.3 -> 3.4 ms; a servo specimen of 2,197: 3.1 -> 1.6 ms.
//
// Every value is computed by lmder2's operations on the same operands, in the same order, so that a
// search's results do not depend on the schedule: speculative points that it does not come to are
// dropped.

#include "sq_warp_plan.cuh"

static const int WS_LANES = 5, WS_POINTS = 6;

// sgn(n) * y for y >= 0 (0 when n is 0, where y is 0 in every use), without the multiplication
__device__ __forceinline__ double signOf(double y, double n) {
  const long long b = __double_as_longlong(n);
  const bool neg = b < 0 && (b << 1) != 0;
  return neg ? -y : y;
}

// One body's shape as a lane of the pair needs it.  k = 0: rows for n.y and p.x, k = 1: n.x, p.y.
struct WShape {
  double rx, ry, rz, e1, e2, a1, i1, i2, rmax;
  double R[9];
  D3 pos;
};

__device__ __forceinline__ void warpShape(const Dev& d, int b, WShape& s) {
  const double4 a = d.shpA[b], x = d.shpB[b], q = d.ori[b];
  s.rx = a.x; s.ry = a.y; s.rz = a.z; s.rmax = a.w; s.e1 = x.x; s.e2 = x.y;
  s.a1 = 2. - x.x; s.i1 = 1 / (2. - x.x); s.i2 = 1 / (2. - x.y);
  const Rot R = quatToRot(q.x, q.y, q.z, q.w);
  for (int i = 0; i < 9; i++) s.R[i] = R.m[i];
  s.pos = xyz(d.pos[b]);
}

// What a round leaves in the lanes of each point's group.
struct WEval {
  double pxy, pz;    // support point of the lane's body: x (k = 0) or y (k = 1), and z
  double fxy, fz;    // p2 - p1: x (k = 0) or y (k = 1), and z
  double sep, nrm;   // c . (p2 - p1), |p2 - p1|
  D3 c;              // contact direction at the point
};

// g0: first lane of the group, r: the lane's place in it (0, 1: body A; 2, 3: body B; 4: v of both);
// G: frame of the angles, if any (the Hertz-Mindlin model's Disfun)
__device__ __forceinline__ void warpEval(const WShape& s, double e1B, int g0, int r, double q0, double q1, WEval& o,
                                         const Rot* G = nullptr) {
  const unsigned FULL = 0xffffffffu;
  const bool isB = r == 2 || r == 3, k = r == 1 || r == 3, extra = r == 4;
  const int mate = extra ? g0 + 1 : g0 + (r ^ 1);
  double sv, cv;
  sincos(k ? q1 : q0, &sv, &cv);
  const double sa0 = __shfl_sync(FULL, sv, g0), ca0 = __shfl_sync(FULL, cv, g0);
  const double sa1 = __shfl_sync(FULL, sv, g0 + 1), ca1 = __shfl_sync(FULL, cv, g0 + 1);
  o.c = d3(ca0 * ca1, sa0 * ca1, sa1);
  if (G) o.c = mulG(*G, o.c);
  // local normal +-R^T c: x on k = 1, y on k = 0, z on both
  double na = (k ? s.R[0] : s.R[1]) * o.c.x + ((k ? s.R[3] : s.R[4]) * o.c.y + (k ? s.R[6] : s.R[7]) * o.c.z);
  double nz = s.R[2] * o.c.x + (s.R[5] * o.c.y + s.R[8] * o.c.z);
  if (isB) { na = -na; nz = -nz; }
  const double nb = __shfl_sync(FULL, na, mate);
  const double nx = k ? na : nb, ny = k ? nb : na;
  const double b1 = fabs(k ? s.rx * nx : s.ry * ny);
  const double v1 = pow(b1, s.i1);   // Y | X
  const double w1 = __shfl_sync(FULL, v1, mate);
  const double ph0 = atan2(signOf(k ? w1 : v1, ny), signOf(k ? v1 : w1, nx));
  double s0, c0;
  sincos(ph0, &s0, &c0);
  const double v2 = pow(extra ? fabs(s0) : k ? b1 : fabs(c0), extra ? s.e1 : k ? s.i2 : s.a1);   // t | W | v of A
  const double s0B = __shfl_sync(FULL, s0, g0 + 2);
  const double v3 = pow(extra ? fabs(s0B) : k ? fabs(c0) : fabs(s.rz * nz * v2), extra ? e1B : k ? s.e1 : s.i2);   // Z | u | v of B
  const double w2 = __shfl_sync(FULL, v2, mate), w3 = __shfl_sync(FULL, v3, mate);
  const double vA = __shfl_sync(FULL, v2, g0 + 4), vB = __shfl_sync(FULL, v3, g0 + 4);
  const double ph1 = atan2(signOf(k ? w3 : v3, nz), k ? v2 : w2);
  double s1, c1;
  sincos(ph1, &s1, &c1);
  const double v4 = pow(fabs(k ? s1 : c1), s.e2);   // |cos phi1|^eps2 | |sin phi1|^eps2
  const double w4 = __shfl_sync(FULL, v4, mate);
  const double pc1 = k ? w4 : v4, ps1 = k ? v4 : w4;
  const double rxy = signOf(k ? s.ry : s.rx, k ? s0 : c0) * (k ? (isB ? vB : vA) : w3) * pc1;
  const double rz = signOf(s.rz, s1) * ps1;
  const double rot = __shfl_sync(FULL, rxy, mate);
  const double rX = k ? rot : rxy, rY = k ? rxy : rot;
  o.pxy = ((k ? s.R[3] : s.R[0]) * rX + ((k ? s.R[4] : s.R[1]) * rY + (k ? s.R[5] : s.R[2]) * rz)) + (k ? s.pos.y : s.pos.x);
  o.pz = (s.R[6] * rX + (s.R[7] * rY + s.R[8] * rz)) + s.pos.z;
  const int ka = k ? 1 : 0;
  o.fxy = __shfl_sync(FULL, o.pxy, g0 + 2 + ka) - __shfl_sync(FULL, o.pxy, g0 + ka);
  o.fz = __shfl_sync(FULL, o.pz, g0 + 2) - __shfl_sync(FULL, o.pz, g0);
  const double m1 = (k ? o.c.y : o.c.x) * o.fxy, m2 = o.c.z * o.fz;
  const double n1 = o.fxy * o.fxy, n2 = o.fz * o.fz;
  const double m1o = __shfl_sync(FULL, m1, mate), n1o = __shfl_sync(FULL, n1, mate);
  o.sep = (k ? m1o : m1) + ((k ? m1 : m1o) + m2);
  o.nrm = sqrt((k ? n1o : n1) + ((k ? n1 : n1o) + n2));
}

// A point of a round, as all lanes of a search read it: its evaluation, and for a trial point the
// step it came from and what follows if it is accepted.
struct WSlot {
  double f[3], nrm, sep, c[3], a[3], b[3];   // p2 - p1, |f|, c . f, direction, support points
  double D0, D1, t0, t1, mu;
  unsigned bits;
};
enum { WB_APART = 1, WB_FINITE = 2, WB_GAIN = 4, WB_SMALL = 8, WB_HUGE = 16 };

// Work lists: which entries a launch takes, in this order.
//   WS_LONG      the long-search queue (fbQueue), its front first
//   WS_DEFERRED  the searches the mixed form's double-float kernels deferred (deferQueue)
//   WS_MAIN      the main queue (lmQueue), longest first
//   WS_TAIL      the searches left after `rounds` rounds of k_wave_trial / k_wave_probe, from there on;
//                the main queue where it is no longer than `few`, which those leave alone
enum { WS_LONG = 0, WS_DEFERRED = 1, WS_MAIN = 2, WS_TAIL = 3 };

// W warps per search.  W = 1: blocks go to the SMs in turn, so that in blocks of one warp fewer
// searches than warps have an SM's FP64 pipes to themselves (64 cycles an instruction, 76 with four
// busy schedulers).  W = 2: a block of two warps, twelve points a round, four trials with their
// probes each: 1.07 rounds an iteration instead of 1.33 for twice the FP64 work, where few searches
// bound the stage and the pipes are otherwise idle (12,800 particles, mixed form: 18.3 -> 15.1 ms for
// five steps; 1,583 in FP64: 3.46 -> 2.82 ms a step; 20,000 polydisperse: 11.1 -> 9.6 for three).
template <int W>
__global__ void __launch_bounds__(W == 1 ? LM_BS : 64, W == 1 ? 3 : 6) k_search_warp(Dev d, int mode, int waveRounds, int few) {
  const unsigned FULL = 0xffffffffu;
  const SceneState& S = *d.S;
  if (mode == WS_TAIL && S.lmCount + S.nmShort <= few) mode = WS_MAIN;
  extern __shared__ WSlot wsSlots[];   // per search of the block: two rounds of WS_POINTS * W (wsShared)
  WSlot (*slots)[2][WS_POINTS * W] = reinterpret_cast<WSlot(*)[2][WS_POINTS * W]>(wsSlots);
  __shared__ int taken[W == 1 ? LM_BS / 32 : 1];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int own = W == 1 ? wib : 0;                 // the search's place in the block
  const bool real = lane < WS_LANES * WS_POINTS;    // lanes 30, 31: the step of trial 0, no point of their own
  const int g0 = real ? lane / WS_LANES * WS_LANES : 0;
  const int r = real ? lane - g0 : lane - WS_LANES * WS_POINTS;
  const int grp = (W == 1 ? 0 : wib * WS_POINTS) + g0 / WS_LANES;
  const int gs = real ? g0 : 30;                    // where the lane's step is computed
  const bool odd = r == 1 || r == 3;
  const int nLong1 = S.vlCount, nLong = S.vlCount + min(d.Q->vl2Count, d.prm->vlongMax);
  const int nFront = S.lmCount;
  const int total = mode == WS_LONG       ? nLong
                    : mode == WS_DEFERRED ? S.fbCount
                    : mode == WS_TAIL     ? d.Q->nT[waveRounds]
                                          : S.lmCount + S.nmShort;
  int* head = mode == WS_LONG ? &d.S->vlHead : mode == WS_DEFERRED ? &d.S->fbHead : mode == WS_TAIL ? &d.Q->tailHead : &d.S->lmHead;
  if ((int)(W == 1 ? blockIdx.x * (blockDim.x >> 5) + wib : blockIdx.x) >= total) return;
  Counters cnt = {0, 0, 0, 0, 0};
  unsigned long long ev64 = 0;
  unsigned roundsMax = 0;
  int flip = 0;
  auto join = [&]() { if (W == 1) __syncwarp(); else __syncthreads(); };
  for (;;) {
    if (lane == 0 && (W == 1 || wib == 0)) taken[own] = atomicAdd(head, 1);
    join();
    const int idx = taken[own];
    join();
    if (idx >= total) break;
    int e;
    WaveState w;
    bool resume = false;   // the call goes on at the pending trial
    if (mode == WS_TAIL) {
      waveLoad(d, ((waveRounds & 1) ? d.waveT1 : d.waveT0)[idx], w);
      e = w.e;
      resume = !w.init;
    } else if (mode == WS_DEFERRED) e = d.deferQueue[idx];
    else if (mode == WS_LONG) e = idx < nLong1 ? d.fbQueue[idx] : d.fbQueue[d.Pcap - 1 - (idx - nLong1)];
    else e = idx < nFront ? d.lmQueue[idx] : d.lmQueue[d.qCap - 1 - (idx - nFront)];
    // start of Ig2_Superquadrics_Superquadrics_SuperquadricsGeom::go up to lmder2
    const unsigned fl = d.A.flags[e];
    int id1, id2;
    entryIds(d, e, fl, id1, id2);
    const bool bodyB = r == 2 || r == 3;
    WShape s;
    {
      warpShape(d, bodyB ? id2 : id1, s);
      if (bodyB) s.pos = s.pos + cellShift(S, d.A.cd[e]);
    }
    const double e1B = d.shpB[id2].x;
    const bool isNew = !(fl & F_GEOM);
    bool fromCenter = isNew;
    double p0 = 0, p1 = 0;
    auto centre = [&]() {
      double para[2];
      centerLine(d3(__shfl_sync(FULL, s.pos.x, 0), __shfl_sync(FULL, s.pos.y, 0), __shfl_sync(FULL, s.pos.z, 0)),
                 d3(__shfl_sync(FULL, s.pos.x, 2), __shfl_sync(FULL, s.pos.y, 2), __shfl_sync(FULL, s.pos.z, 2)), para);
      p0 = para[0]; p1 = para[1];
    };
    if (mode == WS_TAIL) { p0 = w.p0; p1 = w.p1; fromCenter = w.fromCenter; }
    else if (isNew) centre();
    else { const double2 an = d.A.angle[e]; p0 = an.x; p1 = an.y; }
    D3 contact = d3(0, 0, 0), P1 = d3(0, 0, 0), P2 = d3(0, 0, 0);
    int phase = 0;
    unsigned calls = 0, iters = 0, maxit = 0, rounds = 0;
    bool touching = true;
    if (mode == WS_TAIL) { contact = w.contact; phase = (int)w.phase; calls = w.calls; iters = w.iters; maxit = w.maxit; rounds = w.rounds; }
    WSlot* q = slots[own][flip];   // the last round's points
    // evaluates the lane's group's point into the round's slots; the other trial fields are the caller's
    auto round = [&](double q0, double q1, bool trial, double D0, double D1, double t0, double t1, double myMu, double pfL2,
                     double jt0, double jt1, unsigned bits) {
      WEval v;
      warpEval(s, e1B, g0, r, q0, q1, v);
      double muNext = 0;
      if (v.sep > 0) bits |= WB_APART;
      if (isfinite(v.nrm)) bits |= WB_FINITE;
      if (trial) {   // gain ratio and damping update
        const double dm = (odd ? D1 : D0) * (myMu * (odd ? D1 : D0) + (odd ? jt1 : jt0));
        const double dmo = __shfl_sync(FULL, dm, r == 4 ? g0 + 1 : gs + (r ^ 1));
        const double dL = dm + dmo, dF = pfL2 - v.nrm;
        double tmp = dF / dL;
        if (tmp > 0.0) bits |= WB_GAIN;
        tmp = 1.0 - cube(2 * tmp - 1.);
        muNext = myMu * ((tmp >= 0.3333333333333334) ? tmp : 0.3333333333333334);
      }
      flip ^= 1;
      q = slots[own][flip];
      if (real) {
        WSlot& o = q[grp];
        const int k = odd ? 1 : 0;
        if (r < 2) { o.f[k] = v.fxy; o.a[k] = v.pxy; }
        else if (r < 4) o.b[k] = v.pxy;
        if (r == 0) { o.f[2] = v.fz; o.a[2] = v.pz; o.nrm = v.nrm; o.sep = v.sep; }
        if (r == 1) { o.c[0] = v.c.x; o.c[1] = v.c.y; o.c[2] = v.c.z; }
        if (r == 2) o.b[2] = v.pz;
        if (r == 3) { o.D0 = D0; o.D1 = D1; o.t0 = t0; o.t1 = t1; }
        if (r == 4) { o.mu = muNext; o.bits = bits; }
      }
      join();
      rounds++;
    };
    for (;;) {   // one lmder2 call
      touching = true;
      bool stopFlag = false;
      int stop, k = 0, nu = 2;
      double mu = 0, Dp0 = 1e-7, Dp1 = 1e-7, pfL2;
      D3 pf;
      double diag0 = 0, diag1 = 0, j01 = 0, jt0 = 0, jt1 = 0;
      int last = 0, base = 0;       // the group whose evaluation was consumed last; the accepted point's group
      int probe0 = 1, probe1 = 2;   // the groups of the accepted point's probes
      double muRej = 0;             // damping below which trials were last rejected
      bool more;
      // the accepted point of group `base`, then the top of lmder2's loop (lmOuter)
      auto outer = [&]() {
        const WSlot& o = q[base];
        pf = d3(o.f[0], o.f[1], o.f[2]);
        pfL2 = o.nrm;
        if (!(k < 50 && !stop)) { if (k >= 50) stop = 3; return false; }
        if (pfL2 <= 1e-20) { stop = 6; return false; }
        if (stopFlag) { stop = 9; touching = false; return false; }
        contact = d3(o.c[0], o.c[1], o.c[2]);
        if (angleTest(o.sep, pfL2, contact)) { stop = 8; return false; }
        return true;
      };
      auto end = [&](int code) { stop = code; k++; if (k >= 50) stop = 3; };
      if (resume) {
        stopFlag = w.stopFlag; stop = 0; k = w.k; nu = w.nu; mu = w.mu;
        pf = w.pf; pfL2 = w.pfL2;
        diag0 = w.diag0; diag1 = w.diag1; j01 = w.j01; jt0 = w.jt0; jt1 = w.jt1;
        more = true;
      } else {
        // the start point and its two probes
        round(grp == 1 ? p0 + Dp0 : p0, grp == 2 ? p1 + Dp1 : p1, false, 0, 0, 0, 0, 0, 0, 0, 0, 0u);
        ev64 += 3;
        if (q[0].bits & WB_APART) stopFlag = true;
        stop = isfinite(q[0].nrm) ? 0 : 7;
        more = outer();
      }
      while (more) {
        if (!resume) {
          // the two probes at the accepted point: Jacobian and normal equations
          last = probe1;
          if ((q[probe0].bits | q[probe1].bits) & WB_APART) stopFlag = true;
          const int pc = lane % 3, pj = (lane / 3) & 1;   // lanes 0-5: component pc of column pj
          const double f0c = pc == 0 ? pf.x : pc == 1 ? pf.y : pf.z;
          const double J = (q[pj ? probe1 : probe0].f[pc] - f0c) / (pj ? Dp1 : Dp0);
          // lane 3 m + pc: product m of component pc: J0 J0, J0 J1, J1 J1, J0 (-f0), J1 (-f0)
          const int pm = lane / 3;
          const double Ja = __shfl_sync(FULL, J, ((pm == 2 || pm == 4) ? 3 : 0) + pc);
          const double Jb = __shfl_sync(FULL, J, (pm == 0 ? 0 : 3) + pc);
          const double pr = Ja * (pm >= 3 ? -1.0 * f0c : Jb);
          // sums x + (y + z) of product `lane` on lanes 0-4
          const int sm = 3 * (lane < 5 ? lane : 0);
          const double sx = __shfl_sync(FULL, pr, sm), sy = __shfl_sync(FULL, pr, sm + 1), sz = __shfl_sync(FULL, pr, sm + 2);
          const double sum = sx + (sy + sz);
          diag0 = __shfl_sync(FULL, sum, 0); j01 = __shfl_sync(FULL, sum, 1); diag1 = __shfl_sync(FULL, sum, 2);
          jt0 = __shfl_sync(FULL, sum, 3); jt1 = __shfl_sync(FULL, sum, 4);
          const double jinf = (fabs(jt0) > fabs(jt1) ? fabs(jt0) : fabs(jt1));
          if (jinf <= 1e-15) { stop = 1; break; }
          if (k == 0) mu = 1.0 * (diag0 > diag1 ? diag0 : diag1);
        }
        more = false;
        resume = false;
        for (;;) {   // damping loop: the step for mu, and those that follow its rejections
          const int plan = wsPlan<W>(mu, muRej, nu);
          const int trial = real ? wsTrial(plan, grp) : 0, role = wsRole(plan, grp);
          const int trials = wsTrials<W>(plan);
          double myMu = mu;
          for (int j = 0, m = nu; j < trial; j++, m = (int)((unsigned)m << 1)) myMu *= m;
          const double bo = (odd ? diag0 : diag1) + myMu, bx = (odd ? diag1 : diag0) + myMu;   // even lanes: Dp0, odd lanes: Dp1
          const double n_a = bo * bx - j01 * j01;
          const double D = ((odd ? jt1 : jt0) * bo - (odd ? jt0 : jt1) * j01) / n_a;
          const double D0 = __shfl_sync(FULL, D, gs), D1 = __shfl_sync(FULL, D, gs + 1);
          const double DL2 = sqrt(D0 * D0 + D1 * D1);
          const bool small = DL2 < 1e-5;
          // stop 4 compares with (|p| + 1e-3) / 1e-24, which is above 1e20
          bool huge = false;
          if (!(DL2 < 1e20)) huge = DL2 >= (sqrt(p0 * p0 + p1 * p1) + 1e-3) / (1e-12 * 1e-12);
          const unsigned smallB = __ballot_sync(FULL, small), hugeB = __ballot_sync(FULL, huge);
          if (smallB >> 30) { end(2); break; }   // lanes 30, 31: trial 0
          if (hugeB >> 30) { end(4); break; }
          const double t0 = p0 + D0, t1 = p1 + D1;
          round(role == 1 ? t0 + D0 : t0, role == 2 ? t1 + D1 : t1, true, D0, D1, t0, t1, myMu, pfL2, jt0, jt1,
                (small ? WB_SMALL : 0u) | (huge ? WB_HUGE : 0u));
          ev64 += WS_POINTS * W;
          bool ended = false, accepted = false;
          for (int a = 0; a < trials; a++) {
            const int g = wsGroup(plan, a);
            const WSlot& o = q[g];
            if (a > 0 && (o.bits & (WB_SMALL | WB_HUGE))) {   // the step after the last rejection ends the call
              end((o.bits & WB_SMALL) ? 2 : 4);
              ended = true;
              break;
            }
            last = g;
            if (o.bits & WB_APART) stopFlag = true;
            if (!(o.bits & WB_FINITE)) { end(7); ended = true; break; }
            if (o.bits & WB_GAIN) {
              base = g;
              if (mu <= muRej) muRej = 0.5 * mu;
              mu = o.mu;
              nu = 2;
              Dp0 = o.D0; Dp1 = o.D1;
              p0 = o.t0; p1 = o.t1;
              k++;
              more = outer();
              accepted = true;
              // the probes at the accepted trial: in this round's groups, or a round of their own
              const bool have = wsProbed(plan, a);
              probe0 = have ? g + 1 : 0; probe1 = have ? g + 2 : 1;
              if (more && !have) {
                round(grp == 0 ? p0 + Dp0 : p0, grp == 1 ? p1 + Dp1 : p1, false, 0, 0, 0, 0, 0, 0, 0, 0, 0u);
                ev64 += 2;
              }
              break;
            }
            muRej = mu;
            mu *= nu;
            const int nn = (int)((unsigned)nu << 1);
            if (nn <= nu) { end(5); ended = true; break; }
            nu = nn;
          }
          if (ended || accepted) break;
        }
      }
      P1 = d3(q[last].a[0], q[last].a[1], q[last].a[2]);
      P2 = d3(q[last].b[0], q[last].b[1], q[last].b[2]);
      // the restart rules of Superquadrics_Ig2.cpp:2013-2053
      bool again = false;
      for (;;) {
        calls++; iters += k; maxit += (stop == 3);
        bool restart = false;
        if (phase == 0) {
          phase = 1;
          if ((isnan(p0) || isnan(p1) || 7 == stop) && touching) restart = true;
        }
        if (!restart) {
          if (phase == 1) {
            phase = 3;
            const double rmaxA = __shfl_sync(FULL, s.rmax, 0);
            if (touching && 10.0 * nrm(P2 - P1) > rmaxA) {
              // isInside (Superquadrics.cpp:103-108) of the other body's point, each body on its lanes
              SqShape b;
              b.rx = s.rx; b.ry = s.ry; b.rz = s.rz; b.e1 = s.e1; b.e2 = s.e2;
              for (int i = 0; i < 9; i++) b.R.m[i] = s.R[i];
              const D3 rel = (bodyB ? P1 : P2) - s.pos;
              const int fast = insideFast(b, rel);
              const bool mine = __any_sync(FULL, fast < 0) ? isInside(b, rel) : fast == 1;
              const unsigned in = __ballot_sync(FULL, mine);
              if (!(in & 1u) || !(in & 4u)) { phase = 2; restart = true; }
            }
          } else phase = 3;
        }
        if (!restart) break;
        if (!fromCenter) { centre(); fromCenter = true; again = true; break; }
        // a restart from the centre line that the call just ended started from: the same
        // computation, counted as run
      }
      if (!again) break;
    }
    if (threadIdx.x == (W == 1 ? threadIdx.x & ~31 : 0))
      finishSearch(d, e, fl, id1, id2, isNew, p0, p1, touching, P1, P2, contact, calls, iters, maxit, cnt);
    roundsMax = max(roundsMax, rounds);
  }
  flushCounters(d, cnt);
  if (lane == 0 && (W == 1 || wib == 0) && roundsMax) {
    atomicAdd(&d.S->err[E_EVAL64], ev64);
    atomicMax(&d.S->err[E_ROUNDS_MAX], (unsigned long long)roundsMax);
  }
}
