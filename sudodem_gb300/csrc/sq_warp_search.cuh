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

// What a round leaves in the lanes of each point's group.
struct WEval {
  double pxy, pz;    // support point of the lane's body: x (k = 0) or y (k = 1), and z
  double fxy, fz;    // p2 - p1: x (k = 0) or y (k = 1), and z
  double sep, nrm;   // c . (p2 - p1), |p2 - p1|
  D3 c;              // contact direction at the point
};

// g0: first lane of the group, r: the lane's place in it (0, 1: body A; 2, 3: body B; 4: v of both)
__device__ __forceinline__ void warpEval(const WShape& s, double e1B, int g0, int r, double q0, double q1, WEval& o) {
  const unsigned FULL = 0xffffffffu;
  const bool isB = r == 2 || r == 3, k = r == 1 || r == 3, extra = r == 4;
  const int mate = extra ? g0 + 1 : g0 + (r ^ 1);
  double sv, cv;
  sincos(k ? q1 : q0, &sv, &cv);
  const double sa0 = __shfl_sync(FULL, sv, g0), ca0 = __shfl_sync(FULL, cv, g0);
  const double sa1 = __shfl_sync(FULL, sv, g0 + 1), ca1 = __shfl_sync(FULL, cv, g0 + 1);
  o.c = d3(ca0 * ca1, sa0 * ca1, sa1);
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

// Work lists: which entries a launch takes, in this order.
//   WS_LONG      the long-search queue (fbQueue): 64+ iterations at the last step, then 32-63
//   WS_DEFERRED  the searches the mixed form's double-float kernels deferred (deferQueue)
//   WS_ALL       the long-search queue, then the main queue (lmQueue), longest first
//   WS_TAIL      the searches left after `rounds` rounds of k_wave_trial / k_wave_probe, from there on
enum { WS_LONG = 0, WS_DEFERRED = 1, WS_ALL = 2, WS_TAIL = 3 };

// Blocks go to the SMs in turn, so that in blocks of one warp fewer searches than warps have an SM's
// FP64 pipes to themselves (64 cycles an instruction, 76 with four busy schedulers).
__global__ void __launch_bounds__(LM_BS, 3) k_search_warp(Dev d, int mode, int waveRounds) {
  const unsigned FULL = 0xffffffffu;
  const SceneState& S = *d.S;
  const int lane = threadIdx.x & 31;
  const int grp = lane < WS_LANES * WS_POINTS ? lane / WS_LANES : 0;
  const int g0 = grp * WS_LANES;
  const int r = lane < WS_LANES * WS_POINTS ? lane - g0 : lane - WS_LANES * WS_POINTS;   // lanes 30, 31 mirror 0, 1
  const bool odd = r == 1 || r == 3;
  const int nLong1 = S.vlCount, nLong = mode == WS_DEFERRED ? 0 : S.vlCount + d.Q->vl2Count;
  const int nFront = S.lmCount;
  const int total = mode == WS_LONG       ? nLong
                    : mode == WS_DEFERRED ? S.fbCount
                    : mode == WS_TAIL     ? d.Q->nT[waveRounds]
                                          : nLong + S.lmCount + S.nmShort;
  int* head = mode == WS_DEFERRED ? &d.S->fbHead : mode == WS_TAIL ? &d.Q->tailHead : &d.S->vlHead;
  if ((int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) >= total) return;
  Counters cnt = {0, 0, 0, 0, 0};
  unsigned long long ev64 = 0;
  unsigned roundsMax = 0;
  for (;;) {
    int idx = 0;
    if (lane == 0) idx = atomicAdd(head, 1);
    idx = __shfl_sync(FULL, idx, 0);
    if (idx >= total) break;
    int e;
    WaveState w;
    bool resume = false;   // the call goes on at the pending trial
    if (mode == WS_TAIL) {
      waveLoad(d, ((waveRounds & 1) ? d.waveT1 : d.waveT0)[idx], w);
      e = w.e;
      resume = !w.init;
    } else if (mode == WS_DEFERRED) e = d.deferQueue[idx];
    else if (idx < nLong) e = idx < nLong1 ? d.fbQueue[idx] : d.fbQueue[d.Pcap - 1 - (idx - nLong1)];
    else { const int j = idx - nLong; e = j < nFront ? d.lmQueue[j] : d.lmQueue[d.qCap - 1 - (j - nFront)]; }
    // start of Ig2_Superquadrics_Superquadrics_SuperquadricsGeom::go up to lmder2
    const unsigned fl = d.A.flags[e];
    int id1, id2;
    entryIds(d, e, fl, id1, id2);
    const bool bodyB = r == 2 || r == 3;
    WShape s;
    {
      const int b = bodyB ? id2 : id1;
      const double4 a = d.shpA[b], x = d.shpB[b], q = d.ori[b];
      s.rx = a.x; s.ry = a.y; s.rz = a.z; s.rmax = a.w; s.e1 = x.x; s.e2 = x.y;
      s.a1 = 2. - x.x; s.i1 = 1 / (2. - x.x); s.i2 = 1 / (2. - x.y);
      const Rot R = quatToRot(q.x, q.y, q.z, q.w);
      for (int i = 0; i < 9; i++) s.R[i] = R.m[i];
      s.pos = xyz(d.pos[b]);
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
    if (mode == WS_TAIL) { contact = w.contact; phase = (int)w.phase; calls = w.calls; iters = w.iters; maxit = w.maxit; }
    for (;;) {   // one lmder2 call
      touching = true;
      bool stopFlag = false;
      int stop, k = 0, nu = 2;
      double mu = 0, Dp0 = 1e-7, Dp1 = 1e-7, pfL2;
      D3 pf;
      WEval v = {};
      double diag0 = 0, diag1 = 0, j01 = 0, jt0 = 0, jt1 = 0;
      unsigned sepPos = 0;   // bit of a group's first lane: its stop predicate
      int last = 0, base = 0;       // the group whose evaluation was consumed last; the accepted point's group
      int probe0 = 1, probe1 = 2;   // the groups of the accepted point's probes
      double muRej = 0;             // damping below which trials were last rejected
      bool more;
      // the accepted point of group `base`, then the top of lmder2's loop (lmOuter)
      auto outer = [&]() {
        if (!(k < 50 && !stop)) { if (k >= 50) stop = 3; return false; }
        if (pfL2 <= 1e-20) { stop = 6; return false; }
        if (stopFlag) { stop = 9; touching = false; return false; }
        const int l = base * WS_LANES;
        contact = d3(__shfl_sync(FULL, v.c.x, l), __shfl_sync(FULL, v.c.y, l), __shfl_sync(FULL, v.c.z, l));
        if (angleTest(__shfl_sync(FULL, v.sep, l), pfL2, contact)) { stop = 8; return false; }
        return true;
      };
      auto accept = [&]() {
        const int l = base * WS_LANES;
        pf = d3(__shfl_sync(FULL, v.fxy, l), __shfl_sync(FULL, v.fxy, l + 1), __shfl_sync(FULL, v.fz, l));
        pfL2 = __shfl_sync(FULL, v.nrm, l);
      };
      if (resume) {
        stopFlag = w.stopFlag; stop = 0; k = w.k; nu = w.nu; mu = w.mu;
        pf = w.pf; pfL2 = w.pfL2;
        diag0 = w.diag0; diag1 = w.diag1; j01 = w.j01; jt0 = w.jt0; jt1 = w.jt1;
        more = true;
      } else {
        // the start point and its two probes
        warpEval(s, e1B, g0, r, grp == 1 ? p0 + Dp0 : p0, grp == 2 ? p1 + Dp1 : p1, v);
        rounds++;
        ev64 += 3;
        sepPos = __ballot_sync(FULL, v.sep > 0);
        accept();
        if (sepPos & 1u) stopFlag = true;
        stop = isfinite(pfL2) ? 0 : 7;
        more = outer();
      }
      while (more) {
        if (!resume) {
          // the two probes at the accepted point: Jacobian and normal equations
          last = probe1;
          if (((sepPos >> (probe0 * WS_LANES)) | (sepPos >> (probe1 * WS_LANES))) & 1u) stopFlag = true;
          const int pc = lane % 3, pj = (lane / 3) & 1;   // lanes 0-5: component pc of column pj
          const int src = (pj ? probe1 : probe0) * WS_LANES;
          const double fx = __shfl_sync(FULL, v.fxy, pc == 1 ? src + 1 : src), fz = __shfl_sync(FULL, v.fz, src);
          const double f0c = pc == 0 ? pf.x : pc == 1 ? pf.y : pf.z;
          const double J = ((pc == 2 ? fz : fx) - f0c) / (pj ? Dp1 : Dp0);
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
          more = false;
          if (jinf <= 1e-15) { stop = 1; break; }
          if (k == 0) mu = 1.0 * (diag0 > diag1 ? diag0 : diag1);
        }
        more = false;
        resume = false;
        for (;;) {   // damping loop: the step for mu, and those that follow its rejections
          // A slow search divides mu by three at every accepted trial, until trials are rejected
          // (two to five in a row, mu times 2, 4, 8 ...) and mu is above the level again below which
          // it was rejected last, muRej, which moves little: so the trials up to the first above
          // that level take a group each, and that one's probes two more.  plan: the trial whose
          // probes are evaluated with it (0: those of trials 0 and 1; 4: none).
          // group's trial and role (0: the trial point, 1 and 2: its probes)
          int rej = 0;
          for (double m = mu; rej < 4 && m <= muRej; rej++) m *= (double)(2 << rej) * 0.5 * nu;
          const int plan = rej < 2 ? 0 : rej;
          const int trial = plan == 0 ? grp / 3 : plan == 2 ? (grp < 2 ? grp : grp < 5 ? 2 : 3) : plan == 3 ? min(grp, 3) : grp;
          const int role = plan == 0 ? grp % 3 : plan == 4 ? 0 : max(0, min(2, grp - plan)) * (grp < plan + 3 ? 1 : 0);
          const int trials = plan == 0 ? 2 : plan == 4 ? WS_POINTS : 4;
          double myMu = mu;
          for (int j = 0, m = nu; j < trial; j++, m = (int)((unsigned)m << 1)) myMu *= m;
          const double bo = (odd ? diag0 : diag1) + myMu, bx = (odd ? diag1 : diag0) + myMu;   // even lanes: Dp0, odd lanes: Dp1
          const double n_a = bo * bx - j01 * j01;
          const double D = ((odd ? jt1 : jt0) * bo - (odd ? jt0 : jt1) * j01) / n_a;
          const double D0 = __shfl_sync(FULL, D, g0), D1 = __shfl_sync(FULL, D, g0 + 1);
          const double DL2 = sqrt(D0 * D0 + D1 * D1);
          const bool small = DL2 < 1e-5;
          // stop 4 compares with (|p| + 1e-3) / 1e-24, which is above 1e20
          bool huge = false;
          if (!(DL2 < 1e20)) huge = DL2 >= (sqrt(p0 * p0 + p1 * p1) + 1e-3) / (1e-12 * 1e-12);
          const unsigned smallB = __ballot_sync(FULL, small), hugeB = __ballot_sync(FULL, huge);
          if (smallB & 1u) { stop = 2; k++; if (k >= 50) stop = 3; break; }
          if (hugeB & 1u) { stop = 4; k++; if (k >= 50) stop = 3; break; }
          const double t0 = p0 + D0, t1 = p1 + D1;
          warpEval(s, e1B, g0, r, role == 1 ? t0 + D0 : t0, role == 2 ? t1 + D1 : t1, v);
          rounds++;
          ev64 += WS_POINTS;
          // gain ratio and damping update of each group's trial
          const double dm = (odd ? D1 : D0) * (myMu * (odd ? D1 : D0) + (odd ? jt1 : jt0));
          const double dmo = __shfl_sync(FULL, dm, r == 4 ? g0 + 1 : g0 + (r ^ 1));
          const double dL = dm + dmo;
          const double dF = pfL2 - v.nrm;
          double tmp = dF / dL;
          const unsigned gain = __ballot_sync(FULL, tmp > 0.0);
          tmp = 1.0 - cube(2 * tmp - 1.);
          const double muNext = myMu * ((tmp >= 0.3333333333333334) ? tmp : 0.3333333333333334);
          const unsigned fin = __ballot_sync(FULL, isfinite(v.nrm));
          sepPos = __ballot_sync(FULL, v.sep > 0);
          bool ended = false, taken = false;
          for (int a = 0; a < trials; a++) {
            const int g = plan == 0 ? 3 * a : plan == 2 && a == 3 ? 5 : a, l = g * WS_LANES;
            if (a > 0) {   // the step after the last rejection ends the call
              const bool sm = (smallB >> l) & 1u, hu = (hugeB >> l) & 1u;
              if (sm || hu) { stop = sm ? 2 : 4; k++; if (k >= 50) stop = 3; ended = true; break; }
            }
            last = g;
            if ((sepPos >> l) & 1u) stopFlag = true;
            if (!((fin >> l) & 1u)) { stop = 7; k++; if (k >= 50) stop = 3; ended = true; break; }
            if ((gain >> l) & 1u) {
              base = g;
              const double myAcc = mu;
              mu = __shfl_sync(FULL, muNext, l);
              nu = 2;
              Dp0 = __shfl_sync(FULL, D0, l); Dp1 = __shfl_sync(FULL, D1, l);
              p0 = __shfl_sync(FULL, t0, l); p1 = __shfl_sync(FULL, t1, l);
              accept();
              k++;
              more = outer();
              taken = true;
              // the probes at the accepted trial: in this round's groups, or a round of their own
              const bool have = plan == 0 || a == plan;
              probe0 = have ? g + 1 : 0; probe1 = have ? g + 2 : 1;
              if (more && !have) {
                warpEval(s, e1B, g0, r, grp == 0 ? p0 + Dp0 : p0, grp == 1 ? p1 + Dp1 : p1, v);
                rounds++;
                ev64 += 2;
                sepPos = __ballot_sync(FULL, v.sep > 0);
              }
              if (myAcc <= muRej) muRej = 0.5 * myAcc;
              break;
            }
            muRej = mu;
            mu *= nu;
            const int nn = (int)((unsigned)nu << 1);
            if (nn <= nu) { stop = 5; k++; if (k >= 50) stop = 3; ended = true; break; }
            nu = nn;
          }
          if (ended || taken) break;
        }
      }
      {
        const int l = last * WS_LANES;
        P1 = d3(__shfl_sync(FULL, v.pxy, l), __shfl_sync(FULL, v.pxy, l + 1), __shfl_sync(FULL, v.pz, l));
        P2 = d3(__shfl_sync(FULL, v.pxy, l + 2), __shfl_sync(FULL, v.pxy, l + 3), __shfl_sync(FULL, v.pz, l + 2));
      }
      // the restart rules of Superquadrics_Ig2.cpp:2013-2053 (as lmCallEnd)
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
              SqShape q;
              q.rx = s.rx; q.ry = s.ry; q.rz = s.rz; q.e1 = s.e1; q.e2 = s.e2;
              for (int i = 0; i < 9; i++) q.R.m[i] = s.R[i];
              const D3 rel = (bodyB ? P1 : P2) - s.pos;
              const int fast = insideFast(q, rel);
              const bool mine = __any_sync(FULL, fast < 0) ? isInside(q, rel) : fast == 1;
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
    if (lane == 0)
      finishSearch(d, e, fl, id1, id2, isNew, p0, p1, touching, P1, P2, contact, calls, iters, maxit, cnt);
    roundsMax = max(roundsMax, rounds);
  }
  flushCounters(d, cnt);
  if (lane == 0 && roundsMax) {
    atomicAdd(&d.S->err[E_EVAL64], ev64);
    atomicMax(&d.S->err[E_ROUNDS_MAX], (unsigned long long)roundsMax);
  }
}
