// Which points a round of k_search_warp evaluates: the pending trial of lmder2's damping loop, the
// trials its rejections lead to, and probes.  A search on W warps has 6 W groups of lanes, one point
// each.  plan 0: trials with their two probes each, three groups a trial; plan 2 (W = 1): trials 0
// and 1 alone, 2 with its probes, 3 alone.
#pragma once

#define WS_HD __host__ __device__ __forceinline__

// A slow search divides mu by at most three at every accepted trial, until trials are rejected (two to
// five in a row, mu times 2, 4, 8 ...) and mu is above the level again below which it was rejected
// last, muRej, which moves little (to half the mu of a trial accepted at or below it).  So mu > muRej / 3
// and of the trials mu, 2 mu, 8 mu at most the first two are not above the level: the first above it is
// the one likely to be accepted, whose probes are worth evaluating.
template <int W> WS_HD int wsPlan(double mu, double muRej, int nu) { return W == 1 && mu <= muRej && mu * nu <= muRej ? 2 : 0; }
// consecutive trials a round holds
template <int W> WS_HD int wsTrials(int plan) { return plan == 0 ? 2 * W : 4; }
// the trial group grp belongs to, and its point: 0 the trial itself, 1 and 2 its probes
WS_HD int wsTrial(int plan, int grp) { return plan == 0 ? grp / 3 : grp < 2 ? grp : grp < 5 ? 2 : 3; }
WS_HD int wsRole(int plan, int grp) { return plan == 0 ? grp % 3 : grp == 3 || grp == 4 ? grp - 2 : 0; }
// the group of trial a's own point; whether the two groups after it hold its probes
WS_HD int wsGroup(int plan, int a) { return plan == 0 ? 3 * a : a == 3 ? 5 : a; }
WS_HD bool wsProbed(int plan, int a) { return plan == 0 || a == 2; }
