// Host build of the warp search's plan of points (test infrastructure only).
#include "../sudodem_gb300/csrc/sq_warp_plan.cuh"

// out: plan, trials, then per group (trial, role), then per trial (group, probed)
template <int W> static void fill(double mu, double muRej, int nu, int* out) {
  const int plan = wsPlan<W>(mu, muRej, nu), trials = wsTrials<W>(plan);
  *out++ = plan; *out++ = trials;
  for (int g = 0; g < 6 * W; g++) { *out++ = wsTrial(plan, g); *out++ = wsRole(plan, g); }
  for (int a = 0; a < trials; a++) { *out++ = wsGroup(plan, a); *out++ = wsProbed(plan, a); }
}
extern "C" void wph_plan(int W, double mu, double muRej, int nu, int* out) {
  if (W == 1) fill<1>(mu, muRej, nu, out); else fill<2>(mu, muRej, nu, out);
}
