// Host build of the restart rule's isInside and of its FP32 decision (test infrastructure only).
#include "../sudodem_gb300/csrc/sq_device.cuh"

using namespace sqdem;

// per row: rx ry rz eps1 eps2, quaternion (w x y z), point relative to the centre; fast: -1, 0, 1
extern "C" void inh_test(const double* rows12, long n, int* fast, int* exact) {
  for (long i = 0; i < n; i++) {
    const double* r = rows12 + 12 * i;
    SqShape s;
    shapeInit(s, r[0], r[1], r[2], r[3], r[4], 0);
    s.R = quatToRot(r[5], r[6], r[7], r[8]);
    const D3 p = d3(r[9], r[10], r[11]);
    fast[i] = insideFast(s, p);
    exact[i] = isInside(s, p) ? 1 : 0;
  }
}
