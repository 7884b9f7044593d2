// CPU check of the FP64 update's schedule (test infrastructure): the loads and both
// issuers' steps as oz_update_kernel takes them.
#include "../../nemoh_b200/csrc/oz_gemm.cuh"

using namespace nb200;

template <class P>
static void steps(const P& p, int phase, int*& out) {
  for (int k = 0; k < p.count; ++k) {
    const OzStep& t = p.s[k];
    const int v[] = {phase, t.i, t.j, t.slot_i, t.slot_j, t.acc, t.first, t.need, t.retire, t.full};
    for (int x : v) *out++ = x;
  }
}

template <int WHO>
static int plan(int* out) {
  using P = OzPlan<WHO>;
  int* o = out;
  steps(P::p0, 0, o);
  steps(P::p1, 1, o);
  steps(P::p2, 2, o);
  steps(P::p3, 3, o);
  return (int)(o - out) / 10;
}

// loads: OZ_LOADS x (slice, slot, chunk); issuer 0, 1: its steps, ten values each; returns their count
extern "C" int host_schedule_loads(int* loads) {
  for (int l = 0; l < OZ_LOADS; ++l)
    for (int k = 0; k < 3; ++k) loads[3 * l + k] = OZ_LOAD[l][k];
  return OZ_LOADS;
}
extern "C" int host_schedule_steps(int issuer, int* out) { return issuer ? plan<OZ_WHO1>(out) : plan<OZ_WHO0>(out); }
