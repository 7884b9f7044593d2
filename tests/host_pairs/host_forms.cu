// CPU check of the field points' choice of forms (test infrastructure): the
// elevation with the library's own field_forms(), on the host build of the
// field-point Green functions.
#include "host_pairs.cu"

extern "C" int host_forms_free_surface(int np, int nfa, int nsymy, const double* xyz, const int* m1234,
                                       const double* geo, double zer, const double* apd, double g, double depth,
                                       double period, int npts, const double* xy, int nprob, const double* zigb,
                                       const double* zigs, double* eta, int* finite_forms) {
  HostCtx h(np, nfa, nsymy, xyz, m1234, geo, zer, apd);
  OmegaParams om;
  const double W = 2. * kPI / period;
  int nq = 0;
  const int st = frequency_setup(W, g, depth, h.gm, &nq, om);
  if (st) return st;
  const bool fd = field_forms(om, W, g, depth);
  if (finite_forms) *finite_forms = fd;
  if (fd) free_surface<true>(h.gc, om, h.P, W, g, npts, xy, nprob, zigb, zigs, eta);
  else free_surface<false>(h.gc, om, h.P, W, g, npts, xy, nprob, zigb, zigs, eta);
  return h.status;
}
