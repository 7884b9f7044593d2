// CPU check of the wave pass as it evaluates a pair of submerged panels (test
// infrastructure): wave_sym_pair(), the function that the kernel calls, in place
// of the separate parts that host_pairs.cu assembles from.
#include "host_pairs.cu"

namespace {

template <bool FD>
void assemble_in_order(const GreenCtx& g, const OmegaParams& om, const std::vector<PanelRec>& P, double* dp, double* dm,
                       double* sp, double* sm) {
  const int N = (int)P.size(), NJJ = g.nsymy + 1;
  auto entry = [&](int I, int J, const PairOut& o) {
    RealOut r;
    pair_rankine<FD>(g, om, om.ambda, om.ar, P[I].xg, P[I].yg, P[I].zg, P[I].xn, P[I].yn, P[I].zn, I == J, P[J], r);
    const long long q = I + (long long)N * J;
    put(dp, q, r.dp + o.dp_re, o.dp_im);
    put(sp, q, r.sp + o.sp_re, o.sp_im);
    put(dm, q, r.dm + o.dm_re, o.dm_im);
    put(sm, q, r.sm + o.sm_re, o.sm_im);
  };
  for (int J = 0; J < N; ++J)
    for (int I = 0; I <= J; ++I) {
      PairOut oij, oji;
      if (P[I].zg < g.zer && P[J].zg < g.zer) {
        if (!wave_sym_pair<FD>(g, om, P[I], P[J], NJJ, I != J, oij, oji)) set_status(g.status, ST_AKZ_UNDEFINED);
      } else {
        pair_wave_ordered<FD>(g, om, P[I], P[J], oij);
        if (I != J) pair_wave_ordered<FD>(g, om, P[J], P[I], oji);
      }
      entry(I, J, oij);
      if (I != J) entry(J, I, oji);
    }
}

}  // namespace

extern "C" int host_order_assemble(int np, int nfa, int nsymy, const double* xyz, const int* m1234, const double* geo,
                                   double zer, const double* apd, double g, double depth, double omega, int* nq_state,
                                   int* fd_mode, double* dp, double* dm, double* sp, double* sm) {
  HostCtx h(np, nfa, nsymy, xyz, m1234, geo, zer, apd);
  OmegaParams om;
  const double T = 2. * kPI / omega;
  const int st = frequency_setup(2. * kPI / T, g, depth, h.gm, nq_state, om);
  if (st) return st;
  if (om.fd) assemble_in_order<true>(h.gc, om, h.P, dp, dm, sp, sm);
  else assemble_in_order<false>(h.gc, om, h.P, dp, dm, sp, sm);
  if (!nsymy) {
    std::memcpy(dm, dp, sizeof(double) * 2 * (size_t)nfa * nfa);
    std::memcpy(sm, sp, sizeof(double) * 2 * (size_t)nfa * nfa);
  }
  if (fd_mode) *fd_mode = om.fd;
  return h.status;
}
