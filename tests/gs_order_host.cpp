// Host build of the node sweeps' order (nalu-wind_gb300/csrc/gs_order.h) for
// tests/test_gs_order.py.
#include "gs_order.h"

// the classes colour * dof + d in the order visited; returns their number,
// fwd: how many of them belong to the forward sweep
extern "C" int gs_order(int ncol, int dof, int sweep, int* classes, int* fwd) {
  int n = 0;
  *fwd = 0;
  nw::gs_node_passes(ncol, dof, sweep, [&](const nw::GsNodePass& p) {
    for (int t = 0; t < p.nseq; ++t) classes[n++] = p.colour * dof + p.seq[t];
    *fwd += p.nfwd;
  });
  return n;
}
