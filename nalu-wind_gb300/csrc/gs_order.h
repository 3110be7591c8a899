// Order in which a multicolour Gauss-Seidel sweep of a system with several
// rows a node visits the rows, one kernel a colour (gs_node_k, krylov.cu).
// Class (colour, d) holds row d of the colour's nodes; the order is that of
// the class-by-class sweep. Host-callable for the CPU test.
#pragma once

namespace nw {

constexpr int kMaxDof = 3;

// One kernel: the rows 0..dof-1 of its colour's nodes in the order seq, the
// first nfwd of them the forward sweep's.
struct GsNodePass {
  int colour = 0, nseq = 0, nfwd = 0;
  int seq[2 * kMaxDof] = {};
};

// sweep 0: symmetric, the class relaxed last by the forward sweep not
// repeated; 1: forward only; 2: backward only.
template <typename F>
void gs_node_passes(int ncol, int dof, int sweep, F run) {
  auto pass = [&](int c, bool forward, int back) {  // back: rows back-1..0, backward
    GsNodePass p;
    p.colour = c;
    if (forward)
      for (int d = 0; d < dof; ++d) p.seq[p.nseq++] = d;
    p.nfwd = p.nseq;
    for (int d = back - 1; d >= 0; --d) p.seq[p.nseq++] = d;
    run(p);
  };
  if (sweep != 2)
    for (int c = 0; c < ncol; ++c) pass(c, true, sweep == 0 && c == ncol - 1 ? dof - 1 : 0);
  if (sweep != 1)
    for (int c = sweep == 0 ? ncol - 2 : ncol - 1; c >= 0; --c) pass(c, false, dof);
}

}  // namespace nw
