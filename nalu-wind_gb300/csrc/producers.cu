// Input producers of the edge assembly, on the GPU: the per-edge mass flow
// rate (MdotEdgeAlg), the edge-based nodal gradient (NodalGradEdgeAlg with a
// lumped boundary closure) and the per-edge Peclet factor
// (MomentumEdgePecletAlg). They run every nonlinear iteration just before
// the assembly and use the same edge list and incidence lists as the
// handle they are called on; like the assembly kernels they evaluate FP64
// formulas in float-float arithmetic (dd.h) and sum without atomics.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "dd.h"
#include "nw_capi.h"
#include "nw_internal.h"

namespace nw {
namespace {

constexpr int kThreads = 256;
inline unsigned grid_for(int64_t n) { return unsigned((n + kThreads - 1) / kThreads); }

__device__ __forceinline__ dd ldd(const double* p) { return dd_from_double(*p); }

// MdotEdgeAlg::execute (src/ngp_algorithms/MdotEdgeAlg.C:117-190) without
// balanced forcing and GCL terms:
//   tmdot = -projTimeScale (p_R - p_L) |A|^2 / (A.dx)
//         + sum_d (interp rhoU_Ip + (1 - interp) rho_Ip u_Ip + G_Ip)_d A_d
//         - noc sum_d k_d G_Ip,d,   k = A - w dx,  w = |A|^2 / (A.dx)
// evaluated as -(p_R - p_L) w pts + rhoU . A + (1 - noc) G . A + noc w (dx . G):
// with the default noc = 1 the G . A terms cancel before they are formed.
//
// Bound by instruction issue: products stay in float pairs, but sums of FP64
// inputs and rho u are formed in FP64 (ten operations an edge on the
// otherwise idle pipe), each split once. NOC1, TOG1: noc = 1, interp = 1, whose
// terms with 1 - noc and 1 - interp are left out. It also waits for the gathers of
// two random nodes: twelve blocks of 128 (40 registers) took the four producers
// on 1,167,183 edges of tets from 144 us (four of 256) to 137.6; ten 138.2,
// fourteen 141.6. The terms with 1 - noc need 54
// registers, eight blocks: 3.2 M edges of hexes in row order take 109 us with the
// default factors, 127 with noc 0.3, 117 with interp 0.4 (176 for these two as one
// general form with twelve blocks; 152 for each before sums went to FP64).
constexpr int kMdotBlock = 128;
template <bool NOC1, bool TOG1>
__global__ void __launch_bounds__(kMdotBlock, NOC1 ? 12 : 8)
    mdot_k(int64_t E, const int2* __restrict__ edges, const double* __restrict__ coords,
           const double* __restrict__ velocity, const double* __restrict__ Gpdx,
           const double* __restrict__ density, const double* __restrict__ pressure,
           const double* __restrict__ udiag, const double* __restrict__ area, dd noc, dd om_noc,
           double interp, double om_interp, double* __restrict__ mdot) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const int2 lr = edges[e];
  const int64_t L = lr.x, R = lr.y;
  double rhoL = density[L], rhoR = density[R];
  if (!TOG1) {  // 2 (interp rhoU_Ip + (1 - interp) rho_Ip u_Ip) is linear in u_L and u_R
    const double h = om_interp * 0.5 * (rhoL + rhoR);
    rhoL = fma(interp, rhoL, h);
    rhoR = fma(interp, rhoR, h);
  }
  const dd iuL = dd_rcp_fast(ldd(udiag + L)), iuR = dd_rcp_fast(ldd(udiag + R));
  dd av[3], dx[3], m[3], g[3];  // m = 2 rhoU_Ip, g = 2 G_Ip
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    av[d] = dd_from_double_near_z(area[3 * e + d]);
    dx[d] = dd_from_double_z(coords[3 * R + d] - coords[3 * L + d]);
    const double uL = velocity[3 * L + d], uR = velocity[3 * R + d];
    m[d] = dd_from_double_near(fma(rhoR, uR, rhoL * uL));
    g[d] = ldd(Gpdx + 3 * R + d) * iuR + ldd(Gpdx + 3 * L + d) * iuL;
  }
  const dd asq = dd_dot3(av[0], av[0], av[1], av[1], av[2], av[2]);
  const dd axdx = dd_dot3(av[0], dx[0], av[1], dx[1], av[2], dx[2]);
  const dd w = asq * dd_rcp_fast(axdx);
  const dd ma = dd_dot3(m[0], av[0], m[1], av[1], m[2], av[2]);
  dd xg = dd_dot3(dx[0], g[0], dx[1], g[1], dx[2], g[2]);
  if (!NOC1) xg = noc * xg;
  // twice tmdot
  dd t = w * (xg - (iuL + iuR) * dd_from_double(pressure[R] - pressure[L])) + ma;
  if (!NOC1) t = om_noc * dd_dot3(g[0], av[0], g[1], av[1], g[2], av[2]) + t;
  mdot[e] = dd_to_double_int(scale2(t, 0.5f));
}

// acc += a b, renormalised: the product's head and error terms enter the pair
// sum unnormalised (15 operations against 18)
__device__ __forceinline__ void dd_mac(dd& acc, dd a, dd b) {
  const float p = fmul(a.hi, b.hi);
  float e = ffma(a.hi, b.hi, -p);
  e = ffma(a.hi, b.lo, e);
  e = ffma(a.lo, b.hi, e);
  const dd s = two_sum(acc.hi, p);
  acc = fast_two_sum(s.hi, fadd(s.lo, fadd(acc.lo, e)));
}

// NodalGradEdgeAlg::execute (src/ngp_algorithms/NodalGradEdgeAlg.C:85-109):
// grad_L += A phi_Ip / V_L, grad_R -= A phi_Ip / V_R, phi_Ip the edge
// midpoint average, plus bnd_area phi on exposed faces; periodic masters
// and slaves hold the sum. Thread per node row: its incident edges in
// order, then the row's nodes' boundary terms; the result goes to every
// node of the row.
//
// phi_L + phi_R is added in FP64 and split once (twice phi_Ip; the half is
// applied to 1 / V). A row's edges are a chain of three dependent loads each
// (incidence, edge, nodal values), hidden by many warps: 40 a SM or more
// measured better than two to four edges loaded together at fewer. 172,032
// nodes and 1,167,183 edges of tets: 68 -> 43 us (vector), 38 -> 25 (scalar);
// mdot above 58 -> 36, the Peclet factor below 28 -> 23, all with smaller
// errors against 64 bits (splits to the nearest pair).
template <int DIM1>
__global__ void __launch_bounds__(DIM1 == 3 ? 128 : kThreads, DIM1 == 3 ? 10 : 6)
    nodal_grad_k(int64_t R, const int32_t* __restrict__ inc_ptr, const uint32_t* __restrict__ inc,
                 const int2* __restrict__ edges, const int64_t* __restrict__ rn_ptr,
                 const int32_t* __restrict__ rn, const double* __restrict__ phi,
                 const double* __restrict__ area, const double* __restrict__ dualvol,
                 const double* __restrict__ bnd_area, double* __restrict__ grad) {
  const int64_t r = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (r >= R) return;
  dd acc[DIM1][3];
#pragma unroll
  for (int i = 0; i < DIM1; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) acc[i][j] = dd{0.f, 0.f};
  const int32_t end = inc_ptr[r + 1];
  for (int32_t q = inc_ptr[r]; q < end; ++q) {
    const uint32_t w = inc[q];
    const int64_t e = (w & 0x7fffffffu) >> 1;
    const int2 lr = edges[e];
    const uint32_t flip = (w & 1u) << 31;  // the right node's sum takes -A
    dd a[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      a[j] = dd_from_double_near_z(area[3 * e + j]);
      a[j] = dd{u2f(f2u(a[j].hi) ^ flip), u2f(f2u(a[j].lo) ^ flip)};
    }
#pragma unroll
    for (int i = 0; i < DIM1; ++i) {
      const dd p2 = dd_from_double_near(phi[int64_t(DIM1) * lr.x + i] + phi[int64_t(DIM1) * lr.y + i]);
#pragma unroll
      for (int j = 0; j < 3; ++j) dd_mac(acc[i][j], a[j], p2);
    }
  }
  const int64_t n0 = rn_ptr[r], n1 = rn_ptr[r + 1];
  if (bnd_area)
    for (int64_t k = n0; k < n1; ++k) {
      const int64_t nd = rn[k];
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const dd b = scale2(ldd(bnd_area + 3 * nd + j), 2.0f);
#pragma unroll
        for (int i = 0; i < DIM1; ++i) dd_mac(acc[i][j], b, ldd(phi + int64_t(DIM1) * nd + i));
      }
    }
  const dd iv = scale2(dd_rcp_fast(ldd(dualvol + rn[n0])), 0.5f);
  double out[DIM1 * 3];
#pragma unroll
  for (int i = 0; i < DIM1; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) out[3 * i + j] = dd_to_double_int(acc[i][j] * iv);
  for (int64_t k = n0; k < n1; ++k) {
    double* g = grad + int64_t(DIM1 * 3) * rn[k];
#pragma unroll
    for (int c = 0; c < DIM1 * 3; ++c) g[c] = out[c];
  }
}

// MomentumEdgePecletAlg::execute (src/edge_kernels/MomentumEdgePecletAlg.C:
// 74-101) with ClassicPecletFunction / TanhFunction (src/PecletFunction.C:
// 39-45, 66-71):
//   diff_Ip = 0.5 (mu_L / rho_L + mu_R / rho_R), udotx = 0.5 dx . (u_L + u_R)
//   Pe = |udotx| / (diff_Ip + eps),  f = (hf Pe)^2 / (5 + (hf Pe)^2)
//   or f = 0.5 (1 + tanh((Pe - c1) / c2))
__global__ void __launch_bounds__(kThreads)
    peclet_k(int64_t E, const int2* __restrict__ edges, const double* __restrict__ coords,
             const double* __restrict__ density, const double* __restrict__ viscosity,
             const double* __restrict__ vel, nw_peclet_opts o, dd hf, dd eps,
             double* __restrict__ pecnum, double* __restrict__ pecfac) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const int2 lr = edges[e];
  const int64_t L = lr.x, R = lr.y;
  const dd diffIp = scale2(ldd(viscosity + L) * dd_rcp_fast(ldd(density + L)) +
                               ldd(viscosity + R) * dd_rcp_fast(ldd(density + R)),
                           0.5f);
  dd dx[3], us[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    dx[d] = scale2(dd_from_double_near_z(coords[3 * R + d] - coords[3 * L + d]), 0.5f);
    // one FP64 addition and a split; with the tanh form, which fills the FP64
    // pipe, two splits and a pair addition
    us[d] = o.tanh_form ? ldd(vel + 3 * R + d) + ldd(vel + 3 * L + d)
                        : dd_from_double_near(vel[3 * R + d] + vel[3 * L + d]);
  }
  const dd udotx = dd_dot3(dx[0], us[0], dx[1], us[1], dx[2], us[2]);
  const dd pe = dd_abs(udotx) * dd_rcp_fast(diffIp + eps);
  if (pecnum) pecnum[e] = dd_to_double_int(pe);
  double f;
  if (o.tanh_form) {
    f = 0.50 * (1.0 + tanh((dd_to_double_int(pe) - o.tanh_trans) / o.tanh_width));
  } else {
    const dd m = hf * pe;
    const dd m2 = m * m;
    f = dd_to_double_int(m2 * dd_rcp_fast(m2 + 5.0f));
  }
  pecfac[e] = f;
}

template <typename F>
nw_status guard_call(F&& f) {
  try {
    f();
    return NW_OK;
  } catch (const Error& e) {
    set_last_error(e.msg);
    return e.status;
  } catch (const std::exception& e) {
    set_last_error(e.what());
    return NW_INTERNAL;
  }
}

}  // namespace
}  // namespace nw

using nw::dd;
using nw::dd_from_double;

extern "C" nw_status nw_compute_mdot_edges(nw_linsys* ls, const nw_continuity_fields* f,
                                           double noc_fac, double interp_together,
                                           double* mdot) {
  return nw::guard_call([&] {
    const nw::PlanView v = nw::plan_view(ls);
    if (!f || !mdot) nw::fail(NW_INVALID_ARG, "null argument");
    if (!f->coords || !f->velocity || !f->dpdx || !f->density || !f->pressure || !f->udiag ||
        !f->area)
      nw::fail(NW_INVALID_ARG, "null field pointer");
    if (v.num_edges == 0) return;
    auto go = [&](auto kernel) {
      kernel<<<unsigned((v.num_edges + nw::kMdotBlock - 1) / nw::kMdotBlock), nw::kMdotBlock, 0, v.stream>>>(
          v.num_edges, v.edges, f->coords, f->velocity, f->dpdx, f->density, f->pressure, f->udiag, f->area,
          dd_from_double(noc_fac), dd_from_double(1.0 - noc_fac), interp_together, 1.0 - interp_together, mdot);
    };
    if (noc_fac == 1.0)
      interp_together == 1.0 ? go(nw::mdot_k<true, true>) : go(nw::mdot_k<true, false>);
    else
      interp_together == 1.0 ? go(nw::mdot_k<false, true>) : go(nw::mdot_k<false, false>);
    NW_CUDA(cudaGetLastError());
  });
}

extern "C" nw_status nw_compute_nodal_gradient(nw_linsys* ls, int dim1, const double* phi,
                                               const double* area, const double* dualvol,
                                               const double* bnd_area, double* grad) {
  return nw::guard_call([&] {
    const nw::PlanView v = nw::plan_view(ls);
    if (!phi || !area || !dualvol || !grad) nw::fail(NW_INVALID_ARG, "null argument");
    if (dim1 != 1 && dim1 != 3) nw::fail(NW_INVALID_ARG, "dim1 must be 1 or 3");
    if (v.node_rows == 0) return;
    if (dim1 == 1)
      nw::nodal_grad_k<1><<<nw::grid_for(v.node_rows), nw::kThreads, 0, v.stream>>>(
          v.node_rows, v.inc_ptr, v.inc, v.edges, v.row_nodes_ptr, v.row_nodes, phi, area,
          dualvol, bnd_area, grad);
    else
      nw::nodal_grad_k<3><<<unsigned((v.node_rows + 127) / 128), 128, 0, v.stream>>>(
          v.node_rows, v.inc_ptr, v.inc, v.edges, v.row_nodes_ptr, v.row_nodes, phi, area,
          dualvol, bnd_area, grad);
    NW_CUDA(cudaGetLastError());
  });
}

extern "C" nw_status nw_compute_peclet_factor(nw_linsys* ls, const double* coords,
                                              const double* density, const double* viscosity,
                                              const double* velocity, const nw_peclet_opts* o,
                                              double* pecnum, double* pecfac) {
  return nw::guard_call([&] {
    const nw::PlanView v = nw::plan_view(ls);
    if (!coords || !density || !viscosity || !velocity || !o || !pecfac)
      nw::fail(NW_INVALID_ARG, "null argument");
    if (o->tanh_form && !(o->tanh_width != 0.0)) nw::fail(NW_INVALID_ARG, "tanh_width is zero");
    if (v.num_edges == 0) return;
    nw::peclet_k<<<nw::grid_for(v.num_edges), nw::kThreads, 0, v.stream>>>(
        v.num_edges, v.edges, coords, density, viscosity, velocity, *o,
        dd_from_double(o->hybrid_factor), dd_from_double(o->eps), pecnum, pecfac);
    NW_CUDA(cudaGetLastError());
  });
}
