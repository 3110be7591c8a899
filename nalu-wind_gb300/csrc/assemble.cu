// Edge assembly kernels for sm_103a.
//
// The reference computes each edge's local system in a Kokkos team lambda
// (include/AssembleEdgeSolverAlgorithm.h:47-100) and scatters it with FP64
// atomics (TpetraLinearSystem::sum_into, src/TpetraLinearSystem.C:
// 1381-1459), so its summation order is not reproducible on a GPU. Here
// assembly has deterministic phases and no floating-point atomics:
//
//  0. (continuity) node phase: one thread per node computes the node-only
//     factors every incident edge needs (1/udiag, rho u, grad p / udiag);
//  1. edge phase: one thread per edge evaluates the edge physics once and
//     writes its compact coefficients to an edge-major buffer (SoA);
//  2. row phase: one thread per node row walks the row's incident
//     (edge, side) list, sorted by column then edge, accumulates the
//     diagonal block and rhs in registers, stages the row's CSR values in
//     shared memory and the block writes its contiguous CSR range with
//     coalesced stores (or read-add-writes when the system already holds
//     values).
//
// GB300 issues FP64 at about 1/58 of its FP32 rate, so evaluated in FP64
// these kernels are bound by FP64 issue, not by HBM. The momentum and
// continuity kernels therefore evaluate the FP64 formulas in float-float
// arithmetic (dd.h: about 48 significant bits, error within a few 2^-48 of
// the operand magnitudes) on the FP32 pipes, split the FP64 inputs with
// integer operations, keep their edge coefficients as float pairs (8 bytes,
// the size of a double) and widen each finished CSR entry to FP64 once.
// The scalar kernel stays in FP64 (MUFU-seeded reciprocals). Node-only
// factors are computed once per node, and option branches are compile-time
// template parameters.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>

#include "assemble.h"
#include "schedule.h"
#include "dd.h"
#include "nw_internal.h"
#include "row_stage.h"

namespace nw {
namespace {

constexpr int kThreads = 256;
constexpr int kRow1Threads = 128;  // node rows per block, 1-dof row phase
constexpr int kMaxRowSmem = 96 * 1024;  // staging capacity limit per block
constexpr int kSmSmem = 228 * 1024;     // shared memory of a SM

// 1/x from the MUFU approximation (rcp.approx.ftz.f64) refined by a cubic
// step r(1 + e + e^2) and a Newton step r(1 + e), e = 1 - x r: five FP64
// operations. Zero, infinite and denormal inputs return the seed (inf, 0 or
// inf), tested on its bits: a comparison would be two more on the FP64 pipe.
__device__ __forceinline__ double fast_rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const uint32_t h = uint32_t(__double2hiint(r)) & 0x7fffffffu;
  if (h == 0u || h == 0x7ff00000u) return r;
  double e = fma(-x, r, 1.0);
  r = fma(r, fma(e, e, e), r);
  e = fma(-x, r, 1.0);
  return fma(r, e, r);
}

// van Leer limiter 2 (m p + |m p|) / ((m + p)^2 + eps): zero unless m p > 0
__device__ __forceinline__ double van_leer(double dqm, double dqp, double eps) {
  const double p = dqm * dqp, s = dqm + dqp;
  const double v = (4.0 * p) * fast_rcp(fma(s, s, eps));
  return __double_as_longlong(p) <= 0 ? 0.0 : v;  // p <= 0 on the integer pipe
}

// one 32-byte sector, aligned
__device__ __forceinline__ void st32(double* p, double a, double b, double c, double d) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}
// through the read-only path when the buffer is not written during the
// kernel (NC), else a plain load
template <bool NC>
__device__ __forceinline__ void ld32(const double* p, double (&x)[4]) {
  if constexpr (NC)
    asm volatile("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3])
                 : "l"(p));
  else
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3])
                 : "l"(p)
                 : "memory");
}

// ---------------------------------------------------------------------------
// Scalar advection-diffusion: ScalarEdgeSolverAlg::execute
// (src/edge_kernels/ScalarEdgeSolverAlg.C:85-205), in FP64. The local matrix
// is [-a10 w, a01; a10, -a01 w] with w = 1 / relax (the diagonal terms of the
// reference are the opposite off-diagonal ones relaxed) and the rhs
// (-flux, flux); one 32-byte record (a01, a10, flux, -) per edge.
//
// Bound by the FP64 pipe, 64 clocks of a scheduler's unit an instruction, so
// what counts is their number: node diffusivities mu / rho are divided once
// per node, 0.5 dx . grad q enters the non-orthogonal term through the two
// extrapolations, the classic Peclet function (h u)^2 / (5 d^2 + (h u)^2)
// takes one reciprocal for both of its divisions, the tanh form 0.5 (1 +
// tanh x) is 1 / (1 + exp(-2 x)), and with alpha = 0 (the default) only the
// upwind side is extrapolated and limited. 68 FP64 instructions an edge
// against 132 (classic), 104 against 196 (limiter and tanh): 476,280 nodes
// 576 -> 333 us with the row phase. Errors of the entries against extended
// precision (rms, 49 x 40 x 30 hexes, tanh and relax 0.7; 132 and 196
// instructions and now): downwind side 1.88e-16 and 1.59e-16, upwind side
// 8.5e-17 and 7.3e-17, diagonal 1.23e-16 and 1.20e-16.
struct ScalarArgs {
  double alpha, alpha_upw, om_alpha, om_alpha_upw, upw, h, c1, k2;  // h = hf / 2, k2 = -2 / c2
};

__global__ void __launch_bounds__(kThreads)
    scalar_node_k(int64_t N, const double* __restrict__ density, const double* __restrict__ dflux,
                  double* __restrict__ dor) {
  const int64_t n = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (n < N) dor[n] = dflux[n] * fast_rcp(density[n]);
}

// ALPHA: alpha != 0 (central part extrapolated on both sides). Blocks of 64
// spread the FP64 work evenly over the SMs: 346 -> 338 us on 476,280 nodes with
// limiter and tanh (blocks of 256 and 64).
constexpr int kScalarBlock = 64;
template <bool LIMITER, bool TANH, bool ALPHA, bool NODE>
__global__ void __launch_bounds__(kScalarBlock)
    scalar_edge_k(int64_t E, const int2* __restrict__ edges, const double* __restrict__ coords,
                  const double* __restrict__ vrtm, const double* __restrict__ q, const double* __restrict__ dqdx,
                  const double* __restrict__ dflux, const double* __restrict__ dor,
                  const double* __restrict__ area, const double* __restrict__ mdotA, ScalarArgs o,
                  double* __restrict__ buf) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= E) return;
  constexpr double eps = 1.0e-16;
  const int2 lr = edges[e];
  const int64_t L = lr.x, R = lr.y;
  const double mdot = mdotA[e], qL = q[L], qR = q[R];
  const bool up = __double_as_longlong(mdot) > 0;  // mdot > 0 on the integer pipe
  double asq = 0.0, axdx = 0.0, udx = 0.0, dL = 0.0, dR = 0.0, ag = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double av = area[3 * e + d], dx = coords[3 * R + d] - coords[3 * L + d];
    const double gL = dqdx[3 * L + d], gR = dqdx[3 * R + d];
    asq = d ? fma(av, av, asq) : av * av;
    axdx = d ? fma(av, dx, axdx) : av * dx;
    const double vs = vrtm[3 * R + d] + vrtm[3 * L + d];
    udx = d ? fma(dx, vs, udx) : dx * vs;
    dL = d ? fma(dx, gL, dL) : dx * gL;  // twice the left extrapolation
    dR = d ? fma(dx, gR, dR) : dx * gR;
    const double gs = gL + gR;
    ag = d ? fma(av, gs, ag) : av * gs;
  }
  const double w = asq * fast_rcp(axdx);
  const double visc = 0.5 * (dflux[L] + dflux[R]);
  // mu / rho: from the node pre-pass, or (small systems) here from rho
  const double dsum = NODE ? dor[L] + dor[R]
                           : __dadd_rn(__dmul_rn(dflux[L], fast_rcp(dor[L])), __dmul_rn(dflux[R], fast_rcp(dor[R])));
  double pec, om;  // Peclet function and one less it
  if (TANH) {
    const double pe = fabs(udx) * fast_rcp(dsum + 2.0 * eps);  // 0.5 |udx| over the mean diffusivity
    const double ex = exp((pe - o.c1) * o.k2);
    pec = fast_rcp(1.0 + ex);
    // as a product: a difference would lose what the rounding of 1 + ex lost.
    // ex may be infinite where pec is zero (tested on its bits)
    om = __double_as_longlong(pec) == 0 ? 1.0 : ex * pec;
  } else {
    const double den = fma(0.5, dsum, eps), u = o.h * udx, u2 = u * u;
    pec = u2 * fast_rcp(fma(5.0 * den, den, u2));
    om = 1.0 - pec;
  }
  const double dq = qR - qL, qIp = 0.5 * (qL + qR);
  // lhsfac dq + non-orthogonal correction -visc / 2 (A - w dx) . (gL + gR)
  const double lhsfac = -(visc * w);
  const double diff = fma(lhsfac, dq, -(0.5 * visc) * fma(-w, dL + dR, ag));
  // upwind value - mean of the upwind side
  const double half = 0.5 * o.upw;
  double qc = qIp, dU;
  if (!ALPHA) {
    const double dS = up ? dL : dR;
    double f = half * dS;
    if (LIMITER) f *= van_leer(fma(2.0, dS, -dq), dq, eps);
    dU = up ? (qL - qIp) + f : (qR - qIp) - f;
  } else {
    double fL = half * dL, fR = half * dR;
    if (LIMITER) {
      fL *= van_leer(fma(2.0, dL, -dq), dq, eps);
      fR *= van_leer(fma(2.0, dR, -dq), dq, eps);
    }
    const double qIpL = qL + fL, qIpR = qR - fR;
    dU = (up ? qIpL : qIpR) - qIp;
    qc = fma(o.alpha, 0.5 * (qIpL + qIpR), o.om_alpha * qIp);
  }
  // adv = mdot (pec (a_u q_upw + (1 - a_u) qIp) + (1 - pec) q_cds)
  const double pa = pec * o.alpha_upw;  // weight of the upwind deviation
  const double mp = mdot * pa, hm = 0.5 * mdot;
  double adv, a01, a10;
  if (!ALPHA) {
    adv = fma(mp, dU, mdot * qIp);
    if (TANH) {
      // downwind side mdot / 2 (1 - pec a_u), upwind side mdot / 2 (1 + pec a_u)
      const double sh = up ? hm : -hm;
      const double dw = fma(sh, fma(o.alpha_upw, om, o.om_alpha_upw), lhsfac);
      const double uw = lhsfac - fma(sh, pa, sh);
      a01 = up ? dw : uw;
      a10 = up ? uw : dw;
    } else {
      const double mc = fma(-hm, pa, hm);  // mdot / 2 (1 - pec a_u)
      a01 = lhsfac + mc;
      a10 = lhsfac - mc;
    }
  } else {
    adv = fma(mp, dU, mdot * fma(pec, qIp, om * qc));
    const double m0 = hm * o.alpha * om;
    const double mc = hm * fma(pec, o.om_alpha_upw, om * o.om_alpha);
    a01 = (lhsfac + mc) + m0;
    a10 = (lhsfac - mc) - m0;
  }
  if (!TANH || ALPHA) {
    if (up)
      a10 -= mp;
    else
      a01 += mp;
  }
  st32(buf + kScalarCoefs * e, a01, a10, diff + adv, 0.0);
}

// ---------------------------------------------------------------------------
// Continuity / pressure Poisson: ContinuityEdgeSolverAlg::execute
// (src/edge_kernels/ContinuityEdgeSolverAlg.C:109-194), no balanced buoyancy
// and no GCL term. The 2x2 local matrix is [-f, f; f, -f] with
// f = lhsfac, and the rhs is (-tmdot, tmdot); output per edge: f, tmdot.
//
// Fast form (rho u and rho_Ip u_Ip interpolated together, incompressible
// scaling off: the reference defaults): the node phase stores per node
//   n = (1/udiag, rho u_x, rho u_y, rho u_z, g_x, g_y, g_z, p),
//   g = (grad p) / udiag (the edge phase forms p_R - p_L from the FP64
//   pressures, like the coordinate differences),
// so that tmdot = -0.5 (n0_L + n0_R) (p_R - p_L) w
//               + sum_d [0.5 (m_R + m_L) + 0.5 (g_R + g_L)]_d A_d
//               - noc sum_d k_d 0.5 (g_R + g_L)_d,
// w = |A|^2 / (A.dx), k = A - w dx, then tmdot /= tau. This is the
// reference expression regrouped; the parity tests bound the difference by
// eps times the running magnitude of each entry.
//
// The edge phase is bound by its 580 instructions an edge (56 % of the issue
// slots) and the latency of two random records: 88 us on 128x128x64 hexes with
// 16-byte record loads and 4 resident blocks a SM. Records read as 32-byte
// loads and summed on arrival leave 40 registers, 1,536 threads a SM in blocks
// of 128: the whole assembly takes 145 us, 159 before (blocks of 256: four 158,
// five 150, six 147; blocks of 64 147; 32 registers 148.5). PLAIN: the default
// noc = 1 needs no product with it.
constexpr int kNodeStride = 8;  // dd slots (8 bytes each) per node

__device__ __forceinline__ dd ldd(const double* p) { return dd_from_double(*p); }
__device__ __forceinline__ void st4(dd* p, dd a, dd b, dd c, dd d) {
  float4* q = reinterpret_cast<float4*>(p);
  q[0] = make_float4(a.hi, a.lo, b.hi, b.lo);
  q[1] = make_float4(c.hi, c.lo, d.hi, d.lo);
}

// nodes [n0, n1)
__global__ void __launch_bounds__(kThreads)
    continuity_node_k(int64_t n0, int64_t n1, const double* __restrict__ velocity,
                      const double* __restrict__ Gpdx,
                      const double* __restrict__ density,
                      const double* __restrict__ pressure,
                      const double* __restrict__ udiag,
                      dd* __restrict__ nodebuf) {
  const int64_t n = n0 + int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (n >= n1) return;
  const dd iu = dd_rcp(ldd(udiag + n));
  const dd rho = ldd(density + n);
  dd* out = nodebuf + kNodeStride * n;
  st4(out, iu, rho * ldd(velocity + 3 * n), rho * ldd(velocity + 3 * n + 1),
      rho * ldd(velocity + 3 * n + 2));
  st4(out + 4, ldd(Gpdx + 3 * n) * iu, ldd(Gpdx + 3 * n + 1) * iu,
      ldd(Gpdx + 3 * n + 2) * iu, ldd(pressure + n));
}

constexpr int kContinuityBlock = 128;
struct ContinuityNodeFields {
  const double *velocity, *Gpdx, *density, *udiag;
};
template <bool PLAIN, bool NODE>
__global__ void __launch_bounds__(kContinuityBlock, NODE ? 12 : 8)
    continuity_edge_fast_k(int64_t E, const int2* __restrict__ edges,
                           const double* __restrict__ coords,
                           const dd* __restrict__ nodebuf,
                           const double* __restrict__ pressure,
                           const double* __restrict__ area, dd noc,
                           dd inv_tau, dd* __restrict__ buf, ContinuityNodeFields nf) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const int2 lr = edges[e];
  const int64_t L = lr.x, R = lr.y;
  // sums over the two nodes; a record is two 32-byte loads (four 16-byte
  // loads cost twice the L1 lookups)
  dd n[7];
  if constexpr (!NODE) {  // the two records formed here
    const dd iul = dd_rcp(ldd(nf.udiag + L)), iur = dd_rcp(ldd(nf.udiag + R));
    const dd rl = ldd(nf.density + L), rr = ldd(nf.density + R);
    n[0] = iul + iur;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      n[1 + d] = rl * ldd(nf.velocity + 3 * L + d) + rr * ldd(nf.velocity + 3 * R + d);
      n[4 + d] = ldd(nf.Gpdx + 3 * L + d) * iul + ldd(nf.Gpdx + 3 * R + d) * iur;
    }
  } else {
    double a[4], b[4];
    const double* pl = reinterpret_cast<const double*>(nodebuf + kNodeStride * L);
    const double* pr = reinterpret_cast<const double*>(nodebuf + kNodeStride * R);
    auto pair = [](double x) { return dd{__int_as_float(__double2loint(x)), __int_as_float(__double2hiint(x))}; };
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      ld32<true>(pl + 4 * h, a);
      ld32<true>(pr + 4 * h, b);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * h + k < 7) n[4 * h + k] = pair(a[k]) + pair(b[k]);
    }
  }
  dd av[3], dx[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    av[d] = dd_from_double_z(area[3 * e + d]);
    dx[d] = dd_from_double_z(coords[3 * R + d] - coords[3 * L + d]);
  }
  const dd asq = dd_dot3(av[0], av[0], av[1], av[1], av[2], av[2]);
  const dd axdx = dd_dot3(av[0], dx[0], av[1], dx[1], av[2], dx[2]);
  const dd w = asq * dd_rcp(axdx);
  const dd projTimeScale = scale2(n[0], 0.5f);
  dd mg[3], c[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    mg[d] = n[1 + d] + n[4 + d];
    c[d] = av[d] - w * dx[d];
  }
  // sum (rho u + G p / A_p) . A and the non-orthogonal correction
  // sum (A - w dx) . (G p / A_p), as three-term dots
  const dd flux = dd_dot3(mg[0], av[0], mg[1], av[1], mg[2], av[2]);
  dd corr = dd_dot3(c[0], n[4], c[1], n[5], c[2], n[6]);
  if (!PLAIN) corr = noc * corr;
  dd tmdot = -(projTimeScale * dd_from_double(pressure[R] - pressure[L]) * w);
  tmdot = (tmdot + scale2(flux - corr, 0.5f)) * inv_tau;
  const dd f = -(w * projTimeScale * inv_tau);
  reinterpret_cast<float4*>(buf)[e] = make_float4(f.hi, f.lo, tmdot.hi, tmdot.lo);
}

// General options (interpolation blend, incompressible density scaling).
struct ContinuityDD {
  dd noc, inv_tau, interp, om_interp, incomp, om_incomp;
};

__global__ void __launch_bounds__(kThreads)
    continuity_edge_k(int64_t E, const int2* __restrict__ edges,
                      const double* __restrict__ coords,
                      const double* __restrict__ velocity,
                      const double* __restrict__ Gpdx,
                      const double* __restrict__ density,
                      const double* __restrict__ pressure,
                      const double* __restrict__ udiag,
                      const double* __restrict__ area, ContinuityDD c,
                      dd* __restrict__ buf) {
  const int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= E) return;
  const int2 lr = edges[e];
  const int64_t L = lr.x, R = lr.y;
  const dd iuL = dd_rcp(ldd(udiag + L)), iuR = dd_rcp(ldd(udiag + R));
  const dd densityL = ldd(density + L), densityR = ldd(density + R);
  const dd projTimeScale = scale2(iuL + iuR, 0.5f);
  const dd rhoIp = scale2(densityL + densityR, 0.5f);
  const dd denScale = dd_rcp(rhoIp) * c.incomp + c.om_incomp;
  dd av[3], dx[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    av[d] = ldd(area + 3 * e + d);
    dx[d] = dd_from_double(coords[3 * R + d] - coords[3 * L + d]);
  }
  const dd asq = av[0] * av[0] + av[1] * av[1] + av[2] * av[2];
  const dd axdx = av[0] * dx[0] + av[1] * dx[1] + av[2] * dx[2];
  const dd w = asq * dd_rcp(axdx);
  dd tmdot = -(projTimeScale * dd_from_double(pressure[R] - pressure[L]) * w);
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const dd kxj = av[d] - w * dx[d];
    const dd uR = ldd(velocity + 3 * R + d), uL = ldd(velocity + 3 * L + d);
    const dd rhoUjIp = scale2(densityR * uR + densityL * uL, 0.5f);
    const dd ujIp = scale2(uR + uL, 0.5f);
    const dd GjIp = scale2(ldd(Gpdx + 3 * R + d) * iuR + ldd(Gpdx + 3 * L + d) * iuL, 0.5f);
    tmdot = tmdot + ((c.interp * rhoUjIp + c.om_interp * rhoIp * ujIp + GjIp) * av[d] -
                     kxj * GjIp * c.noc);
  }
  tmdot = tmdot * c.inv_tau * denScale;
  const dd f = -(w * projTimeScale * denScale * c.inv_tau);
  reinterpret_cast<float4*>(buf)[e] = make_float4(f.hi, f.lo, tmdot.hi, tmdot.lo);
}

__device__ __forceinline__ dd van_leer_dd(dd dqm, dd dqp, dd eps) {
  const dd p = dqm * dqp;
  const dd s = dqm + dqp;
  return scale2(p + dd_abs(p), 2.0f) * dd_rcp_fast(s * s + eps);
}

// ---------------------------------------------------------------------------
// Momentum: MomentumEdgeSolverAlg::execute (src/edge_kernels/
// MomentumEdgeSolverAlg.C:105-312), VOF off. The 6x6 local matrix has the
// block form
//   LL = cLL I - N/relax,  LR = cLR I + N,  RL = cRL I + N,
//   RR = cRR I - N/relax,  N_ij = -viscIp A_i A_j / (A.dx)
// because the advective and diffusive factors do not depend on the
// component; the rhs is (-tf, +tf), and cLL = -cRL / relax, cRR = -cLR /
// relax. So an off-diagonal CSR entry is N_ij or N_qq + c of one edge, and a
// diagonal block is -(the sum over the row's edges of the opposite block) /
// relax. The edge phase writes the nine distinct entries as the FP64 numbers
// that go into the matrix, widened once here instead of once per row and
// component, and the three fluxes as float pairs: a 96-byte record
//   D_LR0 D_RL0 tf0 N01 | D_LR1 D_RL1 tf1 N12 | D_LR2 D_RL2 tf2 N02
// (D_LRq = N_qq + c_LR), one 32-byte sector per component: what the row
// thread of that component needs but for one entry of N.
//
// Both FP32 issue and the FP64 pipe work here: sums and differences of FP64
// inputs are one FP64 operation each (25 an edge, 64 clocks of a scheduler's
// unit), exact to 53 bits, and replace the pair additions (11 operations) and
// second splits; products stay in float pairs. With g = grad u_L + grad u_R
// and the upwind side's gradient (the only one the default options need) an
// edge takes 1,900 instructions; the form that split every operand and added
// in pairs took 2,200. At 128 x 128 x 64 this kernel went from 309 to 267 us
// (59 % issue, FP64 pipe busy half the time) and the row kernel below from
// 228 to 172; on 734,831 edges of randomly numbered tets, where eleven arrays
// meant eleven sectors an edge and side, from 100 to 76 and from 232 to 59.
// The whole assembly: 542 -> 449 us and 331 -> 139 us, with smaller errors
// against 64 bits in values and rhs.
struct MomentumDD {
  dd alpha, alpha_upw, om_alpha, om_alpha_upw, upw, divu_fac, eps;
};

struct MomentumIn {
  const int2* __restrict__ edges;
  const double* __restrict__ coords;
  const double* __restrict__ vel;
  const double* __restrict__ dudx;
  const double* __restrict__ viscosity;
  const double* __restrict__ mask;
  const double* __restrict__ area;
  const double* __restrict__ mdot;
  const double* __restrict__ pec;
};

__device__ __forceinline__ double pair_bits(dd a) {
  return __hiloint2double(__float_as_int(a.lo), __float_as_int(a.hi));
}

// DEF: the reference's default advection options alpha = 0, alpha_upw = 1,
// upw_factor = 1 (SolutionOptions, src/SolutionOptions.C:31-80): only the
// upwind side's extrapolation enters, as its difference from the edge mean.
template <bool LIMITER, bool DIVU, bool DEF>
__device__ __forceinline__ void momentum_edge(int64_t e, const MomentumIn& in, const MomentumDD& c,
                                              double* __restrict__ rec) {
  const double* __restrict__ coords = in.coords;
  const double* __restrict__ vel = in.vel;
  const double* __restrict__ dudx = in.dudx;
  const int2 lr = in.edges[e];
  // 32-bit node offsets (9 N < 2^32 is checked when the system is
  // finalized): fewer registers than 64-bit ones
  const uint32_t L = uint32_t(lr.x), R = uint32_t(lr.y);
  dd av[3], hdx[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    av[d] = dd_from_double_z(in.area[3 * e + d]);
    hdx[d] = scale2(dd_from_double_z(coords[3 * R + d] - coords[3 * L + d]), 0.5f);
  }
  // the advective flux mdot u carries the largest terms of the rhs: its two
  // factors are split to the nearest pair (errors against 64 bits 1.9e-14 ->
  // 1.3e-14 of the rhs norm at 128 x 128 x 64)
  const dd mdot = dd_from_double_near(in.mdot[e]), pec = ldd(in.pec + e);
  const bool up = dd_gt0(mdot);
  const dd asq = dd_dot3(av[0], av[0], av[1], av[1], av[2], av[2]);
  const dd hinv = dd_rcp_fast(dd_dot3(av[0], hdx[0], av[1], hdx[1], av[2], hdx[2]));  // 2 / (A.dx)
  const dd inv_axdx = scale2(hinv, 0.5f);
  const dd mp = mdot * pec;
  // g: the sum (not the mean) of the two nodal gradients; corr: the factor of
  // the over-relaxed non-orthogonal correction, duidxj = g / 2 + corr A; adv:
  // the advective flux
  dd g[3][3], corr[3], adv[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double uL = vel[3 * L + i], uR = vel[3 * R + i];
    double gl[3], gr[3], gs[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      gl[j] = dudx[9 * L + 3 * i + j];
      gr[j] = dudx[9 * R + 3 * i + j];
      gs[j] = gl[j] + gr[j];
    }
    dd_from_double3(gs, g[i]);
    const dd du = dd_from_double(uR - uL), uip = scale2(dd_from_double_near(uR + uL), 0.5f);
    // 0.5 dx . (grad u_L + grad u_R), the sum of the two sides' increments
    const dd s = dd_dot3(hdx[0], g[i][0], hdx[1], g[i][1], hdx[2], g[i][2]);
    corr[i] = (du - s) * inv_axdx;
    if (DEF) {
      double gu[3];
      dd gd[3];
#pragma unroll
      for (int j = 0; j < 3; ++j) gu[j] = up ? gl[j] : gr[j];
      dd_from_double3(gu, gd);
      dd t = dd_dot3(hdx[0], gd[0], hdx[1], gd[1], hdx[2], gd[2]);
      if (LIMITER) t = t * van_leer_dd(scale2(t, 4.0f) - du, du, c.eps);
      // upwind value - mean: u_L + t - uip = t - du / 2, or -(t - du / 2)
      dd d = t - scale2(du, 0.5f);
      if (!up) d = -d;
      adv[i] = mdot * uip + mp * d;
    } else {
      dd gd[3];
      dd_from_double3(gl, gd);
      const dd duL = dd_dot3(hdx[0], gd[0], hdx[1], gd[1], hdx[2], gd[2]);
      dd_from_double3(gr, gd);
      const dd duR = dd_dot3(hdx[0], gd[0], hdx[1], gd[1], hdx[2], gd[2]);
      dd tL = duL * c.upw, tR = duR * c.upw;
      if (LIMITER) {
        tL = tL * van_leer_dd(scale2(duL, 4.0f) - du, du, c.eps);
        tR = tR * van_leer_dd(scale2(duR, 4.0f) - du, du, c.eps);
      }
      const dd uIpL = dd_from_double(uL) + tL, uIpR = dd_from_double(uR) - tR;
      const dd uiUpw = c.alpha_upw * (up ? uIpL : uIpR) + c.om_alpha_upw * uip;
      const dd uiCds = scale2(c.alpha * (uIpL + uIpR), 0.5f) + c.om_alpha * uip;
      adv[i] = mdot * (pec * uiUpw + (dd{1.0f, 0.0f} - pec) * uiCds);
    }
  }
  // viscous flux: -visc mask sum_j (duidxj + dujdxi) A_j
  //   = -visc mask [corr_i |A|^2 + A_i (corr . A) + sum_j (g_ij + g_ji) A_j / 2]
  const dd visc = scale2(dd_from_double(in.viscosity[L] + in.viscosity[R]), 0.5f);
  const dd vm = visc * dd_min(ldd(in.mask + L), ldd(in.mask + R));
  const dd ca = dd_dot3(corr[0], av[0], corr[1], av[1], corr[2], av[2]);
  dd ga = ca;  // the factor of A_i
  if (DIVU) ga = ca - c.divu_fac * (ca + scale2((g[0][0] + g[1][1]) + g[2][2], 0.5f));
  const dd s01 = scale2(g[0][1] + g[1][0], 0.5f), s02 = scale2(g[0][2] + g[2][0], 0.5f),
           s12 = scale2(g[1][2] + g[2][1], 0.5f);
  dd tf[3];
  tf[0] = adv[0] - vm * (dd_dot3(g[0][0], av[0], s01, av[1], s02, av[2]) + (corr[0] * asq + av[0] * ga));
  tf[1] = adv[1] - vm * (dd_dot3(s01, av[0], g[1][1], av[1], s12, av[2]) + (corr[1] * asq + av[1] * ga));
  tf[2] = adv[2] - vm * (dd_dot3(s02, av[0], s12, av[1], g[2][2], av[2]) + (corr[2] * asq + av[2] * ga));
  // advective constants: the upwind part mdot pec of the upwind side and the
  // central part of both
  const dd hm = scale2(mdot, 0.5f);
  dd x, y;
  if (DEF) {
    const dd aC = hm - scale2(mp, 0.5f);
    const dd w = mp + aC;
    x = up ? aC : w;
    y = up ? w : aC;
  } else {
    const dd om_pec = dd{1.0f, 0.0f} - pec;
    const dd cen = c.alpha * om_pec * hm + hm * (pec * c.om_alpha_upw + om_pec * c.om_alpha);
    const dd ua = mp * c.alpha_upw;
    x = up ? cen : ua + cen;
    y = up ? ua + cen : cen;
  }
  const dd t = -(visc * inv_axdx);
  const dd dl = t * asq;
  const dd ta0 = t * av[0], ta1 = t * av[1], ta2 = t * av[2];
  const double cLR = dd_to_double_int(x + dl), cRL = dd_to_double_int(dl - y);
  const double n00 = dd_to_double_int(ta0 * av[0]), n11 = dd_to_double_int(ta1 * av[1]),
               n22 = dd_to_double_int(ta2 * av[2]);
  st32(rec, n00 + cLR, n00 + cRL, pair_bits(tf[0]), dd_to_double_int(ta0 * av[1]));
  st32(rec + 4, n11 + cLR, n11 + cRL, pair_bits(tf[1]), dd_to_double_int(ta1 * av[2]));
  st32(rec + 8, n22 + cLR, n22 + cRL, pair_bits(tf[2]), dd_to_double_int(ta0 * av[2]));
}

template <bool LIMITER, bool DIVU, bool DEF>
__global__ void __launch_bounds__(kThreads, 4)
    momentum_edge_k(int64_t e0, int64_t e1, MomentumIn in, MomentumDD c, double* __restrict__ buf) {
  const int64_t e = e0 + int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= e1) return;
  momentum_edge<LIMITER, DIVU, DEF>(e, in, c, buf + kMomentumCoefs * e);
}

// ---------------------------------------------------------------------------
// Row phase. Each block owns node rows [r0, r0 + kRowThreads) and therefore
// the contiguous CSR value range [row_ptr[nd r0], row_ptr[nd r1]). Threads
// build their rows in shared memory; the block then writes (or adds) the
// whole range with coalesced accesses. Blocks whose range exceeds the
// staging capacity write straight to global memory.
//
// KIND 0: scalar (FP64 a01, a10, flux), KIND 1: continuity (f, tmdot as float
// pairs). Incident entries come in column order; bit 31
// marks a repeat of the previous column (periodic duplicates).
__device__ __forceinline__ double to_f64(double v) { return v; }
__device__ __forceinline__ double to_f64(dd v) { return dd_to_double_int(v); }

template <int KIND>
__global__ void __launch_bounds__(kRow1Threads)
    row1_k(int64_t R, const int32_t* __restrict__ inc_ptr,
           const uint32_t* __restrict__ inc, const int32_t* __restrict__ diag_pos,
           const int64_t* __restrict__ row_ptr, const double* __restrict__ buf,
           double irelax, double irelax_lo, double* __restrict__ values, double* __restrict__ rhs,
           int accumulate, int smem_bytes) {
  using C = typename std::conditional<KIND == 0, double, dd>::type;
  extern __shared__ __align__(16) double stage[];
  const int64_t r0 = int64_t(blockIdx.x) * kRow1Threads;
  const int64_t r1 = (r0 + kRow1Threads < R) ? r0 + kRow1Threads : R;
  const int64_t base = row_ptr[r0];
  const int64_t cnt = row_ptr[r1] - base;
  const bool staged = cnt * int64_t(sizeof(double)) <= smem_bytes;
  const int64_t r = r0 + threadIdx.x;
  if (r < r1) {
    const int32_t s = inc_ptr[r], t = inc_ptr[r + 1];
    const int64_t rb = row_ptr[r];
    double* out = staged ? stage + (rb - base) : values + rb;
    const bool acc = accumulate && !staged;
    if (s != t) {
      const int dp = diag_pos[r];
      C dg{}, rr{}, off{};
      dd_acc dga, rra;  // continuity: the diagonal and rhs sums, deferred renormalisation
      int slot = -1;
      for (int32_t qi = s; qi < t; ++qi) {
        const uint32_t w = inc[qi];
        const bool dup = (w >> 31) != 0;
        const int64_t e = (w & 0x7fffffffu) >> 1;
        const int side = w & 1u;
        C co, cd, cr;
        if constexpr (KIND == 0) {
          double x[4];
          ld32<true>(buf + kScalarCoefs * e, x);
          co = side ? x[1] : x[0];
          cd = side ? x[0] : x[1];
          cr = side ? x[2] : -x[2];
        } else {
          const float4 q = reinterpret_cast<const float4*>(buf)[e];
          const dd f{q.x, q.y}, tm{q.z, q.w};
          co = f;
          cd = -f;
          cr = side ? tm : -tm;
        }
        if (!dup) {
          if (slot >= 0) {
            double* p = out + (slot < dp ? slot : slot + 1);
            const double v = to_f64(off);
            *p = acc ? *p + v : v;
          }
          ++slot;
          off = co;
        } else {
          off = off + co;
        }
        if constexpr (KIND == 0) {
          dg = dg + cd;
          rr = rr + cr;
        } else {
          acc_add(dga, cd);
          acc_add(rra, cr);
        }
      }
      if constexpr (KIND == 0) {
        // dg / relax rounded once: 1 / relax as a pair (a rounded reciprocal left
        // 1.28e-16 on the diagonal). An infinite sum takes no correction.
        const bool finite = (__double2hiint(dg) & 0x7ff00000) != 0x7ff00000;
        dg = -fma(dg, irelax, finite ? dg * irelax_lo : 0.0);
      }
      if constexpr (KIND == 1) {
        dg = acc_value(dga);
        rr = acc_value(rra);
      }
      double* p = out + (slot < dp ? slot : slot + 1);
      const double v = to_f64(off), vd = to_f64(dg), vr = to_f64(rr);
      *p = acc ? *p + v : v;
      out[dp] = acc ? out[dp] + vd : vd;
      rhs[r] = accumulate ? rhs[r] + vr : vr;
    } else if (!acc) {
      // a row without edges: zero it (its entries are not otherwise written)
      for (int64_t k = 0; k < row_ptr[r + 1] - rb; ++k) out[k] = 0.0;
      if (!accumulate) rhs[r] = 0.0;
    }
  }
  if (!staged) return;
  __syncthreads();
  for (int64_t k = threadIdx.x; k < cnt; k += kRow1Threads)
    values[base + k] = accumulate ? values[base + k] + stage[k] : stage[k];
}

// 3-dof momentum, one thread per CSR row (three neighbouring lanes per node
// row, ten nodes a warp) over the row's incident edges in column order.
// Off-diagonal entries are copied from the edge's record; the diagonal block
// -(sum of the opposite D e_q + sum of N)_q / relax is summed in FP64, the rhs
// in float pairs. Thread q loads sector q of a record with one 32-byte load
// (a record is one line and a warp's ten records eleven or so, where eight-
// byte loads of the same words cost five times the L1 lookups), sums its own
// entry of N and takes the other one it stores from the node's next lane.
// The next record is loaded while one is summed. A warp stages its CSR range in
// shared memory and writes it with one bulk copy, or adds it with one where the
// system holds values: read, added and written by the lanes, repeated assembly of
// 128 x 128 x 64 took 782 us (766 with the kernels of a block a range), 517 now, of
// 1,167,183 tet edges 357 and 229. What it reads and writes (96
// bytes an edge, the matrix) takes 125 us at 128 x 128 x 64; it takes 172,
// with FP64 pipe, issue and L1 each about half busy (24 warps a SM without
// spills measured the same as 36 with).
constexpr int kRow3Warps = 6, kRow3PerSm = 4;
constexpr int kRow3Group = 10;  // node rows of a warp, three lanes each
struct Row3Args {
  int64_t R;  // end of the node rows
  int64_t r_begin;  // first node row (the row kernel's blocks start here)
  int64_t mask;  // edge -> record: e & mask
  const int32_t* __restrict__ inc_ptr;
  const uint32_t* __restrict__ inc;
  const int32_t* __restrict__ diag_pos;
  const int64_t* __restrict__ row_ptr;
  const double* rec;  // not restrict: the single-kernel assembly writes it in flight
  double irelax;
  double* __restrict__ values;
  double* __restrict__ rhs;
  int accumulate, smem_bytes;
};

// *p += x with an addition that stays inside its branch
__device__ __forceinline__ void add64(double* p, double x) {
  double y = *p;
  asm volatile("add.f64 %0, %0, %1;" : "+d"(y) : "d"(x));
  *p = y;
}

// Bulk copy (add: element-wise addition to what is there, rounded as any other)
// of `bytes` (a multiple of 16) from shared to global memory, both 16-byte
// aligned, by one thread after the others' writes have been fenced
// (fence_async) and joined.
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void bulk_store(double* dst, const double* src, int bytes, bool add) {
  if (add)
    asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f64 [%0], [%1], %2;" ::"l"(dst),
                 "r"(uint32_t(__cvta_generic_to_shared(src))), "r"(bytes)
                 : "memory");
  else
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(uint32_t(__cvta_generic_to_shared(src))), "r"(bytes)
                 : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// the calling thread's bulk copies have read their sources
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// Groups g, g + step, ... of kRow3Group node rows from row `first` to `end`,
// by one warp, which stages each group's CSR range and writes it: no block
// barrier. A group starts with a chain of loads (list bounds, list, record),
// as long as the sums themselves at the matrix sizes here, so the next
// group's bounds are loaded with this group's records and its first record
// while this group's rows are finished.
// IDX: the type of the record offsets (uint32_t when 12 E < 2^31: one
// register and one wide multiply-add per record instead of 64-bit
// arithmetic). ACC: 0 overwrite, 1 add to the values present, -1 as
// a.accumulate says (the write mode as a constant drops the read and select
// of every store).
template <bool NC, typename IDX = int64_t, int ACC = -1>
__device__ __forceinline__ void row3_groups(int64_t g, int64_t step, int64_t first, int64_t end_row,
                                            const Row3Args& a, double* stage) {
  const bool accumulate = ACC < 0 ? a.accumulate != 0 : ACC != 0;
  const int lane = threadIdx.x & 31, trio = lane / 3, q = lane - 3 * trio;
  const int next = 3 * trio + (q + 2) % 3;  // the lane that holds the other entry of N
  // columns of thread q's own entry of N (0: N01, 1: N12, 2: N02) and of the
  // other one (0: N02, 1: N01, 2: N12)
  const int cn = q == 0 ? 1 : (q == 1 ? 2 : 0), co = q == 0 ? 2 : (q == 1 ? 0 : 1);
  struct Bounds {
    int64_t base, bq;  // CSR position of the group and of this lane's row
    int32_t s, t, cnt, dp;
  };
  auto bounds = [&](int64_t gr) {
    Bounds b{0, 0, 0, 0, 0, 0};
    const int64_t r0 = first + gr * kRow3Group;
    if (r0 >= end_row) return b;
    const int64_t r1 = r0 + kRow3Group < end_row ? r0 + kRow3Group : end_row, r = r0 + trio;
    b.base = a.row_ptr[3 * r0];
    b.cnt = stage_count(b.base, a.row_ptr[3 * r1]);
    if (trio < kRow3Group && r < r1) {
      b.s = a.inc_ptr[r];
      b.t = a.inc_ptr[r + 1];
      b.bq = a.row_ptr[3 * r + q];
      b.dp = a.diag_pos[r];
    }
    return b;
  };
  auto load = [&](uint32_t w, double (&x)[4]) {
    ld32<NC>(a.rec + IDX(kMomentumCoefs) * IDX(int64_t((w & 0x7fffffffu) >> 1) & a.mask) + 4 * q, x);
  };
  if (first + g * kRow3Group >= end_row) return;
  Bounds b = bounds(g);
  uint32_t w = b.s < b.t ? a.inc[b.s] : 0u, wn = b.s + 1 < b.t ? a.inc[b.s + 1] : 0u;
  double x[4];
  if (b.s < b.t) load(w, x);
  for (;;) {
    const int64_t r = first + g * kRow3Group + trio;
    g += step;
    const Bounds bn = bounds(g);
    if (lane == 0) bulk_wait();  // the previous group's copy has left the stage
    __syncwarp();
    const int s = b.s, t = b.t, dp = b.dp;
    // the staged range keeps the parity of the CSR position, so that both
    // sides of the copy are 16-byte aligned together
    const int odd = int(b.base & 1);
    const bool staged = stage_fits(b.cnt, odd, a.smem_bytes);
    const bool acc = accumulate && !staged;
    double* v = staged ? stage + odd + (b.bq - b.base) : a.values + b.bq;
    if (s == t && trio < kRow3Group && r < end_row && !acc) {
      const int64_t len = a.row_ptr[3 * r + q + 1] - b.bq;
      for (int64_t k = 0; k < len; ++k) v[k] = 0.0;
      if (!accumulate) a.rhs[3 * r + q] = 0.0;
    }
    auto put3 = [&](int k, double d, double n, double o) {
      v[k + q] = acc ? v[k + q] + d : d;
      v[k + cn] = acc ? v[k + cn] + n : n;
      v[k + co] = acc ? v[k + co] + o : o;
    };
    dd_acc rr;
    double sd = 0.0, sn = 0.0;
    int slot = -1;
    // every lane takes the warp's largest number of rounds (the exchange is
    // warp-wide); the next record and the incidence after it are in flight
    // while a record is summed (two records ahead measured the same)
    const int most = __reduce_max_sync(0xffffffffu, t - s);
#pragma unroll 2
    for (int k = 0; k < most; ++k) {
      double xn[4];
      if (s + k + 1 < t) load(wn, xn);
      const uint32_t w2 = s + k + 2 < t ? a.inc[s + k + 2] : 0u;
      const double other = __shfl_sync(0xffffffffu, x[3], next);
      if (s + k < t) {
        const bool side = (w & 1u) != 0, dup = (w >> 31) != 0;
        const double own = side ? x[1] : x[0], opp = side ? x[0] : x[1];
        const dd f{__int_as_float(__double2loint(x[2])), __int_as_float(__double2hiint(x[2]))};
        acc_add(rr, side ? f : -f);
        slot += dup ? 0 : 1;
        const int col = 3 * (slot < dp ? slot : slot + 1);
        if (!dup) {
          put3(col, own, x[3], other);
        } else {  // a repeated column (periodic pairs)
          add64(v + col + q, own);
          add64(v + col + cn, x[3]);
          add64(v + col + co, other);
        }
        sd += opp;
        sn += x[3];
      }
      w = wn;
      wn = w2;
#pragma unroll
      for (int j = 0; j < 4; ++j) x[j] = xn[j];
    }
    // the next group's first incidences, then its first record
    const bool more = bn.s < bn.t;
    w = more ? a.inc[bn.s] : 0u;
    wn = bn.s + 1 < bn.t ? a.inc[bn.s + 1] : 0u;
    const double so = __shfl_sync(0xffffffffu, sn, next);
    if (s != t) {
      put3(3 * dp, -sd * a.irelax, -sn * a.irelax, -so * a.irelax);
      const double d = dd_to_double_int(acc_value(rr));
      a.rhs[3 * r + q] = accumulate ? a.rhs[3 * r + q] + d : d;
    }
    if (more) load(w, x);
    if (staged) {
      double* out = a.values + b.base - odd;
      const int end = b.cnt + odd;
      // the whole 16-byte pairs as one bulk copy, the ends by hand
      fence_async();
      __syncwarp();
      const int by_hand = lane == 1 && odd && end > 1 ? 1 : (lane == 2 && (end & 1) && end > odd ? end - 1 : -1);
      if (by_hand >= 0) out[by_hand] = accumulate ? out[by_hand] + stage[by_hand] : stage[by_hand];
      const int from = 2 * odd, bytes = ((end & ~1) - from) * int(sizeof(double));
      if (lane == 0 && bytes > 0) bulk_store(out + from, stage + from, bytes, accumulate);
    }
    if (first + g * kRow3Group >= end_row) {
      if (lane == 0) bulk_wait();
      return;
    }
    b = bn;
  }
}

template <typename IDX, int ACC>
__global__ void __launch_bounds__(32 * kRow3Warps, kRow3PerSm) row3t_k(Row3Args a) {
  extern __shared__ __align__(16) double stage[];
  row3_groups<true, IDX, ACC>(int64_t(blockIdx.x) * kRow3Warps + (threadIdx.x >> 5),
                              int64_t(gridDim.x) * kRow3Warps, a.r_begin, a.R, a,
                              stage + (threadIdx.x >> 5) * (a.smem_bytes >> 3));
}

// ---------------------------------------------------------------------------
// Single-kernel momentum assembly: a persistent kernel whose blocks take
// edge chunks and row blocks from the work list of schedule.h in ticket
// order. Edge chunks write their records into a ring of slots small enough
// for L2 and row blocks read them from there, so that most of the record
// round trip of the two-kernel form stays out of DRAM. The arithmetic and
// the summation order are those of momentum_edge_k + row3t_k: the CSR
// values are the same bits.
//
// Bound by its barriers and instruction issue. Three blocks a SM (80
// registers, about 100 bytes of spills a thread): at four (64 registers) the
// row part spills 370 bytes a thread, 57 MB over the resident threads, which
// push the 50 MB ring out of L2. 128 x 128 x 64 hexes: 1.22 GB of DRAM traffic and
// 613 us with three, 1.55 GB and 632 us with four (two kernels 1.45 GB and
// 449 us); 734,831 edges of random tets, option set in full: 194 and 227 us.
// Two blocks a SM take 791 and 186 us.
//
// Dependencies are flags holding the launch's generation number: a chunk's
// flag is set once its coefficients are written, a row block's once its
// reads are done. Waits only point to earlier tickets, held by running
// blocks, so they end; each poll is still bounded (kSpinLimit rounds), after
// which the block records the timeout in *err, skips its work, sets its own
// flag and the remaining blocks stop taking tickets.
struct FusedArgs {
  const int32_t* __restrict__ items;
  const int32_t* __restrict__ in_ptr;   // row block k reads chunks in[in_ptr[k] ..]
  const int32_t* __restrict__ in;
  const int32_t* __restrict__ out_ptr;  // chunk c is read by blocks out[out_ptr[c] ..]
  const int32_t* __restrict__ out;
  int* eflag;
  int* rflag;
  int* ticket;
  int* err;
  int64_t num_edges, ring_chunks;
  int nitems, gen;
};

constexpr int kSpinLimit = 1 << 20;

__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_volatile(const int* p) { return *reinterpret_cast<const volatile int*>(p); }

// True once flags[list[0 .. n)] all hold gen. Each thread polls a strided
// share with relaxed loads and, having seen its flags set, issues one
// acquire fence (the flag was set by a release store after the producer's
// writes), then the block agrees at a barrier. False in every thread after a
// timeout, or when another block has reported one.
__device__ bool wait_flags(const int* flags, const int32_t* list, int n, int gen, int* err) {
  bool ok = true, polled = false;
  for (int i = int(threadIdx.x); ok && i < n; i += int(blockDim.x)) {
    const int* fp = flags + list[i];
    polled = true;
    int spins = 0;
    while (ld_relaxed(fp) != gen) {
      if (++spins > kSpinLimit || ((spins & 1023) == 0 && ld_volatile(err) != 0)) {
        ok = false;
        break;
      }
      __nanosleep(64);
    }
  }
  if (polled && ok) fence_acq_rel();
  const bool all = __syncthreads_and(ok) != 0;
  if (!all && threadIdx.x == 0) atomicExch(err, 1);
  return all;
}

constexpr int kFusedPerSm = 3;
template <bool LIMITER, bool DIVU, bool DEF>
__global__ void __launch_bounds__(kFusedChunk, kFusedPerSm)
    momentum_fused_k(FusedArgs f, MomentumIn in, MomentumDD c, Row3Args ra, double* ring) {
  extern __shared__ __align__(16) double stage[];
  __shared__ int s_item[2];
  int next = 0;
  if (threadIdx.x == 0) next = atomicAdd(f.ticket, 1);
  for (int p = 0;; p ^= 1) {
    // double-buffered item word: the barrier of the next item separates
    // this item's reads from the write two items on
    if (threadIdx.x == 0) s_item[p] = (next < f.nitems && ld_volatile(f.err) == 0) ? f.items[next] : -1;
    __syncthreads();
    const int it = s_item[p];
    if (it < 0) return;
    // the next ticket is taken now; its latency hides behind this item
    if (threadIdx.x == 0) next = atomicAdd(f.ticket, 1);
    const int idx = it >> 1;
    if (it & 1) {
      const int b = f.in_ptr[idx];
      if (wait_flags(f.eflag, f.in + b, f.in_ptr[idx + 1] - b, f.gen, f.err))
        row3_groups<false>(threadIdx.x >> 5, kFusedBlock / kRow3Group, int64_t(idx) * kFusedBlock,
                           min(int64_t(idx + 1) * kFusedBlock, ra.R), ra,
                           stage + (threadIdx.x >> 5) * (ra.smem_bytes >> 3));
      __syncthreads();
      if (threadIdx.x == 0) st_release(f.rflag + idx, f.gen);
    } else {
      // the slot's previous chunk must have been read by all its row blocks
      const int64_t prev = int64_t(idx) - f.ring_chunks;
      const bool ok = prev < 0 || wait_flags(f.rflag, f.out + f.out_ptr[prev],
                                             f.out_ptr[prev + 1] - f.out_ptr[prev], f.gen, f.err);
      const int64_t e = int64_t(idx) * kFusedChunk + threadIdx.x;
      if (ok && e < f.num_edges) momentum_edge<LIMITER, DIVU, DEF>(e, in, c, ring + kMomentumCoefs * (e & ra.mask));
      __syncthreads();
      if (threadIdx.x == 0) st_release(f.eflag + idx, f.gen);
    }
  }
}

// applyDirichletBCs / resetRows: identity (or diag_value) rows, LANES lanes a row:
// one thread for a node's rows made one uncoalesced pass over its entries, three
// rows of up to 18 on a hex wall. Few or long rows take eight lanes, many short ones
// four. With one thread a node, 16, 8 and 4 lanes a row (us, the host's wait
// included): walls of 221 hex nodes, 3 unknowns, 28.7, 12.7, 12.7, 13.0; all rows of
// 1.08 M hex nodes, 1 unknown (7 entries a row), 53.5, 148, 85, 51; with 3 unknowns
// (21 entries) 801, 472, 288, 194; of 172,032 tet nodes with 3 unknowns (45 entries)
// 276, 102, 73, 104.
constexpr int64_t kResetFewRows = 4096;
template <int LANES>
__global__ void __launch_bounds__(kThreads)
    reset_rows_k(int64_t n, const int64_t* __restrict__ nodes,
                 const int64_t* __restrict__ node_lid, int num_dof,
                 int begin, int end, const int64_t* __restrict__ row_ptr,
                 const int32_t* __restrict__ col_idx,
                 double* __restrict__ values, double* __restrict__ rhs,
                 double diag_value, double rhs_value,
                 const double* __restrict__ q,
                 const double* __restrict__ bc, int64_t num_nodes,
                 int* __restrict__ err) {
  const int64_t t = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) / LANES;
  const int sub = int(threadIdx.x % LANES), nd = max(end - begin, 1);
  const int64_t k = t / nd;
  if (k >= n) return;
  const int64_t node = nodes[k];
  if (node < 0 || node >= num_nodes) {
    *err = 1;
    return;
  }
  if (end <= begin) return;
  const int d = begin + int(t - k * nd);
  const int64_t row = node_lid[node] + d;
  const int64_t p1 = row_ptr[row + 1];
  for (int64_t p = row_ptr[row] + sub; p < p1; p += LANES)
    values[p] = (col_idx[p] == row) ? diag_value : 0.0;
  if (sub == 0) rhs[row] = bc ? (bc[num_dof * node + d] - q[num_dof * node + d]) : rhs_value;
}

// LinearSystem::sumInto for one host-provided entity block: one thread per
// local row scans its CSR row (sum_into_row semantics).
__global__ void sum_into_block_k(int n_ent, int num_dof,
                                 const int64_t* __restrict__ ent_lid,
                                 const double* __restrict__ lhs,
                                 const double* __restrict__ brhs,
                                 const int64_t* __restrict__ row_ptr,
                                 const int32_t* __restrict__ col_idx,
                                 double* __restrict__ values,
                                 double* __restrict__ rhs) {
  const int nloc = n_ent * num_dof;
  const int i = threadIdx.x;
  if (i >= nloc) return;
  const int64_t row = ent_lid[i / num_dof] + i % num_dof;
  for (int j = 0; j < nloc; ++j) {
    const int32_t col = int32_t(ent_lid[j / num_dof] + j % num_dof);
    for (int64_t p = row_ptr[row]; p < row_ptr[row + 1]; ++p)
      if (col_idx[p] == col) {
        values[p] += lhs[i * nloc + j];
        break;
      }
  }
  rhs[row] += brhs[i];
}

inline unsigned grid_for(int64_t n, int t = kThreads) {
  return unsigned((n + t - 1) / t);
}

int g_smem_set_device = -1, g_sms = 1;
void set_smem_attrs() {
  int dev = 0;
  NW_CUDA(cudaGetDevice(&dev));
  if (g_smem_set_device == dev) return;
  NW_CUDA(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
  NW_CUDA(cudaFuncSetAttribute(row1_k<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxRowSmem));
  NW_CUDA(cudaFuncSetAttribute(row1_k<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxRowSmem));
  NW_CUDA(cudaFuncSetAttribute(row3t_k<uint32_t, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxRowSmem));
  NW_CUDA(cudaFuncSetAttribute(row3t_k<uint32_t, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxRowSmem));
  NW_CUDA(cudaFuncSetAttribute(row3t_k<int64_t, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxRowSmem));
  NW_CUDA(cudaFuncSetAttribute(row3t_k<int64_t, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxRowSmem));
#define NW_FUSED_ATTR(LIM, DIV, DEF)                                                      \
  NW_CUDA(cudaFuncSetAttribute(momentum_fused_k<LIM, DIV, DEF>,                           \
                               cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxRowSmem))
  NW_FUSED_ATTR(false, false, false);
  NW_FUSED_ATTR(false, false, true);
  NW_FUSED_ATTR(false, true, false);
  NW_FUSED_ATTR(false, true, true);
  NW_FUSED_ATTR(true, false, false);
  NW_FUSED_ATTR(true, false, true);
  NW_FUSED_ATTR(true, true, false);
  NW_FUSED_ATTR(true, true, true);
#undef NW_FUSED_ATTR
  g_smem_set_device = dev;
}

}  // namespace

void launch_scalar_edges(cudaStream_t s, int64_t E, int64_t N, const int2* edges,
                         const nw_scalar_fields& f, const ScalarOpts& o,
                         double* buf, double* nodebuf) {
  if (E == 0) return;
  // Small systems skip the node pre-pass: its launch costs more than the two
  // reciprocals an edge it saves. Pass with and without it, default options:
  // 104 k edges 44.0 and 42.6 us, 267 k edges 72.5 and 73.3, 799 k 153 and 163
  const bool node = E > 131072;
  if (node) scalar_node_k<<<grid_for(N), kThreads, 0, s>>>(N, f.density, f.diff_coeff, nodebuf);
  const ScalarArgs a{o.alpha, o.alpha_upw, 1.0 - o.alpha, 1.0 - o.alpha_upw, o.upw_factor,
                     0.5 * o.hybrid_factor, o.tanh_trans, -2.0 / o.tanh_width};
  auto go = [&](auto kernel) {
    kernel<<<grid_for(E, kScalarBlock), kScalarBlock, 0, s>>>(E, edges, f.coords, f.velocity_rtm, f.q, f.dqdx,
                                                              f.diff_coeff, node ? nodebuf : f.density, f.area,
                                                              f.mdot, a, buf);
  };
  const int which = (o.use_limiter ? 8 : 0) + (o.tanh_form ? 4 : 0) + (o.alpha != 0.0 ? 2 : 0) + (node ? 1 : 0);
  switch (which) {
    case 0: go(scalar_edge_k<false, false, false, false>); break;
    case 1: go(scalar_edge_k<false, false, false, true>); break;
    case 2: go(scalar_edge_k<false, false, true, false>); break;
    case 3: go(scalar_edge_k<false, false, true, true>); break;
    case 4: go(scalar_edge_k<false, true, false, false>); break;
    case 5: go(scalar_edge_k<false, true, false, true>); break;
    case 6: go(scalar_edge_k<false, true, true, false>); break;
    case 7: go(scalar_edge_k<false, true, true, true>); break;
    case 8: go(scalar_edge_k<true, false, false, false>); break;
    case 9: go(scalar_edge_k<true, false, false, true>); break;
    case 10: go(scalar_edge_k<true, false, true, false>); break;
    case 11: go(scalar_edge_k<true, false, true, true>); break;
    case 12: go(scalar_edge_k<true, true, false, false>); break;
    case 13: go(scalar_edge_k<true, true, false, true>); break;
    case 14: go(scalar_edge_k<true, true, true, false>); break;
    default: go(scalar_edge_k<true, true, true, true>); break;
  }
}

bool continuity_fast_path(const ContinuityOpts& o) {
  return o.interp_together == 1.0 && o.solve_incompressible == 0.0;
}

dd dd_param(double x) { return dd_from_double(x); }

void launch_continuity_edge_range(cudaStream_t s, int64_t n0, int64_t n1, int64_t e0, int64_t e1,
                                  const int2* edges, const nw_continuity_fields& f,
                                  const ContinuityOpts& o, double* buf, double* nodebuf, bool node) {
  // the edge kernels index edges, area vectors and records from 0: shift
  // the per-edge pointers to the range
  const int64_t n = e1 > e0 ? e1 - e0 : 0;
  dd* b = reinterpret_cast<dd*>(buf) + 2 * e0;
  const int2* er = edges + e0;
  const double* ar = f.area + 3 * e0;
  if (nodebuf && continuity_fast_path(o)) {
    dd* nb = reinterpret_cast<dd*>(nodebuf);
    if (node && n1 > n0)
      continuity_node_k<<<grid_for(n1 - n0), kThreads, 0, s>>>(
          n0, n1, f.velocity, f.dpdx, f.density, f.pressure, f.udiag, nb);
    if (n) {
      auto go = [&](auto kernel) {
        kernel<<<grid_for(n, kContinuityBlock), kContinuityBlock, 0, s>>>(n, er, f.coords, nb, f.pressure, ar, dd_param(o.noc_fac),
                                                dd_param(1.0 / o.tau_scale), b,
                                                ContinuityNodeFields{f.velocity, f.dpdx, f.density, f.udiag});
      };
      const bool plain = o.noc_fac == 1.0;
      if (node)
        plain ? go(continuity_edge_fast_k<true, true>) : go(continuity_edge_fast_k<false, true>);
      else
        plain ? go(continuity_edge_fast_k<true, false>) : go(continuity_edge_fast_k<false, false>);
    }
  } else if (n) {
    ContinuityDD c;
    c.noc = dd_param(o.noc_fac);
    c.inv_tau = dd_param(1.0 / o.tau_scale);
    c.interp = dd_param(o.interp_together);
    c.om_interp = dd_param(1.0 - o.interp_together);
    c.incomp = dd_param(o.solve_incompressible);
    c.om_incomp = dd_param(1.0 - o.solve_incompressible);
    continuity_edge_k<<<grid_for(n), kThreads, 0, s>>>(
        n, er, f.coords, f.velocity, f.dpdx, f.density, f.pressure, f.udiag,
        ar, c, b);
  }
}

void launch_continuity_edges(cudaStream_t s, int64_t E, int64_t N,
                             const int2* edges, const nw_continuity_fields& f,
                             const ContinuityOpts& o, double* buf,
                             double* nodebuf) {
  if (E == 0) return;
  // Small systems form the node records in the edge kernel (the same
  // operations): a launch costs more than the repeated ones. With the pre-pass
  // and without it, hexes in row order: 21 k edges 21.1 and 17.7 us, 86 k 21.2
  // and 19.0, 276 k 27.3 and 25.7, 507 k 35.2 and 35.4, 811 k 49.9 and 56.0,
  // 3.2 M 145.7 and 187.9. Randomly numbered tets: 18 k 25.6 and 24.0, 82 k 27.3
  // and 26.1, 274 k 35.9 and 37.2, 497 k 46.6 and 50.5, 3.2 M 235.0 and 299.5. The
  // forms break even near 0.5 M edges on the first and 0.2 M on the second; the line
  // lies between. Ranges keep the pre-pass, whose records later ranges read.
  launch_continuity_edge_range(s, 0, N, 0, E, edges, f, o, buf, nodebuf, E > 262144);
}

void launch_continuity_edges(cudaStream_t s, int64_t E, const int2* edges,
                             const nw_continuity_fields& f,
                             const ContinuityOpts& o, double* buf) {
  launch_continuity_edges(s, E, 0, edges, f, o, buf, nullptr);
}

namespace {
MomentumDD momentum_dd(const MomentumOpts& o) {
  MomentumDD c;
  c.alpha = dd_param(o.alpha);
  c.alpha_upw = dd_param(o.alpha_upw);
  c.om_alpha = dd_param(1.0 - o.alpha);
  c.om_alpha_upw = dd_param(1.0 - o.alpha_upw);
  c.upw = dd_param(o.upw_factor);
  c.divu_fac = dd_param(2.0 / 3.0 * o.include_div_u);
  c.eps = dd_param(1.0e-16);
  return c;
}
MomentumIn momentum_in(const int2* edges, const nw_momentum_fields& f) {
  return MomentumIn{edges, f.coords, f.velocity, f.dudx, f.viscosity, f.mask, f.area, f.mdot, f.pecfac};
}
Row3Args row3_args(int64_t R, const int32_t* inc_ptr, const uint32_t* inc, const int32_t* diag_pos,
                   const int64_t* row_ptr, const double* buf, double relax, double* values,
                   double* rhs, int accumulate, int smem_bytes) {
  return Row3Args{R, 0, int64_t(-1), inc_ptr, inc, diag_pos, row_ptr, buf, 1.0 / relax, values, rhs,
                  accumulate, smem_bytes};
}
}  // namespace

void launch_momentum_edges(cudaStream_t s, int64_t e0, int64_t e1, const int2* edges,
                           const nw_momentum_fields& f, const MomentumOpts& o,
                           double* buf) {
  if (e1 <= e0) return;
  const MomentumDD c = momentum_dd(o);
  const MomentumIn in = momentum_in(edges, f);
  const bool lim = o.use_limiter != 0, divu = o.include_div_u != 0.0;
  const bool def = o.alpha == 0.0 && o.alpha_upw == 1.0 && o.upw_factor == 1.0;
#define NW_MOM(LIM, DIV, DEF) \
  momentum_edge_k<LIM, DIV, DEF><<<grid_for(e1 - e0), kThreads, 0, s>>>(e0, e1, in, c, buf)
#define NW_MOM2(LIM, DIV) \
  if (def) NW_MOM(LIM, DIV, true); \
  else NW_MOM(LIM, DIV, false)
  if (lim && divu) NW_MOM2(true, true);
  else if (lim) NW_MOM2(true, false);
  else if (divu) NW_MOM2(false, true);
  else NW_MOM2(false, false);
#undef NW_MOM2
#undef NW_MOM
}

int fused_blocks_per_sm(int smem_bytes) {
  set_smem_attrs();
  int occ = 0;
  NW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, momentum_fused_k<false, false, true>,
                                                        kFusedChunk, smem_bytes * (kFusedChunk / 32)));
  return occ;
}

void launch_momentum_fused(cudaStream_t s, const FusedLaunch& L, const int2* edges,
                           const nw_momentum_fields& f, const MomentumOpts& o) {
  if (L.nitems == 0) return;
  set_smem_attrs();
  const MomentumDD c = momentum_dd(o);
  const MomentumIn in = momentum_in(edges, f);
  Row3Args ra = row3_args(L.R, L.inc_ptr, L.inc, L.diag_pos, L.row_ptr, L.ring, o.relax, L.values, L.rhs,
                          L.accumulate, L.smem_bytes);
  ra.mask = L.mask;
  FusedArgs fa{L.items, L.in_ptr, L.in, L.out_ptr, L.out, L.eflag, L.rflag,
               L.ticket, L.err, L.num_edges, L.ring_chunks, int(L.nitems), L.gen};
  NW_CUDA(cudaMemsetAsync(L.ticket, 0, sizeof(int), s));
  const bool lim = o.use_limiter != 0, divu = o.include_div_u != 0.0;
  const bool def = o.alpha == 0.0 && o.alpha_upw == 1.0 && o.upw_factor == 1.0;
#define NW_FUSED(LIM, DIV, DEF) \
  momentum_fused_k<LIM, DIV, DEF><<<L.grid, kFusedChunk, L.smem_bytes * (kFusedChunk / 32), s>>>(fa, in, c, ra, L.ring)
#define NW_FUSED2(LIM, DIV) \
  if (def) NW_FUSED(LIM, DIV, true); \
  else NW_FUSED(LIM, DIV, false)
  if (lim && divu) NW_FUSED2(true, true);
  else if (lim) NW_FUSED2(true, false);
  else if (divu) NW_FUSED2(false, true);
  else NW_FUSED2(false, false);
#undef NW_FUSED2
#undef NW_FUSED
}

int row_block_nodes(int kind) { return kind >= 2 ? kRow3Group : kRow1Threads; }

int row_stage_bytes(int kind, const int64_t* row_ptr_host, int64_t R) {
  const int nb = row_block_nodes(kind);
  const int nd = kind >= 2 ? 3 : 1;
  int64_t mx = 0;
  for (int64_t r0 = 0; r0 < R; r0 += nb) {
    const int64_t r1 = r0 + nb < R ? r0 + nb : R;
    const int64_t c = row_ptr_host[nd * r1] - row_ptr_host[nd * r0];
    if (c > mx) mx = c;
  }
  // kind 2 and 3: bytes of one warp, one more entry so that the range can
  // start at its parity, a multiple of 16; at most its share of the block's.
  // Rows beyond it are written entry by entry: 943,991 edges with 19 block
  // columns a row took 267 us with 12 KB a warp of kind 2 (17 columns fit),
  // 161 with its 16 KB (22 fit).
  if (kind >= 2) {
    const int warps = kind == 2 ? kRow3Warps : kFusedChunk / 32;
    return int(std::min<int64_t>((mx + 2) / 2 * 16, kMaxRowSmem / warps));
  }
  const int64_t bytes = mx * int64_t(sizeof(double));
  return bytes <= kMaxRowSmem ? int(bytes) : kMaxRowSmem;
}

void launch_rows(cudaStream_t s, int kind, int64_t R, const int32_t* inc_ptr,
                 const uint32_t* inc, const int32_t* diag_pos,
                 const int64_t* row_ptr, const double* buf, int64_t E,
                 double relax, double* values, double* rhs, int accumulate,
                 int smem_bytes, int max_inc, int64_t row_begin) {
  if (R <= row_begin) return;
  set_smem_attrs();
  const double irelax = 1.0 / relax, lo = std::fma(-relax, irelax, 1.0) / relax;
  if (kind == 0)
    row1_k<0><<<grid_for(R, kRow1Threads), kRow1Threads, smem_bytes, s>>>(
        R, inc_ptr, inc, diag_pos, row_ptr, buf, irelax, std::isfinite(lo) ? lo : 0.0, values, rhs, accumulate,
        smem_bytes);
  else if (kind == 1)
    row1_k<1><<<grid_for(R, kRow1Threads), kRow1Threads, smem_bytes, s>>>(
        R, inc_ptr, inc, diag_pos, row_ptr, buf, 1.0, 0.0, values, rhs, accumulate, smem_bytes);
  else {
    Row3Args a = row3_args(R, inc_ptr, inc, diag_pos, row_ptr, buf, relax, values, rhs, accumulate, smem_bytes);
    a.r_begin = row_begin;
    // one wave of blocks: registers allow kRow3PerSm a SM, the staging fewer
    const int smem = smem_bytes * kRow3Warps;
    const int occ = std::max(1, std::min(kRow3PerSm, kSmSmem / (smem + 1024)));
    const unsigned grid = std::min(grid_for(R - row_begin, kRow3Group * kRow3Warps), unsigned(occ * g_sms));
    const bool narrow = int64_t(kMomentumCoefs) * E < (int64_t(1) << 31);
    if (narrow && !accumulate)
      row3t_k<uint32_t, 0><<<grid, 32 * kRow3Warps, smem, s>>>(a);
    else if (narrow)
      row3t_k<uint32_t, 1><<<grid, 32 * kRow3Warps, smem, s>>>(a);
    else if (!accumulate)
      row3t_k<int64_t, 0><<<grid, 32 * kRow3Warps, smem, s>>>(a);
    else
      row3t_k<int64_t, 1><<<grid, 32 * kRow3Warps, smem, s>>>(a);
  }
}

void launch_reset_rows(cudaStream_t s, int64_t n, const int64_t* nodes,
                       const int64_t* node_lid, int num_dof, int begin,
                       int end, const int64_t* row_ptr, const int32_t* col_idx,
                       double* values, double* rhs, double diag_value,
                       double rhs_value, const double* q, const double* bc,
                       int64_t num_nodes, double row_length, int* err) {
  if (n == 0) return;
  const int64_t rows = n * std::max(end - begin, 1);
  auto go = [&](auto kernel, int lanes) {
    kernel<<<grid_for(rows * lanes), kThreads, 0, s>>>(n, nodes, node_lid, num_dof, begin, end, row_ptr, col_idx,
                                                       values, rhs, diag_value, rhs_value, q, bc, num_nodes, err);
  };
  rows <= kResetFewRows || row_length >= 32.0 ? go(reset_rows_k<8>, 8) : go(reset_rows_k<4>, 4);
}

void launch_sum_into_block(cudaStream_t s, int n_ent, int num_dof,
                           const int64_t* ent_lid, const double* lhs,
                           const double* rhs_in, const int64_t* row_ptr,
                           const int32_t* col_idx, double* values,
                           double* rhs) {
  sum_into_block_k<<<1, 128, 0, s>>>(n_ent, num_dof, ent_lid, lhs, rhs_in,
                                     row_ptr, col_idx, values, rhs);
}

}  // namespace nw
