// D3Q6x12 step, fused form.  Included by cvlbm3d.cu (shares Ctx3 and the
// per-link helpers).
//
// Node kernels (reference raster order of the active nodes):
//   k3_moments   f0 -> U (all 12 components), collide-time u into `ucol`
//                (u_next), invalid flag; when no sweep is due, u and u* too
//   k3_sweep     u_swept -> u and the trapezoidal u* update, from U and ucol
//                of the node and its six neighbours plus cut-point anchors
//   k3_collide   one thread per node: F repair from the swept u (+-2 star
//                stencil), f0 again, BGK collision with damping/source, repair
//                delta and push streaming to f1; a population whose neighbour
//                is not active leaves through a cut link and is kept per link
//                (link_scratch) for the link kernels; the post-step U of nodes
//                that links read goes to U_need, one 96-byte row each
//   k3_moments_part  the moments of the nodes without / with a cut link,
//                for the optional overlap of the next step with the links
// Per active node this reads f0 twice and writes f1 once (the f0 re-read of
// the collide is what a single-pass 3-D fusion would save; its 3-deep halo
// does not fit shared memory), plus U, u and u* (about 2.1 KB per node
// against the algorithmic 1.2 KB).
//
// Link kernels (the four phases of apply_boundary_reconstruction,
// three_d/curved_boundary_warp3d.py:4339-4399): cvlbm3d_links.cuh for problems with
// packed characteristic tables; without them
//   k3_link_gather   16 lanes per link, one per component: value and
//                    gradient of the characteristic stencil (:2675-2700)
//   k3_link_prepare  one thread per link: boundary value, F predictor, Newton
//                    normal solve, P(F_b) (:2887-3151)
//   k3_link_rows     one thread per (link, row): BFL rows (:3154-3241) that
//                    the characteristic closure does not overwrite
//   k3_link_char     one thread per link: characteristic rows (:2812-2884)
// In the fused step they read the outgoing populations from link_scratch and
// the post-stream f1 instead of a stored post-collision field.
#pragma once

namespace {

struct Fused3 {
  const int32_t* need_slot;  // [N] row of Uneed of a node some link reads, or -1
  const int32_t* char_slot;  // [64*n_links] characteristic samples as Uneed rows
  const int32_t* partner;    // [n_links] link at the same node in direction q_in, or -1
  const int32_t* order;      // [n_links] processing order of one-thread-per-link kernels
  double* scratch;           // [12*n_links] post-collision population leaving through a link
  double* Uneed;             // [n_need*12] post-step U, one 96-byte row per node
};

// Moments with the collision's damping/source half step
// (three_d/curved_boundary_warp3d.py:2192-2260), summed over q in order.
__device__ __forceinline__ void moments3(const Ctx3& c, const double* __restrict__ f, int n,
                                         double* S) {
  const int N = c.N;
#pragma unroll
  for (int a = 0; a < kC3; ++a) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < kQ3; ++q) s += f[(size_t)(q * kC3 + a) * N + n];
    S[a] = s;
  }
  source_half3(c, S);
}

__device__ __forceinline__ void moments_node3(const Ctx3& c, const double* __restrict__ f0,
                                              double* __restrict__ U,
                                              double* __restrict__ ucol,
                                              double* __restrict__ ustar,
                                              int* __restrict__ invalid, int sweep_due, int n);

__global__ void __launch_bounds__(256) k3_moments(Ctx3 c, const double* __restrict__ f0,
                                                  double* __restrict__ U,
                                                  double* __restrict__ ucol,
                                                  double* __restrict__ ustar,
                                                  int* __restrict__ invalid, int sweep_due) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= c.N) return;
  moments_node3(c, f0, U, ucol, ustar, invalid, sweep_due, n);
}

// The moments of part of the nodes: LINKED = 0 the nodes without a cut link
// (one thread per node, the others return), LINKED = 1 the nodes of
// p.link_nodes (one thread per listed node).
template <int LINKED>
__global__ void __launch_bounds__(256) k3_moments_part(Ctx3 c, const double* __restrict__ f0,
                                                       double* __restrict__ U,
                                                       double* __restrict__ ucol,
                                                       double* __restrict__ ustar,
                                                       int* __restrict__ invalid,
                                                       int sweep_due) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const cvlbm3d_problem& p = c.p;
  int n;
  if (LINKED) {
    if (t >= p.n_link_nodes) return;
    n = p.link_nodes[t];
  } else {
    if (t >= c.N || p.node_link_start[t + 1] > p.node_link_start[t]) return;
    n = t;
  }
  moments_node3(c, f0, U, ucol, ustar, invalid, sweep_due, n);
}

__device__ __forceinline__ void moments_node3(const Ctx3& c, const double* __restrict__ f0,
                                              double* __restrict__ U,
                                              double* __restrict__ ucol,
                                              double* __restrict__ ustar,
                                              int* __restrict__ invalid, int sweep_due, int n) {
  const int N = c.N;
  const cvlbm3d_problem& p = c.p;
  double S[kC3];
  moments3(c, f0, n, S);
#pragma unroll
  for (int a = 0; a < kC3; ++a) U[(size_t)a * N + n] = S[a];
  const double hdt = 0.5 * p.dt;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double uu = ustar[(size_t)d * N + n] + hdt * S[d];
    ucol[(size_t)d * N + n] = uu;
    // with a sweep due, k3_sweep writes u* = (uu + hdt v) + (u_swept - uu)
    if (!sweep_due) ustar[(size_t)d * N + n] = uu + hdt * S[d];
  }
  if (det3(S[3], S[4], S[5], S[6], S[7], S[8], S[9], S[10], S[11]) <= c.m.jf) *invalid = 1;
}

// One Jacobi sweep (three_d/curved_boundary_warp3d.py:2402-2540); ucol holds
// the collide-time u of every node, the swept u goes to `u`.
// Loads of values that other blocks of the same launch write (the wavefront
// kernel): through L2 only, so that no stale L1 line is read.
template <bool CG>
__device__ __forceinline__ double ldx(const double* q) {
  if constexpr (CG)
    return __ldcg(q);
  else
    return *q;
}

template <bool CG>
__device__ __forceinline__ void sweep_node3(const Ctx3& c, const double* U, const double* ucol,
                                            double* __restrict__ u, double* __restrict__ ustar,
                                            const double* clock, double t_host, int n) {
  const int N = c.N;
  const cvlbm3d_problem& p = c.p;
  double d[3] = {0.0, 0.0, 0.0}, r[3] = {0.0, 0.0, 0.0};
  const double time = time_of(clock, t_host, 0.5 * p.dt);
  const double w2 = p.weight * p.weight;
  for (int k = p.node_link_start[n]; k < p.node_link_start[n + 1]; ++k) {
    const int ell = p.node_link_list[k];
    const int bid = p.link_bid[ell];
    bool force_all = false;
    if (p.disp_bid >= 0) {
      if (bid != p.disp_bid) continue;
      force_all = true;
    }
    const double x = p.link_xb[ell], y = p.link_yb[ell], z = p.link_zb[ell];
    const double dbx = x - ((double)p.active_i[n] + 0.5) * p.dx;
    const double dby = y - ((double)p.active_j[n] + 0.5) * p.dy;
    const double dbz = z - ((double)p.active_k[n] + 0.5) * p.dz;
    const int mode = p.bc_mode[bid];
    const double* pp = p.bc_params + bid * 16;
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      if (!(force_all || p.bc_comp_kind[comp * kMaxIds3 + bid] == kDirichlet)) continue;
      const double ub = disp3(mode, pp, comp, x, y, z, time);
      const double* F = U + (size_t)(3 + 3 * comp) * N;
      double e0 = ldx<CG>(F + n), e1 = ldx<CG>(F + (size_t)N + n),
             e2 = ldx<CG>(F + 2 * (size_t)N + n);
      if (comp == 0) e0 = e0 - 1.0;
      if (comp == 1) e1 = e1 - 1.0;
      if (comp == 2) e2 = e2 - 1.0;
      const double rhs = ub - (e0 * dbx + e1 * dby + e2 * dbz);
      d[comp] = d[comp] + w2;
      r[comp] = r[comp] + w2 * rhs;
    }
  }
  const double* Ub = U + 3 * (size_t)N;
  double Fs[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) Fs[k] = ldx<CG>(Ub + (size_t)k * N + n);
  int nb[kQ3];
#pragma unroll
  for (int q = 0; q < kQ3; ++q) nb[q] = p.neighbor[(size_t)q * N + n];
  // of (F_x dx + F_y dy + F_z dz) only the term on the direction's axis is formed:
  // the other two are products with an exact zero
  auto add = [&](int q, const double* e, const double* un) {
    const int ax = q % 3;
    const double h = q < 3 ? (ax == 0 ? p.dx : ax == 1 ? p.dy : p.dz)
                           : -(ax == 0 ? p.dx : ax == 1 ? p.dy : p.dz);
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      double v = Fs[3 * comp + ax] + e[comp];
      if (comp == ax) v = v - 2.0;
      r[comp] += un[comp] - 0.5 * (v * h);
      d[comp] += 1.0;
    }
  };
  if ((nb[0] | nb[1] | nb[2] | nb[3] | nb[4] | nb[5]) >= 0) {
    // all six neighbours: no load waits for a sum; the kernel's 64 registers hold only part
    // of the 36 values at once
    double e[kQ3][3], un[kQ3][3];
#pragma unroll
    for (int q = 0; q < kQ3; ++q) {
#pragma unroll
      for (int comp = 0; comp < 3; ++comp) {
        e[q][comp] = ldx<CG>(Ub + (size_t)(3 * comp + q % 3) * N + nb[q]);
        un[q][comp] = ldx<CG>(ucol + (size_t)comp * N + nb[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < kQ3; ++q) add(q, e[q], un[q]);
  } else {
#pragma unroll
    for (int q = 0; q < kQ3; ++q) {
      if (nb[q] < 0) continue;
      double e[3], un[3];
#pragma unroll
      for (int comp = 0; comp < 3; ++comp) {
        e[comp] = ldx<CG>(Ub + (size_t)(3 * comp + q % 3) * N + nb[q]);
        un[comp] = ldx<CG>(ucol + (size_t)comp * N + nb[q]);
      }
      add(q, e, un);
    }
  }
  const double hdt = 0.5 * p.dt;
#pragma unroll
  for (int comp = 0; comp < 3; ++comp) {
    const double uo = ldx<CG>(ucol + (size_t)comp * N + n);
    double un = uo;
    if (d[comp] > 0.0) un = uo + p.relax * (sweep_quot3(c, r[comp], d[comp]) - uo);
    u[(size_t)comp * N + n] = un;
    ustar[(size_t)comp * N + n] = (uo + hdt * ldx<CG>(U + (size_t)comp * N + n)) + (un - uo);
  }
}

// The neighbours' values are scattered loads that miss L1 at the plane neighbours:
// bound by their latency, so warps count (four blocks of 256, 64 registers: shell176
// 4,799 us per four steps against 4,863 with three and 5,057 with two).
__global__ void __launch_bounds__(256, 4) k3_sweep(Ctx3 c, const double* __restrict__ U,
                                                const double* __restrict__ ucol,
                                                double* __restrict__ u,
                                                double* __restrict__ ustar, const double* clock,
                                                double t_host) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= c.N) return;
  sweep_node3<false>(c, U, ucol, u, ustar, clock, t_host, n);
}

// The material of a kernel: the problem's, its law fixed when compiled for one.
template <int MAT>
__device__ __forceinline__ Mat mat3(const Ctx3& c) {
  Mat m = c.m;
  if (MAT >= 0) m.model = MAT;
  return m;
}

// Collision + F repair + push streaming of one node with its state in registers and
// the six directions unrolled (the wavefront kernel's collide items).
//
// The moments come from U, which the moments wrote this step, and P(F), P(F_repaired) are evaluated once per node.  Each direction is then 12
// coalesced loads of f0 and 12 stores to f1 at the neighbour, with the
// direction a compile-time constant: of the three terms s_x f_x + s_y f_y +
// s_z f_z of the equilibrium flux only the one on the direction's axis is
// formed (the others are products with an exact zero, which change no finite
// sum).
struct NodeState3 {
  double S[kC3];
  double Po[9];  // P(F)
  double dP[9];  // P(F_repaired) - P(F)
  double dF[9];  // F_repaired - F
  int nb[kQ3];
  bool repaired;
};

// Moments, neighbours, P(F), the F repair and its Piola difference; the U
// and U_need rows of the node.
template <int MAT, bool CG = false>
__device__ __forceinline__ void node_prologue3(const Ctx3& c, const Fused3& fz, double* U,
                                               const double* u, int do_repair, int store_all,
                                               int n, NodeState3& st) {
  const int N = c.N;
  const cvlbm3d_problem& p = c.p;
  const Mat m = mat3<MAT>(c);
#pragma unroll
  for (int a = 0; a < kC3; ++a) st.S[a] = ldx<CG>(U + (size_t)a * N + n);
#pragma unroll
  for (int q = 0; q < kQ3; ++q) st.nb[q] = p.neighbor[(size_t)q * N + n];
  const double* F = st.S + 3;
  {
    const M3 P = piola3(F, m);
#pragma unroll
    for (int k = 0; k < 9; ++k) st.Po[k] = P.v[k];
  }
  st.repaired = false;
  double nn[9];
  if (do_repair) {
    // I + grad u of the swept u, as du_axis3: centred with both neighbours,
    // second-order one-sided with two on one side, first order with one,
    // zero with none
    double T[9];
#pragma unroll
    for (int comp = 0; comp < 3; ++comp) {
      const double* uc = u + (size_t)comp * N;
      const double u0 = ldx<CG>(uc + n);
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        const int pp = st.nb[ax], pm = st.nb[ax + 3];
        const DivC &h1 = c.h1[ax], &h2 = c.h2[ax];
        double g = 0.0;
        if (pp >= 0 && pm >= 0) {
          g = divc(ldx<CG>(uc + pp) - ldx<CG>(uc + pm), h2);
        } else if (pp >= 0) {
          const int pp2 = p.neighbor[(size_t)ax * N + pp];
          if (pp2 >= 0)
            g = divc(-3.0 * u0 + 4.0 * ldx<CG>(uc + pp) - ldx<CG>(uc + pp2), h2);
          else
            g = divc(ldx<CG>(uc + pp) - u0, h1);
        } else if (pm >= 0) {
          const int pm2 = p.neighbor[(size_t)(ax + 3) * N + pm];
          if (pm2 >= 0)
            g = divc(3.0 * u0 - 4.0 * ldx<CG>(uc + pm) + ldx<CG>(uc + pm2), h2);
          else
            g = divc(u0 - ldx<CG>(uc + pm), h1);
        }
        T[3 * comp + ax] = comp == ax ? 1.0 + g : g;
      }
    }
    const double beta = fmax(0.0, fmin(1.0, p.blend));
#pragma unroll
    for (int k = 0; k < 9; ++k) nn[k] = F[k] + beta * (T[k] - F[k]);
    if (det3v(nn) > m.jf) {
      st.repaired = true;
      const M3 P = piola3(nn, m);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        st.dP[k] = P.v[k] - st.Po[k];
        st.dF[k] = nn[k] - F[k];
      }
    }
  }
  if (st.repaired && store_all) {
#pragma unroll
    for (int k = 0; k < 9; ++k) U[(size_t)(3 + k) * N + n] = nn[k];
  }
  const int slot = fz.need_slot[n];
  if (slot >= 0) {
    double* rowp = fz.Uneed + (size_t)slot * kC3;
    rowp[0] = st.S[0];
    rowp[1] = st.S[1];
    rowp[2] = st.S[2];
#pragma unroll
    for (int k = 0; k < 9; ++k) rowp[3 + k] = st.repaired ? nn[k] : F[k];
  }
}

template <int Q>
__device__ __forceinline__ void collide_dir3(const Ctx3& c, const Fused3& fz,
                                             const NodeState3& st,
                                             const double* __restrict__ f0,
                                             double* __restrict__ f1, int N, int n) {
  constexpr int ax = Q % 3;
  constexpr double s = Q < 3 ? 1.0 : -1.0;
  const cvlbm3d_problem& p = c.p;
  const double k3c = c.k3c, sixth = 1.0 / 6.0, om = p.omega, sw = c.sw, ff = c.ff;
  const int nq = st.nb[Q];
  double* dst;
  size_t stride;  // pointers advance row by row: one 64-bit addition per access
  if (nq >= 0) {
    dst = f1 + (size_t)(Q * kC3) * N + nq;
    stride = (size_t)N;
  } else {
    int ell = -1;
    for (int k = p.node_link_start[n]; k < p.node_link_start[n + 1]; ++k) {
      const int e = p.node_link_list[k];
      if (p.link_q[e] == Q) ell = e;
    }
    if (ell < 0) return;
    dst = fz.scratch + (size_t)ell * kC3;
    stride = 1;
  }
  const double* src = f0 + (size_t)(Q * kC3) * N + n;
  double old[kC3];
#pragma unroll
  for (int a = 0; a < kC3; ++a) {
    old[a] = *src;
    src += N;
  }
#pragma unroll
  for (int a = 0; a < kC3; ++a) {
    double fe;
    if (a < 3) {
      fe = sixth * (st.S[a] + k3c * (s * -st.Po[3 * a + ax]));
    } else if ((a - 3) % 3 == ax) {
      fe = sixth * (st.S[a] + k3c * (s * -st.S[(a - 3) / 3]));
    } else {
      fe = sixth * st.S[a];
    }
    double val = old[a] + om * (fe - old[a]) + sw * source_comp3(a, p.source_mode, p.source, st.S);
    if (st.repaired) {
      if (a < 3)
        val = val - ff * (s * st.dP[3 * a + ax]);
      else
        val = val + sixth * st.dF[a - 3];
    }
    *dst = val;
    dst += stride;
  }
}

// Collision + F repair + push streaming, one thread per node.
//
// Bound by memory and by how much of it is in flight: it moves about 1.3 KB per
// node (f0, f1, U, the swept u, neighbours) at 4.0 TB/s on shell128 (248 us;
// copying 72 such rows alone reaches 5.3 TB/s with the shifted stores).  What the
// layout is after:
//  * little code: the six directions are one loop body, the rows of the axis'
//    column picked at run time, so the kernel fits the instruction cache.  The
//    former form, six unrolled directions with the state in registers (271 us,
//    kept for the wavefront kernel), waited 2.8 of 18 cycles per issue for
//    instructions, and every material law was compiled into one kernel.
//  * the node's state (S, P, the changes of P and F: 39 doubles) in shared memory,
//    a column per thread, so that the loop can index it and the registers hold the
//    populations in flight.
//  * the repair's gradient on a straight path when all six neighbours exist.
//  * L1: 12 warps' worth of staging for all 72 rows (cp.async) left no room in L1
//    for the lines in flight and for the sectors that neighbouring warps share, and
//    was slower (377 us); so were more resident blocks, prefetches to L2, one warp
//    per direction (312 us) and rotating the state through registers (6 to 12 %).
//
// MAT >= 0: compiled for that material law.  MINB resident blocks per SM bound the
// registers per thread.  MOM (a step without sweep and repair): the moments are formed
// here instead of by k3_moments; f0 then crosses HBM once per step and U only on the
// last step (affine3d, 112^3: 57 + 128 us in two kernels).
constexpr int kCT3 = 128;               // nodes per block
constexpr int kCState3 = kC3 + 3 * 9;   // S (12), P(F) (9), change of P (9), change of F / 6 (9)

constexpr int kCollideSmem3 = sizeof(double) * kCState3 * kCT3;

template <int MAT, int MINB, bool MOM>
__global__ void __launch_bounds__(kCT3, MINB)
    k3_collide(Ctx3 c, Fused3 fz, const double* __restrict__ f0, double* __restrict__ f1,
               double* __restrict__ U, const double* __restrict__ u, int do_repair,
               int store_all, double* __restrict__ uw, double* __restrict__ ustar,
               int* __restrict__ invalid) {
  extern __shared__ double sm3[];  // [kCState3][kCT3]; every thread uses its own column
  const int N = c.N, tid = threadIdx.x;
  const int n = blockIdx.x * kCT3 + tid;
  if (n >= N) return;
  const cvlbm3d_problem& p = c.p;
  const double sixth = 1.0 / 6.0;
  double* sS = sm3 + tid;
  double* sP = sS + kC3 * kCT3;
  double* sdP = sP + 9 * kCT3;
  double* sdF = sdP + 9 * kCT3;
  int nb[kQ3];
#pragma unroll
  for (int q = 0; q < kQ3; ++q) nb[q] = p.neighbor[(size_t)q * N + n];
  const int slot = fz.need_slot[n];
  double S[kC3];
  if constexpr (MOM) {
    // neither sweep nor repair this step: the work of k3_moments, the collision's own
    // reads of f0 below then come from L2
    moments3(c, f0, n, S);
    if (store_all) {
#pragma unroll
      for (int a = 0; a < kC3; ++a) U[(size_t)a * N + n] = S[a];
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double uu = ustar[(size_t)d * N + n] + c.hdt * S[d];
      uw[(size_t)d * N + n] = uu;
      ustar[(size_t)d * N + n] = uu + c.hdt * S[d];
    }
    if (det3(S[3], S[4], S[5], S[6], S[7], S[8], S[9], S[10], S[11]) <= c.m.jf) *invalid = 1;
  } else {
    const double* src = U + n;
#pragma unroll
    for (int a = 0; a < kC3; ++a) {
      S[a] = *src;
      src += N;
    }
  }
  bool repaired = false;
  {
    const Mat m = mat3<MAT>(c);
    const double* F = S + 3;
    double nn[9];
    if (do_repair) {
      // I + grad u of the swept u, as du_axis3: centred with both neighbours, second
      // order one-sided with two on one side, first order with one, zero with none
      double* sT = sdF;
      if ((nb[0] | nb[1] | nb[2] | nb[3] | nb[4] | nb[5]) >= 0) {
        double num[9];
        const double* uc = u;
#pragma unroll
        for (int comp = 0; comp < 3; ++comp) {
#pragma unroll
          for (int ax = 0; ax < 3; ++ax) num[3 * comp + ax] = uc[nb[ax]] - uc[nb[ax + 3]];
          uc += N;
        }
#pragma unroll
        for (int k = 0; k < 9; ++k) sT[k * kCT3] = divc(num[k], c.h2[k % 3]);
      } else {
#pragma unroll 1
        for (int ax = 0; ax < 3; ++ax) {
          const int pp = ax == 0 ? nb[0] : ax == 1 ? nb[1] : nb[2];
          const int pm = ax == 0 ? nb[3] : ax == 1 ? nb[4] : nb[5];
          const int pp2 = pp >= 0 && pm < 0 ? p.neighbor[(size_t)ax * N + pp] : -1;
          const int pm2 = pm >= 0 && pp < 0 ? p.neighbor[(size_t)(ax + 3) * N + pm] : -1;
#pragma unroll 1
          for (int comp = 0; comp < 3; ++comp) {
            const double* uc = u + (size_t)comp * N;
            const double u0 = uc[n];
            double num = 0.0;
            bool two = true;  // divided by 2 h (else by h)
            if (pp >= 0 && pm >= 0) {
              num = uc[pp] - uc[pm];
            } else if (pp >= 0) {
              two = pp2 >= 0;
              num = two ? -3.0 * u0 + 4.0 * uc[pp] - uc[pp2] : uc[pp] - u0;
            } else if (pm >= 0) {
              two = pm2 >= 0;
              num = two ? 3.0 * u0 - 4.0 * uc[pm] + uc[pm2] : u0 - uc[pm];
            }
            sT[(3 * comp + ax) * kCT3] = divc(num, two ? c.h2[ax] : c.h1[ax]);
          }
        }
      }
      const double beta = fmax(0.0, fmin(1.0, p.blend));
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        const double g = sT[k * kCT3];
        const double T = k % 4 == 0 ? 1.0 + g : g;
        nn[k] = F[k] + beta * (T - F[k]);
      }
      repaired = det3v(nn) > m.jf;
    }
#pragma unroll
    for (int a = 0; a < kC3; ++a) sS[a * kCT3] = S[a];
    if (slot >= 0) {
      double* rowp = fz.Uneed + (size_t)slot * kC3;
      rowp[0] = S[0];
      rowp[1] = S[1];
      rowp[2] = S[2];
#pragma unroll
      for (int k = 0; k < 9; ++k) rowp[3 + k] = repaired ? nn[k] : F[k];
    }
    if (repaired && store_all) {
#pragma unroll
      for (int k = 0; k < 9; ++k) U[(size_t)(3 + k) * N + n] = nn[k];
    }
    const M3 Po = piola3(F, m);
#pragma unroll
    for (int k = 0; k < 9; ++k) sP[k * kCT3] = Po.v[k];
    if (repaired) {
      const M3 Pn = piola3(nn, m);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        sdP[k * kCT3] = Pn.v[k] - Po.v[k];
        sdF[k * kCT3] = sixth * (nn[k] - F[k]);
      }
    }
  }
  const double k3c = c.k3c, om = p.omega, ff = c.ff;
  const bool src_v = p.source_mode != kSrcNone, src_f = p.source_mode == kSrcConstant;
  // the 12 populations of direction q, the F rows in the order of its columns
  auto load_dir = [&](int q, double* old) {
    const int ax = q < 3 ? q : q - 3;
    const int c1 = ax == 2 ? 0 : ax + 1, c2 = ax == 0 ? 2 : ax - 1;
    const double* src = f0 + (size_t)(q * kC3) * N + n;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      old[a] = *src;
      src += N;
    }
    const size_t o[3] = {(size_t)ax * N, (size_t)c1 * N, (size_t)c2 * N};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
      for (int j = 0; j < 3; ++j) old[3 + 3 * i + j] = src[o[j]];
      src += 3 * (size_t)N;
    }
  };
  auto push_dir = [&](int q, const double* old) {
    const int ax = q < 3 ? q : q - 3;
    const int c1 = ax == 2 ? 0 : ax + 1, c2 = ax == 0 ? 2 : ax - 1;
    const int col[3] = {ax, c1, c2};  // the axis' own F column first
    const int nq = q == 0 ? nb[0] : q == 1 ? nb[1] : q == 2 ? nb[2] : q == 3 ? nb[3] : q == 4 ? nb[4] : nb[5];
    double* d;
    size_t stride = (size_t)N;
    if (nq >= 0) {
      d = f1 + (size_t)(q * kC3) * N + nq;
    } else {
      int ell = -1;
      for (int k = p.node_link_start[n]; k < p.node_link_start[n + 1]; ++k) {
        const int e = p.node_link_list[k];
        if (p.link_q[e] == q) ell = e;
      }
      if (ell < 0) return;
      d = fz.scratch + (size_t)ell * kC3;
      stride = 1;
    }
    // velocity rows: flux -P in the axis' column, its sign that of the direction
    const double s = q < 3 ? 1.0 : -1.0;
    const double* pP = sP + ax * kCT3;
    const double* pdP = sdP + ax * kCT3;
    double vel[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      vel[a] = sS[a * kCT3];
      const double fe = sixth * (vel[a] + k3c * (s * -pP[3 * a * kCT3]));
      double val = old[a] + om * (fe - old[a]);
      if (src_v) val = val + c.sw * source_comp3(a, p.source_mode, p.source, vel);
      if (repaired) val = val - ff * (s * pdP[3 * a * kCT3]);
      *d = val;
      d += stride;
    }
    // F rows: flux -v in the axis' column
    const size_t o[3] = {(size_t)col[0] * stride, (size_t)col[1] * stride, (size_t)col[2] * stride};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int k = 3 * i + col[j];
        const double Sa = sS[(3 + k) * kCT3];
        const double fe = j == 0 ? sixth * (Sa + k3c * (s * -vel[i])) : sixth * Sa;
        const double v = old[3 + 3 * i + j];
        double val = v + om * (fe - v);
        if (src_f) val = val + c.sw * p.source[3 + k];
        if (repaired) val = val + sdF[k * kCT3];
        d[o[j]] = val;
      }
      d += 3 * stride;
    }
  };
  double va[kC3];
#pragma unroll 1
  for (int q = 0; q < kQ3; ++q) {
    load_dir(q, va);
    push_dir(q, va);
  }
}

using CollideFn3 = void (*)(Ctx3, Fused3, const double*, double*, double*, const double*, int, int,
                            double*, double*, int*);

// The collision compiled for the problem's material law.
template <int MINB, bool MOM>
CollideFn3 collide3(int model) {
  switch (model) {
    case kMatSVK: return k3_collide<kMatSVK, MINB, MOM>;
    case kMatNeoHooke: return k3_collide<kMatNeoHooke, MINB, MOM>;
    case kMatLogNeoHooke: return k3_collide<kMatLogNeoHooke, MINB, MOM>;
    case kMatMooneyRivlin: return k3_collide<kMatMooneyRivlin, MINB, MOM>;
    case kMatYeoh: return k3_collide<kMatYeoh, MINB, MOM>;
    case kMatGent: return k3_collide<kMatGent, MINB, MOM>;
    case kMatSix: return k3_collide<kMatSix, MINB, MOM>;
    default: return k3_collide<-1, MINB, MOM>;
  }
}

// ---------------------------------------------------------------------------
// Wavefront form of the node work (node_variant 3): the moments, sweep and
// collide of chunks of one x-plane (the slowest index of the active order)
// in ONE persistent launch.  Blocks take work items from a ticket counter in
// the order  moments(w), sweep(w-1), collide(w-3)  for w = 0, 1, ..., so the
// collide of a plane re-reads f0 a few planes after the moments read it,
// while it is still in L2: f0 crosses HBM once per step instead of twice.
// Dependencies (whole planes): the sweep of plane i needs the moments of
// planes i-1..i+1 (+-x neighbours, same-plane +-y/z); the collide of plane i
// needs the sweep of planes i-2..i+2 (repair stencil +-2) - which also
// orders it after every read of its U by a neighbouring sweep.  A block
// waits only on items with lower tickets, which are held by running blocks,
// so the order cannot deadlock; every wait is bounded all the same, and a
// wait that runs out sets the timeout flag and the invalid flag and goes on
// (a wrong step, never a hung device).  Values other blocks of the launch
// write (U, collide-time u, swept u) are read through L2 only (ldx<true>).
// ---------------------------------------------------------------------------
struct Wave3 {
  const int4* items;         // [n_items] (stage, plane, first active id, end active id)
  int n_items, n_planes;
  const int32_t* chunks;     // [n_planes] items of one stage per plane
  int32_t* sync;             // [2 + 3*n_planes] ticket, timeout flag, done counters
};

// A wait gives up after this many polls (about a quarter of a second); the
// first wait that gives up makes every later wait of the launch return at
// once, so a broken dependency costs one bound, not one per item.
constexpr long long kWaveMaxSpins = 1LL << 20;

template <int MINB>
__global__ void __launch_bounds__(128, MINB)
    k3_wave(Ctx3 c, Fused3 fz, Wave3 wv, const double* __restrict__ f0, double* __restrict__ f1,
            double* U, double* ucol, double* u, double* ustar, int* __restrict__ invalid,
            const double* clock, double t_host, int sweep_due, int do_repair, int store_all) {
  __shared__ int s_item;
  int* ticket = wv.sync;
  int* timeout = wv.sync + 1;
  int* done = wv.sync + 2;
  const int N = c.N;
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(ticket, 1);
    __syncthreads();
    const int it = s_item;
    __syncthreads();  // s_item is rewritten only after every thread has read it
    if (it >= wv.n_items) return;
    const int4 w = wv.items[it];
    const int stage = w.x, plane = w.y;
    if (stage > 0 && threadIdx.x == 0) {
      const int dep = stage - 1;
      const int r = stage == 1 ? 1 : 2;
      const int lo = plane - r < 0 ? 0 : plane - r;
      const int hi = plane + r >= wv.n_planes ? wv.n_planes - 1 : plane + r;
      const volatile int* gave_up = timeout;
      for (int pl = lo; pl <= hi && !*gave_up; ++pl) {
        const int want = wv.chunks[pl];
        const volatile int* d = done + dep * wv.n_planes + pl;
        long long spins = 0;
        while (*d < want && !*gave_up) {
          if (++spins > kWaveMaxSpins) {
            atomicExch(timeout, 1);
            atomicExch(invalid, 1);
            break;
          }
          __nanosleep(64);
        }
      }
      __threadfence();
    }
    __syncthreads();
    const int n = w.z + (int)threadIdx.x;
    if (n < w.w) {
      if (stage == 0) {
        moments_node3(c, f0, U, sweep_due ? ucol : u, ustar, invalid, sweep_due, n);
      } else if (stage == 1) {
        if (sweep_due) sweep_node3<true>(c, U, ucol, u, ustar, clock, t_host, n);
      } else {
        NodeState3 st;
        node_prologue3<-1, true>(c, fz, U, u, do_repair, store_all, n, st);
        collide_dir3<0>(c, fz, st, f0, f1, N, n);
        collide_dir3<1>(c, fz, st, f0, f1, N, n);
        collide_dir3<2>(c, fz, st, f0, f1, N, n);
        collide_dir3<3>(c, fz, st, f0, f1, N, n);
        collide_dir3<4>(c, fz, st, f0, f1, N, n);
        collide_dir3<5>(c, fz, st, f0, f1, N, n);
      }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) atomicAdd(done + stage * wv.n_planes + plane, 1);
  }
}

// -- link kernels -------------------------------------------------------------
constexpr int kGatherLanes = 16;  // lanes per link in the gather (12 components used)

// Value and gradients of the 12 components at a link from its <= 64
// characteristic samples, in slot order (_sparse_characteristic_gather,
// :2675-2700).  A block takes 8 consecutive links: their sample slots and
// weights are staged in shared memory with coalesced loads, then the 12
// lanes of a link read one 96-byte U_need row per sample, 16 samples per
// batch of independent loads.
constexpr int kGatherLinks = 128 / kGatherLanes;

__global__ void __launch_bounds__(128)
    k3_link_gather(Ctx3 c, Fused3 fz, double* __restrict__ char_state) {
  __shared__ int s_slot[kGatherLinks][kChar];
  __shared__ double s_w[kGatherLinks][4][kChar];
  const cvlbm3d_problem& p = c.p;
  const int L = p.n_links;
  const int ell0 = blockIdx.x * kGatherLinks;
  for (int t = threadIdx.x; t < kChar * kGatherLinks; t += blockDim.x) {
    const int mm = t / kGatherLinks, g = t % kGatherLinks;
    const int ell = ell0 + g;
    s_slot[g][mm] = ell < L ? fz.char_slot[(size_t)mm * L + ell] : -1;
#pragma unroll
    for (int k = 0; k < 4; ++k)
      s_w[g][k][mm] = ell < L ? p.char_w[((size_t)k * kChar + mm) * L + ell] : 0.0;
  }
  __syncthreads();
  const int a = threadIdx.x % kGatherLanes;
  const int g = threadIdx.x / kGatherLanes;
  const int ell = ell0 + g;
  if (ell >= L || a >= kC3 || p.char_idx[ell] < 0) return;
  double v0 = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
  constexpr int kChunk = 16;
#pragma unroll 1
  for (int m0 = 0; m0 < kChar; m0 += kChunk) {
    double uv[kChunk];
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
      const int q = s_slot[g][m0 + k];
      uv[k] = q >= 0 ? fz.Uneed[(size_t)q * kC3 + a] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
      const int mm = m0 + k;
      if (s_slot[g][mm] >= 0) {
        v0 += s_w[g][0][mm] * uv[k];
        gx += s_w[g][1][mm] * uv[k];
        gy += s_w[g][2][mm] * uv[k];
        gz += s_w[g][3][mm] * uv[k];
      }
    }
  }
  char_state[((size_t)0 * 12 + a) * L + ell] = v0;
  char_state[((size_t)1 * 12 + a) * L + ell] = gx;
  char_state[((size_t)2 * 12 + a) * L + ell] = gy;
  char_state[((size_t)3 * 12 + a) * L + ell] = gz;
}

// The same gather with 4 lanes per link, 3 components per lane and 32 links
// per block, from the link-major copies of the tables (char_slot_lm
// [n_links][64], char_w_lm [n_links][64][4]): a sample's slot and four
// weights are one 4-byte and two 16-byte loads shared by the link's lanes,
// every lane does useful work (the 16-lane form leaves 4 of 16 idle), and
// each lane runs 12 independent accumulations.  Each of the 48 sums runs
// over the samples in slot order, as in k3_link_gather (the same doubles).
constexpr int kGather4Lanes = 4;
constexpr int kGather4Links = 128 / kGather4Lanes;

__global__ void __launch_bounds__(128)
    k3_link_gather4(Ctx3 c, Fused3 fz, double* __restrict__ char_state) {
  // the block's 32 x 64 sample slots, staged with coalesced 16-byte loads so
  // that each chunk of samples waits for one load level (weights and U rows
  // together) instead of two (the slot, then its U row)
  __shared__ int4 s_slot4[kGather4Links * kChar / 4];
  const cvlbm3d_problem& p = c.p;
  const int L = p.n_links;
  const int ell0 = blockIdx.x * kGather4Links;
  const int nl = L - ell0 < kGather4Links ? L - ell0 : kGather4Links;
  const int4* src = reinterpret_cast<const int4*>(p.char_slot_lm + (size_t)ell0 * kChar);
  for (int t = threadIdx.x; t < kGather4Links * kChar / 4; t += blockDim.x)
    s_slot4[t] = t < nl * (kChar / 4) ? src[t] : make_int4(-1, -1, -1, -1);
  __syncthreads();
  const int lane = threadIdx.x % kGather4Lanes;
  const int g = threadIdx.x / kGather4Lanes;
  const int ell = ell0 + g;
  if (ell >= L || p.char_idx[ell] < 0) return;
  const int a0 = 3 * lane;
  const int* slot = reinterpret_cast<const int*>(s_slot4) + g * kChar;
  const double2* w2 = reinterpret_cast<const double2*>(p.char_w_lm + (size_t)ell * kChar * 4);
  double acc[3][4];
#pragma unroll
  for (int cc = 0; cc < 3; ++cc)
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[cc][k] = 0.0;
  constexpr int kChunk = 8;
#pragma unroll 1
  for (int m0 = 0; m0 < kChar; m0 += kChunk) {
    int q[kChunk];
    double2 wa[kChunk], wb[kChunk];
    double uv[kChunk][3];
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
      q[k] = slot[m0 + k];
      wa[k] = w2[2 * (m0 + k)];
      wb[k] = w2[2 * (m0 + k) + 1];
    }
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
      const double* row = fz.Uneed + (size_t)(q[k] >= 0 ? q[k] : 0) * kC3 + a0;
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) uv[k][cc] = q[k] >= 0 ? row[cc] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
      if (q[k] >= 0) {
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
          acc[cc][0] += wa[k].x * uv[k][cc];
          acc[cc][1] += wa[k].y * uv[k][cc];
          acc[cc][2] += wb[k].x * uv[k][cc];
          acc[cc][3] += wb[k].y * uv[k][cc];
        }
      }
    }
  }
#pragma unroll
  for (int cc = 0; cc < 3; ++cc)
#pragma unroll
    for (int k = 0; k < 4; ++k) char_state[((size_t)k * 12 + a0 + cc) * L + ell] = acc[cc][k];
}

// F predictor of the link from U at the node and its upstream node (BFL and
// compat_bfl reconstructions, :2887-2990), tangential image from the LSQ stencil.
static __device__ __noinline__ void predictor3(const Ctx3& c, const Fused3& fz, int ell,
                                               const double* u, double* F) {
  const cvlbm3d_problem& p = c.p;
  const int N = c.N, n = p.link_p[ell], upid = p.link_up[ell];
  const double eta = p.link_eta[ell];
  const double* Un = fz.Uneed + (size_t)fz.need_slot[n] * kC3;
  for (int k = 0; k < 9; ++k) F[k] = Un[3 + k];
  if (!(p.recon == 2 || p.recon == 4)) return;
  if (upid >= 0) {
    const double* Uu = fz.Uneed + (size_t)fz.need_slot[upid] * kC3;
    for (int k = 0; k < 9; ++k) F[k] = Un[3 + k] + eta * (Un[3 + k] - Uu[3 + k]);
  }
  if (p.recon == 2 && p.has_tangent_lsq && p.lsq_valid[ell] != 0) {
    Frame3 fr = frame3(p.link_nx[ell], p.link_ny[ell], p.link_nz[ell]);
    double du1[3] = {0, 0, 0}, du2[3] = {0, 0, 0}, wt_abs = 0.0;
    for (int mm = 0; mm < kMaxLsq3; ++mm) {
      const int q = p.lsq_p[(size_t)ell * kMaxLsq3 + mm];
      if (q >= 0) {
        const double w1 = p.lsq_wt1[(size_t)ell * kMaxLsq3 + mm];
        const double w2 = p.lsq_wt2[(size_t)ell * kMaxLsq3 + mm];
        for (int r = 0; r < 3; ++r) {
          du1[r] += w1 * u[(size_t)r * N + q];
          du2[r] += w2 * u[(size_t)r * N + q];
        }
        wt_abs += fabs(w1) + fabs(w2);
      }
    }
    if (wt_abs > 0.0) {
      double h[3], g1[3], g2[3];
      for (int r = 0; r < 3; ++r) {
        h[r] = F[3 * r] * fr.n[0] + F[3 * r + 1] * fr.n[1] + F[3 * r + 2] * fr.n[2];
        g1[r] = fr.t1[r] + du1[r];
        g2[r] = fr.t2[r] + du2[r];
      }
      for (int r = 0; r < 3; ++r)
        for (int s = 0; s < 3; ++s)
          F[3 * r + s] = h[r] * fr.n[s] + g1[r] * fr.t1[s] + g2[r] * fr.t2[s];
    }
  }
}

// Boundary value, F predictor, Newton normal solve and P(F_b) of one link;
// the results go to the link buffers (link_kind .. link_Pb), which the
// reference also exposes (three_d/curved_boundary_warp3d.py:4281-4337).
__global__ void __launch_bounds__(128)
    k3_link_prepare(const __grid_constant__ Ctx3 c, const __grid_constant__ Fused3 fz,
                    const double* __restrict__ u, cvlbm3d_fields fl, const double* clock, double t_host, double offset) {
  const cvlbm3d_problem& p = c.p;
  const Mat& m = c.m;
  const int L = p.n_links, N = c.N;
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= L) return;
  const int ell = fz.order ? fz.order[slot] : slot;
  const double t = time_of(clock, t_host, offset);
  const int bid = p.link_bid[ell];
  const int kind = p.bc_kind[bid], mode = p.bc_mode[bid];
  int ck[3];
  for (int r = 0; r < 3; ++r) ck[r] = p.bc_comp_kind[r * kMaxIds3 + bid];
  const double* pp = p.bc_params + bid * 16;
  const double x = p.link_xb[ell], y = p.link_yb[ell], z = p.link_zb[ell];
  const double nx = p.link_nx[ell], ny = p.link_ny[ell], nz = p.link_nz[ell];
  const int n = p.link_p[ell];
  const int upid = p.link_up[ell];
  const double eta = p.link_eta[ell];
  double T[3];
  for (int r = 0; r < 3; ++r) T[r] = value3(r, mode, pp, x, y, z, nx, ny, nz, t, m.jf);
  if (p.dyn_enabled && p.dyn_enabled[ell] != 0)
    for (int r = 0; r < 3; ++r) T[r] = p.dyn_traction[(size_t)r * L + ell];
  double Fb[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  double Pb[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  const bool anyN = ck[0] == kNeumann || ck[1] == kNeumann || ck[2] == kNeumann;
  if (anyN) {
    double F[9];
    if (p.recon != 3) predictor3(c, fz, ell, u, F);
    if (p.recon == 3 && p.has_char && p.char_idx[ell] >= 0)
      for (int k = 0; k < 9; ++k) F[k] = fl.char_state[((size_t)0 * 12 + 3 + k) * L + ell];
    else if (p.recon == 3)
      for (int k = 0; k < 9; ++k) F[k] = 0.0;
    for (int k = 0; k < 9; ++k) Fb[k] = F[k];
    if (ck[0] == kNeumann && ck[1] == kNeumann && ck[2] == kNeumann)
      solve_Fb3(F, nx, ny, nz, T, m, p.normal_solver, Fb);
    else if (ck[0] == kNeumann || ck[1] == kNeumann || ck[2] == kNeumann)
      solve_Fb3_mixed(F, nx, ny, nz, T, ck, m, p.normal_solver, Fb);
    const M3 P = piola3(Fb, m);
    for (int k = 0; k < 9; ++k) Pb[k] = P.v[k];
  }
  fl.link_kind[ell] = kind;
  for (int r = 0; r < 3; ++r) {
    fl.link_comp_kind[(size_t)r * L + ell] = ck[r];
    fl.link_bv[(size_t)r * L + ell] = T[r];
  }
  for (int k = 0; k < 9; ++k) {
    fl.link_Fb[(size_t)k * L + ell] = Fb[k];
    fl.link_Pb[(size_t)k * L + ell] = Pb[k];
  }
}

__device__ __forceinline__ bool char_rows3(const cvlbm3d_problem& p, int ell) {
  return p.has_char && p.char_idx[ell] >= 0;
}

// BFL value of row `a` of one link (:3154-3241) with the outgoing populations
// taken from link_scratch and the post-stream f1.
__global__ void __launch_bounds__(128)
    k3_link_rows(Ctx3 c, Fused3 fz, double* __restrict__ f1, cvlbm3d_fields fl) {
  const cvlbm3d_problem& p = c.p;
  const int L = p.n_links, N = c.N;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)L * kC3) return;
  const int ell = (int)(t / kC3), a = (int)(t - (long long)ell * kC3);
  const int row = a < 3 ? a : (a - 3) / 3;
  const int ckr = fl.link_comp_kind[(size_t)row * L + ell];
  const bool anyN = fl.link_comp_kind[ell] == kNeumann ||
                    fl.link_comp_kind[(size_t)L + ell] == kNeumann ||
                    fl.link_comp_kind[2 * (size_t)L + ell] == kNeumann;
  // rows the characteristic closure overwrites are written by k3_link_char
  if (anyN && ckr == kNeumann && char_rows3(p, ell)) return;
  const int n = p.link_p[ell], upid = p.link_up[ell], qo = p.link_q[ell];
  const int qi = opp3(qo);
  double eta = p.link_eta[ell];
  if (p.recon == 1) eta = 0.5;
  const double din[3] = {(double)dx3(qi), (double)dy3(qi), (double)dz3(qi)};
  double D = 1.0, S = 0.0;
  if (ckr == kDirichlet) {
    const double Tr = fl.link_bv[(size_t)row * L + ell];
    if (a < 3) {
      D = -1.0;
      S = divc(fl.link_bv[(size_t)a * L + ell], c.d3);
    } else {
      const int col = (a - 3) - row * 3;
      S = divc(-din[col] * Tr, c.dc);
    }
  } else {
    if (a < 3) {
      const double* Pb = fl.link_Pb;
      S = divc(-(din[0] * Pb[(size_t)(3 * a) * L + ell] + din[1] * Pb[(size_t)(3 * a + 1) * L + ell] +
                 din[2] * Pb[(size_t)(3 * a + 2) * L + ell]),
               c.dc);
    } else {
      D = -1.0;
      S = divc(fl.link_Fb[(size_t)(a - 3) * L + ell], c.d3);
    }
  }
  const double fo = fz.scratch[(size_t)ell * kC3 + a];
  double val;
  if (eta >= 0.5) {
    const double fi = upid >= 0 ? f1[(size_t)(qi * kC3 + a) * N + upid]
                                : fz.scratch[(size_t)fz.partner[ell] * kC3 + a];
    const double al = 1.0 / (2.0 * eta);
    val = al * (D * fo + S) + (1.0 - al) * fi;
  } else {
    const double up = upid >= 0 ? f1[(size_t)(qo * kC3 + a) * N + n] : fo;
    val = D * (2.0 * eta * fo + (1.0 - 2.0 * eta) * up) + S;
  }
  f1[(size_t)(qi * kC3 + a) * N + n] = val;
}

// Characteristic rows (:2812-2884) of links with a Neumann row.
__global__ void __launch_bounds__(64)
    k3_link_char(Ctx3 c, Fused3 fz, double* __restrict__ f1, cvlbm3d_fields fl) {
  const cvlbm3d_problem& p = c.p;
  const Mat& m = c.m;
  const int L = p.n_links, N = c.N;
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= L) return;
  const int ell = fz.order ? fz.order[slot] : slot;
  if (!char_rows3(p, ell)) return;
  int ck[3];
  for (int r = 0; r < 3; ++r) ck[r] = fl.link_comp_kind[(size_t)r * L + ell];
  if (!(ck[0] == kNeumann || ck[1] == kNeumann || ck[2] == kNeumann)) return;
  const int n = p.link_p[ell], qi = opp3(p.link_q[ell]);
  const double din[3] = {(double)dx3(qi), (double)dy3(qi), (double)dz3(qi)};
  double Ub[12], G[3][12];
  const double* Un = fz.Uneed + (size_t)fz.need_slot[n] * kC3;
  for (int a = 0; a < 3; ++a)
    Ub[a] = ck[a] == kDirichlet ? fl.link_bv[(size_t)a * L + ell] : Un[a];
  for (int k = 0; k < 9; ++k) Ub[3 + k] = fl.link_Fb[(size_t)k * L + ell];
  if (state_det3(Ub) <= m.jf) *fl.invalid = 1;
  for (int d = 0; d < 3; ++d)
    for (int a = 0; a < 12; ++a) G[d][a] = fl.char_state[((size_t)(1 + d) * 12 + a) * L + ell];
  double out[12];
  char_population3(Ub, G[0], G[1], G[2], din, p.link_eta[ell], c, out);
  for (int a = 0; a < 12; ++a) {
    const int row = a < 3 ? a : (a - 3) / 3;
    if (ck[row] == kNeumann) f1[(size_t)(qi * kC3 + a) * N + n] = out[a];
  }
}

}  // namespace
