// D3Q6x12 cut links with packed characteristic tables (char_packed): the four phases
// of apply_boundary_reconstruction (three_d/curved_boundary_warp3d.py:4339-4399) in
// two kernels.  Included by cvlbm3d.cu after cvlbm3d_fused.cuh.
//
//   k3_link_gather_packed  four lanes per link: value and gradients of the
//                          characteristic stencil
//   k3_link_finish         one thread per link: boundary value, normal solve, P(F_b),
//                          characteristic rows, BFL rows
//
// The link work is a long dependent chain per link (about 3,400 FP64 steps) at few
// warps per SM.  The four separate kernels took 22 + 19 + 8 + 31 us at 11,256 links
// and 176 + 57 + 23 + 97 us at 150,800: each loaded the link again, the results went
// through memory between them, and code for every material law, value mode and
// solver sat in one kernel.  One kernel with four lanes per link for everything
// (tangents and evaluations of P spread over the lanes) was 50 us and 498 us: it
// repeats the normal solve on every lane.
// Four lanes per link in k3_link_finish alone (three tangents and P at the state side
// by side) cost 1 us per step more at 3,920 to 11,256 links, 8 at 15,448 and 20 at
// 25,320: the chain's length there is the unique code a warp runs through, not the
// number of tangents.
#pragma once

namespace {

constexpr int kLL3 = 4;                 // gather lanes per link
constexpr int kLinks3 = 32;             // links per gather block
constexpr int kLT3 = kLL3 * kLinks3;
constexpr int kFinish3 = 64;            // threads per block of k3_link_finish
constexpr int kGradSamples = 48, kProbeSamples = kChar - kGradSamples;

// Boundary values of the three components, out of line but for the common modes.
static __device__ __noinline__ void value3_all(int mode, const double* pp, double x, double y,
                                               double z, double nx, double ny, double nz, double t,
                                               double jf, double* T) {
  for (int r = 0; r < 3; ++r) T[r] = value3(r, mode, pp, x, y, z, nx, ny, nz, t, jf);
}

static __device__ __noinline__ void solve_mixed3(const double* F, double nx, double ny, double nz,
                                                 const double* T, const int* ck, const Mat* m,
                                                 int solver, double* Fb) {
  solve_Fb3_mixed(F, nx, ny, nz, T, ck, *m, solver, Fb);
}

// BFL rows of one link (:3154-3241) that the characteristic closure does not
// overwrite, from the link's buffers, link_scratch and the post-stream f1.
static __device__ __noinline__ void bfl_rows3(const Ctx3& c, const Fused3& fz, const cvlbm3d_fields& fl,
                                              double* f1, int ell, bool use_char) {
  const cvlbm3d_problem& p = c.p;
  const int L = p.n_links, N = c.N;
  const int n = p.link_p[ell], upid = p.link_up[ell], qo = p.link_q[ell], qi = opp3(qo);
  double eta = p.link_eta[ell];
  if (p.recon == 1) eta = 0.5;
  const double din[3] = {(double)dx3(qi), (double)dy3(qi), (double)dz3(qi)};
  const double al = 1.0 / (2.0 * eta);
#pragma unroll 1
  for (int row = 0; row < 3; ++row) {
    const int ckr = fl.link_comp_kind[(size_t)row * L + ell];
    if (use_char && ckr == kNeumann) continue;
    const double Tr = fl.link_bv[(size_t)row * L + ell];
    // population `row` (velocity) and the three of F row `row`
    double fo[4], fx[4], S[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int a = j == 0 ? row : 3 * row + 2 + j;
      fo[j] = fz.scratch[(size_t)ell * kC3 + a];
      if (eta >= 0.5)
        fx[j] = upid >= 0 ? f1[(size_t)(qi * kC3 + a) * N + upid]
                          : fz.scratch[(size_t)fz.partner[ell] * kC3 + a];
      else
        fx[j] = upid >= 0 ? f1[(size_t)(qo * kC3 + a) * N + n] : fo[j];
    }
    double D0, D1;
    if (ckr == kDirichlet) {
      D0 = -1.0;
      D1 = 1.0;
      S[0] = divc(Tr, c.d3);
#pragma unroll
      for (int j = 0; j < 3; ++j) S[1 + j] = divc(-din[j] * Tr, c.dc);
    } else {
      D0 = 1.0;
      D1 = -1.0;
      const double* Pb = fl.link_Pb + (size_t)(3 * row) * L + ell;
      S[0] = divc(-(din[0] * Pb[0] + din[1] * Pb[L] + din[2] * Pb[2 * (size_t)L]), c.dc);
#pragma unroll
      for (int j = 0; j < 3; ++j) S[1 + j] = divc(fl.link_Fb[(size_t)(3 * row + j) * L + ell], c.d3);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int a = j == 0 ? row : 3 * row + 2 + j;
      const double D = j == 0 ? D0 : D1;
      double val;
      if (eta >= 0.5)
        val = al * (D * fo[j] + S[j]) + (1.0 - al) * fx[j];
      else
        val = D * (2.0 * eta * fo[j] + (1.0 - 2.0 * eta) * fx[j]) + S[j];
      f1[(size_t)(qi * kC3 + a) * N + n] = val;
    }
  }
}

// One thread per link after the gather: boundary value, normal solve, P(F_b),
// characteristic rows, BFL rows.  One code copy serves the four flux tangents, each
// with its two evaluations of P side by side; what is rare (other value modes, mixed
// rows, BFL rows) is called out of line with its arguments copied, and the kernel's
// structures stay in the parameter bank (__grid_constant__), so that nothing on the
// common path lives in local memory (shell48 914 to 866 us per ten steps).
template <int MAT>
__global__ void __launch_bounds__(kFinish3, 6)
    k3_link_finish(const __grid_constant__ Ctx3 c, const __grid_constant__ Fused3 fz,
                   double* __restrict__ f1, const double* __restrict__ u,
                   const __grid_constant__ cvlbm3d_fields fl, const double* clock, double t_host,
                   double offset) {
  const cvlbm3d_problem& p = c.p;
  const Mat m = mat3<MAT>(c);
  const int L = p.n_links, N = c.N;
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= L) return;
  const int ell = fz.order ? fz.order[slot] : slot;
  const bool gathered = p.char_idx[ell] >= 0;
  const int bid = p.link_bid[ell];
  const int kind = p.bc_kind[bid], mode = p.bc_mode[bid];
  int ck[3];
#pragma unroll
  for (int r = 0; r < 3; ++r) ck[r] = p.bc_comp_kind[r * kMaxIds3 + bid];
  const bool anyN = ck[0] == kNeumann || ck[1] == kNeumann || ck[2] == kNeumann;
  const double nx = p.link_nx[ell], ny = p.link_ny[ell], nz = p.link_nz[ell];
  const double t = time_of(clock, t_host, offset);
  double T[3] = {0.0, 0.0, 0.0};
  if (mode == 208) {
    const double* pp = p.bc_params + bid * 16;
    const double rt = pp[1], amp = pp[0];
    double s = 1.0;
    if (rt > 0.0 && t < rt) s = t / rt;
    T[0] = amp * s * nx;
    T[1] = amp * s * ny;
    T[2] = amp * s * nz;
  } else if (mode != 0) {
    double v[3];
    value3_all(mode, p.bc_params + bid * 16, p.link_xb[ell], p.link_yb[ell], p.link_zb[ell], nx, ny,
               nz, t, m.jf, v);
    T[0] = v[0];
    T[1] = v[1];
    T[2] = v[2];
  }
  if (p.dyn_enabled && p.dyn_enabled[ell] != 0) {
#pragma unroll
    for (int r = 0; r < 3; ++r) T[r] = p.dyn_traction[(size_t)r * L + ell];
  }
  double Fb[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  const double* cs = fl.char_state + ell;  // [48] rows of stride L
  fl.link_kind[ell] = kind;
#pragma unroll
  for (int r = 0; r < 3; ++r) {
    fl.link_comp_kind[(size_t)r * L + ell] = ck[r];
    fl.link_bv[(size_t)r * L + ell] = T[r];
  }
  if (anyN) {
    double F[9];
    if (p.recon == 3) {
#pragma unroll
      for (int k = 0; k < 9; ++k) F[k] = gathered ? cs[(size_t)(3 + k) * L] : 0.0;
    } else {
      double F2[9];
      predictor3(c, fz, ell, u, F2);
#pragma unroll
      for (int k = 0; k < 9; ++k) F[k] = F2[k];
    }
#pragma unroll
    for (int k = 0; k < 9; ++k) Fb[k] = F[k];
    if (ck[0] == kNeumann && ck[1] == kNeumann && ck[2] == kNeumann)
      solve_Fb3(F, nx, ny, nz, T, m, p.normal_solver, Fb);
    else {
      // copies: what a call takes by address lives in local memory
      double F2[9], T2[3], B2[9];
      int c2[3];
      const Mat m2 = m;
#pragma unroll
      for (int k = 0; k < 9; ++k) F2[k] = B2[k] = F[k];
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        T2[r] = T[r];
        c2[r] = ck[r];
      }
      solve_mixed3(F2, nx, ny, nz, T2, c2, &m2, p.normal_solver, B2);
#pragma unroll
      for (int k = 0; k < 9; ++k) Fb[k] = B2[k];
    }
    const M3 P = piola3(Fb, m);
#pragma unroll
    for (int k = 0; k < 9; ++k) fl.link_Pb[(size_t)k * L + ell] = P.v[k];
  } else {
#pragma unroll
    for (int k = 0; k < 9; ++k) fl.link_Pb[(size_t)k * L + ell] = 0.0;
  }
#pragma unroll
  for (int k = 0; k < 9; ++k) fl.link_Fb[(size_t)k * L + ell] = Fb[k];
  const bool use_char = gathered && anyN;
  if (use_char) {
    const int n = p.link_p[ell], qi = opp3(p.link_q[ell]);
    const int ax = qi < 3 ? qi : qi - 3;
    const double sg = qi < 3 ? 1.0 : -1.0;  // incoming direction along axis ax
    const double eta = p.link_eta[ell];
    const double* Un = fz.Uneed + (size_t)fz.need_slot[n] * kC3;
    const double* Gx = cs + (size_t)(12 * (1 + ax)) * L;  // gradient along the incoming axis
    double Uc[12], w[12];
    {
      double Ub[12], shift[12];
#pragma unroll
      for (int a = 0; a < 3; ++a) Ub[a] = ck[a] == kDirichlet ? T[a] : Un[a];
#pragma unroll
      for (int k = 0; k < 9; ++k) Ub[3 + k] = Fb[k];
      if (state_det3(Ub) <= m.jf) *fl.invalid = 1;
      const double kk = eta * p.dt * p.c;
#pragma unroll
      for (int a = 0; a < 12; ++a) shift[a] = kk * (sg * Gx[(size_t)a * L]);
      double chi = 1.0;
#pragma unroll 1
      for (int it = 0; it < 10; ++it) {
#pragma unroll
        for (int a = 0; a < 12; ++a) Uc[a] = Ub[a] + chi * shift[a];
        if (state_det3(Uc) > 10.0 * m.jf) break;
        chi = 0.5 * chi;
      }
#pragma unroll
      for (int a = 0; a < 12; ++a) Uc[a] = Ub[a] + chi * shift[a];
    }
    // w = B - j0 - j1 - j2 + c dG, then the tangent along the incoming axis on w
#pragma unroll
    for (int a = 0; a < 3; ++a) w[a] = source_comp3(a, p.source_mode, p.source, Uc);
    double Aw[3];
#pragma unroll 1
    for (int d = 0; d < 4; ++d) {
      double W[12];
      if (d < 3) {
#pragma unroll
        for (int a = 0; a < 12; ++a) W[a] = cs[(size_t)(12 * (1 + d) + a) * L];
      } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) w[a] = w[a] + p.c * (sg * Gx[(size_t)a * L]);
#pragma unroll
        for (int a = 3; a < 12; ++a)
          w[a] = source_comp3(a, p.source_mode, p.source, Uc) +
                 cs[(size_t)(12 * (1 + (a - 3) % 3) + (a - 3) / 3) * L] +
                 p.c * (sg * Gx[(size_t)a * L]);
#pragma unroll
        for (int a = 0; a < 12; ++a) W[a] = w[a];
      }
      double s = 1.0;
#pragma unroll
      for (int a = 0; a < 12; ++a) s = fmax(s, fabs(W[a]));
      const double eps = 1.0e-6 / s;
      double Fp[9], Fm[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        Fp[k] = Uc[3 + k] + eps * W[3 + k];
        Fm[k] = Uc[3 + k] - eps * W[3 + k];
      }
      const M3 Pp = piola3(Fp, m), Pm = piola3(Fm, m);
      const int col = d < 3 ? d : ax;
      double num[3], jv[3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
        num[i] = col == 0   ? -(Pp.v[3 * i] - Pm.v[3 * i])
                 : col == 1 ? -(Pp.v[3 * i + 1] - Pm.v[3 * i + 1])
                            : -(Pp.v[3 * i + 2] - Pm.v[3 * i + 2]);
      div_n(rcp_of(2.0 * eps), num, jv, 3);
      if (d < 3) {
#pragma unroll
        for (int i = 0; i < 3; ++i) w[i] = w[i] - jv[i];
      } else {
#pragma unroll
        for (int i = 0; i < 3; ++i) Aw[i] = jv[i];
      }
    }
    const M3 P = piola3(Uc + 3, m);
    const double s3 = 3.0 * sg;
    const double kk = p.dt / p.omega, kb = p.dt * (1.0 / p.omega - 0.5);
    double* dst = f1 + (size_t)(qi * kC3) * N + n;
#pragma unroll
    for (int a = 0; a < 12; ++a) {
      const int row = a < 3 ? a : (a - 3) / 3, j = (a - 3) % 3;
      double fla, Awa;
      if (a < 3) {
        fla = -(ax == 0 ? P.v[3 * a] : ax == 1 ? P.v[3 * a + 1] : P.v[3 * a + 2]);
        Awa = Aw[a];
      } else {
        fla = j == ax ? -Uc[row] : 0.0;
        Awa = j == ax ? -w[row] : 0.0;
      }
      const double Ba = source_comp3(a, p.source_mode, p.source, Uc);
      if (ck[row] == kNeumann)
        dst[(size_t)a * N] =
            divc(Uc[a] + divc(s3 * fla, c.dc) - kk * (w[a] + divc(s3 * Awa, c.dc)) + kb * Ba, c.d6);
    }
    if (ck[0] == kNeumann && ck[1] == kNeumann && ck[2] == kNeumann) return;
  }
  bfl_rows3(c, fz, fl, f1, ell, use_char);
}

// Value and gradients of the 12 components at every link (_sparse_characteristic_gather,
// :2675-2700) from the packed tables: lane l of a link's four sums components 3l ..
// 3l + 2, the gradients over slots 0..47 and the value over slots 48..63, in slot
// order (the other weights are zero: their products change no finite sum).  Four
// samples at a time; staging the slots in shared memory or eight samples at a time
// measured the same.
constexpr int kChunk3 = 4;

template <bool PROBE>
__device__ __forceinline__ void gather_chunk3(const int4* __restrict__ slot, const double2* __restrict__ w2,
                                              const double* __restrict__ Ub, int m0, double* av,
                                              double (*ag)[3]) {
  const int4 q4 = slot[m0 / 4], r4 = PROBE ? slot[(kGradSamples + m0) / 4] : make_int4(-1, -1, -1, -1);
  const int q[kChunk3] = {q4.x, q4.y, q4.z, q4.w}, qp[kChunk3] = {r4.x, r4.y, r4.z, r4.w};
  double2 wa[kChunk3], wb[kChunk3];
  double uv[kChunk3][3], up[kChunk3][3];
#pragma unroll
  for (int k = 0; k < kChunk3; ++k) {
    wa[k] = w2[2 * (m0 + k)];
    wb[k] = w2[2 * (m0 + k) + 1];
  }
#pragma unroll
  for (int k = 0; k < kChunk3; ++k) {
    const double* row = Ub + (size_t)(q[k] >= 0 ? q[k] : 0) * kC3;
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) uv[k][cc] = row[cc];
    if (PROBE) {
      const double* rowp = Ub + (size_t)(qp[k] >= 0 ? qp[k] : 0) * kC3;
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) up[k][cc] = rowp[cc];
    }
  }
#pragma unroll
  for (int k = 0; k < kChunk3; ++k) {
    if (q[k] >= 0) {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) {
        ag[0][cc] += wa[k].x * uv[k][cc];
        ag[1][cc] += wa[k].y * uv[k][cc];
        ag[2][cc] += wb[k].x * uv[k][cc];
      }
    }
    if (PROBE && qp[k] >= 0) {
#pragma unroll
      for (int cc = 0; cc < 3; ++cc) av[cc] += wb[k].y * up[k][cc];
    }
  }
}

__global__ void __launch_bounds__(kLT3, 4)
    k3_link_gather_packed(Ctx3 c, Fused3 fz, double* __restrict__ char_state) {
  const cvlbm3d_problem& p = c.p;
  const int L = p.n_links;
  const int lane = threadIdx.x & (kLL3 - 1);
  const int ell = blockIdx.x * kLinks3 + threadIdx.x / kLL3;
  if (ell >= L || p.char_idx[ell] < 0) return;
  const int4* slot = reinterpret_cast<const int4*>(p.char_slot_lm + (size_t)ell * kChar);
  const double2* w2 = reinterpret_cast<const double2*>(p.char_w_lm) + (size_t)ell * kGradSamples * 2;
  const double* Ub = fz.Uneed + 3 * lane;
  double av[3] = {0.0, 0.0, 0.0}, ag[3][3];
#pragma unroll
  for (int k = 0; k < 3; ++k) ag[k][0] = ag[k][1] = ag[k][2] = 0.0;
#pragma unroll 1
  for (int m0 = 0; m0 < kProbeSamples; m0 += kChunk3) gather_chunk3<true>(slot, w2, Ub, m0, av, ag);
#pragma unroll 1
  for (int m0 = kProbeSamples; m0 < kGradSamples; m0 += kChunk3)
    gather_chunk3<false>(slot, w2, Ub, m0, av, ag);
#pragma unroll
  for (int cc = 0; cc < 3; ++cc) {
    const int a = 3 * lane + cc;
    char_state[(size_t)a * L + ell] = av[cc];
#pragma unroll
    for (int d = 0; d < 3; ++d) char_state[((size_t)(1 + d) * 12 + a) * L + ell] = ag[d][cc];
  }
}

using LinkFn3 = void (*)(Ctx3, Fused3, double*, const double*, cvlbm3d_fields, const double*, double,
                         double);

inline LinkFn3 link_finish3(int model) {
  switch (model) {
    case kMatSVK: return k3_link_finish<kMatSVK>;
    case kMatNeoHooke: return k3_link_finish<kMatNeoHooke>;
    case kMatLogNeoHooke: return k3_link_finish<kMatLogNeoHooke>;
    case kMatMooneyRivlin: return k3_link_finish<kMatMooneyRivlin>;
    case kMatYeoh: return k3_link_finish<kMatYeoh>;
    case kMatGent: return k3_link_finish<kMatGent>;
    case kMatSix: return k3_link_finish<kMatSix>;
    default: return k3_link_finish<-1>;
  }
}

}  // namespace
