// The Krylov operator J v at a held linearisation (first-order upwind), tangents only.  Included by
// residual.cu (shares its device helpers).
//
// fv_case_linearise keeps the double pass's gradients, closure fields, d, mass-flux estimate and
// face intermediates, and the off-wall cells' closure and source forms; a product then carries one
// double per quantity, its tangent: half the bytes of dual numbers between the stages, and none of
// the primal arithmetic.  The few places where the tangent is not a short form -- boundary faces,
// the wall functions of wall cells -- evaluate the residual's own formulas in dual numbers, paired
// from the held value and the tangent (TangentOf), in kernels of their own: inside the off-wall
// stages their registers and their divergence cost more than their work (k_closure_lin 141 us,
// k_sum_lin 132 us a product on the 96 x 64 x 64 channel with them inside and dual arrays).
//   k_grad_tangent    cell  compact Green-Gauss (the scheme is linear)
//   k_closure_lin     cell  off the wall: the tabulated forms
//   k_wall_closure    wall cell
//   k_apcoef_tangent  face  interior;  k_apcoef_boundary
//   k_dcoeff_tangent  cell  d = V / a_P
//   k_flux_tangent    face  interior, from the kept intermediates;  k_flux_boundary
//   k_sum_lin         cell  face sums, pin row, off-wall sources
//   k_wall_rows       wall cell  source rows and the omega fixation
// Measured there, linearisation and four products: 4.89 -> 3.97 ms.

// Held values with a product's tangents as dual numbers.
struct TangentOf {
  const double *v, *d;
  __device__ __forceinline__ Dual operator[](long i) const { return {v[i], d[i]}; }
};


// Wall cells: closure tangents.  `cells` lists them.
template <int DIM>
__global__ void __launch_bounds__(128) k_wall_closure(MeshView m, CaseView cv, Src<Dual> st,
                                                      Par<Dual> par, TangentOf G, int n,
                                                      const int* cells, double* cl) {
  stage_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cells[i];
  const long nc = m.nc;
  Dual out[7], gw[DIM];
  closure_cell<Dual, DIM>(m, cv, st, par, G, c, GeoPlain{}, out, gw);
#pragma unroll
  for (int q = 0; q < 7; ++q) cl[q * nc + c] = out[q].d;
}

// Wall cells: the k and omega rows from their face sums in JV.
template <int DIM>
__global__ void __launch_bounds__(128) k_wall_rows(MeshView m, CaseView cv, Src<Dual> st,
                                                   Par<Dual> par, TangentOf cl, TangentOf G, int n,
                                                   const int* cells, double* JV) {
  using L = Layout<DIM, true>;
  stage_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cells[i];
  const long nc = m.nc;
  Dual rk{0.0, JV[L::K * nc + c]}, rw{0.0, JV[L::W * nc + c]};
  // (a wall cell's rows do not read the omega gradient)
  sst_rows<Dual, DIM>(m, cv, st, par, cl, G, G, c, rk, rw);
  JV[L::K * nc + c] = rk.d;
  JV[L::W * nc + c] = rw.d;
}

template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_grad_tangent(MeshView m, CaseView cv, Src<Dual> st,
                                                      Par<Dual> par, double* G, double* Bg,
                                                      double rel) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  stage_begin();
  const int c = stage_cell<double>(m, cv);
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  const double* t = st.t;
  double phic[NF], acc[NF][DIM], own[DIM];  // own (SST): as in k_grad
#pragma unroll
  for (int j = 0; j < DIM; ++j) own[j] = 0.0;
#pragma unroll
  for (int q = 0; q < NF; ++q) {
    phic[q] = t[(long)q * nc + c];
#pragma unroll
    for (int j = 0; j < DIM; ++j) acc[q][j] = 0.0;
  }
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    const bool isnb = (ent & FV_NB_BIT) != 0;
    const double af = m.area[f];
    const double A = isnb ? -af : af;
    double S[DIM], phif[NF];
#pragma unroll
    for (int j = 0; j < DIM; ++j) S[j] = m.normal[(long)j * nf + f] * A;
    if (f < m.nfi) {
      const double g = m.g[f];
      const int other = isnb ? m.owner[f] : m.nb[f];
#pragma unroll
      for (int q = 0; q < NF; ++q) {
        const double po = t[(long)q * nc + other];
        if constexpr (TURB) phif[q] = po;
        else phif[q] = lerp(isnb ? po : phic[q], isnb ? phic[q] : po, g);
      }
      if constexpr (TURB) {
        const double h = 1.0 - g, wo = isnb ? h : g, wc = isnb ? g : h;
#pragma unroll
        for (int j = 0; j < DIM; ++j) {
          own[j] += S[j] * wc;
          S[j] *= wo;
        }
      }
    } else {
      const signed char kind = cv.fkind[f];
#pragma unroll
      for (int j = 0; j < DIM; ++j)
        phif[j] = bvel(cv, nf, f, j, kind, Dual{0.0, phic[j]}, par).d;
      phif[L::P] = bpress(cv, f, kind, Dual{0.0, phic[L::P]}).d;
      if (TURB) {
        const Dual z{0.0, 0.0};
        phif[L::K] = bscalar(cv.kkind[f], cv.kval[f], Dual{0.0, phic[L::K]}, z).d;
        phif[L::W] = bscalar(cv.wkind[f], cv.wval[f], Dual{0.0, phic[L::W]}, z).d;
      }
    }
#pragma unroll
    for (int q = 0; q < NF; ++q)
#pragma unroll
      for (int j = 0; j < DIM; ++j) acc[q][j] += S[j] * phif[q];
  }
  const double inv = rel * m.inv_vol[c];
#pragma unroll
  for (int q = 0; q < NF; ++q)
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const long k = ((long)q * DIM + j) * nc + c;
      const double x = TURB ? acc[q][j] + own[j] * phic[q] : acc[q][j];
      G[k] = x * inv;
      if (Bg) Bg[k] = x;
    }
}

// ---------------------------------------------------------------- linearised SST closure
// Off the wall, the closure fields and the k / omega source terms of a cell depend on the state
// through four scalars only: k, omega, the strain rate S and grad k . grad omega.  At a held
// linearisation their tangents are therefore linear forms in those four tangents, tabulated once
// per linearisation (k_lin_closure_coef) and applied by every Krylov product (k_closure_lin,
// k_sum_lin).
//
// Coefficients per cell (LIN_NCOEF rows of nc): 2 / S (the strain rate's tangent is
// 2 / S sum_ij s_ij (grad u)'_ij, 0 where S = 0), then the linear forms in (k', omega', S',
// (grad k . grad omega)') of nu_t, the k and omega diffusivities and the k and omega sources as
// they enter the face sums.  (The forms of F1 and F2 enter these and nothing else.)
constexpr int LIN_NCOEF = 21;

// weight of a in max(a, b) (min: of a in min(a, b)); a tie takes half of each
__device__ __forceinline__ double max_weight(double a, double b) {
  return a > b ? 1.0 : (a < b ? 0.0 : 0.5);
}

// The forms, by the closure's partial derivatives written out (closure_cell and sst_rows off the
// wall; F1, nu_t and F2 are the pass's own): about 150 fp64 instructions a cell, where a
// four-direction dual number evaluation took 296 us for 393,000 cells.
template <int DIM>
__global__ void __launch_bounds__(128) k_lin_closure_coef(MeshView m, CaseView cv,
                                                          const double* state, const double* G,
                                                          const double* cl, double nu,
                                                          double* cc) {
  using L = Layout<DIM, true>;
  const int c = stage_cell<double>(m, cv);
  if (c >= m.nc || cv.wcell[c]) return;
  const long nc = m.nc;
  const double S = cl[c], F1 = cl[nc + c], nut = cl[2 * nc + c], F2 = cl[6 * nc + c];
  const double k = state[(long)L::K * nc + c], w = state[(long)L::W * nc + c];
  const double id = cv.inv_wd[c], id2 = cv.inv_wd2[c], V = m.vol[c];
  double dot = 0.0;
#pragma unroll
  for (int j = 0; j < DIM; ++j)
    dot += G[((long)L::K * DIM + j) * nc + c] * G[((long)L::W * DIM + j) * nc + c];
  const double kp = pos(k), dk = dpos(k), iw = 1.0 / w;
  constexpr double X = 2.0 * SIGMA_W2;
  const double cd0 = X * dot * iw;
  const double wc = max_weight(cd0, CROSS_FLOOR), cd = cd0 > CROSS_FLOOR ? cd0 : CROSS_FLOOR;
  const double icd = 1.0 / cd;
  const double cd_w = -wc * cd0 * iw, cd_d = wc * X * iw;
  const double sk = kp > 0.0 ? sqrt(kp) : 0.0;
  const double bw = iw * (id / BETA_STAR);
  const double c1 = sk * bw, c1_k = kp > 0.0 ? 0.5 * bw / sk : 0.0, c1_w = -c1 * iw;
  const double vt = (500.0 * id2) * nu * iw, vt_w = -vt * iw;
  const double a = max_weight(c1, vt), inner = c1 > vt ? c1 : vt;
  const double cf = (4.0 * SIGMA_W2 * id2) * icd;
  const double c2 = cf * kp, c2_cd = -c2 * icd;
  const double b = 1.0 - max_weight(inner, c2), arg1 = inner < c2 ? inner : c2;
  const double a2 = arg1 * arg1, f1 = (1.0 - F1 * F1) * 4.0 * (a2 * arg1);
  // d F1 / d (k, omega, dot); F1 does not see S
  const double F1k = f1 * (b * (a * c1_k) + (1.0 - b) * cf * dk);
  const double F1w = f1 * (b * (a * c1_w + (1.0 - a) * vt_w) + (1.0 - b) * (c2_cd * cd_w));
  const double F1d = f1 * ((1.0 - b) * (c2_cd * cd_d));
  const double tc1 = 2.0 * c1, e = max_weight(tc1, vt), arg2 = tc1 > vt ? tc1 : vt;
  const double f2 = (1.0 - F2 * F2) * 2.0 * arg2;
  const double F2k = f2 * (e * 2.0 * c1_k), F2w = f2 * (e * 2.0 * c1_w + (1.0 - e) * vt_w);
  const double ma = A1 * w, mb = S * F2, h = max_weight(ma, mb), iM = 1.0 / (ma > mb ? ma : mb);
  const double hs = (1.0 - h) * S;
  const double nk = (A1 * dk - nut * (hs * F2k)) * iM;
  const double nw = -nut * (h * A1 + hs * F2w) * iM;
  const double ns = -nut * ((1.0 - h) * F2) * iM;
  auto put = [&](int q, double pk, double pw, double ps, double pd) {
    double* o = cc + (1L + 4 * q) * nc + c;
    o[0] = pk;
    o[nc] = pw;
    o[2 * nc] = ps;
    o[3 * nc] = pd;
  };
  cc[c] = S > 0.0 ? 2.0 / S : 0.0;
  put(0, nk, nw, ns, 0.0);
  auto diffusivity = [&](int q, double in, double out) {
    const double x = out + F1 * (in - out), y = (in - out) * nut;
    put(q, x * nk + y * F1k, x * nw + y * F1w, x * ns, y * F1d);
  };
  diffusivity(1, SIGMA_K1, SIGMA_K2);
  diffusivity(2, SIGMA_W1, SIGMA_W2);
  // k source: beta* V k omega - V min(nu_t S^2, limit)
  constexpr double PB = PROD_RATIO * BETA_STAR;
  const double S2 = S * S, prod = nut * S2, limit = PB * kp * w;
  const double lk = PB * dk * w, lw = PB * kp;
  const double p = 1.0 - max_weight(prod, limit);
  put(3, V * (BETA_STAR * w - (p * nk * S2 + (1.0 - p) * lk)),
      V * (BETA_STAR * k - (p * nw * S2 + (1.0 - p) * lw)), -V * p * (ns * S2 + 2.0 * nut * S),
      0.0);
  // omega source: V (beta omega^2 - alpha min(S^2, limit / max(nu_t, floor)) - cross)
  const double nm = max_weight(nut, NUT_FLOOR), inf = 1.0 / (nut > NUT_FLOOR ? nut : NUT_FLOOR);
  const double cap = limit * inf, r = 1.0 - max_weight(S2, cap);
  const double cn = -cap * nm * inf;  // d cap / d nu_t
  const double mn = S2 < cap ? S2 : cap;
  const double alpha = ALPHA_2 + F1 * (ALPHA_1 - ALPHA_2), beta = BETA_2 + F1 * (BETA_1 - BETA_2);
  const double xd = X * iw, cross = xd * (1.0 - F1) * dot;
  // what multiplies d F1
  const double y = (BETA_1 - BETA_2) * (w * w) - (ALPHA_1 - ALPHA_2) * mn + xd * dot;
  put(4, V * (y * F1k - alpha * ((1.0 - r) * (lk * inf + cn * nk))),
      V * (y * F1w + 2.0 * beta * w - alpha * ((1.0 - r) * (lw * inf + cn * nw)) + cross * iw),
      -V * alpha * (r * 2.0 * S + (1.0 - r) * (cn * ns)), V * (y * F1d - xd * (1.0 - F1)));
}

// Off the wall: closure tangents by the tabulated forms, and the k / omega source tangents (src, 2
// rows of nc) for k_sum_lin.  Gp: the held gradients.
template <int DIM>
__global__ void __launch_bounds__(128) k_closure_lin(MeshView m, CaseView cv, Src<Dual> st,
                                                     const double* Gp, const double* Gt,
                                                     const double* cc, double* cl, double* src) {
  using L = Layout<DIM, true>;
  stage_begin();
  const int c = stage_cell<double>(m, cv);
  if (c >= m.nc || cv.wcell[c]) return;
  const long nc = m.nc;
  auto gv = [&](int i, int j) { return Gp[((long)i * DIM + j) * nc + c]; };
  auto gd = [&](int i, int j) { return Gt[((long)i * DIM + j) * nc + c]; };
  double ss = 0.0, off = 0.0, dd = 0.0;  // s_ij (grad u)'_ij, each off-diagonal pair once
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    ss += gv(i, i) * gd(i, i);
#pragma unroll
    for (int j = i + 1; j < DIM; ++j) off += (gv(i, j) + gv(j, i)) * (gd(i, j) + gd(j, i));
  }
  ss += 0.5 * off;
#pragma unroll
  for (int j = 0; j < DIM; ++j) dd += gd(L::K, j) * gv(L::W, j) + gv(L::K, j) * gd(L::W, j);
  const double tk = st.t[(long)L::K * nc + c], tw = st.t[(long)L::W * nc + c], ts = cc[c] * ss;
  auto form = [&](int q) {
    const double* a = cc + (1L + 4 * q) * nc + c;
    double x = a[0] * tk + a[nc] * tw + a[2 * nc] * ts;
    if (q != 0 && q != 3) x += a[3 * nc] * dd;  // nu_t and the k source do not see it
    return x;
  };
  cl[2 * nc + c] = form(0);
  cl[4 * nc + c] = form(1);
  cl[5 * nc + c] = form(2);
  src[c] = form(3);
  src[nc + c] = form(4);
}

// ---------------------------------------------------------------- momentum diagonal and d
// The interior faces' momentum-diagonal coefficients and mass-flux estimate: the momentum-normal
// flux is linear in the velocities and their gradients, the conductance's tangent comes from its
// kept partial derivatives in the cell viscosities, max(., 0) follows the kept sign of the estimate
// (JAX's tie rule).
template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_apcoef_tangent(MeshView m, CaseView cv, Src<Dual> st,
                                                        const double* G, const double* cl,
                                                        const double* aux, const double* mest,
                                                        double* ac_own, double* ac_nb,
                                                        double* me) {
  stage_begin();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nfi) return;
  const long nc = m.nc, nf = m.nf;
  const int o = m.owner[f], n = m.nb[f];
  const double g = m.g[f], A = m.area[f], rho = cv.rho;
  double so = 0.0, sn = 0.0;  // each side's sum (mom_normal)
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    const double nj = m.normal[(long)j * nf + f];
    so += nj * st.t[(long)j * nc + o];
    sn += nj * st.t[(long)j * nc + n];
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
      const double x = m.ns[(long)(j * DIM + q) * nf + f];
      so += x * G[((long)j * DIM + q) * nc + o];
      sn += x * G[((long)j * DIM + q) * nc + n];
    }
  }
  const double met = (rho * lerp(so, sn, g)) * A;
  const double visc = TURB ? rho * (aux[4L * nf + f] * cl[2L * nc + o] +
                                    aux[5L * nf + f] * cl[2L * nc + n])
                           : 0.0;
  const double e = mest[f];
  ac_own[f] = visc + (e > 0.0 ? met : (e < 0.0 ? 0.0 : 0.5 * met));
  ac_nb[f] = visc - (e < 0.0 ? met : (e > 0.0 ? 0.0 : 0.5 * met));
  me[f] = met;
}

template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_apcoef_boundary(MeshView m, CaseView cv, Src<Dual> st,
                                                         Par<Dual> par, TangentOf G, TangentOf cl,
                                                         double* ac_own) {
  stage_begin();
  const int f = m.nfi + blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  Dual ao, an, me;
  apcoef_face<Dual, DIM, TURB>(m, cv, st, par, G, cl, f, GeoPlain{}, ao, an, me);
  ac_own[f] = ao.d;
}

__global__ void k_dcoeff_tangent(MeshView m, const double* ac_own, const double* ac_nb,
                                 const double* dco, double* dt) {
  stage_begin();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  double a = 0.0;
  for (int i = m.cf_ptr[c]; i < m.cf_ptr[c + 1]; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    a += (ent & FV_NB_BIT) ? ac_nb[f] : ac_own[f];
  }
  const double d = dco[c];
  dt[c] = -(d * d) * m.inv_vol[c] * a;
}

// ---------------------------------------------------------------- face fluxes and sums
// The interior faces: the primal face intermediates the double pass kept (mass flux, pressure
// damping, interpolated d, conductances and their partial derivatives in the cell diffusivities,
// the cross-diffusion numerators) stand in for their recomputation, so only the tangent arithmetic
// of flux_face runs -- the forward-mode counterpart of the adjoint's use of the same intermediates.
template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_flux_tangent(MeshView m, CaseView cv, Src<Dual> st,
                                                      const double* G, const double* cl,
                                                      const double* dco, const double* me,
                                                      const double* aux, double* FL) {
  using L = Layout<DIM, TURB>;
  using AX = Aux<DIM, TURB>;
  stage_begin();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nfi) return;
  const long nc = m.nc, nf = m.nf;
  const int o = m.owner[f], n = m.nb[f];
  const double A = m.area[f], g = m.g[f];
  const double rho = cv.rho, irho = cv.irho;
  const double mdot = aux[0L * nf + f], damping = aux[1L * nf + f], dhat = aux[2L * nf + f];
  const double cmo = aux[3L * nf + f];
  double gd = 0.0, gs = 0.0;
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    const double gpf = lerp(G[((long)L::P * DIM + j) * nc + o], G[((long)L::P * DIM + j) * nc + n], g);
    gd += gpf * m.dvec[(long)j * nf + f];
    gs += gpf * m.skew[(long)j * nf + f];
  }
  const double dhat_t = m.nn2[f] * lerp(dco[o], dco[n], g);
  const double po = st.t[(long)L::P * nc + o], pn = st.t[(long)L::P * nc + n];
  const double damp_t = ((pn - po) - gd) * m.inv_nd[f];
  const double mdot_t = me[f] - (rho * A) * (dhat_t * damping + dhat * damp_t);
  const double pA_t = (lerp(po, pn, g) + gs) * A;
  // d(mu + rho nu_t) for a state tangent (the molecular viscosity is a parameter)
  const double cmo_t = TURB ? rho * (aux[4L * nf + f] * cl[2L * nc + o] +
                                     aux[5L * nf + f] * cl[2L * nc + n])
                            : 0.0;
  const bool out = mdot >= 0.0;
  double tP[DIM], tN[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    tP[j] = m.tP[(long)j * nf + f];
    tN[j] = m.tN[(long)j * nf + f];
  }
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    const double uo = st.t[(long)i * nc + o], un = st.t[(long)i * nc + n];
    double cpn_t = un - uo;
#pragma unroll
    for (int j = 0; j < DIM; ++j)
      cpn_t += G[((long)i * DIM + j) * nc + n] * tN[j] - G[((long)i * DIM + j) * nc + o] * tP[j];
    const double up = st.v[(long)i * nc + (out ? o : n)], up_t = out ? uo : un;
    double x = pA_t * m.normal[(long)i * nf + f] - cmo * cpn_t + mdot_t * up + mdot * up_t;
    if (TURB) x -= cmo_t * aux[(long)(AX::CPN + i) * nf + f];
    FL[(long)i * nf + f] = x;
  }
  FL[(long)L::P * nf + f] = mdot_t;
  if (TURB) {
    const double vflux = mdot * irho, vflux_t = mdot_t * irho;
    const bool vout = vflux >= 0.0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int q = s == 0 ? L::K : L::W;
      const long b0 = AX::S0 + 4 * s;
      const double phio = st.t[(long)q * nc + o], phin = st.t[(long)q * nc + n];
      double cpn_t = phin - phio;
#pragma unroll
      for (int j = 0; j < DIM; ++j)
        cpn_t += G[((long)q * DIM + j) * nc + n] * tN[j] - G[((long)q * DIM + j) * nc + o] * tP[j];
      const double cs_t = aux[(b0 + 1) * nf + f] * cl[(4L + s) * nc + o] +
                          aux[(b0 + 2) * nf + f] * cl[(4L + s) * nc + n];
      const double up = st.v[(long)q * nc + (vout ? o : n)], up_t = vout ? phio : phin;
      FL[(long)q * nf + f] = vflux_t * up + vflux * up_t -
                             (cs_t * aux[(b0 + 3) * nf + f] + aux[b0 * nf + f] * cpn_t);
    }
  }
}

// Keeps a flux's tangent.
struct TangentStore {
  double* FL;
  long nf, f;
  __device__ __forceinline__ void operator()(int q, const Dual& x) const { FL[q * nf + f] = x.d; }
};
template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_flux_boundary(MeshView m, CaseView cv, Src<Dual> st,
                                                       Par<Dual> par, TangentOf G, TangentOf cl,
                                                       TangentOf dco, double* FL) {
  stage_begin();
  const int f = m.nfi + blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  flux_face<Dual, DIM, TURB>(m, cv, st, par, G, cl, dco, (const Dual*)nullptr, (const Dual*)nullptr,
                             false, f, TangentStore{FL, m.nf, f}, nullptr);
}

template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_sum_lin(MeshView m, CaseView cv, Src<Dual> st,
                                                 const double* FL, const double* src, double* JV) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  stage_begin();
  const int c = stage_cell<double>(m, cv);
  if (c >= m.nc) return;
  const long nc = m.nc, nf = m.nf;
  double r[NF];
#pragma unroll
  for (int q = 0; q < NF; ++q) r[q] = 0.0;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    const bool isnb = (ent & FV_NB_BIT) != 0;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      const double x = FL[q * nf + f];
      r[q] += isnb ? -x : x;
    }
  }
  if (c == cv.pin) r[L::P] = st.t[(long)L::P * nc + c];
  if (TURB && !cv.wcell[c]) {
    r[L::K] += src[c];
    r[L::W] += src[nc + c];
  }
#pragma unroll
  for (int q = 0; q < NF; ++q) JV[q * nc + c] = r[q];
}

template <int DIM, bool TURB>
int run_linearised(FvCase* cs, const double* state, const double* tangent, double* JV,
                   cudaStream_t s) {
  constexpr int NF = Layout<DIM, TURB>::NFLD;
  const MeshView& m = cs->mesh->view;
  const CaseView& cv = cs->view;
  const long nc = m.nc, nf = m.nf;
  cs->fwd_valid = 0;  // the workspace is about to hold this pass
  Work<double> w = work_layout<double, DIM, TURB>(cs->work, nc, nf, 0);
  const int* tb = cs->tbs;
  auto bc = [&](int k) { return fv_blocks(nc, tb[k]); };
  const int nfi = m.nfi, nfb = m.nf - m.nfi, nw = cs->n_wall_cells;
  const double irho = 1.0 / cs->desc.rho;
  const Src<Dual> st{state, tangent};
  const Par<Dual> par{{cs->mu, 0.0}, {cs->inlet_scale, 0.0}, {cs->mu * irho, 0.0}};
  fv_prof_mark(cs, 0, s);
  const int sweeps = cs->desc.gradient_sweeps;
  const double rel = sweeps >= 1 ? cs->desc.gradient_relaxation : 1.0;
  double* x0 = sweeps <= 1 || (sweeps - 1) % 2 == 0 ? w.G : w.Galt;
  stage(k_grad_tangent<DIM, TURB>, bc(0), tb[0], s, m, cv, st, par, x0,
        sweeps <= 1 ? nullptr : w.Bg, rel);
  if (sweeps > 1)
    gg_sweeps<double, DIM, NF>(m, sweeps, rel, w.Bg, x0, x0 == w.G ? w.Galt : w.G, w.FL, s);
  const TangentOf G{cs->lin_g, w.G}, cl{cs->lin_cl, w.cl}, dco{cs->lin_d, w.dco};
  fv_prof_mark(cs, 1, s);
  if constexpr (TURB) {
    stage(k_closure_lin<DIM>, bc(1), tb[1], s, m, cv, st, cs->lin_g, w.G, cs->lin_cc, w.cl,
          cs->lin_src);
    if (nw > 0)
      stage(k_wall_closure<DIM>, fv_blocks(nw, 64), 64, s, m, cv, st, par, G, nw, cs->wall_cells,
            w.cl);
  }
  fv_prof_mark(cs, 2, s);
  if (nfi > 0)
    stage(k_apcoef_tangent<DIM, TURB>, fv_blocks(nfi, tb[2]), tb[2], s, m, cv, st, w.G, w.cl,
          cs->lin_aux, cs->lin_me, w.acown, w.acnb, w.me);
  if (nfb > 0)
    stage(k_apcoef_boundary<DIM, TURB>, fv_blocks(nfb, 64), 64, s, m, cv, st, par, G, cl, w.acown);
  fv_prof_mark(cs, 3, s);
  stage(k_dcoeff_tangent, bc(3), tb[3], s, m, w.acown, w.acnb, cs->lin_d, w.dco);
  fv_prof_mark(cs, 4, s);
  if (nfi > 0)
    stage(k_flux_tangent<DIM, TURB>, fv_blocks(nfi, tb[4]), tb[4], s, m, cv, st, w.G, w.cl, w.dco,
          w.me, cs->lin_aux, w.FL);
  if (nfb > 0)
    stage(k_flux_boundary<DIM, TURB>, fv_blocks(nfb, 64), 64, s, m, cv, st, par, G, cl, dco, w.FL);
  fv_prof_mark(cs, 5, s);
  stage(k_sum_lin<DIM, TURB>, bc(5), tb[5], s, m, cv, st, w.FL, cs->lin_src, JV);
  if constexpr (TURB) {
    if (nw > 0)
      stage(k_wall_rows<DIM>, fv_blocks(nw, 64), 64, s, m, cv, st, par, cl, G, nw, cs->wall_cells,
            JV);
  }
  fv_prof_mark(cs, 6, s);
  fv_prof_end_run(cs);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}
