// Mesh-coordinate adjoint: dL/dnodes of L = w . R(state, nodes), the node-coordinate part of
// theta_bar = -(dR/dtheta)^T lambda in _implicit_solve_bwd (aquaflux/solve/implicit.py:733-761).
// Included by residual.cu after the state adjoint (it reuses that adjoint's cotangents).
//
// Reverse mode over the stages, written out by hand from the forward formulas and the cotangents
// that the state adjoint left:
//   face fluxes           FL_bar = Wt_P - Wt_N, with the a_P face coefficients
//                         (a_bar = -d_bar d^2 / V of the owner / neighbour)     (k_nadj_face)
//   Green-Gauss gradients G_bar (linear in S_f, g, 1/V)                        (k_nadj_grad_*)
//   SST closure           (S, F1, nu_t, shear, imposed omega gradient)_bar     (k_nadj_closure)
//   SST sources           w on the k and omega rows                           (k_nadj_src)
//   d = V / a_P           d_bar d / V                                          (k_nadj_dcoeff)
// then back through the geometry formulas of geom.cuh, again by hand: the per-face factors (normal,
// face and cell centroids), the wall distance (nearest wall-face centroid) and its Green-Gauss
// gradient, the cell volumes / centroids (face areas, normals, centroids) and the face geometry
// (node coordinates; the owner-outward flip is a constant sign).  Wall-function cells and the
// limiters (a few per cent of the cells, and a formula with many branches) keep a seeded
// dual-number evaluation of the forward formula per geometric input (GeoSeed).
// The reverse pass costs a face about one flux evaluation; seeding every geometric input of every
// face cost 31 dual-number flux evaluations per face, FP64-bound (48^3 SST channel, GB300: the
// whole node VJP 21.9 ms seeded, 1.73 ms written out).  Every scatter is a gather over a precomputed
// incidence list: deterministic.
// Advection: first-order upwind and the limited linear upwind reconstruction (the centroids it
// reads, and the Venkatakrishnan limiters' geometry by seeded dual evaluations, k_nadj_limiter).
// Gradients: the compact scheme (with its relaxation) and the corrected scheme's swept solve
// (aquaflux/schemes/gradient.py:618-705, 1122-1337): the forward iterates X_0 .. X_{S-2} are
// recomputed, the sweeps reversed once more, and each sweep X' = X + rel (B - V X + C(X)) / V
// contributes the cotangents of 1/V, V and of C(X) = sum_f +-S_f ((1 - g) skew . X_P +
// g skew . X_N) (S_f, g, skew) at its own input; the numerator B takes rel X0_bar / V plus the
// sweeps' share (k_nadj_numerator_bar).  The SST wall-distance gradient is reversed the same way.


namespace {

// Rows of the face cotangents Fb (each nf long): face area, owner-outward normal, interpolation
// factor g, skew vector, face centroid, owner and neighbour cell centroid.  k_nadj_face folds the
// other per-face factors (dvec, dpn, dnn, nd, nn2, tP, tN, n x skew) into these; k_nadj_factors
// does g and the skew vector, to which the gradient stages add first.
template <int DIM>
struct FaceBar {
  static constexpr int A = 0, N = 1, G = 1 + DIM, SK = 2 + DIM, XF = 2 + 2 * DIM, XO = 2 + 3 * DIM,
                       XN = 2 + 4 * DIM, COUNT = 2 + 5 * DIM;
};

// A double array read as dual numbers with zero tangents.
struct Lifted {
  const double* p;
  __device__ __forceinline__ Dual operator[](long i) const { return {p[i], 0.0}; }
};

// The face fluxes' and the a_P face coefficients' geometry cotangents of one face, from the
// forward pass's kept intermediates (aux).  Interior face (o owner, n neighbour, lerp with g):
//   v_j = lerp(u_j) + skew . lerp(grad u_j),  mn = n . v,  me = rho mn A
//   damping = ((p_n - p_o) - gpf . dvec) / nd,  mdot = me - rho A nn2 lerp(d) damping
//   F_i = (lerp(p) + gpf . skew) A n_i - c (u_n - u_o + G_n . tN - G_o . tP) + mdot up_i
//   c = m_o m_n A / (dpn m_n - m_o dnn);  ac_own = c + max(me, 0), ac_nb = c + max(-me, 0)
// wdf: the cotangent of the owner's wall distance through the wall functions (boundary faces).
// FP64-bound: about 330 FP64 instructions for an interior SST face in 3D.
template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_nadj_face(MeshView m, CaseView cv, const double* state,
                                                   Par<double> par, const double* G,
                                                   const double* cl, const double* dco,
                                                   const double* me, const double* aux, AdjWork aw,
                                                   double* Fb, double* wdf) {
  using L = Layout<DIM, TURB>;
  using AX = Aux<DIM, TURB>;
  using R = FaceBar<DIM>;
  constexpr int NF = L::NFLD;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nc = m.nc, nf = m.nf;
  const int o = m.owner[f];
  const bool interior = f < m.nfi;
  const int n = interior ? m.nb[f] : o;
  const double A = m.area[f], rho = cv.rho, irho = cv.irho, nu = par.nu;
  auto st = [&](int q, int c) { return state[(long)q * nc + c]; };
  auto gr = [&](int q, int j, int c) { return G[((long)q * DIM + j) * nc + c]; };
  double nrm[DIM], dp[DIM], FLb[NF];
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    nrm[j] = m.normal[(long)j * nf + f];
    dp[j] = m.xf[(long)j * nf + f] - m.xc[(long)j * nc + o];
  }
#pragma unroll
  for (int q = 0; q < NF; ++q)
    FLb[q] = aw.Wt[(long)q * nc + o] - (interior ? aw.Wt[(long)q * nc + n] : 0.0) +
             (aw.FLx ? aw.FLx[(long)q * nf + f] : 0.0);
  double Ab = 0.0, gb = 0.0, dpnb = 0.0, wdb = 0.0;
  double nb_[DIM], skb[DIM], xfb[DIM], xob[DIM], xnb[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) nb_[j] = skb[j] = xfb[j] = xob[j] = xnb[j] = 0.0;
  const double abo = aw.apb[o];
  const double mest = me[f];
  // the cotangent of a limited reconstruction at upwind cell cu (psi itself: k_nadj_limiter)
  auto rec_adj = [&](int a, int q, bool own, double t) {
    const int cu = own ? o : n;
    const double ps = t * aw.psi[(long)a * nc + cu];
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double x = ps * gr(q, j, cu);
      xfb[j] += x;
      (own ? xob[j] : xnb[j]) -= x;
    }
  };
  if (interior) {
    const double g = m.g[f];
    const double mo = TURB ? par.mu + rho * cl[2L * nc + o] : mu_at(par, cv, o);
    const double mn_ = TURB ? par.mu + rho * cl[2L * nc + n] : mu_at(par, cv, n);
    const double dpn = m.dpn[f], dnn = m.dnn[f], inv_nd = m.inv_nd[f], nn2 = m.nn2[f];
    const double mdot = aux[f], damping = aux[1L * nf + f], dhat = aux[2L * nf + f];
    const double abn = aw.apb[n];
    const bool out = mdot >= 0.0;
    double dv[DIM], sk[DIM], tPb[DIM], tNb[DIM], gpfb[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      dv[j] = m.dvec[(long)j * nf + f];
      sk[j] = m.skew[(long)j * nf + f];
      tPb[j] = tNb[j] = 0.0;
    }
    // F_i
    double mdotb = FLb[L::P], pAb = 0.0, cb = abo + abn;
    double pf = lerp(st(L::P, o), st(L::P, n), g);
#pragma unroll
    for (int j = 0; j < DIM; ++j) pf += lerp(gr(L::P, j, o), gr(L::P, j, n), g) * sk[j];
    const double c = aux[3L * nf + f];
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      const double fb = FLb[i];
      double up = out ? st(i, o) : st(i, n);
      if (aw.psi && cv.rec_mom) {
        const int cu = out ? o : n;
        up += aw.psi[(long)i * nc + cu] * rec_dot<DIM>(m, G, i, f, cu);
        rec_adj(i, i, out, fb * mdot);
      }
      mdotb += fb * up;
      pAb += fb * nrm[i];
      nb_[i] += fb * (pf * A);
      cb -= fb * aux[(long)(AX::CPN + i) * nf + f];
      const double k1 = fb * c;
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        tPb[j] += k1 * gr(i, j, o);
        tNb[j] -= k1 * gr(i, j, n);
      }
    }
    Ab += pAb * pf;
    const double pfb = pAb * A;
    double dnnb = 0.0;
    // c = m_o m_n A / (dpn m_n - m_o dnn) and its cotangent
    auto conductance_bar = [&](double go, double gn, double cbar) {
      const double iden = 1.0 / (dpn * gn - go * dnn);
      const double t = cbar * (go * gn * iden);
      Ab += t;
      const double denb = t * A * iden;
      dpnb -= denb * gn;
      dnnb += denb * go;
    };
    conductance_bar(mo, mn_, cb);
    if constexpr (TURB) {
      const double vflux = mdot * irho;
      const bool vout = vflux >= 0.0;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int q = s == 0 ? L::K : L::W;
        const long b0 = AX::S0 + 4 * s;
        const double fb = FLb[q];
        double up = vout ? st(q, o) : st(q, n);
        if (aw.psi && cv.rec_sca) {
          const int cu = vout ? o : n;
          up += aw.psi[(long)(DIM + s) * nc + cu] * rec_dot<DIM>(m, G, q, f, cu);
          rec_adj(DIM + s, q, vout, fb * vflux);
        }
        mdotb += fb * up * irho;
        const double k1 = fb * aux[b0 * nf + f];
#pragma unroll
        for (int j = 0; j < DIM; ++j) {
          tPb[j] += k1 * gr(q, j, o);
          tNb[j] -= k1 * gr(q, j, n);
        }
        conductance_bar(cl[(4L + s) * nc + o], cl[(4L + s) * nc + n],
                        -fb * aux[(b0 + 3) * nf + f]);
      }
    }
    // mdot = me - rho A dhat damping
    const double rA = rho * A;
    Ab -= mdotb * rho * (dhat * damping);
    const double dhatb = -mdotb * rA * damping, dampb = -mdotb * rA * dhat;
    const double gdb = -dampb * inv_nd;
    // damping = num / nd: nd's cotangent (nd = dvec . n)
    const double ndb = gdb * damping;
    gb += pfb * (st(L::P, n) - st(L::P, o)) + dhatb * nn2 * (dco[n] - dco[o]);
    const double nn2b = 2.0 * (dhatb * lerp(dco[o], dco[n], g));
    // me = rho A mn
    const double meb = mdotb + (abo * dpos(mest) - abn * dpos(-mest));
    const double mnb = meb * rA;
    double mn = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double du = st(j, n) - st(j, o);
      double v = fma(g, du, st(j, o)), dvj = du;
      const double mj = mnb * nrm[j];
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
        const double go = gr(j, q, o), dg = gr(j, q, n) - go;
        const double gf = fma(g, dg, go);
        v += gf * sk[q];
        dvj += dg * sk[q];
        skb[q] += mj * gf;
      }
      mn += nrm[j] * v;
      nb_[j] += mnb * v + nn2b * nrm[j] + ndb * dv[j];
      gb += mj * dvj;
    }
    Ab += meb * rho * mn;
    // gpf, dvec; tP = dp - n dpn, tN = dn - n dnn (dn = dp - dvec); dpn = dp . n, dnn = dn . n
    double tpn = 0.0, tnn = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double po = gr(L::P, j, o), dpg = gr(L::P, j, n) - po, gpf = fma(g, dpg, po);
      skb[j] += pfb * gpf;
      gpfb[j] = pfb * sk[j] + gdb * dv[j];
      gb += gpfb[j] * dpg;
      const double db = gdb * gpf + ndb * nrm[j];
      xnb[j] += db;
      xob[j] -= db;
      tpn += tPb[j] * nrm[j];
      tnn += tNb[j] * nrm[j];
    }
    dpnb -= tpn;
    dnnb -= tnn;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double dn = dp[j] - dv[j];
      nb_[j] += dpnb * dp[j] + dnnb * dn - tPb[j] * dpn - tNb[j] * dnn;
      const double pb = tPb[j] + dpnb * nrm[j], qb = tNb[j] + dnnb * nrm[j];
      xfb[j] += pb + qb;
      xob[j] -= pb;
      xnb[j] -= qb;
    }
  } else {
    const signed char kind = cv.fkind[f];
    const double dpn = m.dpn[f], inv_nd = m.inv_nd[f], inv_dpn = m.inv_dpn[f];
    const double po = st(L::P, o);
    double bu[DIM], tPb[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      bu[j] = bvel(cv, nf, f, j, kind, st(j, o), par);
      tPb[j] = 0.0;
    }
    double un = 0.0, interp = 0.0, compact = 0.0, mdot = 0.0;
    if (kind == 2 || kind == 3) {
#pragma unroll
      for (int j = 0; j < DIM; ++j) un += bu[j] * nrm[j];
      if (kind == 3) {
#pragma unroll
        for (int j = 0; j < DIM; ++j) interp += gr(L::P, j, o) * nrm[j];
        compact = (cv.fp[f] - po) * inv_nd;
        un -= m.nn2[f] * dco[o] * (compact - interp);
      }
      mdot = (rho * A) * un;
    }
    const bool out = mdot >= 0.0;
    const double pf = bpress(cv, f, kind, po);
    double gbv = TURB ? par.mu + rho * cl[2L * nc + o] : mu_at(par, cv, o), dgb_dd = 0.0;
    const double vob_visc = gbv;  // inlet faces: the cell's own viscosity
    if (TURB && (kind == 0 || kind == 1)) {
      Dual nw{0.0, 0.0};
      if (cv.swall[f])
        nw = nut_wall(Dual{nu, 0.0}, Dual{cv.wd[o], 1.0}, Dual{st(L::K, o), 0.0});
      gbv = par.mu + rho * nw.v;
      dgb_dd = rho * nw.d;
    }
    const double gA = gbv * (A * inv_dpn);
    double mdotb = FLb[L::P], pAb = 0.0, gAb = 0.0;
    double inv_dpnb = 0.0;
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      const double fb = FLb[i], uo = st(i, o);
      double cp = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) cp += gr(i, j, o) * m.tP[(long)j * nf + f];
      double up = out ? uo : bu[i];
      if (out && aw.psi && cv.rec_mom) {
        up += aw.psi[(long)i * nc + o] * rec_dot<DIM>(m, G, i, f, o);
        rec_adj(i, i, true, fb * mdot);
      }
      mdotb += fb * up;
      pAb += fb * nrm[i];
      nb_[i] += fb * (pf * A);
      gAb -= fb * (bu[i] - uo - cp);
#pragma unroll
      for (int j = 0; j < DIM; ++j) tPb[j] += fb * gA * gr(i, j, o);
    }
    Ab += pAb * pf + gAb * (gbv * inv_dpn);
    inv_dpnb += gAb * (gbv * A);
    wdb += gAb * (A * inv_dpn) * dgb_dd;
    if constexpr (TURB) {
      const double vflux = mdot * irho;
      const bool vout = vflux >= 0.0;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int q = s == 0 ? L::K : L::W;
        const double fb = FLb[q], phio = st(q, o), go = cl[(4L + s) * nc + o];
        double cp = 0.0;
#pragma unroll
        for (int j = 0; j < DIM; ++j) cp += gr(q, j, o) * m.tP[(long)j * nf + f];
        const signed char sk = s == 0 ? cv.kkind[f] : cv.wkind[f];
        const double bphi = bscalar(sk, s == 0 ? cv.kval[f] : cv.wval[f], phio, cp);
        double gface = go, dgf_dd = 0.0;
        if (s == 0 && cv.swall[f]) {
          const Dual ww = wall_weight(Dual{nu, 0.0}, Dual{cv.wd[o], 1.0}, Dual{phio, 0.0});
          gface = (1.0 - ww.v) * go;
          dgf_dd = -ww.d * go;
        }
        double up = vout ? phio : bphi;
        if (vout && aw.psi && cv.rec_sca) {
          up += aw.psi[(long)(DIM + s) * nc + o] * rec_dot<DIM>(m, G, q, f, o);
          rec_adj(DIM + s, q, true, fb * vflux);
        }
        mdotb += fb * up * irho;
        const double num = bphi - phio - cp, Ad = A * inv_dpn;
        const double numb = -fb * gface * Ad, Adb = -fb * num * gface;
        Ab += Adb * inv_dpn;
        inv_dpnb += Adb * A;
        wdb += -fb * num * Ad * dgf_dd;
        // num = bphi - phi_o - cp and (zero gradient) bphi = phi_o + cp
        const double cpb = sk == 1 ? (vout ? 0.0 : fb * vflux) : -numb;
#pragma unroll
        for (int j = 0; j < DIM; ++j) tPb[j] += cpb * gr(q, j, o);
      }
    }
    // the a_P coefficient: vo = mu A / nd (walls, inlet), max(me, 0) (inlet, outlet)
    const double vob = (kind >= 0 && kind <= 2) ? abo : 0.0;
    const double bv = (TURB && (kind == 0 || kind == 1)) ? gbv : vob_visc;
    Ab += vob * bv * inv_nd;
    double inv_ndb = vob * bv * A;
    wdb += vob * (A * inv_nd) * dgb_dd;
    const double meb = ((kind == 2 || kind == 3) ? abo : 0.0) * dpos(mest);
    const double mnb = meb * rho * A;
    double mn = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      double v = st(j, o);
      const double mj = mnb * nrm[j];
#pragma unroll
      for (int q = 0; q < DIM; ++q) {
        v += gr(j, q, o) * m.skew[(long)q * nf + f];
        skb[q] += mj * gr(j, q, o);
      }
      mn += nrm[j] * v;
      nb_[j] += mnb * v;
    }
    Ab += meb * rho * mn;
    // the mass flux
    if (kind == 2 || kind == 3) {
      Ab += mdotb * rho * un;
      const double ub = mdotb * rho * A;
      double gpb = 0.0, nn2b = 0.0;
      if (kind == 3) {
        const double dh = m.nn2[f] * dco[o];
        nn2b = -2.0 * (ub * (compact - interp) * dco[o]);
        inv_ndb -= ub * dh * (cv.fp[f] - po);
        gpb = ub * dh;
      }
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        nb_[j] += ub * bu[j] + nn2b * nrm[j];
        if (kind == 3) nb_[j] += gpb * gr(L::P, j, o);
      }
    }
    // nd = dpn on a boundary face; tP = dp - n dpn, dpn = dp . n
    double tpn = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) tpn += tPb[j] * nrm[j];
    dpnb = -inv_ndb * inv_nd * inv_nd - inv_dpnb * inv_dpn * inv_dpn - tpn;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      nb_[j] += dpnb * dp[j] - tPb[j] * dpn;
      const double pb = tPb[j] + dpnb * nrm[j];
      xfb[j] += pb;
      xob[j] -= pb;
    }
  }
  Fb[(long)R::A * nf + f] = Ab;
  Fb[(long)R::G * nf + f] = gb;
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    Fb[(long)(R::N + j) * nf + f] = nb_[j];
    Fb[(long)(R::SK + j) * nf + f] = skb[j];
    Fb[(long)(R::XF + j) * nf + f] = xfb[j];
    Fb[(long)(R::XO + j) * nf + f] = xob[j];
    Fb[(long)(R::XN + j) * nf + f] = xnb[j];
  }
  if (TURB) wdf[f] = wdb;
}

// The Venkatakrishnan limiters' geometry (limiter_cell reads x_f, x_c and V): per cell and
// advected field with a limiter, d psi / d(geometry) by seeded dual evaluations contracted with
// psi_bar -- into Vb, limxc (DIM, nc) and limxf (DIM, ncf: per cell-face entry).
template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_nadj_limiter(MeshView m, const double* state,
                                                      const double* G, double Km, double Ks,
                                                      const double* psib, double* Vb,
                                                      double* limxc, double* limxf, long ncf) {
  constexpr int NA = DIM + (TURB ? 2 : 0);
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
#pragma unroll 1
  for (int a = 0; a < NA; ++a) {
    const double K = a < DIM ? Km : Ks;
    const double pb = psib[(long)a * nc + c];
    if (!(K > 0.0) || pb == 0.0) continue;
    const int q = advected_field<DIM, TURB>(a);
    auto eval = [&](const GeoSeed& gs) {
      auto phi = [&](int cell) { return Dual{state[(long)q * nc + cell], 0.0}; };
      auto grad = [&](int j) { return Dual{G[((long)q * DIM + j) * nc + c], 0.0}; };
      return limiter_cell<Dual, DIM>(m, c, K, phi, grad, gs).d;
    };
    Vb[c] += pb * eval(GeoSeed{-1, GC_VOL, -1, c});
#pragma unroll 1
    for (int j = 0; j < DIM; ++j) limxc[(long)j * nc + c] += pb * eval(GeoSeed{-1, GC_XC + j, -1, c});
#pragma unroll 1
    for (int i = b; i < e; ++i) {
      const int f = (int)(m.cf_face[i] & ~FV_NB_BIT);
      for (int j = 0; j < DIM; ++j) limxf[(long)j * ncf + i] += pb * eval(GeoSeed{GF_XF + j, -1, f, -1});
    }
  }
}

// Cell-centroid cotangents of the limiters (limxc), added to xcb.
__global__ void k_nadj_add(long n, const double* a, double* b) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] += a[i];
}

// Green-Gauss: G_c = (1/V_c) sum_f +-S_f phi_f, S_f = n_f A_f, phi_f = lerp(phi_P, phi_N, g_f) or
// the leading-order boundary value.
// nbar: the cotangent of the Green-Gauss numerator B phi per cell, (NF, DIM, nc).
template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_nadj_grad_face(MeshView m, CaseView cv,
                                                        const double* state, Par<double> par,
                                                        const double* nbar, double* Fb) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nc = m.nc, nf = m.nf;
  const int o = m.owner[f];
  const double A = m.area[f];
  double nrm[DIM], Sb[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    nrm[j] = m.normal[(long)j * nf + f];
    Sb[j] = 0.0;
  }
  if (f < m.nfi) {
    const int n = m.nb[f];
    const double g = m.g[f];
    double gb = 0.0;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      const double po = state[(long)q * nc + o], pn = state[(long)q * nc + n];
      const double pf = lerp(po, pn, g);
      double pbar = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        const double y = nbar[((long)q * DIM + j) * nc + o] - nbar[((long)q * DIM + j) * nc + n];
        Sb[j] += pf * y;
        pbar += nrm[j] * A * y;
      }
      gb += pbar * (pn - po);
    }
    Fb[(long)FaceBar<DIM>::G * nf + f] += gb;
  } else {
    const signed char kind = cv.fkind[f];
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      const double po = state[(long)q * nc + o];
      double pb;
      if (q < DIM) pb = bvel(cv, nf, f, q, kind, po, par);
      else if (q == L::P) pb = bpress(cv, f, kind, po);
      else if (q == L::K) pb = bscalar(cv.kkind[f], cv.kval[f], po, 0.0);
      else pb = bscalar(cv.wkind[f], cv.wval[f], po, 0.0);
#pragma unroll
      for (int j = 0; j < DIM; ++j) Sb[j] += pb * nbar[((long)q * DIM + j) * nc + o];
    }
  }
  double ab = 0.0;
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    ab += Sb[j] * nrm[j];
    Fb[(long)(FaceBar<DIM>::N + j) * nf + f] += Sb[j] * A;
  }
  Fb[(long)FaceBar<DIM>::A * nf + f] += ab;
}

// The numerator cotangent of NQ Green-Gauss fields: X0 = rel B / V (the gradient itself for the
// compact scheme), so B_bar = rel X0_bar / V, plus the swept sweeps' share Bsw (may be null).
template <int DIM, int NQ>
__global__ void k_nadj_numerator_bar(MeshView m, const double* X0b, const double* Bsw, double rel,
                                     double* nbar) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc;
  const double r = rel * m.inv_vol[c];
  for (int k = 0; k < NQ * DIM; ++k) {
    const long i = (long)k * nc + c;
    nbar[i] = X0b[i] * r + (Bsw ? Bsw[i] : 0.0);
  }
}

// 1/V part of the first gradient iterate X0 = rel B / V: ivb += rel X0_bar . B, with B = X0 V / rel
// for the compact scheme (Bnum null) or the stored numerator.
template <int DIM, int NQ>
__global__ void k_nadj_grad_cell(MeshView m, const double* X0b, const double* X0,
                                 const double* Bnum, double rel, double* ivb) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc;
  double acc = 0.0;
  for (int k = 0; k < NQ * DIM; ++k) acc += X0b[(long)k * nc + c] * (Bnum ? Bnum[(long)k * nc + c] : X0[(long)k * nc + c]);
  ivb[c] += Bnum ? rel * acc : acc * m.vol[c];
}

// d = V / a_P: the volume part.
__global__ void k_nadj_dcoeff(MeshView m, const double* dco, const double* dcob, double* Cb) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  Cb[(long)GC_VOL * m.nc + c] += dcob[c] * dco[c] / m.vol[c];
}

// X0 = rel B / V.
template <int DIM, int NQ>
__global__ void k_nadj_x0(MeshView m, const double* B, double rel, double* X0) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc;
  const double iv = m.inv_vol[c];
  for (int k = 0; k < NQ * DIM; ++k) X0[(long)k * nc + c] = rel * (B[(long)k * nc + c] * iv);
}

// One swept sweep X' = X + rel (B - (V X - C(X))) / V, its geometry cotangents at input X with
// output cotangent Y.  Face part (interior faces): w_f = (1 - g) skew . X_P + g skew . X_N (kept
// in wface for the cell part) and the cotangents of S_f, g, skew from C = sum +-S_f w_f.
template <int DIM, int NQ>
__global__ void __launch_bounds__(128) k_nadj_sweep_face(MeshView m, const double* X,
                                                         const double* Y, double rel, double* Fb,
                                                         double* wface) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nfi) return;
  const int nc = m.nc, nf = m.nf;
  const int o = m.owner[f], n = m.nb[f];
  const double A = m.area[f], g = m.g[f];
  const double ro = rel * m.inv_vol[o], rn = rel * m.inv_vol[n];
  double nrm[DIM], sk[DIM], Sb[DIM], skb[DIM];
  for (int j = 0; j < DIM; ++j) {
    nrm[j] = m.normal[(long)j * nf + f];
    sk[j] = m.skew[(long)j * nf + f];
    Sb[j] = 0.0;
    skb[j] = 0.0;
  }
  double gb = 0.0;
  for (int q = 0; q < NQ; ++q) {
    double so = 0.0, sn = 0.0;
    for (int j = 0; j < DIM; ++j) {
      so += sk[j] * X[((long)q * DIM + j) * nc + o];
      sn += sk[j] * X[((long)q * DIM + j) * nc + n];
    }
    const double w = (1.0 - g) * so + g * sn;
    wface[(long)q * nf + f] = w;
    double wb = 0.0;
    for (int j = 0; j < DIM; ++j) {
      const double D = Y[((long)q * DIM + j) * nc + o] * ro - Y[((long)q * DIM + j) * nc + n] * rn;
      Sb[j] += D * w;
      wb += D * nrm[j] * A;
    }
    gb += wb * (sn - so);
    for (int j = 0; j < DIM; ++j)
      skb[j] += wb * ((1.0 - g) * X[((long)q * DIM + j) * nc + o] + g * X[((long)q * DIM + j) * nc + n]);
  }
  double ab = 0.0;
  for (int j = 0; j < DIM; ++j) {
    ab += Sb[j] * nrm[j];
    Fb[(long)(FaceBar<DIM>::N + j) * nf + f] += Sb[j] * A;
    Fb[(long)(FaceBar<DIM>::SK + j) * nf + f] += skb[j];
  }
  Fb[(long)FaceBar<DIM>::A * nf + f] += ab;
  Fb[(long)FaceBar<DIM>::G * nf + f] += gb;
}

// ... cell part: C(X) from wface, then the cotangents of 1/V (rel (B - V X + C) . Y) and of V
// (-rel X . Y / V).
template <int DIM, int NQ>
__global__ void __launch_bounds__(128) k_nadj_sweep_cell(MeshView m, const double* X,
                                                         const double* Y, const double* B,
                                                         const double* wface, double rel,
                                                         double* ivb, double* Vb) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  double corr[NQ][DIM];
  for (int q = 0; q < NQ; ++q)
    for (int j = 0; j < DIM; ++j) corr[q][j] = 0.0;
  bool any = false;
  for (int i = m.cf_ptr[c]; i < m.cf_ptr[c + 1]; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    if (f >= m.nfi) continue;
    any = true;
    const double A = (ent & FV_NB_BIT) ? -m.area[f] : m.area[f];
    for (int q = 0; q < NQ; ++q)
      for (int j = 0; j < DIM; ++j) corr[q][j] += (m.normal[(long)j * nf + f] * A) * wface[(long)q * nf + f];
  }
  const double V = m.vol[c];
  double aiv = 0.0, av = 0.0;
  for (int q = 0; q < NQ; ++q)
    for (int j = 0; j < DIM; ++j) {
      const long k = ((long)q * DIM + j) * nc + c;
      const double x = X[k], y = Y[k];
      const double ax = any ? x * V - corr[q][j] : x * V;
      aiv += (B[k] - ax) * y;
      av += x * y;
    }
  ivb[c] += rel * aiv;
  Vb[c] += -rel * m.inv_vol[c] * av;
}

// Buffers of the swept reversal for NQ fields: S - 1 forward iterates, two cotangents, a
// numerator-sweep accumulator, and the face values.
struct SweepBufs {
  double* X;     // (S - 1) iterates X_0 .. X_{S-2}, each (NQ, DIM, nc)
  double* Y0;
  double* Y1;
  double* Bsw;   // sum over the sweeps of rel Y / V: the numerator's share
  double* nbar;
  double* wface; // (NQ, nf)
};

SweepBufs sweep_layout(double* p, int sweeps, int nq, int dim, long nc, long nf) {
  const long blk = (long)nq * dim * nc;
  SweepBufs b;
  b.X = p; p += (long)std::max(sweeps - 1, 1) * blk;
  b.Y0 = p; p += blk;
  b.Y1 = p; p += blk;
  b.Bsw = p; p += blk;
  b.nbar = p; p += blk;
  b.wface = p;
  return b;
}

size_t sweep_doubles(int sweeps, int nq, int dim, long nc, long nf) {
  return (size_t)(std::max(sweeps - 1, 1) + 4) * nq * dim * nc + (size_t)nq * nf;
}

// The corrected scheme's reversal for NQ fields with numerator B (stored) and the cotangent Gb of
// the last iterate: contributions of every sweep to Fb / ivb / Vb; on return bf.nbar holds the
// numerator's cotangent and ivb the first iterate's 1/V part.
template <int DIM, int NQ>
int sweeps_geometry(const MeshView& m, int sweeps, double rel, const double* B, const double* Gb,
                    const SweepBufs& bf, double* Fb, double* ivb, double* Vb, cudaStream_t s) {
  constexpr int TB = 128;
  const long blk = (long)NQ * DIM * m.nc;
  const int bc = fv_blocks(m.nc, TB), bfi = fv_blocks(m.nfi > 0 ? m.nfi : 1, TB);
  // forward iterates X_0 .. X_{S-2}
  k_nadj_x0<DIM, NQ><<<bc, TB, 0, s>>>(m, B, rel, bf.X);
  for (int it = 1; it < sweeps - 1; ++it) {
    if (m.nfi > 0) k_gg_skew<double, DIM, NQ><<<bfi, TB, 0, s>>>(m, bf.X + (it - 1) * blk, bf.wface);
    k_gg_sweep<double, DIM, NQ><<<bc, TB, 0, s>>>(m, B, bf.X + (it - 1) * blk, bf.wface, rel,
                                                   bf.X + it * blk);
  }
  // backward: sweep k maps X_{k-1} to X_k; Y holds X_k's cotangent
  FV_CUDA_TRY(cudaMemcpyAsync(bf.Y0, Gb, sizeof(double) * blk, cudaMemcpyDeviceToDevice, s));
  double* Y = bf.Y0;
  double* Yn = bf.Y1;
  MeshView mv = m;
  for (int k = sweeps - 1; k >= 1; --k) {
    const double* Xin = bf.X + (k - 1) * blk;
    if (m.nfi > 0) k_nadj_sweep_face<DIM, NQ><<<bfi, TB, 0, s>>>(mv, Xin, Y, rel, Fb, bf.wface);
    k_nadj_sweep_cell<DIM, NQ><<<bc, TB, 0, s>>>(mv, Xin, Y, B, bf.wface, rel, ivb, Vb);
    if (m.nfi > 0) a_gg_skew<DIM, NQ><<<bfi, TB, 0, s>>>(mv, Y, rel, bf.wface);
    a_gg_sweep<DIM, NQ><<<bc, TB, 0, s>>>(mv, Y, bf.wface, rel, k == sweeps - 1, bf.Bsw, Yn);
    double* t = Y;
    Y = Yn;
    Yn = t;
  }
  // Y = X0_bar
  k_nadj_numerator_bar<DIM, NQ><<<bc, TB, 0, s>>>(mv, Y, bf.Bsw, rel, bf.nbar);
  k_nadj_grad_cell<DIM, NQ><<<bc, TB, 0, s>>>(mv, Y, bf.X, B, rel, ivb);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

// The wall-distance gradient's numerator sum_f +-S_f d_f (d_f the interpolated distance, 0 on SST
// walls, the owner's value on other boundaries), (DIM, nc).
template <int DIM>
__global__ void k_nadj_wd_numerator(MeshView m, CaseView cv, double* num) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  double acc[DIM];
  for (int j = 0; j < DIM; ++j) acc[j] = 0.0;
  const double phic = cv.wd[c];
  for (int i = m.cf_ptr[c]; i < m.cf_ptr[c + 1]; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    double phif;
    if (f < m.nfi) {
      const double g = m.g[f];
      phif = (1.0 - g) * cv.wd[m.owner[f]] + g * cv.wd[m.nb[f]];
    } else {
      phif = cv.swall[f] ? 0.0 : phic;
    }
    const double sgn = (ent & FV_NB_BIT) ? -phif : phif;
    for (int j = 0; j < DIM; ++j) acc[j] += (m.normal[(long)j * nf + f] * m.area[f]) * sgn;
  }
  for (int j = 0; j < DIM; ++j) num[(long)j * nc + c] = acc[j];
}

// Wall cells: the closure's wall-distance inputs and the wall faces' areas by seeded evaluations,
// one per thread (blockIdx.y picks the input; a cell's seven seeded closures in one thread were one
// serial chain: 385 us of the 48^3 channel's node VJP against 141 us).  Off the wall only 1/d and
// 1/d^2 enter, through c1 = sqrt(k) / (beta* w d), vt = 500 nu / (d^2 w) and
// c2 = 4 sigma_w2 k / (cd d^2): the reverse of F1 = tanh(min(max(c1, vt), c2)^4) and
// nu_t = A1 k / max(A1 w, S tanh(max(2 c1, vt)^2)), as in a_closure.
template <int DIM>
__global__ void __launch_bounds__(128) k_nadj_closure(MeshView m, CaseView cv, const double* state,
                                                      Par<Dual> par, const double* G,
                                                      const double* cl, const double* Gwi,
                                                      const double* clb, const double* Gwib,
                                                      double* Cb, double* Fb) {
  using L = Layout<DIM, true>;
  const int c = stage_cell(m, cv);
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  if (cv.wcell[c]) {
    const Src<Dual> st{state, nullptr};
    auto contract = [&](const GeoSeed& gs) {
      Dual out[7], gw[DIM];
      closure_cell<Dual, DIM>(m, cv, st, par, Lifted{G}, c, gs, out, gw);
      double acc = 0.0;
      for (int i = 0; i < 4; ++i) acc += clb[(long)i * nc + c] * out[i].d;
      for (int j = 0; j < DIM; ++j) acc += Gwib[(long)j * nc + c] * gw[j].d;
      return acc;
    };
    const int comp = GC_WD + blockIdx.y;
    if (comp < GC_WDG + DIM) {
      Cb[(long)comp * nc + c] += contract(GeoSeed{-1, comp, -1, c});
      return;
    }
    const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
    for (int i = b; i < e; ++i) {
      const int f = (int)(m.cf_face[i] & ~FV_NB_BIT);
      if (f < m.nfi || !cv.swall[f]) continue;
      Fb[(long)FaceBar<DIM>::A * nf + f] += contract(GeoSeed{GF_AREA, -1, f, -1});
    }
    return;
  }
  if (blockIdx.y != 0) return;
  const double kp = fmax(state[(long)L::K * nc + c], 0.0), w = state[(long)L::W * nc + c];
  const double S = cl[c], F1 = cl[(long)nc + c], F2 = cl[6L * nc + c], nu = par.nu.v;
  const double id = cv.inv_wd[c], id2 = cv.inv_wd2[c], iw = 1.0 / w;
  double dot = 0.0;
#pragma unroll
  for (int j = 0; j < DIM; ++j)
    dot += G[((long)L::K * DIM + j) * nc + c] * Gwi[(long)j * nc + c];
  const double icd = 1.0 / fmax((2.0 * SIGMA_W2) * dot * iw, CROSS_FLOOR);
  const double siw = (kp > 0.0 ? sqrt(kp) : 0.0) * iw * (1.0 / BETA_STAR);
  const double nuw = 500.0 * nu * iw, kcd = (4.0 * SIGMA_W2) * kp * icd;
  const double c1 = siw * id, vt = nuw * id2, c2 = kcd * id2;
  double c1b = 0.0, vtb = 0.0, c2b = 0.0;
  const double iMx = 1.0 / fmax(A1 * w, S * F2);
  const double Mb = -clb[2L * nc + c] * (A1 * kp) * iMx * iMx;
  double awb = 0.0, sfb = 0.0, a2b = 0.0, innerb = 0.0;
  split_ext(A1 * w, S * F2, Mb, false, &awb, &sfb);
  const double a2 = 2.0 * c1, arg2 = fmax(a2, vt);
  split_ext(a2, vt, sfb * S * (1.0 - F2 * F2) * 2.0 * arg2, false, &a2b, &vtb);
  const double inner = fmax(c1, vt), arg1 = fmin(inner, c2);
  split_ext(inner, c2, clb[(long)nc + c] * (1.0 - F1 * F1) * 4.0 * (arg1 * arg1 * arg1), true,
            &innerb, &c2b);
  split_ext(c1, vt, innerb, false, &c1b, &vtb);
  c1b += 2.0 * a2b;
  Cb[(long)GC_INV_WD * nc + c] += c1b * siw;
  Cb[(long)GC_INV_WD2 * nc + c] += vtb * nuw + c2b * kcd;
}

// The k and omega source rows: off the wall V times a density, so the volume part is the rows' own
// value over V; wall cells by seeded evaluations (blockIdx.y: V, the wall functions' distance).
template <int DIM>
__global__ void __launch_bounds__(128) k_nadj_src(MeshView m, CaseView cv, const double* state,
                                                  Par<Dual> par, const double* cl, const double* G,
                                                  const double* Gwi, const double* W, double* Cb) {
  using L = Layout<DIM, true>;
  const int c = stage_cell(m, cv);
  if (c >= m.nc) return;
  const int nc = m.nc;
  const double wk = W[(long)L::K * nc + c], ww = W[(long)L::W * nc + c];
  if (!cv.wcell[c]) {
    if (blockIdx.y != 0) return;
    const Src<double> st{state};
    const Par<double> pd{par.mu.v, par.iscale.v, par.nu.v};
    double rk = 0.0, rw = 0.0;
    sst_rows<double, DIM>(m, cv, st, pd, cl, G, Gwi, c, rk, rw);
    Cb[(long)GC_VOL * nc + c] += (wk * rk + ww * rw) * m.inv_vol[c];
    return;
  }
  const Src<Dual> st{state, nullptr};
  const int comp = GC_VOL + blockIdx.y;
  Dual rk{0.0, 0.0}, rw{0.0, 0.0};
  sst_rows<Dual, DIM>(m, cv, st, par, Lifted{cl}, Lifted{G}, Lifted{Gwi}, c, rk, rw,
                      GeoSeed{-1, comp, -1, c});
  Cb[(long)comp * nc + c] += wk * rk.d + ww * rw.d;
}

// Wall-distance gradient (compact Green-Gauss of d: Dirichlet 0 on SST walls, the owner value on
// other boundaries): face part.
// nb: the cotangent of the gradient's numerator per cell, (DIM, nc).
template <int DIM>
__global__ void k_nadj_wdg_face(MeshView m, CaseView cv, const double* nb, double* Fb,
                                double* dpart) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nc = m.nc, nf = m.nf;
  const int o = m.owner[f];
  const double A = m.area[f];
  double nrm[DIM], Sb[DIM];
  for (int j = 0; j < DIM; ++j) {
    nrm[j] = m.normal[(long)j * nf + f];
    Sb[j] = 0.0;
  }
  double pbar = 0.0, d_o = 0.0, d_n = 0.0, po = 0.0, pn = 0.0;
  if (f < m.nfi) {
    const int n = m.nb[f];
    const double g = m.g[f];
    d_o = cv.wd[o];
    d_n = cv.wd[n];
    const double df = (1.0 - g) * d_o + g * d_n;
    for (int j = 0; j < DIM; ++j) {
      const double y = nb[(long)j * nc + o] - nb[(long)j * nc + n];
      Sb[j] += df * y;
      pbar += nrm[j] * A * y;
    }
    Fb[(long)FaceBar<DIM>::G * nf + f] += pbar * (d_n - d_o);
    po = (1.0 - g) * pbar;
    pn = g * pbar;
  } else {
    const double df = cv.swall[f] ? 0.0 : cv.wd[o];
    for (int j = 0; j < DIM; ++j) {
      const double y = nb[(long)j * nc + o];
      Sb[j] += df * y;
      pbar += nrm[j] * A * y;
    }
    po = cv.swall[f] ? 0.0 : pbar;
  }
  double ab = 0.0;
  for (int j = 0; j < DIM; ++j) {
    ab += Sb[j] * nrm[j];
    Fb[(long)(FaceBar<DIM>::N + j) * nf + f] += Sb[j] * A;
  }
  Fb[(long)FaceBar<DIM>::A * nf + f] += ab;
  dpart[f] = po;
  dpart[(long)nf + f] = pn;
}

// ... cell part: the d cotangent from the faces (the 1/V part goes through ivb).
template <int DIM>
__global__ void k_nadj_wdg_cell(MeshView m, CaseView cv, const double* dpart, double* Cb) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  double db = 0.0;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    db += (ent & FV_NB_BIT) ? dpart[(long)nf + f] : dpart[f];
  }
  Cb[(long)GC_WD * nc + c] += db;
}

// Cell scalars: V_bar (with the 1/V cotangent) and the wall-distance cotangent; the nearest wall
// face's centroid and the cell centroid take d_bar (x_c - x_w) / d.
template <int DIM, bool TURB>
__global__ void k_nadj_cell_chain(MeshView m, CaseView cv, const double* Cb, const double* ivb,
                                  const double* wdf, const int* wnear, double* Vb, double* xcb,
                                  double* wcon) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  const double iv = m.inv_vol[c];
  Vb[c] += Cb[(long)GC_VOL * nc + c] - ivb[c] * iv * iv;
  for (int j = 0; j < DIM; ++j) xcb[(long)j * nc + c] = 0.0;
  if (!TURB) return;
  double db = Cb[(long)GC_WD * nc + c];
  const double i1 = cv.inv_wd[c], i2 = cv.inv_wd2[c];
  db += -Cb[(long)GC_INV_WD * nc + c] * i1 * i1 - 2.0 * Cb[(long)GC_INV_WD2 * nc + c] * i1 * i2;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const int f = (int)(m.cf_face[i] & ~FV_NB_BIT);
    if (f >= m.nfi && m.owner[f] == c) db += wdf[f];
  }
  const int w = wnear[c];
  const double d = cv.wd[c];
  for (int j = 0; j < DIM; ++j) {
    const double t = d > 0.0 ? db * (m.xc[(long)j * nc + c] - m.xf[(long)j * nf + w]) / d : 0.0;
    xcb[(long)j * nc + c] = t;
    wcon[(long)j * nc + c] = t;
  }
}

template <int DIM>
__global__ void k_nadj_wall_face(MeshView m, const int* wall_ptr, const int* wall_cell,
                                 const double* wcon, double* xfb) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nc = m.nc, nf = m.nf;
  for (int i = wall_ptr[f]; i < wall_ptr[f + 1]; ++i) {
    const int c = wall_cell[i];
    for (int j = 0; j < DIM; ++j) xfb[(long)j * nf + f] -= wcon[(long)j * nc + c];
  }
}

// Interpolation factor and skew vector -> face centroid and the two cell centroids:
// skew = x_f - (x_o + g d), g = (x_f - x_o) . d / d . d, d = x_n - x_o (boundary: d = 0, g = 0).
// Adds the rows' own centroid parts; xcpart is Fb's owner / neighbour centroid rows, in place.
template <int DIM>
__global__ void __launch_bounds__(128) k_nadj_factors(MeshView m, double* Fb, double* xfb) {
  using R = FaceBar<DIM>;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nc = m.nc, nf = m.nf;
  double skb[DIM], db[DIM], dpb[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    dpb[j] = skb[j] = Fb[(long)(R::SK + j) * nf + f];
    db[j] = 0.0;
  }
  if (f < m.nfi) {
    const int o = m.owner[f];
    const double g = m.g[f];
    double gb = Fb[(long)R::G * nf + f], dd = 0.0, d[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      d[j] = m.dvec[(long)j * nf + f];
      dd += d[j] * d[j];
      gb -= skb[j] * d[j];
    }
    const double fdb = gb / dd, ddb2 = -2.0 * fdb * g;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double dp = m.xf[(long)j * nf + f] - m.xc[(long)j * nc + o];
      db[j] = fdb * dp + ddb2 * d[j] - skb[j] * g;
      dpb[j] += fdb * d[j];
    }
  }
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    xfb[(long)j * nf + f] += Fb[(long)(R::XF + j) * nf + f] + dpb[j];
    Fb[(long)(R::XO + j) * nf + f] -= dpb[j] + db[j];
    Fb[(long)(R::XN + j) * nf + f] += db[j];
  }
}

template <int DIM>
__global__ void k_nadj_xc_gather(MeshView m, const double* xcpart, double* xcb) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  double acc[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) acc[j] = xcb[(long)j * nc + c];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    const long base = (ent & FV_NB_BIT) ? (long)DIM * nf : 0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) acc[j] += xcpart[base + (long)j * nf + f];
  }
#pragma unroll
  for (int j = 0; j < DIM; ++j) xcb[(long)j * nc + c] = acc[j];
}

// Cell volume and centroid -> the areas, normals and centroids of the cell's faces, the reverse of
// cell_geom: a = mean x_f, loc = x_f - a, fl = +-(loc . n) A, V = sum fl / D,
// x_c = sum fl loc / ((D + 1) V) + a.
template <int DIM>
__global__ void __launch_bounds__(128) k_nadj_cell_geom(MeshView m, const double* Vb,
                                                        const double* xcb, double* cfA,
                                                        double* cfN, double* cfX, long ncf) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  const double iv = m.inv_vol[c], inv_k = 1.0 / (double)(e - b);
  double a[DIM], csb[DIM], ab[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) a[j] = 0.0;
  for (int i = b; i < e; ++i) {
    const int f = (int)(m.cf_face[i] & ~FV_NB_BIT);
#pragma unroll
    for (int j = 0; j < DIM; ++j) a[j] += m.xf[(long)j * nf + f];
  }
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    a[j] *= inv_k;
    ab[j] = xcb[(long)j * nc + c];
    csb[j] = ab[j] * iv * (1.0 / (DIM + 1));
  }
  double dotx = 0.0;  // sum fl loc . csb: x_c's cotangent on 1 / ((D + 1) V), times that factor
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    double dn = 0.0, dc = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double loc = m.xf[(long)j * nf + f] - a[j];
      dn += loc * m.normal[(long)j * nf + f];
      dc += loc * csb[j];
    }
    dotx += ((ent & FV_NB_BIT) ? -dn : dn) * m.area[f] * dc;
  }
  const double vb = (Vb[c] - dotx * iv) * (1.0 / DIM);
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    const double A = (ent & FV_NB_BIT) ? -m.area[f] : m.area[f];
    double loc[DIM], n[DIM], dn = 0.0, flb = vb;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      loc[j] = m.xf[(long)j * nf + f] - a[j];
      n[j] = m.normal[(long)j * nf + f];
      dn += loc[j] * n[j];
      flb += csb[j] * loc[j];
    }
    const double fl = dn * A, dnb = A * flb;
    cfA[i] = (ent & FV_NB_BIT) ? -dn * flb : dn * flb;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double lb = csb[j] * fl + dnb * n[j];
      cfN[(long)j * ncf + i] = dnb * loc[j];
      cfX[(long)j * ncf + i] = lb;
      ab[j] -= lb;
    }
  }
  for (int i = b; i < e; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) cfX[(long)j * ncf + i] += ab[j] * inv_k;
}

__device__ __forceinline__ int cf_entry(const MeshView& m, int c, int f, bool nb) {
  const unsigned want = (unsigned)f | (nb ? FV_NB_BIT : 0u);
  for (int i = m.cf_ptr[c]; i < m.cf_ptr[c + 1]; ++i)
    if (m.cf_face[i] == want) return i;
  return -1;
}

// Totals of the face primitives' cotangents (residual stages + factors + cell geometry).
template <int DIM>
__global__ void k_nadj_cf_gather(MeshView m, const double* Fb, const double* cfA, const double* cfN,
                                 const double* cfX, const double* limxf, long ncf, double* Ab,
                                 double* nbt, double* xfb) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nf = m.nf;
  const int eo = cf_entry(m, m.owner[f], f, false);
  const int en = f < m.nfi ? cf_entry(m, m.nb[f], f, true) : -1;
  double a = Fb[(long)FaceBar<DIM>::A * nf + f];
  if (eo >= 0) a += cfA[eo];
  if (en >= 0) a += cfA[en];
  Ab[f] = a;
  for (int j = 0; j < DIM; ++j) {
    double nb = 0.0, xb = 0.0;
    if (eo >= 0) {
      nb += cfN[(long)j * ncf + eo];
      xb += cfX[(long)j * ncf + eo];
      if (limxf) xb += limxf[(long)j * ncf + eo];
    }
    if (en >= 0) {
      nb += cfN[(long)j * ncf + en];
      xb += cfX[(long)j * ncf + en];
      if (limxf) xb += limxf[(long)j * ncf + en];
    }
    nbt[(long)j * nf + f] = Fb[(long)(FaceBar<DIM>::N + j) * nf + f] + nb;
    xfb[(long)j * nf + f] += xb;
  }
}

// Face area / normal / centroid -> the face's node coordinates, the reverse of face_geom.
// 3D fan over k triangles (p_i, p_i+1, pa = mean p): d_i = (p_i - pa) x (p_i+1 - pa) / 2, S = sum d_i,
// A = |S|, n = S / A, x_f = sum (d_i . n) t_i / A, t_i = (pa + p_i + p_i+1) / 3.  K > 0: a
// compile-time node count (quads; the nodes and their cotangents in registers), K = 0: any.
template <int K>
__device__ __forceinline__ void face_geom_bar_3d(int k, const double* nodes, const int* idx,
                                                 const double* ns, double ab, const double* nbs,
                                                 const double* xb, double* out) {
  const int kk = K > 0 ? K : k;
  double local[K > 0 ? 3 * K : 1], nodel[K > 0 ? 3 * K : 1];  // K = 0: unused
  double* acc = K > 0 ? local : out;
  if constexpr (K > 0) {
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) nodel[3 * i + j] = nodes[3L * idx[i] + j];
  }
  auto P = [&](int i, int j) {
    if constexpr (K > 0) return nodel[3 * i + j];
    else return nodes[3L * idx[i] + j];
  };
  double pa[3] = {0.0, 0.0, 0.0}, S[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 0; i < kk; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      pa[j] += P(i, j);
      acc[3 * i + j] = 0.0;
    }
  const double inv = 1.0 / (double)kk;
#pragma unroll
  for (int j = 0; j < 3; ++j) pa[j] *= inv;
  auto tri = [&](int i, double* u, double* v, double* d) {
    const int i1 = i + 1 == kk ? 0 : i + 1;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      u[j] = P(i, j) - pa[j];
      v[j] = P(i1, j) - pa[j];
    }
    d[0] = 0.5 * (u[1] * v[2] - u[2] * v[1]);
    d[1] = 0.5 * (u[2] * v[0] - u[0] * v[2]);
    d[2] = 0.5 * (u[0] * v[1] - u[1] * v[0]);
  };
#pragma unroll
  for (int i = 0; i < kk; ++i) {
    double u[3], v[3], d[3];
    tri(i, u, v, d);
#pragma unroll
    for (int j = 0; j < 3; ++j) S[j] += d[j];
  }
  const double sq = S[0] * S[0] + S[1] * S[1] + S[2] * S[2];
  if (sq > 0.0) {
    const double a = sqrt(sq), ia = 1.0 / a;
    const double n[3] = {S[0] * ia, S[1] * ia, S[2] * ia};
    const double sgn = n[0] * ns[0] + n[1] * ns[1] + n[2] * ns[2] < 0.0 ? -1.0 : 1.0;
    double cb[3], nb[3], c[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cb[j] = xb[j] * ia;
      nb[j] = sgn * nbs[j];
    }
    // t_i = pa + (u_i + v_i) / 3 and sum (d_i . n) = A: x_f = pa + sum (d_i . n) (u_i + v_i) / 3 A,
    // the same centroid about pa (no cancellation of the face's position)
    auto weight_bar = [&](const double* u, const double* v) {
      return (cb[0] * (u[0] + v[0]) + cb[1] * (u[1] + v[1]) + cb[2] * (u[2] + v[2])) * (1.0 / 3.0);
    };
#pragma unroll
    for (int i = 0; i < kk; ++i) {
      double u[3], v[3], d[3];
      tri(i, u, v, d);
      const double w = d[0] * n[0] + d[1] * n[1] + d[2] * n[2];
      const double wb = weight_bar(u, v);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        nb[j] += wb * d[j];
        c[j] += w * ((u[j] + v[j]) * (1.0 / 3.0));
      }
    }
    double abt = ab;
#pragma unroll
    for (int j = 0; j < 3; ++j) abt -= (cb[j] * c[j] + nb[j] * n[j]) * ia;
    double Sb[3], pab[3] = {xb[0], xb[1], xb[2]};
#pragma unroll
    for (int j = 0; j < 3; ++j) Sb[j] = nb[j] * ia + abt * n[j];
#pragma unroll
    for (int i = 0; i < kk; ++i) {
      const int i1 = i + 1 == kk ? 0 : i + 1;
      double u[3], v[3], d[3], db[3];
      tri(i, u, v, d);
      const double w3 = (d[0] * n[0] + d[1] * n[1] + d[2] * n[2]) * (1.0 / 3.0);
      const double wb = weight_bar(u, v);
#pragma unroll
      for (int j = 0; j < 3; ++j) db[j] = 0.5 * (Sb[j] + wb * n[j]);
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const int p = (j + 1) % 3, q = (j + 2) % 3;
        const double tb = cb[j] * w3;
        const double ub = v[p] * db[q] - v[q] * db[p] + tb;
        const double vb = db[p] * u[q] - db[q] * u[p] + tb;
        acc[3 * i + j] += ub;
        acc[3 * i1 + j] += vb;
        pab[j] -= ub + vb;
      }
    }
#pragma unroll
    for (int i = 0; i < kk; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) acc[3 * i + j] += pab[j] * inv;
  }
  if constexpr (K > 0) {
#pragma unroll
    for (int i = 0; i < 3 * K; ++i) out[i] = local[i];
  }
}

template <int DIM>
__global__ void __launch_bounds__(128) k_nadj_face_geom(MeshView m, const double* Ab,
                                                        const double* nbt, const double* xfb,
                                                        double* nodepart) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nf = m.nf;
  const int b = m.fn_ptr[f], e = m.fn_ptr[f + 1];
  double ns[DIM], nb[DIM], xb[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    ns[j] = m.normal[(long)j * nf + f];
    nb[j] = nbt[(long)j * nf + f];
    xb[j] = xfb[(long)j * nf + f];
  }
  double* out = nodepart + (long)b * DIM;
  const int* idx = m.fn_idx + b;
  if constexpr (DIM == 3) {
    if (e - b == 4) face_geom_bar_3d<4>(4, m.nodes, idx, ns, Ab[f], nb, xb, out);
    else face_geom_bar_3d<0>(e - b, m.nodes, idx, ns, Ab[f], nb, xb, out);
  } else {
    const double dx = m.nodes[2L * idx[1]] - m.nodes[2L * idx[0]];
    const double dy = m.nodes[2L * idx[1] + 1] - m.nodes[2L * idx[0] + 1];
    const double sq = dx * dx + dy * dy;
    double xs = 0.0, ys = 0.0;
    if (sq > 0.0) {  // n = (dy, -dx) / A up to the owner-outward sign, A = |(dx, dy)|
      const double ia = 1.0 / sqrt(sq), n0 = dy * ia, n1 = -dx * ia;
      const double sgn = n0 * ns[0] + n1 * ns[1] < 0.0 ? -1.0 : 1.0;
      const double b0 = sgn * nb[0], b1 = sgn * nb[1];
      const double abt = Ab[f] - (b0 * n0 + b1 * n1) * ia;
      xs = -b1 * ia - abt * n1;
      ys = b0 * ia + abt * n0;
    }
    out[0] = 0.5 * xb[0] - xs;
    out[1] = 0.5 * xb[1] - ys;
    out[2] = 0.5 * xb[0] + xs;
    out[3] = 0.5 * xb[1] + ys;
    for (int i = 4; i < 2 * (e - b); ++i) out[i] = 0.0;
  }
}

__global__ void k_nadj_nodes(int nn, int dim, const int* node_ptr, const int* node_ent,
                             const double* nodepart, double* dnodes) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nn) return;
  for (int j = 0; j < dim; ++j) {
    double acc = 0.0;
    for (int i = node_ptr[v]; i < node_ptr[v + 1]; ++i)
      acc += nodepart[(long)node_ent[i] * dim + j];
    dnodes[(long)v * dim + j] = acc;
  }
}

// The pressure part sum_i w_i p_f A n_i of a viscous-only functional on boundary faces: its
// geometry cotangents are subtracted (p_f = the owner pressure, or the outlet value).
template <int DIM, bool TURB>
__global__ void k_nadj_pressure_term(MeshView m, CaseView cv, const double* state,
                                     const double* FLx, double* Fb) {
  using L = Layout<DIM, TURB>;
  const int f = m.nfi + blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const int nf = m.nf;
  const int o = m.owner[f];
  const double pf = bpress(cv, f, cv.fkind[f], state[(long)L::P * m.nc + o]);
  const double A = m.area[f];
  double ab = 0.0;
  for (int i = 0; i < DIM; ++i) {
    const double wi = FLx[(long)i * nf + f];
    ab += wi * pf * m.normal[(long)i * nf + f];
    Fb[(long)(FaceBar<DIM>::N + i) * nf + f] -= wi * pf * A;
  }
  Fb[(long)FaceBar<DIM>::A * nf + f] -= ab;
}

struct NadjBuffers {
  double *Fb, *Cb, *ivb, *wdf, *dpart, *Vb, *Ab, *nbt, *xfb, *xcb, *wcon, *cfA, *cfN, *cfX,
      *nodepart;
};

NadjBuffers nadj_layout(double* p, int dim, long nc, long nf, long ncf, long nfn) {
  NadjBuffers B;
  B.Fb = p; p += (long)(2 + 5 * dim) * nf;  // FaceBar
  B.Cb = p; p += (long)GC_COUNT * nc;
  B.ivb = p; p += nc;
  B.wdf = p; p += nf;
  B.dpart = p; p += 2 * nf;
  B.Vb = p; p += nc;
  B.Ab = p; p += nf;
  B.nbt = p; p += (long)dim * nf;
  B.xfb = p; p += (long)dim * nf;
  B.xcb = p; p += (long)dim * nc;
  B.wcon = p; p += (long)dim * nc;
  B.cfA = p; p += ncf;
  B.cfN = p; p += (long)dim * ncf;
  B.cfX = p; p += (long)dim * ncf;
  B.nodepart = p;
  return B;
}

size_t nadj_doubles(int dim, long nc, long nf, long ncf, long nfn) {
  return (size_t)(2 + 5 * dim) * nf + (size_t)GC_COUNT * nc + 2 * nc + 4 * nf + 2 * dim * nf +
         2 * dim * nc + ncf * (1 + 2 * dim) + (size_t)dim * nfn;
}

int nadj_setup(FvCase* cs, cudaStream_t s) {
  if (cs->nadj) return FV_OK;
  FvMesh* M = cs->mesh;
  const int dim = M->dim;
  const long nc = M->nc, nf = M->nf;
  const long ncf = M->h_cf_ptr[nc];
  std::vector<int> fp(nf + 1);
  FV_CUDA_TRY(cudaMemcpyAsync(fp.data(), M->fn_ptr, sizeof(int) * (nf + 1), cudaMemcpyDeviceToHost, s));
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  const long nfn = fp[nf];
  std::vector<int> fi(nfn);
  FV_CUDA_TRY(cudaMemcpy(fi.data(), M->fn_idx, sizeof(int) * nfn, cudaMemcpyDeviceToHost));
  // node -> entries of fn_idx (ascending)
  std::vector<int> np(M->nn + 1, 0), ne(nfn);
  for (long i = 0; i < nfn; ++i) np[fi[i] + 1]++;
  for (int v = 0; v < M->nn; ++v) np[v + 1] += np[v];
  std::vector<int> fill(np.begin(), np.end() - 1);
  for (long i = 0; i < nfn; ++i) ne[fill[fi[i]]++] = (int)i;
  // face -> cells whose nearest wall face it is
  std::vector<int> wp(nf + 1, 0), wc;
  if (cs->desc.turbulent) {
    std::vector<int> near(nc);
    FV_CUDA_TRY(cudaMemcpy(near.data(), cs->wnear, sizeof(int) * nc, cudaMemcpyDeviceToHost));
    for (long c = 0; c < nc; ++c) wp[near[c] + 1]++;
    for (long f = 0; f < nf; ++f) wp[f + 1] += wp[f];
    wc.assign(nc, 0);
    std::vector<int> wf(wp.begin(), wp.end() - 1);
    for (long c = 0; c < nc; ++c) wc[wf[near[c]]++] = (int)c;
  }
  NodeAdjoint* na = new NodeAdjoint();
  cs->nadj = na;
  FV_CUDA_TRY(cudaMalloc(&na->buf, sizeof(double) * nadj_doubles(dim, nc, nf, ncf, nfn)));
  {
    // gradient reversal: the saved last-iterate cotangent (nfld, dim, nc), the wall-distance
    // numerator (dim, nc) and the sweep buffers of the flow fields
    const int sweeps = std::max(cs->desc.gradient_sweeps, 1);
    const size_t n = (size_t)cs->nfld * dim * nc + (size_t)dim * nc +
                     sweep_doubles(sweeps, cs->nfld, dim, nc, nf);
    FV_CUDA_TRY(cudaMalloc(&na->sweep, sizeof(double) * n));
  }
  if (cs->view.rec_mom || cs->view.rec_sca)  // limxc (dim, nc), limxf (dim, ncf)
    FV_CUDA_TRY(cudaMalloc(&na->rec, sizeof(double) * (size_t)dim * (nc + ncf)));
  FV_CUDA_TRY(cudaMalloc(&na->node_ptr, sizeof(int) * np.size()));
  FV_CUDA_TRY(cudaMalloc(&na->node_ent, sizeof(int) * std::max<long>(nfn, 1)));
  FV_CUDA_TRY(cudaMalloc(&na->wall_ptr, sizeof(int) * wp.size()));
  FV_CUDA_TRY(cudaMalloc(&na->wall_cell, sizeof(int) * std::max<size_t>(wc.size(), 1)));
  FV_CUDA_TRY(cudaMemcpyAsync(na->node_ptr, np.data(), sizeof(int) * np.size(), cudaMemcpyHostToDevice, s));
  FV_CUDA_TRY(cudaMemcpyAsync(na->node_ent, ne.data(), sizeof(int) * nfn, cudaMemcpyHostToDevice, s));
  FV_CUDA_TRY(cudaMemcpyAsync(na->wall_ptr, wp.data(), sizeof(int) * wp.size(), cudaMemcpyHostToDevice, s));
  if (!wc.empty())
    FV_CUDA_TRY(cudaMemcpyAsync(na->wall_cell, wc.data(), sizeof(int) * wc.size(), cudaMemcpyHostToDevice, s));
  FV_CUDA_TRY(cudaStreamSynchronize(s));
  return FV_OK;
}

template <int DIM, bool TURB>
int node_vjp(FvCase* cs, const double* state, const double* W, double* dnodes, cudaStream_t s) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  NodeAdjoint* na0 = cs->nadj;
  const int sweeps = cs->desc.gradient_sweeps;
  const double rel = sweeps >= 1 ? cs->desc.gradient_relaxation : 1.0;
  double* gb_last = na0->sweep;                                  // (NF, DIM, nc)
  double* wd_num = gb_last + (long)NF * DIM * cs->mesh->nc;      // (DIM, nc)
  double* sweep_area = wd_num + (long)DIM * cs->mesh->nc;
  // cotangents of every stage (the gradient's saved before the backward sweeps overwrite it)
  int rc = run_vjp<DIM, TURB>(cs, state, W, nullptr, cs->tmp2, s, sweeps >= 2 ? gb_last : nullptr);
  if (rc != FV_OK) return rc;
  FvMesh* M = cs->mesh;
  const MeshView& m = M->view;
  const CaseView& cv = cs->view;
  const long nc = m.nc, nf = m.nf;
  const long ncf = M->h_cf_ptr[nc];
  NodeAdjoint* na = cs->nadj;
  Work<double> fw = work_layout<double, DIM, TURB>(cs->work, nc, nf, psi_count<DIM, TURB>(cs));
  AdjWork aw = adj_layout<DIM, TURB>(cs);
  NadjBuffers B = nadj_layout(na->buf, DIM, nc, nf, ncf, 0);
  constexpr int TB = 128;
  const int bc = fv_blocks(nc, TB), bf = fv_blocks(nf, TB);
  const long npsi = psi_count<DIM, TURB>(cs);
  double* limxc = na->rec;
  double* limxf = limxc ? limxc + (long)DIM * nc : nullptr;
  if (npsi) {
    aw.psi = fw.psi;
    FV_CUDA_TRY(cudaMemsetAsync(limxc, 0, sizeof(double) * ((size_t)DIM * nc + (size_t)DIM * ncf), s));
  }
  FV_CUDA_TRY(cudaMemsetAsync(B.Cb, 0, sizeof(double) * ((size_t)GC_COUNT * nc + nc), s));  // and ivb
  FV_CUDA_TRY(cudaMemsetAsync(B.Vb, 0, sizeof(double) * nc, s));
  FV_CUDA_TRY(cudaMemsetAsync(B.xfb, 0, sizeof(double) * DIM * nf, s));
  const double irho = 1.0 / cs->desc.rho;
  const Par<Dual> pd{{cs->mu, 0.0}, {cs->inlet_scale, 0.0}, {cs->mu * irho, 0.0}};
  const Par<double> pdd{cs->mu, cs->inlet_scale, cs->mu * irho};
  k_nadj_face<DIM, TURB><<<bf, TB, 0, s>>>(m, cv, state, pdd, fw.G, fw.cl, fw.dco, fw.me, cs->aux,
                                           aw, B.Fb, B.wdf);
  if (aw.FLx && cs->flx_viscous)
    k_nadj_pressure_term<DIM, TURB><<<bf, TB, 0, s>>>(m, cv, state, aw.FLx, B.Fb);
  // Green-Gauss gradients of the fields: the swept sweeps' geometry, then the numerator's
  {
    SweepBufs sb = sweep_layout(sweep_area, std::max(sweeps, 1), NF, DIM, nc, nf);
    if (sweeps >= 2) {
      rc = sweeps_geometry<DIM, NF>(m, sweeps, rel, fw.Bg, gb_last, sb, B.Fb, B.ivb, B.Vb, s);
      if (rc != FV_OK) return rc;
    } else {
      k_nadj_numerator_bar<DIM, NF><<<bc, TB, 0, s>>>(m, aw.Gb, nullptr, rel, sb.nbar);
      k_nadj_grad_cell<DIM, NF><<<bc, TB, 0, s>>>(m, aw.Gb, fw.G, nullptr, rel, B.ivb);
    }
    k_nadj_grad_face<DIM, TURB><<<bf, TB, 0, s>>>(m, cv, state, pdd, sb.nbar, B.Fb);
  }
  k_nadj_dcoeff<<<bc, TB, 0, s>>>(m, fw.dco, aw.dcob, B.Cb);
  if constexpr (TURB) {
    // one block row per seeded input of a wall cell: GC_WD .. GC_WDG + DIM - 1, and the face areas
    k_nadj_closure<DIM><<<dim3(bc, GC_WDG + DIM - GC_WD + 1), TB, 0, s>>>(
        m, cv, state, pd, fw.G, fw.cl, fw.Gwi, aw.clb, aw.Gwib, B.Cb, B.Fb);
    k_nadj_src<DIM><<<dim3(bc, 2), TB, 0, s>>>(m, cv, state, pd, fw.cl, fw.G, fw.Gwi, W, B.Cb);
    // the wall-distance gradient, the same scheme as the fields'
    SweepBufs sd = sweep_layout(sweep_area, std::max(sweeps, 1), 1, DIM, nc, nf);
    const double* yb = B.Cb + (long)GC_WDG * nc;
    if (sweeps >= 2) {
      k_nadj_wd_numerator<DIM><<<bc, TB, 0, s>>>(m, cv, wd_num);
      rc = sweeps_geometry<DIM, 1>(m, sweeps, rel, wd_num, yb, sd, B.Fb, B.ivb, B.Vb, s);
      if (rc != FV_OK) return rc;
    } else {
      k_nadj_numerator_bar<DIM, 1><<<bc, TB, 0, s>>>(m, yb, nullptr, rel, sd.nbar);
      k_nadj_grad_cell<DIM, 1><<<bc, TB, 0, s>>>(m, yb, cv.wdg, nullptr, rel, B.ivb);
    }
    k_nadj_wdg_face<DIM><<<bf, TB, 0, s>>>(m, cv, sd.nbar, B.Fb, B.dpart);
    k_nadj_wdg_cell<DIM><<<bc, TB, 0, s>>>(m, cv, B.dpart, B.Cb);
  }
  if (npsi && (cv.lim_km > 0.0 || cv.lim_ks > 0.0))
    k_nadj_limiter<DIM, TURB><<<bc, TB, 0, s>>>(m, state, fw.G, cv.lim_km, cv.lim_ks, aw.psib,
                                                B.Vb, limxc, limxf, ncf);
  k_nadj_cell_chain<DIM, TURB><<<bc, TB, 0, s>>>(m, cv, B.Cb, B.ivb, B.wdf, cs->wnear, B.Vb, B.xcb,
                                                 B.wcon);
  if (npsi) k_nadj_add<<<fv_blocks((long)DIM * nc, 256), 256, 0, s>>>((long)DIM * nc, limxc, B.xcb);
  if constexpr (TURB)
    k_nadj_wall_face<DIM><<<bf, TB, 0, s>>>(m, na->wall_ptr, na->wall_cell, B.wcon, B.xfb);
  k_nadj_factors<DIM><<<bf, TB, 0, s>>>(m, B.Fb, B.xfb);
  k_nadj_xc_gather<DIM><<<bc, TB, 0, s>>>(m, B.Fb + (long)FaceBar<DIM>::XO * nf, B.xcb);
  k_nadj_cell_geom<DIM><<<bc, TB, 0, s>>>(m, B.Vb, B.xcb, B.cfA, B.cfN, B.cfX, ncf);
  k_nadj_cf_gather<DIM><<<bf, TB, 0, s>>>(m, B.Fb, B.cfA, B.cfN, B.cfX, npsi ? limxf : nullptr, ncf,
                                          B.Ab, B.nbt, B.xfb);
  k_nadj_face_geom<DIM><<<bf, TB, 0, s>>>(m, B.Ab, B.nbt, B.xfb, B.nodepart);
  k_nadj_nodes<<<fv_blocks(M->nn, 256), 256, 0, s>>>(M->nn, DIM, na->node_ptr, na->node_ent,
                                                    B.nodepart, dnodes);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

}  // namespace

int fv_case_node_vjp(FvCase* cs, const double* state, const double* w, double* dnodes,
                     cudaStream_t s) {
  if (cs->wd_external) {
    fv_set_error("fv_node_vjp: the wall distance was set by the caller (fv_case_set_wall_distance), "
                 "so its dependence on the nodes is unknown here");
    return FV_ERR_ARG;
  }
  int rc = nadj_setup(cs, s);
  if (rc != FV_OK) return rc;
  const int dim = cs->mesh->dim;
  const bool turb = cs->desc.turbulent != 0;
  if (dim == 2)
    return turb ? node_vjp<2, true>(cs, state, w, dnodes, s) : node_vjp<2, false>(cs, state, w, dnodes, s);
  return turb ? node_vjp<3, true>(cs, state, w, dnodes, s) : node_vjp<3, false>(cs, state, w, dnodes, s);
}

void fv_node_adjoint_free(FvCase* cs) {
  NodeAdjoint* na = cs->nadj;
  if (!na) return;
  cudaFree(na->buf);
  cudaFree(na->node_ptr);
  cudaFree(na->node_ent);
  cudaFree(na->wall_ptr);
  cudaFree(na->wall_cell);
  cudaFree(na->sweep);
  cudaFree(na->rec);
  delete na;
  cs->nadj = nullptr;
}

// ------------------------------------------------------------------------ face-flux functionals
// J = sum_f sum_q w_qf FL_q(f), optionally less the pressure part sum_i w_if p_f A_f n_if on
// boundary faces (the viscous, "wall shear" force): the outlet mass flux (w = 1 on the
// continuity flux of the outlet faces) and the wall shear force (w = 1 on a momentum component of
// the wall faces) of the 3D channel's adjoint objectives.  Value, dJ/dstate (the state adjoint
// with w as an extra face-flux cotangent), the parameter partials (forward tangents of the face
// fluxes) and dJ/dnodes (the mesh-coordinate adjoint with the same extra cotangent).
namespace {

constexpr int kFnBlocks = 304;

__global__ void k_face_in(int nf, int nfld, const int* face_old, const double* w_ref,
                          double* w_int) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= nf) return;
  const int r = face_old[f];
  for (int q = 0; q < nfld; ++q) w_int[(long)q * nf + f] = w_ref[(long)q * nf + r];
}

template <class T>
__device__ __forceinline__ double part_of(const T& x, bool tangent);
template <>
__device__ __forceinline__ double part_of<double>(const double& x, bool) { return x; }
template <>
__device__ __forceinline__ double part_of<Dual>(const Dual& x, bool tangent) {
  return tangent ? x.d : x.v;
}

template <int DIM, bool TURB, class T>
__global__ void __launch_bounds__(256) k_functional_partial(MeshView m, CaseView cv,
                                                            const double* state, const double* w,
                                                            const T* FL, int viscous, int tangent,
                                                            double* part) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  __shared__ double red[256];
  const int nf = m.nf;
  double acc = 0.0;
  for (long f = (long)blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += (long)gridDim.x * blockDim.x) {
    double a = 0.0;
    for (int q = 0; q < NF; ++q) {
      const double wq = w[(long)q * nf + f];
      if (wq != 0.0) a += wq * part_of(FL[(long)q * nf + f], tangent != 0);
    }
    if (viscous && !tangent && f >= m.nfi) {
      const int o = m.owner[f];
      const double pf = bpress(cv, (int)f, cv.fkind[f], state[(long)L::P * m.nc + o]);
      for (int i = 0; i < DIM; ++i)
        a -= w[(long)i * nf + f] * pf * m.area[f] * m.normal[(long)i * nf + f];
    }
    acc += a;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_functional_final(int nparts, const double* part, double* out) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double acc = 0.0;
  for (int i = 0; i < nparts; ++i) acc += part[i];
  *out = acc;
}

// d(pressure part)/d(owner pressure) on boundary faces whose pressure is the owner's.
template <int DIM, bool TURB>
__global__ void k_functional_pressure_state(MeshView m, CaseView cv, const double* w,
                                            double* dstate) {
  using L = Layout<DIM, TURB>;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nf = m.nf;
  double acc = 0.0;
  for (int i = m.cf_ptr[c]; i < m.cf_ptr[c + 1]; ++i) {
    const int f = (int)(m.cf_face[i] & ~FV_NB_BIT);
    const signed char kind = cv.fkind[f];
    if (f < m.nfi || kind < 0 || kind > 2) continue;
    for (int j = 0; j < DIM; ++j) acc += w[(long)j * nf + f] * m.area[f] * m.normal[(long)j * nf + f];
  }
  dstate[(long)L::P * m.nc + c] -= acc;
}

template <int DIM, bool TURB>
int face_functional(FvCase* cs, const double* state, const double* wref, int viscous,
                    double* value, double* dstate, double* dparams, double* dnodes,
                    cudaStream_t s) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  const MeshView& m = cs->mesh->view;
  const CaseView& cv = cs->view;
  const long nc = m.nc, nf = m.nf, n = (long)NF * nc;
  if (!cs->flx) FV_CUDA_TRY(cudaMalloc(&cs->flx, sizeof(double) * ((size_t)NF * nf + n)));
  if (!cs->red) FV_CUDA_TRY(cudaMalloc(&cs->red, sizeof(double) * kFnBlocks));
  double* zeros = cs->flx + (long)NF * nf;
  FV_CUDA_TRY(cudaMemsetAsync(zeros, 0, sizeof(double) * n, s));
  k_face_in<<<fv_blocks(nf, 256), 256, 0, s>>>((int)nf, NF, cs->mesh->face_old, wref, cs->flx);
  // value
  int rc = fv_case_run(cs, state, nullptr, FV_TAN_NONE, cs->tmp, nullptr, s);
  if (rc != FV_OK) return rc;
  {
    Work<double> fw = work_layout<double, DIM, TURB>(cs->work, nc, nf, psi_count<DIM, TURB>(cs));
    k_functional_partial<DIM, TURB, double><<<kFnBlocks, 256, 0, s>>>(m, cv, state, cs->flx, fw.FL,
                                                                      viscous, 0, cs->red);
    k_functional_final<<<1, 32, 0, s>>>(kFnBlocks, cs->red, value);
  }
  // parameter partials at fixed state
  if (dparams) {
    const int kinds[2] = {FV_TAN_MU, FV_TAN_INLET};
    for (int i = 0; i < 2; ++i) {
      rc = fv_case_run(cs, state, nullptr, kinds[i], nullptr, cs->tmp2, s);
      if (rc != FV_OK) return rc;
      cs->fwd_valid = 0;  // the workspace is about to hold a dual-number pass
      Work<Dual> dw = work_layout<Dual, DIM, TURB>(cs->work, nc, nf, psi_count<DIM, TURB>(cs));
      k_functional_partial<DIM, TURB, Dual><<<kFnBlocks, 256, 0, s>>>(m, cv, state, cs->flx, dw.FL,
                                                                      0, 1, cs->red);
      k_functional_final<<<1, 32, 0, s>>>(kFnBlocks, cs->red, dparams + i);
    }
  }
  // state partial: the adjoint with no residual cotangent and w on the face fluxes
  cs->flx_active = true;
  cs->flx_viscous = viscous != 0;
  rc = run_vjp<DIM, TURB>(cs, state, zeros, nullptr, dstate, s);
  if (rc == FV_OK && viscous)
    k_functional_pressure_state<DIM, TURB><<<fv_blocks(nc, 128), 128, 0, s>>>(m, cv, cs->flx, dstate);
  if (rc == FV_OK && dnodes) rc = fv_case_node_vjp(cs, state, zeros, dnodes, s);
  cs->flx_active = false;
  cs->flx_viscous = false;
  if (rc != FV_OK) return rc;
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

}  // namespace

int fv_case_face_functional(FvCase* cs, const double* state, const double* weights_ref,
                            int viscous_only, double* value, double* dstate, double* dparams,
                            double* dnodes, cudaStream_t s) {
  const int dim = cs->mesh->dim;
  const bool turb = cs->desc.turbulent != 0;
  if (dim == 2)
    return turb ? face_functional<2, true>(cs, state, weights_ref, viscous_only, value, dstate, dparams, dnodes, s)
                : face_functional<2, false>(cs, state, weights_ref, viscous_only, value, dstate, dparams, dnodes, s);
  return turb ? face_functional<3, true>(cs, state, weights_ref, viscous_only, value, dstate, dparams, dnodes, s)
              : face_functional<3, false>(cs, state, weights_ref, viscous_only, value, dstate, dparams, dnodes, s);
}
