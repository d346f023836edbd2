// The frozen (reach-1) block Jacobian J_direct in fp64, by the derivatives written out.  Included by
// residual.cu (shares its device helpers); assemble.inc.cuh holds the fp32 form and says what is
// frozen.
//
// With the gradients, the closure and d held, the flux of field q through an interior face is
//   mdot up_q + (pressure part) - conductance (phi_N - phi_P + const),
// mdot linear in the two cells' velocities and pressures.  A face's derivative blocks are therefore
// up_q times one row vector, a diagonal and (momentum rows) a pressure column: about 20 products a
// block row, where differentiating the flux code once per unknown evaluated it 2 NF = 12 times (all
// of it fp64 issue: 5.2 of 6.7 ms on the 80 x 63 x 51 SST channel) and kept 2 NF^2 doubles per
// face between the face and the cell pass (0.46 GB written and read).
//   k_jac_coef  face  mass flux, its pressure derivative, the fields' conductances (NCO rows of nf)
//   k_jac_src   cell  2 x 2 derivatives of the k / omega source rows (off the wall written out; the
//                     wall functions by seeded dual numbers)
//   k_jac_rows  one thread per block row and field: the field's scalar rows of the cell's blocks,
//               the diagonal block accumulated in registers over the cell's faces, each other block
//               written once, nothing zeroed beforehand.  A thread per cell would write 8 bytes
//               per 288; adjacent rows make a warp's stores contiguous.

// Where a factor of a flux or of a source is not finite, every derivative of that row through it is
// NaN, as it is with dual numbers (a zero tangent times it): the probes and this assembly then agree
// on which blocks a state such as omega = 0 spoils.
__device__ __forceinline__ bool finite_bits(double x) {  // no fp64 comparison
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

template <int DIM, bool TURB>
struct JacCoef {
  static constexpr int N = 3 + (TURB ? 2 : 0);  // mdot, d mdot / d p_owner, momentum, k, omega
};

template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_jac_coef(MeshView m, CaseView cv, const double* state,
                                                  Par<double> par, const double* G,
                                                  const double* cl, const double* dco,
                                                  const double* me, double* co) {
  using L = Layout<DIM, TURB>;
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nf) return;
  const long nc = m.nc, nf = m.nf;
  const int o = m.owner[f];
  const double A = m.area[f], rho = cv.rho, rA = rho * A;
  const double mo = mu_eff<double, TURB>(par, cv, rho, cl, m.nc, o);
  if (f < m.nfi) {
    const int n = m.nb[f];
    const double g = m.g[f], dpn = m.dpn[f], dnn = m.dnn[f];
    double gd = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j)
      gd += lerp(G[((long)L::P * DIM + j) * nc + o], G[((long)L::P * DIM + j) * nc + n], g) *
            m.dvec[(long)j * nf + f];
    const double mp = rA * (m.nn2[f] * lerp(dco[o], dco[n], g)) * m.inv_nd[f];
    co[f] = me[f] - mp * ((state[(long)L::P * nc + n] - state[(long)L::P * nc + o]) - gd);
    co[nf + f] = mp;
    co[2 * nf + f] =
        conductance(mo, mu_eff<double, TURB>(par, cv, rho, cl, m.nc, n), A, dpn, dnn);
    if (TURB) {
#pragma unroll
      for (int s = 0; s < 2; ++s)
        co[(3L + s) * nf + f] =
            conductance(cl[(4L + s) * nc + o], cl[(4L + s) * nc + n], A, dpn, dnn);
    }
    return;
  }
  const signed char kind = cv.fkind[f];
  double mdot = 0.0, mp = 0.0;
  if (kind == 2) {
#pragma unroll
    for (int j = 0; j < DIM; ++j)
      mdot += (cv.fvel[(long)j * nf + f] * par.iscale) * m.normal[(long)j * nf + f];
    mdot *= rA;
  } else if (kind == 3) {
    double un = 0.0, interp = 0.0;
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const double nj = m.normal[(long)j * nf + f];
      un += state[(long)j * nc + o] * nj;
      interp += G[((long)L::P * DIM + j) * nc + o] * nj;
    }
    const double dh = m.nn2[f] * dco[o];
    mdot = rA * (un - dh * ((cv.fp[f] - state[(long)L::P * nc + o]) * m.inv_nd[f] - interp));
    mp = rA * dh * m.inv_nd[f];
  }
  co[f] = mdot;
  co[nf + f] = mp;
  double gb = mo;
  const bool wall = TURB && cv.swall[f];
  if (TURB && (kind == 0 || kind == 1))
    gb = par.mu + rho * (wall ? nut_wall(par.nu, cv.wd[o], state[(long)L::K * nc + o]) : 0.0);
  const double Ai = A * m.inv_dpn[f];
  co[2 * nf + f] = gb * Ai;
  if (TURB) {
    const double gk = cl[4L * nc + o];
    co[3 * nf + f] =
        (wall ? (1.0 - wall_weight(par.nu, cv.wd[o], state[(long)L::K * nc + o])) * gk : gk) * Ai;
    co[4 * nf + f] = cl[5L * nc + o] * Ai;
  }
}

// Values as dual numbers without a tangent.
struct FrozenDual {
  const double* p;
  __device__ __forceinline__ Dual operator[](long i) const { return {p[i], 0.0}; }
};

// The closure of the cells where its inputs are not finite or 1 / omega is not, again by dual
// numbers: their max / min keep a NaN that the plain ones may drop.
template <int DIM>
__global__ void __launch_bounds__(128) k_jac_closure_nan(MeshView m, CaseView cv,
                                                         const double* state, Par<double> par,
                                                         const double* G, double* cl,
                                                         double* Gwi) {
  using L = Layout<DIM, true>;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const long nc = m.nc;
  const double w = state[(long)L::W * nc + c];
  bool ok = finite_bits(w) && (__double2hiint(w) & 0x7ff00000) != 0 &&
            finite_bits(state[(long)L::K * nc + c]) && finite_bits(cl[c]);
#pragma unroll
  for (int j = 0; j < 2 * DIM; ++j) ok = ok && finite_bits(G[((long)L::K * DIM + j) * nc + c]);
  if (ok) return;
  const Par<Dual> pd{{par.mu, 0.0}, {par.iscale, 0.0}, {par.nu, 0.0}};
  Dual out[7], gw[DIM];
  closure_cell<Dual, DIM>(m, cv, Src<Dual>{state, nullptr}, pd, FrozenDual{G}, c, GeoPlain{}, out,
                          gw);
#pragma unroll
  for (int i = 0; i < 7; ++i) cl[i * nc + c] = out[i].v;
#pragma unroll
  for (int j = 0; j < DIM; ++j) Gwi[j * nc + c] = gw[j].v;
}

// src = d(k row, omega row) / d(k, omega) of the cell's source terms: rows kk, kw, wk, ww of nc.
template <int DIM>
__global__ void __launch_bounds__(128) k_jac_src(MeshView m, CaseView cv, const double* state,
                                                 Par<double> par, const double* G,
                                                 const double* cl, const double* Gwi,
                                                 double* src) {
  using L = Layout<DIM, true>;
  const int c = stage_cell<double>(m, cv);
  if (c >= m.nc) return;
  const long nc = m.nc;
  if (cv.wcell[c]) {
    const Par<Dual> pd{{par.mu, 0.0}, {par.iscale, 0.0}, {par.nu, 0.0}};
#pragma unroll 1
    for (int r = 0; r < 2; ++r) {
      const SeedSrc<Dual> st{state, (r ? (long)L::W : (long)L::K) * nc + c};
      Dual rk{0.0, 0.0}, rw{0.0, 0.0};
      sst_rows<Dual, DIM>(m, cv, st, pd, FrozenDual{cl}, FrozenDual{G}, FrozenDual{Gwi}, c, rk, rw);
      src[r * nc + c] = rk.d;
      src[(2 + r) * nc + c] = rw.d;
    }
    return;
  }
  // sst_rows: the production limiter and its cap are minima (a tie takes half the derivative)
  const double V = m.vol[c], k = state[(long)L::K * nc + c], w = state[(long)L::W * nc + c];
  const double S2 = cl[c] * cl[c], F1 = cl[nc + c], nut = cl[2 * nc + c];
  constexpr double PB = PROD_RATIO * BETA_STAR;
  const double kp = pos(k), limit = PB * kp * w, t1 = nut * S2;
  const double lk = PB * dpos(k) * w, lw = PB * kp;  // the limit's derivatives
  const double sel = t1 > limit ? 1.0 : (t1 < limit ? 0.0 : 0.5);
  src[c] = V * (BETA_STAR * w - sel * lk);
  src[nc + c] = V * (BETA_STAR * k - sel * lw);
  double dkw = 0.0;
#pragma unroll
  for (int j = 0; j < DIM; ++j)
    dkw += G[((long)L::K * DIM + j) * nc + c] * Gwi[(long)j * nc + c];
  const double inv = 1.0 / (nut > NUT_FLOOR ? nut : NUT_FLOOR), cap = limit * inv;
  const double alpha = ALPHA_2 + F1 * (ALPHA_1 - ALPHA_2), beta = BETA_2 + F1 * (BETA_1 - BETA_2);
  const double cut = alpha * inv * (S2 > cap ? 1.0 : (S2 < cap ? 0.0 : 0.5));
  const double iw = 1.0 / w, cross = (2.0 * SIGMA_W2) * (1.0 - F1) * dkw * iw;
  const double bad = __longlong_as_double(0x7ff8000000000000LL);
  const bool ok = finite_bits(nut) && finite_bits(S2);
  if (!ok) src[c] = src[nc + c] = bad;
  const bool okw = ok && finite_bits(cross);
  src[2 * nc + c] = okw ? -V * (cut * lk) : bad;
  src[3 * nc + c] = okw ? V * (2.0 * beta * w - cut * lw + cross * iw) : bad;
}

// -x where `neg`, by the sign bit (no fp64 instruction).
__device__ __forceinline__ double flip(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? 0x80000000 : 0), __double2loint(x));
}
template <int NF>
__device__ __forceinline__ void store_row(double* p, const double (&x)[NF], bool vec) {
  if (NF % 2 == 0 && vec) {
#pragma unroll
    for (int r = 0; r + 1 < NF; r += 2) *reinterpret_cast<double2*>(p + r) = make_double2(x[r], x[r + 1]);
  } else {
#pragma unroll
    for (int r = 0; r < NF; ++r) p[r] = x[r];
  }
}

template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_jac_rows(MeshView m, CaseView cv, const double* state,
                                                  Par<double> par, const double* G,
                                                  const double* cl, const double* psi,
                                                  const double* co, const double* src,
                                                  const int* indptr, const int* indices,
                                                  double* values, bool vec) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  const long t = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long)m.nc * NF) return;
  const int q = (int)(t % NF), at = (int)(t / NF);
  const int c = cv.sched != nullptr ? __ldg(cv.sched + at) : at;
  const long nc = m.nc, nf = m.nf;
  const GeoPlain gv{};
  const int bp = indptr[c], be = indptr[c + 1];
  const bool mom = q < DIM, cont = q == L::P;
  // rows without the face sum: the pinned pressure row, the omega wall-cell row
  bool skip = cont && c == cv.pin;
  if constexpr (TURB) skip = skip || (q == L::W && cv.wcell[c] != 0);
  const double rho = cv.rho, irho = cv.irho;
  const double* rec = mom ? (cv.rec_mom ? psi : nullptr) : (cv.rec_sca ? psi : nullptr);
  const int adv = mom ? q : q - 1;  // index among the advected fields
  // the diagonal block's row; its own field's column (one fp64 addition a face, not one for every
  // field a warp's rows hold) is added at the end
  double dg[NF], dq = 0.0;
#pragma unroll
  for (int r = 0; r < NF; ++r) dg[r] = 0.0;
  unsigned long long written = 0;  // slots of the block row, the first 64
  double* row = values + ((long)bp * NF + q) * NF;
  const double zero[NF] = {};
  if (be - bp > 64)
    for (int p = 0; p < be - bp; ++p) store_row<NF>(row + (long)p * NF * NF, zero, vec);
  auto spoil = [](double (&x)[NF]) {
#pragma unroll
    for (int r = 0; r < NF; ++r) x[r] = __longlong_as_double(0x7ff8000000000000LL);
  };
  const int fb = m.cf_ptr[c], fe = skip ? fb : m.cf_ptr[c + 1];
  for (int i = fb; i < fe; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    const bool isnb = (ent & FV_NB_BIT) != 0;
    const double A = m.area[f], mdot = co[f];
    const bool out = mdot >= 0.0;
    double nrm[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) nrm[j] = m.normal[(long)j * nf + f];
    if (f < m.nfi) {
      const int o = m.owner[f], n = m.nb[f];
      const double g = m.g[f], h = 1.0 - g;
      const double ws = isnb ? g : h, wo = isnb ? h : g;  // this cell's weight, the other's
      double up = isnb ? -1.0 : 1.0;  // d flux / d mdot, with the sum's sign
      double cond = 0.0, flux = 0.0;
      if (!cont) {
        const int cu = out ? o : n;
        up = upwind_rec<double, DIM>(m, G, rec, adv, q, f, cu, state[(long)q * nc + cu], gv);
        flux = mdot;
        if (!mom) {
          up *= irho;
          flux *= irho;
        }
        up = flip(up, isnb);
        flux = flip(flux, isnb);
        cond = co[(mom ? 2L : (long)q - DIM + 2) * nf + f];
      }
      double oth[NF];
#pragma unroll
      for (int r = 0; r < NF; ++r) oth[r] = 0.0;
      const double ur = up * (rho * A);
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        const double x = ur * nrm[j];
        dg[j] = fma(ws, x, dg[j]);
        oth[j] = wo * x;
      }
      const double x = flip(up * co[nf + f], isnb);
      double ps = x, po = -x;
      double nq = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) nq = q == j ? nrm[j] : nq;
      if (mom) {
        const double y = flip(A * nq, isnb);
        ps = fma(ws, y, ps);
        po = fma(wo, y, po);
      }
      dg[L::P] += ps;
      oth[L::P] = po;
      const bool mine = out != isnb;  // this cell is the upwind one
      const double ds = mine ? cond + flux : cond, dn = mine ? -cond : flux - cond;
      if (!cont) {
        dq += ds;
        double own = oth[0];
#pragma unroll
        for (int r = 1; r < NF; ++r) own = r == q ? oth[r] : own;
        own += dn;
#pragma unroll
        for (int r = 0; r < NF; ++r) oth[r] = r == q ? own : oth[r];
      }
      if (!finite_bits(co[nf + f]) ||
          (!cont && !(finite_bits(mdot) && finite_bits(cond) && finite_bits(up)))) {
        spoil(dg);
        spoil(oth);
      }
      const int other = isnb ? o : n;
      int slot = -1;
      for (int p = bp; p < be; ++p)
        if (indices[p] == other) {
          slot = p - bp;
          break;
        }
      if (slot >= 0) {
        double* d = row + (long)slot * NF * NF;
        const bool add = slot >= 64 || be - bp > 64 || ((written >> slot) & 1ull);
        if (add) {  // a second face between the two cells
#pragma unroll
          for (int r = 0; r < NF; ++r) oth[r] += d[r];
        }
        store_row<NF>(d, oth, vec);
        if (slot < 64) written |= 1ull << slot;
      }
      continue;
    }
    const int o = c;
    const signed char kind = cv.fkind[f];
    double up = 1.0;
    if (mom) {
      const double uo = state[(long)q * nc + o];
      const double bu = bvel(cv, m.nf, f, q, kind, uo, par);
      up = out ? upwind_rec<double, DIM>(m, G, rec, adv, q, f, o, uo, gv) : bu;
      const bool free = kind == 3;  // the boundary velocity is the cell's
      double d = free ? 0.0 : co[2 * nf + f];
      if (out || free) d += mdot;
      double nq = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) nq = q == j ? nrm[j] : nq;
      dq += d;
      if (kind >= 0 && kind != 3) dg[L::P] += A * nq;
      if constexpr (TURB) {
        if ((kind == 0 || kind == 1) && cv.swall[f]) {
          const Dual nw = nut_wall(Dual{par.nu, 0.0}, cv.wd[o], Dual{state[(long)L::K * nc + o], 1.0});
          double cp = 0.0;
#pragma unroll
          for (int j = 0; j < DIM; ++j)
            cp += G[((long)q * DIM + j) * nc + o] * m.tP[(long)j * nf + f];
          dg[L::K] -= (rho * nw.d) * (A * m.inv_dpn[f]) * (bu - uo - cp);
        }
      }
    } else if (TURB && !cont) {
      const bool is_k = q == L::K;
      const signed char sk = is_k ? cv.kkind[f] : cv.wkind[f];
      const double phi = state[(long)q * nc + o];
      double cp = 0.0;
#pragma unroll
      for (int j = 0; j < DIM; ++j) cp += G[((long)q * DIM + j) * nc + o] * m.tP[(long)j * nf + f];
      const double bphi = bscalar(sk, is_k ? cv.kval[f] : cv.wval[f], phi, cp);
      up = irho * (out ? upwind_rec<double, DIM>(m, G, rec, adv, q, f, o, phi, gv) : bphi);
      const bool free = sk == 1;  // zero gradient
      double d = free ? 0.0 : co[(is_k ? 3L : 4L) * nf + f];
      if (out || free) d += mdot * irho;
      if constexpr (TURB) {
        if (is_k && cv.swall[f]) {
          const Dual wt = wall_weight(Dual{par.nu, 0.0}, cv.wd[o], Dual{phi, 1.0});
          d += wt.d * cl[4L * nc + o] * (A * m.inv_dpn[f]) * (bphi - phi - cp);
        }
      }
      dq += d;
    }
    if (!finite_bits(co[nf + f]) ||
        (!cont && !(finite_bits(mdot) && finite_bits(up) &&
                    finite_bits(co[(mom ? 2L : (long)q - DIM + 2) * nf + f]))))
      spoil(dg);
    if (kind == 3) {  // the outlet's mass flux follows the cell's velocity and pressure
      const double ur = up * (rho * A);
#pragma unroll
      for (int j = 0; j < DIM; ++j) dg[j] = fma(ur, nrm[j], dg[j]);
      dg[L::P] = fma(up, co[nf + f], dg[L::P]);
    }
  }
#pragma unroll
  for (int r = 0; r < NF; ++r)
    if (r == q) dg[r] += dq;
  if (cont && c == cv.pin) dg[L::P] = 1.0;
  if constexpr (TURB) {
    if (q >= L::K) {
      const double* s = src + 2L * (q - L::K) * nc + c;
      dg[L::K] += s[0];
      dg[L::W] += s[nc];
    }
  }
  for (int p = 0; p < be - bp; ++p) {
    double* d = row + (long)p * NF * NF;
    if (indices[bp + p] == c) store_row<NF>(d, dg, vec);
    else if (p < 64 && be - bp <= 64 && !((written >> p) & 1ull)) store_row<NF>(d, zero, vec);
  }
}

// The fp64 blocks of J_direct; `src` holds 4 nc doubles.
// Measured (80 x 63 x 51 SST channel): 6.73 -> 1.09 ms, 0.6 of it k_jac_rows.
template <int DIM, bool TURB>
int assemble_frozen64(FvCase* cs, const double* state, const int* indptr, const int* indices,
                      double* values, double* src, cudaStream_t s) {
  const MeshView& m = cs->mesh->view;
  const CaseView& cv = cs->view;
  const long nc = m.nc, nf = m.nf;
  constexpr int NF = Layout<DIM, TURB>::NFLD;
  static_assert(JacCoef<DIM, TURB>::N <= NF, "the coefficients use the flux rows of the workspace");
  cs->fwd_valid = 0;  // the workspace is about to hold this pass
  const long npsi = psi_count<DIM, TURB>(cs);
  Work<double> w = work_layout<double, DIM, TURB>(cs->work, nc, nf, npsi);
  const Src<double> st{state};
  const Par<double> par{cs->mu, cs->inlet_scale, cs->mu * (1.0 / cs->desc.rho)};
  constexpr int TB = 128;
  const int bc = fv_blocks(nc, TB), bf = fv_blocks(nf, TB);
  gradient_stage<double, DIM, TURB>(cs, st, par, w, s);
  if constexpr (TURB) {
    k_closure<double, DIM><<<bc, TB, 0, s>>>(m, cv, st, par, w.G, w.cl, w.Gwi);
    k_jac_closure_nan<DIM><<<bc, TB, 0, s>>>(m, cv, state, par, w.G, w.cl, w.Gwi);
  }
  k_apcoef<double, DIM, TURB><<<bf, TB, 0, s>>>(m, cv, st, par, w.G, w.cl, w.acown, w.acnb, w.me);
  k_dcoeff<double><<<bc, TB, 0, s>>>(m, w.acown, w.acnb, w.dco);
  if (npsi)
    k_limiter<double, DIM, TURB><<<bc, TB, 0, s>>>(m, st, w.G, cv.lim_km, cv.lim_ks, w.psi);
  k_jac_coef<DIM, TURB><<<bf, TB, 0, s>>>(m, cv, state, par, w.G, w.cl, w.dco, w.me, w.FL);
  if constexpr (TURB)
    k_jac_src<DIM><<<bc, TB, 0, s>>>(m, cv, state, par, w.G, w.cl, w.Gwi, src);
  k_jac_rows<DIM, TURB><<<fv_blocks(nc * NF, TB), TB, 0, s>>>(
      m, cv, state, par, w.G, w.cl, npsi ? w.psi : nullptr, w.FL, src, indptr, indices, values,
      (uintptr_t)values % 16 == 0);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}
