// The finite-volume residual pipeline (laminar Rhie-Chow momentum/continuity, optionally coupled
// to k-omega SST), written once as templates over the scalar type:
//   T = double -> R(state)
//   T = Dual   -> R(state) and J v (forward-mode tangent through the same arithmetic)
//
// Pipeline (each stage one kernel; face stages run one thread per face in the internal face
// order, cell stages one thread per cell summing its faces in ascending order, so every
// face-to-cell accumulation is deterministic without atomics):
//   k_grad      cell  compact Green-Gauss gradients of every field
//               (aquaflux/schemes/gradient.py:129-153 with the leading-order boundary values of
//               aquaflux/flow/momentum.py:445-469 / discretization/residual.py:252-291)
//   k_closure   cell  SST closure: strain with the wall-cell log-layer blend, imposed wall-cell
//               omega gradient, F1, nu_t, wall shear rate (aquaflux/turbulence/transport.py:369-579)
//   k_apcoef    face  momentum-diagonal face coefficients: flux-continuous viscous conductance +
//               upwind part of the lagged mass-flux estimate, boundary closures
//               (aquaflux/flow/momentum.py:556-693, aquaflux/flow/rhie_chow.py:81-271)
//   k_dcoeff    cell  a_P and d = V / a_P
//   k_flux      face  Rhie-Chow mass flux (rhie_chow.py:274-353, flow/boundary.py:381-435), face
//               pressure, momentum diffusion + pressure + upwind advection fluxes, k / omega
//               advection + diffusion fluxes (discretization/diffusion.py:163-199,
//               advection.py:99-187, turbulence/transport.py:581-718)
//   k_sum       cell  conservative face-to-cell sums, pressure pin, SST sources and the omega
//               wall-cell fixation (turbulence/sources.py:60-412, fixed_value.py:124-158)
#include <cooperative_groups.h>
#include <type_traits>

#include "geom.cuh"
#include "internal.cuh"

namespace {

// The stages of a pass are launched with programmatic dependent launch: a stage's blocks may be
// placed before the stage before has ended, and wait for it before their first read.  On small
// meshes a pass is a dozen kernels of 2-6 us with 1-3 us between them (64 x 64 cavity, residual +
// VJP: 79 -> 61 us).  The next stage is let in at once where its blocks find SMs of their own
// beside this one's, or where there are many waves of them; between, blocks placed around a stage
// that still runs would crowd the SMs it left free (10,000-cell JVP: 41 -> 43 us), so the next
// stage comes as this one's blocks end.
__device__ __forceinline__ void stage_begin() {
  const unsigned threads = gridDim.x * blockDim.x;
  if (threads <= 8192u || threads >= 262144u)
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class K, class... Args>
void stage(K kern, int grid, int block, cudaStream_t s, Args... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, args...);
}

// SST constants, aquaflux/turbulence/sst.py:69-82 and sources.py:52-57.
constexpr double A1 = 0.31, BETA_STAR = 0.09, ALPHA_1 = 5.0 / 9.0, BETA_1 = 3.0 / 40.0;
constexpr double SIGMA_K1 = 0.85, SIGMA_W1 = 0.5, ALPHA_2 = 0.44, BETA_2 = 0.0828;
constexpr double SIGMA_K2 = 1.0, SIGMA_W2 = 0.856, KAPPA = 0.41, E_WALL = 9.8;
constexpr double CROSS_FLOOR = 1e-10, PROD_RATIO = 10.0, NUT_FLOOR = 1e-30;

struct SstConst {
  double bs4;   // beta_star ** 0.25
  double ylam;  // laminar-sublayer y* (fixed point of y = ln(E y) / kappa, 10 sweeps from 11)
};
__constant__ SstConst c_sst;

// fp32 passes (T = DualF) read the fp32 mirrors of the geometry and of the state, so that their
// arithmetic stays off the fp64 pipe; GS<T> is the scalar type of the geometry a pass reads.
template <class T>
struct IsF32 : std::false_type {};
template <>
struct IsF32<DualF> : std::true_type {};
template <class T>
using GS = typename std::conditional<IsF32<T>::value, float, double>::type;
// The cell a thread of a cell-centric stage evaluates.  With the case's warp-coherent order the
// threads walk the cells grouped by the pattern of their face lists (owner / neighbour / boundary
// kind at each position), so the 32 lanes of a warp take the same branches; without it, the
// natural order.  A cell's arithmetic does not depend on which thread runs it, so both orders give
// bitwise the same result.  The fp32 dual-number passes keep the natural order: they are not
// bound by the floating-point issue rate that divergence wastes, and the indirection costs them.
template <class T = double>
__device__ __forceinline__ int stage_cell(const MeshView& m, const CaseView& cv) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if constexpr (IsF32<T>::value) return t;
  else return (cv.sched != nullptr && t < m.nc) ? __ldg(cv.sched + t) : t;
}

template <class T>
__device__ __forceinline__ GS<T> gx(const double* d, const float* f, long i) {
  if constexpr (IsF32<T>::value) return f[i];
  else return d[i];
}
template <class T>
__device__ __forceinline__ GS<T> rho_of(const CaseView& cv) {
  if constexpr (IsF32<T>::value) return cv.f_rho;
  else return cv.rho;
}

template <class T>
struct Src;
template <>
struct Src<double> {
  const double* v;
  __device__ __forceinline__ double operator()(long i) const { return v[i]; }
};
template <>
struct Src<Dual> {
  const double* v;
  const double* t;  // may be null: zero tangent
  __device__ __forceinline__ Dual operator()(long i) const { return {v[i], t ? t[i] : 0.0}; }
};
template <>
struct Src<DualF> {
  const float* v;  // the fp32 copy of the state
  const float* t;  // of the tangent; may be null: zero tangent
  __device__ __forceinline__ DualF operator()(long i) const { return {v[i], t ? t[i] : 0.0f}; }
};

template <class T>
struct Par {
  T mu;      // molecular dynamic viscosity
  T iscale;  // inlet-velocity factor
  T nu;      // molecular kinematic viscosity mu / rho
};

template <class T>
__device__ __forceinline__ void put(double* r, double* t, long i, const T& x);
template <>
__device__ __forceinline__ void put<double>(double* r, double*, long i, const double& x) {
  r[i] = x;
}
template <>
__device__ __forceinline__ void put<Dual>(double* r, double* t, long i, const Dual& x) {
  if (r) r[i] = x.v;
  t[i] = x.d;
}
template <>
__device__ __forceinline__ void put<DualF>(double* r, double* t, long i, const DualF& x) {
  if (r) r[i] = x.v;
  t[i] = x.d;
}

// ---------------------------------------------------------------- SST wall functions
// aquaflux/turbulence/boundary.py:45-589.
template <class T, class D>
__device__ __forceinline__ T y_star(T nu, D d, T k) {
  return c_sst.bs4 * safe_sqrt(pos(k)) * d / nu;
}
template <class T, class D>
__device__ __forceinline__ T wall_weight(T nu, D d, T k) {
  T r = y_star(nu, d, k) / c_sst.ylam;
  T r2 = r * r;
  return fv_tanh(r2 * r2);
}
template <class T, class D>
__device__ __forceinline__ T log_shear(D d, T k) {
  return c_sst.bs4 * safe_sqrt(pos(k)) / (KAPPA * d);
}
template <class T, class D>
__device__ __forceinline__ T omega_wall(T nu, D d, T k) {
  T vis = 6.0 * nu / (BETA_1 * (d * d));
  T lg = safe_sqrt(pos(k)) / (c_sst.bs4 * KAPPA * d);
  T m = fv_max(vis, lg);
  T ra = vis / m, rb = lg / m;
  T bt = val(rb) > 0.0 ? rb * rb : cst(0.0, rb);
  return m * fv_sqrt(ra * ra + bt);
}
template <class T, class D>
__device__ __forceinline__ T nut_wall(T nu, D d, T k) {
  T ys = y_star(nu, d, k);
  T arg = E_WALL * fv_max(ys, cst(c_sst.ylam, ys));
  T ratio = ys * KAPPA / fv_log(arg) - 1.0;
  return val(ys) > c_sst.ylam ? nu * ratio : cst(0.0, ys);
}
// d omega_wall / d d and d omega_wall / d k in closed form (the reference obtains them with
// jax.grad, boundary.py:585-589); written in T so the JVP differentiates them once more.
template <class T, class D>
__device__ __forceinline__ void omega_wall_partials(T nu, D d, T k, T* dwdd, T* dwdk) {
  T vis = 6.0 * nu / (BETA_1 * (d * d));
  T kp = pos(k);
  T sk = safe_sqrt(kp);
  double c = c_sst.bs4 * KAPPA;
  T lg = sk / (c * d);
  T w = omega_wall(nu, d, k);
  T dvis_dd = -2.0 * vis / d;
  T dlog_dd = -lg / d;
  T dsk = val(kp) > 0.0 ? 0.5 / sk : cst(0.0, sk);
  T dlog_dk = dsk / (c * d);
  T a = vis / w, b = lg / w;
  *dwdd = a * dvis_dd + b * dlog_dd;
  *dwdk = b * dlog_dk;
}

// ---------------------------------------------------------------- boundary values
// Leading-order flow boundary velocity / pressure (aquaflux/flow/boundary.py:43-120, 278-446).
template <class T>
__device__ __forceinline__ T bvel(const CaseView& cv, int nf, int f, int j, signed char kind,
                                  T u_owner, const Par<T>& par) {
  if (kind == 1) return cst(cv.fvel[(long)j * nf + f], u_owner);
  if (kind == 2) return cv.fvel[(long)j * nf + f] * par.iscale;
  if (kind == 3) return u_owner;
  return cst(0.0, u_owner);
}
template <class T>
__device__ __forceinline__ T bpress(const CaseView& cv, int f, signed char kind, T p_owner) {
  if (kind == 3) return cst(cv.fp[f], p_owner);
  if (kind >= 0) return p_owner;
  return cst(0.0, p_owner);
}
// Scalar closure Dirichlet / ZeroGradient (aquaflux/boundary/conditions.py:111-160); `corr` is
// the tangential correction (zero for the leading-order values used by the gradient).
template <class T>
__device__ __forceinline__ T bscalar(signed char kind, double value, T phi_owner, T corr) {
  if (kind == 0) return cst(value, phi_owner);
  if (kind == 1) return phi_owner + corr;
  return cst(0.0, phi_owner);
}

// ---------------------------------------------------------------- geometry accessors
// The face and cell formulas read the mesh geometry through an accessor: GeoPlain returns the
// stored doubles; GeoSeed returns dual numbers whose tangent is 1 on one geometric input (one
// component, on every face / cell or on one of them), which lets the mesh-coordinate adjoint
// differentiate the closure, source and limiter formulas by local forward mode where it does not
// write the reverse out.
enum GeoFace { GF_AREA = 0 };
enum GeoCell { GC_VOL = 0, GC_WD = 1, GC_INV_WD = 2, GC_INV_WD2 = 3, GC_WDG = 4, GC_COUNT = 7 };
// Centroid seeds (not stored per-factor cotangent rows): face centroid component j of the seeded
// face (fcomp = GF_XF + j), cell centroid component j of the seeded cell (ccomp = GC_XC + j).
enum GeoCentroid { GF_XF = 40, GC_XC = 50 };

struct GeoPlain {
  __device__ __forceinline__ double area(const MeshView& m, int f) const { return m.area[f]; }
  __device__ __forceinline__ double normal(const MeshView& m, int j, int f) const {
    return m.normal[(long)j * m.nf + f];
  }
  __device__ __forceinline__ double tP(const MeshView& m, int j, int f) const {
    return m.tP[(long)j * m.nf + f];
  }
  __device__ __forceinline__ double tN(const MeshView& m, int j, int f) const {
    return m.tN[(long)j * m.nf + f];
  }
  __device__ __forceinline__ double g(const MeshView& m, int f) const { return m.g[f]; }
  __device__ __forceinline__ double dvec(const MeshView& m, int j, int f) const {
    return m.dvec[(long)j * m.nf + f];
  }
  __device__ __forceinline__ double skew(const MeshView& m, int j, int f) const {
    return m.skew[(long)j * m.nf + f];
  }
  __device__ __forceinline__ double nn2(const MeshView& m, int f) const { return m.nn2[f]; }
  __device__ __forceinline__ double inv_nd(const MeshView& m, int f) const { return m.inv_nd[f]; }
  __device__ __forceinline__ double inv_dpn(const MeshView& m, int f) const {
    return m.inv_dpn[f];
  }
  __device__ __forceinline__ double dpn(const MeshView& m, int f) const { return m.dpn[f]; }
  __device__ __forceinline__ double dnn(const MeshView& m, int f) const { return m.dnn[f]; }
  __device__ __forceinline__ double ns(const MeshView& m, int jq, int f) const {
    return m.ns[(long)jq * m.nf + f];
  }
  __device__ __forceinline__ double vol(const MeshView& m, int c) const { return m.vol[c]; }
  __device__ __forceinline__ double wd(const CaseView& cv, int c) const { return cv.wd[c]; }
  __device__ __forceinline__ double inv_wd(const CaseView& cv, int c) const {
    return cv.inv_wd[c];
  }
  __device__ __forceinline__ double inv_wd2(const CaseView& cv, int c) const {
    return cv.inv_wd2[c];
  }
  __device__ __forceinline__ double wdg(const CaseView& cv, int nc, int j, int c) const {
    return cv.wdg[(long)j * nc + c];
  }
  __device__ __forceinline__ double xf(const MeshView& m, int j, int f) const {
    return m.xf[(long)j * m.nf + f];
  }
  __device__ __forceinline__ double xc(const MeshView& m, int j, int c) const {
    return m.xc[(long)j * m.nc + c];
  }
};

// The fp32 mirror (fp32 passes).
struct GeoPlainF {
  __device__ __forceinline__ float area(const MeshView& m, int f) const { return m.f_area[f]; }
  __device__ __forceinline__ float normal(const MeshView& m, int j, int f) const {
    return m.f_normal[(long)j * m.nf + f];
  }
  __device__ __forceinline__ float tP(const MeshView& m, int j, int f) const {
    return m.f_tP[(long)j * m.nf + f];
  }
  __device__ __forceinline__ float tN(const MeshView& m, int j, int f) const {
    return m.f_tN[(long)j * m.nf + f];
  }
  __device__ __forceinline__ float g(const MeshView& m, int f) const { return m.f_g[f]; }
  __device__ __forceinline__ float dvec(const MeshView& m, int j, int f) const {
    return m.f_dvec[(long)j * m.nf + f];
  }
  __device__ __forceinline__ float skew(const MeshView& m, int j, int f) const {
    return m.f_skew[(long)j * m.nf + f];
  }
  __device__ __forceinline__ float nn2(const MeshView& m, int f) const { return m.f_nn2[f]; }
  __device__ __forceinline__ float inv_nd(const MeshView& m, int f) const { return m.f_inv_nd[f]; }
  __device__ __forceinline__ float inv_dpn(const MeshView& m, int f) const {
    return m.f_inv_dpn[f];
  }
  __device__ __forceinline__ float dpn(const MeshView& m, int f) const { return m.f_dpn[f]; }
  __device__ __forceinline__ float dnn(const MeshView& m, int f) const { return m.f_dnn[f]; }
  __device__ __forceinline__ float ns(const MeshView& m, int jq, int f) const {
    return m.f_ns[(long)jq * m.nf + f];
  }
  __device__ __forceinline__ float vol(const MeshView& m, int c) const { return m.f_vol[c]; }
  __device__ __forceinline__ float wd(const CaseView& cv, int c) const { return cv.f_wd[c]; }
  __device__ __forceinline__ float inv_wd(const CaseView& cv, int c) const {
    return cv.f_inv_wd[c];
  }
  __device__ __forceinline__ float inv_wd2(const CaseView& cv, int c) const {
    return cv.f_inv_wd2[c];
  }
  __device__ __forceinline__ float wdg(const CaseView& cv, int nc, int j, int c) const {
    return cv.f_wdg[(long)j * nc + c];
  }
  __device__ __forceinline__ float xf(const MeshView& m, int j, int f) const {
    return m.f_xf[(long)j * m.nf + f];
  }
  __device__ __forceinline__ float xc(const MeshView& m, int j, int c) const {
    return m.f_xc[(long)j * m.nc + c];
  }
};

// The plain accessor of a pass's scalar type.
template <class T>
struct GeoOf {
  using type = GeoPlain;
};
template <>
struct GeoOf<DualF> {
  using type = GeoPlainF;
};

struct GeoSeed {
  int fcomp;  // seeded face component (GeoFace), -1 for none
  int ccomp;  // seeded cell component (GeoCell), -1 for none
  int face;   // the one seeded face, -1 for every face
  int cell;   // the one seeded cell, -1 for every cell
  __device__ __forceinline__ double hf(int id, int f) const {
    return (fcomp == id && (face < 0 || face == f)) ? 1.0 : 0.0;
  }
  __device__ __forceinline__ double hc(int id, int c) const {
    return (ccomp == id && (cell < 0 || cell == c)) ? 1.0 : 0.0;
  }
  __device__ __forceinline__ Dual area(const MeshView& m, int f) const {
    return {m.area[f], hf(GF_AREA, f)};
  }
  __device__ __forceinline__ Dual vol(const MeshView& m, int c) const {
    return {m.vol[c], hc(GC_VOL, c)};
  }
  __device__ __forceinline__ Dual wd(const CaseView& cv, int c) const {
    return {cv.wd[c], hc(GC_WD, c)};
  }
  __device__ __forceinline__ Dual inv_wd(const CaseView& cv, int c) const {
    return {cv.inv_wd[c], hc(GC_INV_WD, c)};
  }
  __device__ __forceinline__ Dual inv_wd2(const CaseView& cv, int c) const {
    return {cv.inv_wd2[c], hc(GC_INV_WD2, c)};
  }
  __device__ __forceinline__ Dual wdg(const CaseView& cv, int nc, int j, int c) const {
    return {cv.wdg[(long)j * nc + c], hc(GC_WDG + j, c)};
  }
  __device__ __forceinline__ Dual xf(const MeshView& m, int j, int f) const {
    return {m.xf[(long)j * m.nf + f], hf(GF_XF + j, f)};
  }
  __device__ __forceinline__ Dual xc(const MeshView& m, int j, int c) const {
    return {m.xc[(long)j * m.nc + c], hc(GC_XC + j, c)};
  }
};

template <int DIM, bool TURB>
struct Layout {
  static constexpr int NFLD = DIM + 1 + (TURB ? 2 : 0);
  static constexpr int P = DIM, K = DIM + 1, W = DIM + 2;
};

// ---------------------------------------------------------------- workspace
// Forward workspace of one residual evaluation (elements of type T), carved from FvCase::work.
template <class T>
struct Work {
  T* G;      // (NF, DIM, nc) gradients
  T* cl;     // (7, nc) strain, F1, nu_t, wall shear rate, k diffusivity, omega diffusivity, F2
  T* Gwi;    // (DIM, nc) omega gradient with the wall-cell value imposed
  T* acown;  // (nf) momentum-diagonal coefficient, owner side
  T* acnb;   // (nf) neighbour side
  T* dco;    // (nc) d = V / a_P
  T* psi;    // (NA, nc) slope limiter of each advected field (limited upwind only)
  T* me;     // (nf) lagged mass-flux estimate (rho u)_f . n A
  T* FL;     // (NF, nf) face fluxes (also the face scratch of the gradient sweeps)
  T* Bg;     // (NF, DIM, nc) corrected Green-Gauss right-hand side B phi (swept cases only)
  T* Galt;   // (NF, DIM, nc) second iterate buffer of the sweeps (swept cases only)
};
// Number of advected fields (the momentum components, and k and omega) and the limiter storage a
// case needs (limited linear upwind only).
template <int DIM, bool TURB>
__host__ __device__ constexpr int n_advected() {
  return DIM + (TURB ? 2 : 0);
}
template <int DIM, bool TURB>
long psi_count(const FvCase* cs) {
  return (cs->view.rec_mom || cs->view.rec_sca) ? (long)n_advected<DIM, TURB>() * cs->mesh->nc : 0;
}

template <class T, int DIM, bool TURB>
Work<T> work_layout(void* base, long nc, long nf, long npsi = 0) {
  constexpr int NF = Layout<DIM, TURB>::NFLD;
  T* p = (T*)base;
  Work<T> w;
  w.G = p; p += (long)NF * DIM * nc;
  w.cl = p; p += 7 * nc;
  w.Gwi = p; p += DIM * nc;
  w.acown = p; p += nf;
  w.acnb = p; p += nf;
  w.dco = p; p += nc;
  w.psi = p; p += npsi;
  w.me = p; p += nf;
  w.FL = p; p += (long)NF * nf;
  w.Bg = p; p += (long)NF * DIM * nc;
  w.Galt = p;
  return w;
}

// ---------------------------------------------------------------- k_grad
// G = rel * (B phi / V) with B phi the compact Green-Gauss numerator; Bg (may be null) receives
// B phi itself (the right-hand side of the corrected scheme's sweeps).  rel = 1 and Bg = null is
// the compact scheme.
template <class T, int DIM, bool TURB>
__device__ __forceinline__ void k_grad_at(const int c, MeshView m, CaseView cv, Src<T> st, Par<T> par, T* G,
                                              T* Bg, double rel) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  T phic[NF];
#pragma unroll
  for (int q = 0; q < NF; ++q) phic[q] = st((long)q * nc + c);
  T acc[NF][DIM];
#pragma unroll
  for (int q = 0; q < NF; ++q)
#pragma unroll
    for (int j = 0; j < DIM; ++j) acc[q][j] = cst(0.0, phic[0]);
  // fp64 with SST: the cell's own values leave the face sum (own = sum S w_c is one vector for all
  // fields; 3D: 28 fp64 instructions a side, not 34: 128^3 818 -> 775 us).  With four fields or
  // fewer it saves nothing (64 laminar 2D channels 0.3 % slower).
  constexpr bool kOwn = TURB && !IsF32<T>::value;
  GS<T> own[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) own[j] = GS<T>(0);
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    const bool isnb = (ent & FV_NB_BIT) != 0;
    const GS<T> af = gx<T>(m.area, m.f_area, f);
    const GS<T> A = isnb ? -af : af;  // the neighbour takes -S_f phi_f
    GS<T> S[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) S[j] = gx<T>(m.normal, m.f_normal, (long)j * nf + f) * A;
    T phif[NF];
    if (f < m.nfi) {
      const GS<T> g = gx<T>(m.g, m.f_g, f);
      const int other = isnb ? m.owner[f] : m.nb[f];
      if constexpr (kOwn) {
        const GS<T> h = GS<T>(1) - g, wo = isnb ? h : g, wc = isnb ? g : h;
#pragma unroll
        for (int j = 0; j < DIM; ++j) {
          own[j] += S[j] * wc;
          S[j] = S[j] * wo;
        }
      }
      // owner value first: the operands are selected, not the interpolation (one code path for
      // both sides of a face, no if-converted duplicate of the dual-number arithmetic)
#pragma unroll
      for (int q = 0; q < NF; ++q) {
        const T po = st((long)q * nc + other);
        if constexpr (kOwn) phif[q] = po;
        else phif[q] = lerp(isnb ? po : phic[q], isnb ? phic[q] : po, g);
      }
    } else {
      const signed char kind = cv.fkind[f];
#pragma unroll
      for (int j = 0; j < DIM; ++j) phif[j] = bvel(cv, nf, f, j, kind, phic[j], par);
      phif[L::P] = bpress(cv, f, kind, phic[L::P]);
      if (TURB) {
        T z = cst(0.0, phic[0]);
        phif[L::K] = bscalar(cv.kkind[f], cv.kval[f], phic[L::K], z);
        phif[L::W] = bscalar(cv.wkind[f], cv.wval[f], phic[L::W], z);
      }
    }
#pragma unroll
    for (int q = 0; q < NF; ++q)
#pragma unroll
      for (int j = 0; j < DIM; ++j) acc[q][j] += S[j] * phif[q];
  }
  if constexpr (kOwn) {
#pragma unroll
    for (int q = 0; q < NF; ++q)
#pragma unroll
      for (int j = 0; j < DIM; ++j) acc[q][j] += own[j] * phic[q];
  }
  const GS<T> inv = gx<T>(m.inv_vol, m.f_inv_vol, c);
  if (Bg) {
#pragma unroll
    for (int q = 0; q < NF; ++q)
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        Bg[((long)q * DIM + j) * nc + c] = acc[q][j];
        G[((long)q * DIM + j) * nc + c] = rel * (acc[q][j] * inv);
      }
  } else if (rel != 1.0) {
#pragma unroll
    for (int q = 0; q < NF; ++q)
#pragma unroll
      for (int j = 0; j < DIM; ++j) G[((long)q * DIM + j) * nc + c] = rel * (acc[q][j] * inv);
  } else {
#pragma unroll
    for (int q = 0; q < NF; ++q)
#pragma unroll
      for (int j = 0; j < DIM; ++j) G[((long)q * DIM + j) * nc + c] = acc[q][j] * inv;
  }
}

template <class T, int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_grad(MeshView m, CaseView cv, Src<T> st, Par<T> par, T* G,
                                              T* Bg, double rel) {
  stage_begin();
  k_grad_at<T, DIM, TURB>(stage_cell<T>(m, cv), m, cv, st, par, G, Bg, rel);
}

// ---------------------------------------------------------------- corrected Green-Gauss sweeps
// CorrectedGreenGauss (aquaflux/schemes/gradient.py:1122-1337) by SweptGradientSolve
// (gradient.py:618-705): A_g G = V G - C(G), C(G)_c = sum over the interior faces of c of
// +-S_f w_f, w_f = (1 - g) skew . G_P + g skew . G_N; every sweep after the peeled first one is
// X <- X + rel (B phi - A_g X) / V.  Gradients are field-major (NQ, DIM, nc).
//
// w_f for every field (face pass, interior faces).
template <class T, int DIM, int NQ>
__global__ void __launch_bounds__(128) k_gg_skew(MeshView m, const T* X, T* w) {
  stage_begin();
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.nfi) return;
  const int nc = m.nc, nf = m.nf;
  const int o = m.owner[f], n = m.nb[f];
  const GS<T> g = gx<T>(m.g, m.f_g, f);
  GS<T> sk[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) sk[j] = gx<T>(m.skew, m.f_skew, (long)j * nf + f);
  GS<T> ko[DIM], kn[DIM];  // the blend's weights folded into the skew vector, once for all fields
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    ko[j] = (GS<T>(1) - g) * sk[j];
    kn[j] = g * sk[j];
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    T wq = ko[0] * X[((long)q * DIM) * nc + o] + kn[0] * X[((long)q * DIM) * nc + n];
#pragma unroll
    for (int j = 1; j < DIM; ++j) {
      wq = wq + ko[j] * X[((long)q * DIM + j) * nc + o];
      wq = wq + kn[j] * X[((long)q * DIM + j) * nc + n];
    }
    w[(long)q * nf + f] = wq;
  }
}

// One sweep (cell pass): Xn = X + rel (Bg - (V X - C(X))) / V, as X + rel ((Bg + C(X)) / V - X):
// for rel = 1, the usual one, X itself drops out.  The sums are multiply-adds from zero.  fp64 issue
// bounds it (dual numbers, 5 fields in 2D: 280 -> 120 fp64 instructions a cell; 130,000 cells,
// three sweeps 345 -> 165 us, k_gg_skew 142 -> 105 us).
template <class T, int DIM, int NQ>
__global__ void __launch_bounds__(128) k_gg_sweep(MeshView m, const T* Bg, const T* X, const T* w,
                                                  double rel, T* Xn) {
  stage_begin();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  T corr[NQ][DIM];
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int j = 0; j < DIM; ++j) corr[q][j] = T{};
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    if (f >= m.nfi) continue;  // the correction vanishes on boundary faces
    const GS<T> af = gx<T>(m.area, m.f_area, f);
    const GS<T> A = (ent & FV_NB_BIT) ? -af : af;
    GS<T> S[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) S[j] = gx<T>(m.normal, m.f_normal, (long)j * nf + f) * A;
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const T wq = w[(long)q * nf + f];
#pragma unroll
      for (int j = 0; j < DIM; ++j) corr[q][j] = corr[q][j] + S[j] * wq;
    }
  }
  const GS<T> inv = gx<T>(m.inv_vol, m.f_inv_vol, c);
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const long k = ((long)q * DIM + j) * nc + c;
      T y = (Bg[k] + corr[q][j]) * inv;
      if (rel != 1.0) {
        const T x = X[k];
        y = x + rel * (y - x);
      }
      Xn[k] = y;
    }
}

// The swept gradients of NQ fields: on entry G0 holds rel * B phi / V and Bg holds B phi; the
// iterates alternate between G0 and Galt so that the last one lands in G (= G0 or Galt, chosen by
// the caller from the parity of the sweep count).
template <class T, int DIM, int NQ>
void gg_sweeps(const MeshView& m, int sweeps, double rel, const T* Bg, T* G0, T* Galt, T* wface,
               cudaStream_t s) {
  constexpr int TB = 128;
  const int bc = fv_blocks(m.nc, TB), bfi = fv_blocks(m.nfi > 0 ? m.nfi : 1, TB);
  T* cur = G0;
  T* nxt = Galt;
  for (int it = 1; it < sweeps; ++it) {
    if (m.nfi > 0) stage(k_gg_skew<T, DIM, NQ>, bfi, TB, s, m, cur, wface);
    stage(k_gg_sweep<T, DIM, NQ>, bc, TB, s, m, Bg, cur, wface, rel, nxt);
    T* t = cur;
    cur = nxt;
    nxt = t;
  }
}

// ---------------------------------------------------------------- k_closure (SST)
// 2 s_ij s_ij of the strain rate s = sym grad u, each pair of off-diagonal entries once (10 fp64
// instructions in 3D, 28 entry by entry).
template <class T, int DIM>
__device__ __forceinline__ T strain2(const T (&gu)[DIM][DIM]) {
  T diag = cst(0.0, gu[0][0]), off = diag;
#pragma unroll
  for (int i = 0; i < DIM; ++i) {
    diag += gu[i][i] * gu[i][i];
#pragma unroll
    for (int j = i + 1; j < DIM; ++j) {
      const T x = gu[i][j] + gu[j][i];
      off += x * x;
    }
  }
  return 2.0 * diag + off;
}

// The closure of cell c: out = (S, F1, nu_t, wall shear rate, k diffusivity, omega diffusivity,
// F2), gw = the omega gradient with the wall-cell value imposed.
template <class T, int DIM, class S_, class GV, class GP>
__device__ __forceinline__ void closure_cell(const MeshView& m, const CaseView& cv, const S_& st,
                                             const Par<T>& par, const GP& G, int c, const GV& gv,
                                             T* out, T* gw) {
  using L = Layout<DIM, true>;
  using GT = decltype(gv.area(m, 0));
  const int nc = m.nc, nf = m.nf;
  T gu[DIM][DIM];
#pragma unroll
  for (int i = 0; i < DIM; ++i)
#pragma unroll
    for (int j = 0; j < DIM; ++j) gu[i][j] = G[((long)i * DIM + j) * nc + c];
  T S;
  if constexpr (!IsF32<T>::value) {
    S = safe_sqrt(strain2<T, DIM>(gu));
  } else {
    T sum = cst(0.0, gu[0][0]);
#pragma unroll
    for (int i = 0; i < DIM; ++i)
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        T sij = 0.5 * (gu[i][j] + gu[j][i]);
        sum += sij * sij;
      }
    S = safe_sqrt(2.0 * sum);
  }
  const T k = st((long)L::K * nc + c);
  const T w = st((long)L::W * nc + c);
  const T nu = par.nu;
  const GT d = gv.wd(cv, c), id = gv.inv_wd(cv, c), id2 = gv.inv_wd2(cv, c);
  T gk[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    gk[j] = G[((long)L::K * DIM + j) * nc + c];
    gw[j] = G[((long)L::W * DIM + j) * nc + c];
  }
  T shear = cst(0.0, k);
  if (cv.wcell[c]) {
    T wgt = wall_weight(nu, d, k);
    S = (1.0 - wgt) * S + wgt * log_shear(d, k);
    T dwdd, dwdk;
    omega_wall_partials(nu, d, k, &dwdd, &dwdk);
#pragma unroll
    for (int j = 0; j < DIM; ++j) gw[j] = gv.wdg(cv, nc, j, c) * dwdd + gk[j] * dwdk;
    T num = cst(0.0, k);
    GT den{};
    T u[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) u[j] = st((long)j * nc + c);
    const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
    for (int i = b; i < e; ++i) {
      const int f = (int)(m.cf_face[i] & ~FV_NB_BIT);
      if (f < m.nfi || !cv.swall[f]) continue;
      const signed char kind = cv.fkind[f];
      T s2 = cst(0.0, k);
#pragma unroll
      for (int j = 0; j < DIM; ++j) {
        T sl = u[j] - bvel(cv, nf, f, j, kind, u[j], par);
        s2 += sl * sl;
      }
      const GT af = gv.area(m, f);
      num += safe_sqrt(s2) * af;
      den += af;
    }
    shear = num * (id / den);
  }
  // F1 (sst.py:166-202) and the eddy viscosity with F2 (sst.py:152-164, 204-239)
  const T kp = pos(k);
  const T iw = 1.0 / w;
  T dot_kw = gk[0] * gw[0];
#pragma unroll
  for (int j = 1; j < DIM; ++j) dot_kw += gk[j] * gw[j];
  const T cd = fv_max((2.0 * SIGMA_W2) * dot_kw * iw, cst(CROSS_FLOOR, w));
  const T sk = safe_sqrt(kp);
  const T vt = (500.0 * id2) * nu * iw;
  const T c1 = sk * iw * (id / BETA_STAR);
  const T arg1 = fv_min(fv_max(c1, vt), (4.0 * SIGMA_W2 * id2) * kp / cd);
  const T a1sq = arg1 * arg1;
  const T F1 = fv_tanh(a1sq * a1sq);
  const T arg2 = fv_max(2.0 * c1, vt);
  const T F2 = fv_tanh(arg2 * arg2);
  const T nut = A1 * kp / fv_max(A1 * w, S * F2);
  out[0] = S;
  out[1] = F1;
  out[2] = nut;
  out[3] = shear;
  out[4] = nu + (SIGMA_K2 + F1 * (SIGMA_K1 - SIGMA_K2)) * nut;
  out[5] = nu + (SIGMA_W2 + F1 * (SIGMA_W1 - SIGMA_W2)) * nut;
  out[6] = F2;
}

template <class T, int DIM>
__device__ __forceinline__ void k_closure_at(const int c, MeshView m, CaseView cv, Src<T> st, Par<T> par,
                                                 const T* G, T* cl, T* Gwi) {
  if (c >= m.nc) return;
  const int nc = m.nc;
  T out[7], gw[DIM];
  closure_cell<T, DIM>(m, cv, st, par, G, c, typename GeoOf<T>::type{}, out, gw);
#pragma unroll
  for (int i = 0; i < 7; ++i) cl[(long)i * nc + c] = out[i];
#pragma unroll
  for (int j = 0; j < DIM; ++j) Gwi[(long)j * nc + c] = gw[j];
}

template <class T, int DIM>
__global__ void __launch_bounds__(128) k_closure(MeshView m, CaseView cv, Src<T> st, Par<T> par,
                                                 const T* G, T* cl, T* Gwi) {
  stage_begin();
  k_closure_at<T, DIM>(stage_cell<T>(m, cv), m, cv, st, par, G, cl, Gwi);
}

// effective dynamic viscosity mu + rho nu_t (aquaflux/flow/momentum.py:357-368)
// molecular viscosity of cell c: the case constant, or a per-cell field (laminar batched
// instances) whose tangent under the viscosity seed is the constant's
__device__ __forceinline__ double mu_at(const Par<double>& par, const CaseView& cv, int c) {
  return cv.mu_cell ? cv.mu_cell[c] : par.mu;
}
__device__ __forceinline__ Dual mu_at(const Par<Dual>& par, const CaseView& cv, int c) {
  return cv.mu_cell ? Dual{cv.mu_cell[c], par.mu.d} : par.mu;
}
__device__ __forceinline__ DualF mu_at(const Par<DualF>& par, const CaseView& cv, int c) {
  return cv.mu_cell ? DualF{cv.f_mu_cell[c], par.mu.d} : par.mu;
}
template <class T, bool TURB, class CP>
__device__ __forceinline__ T mu_eff(const Par<T>& par, const CaseView& cv, GS<T> rho, const CP& cl,
                                    int nc, int c) {
  if (TURB) return par.mu + rho * cl[2L * nc + c];
  return mu_at(par, cv, c);
}

// lagged advective momentum flux (rho u)_f . n with the skew-corrected face value
// (aquaflux/flow/rhie_chow.py:220-271): rho (sum_j n_j u_j,f + sum_jq n_j skew_q (grad u)_jq,f)
template <class T, int DIM, bool TURB, class S, class GP, class GV, class GT>
__device__ __forceinline__ T mom_normal(const MeshView& m, const S& st, const GP& G, GS<T> rho,
                                        int f, int o, int n, GT g, const GV& gv) {
  const int nc = m.nc;
  if constexpr (IsF32<T>::value) {
    T mn = cst(0.0, st(o));
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      mn += gv.normal(m, j, f) * lerp(st((long)j * nc + o), st((long)j * nc + n), g);
#pragma unroll
      for (int q = 0; q < DIM; ++q)
        mn += gv.ns(m, j * DIM + q, f) *
              lerp(G[((long)j * DIM + q) * nc + o], G[((long)j * DIM + q) * nc + n], g);
    }
    return rho * mn;
  }
  // fp64: each side's sum, then one blend of the two (3D: 26 fp64 instructions for 36)
  T mo = gv.normal(m, 0, f) * st(o), mn = gv.normal(m, 0, f) * st(n);
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    if (j > 0) {
      mo += gv.normal(m, j, f) * st((long)j * nc + o);
      mn += gv.normal(m, j, f) * st((long)j * nc + n);
    }
#pragma unroll
    for (int q = 0; q < DIM; ++q) {
      mo += gv.ns(m, j * DIM + q, f) * G[((long)j * DIM + q) * nc + o];
      mn += gv.ns(m, j * DIM + q, f) * G[((long)j * DIM + q) * nc + n];
    }
  }
  return rho * lerp(mo, mn, g);
}

// flux-continuous conductance g_o A / (dpn - g_o / g_n dnn), one division
// (aquaflux/discretization/diffusion.py:85-134)
template <class T, class GT>
__device__ __forceinline__ T conductance(T go, T gn, GT A, GT dpn, GT dnn) {
  return go * gn * A / (dpn * gn - go * dnn);
}

// The conductance c = g_o g_n A / den, den = dpn g_n - g_o dnn, of a flux stage, and its derivatives
// in g_o and g_n, d c / d g_o = A dpn (g_n / den)^2 and d c / d g_n = -A dnn (g_o / den)^2: two
// products each behind the ratios, where c's own form costs five.
template <class T>
struct Conduct {
  T c, ro, rn;  // ro = g_o / den, rn = g_n / den
  double ao, an;
  template <class GT>
  __device__ __forceinline__ Conduct(const T& go, const T& gn, GT A, GT dpn, GT dnn) {
    const T iden = 1.0 / (dpn * gn - go * dnn);
    if constexpr (IsF32<T>::value) {
      c = go * gn * A * iden;
    } else {
      rn = gn * iden;
      c = go * rn * A;
      if constexpr (std::is_same<T, double>::value) {
        ro = go * iden;
        ao = A * dpn;
        an = A * dnn;
      }
    }
  }
  __device__ __forceinline__ double d_owner() const { return ao * rn * rn; }
  __device__ __forceinline__ double d_neighbour() const { return -(an * ro * ro); }
};

// ---------------------------------------------------------------- slope limiter
// VenkatakrishnanLimiter.limit (aquaflux/schemes/limiter.py:78-117) of one field at cell c:
// psi = clip(min over the cell's faces of psi_face, 0, 1), psi_face from the unlimited increment
// dm = grad . (x_f - x_c) (regularised away from 0) and the headroom to the extrema over the cell
// and its face neighbours, eps^2 = V K^3.  phi(cell) and grad(j) read the field (either may carry
// a tangent).
template <class T, int DIM, class PhiFn, class GradFn, class GV = typename GeoOf<T>::type>
__device__ __forceinline__ T limiter_cell(const MeshView& m, int c, double K, const PhiFn& phi,
                                          const GradFn& grad, const GV& gv = GV{}) {
  const int nc = m.nc, nf = m.nf;
  const T pc = phi(c);
  T pmax = pc, pmin = pc;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    if (f >= m.nfi) continue;
    const T po = phi((ent & FV_NB_BIT) ? m.owner[f] : m.nb[f]);
    pmax = fv_max(pmax, po);
    pmin = fv_min(pmin, po);
  }
  using GT = decltype(gv.vol(m, 0));
  using KT = typename std::conditional<std::is_same<GT, float>::value, float, double>::type;
  const GT e2 = gv.vol(m, c) * KT(K * K * K);
  T psi = cst(1.0, pc);
  for (int i = b; i < e; ++i) {
    const int f = (int)(m.cf_face[i] & ~FV_NB_BIT);
    T dm = grad(0) * (gv.xf(m, 0, f) - gv.xc(m, 0, c));
#pragma unroll
    for (int j = 1; j < DIM; ++j) dm = dm + grad(j) * (gv.xf(m, j, f) - gv.xc(m, j, c));
    const double sign = val(dm) >= 0.0 ? 1.0 : -1.0;
    dm = sign * (fv_abs(dm) + 1e-12);
    const T head = val(dm) > 0.0 ? pmax - pc : pmin - pc;
    const T num = (head * head + e2) * dm + 2.0 * (dm * dm) * head;
    const T den = (head * head + 2.0 * (dm * dm) + head * dm + e2) * dm;
    const T pf = num / den;
    psi = i == b ? pf : fv_min(psi, pf);
  }
  return fv_min(fv_max(psi, cst(0.0, psi)), cst(1.0, psi));
}

// Field index of advected field a: the momentum components, then k and omega.
template <int DIM, bool TURB>
__device__ __forceinline__ int advected_field(int a) {
  return a < DIM ? a : (a == DIM ? Layout<DIM, TURB>::K : Layout<DIM, TURB>::W);
}

// Km / Ks: the limiter constants of the momentum components / of k and omega (0: psi = 1).
template <class T, int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_limiter(MeshView m, Src<T> st, const T* G, double Km,
                                                 double Ks, T* psi) {
  stage_begin();
  constexpr int NA = n_advected<DIM, TURB>();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.nc) return;
  const int nc = m.nc;
#pragma unroll 1
  for (int a = 0; a < NA; ++a) {
    const int q = advected_field<DIM, TURB>(a);
    const double K = a < DIM ? Km : Ks;
    T v;
    if (K > 0.0) {
      auto phi = [&](int cell) { return st((long)q * nc + cell); };
      auto grad = [&](int j) { return G[((long)q * DIM + j) * nc + c]; };
      v = limiter_cell<T, DIM>(m, c, K, phi, grad);
    } else {
      v = cst(1.0, st((long)q * nc + c));
    }
    psi[(long)a * nc + c] = v;
  }
}

// The advected face value of field q through face f from the upwind cell cu (upwind_value, the
// cell value; with a limiter, plus psi grad . (x_f - x_cu)).
template <class T, int DIM, class GP, class GV>
__device__ __forceinline__ T upwind_rec(const MeshView& m, const GP& G, const T* psi, int a, int q,
                                        int f, int cu, const T& value, const GV& gv) {
  if (!psi) return value;
  const int nc = m.nc;
  T d = G[((long)q * DIM) * nc + cu] * (gv.xf(m, 0, f) - gv.xc(m, 0, cu));
#pragma unroll
  for (int j = 1; j < DIM; ++j)
    d = d + G[((long)q * DIM + j) * nc + cu] * (gv.xf(m, j, f) - gv.xc(m, j, cu));
  return value + psi[(long)a * nc + cu] * d;
}

// ---------------------------------------------------------------- k_apcoef
// The momentum-diagonal face coefficients of face f (owner side, neighbour side) and the lagged
// mass-flux estimate me.
template <class T, int DIM, bool TURB, class S_, class GP, class CP, class GV>
__device__ __forceinline__ void apcoef_face(const MeshView& m, const CaseView& cv, const S_& st,
                                            const Par<T>& par, const GP& G, const CP& cl, int f,
                                            const GV& gv, T& ac_own, T& ac_nb, T& me) {
  using L = Layout<DIM, TURB>;
  using GT = decltype(gv.area(m, 0));
  const int nc = m.nc;
  const int o = m.owner[f];
  const bool interior = f < m.nfi;
  const int n = interior ? m.nb[f] : o;
  const GT g = gv.g(m, f), A = gv.area(m, f);
  const GS<T> rho = rho_of<T>(cv);
  const T mdot = mom_normal<T, DIM, TURB>(m, st, G, rho, f, o, n, g, gv) * A;
  me = mdot;
  const T mo = mu_eff<T, TURB>(par, cv, rho, cl, nc, o);
  if (interior) {
    const T mnb = mu_eff<T, TURB>(par, cv, rho, cl, nc, n);
    const T visc = conductance(mo, mnb, A, gv.dpn(m, f), gv.dnn(m, f));
    ac_own = visc + pos(mdot);
    ac_nb = visc + pos(-mdot);
  } else {
    const signed char kind = cv.fkind[f];
    T bv = mo;
    if (TURB && (kind == 0 || kind == 1)) {
      T nutw = cst(0.0, mo);
      if (cv.swall[f]) nutw = nut_wall(par.nu, gv.wd(cv, o), st((long)L::K * nc + o));
      bv = par.mu + rho * nutw;
    }
    const T vo = bv * (A * gv.inv_nd(m, f));
    const T conv = pos(mdot);
    ac_own = kind == 0 || kind == 1 ? vo : (kind == 2 ? vo + conv : (kind == 3 ? conv : cst(0.0, vo)));
    ac_nb = cst(0.0, vo);
  }
}

template <class T, int DIM, bool TURB>
__device__ __forceinline__ void k_apcoef_at(const int f, MeshView m, CaseView cv, Src<T> st, Par<T> par,
                                                const T* G, const T* cl, T* ac_own, T* ac_nb,
                                                T* me) {
  if (f >= m.nf) return;
  T ao, an, mf;
  apcoef_face<T, DIM, TURB>(m, cv, st, par, G, cl, f, typename GeoOf<T>::type{}, ao, an, mf);
  ac_own[f] = ao;
  ac_nb[f] = an;
  me[f] = mf;
}

template <class T, int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_apcoef(MeshView m, CaseView cv, Src<T> st, Par<T> par,
                                                const T* G, const T* cl, T* ac_own, T* ac_nb,
                                                T* me) {
  stage_begin();
  k_apcoef_at<T, DIM, TURB>(blockIdx.x * blockDim.x + threadIdx.x, m, cv, st, par, G, cl, ac_own,
                            ac_nb, me);
}

// ---------------------------------------------------------------- k_dcoeff
template <class T>
__device__ __forceinline__ void k_dcoeff_at(const int c, MeshView m, const T* ac_own, const T* ac_nb, T* dco) {
  if (c >= m.nc) return;
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  T a;
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    T x = (ent & FV_NB_BIT) ? ac_nb[f] : ac_own[f];
    a = i == b ? x : a + x;
  }
  dco[c] = gx<T>(m.vol, m.f_vol, c) / a;
}

template <class T>
__global__ void k_dcoeff(MeshView m, const T* ac_own, const T* ac_nb, T* dco) {
  stage_begin();
  k_dcoeff_at<T>(blockIdx.x * blockDim.x + threadIdx.x, m, ac_own, ac_nb, dco);
}

// ---------------------------------------------------------------- k_flux
// Face intermediates kept for the adjoint (double forward pass only), (FV_AUX_N, nf):
//   0 mdot, 1 damping, 2 dhat, 3 c (momentum conductance), 4 dc/dm_o, 5 dc/dm_n,
//   6.. 6+DIM-1 diffusion numerators of the velocity components, then for k and omega:
//   conductance, d/dgamma_o, d/dgamma_n, numerator.
template <int DIM, bool TURB>
struct Aux {
  static constexpr int N = 6 + DIM + (TURB ? 8 : 0);
  static constexpr int CPN = 6, S0 = 6 + DIM;
};

// The fluxes of face f, handed to wr(q, flux_q) for every field q.  `st` reads the state (Src, or
// a seeded accessor in the Jacobian assembly); aux (double only) receives the face intermediates.
template <class T, int DIM, bool TURB, class S, class GP, class CP, class DP, class Wr,
          class GV = typename GeoOf<T>::type>
__device__ __forceinline__ void flux_face(const MeshView& m, const CaseView& cv, const S& st,
                                          const Par<T>& par, const GP& G, const CP& cl, const DP& dco,
                                          const T* me, const T* psi, bool recompute_me, int f,
                                          const Wr& wr, double* aux, const GV& gv = GV{}) {
  using GT = decltype(gv.area(m, 0));
  constexpr bool KEEP = std::is_same<T, double>::value && std::is_same<GT, double>::value;
  using L = Layout<DIM, TURB>;
  const int nc = m.nc, nf = m.nf;
  const int o = m.owner[f];
  const GT A = gv.area(m, f);
  const GS<T> rho = rho_of<T>(cv);
  GS<T> irho;
  if constexpr (IsF32<T>::value) irho = 1.0f / rho;
  else irho = cv.irho;
  GT nrm[DIM], tP[DIM];
#pragma unroll
  for (int j = 0; j < DIM; ++j) {
    nrm[j] = gv.normal(m, j, f);
    tP[j] = gv.tP(m, j, f);
  }
  const T po = st((long)L::P * nc + o);
  const T mo = mu_eff<T, TURB>(par, cv, rho, cl, nc, o);
  if (f < m.nfi) {
    const int n = m.nb[f];
    const GT g = gv.g(m, f);
    GT tN[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) tN[j] = gv.tN(m, j, f);
    const T pn = st((long)L::P * nc + n);
    const T mest = recompute_me ? mom_normal<T, DIM, TURB>(m, st, G, rho, f, o, n, g, gv) * A : me[f];
    T gd = cst(0.0, po), gs = cst(0.0, po);
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      const T gpf = lerp(G[((long)L::P * DIM + j) * nc + o], G[((long)L::P * DIM + j) * nc + n], g);
      gd += gpf * gv.dvec(m, j, f);
      gs += gpf * gv.skew(m, j, f);
    }
    const T dhat = gv.nn2(m, f) * lerp(dco[o], dco[n], g);
    const T damping = ((pn - po) - gd) * gv.inv_nd(m, f);
    const T mdot = mest - (rho * A) * dhat * damping;
    const T pf = lerp(po, pn, g) + gs;
    const T mnb = mu_eff<T, TURB>(par, cv, rho, cl, nc, n);
    const Conduct<T> cm(mo, mnb, A, gv.dpn(m, f), gv.dnn(m, f));
    const T cmo = cm.c;
    const bool out = val(mdot) >= 0.0;
    const T pA = pf * A;
    using AX = Aux<DIM, TURB>;
    if constexpr (KEEP) {
      if (aux) {
        aux[0L * nf + f] = mdot;
        aux[1L * nf + f] = damping;
        aux[2L * nf + f] = dhat;
        aux[3L * nf + f] = cmo;
        aux[4L * nf + f] = cm.d_owner();
        aux[5L * nf + f] = cm.d_neighbour();
      }
    }
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      const T uo = st((long)i * nc + o), un = st((long)i * nc + n);
      T cpn = (un - uo);
#pragma unroll
      for (int j = 0; j < DIM; ++j)
        cpn += G[((long)i * DIM + j) * nc + n] * tN[j] - G[((long)i * DIM + j) * nc + o] * tP[j];
      const T* pm = cv.rec_mom ? psi : nullptr;
      const T up = out ? upwind_rec<T, DIM>(m, G, pm, i, i, f, o, uo, gv)
                       : upwind_rec<T, DIM>(m, G, pm, i, i, f, n, un, gv);
      wr(i, (pA * nrm[i] - cmo * cpn) + mdot * up);
      if constexpr (KEEP) {
        if (aux) aux[(long)(AX::CPN + i) * nf + f] = cpn;
      }
    }
    wr(L::P, mdot);
    if (TURB) {
      const T vflux = mdot * irho;
      const bool vout = val(vflux) >= 0.0;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int q = s == 0 ? L::K : L::W;
        const T go = cl[(4L + s) * nc + o], gn = cl[(4L + s) * nc + n];
        const T phio = st((long)q * nc + o), phin = st((long)q * nc + n);
        T cpn = (phin - phio);
#pragma unroll
        for (int j = 0; j < DIM; ++j)
          cpn += G[((long)q * DIM + j) * nc + n] * tN[j] - G[((long)q * DIM + j) * nc + o] * tP[j];
        const Conduct<T> cq(go, gn, A, gv.dpn(m, f), gv.dnn(m, f));
        const T cs_ = cq.c;
        const T* ps = cv.rec_sca ? psi : nullptr;
        const T up = vout ? upwind_rec<T, DIM>(m, G, ps, DIM + s, q, f, o, phio, gv)
                          : upwind_rec<T, DIM>(m, G, ps, DIM + s, q, f, n, phin, gv);
        wr(q, vflux * up - cs_ * cpn);
        if constexpr (KEEP) {
          if (aux) {
            const long b0 = AX::S0 + 4 * s;
            aux[b0 * nf + f] = cs_;
            aux[(b0 + 1) * nf + f] = cq.d_owner();
            aux[(b0 + 2) * nf + f] = cq.d_neighbour();
            aux[(b0 + 3) * nf + f] = cpn;
          }
        }
      }
    }
  } else {
    const signed char kind = cv.fkind[f];
    T uo[DIM], bu[DIM];
#pragma unroll
    for (int j = 0; j < DIM; ++j) {
      uo[j] = st((long)j * nc + o);
      bu[j] = bvel(cv, nf, f, j, kind, uo[j], par);
    }
    T mdot;
    if (kind == 2) {
      T un = bu[0] * nrm[0];
#pragma unroll
      for (int j = 1; j < DIM; ++j) un += bu[j] * nrm[j];
      mdot = (rho * A) * un;
    } else if (kind == 3) {
      T un = uo[0] * nrm[0];
      T interp = G[((long)L::P * DIM) * nc + o] * nrm[0];
#pragma unroll
      for (int j = 1; j < DIM; ++j) {
        un += uo[j] * nrm[j];
        interp += G[((long)L::P * DIM + j) * nc + o] * nrm[j];
      }
      const T dh = gv.nn2(m, f) * dco[o];
      const T compact = (cv.fp[f] - po) * gv.inv_nd(m, f);
      mdot = (rho * A) * (un - dh * (compact - interp));
    } else {
      mdot = cst(0.0, po);
    }
    const T pf = bpress(cv, f, kind, po);
    T gb = mo;
    if (TURB && (kind == 0 || kind == 1)) {
      T nutw = cst(0.0, mo);
      if (cv.swall[f]) nutw = nut_wall(par.nu, gv.wd(cv, o), st((long)L::K * nc + o));
      gb = par.mu + rho * nutw;
    }
    const T gA = gb * (A * gv.inv_dpn(m, f));
    const bool out = val(mdot) >= 0.0;
    const T pA = pf * A;
#pragma unroll
    for (int i = 0; i < DIM; ++i) {
      T cp = G[((long)i * DIM) * nc + o] * tP[0];
#pragma unroll
      for (int j = 1; j < DIM; ++j) cp += G[((long)i * DIM + j) * nc + o] * tP[j];
      const T up = out ? upwind_rec<T, DIM>(m, G, cv.rec_mom ? psi : nullptr, i, i, f, o, uo[i], gv)
                       : bu[i];
      wr(i, (pA * nrm[i] - gA * (bu[i] - uo[i] - cp)) + mdot * up);
    }
    wr(L::P, mdot);
    if (TURB) {
      const T vflux = mdot * irho;
      const bool vout = val(vflux) >= 0.0;
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int q = s == 0 ? L::K : L::W;
        const T go = cl[(4L + s) * nc + o];
        const T phio = st((long)q * nc + o);
        T cp = G[((long)q * DIM) * nc + o] * tP[0];
#pragma unroll
        for (int j = 1; j < DIM; ++j) cp += G[((long)q * DIM + j) * nc + o] * tP[j];
        const T bphi = s == 0 ? bscalar(cv.kkind[f], cv.kval[f], phio, cp)
                              : bscalar(cv.wkind[f], cv.wval[f], phio, cp);
        T gface = go;
        if (s == 0 && cv.swall[f]) gface = (1.0 - wall_weight(par.nu, gv.wd(cv, o), phio)) * go;
        const T up = vout ? upwind_rec<T, DIM>(m, G, cv.rec_sca ? psi : nullptr, DIM + s, q, f, o,
                                               phio, gv)
                          : bphi;
        wr(q, vflux * up - gface * (A * gv.inv_dpn(m, f)) * (bphi - phio - cp));
      }
    }
  }
}

template <class T>
struct FluxStore {
  T* FL;
  int nf, f;
  __device__ __forceinline__ void operator()(int q, const T& x) const { FL[(long)q * nf + f] = x; }
};

template <class T, int DIM, bool TURB>
__device__ __forceinline__ void k_flux_at(const int f, MeshView m, CaseView cv, Src<T> st, Par<T> par,
                                              const T* G, const T* cl, const T* dco, const T* me,
                                              const T* psi, bool recompute_me, T* FL, double* aux) {
  if (f >= m.nf) return;
  flux_face<T, DIM, TURB>(m, cv, st, par, G, cl, dco, me, psi, recompute_me, f,
                          FluxStore<T>{FL, m.nf, f}, aux);
}

template <class T, int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_flux(MeshView m, CaseView cv, Src<T> st, Par<T> par,
                                              const T* G, const T* cl, const T* dco, const T* me,
                                              const T* psi, bool recompute_me, T* FL, double* aux) {
  stage_begin();
  k_flux_at<T, DIM, TURB>(blockIdx.x * blockDim.x + threadIdx.x, m, cv, st, par, G, cl, dco, me, psi,
                          recompute_me, FL, aux);
}

// ---------------------------------------------------------------- k_sum
// SST rows of cell c: k and omega source terms added to the face sums rk / rw, and the omega
// wall-cell fixation (aquaflux/turbulence/sources.py:60-412, fixed_value.py:124-158).
template <class T, int DIM, class Acc, class GP, class GV = typename GeoOf<T>::type>
__device__ __forceinline__ void sst_rows(const MeshView& m, const CaseView& cv, const Acc& st,
                                         const Par<T>& par, const GP& cl, const GP& G,
                                         const GP& Gwi, int c, T& rk, T& rw, const GV& gv = GV{}) {
  using L = Layout<DIM, true>;
  using GT = decltype(gv.area(m, 0));
  const int nc = m.nc;
  const GT V = gv.vol(m, c);
  const T k = st((long)L::K * nc + c), w = st((long)L::W * nc + c);
  const T S = cl[c], F1 = cl[(long)nc + c], nut = cl[2L * nc + c];
  const T nu = par.nu;
  const GT d = gv.wd(cv, c);
  const bool wall = cv.wcell[c] != 0;
  const T kp = pos(k);
  const T limit = (PROD_RATIO * BETA_STAR) * kp * w;
  T lim = fv_min(nut * (S * S), limit);
  T weff = w;
  if (wall) {
    const T lw = wall_weight(nu, d, k);
    const T pw = (nu + nut_wall(nu, d, k)) * cl[3L * nc + c] * log_shear(d, k);
    lim = (1.0 - lw) * lim + lw * pw;
    weff = omega_wall(nu, d, k);
  }
  rk = rk - lim * V;
  rk = rk + BETA_STAR * V * k * weff;
  if (wall) {
    // DifferenceRow w - omega_wall, or LogRatioRow log(w / omega_wall) for a log-solved omega
    // (aquaflux/discretization/fixed_value.py:80-120)
    rw = cv.log_w ? fv_log(w / omega_wall(nu, d, k)) : w - omega_wall(nu, d, k);
  } else {
    const T alpha = ALPHA_2 + F1 * (ALPHA_1 - ALPHA_2);
    const T cap = limit / fv_max(nut, cst(NUT_FLOOR, nut));
    const T beta = BETA_2 + F1 * (BETA_1 - BETA_2);
    T dkw = G[((long)L::K * DIM) * nc + c] * Gwi[c];
#pragma unroll
    for (int j = 1; j < DIM; ++j) dkw += G[((long)L::K * DIM + j) * nc + c] * Gwi[(long)j * nc + c];
    const T cross = (2.0 * SIGMA_W2) * (1.0 - F1) * dkw / w;
    rw = rw + V * (beta * (w * w) - alpha * fv_min(S * S, cap) - cross);
  }
}

template <class T, int DIM, bool TURB>
__device__ __forceinline__ void k_sum_at(const int c, MeshView m, CaseView cv, Src<T> st, Par<T> par, const T* FL, const T* cl,
                                             const T* G, const T* Gwi, double* R, double* JV) {
  using L = Layout<DIM, TURB>;
  constexpr int NF = L::NFLD;
  if (c >= m.nc) return;
  const int nc = m.nc, nf = m.nf;
  T r[NF];
  const int b = m.cf_ptr[c], e = m.cf_ptr[c + 1];
  for (int i = b; i < e; ++i) {
    const unsigned ent = m.cf_face[i];
    const int f = (int)(ent & ~FV_NB_BIT);
    const bool isnb = (ent & FV_NB_BIT) != 0;
#pragma unroll
    for (int q = 0; q < NF; ++q) {
      T x = FL[(long)q * nf + f];
      if (isnb) x = -x;
      r[q] = i == b ? x : r[q] + x;
    }
  }
  if (c == cv.pin) r[L::P] = st((long)L::P * nc + c) - cv.pin_value;
  if constexpr (TURB) sst_rows<T, DIM>(m, cv, st, par, cl, G, Gwi, c, r[L::K], r[L::W]);
#pragma unroll
  for (int q = 0; q < NF; ++q) put<T>(R, JV, (long)q * nc + c, r[q]);
}

template <class T, int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_sum(MeshView m, CaseView cv, Src<T> st, Par<T> par, const T* FL, const T* cl,
                                             const T* G, const T* Gwi, double* R, double* JV) {
  stage_begin();
  k_sum_at<T, DIM, TURB>(stage_cell<T>(m, cv), m, cv, st, par, FL, cl, G, Gwi, R, JV);
}

// Zero the tangent of n dual values (the "frozen" JVP holds gradients, closure and a_P fixed).
__global__ void k_freeze(long n, Dual* x) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i].d = 0.0;
}
template <class T>
void freeze(T*, long, cudaStream_t) {}
template <>
void freeze<Dual>(Dual* x, long n, cudaStream_t s) {
  k_freeze<<<fv_blocks(n, 256), 256, 0, s>>>(n, x);
}
__global__ void k_freeze_f(long n, DualF* x) {
  long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) x[i].d = 0.0f;
}
template <>
void freeze<DualF>(DualF* x, long n, cudaStream_t s) {
  k_freeze_f<<<fv_blocks(n, 256), 256, 0, s>>>(n, x);
}

// Every field's gradient with the case's scheme, into w.G.
template <class T, int DIM, bool TURB>
void gradient_stage(FvCase* cs, Src<T> st, Par<T> par, const Work<T>& w, cudaStream_t s) {
  const MeshView& m = cs->mesh->view;
  const CaseView& cv = cs->view;
  constexpr int NF = Layout<DIM, TURB>::NFLD;
  const int TB = cs->tbs[0];
  const int bc = fv_blocks(m.nc, TB);
  const int sweeps = cs->desc.gradient_sweeps;
  const double rel = sweeps >= 1 ? cs->desc.gradient_relaxation : 1.0;
  if (sweeps <= 1) {
    stage(k_grad<T, DIM, TURB>, bc, TB, s, m, cv, st, par, w.G, nullptr, rel);
    return;
  }
  T* x0 = ((sweeps - 1) % 2 == 0) ? w.G : w.Galt;
  T* x1 = x0 == w.G ? w.Galt : w.G;
  stage(k_grad<T, DIM, TURB>, bc, TB, s, m, cv, st, par, x0, w.Bg, rel);
  gg_sweeps<T, DIM, NF>(m, sweeps, rel, w.Bg, x0, x1, w.FL, s);
}

template <class T, int DIM, bool TURB>
int run(FvCase* cs, Src<T> st, Par<T> par, double* R, double* JV, cudaStream_t s,
        bool frozen = false, bool end_profile_run = true, double* aux = nullptr,
        const Work<T>* into = nullptr) {  // into: where its arrays go, in place of the workspace
  const MeshView& m = cs->mesh->view;
  const CaseView& cv = cs->view;
  const long nc = m.nc, nf = m.nf;
  cs->fwd_valid = 0;  // the workspace is about to hold this pass
  const Work<T> w =
      into ? *into : work_layout<T, DIM, TURB>(cs->work, nc, nf, psi_count<DIM, TURB>(cs));
  // each stage at its own block size (the index is the stage's profiling mark)
  const int* tb = cs->tbs;
  auto bc = [&](int k) { return fv_blocks(nc, tb[k]); };
  auto bf = [&](int k) { return fv_blocks(nf, tb[k]); };
  fv_prof_mark(cs, 0, s);
  gradient_stage<T, DIM, TURB>(cs, st, par, w, s);
  fv_prof_mark(cs, 1, s);
  if (TURB) stage(k_closure<T, DIM>, bc(1), tb[1], s, m, cv, st, par, w.G, w.cl, w.Gwi);
  fv_prof_mark(cs, 2, s);
  stage(k_apcoef<T, DIM, TURB>, bf(2), tb[2], s, m, cv, st, par, w.G, w.cl, w.acown, w.acnb, w.me);
  fv_prof_mark(cs, 3, s);
  stage(k_dcoeff<T>, bc(3), tb[3], s, m, w.acown, w.acnb, w.dco);
  const long npsi = psi_count<DIM, TURB>(cs);
  if (npsi)
    stage(k_limiter<T, DIM, TURB>, bc(3), tb[3], s, m, st, w.G, cv.lim_km, cv.lim_ks, w.psi);
  // G, closure, Gwi, a_P, d and the slope limiters
  if (frozen) freeze<T>(w.G, (long)(w.psi + npsi - w.G), s);
  fv_prof_mark(cs, 4, s);
  stage(k_flux<T, DIM, TURB>, bf(4), tb[4], s, m, cv, st, par, w.G, w.cl, w.dco, w.me,
        npsi ? w.psi : nullptr, frozen, w.FL, aux);
  fv_prof_mark(cs, 5, s);
  stage(k_sum<T, DIM, TURB>, bc(5), tb[5], s, m, cv, st, par, w.FL, w.cl, w.G, w.Gwi, R, JV);
  fv_prof_mark(cs, 6, s);
  if (end_profile_run) fv_prof_end_run(cs);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

#include "adjoint.inc.cuh"
#include "assemble.inc.cuh"
#include "jacobian.inc.cuh"
#include "linearised.inc.cuh"

template <int DIM, bool TURB>
int dispatch_t(FvCase* cs, const double* state, const double* tangent, int kind, double* R,
               double* JV, cudaStream_t s) {
  const double irho = 1.0 / cs->desc.rho;
  if (kind == FV_TAN_NONE) {
    return run<double, DIM, TURB>(
        cs, Src<double>{state}, Par<double>{cs->mu, cs->inlet_scale, cs->mu * irho}, R, nullptr, s);
  }
  if (kind == FV_TAN_STATE32 || kind == FV_TAN_FROZEN32) {
    constexpr int NF = Layout<DIM, TURB>::NFLD;
    const long n = (long)NF * cs->mesh->nc;
    int rc = fv_case_ensure_f32(cs, s);
    if (rc == FV_OK) rc = fv_d2f(n, state, cs->f_state, s);
    if (rc == FV_OK && tangent) rc = fv_d2f(n, tangent, cs->f_tangent, s);
    if (rc != FV_OK) return rc;
    Par<DualF> pf{{(float)cs->mu, 0.0f}, {(float)cs->inlet_scale, 0.0f},
                  {(float)(cs->mu * irho), 0.0f}};
    return run<DualF, DIM, TURB>(cs, Src<DualF>{cs->f_state, tangent ? cs->f_tangent : nullptr},
                                 pf, R, JV, s, kind == FV_TAN_FROZEN32);
  }
  if (kind == FV_TAN_STATE && cs->lin_use) {
    return run_linearised<DIM, TURB>(cs, state, tangent, JV, s);
  }
  const double dmu = kind == FV_TAN_MU ? 1.0 : 0.0;
  Par<Dual> par{{cs->mu, dmu}, {cs->inlet_scale, kind == FV_TAN_INLET ? 1.0 : 0.0},
                {cs->mu * irho, dmu * irho}};
  Src<Dual> st{state, (kind == FV_TAN_STATE || kind == FV_TAN_FROZEN) ? tangent : nullptr};
  return run<Dual, DIM, TURB>(cs, st, par, R, JV, s, kind == FV_TAN_FROZEN);
}


template <int DIM, bool TURB>
AdjWork adj_layout(FvCase* cs) {
  using L = Layout<DIM, TURB>;
  const long nc = cs->mesh->view.nc;
  AdjWork aw;
  double* p = cs->adj;
  aw.Wt = p; p += L::NFLD * nc;
  aw.sb = p; p += L::NFLD * nc;
  aw.Gb = p; p += L::NFLD * DIM * nc;
  aw.dcob = p; p += nc;
  aw.apb = p; p += nc;
  aw.clb = p; p += 4 * nc;
  aw.Gwib = p; p += DIM * nc;
  aw.Gb2 = p; p += L::NFLD * DIM * nc;  // present when the case is swept
  aw.Bb = p;
  aw.FLx = cs->flx_active ? cs->flx : nullptr;
  p += L::NFLD * DIM * nc;  // Bb
  constexpr int NA = n_advected<DIM, TURB>();
  aw.psi = nullptr;
  aw.psib = p; p += (long)NA * nc;
  aw.lnb = p;
  return aw;
}

// ---------------------------------------------------------------- one persistent launch
// The whole residual + VJP evaluation of a case with compact gradients and first-order upwind
// advection as ONE cooperative launch: the stages of run<double> and of the adjoint in order, each
// over its cells or faces, separated by grid-wide barriers (cooperative_groups grid sync; the
// cooperative launch guarantees every block is resident).  Each thread takes `chunk` consecutive
// cells / faces per step of a grid-stride loop.  Every cell or face is computed by the same body
// as in the stage-per-launch path, so the result is bitwise the same.
struct PersistentVjp {
  Work<double> w;
  AdjWork aw;
  const double* W;
  double* aux;
  double* R;
  double* out;
  double rel;
  int chunk;
};

template <int DIM, bool TURB>
__global__ void __launch_bounds__(128) k_persistent_vjp(MeshView m, CaseView cv, Src<double> st,
                                                        Par<double> par, PersistentVjp a) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  const long nthr = (long)gridDim.x * blockDim.x;
  const long tid = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const int chunk = a.chunk;
  auto each = [&](long n, auto&& fn) {
    for (long base = tid * chunk; base < n; base += nthr * chunk)
      for (int k = 0; k < chunk && base + k < n; ++k) fn((int)(base + k));
  };
  const Work<double>& w = a.w;
  const AdjWork& aw = a.aw;
  each(m.nc, [&](int c) { k_grad_at<double, DIM, TURB>(c, m, cv, st, par, w.G, nullptr, a.rel); });
  grid.sync();
  if constexpr (TURB) {
    each(m.nc, [&](int c) { k_closure_at<double, DIM>(c, m, cv, st, par, w.G, w.cl, w.Gwi); });
    grid.sync();
  }
  each(m.nf, [&](int f) {
    k_apcoef_at<double, DIM, TURB>(f, m, cv, st, par, w.G, w.cl, w.acown, w.acnb, w.me);
  });
  grid.sync();
  each(m.nc, [&](int c) { k_dcoeff_at<double>(c, m, w.acown, w.acnb, w.dco); });
  grid.sync();
  each(m.nf, [&](int f) {
    k_flux_at<double, DIM, TURB>(f, m, cv, st, par, w.G, w.cl, w.dco, w.me, nullptr, false, w.FL,
                                 a.aux);
  });
  grid.sync();
  each(m.nc, [&](int c) {
    k_sum_at<double, DIM, TURB>(c, m, cv, st, par, w.FL, w.cl, w.G, w.Gwi, a.R, nullptr);
  });
  grid.sync();
  each(m.nc, [&](int c) { a_sum_at<DIM, TURB>(c, m, cv, st, par, a.W, w.cl, w.G, w.Gwi, aw); });
  grid.sync();
  each(m.nc, [&](int c) {
    a_flux_at<DIM, TURB>(c, m, cv, st, par, w.G, w.cl, w.dco, w.me, a.aux, aw);
  });
  grid.sync();
  each(m.nc, [&](int c) {
    a_apcoef_at<DIM, TURB>(c, m, cv, st, par, w.G, w.cl, w.dco, w.me, a.aux, aw);
  });
  grid.sync();
  if constexpr (TURB) {
    each(m.nc, [&](int c) { a_closure_at<DIM>(c, m, cv, st, par, w.G, w.cl, aw); });
    grid.sync();
  }
  each(m.nf, [&](int f) { a_grad_face_at<DIM, TURB>(f, m, cv, aw, aw.Gb, nullptr, a.rel, w.FL); });
  grid.sync();
  each(m.nc, [&](int c) { a_grad_at<DIM, TURB>(c, m, cv, aw, w.FL, a.out); });
}

// Whether the case's schemes are those the persistent kernel runs.
bool persistent_supported(const FvCase* cs) {
  return cs->desc.gradient_sweeps <= 1 && !cs->view.rec_mom && !cs->view.rec_sca &&
         !cs->flx_active;
}

template <int DIM, bool TURB>
int run_vjp_persistent(FvCase* cs, const double* state, const double* W, double* R, double* out,
                       cudaStream_t s) {
  const MeshView& m = cs->mesh->view;
  const long nc = m.nc, nf = m.nf;
  PersistentVjp a;
  a.w = work_layout<double, DIM, TURB>(cs->work, nc, nf, 0);
  a.aw = adj_layout<DIM, TURB>(cs);
  a.W = W;
  a.aux = cs->aux;
  a.R = R ? R : cs->tmp;
  a.out = out;
  a.rel = cs->desc.gradient_sweeps >= 1 ? cs->desc.gradient_relaxation : 1.0;
  a.chunk = cs->pchunk;
  Src<double> st{state};
  Par<double> par{cs->mu, cs->inlet_scale, cs->mu / cs->desc.rho};
  const MeshView mv = m;
  const CaseView cv = cs->view;
  auto kern = k_persistent_vjp<DIM, TURB>;
  int dev = 0, sms = 0, per_sm = 0;
  FV_CUDA_TRY(cudaGetDevice(&dev));
  FV_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  FV_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, cs->pblock, 0));
  if (per_sm < 1) {
    fv_set_error("persistent residual + VJP: no block of %d threads fits on an SM", cs->pblock);
    return FV_ERR_ARG;
  }
  void* args[] = {(void*)&mv, (void*)&cv, (void*)&st, (void*)&par, (void*)&a};
  FV_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)kern, dim3(per_sm * sms),
                                          dim3(cs->pblock), args, 0, s));
  return FV_OK;
}

// gb_save (optional, (NF, DIM, nc)): receives the gradient cotangent before the corrected
// scheme's backward sweeps overwrite it (the mesh-coordinate adjoint re-runs them).
template <int DIM, bool TURB>
int run_vjp(FvCase* cs, const double* state, const double* W, double* R, double* out,
            cudaStream_t s, double* gb_save = nullptr, bool held = false) {
  if (held) {
    if (!cs->fwd_valid) {
      fv_set_error("fv_vjp_held: no forward pass held; call fv_hold_forward at this state (again "
                   "after any other evaluation or a parameter, viscosity-field, wall-distance or "
                   "geometry change)");
      return FV_ERR_ARG;
    }
  } else if (cs->persistent && !gb_save && persistent_supported(cs)) {
    cs->fwd_valid = 0;
    return run_vjp_persistent<DIM, TURB>(cs, state, W, R, out, s);
  }
  using L = Layout<DIM, TURB>;
  const MeshView& m = cs->mesh->view;
  const CaseView& cv = cs->view;
  const long nc = m.nc, nf = m.nf;
  Src<double> st{state};
  Par<double> par{cs->mu, cs->inlet_scale, cs->mu / cs->desc.rho};
  if (held) {
    // the forward stages' profiling marks at one instant: they took no time in this call
    for (int k = 0; k <= 6; ++k) fv_prof_mark(cs, k, s);
  } else {
    int rc = run<double, DIM, TURB>(cs, st, par, R ? R : cs->tmp, nullptr, s, false, false,
                                    cs->aux);
    if (rc != FV_OK) return rc;
    cs->fwd_valid = 1;  // the adjoint stages below read but do not change it
  }
  // forward workspace (double layout, as written by run<double>)
  Work<double> fw = work_layout<double, DIM, TURB>(cs->work, nc, nf, psi_count<DIM, TURB>(cs));
  double* G = fw.G;
  double* cl = fw.cl;
  double* Gwi = fw.Gwi;
  double* dco = fw.dco;
  AdjWork aw = adj_layout<DIM, TURB>(cs);
  const int* tb = cs->tbs;  // each stage at its own block size (its profiling mark's index)
  auto bc = [&](int k) { return fv_blocks(nc, tb[k]); };
  stage(a_sum<DIM, TURB>, bc(6), tb[6], s, m, cv, st, par, W, cl, G, Gwi, aw);
  fv_prof_mark(cs, 7, s);
  const bool lim = psi_count<DIM, TURB>(cs) > 0;
  if (lim) aw.psi = fw.psi;
  if (aw.FLx && lim)
    stage(a_flux<DIM, TURB, true, true>, bc(7), tb[7], s, m, cv, st, par, G, cl, dco, fw.me,
          cs->aux, aw);
  else if (aw.FLx)
    stage(a_flux<DIM, TURB, true>, bc(7), tb[7], s, m, cv, st, par, G, cl, dco, fw.me, cs->aux,
          aw);
  else if (lim)
    stage(a_flux<DIM, TURB, false, true>, bc(7), tb[7], s, m, cv, st, par, G, cl, dco, fw.me,
          cs->aux, aw);
  else
    stage(a_flux<DIM, TURB>, bc(7), tb[7], s, m, cv, st, par, G, cl, dco, fw.me, cs->aux, aw);
  if (lim && (cv.lim_km > 0.0 || cv.lim_ks > 0.0)) {
    stage(a_limiter<DIM, TURB>, bc(7), tb[7], s, m, st, G, cv.lim_km, cv.lim_ks, aw);
    stage(a_limiter_gather<DIM, TURB>, bc(7), tb[7], s, m, aw);
  }
  fv_prof_mark(cs, 8, s);
  stage(a_apcoef<DIM, TURB>, bc(8), tb[8], s, m, cv, st, par, G, cl, dco, fw.me, cs->aux, aw);
  fv_prof_mark(cs, 9, s);
  if (TURB) stage(a_closure<DIM>, bc(9), tb[9], s, m, cv, st, par, G, cl, aw);
  fv_prof_mark(cs, 10, s);
  const int sweeps = cs->desc.gradient_sweeps;
  const double rel = sweeps >= 1 ? cs->desc.gradient_relaxation : 1.0;
  const double* gb0 = aw.Gb;
  if (gb_save)
    FV_CUDA_TRY(cudaMemcpyAsync(gb_save, aw.Gb, sizeof(double) * L::NFLD * DIM * nc,
                                cudaMemcpyDeviceToDevice, s));
  if (sweeps >= 2) gb0 = gg_sweeps_adjoint<DIM, L::NFLD>(m, sweeps, rel, aw, fw.FL, s);
  stage(a_grad_face<DIM, TURB>, fv_blocks(nf, tb[10]), tb[10], s, m, cv, aw, gb0,
        sweeps >= 2 ? aw.Bb : nullptr, rel, fw.FL);
  stage(a_grad<DIM, TURB>, bc(10), tb[10], s, m, cv, aw, fw.FL, out);
  fv_prof_mark(cs, 11, s);
  fv_prof_end_run(cs);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

bool g_const_ready = false;

}  // namespace

#include "node_adjoint.inc.cuh"

size_t fv_adjoint_work_bytes(int dim, int turb, long nc, long nf, int sweeps, int advection) {
  long nfld = dim + 1 + (turb ? 2 : 0);
  long n = 2 * nfld * nc + nfld * dim * nc + 2 * nc + 4 * nc + dim * nc;
  // the sweeps' second iterate cotangent and B phi's (the limiter buffers follow them)
  if (sweeps >= 1 || advection >= 1) n += 2 * nfld * dim * nc;
  if (advection >= 1) n += (long)(dim + (turb ? 2 : 0)) * (nc + 2 * nf);
  return sizeof(double) * (size_t)n;
}

size_t fv_aux_bytes(int dim, int turb, long nf) {
  return sizeof(double) * (size_t)(6 + dim + (turb ? 8 : 0)) * nf;
}

int fv_case_vjp_run(FvCase* cs, const double* state, const double* W, double* R, double* out,
                    cudaStream_t s) {
  const int dim = cs->mesh->dim;
  const bool turb = cs->desc.turbulent != 0;
  if (dim == 2)
    return turb ? run_vjp<2, true>(cs, state, W, R, out, s) : run_vjp<2, false>(cs, state, W, R, out, s);
  return turb ? run_vjp<3, true>(cs, state, W, R, out, s) : run_vjp<3, false>(cs, state, W, R, out, s);
}

namespace {
template <int DIM, bool TURB>
int hold_forward(FvCase* cs, const double* state, double* R, cudaStream_t s) {
  Par<double> par{cs->mu, cs->inlet_scale, cs->mu / cs->desc.rho};
  int rc = run<double, DIM, TURB>(cs, Src<double>{state}, par, R ? R : cs->tmp, nullptr, s, false,
                                  true, cs->aux);
  if (rc == FV_OK) cs->fwd_valid = 1;
  return rc;
}
}  // namespace

int fv_case_hold_forward(FvCase* cs, const double* state, double* R, cudaStream_t s) {
  if (cs->wd_missing) {
    fv_set_error("turbulent case without SST wall faces: set its wall distance first "
                 "(fv_case_set_wall_distance)");
    return FV_ERR_ARG;
  }
  const int dim = cs->mesh->dim;
  const bool turb = cs->desc.turbulent != 0;
  if (dim == 2) return turb ? hold_forward<2, true>(cs, state, R, s) : hold_forward<2, false>(cs, state, R, s);
  return turb ? hold_forward<3, true>(cs, state, R, s) : hold_forward<3, false>(cs, state, R, s);
}

int fv_case_vjp_held(FvCase* cs, const double* state, const double* W, double* out,
                     cudaStream_t s) {
  const int dim = cs->mesh->dim;
  const bool turb = cs->desc.turbulent != 0;
  if (dim == 2)
    return turb ? run_vjp<2, true>(cs, state, W, nullptr, out, s, nullptr, true)
                : run_vjp<2, false>(cs, state, W, nullptr, out, s, nullptr, true);
  return turb ? run_vjp<3, true>(cs, state, W, nullptr, out, s, nullptr, true)
              : run_vjp<3, false>(cs, state, W, nullptr, out, s, nullptr, true);
}

namespace {
template <int DIM, bool TURB>
int linearise(FvCase* cs, const double* state, double* R, cudaStream_t s) {
  const long nc = cs->mesh->nc, nf = cs->mesh->nf;
  constexpr int NF = Layout<DIM, TURB>::NFLD;
  if (psi_count<DIM, TURB>(cs) > 0) {
    fv_set_error("fv_case_linearise: the linearised JVP covers first-order upwind advection only");
    return FV_ERR_ARG;
  }
  auto ensure = [](double** p, long n) {
    return *p || cudaMalloc(p, sizeof(double) * (size_t)n) == cudaSuccess;
  };
  if ((!cs->lin_aux && cudaMalloc(&cs->lin_aux, fv_aux_bytes(DIM, TURB, nf)) != cudaSuccess) ||
      !ensure(&cs->lin_me, nf) || !ensure(&cs->lin_d, nc) || !ensure(&cs->lin_g, NF * DIM * nc) ||
      !ensure(&cs->lin_r, NF * nc) ||
      (TURB && (!ensure(&cs->lin_cl, 7 * nc) || !ensure(&cs->lin_cc, LIN_NCOEF * nc) ||
                !ensure(&cs->lin_src, 2 * nc)))) {
    fv_set_error("fv_case_linearise: %s", cudaGetErrorString(cudaGetLastError()));
    return FV_ERR_CUDA;
  }
  if (TURB && cs->n_wall_cells < 0) {  // the wall cells, listed once a case
    std::vector<unsigned char> wall(nc);
    FV_CUDA_TRY(cudaMemcpyAsync(wall.data(), cs->wcell, nc, cudaMemcpyDeviceToHost, s));
    FV_CUDA_TRY(cudaStreamSynchronize(s));
    std::vector<int> cells;
    for (long c = 0; c < nc; ++c)
      if (wall[c]) cells.push_back((int)c);
    FV_CUDA_TRY(cudaMalloc(&cs->wall_cells, sizeof(int) * (cells.size() + 1)));
    FV_CUDA_TRY(cudaMemcpyAsync(cs->wall_cells, cells.data(), sizeof(int) * cells.size(),
                                cudaMemcpyHostToDevice, s));
    FV_CUDA_TRY(cudaStreamSynchronize(s));
    cs->n_wall_cells = (int)cells.size();
  }
  cs->lin_valid = 0;
  const double irho = 1.0 / cs->desc.rho;
  // the pass writes what is held where it stays
  Work<double> w = work_layout<double, DIM, TURB>(cs->work, nc, nf, psi_count<DIM, TURB>(cs));
  w.G = cs->lin_g;
  if (TURB) w.cl = cs->lin_cl;
  w.me = cs->lin_me;
  w.dco = cs->lin_d;
  int rc = run<double, DIM, TURB>(cs, Src<double>{state},
                                  Par<double>{cs->mu, cs->inlet_scale, cs->mu * irho}, R, nullptr,
                                  s, false, true, cs->lin_aux, &w);
  if (rc != FV_OK) return rc;
  FV_CUDA_TRY(cudaMemcpyAsync(cs->lin_r, R, sizeof(double) * NF * nc, cudaMemcpyDeviceToDevice, s));
  if constexpr (TURB) {
    k_lin_closure_coef<DIM><<<fv_blocks(nc, 128), 128, 0, s>>>(
        cs->mesh->view, cs->view, state, w.G, w.cl, cs->mu * irho, cs->lin_cc);
    FV_CUDA_TRY(cudaGetLastError());
  }
  cs->lin_valid = 1;
  return FV_OK;
}
}  // namespace

int fv_case_linearise(FvCase* cs, const double* state, double* R, cudaStream_t s) {
  if (cs->wd_missing) {
    fv_set_error("turbulent case without SST wall faces: set its wall distance first "
                 "(fv_case_set_wall_distance)");
    return FV_ERR_ARG;
  }
  const int dim = cs->mesh->dim;
  const bool turb = cs->desc.turbulent != 0;
  if (dim == 2) return turb ? linearise<2, true>(cs, state, R, s) : linearise<2, false>(cs, state, R, s);
  return turb ? linearise<3, true>(cs, state, R, s) : linearise<3, false>(cs, state, R, s);
}

size_t fv_residual_work_bytes(int dim, int turb, long nc, long nf, int sweeps, int advection) {
  long nfld = dim + 1 + (turb ? 2 : 0);
  long n = nfld * dim * nc + 7 * nc + dim * nc + 3 * nf + nc + nfld * nf;
  if (advection >= 1) n += (long)(dim + (turb ? 2 : 0)) * nc;  // slope limiters
  if (sweeps >= 2) n += 2 * nfld * dim * nc;  // B phi and the second sweep iterate
  return (size_t)n * sizeof(Dual);
}

// fp32: the face derivatives; fp64: the source rows' 4 doubles per cell (fewer: nc < nf).
size_t fv_jac_face_bytes(int dim, int turb, long nf) {
  long nfld = dim + 1 + (turb ? 2 : 0);
  return sizeof(float) * (size_t)(2 * nfld * nfld) * nf;
}

int fv_case_assemble_frozen(FvCase* cs, const double* state, const int* indptr,
                            const int* indices, void* values, void* D, int fp32,
                            cudaStream_t s) {
  auto go = [&](auto dim, auto turb) {
    constexpr int DIM = decltype(dim)::value;
    constexpr bool TURB = decltype(turb)::value;
    if (fp32)
      return assemble_frozen<DualF, DIM, TURB>(cs, state, indptr, indices, (float*)values,
                                               (float*)D, s);
    return assemble_frozen64<DIM, TURB>(cs, state, indptr, indices, (double*)values, (double*)D, s);
  };
  using D2 = std::integral_constant<int, 2>;
  using D3 = std::integral_constant<int, 3>;
  const bool turb = cs->desc.turbulent != 0;
  if (cs->mesh->dim == 2) return turb ? go(D2{}, std::true_type{}) : go(D2{}, std::false_type{});
  return turb ? go(D3{}, std::true_type{}) : go(D3{}, std::false_type{});
}

int fv_gg_sweeps_scalar(const MeshView& m, int sweeps, double rel, const double* num, double* x0,
                        double* x1, double* wface, cudaStream_t s) {
  if (m.dim == 2)
    gg_sweeps<double, 2, 1>(m, sweeps, rel, num, x0, x1, wface, s);
  else
    gg_sweeps<double, 3, 1>(m, sweeps, rel, num, x0, x1, wface, s);
  FV_CUDA_TRY(cudaGetLastError());
  return FV_OK;
}

int fv_residual_init_constants() {
  if (g_const_ready) return FV_OK;
  SstConst h;
  h.bs4 = pow(BETA_STAR, 0.25);
  double y = 11.0;
  for (int i = 0; i < 10; ++i) y = log(E_WALL * y) / KAPPA;
  h.ylam = y;
  FV_CUDA_TRY(cudaMemcpyToSymbol(c_sst, &h, sizeof(h)));
  g_const_ready = true;
  return FV_OK;
}

int fv_case_ensure_f32(FvCase* c, cudaStream_t s) {
  FvMesh* m = c->mesh;
  int rc = fv_mesh_ensure_f32(m, s);
  if (rc != FV_OK) return rc;
  const long nc = m->nc, dim = m->dim;
  if (!c->f32) {
    // wd (nc), wdg (dim nc), 1/wd and 1/wd^2 (2 nc), per-cell viscosity (nc)
    FV_CUDA_TRY(cudaMalloc(&c->f32, sizeof(float) * (size_t)(nc * (4 + dim))));
    FV_CUDA_TRY(cudaMalloc(&c->f_state, sizeof(float) * (size_t)c->nfld * nc));
    FV_CUDA_TRY(cudaMalloc(&c->f_tangent, sizeof(float) * (size_t)c->nfld * nc));
    float* p = c->f32;
    if ((rc = fv_d2f(nc, c->wd, p, s)) != FV_OK) return rc;
    if ((rc = fv_d2f(dim * nc, c->wdg, p + nc, s)) != FV_OK) return rc;
    if ((rc = fv_d2f(2 * nc, c->inv_wd, p + (1 + dim) * nc, s)) != FV_OK) return rc;
    CaseView& v = c->view;
    v.f_wd = p;
    v.f_wdg = p + nc;
    v.f_inv_wd = p + (1 + dim) * nc;
    v.f_inv_wd2 = p + (2 + dim) * nc;
    v.f_rho = (float)c->desc.rho;
  }
  if (c->mu_cell) {  // the per-cell viscosity can change between calls
    if ((rc = fv_d2f(nc, c->mu_cell, c->f32 + (3 + dim) * nc, s)) != FV_OK) return rc;
    c->view.f_mu_cell = c->f32 + (3 + dim) * nc;
  }
  return FV_OK;
}

// nu_t of a (physical) state: one residual evaluation, then the closure's eddy-viscosity row.
int fv_case_eddy_viscosity(FvCase* cs, const double* state, double* nut, cudaStream_t s) {
  const int dim = cs->mesh->dim;
  const long nc = cs->mesh->nc, nf = cs->mesh->nf;
  int rc = fv_case_run(cs, state, nullptr, FV_TAN_NONE, cs->tmp, nullptr, s);
  if (rc != FV_OK) return rc;
  const double* cl = dim == 2 ? work_layout<double, 2, true>(cs->work, nc, nf, psi_count<2, true>(cs)).cl
                              : work_layout<double, 3, true>(cs->work, nc, nf, psi_count<3, true>(cs)).cl;
  FV_CUDA_TRY(cudaMemcpyAsync(nut, cl + 2 * nc, sizeof(double) * nc, cudaMemcpyDeviceToDevice, s));
  return FV_OK;
}

int fv_case_run(FvCase* cs, const double* state, const double* tangent, int kind, double* R,
                double* JV, cudaStream_t s) {
  if (cs->wd_missing) {
    fv_set_error("turbulent case without SST wall faces: set its wall distance first "
                 "(fv_case_set_wall_distance)");
    return FV_ERR_ARG;
  }
  const int dim = cs->mesh->dim;
  const bool turb = cs->desc.turbulent != 0;
  if (dim == 2) {
    return turb ? dispatch_t<2, true>(cs, state, tangent, kind, R, JV, s)
                : dispatch_t<2, false>(cs, state, tangent, kind, R, JV, s);
  }
  return turb ? dispatch_t<3, true>(cs, state, tangent, kind, R, JV, s)
              : dispatch_t<3, false>(cs, state, tangent, kind, R, JV, s);
}
