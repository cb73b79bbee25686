// k_scalar.cu - node-centred scalar transport and turbulence of INTERNAL_STEP:
// ADV_Q/FCT_Q2/FCT_Q2L (adv_q.F, fct_q2.F, fct_q2l.F), VDIF_Q with the MY2.5 closure
// (vdif_q.F), ADV_T/ADV_S with FCT_T/FCT_S (adv_t.F, adv_s.F, fct_t.F, fct_s.F), VDIF_TS
// (vdif_ts.F), BCOND_TS (bcond_ts.F, mod_obcs.F:1223-1373), DENS2 (eqs_of_state.F) and the
// end-of-step shifts (internal_step.F:1034-1590).
//
// The node-ring gradients (PTPX.. over NBSN) and the ring extrema of the advected field
// are formed once per (node, layer) by k_grad into scratch fields.  Horizontal advection
// then runs in two phases: k_he_adv evaluates each control-volume half-edge flux once
// (one thread per cell and layer, the cell's three half-edges), and k_gather_q/_ts sum
// each node's half-edge fluxes with their signs in ascending half-edge order, which
// reproduces the reference's scatter sums bit for bit.  T and S (and Q2 and Q2L) are
// transported in the same launches since neither reads the other's update.
#include <cuda_bf16.h>

#include "fvg_model.h"

// The FP32 instantiations of the precision form's flux kernels are compiled from this
// same source a second time with -DFVG_F32_TU and multiply-add contraction (build.py),
// into namespace fvg_f32; the FP64 translation unit forwards their launches there.
#ifdef FVG_F32_TU
namespace fvg_f32 {
using namespace fvg;
#else
namespace fvg {
#endif

#define ONE_THIRD (1.0 / 3.0)
constexpr int kMaxKBs = 64;

static inline int nblk(int n, int b) { return (n + b - 1) / b; }

__device__ inline double F4(double x) { return (double)(float)x; }
__device__ inline int NBSN(const Dev& P, int i, int j) { return P.nbsn[(size_t)(j - 1) * (P.M + 1) + i]; }
__device__ inline double TRIEX(const Dev& P, int i, int j) { return P.dltxtrie[(size_t)(j - 1) * (P.M + 1) + i]; }
__device__ inline double TRIEY(const Dev& P, int i, int j) { return P.dltytrie[(size_t)(j - 1) * (P.M + 1) + i]; }

// One tracer's node data on layer k: value, ring gradients, ring extrema.
template <typename R>
struct TRec {
  R q, px, py, pxd, pyd, rmin, rmax;
  R vf;  // FP32 records: the node's VISCOFH on the record's layer or level (else unused)
};

// Storage of the ring gradients and extrema by arithmetic type.  FP64: six arrays per
// tracer (P.gq, P.gt).  FP32: one 32-byte record per tracer and (node, layer) in P.f.npk,
// record r = (K-1)*ms + I holding {value, PX, PY, PXD, PYD, min, max, VF} for tracer t at
// floats 16r + 8t, read and written as two float4; VF is the node's VISCOFH on the layer
// (T, S) or interpolated to the level (Q2, Q2L) as the half-edge fluxes take it, so that
// they need not gather it.
template <typename R> struct NodeRec;
template <> struct NodeRec<double> {
  __device__ static void store(const Dev& P, int mode, int t, size_t q, double, double px, double py, double pxd,
                               double pyd, double mn, double mx, double) {
    double* const* G = mode == 0 ? P.gq[t] : P.gt[t];
    G[0][q] = px;
    G[1][q] = py;
    G[2][q] = pxd;
    G[3][q] = pyd;
    G[4][q] = mn;
    G[5][q] = mx;
  }
  __device__ static TRec<double> load(const Dev& P, int mode, int t, size_t q, double qv) {
    double* const* G = mode == 0 ? P.gq[t] : P.gt[t];
    return TRec<double>{qv, G[0][q], G[1][q], G[2][q], G[3][q], G[4][q], G[5][q], 0.0};
  }
  __device__ static void minmax(const Dev& P, int mode, int t, size_t q, double& mn, double& mx) {
    double* const* G = mode == 0 ? P.gq[t] : P.gt[t];
    mn = G[4][q];
    mx = G[5][q];
  }
};
template <> struct NodeRec<float> {
  __device__ static float4* rec(const Dev& P, int t, size_t q) {
    return reinterpret_cast<float4*>(P.f.npk + 16 * q + 8 * t);
  }
  __device__ static void store(const Dev& P, int, int t, size_t q, float qv, float px, float py, float pxd,
                               float pyd, float mn, float mx, float vf) {
    float4* r = rec(P, t, q);
    r[0] = make_float4(qv, px, py, pxd);
    r[1] = make_float4(pyd, mn, mx, vf);
  }
  __device__ static TRec<float> load(const Dev& P, int, int t, size_t q, double) {
    const float4* r = rec(P, t, q);
    const float4 a = r[0], b = r[1];
    return TRec<float>{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  }
  __device__ static void minmax(const Dev& P, int, int t, size_t q, double& mn, double& mx) {
    const float4 b = rec(P, t, q)[1];
    mn = (double)b.y;
    mx = (double)b.z;
  }
};

template <typename R, int MODE>
__device__ inline TRec<R> load_trec(const Dev& P, int n, int k, int t) {
  const size_t q = N3(P, n, k);
  if (sizeof(R) == 8) {
    const double* Q = MODE == 0 ? (t == 0 ? P.q2 : P.q2l) : (t == 0 ? P.t1 : P.s1);
    return NodeRec<R>::load(P, MODE, t, q, Q[q]);
  }
  return NodeRec<R>::load(P, MODE, t, q, 0.0);
}

// -------------------------------------------------------------------------------------
// Ring gradients and extrema.  which == 0: Q2 and Q2L on K=2..KBM1 (adv_q.F:161-235);
// which == 1: T1 and S1 on K=1..KBM1 with the wet/dry substitution of adv_t.F:214-376,
// plus PFPXB/PFPYB and AH_BOTTOM at K=KBM1 (adv_t.F:394-408).
// -------------------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(256) k_grad(const Dev P, int which) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) return;
  int kb, ke;
  col_range(P, which == 0 ? 2 : 1, P.KBM1, kb, ke);
  const int nt = P.ntsn[i];
  const R art2 = (R)P.art2[i];
  const R half = (R)0.5;
  const R qmean = (R)F4(1.e-8);
  // One walk of the ring per layer serves both tracers: the ring node, its wet flag and
  // the ring-edge metrics are loaded once, and each neighbour's values are carried to
  // the next ring edge.  Per tracer the arithmetic is the reference's, term by term.
  for (int k = kb; k <= ke; ++k) {
    const double* Q[2];
    const double* QM[2] = {nullptr, nullptr};
    if (which == 0) {
      Q[0] = P.q2 + N3(P, 0, k);
      Q[1] = P.q2l + N3(P, 0, k);
    } else {
      Q[0] = P.t1 + N3(P, 0, k);
      Q[1] = P.s1 + N3(P, 0, k);
      QM[0] = P.tmean1 + N3(P, 0, k);
      QM[1] = P.smean1 + N3(P, 0, k);
    }
    R qi[2], qmi[2] = {0, 0}, q1[2], qm1[2] = {0, 0};
    R px[2] = {0, 0}, py[2] = {0, 0}, pxd[2] = {0, 0}, pyd[2] = {0, 0}, rmin[2], rmax[2];
    int i1 = NBSN(P, i, 1);
    int w1 = which == 0 ? 1 : P.iswetn[i1];
    for (int t = 0; t < 2; ++t) {
      qi[t] = (R)Q[t][i];
      q1[t] = (R)Q[t][i1];
      if (which != 0) {
        qmi[t] = (R)QM[t][i];
        qm1[t] = (R)QM[t][i1];
      }
      rmin[t] = q1[t];
      rmax[t] = q1[t];
    }
    for (int j = 1; j <= nt - 1; ++j) {
      const int i2 = NBSN(P, i, j + 1);
      const int w2 = which == 0 ? 1 : P.iswetn[i2];
      R ty, tx;
      if constexpr (sizeof(R) == 4) {
        const float2 tr = P.f.trie[(size_t)(j - 1) * (P.M + 1) + i];
        ty = tr.x;
        tx = tr.y;
      } else {
        ty = TRIEY(P, i, j);
        tx = TRIEX(P, i, j);
      }
      for (int t = 0; t < 2; ++t) {
        const R q2 = (R)Q[t][i2];
        if (j >= 2) {
          rmin[t] = fmin(rmin[t], q1[t]);
          rmax[t] = fmax(rmax[t], q1[t]);
        }
        R ffd, ff1;
        if (which == 0) {
          ffd = half * (q1[t] + q2 - qmean - qmean);
          ff1 = half * (q1[t] + q2);
        } else {
          const R qm2 = (R)QM[t][i2];
          R qa = q1[t], qb = q2, qma = qm1[t], qmb = qm2;
          if (w1 == 0 && w2 == 1) { qa = qi[t]; qma = qmi[t]; }
          else if (w1 == 1 && w2 == 0) { qb = qi[t]; qmb = qmi[t]; }
          else if (w1 == 0 && w2 == 0) { qa = qi[t]; qb = qi[t]; qma = qmi[t]; qmb = qmi[t]; }
          ffd = half * (qa + qb - qma - qmb);
          ff1 = half * (qa + qb);
          qm1[t] = qm2;
        }
        px[t] = px[t] + ff1 * ty;
        py[t] = py[t] + ff1 * tx;
        pxd[t] = pxd[t] + ffd * ty;
        pyd[t] = pyd[t] + ffd * tx;
        q1[t] = q2;
      }
      w1 = w2;
    }
    const size_t q = N3(P, i, k);
    // the node's mixing coefficient as the half-edge fluxes take it: VISCOFH on the layer or
    // interpolated to the level, in the FP32 records, and times NN_HVC in the plane gvn in FP64
    R vf;
    if (which == 0) {
      const size_t qm = N3(P, i, k - 1);
      const double za = P.dz(i, k - 1), zb = P.dz(i, k);
      vf = (R)((P.viscofh[q] * za + P.viscofh[qm] * zb) / (zb + za));
    } else {
      vf = (R)P.viscofh[q];
    }
    if (sizeof(R) == 8) P.gvn[q] = vf * P.nn_hvc[i];
    for (int t = 0; t < 2; ++t) {
      const R gx = px[t] / art2, gy = py[t] / art2, gxd = pxd[t] / art2, gyd = pyd[t] / art2;
      NodeRec<R>::store(P, which, t, q, qi[t], gx, gy, gxd, gyd, rmin[t], rmax[t], vf);
      if (which == 1 && k == P.KBM1) {
        if (t == 0) { P.pfpxb_t[i] = (double)gx; P.pfpyb_t[i] = (double)gy; }
        else { P.pfpxb_s[i] = (double)gx; P.pfpyb_s[i] = (double)gy; }
        double ah = (P.fact * P.viscofh[N3(P, i, P.KBM1)] + P.fm1) * P.nn_hvc[i];
        if (t == 0) P.ah_bottom_t[i] = ah;
        else P.ah_bottom_s[i] = ah;
      }
    }
  }
}

// Vertical-neighbour bound of FCT on sigma layers (fct_t.F:78-97) and on interfaces
// (fct_q2.F:73-92).
__device__ inline void fct_layer_bounds(const Dev& P, int i, int k, const double* F, double& fmax_, double& fmin_) {
  const double z = P.dz(i, k), zm = k > 1 ? P.dz(i, k - 1) : 0.0, zp = k < P.KBM1 ? P.dz(i, k + 1) : 0.0;
  size_t q = N3(P, i, k);
  if (k == 1) {
    size_t qp = N3(P, i, k + 1);
    double a = (F[q] * zp + F[qp] * z) / (z + zp);
    fmax_ = fmax(fmax_, a);
    fmin_ = fmin(fmin_, a);
  } else if (k == P.KBM1) {
    size_t qm = N3(P, i, k - 1);
    double a = (F[q] * zm + F[qm] * z) / (z + zm);
    fmax_ = fmax(fmax_, a);
    fmin_ = fmin(fmin_, a);
  } else {
    size_t qm = N3(P, i, k - 1), qp = N3(P, i, k + 1);
    double a = (F[q] * zm + F[qm] * z) / (z + zm);
    double b = (F[q] * zp + F[qp] * z) / (z + zp);
    fmax_ = fmax(fmax(fmax_, a), b);
    fmin_ = fmin(fmin(fmin_, a), b);
  }
}
__device__ inline void fct_level_bounds(const Dev& P, int i, int k, const double* F, double& fmax_, double& fmin_) {
  const double z = P.dzz(i, k), zm = P.dzz(i, k - 1), zmm = k > 2 ? P.dzz(i, k - 2) : 0.0;
  size_t q = N3(P, i, k), qm = N3(P, i, k - 1), qp = N3(P, i, k + 1);
  if (k == 2) {
    double a = (F[q] * z + F[qp] * zm) / (z + zm);
    fmax_ = fmax(fmax_, a);
    fmin_ = fmin(fmin_, a);
  } else if (k == P.KBM1) {
    size_t qmm = N3(P, i, k - 2);
    double a = (F[q] * zmm + F[qm] * zm) / (zm + zmm);
    fmax_ = fmax(fmax_, a);
    fmin_ = fmin(fmin_, a);
  } else {
    size_t qmm = N3(P, i, k - 2);
    double a = (F[q] * zmm + F[qm] * zm) / (zm + zmm);
    double b = (F[q] * z + F[qp] * zm) / (z + zm);
    fmax_ = fmax(fmax(fmax_, a), b);
    fmin_ = fmin(fmin(fmin_, a), b);
  }
}

// -------------------------------------------------------------------------------------
// Half-edge fluxes of ADV_Q (adv_q.F:250-342) and ADV_T/ADV_S (adv_t.F:411-556).
//
// Phase 1 (k_he_adv, one thread per cell and layer): a cell's three control-volume
// half-edges run from its centroid to its edge midpoints and each separates two of the
// cell's own nodes, so the node data (tracer value, ring gradients and extrema, mixing
// coefficient) is loaded once for the three half-edges.  Each half-edge flux EXFLUX is
// evaluated once, in the reference's expression order, and stored at the half-edge's
// position slot*ns + cell.
// Phase 2 (k_gather_*, one thread per node and layer) sums the node's half-edge fluxes
// with their signs in ascending half-edge order -- the order of the reference's scatter --
// and applies the vertical flux, the update and the FCT clamp.
// MODE 0: Q2 and Q2L on interfaces K=2..KBM1; MODE 1: T and S on layers K=1..KBM1.
// -------------------------------------------------------------------------------------
// A cell's half-edge in slot s separates two of its nodes; the cell's nodes are taken in the
// order X0, X1, X2 (hex) in which slot s separates X(s) and X(s+1 mod 3), so that every node
// record has a fixed place and no value is selected at run time (the selects between the
// records were a third of the kernel's instructions, which bound it).  Bit s of the order's
// fourth word tells that NIEC(he,1) is X(s+1): the two sides then swap roles, which the
// upwind weights alone see.
template <typename R>
struct HeCell {
  R uq, vq, dtij;
};

// Cell data of the half-edge fluxes on layer k, formed in FP64 and rounded to R.
template <typename R, int MODE>
__device__ inline void he_cell_load(const Dev& P, int c, int k, HeCell<R>& hc) {
  size_t ck = C3(P, c, k);
  if (MODE == 0) {
    size_t ckm = C3(P, c, k - 1);
    const double za = P.dz1(c, k - 1), zb = P.dz1(c, k), zs = zb + za;
    hc.uq = (R)((P.u[ck] * za + P.u[ckm] * zb) / zs);
    hc.vq = (R)((P.v[ck] * za + P.v[ckm] * zb) / zs);
    hc.dtij = (R)(P.dt1[c] * P.dzz1(c, k - 1));
  } else {
    hc.uq = (R)P.u[ck];
    hc.vq = (R)P.v[ck];
    hc.dtij = (R)(P.dt1[c] * P.dz1(c, k));
  }
}

// Metrics of one half-edge (DLTXE, DLTYE and the DLTXNCVE/DLTYNCVE of X(s) and X(s+1)), read
// by position (coalesced over the threads of consecutive cells).
template <typename R>
struct HeGeo {
  R dx, dy, xa, ya, xb, yb;
};
template <typename R>
__device__ inline HeGeo<R> he_geo(const Dev& P, size_t pos) {
  typedef Mesh<R> Mh;
  if constexpr (sizeof(R) == 4) {
    const float4 a = P.f.hg4[pos];
    const float2 b = P.f.hg2[pos];
    return HeGeo<R>{a.x, a.y, a.z, a.w, b.x, b.y};
  } else {
    return HeGeo<R>{Mh::hg(P, 0, pos), Mh::hg(P, 1, pos), Mh::hg(P, 2, pos),
                    Mh::hg(P, 3, pos), Mh::hg(P, 4, pos), Mh::hg(P, 5, pos)};
  }
}

// VISCOFH*NN_HVC of a node as the half-edge fluxes take it (in FP32 from its record).
template <typename R>
__device__ inline R he_vn(const Dev& P, int n, int k, R nn, R vf) {
  if constexpr (sizeof(R) == 4)
    return vf * nn;
  else
    return P.gvn[N3(P, n, k)];
}
// Horizontal viscosity of a half-edge from its nodes' VISCOFH*NN_HVC and NN_HVC.
template <typename R, int MODE>
__device__ inline R he_visc(const Dev& P, R vna, R vnb, R nna, R nnb) {
  const R half = (R)0.5;
  R viscof = (R)P.fact * half * (vna + vnb) + (R)P.fm1 * half * (nna + nnb);
  if (MODE == 0 && P.hprnu != 1.0) viscof = viscof / (R)P.hprnu;
  return viscof;
}
// The bounds of a node's face values: its ring and itself.
template <typename R>
__device__ inline void he_bounds(TRec<R>& r) {
  r.rmin = fmin(r.rmin, r.q);
  r.rmax = fmax(r.rmax, r.q);
}

// EXFLUX of a half-edge with metrics g for one tracer, in R; ra and rb are the records of
// X(s) and X(s+1) with their bounds (he_bounds), flip the slot's bit of hex, viscof its
// viscosity.  xadv receives EXFLUX-FXX-FYY.
template <typename R>
__device__ inline R he_flux(const HeCell<R>& hc, const HeGeo<R>& g, int flip, const TRec<R>& ra, const TRec<R>& rb,
                            R viscof, R* xadv) {
  const R half = (R)0.5, one = (R)1.0;
  const R dltxe = g.dx, dltye = g.dy;
  R un = hc.vq * dltxe - hc.uq * dltye;
  R fa = ra.q + g.xa * ra.px + g.ya * ra.py;
  R fb = rb.q + g.xb * rb.px + g.yb * rb.py;
  if (fa < ra.rmin) fa = ra.rmin;
  if (fa > ra.rmax) fa = ra.rmax;
  if (fb < rb.rmin) fb = rb.rmin;
  if (fb > rb.rmax) fb = rb.rmax;
  R txx = half * (ra.pxd + rb.pxd) * viscof;
  R tyy = half * (ra.pyd + rb.pyd) * viscof;
  R fxx = -hc.dtij * txx * dltye;
  R fyy = hc.dtij * tyy * dltxe;
  R sg = fsign1(un);
  if (flip) sg = -sg;
  R exflux = -un * hc.dtij * ((one + sg) * fb + (one - sg) * fa) * half + fxx + fyy;
  if (xadv) *xadv = exflux - fxx - fyy;
  return exflux;
}

// Largest block of k_he_adv.  The FP32 form takes 64 registers and eight blocks per SM: 200 k
// nodes, six -> eight blocks, ADV_Q 716 -> 682 us.  In FP64 five blocks (96 registers) suit T and
// S (28 bytes spilled); Q2 and Q2L, with the level interpolation, spill 72 and keep four (ADV_Q
// 1186 against 1258 us).
constexpr int kHeThreads = 128;
template <typename R, int MODE>
__global__ void __launch_bounds__(kHeThreads, sizeof(R) == 4 ? 8 : (MODE == 1 ? 5 : 4)) k_he_adv(const Dev P, int parts) {
  typedef typename Mesh<R>::R2 R2;
  int c = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (c > P.N) return;
  int kb, ke;
  col_range(P, MODE == 0 ? 2 : 1, P.KBM1, kb, ke);
  const bool do0 = parts & (MODE == 0 ? AD_Q2 : AD_T), do1 = parts & (MODE == 0 ? AD_Q2L : AD_S);
  const int4 hx = P.hex[c];
  const R nn0 = (R)P.nn_hvc[hx.x], nn1 = (R)P.nn_hvc[hx.y], nn2 = (R)P.nn_hvc[hx.z];
  // Each node's record is loaded once per tracer and layer and serves its two half-edges.
  HeCell<R> hc;
  for (int k = kb; k <= ke; ++k) {
    he_cell_load<R, MODE>(P, c, k, hc);
    R2* EX = Mesh<R>::ex2(P) + (size_t)(k - 1) * P.ncvs + c;
    R e[2][3] = {{0, 0, 0}, {0, 0, 0}};
    R vs0 = 0, vs1 = 0, vs2 = 0;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!(t == 0 ? do0 : do1)) continue;
      TRec<R> r0 = load_trec<R, MODE>(P, hx.x, k, t);
      TRec<R> r1 = load_trec<R, MODE>(P, hx.y, k, t);
      TRec<R> r2 = load_trec<R, MODE>(P, hx.z, k, t);
      if (t == 0 || !do0) {  // the mixing is the same for both tracers
        const R v0 = he_vn<R>(P, hx.x, k, nn0, r0.vf), v1 = he_vn<R>(P, hx.y, k, nn1, r1.vf),
                v2 = he_vn<R>(P, hx.z, k, nn2, r2.vf);
        vs0 = he_visc<R, MODE>(P, v0, v1, nn0, nn1);
        vs1 = he_visc<R, MODE>(P, v1, v2, nn1, nn2);
        vs2 = he_visc<R, MODE>(P, v2, v0, nn2, nn0);
      }
      he_bounds(r0);
      he_bounds(r1);
      he_bounds(r2);
      e[t][0] = he_flux<R>(hc, he_geo<R>(P, c), hx.w & 1, r0, r1, vs0, nullptr);
      e[t][1] = he_flux<R>(hc, he_geo<R>(P, (size_t)P.ns + c), hx.w & 2, r1, r2, vs1, nullptr);
      e[t][2] = he_flux<R>(hc, he_geo<R>(P, (size_t)2 * P.ns + c), hx.w & 4, r2, r0, vs2, nullptr);
    }
    for (int s = 0; s < 3; ++s) EX[(size_t)s * P.ns] = mk2(e[0][s], e[1][s]);
  }
}

// The same where a cell's half-edges do not go round its nodes (Dev::closed): both nodes of each
// half-edge from NIEC.
template <typename R, int MODE>
__global__ void __launch_bounds__(kHeThreads) k_he_adv_listed(const Dev P, int parts) {
  typedef typename Mesh<R>::R2 R2;
  const int c = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (c > P.N) return;
  int kb, ke;
  col_range(P, MODE == 0 ? 2 : 1, P.KBM1, kb, ke);
  const bool on[2] = {(parts & (MODE == 0 ? AD_Q2 : AD_T)) != 0, (parts & (MODE == 0 ? AD_Q2L : AD_S)) != 0};
  HeCell<R> hc;
  for (int k = kb; k <= ke; ++k) {
    he_cell_load<R, MODE>(P, c, k, hc);
    for (int s = 0; s < 3; ++s) {
      const int he = P.cell_he[3 * c + s], na = P.niec[he], nb = P.niec[P.NCV + 1 + he];
      const size_t pos = (size_t)s * P.ns + c;
      const R nna = (R)P.nn_hvc[na], nnb = (R)P.nn_hvc[nb];
      R e[2] = {0, 0};
      for (int t = 0; t < 2; ++t) {
        if (!on[t]) continue;
        TRec<R> ra = load_trec<R, MODE>(P, na, k, t), rb = load_trec<R, MODE>(P, nb, k, t);
        const R visc = he_visc<R, MODE>(P, he_vn<R>(P, na, k, nna, ra.vf), he_vn<R>(P, nb, k, nnb, rb.vf), nna, nnb);
        he_bounds(ra);
        he_bounds(rb);
        e[t] = he_flux<R>(hc, he_geo<R>(P, pos), 0, ra, rb, visc, nullptr);
      }
      Mesh<R>::ex2(P)[(size_t)(k - 1) * P.ncvs + pos] = mk2(e[0], e[1]);
    }
  }
}

// XFLUX_ADV of one open-boundary node (adv_t.F:510-511, 572-579): the advective parts of
// its half-edge fluxes, recomputed with the same arithmetic as phase 1.
template <typename R>
__device__ inline double obc_xflux_adv(const Dev& P, int i, int k, int t) {
  R xa = 0;
  for (int q = P.node_he_ptr[i]; q < P.node_he_ptr[i + 1]; ++q) {
    int code = P.node_he[q];
    int he = code >> 1;
    int c = P.ntrg[he];
    const int sl = P.cell_he[3 * c] == he ? 0 : (P.cell_he[3 * c + 1] == he ? 1 : 2);
    const int flip = (P.closed & 2) ? (P.hex[c].w >> sl) & 1 : 0, n1 = P.niec[he], n2 = P.niec[P.NCV + 1 + he];
    const int na = flip ? n2 : n1, nb = flip ? n1 : n2;
    HeCell<R> hc;
    he_cell_load<R, 1>(P, c, k, hc);
    TRec<R> ra = load_trec<R, 1>(P, na, k, t), rb = load_trec<R, 1>(P, nb, k, t);
    const R nna = (R)P.nn_hvc[na], nnb = (R)P.nn_hvc[nb];
    const R visc = he_visc<R, 1>(P, he_vn<R>(P, na, k, nna, ra.vf), he_vn<R>(P, nb, k, nnb, rb.vf), nna, nnb);
    he_bounds(ra);
    he_bounds(rb);
    R part;
    he_flux<R>(hc, he_geo<R>(P, (size_t)sl * P.ns + c), flip, ra, rb, visc, &part);
    xa = (code & 1) ? xa - part : xa + part;
  }
  return (double)xa;
}

// XFLUX_OBC of every open-boundary node, layer and tracer (adv_t.F:572-579), one thread
// each (blockIdx.y: the layer, blockIdx.z: the tracer).  The recomputation is a long chain
// for few nodes: inside the node gather it held every block with an open-boundary node
// back and cost all of them its registers (102 against 64-78).
template <typename R>
__global__ void __launch_bounds__(64) k_obc_xflux(const Dev P, int parts) {
  const int ob = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1, t = blockIdx.z;
  if (ob > P.iobcn || !(parts & (t == 0 ? AD_T : AD_S))) return;
  (t == 0 ? P.xflux_obc_t : P.xflux_obc_s)[(size_t)(k - 1) * (P.iobcn + 1) + ob] =
      obc_xflux_adv<R>(P, P.i_obc_n[ob], k, t);
}

// Signed sum of a node's half-edge fluxes on layer k, both tracers, in ascending
// half-edge order (the order of the reference's scatter into XFLUX).
// The loads are issued kHeBat entries at a time (codes, then fluxes) and added in order; a
// node of six cells has twelve.  Four, six and eight entries with the node gathers at 200 k
// nodes x 30 layers: ADV_Q 1094, 1090, 1085 us in FP64, 751, 722, 716 in FP32.
constexpr int kHeBat = 8;
// Largest block of the node gathers.  Four FP64 and six FP32 blocks per SM leave them 128 and
// 80 registers; six and seven spill 140 and 76 bytes (FP64 step 9900 against 9840 us).
constexpr int kGatherThreads = 128;
template <typename R>
__device__ inline double2 gather_he(const Dev& P, int i, int n, int k) {
  typedef typename Mesh<R>::R2 R2;
  const R2* EX = Mesh<R>::ex2(P) + (size_t)(k - 1) * P.ncvs;
  const int* L = P.node_vpos_ell + i;
  const size_t ms = P.ms;
  R x0 = 0, x1 = 0;
  auto add = [&](int code, R2 e) {
    if (code & 1) {
      x0 = x0 - e.x;
      x1 = x1 - e.y;
    } else {
      x0 = x0 + e.x;
      x1 = x1 + e.y;
    }
  };
  for (int j = 0; j < n; j += kHeBat) {
    int c[kHeBat];
    R2 e[kHeBat];
#pragma unroll
    for (int b = 0; b < kHeBat; ++b) c[b] = L[(j + b < n ? j + b : j) * ms];
#pragma unroll
    for (int b = 0; b < kHeBat; ++b) e[b] = EX[c[b] >> 1];
#pragma unroll
    for (int b = 0; b < kHeBat; ++b)
      if (j + b < n) add(c[b], e[b]);
  }
  return make_double2((double)x0, (double)x1);
}

// Phase 2 of ADV_Q(Q2,Q2F)/ADV_Q(Q2L,Q2LF) (adv_q.F:114-401) with FCT_Q2/FCT_Q2L.
// Latency bounds the node gathers (30 % of the issue slots at 28 % occupancy), so a layer's loads
// of both tracers stand before its first store, and what two neighbouring layers share -- the
// values beside the interface, the value on it (the lower layer's upper bound is the same sum
// with its two terms swapped) and the vertical flux through it -- is formed once and handed
// down.  That and the node's quotients taken out of the loop halve the divisions (14 -> 7 per
// layer in the T/S gather).  At 200 k nodes x 30 layers ADV_Q went 1187 -> 1086 us and ADV_TS
// 1125 -> 1009 in FP64, 802 -> 682 and 805 -> 653 in FP32 (with k_he_adv's blocks).
template <typename R>
__global__ void __launch_bounds__(kGatherThreads, sizeof(R) == 4 ? 6 : 4) k_gather_q(const Dev P, int parts) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) return;
  int kb, ke;
  col_range(P, 2, P.KBM1, kb, ke);
  if (kb > ke) return;
  const bool wet = P.iswetn[i] * P.iswetnt[i] == 1;
  const bool fct = (parts & AD_FCT) && !P.riv_skip[i];
  const int nhe = P.node_he_ptr[i + 1] - P.node_he_ptr[i], KBM1 = P.KBM1;
  const double art1 = P.art1[i], dt = P.dt[i], dr = dt / P.d[i];
  const bool on[2] = {(parts & AD_Q2) != 0, (parts & AD_Q2L) != 0};
  const double* Q[2] = {P.q2, P.q2l};
  double* QF[2] = {P.q2f, P.q2lf};
  // f, fp: Q on levels k and k+1; wf, wfm: WTS*Q on levels k and k-1; face: the bound between
  // levels k-1 and k, which is level k-1's lower and level k's upper one
  double f[2], wf[2], wfm[2], face[2] = {0.0, 0.0};
  {
    const size_t q = N3(P, i, kb), qm = N3(P, i, kb - 1);
    const double w = P.wts[q], wm = P.wts[qm];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!on[t]) continue;
      const double fm = Q[t][qm];
      f[t] = Q[t][q];
      wfm[t] = wm * fm;
      wf[t] = w * f[t];
      if (fct && kb > 2) {
        const double zm = P.dzz(i, kb - 1), zmm = P.dzz(i, kb - 2);
        face[t] = (f[t] * zmm + fm * zm) / (zm + zmm);
      }
    }
  }
  for (int k = kb; k <= ke; ++k) {
    const size_t q = N3(P, i, k), qp = N3(P, i, k + 1);
    const double z = P.dzz(i, k), zm = P.dzz(i, k - 1), zl = P.dz(i, k - 1) + P.dz(i, k);
    const double wp = P.wts[qp];
    double fp[2], qmin[2], qmax[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!on[t]) continue;
      fp[t] = Q[t][qp];
      if (fct) NodeRec<R>::minmax(P, 0, t, q, qmin[t], qmax[t]);
    }
    const double2 xs = gather_he<R>(P, i, nhe, k);
    const double rt = P.dti / (dt * zm);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!on[t]) continue;
      if (k == 2) {
        // QF = 0 on every level before the interior levels are set (adv_q.F:114)
        QF[t][N3(P, i, 1)] = 0.0;
        QF[t][N3(P, i, P.KB)] = 0.0;
      }
      double x = t == 0 ? xs.x : xs.y;
      const double wfp = wp * fp[t];
      double qf = f[t];
      if (wet) {
        const double temp = wfm[t] - wfp;
        x = x + temp * art1 * zm / zl;
        qf = (f[t] - x / art1 * rt) * dr;
      }
      if (fct) {
        if (k > 2) {
          qmax[t] = fmax(qmax[t], face[t]);
          qmin[t] = fmin(qmin[t], face[t]);
        }
        if (k == 2 || k < KBM1) {
          face[t] = (f[t] * z + fp[t] * zm) / (z + zm);
          qmax[t] = fmax(qmax[t], face[t]);
          qmin[t] = fmin(qmin[t], face[t]);
        }
        if (qmin[t] - qf > 0.0) qf = qmin[t];
        if (qf - qmax[t] > 0.0) qf = qmax[t];
      }
      QF[t][q] = qf;
      wfm[t] = wf[t];
      wf[t] = wfp;
      f[t] = fp[t];
    }
  }
}

// FCT_Q2 / FCT_Q2L alone (fct_q2.F:51-99) on QF already in memory.
__global__ void __launch_bounds__(256) k_fct_q(const Dev P, int parts) {
  int i = blockIdx.x * 32 + threadIdx.x + 1;
  int k = blockIdx.y * 8 + threadIdx.y + 2;
  if (i > P.M || k > P.KBM1 || P.riv_skip[i]) return;
  for (int t = 0; t < 2; ++t) {
    if (!(parts & (t == 0 ? AD_Q2 : AD_Q2L))) continue;
    const double* Q = (t == 0 ? P.q2 : P.q2l);
    double* QF = (t == 0 ? P.q2f : P.q2lf);
    size_t q = N3(P, i, k);
    double qmax = Q[N3(P, NBSN(P, i, 1), k)], qmin = qmax;
    for (int j = 2; j <= P.ntsn[i]; ++j) {
      double v = Q[N3(P, NBSN(P, i, j), k)];
      qmax = fmax(qmax, v);
      qmin = fmin(qmin, v);
    }
    fct_level_bounds(P, i, k, Q, qmax, qmin);
    double qf = QF[q];
    if (qmin - qf > 0.0) qf = qmin;
    if (qf - qmax > 0.0) qf = qmax;
    QF[q] = qf;
  }
}

// -------------------------------------------------------------------------------------
// VDIF_Q, MY2.5 (vdif_q.F:119-513), one thread per node column.  With copy_back the
// end-of-closure shift Q2=Q2F, Q2L=Q2LF (internal_step.F:1034-1035) follows.
// -------------------------------------------------------------------------------------
// VDIF_Q in three passes.  The reference's column loop (one node at a time) has only two
// truly sequential parts, the tridiagonal sweeps of the q2 and q2l equations; everything
// else is per level.  k_vdif_q_levels forms, per (node, level), every input of the sweeps
// (the positivity fixes, BOYGR, the shear production PROD, the length scale L and its
// limits, GH, DTEF and the q2l wall-function DTEF); k_vdif_q_sweep runs the two sweeps per
// column; k_vdif_q_coef applies the stability functions per (node, level).  Each value is
// computed with the reference's expression, so the result is bitwise that of the column
// loop.
namespace vq {
constexpr double A1 = 0.92, B1 = 16.6, A2 = 0.74, B2 = 10.1, C1 = 0.08;
constexpr double E1 = 1.80, E2 = 1.33, SEF = 1.00, KAPPA = 0.40;
constexpr double SMALL = 1.e-8, GH_MAX = .0233, GH_MIN = -.281;
constexpr double SURFL = 2.e+5, GHC = -6.0;
}  // namespace vq

// Surface stress magnitude UTAU2 and bottom stress magnitude of node i (vdif_q.F:172-246),
// the NBVE means in ring order.
__device__ inline void vq_stress(const Dev& P, int i, double& utau2, double& wub, double& wvb) {
  const size_t m1 = P.M + 1;
  const int nt = P.ntve[i];
  double wus = 0.0, wvs = 0.0;
  wub = 0.0;
  wvb = 0.0;
  for (int j = 1; j <= nt; ++j) {
    int c = P.nbve[(size_t)(j - 1) * m1 + i];
    wus = wus + P.wusurf[c];
    wvs = wvs + P.wvsurf[c];
  }
  const double fn = (double)(float)nt;
  wus = wus / fn;
  wvs = wvs / fn;
  utau2 = sqrt(wus * wus + wvs * wvs);
  for (int j = 1; j <= nt; ++j) {
    int c = P.nbve[(size_t)(j - 1) * m1 + i];
    wub = wub + P.wubot[c];
    wvb = wvb + P.wvbot[c];
  }
  wub = wub / fn;
  wvb = wvb / fn;
}

// AUX bit 1: the learned closure's inputs are written (P.closure); bit 2: the closure
// samples (P.clos_samp).  Each combination is its own instantiation, so that the plain
// step carries none of the other paths' registers.  Every instantiation is held to 64
// registers (four blocks per SM): with the closure's inputs that spills 20 bytes, and
// still measured faster than 80 registers and three blocks (1.30 against 1.37 ms per
// step for VDIF_Q on the 200k-node mesh).
template <int AUX>
__global__ void __launch_bounds__(256, 4) k_vdif_q_levels(const Dev P) {
  using namespace vq;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) return;
  int kb, ke;
  col_range(P, 1, P.KB, kb, ke);
  const int KB = P.KB, KBM1 = P.KBM1;
  const double d = P.d[i];
  const bool wet = P.iswetn[i] == 1;
  double* Q2 = P.q2;
  double* Q2L = P.q2l;
  double* L = P.l;
  auto n3 = [&](int k) { return N3(P, i, k); };
  double utau2, wub, wvb;
  vq_stress(P, i, utau2, wub, wvb);
  const double l0 = SURFL * utau2 / P.grav_n[i];
  if (kb == 1) P.vq_ut[i] = utau2;
  if (ke == KB) P.q2f[n3(KB)] = sqrt(wub * wub + wvb * wvb) * P.const1;
  float* const cs = (AUX & 2) ? P.clos_samp : nullptr;
  const size_t ss = (size_t)P.M * (size_t)(KBM1 - 1);
  auto samp = [&](int f, int k, double v) { cs[(size_t)f * ss + (size_t)(k - 2) * P.M + (i - 1)] = (float)v; };
  // ring means of U, V on the level above the first interior level of the chunk
  const size_t m1 = P.M + 1;
  const int nt = P.ntve[i];
  const double fn = (double)(float)nt;
  auto ring_mean = [&](int k, double& um, double& vm) {
    double su = 0.0, sv = 0.0;
    for (int j = 1; j <= nt; ++j) {
      int c = P.nbve[(size_t)(j - 1) * m1 + i];
      su = su + P.u[C3(P, c, k)];
      sv = sv + P.v[C3(P, c, k)];
    }
    um = su / fn;
    vm = sv / fn;
  };
  double ukm1 = 0.0, vkm1 = 0.0;
  if (wet && kb <= KBM1) ring_mean(kb >= 2 ? kb - 1 : 1, ukm1, vkm1);
  bool chunk_inside = wet;  // every interior level of this chunk inside the closure's envelope
  double rhom = kb >= 2 ? P.rho1[n3(kb - 1)] : 0.0;  // RHO1 above the level
  for (int k = kb; k <= ke; ++k) {
    const size_t q = n3(k);
    const bool inner = k >= 2 && k <= KBM1;
    // the level's loads stand before its first store, which none of them could pass otherwise
    // (200 k nodes x 30 layers: VDIF_Q 839 -> 800 us)
    const double rho = P.rho1[q], q20 = Q2[q], q2l0 = Q2L[q];
    double q2f = 1.0, q2lf = 1.0, km = 0.0, kh = 0.0, uk = 0.0, vk = 0.0;
    if (inner) {
      q2f = P.q2f[q];
      q2lf = P.q2lf[q];
      km = P.km[q];
      kh = P.kh[q];
      if (wet) ring_mean(k, uk, vk);
    }
    // positivity of the previous Q2F/Q2LF (vdif_q.F:144-149)
    if (inner && (q2f <= SMALL || q2lf <= SMALL)) {
      P.q2f[q] = SMALL;
      P.q2lf[q] = SMALL;
    }
    const double q2 = fabs(q20 + SMALL);
    double q2l = fabs(q2l0);
    Q2[q] = q2;
    double boygr = 0.0, prod = 0.0, lk;
    if (k >= 2 && k <= KBM1) {
      if (wet) {
        const double den = P.dzz(i, k - 1) * d;
        boygr = P.grav_n[i] * (rhom - rho) / den;
        // the reference's internal-wave term carries a weight of zero and is not evaluated
        const double shear2 = ((uk - ukm1) * (uk - ukm1) + (vk - vkm1) * (vk - vkm1)) / (den * den);
        if (AUX & 1) {
          // the network's inputs: inside the envelope or not, then transformed,
          // standardised and rounded to BF16 as the MMA takes them
          const float fv[CLOS_IN] = {(float)boygr, (float)shear2, (float)d, (float)P.z(i, k), (float)sqrt(utau2),
                                     (float)sqrt(sqrt(wub * wub + wvb * wvb)), (float)q2, (float)q2l};
          uint32_t packed[4];
          for (int f = 0; f < CLOS_IN; ++f) {
            if (!(fv[f] >= P.clos_norm.lo[f] && fv[f] <= P.clos_norm.hi[f])) chunk_inside = false;
          }
          for (int f = 0; f < CLOS_IN; f += 2) {
            const __nv_bfloat162 b = __floats2bfloat162_rn(clos_feat_transform(P.clos_norm, f, fv[f]),
                                                           clos_feat_transform(P.clos_norm, f + 1, fv[f + 1]));
            packed[f / 2] = *reinterpret_cast<const uint32_t*>(&b);
          }
          P.clos_feat[(size_t)(k - 2) * P.M + (i - 1)] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        }
        if (AUX & 2) {
          samp(0, k, boygr);
          samp(1, k, shear2);
          samp(2, k, d);
          samp(3, k, P.z(i, k));
          samp(4, k, sqrt(utau2));
          samp(5, k, sqrt(sqrt(wub * wub + wvb * wvb)));
          samp(6, k, q2);
          samp(7, k, q2l);
        }
        prod = km * SEF * ((uk - ukm1) * (uk - ukm1) + (vk - vkm1) * (vk - vkm1)) / (den * den);
        prod = prod + kh * boygr;
        ukm1 = uk;
        vkm1 = vk;
      }
      // length scale and its limits (vdif_q.F:300-331)
      lk = q2l / q2;
      if (P.z(i, k) > -0.5) lk = fmax(lk, KAPPA * l0);
      if (boygr < 0.0) {
        double lmax = sqrt(fabs(GH_MIN) * q2 / (-boygr + SMALL));
        lk = fmin(lk, lmax);
        q2l = q2 * lk;
      }
    } else {
      lk = k == 1 ? KAPPA * l0 : 0.0;
    }
    Q2L[q] = q2l;
    L[q] = lk;
    double gh = 0.0;
    if (k >= 2 && k <= KBM1) gh = fmin((lk * lk / q2) * boygr, GH_MAX);
    double stf = 1.0;
    if (gh < 0.0) stf = 1.0 - F4(0.9) * pow(gh / GHC, 1.5);
    if (gh < GHC) stf = F4(0.1);
    const double dtef = sqrt(q2) / (B1 * lk + SMALL) * stf;
    P.vq_prod[q] = prod;
    P.vq_gh[q] = gh;
    P.vq_stf[q] = stf;
    P.vq_dtef[q] = dtef;
    rhom = rho;
    if (wet && k >= 2 && k <= KBM1) {
      const double x = (1. / fabs(P.z(i, k) - P.z(i, 1)) + 1. / fabs(P.z(i, k) - P.z(i, KB))) * lk / (d * KAPPA);
      P.vq_dtefl[q] = dtef * (1. + E2 * (x * x));
    }
  }
  if (AUX & 1) P.clos_envc[(size_t)blockIdx.y * (P.M + 1) + i] = chunk_inside ? 1 : 0;
}

// The q2 and q2l tridiagonal sweeps of one column (vdif_q.F:372-431), and the column's
// envelope flag of the learned closure.  The two sweeps are independent: blockIdx.y = 0
// runs the q2 sweep, 1 the q2l sweep.  The forward elimination loads the coefficients of
// four levels before it runs their (serial) recurrence.
__global__ void __launch_bounds__(128) k_vdif_q_sweep(const Dev P) {
  using namespace vq;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) return;
  const int KB = P.KB, KBM1 = P.KBM1;
  const double DTI = P.dti;
  const double d = P.d[i];
  const bool wet = P.iswetn[i] == 1;
  const bool q2l = blockIdx.y == 1;
  auto n3 = [&](int k) { return N3(P, i, k); };
  if (P.closure && !q2l) {
    // the column's envelope flag from the level kernel's per-chunk flags
    bool in_env = wet;
    const int nch = (P.KB + P.col_lc - 1) / P.col_lc;
    for (int c = 0; c < nch && in_env; ++c) in_env = P.clos_envc[(size_t)c * (P.M + 1) + i] != 0;
    P.clos_env[i] = in_env ? 1 : 0;
  }
  if (!wet) return;
  double vh[kMaxKBs], vhp[kMaxKBs];
  vh[1] = 0.0;
  vhp[1] = q2l ? 0.0 : P.vhp1c * P.vq_ut[i];
  double* QF = q2l ? P.q2lf : P.q2f;
  // the coefficients of level k: A, C, the diagonal term and the source of the equation
  auto coef = [&](int k, double& a, double& c, double& e, double& r, double& qf) {
    a = -0.5 * DTI * (P.kq[n3(k + 1)] + P.kq[n3(k)] + 2.0 * P.umol) / (P.dzz(i, k - 1) * P.dz(i, k) * d * d);
    c = -0.5 * DTI * (P.kq[n3(k - 1)] + P.kq[n3(k)] + 2.0 * P.umol) / (P.dzz(i, k - 1) * P.dz(i, k - 1) * d * d);
    if (q2l) {
      e = DTI * P.vq_dtefl[n3(k)] + 1.;
      r = DTI * (-P.vq_prod[n3(k)] * P.l[n3(k)] * E1);
    } else {
      e = 2. * DTI * P.vq_dtef[n3(k)] + 1.;
      r = -2. * DTI * P.vq_prod[n3(k)];
    }
    qf = QF[n3(k)];
  };
  auto step = [&](int k, double a, double c, double e, double r, double qf) {
    const double p = 1. / (a + c * (1. - vh[k - 1]) - e);
    vh[k] = a * p;
    vhp[k] = (r + c * vhp[k - 1] - qf) * p;
  };
  int k = 2;
  for (; k + 3 <= KBM1; k += 4) {
    double a[4], c[4], e[4], r[4], qf[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) coef(k + u, a[u], c[u], e[u], r[u], qf[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u) step(k + u, a[u], c[u], e[u], r[u], qf[u]);
  }
  for (; k <= KBM1; ++k) {
    double a, c, e, r, qf;
    coef(k, a, c, e, r, qf);
    step(k, a, c, e, r, qf);
  }
  for (int k = 1; k <= KBM1; ++k) {
    int ki = KB - k;
    QF[n3(ki)] = vh[ki] * QF[n3(ki + 1)] + vhp[ki];
  }
}

// Positivity of the new Q2F/Q2LF, the stability functions and KQ, KM, KH
// (vdif_q.F:443-491), per (node, level); then Q2 = Q2F, Q2L = Q2LF.  AUX as for
// k_vdif_q_levels; with the learned closure the interior levels of a column on the network
// skip the stability functions, which k_closure_mlp replaces.
template <int AUX>
__global__ void __launch_bounds__(256) k_vdif_q_coef(const Dev P, int copy_back) {
  using namespace vq;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) return;
  int kb, ke;
  col_range(P, 1, P.KB, kb, ke);
  const int KBM1 = P.KBM1;
  const double COEF4 = 18.0 * A1 * A1 + 9.0 * A1 * A2;
  const double COEF5 = 9.0 * A1 * A2;
  const bool wet = P.iswetn[i] == 1;
  float* const cs = (AUX & 2) ? P.clos_samp : nullptr;
  const size_t ss = (size_t)P.M * (size_t)(KBM1 - 1);
  auto samp = [&](int f, int k, double v) { cs[(size_t)f * ss + (size_t)(k - 2) * P.M + (i - 1)] = (float)v; };
  // interior levels of a column inside the envelope are finished by the network kernel
  // (k_closure_mlp); every other column keeps MY2.5 here
  const bool on_network = (AUX & 1) && P.clos_env[i] != 0;
  for (int k = kb; k <= ke; ++k) {
    const size_t q = N3(P, i, k);
    if (k >= 2 && k <= KBM1 && (P.q2f[q] <= SMALL || P.q2lf[q] <= SMALL)) {
      P.q2f[q] = SMALL;
      P.q2lf[q] = SMALL;
    }
    if (!(AUX & 2) && on_network && k >= 2 && k <= KBM1) {
      if (copy_back) {
        P.q2[q] = P.q2f[q];
        P.q2l[q] = P.q2lf[q];
      }
      continue;
    }
    const double gh = P.vq_gh[q];
    const double stf = P.vq_stf[q];
    double coef1 = A2 * (1.0 - 6.0 * A1 / B1 * stf);
    double coef2 = 3.0 * A2 * B2 / stf + 18.0 * A1 * A2;
    double coef3 = A1 * (1.0 - 3.0 * C1 - 6.0 * A1 / B1 * stf);
    double sh = coef1 / (1.0 - coef2 * gh);
    double sm = (coef3 + sh * COEF4 * gh) / (1. - COEF5 * gh);
    double kn = P.l[q] * sqrt(P.q2[q]);
    bool interior_by_network = false;
    if (k >= 2 && k <= KBM1) {
      if (AUX & 2) {
        samp(8, k, kn * KAPPA * sm);
        samp(9, k, kn * sm);
        samp(10, k, kn * sh * P.vprnu);
        samp(11, k, wet ? 1.0 : 0.0);
      }
      interior_by_network = on_network;
    }
    if (!interior_by_network) {
      P.kq[q] = 0.5 * (kn * KAPPA * sm + P.kq[q]);
      P.km[q] = 0.5 * (kn * sm + P.km[q]);
      P.kh[q] = 0.5 * (kn * sh * P.vprnu + P.kh[q]);
    }
    if (copy_back) {
      P.q2[q] = P.q2f[q];
      P.q2l[q] = P.q2lf[q];
    }
  }
}

// Q2=Q2F, Q2L=Q2LF on every node and level; N2E3D(KM,KM1) (internal_step.F:1034-1053).
__global__ void __launch_bounds__(256) k_turb_update(const Dev P) {
  int i = blockIdx.x * 32 + threadIdx.x;
  int k = blockIdx.y * 8 + threadIdx.y + 1;
  if (k > P.KB) return;
  if (i <= P.M) {
    size_t q = N3(P, i, k);
    P.q2[q] = P.q2f[q];
    P.q2l[q] = P.q2lf[q];
  }
  if (i >= 1 && i <= P.N) {
    const size_t n1 = P.N + 1;
    P.km1[C3(P, i, k)] = ONE_THIRD * (P.km[N3(P, P.nv[i], k)] + P.km[N3(P, P.nv[n1 + i], k)] + P.km[N3(P, P.nv[2 * n1 + i], k)]);
  }
}

// -------------------------------------------------------------------------------------
// Phase 2 of ADV_T / ADV_S (adv_t.F:124-1042, adv_s.F) with FCT_T / FCT_S (fct_t.F:51-104,
// fct_s.F:50-108) on the same (node, layer) thread.
// -------------------------------------------------------------------------------------
template <typename R>
__global__ void __launch_bounds__(kGatherThreads, sizeof(R) == 4 ? 6 : 4) k_gather_ts(const Dev P, int parts) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) return;
  int kb, ke;
  col_range(P, 1, P.KBM1, kb, ke);
  if (kb > ke) return;
  const bool wet = P.iswetn[i] * P.iswetnt[i] == 1;
  const bool fct = (parts & AD_FCT) && !P.riv_skip[i];
  const bool open = P.isonb[i] == 2;
  const int nhe = P.node_he_ptr[i + 1] - P.node_he_ptr[i], KBM1 = P.KBM1;
  const double art1 = P.art1[i], dt = P.dt[i], dr = dt / P.dtfa[i];
  const bool on[2] = {(parts & AD_T) != 0, (parts & AD_S) != 0};
  const double* F1[2] = {P.t1, P.s1};
  double* FF1[2] = {P.tf1, P.sf1};
  // f, fp: the tracer on layers k and k+1; face, flux: the value on the interface between layers
  // k-1 and k and the vertical flux through it, layer k-1's lower and layer k's upper ones
  double f[2], face[2] = {0.0, 0.0}, flux[2] = {0.0, 0.0};
  {
    const size_t q = N3(P, i, kb);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!on[t]) continue;
      f[t] = F1[t][q];
      if (kb > 1) {
        const double z = P.dz(i, kb), zm = P.dz(i, kb - 1);
        const double sum = f[t] * zm + F1[t][N3(P, i, kb - 1)] * z;
        face[t] = sum / (z + zm);
        flux[t] = P.wts[q] * sum / (z + zm);
      }
    }
  }
  for (int k = kb; k <= ke; ++k) {
    const size_t q = N3(P, i, k), qp = N3(P, i, k + 1);
    const double z = P.dz(i, k), zp = k < KBM1 ? P.dz(i, k + 1) : 0.0;
    const bool lower = k == 1 || k < KBM1;
    const double wp = lower ? P.wts[qp] : 0.0;
    double fp[2], fmn[2], fmx[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!on[t]) continue;
      fp[t] = lower ? F1[t][qp] : 0.0;
      if (fct) NodeRec<R>::minmax(P, 1, t, q, fmn[t], fmx[t]);
    }
    const double2 xs = gather_he<R>(P, i, nhe, k);
    const double rt = P.dti / (dt * z);
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      if (!on[t]) continue;
      double x = t == 0 ? xs.x : xs.y;
      const double up = flux[t], fa = face[t];
      if (lower) {
        const double sum = f[t] * zp + fp[t] * z;
        face[t] = sum / (z + zp);
        flux[t] = wp * sum / (z + zp);
      }
      double ff = f[t];
      if (wet) {
        const double temp = k == 1 ? -flux[t] : (lower ? up - flux[t] : up);
        if (open)
          x = temp * art1;
        else
          x = x + temp * art1;
        ff = (f[t] - x / art1 * rt) * dr;
      }
      if (fct) {
        if (k > 1) {
          fmx[t] = fmax(fmx[t], fa);
          fmn[t] = fmin(fmn[t], fa);
        }
        if (lower) {
          fmx[t] = fmax(fmx[t], face[t]);
          fmn[t] = fmin(fmn[t], face[t]);
        }
        if (fmn[t] - ff > 0.0) ff = fmn[t];
        if (ff - fmx[t] > 0.0) ff = fmx[t];
      }
      if ((parts & AD_FCT) && t == 1 && ff < 0.0) ff = 0.0;
      FF1[t][q] = ff;
      f[t] = fp[t];
    }
  }
}

// FCT_T / FCT_S alone (fct_t.F:51-104, fct_s.F:50-108) on TF1/SF1 in memory.
__global__ void __launch_bounds__(256) k_fct_ts(const Dev P, int parts) {
  int i = blockIdx.x * 32 + threadIdx.x + 1;
  int k = blockIdx.y * 8 + threadIdx.y + 1;
  if (i > P.M || k > P.KBM1) return;
  for (int t = 0; t < 2; ++t) {
    if (!(parts & (t == 0 ? AD_T : AD_S))) continue;
    const double* F1 = (t == 0 ? P.t1 : P.s1);
    double* FF1 = (t == 0 ? P.tf1 : P.sf1);
    size_t q = N3(P, i, k);
    double ff = FF1[q];
    if (!P.riv_skip[i]) {
      double fmx = F1[N3(P, NBSN(P, i, 1), k)], fmn = fmx;
      for (int j = 2; j <= P.ntsn[i]; ++j) {
        double v = F1[N3(P, NBSN(P, i, j), k)];
        fmx = fmax(fmx, v);
        fmn = fmin(fmn, v);
      }
      fct_layer_bounds(P, i, k, F1, fmx, fmn);
      if (fmn - ff > 0.0) ff = fmn;
      if (ff - fmx > 0.0) ff = fmx;
    }
    if (t == 1 && ff < 0.0) ff = 0.0;
    FF1[q] = ff;
  }
}

// -------------------------------------------------------------------------------------
// VDIF_TS(1,TF1) and VDIF_TS(2,SF1) (vdif_ts.F:78-337), one thread per node column and
// tracer (blockIdx.y 0: T, 1: S).
// With surface heating (HEATING_TYPE 'flux', vdif_ts.F:118-150) the temperature column
// takes the net heat flux WTSURF, held at zero while cooling water at or below -2 C,
// and the short-wave flux RAD(K) = SWRAD*(RHEAT*EXP(Z*D/ZETA1) + (1-RHEAT)*EXP(Z*D/ZETA2))
// absorbed between levels; WTSURF and SWRAD are the forcing in W/m^2 times RAMP over
// -SPCP*ROSEA (BCOND_GCN(8), bcond_gcn.F:683-694).  Without heating every term is zero
// and the kernel is instantiated without them (HEAT = false).
// -------------------------------------------------------------------------------------
template <bool HEAT>
__global__ void __launch_bounds__(128) k_vdif_ts(const Dev P, int parts) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M || P.iswetn[i] != 1) return;
  const int KB = P.KB, KBM1 = P.KBM1, KBM2 = P.KBM2;
  const double DTI = P.dti, UMOLPR = P.umol * 1.e0, GW = 0.0;
  const double d = P.d[i];
  auto n3 = [&](int k) { return N3(P, i, k); };
  auto AF = [&](int k) { double fkh = P.kh[n3(k + 1)]; return -DTI * (fkh + UMOLPR) / (P.dz(i, k) * P.dzz(i, k) * d * d); };
  auto CF = [&](int k) { double fkh = P.kh[n3(k)]; return -DTI * (fkh + UMOLPR) / (P.dz(i, k) * P.dzz(i, k - 1) * d * d); };
  const double khbottom = P.kh[n3(KBM1)];
  const bool update = P.iswetn[i] * P.iswetnt[i] == 1;
  {
    const int t = blockIdx.y;  // 0: temperature, 1: salinity (independent columns)
    if (!(parts & (t == 0 ? AD_T : AD_S))) return;
    double* F = (t == 0 ? P.tf1 : P.sf1);
    double vhf[kMaxKBs], vhpf[kMaxKBs];
    const double sasurf = 0.0;
    double wfsurf = 0.0, swradf = 0.0;
    const bool heat = HEAT && t == 0;
    if (heat) {
      const double spro = 4.2174E3 * 1.023E3;
      const double ramp = ramp_int(P);
      wfsurf = -(P.wtsurf_w[i] * ramp) / spro;
      swradf = -(P.swrad_w[i] * ramp) / spro;
      const double wftmp1 = -2.0, wftmp2 = wfsurf;
      const double wftmp3 = 0.5 * (1.0 + fsign1(wftmp1 - F[n3(1)]));
      wfsurf = wftmp2 - wftmp3 * 0.5 * (wftmp2 + fabs(wftmp2));
    }
    // RAD at level k; zero without heating
    auto RAD = [&](int k) {
      if (!heat) return 0.0;
      const double zdep = P.z(i, k) * d;
      return swradf * (P.rheat * exp(zdep / P.zeta1) + (1 - P.rheat) * exp(zdep / P.zeta2));
    };
    double rad_k = RAD(1), rad_k1 = RAD(2);
    double af1 = AF(1);
    vhf[1] = af1 / (af1 - 1.);
    vhpf[1] = -DTI * (sasurf + wfsurf - swradf + rad_k - rad_k1) / (-P.dz(i, 1) * d) - F[n3(1)];
    vhpf[1] = vhpf[1] / (af1 - 1.);
    // level k's coefficients and source, then its step of the (serial) recurrence; the
    // loads of four levels are issued before their steps
    auto coef = [&](int k, double& af, double& cf, double& fk, double& r) {
      rad_k = rad_k1;
      rad_k1 = RAD(k + 1);
      af = AF(k);
      cf = CF(k);
      fk = F[n3(k)];
      r = DTI * (rad_k - rad_k1) / (d * P.dz(i, k));
    };
    auto step = [&](int k, double af, double cf, double fk, double r) {
      double p = 1. / (af + cf * (1. - vhf[k - 1]) - 1.);
      vhf[k] = af * p;
      vhpf[k] = (cf * vhpf[k - 1] - fk + r) * p;
    };
    int k = 2;
    for (; k + 3 <= KBM2; k += 4) {
      double af[4], cf[4], fk[4], r[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) coef(k + u, af[u], cf[u], fk[u], r[u]);
#pragma unroll
      for (int u = 0; u < 4; ++u) step(k + u, af[u], cf[u], fk[u], r[u]);
    }
    for (; k <= KBM2; ++k) {
      double af, cf, fk, r;
      coef(k, af, cf, fk, r);
      step(k, af, cf, fk, r);
    }
    if (P.isonb[i] != 2 && update) {
      double pfx = t == 0 ? P.pfpxb_t[i] : P.pfpxb_s[i];
      double pfy = t == 0 ? P.pfpyb_t[i] : P.pfpyb_s[i];
      double ah = t == 0 ? P.ah_bottom_t[i] : P.ah_bottom_s[i];
      double tmp1 = pfx * P.cos_sita[i] + pfy * P.sin_sita[i];
      double tmp2 = ah * P.phpn[i];
      double tmp3 = khbottom + UMOLPR + ah * P.phpn[i] * P.phpn[i];
      double tmp = tmp1 * tmp2 / tmp3 * (khbottom + UMOLPR);
      if (t == 0) {
        if (tmp1 > 0.0) tmp = 0.0;
      } else {
        if (tmp1 < 0.0) tmp = 0.0;
        tmp = -tmp;
      }
      double cfb = CF(KBM1);
      const double rad_b = RAD(KBM1), rad_kb = RAD(KB);
      double ff = (cfb * vhpf[KBM2] - F[n3(KBM1)] - GW + DTI * (rad_b - rad_kb - tmp) / (d * P.dz(i, KBM1))) /
                  (cfb * (1. - vhf[KBM2]) - 1.);
      F[n3(KBM1)] = ff;
      for (int k = 2; k <= KBM1; ++k) {
        int ki = KB - k;
        ff = (vhf[ki] * ff + vhpf[ki]);
        F[n3(ki)] = ff;
      }
    }
  }
}

// -------------------------------------------------------------------------------------
// BCOND_TS(1) and BCOND_TS(2) (bcond_ts.F:60-262): river nodes take the river T/S; open
// boundary nodes take the outflow estimate with the radiation perturbation of
// OBC_TS_TYPE and the neighbour clamp, or keep T1/S1 on inflow.
// -------------------------------------------------------------------------------------
// One block per layer, its threads over the rivers; a node of several rivers is the last one's
// (riv_ts).
__global__ void k_bcond_ts_riv(const Dev P) {
  const int k = blockIdx.x + 1;
  for (int r = threadIdx.x + 1; r <= P.numqbc; r += blockDim.x) {
    const int2 n = P.riv_ts[r];
    const double t = P.tdis[r], s = P.sdis[r];
    if (n.x > 0) {
      P.tf1[N3(P, n.x, k)] = t;
      P.sf1[N3(P, n.x, k)] = s;
    }
    if (n.y > 0) {
      P.tf1[N3(P, n.y, k)] = t;
      P.sf1[N3(P, n.y, k)] = s;
    }
  }
}

// Open-boundary part: one block per (open-boundary node, tracer), one thread per layer.
// The nodes are independent: each reads the old field, its own XFLUX_OBC and TF1/SF1 of
// its interior neighbour NEXT_OBC, which is not an open-boundary node.  Only the three
// depth sums are sequential: the layers' terms go through shared memory and three threads
// add them in layer order, one sum each.
__global__ void __launch_bounds__(64) k_bcond_ts_obc(const Dev P, int parts) {
  __shared__ double term[3][64];
  __shared__ double sum[3];
  const int KBM1 = P.KBM1;
  const int ob = blockIdx.x + 1, t = blockIdx.y, k = threadIdx.x + 1;
  if (!(parts & (t == 0 ? AD_T : AD_S))) return;
  const int j = P.i_obc_n[ob], j1 = P.next_obc[ob];
  const double* F1 = t == 0 ? P.t1 : P.s1;
  double* FF1 = t == 0 ? P.tf1 : P.sf1;
  const double* XO = t == 0 ? P.xflux_obc_t : P.xflux_obc_s;
  const bool live = k <= KBM1;
  const size_t q = N3(P, j, k), q1 = N3(P, j1, k);
  if (!(P.uard_obcn[ob] > 0.0)) {
    if (live) FF1[q] = F1[q];
    return;
  }
  double f1 = 0.0, fnext = 0.0;
  if (live) {
    f1 = F1[q];
    fnext = FF1[q1];
    term[0][k - 1] = f1 * P.dz(j, k);
    term[1][k - 1] = fnext * P.dz(j1, k);
    term[2][k - 1] = XO[(size_t)(k - 1) * (P.iobcn + 1) + ob];
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double s = 0.0;
    for (int l = 0; l < KBM1; ++l) s = s + term[threadIdx.x][l];
    sum[threadIdx.x] = s;
  }
  __syncthreads();
  if (!live) return;
  const double t2d = sum[0], t2dn = sum[1], xf2d = sum[2];
  const double tmp = xf2d + t2d * P.uard_obcn[ob];
  const double t2d_obc = (t2d * P.dt[j] - tmp * P.dti / P.art1[j]) / P.d[j];
  double cc = 0.0, cp = 1.0;
  if (P.obc_ts_type != 1) {
    cc = sqrt(P.grav_n[j] * P.h[j]) * P.dti / P.dltn_obc[ob];
    cp = cc + 1.0;
  }
  double ttmp;
  const double pert_next = fnext - t2dn;
  if (P.obc_ts_type == 1) {
    ttmp = pert_next;
  } else if (P.obc_ts_type == 2) {
    const double pert = f1 - t2d;
    ttmp = (cc * pert_next + pert) / cp;
  } else {
    const double pert = f1 - t2d;
    ttmp = (cc * pert_next + pert * (1.0 - P.dti / 10800.0)) / cp;
  }
  double ff = t2d_obc + ttmp;
  double fmx = F1[N3(P, NBSN(P, j, 1), k)], fmn = fmx;
  for (int jj = 2; jj <= P.ntsn[j]; ++jj) {
    const double v = F1[N3(P, NBSN(P, j, jj), k)];
    fmx = fmax(fmx, v);
    fmn = fmin(fmn, v);
  }
  fct_layer_bounds(P, j, k, F1, fmx, fmn);
  if (fmn - ff > 0.0) ff = fmn;
  if (ff - fmx > 0.0) ff = fmx;
  FF1[q] = ff;
}

// DENS2_2D (eqs_of_state.F:290-319), same operation order.
__device__ inline double dens2(double S, double T) {
  double r = S * S * S * 6.76786136E-6 - S * S * 4.8249614E-4 + S * 8.14876577E-1 - 0.22584586E0;
  r = r * (T * T * T * 1.667E-8 - T * T * 8.164E-7 + T * 1.803E-5);
  r = r + 1.0 - T * T * T * 1.0843E-6 + T * T * 9.8185E-5 - T * 4.786E-3;
  r = r * (S * S * S * 6.76786136E-6 - S * S * 4.8249614E-4 + S * 8.14876577E-1 + 3.895414E-2);
  r = r - (T - 3.98) * (T - 3.98) * (T + 283.0) / (503.57 * (T + 67.26));
  return r * 1.e-3;
}

// -------------------------------------------------------------------------------------
// End of the internal step: T1=TF1, S1=SF1, N2E3D to T/S, DENS2 with N2E3D(RHO1,RHO),
// N2E3D(KM,KM1), U=UF, V=VF, ET=EL, DT=D, ET1=EL1, DT1=D1, WD_UPDATE(3)
// (internal_step.F:1053-1590).  Threads over (max(M,N)+1) x KB, or over the nodes alone
// (cells = 0) where k_final_cells follows.
// -------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_final(const Dev P, int parts, int cells) {
  int i = blockIdx.x * 32 + threadIdx.x;
  int k = blockIdx.y * 8 + threadIdx.y + 1;
  if (k > P.KB) return;
  const double* Tn = (parts & FI_T) ? P.tf1 : P.t1;
  const double* Sn = (parts & FI_S) ? P.sf1 : P.s1;
  if (i <= P.M) {
    size_t q = N3(P, i, k);
    if (parts & FI_T) P.t1[q] = P.tf1[q];
    if (parts & FI_S) P.s1[q] = P.sf1[q];
    if (parts & FI_DENS) P.rho1[q] = (k == P.KB || i == 0) ? 0.0 : dens2(Sn[q], Tn[q]);
    if ((parts & FI_SHIFT) && k == 1) {
      P.et[i] = P.el[i];
      P.dt[i] = P.d[i];
      if (P.wetting_drying_on) P.iswetnt[i] = P.iswetn[i];
    }
  }
  if (cells && i >= 1 && i <= P.N) {
    const size_t n1 = P.N + 1;
    int a = P.nv[i], b = P.nv[n1 + i], c = P.nv[2 * n1 + i];
    size_t qa = N3(P, a, k), qb = N3(P, b, k), qc = N3(P, c, k);
    size_t q = C3(P, i, k);
    if (parts & FI_T) P.t[q] = ONE_THIRD * (P.tf1[qa] + P.tf1[qb] + P.tf1[qc]);
    if (parts & FI_S) P.s[q] = ONE_THIRD * (P.sf1[qa] + P.sf1[qb] + P.sf1[qc]);
    if (parts & FI_DENS) {
      double ra = k == P.KB ? 0.0 : dens2(Sn[qa], Tn[qa]);
      double rb = k == P.KB ? 0.0 : dens2(Sn[qb], Tn[qb]);
      double rc = k == P.KB ? 0.0 : dens2(Sn[qc], Tn[qc]);
      P.rho[q] = ONE_THIRD * (ra + rb + rc);
    }
    if (parts & FI_KM1) P.km1[q] = ONE_THIRD * (P.km[qa] + P.km[qb] + P.km[qc]);
    if (parts & FI_SHIFT) {
      P.u[q] = P.uf[q];
      P.v[q] = P.vf[q];
      if (k == 1) {
        P.et1[i] = P.el1[i];
        P.dt1[i] = P.d1[i];
        if (P.wetting_drying_on) P.iswetct[i] = P.iswetc[i];
      }
    }
  }
}

// The cells' part of k_final alone, after k_final has written RHO1: one thread per cell walks a
// chunk of levels, the inputs of kFinBat levels loaded before they are stored.  In one kernel
// a cell cannot read RHO1 that another block writes and evaluates the density of its three
// nodes itself, seven evaluations per node instead of one, which bound it (98 us at 50 k nodes x 30
// layers for about 270 MB, 41 us at the copy rate).  kFinSplit: from this many cells x levels
// on the second launch pays.  One kernel and two: 4 k cells x 11 levels 10.2 and 11.6 us, 12 k x 24
// 16.8 and 19.4, 39 k x 20 33.0 and 27.7, 99 k x 31 98 and 77, 396 k x 31 398 and 279.
constexpr int kFinBat = 2;
constexpr long kFinSplit = 500000;
__global__ void __launch_bounds__(128) k_final_cells(const Dev P, int parts) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.N) return;
  int kb, ke;
  col_range(P, 1, P.KB, kb, ke);
  const size_t n1 = P.N + 1;
  const int nd[3] = {P.nv[i], P.nv[n1 + i], P.nv[2 * n1 + i]};
  const bool ft = parts & FI_T, fs = parts & FI_S, fd = parts & FI_DENS, fk = parts & FI_KM1, fu = parts & FI_SHIFT;
  for (int k0 = kb; k0 <= ke; k0 += kFinBat) {
    double t[kFinBat][3], s[kFinBat][3], r[kFinBat][3], m[kFinBat][3], u[kFinBat], v[kFinBat];
#pragma unroll
    for (int b = 0; b < kFinBat; ++b) {
      const int k = k0 + b <= ke ? k0 + b : ke;
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const size_t q = N3(P, nd[j], k);
        if (ft) t[b][j] = P.tf1[q];
        if (fs) s[b][j] = P.sf1[q];
        if (fd) r[b][j] = P.rho1[q];
        if (fk) m[b][j] = P.km[q];
      }
      if (fu) {
        u[b] = P.uf[C3(P, i, k)];
        v[b] = P.vf[C3(P, i, k)];
      }
    }
#pragma unroll
    for (int b = 0; b < kFinBat; ++b) {
      if (k0 + b > ke) break;
      const size_t q = C3(P, i, k0 + b);
      if (ft) P.t[q] = ONE_THIRD * (t[b][0] + t[b][1] + t[b][2]);
      if (fs) P.s[q] = ONE_THIRD * (s[b][0] + s[b][1] + s[b][2]);
      if (fd) P.rho[q] = ONE_THIRD * (r[b][0] + r[b][1] + r[b][2]);
      if (fk) P.km1[q] = ONE_THIRD * (m[b][0] + m[b][1] + m[b][2]);
      if (fu) {
        P.u[q] = u[b];
        P.v[q] = v[b];
      }
    }
  }
  if (fu && kb == 1) {
    P.et1[i] = P.el1[i];
    P.dt1[i] = P.d1[i];
    if (P.wetting_drying_on) P.iswetct[i] = P.iswetc[i];
  }
}

// FP64 budgets over node control volumes, fixed-order two-level reduction.
__global__ void k_budget_partial(const Dev P, double* part) {
  __shared__ double sv[256], sh[256], ss[256];
  int tid = threadIdx.x;
  double v = 0.0, hh = 0.0, s = 0.0;
  for (int i = blockIdx.x * blockDim.x + tid + 1; i <= P.M; i += gridDim.x * blockDim.x) {
    double dd = P.d[i] * P.art1[i];
    double ct = 0.0, cs = 0.0;
    for (int k = 1; k <= P.KBM1; ++k) {
      ct = ct + P.t1[N3(P, i, k)] * P.dz(i, k);
      cs = cs + P.s1[N3(P, i, k)] * P.dz(i, k);
    }
    v = v + dd;
    hh = hh + ct * dd;
    s = s + cs * dd;
  }
  sv[tid] = v; sh[tid] = hh; ss[tid] = s;
  __syncthreads();
  for (int st = 128; st > 0; st >>= 1) {
    if (tid < st) { sv[tid] += sv[tid + st]; sh[tid] += sh[tid + st]; ss[tid] += ss[tid + st]; }
    __syncthreads();
  }
  if (tid == 0) { part[3 * blockIdx.x] = sv[0]; part[3 * blockIdx.x + 1] = sh[0]; part[3 * blockIdx.x + 2] = ss[0]; }
}
__global__ void k_budget_final(const double* part, int nb, double* out) {
  if (threadIdx.x != 0) return;
  double a = 0.0, b = 0.0, c = 0.0;
  for (int j = 0; j < nb; ++j) { a += part[3 * j]; b += part[3 * j + 1]; c += part[3 * j + 2]; }
  out[0] = a; out[1] = b; out[2] = c;
}

void launch_grad(const Dev& P, cudaStream_t s, int which) {
  FVG_F32_FORWARD(launch_grad(P, s, which));
  const int nl = which == 0 ? P.KBM1 - 1 : P.KBM1;
  const Dev Q = col_shape(P, P.M, nl);
  k_grad<RF><<<col_grid(Q, P.M, nl), Q.col_bc, 0, s>>>(Q, which);
}
void launch_adv_q(const Dev& P, cudaStream_t s, int parts) {
  FVG_F32_FORWARD(launch_adv_q(P, s, parts));
  const int nl = P.KBM1 - 1;
  Dev Q = col_shape(P, P.N, nl);
  if (Q.col_bc > kHeThreads) Q.col_bc = kHeThreads;
  Dev G = col_shape(P, P.M, nl);
  if (G.col_bc > kGatherThreads) G.col_bc = kGatherThreads;
  ((P.closed & 2) ? k_he_adv<RF, 0> : k_he_adv_listed<RF, 0>)<<<col_grid(Q, P.N, nl), Q.col_bc, 0, s>>>(Q, parts);
  k_gather_q<RF><<<col_grid(G, P.M, nl), G.col_bc, 0, s>>>(G, parts);
}
void launch_fct_q(const Dev& P, cudaStream_t s, int parts) {
  dim3 b(32, 8), g(nblk(P.M, 32), nblk(P.KBM1 - 1, 8));
  k_fct_q<<<g, b, 0, s>>>(P, parts);
}
void launch_vdif_q(const Dev& P, cudaStream_t s, int copy_back) {
  const int aux = (P.closure ? 1 : 0) | (P.clos_samp ? 2 : 0);
  void (*lv)(const Dev) = aux == 0 ? k_vdif_q_levels<0> : aux == 1 ? k_vdif_q_levels<1>
                        : aux == 2 ? k_vdif_q_levels<2> : k_vdif_q_levels<3>;
  void (*cf)(const Dev, int) = aux == 0 ? k_vdif_q_coef<0> : aux == 1 ? k_vdif_q_coef<1>
                             : aux == 2 ? k_vdif_q_coef<2> : k_vdif_q_coef<3>;
  const Dev Q = col_shape(P, P.M, P.KB);  // one shape: the sweep reads the level kernel's chunk flags
  const int b = col_threads(P, P.M, 128);
  lv<<<col_grid(Q, P.M, P.KB), Q.col_bc, 0, s>>>(Q);
  k_vdif_q_sweep<<<dim3(nblk(P.M, b), 2), b, 0, s>>>(Q);
  cf<<<col_grid(Q, P.M, P.KB), Q.col_bc, 0, s>>>(Q, copy_back);
  if (!P.closure) launch_vdif_q_shallow(P, s);
}
void launch_turb_update(const Dev& P, cudaStream_t s) {
  int n = (P.M > P.N ? P.M : P.N) + 1;
  dim3 b(32, 8), g(nblk(n, 32), nblk(P.KB, 8));
  k_turb_update<<<g, b, 0, s>>>(P);
}
void launch_adv_ts(const Dev& P, cudaStream_t s, int parts) {
  FVG_F32_FORWARD(launch_adv_ts(P, s, parts));
  Dev Q = col_shape(P, P.N, P.KBM1);
  if (Q.col_bc > kHeThreads) Q.col_bc = kHeThreads;
  Dev G = col_shape(P, P.M, P.KBM1);
  if (G.col_bc > kGatherThreads) G.col_bc = kGatherThreads;
  ((P.closed & 2) ? k_he_adv<RF, 1> : k_he_adv_listed<RF, 1>)<<<col_grid(Q, P.N, P.KBM1), Q.col_bc, 0, s>>>(Q, parts);
  if (P.iobcn > 0) k_obc_xflux<RF><<<dim3(nblk(P.iobcn, 64), P.KBM1, 2), 64, 0, s>>>(P, parts);
  k_gather_ts<RF><<<col_grid(G, P.M, P.KBM1), G.col_bc, 0, s>>>(G, parts);
}
void launch_fct_ts(const Dev& P, cudaStream_t s, int parts) {
  dim3 b(32, 8), g(nblk(P.M, 32), nblk(P.KBM1, 8));
  k_fct_ts<<<g, b, 0, s>>>(P, parts);
}
void launch_vdif_ts(const Dev& P, cudaStream_t s, int parts) {
  const int b = col_threads(P, P.M, 128);
  if (P.heating_on)
    k_vdif_ts<true><<<dim3(nblk(P.M, b), 2), b, 0, s>>>(P, parts);
  else
    k_vdif_ts<false><<<dim3(nblk(P.M, b), 2), b, 0, s>>>(P, parts);
}
void launch_bcond_ts(const Dev& P, cudaStream_t s, int parts) {
  if (P.numqbc > 0) k_bcond_ts_riv<<<P.KBM1, 128, 0, s>>>(P);
  if (P.iobcn > 0) k_bcond_ts_obc<<<dim3(P.iobcn, 2), 64, 0, s>>>(P, parts);
}
static bool final_split(const Dev& P) { return (long)P.N * P.KB >= kFinSplit; }
int final_launches(const Dev& P) { return final_split(P) ? 2 : 1; }
void launch_final(const Dev& P, cudaStream_t s, int parts) {
  const bool split = final_split(P);
  const int n = (split ? P.M : P.M > P.N ? P.M : P.N) + 1;
  dim3 b(32, 8), g(nblk(n, 32), nblk(P.KB, 8));
  k_final<<<g, b, 0, s>>>(P, parts, split ? 0 : 1);
  if (!split) return;
  Dev Q = col_shape(P, P.N, P.KB);
  if (Q.col_bc > 128) Q.col_bc = 128;
  k_final_cells<<<col_grid(Q, P.N, P.KB), Q.col_bc, 0, s>>>(Q, parts);
}
void launch_budget(const Dev& P, cudaStream_t s) {
  const int nb = 148;
  k_budget_partial<<<nb, 256, 0, s>>>(P, P.budget + 3);
  k_budget_final<<<1, 32, 0, s>>>(P.budget + 3, nb, P.budget);
}

}  // namespace fvg / fvg_f32
