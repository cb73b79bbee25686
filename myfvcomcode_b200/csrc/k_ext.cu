// k_ext.cu - external (2-D) mode kernels: one EXTERNAL_STEP Runge-Kutta stage is
//   k_ext_node   EXTEL_EDGE(K) + BCOND_GCN(1,K) + RK blend      (per node, half-edge gather)
//   k_wet_*      WET_JUDGE                                      (wetting/drying only)
//   k_ext_cell   N2E2D + FLUX_OBN + ADVAVE_EDGE_GCN + EXTUV_EDGE + BCOND_GCN(2,K)  (per cell)
//   k_ext_update external_step.F:333-436 (EL=ELF, D, D1, UA=UAF, UARD/EGF sums)
// and, on meshes whose metrics are the ones their coordinates define, the same on packed records:
//   k_stage_node, k_stage_cell (one stage), k_ext_loop (every stage of an internal step)
// Reference: FVCOM_source/external_step.F:30-443 and the routines cited per kernel.
// Arithmetic is kept in the reference's expression order; the library is compiled with
// --fmad=false so no multiply-add is contracted.
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

// Programmatic dependent launch: wait until the previous kernel in the stream has
// completed and its writes are visible (a no-op when the kernel was launched without the
// attribute), then let the next kernel's blocks be scheduled during this one's tail.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <typename... KArgs, typename... Args>
static void launch_maybe_pdl(int pdl, void (*k)(KArgs...), dim3 grid, dim3 block, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = pdl ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k, args...);
}

__device__ __constant__ double dAlphaRK[5] = {0.0, 0.25, 1.0 / 3.0, 0.5, 1.0};
#ifndef FVG_F32_TU
const double kAlphaRK[5] = {0.0, 0.25, 1.0 / 3.0, 0.5, 1.0};
#endif
#define ONE_THIRD (1.0 / 3.0)

__device__ inline const double* sched_row(const Dev& P) {
  return P.sched + (size_t)P.ctl[0] * P.sl.len;
}

// -------------------------------------------------------------------------------------
// Least-squares velocity gradient of one cell from itself and its three neighbours
// (advave_edge_gcn.F:634-637, 699-702): COFA1/COFA2 for UA, COFA5/COFA6 for VA.
// -------------------------------------------------------------------------------------
template <typename R>
struct Grad {
  R ux, uy, vx, vy;
};

// a*b and a*b + c in separate roundings, also where this file is compiled with
// contraction: the node part of a stage is the same in the stage kernels (compiled
// without) and in the precision form's resident loop (compiled with).
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
template <typename R>
__device__ __forceinline__ R dot4(R a, R u, R b, R v, R c, R w, R d, R x) {
  return add_rn(add_rn(add_rn(mul_rn(a, u), mul_rn(b, v)), mul_rn(c, w)), mul_rn(d, x));
}

template <typename R, bool CS = false>
__device__ inline Grad<R> cell_grad(const Dev& P, int c, const double* U, const double* V) {
  typedef Mesh<R> Mh;
  int k1, k2, k3;
  R A[4], B[4];
  lsq_coef<R, CS>(P, c, k1, k2, k3, A, B);
  const R a1 = A[0], a2 = A[1], a3 = A[2], a4 = A[3], b1 = B[0], b2 = B[1], b3 = B[2], b4 = B[3];
  R u0 = (R)U[c], u1 = (R)U[k1], u2 = (R)U[k2], u3 = (R)U[k3];
  R v0 = (R)V[c], v1 = (R)V[k1], v2 = (R)V[k2], v3 = (R)V[k3];
  if (P.gcy && (k1 == 0 || k2 == 0 || k3 == 0)) {
    double gu, gv;
    if (k1 == 0) { ghost_uv(P, U, V, c, 1, gu, gv); u1 = (R)gu; v1 = (R)gv; }
    if (k2 == 0) { ghost_uv(P, U, V, c, 2, gu, gv); u2 = (R)gu; v2 = (R)gv; }
    if (k3 == 0) { ghost_uv(P, U, V, c, 3, gu, gv); u3 = (R)gu; v3 = (R)gv; }
  }
  Grad<R> g;
  g.ux = dot4(a1, u0, a2, u1, a3, u2, a4, u3);
  g.uy = dot4(b1, u0, b2, u1, b3, u2, b4, u3);
  g.vx = dot4(a1, v0, a2, v1, a3, v2, a4, v3);
  g.vy = dot4(b1, v0, b2, v1, b3, v2, b4, v3);
  return g;
}
// Least-squares gradient of UA, VA of cell c (advave_edge_gcn.F:634-637, 699-702) and the
// cell's part ART*|grad|*CC_HVC of its three edges' viscosity, stored for the edge loop of the
// next ADVAVE call in the handle's precision.
template <typename R, bool CS>
__device__ inline void store_grad_t(const Dev& P, int c) {
  typedef Mesh<R> Mh;
  Grad<R> g = cell_grad<R, CS>(P, c, P.ua, P.va);
  const R half = (R)0.5;
  reinterpret_cast<R*>(P.xvc)[c] = Mh::art(P, c) *
      sqrt(g.ux * g.ux + g.vy * g.vy + half * ((g.uy + g.vx) * (g.uy + g.vx))) * Mh::cc_hvc(P, c);
  if constexpr (sizeof(R) == 4) {
    P.f.g2d4[c] = make_float4(g.ux, g.uy, g.vx, g.vy);
  } else {
    Mesh<R>::g2d(P, 0)[c] = g.ux;
    Mesh<R>::g2d(P, 1)[c] = g.uy;
    Mesh<R>::g2d(P, 2)[c] = g.vx;
    Mesh<R>::g2d(P, 3)[c] = g.vy;
  }
}
template <bool CS>
__device__ inline void store_grad(const Dev& P, int c) {
  if (P.prec) store_grad_t<float, CS>(P, c);
  else store_grad_t<double, CS>(P, c);
}
template <typename R>
__device__ inline Grad<R> load_grad(const Dev& P, int c) {
  Grad<R> g;
  if constexpr (sizeof(R) == 4) {
    const float4 a = P.f.g2d4[c];
    g.ux = a.x;
    g.uy = a.y;
    g.vx = a.z;
    g.vy = a.w;
  } else {
    g.ux = Mesh<R>::g2d(P, 0)[c];
    g.uy = Mesh<R>::g2d(P, 1)[c];
    g.vx = Mesh<R>::g2d(P, 2)[c];
    g.vy = Mesh<R>::g2d(P, 3)[c];
  }
  return g;
}
// EXTEL_EDGE half-edge flux EXFLUX = DIJ*(-UIJ*DLTYE+VIJ*DLTXE) (extel_edge.F:86-94) of the
// three half-edges owned by cell c, from the cell's own D1, UA, VA.
__device__ inline void store_exf(const Dev& P, int c) {
  double d1 = P.d1[c], u = P.ua[c], v = P.va[c];
  for (int s = 0; s < 3; ++s) {
    const size_t pos = (size_t)s * P.ns + c;
    P.exf2d[pos] = d1 * (-u * Mesh<double>::hg(P, 1, pos) + v * Mesh<double>::hg(P, 0, pos));
  }
}

// -------------------------------------------------------------------------------------
// EXTEL_EDGE(K) (extel_edge.F:76-180) and BCOND_GCN(1,K) -> BCOND_ASL/BCOND_ASL_CLP
// (mod_obcs.F:509-617) with the Runge-Kutta blend of the specified-elevation nodes
// (external_step.F:262-266).  One thread per node; the node's control-volume half-edges
// are gathered in ascending half-edge number, the order of the reference's scatter.
// Node part of WET_JUDGE for node i from the cell flags cwet of the same judgement.
template <bool CS = false>
__device__ inline void wet_node(const Dev& P, int i, const int* cwet) {
  double e = P.elf[i];
  int wet = ((P.h[i] + e - P.min_depth) < 1.0e-5) ? 0 : 1;
  // the ring's cell flags, four entries' indices and then their flags loaded at a time
  const int nt = ld1<CS>(P.ntve + i);
  const size_t m1 = P.M + 1;
  const int* L = P.nbve + i;
  int s = 0, j = 0;
  for (; j + 4 <= nt; j += 4) {
    const int c0 = ld1<CS>(L + j * m1), c1 = ld1<CS>(L + (j + 1) * m1), c2 = ld1<CS>(L + (j + 2) * m1),
              c3 = ld1<CS>(L + (j + 3) * m1);
    s += cwet[c0] + cwet[c1] + cwet[c2] + cwet[c3];
  }
  for (; j < nt; ++j) s += cwet[ld1<CS>(L + j * m1)];
  if (s == 0) wet = 0;
  P.iswetn[i] = wet;
  P.elf[i] = fmax(e, -P.h[i] + P.min_depth);
}

// -------------------------------------------------------------------------------------
// Node part of the update after stage K (external_step.F:333-436): EL = ELF, D, DTFA, and
// the K == 3 and K == 4 sums.
template <bool CS = false>
__device__ inline void ext_update_node(const Dev& P, int i, int K) {
  double e = P.elf[i];
  P.el[i] = e;
  double dd = P.h[i] + e;
  P.d[i] = dd;
  P.dtfa[i] = dd;
  if (K == 3) P.egf[i] = ld1<CS>(P.egf + i) + e / (double)P.isplit;
  if (K == 4) {
    int ob = ld1<CS>(P.node_obc + i);
    if (ob > 0) {
      double tmp = -(P.elf[i] - P.elrk[i]) * P.art1[i] / P.dte - P.xflux_obcn[ob];
      P.uard_obcn[ob] = P.uard_obcn[ob] + tmp / (double)(float)P.isplit;
    }
  }
}

// Cell part of the update after stage K with the new UA, VA: EL1, D1, the K == 3 sums and
// the half-edge continuity fluxes of the next stage.
__device__ inline void ext_update_cell(const Dev& P, int i, int K, double e1, double u, double v) {
  P.el1[i] = e1;
  double dd1 = P.h1[i] + e1;
  P.d1[i] = dd1;
  if (K == 3) {
    P.uard[i] = P.uard[i] + u * dd1;
    P.vard[i] = P.vard[i] + v * dd1;
  }
  for (int s = 0; s < 3; ++s) {
    const size_t pos = (size_t)s * P.ns + i;
    P.exf2d[pos] = dd1 * (-u * Mesh<double>::hg(P, 1, pos) + v * Mesh<double>::hg(P, 0, pos));
  }
}

// Slope limiters UALFA, VALFA of each cell for the limited ADVAVE (advave_edge_gcn.F:141-318):
// the cell's three edges with a wet side, in any order (a minimum), from the cell's own
// gradient and the two cells' UA, VA.  After WET_JUDGE, before the stage's ADVAVE.
template <typename R>
__global__ void k_alfa2(const Dev P) {
  typedef Mesh<R> Mh;
  const int c = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (c > P.N) return;
  const size_t n1 = P.N + 1;
  const Grad<R> g = load_grad<R>(P, c);
  R au = (R)1, av = (R)1;
  for (int s = 0; s < 3; ++s) {
    const size_t q = (size_t)s * n1 + c;
    const int ia = P.ce_ia[q], ib = P.ce_ib[q];
    if (!(P.iswetce[ia] * P.iswetc[ia] == 1 || P.iswetce[ib] * P.iswetc[ib] == 1)) continue;
    const bool a_side = (P.ce_code[q] & 1) == 0;
    const R x = a_side ? Mh::s_xoa(P, q) : Mh::s_xob(P, q);
    const R y = a_side ? Mh::s_yoa(P, q) : Mh::s_yob(P, q);
    lim_alfa<R>(fabs((R)P.ua[ia] - (R)P.ua[ib]), g.ux * x + g.uy * y, au);
    lim_alfa<R>(fabs((R)P.va[ia] - (R)P.va[ib]), g.vx * x + g.vy * y, av);
  }
  Mh::alfa2(P, 0)[c] = au;
  Mh::alfa2(P, 1)[c] = av;
}

// CS: the arrays the kernel reads once per stage (gather lists, pointers, per-node and
// per-cell coefficients) are loaded evict-first (ld1).
template <bool CS>
__device__ __forceinline__ void ext_node_job(const Dev& P, const int i, int iext, int K, int parts) {
  // jobs 1..M are the nodes, jobs M+1..M+N the cells' least-squares gradients of the
  // current UA, VA for ADVAVE of this stage
  if (i > P.M) {
    const int c = i - P.M;
    if ((parts & EN_GRAD) && c <= P.N) store_grad<CS>(P, c);
    return;
  }
  // EXTEL's sum first: its loads (the previous cell kernel's half-edge fluxes) do not
  // depend on the node updates below, which then overlap with them
  double x = 0.0;
  if (parts & EN_EXTEL) {
    // the half-edge fluxes in ascending half-edge order; four entries' codes and then
    // their fluxes are loaded at a time, and added in order
    const int n = ld1<CS>(P.node_he_ptr + i + 1) - ld1<CS>(P.node_he_ptr + i);
    const int* L = P.node_vpos_ell + i;
    const size_t ms = P.ms;
    int j = 0;
    for (; j + 4 <= n; j += 4) {
      const int e0 = ld1<CS>(L + j * ms), e1 = ld1<CS>(L + (j + 1) * ms), e2 = ld1<CS>(L + (j + 2) * ms),
                e3 = ld1<CS>(L + (j + 3) * ms);
      const double f0 = P.exf2d[e0 >> 1], f1 = P.exf2d[e1 >> 1], f2 = P.exf2d[e2 >> 1], f3 = P.exf2d[e3 >> 1];
      x = (e0 & 1) ? x + f0 : x - f0;
      x = (e1 & 1) ? x + f1 : x - f1;
      x = (e2 & 1) ? x + f2 : x - f2;
      x = (e3 & 1) ? x + f3 : x - f3;
    }
    for (; j < n; ++j) {
      const int e = ld1<CS>(L + j * ms);
      const double exflux = P.exf2d[e >> 1];
      x = (e & 1) ? x + exflux : x - exflux;
    }
  }
  // the previous stage's ELF clamp (WET_JUDGE) and update (ext_update_node); ISWETN and DTFA,
  // which nothing inside the loop reads, are left to k_ext_finish
  double e = 0.0;
  const int ob = ld1<CS>(P.node_obc + i);
  if (parts & EN_FINISH_PREV) {
    const double h = P.h[i];
    const int Kp = (parts >> 8) & 7;
    e = P.elf[i];
    if (parts & EN_WET_PREV) e = fmax(e, -h + P.min_depth);
    P.el[i] = e;
    P.d[i] = h + e;
    if (Kp == 3) P.egf[i] = ld1<CS>(P.egf + i) + e / (double)P.isplit;
    if (Kp == 4 && ob > 0) {
      const double tmp = -(e - P.elrk[i]) * P.art1[i] / P.dte - P.xflux_obcn[ob];
      P.uard_obcn[ob] = P.uard_obcn[ob] + tmp / (double)(float)P.isplit;
    }
  } else if (parts & EN_COPY_ELRK) {
    e = P.el[i];
  }
  double elrk;
  if (parts & EN_COPY_ELRK) {
    elrk = e;
    P.elrk[i] = e;
  } else {
    elrk = ld1<CS>(P.elrk + i);
  }
  const double alpha = dAlphaRK[K];
  double elf = 0.0;
  if (parts & EN_EXTEL) {
    if (ob > 0) {
      P.xflux_obcn[ob] = x;
      x = 0.0;
    }
    for (int q = P.node_riv_ptr[i]; q < P.node_riv_ptr[i + 1]; ++q) {
      int r = P.node_riv[q];
      int j = r >> 1;
      if (P.river_location == 0)
        x = x - P.qdis[j];
      else
        x = x - P.qdis[j] * P.rdisq[(size_t)(r & 1) * (P.numqbc + 1) + j];
    }
    double dtk = alpha * P.dte;
    elf = elrk - dtk * x / ld1<CS>(P.art1 + i);
  } else {
    elf = P.elf[i];
  }
  if ((parts & EN_BC) && ob > 0) {
    int kind = P.obc_kind[ob];
    if (kind == 1) {
      if (P.obc_elev_on && (parts & EN_TABLE)) {
        elf = P.obf[(size_t)((iext - 1) * 4 + K - 1) * (P.iobcn + 1) + ob];
      } else if (P.obc_elev_on) {
        const double* row = sched_row(P);
        double force = 0.0;
        for (int j = 0; j < P.ntide; ++j) {
          size_t q = (size_t)j * (P.iobcn + 1) + ob;
          double targ = row[P.sl.targ(iext, K, j)];
          force = add_rn(mul_rn(P.apt[q], cos(targ - P.phai_rad[q])), force);
        }
        force = force + P.emean[ob];
        elf = force * row[P.sl.ramp_ext(iext)];
      }
      elf = add_rn(elrk, mul_rn(alpha, elf - elrk));
    } else if (kind == 2) {
      elf = 0.0;
    }
  }
  P.elf[i] = elf;
}

// One job per thread, 48 registers (five blocks of 256 per SM; at 40 registers it
// spills).  Measured slower on the 200k-node mesh: a grid of five blocks per SM whose
// threads walk the jobs (1.14 -> 1.29 ms per step), and blocks that each mix three warps
// of node jobs with five of gradient jobs (1.13 -> 1.45 ms).
template <bool CS>
__global__ void __launch_bounds__(256, 5) k_ext_node(const Dev P, int iext, int K, int parts) {
  pdl_enter();
  const int n = (parts & EN_GRAD) ? P.M + P.N : P.M;
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i <= n) ext_node_job<CS>(P, i, iext, K, parts);
}

// -------------------------------------------------------------------------------------
// WET_JUDGE (mod_wd.F:193-284) in two passes.  Cells first: the cell flag uses the
// unclamped ELF of its nodes, and ELF1 is the mean of the clamped ELF, which each cell
// forms itself from h and ELF.  Then nodes: the node flag and the clamp of ELF.
// -------------------------------------------------------------------------------------
template <bool CS>
__device__ __forceinline__ int wet_cell(const Dev& P, const int i, double& elf1) {
  int n1 = ld1<CS>(P.nv + i), n2 = ld1<CS>(P.nv + (size_t)(P.N + 1) + i), n3 = ld1<CS>(P.nv + (size_t)2 * (P.N + 1) + i);
  double e1 = P.elf[n1], e2 = P.elf[n2], e3 = P.elf[n3];
  double dtmp = fmax(fmax(e1, e2), e3) + fmin(fmin(P.h[n1], P.h[n2]), P.h[n3]);
  const int wet = ((dtmp - P.min_depth) < 1.0e-5) ? 0 : 1;
  P.iswetc[i] = wet;
  double c1 = fmax(e1, -P.h[n1] + P.min_depth);
  double c2 = fmax(e2, -P.h[n2] + P.min_depth);
  double c3 = fmax(e3, -P.h[n3] + P.min_depth);
  elf1 = ONE_THIRD * (c1 + c2 + c3);
  P.elf1[i] = elf1;
  return wet;
}
template <bool CS>
__global__ void k_wet_cells(const Dev P) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  double elf1;
  if (i <= P.N) wet_cell<CS>(P, i, elf1);
}

__global__ void k_wet_nodes(const Dev P) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) return;
  wet_node(P, i, P.iswetc);
}

// Whether cell o on the other side of slot s (nodes j1, j2) of cell i counts as wet,
// ISWETCE*ISWETC.  judge: WET_JUDGE's cell part runs in the same kernel (EC_WET), so the flag
// of this stage is formed from the neighbour's three nodes, its node off the edge in wfar, as
// wet_cell forms it.  A cell that is wet itself needs no neighbour's flag, so that only dry
// cells pay for this.
__device__ inline bool wet_other(const Dev& P, bool judge, int i, int s, int o, int j1, int j2) {
  if (judge && o != 0) {
    const double e = fmax(fmax(P.elf[j1], P.elf[j2]), P.elf[P.wfar[(size_t)s * (P.N + 1) + i]]);
    return (((e + P.hmin[o]) - P.min_depth) < 1.0e-5 ? 0 : 1) * P.iswetce[o] == 1;
  }
  return P.iswetce[o] * P.iswetc[o] == 1;
}

// ADVAVE_EDGE_GCN for one cell (advave_edge_gcn.F:115-1003), over the cell's slot table.
// EDGES: the edges as the cell sees them, or each by its own list entry (per_edge), plain or
// limited.  The edge fluxes are evaluated in R; the surface-slope pressure gradient PSTX/PSTY
// stays FP64.
enum Edges { kSeen, kListed, kLimitedEdges };
template <typename R, Edges EDGES>
__device__ inline void advave_cell(const Dev& P, int i, int weti, bool judge, double& xfo, double& yfo, double& px,
                                   double& py) {
  typedef Mesh<R> Mh;
  const R half = (R)0.5, one = (R)1.0;
  R xf = 0, yf = 0;
  px = 0.0; py = 0.0;
  const size_t n1 = P.N + 1;
  const R epor = (R)P.epor[i], iucp = (R)P.iucp[i];
  const Grad<R> gi = load_grad<R>(P, i);
  const R ui = (R)P.ua[i], vi = (R)P.va[i];
  const double ged1 = P.grav_e[i] * P.d1[i];
  if constexpr (EDGES == kSeen) {
    // Each edge as the cell sees it: its own side from the values above, sums that commute
    // without regard to the sides, the upwind weights with the side as a sign, and both
    // cells' ART*|grad|*CC_HVC from the gradient job (xvc), so that the values and their
    // order are the reference's and the square roots are one per cell instead of six.
    const R* VC = reinterpret_cast<const R*>(P.xvc);
    const R vci = VC[i];
    const int4 xn = P.loopx[i], oo = P.loopo[i];
    const int xs[3] = {xn.x, xn.y, xn.z}, os[3] = {oo.x, oo.y, oo.z};
    const int bits = xn.w;
    const double dn[3] = {P.d[xs[0]], P.d[xs[1]], P.d[xs[2]]};
    const double en[3] = {P.el[xs[0]], P.el[xs[1]], P.el[xs[2]]};
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const int side = (bits >> s) & 1, o = os[s];
      const size_t q = (size_t)s * n1 + i;
      const double edx = P.ce_dx[q], edy = P.ce_dy[q];
      if (weti == 1 || wet_other(P, judge, i, s, o, xs[s], xs[(s + 1) % 3])) {
        const R dij = (R)(0.5 * (dn[s] + dn[(s + 1) % 3]));
        R xi, yi, xo, yo, dx, dy;
        if constexpr (sizeof(R) == 4) {
          const float4 G = P.f.ce_geo[q];  // XOA, YOA, XOB, YOB
          const float2 D = P.f.ce_dd[q];
          xi = side ? G.z : G.x;
          yi = side ? G.w : G.y;
          xo = side ? G.x : G.z;
          yo = side ? G.y : G.w;
          dx = D.x;
          dy = D.y;
        } else {
          xi = (side ? P.ce_xob : P.ce_xoa)[q];
          yi = (side ? P.ce_yob : P.ce_yoa)[q];
          xo = (side ? P.ce_xoa : P.ce_xob)[q];
          yo = (side ? P.ce_yoa : P.ce_yob)[q];
          dx = edx;
          dy = edy;
        }
        const Grad<R> go = load_grad<R>(P, o);
        const R uo = (R)P.ua[o], vo = (R)P.va[o], vco = VC[o];
        const R uown = ui + gi.ux * xi + gi.uy * yi, vown = vi + gi.vx * xi + gi.vy * yi;
        const R uoth = uo + go.ux * xo + go.uy * yo, voth = vo + go.vx * xo + go.vy * yo;
        const R uij = half * (uown + uoth), vij = half * (vown + voth);
        const R un = -uij * dy + vij * dx;
        R viscof = (R)P.fact * half * (vci + vco);
        viscof = viscof + (R)P.fm1 * half * (P.fm1 != 0.0 ? Mh::cc_hvc(P, i) + Mh::cc_hvc(P, o) : (R)0);
        if (P.hprnu != 1.0) viscof = viscof / (R)P.hprnu;
        const R vxa = side ? go.vx : gi.vx, vxb = side ? gi.vx : go.vx;
        const R txx = (gi.ux + go.ux) * viscof;
        const R tyy = (gi.vy + go.vy) * viscof;
        const R txy = half * (gi.uy + go.uy + vxa + vxb) * viscof;
        const R fxx = dij * (txx * dy - txy * dx);
        const R fyy = dij * (txy * dy - tyy * dx);
        const R sg = fsign1(un), so = side ? -sg : sg;
        const R xadv = dij * un * ((one - so) * uoth + (one + so) * uown) * half;
        const R yadv = dij * un * ((one - so) * voth + (one + so) * vown) * half;
        const R nb = one - (R)((bits >> (3 + s)) & 1);
        const R ax = (xadv + fxx * epor) * nb * iucp, ay = (yadv + fyy * epor) * nb * iucp;
        xf = side ? xf - ax : xf + ax;
        yf = side ? yf - ay : yf + ay;
      }
      const double elij = 0.5 * (en[s] + en[(s + 1) % 3]);
      const double tx = ged1 * elij * edy, ty = ged1 * elij * edx;
      px = side ? px + tx : px - tx;
      py = side ? py - ty : py + ty;
    }
  } else {
    for (int s = 0; s < 3; ++s) {
      const size_t q = (size_t)s * n1 + i;
      const int4 ci = P.ce_i4[q];  // {code, IA, IB, J1}
      const int code = ci.x;
      const int side = code & 1;
      const int ia = ci.y, ib = ci.z;
      const int j1 = ci.w, j2 = P.ce_j2[q];
      R dij = (R)(0.5 * (P.d[j1] + P.d[j2]));
      double elij = 0.5 * (P.el[j1] + P.el[j2]);
      const int o = side == 0 ? ib : ia;  // the other cell of the edge
      if (weti == 1 || P.iswetce[o] * P.iswetc[o] == 1) {
        R uij1, vij1, uij2, vij2;
        const R arta = Mh::art(P, ia), artb = Mh::art(P, ib);
        const R cca = Mh::cc_hvc(P, ia), ccb = Mh::cc_hvc(P, ib);
        const Grad<R> ga = load_grad<R>(P, ia), gb = load_grad<R>(P, ib);
        const R xija = Mh::s_xoa(P, q), yija = Mh::s_yoa(P, q);
        const R xijb = Mh::s_xob(P, q), yijb = Mh::s_yob(P, q);
        if constexpr (EDGES == kLimitedEdges) {
          lim_faces<R>(P.limiter, (R)P.ua[ia], (R)P.ua[ib], ga.ux * xija + ga.uy * yija, gb.ux * xijb + gb.uy * yijb,
                       Mh::alfa2(P, 0)[ia], Mh::alfa2(P, 0)[ib], uij1, uij2);
          lim_faces<R>(P.limiter, (R)P.va[ia], (R)P.va[ib], ga.vx * xija + ga.vy * yija, gb.vx * xijb + gb.vy * yijb,
                       Mh::alfa2(P, 1)[ia], Mh::alfa2(P, 1)[ib], vij1, vij2);
        } else {
          uij1 = (R)P.ua[ia] + ga.ux * xija + ga.uy * yija;
          uij2 = (R)P.ua[ib] + gb.ux * xijb + gb.uy * yijb;
          vij1 = (R)P.va[ia] + ga.vx * xija + ga.vy * yija;
          vij2 = (R)P.va[ib] + gb.vx * xijb + gb.vy * yijb;
        }
        R uij = half * (uij1 + uij2);
        R vij = half * (vij1 + vij2);
        const auto DD = Mh::s_dd(P, q);
        const R dltxc = DD.x, dltyc = DD.y;
        R un = -uij * dltyc + vij * dltxc;
        R viscof1 = arta * sqrt(ga.ux * ga.ux + ga.vy * ga.vy + half * ((ga.uy + ga.vx) * (ga.uy + ga.vx)));
        R viscof2 = artb * sqrt(gb.ux * gb.ux + gb.vy * gb.vy + half * ((gb.uy + gb.vx) * (gb.uy + gb.vx)));
        R viscof = ((R)P.fact * half * (viscof1 * cca + viscof2 * ccb) + (R)P.fm1 * half * (cca + ccb)) / (R)P.hprnu;
        R txx = (ga.ux + gb.ux) * viscof;
        R tyy = (ga.vy + gb.vy) * viscof;
        R txy = half * (ga.uy + gb.uy + ga.vx + gb.vx) * viscof;
        R fxx = dij * (txx * dltyc - txy * dltxc);
        R fyy = dij * (txy * dltyc - tyy * dltxc);
        R sg = fsign1(un);
        R xadv = dij * un * ((one - sg) * uij2 + (one + sg) * uij1) * half;
        R yadv = dij * un * ((one - sg) * vij2 + (one + sg) * vij1) * half;
        R nb = one - (R)((code >> 1) & 1);
        if (side == 0) {
          xf = xf + (xadv + fxx * epor) * nb * iucp;
          yf = yf + (yadv + fyy * epor) * nb * iucp;
        } else {
          xf = xf - (xadv + fxx * epor) * nb * iucp;
          yf = yf - (yadv + fyy * epor) * nb * iucp;
        }
      }
      const double edx = P.ce_dx[q], edy = P.ce_dy[q];
      if (side == 0) {
        px = px - ged1 * elij * edy;
        py = py + ged1 * elij * edx;
      } else {
        px = px + ged1 * elij * edy;
        py = py - ged1 * elij * edx;
      }
    }
  }
  R w = (R)weti;
  xfo = (double)(xf * w);
  yfo = (double)(yf * w);
}

// FLUX_OBN (mod_obcs.F:1181-1215) value on one open-boundary cell.
__device__ inline double fluxobn_cell(const Dev& P, int i, int K) {
  double f = 0.0;
  for (int q = P.cell_obc_ptr[i]; q < P.cell_obc_ptr[i + 1]; ++q) {
    int code = P.cell_obc[q];
    int ob = code >> 1, slot = code & 1;
    int j = P.i_obc_n[ob];
    // ELF as WET_JUDGE leaves it (its node part may still be pending in a fused loop;
    // the clamp is idempotent)
    double ej = P.wetting_drying_on ? fmax(P.elf[j], -P.h[j] + P.min_depth) : P.elf[j];
    double flux = -(ej - P.elrk[j]) * P.art1[j] / (dAlphaRK[K] * P.dte) - P.xflux_obcn[ob];
    f = f + P.fluxf_obc[(size_t)slot * (P.iobcn + 1) + ob] * flux;
  }
  return f;
}

// River clamp / tangential projection of a solid-boundary cell (bcond_gcn.F:345-405).
__device__ inline void bc_solid(const Dev& P, int i, int rj, double& uu, double& vv) {
  if (rj > 0) {
    double ca = P.cos_angleq[rj], sa = P.sin_angleq[rj];
    double untmp = uu * ca + vv * sa;
    double vntmp = -uu * sa + vv * ca;
    untmp = fmax(untmp, 0.0);
    uu = untmp * ca - vntmp * sa;
    vv = untmp * sa + vntmp * ca;
  } else {
    double sa = P.sin_alpha[i], ca = P.cos_alpha[i];
    double ui = uu * (sa * sa) - vv * sa * ca;
    double vi = -uu * sa * ca + vv * (ca * ca);
    uu = ui;
    vv = vi;
  }
}

// EXTUV's terms that stay fixed over the coming external loop, packed for its stages.  FP64:
// six pairs per cell (exd), read as they are.  FP32 form: summed in FP64 (exc0, exc1), which
// that form's rounding allows.
template <typename R>
__device__ inline void store_fixed(const Dev& P, int i, double adx, double ady) {
  const size_t n1 = P.N + 1;
  const double art = P.art[i], wx = P.have_wind ? P.wsx[i] : 0.0, wy = P.have_wind ? P.wsy[i] : 0.0;
  if constexpr (sizeof(R) == 4) {
    P.f.exc0[i] = make_double4(adx + P.drx2d[i] - P.wubot[i] * art, ady + P.dry2d[i] - P.wvbot[i] * art,
                               0.001 * wx * art, 0.001 * wy * art);
    P.f.exc1[i] = make_double4(P.cor[i] * art, art, P.h1[i], P.grav_e[i]);
  } else {
    P.exd[i] = make_double2(adx, P.drx2d[i]);
    P.exd[n1 + i] = make_double2(ady, P.dry2d[i]);
    P.exd[2 * n1 + i] = make_double2(P.wubot[i], P.wvbot[i]);
    P.exd[3 * n1 + i] = make_double2(wx, wy);
    P.exd[4 * n1 + i] = make_double2(P.cor[i], art);
    P.exd[5 * n1 + i] = make_double2(P.h1[i], P.grav_e[i]);
  }
}

// -------------------------------------------------------------------------------------
// Per-cell part of one RK stage.  EC_INT_ADVAVE is the internal-step call of ADVAVE
// followed by ADX2D -= ADVUA (internal_step.F:387-392).
// -------------------------------------------------------------------------------------
template <typename R, Edges EDGES>
__global__ void __launch_bounds__(128, sizeof(R) == 4 ? 8 : (EDGES == kSeen ? 5 : 1)) k_ext_cell(const Dev P, int iext, int K, int parts) {
  pdl_enter();
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.N) return;
  const size_t n1 = P.N + 1;
  if (parts & EC_COPY_RK) {
    P.uark[i] = P.ua[i];
    P.vark[i] = P.va[i];
    P.elrk1[i] = P.el1[i];
  }
  double elf1;
  if (parts & EC_N2E) {
    elf1 = ONE_THIRD * (P.elf[P.nv[i]] + P.elf[P.nv[n1 + i]] + P.elf[P.nv[2 * n1 + i]]);
    P.elf1[i] = elf1;
  }
  const int weti = P.iswetce[i] * ((parts & EC_WET) ? wet_cell<false>(P, i, elf1) : P.iswetc[i]);
  if (!(parts & (EC_N2E | EC_WET))) elf1 = P.elf1[i];
  double fob = 0.0;
  if (parts & EC_FLUXOBN) {
    fob = fluxobn_cell(P, i, K);
    P.fluxobn[i] = fob;
  } else if (P.isbce[i] == 2) {
    fob = P.fluxobn[i];
  }
  double xf, yf, px, py;
  if (parts & (EC_ADVAVE | EC_INT_ADVAVE)) {
    advave_cell<R, EDGES>(P, i, weti, parts & EC_WET, xf, yf, px, py);
    if (P.isbce[i] == 2) {
      if (P.gcy) {  // advave_edge_gcy.F
        xf = xf + fob * P.ua[i] * P.iucp[i];
        yf = yf + fob * P.va[i] * P.iucp[i];
      } else {
        xf = (xf + fob * P.ua[i]) * P.iucp[i];
        yf = (yf + fob * P.va[i]) * P.iucp[i];
      }
    }
    for (int q = P.cell_riv_ptr[i]; q < P.cell_riv_ptr[i + 1]; ++q) {
      int k = P.cell_riv[q] >> 1;
      double vlctyq = P.qdis[k] / P.qarea[k];
      if (P.river_location == 0) {
        xf = xf - 0.5 * P.qdis[k] * vlctyq * P.cos_angleq[k];
        yf = yf - 0.5 * P.qdis[k] * vlctyq * P.sin_angleq[k];
      } else {
        double temp = P.qdis[k] * vlctyq;
        xf = xf - temp * P.cos_angleq[k];
        yf = yf - temp * P.sin_angleq[k];
      }
    }
    P.advua[i] = xf;
    P.advva[i] = yf;
    P.pstx[i] = px;
    P.psty[i] = py;
    if (parts & EC_INT_ADVAVE) {
      const double adx = P.adx2d[i] - xf, ady = P.ady2d[i] - yf;
      P.adx2d[i] = adx;
      P.ady2d[i] = ady;
      if (P.xform) store_fixed<R>(P, i, adx, ady);
    }
  } else {
    xf = P.advua[i];
    yf = P.advva[i];
    px = P.pstx[i];
    py = P.psty[i];
  }
  if (parts & (EC_EXTUV | EC_BC2)) {
    double uaf, vaf;
    if (parts & EC_EXTUV) {
      // EXTUV_EDGE(K) (extuv_edge.F:106-163)
      if (weti == 1) {
        double ramp = sched_row(P)[P.sl.ramp_ext(iext)];
        double wus = P.have_wind ? P.wsx[i] * ramp * 0.001 : 0.0;
        double wvs = P.have_wind ? P.wsy[i] * ramp * 0.001 : 0.0;
        double resx = P.adx2d[i] + xf + P.drx2d[i] + px - P.cor[i] * P.va[i] * P.d1[i] * P.art[i] -
                      (wus + P.wubot[i]) * P.art[i];
        double resy = P.ady2d[i] + yf + P.dry2d[i] + py + P.cor[i] * P.ua[i] * P.d1[i] * P.art[i] -
                      (wvs + P.wvbot[i]) * P.art[i];
        double a = dAlphaRK[K];
        uaf = (P.uark[i] * (P.h1[i] + P.elrk1[i]) - a * P.dte * resx / P.art[i]) / (P.h1[i] + elf1);
        vaf = (P.vark[i] * (P.h1[i] + P.elrk1[i]) - a * P.dte * resy / P.art[i]) / (P.h1[i] + elf1);
      } else {
        uaf = 0.0;
        vaf = 0.0;
      }
      const double sp = P.cc_sponge[i];
      if (sp != 0.0) {
        uaf = uaf / (1.0 + sp * (uaf * uaf));
        vaf = vaf / (1.0 + sp * (vaf * vaf));
      }
    } else {
      uaf = P.uaf[i];
      vaf = P.vaf[i];
    }
    if (parts & EC_BC2) {
      // BCOND_GCN(2,K) (bcond_gcn.F:325-406)
      int b = P.isbce[i];
      // GCY (bcond_gcy.F): the river clamp only, no tangential projection or corner zero
      if (b == 3 && !P.gcy) { uaf = 0.0; vaf = 0.0; }
      if (b == 1 && (!P.gcy || P.cell_bcriv[i] > 0)) bc_solid(P, i, P.cell_bcriv[i], uaf, vaf);
    }
    P.uaf[i] = uaf;
    P.vaf[i] = vaf;
    if (parts & EC_FINISH) ext_update_cell(P, i, K, elf1, uaf, vaf);
  }
}


// -------------------------------------------------------------------------------------
// The external stages on packed records (Dev::xform), two phases per Runge-Kutta stage:
//   node phase   the update of the previous stage, EXTEL_EDGE and the boundary elevation of
//                a node; the least-squares gradient of a cell and its viscosity term
//                ART*|grad|*CC_HVC, which its neighbours' edges share;
//   cell phase   WET_JUDGE's cell part (a dry cell forms its neighbours' flags itself),
//                ADVAVE, EXTUV, BCOND_GCN(2) and the update of a cell.
// A stage waits on loads, not on arithmetic or bandwidth, so a phase loads all it needs before
// it computes: values of neighbours and nodes are packed in pairs (xuv, xg, xnd), the edge
// geometry is formed from coordinates (seven pairs instead of twenty-four doubles), EXTUV's
// fixed terms are pairs too.  ISWETN, DTFA, EL and D, which nothing inside the loop reads from
// their own arrays, are left to k_ext_finish; ADVUA, ADVVA, PSTX, PSTY to the last stage.  In
// FP64 every value is formed as the general stage kernels form it, with the sums that commute
// taken in the cell's own order: results are theirs bit for bit.
//
// k_ext_loop runs the whole external loop as one kernel, for meshes with at most one cell and
// one node per thread of a grid of one block per SM (launched cooperatively, so that all its
// blocks are resident), with a grid barrier behind each phase: there a stage kernel is one wave
// behind a launch, and 80 to 120 launches were half of the step.  k_stage_node and k_stage_cell
// are the same phases as kernels, for larger meshes.
// -------------------------------------------------------------------------------------
// A load of what other threads exchange: in L2 inside the resident loop, whose L1 lines go
// stale; through L1 in the stage kernels, where neighbouring cells share it.
template <bool RES, class T>
__device__ __forceinline__ T ldx(const T* p) {
  if constexpr (RES) return __ldcg(p);
  return *p;
}
template <typename R, bool RES>
__device__ __forceinline__ Grad<R> ld_xg(const Dev& P, int c) {
  if constexpr (sizeof(R) == 4) {
    const float4 a = ldx<RES>(P.f.g2d4 + c);
    return Grad<R>{a.x, a.y, a.z, a.w};
  } else {
    const double2* g = reinterpret_cast<const double2*>(P.xg) + 2 * (size_t)c;
    const double2 a = ldx<RES>(g), b = ldx<RES>(g + 1);
    return Grad<R>{a.x, a.y, b.x, b.y};
  }
}
template <typename R>
__device__ __forceinline__ void st_xg(const Dev& P, int c, const Grad<R>& g) {
  if constexpr (sizeof(R) == 4) {
    P.f.g2d4[c] = make_float4(g.ux, g.uy, g.vx, g.vy);
  } else {
    double2* q = reinterpret_cast<double2*>(P.xg) + 2 * (size_t)c;
    q[0] = make_double2(g.ux, g.uy);
    q[1] = make_double2(g.vx, g.vy);
  }
}

// What a thread of the resident loop reads every stage and nothing changes in between, in
// shared memory, one column per thread (T threads): a grid barrier empties L1, and these were
// half of a phase's loads from L2.  Pairs: VX,VY of X0..X2, XC,YC of the cell and of the other
// cells, EXTUV's fixed terms; doubles: hmin, H of X0..X2, CC_SPONGE; the gradient's
// coefficients, ART and CC_HVC in the form's type; the first kLoopList entries of the node's
// half-edge list and the cell's NBE.
constexpr int kLoopList = 14;
template <typename R, int T>
struct LoopShared {
  double2 p2[13][T];
  double p1[5][T];
  // the cell's own state, written back after the last stage: D1, EL1, ELRK1, UARK, VARK, UARD, VARD
  double own[7][T];
  R ab[10][T];
  int list[kLoopList][T];
  int nb[3][T];
};
template <typename R, int T>
__device__ __forceinline__ LoopShared<R, T>& loop_shared() {
  extern __shared__ __align__(16) unsigned char loop_sm[];
  return *reinterpret_cast<LoopShared<R, T>*>(loop_sm);
}

// ISWETCE*ISWETC of cell o on the other side of slot s of a dry cell c at a stage with flag
// buffers wp (the stage before) and wn (this one): the neighbour's flag of this stage is formed
// from its three nodes, e the larger ELF of the edge's two, as WET_JUDGE forms it.
template <bool RES>
__device__ __forceinline__ bool stage_wet_other(const Dev& P, int c, int s, int o, const int* wp, const int* wn, double e) {
  int wo = wp[o];
  if (P.wetting_drying_on && o != 0) {
    const double m = fmax(e, ldx<RES>(P.elf + P.wfar[(size_t)s * (P.N + 1) + c]));
    wo = wo * (((m + P.hmin[o]) - P.min_depth) < 1.0e-5 ? 0 : 1);
  } else {
    wo = wo * (P.wetting_drying_on ? wn[0] : P.iswetc[o]);
  }
  return wo == 1;
}

// Gradient and viscosity term of cell c (neighbours nb) with velocity u, v at stage st.
// T: threads per block of the resident loop, 0 in a stage kernel.
template <typename R, bool CS, int T>
__device__ __forceinline__ Grad<R> grad_job(const Dev& P, int c, int st, double u, double v, R& vc) {
  typedef Mesh<R> Mh;
  constexpr bool RES = T > 0;
  const double2* const uv = P.xuv + (st & 1) * (size_t)(P.N + 1);
  int k1, k2, k3;
  R A[4], B[4], art, cc;
  if constexpr (RES) {
    const LoopShared<R, T>& sm = loop_shared<R, T>();
    k1 = sm.nb[0][threadIdx.x];
    k2 = sm.nb[1][threadIdx.x];
    k3 = sm.nb[2][threadIdx.x];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      A[j] = sm.ab[j][threadIdx.x];
      B[j] = sm.ab[4 + j][threadIdx.x];
    }
    art = sm.ab[8][threadIdx.x];
    cc = sm.ab[9][threadIdx.x];
  } else {
    lsq_coef<R, CS>(P, c, k1, k2, k3, A, B);
    art = Mh::art(P, c);
    cc = Mh::cc_hvc(P, c);
  }
  const double2 b1 = ldx<RES>(uv + k1), b2 = ldx<RES>(uv + k2), b3 = ldx<RES>(uv + k3);
  const R half = (R)0.5;
  R u1 = (R)b1.x, u2 = (R)b2.x, u3 = (R)b3.x, v1 = (R)b1.y, v2 = (R)b2.y, v3 = (R)b3.y;
  if (P.gcy && (k1 == 0 || k2 == 0 || k3 == 0)) {
    double gu, gv;
    if (k1 == 0) { ghost_uv1(P, u, v, c, 1, gu, gv); u1 = (R)gu; v1 = (R)gv; }
    if (k2 == 0) { ghost_uv1(P, u, v, c, 2, gu, gv); u2 = (R)gu; v2 = (R)gv; }
    if (k3 == 0) { ghost_uv1(P, u, v, c, 3, gu, gv); u3 = (R)gu; v3 = (R)gv; }
  }
  Grad<R> g;
  g.ux = dot4(A[0], (R)u, A[1], u1, A[2], u2, A[3], u3);
  g.uy = dot4(B[0], (R)u, B[1], u1, B[2], u2, B[3], u3);
  g.vx = dot4(A[0], (R)v, A[1], v1, A[2], v2, A[3], v3);
  g.vy = dot4(B[0], (R)v, B[1], v1, B[2], v2, B[3], v3);
  st_xg<R>(P, c, g);
  vc = art * sqrt(g.ux * g.ux + g.vy * g.vy + half * ((g.uy + g.vx) * (g.uy + g.vx))) * cc;
  reinterpret_cast<R*>(P.xvc)[c] = vc;
  return g;
}

// What the resident loop keeps of a node between stages; the launched phases load it.
struct NodeKeep {
  double elf, el, elrk, d, egf, h, art1, riv[2];
  int ob, kind, nhe, nriv;
};
// EXTEL_EDGE, the boundary elevation and the previous stage's update of node i.  RES: the
// resident loop, whose z lives in registers.
template <typename R, bool CS, int T>
__device__ __forceinline__ void node_phase(const Dev& P, int i, int st, NodeKeep& z) {
  constexpr bool RES = T > 0;
  const int K = st % 4 + 1;
  const size_t ms = P.ms;
  if constexpr (!RES) {
    z.ob = ld1<CS>(P.node_obc + i);
    z.nhe = ld1<CS>(P.node_he_ptr + i + 1) - ld1<CS>(P.node_he_ptr + i);
    z.h = ld1<CS>(P.h + i);
    z.art1 = ld1<CS>(P.art1 + i);
    z.elf = st > 0 ? P.elf[i] : 0.0;
    z.el = st == 0 ? P.el[i] : 0.0;
    z.d = st == 0 ? P.d[i] : 0.0;
    z.elrk = st > 0 ? ld1<CS>(P.elrk + i) : 0.0;
    z.egf = K == 4 ? ld1<CS>(P.egf + i) : 0.0;
    z.nriv = P.numqbc > 0 ? P.node_riv_ptr[i + 1] - P.node_riv_ptr[i] : 0;
  }
  double x = 0.0;
  const int* L = P.node_vpos_ell + i;
  int j = 0;
  if constexpr (RES) {
    // the list's first entries at once
    const LoopShared<R, T>& sm = loop_shared<R, T>();
    int e[kLoopList];
    double f[kLoopList];
#pragma unroll
    for (int q = 0; q < kLoopList; ++q) e[q] = q < z.nhe ? sm.list[q][threadIdx.x] : 0;
#pragma unroll
    for (int q = 0; q < kLoopList; ++q) f[q] = q < z.nhe ? ldx<RES>(P.exf2d + (e[q] >> 1)) : 0.0;
#pragma unroll
    for (int q = 0; q < kLoopList; ++q)
      if (q < z.nhe) x = (e[q] & 1) ? x + f[q] : x - f[q];
    j = kLoopList;
  }
  for (; j + 6 <= z.nhe; j += 6) {
    int e[6];
    double f[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) e[q] = ld1<CS>(L + (j + q) * ms);
#pragma unroll
    for (int q = 0; q < 6; ++q) f[q] = ldx<RES>(P.exf2d + (e[q] >> 1));
#pragma unroll
    for (int q = 0; q < 6; ++q) x = (e[q] & 1) ? x + f[q] : x - f[q];
  }
  for (; j + 2 <= z.nhe; j += 2) {
    const int e0 = ld1<CS>(L + j * ms), e1 = ld1<CS>(L + (j + 1) * ms);
    const double f0 = ldx<RES>(P.exf2d + (e0 >> 1)), f1 = ldx<RES>(P.exf2d + (e1 >> 1));
    x = (e0 & 1) ? x + f0 : x - f0;
    x = (e1 & 1) ? x + f1 : x - f1;
  }
  if (j < z.nhe) {
    const int e0 = ld1<CS>(L + j * ms);
    const double f0 = ldx<RES>(P.exf2d + (e0 >> 1));
    x = (e0 & 1) ? x + f0 : x - f0;
  }
  if (st > 0) {
    // the previous stage's clamp (WET_JUDGE) and update (ext_update_node)
    if (P.wetting_drying_on) z.elf = fmax(z.elf, -z.h + P.min_depth);
    z.el = z.elf;
    z.d = z.h + z.elf;
    if (K == 4) {  // previous stage 3
      z.egf = z.egf + z.elf / (double)P.isplit;
      if constexpr (!RES) P.egf[i] = z.egf;
    }
    if (K == 1 && z.ob > 0) {
      const double tmp = -(z.elf - z.elrk) * z.art1 / P.dte - P.xflux_obcn[z.ob];
      P.uard_obcn[z.ob] = P.uard_obcn[z.ob] + tmp / (double)(float)P.isplit;
    }
  }
  if (K == 1) {
    z.elrk = z.el;
    if constexpr (!RES) P.elrk[i] = z.elrk;
  }
  if (z.ob > 0) {
    P.xflux_obcn[z.ob] = x;
    x = 0.0;
  }
  if (z.nriv > 0) {
    int q0 = P.node_riv_ptr[i];
    if constexpr (RES) {
      x = x - z.riv[0];
      if (z.nriv > 1) x = x - z.riv[1];
      q0 += 2;
    }
    for (int q = q0; q < P.node_riv_ptr[i + 1]; ++q) {
      const int r = P.node_riv[q], jr = r >> 1;
      x = x - (P.river_location == 0 ? P.qdis[jr] : P.qdis[jr] * P.rdisq[(size_t)(r & 1) * (P.numqbc + 1) + jr]);
    }
  }
  const double alpha = dAlphaRK[K], dtk = alpha * P.dte;
  z.elf = z.elrk - dtk * x / z.art1;
  if (z.ob > 0) {
    if constexpr (!RES) z.kind = P.obc_kind[z.ob];
    if (z.kind == 1) {
      if (P.obc_elev_on) z.elf = P.obf[(size_t)st * (P.iobcn + 1) + z.ob];
      z.elf = add_rn(z.elrk, mul_rn(alpha, z.elf - z.elrk));
    } else if (z.kind == 2) {
      z.elf = 0.0;
    }
    if constexpr (RES) P.elrk[i] = z.elrk;
  }
  P.elf[i] = z.elf;
  P.xnd[i] = make_double2(z.el, z.d);
}

// Slope limiters UALFA, VALFA of cell c for the limited ADVAVE (advave_edge_gcn.F:141-318), a
// phase of its own between the two: WET_JUDGE's cell flag, then the cell's three edges with a
// wet side, from its own gradient g and the two cells' velocities.
template <typename R, bool CS, int T>
__device__ __forceinline__ void alfa_phase(const Dev& P, int c, int st, const int4 xn, const int4 oo, int wce, double u,
                                           double v, const Grad<R>& g) {
  constexpr bool RES = T > 0;
  const size_t n1 = P.N + 1;
  const double2* const uv = P.xuv + (st & 1) * n1;
  const int* const wp = P.xw + ((st + 1) & 1) * n1;
  const int* const wn = P.xw + (st & 1) * n1;
  const bool wd = P.wetting_drying_on != 0;
  const int xs[3] = {xn.x, xn.y, xn.z}, os[3] = {oo.x, oo.y, oo.z};
  double2 ou[3];
  double en[3];
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    ou[s] = ldx<RES>(uv + os[s]);
    en[s] = ldx<RES>(P.elf + xs[s]);
  }
  int wetc = wd ? 0 : P.iswetc[c];
  if (wd) {
    const double dtmp = fmax(fmax(en[0], en[1]), en[2]) + P.hmin[c];
    wetc = ((dtmp - P.min_depth) < 1.0e-5) ? 0 : 1;
  }
  const bool wet = wce * wetc == 1;
  const double2 ci = P.xyc[c];
  R au = (R)1, av = (R)1;
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int o = os[s];
    if (!(wet || stage_wet_other<RES>(P, c, s, o, wp, wn, fmax(en[s], en[(s + 1) % 3])))) continue;
    const double2 v1 = P.vxy[xs[s]], v2 = P.vxy[xs[(s + 1) % 3]];
    const R x = (R)((v1.x + v2.x) * 0.5 - ci.x), y = (R)((v1.y + v2.y) * 0.5 - ci.y);
    lim_alfa<R>(fabs((R)u - (R)ou[s].x), g.ux * x + g.uy * y, au);
    lim_alfa<R>(fabs((R)v - (R)ou[s].y), g.vx * x + g.vy * y, av);
  }
  P.xal[c] = make_double2(au, av);
}

// What the resident loop keeps of a cell between stages; the launched phases load it.
template <typename R>
struct CellKeep {
  int4 xn, oo;  // loopx, loopo
  double u, v;
  Grad<R> g;
  R vc;
  // the resident loop's river and open-boundary entries (up to two of each)
  int bcriv, nobc, nriv, wce, wci, ob[2], obn[2];
  double obf[2], rvx[2], rvy[2];
};
template <typename R, bool CS, int T, bool LIM>
__device__ __forceinline__ void cell_phase(const Dev& P, int c, int st, CellKeep<R>& z) {
  typedef Mesh<R> Mh;
  constexpr bool RES = T > 0;
  LoopShared<R, RES ? T : 1>& sm = loop_shared<R, RES ? T : 1>();
  const int me = RES ? threadIdx.x : 0;
  const R half = (R)0.5, one = (R)1.0;
  const int iext = st / 4 + 1, K = st % 4 + 1, last = 4 * P.isplit - 1;
  const size_t n1 = P.N + 1, ns = P.ns;
  const double2* const uv = P.xuv + (st & 1) * n1;
  double2* const uvn = P.xuv + ((st + 1) & 1) * n1;
  int* const wn = P.xw + (st & 1) * n1;
  const int* const wp = P.xw + ((st + 1) & 1) * n1;
  const R* const xvc = reinterpret_cast<const R*>(P.xvc);
  const bool wd = P.wetting_drying_on != 0;
  if constexpr (!RES) {
    z.xn = ld1<CS>(P.loopx + c);
    z.oo = ld1<CS>(P.loopo + c);
  }
  // RES: what other threads wrote is loaded before the arithmetic and the stores, the rest comes
  // from shared memory; the launched phase, with many warps per SM and fewer registers, loads
  // the neighbours where they are used
  const int xs[3] = {z.xn.x, z.xn.y, z.xn.z}, os[3] = {z.oo.x, z.oo.y, z.oo.z};
  const int bits = z.xn.w, fl = z.oo.w, isbce = fl & 3;
  double2 nd[3], ou[3];
  double en[3], hn3[3];
  Grad<R> go[3];
  R vo[3];
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    nd[s] = ldx<RES>(P.xnd + xs[s]);
    en[s] = ldx<RES>(P.elf + xs[s]);
    if constexpr (RES) {
      ou[s] = ldx<RES>(uv + os[s]);
      go[s] = ld_xg<R, RES>(P, os[s]);
      vo[s] = ldx<RES>(xvc + os[s]);
    }
  }
  if constexpr (!RES) {
    const double2 own = uv[c];
    z.u = own.x;
    z.v = own.y;
    z.g = ld_xg<R, RES>(P, c);
    z.vc = xvc[c];
  }
  const double2 ci = RES ? sm.p2[3][me] : P.xyc[c];
#pragma unroll
  for (int s = 0; s < 3; ++s) hn3[s] = RES ? sm.p1[1 + s][me] : (wd ? P.h[xs[s]] : 0.0);
  const double u = z.u, v = z.v;
  const double d1i = RES ? sm.own[0][me] : ld1<CS>(P.d1 + c);
  const double2 rk = K == 1 ? make_double2(u, v)
                            : (RES ? make_double2(sm.own[3][me], sm.own[4][me]) : ld1<CS>(P.xrk + c));
  const double elrk1 = RES ? sm.own[K == 1 ? 1 : 2][me] : ld1<CS>((K == 1 ? P.el1 : P.elrk1) + c);
  const int wce = RES ? z.wce : wp[c], wci = wd ? 0 : (RES ? z.wci : P.iswetc[c]);  // ISWETCE; a fixed ISWETC
  const double hmin = RES ? sm.p1[0][me] : (wd ? ld1<CS>(P.hmin + c) : 0.0);
  double uard = 0.0, vard = 0.0;
  if (!RES && K == 3) {
    uard = ld1<CS>(P.uard + c);
    vard = ld1<CS>(P.vard + c);
  }
  const double ramp = sched_row(P)[P.sl.ramp_ext(iext)];
  // EXTUV's terms that stay fixed over the loop (store_fixed)
  double4 e0, e1;
  double2 ax2, ay2, wb, ws;
  double art, cor, h1i, grav;
  if constexpr (sizeof(R) == 4) {
    if constexpr (RES) {
      const double2 a = sm.p2[9][me], b = sm.p2[10][me];
      e1 = make_double4(a.x, a.y, b.x, b.y);
    } else {
      e1 = ld1<CS>(P.f.exc1 + c);
    }
    cor = e1.x;
    art = e1.y;
    h1i = e1.z;
    grav = e1.w;
  } else {
    const double2 hg = RES ? sm.p2[12][me] : ld1<CS>(P.exd + 5 * n1 + c);
    h1i = hg.x;
    grav = hg.y;
  }
  auto load_fixed = [&]() {
    if constexpr (sizeof(R) == 4) {
      if constexpr (RES) {
        const double2 a = sm.p2[7][me], b = sm.p2[8][me];
        e0 = make_double4(a.x, a.y, b.x, b.y);
      } else {
        e0 = ld1<CS>(P.f.exc0 + c);
      }
    } else {
      ax2 = RES ? sm.p2[7][me] : ld1<CS>(P.exd + c);
      ay2 = RES ? sm.p2[8][me] : ld1<CS>(P.exd + n1 + c);
      wb = RES ? sm.p2[9][me] : ld1<CS>(P.exd + 2 * n1 + c);
      ws = RES ? sm.p2[10][me] : ld1<CS>(P.exd + 3 * n1 + c);
      const double2 ca = RES ? sm.p2[11][me] : ld1<CS>(P.exd + 4 * n1 + c);
      cor = ca.x;
      art = ca.y;
    }
  };
  const double ged1 = grav * d1i;
  // WET_JUDGE's cell part, or N2E2D; the mean in NV order (its last node's place in bits)
  const int k3 = (bits >> 6) & 3;
  double cl[3] = {en[0], en[1], en[2]};
  int wetc = wci;
  if (wd) {
    const double md = P.min_depth;
    const double dtmp = fmax(fmax(en[0], en[1]), en[2]) + hmin;
    wetc = ((dtmp - md) < 1.0e-5) ? 0 : 1;
#pragma unroll
    for (int s = 0; s < 3; ++s) cl[s] = fmax(en[s], -hn3[s] + md);
  }
  const double l3 = k3 == 0 ? cl[0] : (k3 == 1 ? cl[1] : cl[2]);
  const double l12 = k3 == 0 ? cl[1] + cl[2] : (k3 == 1 ? cl[0] + cl[2] : cl[0] + cl[1]);
  const double elf1 = ONE_THIRD * (l12 + l3);
  const int weti = wce * wetc;
  // FLUX_OBN
  double fob = 0.0;
  if (fl & 8) {
    if (RES && z.nobc <= 2) {
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        if (q < z.nobc) {
          const int j = z.obn[q];
          const double ej0 = ldx<RES>(P.elf + j);
          const double ej = wd ? fmax(ej0, -P.h[j] + P.min_depth) : ej0;
          const double flux =
              -(ej - ldx<RES>(P.elrk + j)) * P.art1[j] / (dAlphaRK[K] * P.dte) - ldx<RES>(P.xflux_obcn + z.ob[q]);
          fob = fob + z.obf[q] * flux;
        }
      }
    } else {
      fob = fluxobn_cell(P, c, K);
    }
  }
  if ((fl & 8) || st == 0) P.fluxobn[c] = fob;
  if (K == 1) {
    if constexpr (RES) {
      sm.own[2][me] = elrk1;
      sm.own[3][me] = u;
      sm.own[4][me] = v;
    } else {
      P.elrk1[c] = elrk1;
      P.xrk[c] = rk;
    }
  }
  R xr = 0, yr = 0;
  double px = 0.0, py = 0.0;
  double exx[3], exy[3];  // XIJC-XC, YIJC-YC of the cell, which are DLTXE, DLTYE too
  const R epor = (fl & 32) ? one : (R)0, iucp = (fl & 64) ? one : (R)0;
  const R ui = (R)u, vi = (R)v, vci = z.vc;
  const Grad<R> gi = z.g;
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int side = (bits >> s) & 1, isbc = (bits >> (3 + s)) & 1, turn = (bits >> (8 + s)) & 1, o = os[s];
    const double2 na = nd[s], nbb = nd[(s + 1) % 3];
    const double2 v1 = RES ? sm.p2[s][me] : P.vxy[xs[s]];
    const double2 v2 = RES ? sm.p2[(s + 1) % 3][me] : P.vxy[xs[(s + 1) % 3]];
    const double xij = (v1.x + v2.x) * 0.5, yij = (v1.y + v2.y) * 0.5;
    const double edx = turn ? v1.x - v2.x : v2.x - v1.x, edy = turn ? v1.y - v2.y : v2.y - v1.y;
    exx[s] = xij - ci.x;
    exy[s] = yij - ci.y;
    const R dij = (R)(0.5 * (na.y + nbb.y));
    const double elij = 0.5 * (na.x + nbb.x);
    bool on = weti == 1;
    if (!on) on = stage_wet_other<RES>(P, c, s, o, wp, wn, fmax(en[s], en[(s + 1) % 3]));
    if (on) {
      const R dx = (R)edx, dy = (R)edy;
      const double2 co = RES ? sm.p2[4 + s][me] : P.xyc[o];
      const R xi = (R)exx[s], yi = (R)exy[s], xo = (R)(xij - co.x), yo = (R)(yij - co.y);
      const double2 uvo = RES ? ou[s] : uv[o];
      const Grad<R> gs = RES ? go[s] : ld_xg<R, RES>(P, o);
      const R uo = (R)uvo.x, vv = (R)uvo.y, vco = RES ? vo[s] : xvc[o];
      R uown, vown, uoth, voth;
      if constexpr (LIM) {
        const double2 ai = ldx<RES>(P.xal + c), ao = ldx<RES>(P.xal + o);
        lim_faces<R>(P.limiter, ui, uo, gi.ux * xi + gi.uy * yi, gs.ux * xo + gs.uy * yo, ai.x, ao.x, uown, uoth);
        lim_faces<R>(P.limiter, vi, vv, gi.vx * xi + gi.vy * yi, gs.vx * xo + gs.vy * yo, ai.y, ao.y, vown, voth);
      } else {
        uown = ui + gi.ux * xi + gi.uy * yi;
        vown = vi + gi.vx * xi + gi.vy * yi;
        uoth = uo + gs.ux * xo + gs.uy * yo;
        voth = vv + gs.vx * xo + gs.vy * yo;
      }
      const R uij = half * (uown + uoth), vij = half * (vown + voth);
      const R un = -uij * dy + vij * dx;
      R viscof = (R)P.fact * half * (vci + vco);
      viscof = viscof + (R)P.fm1 * half * (P.fm1 != 0.0 ? Mh::cc_hvc(P, c) + Mh::cc_hvc(P, o) : (R)0);
      if (P.hprnu != 1.0) viscof = viscof / (R)P.hprnu;
      const R vxa = side ? gs.vx : gi.vx, vxb = side ? gi.vx : gs.vx;
      const R txx = (gi.ux + gs.ux) * viscof;
      const R tyy = (gi.vy + gs.vy) * viscof;
      const R txy = half * (gi.uy + gs.uy + vxa + vxb) * viscof;
      const R fxx = dij * (txx * dy - txy * dx);
      const R fyy = dij * (txy * dy - tyy * dx);
      const R sg = fsign1(un), sgo = side ? -sg : sg;
      const R xadv = dij * un * ((one - sgo) * uoth + (one + sgo) * uown) * half;
      const R yadv = dij * un * ((one - sgo) * voth + (one + sgo) * vown) * half;
      const R nbd = one - (R)isbc;
      const R ax = (xadv + fxx * epor) * nbd * iucp, ay = (yadv + fyy * epor) * nbd * iucp;
      xr = side ? xr - ax : xr + ax;
      yr = side ? yr - ay : yr + ay;
    }
    const double tx = ged1 * elij * edy, ty = ged1 * elij * edx;
    px = side ? px + tx : px - tx;
    py = side ? py - ty : py + ty;
  }
  const R w = (R)weti;
  double xf = (double)(xr * w), yf = (double)(yr * w);
  if (isbce == 2) {
    const double iu = (fl & 64) ? 1.0 : 0.0;
    if (P.gcy) {
      xf = xf + fob * u * iu;
      yf = yf + fob * v * iu;
    } else {
      xf = (xf + fob * u) * iu;
      yf = (yf + fob * v) * iu;
    }
  }
  if (fl & 4) {
    int q0 = P.cell_riv_ptr[c];
    if constexpr (RES) {
      xf = xf - z.rvx[0];
      yf = yf - z.rvy[0];
      if (z.nriv > 1) {
        xf = xf - z.rvx[1];
        yf = yf - z.rvy[1];
      }
      q0 += 2;
    }
    for (int q = q0; q < P.cell_riv_ptr[c + 1]; ++q) {
      const int k = P.cell_riv[q] >> 1;
      const double vl = P.qdis[k] / P.qarea[k];
      const double t = P.river_location == 0 ? 0.5 * P.qdis[k] * vl : P.qdis[k] * vl;
      xf = xf - t * P.cos_angleq[k];
      yf = yf - t * P.sin_angleq[k];
    }
  }
  if (st == last) {
    P.advua[c] = xf;
    P.advva[c] = yf;
    P.pstx[c] = px;
    P.psty[c] = py;
  }
  double uaf = 0.0, vaf = 0.0;
  if (weti == 1) {
    const double a = dAlphaRK[K];
    load_fixed();
    double resx, resy;
    if constexpr (sizeof(R) == 4) {
      resx = e0.x + xf + px - cor * v * d1i - ramp * e0.z;
      resy = e0.y + yf + py + cor * u * d1i - ramp * e0.w;
    } else {
      const double wus = P.have_wind ? ws.x * ramp * 0.001 : 0.0;
      const double wvs = P.have_wind ? ws.y * ramp * 0.001 : 0.0;
      resx = ax2.x + xf + ax2.y + px - cor * v * d1i * art - (wus + wb.x) * art;
      resy = ay2.x + yf + ay2.y + py + cor * u * d1i * art - (wvs + wb.y) * art;
    }
    uaf = (rk.x * (h1i + elrk1) - a * P.dte * resx / art) / (h1i + elf1);
    vaf = (rk.y * (h1i + elrk1) - a * P.dte * resy / art) / (h1i + elf1);
  }
  if (fl & 16) {
    const double sp = RES ? sm.p1[4][me] : P.cc_sponge[c];
    uaf = uaf / (1.0 + sp * (uaf * uaf));
    vaf = vaf / (1.0 + sp * (vaf * vaf));
  }
  if (isbce == 3 && !P.gcy) { uaf = 0.0; vaf = 0.0; }
  if (isbce == 1) {
    const int rj = RES ? z.bcriv : P.cell_bcriv[c];
    if (!P.gcy || rj > 0) bc_solid(P, c, rj, uaf, vaf);
  }
  z.u = uaf;
  z.v = vaf;
  uvn[c] = make_double2(uaf, vaf);
  if (wd) wn[c] = wetc;
  else if (!RES || st < 2) wn[c] = wce;
  const double dd1 = h1i + elf1;
  if constexpr (RES) {
    z.wce = wd ? wetc : wce;
    sm.own[0][me] = dd1;
    sm.own[1][me] = elf1;
    if (K == 3) {
      sm.own[5][me] = sm.own[5][me] + uaf * dd1;
      sm.own[6][me] = sm.own[6][me] + vaf * dd1;
    }
  } else {
    P.el1[c] = elf1;
    P.d1[c] = dd1;
    if (K == 3) {
      P.uard[c] = uard + uaf * dd1;
      P.vard[c] = vard + vaf * dd1;
    }
  }
#pragma unroll
  for (int s = 0; s < 3; ++s) P.exf2d[(size_t)s * ns + c] = dd1 * (-uaf * exy[s] + vaf * exx[s]);
  if (st == last) {
    // as the general loop leaves its arrays before k_ext_finish
    P.elf1[c] = elf1;
    P.ua[c] = uaf;
    P.va[c] = vaf;
    P.uark[c] = rk.x;
    P.vark[c] = rk.y;
    if (wd) P.iswetce[c] = wetc;
    if constexpr (RES) {
      P.el1[c] = elf1;
      P.d1[c] = dd1;
      P.elrk1[c] = elrk1;
      P.uard[c] = sm.own[5][me];
      P.vard[c] = sm.own[6][me];
    }
  }
}

// One job per thread: nodes 1..M, then the cells' gradients.
template <typename R, bool CS>
__global__ void __launch_bounds__(256, 5) k_stage_node(const Dev P, int st) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.M) {
    const int c = i - P.M;
    if (c > P.N) return;
    const double2 own = P.xuv[(st & 1) * (size_t)(P.N + 1) + c];
    R vc;
    grad_job<R, CS, 0>(P, c, st, own.x, own.y, vc);
  } else {
    NodeKeep z;
    node_phase<R, CS, 0>(P, i, st, z);
  }
}
// Resident blocks per SM of the stage cell kernel, external mode of a step: FP64 four blocks of
// 128 registers 2,524 us against five of 96 (spilling 100 bytes) 2,905 (200k nodes; 50k 1,024
// against 1,122); FP32 six 923, seven 966, eight 996, five 1,005 (50k; 200k 2,302, 2,267,
// 2,447, 2,200).  One count serves every size: six lose 5 % of the external mode to five at
// 200k, five lose 9 % to six at 50k, whose cells fill one round of six and not of five.
template <typename R>
constexpr int kStageBlocks = sizeof(R) == 4 ? 6 : 4;
// WALK: one wave of blocks whose threads walk the cells.
template <typename R, bool CS, bool WALK, bool LIM>
__global__ void __launch_bounds__(128, kStageBlocks<R>) k_stage_cell(const Dev P, int st) {
  pdl_enter();
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  do {
    if (i > P.N) return;
    CellKeep<R> z;
    cell_phase<R, CS, 0, LIM>(P, i, st, z);
    i += gridDim.x * blockDim.x;
  } while (WALK);
}

template <typename R, bool CS>
__global__ void __launch_bounds__(128) k_stage_alfa(const Dev P, int st) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i > P.N) return;
  const size_t n1 = P.N + 1;
  const double2 own = P.xuv[(st & 1) * n1 + i];
  alfa_phase<R, CS, 0>(P, i, st, ld1<CS>(P.loopx + i), ld1<CS>(P.loopo + i), P.xw[((st + 1) & 1) * n1 + i], own.x, own.y,
                       ld_xg<R, false>(P, i));
}

// Barrier over the grid: every block adds one to the counter (zeroed by k_begin_step) and
// waits until all have, for at most bar_polls polls.  A block whose wait runs out reports it,
// sets the counter's top bit and leaves; the others leave at that bit, and so do the loops of
// the steps already queued behind (k_begin_step keeps it), whose state is that of a half-done
// stage.
__device__ __forceinline__ bool grid_barrier(const Dev& P, unsigned target) {
  __syncthreads();
  int ok = 1;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.bar) : "memory");
    unsigned seen = 0;
    int it = 0;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(P.bar) : "memory");
    } while (seen < target && ++it < P.bar_polls);
    if (seen < target || (seen & kBarStopped) || P.bar_polls == 0) {
      ok = 0;
      asm volatile("red.relaxed.gpu.global.or.b32 [%0], %1;" ::"l"(P.bar), "r"(kBarStopped) : "memory");
      *P.bar_err = 1;
    }
  }
  return __syncthreads_and(ok);
}

// SPLIT: the block's first half of threads holds its cells and the second half its nodes, so
// that the two jobs of a node phase run side by side on different warps.
template <typename R, int T, bool SPLIT, bool LIM>
__global__ void __launch_bounds__(T, 1) k_ext_loop(const __grid_constant__ Dev P) {
  const int tid = threadIdx.x, tn = SPLIT ? tid - T / 2 : tid;
  const int c = blockIdx.x * P.loop_cells + tid + 1, i = blockIdx.x * P.loop_nodes + tn + 1;
  const bool hc = tid < P.loop_cells && c <= P.N, hn = tn >= 0 && tn < P.loop_nodes && i <= P.M;
  LoopShared<R, T>& sm = loop_shared<R, T>();
  CellKeep<R> z;
  if (hc) {
    z.xn = P.loopx[c];
    z.oo = P.loopo[c];
    z.bcriv = (z.oo.w & 3) == 1 ? P.cell_bcriv[c] : 0;
    const int q0 = P.cell_obc_ptr[c];
    z.nobc = P.cell_obc_ptr[c + 1] - q0;
    for (int q = 0; q < 2; ++q) {
      z.ob[q] = z.obn[q] = 0;
      z.obf[q] = z.rvx[q] = z.rvy[q] = 0.0;
      if (q < z.nobc) {
        const int code = P.cell_obc[q0 + q];
        z.ob[q] = code >> 1;
        z.obn[q] = P.i_obc_n[code >> 1];
        z.obf[q] = P.fluxf_obc[(size_t)(code & 1) * (P.iobcn + 1) + (code >> 1)];
      }
    }
    const int r0 = P.cell_riv_ptr[c];
    z.nriv = P.cell_riv_ptr[c + 1] - r0;
    for (int q = 0; q < z.nriv && q < 2; ++q) {
      const int k = P.cell_riv[r0 + q] >> 1;
      const double vlctyq = P.qdis[k] / P.qarea[k];
      const double t = P.river_location == 0 ? 0.5 * P.qdis[k] * vlctyq : P.qdis[k] * vlctyq;
      z.rvx[q] = t * P.cos_angleq[k];
      z.rvy[q] = t * P.sin_angleq[k];
    }
    z.u = P.ua[c];
    z.v = P.va[c];
    const size_t n1 = P.N + 1;
    const int xs[3] = {z.xn.x, z.xn.y, z.xn.z}, os[3] = {z.oo.x, z.oo.y, z.oo.z};
    z.wce = P.iswetce[c];
    z.wci = P.iswetc[c];
    sm.own[0][tid] = P.d1[c];
    sm.own[1][tid] = P.el1[c];
    sm.own[5][tid] = P.uard[c];
    sm.own[6][tid] = P.vard[c];
    sm.p2[3][tid] = P.xyc[c];
    sm.p1[0][tid] = P.hmin[c];
    sm.p1[4][tid] = P.cc_sponge[c];
    for (int s = 0; s < 3; ++s) {
      sm.p2[s][tid] = P.vxy[xs[s]];
      sm.p2[4 + s][tid] = P.xyc[os[s]];
      sm.p1[1 + s][tid] = P.h[xs[s]];
    }
    if constexpr (sizeof(R) == 4) {
      const double4 e0 = P.f.exc0[c], e1 = P.f.exc1[c];
      sm.p2[7][tid] = make_double2(e0.x, e0.y);
      sm.p2[8][tid] = make_double2(e0.z, e0.w);
      sm.p2[9][tid] = make_double2(e1.x, e1.y);
      sm.p2[10][tid] = make_double2(e1.z, e1.w);
    } else {
      for (int q = 0; q < 6; ++q) sm.p2[7 + q][tid] = P.exd[q * n1 + c];
    }
    int k1, k2, k3;
    R A[4], B[4];
    lsq_coef<R>(P, c, k1, k2, k3, A, B);
    sm.nb[0][tid] = k1;
    sm.nb[1][tid] = k2;
    sm.nb[2][tid] = k3;
    for (int j = 0; j < 4; ++j) {
      sm.ab[j][tid] = A[j];
      sm.ab[4 + j][tid] = B[j];
    }
    sm.ab[8][tid] = Mesh<R>::art(P, c);
    sm.ab[9][tid] = Mesh<R>::cc_hvc(P, c);
  }
  NodeKeep y;
  if (hn) {
    y.elf = P.elf[i];
    y.el = P.el[i];
    y.d = P.d[i];
    y.elrk = 0.0;
    y.egf = P.egf[i];
    y.h = P.h[i];
    y.art1 = P.art1[i];
    y.ob = P.node_obc[i];
    y.kind = y.ob > 0 ? P.obc_kind[y.ob] : 0;
    y.nhe = P.node_he_ptr[i + 1] - P.node_he_ptr[i];
    for (int q = 0; q < kLoopList && q < y.nhe; ++q) sm.list[q][tid] = P.node_vpos_ell[q * (size_t)P.ms + i];
    const int r0 = P.node_riv_ptr[i];
    y.nriv = P.node_riv_ptr[i + 1] - r0;
    y.riv[0] = y.riv[1] = 0.0;
    for (int q = 0; q < y.nriv && q < 2; ++q) {
      const int r = P.node_riv[r0 + q], j = r >> 1;
      y.riv[q] = P.river_location == 0 ? P.qdis[j] : P.qdis[j] * P.rdisq[(size_t)(r & 1) * (P.numqbc + 1) + j];
    }
  }
  unsigned target = 0;
  const int nst = 4 * P.isplit;
  for (int st = 0; st < nst; ++st) {
    if (hn) node_phase<R, false, T>(P, i, st, y);
    if (hc) z.g = grad_job<R, false, T>(P, c, st, z.u, z.v, z.vc);
    if (!grid_barrier(P, target += gridDim.x)) return;
    if constexpr (LIM) {
      if (hc) alfa_phase<R, false, T>(P, c, st, z.xn, z.oo, z.wce, z.u, z.v, z.g);
      if (!grid_barrier(P, target += gridDim.x)) return;
    }
    if (hc) cell_phase<R, false, T, LIM>(P, c, st, z);
    if (st < nst - 1 && !grid_barrier(P, target += gridDim.x)) return;
  }
  if (hn) {
    P.el[i] = y.el;
    P.d[i] = y.d;
    P.egf[i] = y.egf;
    P.elrk[i] = y.elrk;
  }
}

// -------------------------------------------------------------------------------------
// external_step.F:333-436: EL=ELF, EL1=N2E2D(EL), D, D1, UA=UAF, DTFA, the K==3 sums
// for the 3-D correction, the K==4 open-boundary transport and WD_UPDATE(1).
// -------------------------------------------------------------------------------------
__global__ void k_ext_update(const Dev P, int K) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i <= P.M) ext_update_node(P, i, K);
  if (i <= P.N) {
    double u = P.uaf[i], v = P.vaf[i];
    P.ua[i] = u;
    P.va[i] = v;
    if (P.wetting_drying_on) P.iswetce[i] = P.iswetc[i];
    ext_update_cell(P, i, K, P.elf1[i], u, v);
  }
}

// After the last stage of a fused external loop: the node part of its update, and UAF,
// VAF, ISWETC made equal to UA, VA, ISWETCE as the copying update leaves them.
__global__ void k_ext_finish(const Dev P, int K, int wet_prev) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (i <= P.M) {
    if (wet_prev) wet_node(P, i, P.iswetce);
    ext_update_node(P, i, K);
  }
  if (i <= P.N) {
    P.uaf[i] = P.ua[i];
    P.vaf[i] = P.va[i];
    P.iswetc[i] = P.iswetce[i];
  }
}
// The specified elevation of every open-boundary node and stage of the external loop
// (BCOND_ASL, mod_obcs.F:554-583), for the loop's node phase: inside it the cosines were the
// longest chain of a stage, on a few threads.
__device__ inline void tide_entry(const Dev& P, int st, int ob) {
  if (P.obc_kind[ob] != 1) return;
  const int iext = st / 4 + 1, K = st % 4 + 1;
  const double* row = sched_row(P);
  double force = 0.0;
  for (int j = 0; j < P.ntide; ++j) {
    const size_t q = (size_t)j * (P.iobcn + 1) + ob;
    const double targ = row[P.sl.targ(iext, K, j)];
    force = add_rn(mul_rn(P.apt[q], cos(targ - P.phai_rad[q])), force);
  }
  force = force + P.emean[ob];
  P.obf[(size_t)st * (P.iobcn + 1) + ob] = force * row[P.sl.ramp_ext(iext)];
}
__global__ void k_ext_prep(const Dev P) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1;
  if (P.obc_elev_on)
    for (int q = i - 1; q < 4 * P.isplit * P.iobcn; q += gridDim.x * blockDim.x)
      tide_entry(P, q / P.iobcn, q % P.iobcn + 1);
  if (i > P.N) return;
  if (i == 1) {
    // the viscosity beside a boundary edge, in the form's type: the other form's values lie over it
    if (P.prec) reinterpret_cast<float*>(P.xvc)[0] = 0.f;
    else P.xvc[0] = 0.0;
  }
  store_grad<false>(P, i);
  store_exf(P, i);
  if (P.xform) {
    // the stages' exchange buffers: the loop reads buffer 0 first, and its flags in buffer 1
    const size_t n1 = P.N + 1;
    P.xuv[i] = make_double2(P.ua[i], P.va[i]);
    P.xw[n1 + i] = P.iswetce[i];
    if (i == 1) {  // the ghost cell 0 of both buffers and its gradient
      P.xuv[0] = make_double2(P.ua[0], P.va[0]);
      P.xuv[n1] = make_double2(P.uaf[0], P.vaf[0]);
      P.xw[0] = P.iswetc[0];
      P.xw[n1] = P.iswetce[0];
      if (P.limiter) P.xal[0] = make_double2(1.0, 1.0);
      if (!P.prec) {
        P.xg[0] = P.g2d[0][0];
        P.xg[1] = P.g2d[1][0];
        P.xg[2] = P.g2d[2][0];
        P.xg[3] = P.g2d[3][0];
      }
    }
  }
}

// Start of an internal step: advance the schedule slot, then BCOND_GCN(8,0)'s river ramp
// QDIS = QDIS*RAMP (bcond_gcn.F:645-648).
__global__ void k_begin_step(const Dev P, int advance) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const unsigned stopped = *P.bar & kBarStopped;  // a wait ran out: see grid_barrier
  int slot = P.ctl[0] + advance;
  P.ctl[0] = slot;
  *P.bar = stopped;
  double ramp = P.sched[(size_t)slot * P.sl.len];
  for (int j = 1; j <= P.numqbc; ++j) P.qdis[j] = P.qdis0[j] * ramp;
}

static inline int nblk(int n, int b) { return (n + b - 1) / b; }

void launch_ext_node(const Dev& P, cudaStream_t s, int iext, int K, int parts, int pdl) {
  const int n = (parts & EN_GRAD) ? P.M + P.N : P.M;
  const int b = col_threads(P, n, 256);
  launch_maybe_pdl(pdl, P.ldcs ? k_ext_node<true> : k_ext_node<false>, dim3(nblk(n, b)), dim3(b), s, P, iext, K,
                   parts);
}
void launch_ext_prep(const Dev& P, cudaStream_t s) { k_ext_prep<<<nblk(P.N, 256), 256, 0, s>>>(P); }
void launch_alfa2(const Dev& P, cudaStream_t s) {
  FVG_F32_FORWARD(launch_alfa2(P, s));
  k_alfa2<RF><<<nblk(P.N, 128), 128, 0, s>>>(P);
}

// FP32 copies of the mesh metrics the precision form's flux kernels read.
__global__ void k_d2f(const double* __restrict__ src, float* __restrict__ dst, size_t n) {
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x)
    dst[q] = (float)src[q];
}
__global__ void k_edge_offsets_f32(const Dev P) {
  int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e > P.NE) return;
  const size_t e1 = P.NE + 1;
  float xa = 0.f, ya = 0.f, xb = 0.f, yb = 0.f;
  if (e >= 1) {
    int ia = P.iec[e], ib = P.iec[e1 + e];
    xa = (float)(P.xijc[e] - P.xc[ia]);
    ya = (float)(P.yijc[e] - P.yc[ia]);
    xb = (float)(P.xijc[e] - P.xc[ib]);
    yb = (float)(P.yijc[e] - P.yc[ib]);
  }
  P.f.xo[e] = xa;
  P.f.yo[e] = ya;
  P.f.xo[e1 + e] = xb;
  P.f.yo[e1 + e] = yb;
}
// FP32 slot metrics packed per slot, each value rounded once from FP64
__global__ void k_pack_slots_f32(const Dev P) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= 3 * (size_t)(P.N + 1)) return;
  P.f.ce_geo[q] = make_float4((float)P.ce_xoa[q], (float)P.ce_yoa[q], (float)P.ce_xob[q], (float)P.ce_yob[q]);
  P.f.ce_dd[q] = make_float2((float)P.ce_dx[q], (float)P.ce_dy[q]);
}
// FP32 half-edge metrics per position and ring-edge metrics, packed, rounded once
__global__ void k_pack_he_f32(const Dev P) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t pl = P.ncvs;
  if (q < pl) {
    P.f.hg4[q] = make_float4((float)P.hg[q], (float)P.hg[pl + q], (float)P.hg[2 * pl + q], (float)P.hg[3 * pl + q]);
    P.f.hg2[q] = make_float2((float)P.hg[4 * pl + q], (float)P.hg[5 * pl + q]);
  }
  if (q < (size_t)P.trie_n) P.f.trie[q] = make_float2((float)P.dltytrie[q], (float)P.dltxtrie[q]);
  const size_t n1 = P.N + 1;
  if (q < n1) {
    P.f.a1u4[q] = make_float4((float)P.a1u[q], (float)P.a1u[n1 + q], (float)P.a1u[2 * n1 + q], (float)P.a1u[3 * n1 + q]);
    P.f.a2u4[q] = make_float4((float)P.a2u[q], (float)P.a2u[n1 + q], (float)P.a2u[2 * n1 + q], (float)P.a2u[3 * n1 + q]);
  }
}
void launch_make_f32(const Dev& P, cudaStream_t s) {
  auto cvt = [&](const double* a, float* b, size_t n) { k_d2f<<<296, 256, 0, s>>>(a, b, n); };
  const size_t n1 = P.N + 1, e1 = P.NE + 1;
  k_edge_offsets_f32<<<nblk(P.NE + 1, 256), 256, 0, s>>>(P);
  cvt(P.dltxc, P.f.dltxc, e1);
  cvt(P.dltyc, P.f.dltyc, e1);
  cvt(P.art, P.f.art, n1);
  cvt(P.cc_hvc, P.f.cc_hvc, n1);
  cvt(P.a1u, P.f.a1u, 4 * n1);
  cvt(P.a2u, P.f.a2u, 4 * n1);
  cvt(P.ce_xoa, P.f.ce_xoa, 3 * n1);
  cvt(P.ce_yoa, P.f.ce_yoa, 3 * n1);
  cvt(P.ce_xob, P.f.ce_xob, 3 * n1);
  cvt(P.ce_yob, P.f.ce_yob, 3 * n1);
  cvt(P.ce_dx, P.f.ce_dx, 3 * n1);
  cvt(P.ce_dy, P.f.ce_dy, 3 * n1);
  k_pack_slots_f32<<<nblk(3 * (P.N + 1), 256), 256, 0, s>>>(P);
  size_t npk = P.ncvs > P.trie_n ? P.ncvs : P.trie_n;
  if ((size_t)P.N + 1 > npk) npk = P.N + 1;
  k_pack_he_f32<<<nblk(npk, 256), 256, 0, s>>>(P);
}
void launch_wet_judge(const Dev& P, cudaStream_t s) {
  k_wet_cells<false><<<nblk(P.N, 256), 256, 0, s>>>(P);
  k_wet_nodes<<<nblk(P.M, 256), 256, 0, s>>>(P);
}
void launch_wet_cells(const Dev& P, cudaStream_t s, int pdl) {
  const int b = col_threads(P, P.N, 256);
  launch_maybe_pdl(pdl, P.ldcs ? k_wet_cells<true> : k_wet_cells<false>, dim3(nblk(P.N, b)), dim3(b), s, P);
}
void launch_ext_cell(const Dev& P, cudaStream_t s, int iext, int K, int parts, int pdl) {
  FVG_F32_FORWARD(launch_ext_cell(P, s, iext, K, parts, pdl));
  void (*k)(const Dev, int, int, int);
  k = P.limiter ? k_ext_cell<RF, kLimitedEdges> : per_edge(P) ? k_ext_cell<RF, kListed> : k_ext_cell<RF, kSeen>;
  const int b = col_threads(P, P.N, 128);
  launch_maybe_pdl(pdl, k, dim3(nblk(P.N, b)), dim3(b), s, P, iext, K, parts);
}
void launch_ext_update(const Dev& P, cudaStream_t s, int K) {
  int n = P.M > P.N ? P.M : P.N;
  k_ext_update<<<nblk(n, 256), 256, 0, s>>>(P, K);
}
void launch_ext_finish(const Dev& P, cudaStream_t s, int K, int wet_prev) {
  int n = P.M > P.N ? P.M : P.N;
  k_ext_finish<<<nblk(n, 256), 256, 0, s>>>(P, K, wet_prev);
}
// A limited scheme runs on the packed records in FP64 only.  LIMITED_1's clamp is
// discontinuous: the packed FP32 form's rounding (a few 1e-9 of the fields) would switch it on
// other edges, so that form keeps the general kernels.
constexpr bool kLimited = sizeof(RF) == 8;
template <int T, bool SPLIT>
static void loop_launch(const Dev& P, cudaStream_t s, int grid) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(T);
  cfg.dynamicSmemBytes = sizeof(LoopShared<RF, T>);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  Dev Q = P;
  Q.loop_cells = nblk(P.N, grid);
  Q.loop_nodes = nblk(P.M, grid);
  void (*k)(const Dev) = k_ext_loop<RF, T, SPLIT, false>;
  if constexpr (kLimited) {
    if (P.limiter) k = k_ext_loop<RF, T, SPLIT, true>;
  }
  cudaLaunchKernelEx(&cfg, k, Q);
}
// Shared memory of the resident loop's blocks (once, before any launch or capture); 0 on success.
template <int T, bool SPLIT>
static int loop_attr() {
  int bad = 0;
  for (auto k : {k_ext_loop<RF, T, SPLIT, false>, k_ext_loop<RF, T, SPLIT, kLimited>})
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LoopShared<RF, T>)) != cudaSuccess)
      bad = 1;
  return bad;
}
int ext_loop_setup() { return loop_attr<256, true>() | loop_attr<256, false>() | loop_attr<kLoopThreads, false>(); }
// One block per SM at most, the smallest that then holds a cell and a node per thread, so that
// the threads spread over the SMs.  256 threads take 250 registers each and spill nothing; up
// to 128 cells per SM they leave half of the threads to the nodes.  One cluster of sixteen
// blocks with its hardware barrier in place of the grid's measured no faster (2,121 nodes 492
// against 491 us per step): a phase waits on its own loads and arithmetic more than on the
// barrier.
void launch_ext_loop(const Dev& P, cudaStream_t s) {
  FVG_F32_FORWARD(launch_ext_loop(P, s));
  const int most = P.N > P.M ? P.N : P.M, need = nblk(most, P.nsm);
  if (need <= 128)
    loop_launch<256, true>(P, s, nblk(most, 128));
  else if (need <= 256)
    loop_launch<256, false>(P, s, P.nsm);
  else
    loop_launch<kLoopThreads, false>(P, s, P.nsm);
}
// Stage st of the launched loop: its two phases as kernels, each a programmatic dependent of
// the one before (not the first).
void launch_ext_stage(const Dev& P, cudaStream_t s, int st) {
  FVG_F32_FORWARD(launch_ext_stage(P, s, st));
  const int n = P.M + P.N, bn = col_threads(P, n, 256);
  launch_maybe_pdl(st > 0, P.ldcs ? k_stage_node<RF, true> : k_stage_node<RF, false>, dim3(nblk(n, bn)), dim3(bn), s,
                   P, st);
  const int b = col_threads(P, P.N, 128), nb = nblk(P.N, b);
  if constexpr (kLimited) {
    if (P.limiter)
      launch_maybe_pdl(1, P.ldcs ? k_stage_alfa<RF, true> : k_stage_alfa<RF, false>, dim3(nb), dim3(b), s, P, st);
  }
  const int wave = (P.ext_grid < kStageBlocks<RF> ? P.ext_grid : kStageBlocks<RF>)*P.nsm;
  const bool walk = P.ext_grid > 0 && nb > wave;
  auto k = [&](auto lim) {
    constexpr bool L = decltype(lim)::value;
    return walk ? (P.ldcs ? k_stage_cell<RF, true, true, L> : k_stage_cell<RF, false, true, L>)
                : (P.ldcs ? k_stage_cell<RF, true, false, L> : k_stage_cell<RF, false, false, L>);
  };
  launch_maybe_pdl(1, P.limiter ? k(std::bool_constant<kLimited>()) : k(std::false_type()), dim3(walk ? wave : nb),
                   dim3(b), s, P, st);
}
void launch_begin_step(const Dev& P, cudaStream_t s) { k_begin_step<<<1, 32, 0, s>>>(P, 1); }
void launch_set_qdis(const Dev& P, cudaStream_t s) { k_begin_step<<<1, 32, 0, s>>>(P, 0); }

}  // namespace fvg / fvg_f32
