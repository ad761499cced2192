// CUDA kernels of the GAMERA-OP single-domain MHD step for B200 (sm_100a).
//
// One step (src/solver_solve.c:103-508) is a fixed sequence of launches on
// one stream, all reading dt and the AB2 coefficient from device memory so
// the sequence can be captured in a CUDA graph and replayed without host
// synchronisation:
//
//   ab2       W_h, mags, mags_h, B_h over the ghost-extended grid
//   flux      PDM reconstruction + Rusanov flux + Maxwell stress per face; the
//             first centre-to-edge sweep where it has the face's states
//   c2c       centre-to-edge velocity, first sweep, in the ghost layers of
//             axes that are not periodic (3 edge directions)
//   emf       centre-to-edge second sweep, face-B reconstruction, edge EMF
//   update    divergence, sources, constrained transport, cons->prim,
//             floors, Alfven/Boris correction, next CFL dt, max|div B|
//   ghost     periodic wrap and boundary fills of the new state; its last
//             block ends the step (the written buffer becomes the current
//             state) and opens the next one: dt <- running CFL minimum, time
//             += dt, c = dt/(2 dt0)
//
// (the first step of a call is opened by k_arm, which sets its budget)
//
// Every stage is a per-point body function of a kernel whose launch grid
// covers one grid; a batch of grids captures each member's launches on
// parallel branches of one CUDA graph.
//
// R is the arithmetic type of the reconstruction / flux / EMF stages
// (double: plain path; float: mixed path).  The state, the AB2
// extrapolation, the conservative update and the pressure recovery are FP64
// in both.
#include "gop_device.cuh"
#include "gop_kernels.h"
#include "gop_stage.cuh"
#include "gop_update.cuh"

#include <algorithm>
#include <type_traits>
#include <atomic>
#include <cfloat>

namespace gop {

// ------------------------------------------------------------------ utils


// rows of cells whose state or face field the pole ring average changes
// (the ring rows and the rows of the faces its EMF-like field touches)
__device__ __forceinline__ bool ring_band_row(const Params& P, int j) {
  const int jm = P.ring_jmax;
  return ((P.ring & 1) && j >= NGH && j <= NGH + jm + 1) ||
         ((P.ring & 2) && j >= NGH + P.n[1] - 2 - jm && j <= NGH + P.n[1] - 1);
}

// cell-centred B from the two faces along each axis (src/solver_func.c:311-322)
__device__ __forceinline__ double mags_at(const Params& P, const double* B, int a, int i, int j,
                                          int k) {
  long long c = lin(P, i, j, k);
  int idx = a == 0 ? i : (a == 1 ? j : k);
  const double* f = B + (size_t)a * P.fs;
  return f[c] * tb(P, a, T_MA, idx) + f[c + stride(P, a)] * tb(P, a, T_MB, idx);
}

template <int AX>
__device__ __forceinline__ long long sd(const Params& P) {
  return AX == 0 ? 1LL : (AX == 1 ? P.sj : P.sk);
}

// v[0..7] = a[(t-4)*s]: cells f-4..f+3 along stride s, a pointing at cell f
template <typename R, typename T>
__device__ __forceinline__ void line8(const T* __restrict__ a, long long s, R v[8]) {
#pragma unroll
  for (int t = 0; t < 8; t++) v[t] = (R)a[(t - 4) * s];
}



__device__ __forceinline__ Pos grid_pos() {
  return {(int)(blockIdx.x * blockDim.x + threadIdx.x), (int)(blockIdx.y * blockDim.y + threadIdx.y),
          (int)(blockIdx.z * blockDim.z + threadIdx.z)};
}
// ---------------------------------------------------------- step control

// open the step (src/solver_solve.c:103-107, src/solver_func.c:385-491):
// dt from the running CFL minimum, time, AB2 coefficient; stop once the
// previous step passed time_stop or the step budget is spent
__device__ __forceinline__ void begin_body(const Params& P) {
  double* s = P.scal;
  if (s[S_STOP] != 0.0) return;
  if (s[S_TIME] > s[S_TSTOP] || s[S_BUDGET] <= 0.0) {
    s[S_STOP] = 1.0;
    return;
  }
  s[S_BUDGET] = s[S_BUDGET] - 1.0;
  const double dt = s[S_NEXT_DT];
  if ((!(dt > 0.0) || !isfinite(dt)) && s[S_FLAGS] == 0.0) s[S_FLAGS] = 1.0;  // (one thread: no atomic)
  s[S_DT] = dt;
  s[S_TIME] = s[S_TIME] + dt;
  s[S_CAB2] = 0.5 * dt / s[S_DT0];
  s[S_DT0] = dt;
  s[S_NEXT_DT] = DBL_MAX;
  s[S_DIVB] = 0.0;
  s[S_STEPS] = s[S_STEPS] + 1.0;
}

// close the step: the buffer written by this step becomes the current state
__device__ __forceinline__ void end_body(const Params& P) {
  if (P.scal[S_STOP] != 0.0) return;
  P.scal[S_PAR] = P.scal[S_PAR] != 0.0 ? 0.0 : 1.0;
}

__device__ __forceinline__ void arm_body(const Params& P, double tstop, double budget) {
  P.scal[S_TSTOP] = tstop;
  P.scal[S_BUDGET] = budget;
  P.scal[S_STOP] = 0.0;
}

// ------------------------------------------------------------------- AB2

// W_h = W + c (W - W_old), mags and mags_h from the faces, B_h on faces
// (src/solver_func.c:385-449) over the whole ghost-extended grid; PSL false:
// p_S and its extrapolation stay zero (Params::ps_live) and are not touched
template <typename R, bool PSL>
__device__ __forceinline__ void ab2_body(const Params& P, const Work<R>& w, Pos t) {
  const int i = t.x, j = t.y, k = t.z;
  if (i >= P.N[0] || j >= P.N[1] || k >= P.N[2]) return;
  const int cb = cur_buf(P);
  const double* __restrict__ W = P.Wbuf[cb];
  const double* __restrict__ Wo = P.Wbuf[1 - cb];
  const double* __restrict__ B = P.Bbuf[cb];
  const double* __restrict__ Bo = P.Bbuf[1 - cb];
  const double c = P.scal[S_CAB2];
  const long long x = lin(P, i, j, k);
  const size_t fs = P.fs;
  const bool ci = i < P.N[0] - 1, cj = j < P.N[1] - 1, ck = k < P.N[2] - 1;
  // all loads first, then the stores: with FP64 work arrays the compiler
  // cannot tell them from the state, and a store between two loads would
  // keep the second from being issued ahead
  constexpr int NW = PSL ? 6 : 5;
  const bool inner = ci && cj && ck;
  double v[NW], vo[NW], ms[3], mo[3], b[3], bo[3];
  bool ok[3];
  if (inner) {
#pragma unroll
    for (int m = 0; m < NW; m++) {
      v[m] = W[x + m * fs];
      vo[m] = Wo[x + m * fs];
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      ms[a] = mags_at(P, B, a, i, j, k);
      mo[a] = mags_at(P, Bo, a, i, j, k);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    ok[a] = (a == 0 || ci) && (a == 1 || cj) && (a == 2 || ck);
    if (ok[a]) {
      b[a] = B[x + a * fs];
      bo[a] = Bo[x + a * fs];
    }
  }
  if (inner) {
#pragma unroll
    for (int m = 0; m < NW; m++) {
      w.Wh[x + m * fs] = (R)(v[m] + c * (v[m] - vo[m]));
      if constexpr (sizeof(R) == 4) w.Wl[x + m * fs] = (R)v[m];
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      w.Ms[x + a * fs] = (R)ms[a];
      w.Msh[x + a * fs] = (R)(ms[a] + c * (ms[a] - mo[a]));
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    if (ok[a]) {
      w.Bh[x + a * fs] = (R)(b[a] + c * (b[a] - bo[a]));
      if constexpr (sizeof(R) == 4) w.Bl[x + a * fs] = (R)b[a];
    }
  }
}

// ------------------------------------------------------------- edge EMF

// First centre-to-edge sweep of center2corner_{jk,ki,ij}
// (src/solver_func.c:686-778): for edges along D, velocity components
// p=(D+1)%3 and q=(D+2)%3 reconstructed along p (limiter on the step-start
// velocity) and averaged, at D active, p faces lo..hi+1, q over all cells
// including ghosts.  Over the active q range these are exactly the
// velocity states the face flux along p reconstructs (same inputs, same
// weights), so the flux stage writes them there and this kernel covers only
// the 2*NGH ghost layers of q.
template <typename R, int D>
__device__ __forceinline__ void c2c_body(const Params& P, const Work<R>& wk, Pos t) {
  constexpr int p = (D + 1) % 3, q = (D + 2) % 3;
  int ijk[3] = {t.x, t.y, t.z};
  int cnt[3], lo[3];
  lo[D] = NGH; cnt[D] = P.n[D];
  lo[p] = NGH; cnt[p] = P.n[p] + 1;
  lo[q] = 0;   cnt[q] = 2 * NGH;
  if (ijk[0] >= cnt[0] || ijk[1] >= cnt[1] || ijk[2] >= cnt[2]) return;
  if (ijk[q] >= NGH) ijk[q] += P.n[q];  // upper ghost layers
  const int i = ijk[0] + lo[0], j = ijk[1] + lo[1], k = ijk[2] + lo[2];
  const int f = p == 0 ? i : (p == 1 ? j : k);
  const long long x = lin(P, i, j, k), s = sd<p>(P);
  const size_t fs = P.fs;
  const R* __restrict__ W = lim_w<R>(P, wk) + x;
  FaceWeights<R> Wt;
  load_face_weights<p, R>(wk.tab, wk.fw, P.tmax, f, Wt);
#pragma unroll
  for (int cc = 0; cc < 2; cc++) {
    const int comp = cc == 0 ? p : q;
    R v[8], lim[4], L, Rr;
    line8<R, R>(wk.Wh + (size_t)(V1 + comp) * fs + x, s, v);
#pragma unroll
    for (int u = 0; u < 4; u++) lim[u] = W[(V1 + comp) * fs + (u - 2) * s];
    recon_lr<p == 1>(v, lim, Wt, L, Rr);
    wk.V[x + (size_t)(2 * D + cc) * fs] = R(0.5) * (L + Rr);
  }
}

// Second sweep, face-field reconstruction and the edge EMF
// (src/solver_func.c:779-902) for edges along D: D active, p and q faces.
template <typename R, int D, bool BG>
__device__ __forceinline__ void emf_body(const Params& P, const Work<R>& wk, Pos t) {
  constexpr int p = (D + 1) % 3, q = (D + 2) % 3;
  const int ijk[3] = {t.x, t.y, t.z};
  int cnt[3];
  cnt[D] = P.n[D];
  cnt[p] = P.n[p] + 1;
  cnt[q] = P.n[q] + 1;
  if (ijk[0] >= cnt[0] || ijk[1] >= cnt[1] || ijk[2] >= cnt[2]) return;
  const int i = ijk[0] + NGH, j = ijk[1] + NGH, k = ijk[2] + NGH;
  const int pos[3] = {i, j, k};
  const long long x = lin(P, i, j, k), sp = sd<p>(P), sq = sd<q>(P);
  const size_t fs = P.fs;
  const R* __restrict__ B = lim_b<R>(P, wk) + x;
  R vav[2], bpl, bpr, bql, bqr;
  {
    FaceWeights<R> Wt;
    load_face_weights<q, R>(wk.tab, wk.fw, P.tmax, pos[q], Wt);
#pragma unroll
    for (int cc = 0; cc < 2; cc++) {
      R v[8], lim[4], L, Rr;
      line8<R, R>(wk.V + (size_t)(2 * D + cc) * fs + x, sq, v);
#pragma unroll
      for (int u = 0; u < 4; u++) lim[u] = v[u + 2];
      recon_lr<q == 1>(v, lim, Wt, L, Rr);
      vav[cc] = R(0.5) * (L + Rr);
    }
    // B_p along q
    R v[8], lim[4];
    line8<R, R>(wk.Bh + (size_t)p * fs + x, sq, v);
#pragma unroll
    for (int u = 0; u < 4; u++) lim[u] = B[p * fs + (u - 2) * sq];
    recon_lr<q == 1>(v, lim, Wt, bpl, bpr);
  }
  {
    // B_q along p
    FaceWeights<R> Wt;
    load_face_weights<p, R>(wk.tab, wk.fw, P.tmax, pos[p], Wt);
    R v[8], lim[4];
    line8<R, R>(wk.Bh + (size_t)q * fs + x, sp, v);
#pragma unroll
    for (int u = 0; u < 4; u++) lim[u] = B[q * fs + (u - 2) * sp];
    recon_lr<p == 1>(v, lim, Wt, bql, bqr);
  }
  R b0p = R(0), b0q = R(0);
  if constexpr (BG) {  // B0 averaged along the edge (B0Aedge*)
    b0p = (R)P.bg[(size_t)(BG_EDGE + 3 * D + p) * fs + x];
    b0q = (R)P.bg[(size_t)(BG_EDGE + 3 * D + q) * fs + x];
  }
  const R* rh = wk.Wh + x;  // density slot
  // the reference sums the four densities around the edge in (i,j,k) order
  const R rho4 = D == 1 ? rh[-sq - sp] + rh[-sq] + rh[-sp] + rh[0]
                        : rh[-sp - sq] + rh[-sp] + rh[-sq] + rh[0];
  const R e = emf_finish<R, BG>(P, vav[0], vav[1], bpl, bpr, bql, bqr, b0p, b0q, rho4);
  wk.E[x + (size_t)D * fs] = e;
}

// ------------------------------------------------------------ face flux


// PDM reconstruction of the 9 face states, then flux_out: one thread per face
// (PSL: the entropy channel p_S is live, Params::ps_live)
template <typename R, int D, bool BG, bool PSL>
__device__ __forceinline__ void flux_body(const Params& P, const Work<R>& wk, Pos t) {
  const int i = NGH + t.x, j = NGH + t.y, k = NGH + t.z;
  if (i >= NGH + P.n[0] + (D == 0) || j >= NGH + P.n[1] + (D == 1) ||
      k >= NGH + P.n[2] + (D == 2))
    return;
  const int f = D == 0 ? i : (D == 1 ? j : k);
  const long long x = lin(P, i, j, k), s = sd<D>(P);
  const size_t fs = P.fs;
  const R* __restrict__ W = lim_w<R>(P, wk) + x;
  FaceWeights<R> Wt;
  load_face_weights<D, R>(wk.tab, wk.fw, P.tmax, f, Wt);
  R L[6], Rt[6], mL[3], mR[3];
  // PSL false: p_S is identically zero (Params::ps_live), its face states
  // are zero and flux_out's zero path gives the zero entropy flux that
  // reconstructing the zero line would give
  L[PS] = Rt[PS] = R(0);
#pragma unroll
  for (int m = 0; m < 6; m++) {
    if (m == PS && !PSL) continue;
    R v[8], lim[4];
    line8<R, R>(wk.Wh + (size_t)m * fs + x, s, v);
#pragma unroll
    for (int u = 0; u < 4; u++) lim[u] = W[m * fs + (u - 2) * s];
    recon_lr<D == 1>(v, lim, Wt, L[m], Rt[m]);
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    R v[8], lim[4];
    line8<R, R>(wk.Msh + (size_t)a * fs + x, s, v);
    const R* ms = wk.Ms + (size_t)a * fs + x;
#pragma unroll
    for (int u = 0; u < 4; u++) lim[u] = ms[(u - 2) * s];
    recon_lr<D == 1>(v, lim, Wt, mL[a], mR[a]);
  }
  flux_out<R, D, BG, PSL>(P, wk, (int)x, D == 0 ? j : (D == 1 ? k : i), L, Rt, mL, mR,
                          lim_b<R>(P, wk)[x + D * fs]);
}

// --------------------------------------------------------------- update

// new face field of component A at face (i,j,k) by constrained transport
// (src/solver_solve.c:263-306)
template <int COORD, int A, typename R>
__device__ __forceinline__ double ct_face(const Params& P, const double* __restrict__ B,
                                          const R* __restrict__ E, int i, int j, int k,
                                          double dt) {
  constexpr int p = (A + 1) % 3, q = (A + 2) % 3;
  const long long x = lin(P, i, j, k), sp = sd<p>(P), sq = sd<q>(P);
  const int ip = i + (p == 0), jp = j + (p == 1), kp = k + (p == 2);
  const int iq = i + (q == 0), jq = j + (q == 1), kq = k + (q == 2);
  const size_t fs = P.fs;
  const double cq = (double)E[x + sp + q * fs] * Geo<COORD>::edge(P, q, ip, jp, kp) -
                    (double)E[x + q * fs] * Geo<COORD>::edge(P, q, i, j, k);
  const double cp = (double)E[x + sq + p * fs] * Geo<COORD>::edge(P, p, iq, jq, kq) -
                    (double)E[x + p * fs] * Geo<COORD>::edge(P, p, i, j, k);
  return B[x + A * fs] - dt * (cq - cp) / Geo<COORD>::face(P, A, i, j, k);
}

// Constrained transport of a spherical grid (src/solver_solve.c:263-306) in a
// launch of its own before the update: with the pole ring average, whose pole
// faces take their field from faces half a turn away, and on the mixed path
// (see update_sph).  Every active cell writes its three lower
// faces, the last cell along an axis also the upper boundary face, so each
// face (with its division by the face area) is computed once
template <int COORD, typename R>
__device__ __forceinline__ void ct_body(const Params& P, const Work<R>& wk, Pos t) {
  const int i = NGH + t.x, j = NGH + t.y, k = NGH + t.z;
  if (i >= NGH + P.n[0] || j >= NGH + P.n[1] || k >= NGH + P.n[2]) return;
  const size_t fs = P.fs;
  const double dt = P.scal[S_DT];
  const int cb = cur_buf(P);
  const double* __restrict__ B = P.Bbuf[cb];
  double* __restrict__ Bn = P.Bbuf[1 - cb];
  const R* __restrict__ E = wk.E;
  const long long x = lin(P, i, j, k);
  const bool last[3] = {i == NGH + P.n[0] - 1, j == NGH + P.n[1] - 1, k == NGH + P.n[2] - 1};
  double bl[3], bu[3] = {0.0, 0.0, 0.0};
  bl[0] = ct_face<COORD, 0, R>(P, B, E, i, j, k, dt);
  bl[1] = ct_face<COORD, 1, R>(P, B, E, i, j, k, dt);
  bl[2] = ct_face<COORD, 2, R>(P, B, E, i, j, k, dt);
  if (last[0]) bu[0] = ct_face<COORD, 0, R>(P, B, E, i + 1, j, k, dt);
  if (last[1]) bu[1] = ct_face<COORD, 1, R>(P, B, E, i, j + 1, k, dt);
  if (last[2]) bu[2] = ct_face<COORD, 2, R>(P, B, E, i, j, k + 1, dt);
  if (COORD == 2 && P.ring) {
    // B_j on a pole face (zero area) from the face next to it and the one
    // half a turn away in phi (tackle_Magfield_pole,
    // spherical_RingAverage.c:205-233)
    const int ko = NGH + (k - NGH + P.n[2] / 2) % P.n[2];
    if ((P.ring & 1) && j == NGH)
      bl[1] = 0.5 * (ct_face<COORD, 1, R>(P, B, E, i, j + 1, k, dt) -
                     ct_face<COORD, 1, R>(P, B, E, i, j + 1, ko, dt));
    if ((P.ring & 2) && last[1])
      bu[1] = 0.5 * (bl[1] - ct_face<COORD, 1, R>(P, B, E, i, j, ko, dt));
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    Bn[x + a * fs] = bl[a];
    if (last[a]) Bn[x + stride(P, a) + a * fs] = bu[a];
  }
}

// one active cell: returns its CFL rate and |div B| of the new state.  After
// k_ct (spherical grids, see update_sph): the
// flux divergence, the geometric sources, the Alfven/Boris correction and
// the CFL estimate are in R (FP32 on the mixed path); the face fields, the
// conservative update and the pressure recovery are FP64.
template <int COORD, typename R, bool BG, bool PSL, bool CT>
__device__ __forceinline__ void update_body(const Params& P, const Work<R>& wk, Pos t,
                                            double& rate, double& dbmax) {
  if constexpr (COORD == 0) {
    const int ci = NGH + t.x, cj = NGH + t.y, ck = NGH + t.z;
    if (ci >= NGH + P.n[0] || cj >= NGH + P.n[1] || ck >= NGH + P.n[2]) return;
    update_cart<R, BG, PSL>(P, PointReader<R>(P, wk, ci, cj, ck), ci, cj, ck, rate, dbmax);
    return;
  } else if constexpr (COORD == 2 && !CT && sizeof(R) == 8) {
    const int ci = NGH + t.x, cj = NGH + t.y, ck = NGH + t.z;
    if (ci >= NGH + P.n[0] || cj >= NGH + P.n[1] || ck >= NGH + P.n[2]) return;
    update_sph<BG, PSL>(P, wk, PointReader<R>(P, wk, ci, cj, ck), ci, cj, ck, rate, dbmax);
    return;
  }
  const int i = NGH + t.x, j = NGH + t.y, k = NGH + t.z;
  if (i >= NGH + P.n[0] || j >= NGH + P.n[1] || k >= NGH + P.n[2]) return;
  const size_t fs = P.fs;
  const double dt = P.scal[S_DT];
  const int cb = cur_buf(P);
  const double* __restrict__ W = P.Wbuf[cb];
  const double* __restrict__ B = P.Bbuf[cb];
  double* __restrict__ Wn = P.Wbuf[1 - cb];
  double* __restrict__ Bn = P.Bbuf[1 - cb];
  const R* __restrict__ F = wk.F;
  const long long x = lin(P, i, j, k);
  const double vol = Geo<COORD>::vol(P, i, j, k);
  const double ivol = 1.0 / vol;
  const R rivol = (R)ivol;
  R du[6], dm[3];
  double fl[3], fu[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const long long s = stride(P, d);
    const int i1 = i + (d == 0), j1 = j + (d == 1), k1 = k + (d == 2);
    fl[d] = Geo<COORD>::face(P, d, i, j, k);
    fu[d] = Geo<COORD>::face(P, d, i1, j1, k1);
    const R* Fd = F + (size_t)(9 * d) * fs + x;
#pragma unroll
    for (int m = 0; m < 6; m++) {
      if (m == PS && !PSL) continue;
      const R v = ((R)Fd[s + m * fs] * (R)fu[d] - (R)Fd[m * fs] * (R)fl[d]) * rivol;
      du[m] = d == 0 ? v : du[m] + v;
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const R v = ((R)Fd[s + (6 + a) * fs] * (R)fu[d] - (R)Fd[(6 + a) * fs] * (R)fl[d]) * rivol;
      dm[a] = d == 0 ? v : dm[a] + v;
    }
  }
  if constexpr (BG) {  // + the Lorentz force of B0 (src/solver_solve.c:312-324)
#pragma unroll
    for (int a = 0; a < 3; a++) dm[a] += (R)P.bg[(size_t)(BG_LOR + a) * fs + x];
  }
  // spherical geometric sources (src/spherical/spherical_general.c:605-681)
  R sh[3] = {R(0), R(0), R(0)}, sb[3] = {R(0), R(0), R(0)};
  if (COORD == 2) {
    const long long si = 1, sjj = P.sj;
    const R fi0 = (R)fl[0], fi1 = (R)fu[0], fj0 = (R)fl[1], fj1 = (R)fu[1];
    const R dr = (R)tb(P, 0, T_DX, i), rc = (R)tb(P, 0, T_G3, i);
    const R* Wh = wk.Wh + x;
    const R ph = (R)Wh[PR * fs], rh = (R)Wh[RHO * fs], v2h = (R)Wh[V2 * fs], v3h = (R)Wh[V3 * fs];
    const R m22 = ph + rh * v2h * v2h, m33 = ph + rh * v3h * v3h;
    const R* Fi = F + x;
    const R* Fj = F + (size_t)9 * fs + x;
    const R geo = dr / rc / R(2) * rivol;
    sh[0] = R(0.5) * (m22 + m33) * (fi1 - fi0) * rivol;
    sh[1] = -((R)Fi[2 * fs] * fi0 + (R)Fi[si + 2 * fs] * fi1) * geo + (fj1 - fj0) * rivol * m33;
    sh[2] = -((R)Fi[3 * fs] * fi0 + (R)Fi[si + 3 * fs] * fi1) * geo;
    const R sr = (R)tb(P, 1, T_G3, j) / (R)tb(P, 1, T_G4, j) * rivol;
    sh[2] += -((R)Fj[3 * fs] * fj0 + (R)Fj[sjj + 3 * fs] * fj1) * sr;
    const R* Msh = wk.Msh + x;
    const R b1 = (R)Msh[0], b2 = (R)Msh[fs], b3 = (R)Msh[2 * fs];
    R bsq = b1 * b1 + b2 * b2 + b3 * b3;
    R n22 = R(0.5) * bsq - b2 * b2, n33 = R(0.5) * bsq - b3 * b3;
    if constexpr (BG) {  // with the B0 cross terms (spherical_general.c:634-638)
      const double* c0 = P.bg + (size_t)BG_B0 * fs + x;
      const R g1 = (R)c0[0], g2 = (R)c0[fs], g3 = (R)c0[2 * fs];
      bsq = b1 * b1 + b2 * b2 + b3 * b3 + R(2) * (b1 * g1 + b2 * g2 + b3 * g3);
      n22 = R(0.5) * bsq - (b2 + g2) * b2 - b2 * g2;
      n33 = R(0.5) * bsq - (b3 + g3) * b3 - b3 * g3;
    }
    sb[0] = R(0.5) * (n22 + n33) * (fi1 - fi0) * rivol;
    sb[1] = -((R)Fi[7 * fs] * fi0 + (R)Fi[si + 7 * fs] * fi1) * geo + (fj1 - fj0) * rivol * n33;
    sb[2] = -((R)Fi[8 * fs] * fi0 + (R)Fi[si + 8 * fs] * fi1) * geo;
    sb[2] += -((R)Fj[8 * fs] * fj0 + (R)Fj[sjj + 8 * fs] * fj1) * sr;
  }
  // the new face fields of this cell's lower and upper faces, written by
  // k_ct before this launch
  double bl[3], bu[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    bl[a] = Bn[x + a * fs];
    bu[a] = Bn[x + stride(P, a) + a * fs];
  }
  // U^n from W^n (src/solver_func.c:356-382)
  const double gm1 = P.gm1;
  const double r0 = W[x], u0 = W[x + fs], v0 = W[x + 2 * fs], w0 = W[x + 3 * fs],
               p0 = W[x + 4 * fs];
  double U[6];
  U[0] = r0;
  U[1] = r0 * u0;
  U[2] = r0 * v0;
  U[3] = r0 * w0;
  U[4] = 0.5 * r0 * (u0 * u0 + v0 * v0 + w0 * w0) + p0 * P.inv_gm1;
  U[5] = 0.0;
  if constexpr (PSL) {
    const double ps0 = W[x + 5 * fs];
    U[5] = (ps0 == 0.0 && r0 > 0.0) ? ps0 : ps0 / pow(r0, gm1);
  }
  const double U0[3] = {U[1], U[2], U[3]};
  // conservative update and cons->prim (src/solver_solve.c:326-377)
  U[0] -= dt * (double)du[0];
#pragma unroll
  for (int a = 0; a < 3; a++) U[1 + a] = U[1 + a] - dt * (double)du[1 + a] + dt * (double)sh[a];
  U[4] -= dt * (double)du[4];
  double rho = U[0];
  const double irho = 1.0 / U[0];
  double vv[3] = {U[1] * irho, U[2] * irho, U[3] * irho};
  double p = (U[4] - 0.5 * (vv[0] * vv[0] + vv[1] * vv[1] + vv[2] * vv[2]) * rho) * gm1;
  double pS = 0.0;
  if constexpr (PSL) {
    U[5] -= dt * (double)du[5];
    pS = (U[5] == 0.0 && U[0] > 0.0) ? U[5] : U[5] * pow(U[0], gm1);
  }
  // positivity floors (src/solver_func.c:2117-2135)
  if (rho < P.rho_floor) {
    rho = P.rho_floor;
    p = P.p_floor;
  }
  if (p < P.p_floor) p = P.p_floor;
  // mags^{n+1}, time-centred field, Alfven/Boris correction
  // (src/solver_solve.c:385-484)
  double mt[3], mn[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const int idx = a == 0 ? i : (a == 1 ? j : k);
    mn[a] = bl[a] * tb(P, a, T_MA, idx) + bu[a] * tb(P, a, T_MB, idx);
    mt[a] = 0.5 * (mn[a] + mags_at(P, B, a, i, j, k));
    if constexpr (BG) {  // magtot = mags + B0
      const double c0 = P.bg[(size_t)(BG_B0 + a) * fs + x];
      mt[a] += c0;
      mn[a] += c0;  // the next step's magtot, for its CFL dt
    }
  }
  const R mr[3] = {(R)mt[0], (R)mt[1], (R)mt[2]};
  const R bsq = mr[0] * mr[0] + mr[1] * mr[1] + mr[2] * mr[2];
  const R alf = bsq / (R)rho / (R)P.ca2;
  const R perp = R(1) / (R(1) + alf);
  const R rdt = (R)dt;
  const R drho = -rdt * du[0];
  const R dva = alf * drho;
  R tv[3], wv[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    wv[a] = (R)W[x + (1 + a) * fs];
    tv[a] = alf * (-rdt * du[1 + a] + rdt * sh[a] - drho * wv[a]);
  }
  R bdv = mr[0] * tv[0] + mr[1] * tv[1] + mr[2] * tv[2];
  bdv = bdv / (bsq + R(1e-10));
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const R inc = perp * ((-rdt * du[1 + a] + rdt * sh[a]) + (-rdt * dm[a] + rdt * sb[a]) +
                          dva * wv[a] + mr[a] * bdv);
    vv[a] = (U0[a] + (double)inc) * irho;
  }
  Wn[x] = rho;
  Wn[x + fs] = vv[0];
  Wn[x + 2 * fs] = vv[1];
  Wn[x + 3 * fs] = vv[2];
  Wn[x + 4 * fs] = p;
  if constexpr (PSL) Wn[x + 5 * fs] = pS;
  // CFL rate of the new state (magtot = mags^{n+1}) and max|div B^{n+1}|
  rate = cfl_cell<COORD, R>(P, i, j, k, rho, vv[0], vv[1], vv[2], p, mn[0], mn[1], mn[2]);
  double b0l[3] = {0.0, 0.0, 0.0}, b0u[3] = {0.0, 0.0, 0.0};
  if constexpr (BG) {  // div of B + B0 (face-normal B0, src/solver_func.c:324-343)
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const double* f = P.bg + (size_t)(BG_FACE + 4 * a) * fs + x;
      b0l[a] = f[0];
      b0u[a] = f[stride(P, a)];
    }
  }
  const double dvb = ((bu[0] + b0u[0]) * fu[0] - (bl[0] + b0l[0]) * fl[0]) * ivol +
                     ((bu[1] + b0u[1]) * fu[1] - (bl[1] + b0l[1]) * fl[1]) * ivol +
                     ((bu[2] + b0u[2]) * fu[2] - (bl[2] + b0l[2]) * fl[2]) * ivol;
  dbmax = fabs(dvb);
  if (bad_rate(rate) || !isfinite(p) || !isfinite(rho) || !isfinite(vv[0] + vv[1] + vv[2]))
    flag_numeric(P);
  if (COORD == 2 && P.ring && ring_band_row(P, j)) {
    // the ring average still changes this row: k_ring_dt takes its CFL dt
    // and div B afterwards
    rate = 0.0;
    dbmax = 0.0;
  }
}

// CFL dt and |div B| of one cell of the current state (prepare).  The dt
// takes the form and arithmetic R of the step's own estimate (the FP32
// estimate on the mixed path; FP64 in the rows of the pole ring average),
// so a restarted run takes exactly the step the uninterrupted one would.
template <int COORD, bool BG, typename R>
__device__ __forceinline__ void dt_body(const Params& P, Pos t, double& dtc, double& db) {
  const int i = NGH + t.x, j = NGH + t.y, k = NGH + t.z;
  if (i >= NGH + P.n[0] || j >= NGH + P.n[1] || k >= NGH + P.n[2]) return;
  const double* __restrict__ W = P.Wbuf[cur_buf(P)];
  const double* __restrict__ B = P.Bbuf[cur_buf(P)];
  const long long c = lin(P, i, j, k);
  double b1 = mags_at(P, B, 0, i, j, k), b2 = mags_at(P, B, 1, i, j, k),
         b3 = mags_at(P, B, 2, i, j, k);
  if constexpr (BG) {  // magtot = mags + B0 (src/solver_func.c:345-353)
    b1 += P.bg[(size_t)BG_B0 * P.fs + c];
    b2 += P.bg[(size_t)(BG_B0 + 1) * P.fs + c];
    b3 += P.bg[(size_t)(BG_B0 + 2) * P.fs + c];
  }
  if constexpr (COORD == 0) {  // as update_cart
    using RC = typename std::conditional<sizeof(R) == 8 || GOP_MX_CFL64, double, R>::type;
    const double il[3] = {tb(P, 0, T_IDX, i), tb(P, 1, T_IDX, j), tb(P, 2, T_IDX, k)};
    dtc = step_of<RC>(P, cfl_cart<RC>(P, il, W[c], W[c + P.fs], W[c + 2 * P.fs], W[c + 3 * P.fs],
                                      W[c + 4 * P.fs], b1 * b1 + b2 * b2 + b3 * b3));
  } else if (P.ring && ring_band_row(P, j)) {  // as k_ring_dt
    dtc = step_of<double>(P, cfl_cell<COORD>(P, i, j, k, W[c], W[c + P.fs], W[c + 2 * P.fs], W[c + 3 * P.fs],
                                             W[c + 4 * P.fs], b1, b2, b3));
  } else {  // as the curvilinear update
    dtc = step_of<R>(P, cfl_cell<COORD, R>(P, i, j, k, W[c], W[c + P.fs], W[c + 2 * P.fs], W[c + 3 * P.fs],
                                           W[c + 4 * P.fs], b1, b2, b3));
  }
  const double vol = Geo<COORD>::vol(P, i, j, k);
  double d = 0.0;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const double* f = B + (size_t)a * P.fs;
    const long long s = stride(P, a);
    const int i1 = i + (a == 0), j1 = j + (a == 1), k1 = k + (a == 2);
    double bu = f[c + s], bl = f[c];
    if constexpr (BG) {
      const double* g = P.bg + (size_t)(BG_FACE + 4 * a) * P.fs;
      bu += g[c + s];
      bl += g[c];
    }
    d += (bu * Geo<COORD>::face(P, a, i1, j1, k1) - bl * Geo<COORD>::face(P, a, i, j, k)) / vol;
  }
  db = fabs(d);
}

// ---------------------------------------------------------------- ghosts

// The reference fills its ghost layers axis by axis: the periodic halos along
// i, j and k (src/boundary_exchange.c, index sets of src/setup_mpi.c:62-253),
// then the problem's fills face by face (src/boundary_conditions.c: gas_bc_*
// and gem_bc_*), each over the full transverse extent, so that later fills
// copy what earlier ones wrote at edges and corners.  Here every ghost point
// finds the value it ends with: going back through the fills from the last,
// each fill whose target holds the point moves it to that fill's source (with
// its sign), until no fill applies.  That source is written by no fill, so
// all points go at once, in one launch, where the fills took one each (6 for
// a shell open on all sides: 52 -> 38 us of a 192x128x128 step on B200).

// Where the value of a cell field (fa < 0) or of the face field along axis fa
// at point x comes from: x moves to the source.  False: no fill writes the
// point.  neg: the axes whose 'r' fills reflect the point (bit a) and, bit 3,
// pole fills; fixed: the face of a fixed-state fill (-1: none); entropy: for
// p_S, which the fixed-state fills leave alone.
template <bool PERIODIC>
__device__ __forceinline__ bool ghost_source(const Params& P, const GhostFill& G, const char* kind, int fa,
                                             int x[3], int& neg, int& fixed, bool entropy = false) {
  bool any = false;
  neg = 0;
  fixed = -1;
  if constexpr (!PERIODIC) {
#pragma unroll
    for (int face = 5; face >= 0; face--) {
      const int a = face / 2, side = face % 2, n = P.n[a], o = fa == a;
      const int kd = kind[face];
      const int l = side ? x[a] - (n + NGH + o) : x[a];
      if (fixed >= 0 || G.per[a] || l < 0 || l >= NGH || kd == 'n') continue;
      if ((fa >= 0 && kd == 'r') || (entropy && kd == 'f')) continue;  // gem_bc_reflective_* are empty
      any = true;
      if (kd == 'f') {
        fixed = face;
      } else if (kd == 'e') {
        x[a] = side ? n + NGH - 1 + o : NGH;
      } else {
        x[a] = side ? n + NGH - 1 - l : 2 * NGH - 1 - l + o;
        if (kd == 'r') neg ^= 1 << a;
        // pole (j faces): mirrored across the axis half a turn away in phi
        // (src/spherical/spherical_boundary.c:23-138)
        if (kd == 'o') {
          x[2] = NGH + (x[2] - NGH + P.n[2] / 2) % P.n[2];
          neg ^= 8;
        }
      }
    }
  }
#pragma unroll
  for (int a = 2; a >= 0; a--) {
    const int n = P.n[a], o = fa == a;
    if (fixed >= 0 || !(PERIODIC || G.per[a])) continue;
    if (x[a] < NGH) {
      x[a] += n;
      any = true;
    } else if (x[a] >= n + NGH + o && x[a] < n + 2 * NGH + o) {
      x[a] -= n;
      any = true;
    }
  }
  return any;
}

// Thread g runs over three slabs, axis a's 9 layers (4 ghost layers below, 5
// points above: the cell fields' 4 ghost layers and the padding point, or the
// upper boundary face and the face field's 4 ghost layers) times all points
// of the other two axes; a point belongs to the slab of the lowest axis whose
// layers hold it.
template <bool PERIODIC>
__device__ __forceinline__ void ghost_body(const Params& P, const GhostFill& G, int which, unsigned g) {
  // (32 bits: the slabs of a grid of fewer than 2^29 points, see lin32)
  const unsigned N0 = P.N[0], N1 = P.N[1], N2 = P.N[2];
  const unsigned s0 = 9 * N1 * N2, s1 = N0 * 9 * N2, s2 = N0 * N1 * 9;
  int a, x[3];
  if (g < s0) {
    a = 0;
    x[0] = (int)(g % 9);
    const unsigned r = g / 9;
    x[1] = (int)(r % N1);
    x[2] = (int)(r / N1);
  } else if (g < s0 + s1) {
    a = 1;
    const unsigned r = g - s0;
    x[0] = (int)(r % N0);
    x[1] = (int)((r / N0) % 9);
    x[2] = (int)(r / N0 / 9);
  } else if (g < s0 + s1 + s2) {
    a = 2;
    const unsigned r = g - s0 - s1;
    x[0] = (int)(r % N0);
    x[1] = (int)((r / N0) % N1);
    x[2] = (int)(r / N0 / N1);
  } else {
    return;
  }
  if (x[a] >= NGH) x[a] += P.n[a];  // the 5 points above the active range
  for (int b = 0; b < a; b++)
    if (x[b] < NGH || x[b] >= NGH + P.n[b]) return;
  const int bsel = which ? cur_buf(P) : 1 - cur_buf(P);
  double* __restrict__ W = P.Wbuf[bsel];
  double* __restrict__ B = P.Bbuf[bsel];
  const bool ps = P.ps_live != 0;  // p_S zero everywhere stays so: skipped
  const int dst = lin32(P, x[0], x[1], x[2]);
  // all loads before the stores
  double v[9];
  bool on[9];
  {
    int y[3] = {x[0], x[1], x[2]}, neg, fixed;
    const bool any = ghost_source<PERIODIC>(P, G, G.gas, -1, y, neg, fixed);
    const int src = lin32(P, y[0], y[1], y[2]);
#pragma unroll
    for (int f = 0; f < PS; f++) {
      on[f] = any;
      if (!any) continue;
      if (fixed < 0) {
        v[f] = W[(size_t)f * P.fs + src];
      } else {  // gas_bc_fixed_*
        v[f] = f == RHO ? (fixed == 2 ? 2.0 : 1.0) : (f == PR ? (fixed == 3 ? 2.5 : 1.0) : 0.0);
      }
      // a reflective fill turns the velocity along its axis, the pole fill
      // theta and phi components
      const bool flip = f >= V1 && f <= V3 && ((neg >> (f - V1) & 1) != (f != V1 && (neg & 8)));
      if (flip) v[f] = -v[f];
    }
  }
  on[PS] = false;
  if (ps) {
    int y[3] = {x[0], x[1], x[2]}, neg, fixed;
    on[PS] = ghost_source<PERIODIC>(P, G, G.gas, -1, y, neg, fixed, true);
    if (on[PS]) v[PS] = W[(size_t)PS * P.fs + lin32(P, y[0], y[1], y[2])];
  }
#pragma unroll
  for (int c = 0; c < 3; c++) {
    int y[3] = {x[0], x[1], x[2]}, neg, fixed;
    on[6 + c] = ghost_source<PERIODIC>(P, G, G.gem, c, y, neg, fixed);
    if (!on[6 + c]) continue;
    v[6 + c] = fixed < 0 ? B[(size_t)c * P.fs + lin32(P, y[0], y[1], y[2])] : 0.0;
    if (c != 0 && (neg & 8)) v[6 + c] = -v[6 + c];
  }
#pragma unroll
  for (int f = 0; f < 9; f++)
    if (on[f]) (f < 6 ? W + (size_t)f * P.fs : B + (size_t)(f - 6) * P.fs)[dst] = v[f];
}

// ------------------------------------------------- single-instance kernels

// Resident 256-thread blocks per SM each kernel is compiled for (caps its
// registers at 65536 / (256 * n)), per stage and arithmetic type; the
// defaults are the fastest of 1..4 timed on B200 (blast 256^3).
#ifndef GOP_MINB_AB2_F64
#define GOP_MINB_AB2_F64 1
#endif
#ifndef GOP_MINB_AB2_F32
#define GOP_MINB_AB2_F32 1
#endif
#ifndef GOP_MINB_C2C_F64
#define GOP_MINB_C2C_F64 3
#endif
#ifndef GOP_MINB_C2C_F32
#define GOP_MINB_C2C_F32 4
#endif
#ifndef GOP_MINB_EMF_F64
#define GOP_MINB_EMF_F64 2
#endif
#ifndef GOP_MINB_EMF_F32
#define GOP_MINB_EMF_F32 4
#endif
#ifndef GOP_MINB_FLUX_F64
#define GOP_MINB_FLUX_F64 2
#endif
#ifndef GOP_MINB_FLUX_F32
#define GOP_MINB_FLUX_F32 4
#endif
#ifndef GOP_MINB_UPDATE_F64
#define GOP_MINB_UPDATE_F64 2
#endif
#ifndef GOP_MINB_UPDATE_F32
#define GOP_MINB_UPDATE_F32 4
#endif
#ifndef GOP_MINB_UPDATE_SPH_F64
#define GOP_MINB_UPDATE_SPH_F64 2
#endif
#ifndef GOP_MINB_UPDATE_SPH_F32
#define GOP_MINB_UPDATE_SPH_F32 2
#endif
#ifndef GOP_MINB_CT
#define GOP_MINB_CT 4
#endif
#define GOP_MINB(STAGE, R) (sizeof(R) == 8 ? GOP_MINB_##STAGE##_F64 : GOP_MINB_##STAGE##_F32)
#define GOP_UPD_MINB(COORD, R) ((COORD) == 0 ? GOP_MINB(UPDATE, R) : GOP_MINB(UPDATE_SPH, R))

__global__ void k_arm(Params P, double tstop, double budget) {
  pdl_enter();
  arm_body(P, tstop, budget);
  begin_body(P);
}
// between two steps of a call: the buffer just written becomes the current
// state, the next step is opened
__device__ __forceinline__ void turn_body(const Params& P) {
  end_body(P);
  begin_body(P);
}
__global__ void k_turn(Params P) {
  pdl_enter();
  turn_body(P);
}

// At the points the AB2 stage reads (every point but the last plane of each
// axis): S_PSNZ <- 1 if p_S of either state buffer is nonzero; with an uploaded
// history (in buffer 1) S_HISTG <- 1 if its velocities in the ghost layers of
// the axes in P.per are not those of the cells the layers repeat
__global__ void k_state_check(Params P, bool history) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  bool nz = false;
  if (i < P.N[0] - 1 && j < P.N[1] - 1 && k < P.N[2] - 1) {
    const long long x = lin(P, i, j, k) + (long long)PS * P.fs;
    nz = P.Wbuf[0][x] != 0.0 || P.Wbuf[1][x] != 0.0;
  }
  if (__any_sync(0xffffffffu, nz) && (threadIdx.x & 31) == 0) P.scal[S_PSNZ] = 1.0;
  if (!history) return;
  bool other = false;
  if (i < P.N[0] - 1 && j < P.N[1] - 1 && k < P.N[2] - 1) {
    const int x[3] = {i, j, k};
    for (int a = 0; a < 3; a++) {
      if (!P.per[a] || (x[a] >= NGH && x[a] < NGH + P.n[a])) continue;
      const double* h = P.Wbuf[1] + lin(P, i, j, k);
      const long long s = (x[a] < NGH ? P.n[a] : -P.n[a]) * stride(P, a);
      for (int m = V1; m <= V3; m++)
        other = other || !(h[(long long)m * P.fs] == h[(long long)m * P.fs + s]);
    }
  }
  if (__any_sync(0xffffffffu, other) && (threadIdx.x & 31) == 0) P.scal[S_HISTG] = 1.0;
}

template <int COORD, bool BG, typename R>
__global__ void k_dt(Params P) {
  pdl_enter();
  double dtc = DBL_MAX, db = 0.0;
  dt_body<COORD, BG, R>(P, grid_pos(), dtc, db);
  dtc = warp_min(dtc);
  db = warp_max(db);
  if (((threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)) & 31) == 0) {
    if (dtc < DBL_MAX) atomic_min_pos(P.scal + S_NEXT_DT, dtc);
    if (db > 0.0) atomic_max_pos(P.scal + S_DIVB, db);
  }
}

// CFL dt and |div B| of the ring band rows of the new state, after the pole
// ring average (get_derived_variables and get_dt_ring of the next step,
// src/solver_func.c:308-343, src/spherical/spherical_general.c:700-743);
// thread (i, band row, k)
__global__ void k_ring_dt(Params P) {
  pdl_enter();
  double rate = 0.0, db = 0.0;
  const int i = NGH + blockIdx.x * blockDim.x + threadIdx.x;
  const int k = NGH + blockIdx.z * blockDim.z + threadIdx.z;
  const int slot = blockIdx.y * blockDim.y + threadIdx.y;
  const int jm = P.ring_jmax, nrow = jm + 2, pole = slot / nrow, rr = slot % nrow;
  const int j = pole == 0 ? NGH + rr : NGH + P.n[1] - 2 - jm + rr;
  if (!stopped(P) && pole <= 1 && (P.ring & (1 << pole)) && i < NGH + P.n[0] &&
      k < NGH + P.n[2]) {
    const int nb = 1 - cur_buf(P);  // this step's result
    const double* __restrict__ W = P.Wbuf[nb];
    const double* __restrict__ B = P.Bbuf[nb];
    const long long c = lin(P, i, j, k);
    double b[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      b[a] = mags_at(P, B, a, i, j, k);
      if (P.bg) b[a] += P.bg[(size_t)(BG_B0 + a) * P.fs + c];
    }
    rate = cfl_cell<2>(P, i, j, k, W[c], W[c + P.fs], W[c + 2 * P.fs], W[c + 3 * P.fs],
                      W[c + 4 * P.fs], b[0], b[1], b[2]);
    const double vol = Geo<2>::vol(P, i, j, k);
    double d = 0.0;
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const double* f = B + (size_t)a * P.fs;
      const long long s = stride(P, a);
      double bu = f[c + s], bl = f[c];
      if (P.bg) {
        const double* g = P.bg + (size_t)(BG_FACE + 4 * a) * P.fs;
        bu += g[c + s];
        bl += g[c];
      }
      const int i1 = i + (a == 0), j1 = j + (a == 1), k1 = k + (a == 2);
      d += (bu * Geo<2>::face(P, a, i1, j1, k1) - bl * Geo<2>::face(P, a, i, j, k)) / vol;
    }
    db = fabs(d);
  }
  block_commit<double>(P, rate, db);
}

template <typename R, bool PSL>
__global__ void __launch_bounds__(256, GOP_MINB(AB2, R)) k_ab2(Params P, Work<R> w) {
  pdl_enter();
  if (stopped(P)) return;
  ab2_body<R, PSL>(P, w, grid_pos());
}
// The ghost layers of the axes that are not periodic, for the edges of all
// three directions in one launch: threads first[D] .. first[D + 1] - 1 take the
// edges along D.  (Three launches of a few thousand points each took 3 to 5 us
// a step apiece: shell 96x64x48 on B200, stage 13.9 -> 8.6 us.)
struct C2cRange {
  unsigned first[4];
};
template <typename R>
__global__ void __launch_bounds__(256, GOP_MINB(C2C, R)) k_c2c(Params P, Work<R> w, C2cRange G) {
  pdl_enter();
  if (stopped(P)) return;
  const unsigned g = blockIdx.x * blockDim.x + threadIdx.x;
  // r = x + ex (y + ey z) over the points of a direction
  auto at = [](unsigned r, unsigned ex, unsigned ey) {
    const unsigned q = r / ex;
    return Pos{(int)(r - q * ex), (int)(q % ey), (int)(q / ey)};
  };
  if (g < G.first[1]) c2c_body<R, 0>(P, w, at(g, P.n[0], P.n[1] + 1));
  else if (g < G.first[2]) c2c_body<R, 1>(P, w, at(g - G.first[1], 2 * NGH, P.n[1]));
  else if (g < G.first[3]) c2c_body<R, 2>(P, w, at(g - G.first[2], P.n[0] + 1, 2 * NGH));
}
// BG: with the background-field terms (Params::bg set)
template <typename R, int D, bool BG>
__global__ void __launch_bounds__(256, GOP_MINB(EMF, R)) k_emf(Params P, Work<R> w) {
  pdl_enter();
  if (stopped(P)) return;
  emf_body<R, D, BG>(P, w, grid_pos());
}
template <typename R, int D, bool BG, bool PSL>
__global__ void __launch_bounds__(256, GOP_MINB(FLUX, R)) k_flux(Params P, Work<R> w) {
  pdl_enter();
  if (stopped(P)) return;
  flux_body<R, D, BG, PSL>(P, w, grid_pos());
}
template <int COORD, typename R>
__global__ void __launch_bounds__(256, GOP_MINB_CT) k_ct(Params P, Work<R> w) {
  pdl_enter();
  if (stopped(P)) return;
  ct_body<COORD, R>(P, w, grid_pos());
}
// CT: k_ct has transported the face field (spherical grids, but for FP64 without
// the pole ring average)
template <int COORD, typename R, bool BG, bool PSL, bool CT = false>
__global__ void __launch_bounds__(256, GOP_UPD_MINB(COORD, R)) k_update(Params P, Work<R> w) {
  pdl_enter();
  if (stopped(P)) return;
  double rate = 0.0, db = 0.0;
  update_body<COORD, R, BG, PSL, CT>(P, w, grid_pos(), rate, db);
  block_commit<typename std::conditional<COORD == 0 && GOP_MX_CFL64, double, R>::type>(P, rate, db);
}
// Ghost fill of the state just written (which 0) or of the current state.
// After a step's fill the block that finishes last turns to the next step: a
// launch of one thread for the end of the step and one for the begin of the
// next took 2.4 us each.
template <bool PERIODIC>
__global__ void __launch_bounds__(256) k_ghost(Params P, GhostFill G, int which) {
  pdl_enter();
  if (!which && stopped(P)) return;
  ghost_body<PERIODIC>(P, G, which, blockIdx.x * blockDim.x + threadIdx.x);
  if (which) return;
  // every thread of the block has read S_PAR and written its points
  __syncthreads();
  if (threadIdx.x != 0) return;
  unsigned* done = reinterpret_cast<unsigned*>(P.scal + S_TILE) + 1;
  __threadfence();
  if (atomicAdd(done, 1u) == gridDim.x - 1) {
    *done = 0;
    turn_body(P);
  }
}

// ------------------------------------------------------ layout transposes

// reference layout [i][j][k] (k fastest) <-> device layout of one field: the
// (i, k) plane of each j in 32 x 32 tiles through shared memory (padded by one
// column against bank conflicts), so both sides move whole lines.  Threads
// along i that read k-fastest memory directly touch one 32-byte sector per
// value.  Blocks of 32 x 8 threads over (k tiles, i tiles, rows j).
constexpr int kXT = 32, kXR = 8;
template <bool TO_REF>
__global__ void __launch_bounds__(kXT* kXR) k_transpose(Params P, const double* __restrict__ src,
                                                        double* __restrict__ dst) {
  pdl_enter();
  __shared__ double tile[kXT][kXT + 1];
  const int N0 = P.N[0], N1 = P.N[1], N2 = P.N[2];
  const int k0 = blockIdx.x * kXT, i0 = blockIdx.y * kXT, tx = threadIdx.x, ty = threadIdx.y;
  for (int j = blockIdx.z; j < N1; j += gridDim.z) {
    __syncthreads();  // the tile of the row before has been read
#pragma unroll
    for (int r = 0; r < kXT; r += kXR) {
      if (TO_REF) {  // lanes along i
        const int i = i0 + tx, k = k0 + ty + r;
        if (i < N0 && k < N2) tile[ty + r][tx] = src[lin(P, i, j, k)];
      } else {  // lanes along k
        const int i = i0 + ty + r, k = k0 + tx;
        if (i < N0 && k < N2) tile[tx][ty + r] = src[((size_t)i * N1 + j) * N2 + k];
      }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kXT; r += kXR) {
      if (TO_REF) {
        const int i = i0 + ty + r, k = k0 + tx;
        if (i < N0 && k < N2) dst[((size_t)i * N1 + j) * N2 + k] = tile[tx][ty + r];
      } else {
        const int i = i0 + tx, k = k0 + ty + r;
        if (i < N0 && k < N2) dst[lin(P, i, j, k)] = tile[ty + r][tx];
      }
    }
  }
}

template <typename R>
__global__ void k_widen(Params P, int nf, const R* __restrict__ src, double* __restrict__ dst) {
  pdl_enter();
  const size_t n = (size_t)nf * P.fs;
  for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
    dst[t] = (double)src[t];
}

// mags over the ghost range from face fields (for downloads)
__global__ void k_mags(Params P, const double* __restrict__ B, double* __restrict__ out) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  const int k = blockIdx.z * blockDim.z + threadIdx.z;
  if (i >= P.N[0] - 1 || j >= P.N[1] - 1 || k >= P.N[2] - 1) return;
  const long long x = lin(P, i, j, k);
  for (int a = 0; a < 3; a++) out[x + a * P.fs] = mags_at(P, B, a, i, j, k);
}

// ----------------------------------------------------------- launchers

// launches by this process (any host thread)
static std::atomic<int64_t> g_launches{0};
int64_t launches() { return g_launches.load(); }
void count_launches(int64_t n) { g_launches += n; }

static dim3 grid3(int a, int b, int c, dim3 blk) {
  return dim3((a + blk.x - 1) / blk.x, (b + blk.y - 1) / blk.y, (c + blk.z - 1) / blk.z);
}

// 1: step kernels go out with programmatic dependent launch
#ifndef GOP_PDL
#define GOP_PDL 1
#endif
// 1: also the first kernel after the tile-staged flux sweeps.  Off: placed
// early, its blocks (and the blocks launched early after them) start on SMs
// still configured for the sweep's 213 KB of shared memory, with a short
// L1, and the L1-bound edge-EMF stage slows down (blast 256^3 FP64 step
// 9.49 vs 8.09 ms on B200)
#ifndef GOP_PDL_AFTER_SWEEP
#define GOP_PDL_AFTER_SWEEP 0
#endif

#define LAUNCH_PDL(pdl, kern, grd, blk, st, ...)                                 \
  do {                                                                           \
    cudaLaunchAttribute at_[1];                                                  \
    at_[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;              \
    at_[0].val.programmaticStreamSerializationAllowed = 1;                       \
    cudaLaunchConfig_t cfg_ = {};                                                \
    cfg_.gridDim = dim3(grd);                                                    \
    cfg_.blockDim = dim3(blk);                                                   \
    cfg_.stream = st;                                                            \
    cfg_.attrs = at_;                                                            \
    cfg_.numAttrs = (GOP_PDL && (pdl)) ? 1 : 0;                                  \
    cudaLaunchKernelEx(&cfg_, kern, __VA_ARGS__);                                \
    g_launches++;                                                                \
  } while (0)
#define LAUNCH(kern, grd, blk, st, ...) LAUNCH_PDL(true, kern, grd, blk, st, __VA_ARGS__)

Tune::Tune() {
  // defaults: warps along i; the sweeps of D=1 / D=2 kernels run along the
  // block's longer transverse side so neighbouring rows share L1 lines
  for (int t = 0; t < NTUNE; t++) blk[t] = dim3(32, 4, 2);
  blk[K_EMF1] = blk[K_FLUX1] = dim3(32, 8, 1);
  blk[K_EMF2] = blk[K_FLUX2] = dim3(32, 1, 8);
  for (int d = 0; d < 3; d++) {
    flux_order[d] = emf_order[d] = d;
  }
  flux_sweep = emf_sweep = update_sweep = true;
}

dim3 launch_space(const Params& P, int slot) {
  if (slot == K_AB2) return dim3(P.N[0], P.N[1], P.N[2]);
  if (slot == K_UPDATE) return dim3(P.n[0], P.n[1], P.n[2]);
  if (slot < K_EMF0 || slot > K_FLUX2) return dim3(0, 0, 0);
  const bool emf = slot < K_FLUX0;
  const int D = emf ? slot - K_EMF0 : slot - K_FLUX0;
  int cnt[3] = {P.n[0], P.n[1], P.n[2]};
  if (emf) {  // D cells, faces of the other two axes
    cnt[(D + 1) % 3] += 1;
    cnt[(D + 2) % 3] += 1;
  } else {
    cnt[D] += 1;
  }
  return dim3(cnt[0], cnt[1], cnt[2]);
}

void launch_arm(const Params& P, double tstop, double budget, cudaStream_t st) {
  LAUNCH(k_arm, 1, 1, st, P, tstop, budget);
}

void launch_state_check(const Params& P, bool history, cudaStream_t st) {
  const int nx = (P.N[0] - 1 + 31) / 32 * 32;
  const dim3 blk(std::min(nx, 256), 1, 1);
  LAUNCH(k_state_check, dim3((nx + blk.x - 1) / blk.x, P.N[1] - 1, P.N[2] - 1), blk, st, P, history);
}

template <typename R>
static void launch_dt_r(const Params& P, int coord, cudaStream_t st) {
  const dim3 blk(32, 4, 2);
  const dim3 g = grid3(P.n[0], P.n[1], P.n[2], blk);
  const bool bg = P.bg != nullptr;
  if (coord == 0) {
    if (bg) LAUNCH((k_dt<0, true, R>), g, blk, st, P);
    else LAUNCH((k_dt<0, false, R>), g, blk, st, P);
  } else {
    if (bg) LAUNCH((k_dt<2, true, R>), g, blk, st, P);
    else LAUNCH((k_dt<2, false, R>), g, blk, st, P);
  }
}

void launch_dt(const Params& P, int coord, bool mixed, cudaStream_t st) {
  if (mixed) launch_dt_r<float>(P, coord, st);
  else launch_dt_r<double>(P, coord, st);
}

// the face field of this grid is transported by k_ct before the update
template <typename R>
static bool ct_apart(const Params& P) {
  return P.coord != 0 && (P.ring || sizeof(R) == 4);
}

template <typename R, bool BG>
static void launch_slot_bg(const Params& P, int coord, const Work<R>& w, int slot, dim3 blk,
                           cudaStream_t st, bool pdl) {
  const dim3 sp = launch_space(P, slot);
  if (sp.x == 0) return;
  const dim3 g = grid3(sp.x, sp.y, sp.z, blk);
  switch (slot) {
    case K_AB2:
      if (P.ps_live) LAUNCH((k_ab2<R, true>), g, blk, st, P, w);
      else LAUNCH((k_ab2<R, false>), g, blk, st, P, w);
      break;
    case K_EMF0: LAUNCH_PDL(pdl, (k_emf<R, 0, BG>), g, blk, st, P, w); break;
    case K_EMF1: LAUNCH_PDL(pdl, (k_emf<R, 1, BG>), g, blk, st, P, w); break;
    case K_EMF2: LAUNCH_PDL(pdl, (k_emf<R, 2, BG>), g, blk, st, P, w); break;
    case K_FLUX0:
      if (P.ps_live) LAUNCH((k_flux<R, 0, BG, true>), g, blk, st, P, w);
      else LAUNCH((k_flux<R, 0, BG, false>), g, blk, st, P, w);
      break;
    case K_FLUX1:
      if (P.ps_live) LAUNCH((k_flux<R, 1, BG, true>), g, blk, st, P, w);
      else LAUNCH((k_flux<R, 1, BG, false>), g, blk, st, P, w);
      break;
    case K_FLUX2:
      if (P.ps_live) LAUNCH((k_flux<R, 2, BG, true>), g, blk, st, P, w);
      else LAUNCH((k_flux<R, 2, BG, false>), g, blk, st, P, w);
      break;
    case K_UPDATE:
      if (coord == 0) {
        if (P.ps_live) LAUNCH_PDL(pdl, (k_update<0, R, BG, true>), g, blk, st, P, w);
        else LAUNCH_PDL(pdl, (k_update<0, R, BG, false>), g, blk, st, P, w);
      } else {
        if (ct_apart<R>(P) && P.ps_live) LAUNCH_PDL(pdl, (k_update<2, R, BG, true, true>), g, blk, st, P, w);
        else if (ct_apart<R>(P)) LAUNCH_PDL(pdl, (k_update<2, R, BG, false, true>), g, blk, st, P, w);
        else if constexpr (sizeof(R) == 8) {
          if (P.ps_live) LAUNCH_PDL(pdl, (k_update<2, R, BG, true>), g, blk, st, P, w);
          else LAUNCH_PDL(pdl, (k_update<2, R, BG, false>), g, blk, st, P, w);
        }
      }
      break;
    default: break;
  }
}

template <typename R>
void launch_slot(const Params& P, int coord, const Work<R>& w, int slot, dim3 blk,
                 cudaStream_t st, bool pdl) {
  if (P.bg) launch_slot_bg<R, true>(P, coord, w, slot, blk, st, pdl);
  else launch_slot_bg<R, false>(P, coord, w, slot, blk, st, pdl);
}

template void launch_slot<double>(const Params&, int, const Work<double>&, int, dim3, cudaStream_t, bool);
template void launch_slot<float>(const Params&, int, const Work<float>&, int, dim3, cudaStream_t, bool);

template <typename R>
void launch_step_body(const Params& P, int coord, const Work<R>& w, cudaStream_t st,
                      const Tune& tune, const SweepSet* sw, const Hook& hook) {
  hook(G_AB2, 1);
  launch_slot<R>(P, coord, w, K_AB2, tune.blk[K_AB2], st);
  hook(G_AB2, 0);
  // flux first: it also writes the edge velocities of the active range and
  // of the ghost layers of periodic axes.  The axes of a stage are
  // independent (each writes its own fluxes, edge velocities or EMFs), so
  // their order (Tune) changes no result.  The launch after a persistent
  // sweep grid waits for it to finish instead of being placed early on SMs
  // still configured for the sweep's shared memory (and its short L1).
  hook(G_FLUX, 1);
  bool after_sweep = tune.flux_sweep && launch_flux_sweep<R>(sw, P, w, tune.flux_order, st);
  if (!after_sweep)
    for (int n = 0; n < 3; n++) {
      const int slot = K_FLUX0 + tune.flux_order[n];
      launch_slot<R>(P, coord, w, slot, tune.blk[slot], st);
    }
  hook(G_FLUX, 0);
  hook(G_C2C, 1);
  {
    C2cRange G;
    G.first[0] = 0;
    const unsigned n0 = P.n[0], n1 = P.n[1], n2 = P.n[2];
    const unsigned pts[3] = {n0 * (n1 + 1) * 2 * NGH, 2 * NGH * n1 * (n2 + 1), (n0 + 1) * 2 * NGH * n2};
    for (int d = 0; d < 3; d++)  // (where q is periodic the flux stage has written the layers)
      G.first[d + 1] = G.first[d] + (P.per[(d + 2) % 3] ? 0u : pts[d]);
    if (G.first[3]) {
      LAUNCH_PDL(!after_sweep || GOP_PDL_AFTER_SWEEP, k_c2c<R>, dim3((G.first[3] + 255) / 256), dim3(256), st,
                 P, w, G);
      after_sweep = false;
    }
  }
  hook(G_C2C, 0);
  hook(G_EMF, 1);
  if (tune.emf_sweep && launch_emf_sweep<R>(sw, P, w, tune.emf_order, st)) {
    after_sweep = true;
  } else {
    for (int n = 0; n < 3; n++) {
      const int slot = K_EMF0 + tune.emf_order[n];
      launch_slot<R>(P, coord, w, slot, tune.blk[slot], st, !after_sweep || GOP_PDL_AFTER_SWEEP);
      after_sweep = false;
    }
  }
  hook(G_EMF, 0);
  hook(G_UPDATE, 1);
  const bool after_emf_sweep = after_sweep && !GOP_PDL_AFTER_SWEEP;
  launch_pole_emf<R>(P, w, st);  // pole ring average only
  if (ct_apart<R>(P)) {  // the face fields in their own launch
    const dim3 blk = tune.blk[K_UPDATE];
    LAUNCH_PDL(!after_emf_sweep, (k_ct<2, R>), grid3(P.n[0], P.n[1], P.n[2], blk), blk, st, P, w);
  }
  if (!(tune.update_sweep && launch_update_sweep<R>(sw, P, w, st)))
    launch_slot<R>(P, coord, w, K_UPDATE, tune.blk[K_UPDATE], st, ct_apart<R>(P) || !after_emf_sweep);
  // the work arrays are free after the update: 2 fields of doubles of scratch
  if (P.ring) {
    launch_ring_average(P, reinterpret_cast<double*>(w.Wh), st);
    const int jm = P.ring_jmax;
    const dim3 blk(32, 2, 4);
    LAUNCH(k_ring_dt, grid3(P.n[0], 2 * (jm + 2), P.n[2], blk), blk, st, P);
  }
  hook(G_UPDATE, 0);
}

template void launch_step_body<double>(const Params&, int, const Work<double>&, cudaStream_t,
                                       const Tune&, const SweepSet*, const Hook&);
template void launch_step_body<float>(const Params&, int, const Work<float>&, cudaStream_t,
                                      const Tune&, const SweepSet*, const Hook&);

void launch_ghosts(const Params& P, const char bc[6], const char gem_bc[6], int which,
                   cudaStream_t st) {
  GhostFill G;
  bool any = false, all = true;
  for (int f = 0; f < 6; f++) {
    G.gas[f] = bc[f];
    G.gem[f] = gem_bc[f];
    any = any || bc[f] != 'n' || (gem_bc[f] != 'n' && gem_bc[f] != 'r');
  }
  for (int a = 0; a < 3; a++) {
    G.per[a] = bc[2 * a] == 'p' && bc[2 * a + 1] == 'p';
    all = all && G.per[a];
  }
  if (!any) {
    if (!which) LAUNCH(k_turn, 1, 1, st, P);
    return;
  }
  const long long N0 = P.N[0], N1 = P.N[1], N2 = P.N[2];
  const long long pts = 9 * (N1 * N2 + N0 * N2 + N0 * N1);
  const dim3 g((unsigned)((pts + 255) / 256));
  if (all) LAUNCH(k_ghost<true>, g, dim3(256), st, P, G, which);
  else LAUNCH(k_ghost<false>, g, dim3(256), st, P, G, which);
}

static dim3 transpose_grid(const Params& P) {
  return dim3((P.N[2] + kXT - 1) / kXT, (P.N[0] + kXT - 1) / kXT, std::min(P.N[1], 65535));
}
void launch_from_ref(const Params& P, const double* src, double* dst, cudaStream_t st) {
  LAUNCH(k_transpose<false>, transpose_grid(P), dim3(kXT, kXR), st, P, src, dst);
}
void launch_to_ref(const Params& P, const double* src, double* dst, cudaStream_t st) {
  LAUNCH(k_transpose<true>, transpose_grid(P), dim3(kXT, kXR), st, P, src, dst);
}

template <typename R>
void launch_widen(const Params& P, int nf, const R* src, double* dst, cudaStream_t st) {
  LAUNCH(k_widen<R>, 1184, 256, st, P, nf, src, dst);
}
template void launch_widen<double>(const Params&, int, const double*, double*, cudaStream_t);
template void launch_widen<float>(const Params&, int, const float*, double*, cudaStream_t);

void launch_mags(const Params& P, const double* B, double* out, cudaStream_t st) {
  const dim3 blk(32, 4, 2);
  LAUNCH(k_mags, grid3(P.N[0], P.N[1], P.N[2], blk), blk, st, P, B, out);
}

}  // namespace gop
