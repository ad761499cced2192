// The cell update of a Cartesian or spherical grid and the reductions of the
// CFL step and of |div B|, shared by the per-cell kernel (gop_kernels.cu) and the
// tile-staged one (gop_sweep.cu).
#pragma once

#include <cfloat>
#include <type_traits>

#include "gop_stage.cuh"

namespace gop {

// Options of the mixed path's Cartesian update (0: FP32 as documented): run
// the flux divergence, the Alfven/Boris correction or the CFL estimate in
// FP64 instead
#ifndef GOP_MX_DIV64
#define GOP_MX_DIV64 0
#endif
#ifndef GOP_MX_ALF64
#define GOP_MX_ALF64 0
#endif
#ifndef GOP_MX_CFL64
#define GOP_MX_CFL64 0
#endif

// thread coordinates in a launch space
struct Pos {
  int x, y, z;
};

__device__ __forceinline__ void atomic_min_pos(double* slot, double v) {
  // positive doubles order like their bit patterns
  atomicMin(reinterpret_cast<unsigned long long*>(slot), (unsigned long long)__double_as_longlong(v));
}
__device__ __forceinline__ void atomic_max_pos(double* slot, double v) {
  atomicMax(reinterpret_cast<unsigned long long*>(slot), (unsigned long long)__double_as_longlong(v));
}

__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// The block's largest CFL rate and |div B|; one thread commits the time step
// of the rate (cfl / rate, in the arithmetic R of the rates: one division per
// block instead of one per cell, the quotient being monotone) and |div B| with
// one atomic each.  A rate of zero is no limit.
template <typename R>
__device__ __forceinline__ double step_of(const Params& P, double rate) {
  return rate > 0.0 ? fmin((double)((R)P.cfl / (R)rate), DBL_MAX) : DBL_MAX;
}
template <typename R>
__device__ __forceinline__ void block_commit(const Params& P, double a, double b) {
  double* smin = P.scal + S_NEXT_DT;
  double* smax = P.scal + S_DIVB;
  __shared__ double sa[32], sb[32];
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nw = (blockDim.x * blockDim.y * blockDim.z + 31) / 32;
  const int w = tid / 32, lane = tid & 31;
  a = warp_max(a);
  b = warp_max(b);
  if (lane == 0) {
    sa[w] = a;
    sb[w] = b;
  }
  __syncthreads();
  if (w == 0) {
    a = lane < nw ? sa[lane] : 0.0;
    b = lane < nw ? sb[lane] : 0.0;
    a = warp_max(a);
    b = warp_max(b);
    if (lane == 0) {
      if (a > 0.0) atomic_min_pos(smin, step_of<R>(P, a));
      if (b > 0.0) atomic_max_pos(smax, b);
    }
  }
}

// a non-finite or non-positive state was seen (1; the flag of a timed-out wait,
// 2, says that the state is none at all and stays)
__device__ __forceinline__ void flag_numeric(const Params& P) {
  if (P.scal[S_FLAGS] == 0.0) atomic_max_pos(P.scal + S_FLAGS, 1.0);
}
// A rate that gives no positive time step
__device__ __forceinline__ bool bad_rate(double rate) { return !(rate >= 0.0 && rate <= DBL_MAX); }

// Fast signal speed |v| + sqrt(cs^2 + va^2) of a cell (src/solver_func.c:
// 255-298): FP64 in the form of fast_speed, FP32 (the mixed path's estimate)
// term by term
__device__ __forceinline__ double signal_speed(const Params& P, double r, double u, double v, double w,
                                               double p, double bsq) {
  return sqrt(u * u + v * v + w * w) + fast_speed(P, P.gamma * p, r, bsq);
}
__device__ __forceinline__ float signal_speed(const Params& P, float r, float u, float v, float w, float p,
                                              float bsq) {
  const float va = sqrt(bsq / r);
  const float vae = va * (float)P.ca / sqrt(va * va + (float)P.ca2);
  const float vf = sqrt(u * u + v * v + w * w);
  const float vs = sqrt((float)P.gamma * p / r);
  return vf + sqrt(vs * vs + vae * vae);
}

// vc (1/di + 1/dj + 1/dk)
__device__ __forceinline__ double cfl_sph(double vc, double di, double dj, double dk) {
  return vc * ((dj * dk + di * dk + di * dj) / (di * dj * dk));
}
// CFL rate (signal speed over the cell's lengths) of one cell of a
// curvilinear grid, in T arithmetic (FP32 for the mixed path's estimate)
template <int COORD, typename T = double>
__device__ __forceinline__ double cfl_cell(const Params& P, int i, int j, int k, double rho,
                                           double u, double v, double w, double p, double b1,
                                           double b2, double b3) {
  const T x1 = (T)b1, x2 = (T)b2, x3 = (T)b3;
  const T vc = signal_speed(P, (T)rho, (T)u, (T)v, (T)w, (T)p, x1 * x1 + x2 * x2 + x3 * x3);
  T dk = (T)Geo<COORD>::dl(P, 2, i, j, k);
  // the phi length of the pole rings is nk / nchunk times longer (dxk_ring,
  // spherical_RingAverage.c:110-138; get_dt_ring, spherical_general.c:700-743)
  if (COORD == 2 && P.ring) dk = (T)P.ringtab[2 * P.n[2] + j] * dk;
  const T di = (T)Geo<COORD>::dl(P, 0, i, j, k), dj = (T)Geo<COORD>::dl(P, 1, i, j, k);
  if constexpr (sizeof(T) == 8) return cfl_sph(vc, di, dj, dk);
  return (double)(vc / di + vc / dj + vc / dk);
}
// CFL rate (signal speed over the cell's lengths) of a cell of a Cartesian
// grid, il the inverse lengths, in T arithmetic (FP32 for the mixed path's
// estimate)
template <typename T>
__device__ __forceinline__ double cfl_cart(const Params& P, const double il[3], double rho, double u,
                                           double v, double w, double p, double bsq) {
  const T vc = signal_speed(P, (T)rho, (T)u, (T)v, (T)w, (T)p, (T)bsq);
  return (double)(vc * (T)il[0] + vc * (T)il[1] + vc * (T)il[2]);
}

// alf = b^2 / (rho ca^2) and perp = 1 / (1 + alf) by one division
__device__ __forceinline__ void boris(const Params& P, double rho, double bsq, double& alf, double& perp) {
  const double rc = rho * P.ca2m, bs = bsq * P.ca2s, q = fma(bsq, P.ca2s, rc), t = rc * q, inv = 1.0 / t;
  alf = bs * q * inv;
  perp = rc * rc * inv;
}

// What a cell's update reads, from global memory: the fluxes of its faces,
// the EMFs of its edges, its face field and its state
template <typename R>
struct PointReader {
  const Params& P;
  const Work<R>& wk;
  const double *W, *B;  // step-start state
  // byte offsets of the cell and of its upper neighbours along j and k: o
  // in the FP64 state, r in the stage arrays
  unsigned o, oj, ok, r, rj, rk;
  int x[3];
  static constexpr unsigned RS = sizeof(R);
  __device__ __forceinline__ PointReader(const Params& p, const Work<R>& w, int i, int j, int k)
      : P(p), wk(w), W(p.Wbuf[cur_buf(p)]), B(p.Bbuf[cur_buf(p)]), x{i, j, k} {
    const unsigned c = lin32(P, i, j, k);
    o = 8 * c, oj = 8 * (unsigned)P.sj, ok = 8 * (unsigned)P.sk;
    r = RS * c, rj = RS * (unsigned)P.sj, rk = RS * (unsigned)P.sk;
  }
  // flux m at the lower (u = 0) or upper face along axis d
  __device__ __forceinline__ R flux(int d, int m, int u) const {
    const unsigned s = d == 0 ? RS : (d == 1 ? rj : rk);
    return at_byte(static_cast<const R*>(wk.F) + (size_t)(9 * d + m) * P.fs, u ? r + s : r);
  }
  // EMF along a at the edge di, dj, dk cells up
  __device__ __forceinline__ double emf(int a, int di, int dj, int dk) const {
    return (double)at_byte(static_cast<const R*>(wk.E) + a * P.fs, r + di * RS + dj * rj + dk * rk);
  }
  __device__ __forceinline__ double face(int a, int u) const {
    return at_byte(B + a * P.fs, u ? o + (a == 0 ? 8u : (a == 1 ? oj : ok)) : o);
  }
  __device__ __forceinline__ double state(int m) const { return at_byte(W + m * P.fs, o); }
  // table t of axis a at the cell, or at the next one
  __device__ __forceinline__ double tab(int a, int t, int up = 0) const { return tb(P, a, t, x[a] + up); }
};

// One active cell of a Cartesian grid (src/solver_solve.c:263-484 with the
// Cartesian geometry of src/cartesian/cartesian_general.c): every face of
// the cell has the area of its axis, every edge along axis a the length
// dx_a, and the geometric sources vanish, so the whole cell needs dx_i,
// dx_j, dx_k and one division.  Face fields, constrained transport, the
// conservative update and the pressure recovery are FP64; with R = float
// the flux divergence, the Alfven/Boris correction and the CFL estimate are
// FP32.  Returns the cell's CFL rate and |div B| of the new state.
// in: the PointReader of cell (i, j, k), or one like it.
template <typename R, bool BG, bool PSL, class Reader>
__device__ __forceinline__ void update_cart(const Params& P, const Reader& in, int i, int j, int k,
                                            double& rate, double& dbmax) {
  // arithmetic of the stages the mixed path runs in FP32 (FP64 when their
  // option is on, and always on the plain path)
  using RD = typename std::conditional<sizeof(R) == 8 || GOP_MX_DIV64, double, R>::type;
  using RA = typename std::conditional<sizeof(R) == 8 || GOP_MX_ALF64, double, R>::type;
  using RC = typename std::conditional<sizeof(R) == 8 || GOP_MX_CFL64, double, R>::type;
  const size_t fs = P.fs;
  const double dt = P.scal[S_DT];
  const int nb = 1 - cur_buf(P);
  double* Wn = P.Wbuf[nb];
  double* Bn = P.Bbuf[nb];
  const unsigned x = lin32(P, i, j, k), o = 8 * x, oj = 8 * (unsigned)P.sj, ok = 8 * (unsigned)P.sk;
  const double il[3] = {in.tab(0, T_IDX), in.tab(1, T_IDX), in.tab(2, T_IDX)};

  // flux divergence: 5 hydro (6 with the entropy channel) and 3 stress
  // components, the difference of the two faces over the cell's length (every
  // face of a Cartesian cell has the area of its axis).  First, so that its 48
  // loads run ahead of everything else.
  RD du[6], dm[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
#pragma unroll
    for (int m = 0; m < 9; m++) {
      if (m == PS && !PSL) continue;
      const R fu = in.flux(d, m, 1), fl = in.flux(d, m, 0);
      const RD v = ((RD)fu - (RD)fl) * (RD)il[d];
      if (m < 6) du[m] = d == 0 ? v : du[m] + v;
      else dm[m - 6] = d == 0 ? v : dm[m - 6] + v;
    }
  }
  if constexpr (BG) {  // + the Lorentz force of B0 (src/solver_solve.c:312-324)
#pragma unroll
    for (int a = 0; a < 3; a++) dm[a] += (RD)P.bg[(size_t)(BG_LOR + a) * fs + x];
  }

  // constrained transport: face A gets -dt (curl E)_A from the differences of
  // the edge EMFs, in FP64 (src/solver_solve.c:263-306; the edge lengths over
  // the face area are inverse cell lengths)
  const double e0 = in.emf(0, 0, 0, 0), e0j = in.emf(0, 0, 1, 0), e0k = in.emf(0, 0, 0, 1),
               e0jk = in.emf(0, 0, 1, 1);
  const double e1 = in.emf(1, 0, 0, 0), e1i = in.emf(1, 1, 0, 0), e1k = in.emf(1, 0, 0, 1),
               e1ik = in.emf(1, 1, 0, 1);
  const double e2 = in.emf(2, 0, 0, 0), e2i = in.emf(2, 1, 0, 0), e2j = in.emf(2, 0, 1, 0),
               e2ij = in.emf(2, 1, 1, 0);
  const double b0l = in.face(0, 0), b0u = in.face(0, 1);
  const double b1l = in.face(1, 0), b1u = in.face(1, 1);
  const double b2l = in.face(2, 0), b2u = in.face(2, 1);
  double bl[3], bu[3], mo[3];
  bl[0] = b0l - dt * ((e2j - e2) * il[1] - (e1k - e1) * il[2]);
  bl[1] = b1l - dt * ((e0k - e0) * il[2] - (e2i - e2) * il[0]);
  bl[2] = b2l - dt * ((e1i - e1) * il[0] - (e0j - e0) * il[1]);
  bu[0] = b0u - dt * ((e2ij - e2i) * il[1] - (e1ik - e1i) * il[2]);
  bu[1] = b1u - dt * ((e0jk - e0j) * il[2] - (e2ij - e2j) * il[0]);
  bu[2] = b2u - dt * ((e1ik - e1k) * il[0] - (e0jk - e0k) * il[1]);
  // mags^n for the time-centred field
  mo[0] = b0l * in.tab(0, T_MA) + b0u * in.tab(0, T_MB);
  mo[1] = b1l * in.tab(1, T_MA) + b1u * in.tab(1, T_MB);
  mo[2] = b2l * in.tab(2, T_MA) + b2u * in.tab(2, T_MB);
  at_byte(Bn, o) = bl[0];
  at_byte(Bn + fs, o) = bl[1];
  at_byte(Bn + 2 * fs, o) = bl[2];
  if (i == NGH + P.n[0] - 1) at_byte(Bn, o + 8) = bu[0];
  if (j == NGH + P.n[1] - 1) at_byte(Bn + fs, o + oj) = bu[1];
  if (k == NGH + P.n[2] - 1) at_byte(Bn + 2 * fs, o + ok) = bu[2];
  if constexpr (BG) {  // div of B + B0 (face-normal B0, src/solver_func.c:324-343)
    const double* f0 = P.bg + (size_t)BG_FACE * fs;
    const double* f1 = P.bg + (size_t)(BG_FACE + 4) * fs;
    const double* f2 = P.bg + (size_t)(BG_FACE + 8) * fs;
    dbmax = fabs(((bu[0] + at_byte(f0, o + 8)) - (bl[0] + at_byte(f0, o))) * il[0] +
                 ((bu[1] + at_byte(f1, o + oj)) - (bl[1] + at_byte(f1, o))) * il[1] +
                 ((bu[2] + at_byte(f2, o + ok)) - (bl[2] + at_byte(f2, o))) * il[2]);
  } else {
    dbmax = fabs((bu[0] - bl[0]) * il[0] + (bu[1] - bl[1]) * il[1] + (bu[2] - bl[2]) * il[2]);
  }
  // cell-centred B0 (magtot = mags + B0)
  double c0[3] = {0.0, 0.0, 0.0};
  if constexpr (BG) {
#pragma unroll
    for (int a = 0; a < 3; a++) c0[a] = at_byte(P.bg + (size_t)(BG_B0 + a) * fs, o);
  }
  double mn[3], mt[3];
  mn[0] = bl[0] * in.tab(0, T_MA) + bu[0] * in.tab(0, T_MB);
  mn[1] = bl[1] * in.tab(1, T_MA) + bu[1] * in.tab(1, T_MB);
  mn[2] = bl[2] * in.tab(2, T_MA) + bu[2] * in.tab(2, T_MB);
#pragma unroll
  for (int a = 0; a < 3; a++) mt[a] = BG ? 0.5 * (mn[a] + mo[a]) + c0[a] : 0.5 * (mn[a] + mo[a]);

  // U^n from W^n, conservative update, cons->prim in FP64
  // (src/solver_func.c:356-382, src/solver_solve.c:326-377)
  const double gm1 = P.gm1;
  const double r0 = in.state(0), p0 = in.state(4);
  double w0[3];
#pragma unroll
  for (int a = 0; a < 3; a++) w0[a] = in.state(1 + a);
  const double U0[3] = {r0 * w0[0], r0 * w0[1], r0 * w0[2]};
  // (p / (gamma - 1) rounded by itself: the way back multiplies by gamma - 1,
  // and with the product inside the sum the pressure of a 128^3 blast was
  // 4.6e-16 off after 40 steps, relative L2, against 1.4e-16)
  const double E0n = fma(0.5 * r0, w0[0] * w0[0] + w0[1] * w0[1] + w0[2] * w0[2], __dmul_rn(p0, P.inv_gm1));
  const double Ur = r0 - dt * (double)du[0];
  double Um[3];
#pragma unroll
  for (int a = 0; a < 3; a++) Um[a] = U0[a] - dt * (double)du[1 + a];
  const double Ue = E0n - dt * (double)du[4];
  double rho = Ur;
  const double irho = 1.0 / Ur;
  double vv[3] = {Um[0] * irho, Um[1] * irho, Um[2] * irho};
  double p = (Ue - 0.5 * (vv[0] * vv[0] + vv[1] * vv[1] + vv[2] * vv[2]) * rho) * gm1;
  double pS = 0.0;
  if constexpr (PSL) {  // entropy S = p_S / rho^(gamma-1), updated and back
    const double ps0 = in.state(5);
    const double S0 = (ps0 == 0.0 && r0 > 0.0) ? ps0 : ps0 / pow(r0, gm1);
    const double Us = S0 - dt * (double)du[5];
    pS = (Us == 0.0 && Ur > 0.0) ? Us : Us * pow(Ur, gm1);
  }
  // positivity floors (src/solver_func.c:2117-2135)
  if (rho < P.rho_floor) {
    rho = P.rho_floor;
    p = P.p_floor;
  }
  if (p < P.p_floor) p = P.p_floor;

  // Alfven/Boris correction of the momentum (src/solver_solve.c:385-484)
  {
    const RA bsq = (RA)(mt[0] * mt[0] + mt[1] * mt[1] + mt[2] * mt[2]);
    RA alf, perp;
    if constexpr (sizeof(RA) == 8) {
      boris(P, rho, bsq, alf, perp);
    } else {
      alf = bsq / ((RA)rho * (RA)P.ca2);
      perp = RA(1) / (RA(1) + alf);
    }
    const RA rdt = (RA)dt;
    const RA drho = -rdt * (RA)du[0];
    const RA dva = alf * drho;
    RA tv[3], wv[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      wv[a] = (RA)w0[a];
      tv[a] = alf * (-rdt * (RA)du[1 + a] - drho * wv[a]);
    }
    RA bdv = (RA)mt[0] * tv[0] + (RA)mt[1] * tv[1] + (RA)mt[2] * tv[2];
    bdv = bdv / (bsq + RA(1e-10));
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const RA inc = perp * ((-rdt * (RA)du[1 + a]) + (-rdt * (RA)dm[a]) + dva * wv[a] + (RA)mt[a] * bdv);
      vv[a] = (U0[a] + (double)inc) * irho;
    }
  }
  at_byte(Wn, o) = rho;
#pragma unroll
  for (int a = 0; a < 3; a++) at_byte(Wn + (1 + a) * fs, o) = vv[a];
  at_byte(Wn + 4 * fs, o) = p;
  if constexpr (PSL) at_byte(Wn + 5 * fs, o) = pS;  // else it stays zero in both buffers

  // CFL rate of the new state with magtot = mags^{n+1} (src/solver_func.c:255-298)
  {
    const double t0 = mn[0] + c0[0], t1 = mn[1] + c0[1], t2 = mn[2] + c0[2];
    rate = cfl_cart<RC>(P, il, rho, vv[0], vv[1], vv[2], p, t0 * t0 + t1 * t1 + t2 * t2);
  }
  if (bad_rate(rate) || !isfinite(p) || !isfinite(rho) || !isfinite(vv[0] + vv[1] + vv[2]))
    flag_numeric(P);
}

// One active cell of a spherical grid without the pole ring average
// (src/solver_solve.c:263-484, src/spherical/spherical_general.c:42-316,
// 605-698).  The areas, edges and volumes are separable, and what the update
// takes of them are quotients: an edge over a face in the transport, a face
// over the volume in the divergence.  They come from tables (T_U0..T_U5), so
// there is no division for the geometry and the cell transports its six
// faces itself (k_ct, a launch of its own, moved the new face field to memory
// and back to save the divisions): 192x128x128 on B200, transport and update
// 469 -> 327 us.  FP64 only: the mixed path's FP32 roundings follow the last
// bits of areas, volumes and face field, and it keeps the reference's products
// and quotients in k_ct and the kernel after it.
template <bool BG, bool PSL, class Reader>
__device__ __forceinline__ void update_sph(const Params& P, const Work<double>& wk, const Reader& in, int i, int j,
                                           int k, double& rate, double& dbmax) {
  using R = double;
  const size_t fs = P.fs;
  const double dt = P.scal[S_DT];
  const int nb = 1 - cur_buf(P);
  double* Wn = P.Wbuf[nb];
  double* Bn = P.Bbuf[nb];
  const unsigned x = lin32(P, i, j, k), o = 8 * x, oj = 8 * (unsigned)P.sj, ok = 8 * (unsigned)P.sk;
  // half-step values of the geometric sources
  const R *Wh = wk.Wh, *Mh = wk.Msh;
  const R rh = at_byte(Wh + RHO * fs, o), v2h = at_byte(Wh + V2 * fs, o), v3h = at_byte(Wh + V3 * fs, o),
          ph = at_byte(Wh + PR * fs, o);
  const R m1h = at_byte(Mh, o), m2h = at_byte(Mh + fs, o), m3h = at_byte(Mh + 2 * fs, o);
  // face over volume: radial lower and upper, h times the theta factors, h w
  // idp in phi
  const double a0 = in.tab(0, T_U0), a1 = in.tab(0, T_U1), h = in.tab(0, T_U2);
  const double s0 = in.tab(1, T_U0), s1 = in.tab(1, T_U1), w = in.tab(1, T_U2);
  const double idp = in.tab(2, T_IDX);

  // flux divergence and the geometric sources (spherical_general.c:605-681)
  R du[6], dm[3], sh[3], sb[3];
  const R m22 = ph + rh * v2h * v2h, m33 = ph + rh * v3h * v3h;
  R bsqh = m1h * m1h + m2h * m2h + m3h * m3h;
  R n22 = R(0.5) * bsqh - m2h * m2h, n33 = R(0.5) * bsqh - m3h * m3h;
  if constexpr (BG) {  // with the B0 cross terms (spherical_general.c:634-638)
    const double* c0 = P.bg + (size_t)BG_B0 * fs;
    const R g1 = (R)at_byte(c0, o), g2 = (R)at_byte(c0 + fs, o), g3 = (R)at_byte(c0 + 2 * fs, o);
    bsqh = m1h * m1h + m2h * m2h + m3h * m3h + R(2) * (m1h * g1 + m2h * g2 + m3h * g3);
    n22 = R(0.5) * bsqh - (m2h + g2) * m2h - m2h * g2;
    n33 = R(0.5) * bsqh - (m3h + g3) * m3h - m3h * g3;
  }
  const R up[3] = {a1, h * s1, h * w * idp}, lo[3] = {a0, h * s0, h * w * idp};
  const R gr = in.tab(0, T_U3), gt = in.tab(1, T_U3);
#pragma unroll
  for (int d = 0; d < 3; d++) {
#pragma unroll
    for (int m = 0; m < 9; m++) {
      if (m == PS && !PSL) continue;
      const R fu = in.flux(d, m, 1) * up[d], fl = in.flux(d, m, 0) * lo[d], v = fu - fl;
      if (m < 6) du[m] = d == 0 ? v : du[m] + v;
      else dm[m - 6] = d == 0 ? v : dm[m - 6] + v;
      if (d == 0 && (m == 2 || m == 3)) sh[m - 1] = -(fl + fu) * gr;
      if (d == 0 && (m == 7 || m == 8)) sb[m - 6] = -(fl + fu) * gr;
      if (d == 1 && m == 3) sh[2] -= (fl + fu) * gt;
      if (d == 1 && m == 8) sb[2] -= (fl + fu) * gt;
    }
  }
  const R dr = R(0.5) * (a1 - a0), dth = h * (s1 - s0);
  sh[0] = (m22 + m33) * dr;
  sh[1] += dth * m33;
  sb[0] = (n22 + n33) * dr;
  sb[1] += dth * n33;
  if constexpr (BG) {  // + the Lorentz force of B0 (src/solver_solve.c:312-324)
#pragma unroll
    for (int a = 0; a < 3; a++) dm[a] += (R)P.bg[(size_t)(BG_LOR + a) * fs + x];
  }

  // constrained transport of the six faces, FP64: curl E over the face from
  // edge over face lengths
  const double b0l = in.face(0, 0), b0u = in.face(0, 1);
  const double b1l = in.face(1, 0), b1u = in.face(1, 1);
  const double b2l = in.face(2, 0), b2u = in.face(2, 1);
  double bl[3], bu[3];
  {
    const double e0 = in.emf(0, 0, 0, 0), e0j = in.emf(0, 0, 1, 0), e0k = in.emf(0, 0, 0, 1),
                 e0jk = in.emf(0, 0, 1, 1);
    const double e1 = in.emf(1, 0, 0, 0), e1i = in.emf(1, 1, 0, 0), e1k = in.emf(1, 0, 0, 1),
                 e1ik = in.emf(1, 1, 0, 1);
    const double e2 = in.emf(2, 0, 0, 0), e2i = in.emf(2, 1, 0, 0), e2j = in.emf(2, 0, 1, 0),
                 e2ij = in.emf(2, 1, 1, 0);
    const double r0 = in.tab(0, T_X), r1 = in.tab(0, T_X, 1), dr = in.tab(0, T_DX);
    const double ir0 = in.tab(0, T_U4), ir1 = in.tab(0, T_U4, 1), ig = in.tab(0, T_U5);
    const double drt = dr * in.tab(1, T_IDX), wp = w * idp;
    const double q0 = dr * idp * in.tab(1, T_U4), q1 = dr * idp * in.tab(1, T_U4, 1);
    bl[0] = b0l - dt * ir0 * ((e2j * s1 - e2 * s0) - (e1k - e1) * wp);
    bu[0] = b0u - dt * ir1 * ((e2ij * s1 - e2i * s0) - (e1ik - e1i) * wp);
    bl[1] = b1l - dt * ig * ((e0k - e0) * q0 - (e2i * r1 - e2 * r0));
    bu[1] = b1u - dt * ig * ((e0jk - e0j) * q1 - (e2ij * r1 - e2j * r0));
    bl[2] = b2l - dt * ig * ((e1i * r1 - e1 * r0) - (e0j - e0) * drt);
    bu[2] = b2u - dt * ig * ((e1ik * r1 - e1k * r0) - (e0jk - e0k) * drt);
  }
  double mo[3], mn[3], mt[3];
  {
    const double ma0 = in.tab(0, T_MA), mb0 = in.tab(0, T_MB), ma1 = in.tab(1, T_MA),
                 mb1 = in.tab(1, T_MB), ma2 = in.tab(2, T_MA), mb2 = in.tab(2, T_MB);
    mo[0] = b0l * ma0 + b0u * mb0;
    mo[1] = b1l * ma1 + b1u * mb1;
    mo[2] = b2l * ma2 + b2u * mb2;
    mn[0] = bl[0] * ma0 + bu[0] * mb0;
    mn[1] = bl[1] * ma1 + bu[1] * mb1;
    mn[2] = bl[2] * ma2 + bu[2] * mb2;
  }
  at_byte(Bn, o) = bl[0];
  at_byte(Bn + fs, o) = bl[1];
  at_byte(Bn + 2 * fs, o) = bl[2];
  if (i == NGH + P.n[0] - 1) at_byte(Bn, o + 8) = bu[0];
  if (j == NGH + P.n[1] - 1) at_byte(Bn + fs, o + oj) = bu[1];
  if (k == NGH + P.n[2] - 1) at_byte(Bn + 2 * fs, o + ok) = bu[2];
  if constexpr (BG) {  // div of B + B0 (face-normal B0, src/solver_func.c:324-343)
    const double* f0 = P.bg + (size_t)BG_FACE * fs;
    const double* f1 = P.bg + (size_t)(BG_FACE + 4) * fs;
    const double* f2 = P.bg + (size_t)(BG_FACE + 8) * fs;
    const double l0 = bl[0] + at_byte(f0, o), u0 = bu[0] + at_byte(f0, o + 8);
    const double l1 = bl[1] + at_byte(f1, o), u1 = bu[1] + at_byte(f1, o + oj);
    const double l2 = bl[2] + at_byte(f2, o), u2 = bu[2] + at_byte(f2, o + ok);
    dbmax = fabs((u0 * a1 - l0 * a0) + h * (u1 * s1 - l1 * s0) + h * w * idp * (u2 - l2));
  } else {
    dbmax = fabs((bu[0] * a1 - bl[0] * a0) + h * (bu[1] * s1 - bl[1] * s0) + h * w * idp * (bu[2] - bl[2]));
  }
#pragma unroll
  for (int a = 0; a < 3; a++) {
    mt[a] = 0.5 * (mn[a] + mo[a]);
    if constexpr (BG) {  // magtot = mags + B0
      const double c0 = at_byte(P.bg + (size_t)(BG_B0 + a) * fs, o);
      mt[a] += c0;
      mn[a] += c0;  // the next step's magtot, for its CFL rate
    }
  }

  // U^n from W^n, conservative update, cons->prim in FP64
  // (src/solver_func.c:356-382, src/solver_solve.c:326-377)
  const double gm1 = P.gm1;
  const double rn = in.state(0), pn = in.state(4);
  const double wn[3] = {in.state(1), in.state(2), in.state(3)};
  const double U0[3] = {rn * wn[0], rn * wn[1], rn * wn[2]};
  const double Ur = rn - dt * (double)du[0];
  double Um[3];
#pragma unroll
  for (int a = 0; a < 3; a++) Um[a] = U0[a] - dt * (double)du[1 + a] + dt * (double)sh[a];
  const double E0n = fma(0.5 * rn, wn[0] * wn[0] + wn[1] * wn[1] + wn[2] * wn[2],
                         __dmul_rn(pn, P.inv_gm1));  // as update_cart
  const double Ue = E0n - dt * (double)du[4];
  double rho = Ur;
  const double irho = 1.0 / Ur;
  double vv[3] = {Um[0] * irho, Um[1] * irho, Um[2] * irho};
  double p = (Ue - 0.5 * (vv[0] * vv[0] + vv[1] * vv[1] + vv[2] * vv[2]) * rho) * gm1;
  double pS = 0.0;
  if constexpr (PSL) {  // entropy S = p_S / rho^(gamma-1), updated and back
    const double ps0 = in.state(5);
    const double S0 = (ps0 == 0.0 && rn > 0.0) ? ps0 : ps0 / pow(rn, gm1);
    const double Us = S0 - dt * (double)du[5];
    pS = (Us == 0.0 && Ur > 0.0) ? Us : Us * pow(Ur, gm1);
  }
  // positivity floors (src/solver_func.c:2117-2135)
  if (rho < P.rho_floor) {
    rho = P.rho_floor;
    p = P.p_floor;
  }
  if (p < P.p_floor) p = P.p_floor;
  // Alfven/Boris correction (src/solver_solve.c:385-484)
  const R mr[3] = {(R)mt[0], (R)mt[1], (R)mt[2]};
  const R bsq = mr[0] * mr[0] + mr[1] * mr[1] + mr[2] * mr[2];
  R alf, perp;
  boris(P, rho, bsq, alf, perp);
  const R rdt = (R)dt;
  const R drho = -rdt * du[0];
  const R dva = alf * drho;
  R tv[3], wv[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    wv[a] = (R)wn[a];
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
  at_byte(Wn, o) = rho;
#pragma unroll
  for (int a = 0; a < 3; a++) at_byte(Wn + (1 + a) * fs, o) = vv[a];
  at_byte(Wn + 4 * fs, o) = p;
  if constexpr (PSL) at_byte(Wn + 5 * fs, o) = pS;
  // CFL rate of the new state (magtot = mags^{n+1})
  // (lengths dr, r_c dtheta, r_c sin(theta_c) dphi, as cfl_cell)
  const double vc = signal_speed(P, rho, vv[0], vv[1], vv[2], p, mn[0] * mn[0] + mn[1] * mn[1] + mn[2] * mn[2]);
  const double rctr = in.tab(0, T_G3);
  rate = cfl_sph(vc, in.tab(0, T_DX), rctr * in.tab(1, T_DX), rctr * in.tab(1, T_G2) * in.tab(2, T_DX));
  if (bad_rate(rate) || !isfinite(p) || !isfinite(rho) || !isfinite(vv[0] + vv[1] + vv[2]))
    flag_numeric(P);
}

}  // namespace gop
