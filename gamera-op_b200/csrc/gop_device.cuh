// Device-side data layout, geometry and per-face numerics of the GAMERA-OP
// MHD step on B200 (sm_100a).
//
// Layout in HBM: structure of arrays, one 3-D array per field, i fastest,
// each axis ghost-extended exactly like the reference (n + 2*4 + 1 points,
// active cells at 4..n+3, the extra point holds the upper boundary face).
// Rows are padded to a multiple of 8 doubles so every row starts on a
// 64-byte boundary and warps along i issue coalesced loads.
//
// Geometry is separable in both supported coordinate systems, so the device
// never stores 3-D geometry: face areas, volumes and edge lengths are
// products of per-axis 1-D tables evaluated in the reference's
// multiplication order (src/cartesian/cartesian_general.c:42-283,
// src/spherical/spherical_general.c:42-316).  PDM weights and the PDM
// limiter's geometric coefficients are per-face 1-D tables.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gop {

constexpr int NGH = 4;
// the reference's PDMB (src/config.c:89); the PDM limiter below blends its
// two slopes with a1 = PDMB/(PDMB+1) = 1/2 and a2 = 1 - a1 = 1/2
constexpr double PDMB = 1.0;

// per-axis 1-D tables (index = position along the axis)
enum Tab : int {
  T_X = 0,     // face coordinate x[f]
  T_DX,        // x[f+1] - x[f]
  T_IDX,       // 1 / T_DX
  T_MA,        // (x[c+1] - xctr[c]) / dx[c]: weight of the lower face in mags
  T_MB,        // (xctr[c] - x[c]) / dx[c]: weight of the upper face
  T_WL0,       // 7 left PDM weights at face f (applied to cells f-4..f+2)
  T_WR0 = T_WL0 + 7,  // 7 right weights (applied to cells f+3..f-3)
  T_CL1 = T_WR0 + 7,  // PDM limiter coefficients of the left state
  T_CL2,
  T_CR1,       // ... of the right state
  T_CR2,
  T_G0,        // coordinate-specific factors (see Geo below)
  T_G1,
  T_G2,
  T_G3,
  T_G4,
  // spherical: quotients of the factors above that the update takes (see
  // update_sph); axis 0 | axis 1, with V = G1 of axis 0, C = cos(t0) - cos(t1)
  T_U0,        // r^2 / V             | sin(t) / C
  T_U1,        // r1^2 / V            | sin(t1) / C
  T_U2,        // G2 / V              | (t1 - t0) / C
  T_U3,        // dr / (2 r_c)        | G3 / G4
  T_U4,        // 1 / r               | 1 / sin(t)
  T_U5,        // 1 / G2              |
  NTAB
};

// The PDM weights and limiter coefficients of one face packed together
// after the per-axis tables: fw[(axis * tmax + f) * FW + t], t = 0..6 left
// weights, 7..13 right weights, 14..17 cl1 cl2 cr1 cr2, 18..19 zero, so one
// face's 18 values come in five 16-byte loads (FP32) from one address.
// tmax is a multiple of 4, which keeps every face record 16-byte aligned.
constexpr int FW = 20;
__host__ __device__ constexpr size_t fw_offset(int tmax) { return (size_t)3 * NTAB * tmax; }
__host__ __device__ constexpr size_t tab_elems(int tmax) { return (size_t)3 * (NTAB + FW) * tmax; }

// device scalars (one double slot each)
enum Scal : int {
  S_DT = 0,      // dt of the current step
  S_DT0,         // dt of the previous step (AB2)
  S_TIME,        // time_sim
  S_CAB2,        // 0.5*dt/dt0 of the current step
  S_NEXT_DT,     // bit pattern of the running CFL minimum (uint64 atomicMin)
  S_DIVB,        // bit pattern of max|div B| (uint64 atomicMax)
  S_STEPS,       // steps taken (as double)
  S_STOP,        // nonzero: time_stop reached, kernels return at once
  S_TSTOP,       // time_stop of the current gop_step call
  S_FLAGS,       // 1: non-finite / non-positive state seen; 2: a pipeline wait
                 // timed out (stays, whatever is seen after it)
  S_PAR,         // which of the two state buffers holds the current state
  S_BUDGET,      // steps left in the current gop_step call
  S_PSNZ,        // gop_prepare's check: nonzero if some p_S of the state or
                 // of its AB2 history is nonzero
  S_HISTG,       // gop_prepare's check of an uploaded AB2 history: nonzero if a
                 // velocity in a periodic ghost layer is not that of the cell
                 // the layer repeats
  S_TILE,        // two 32-bit counters of the running launch: tiles handed
                 // out (sweeps), blocks done; zero between launches
  NSCAL
};

struct Params {
  int n[3];           // active cells
  int N[3];           // ghost-extended points
  int pitch;          // row pitch (elements)
  int coord;          // 0: Cartesian, 2: spherical (batched kernels select on it)
  int per[3];         // 1: the axis is periodic and its ghost layers repeat the active cells, in
                      // the AB2 history too (gop_prepare looks)
  long long sj, sk;   // strides of j and k (stride of i is 1)
  long long fs;       // stride between fields
  const double* tab;  // [3][NTAB][tmax]
  int tmax;
  double gamma, gm1, cfl, ca, ca2, rho_floor, p_floor;
  double ca2m, ca2s;      // ca^2 = ca2m / ca2s (split_ca2)
  double inv_gm1;         // 1/(gamma-1)
  double q_ca;            // 1/(4 CA): Boris diffusion coefficient of the stress
  double* scal;           // device scalars
  double* Wbuf[2];        // two 6-field primitive buffers (current / next)
  double* Bbuf[2];        // two 3-field face-B buffers
  const double* bg;       // background field block (BG_NF fields) or null
  // 1 if p_S (the entropy channel) is nonzero somewhere in the state or its
  // AB2 history; 0 keeps it zero for good (zero states give a zero entropy
  // flux and every fill copies), and the flux kernels skip it
  int ps_live;
  // pole ring average (spherical): bit 0 a pole at theta = 0 (j face NGH),
  // bit 1 at theta = pi (j face NGH + nj); 0 off
  int ring;
  int ring_jmax;          // ring rows per pole - 1
  int nchunk[16];         // phi blocks of ring row r
  const double* ringtab;  // cos, sin of (k + 1/2) 2 pi / nk; then per j the
                          // factor of the CFL length in phi (N[1] values)
};

// Background field B0 (src/solver_func.c:1851-2077), BG_NF fields of the
// state's layout: B0 at the cell centre (B0_b1..3), the Lorentz force of B0
// (dmagsf_G), B0 averaged over the faces normal to axis d (B0Aface*_b1..3,
// field BG_FACE + 3d + c) and along the edges of axis d (B0Aedge*_b1..3,
// field BG_EDGE + 3d + c).
enum BgField : int { BG_B0 = 0, BG_LOR = 3, BG_FACE = 6, BG_EDGE = 15, BG_NF = 24 };

__device__ __forceinline__ int cur_buf(const Params& P) { return P.scal[S_PAR] != 0.0 ? 1 : 0; }

__device__ __forceinline__ double tb(const Params& P, int axis, int t, int idx) {
  return __ldg(P.tab + ((size_t)axis * NTAB + t) * P.tmax + idx);
}

__device__ __forceinline__ long long lin(const Params& P, int i, int j, int k) {
  return (long long)k * P.sk + (long long)j * P.sj + i;
}

// the same in 32 bits: a field has fewer than 2^29 points (gop_create refuses
// more: at 432 bytes per point and up an instance would hold 232 GB)
constexpr long long kMaxField = 1LL << 29;
__device__ __forceinline__ int lin32(const Params& P, int i, int j, int k) {
  return (k * P.N[1] + j) * P.pitch + i;
}

// base[off / sizeof(T)] of a field for a byte offset (below 2^32, see lin32):
// one address register for all the fields a thread reads at a point, where an
// index of 64 bits takes two additions per field
template <typename T>
__device__ __forceinline__ T at_byte(const T* base, unsigned off) {
  return __ldg(reinterpret_cast<const T*>(reinterpret_cast<const char*>(base) + off));
}
template <typename T>
__device__ __forceinline__ T& at_byte(T* base, unsigned off) {
  return *reinterpret_cast<T*>(reinterpret_cast<char*>(base) + off);
}

__device__ __forceinline__ long long stride(const Params& P, int axis) {
  return axis == 0 ? 1LL : (axis == 1 ? P.sj : P.sk);
}

// Geometry policy.  Cartesian: the reference's uniform-grid arrays
// (dx_a, face_i = dx2*dx3, vol = dx1*dx2*dx3).  Spherical (r, theta, phi):
// G0..G4 of axis 0 = -r^2, (r1^3-r0^3)/3, (r1^2-r0^2)/2, r_c;
// of axis 1 = cos(t1)-cos(t0), sin(t), sin(t_c), sin(t1)-sin(t0),
// sin(t1)+sin(t0).
template <int COORD>
struct Geo {
  __device__ static __forceinline__ double face(const Params& P, int a, int i, int j, int k) {
    if (COORD == 0) {
      if (a == 0) return tb(P, 1, T_DX, j) * tb(P, 2, T_DX, k);
      if (a == 1) return tb(P, 0, T_DX, i) * tb(P, 2, T_DX, k);
      return tb(P, 0, T_DX, i) * tb(P, 1, T_DX, j);
    } else {
      if (a == 0) return tb(P, 0, T_G0, i) * tb(P, 1, T_G0, j) * tb(P, 2, T_DX, k);
      if (a == 1) return tb(P, 0, T_G2, i) * tb(P, 1, T_G1, j) * tb(P, 2, T_DX, k);
      return tb(P, 0, T_G2, i) * tb(P, 1, T_DX, j);
    }
  }
  __device__ static __forceinline__ double vol(const Params& P, int i, int j, int k) {
    if (COORD == 0) return tb(P, 0, T_DX, i) * tb(P, 1, T_DX, j) * tb(P, 2, T_DX, k);
    return fabs(tb(P, 0, T_G1, i) * tb(P, 1, T_G0, j) * tb(P, 2, T_DX, k));
  }
  // edge length of the edge along axis a at (i,j,k)
  __device__ static __forceinline__ double edge(const Params& P, int a, int i, int j, int k) {
    if (COORD == 0 || a == 0) return tb(P, a, T_DX, a == 0 ? i : (a == 1 ? j : k));
    if (a == 1) return tb(P, 0, T_X, i) * tb(P, 1, T_DX, j);
    return tb(P, 0, T_X, i) * tb(P, 1, T_G1, j) * tb(P, 2, T_DX, k);
  }
  // CFL length of cell (i,j,k) along axis a (geo[dxi..dxk])
  __device__ static __forceinline__ double dl(const Params& P, int a, int i, int j, int k) {
    if (COORD == 0 || a == 0) return tb(P, a, T_DX, a == 0 ? i : (a == 1 ? j : k));
    if (a == 1) return tb(P, 0, T_G3, i) * tb(P, 1, T_DX, j);
    return tb(P, 0, T_G3, i) * tb(P, 1, T_G2, j) * tb(P, 2, T_DX, k);
  }
};

// Left and right states at face f of a line v[0..7] = cells f-4..f+3, with
// the limiter on lim[0..3] = cells f-2..f+1.
template <typename R>
struct FaceWeights {
  R wl[7], wr[7];
  R cl1, cl2, cr1, cr2;  // the limiter coefficients times a1
  // from the tables' coefficients (a1 = 1/2: exact)
  __device__ __forceinline__ void set_limiter(R l1, R l2, R r1, R r2) {
    cl1 = R(0.5) * l1;
    cl2 = R(0.5) * l2;
    cr1 = R(0.5) * r1;
    cr2 = R(0.5) * r2;
  }
};

// tab: the per-axis tables in the stage type R (layout of Params::tab)
template <typename R>
__device__ __forceinline__ void load_weights(const R* __restrict__ tab, int tmax, int axis, int f,
                                             FaceWeights<R>& W) {
  const R* t0 = tab + (size_t)axis * NTAB * tmax + f;
#pragma unroll
  for (int t = 0; t < 7; t++) {
    W.wl[t] = __ldg(t0 + (size_t)(T_WL0 + t) * tmax);
    W.wr[t] = __ldg(t0 + (size_t)(T_WR0 + t) * tmax);
  }
  W.set_limiter(__ldg(t0 + (size_t)T_CL1 * tmax), __ldg(t0 + (size_t)T_CL2 * tmax),
                __ldg(t0 + (size_t)T_CR1 * tmax), __ldg(t0 + (size_t)T_CR2 * tmax));
}

// the same from the packed face records (fw = the packed region): one
// address and five (FP32) or nine (FP64) vector loads per face
__device__ __forceinline__ void load_fw(const float* __restrict__ fw, int tmax, int axis, int f,
                                        FaceWeights<float>& W) {
  const float4* p = reinterpret_cast<const float4*>(fw + ((size_t)axis * tmax + f) * FW);
  const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2), d = __ldg(p + 3), e = __ldg(p + 4);
  W.wl[0] = a.x; W.wl[1] = a.y; W.wl[2] = a.z; W.wl[3] = a.w;
  W.wl[4] = b.x; W.wl[5] = b.y; W.wl[6] = b.z; W.wr[0] = b.w;
  W.wr[1] = c.x; W.wr[2] = c.y; W.wr[3] = c.z; W.wr[4] = c.w;
  W.wr[5] = d.x; W.wr[6] = d.y;
  W.set_limiter(d.z, d.w, e.x, e.y);
}
__device__ __forceinline__ void load_fw(const double* __restrict__ fw, int tmax, int axis, int f,
                                        FaceWeights<double>& W) {
  const double2* p = reinterpret_cast<const double2*>(fw + ((size_t)axis * tmax + f) * FW);
  double v[18];
#pragma unroll
  for (int t = 0; t < 9; t++) {
    const double2 q = __ldg(p + t);
    v[2 * t] = q.x;
    v[2 * t + 1] = q.y;
  }
#pragma unroll
  for (int t = 0; t < 7; t++) {
    W.wl[t] = v[t];
    W.wr[t] = v[7 + t];
  }
  W.set_limiter(v[14], v[15], v[16], v[17]);
}

// the same from a record in shared memory (16-byte aligned; the whole warp
// reads one record)
__device__ __forceinline__ void load_fw_smem(const float* rec, FaceWeights<float>& W) {
  const float4* p = reinterpret_cast<const float4*>(rec);
  const float4 a = p[0], b = p[1], c = p[2], d = p[3], e = p[4];
  W.wl[0] = a.x; W.wl[1] = a.y; W.wl[2] = a.z; W.wl[3] = a.w;
  W.wl[4] = b.x; W.wl[5] = b.y; W.wl[6] = b.z; W.wr[0] = b.w;
  W.wr[1] = c.x; W.wr[2] = c.y; W.wr[3] = c.z; W.wr[4] = c.w;
  W.wr[5] = d.x; W.wr[6] = d.y;
  W.set_limiter(d.z, d.w, e.x, e.y);
}
__device__ __forceinline__ void load_fw_smem(const double* rec, FaceWeights<double>& W) {
  const double2* p = reinterpret_cast<const double2*>(rec);
  double v[18];
#pragma unroll
  for (int t = 0; t < 9; t++) {
    const double2 q = p[t];
    v[2 * t] = q.x;
    v[2 * t + 1] = q.y;
  }
#pragma unroll
  for (int t = 0; t < 7; t++) {
    W.wl[t] = v[t];
    W.wr[t] = v[7 + t];
  }
  W.set_limiter(v[14], v[15], v[16], v[17]);
}

// Both states of a face: two evaluations of PDMU7 (src/solver_func.c:215-253),
// from the half-step line v[0..7] = cells f-4..f+3 and the step-start values
// lim[0..3] = cells f-2..f+1.  The left state is a 7-tap interpolation of
// v[0..6], clamped to the two step-start values l1, l2 next to the face, then
// limited: with d1 = l2 - l1, dm = l1 - l0, s1 = sgn d1 and
//   q = |sgn dm + s1| (a1/2 |c1 l1 + c2 l0| + a2 |dm|)
// it is f - s1 max(0, |f - l1| - q); the right state is the mirror image.
//
// What it costs is instructions: 8 of these pairs are two thirds of a face's
// work, and the sweeps that call it issue on 60-70 % of the cycles.  So the
// signs are read from sign bits and every sign that cannot matter is left
// out.  For d1 = 0 the clamp has already set f = l1 and the limiter has
// nothing to take off, so s1 may be +1 there; |sgn dm + s1| is then 0 where
// dm has the other sign, 1 where dm is zero and 2 otherwise, and 2 (a1/2 |g| +
// a2 |dm|) is |a1 g| + |dm| exactly (a1 = a2 = 1/2; the powers of two only
// move exponents): the weights carry the a1.
static_assert(PDMB == 1.0, "the limiter's factors below are those of PDMB = 1");

// x is +0 or -0
__device__ __forceinline__ bool is_zero(double x) {
  return ((__double2hiint(x) & 0x7fffffff) | __double2loint(x)) == 0;
}

// FP64: there is no 64-bit min/max or select instruction, and fmin, fmax and
// sgn each become about six instructions, so the state is taken as the
// interpolated value held between l1 and a bound, two comparisons: what the
// limiter leaves of a value beyond q is l1 + s1 q (one rounding where f -
// s1 (|f - l1| - q) has two), or l2 where that is nearer.  fmin and
// fmax put the larger neighbour for a tap that is no number: so do the comparisons
// below, ordered for the left state and not for the right one.
// On B200, blast 256^3 FP64: flux stage 3.09 -> 2.56, EMF stage 1.88 -> 1.72 ms
// per step.
// POLE (faces along axis 1, one of which may lie on a pole): the theta face on
// a pole has no area, the limiter's coefficients there are infinite and q is, or
// is no number: nothing is taken off then, whatever the signs (sgn dm + s1 = 0
// times infinity is no number either), and the state is the value held between
// l1 and l2.
template <bool RIGHT, bool POLE>
__device__ __forceinline__ double pdm_side(double fi, double near, double opp, double d, double d1,
                                           bool neg, double ag) {
  const int sg = __double2hiint(d1) & 0x80000000;
  const bool z = is_zero(d);
  const double q2 = fabs(ag) + fabs(d);
  // s1, halved where d is zero (there |sgn d + s1| is 1)
  const double s = __hiloint2double((z ? 0x3fe00000 : 0x3ff00000) | sg, 0);
  const double u = fma(RIGHT ? -s : s, q2, near);
  // the face's other neighbour where it is nearer than u (RIGHT: the
  // directions are those of -s1, and what is no number counts as larger)
  const bool free = POLE && (unsigned)__double2hiint(q2) >= 0x7ff00000u;
  const bool in = (RIGHT ? !(u <= opp) != neg : (u < opp) != neg) && !free;
  const double bound = in ? u : opp;
  const bool off = ((__double2hiint(d) ^ __double2hiint(d1)) < 0 && !z && !free) ||
                   (RIGHT ? !(fi <= near) != neg : (fi < near) != neg);
  const bool beyond = RIGHT ? !(fi < bound) == neg : (fi <= bound) == neg;
  return off ? near : (beyond ? bound : fi);
}
template <bool POLE>
__device__ __forceinline__ void recon_lr(const double v[8], const double lim[4],
                                         const FaceWeights<double>& W, double& L, double& Rr) {
  const double dm = lim[1] - lim[0], d1 = lim[2] - lim[1], dp = lim[3] - lim[2];
  const bool neg = __double2hiint(d1) < 0;
  double fl = v[0] * W.wl[0], fr = v[7] * W.wr[0];
#pragma unroll
  for (int t = 1; t < 7; t++) {
    fl = fma(v[t], W.wl[t], fl);
    fr = fma(v[7 - t], W.wr[t], fr);
  }
  L = pdm_side<false, POLE>(fl, lim[1], lim[2], dm, d1, neg, W.cl1 * lim[1] + W.cl2 * lim[0]);
  Rr = pdm_side<true, POLE>(fr, lim[2], lim[1], dp, d1, neg, W.cr1 * lim[2] + W.cr2 * lim[3]);
}

// FP32: min and max are one instruction each, and every rounding is the
// reference's (flux stage 1.80 -> 1.70, EMF stage 1.09 -> 1.03 ms per blast
// 256^3 step).
__device__ __forceinline__ float pdm_limit(float fi, float near, float hi, float lo, float d,
                                           float d1, float s, float ag) {
  const float f = fmaxf(lo, fminf(fi, hi));
  const float q2 = fabsf(ag) + fabsf(d);
  const bool other = (__float_as_int(d) ^ __float_as_int(d1)) < 0;
  const float w = d == 0.0f ? 0.5f : (other ? 0.0f : 1.0f);
  return fmaf(-s, fmaxf(0.0f, fabsf(f - near) - w * q2), f);
}
template <bool POLE>
__device__ __forceinline__ void recon_lr(const float v[8], const float lim[4],
                                         const FaceWeights<float>& W, float& L, float& Rr) {
  const float dm = lim[1] - lim[0], d1 = lim[2] - lim[1], dp = lim[3] - lim[2];
  const float s1 = copysignf(1.0f, d1);
  const float hi = fmaxf(lim[1], lim[2]), lo = fminf(lim[1], lim[2]);
  float fl = v[0] * W.wl[0], fr = v[7] * W.wr[0];
#pragma unroll
  for (int t = 1; t < 7; t++) {
    fl = fmaf(v[t], W.wl[t], fl);
    fr = fmaf(v[7 - t], W.wr[t], fr);
  }
  L = pdm_limit(fl, lim[1], hi, lo, dm, d1, s1, W.cl1 * lim[1] + W.cl2 * lim[0]);
  Rr = pdm_limit(fr, lim[2], hi, lo, dp, d1, -s1, W.cr1 * lim[2] + W.cr2 * lim[3]);
}

// Weights of face f on axis AX for a warp whose lanes run along i: along
// i every lane has its own face, and the tap-major tables give coalesced
// loads; along j or k the whole warp shares one face record.
template <int AX, typename R>
__device__ __forceinline__ void load_face_weights(const R* __restrict__ tab, const R* __restrict__ fw,
                                                  int tmax, int f, FaceWeights<R>& W) {
  if constexpr (AX == 0) load_weights<R>(tab, tmax, 0, f, W);
  else load_fw(fw, tmax, AX, f, W);
}

}  // namespace gop
