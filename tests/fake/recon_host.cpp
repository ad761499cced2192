// The reconstruction of gop_device.cuh as host code: the device intrinsics it
// uses stand here, and an array of lines goes through it.
#include <cmath>
#include <cstring>

#include <cuda_runtime.h>

static inline int __double2hiint(double x) { long long b; memcpy(&b, &x, 8); return (int)(b >> 32); }
static inline int __double2loint(double x) { long long b; memcpy(&b, &x, 8); return (int)b; }
static inline double __hiloint2double(int hi, int lo) {
  const long long b = ((long long)hi << 32) | (unsigned)lo;
  double x;
  memcpy(&x, &b, 8);
  return x;
}
static inline int __float_as_int(float x) { int b; memcpy(&b, &x, 4); return b; }
template <typename T>
static inline T __ldg(const T* p) { return *p; }
using std::fabs;
using std::fma;

#include "gop_device.cuh"

template <typename R>
static void lines(int n, const double* v, const double* lim, const double* w, double* out) {
  for (int m = 0; m < n; m++, v += 8, lim += 4, w += 18, out += 2) {
    R a[8], b[4], L, Rr;
    gop::FaceWeights<R> W;
    for (int t = 0; t < 8; t++) a[t] = (R)v[t];
    for (int t = 0; t < 4; t++) b[t] = (R)lim[t];
    for (int t = 0; t < 7; t++) W.wl[t] = (R)w[t], W.wr[t] = (R)w[7 + t];
    W.set_limiter((R)w[14], (R)w[15], (R)w[16], (R)w[17]);
    gop::recon_lr<RECON_AXIS == 1>(a, b, W, L, Rr);
    out[0] = L, out[1] = Rr;
  }
}
extern "C" void recon64(int n, const double* v, const double* lim, const double* w, double* out) {
  lines<double>(n, v, lim, w, out);
}
extern "C" void recon32(int n, const double* v, const double* lim, const double* w, double* out) {
  lines<float>(n, v, lim, w, out);
}
