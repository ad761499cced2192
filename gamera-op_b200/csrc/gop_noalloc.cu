// CFL time step and max|div B| of a caller-owned device state, computed
// without allocating any memory.
//
// Who needs this: a host that already keeps its grid in device memory and
// has to ask "what dt does this state allow?" where it may not allocate --
// a serving loop whose device memory was reserved once at start-up and may
// not grow (an allocation there can fail, or wait for the whole device,
// since cudaMalloc and cudaFree synchronise with running work), or a host
// program that owns all of its device buffers and hands the library only
// pointers.  The instance API (gop_create / gop_prepare) needs its own
// buffers; this entry point needs none.
//
// Its only scratch is g_cfl_scratch below: a file-scope device array of
// GOP_NOALLOC_SCRATCH_DOUBLES doubles (64 KiB) that every GPU loading this
// library holds until the process exits.  It stores the three coordinate
// arrays of the call (at most GOP_NOALLOC_MAX_N active cells per axis) and
// one (dt, div B) partial per block of the reduction.  Every call overwrites
// what it reads, so nothing has to start at zero; but all calls share the
// one array, so two calls whose kernels overlap on the GPU (different
// streams, or different host threads) race on it.
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <mutex>

#include "gamera_op.h"
#include "gop_internal.h"

namespace {

constexpr int kMaxN = GOP_NOALLOC_MAX_N;               // active cells per axis
constexpr int kStride = kMaxN + 16;                    // coordinate slot length
constexpr int kMaxBlocks = 2048;                       // reduction partials
constexpr int kScratch = GOP_NOALLOC_SCRATCH_DOUBLES;  // 3 slots + 2 * blocks
static_assert(3 * kStride + 2 * kMaxBlocks <= kScratch, "scratch layout");

__device__ __align__(256) double g_cfl_scratch[kScratch];

constexpr int NG = 4;
constexpr int kThreads = 256;

struct Args {
  int n[3], N[3];
  int sph;
  double gamma, cfl, ca;
  double ca2m, ca2s;  // ca^2 = ca2m / ca2s (split_ca2)
  const double* gas;  // [6][NI][NJ][NK], k fastest (reference layout)
  const double* fb;   // [3][NI][NJ][NK]
  const double* b0;   // background field at the cell centroid [3][NI][NJ][NK], or null
  const double* b0f;  // background field averaged over the faces [9][NI][NJ][NK], or null
  double* scratch;    // device address of g_cfl_scratch on this device
  double* out;        // out[0] = dt, out[1] = max|div B|
  int nblocks;
  int rows;           // rows of cells along k per block
};

__device__ __forceinline__ const double* coord(const Args& A, int a) {
  return A.scratch + (size_t)a * kStride;
}

// position of the volume centroid along axis a in cell c (x1ctr / x2ctr /
// x3ctr of src/cartesian/cartesian_general.c:190-201 and
// src/spherical/spherical_general.c:205-234)
__device__ double centroid(const Args& A, int a, int c) {
  const double* x = coord(A, a);
  double x0 = x[c], x1 = x[c + 1], xc = 0.5 * (x0 + x1), dx = x1 - x0;
  if (!A.sph || a == 2) return xc;
  if (a == 0) return xc + 2.0 * xc * dx * dx / (12.0 * xc * xc + dx * dx);
  return (sin(x1) - sin(x0) - (x1 * cos(x1) - x0 * cos(x0))) / (-cos(x1) + cos(x0));
}

// What a row of cells along k shares.  The geometry is separable, so a
// cell's centred field, div B and inverse CFL length are products of these
// with the k table below.
struct Row {
  double lo1, hi1, lo2, hi2;  // weights of the lower and upper face in the centred field
  double d1l, d1u, d2l, d2u;  // div B = b1u d1u - b1l d1l + b2u d2u - b2l d2l
  double d3;                  //         + (b3u - b3l) d3 / dx3
  double il, il3;             // 1/l1 + 1/l2 + 1/l3 = il + il3 / dx3
  size_t cell;                // its first active cell
};
__device__ void row_of(const Args& A, int i, int j, Row& R) {
  R.cell = ((size_t)i * A.N[1] + j) * A.N[2] + NG;
  const double *x1 = coord(A, 0), *x2 = coord(A, 1);
  const double a0 = x1[i], a1 = x1[i + 1], b0 = x2[j], b1 = x2[j + 1];
  const double i1 = 1.0 / (a1 - a0), i2 = 1.0 / (b1 - b0);
  const double ca = centroid(A, 0, i), cb = centroid(A, 1, j);
  // cell-centred field from the faces (src/solver_func.c:311-322)
  R.lo1 = (a1 - ca) * i1;
  R.hi1 = (ca - a0) * i1;
  R.lo2 = (b1 - cb) * i2;
  R.hi2 = (cb - b0) * i2;
  if (!A.sph) {
    R.d1l = R.d1u = i1;
    R.d2l = R.d2u = i2;
    R.d3 = R.il3 = 1.0;
    R.il = i1 + i2;
    return;
  }
  // face areas over the volume (spherical_general.c:42-201)
  const double h = 0.5 * (a1 * a1 - a0 * a0);
  const double iv = 3.0 / (a1 * a1 * a1 - a0 * a0 * a0), ic = 1.0 / (cos(b0) - cos(b1));
  R.d1l = a0 * a0 * iv;
  R.d1u = a1 * a1 * iv;
  R.d2l = h * sin(b0) * iv * ic;
  R.d2u = h * sin(b1) * iv * ic;
  R.d3 = h * (b1 - b0) * iv * ic;
  const double rc = 0.5 * (a0 + a1), irc = 1.0 / rc;
  R.il = i1 + irc * i2;
  R.il3 = irc / sin(0.5 * (b0 + b1));
}

// vc times the cell's inverse CFL length (get_dt_normal,
// src/solver_func.c:255-298) and |div B| (src/solver_func.c:324-343) of cell
// c; s1, s2 the strides along i and j, n3 between fields, k the place in the
// k table (lo3, hi3, 1 / dx3)
__device__ __forceinline__ void cell_rate_divb(const Args& A, size_t c, size_t s1, size_t s2, size_t n3,
                                               const Row& R, double lo3, double hi3, double id3,
                                               double& rate, double& divb) {
  const double *g = A.gas + c, *b = A.fb + c;
  const double rho = g[0], u = g[n3], v = g[2 * n3], w = g[3 * n3], p = g[4 * n3];
  double bl[3] = {b[0], b[n3], b[2 * n3]};
  double bu[3] = {b[s1], b[n3 + s2], b[2 * n3 + 1]};
  double m1 = bl[0] * R.lo1 + bu[0] * R.hi1;
  double m2 = bl[1] * R.lo2 + bu[1] * R.hi2;
  double m3 = bl[2] * lo3 + bu[2] * hi3;
  if (A.b0) {
    // magtot = mags + B0 (src/solver_func.c:345-353); the face-normal field
    // plus the face-averaged background normal component (B0AfaceI/J/K_bn)
    m1 += A.b0[c];
    m2 += A.b0[n3 + c];
    m3 += A.b0[2 * n3 + c];
    const double* f0 = A.b0f + c;           // faces normal to i, component i
    const double* f1 = A.b0f + 4 * n3 + c;  // faces normal to j, component j
    const double* f2 = A.b0f + 8 * n3 + c;  // faces normal to k, component k
    bl[0] += f0[0];
    bu[0] += f0[s1];
    bl[1] += f1[0];
    bu[1] += f1[s2];
    bl[2] += f2[0];
    bu[2] += f2[1];
  }
  // |v| + sqrt(cs^2 + va^2) with va^2 = v^2 ca^2 / (v^2 + ca^2), v^2 = b^2 /
  // rho, over the common denominator; by the separate roots (which decide whether
  // there is a speed) where the density or the pressure is not above zero or
  // the product leaves the range of a double
  const double b2 = m1 * m1 + m2 * m2 + m3 * m3, r = A.ca2m * rho, q = fma(A.ca2m, rho, b2 * A.ca2s);
  const double num = A.gamma * p * q + b2 * r, t = num * (rho * q);
  double f = num * rsqrt(t);
  if (!(t >= DBL_MIN && t <= DBL_MAX && rho > 0.0 && p >= 0.0)) {
    const double vs = sqrt(A.gamma * p / rho), va = sqrt(b2 / rho), ve = va * A.ca / sqrt(va * va + A.ca * A.ca);
    f = sqrt(vs * vs + ve * ve);
  }
  rate = (sqrt(u * u + v * v + w * w) + f) * (R.il + R.il3 * id3);
  divb = fabs((bu[0] * R.d1u - bl[0] * R.d1l) + (bu[1] * R.d2u - bl[1] * R.d2l) +
              (bu[2] - bl[2]) * (R.d3 * id3));
}

// Per-block (min dt, max |div B|) into the scratch partials.  The block takes
// A.rows rows of cells along k (k contiguous in memory), kRows at a time: what
// depends on i and j alone is worked out once per row, what depends on k once
// per block, and a cell is left with a root, a reciprocal root and no
// division.  Before, every cell evaluated its geometry with about 18 divisions
// and roots and two 64-bit index divisions, which bound the kernel: 192^3 on
// B200 414 -> 103 us a call (4.4 TB/s of the 8 fields read once).
constexpr int kRows = 16;
__global__ void __launch_bounds__(kThreads) k_cfl_partial(Args A) {
  __shared__ double sdt[kThreads / 32], sdb[kThreads / 32];
  __shared__ double lo3[kMaxN], hi3[kMaxN], id3[kMaxN];
  __shared__ Row rows[kRows];
  const int nk = A.n[2], nj = A.n[1];
  const size_t s2 = A.N[2], s1 = (size_t)A.N[1] * A.N[2], n3 = (size_t)A.N[0] * s1;
  const double* x3 = coord(A, 2);
  for (int k = threadIdx.x; k < nk; k += kThreads) {
    const double z0 = x3[k + NG], z1 = x3[k + NG + 1], zc = 0.5 * (z0 + z1), id = 1.0 / (z1 - z0);
    lo3[k] = (z1 - zc) * id;
    hi3[k] = (zc - z0) * id;
    id3[k] = id;
  }
  // a thread's cells of the row set: (row, k), kThreads apart
  const int dr = kThreads / nk, dk = kThreads % nk;
  const int first = blockIdx.x * A.rows, last = min(first + A.rows, A.n[0] * nj);
  double rate = 0.0, db = 0.0;
  for (int r0 = first; r0 < last; r0 += kRows) {
    const int nr = min(kRows, last - r0);
    __syncthreads();  // the rows before have been used, the k table is written
    if (threadIdx.x < nr) {
      const int row = r0 + threadIdx.x;
      row_of(A, row / nj + NG, row % nj + NG, rows[threadIdx.x]);
    }
    __syncthreads();
    int r = threadIdx.x / nk, k = threadIdx.x % nk;
    while (r < nr) {
      double c_rate, c_db;
      cell_rate_divb(A, rows[r].cell + k, s1, s2, n3, rows[r], lo3[k], hi3[k], id3[k], c_rate, c_db);
      rate = fmax(rate, c_rate);
      db = fmax(db, c_db);
      r += dr;
      k += dk;
      if (k >= nk) {
        k -= nk;
        r++;
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    rate = fmax(rate, __shfl_xor_sync(0xffffffffu, rate, o));
    db = fmax(db, __shfl_xor_sync(0xffffffffu, db, o));
  }
  if ((threadIdx.x & 31) == 0) {
    sdt[threadIdx.x / 32] = rate;
    sdb[threadIdx.x / 32] = db;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kThreads / 32; w++) {
      rate = fmax(rate, sdt[w]);
      db = fmax(db, sdb[w]);
    }
    double* part = A.scratch + 3 * kStride;
    part[2 * blockIdx.x] = rate > 0.0 ? fmin(A.cfl / rate, DBL_MAX) : DBL_MAX;
    part[2 * blockIdx.x + 1] = db;
  }
}

// one block folds the partials written by this call into out[0..1]
__global__ void __launch_bounds__(kThreads) k_cfl_final(Args A) {
  __shared__ double sdt[kThreads / 32], sdb[kThreads / 32];
  const double* part = A.scratch + 3 * kStride;
  double dt = DBL_MAX, db = 0.0;
  for (int t = threadIdx.x; t < A.nblocks; t += blockDim.x) {
    dt = fmin(dt, part[2 * t]);
    db = fmax(db, part[2 * t + 1]);
  }
  for (int o = 16; o > 0; o >>= 1) {
    dt = fmin(dt, __shfl_xor_sync(0xffffffffu, dt, o));
    db = fmax(db, __shfl_xor_sync(0xffffffffu, db, o));
  }
  if ((threadIdx.x & 31) == 0) {
    sdt[threadIdx.x / 32] = dt;
    sdb[threadIdx.x / 32] = db;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kThreads / 32; w++) {
      dt = fmin(dt, sdt[w]);
      db = fmax(db, sdb[w]);
    }
    A.out[0] = dt;
    A.out[1] = db;
  }
}

// device address of g_cfl_scratch, looked up once per device
std::mutex g_mu;
double* g_addr[64] = {};

}  // namespace

extern "C" int gop_cfl_dt_noalloc(const gop_desc* desc, const double* gas, const double* face_b,
                                  const double* b0, const double* b0_face, double* out,
                                  void* stream) {
  int rc = gop::check_desc(desc);
  if (rc) return rc;
  if (!gas || !face_b || !out) return gop::set_error(GOP_EINVAL, "gop_cfl_dt_noalloc: NULL array");
  if ((b0 == nullptr) != (b0_face == nullptr))
    return gop::set_error(GOP_EINVAL, "gop_cfl_dt_noalloc: b0 and b0_face go together");
  // ring-averaged grids take the CFL length of their pole rows from the
  // ring average (get_dt_ring), which this call does not compute
  if (desc->ring_average)
    return gop::set_error(GOP_EINVAL, "gop_cfl_dt_noalloc: grids with the pole ring average are not supported");
  if (desc->ni > kMaxN || desc->nj > kMaxN || desc->nk > kMaxN)
    return gop::set_error(GOP_EINVAL,
                          "gop_cfl_dt_noalloc: grid %dx%dx%d exceeds the static scratch limit of %d "
                          "active cells per axis",
                          desc->ni, desc->nj, desc->nk, kMaxN);
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64)
    return gop::set_error(GOP_ECUDA, "gop_cfl_dt_noalloc: cudaGetDevice: %s", cudaGetErrorString(e));
  double* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_mu);
    if (!g_addr[dev]) {
      // first call on this device: resolve the array's device address
      e = cudaGetSymbolAddress((void**)&g_addr[dev], g_cfl_scratch);
      if (e != cudaSuccess) {
        g_addr[dev] = nullptr;
        return gop::set_error(GOP_ECUDA, "gop_cfl_dt_noalloc: cudaGetSymbolAddress: %s",
                              cudaGetErrorString(e));
      }
    }
    scratch = g_addr[dev];
  }
  cudaStream_t st = (cudaStream_t)stream;
  Args A;
  A.n[0] = desc->ni;
  A.n[1] = desc->nj;
  A.n[2] = desc->nk;
  for (int a = 0; a < 3; a++) A.N[a] = A.n[a] + 2 * NG + 1;
  A.sph = desc->coord == GOP_COORD_SPHERICAL;
  A.gamma = desc->gamma != 0 ? desc->gamma : 5.0 / 3.0;
  A.cfl = desc->cfl != 0 ? desc->cfl : 0.3;
  A.ca = desc->ca != 0 ? desc->ca : 10.0;
  gop::split_ca2(A.ca, A.ca2m, A.ca2s);
  A.gas = gas;
  A.fb = face_b;
  A.b0 = b0;
  A.b0f = b0_face;
  A.scratch = scratch;
  A.out = out;
  const double* xs[3] = {desc->x1, desc->x2, desc->x3};
  for (int a = 0; a < 3; a++) {
    e = cudaMemcpyAsync(scratch + (size_t)a * kStride, xs[a], sizeof(double) * A.N[a],
                        cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess)
      return gop::set_error(GOP_ECUDA, "gop_cfl_dt_noalloc: coordinate copy: %s", cudaGetErrorString(e));
  }
  // at least 4 cells a thread, at most kMaxBlocks blocks
  const int nrows = A.n[0] * A.n[1];
  const int fill = (4 * kThreads + A.n[2] - 1) / A.n[2], spread = (nrows + kMaxBlocks - 1) / kMaxBlocks;
  A.rows = fill > spread ? fill : spread;
  A.nblocks = (nrows + A.rows - 1) / A.rows;
  k_cfl_partial<<<A.nblocks, kThreads, 0, st>>>(A);
  k_cfl_final<<<1, kThreads, 0, st>>>(A);
  e = cudaGetLastError();
  if (e != cudaSuccess)
    return gop::set_error(GOP_ECUDA, "gop_cfl_dt_noalloc: launch: %s", cudaGetErrorString(e));
  return GOP_OK;
}
