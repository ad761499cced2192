// Tile-staged sweeps of the MHD step for B200 (sm_100a): the face flux and
// the edge EMF, the step's two stencil stages, computed from shared-memory
// tiles that the Tensor Memory Accelerator streams in ahead of the
// arithmetic.
//
// Face flux along axis D: PDM reconstruction of the 8 face states, Rusanov
// flux and Maxwell stress (src/solver_func.c:215-253,503-685,934-1529).
// Edge EMF along axis D: the second centre-to-edge sweep, the two face-field
// reconstructions and the EMF (src/solver_func.c:686-902).  Their per-point
// forms (k_flux, k_emf in gop_kernels.cu) gather each output's 8-point
// stencils with dozens of global loads through L1; the loads' 64-bit
// address arithmetic and latency, not the FP64 arithmetic, bound them.
// Here each block is persistent and runs a copy pipeline:
//
//   copies   one elected thread streams tiles into a ring of 2-4
//            shared-memory slots (as many as fit the SM at the kernel's
//            residency) with cp.async.bulk.tensor (one TMA box per
//            input array and tile: stencil windows, limiter windows, PDM
//            weights), completing on the slot's "full" mbarrier;
//   compute  8 warps compute one face, or one or two edges, per thread from
//            shared memory (every stencil tap is a load at a compile-time
//            offset from one per-thread base) and release the slot on its
//            "empty" mbarrier; the feeding thread refills a released slot
//            with the next tile not yet taken, a ring's length ahead.
//
// So the global-memory latency of tile n+1 overlaps the arithmetic of tile
// n, and the stencil re-reads come from shared memory instead of L1.  The
// per-point arithmetic is the per-point kernels' own (recon_lr, flux_out,
// emf_finish), in the same order, so both forms give the same results (to a
// multiply-add the compiler contracts in one and not in the other).
//
// Lanes always run along i (x, the TMA box's contiguous axis); a tile is 32
// lanes x 8 or 16 rows, a warp's row along the stage's sweep axis or its
// third axis.  Every box starts at an x of 32 t or 4 + 32 t, so x times the
// element size is a multiple of 16 bytes (the TMA's alignment rule); no
// coordinate is negative.  Boxes reaching past the grid are filled with
// zeros by the TMA and only feed threads outside the grid, which store
// nothing.  Tiles are numbered with the x tile fastest, then the tile along
// the warps, so the blocks in flight at any time share their halo rows in
// L2.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "gop_stage.cuh"
#include "gop_tma.cuh"
#include "gop_update.cuh"

namespace gop {

constexpr int kWarps = 8;
constexpr int kSweepThreads = 32 * kWarps;

// shared-memory ring and residency per arithmetic type: at least two slots;
// two blocks per SM in FP64 (128 registers), three in FP32 (the flux; the
// EMF below)
#ifndef GOP_SWEEP_STAGES_F64
#define GOP_SWEEP_STAGES_F64 2
#endif
#ifndef GOP_SWEEP_STAGES_F32
#define GOP_SWEEP_STAGES_F32 2
#endif
#ifndef GOP_SWEEP_CTAS_F64
#define GOP_SWEEP_CTAS_F64 2
#endif
#ifndef GOP_SWEEP_CTAS_F32
#define GOP_SWEEP_CTAS_F32 3
#endif
// blocks per SM of the edge-EMF sweeps (smaller slots than the flux
// sweeps); FP32: four (64 registers, no spills) measured 1.06 ms per 256^3
// step on B200 against 1.13 ms with three
#ifndef GOP_SWEEP_EMF_CTAS_F64
#define GOP_SWEEP_EMF_CTAS_F64 GOP_SWEEP_CTAS_F64
#endif
#ifndef GOP_SWEEP_EMF_CTAS_F32
#define GOP_SWEEP_EMF_CTAS_F32 4
#endif
// 1: the sweeps go out with programmatic dependent launch like the other
// step kernels.  Off: a sweep grid placed early onto SMs that still run the
// previous kernel (persistent blocks, no room to spare) measured 2-20 %
// slower on B200 (blast 256^3: FP32 flux 2.47 vs 2.06 ms per step)
#ifndef GOP_SWEEP_PDL
#define GOP_SWEEP_PDL 0
#endif
template <typename R, bool EMF>
struct SweepCfg {
  // the least number of slots; a kernel whose slots are small takes more
  // (ring_slots below)
  static constexpr int STAGES = sizeof(R) == 8 ? GOP_SWEEP_STAGES_F64 : GOP_SWEEP_STAGES_F32;
  static constexpr int CTAS = EMF ? (sizeof(R) == 8 ? GOP_SWEEP_EMF_CTAS_F64 : GOP_SWEEP_EMF_CTAS_F32)
                                  : (sizeof(R) == 8 ? GOP_SWEEP_CTAS_F64 : GOP_SWEEP_CTAS_F32);
};
#ifndef GOP_SWEEP_MAX_STAGES
#define GOP_SWEEP_MAX_STAGES 4
#endif

// a box of the slot: extents (x, y, z, fields) and elements, rounded up to
// 32 so every box starts on a 128-byte boundary in FP32 and FP64
struct Box {
  int x, y, z, f;
  __host__ __device__ constexpr int elems() const { return x * y * z * f; }
  __host__ __device__ constexpr int padded() const { return (elems() + 31) / 32 * 32; }
};
// n packed face records
constexpr Box rec(int n) { return Box{FW, n, 1, 1}; }
// tap-major weights (T_WL0..T_CR2) of the 32 faces of a warp row and of the
// face after them (the sweeps on i faces, below)
constexpr Box kTap40{40, 18, 1, 1};

// The sweeps whose lanes run along i over the n+1 faces of an i row (the flux
// along i, the EMFs along j and k) tile the row in ceil(n/32) tiles of 32
// faces; when 32 divides n the last face of the row, the upper boundary
// face, is left over.  The last tile of the row then computes it too, in
// one extra pass of one warp whose lanes take the tile's 8 rows (its boxes
// are 40 wide along i, so that face's stencil is in the slot), where a
// ninth tile would cost eight warp passes with one live lane each.  The pass
// is a second trip through the same code (a second copy of a face's
// arithmetic, or a call, cost the flux more than it saved).
__device__ __forceinline__ bool row_end_face(const Params& P, int x0) { return x0 + 32 == NGH + P.n[0]; }

// the weights of one face of the tile (tap-major rows of X faces in shared
// memory)
template <int X, typename R>
__device__ __forceinline__ void load_tap(const R* w, FaceWeights<R>& W) {
#pragma unroll
  for (int u = 0; u < 7; u++) {
    W.wl[u] = w[u * X];
    W.wr[u] = w[(7 + u) * X];
  }
  W.set_limiter(w[14 * X], w[15 * X], w[16 * X], w[17 * X]);
}

// ------------------------------------------------------------------ flux

template <int D>
struct FluxTile {
  static constexpr int NG = 5;  // gas fields (the entropy channel is off)
  // stencil and limiter windows of the tile's faces
  static constexpr Box S = D == 0 ? Box{40, 8, 1, 1} : (D == 1 ? Box{32, 15, 1, 1} : Box{32, 1, 15, 1});
  static constexpr Box L = D == 0 ? Box{40, 8, 1, 1} : (D == 1 ? Box{32, 11, 1, 1} : Box{32, 1, 11, 1});
  static constexpr int ROWS = kWarps;
  static constexpr Box WT = D == 0 ? kTap40 : rec(8);
  static constexpr Box BN = D == 0 ? Box{40, 8, 1, 1} : (D == 2 ? Box{32, 1, 8, 1} : Box{32, 8, 1, 1});
  static constexpr int SB = S.elems(), LB = L.elems();
  // slot layout in elements: W_h, limiter W, mags_h, mags, weights, B_n
  static constexpr int OFF_WH = 0;
  static constexpr int OFF_WL = OFF_WH + NG * SB;
  static constexpr int OFF_MSH = OFF_WL + NG * LB;
  static constexpr int OFF_MS = OFF_MSH + 3 * SB;
  static constexpr int OFF_W = OFF_MS + 3 * LB;
  static constexpr int OFF_BN = OFF_W + WT.padded();
  static constexpr int ELEMS = OFF_BN + BN.padded();
  // elements the TMA delivers into a slot (the barrier's transaction count)
  static constexpr int TX = NG * SB + NG * LB + 3 * SB + 3 * LB + WT.elems() + BN.elems();
  static_assert((NG * SB) % 32 == 0 && (NG * LB) % 32 == 0 && (3 * SB) % 32 == 0 &&
                    (3 * LB) % 32 == 0,
                "flux boxes on 128-byte boundaries");
};

struct alignas(64) FluxMaps {
  CUtensorMap wh;     // W_h, stencil box
  CUtensorMap wl[2];  // limiter reference: FP64 the state buffer of each parity, FP32 its copy
  CUtensorMap msh;    // mags_h, stencil box
  CUtensorMap ms;     // mags, limiter box
  CUtensorMap wt;     // PDM weights of the tile's faces
  CUtensorMap bn[2];  // step-start face field (as wl: per parity in FP64)
  int nt[3];          // tiles: x, along the warps, third axis
  uint64_t inv[2];    // inverse_of(nt[0]), inverse_of(nt[1])
};

// a tile: its axis, its first cell or face on each axis, and the warp that
// takes the row's upper boundary face (-1: not this tile's)
struct alignas(16) Tile {
  short D, end_warp;
  int x0, y0, z0;
};
// n / d for d > 1 from inv = floor(2^64 / d) + 1: exact while n d < 2^64
__host__ __device__ constexpr uint64_t inverse_of(int d) { return d > 1 ? ~0ull / (uint64_t)d + 1 : 0; }
__device__ __forceinline__ int div_by(int n, int d, uint64_t inv) {
  return d > 1 ? (int)__umul64hi((uint64_t)n, inv) : n;
}
// Tile r of the nt[0] x nt[1] x nt[2] tiles of a stage, x fastest, as its three
// digits.  The feeding thread works this out and the others read the tile from
// shared memory; its warp is the last of the block at every tile, so the two
// divisions are products with the counts' inverses (FP64 EMF stage 1.81 ->
// 1.76 ms per blast 256^3 step on B200).
template <class Maps>
__device__ __forceinline__ int3 tile_digits(const Maps& m, int r) {
  const int* nt = m.nt;
  const int q = div_by(r, nt[0], m.inv[0]), c = div_by(q, nt[1], m.inv[1]);
  return make_int3(r - q * nt[0], q - c * nt[1], c);
}
// a tile of a sweep along D
template <int D, bool EMF, int ROWS, class Maps>
__device__ __forceinline__ Tile sweep_tile(const Params& P, const Maps& m, int r) {
  const int3 d = tile_digits(m, r);
  Tile T;
  T.D = D;
  T.x0 = NGH + 32 * d.x;
  // the rows of a tile run along k where its windows do (flux along k, EMFs
  // along i and j), along j otherwise
  if constexpr (EMF ? D != 2 : D == 2) {
    T.y0 = NGH + d.z;
    T.z0 = NGH + ROWS * d.y;
  } else {
    T.y0 = NGH + ROWS * d.y;
    T.z0 = NGH + d.z;
  }
  // the warp of the row-end pass rotates over the row sets
  constexpr bool ends = EMF ? D != 0 : D == 0;
  T.end_warp = ends && row_end_face(P, T.x0) ? (short)((d.y + m.nt[1] * d.z) & (kWarps - 1)) : (short)-1;
  return T;
}
// what a thread gathers over its tiles (the update)
struct Gather {
  double rate = 0.0, divb = 0.0;
};

template <typename R, int D, bool BG, bool POLE>
struct FluxStage {
  using F = FluxTile<D>;
  using Maps = FluxMaps;
  static constexpr int ELEMS = F::ELEMS, ROWS = F::ROWS;
  static constexpr int BYTES = F::TX * (int)sizeof(R);
  __device__ static Tile place(const Params& P, const Maps& m, int r) {
    return sweep_tile<D, false, ROWS>(P, m, r);
  }
  static constexpr int TX = F::TX;

  __device__ static void issue(const Params& P, const Maps& m, int par, const Tile& T, R* s,
                               uint64_t* bar) {
    const int f0 = D == 0 ? T.x0 : (D == 1 ? T.y0 : T.z0);  // first face along D
    // stencil windows start 4 cells before the first face, limiter windows
    // 2 (along i both start 4 before, keeping x aligned)
    const int sx = D == 0 ? T.x0 - 4 : T.x0, sy = D == 1 ? T.y0 - 4 : T.y0, sz = D == 2 ? T.z0 - 4 : T.z0;
    const int ly = D == 1 ? T.y0 - 2 : T.y0, lz = D == 2 ? T.z0 - 2 : T.z0;
    tma_load_4d(s + F::OFF_WH, &m.wh, bar, sx, sy, sz, 0);
    tma_load_4d(s + F::OFF_WL, &m.wl[par], bar, sx, ly, lz, 0);
    tma_load_4d(s + F::OFF_MSH, &m.msh, bar, sx, sy, sz, 0);
    tma_load_4d(s + F::OFF_MS, &m.ms, bar, sx, ly, lz, 0);
    if constexpr (D == 0) tma_load_4d(s + F::OFF_W, &m.wt, bar, f0, T_WL0, 0, 0);
    else tma_load_4d(s + F::OFF_W, &m.wt, bar, 0, D * P.tmax + f0, 0, 0);
    tma_load_4d(s + F::OFF_BN, &m.bn[par], bar, T.x0, T.y0, T.z0, D);
  }

  // the face in tile row `row` (a warp's row), column `col` (a lane's face)
  __device__ __forceinline__ static void point(const Params& P, const Work<R>& wk, const R* s,
                                               const Tile& T, int row, int col, Gather&) {
    const int i = T.x0 + col, j = T.y0 + (D == 2 ? 0 : row), k = T.z0 + (D == 2 ? row : 0);
    if (!(i < NGH + P.n[0] + (D == 0) && j < NGH + P.n[1] + (D == 1) && k < NGH + P.n[2] + (D == 2)))
      return;
    // per-thread bases: tap u of field f is then at a compile-time offset
    const R *wh, *wl, *msh, *ms;
    if constexpr (D == 0) {
      const int b = row * 40 + col;
      wh = s + F::OFF_WH + b;
      wl = s + F::OFF_WL + b + 2;  // the limiter cells f-2..f+1 start 2 cells in
      msh = s + F::OFF_MSH + b;
      ms = s + F::OFF_MS + b + 2;
    } else {
      const int b = row * 32 + col;
      wh = s + F::OFF_WH + b;
      wl = s + F::OFF_WL + b;
      msh = s + F::OFF_MSH + b;
      ms = s + F::OFF_MS + b;
    }
    constexpr int TS = D == 0 ? 1 : 32;  // stride of one stencil tap in the slot
    FaceWeights<R> Wt;
    if constexpr (D == 0) load_tap<40>(s + F::OFF_W + col, Wt);
    else load_fw_smem(s + F::OFF_W + row * FW, Wt);
    const R bn = s[F::OFF_BN + row * F::BN.x + col];
    R L[6], Rt[6], mL[3], mR[3];
    L[PS] = Rt[PS] = R(0);
#pragma unroll
    for (int f = 0; f < F::NG; f++) {
      R v[8], lim[4];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = wh[f * F::SB + u * TS];
#pragma unroll
      for (int u = 0; u < 4; u++) lim[u] = wl[f * F::LB + u * TS];
      recon_lr<POLE && D == 1>(v, lim, Wt, L[f], Rt[f]);
    }
#pragma unroll
    for (int a = 0; a < 3; a++) {
      R v[8], lim[4];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = msh[a * F::SB + u * TS];
#pragma unroll
      for (int u = 0; u < 4; u++) lim[u] = ms[a * F::LB + u * TS];
      recon_lr<POLE && D == 1>(v, lim, Wt, mL[a], mR[a]);
    }
    flux_out<R, D, BG, false>(P, wk, lin32(P, i, j, k), D == 0 ? j : (D == 1 ? k : i), L, Rt, mL, mR,
                              bn);
  }
};

// ------------------------------------------------------------------- EMF

// Edge EMF along D, p = D+1, q = D+2 (mod 3).  Inputs per edge: the two
// first-sweep velocities along q (V, 8 cells; limited against themselves),
// B_p along q (8 half-step, 4 step-start values), B_q along p (8 + 4), the
// four half-step densities around the edge, the weights of its q and p faces.
//   D = 0 (p = j, q = k): lanes cells along i, warps k faces, one j face
//   D = 1 (p = k, q = i): lanes i faces, warps k faces, one j cell
//   D = 2 (p = i, q = j): lanes i faces, warps j faces, one k cell
template <int D>
struct EmfTile {
  // Rows of edges per tile.  A tile's fixed costs (its number, its eight
  // copies, the barrier waits, the row halo of the windows) weigh on an edge's
  // 530 instructions: two rows per warp share them, 16 instead of 8 taking
  // the EMF stage of a blast 256^3 step on B200 from 1.76 to 1.55 ms (FP64)
  // and 0.93 to 0.85 (FP32).  Along i 16 rows would leave no room for a
  // second slot.
  static constexpr int ROWS = D == 0 ? 8 : 16;
  static constexpr int H7 = ROWS + 7, H3 = ROWS + 3, H1 = ROWS + 1;  // rows with the windows' halos
  static constexpr Box V = D == 0 ? Box{32, 1, H7, 2} : (D == 1 ? Box{40, 1, ROWS, 2} : Box{40, H7, 1, 2});
  static constexpr Box BHP = D == 0 ? Box{32, 1, H7, 1} : (D == 1 ? Box{40, 1, ROWS, 1} : Box{40, H7, 1, 1});
  static constexpr Box BLP = D == 0 ? Box{32, 1, H3, 1} : (D == 1 ? Box{40, 1, ROWS, 1} : Box{40, H3, 1, 1});
  static constexpr Box BHQ = D == 0 ? Box{32, 8, ROWS, 1} : (D == 1 ? Box{40, 1, H7, 1} : Box{40, ROWS, 1, 1});
  static constexpr Box BLQ = D == 0 ? Box{32, 4, ROWS, 1} : (D == 1 ? Box{40, 1, H3, 1} : Box{40, ROWS, 1, 1});
  static constexpr Box RHO = D == 0 ? Box{32, 2, H1, 1} : (D == 1 ? Box{40, 1, H1, 1} : Box{40, H1, 1, 1});
  static constexpr Box WQ = D == 1 ? kTap40 : rec(ROWS);
  static constexpr Box WP = D == 0 ? rec(1) : (D == 1 ? rec(ROWS) : kTap40);
  static constexpr int VF = V.x * V.y * V.z;  // elements of one V field
  static constexpr int OFF_V = 0;
  static constexpr int OFF_BHP = OFF_V + V.padded();
  static constexpr int OFF_BLP = OFF_BHP + BHP.padded();
  static constexpr int OFF_BHQ = OFF_BLP + BLP.padded();
  static constexpr int OFF_BLQ = OFF_BHQ + BHQ.padded();
  static constexpr int OFF_RHO = OFF_BLQ + BLQ.padded();
  static constexpr int OFF_WQ = OFF_RHO + RHO.padded();
  static constexpr int OFF_WP = OFF_WQ + WQ.padded();
  static constexpr int ELEMS = OFF_WP + WP.padded();
  // elements the TMA delivers into a slot (the barrier's transaction count)
  static constexpr int TX = V.elems() + BHP.elems() + BLP.elems() + BHQ.elems() + BLQ.elems() +
                            RHO.elems() + WQ.elems() + WP.elems();
};

struct alignas(64) EmfMaps {
  CUtensorMap v;       // first-sweep velocities V (2 of its 6 fields)
  CUtensorMap bhp;     // B_h, component p, window along q
  CUtensorMap blp[2];  // step-start B (per parity in FP64), component p
  CUtensorMap bhq;     // B_h, component q, window along p
  CUtensorMap blq[2];  // step-start B, component q
  CUtensorMap rho;     // W_h density around the edges
  CUtensorMap wq;      // weights of the q faces
  CUtensorMap wp;      // weights of the p faces
  int nt[3];
  uint64_t inv[2];
};

template <typename R, int D, bool BG, bool POLE>
struct EmfStage {
  using E = EmfTile<D>;
  using Maps = EmfMaps;
  static constexpr int ELEMS = E::ELEMS, ROWS = E::ROWS;
  static constexpr int BYTES = E::TX * (int)sizeof(R);
  __device__ static Tile place(const Params& P, const Maps& m, int r) {
    return sweep_tile<D, true, ROWS>(P, m, r);
  }
  static constexpr int TX = E::TX;
  static constexpr int p = (D + 1) % 3, q = (D + 2) % 3;

  __device__ static void issue(const Params& P, const Maps& m, int par, const Tile& T, R* s,
                               uint64_t* bar) {
    const int x0 = T.x0, y0 = T.y0, z0 = T.z0;
    if constexpr (D == 0) {  // i cells, j face y0, k faces z0..
      tma_load_4d(s + E::OFF_V, &m.v, bar, x0, y0, z0 - 4, 0);
      tma_load_4d(s + E::OFF_BHP, &m.bhp, bar, x0, y0, z0 - 4, 1);
      tma_load_4d(s + E::OFF_BLP, &m.blp[par], bar, x0, y0, z0 - 2, 1);
      tma_load_4d(s + E::OFF_BHQ, &m.bhq, bar, x0, y0 - 4, z0, 2);
      tma_load_4d(s + E::OFF_BLQ, &m.blq[par], bar, x0, y0 - 2, z0, 2);
      tma_load_4d(s + E::OFF_RHO, &m.rho, bar, x0, y0 - 1, z0 - 1, 0);
      tma_load_4d(s + E::OFF_WQ, &m.wq, bar, 0, 2 * P.tmax + z0, 0, 0);
      tma_load_4d(s + E::OFF_WP, &m.wp, bar, 0, P.tmax + y0, 0, 0);
    } else if constexpr (D == 1) {  // i faces, j cell y0, k faces z0..
      tma_load_4d(s + E::OFF_V, &m.v, bar, x0 - 4, y0, z0, 2);
      tma_load_4d(s + E::OFF_BHP, &m.bhp, bar, x0 - 4, y0, z0, 2);
      tma_load_4d(s + E::OFF_BLP, &m.blp[par], bar, x0 - 4, y0, z0, 2);
      tma_load_4d(s + E::OFF_BHQ, &m.bhq, bar, x0, y0, z0 - 4, 0);
      tma_load_4d(s + E::OFF_BLQ, &m.blq[par], bar, x0, y0, z0 - 2, 0);
      tma_load_4d(s + E::OFF_RHO, &m.rho, bar, x0 - 4, y0, z0 - 1, 0);
      tma_load_4d(s + E::OFF_WQ, &m.wq, bar, x0, T_WL0, 0, 0);
      tma_load_4d(s + E::OFF_WP, &m.wp, bar, 0, 2 * P.tmax + z0, 0, 0);
    } else {  // i faces, j faces y0.., k cell z0
      tma_load_4d(s + E::OFF_V, &m.v, bar, x0, y0 - 4, z0, 4);
      tma_load_4d(s + E::OFF_BHP, &m.bhp, bar, x0, y0 - 4, z0, 0);
      tma_load_4d(s + E::OFF_BLP, &m.blp[par], bar, x0, y0 - 2, z0, 0);
      tma_load_4d(s + E::OFF_BHQ, &m.bhq, bar, x0 - 4, y0, z0, 1);
      tma_load_4d(s + E::OFF_BLQ, &m.blq[par], bar, x0 - 4, y0, z0, 1);
      tma_load_4d(s + E::OFF_RHO, &m.rho, bar, x0 - 4, y0 - 1, z0, 0);
      tma_load_4d(s + E::OFF_WQ, &m.wq, bar, 0, P.tmax + y0, 0, 0);
      tma_load_4d(s + E::OFF_WP, &m.wp, bar, x0, T_WL0, 0, 0);
    }
  }

  // the edge in tile row `warp` (a warp's row), column `lane` (a lane's edge)
  __device__ __forceinline__ static void point(const Params& P, const Work<R>& wk, const R* s,
                                               const Tile& T, int warp, int lane, Gather&) {
    const int i = T.x0 + lane, j = T.y0 + (D == 2 ? warp : 0), k = T.z0 + (D == 2 ? 0 : warp);
    if (!(i < NGH + P.n[0] + (D != 0) && j < NGH + P.n[1] + (D != 1) && k < NGH + P.n[2] + (D != 2)))
      return;
    // stencil bases and tap strides of the windows along q and along p (the
    // boxes whose rows run along i on i faces are 40 wide)
    const R *v0, *bp, *bpl, *bq, *bql;
    constexpr int tq = D == 1 ? 1 : (D == 2 ? 40 : 32);  // slot stride of one tap along q
    constexpr int tp = D == 2 ? 1 : (D == 1 ? 40 : 32);  // ... along p
    R rho4;
    const R* rh = s + E::OFF_RHO;
    FaceWeights<R> Wq, Wp;
    if constexpr (D == 0) {  // q = k rows of 32; p = j rows of 32 in the warp's k face
      v0 = s + E::OFF_V + warp * 32 + lane;
      bp = s + E::OFF_BHP + warp * 32 + lane;
      bpl = s + E::OFF_BLP + warp * 32 + lane;
      bq = s + E::OFF_BHQ + warp * 8 * 32 + lane;
      bql = s + E::OFF_BLQ + warp * 4 * 32 + lane;
      // (j-1,k-1) + (j-1,k) + (j,k-1) + (j,k); box rows [k][j]
      const R* r = rh + lane;
      rho4 = r[(warp * 2 + 0) * 32] + r[((warp + 1) * 2 + 0) * 32] + r[(warp * 2 + 1) * 32] +
             r[((warp + 1) * 2 + 1) * 32];
      load_fw_smem(s + E::OFF_WQ + warp * FW, Wq);
      load_fw_smem(s + E::OFF_WP, Wp);
    } else if constexpr (D == 1) {  // q = i in a row of 40; p = k rows of 40
      v0 = s + E::OFF_V + warp * 40 + lane;
      bp = s + E::OFF_BHP + warp * 40 + lane;
      bpl = s + E::OFF_BLP + warp * 40 + lane + 2;
      bq = s + E::OFF_BHQ + warp * 40 + lane;
      bql = s + E::OFF_BLQ + warp * 40 + lane;
      // (i-1,k-1) + (i-1,k) + (i,k-1) + (i,k); box rows of 40 along k
      const R* r = rh + lane + 3;
      rho4 = r[warp * 40] + r[(warp + 1) * 40] + r[warp * 40 + 1] + r[(warp + 1) * 40 + 1];
      load_tap<40>(s + E::OFF_WQ + lane, Wq);
      load_fw_smem(s + E::OFF_WP + warp * FW, Wp);
    } else {  // q = j rows of 40; p = i in a row of 40
      v0 = s + E::OFF_V + warp * 40 + lane;
      bp = s + E::OFF_BHP + warp * 40 + lane;
      bpl = s + E::OFF_BLP + warp * 40 + lane;
      bq = s + E::OFF_BHQ + warp * 40 + lane;
      bql = s + E::OFF_BLQ + warp * 40 + lane + 2;
      // (i-1,j-1) + (i-1,j) + (i,j-1) + (i,j); box rows of 40 along j
      const R* r = rh + lane + 3;
      rho4 = r[warp * 40] + r[(warp + 1) * 40] + r[warp * 40 + 1] + r[(warp + 1) * 40 + 1];
      load_fw_smem(s + E::OFF_WQ + warp * FW, Wq);
      load_tap<40>(s + E::OFF_WP + lane, Wp);
    }
    R vav[2], bpL, bpR, bqL, bqR;
#pragma unroll
    for (int cc = 0; cc < 2; cc++) {  // second sweep along q, limited against itself
      R v[8], lim[4], L, Rr;
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = v0[cc * E::VF + u * tq];
#pragma unroll
      for (int u = 0; u < 4; u++) lim[u] = v[u + 2];
      recon_lr<POLE && q == 1>(v, lim, Wq, L, Rr);
      vav[cc] = R(0.5) * (L + Rr);
    }
    {  // B_p along q
      R v[8], lim[4];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = bp[u * tq];
#pragma unroll
      for (int u = 0; u < 4; u++) lim[u] = bpl[u * tq];
      recon_lr<POLE && q == 1>(v, lim, Wq, bpL, bpR);
    }
    {  // B_q along p
      R v[8], lim[4];
#pragma unroll
      for (int u = 0; u < 8; u++) v[u] = bq[u * tp];
#pragma unroll
      for (int u = 0; u < 4; u++) lim[u] = bql[u * tp];
      recon_lr<POLE && p == 1>(v, lim, Wp, bqL, bqR);
    }
    const int x = lin32(P, i, j, k);
    const size_t fs = P.fs;
    R b0p = R(0), b0q = R(0);
    if constexpr (BG) {  // B0 averaged along the edge (B0Aedge*)
      b0p = (R)P.bg[(size_t)(BG_EDGE + 3 * D + p) * fs + x];
      b0q = (R)P.bg[(size_t)(BG_EDGE + 3 * D + q) * fs + x];
    }
    wk.E[x + (size_t)D * fs] =
        emf_finish<R, BG>(P, vav[0], vav[1], bpL, bpR, bqL, bqR, b0p, b0q, rho4);
  }
};

// ------------------------------------------------------------- pipeline

// A stage's three sweeps as one launch: the stage of each axis, their tensor
// maps, and the order in which the axes' tiles are taken.
// MASK: the axes it is compiled for (bit d).  POLE: with the look at pole faces
// (recon_lr), for grids with the pole ring average alone: those without have no
// face without an area, and it costs the FP64 flux stage 1 to 2 % (128^3 325 -> 329 us).
template <typename R, bool EMF_, bool BG, unsigned MASK_, bool POLE>
struct Sweep {
  static constexpr bool EMF = EMF_, STATE = false;
  static constexpr unsigned MASK = MASK_;
  static constexpr bool H0 = MASK & 1, H1 = MASK >> 1 & 1, H2 = MASK >> 2 & 1;
  template <int D>
  using Stage = typename std::conditional<EMF, EmfStage<R, D, BG, POLE>, FluxStage<R, D, BG, POLE>>::type;
  using Maps = typename Stage<0>::Maps;
  static constexpr int max3(int a, int b, int c) { return a > b ? (a > c ? a : c) : (b > c ? b : c); }
  // a slot holds the tile of any axis
  static constexpr int ELEMS = max3(H0 ? Stage<0>::ELEMS : 0, H1 ? Stage<1>::ELEMS : 0,
                                    H2 ? Stage<2>::ELEMS : 0);
  static constexpr int SLOT = ELEMS * (int)sizeof(R);
  static constexpr int CTAS = SweepCfg<R, EMF>::CTAS;
  // Slots in a block's ring: as many as fit the SM's 228 KB of shared memory
  // at CTAS blocks per SM (each block also reserves 1 KB), at least
  // SweepCfg::STAGES, at most GOP_SWEEP_MAX_STAGES
  static constexpr int fit = (228 * 1024 / CTAS - 1024 - 128 - 256) / SLOT;
  static constexpr int S = fit < SweepCfg<R, EMF>::STAGES
                               ? SweepCfg<R, EMF>::STAGES
                               : (fit > GOP_SWEEP_MAX_STAGES ? GOP_SWEEP_MAX_STAGES : fit);
  static constexpr int SMEM = S * SLOT + S * (2 * 8 + (int)sizeof(Tile)) + 128;
};
template <class Maps>
struct alignas(64) SweepMaps {
  Maps m[3];
  int first[4];  // the tiles of axis order[g] are first[g] .. first[g + 1] - 1
  int order[3];
};

// Persistent sweep: lane 0 of warp 0 also feeds the ring.  It fills the
// first S slots, and after each tile waits until all 8 warps have released
// that tile's slot, then issues the next tile into it; the
// other warps meanwhile compute the tile whose copies were issued S - 1 tiles
// earlier.  Always the same warp: it runs a little behind the others and so
// finds the slot released (with the warps taking turns every tile waited for
// its slowest warp: FP64 flux 2.34 -> 2.90 ms per blast 256^3 step on B200).
// Every wait is bounded; a block that gives up records the failure in S_FLAGS
// (2) and waits for its copies in flight before it exits.
//
// The tiles of several axes run through one launch.  Their number is rarely
// a multiple of the blocks the GPU holds, so three launches leave three
// partly filled last waves, and each starts with an empty ring (a barrier
// set-up and a copy's latency, about 5 us): flux and EMF stage of an FP64 step
// on B200, Orszag-Tang 64x64x4 32 + 21 -> 13 + 13 us, blast 64^3 84 + 54 -> 54
// + 41 us.
//
// A block takes its first tile by its number and each further one from a
// counter (S_TILE), so the tiles in flight at any time are neighbours.  With
// tiles dealt out in turn (t + grid, t + 2 grid, ...) the blocks whose tiles
// take longer -- always the same ones where the row's tiles divide the grid:
// the row-end tiles -- fell behind, and neighbours along i, which share
// memory lines at their common edge, met them at different times (FP64 flux
// stage of a blast 256^3 step 3.16 ms, with the counter 2.40).  In a batch a block that starts late finds less work left.
template <class SW, typename R>
__device__ __forceinline__ void sweep_run(const Params& P, const Work<R>& wk,
                                          const SweepMaps<typename SW::Maps>& maps, Gather& gather) {
  if (stopped(P)) return;
  constexpr int S = SW::S;
  using S0 = typename SW::template Stage<0>;
  using S1 = typename SW::template Stage<1>;
  using S2 = typename SW::template Stage<2>;
  static_assert((!SW::H0 || S0::BYTES <= SW::SLOT) && (!SW::H1 || S1::BYTES <= SW::SLOT) &&
                    (!SW::H2 || S2::BYTES <= SW::SLOT),
                "slot holds its boxes");
  extern __shared__ unsigned char smem_dyn[];
  // TMA destinations on 128-byte boundaries (the launch adds 128 bytes)
  unsigned char* base = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 127) & ~static_cast<uintptr_t>(127));
  R* slots = reinterpret_cast<R*>(base);
  Tile* tiles = reinterpret_cast<Tile*>(base + S * SW::SLOT);
  uint64_t* full = reinterpret_cast<uint64_t*>(tiles + S);
  uint64_t* empty = full + S;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ntiles = maps.first[3];
  const int par = SW::STATE || sizeof(R) == 8 ? cur_buf(P) : 0;
  // the feeder: tile t into slot q
  auto issue = [&](int q, int t) {
    const int g = (t >= maps.first[1]) + (t >= maps.first[2]), r = t - maps.first[g];
    R* slot = slots + (size_t)q * SW::ELEMS;
    uint64_t* bar = &full[q];
    auto go = [&](auto stage, auto d) {
      using St = decltype(stage);
      constexpr int D = decltype(d)::value;
      if constexpr (!(SW::MASK >> D & 1)) return;
      const Tile T = St::place(P, maps.m[D], r);
      tiles[q] = T;
      mbar_arrive_expect_tx(bar, St::BYTES);
      St::issue(P, maps.m[D], par, T, slot, bar);
    };
    const int D = maps.order[g];
    if (SW::H0 && (SW::MASK == 1 || D == 0)) go(S0{}, std::integral_constant<int, 0>{});
    else if (SW::H1 && (SW::MASK == 2 || D == 1)) go(S1{}, std::integral_constant<int, 1>{});
    else go(S2{}, std::integral_constant<int, 2>{});
  };
  // the two counters of S_TILE: tiles handed out beyond the first of each
  // block, blocks done
  unsigned* counters = reinterpret_cast<unsigned*>(P.scal + S_TILE);
  const bool feeder = threadIdx.x == 0;
  int next = blockIdx.x;  // feeder only: the next tile to issue
  // After a pipeline wait that timed out (flag 2, which another block may be
  // setting now) there is no work.  The feeder looks for all of the block: the
  // ring is set up and carries the end at once, so that no thread reads a tile or
  // waits at a barrier that nobody has written, and the block counts itself like
  // the others, so that the counters end at zero.
  if (feeder && P.scal[S_FLAGS] == 2.0) next = ntiles;
  int issued = 0;         // feeder only: tiles whose copies were issued
  bool more = true;       // feeder only: the end has not been passed on
  // the feeder: the next tile into slot q, or the end of the work
  auto feed = [&](int q) {
    if (next < ntiles) {
      const int t = next;
      next = gridDim.x + (int)atomicAdd(counters, 1u);  // used a tile later
      issue(q, t);
      issued++;
    } else {
      tiles[q].D = -1;
      mbar_arrive(&full[q]);
      more = false;
    }
  };
  if (feeder) {
    for (int q = 0; q < S; q++) {
      mbar_init(&full[q], 1);
      mbar_init(&empty[q], kWarps);
    }
    fence_mbar_init();
    for (int q = 0; q < S && more; q++) feed(q);
  }
  __syncthreads();
  bool ok = true;
  int q = 0;
  uint32_t ph = 0;
  for (;;) {
    if (!mbar_wait(&full[q], ph)) {
      ok = false;
      break;
    }
    const Tile T = tiles[q];
    if (T.D < 0) break;
    const R* slot = slots + (size_t)q * SW::ELEMS;
    auto rows = [&](auto stage) {
      using St = decltype(stage);
      int row = warp, col = lane;
#pragma unroll 1
      for (;;) {
        St::point(P, wk, slot, T, row, col, gather);
        if (St::ROWS > kWarps && col < 32 && row + kWarps < St::ROWS) {
          row += kWarps;
          continue;
        }
        // the row-end pass: column 32 of the tile's rows
        if (warp != T.end_warp || col == 32 || lane >= St::ROWS) break;
        row = lane;
        col = 32;
      }
    };
    if constexpr (SW::MASK == 1) rows(S0{});
    else if constexpr (SW::MASK == 2) rows(S1{});
    else if constexpr (SW::MASK == 4) rows(S2{});
    else {
      if (SW::H0 && T.D == 0) rows(S0{});
      else if (T.D == 1) rows(S1{});
      else rows(S2{});
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[q]);
    if (feeder && more) {
      // every warp has released this slot: refill it
      if (!mbar_wait(&empty[q], ph)) {
        ok = false;
        break;
      }
      feed(q);
    }
    if (++q == S) {
      q = 0;
      ph ^= 1;
    }
  }
  if (feeder) {
    // A block that gave up lets the copies of the tiles issued last land
    // before it exits (at the end of the work all have been waited for; the
    // slot that carries the end had been released)
    if (!ok) {
      const int k0 = issued - S + (more ? 0 : 1);
      for (int k = k0 > 0 ? k0 : 0; k < issued; k++) mbar_wait(&full[k % S], (k / S) & 1);
    }
    // the last block leaves the counters at zero for the next launch
    if (atomicAdd(counters + 1, 1u) == gridDim.x - 1) {
      counters[0] = 0;
      counters[1] = 0;
    }
  }
  if (!ok) P.scal[S_FLAGS] = 2.0;
}

template <typename R, bool EMF, bool BG, unsigned MASK, bool POLE>
__global__ void __launch_bounds__(kSweepThreads, (SweepCfg<R, EMF>::CTAS))
    k_sweep(Params P, Work<R> wk,
            const __grid_constant__ SweepMaps<typename Sweep<R, EMF, BG, MASK, POLE>::Maps> maps) {
  pdl_enter();
  Gather none;
  sweep_run<Sweep<R, EMF, BG, MASK, POLE>, R>(P, wk, maps, none);
}

// ---------------------------------------------------------------- update

// The update (Cartesian, or as update_sph) from tiles of 32 x 4 x 2 cells (a warp per row along
// i): everything a cell reads -- 24 face fluxes with their upper neighbours, 12
// edge EMFs, 6 face and 5 state values, the axes' tables (beside 220 KB of slots
// the L1 keeps little) -- comes by the tile's 16 copies.  The
// per-cell kernel waits for its 71 loads a few at a time (long-scoreboard
// stalls 5.6 per instruction, 4.5 TB/s at 256^3 FP64).
template <typename R, int COORD>
struct UpdTile {
  // the faces along each axis, the edges along each axis
  __host__ __device__ static constexpr Box F(int d) {
    return d == 0 ? Box{36, 4, 2, 1} : (d == 1 ? Box{32, 5, 2, 1} : Box{32, 4, 3, 1});
  }
  __host__ __device__ static constexpr Box E(int d) {
    return d == 0 ? Box{32, 5, 3, 1} : (d == 1 ? Box{36, 4, 3, 1} : Box{36, 5, 2, 1});
  }
  static constexpr Box W{32, 4, 2, 5};
  __host__ __device__ static constexpr int up(int bytes) { return (bytes + 127) / 128 * 128; }
  static constexpr int RS = sizeof(R);
  // byte offsets in the slot: the 5 hydro and the 3 stress fluxes of each
  // axis, the EMFs, the face field (FP64), the state (FP64)
  __host__ __device__ static constexpr int f(int d) {
    int o = 0;
    for (int a = 0; a < d; a++) o += up(5 * F(a).elems() * RS) + up(3 * F(a).elems() * RS);
    return o;
  }
  __host__ __device__ static constexpr int g(int d) { return f(d) + up(5 * F(d).elems() * RS); }
  __host__ __device__ static constexpr int e(int d) {
    int o = f(3);
    for (int a = 0; a < d; a++) o += up(E(a).elems() * RS);
    return o;
  }
  __host__ __device__ static constexpr int b(int d) {
    int o = e(3);
    for (int a = 0; a < d; a++) o += up(F(a).elems() * 8);
    return o;
  }
  __host__ __device__ static constexpr int w() { return b(3); }
  // the axes' tables at the tile's columns, rows and planes (spherical: and
  // the next ones): 1 / dx and the centring weights of a Cartesian grid, all
  // but the reconstruction's of a spherical one (two groups of rows)
  static constexpr int T0 = COORD == 0 ? T_IDX : T_X, TN = T_MB + 1 - T0;
  static constexpr int TG = COORD == 0 ? 0 : NTAB - T_G0;
  __host__ __device__ static constexpr int tw(int d) {
    return COORD == 0 ? (d == 0 ? 32 : (d == 1 ? 4 : 2)) : (d == 0 ? 36 : (d == 1 ? 6 : 2));
  }
  __host__ __device__ static constexpr int t(int d) {
    int o = w() + up(W.elems() * 8);
    for (int a = 0; a < d; a++) o += up(tw(a) * TN * 8) + up(tw(a) * TG * 8);
    return o;
  }
  __host__ __device__ static constexpr int tg(int d) { return t(d) + up(tw(d) * TN * 8); }
  static constexpr int SLOT = t(3);
  static constexpr int BYTES = 8 * (F(0).elems() + F(1).elems() + F(2).elems()) * (RS + 1) +
                               (E(0).elems() + E(1).elems() + E(2).elems()) * RS + W.elems() * 8 +
                               (tw(0) + tw(1) + tw(2)) * (TN + TG) * 8;
};

struct alignas(64) UpdMaps {
  CUtensorMap f[3], g[3];  // fluxes along each axis: hydro, stress
  CUtensorMap e[3];        // EMFs
  CUtensorMap b[3][2];     // step-start face field, of either parity
  CUtensorMap w[2];        // step-start state
  CUtensorMap t[3], g2[3]; // tables: T0.., T_G0..
  int nt[3];
  uint64_t inv[2];
};

// the reader of update_cart and update_sph on a slot: column c, row (jj, kk) of the tile
template <typename R, int COORD>
struct TileReader {
  using U = UpdTile<R, COORD>;
  const unsigned char* s;
  int c, jj, kk;
  template <typename T>
  __device__ __forceinline__ T at(int off, int idx) const {
    return reinterpret_cast<const T*>(s + off)[idx];
  }
  __device__ __forceinline__ int face_at(int d, int u) const {
    return d == 0 ? (kk * 4 + jj) * 36 + c + u
                  : (d == 1 ? (kk * 5 + jj + u) * 32 + c : ((kk + u) * 4 + jj) * 32 + c);
  }
  __device__ __forceinline__ R flux(int d, int m, int u) const {
    constexpr int f[3] = {U::f(0), U::f(1), U::f(2)}, g[3] = {U::g(0), U::g(1), U::g(2)};
    constexpr int n[3] = {U::F(0).elems(), U::F(1).elems(), U::F(2).elems()};
    return m < 5 ? at<R>(f[d], m * n[d] + face_at(d, u)) : at<R>(g[d], (m - 6) * n[d] + face_at(d, u));
  }
  __device__ __forceinline__ double emf(int a, int di, int dj, int dk) const {
    constexpr int e[3] = {U::e(0), U::e(1), U::e(2)};
    const int idx = a == 0 ? ((kk + dk) * 5 + jj + dj) * 32 + c
                           : (a == 1 ? ((kk + dk) * 4 + jj) * 36 + c + di : (kk * 5 + jj + dj) * 36 + c + di);
    return (double)at<R>(e[a], idx);
  }
  __device__ __forceinline__ double face(int a, int u) const {
    constexpr int b[3] = {U::b(0), U::b(1), U::b(2)};
    return at<double>(b[a], face_at(a, u));
  }
  __device__ __forceinline__ double state(int m) const {
    return at<double>(U::w(), ((m * 2 + kk) * 4 + jj) * 32 + c);
  }
  __device__ __forceinline__ double tab(int a, int t, int up = 0) const {
    constexpr int o[3] = {U::t(0), U::t(1), U::t(2)}, g[3] = {U::tg(0), U::tg(1), U::tg(2)};
    const int x = (a == 0 ? c : (a == 1 ? jj : kk)) + up;
    return t <= T_MB ? at<double>(o[a], (t - U::T0) * U::tw(a) + x) : at<double>(g[a], (t - T_G0) * U::tw(a) + x);
  }
};

template <typename R, bool BG, int COORD>
struct UpdStage {
  using U = UpdTile<R, COORD>;
  using Maps = UpdMaps;
  static constexpr int ELEMS = U::SLOT / (int)sizeof(R), ROWS = kWarps, BYTES = U::BYTES;
  __device__ static Tile place(const Params& P, const Maps& m, int r) {
    const int3 d = tile_digits(m, r);
    return Tile{0, -1, NGH + 32 * d.x, NGH + 4 * d.y, NGH + 2 * d.z};
  }
  __device__ static void issue(const Params& P, const Maps& m, int par, const Tile& T, R* slot,
                               uint64_t* bar) {
    unsigned char* s = reinterpret_cast<unsigned char*>(slot);
    const int x = T.x0, y = T.y0, z = T.z0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      tma_load_4d(s + U::f(d), &m.f[d], bar, x, y, z, 9 * d);
      tma_load_4d(s + U::g(d), &m.g[d], bar, x, y, z, 9 * d + 6);
      tma_load_4d(s + U::e(d), &m.e[d], bar, x, y, z, d);
      tma_load_4d(s + U::b(d), &m.b[d][par], bar, x, y, z, d);
      const int at = d == 0 ? x : (d == 1 ? y : z);
      tma_load_4d(s + U::t(d), &m.t[d], bar, at, U::T0, d, 0);
      if constexpr (COORD != 0) tma_load_4d(s + U::tg(d), &m.g2[d], bar, at, T_G0, d, 0);
    }
    tma_load_4d(s + U::w(), &m.w[par], bar, x, y, z, 0);
  }
  __device__ __forceinline__ static void point(const Params& P, const Work<R>& wk, const R* slot,
                                               const Tile& T, int row, int col, Gather& out) {
    const int jj = row & 3, kk = row >> 2;
    const int i = T.x0 + col, j = T.y0 + jj, k = T.z0 + kk;
    if (!(i < NGH + P.n[0] && j < NGH + P.n[1] && k < NGH + P.n[2])) return;
    double rate, divb;
    const TileReader<R, COORD> in{reinterpret_cast<const unsigned char*>(slot), col, jj, kk};
    if constexpr (COORD == 0) update_cart<R, BG, false>(P, in, i, j, k, rate, divb);
    else update_sph<BG, false>(P, wk, in, i, j, k, rate, divb);
    out.rate = fmax(out.rate, rate);
    out.divb = fmax(out.divb, divb);
  }
};

// Two slots, as many blocks per SM as then fit: one in FP64 (90 KB a slot, 8
// warps of up to 255 registers), two in FP32.  What bounds it is that the
// copies run ahead: with one slot a block loads and computes in turn.  Blast
// 256^3 on B200, us a launch: FP64 one slot and two blocks 1256, two slots and
// one block 1108 (per cell 1275); FP32 one slot and three or four blocks 930,
// 1055, two slots and two blocks 886 (per cell 983).  The tables in the slot
// instead of the little L1 beside it: 1089 and 752.
template <typename R, bool BG, int COORD>
struct UpdSweep {
  static constexpr bool EMF = false, STATE = true;
  static constexpr unsigned MASK = 1;
  static constexpr bool H0 = true, H1 = false, H2 = false;
  template <int D>
  using Stage = UpdStage<R, BG, COORD>;
  using Maps = UpdMaps;
  static constexpr int ELEMS = Stage<0>::ELEMS, SLOT = UpdTile<R, COORD>::SLOT;
  static constexpr int CTAS = sizeof(R) == 8 ? 1 : 2, S = 2;
  static constexpr int SMEM = S * SLOT + S * (2 * 8 + (int)sizeof(Tile)) + 128;
  static_assert((SMEM + 1024) * CTAS <= 228 * 1024, "update blocks per SM");
};

template <typename R, bool BG, int COORD>
__global__ void __launch_bounds__(kSweepThreads, (UpdSweep<R, BG, COORD>::CTAS))
    k_update_sweep(Params P, Work<R> wk, const __grid_constant__ SweepMaps<UpdMaps> maps) {
  pdl_enter();
  if (stopped(P)) return;
  Gather g;
  sweep_run<UpdSweep<R, BG, COORD>, R>(P, wk, maps, g);
  using RC = typename std::conditional<COORD == 0 && GOP_MX_CFL64, double, R>::type;
  block_commit<RC>(P, g.rate, g.divb);
}

template <typename R, unsigned MASK>
constexpr bool smem_fits() {
  using F = Sweep<R, false, false, MASK, false>;
  using E = Sweep<R, true, false, MASK, false>;
  return (F::SMEM + 1024) * F::CTAS <= 228 * 1024 && (E::SMEM + 1024) * E::CTAS <= 228 * 1024;
}
static_assert(smem_fits<double, 7>() && smem_fits<double, 1>(), "FP64 sweep blocks per SM");
static_assert(smem_fits<float, 7>() && smem_fits<float, 1>(), "FP32 sweep blocks per SM");

// ------------------------------------------------------------------ host

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  });
  return fn;
}

// a 4-D map over a dense array of dims d[0..3] (elements, d[0] fastest;
// strides in bytes), read in boxes b
template <typename R>
static bool encode(CUtensorMap* m, const R* base, const cuuint64_t d[4], const cuuint64_t st[3],
                   const Box& b) {
  EncodeTiledFn fn = encode_fn();
  if (!fn || !base) return false;
  const cuuint32_t bx[4] = {(cuuint32_t)b.x, (cuuint32_t)b.y, (cuuint32_t)b.z, (cuuint32_t)b.f};
  const cuuint32_t el[4] = {1, 1, 1, 1};
  const CUresult r =
      fn(m, sizeof(R) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4,
         const_cast<R*>(base), d, st, bx, el, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
         CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

// nf fields of one array in the state's layout (i, j, k, field)
template <typename R>
static bool field_map(CUtensorMap* m, const R* base, int nf, const Params& P, const Box& b) {
  const cuuint64_t es = sizeof(R);
  const cuuint64_t d[4] = {(cuuint64_t)P.N[0], (cuuint64_t)P.N[1], (cuuint64_t)P.N[2], (cuuint64_t)nf};
  const cuuint64_t st[3] = {(cuuint64_t)P.pitch * es, (cuuint64_t)P.sk * es, (cuuint64_t)P.fs * es};
  return encode<R>(m, base, d, st, b);
}

// PDM weights: the per-axis tables [axis][NTAB][tmax] for tap-major boxes,
// the packed face records [axis * tmax + f][FW] otherwise
template <typename R>
static bool weight_map(CUtensorMap* m, const Work<R>& w, const Params& P, const Box& b) {
  const cuuint64_t es = sizeof(R), tm = (cuuint64_t)P.tmax;
  if (b.y == kTap40.y && b.x == kTap40.x) {
    const cuuint64_t d[4] = {tm, (cuuint64_t)NTAB, 3, 1};
    const cuuint64_t st[3] = {tm * es, tm * NTAB * es, tm * NTAB * 3 * es};
    return encode<R>(m, w.tab, d, st, b);
  }
  const cuuint64_t d[4] = {(cuuint64_t)FW, 3 * tm, 1, 1};
  const cuuint64_t st[3] = {FW * es, FW * 3 * tm * es, FW * 3 * tm * es};
  return encode<R>(m, w.fw, d, st, b);
}

// the limiters' step-start references: FP64 the state buffer of parity b,
// FP32 its copy (the same for both parities)
template <typename R>
static const R* lim_state(const Params& P, const Work<R>& w, int b) {
  return sizeof(R) == 8 ? reinterpret_cast<const R*>(P.Wbuf[b]) : w.Wl;
}
template <typename R>
static const R* lim_face(const Params& P, const Work<R>& w, int b) {
  return sizeof(R) == 8 ? reinterpret_cast<const R*>(P.Bbuf[b]) : w.Bl;
}

template <typename R, int D>
static bool make_flux_maps(FluxMaps& m, const Params& P, const Work<R>& w) {
  using F = FluxTile<D>;
  const Box S5{F::S.x, F::S.y, F::S.z, F::NG}, L5{F::L.x, F::L.y, F::L.z, F::NG};
  const Box S3{F::S.x, F::S.y, F::S.z, 3}, L3{F::L.x, F::L.y, F::L.z, 3};
  bool ok = field_map<R>(&m.wh, w.Wh, 6, P, S5) && field_map<R>(&m.msh, w.Msh, 3, P, S3) &&
            field_map<R>(&m.ms, w.Ms, 3, P, L3) && weight_map<R>(&m.wt, w, P, F::WT);
  for (int b = 0; b < 2 && ok; b++)
    ok = field_map<R>(&m.wl[b], lim_state<R>(P, w, b), 6, P, L5) &&
         field_map<R>(&m.bn[b], lim_face<R>(P, w, b), 3, P, F::BN);
  const int n0 = P.n[0], n1 = P.n[1], n2 = P.n[2];
  if (D == 0) {  // i-face tiles (the row-end face in the last), j-row tiles, k planes
    m.nt[0] = (n0 + 31) / 32;
    m.nt[1] = (n1 + 7) / 8;
    m.nt[2] = n2;
  } else if (D == 1) {  // i tiles, j-face tiles, k planes
    m.nt[0] = (n0 + 31) / 32;
    m.nt[1] = (n1 + 1 + 7) / 8;
    m.nt[2] = n2;
  } else {  // i tiles, k-face tiles, j rows
    m.nt[0] = (n0 + 31) / 32;
    m.nt[1] = (n2 + 1 + 7) / 8;
    m.nt[2] = n1;
  }
  for (int a = 0; a < 2; a++) m.inv[a] = inverse_of(m.nt[a]);
  return ok;
}

template <typename R, int D>
static bool make_emf_maps(EmfMaps& m, const Params& P, const Work<R>& w) {
  using E = EmfTile<D>;
  bool ok = field_map<R>(&m.v, w.V, 6, P, E::V) && field_map<R>(&m.bhp, w.Bh, 3, P, E::BHP) &&
            field_map<R>(&m.bhq, w.Bh, 3, P, E::BHQ) && field_map<R>(&m.rho, w.Wh, 6, P, E::RHO) &&
            weight_map<R>(&m.wq, w, P, E::WQ) && weight_map<R>(&m.wp, w, P, E::WP);
  for (int b = 0; b < 2 && ok; b++)
    ok = field_map<R>(&m.blp[b], lim_face<R>(P, w, b), 3, P, E::BLP) &&
         field_map<R>(&m.blq[b], lim_face<R>(P, w, b), 3, P, E::BLQ);
  const int n0 = P.n[0], n1 = P.n[1], n2 = P.n[2];
  if (D == 0) {  // i-cell tiles, k-face tiles, j faces
    m.nt[0] = (n0 + 31) / 32;
    m.nt[1] = (n2 + E::ROWS) / E::ROWS;
    m.nt[2] = n1 + 1;
  } else if (D == 1) {  // i-face tiles (the row-end face in the last), k-face tiles, j cells
    m.nt[0] = (n0 + 31) / 32;
    m.nt[1] = (n2 + E::ROWS) / E::ROWS;
    m.nt[2] = n1;
  } else {  // i-face tiles (the row-end face in the last), j-face tiles, k cells
    m.nt[0] = (n0 + 31) / 32;
    m.nt[1] = (n1 + E::ROWS) / E::ROWS;
    m.nt[2] = n2;
  }
  for (int a = 0; a < 2; a++) m.inv[a] = inverse_of(m.nt[a]);
  return ok;
}

template <typename R, int COORD>
static bool make_upd_maps(UpdMaps& m, const Params& P, const Work<R>& w) {
  using U = UpdTile<R, COORD>;
  bool ok = true;
  for (int d = 0; d < 3 && ok; d++) {
    Box f = U::F(d), g = U::F(d);
    f.f = 5;
    g.f = 3;
    ok = field_map<R>(&m.f[d], w.F, 27, P, f) && field_map<R>(&m.g[d], w.F, 27, P, g) &&
         field_map<R>(&m.e[d], w.E, 3, P, U::E(d));
    const cuuint64_t tm = (cuuint64_t)P.tmax, td[4] = {tm, (cuuint64_t)NTAB, 3, 1};
    const cuuint64_t ts[3] = {tm * 8, tm * NTAB * 8, tm * NTAB * 3 * 8};
    ok = ok && encode<double>(&m.t[d], P.tab, td, ts, Box{U::tw(d), U::TN, 1, 1});
    if constexpr (COORD != 0) ok = ok && encode<double>(&m.g2[d], P.tab, td, ts, Box{U::tw(d), U::TG, 1, 1});
    for (int b = 0; b < 2 && ok; b++) ok = field_map<double>(&m.b[d][b], P.Bbuf[b], 3, P, U::F(d));
  }
  for (int b = 0; b < 2 && ok; b++) ok = field_map<double>(&m.w[b], P.Wbuf[b], 6, P, U::W);
  m.nt[0] = (P.n[0] + 31) / 32;
  m.nt[1] = (P.n[1] + 3) / 4;
  m.nt[2] = (P.n[2] + 1) / 2;
  for (int a = 0; a < 2; a++) m.inv[a] = inverse_of(m.nt[a]);
  return ok;
}

struct SweepSet {
  SweepMaps<FluxMaps> flux;
  SweepMaps<EmfMaps> emf;
  SweepMaps<UpdMaps> upd;
  int sms = 0;
};

// the kernels that may have a face on a pole to look at
template <typename R, unsigned MASK>
constexpr bool kPole = sizeof(R) == 8 && (MASK >> 1 & 1);
template <typename R, bool EMF, bool BG, unsigned MASK>
static bool allow_smem() {
  constexpr bool pole = kPole<R, MASK>;
  return cudaFuncSetAttribute(k_sweep<R, EMF, BG, MASK, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              Sweep<R, EMF, BG, MASK, false>::SMEM) == cudaSuccess &&
         (!pole || cudaFuncSetAttribute(k_sweep<R, EMF, BG, MASK, pole>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        Sweep<R, EMF, BG, MASK, pole>::SMEM) == cudaSuccess);
}
template <typename R, bool BG>
static bool allow_smem() {
  return allow_smem<R, false, BG, 1>() && allow_smem<R, false, BG, 2>() && allow_smem<R, false, BG, 4>() &&
         allow_smem<R, false, BG, 7>() && allow_smem<R, true, BG, 7>() &&
         cudaFuncSetAttribute(k_update_sweep<R, BG, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              UpdSweep<R, BG, 0>::SMEM) == cudaSuccess &&
         (sizeof(R) == 4 ||
          cudaFuncSetAttribute(k_update_sweep<double, BG, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               UpdSweep<double, BG, 2>::SMEM) == cudaSuccess);
}

template <typename R>
SweepSet* sweep_create(const Params& P, const Work<R>& w) {
  SweepSet* s = new (std::nothrow) SweepSet();
  if (!s) return nullptr;
  int dev = 0;
  bool ok = cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&s->sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
  ok = ok && make_flux_maps<R, 0>(s->flux.m[0], P, w) && make_flux_maps<R, 1>(s->flux.m[1], P, w) &&
       make_flux_maps<R, 2>(s->flux.m[2], P, w) && make_emf_maps<R, 0>(s->emf.m[0], P, w) &&
       make_emf_maps<R, 1>(s->emf.m[1], P, w) && make_emf_maps<R, 2>(s->emf.m[2], P, w);
  ok = ok && (P.coord == 0 ? make_upd_maps<R, 0>(s->upd.m[0], P, w) : make_upd_maps<R, 2>(s->upd.m[0], P, w)) &&
       allow_smem<R, false>() && allow_smem<R, true>();
  if (!ok) {
    cudaGetLastError();
    delete s;
    return nullptr;
  }
  return s;
}
template SweepSet* sweep_create<double>(const Params&, const Work<double>&);
template SweepSet* sweep_create<float>(const Params&, const Work<float>&);

void sweep_destroy(SweepSet* s) { delete s; }

// the tiles of the axes SW is compiled for, in the given order
template <class SW, typename R, class K>
static void launch_persistent(K kern, const SweepSet* sw, const Params& P, const Work<R>& w,
                              SweepMaps<typename SW::Maps> m, const int order[3], cudaStream_t st) {
  m.first[0] = 0;
  for (int g = 0; g < 3; g++) {
    const int D = m.order[g] = order[g], *nt = m.m[D].nt;
    m.first[g + 1] = m.first[g] + (SW::MASK >> D & 1 ? nt[0] * nt[1] * nt[2] : 0);
  }
  const int grid = std::min(m.first[3], sw->sms * SW::CTAS);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kSweepThreads);
  cfg.dynamicSmemBytes = SW::SMEM;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = GOP_SWEEP_PDL ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kern, P, w, m);
  count_launches(1);
}

template <typename R, bool EMF, bool BG, unsigned MASK, class Maps>
static void launch_mask(const SweepSet* sw, const Params& P, const Work<R>& w, const Maps& m,
                        const int order[3], cudaStream_t st) {
  constexpr bool pole = kPole<R, MASK>;
  if (pole && P.ring)
    launch_persistent<Sweep<R, EMF, BG, MASK, pole>, R>(k_sweep<R, EMF, BG, MASK, pole>, sw, P, w, m, order, st);
  else
    launch_persistent<Sweep<R, EMF, BG, MASK, false>, R>(k_sweep<R, EMF, BG, MASK, false>, sw, P, w, m, order, st);
}
// The axes of a stage in one launch, or (flux) one launch each where each
// axis alone keeps the GPU busy for long: the kernels of one axis are about 3 %
// faster per tile (a third of the code, registers left over), which beats the
// two waves and fills saved from about 128 tiles per resident block on.  Blast
// on B200, flux stage per step, one launch / three: FP64 128^3 321 / 335 us,
// 192^3 1048 / 1022, 256^3 2443 / 2350; FP32 216 / 226, 693 / 681, 1616 / 1560.
// EMF tiles are shorter and gain by the common launch at every size (FP32
// 128^3 120 / 137, 256^3 854 / 851).
constexpr int kTilesApart = 128;
template <typename R, bool EMF, bool BG, class Maps>
static void launch_axes(const SweepSet* sw, const Params& P, const Work<R>& w, const Maps& m,
                        const int order[3], cudaStream_t st) {
  if constexpr (!EMF) {
    long long tiles = 0;
    for (int d = 0; d < 3; d++) tiles += (long long)m.m[d].nt[0] * m.m[d].nt[1] * m.m[d].nt[2];
    if (tiles >= (long long)kTilesApart * sw->sms * SweepCfg<R, false>::CTAS) {
      for (int g = 0; g < 3; g++) {
        if (order[g] == 0) launch_mask<R, EMF, BG, 1>(sw, P, w, m, order, st);
        else if (order[g] == 1) launch_mask<R, EMF, BG, 2>(sw, P, w, m, order, st);
        else launch_mask<R, EMF, BG, 4>(sw, P, w, m, order, st);
      }
      return;
    }
  }
  launch_mask<R, EMF, BG, 7>(sw, P, w, m, order, st);
}

template <typename R>
bool launch_flux_sweep(const SweepSet* sw, const Params& P, const Work<R>& w, const int order[3],
                       cudaStream_t st) {
  if (!sw || P.ps_live) return false;  // the entropy channel runs the per-face kernels
  if (P.bg) launch_axes<R, false, true>(sw, P, w, sw->flux, order, st);
  else launch_axes<R, false, false>(sw, P, w, sw->flux, order, st);
  return true;
}
template <typename R>
bool launch_emf_sweep(const SweepSet* sw, const Params& P, const Work<R>& w, const int order[3],
                      cudaStream_t st) {
  if (!sw) return false;
  if (P.bg) launch_axes<R, true, true>(sw, P, w, sw->emf, order, st);
  else launch_axes<R, true, false>(sw, P, w, sw->emf, order, st);
  return true;
}
// Tiles a block needs: with fewer its ring is hardly filled before it ends and
// the per-cell kernel is as fast or faster (B200, us, tiles / per cell.  FP64, by
// tiles a block: 2.7 (blast 77x45x21) 16.9 / 15.2, 3.2 23.0 / 20.7, 6.9 (64^3) 27.5
// / 31, 55 (128^3) 144 / 171; FP32: 1.7 15.0 / 15.2, 3.5 (64^3) 27.2 / 29.1,
// (Orszag-Tang 256x256x4) 23.7 / 26.7, 28 105 / 134).
template <typename R>
constexpr int upd_tiles() {
  return sizeof(R) == 8 ? 6 : 3;
}
template <typename R, bool BG, int COORD>
static void launch_update_c(const SweepSet* sw, const Params& P, const Work<R>& w, cudaStream_t st) {
  static const int order[3] = {0, 1, 2};
  launch_persistent<UpdSweep<R, BG, COORD>, R>(k_update_sweep<R, BG, COORD>, sw, P, w, sw->upd, order, st);
}
template <typename R>
bool update_sweep_applies(const SweepSet* sw, const Params& P) {
  if (!sw || P.ps_live || P.ring || (P.coord != 0 && sizeof(R) == 4)) return false;
  const int* nt = sw->upd.m[0].nt;
  return (long long)nt[0] * nt[1] * nt[2] >= (long long)upd_tiles<R>() * sw->sms * UpdSweep<R, false, 0>::CTAS;
}
template <typename R>
bool launch_update_sweep(const SweepSet* sw, const Params& P, const Work<R>& w, cudaStream_t st) {
  if (!update_sweep_applies<R>(sw, P)) return false;
  const bool bg = P.bg != nullptr;
  if (P.coord == 0) bg ? launch_update_c<R, true, 0>(sw, P, w, st) : launch_update_c<R, false, 0>(sw, P, w, st);
  else if constexpr (sizeof(R) == 8)
    bg ? launch_update_c<R, true, 2>(sw, P, w, st) : launch_update_c<R, false, 2>(sw, P, w, st);
  return true;
}
#define GOP_INST(R)                                                                            \
  template bool update_sweep_applies<R>(const SweepSet*, const Params&);                        \
  template bool launch_update_sweep<R>(const SweepSet*, const Params&, const Work<R>&, cudaStream_t); \
  template bool launch_flux_sweep<R>(const SweepSet*, const Params&, const Work<R>&,            \
                                     const int[3], cudaStream_t);                     \
  template bool launch_emf_sweep<R>(const SweepSet*, const Params&, const Work<R>&,             \
                                    const int[3], cudaStream_t);
GOP_INST(double)
GOP_INST(float)
#undef GOP_INST

}  // namespace gop
