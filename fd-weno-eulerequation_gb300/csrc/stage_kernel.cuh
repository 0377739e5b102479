// One RK stage of the WENO-FD hot path as a single fused tile kernel:
// halo load, x sweep (flux split, characteristic WENO faces), y sweep, flux
// differences, source term and the RK combination, with nothing but the
// state in global memory.
//
// Replaces, per stage: assembleRHS (src/WENOFD.cpp:454-465) with
// assembleBoundaryTerm's x sweep (513-649) and y sweep (652-797),
// assembleSourceTerm (800-821), and the stage update of RunRK1/2/3
// (301-396).  The boundary fill runs before it (k_bc_fill).
//
// Tile: TI nodes in x by TJ = 32 nodes in y (y is the contiguous axis, so a
// warp spans one tile row).  The block stages the state of the tile plus a
// 3-node halo in shared memory, computes the split fluxes of every node the
// tile's faces need once, then the (TI+1) x TJ x-faces and TI x (TJ+1)
// y-faces, and keeps the per-node x term in registers between the sweeps.
// Shared-memory regions for the split fluxes and face fluxes are reused by
// the y sweep.
//
// This file holds the FP64 tile (bitwise the reference) and the kernel and
// launcher shared by both precisions; the FP32 tile (FP32 form and learned
// form) is stage_f32.cuh.
#pragma once

#include "convert.cuh"
#include "physics.cuh"
#include "stage_f32.cuh"

namespace wenofd {
namespace dev {

// Shared memory of the FP64 tile, structure of arrays [component][row][col].
// The state tile's rows are kBoxJ = 40 doubles wide, halo node hj at column
// hj + 1: the TMA box of the per-solve kernel (40 columns from the even,
// 16-byte aligned column before the halo, TI + 6 rows, 4 planes) lands in
// place, with no copy; the batched kernel's per-thread loads use the same
// layout.
template <int TI, int TJ>
struct StageSmem {
  static constexpr int HI = TI + 6, HJ = TJ + 6;
  static constexpr int kBoxJ = 40;
  static_assert(HJ + 2 <= kBoxJ, "box width");
  static constexpr int kU = 4 * HI * kBoxJ;                                 // state + halo
  static constexpr unsigned kBoxBytes = unsigned(kU) * 8u;
  static constexpr int kSplit = 4 * (HI * TJ > TI * HJ ? HI * TJ : TI * HJ);  // one of F+, F-
  static constexpr int kFace = 4 * ((TI + 1) * TJ > TI * (TJ + 1) ? (TI + 1) * TJ : TI * (TJ + 1));
  // 128 bytes of slack: the base is rounded up to 128 bytes (TMA destination)
  static constexpr size_t bytes = 128 + sizeof(double) * (size_t(kU) + 2 * kSplit + kFace);
  // index of state component r at halo node (hi, hj)
  static __device__ __forceinline__ int u(int r, int hi, int hj) { return (r * HI + hi) * kBoxJ + hj + 1; }
};

// One FP64 tile (TI x TJ interior nodes starting at i0, j0) of one RK stage,
// executed by all NT threads of a block; smem_raw holds StageSmem::bytes.
// Every operation follows the reference's evaluation order (the unit is
// compiled with -fmad=false).  Shared by the per-solve kernel k_stage and
// the persistent batched kernel.  COH: the tile's inputs may have been
// written earlier in the same kernel by other blocks (the persistent batched
// kernel): loads then go through L2 only (ld.global.cg) instead of the
// non-coherent read-only path.  TMA (the per-solve kernel): the halo box
// arrives by TMA through the map in `tma` (one thread issues it; a bounded
// wait, on give-up the block records the error in a.wait_error and leaves
// the tile); otherwise every thread loads nodes.  rows: nodes of the tile in
// x, at most TI; pair: two lanes per face (Fp64Split).
template <int SCHEME, int TI, int TJ, int NT, bool COH = false, bool TMA = false>
__device__ __forceinline__ void stage_tile_f64(const Geom &g, const StageArgs &a, const int i0, const int j0,
                                               const int rows, const bool pair, unsigned char *smem_raw,
                                               const StageTma *tma = nullptr) {
  using T = double;
  using S = StageSmem<TI, TJ>;
  constexpr int HI = S::HI, HJ = S::HJ;
  unsigned char *base = smem_raw + (((tma_smem_addr(smem_raw) + 127u) & ~127u) - tma_smem_addr(smem_raw));
  T *Us = reinterpret_cast<T *>(base);
  T *Fp = Us + S::kU;
  T *Fm = Fp + S::kSplit;
  T *Hf = Fm + S::kSplit;
  const T gamma = g.gamma, zpl = g.zp_lambda;

  // --- state tile with halo: nodes ei = 4+i0-3+hi, ej = 4+j0-3+hj.
  if constexpr (TMA) {
    // box column c = ghosted column j0 + c = halo node hj = c - 1; box row 0 =
    // ghosted row 1 + i0 (rows or columns past the array read as zero, like
    // the per-thread loads, and feed only faces that are not computed)
    __shared__ __align__(8) unsigned long long tma_bar;
    if (threadIdx.x == 0) tma_bar_init(tma_smem_addr(&tma_bar), 1);
    __syncthreads();
    if (threadIdx.x == 0) {
      const unsigned bar = tma_smem_addr(&tma_bar);
      tma_fence_proxy();
      tma_bar_expect(bar, S::kBoxBytes);
      // first coordinate x * 8 bytes a multiple of 16 (j0 is a multiple of
      // 32; an unissued copy leaves the wait below to give up)
      if (WENOFD_REQUIRE(g.guard, (j0 & 1) == 0, j0, 2)) tma_load_3d(tma_smem_addr(Us), &tma->u, j0, 1 + i0, 0, bar);
    }
    const bool ok = tma_bar_wait(tma_smem_addr(&tma_bar), 0, kTmaWaitLimit);
    if (__syncthreads_or(!ok)) {
      if (threadIdx.x == 0) {
        if (a.wait_error) atomicExch(a.wait_error, 1);
        tma_bar_wait(tma_smem_addr(&tma_bar), 0, kTmaWaitLimit);
      }
      __syncthreads();
      return;
    }
  } else {
    // All of a thread's loads are issued before any is used, so they are in
    // flight together.
    constexpr int NLD = (4 * HI * HJ + NT - 1) / NT;
    double v[NLD];
#pragma unroll
    for (int k = 0; k < NLD; ++k) {
      const int t = threadIdx.x + k * NT;
      const int r = t / (HI * HJ);
      const int rem = t - r * (HI * HJ);
      const int hi = rem / HJ, hj = rem - hi * HJ;
      const int ei = 1 + i0 + hi, ej = 1 + j0 + hj;
      const bool ok = t < 4 * HI * HJ && hi < rows + 6 && ei < g.nxt && ej < g.nyt;
      if constexpr (COH) v[k] = ok ? __ldcg(&a.uin[WENOFD_STATE(g, r * g.plane + WENOFD_GNODE(g, ei, ej))]) : 0.0;
      else v[k] = ok ? __ldg(&a.uin[WENOFD_STATE(g, r * g.plane + WENOFD_GNODE(g, ei, ej))]) : 0.0;
    }
#pragma unroll
    for (int k = 0; k < NLD; ++k) {
      const int t = threadIdx.x + k * NT;
      if (t < 4 * HI * HJ) {
        const int r = t / (HI * HJ);
        const int rem = t - r * (HI * HJ);
        const int hi = rem / HJ, hj = rem - hi * HJ;
        Us[WENOFD_IX(g.guard, S::u(r, hi, hj), S::kU)] = v[k];
      }
    }
  }
  __syncthreads();

  // --- the x sweep, then the y sweep, one body: most of it is integer
  // instructions (int_f64.cuh), and two copies would not fit the instruction
  // caches.
  // Bound: the FP64 pipe, with the integer pipes close behind.  At 1024^2
  // (WENO-Z, one stage): all arithmetic on the FP64 pipe 98.7 M warp
  // instructions on it and 6.11 ms; with fewer operations, still all there, 79.9
  // M and 4.95 ms; with products, quotients and roots on the integer pipes 33.0
  // M and 2.47 ms.  Counters at 2048^2, 9.39 ms: FP64 pipe at 84 % of the rate it
  // reaches, ALU pipe 58 %, FMA pipe 22 %, issue 50 %.  4096^2 SSP-RK3 step: 285 ->
  // 112 ms.
  constexpr int PPT = (TI * TJ + NT - 1) / NT;
  T rhs[PPT][4];
#pragma unroll
  for (int k = 0; k < PPT; ++k)
#pragma unroll
    for (int r = 0; r < 4; ++r) rhs[k][r] = T(0.0);
#pragma unroll 1
  for (int dir = 0; dir < 2; ++dir) {
    const bool xdir = dir == 0;
    // split fluxes: x, halo rows 0..rows+5 of the tile's columns; y, halo
    // columns 0..HJ-1 of the tile's rows
    const int sw = xdir ? TJ : HJ, scount = xdir ? (rows + 6) * TJ : rows * HJ;
    bool outside = false;  // a split flux outside the integer forms' range
    for (int t = threadIdx.x; t < scount; t += NT) {
      const int row = t / sw, col = t - row * sw;
      const int hi = xdir ? row : row + 3, hj = xdir ? col + 3 : col;
      T q[4], fm[4] = {0, 0, 0, 0}, fp[4] = {0, 0, 0, 0};
#pragma unroll
      for (int r = 0; r < 4; ++r) q[r] = Us[WENOFD_IX(g.guard, S::u(r, hi, hj), S::kU)];
      // (nodes past the array, which no face of the grid needs, stay zero)
      if (1 + i0 + hi < g.nxt && 1 + j0 + hj < g.nyt) outside = !flux_split_f64(dir, gamma, q, fm, fp) || outside;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        Fp[WENOFD_IX(g.guard, r * scount + t, S::kSplit)] = fp[r];
        Fm[WENOFD_IX(g.guard, r * scount + t, S::kSplit)] = fm[r];
      }
    }
    const bool plain = __syncthreads_or(outside);
    // faces: x, f = 0..rows between tile nodes f-1 and f (halo rows f+2, f+3);
    // y, f = 0..TJ of row i
    const int fw = xdir ? TJ : TJ + 1, fcount = xdir ? (rows + 1) * TJ : rows * (TJ + 1);
    const int ss = xdir ? TJ : 1;  // stencil nodes apart; components scount apart
    // pair: two lanes a face, whole warps (a lane without a face repeats the
    // tile's first and stores nothing)
    const int lanes = pair ? 2 : 1, work = pair ? (2 * fcount + 31) & ~31 : fcount;
    for (int w = threadIdx.x; w < work; w += NT) {
      int t = w / lanes;
      int row = t / fw, col = t - row * fw;
      // x: i0 + row is the face, j0 + col the node; y: the other way round
      const bool inside = t < fcount && i0 + row < g.nx + (xdir ? 1 : 0) && j0 + col < g.ny + (xdir ? 0 : 1);
      if (!inside) {
        if (!pair) continue;
        t = row = col = 0;
      }
      const int hi = xdir ? row + 2 : row + 3, hj = xdir ? col + 3 : col + 2;
      T um[4], u0[4], out[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        um[r] = Us[WENOFD_IX(g.guard, S::u(r, hi, hj), S::kU)];
        u0[r] = Us[WENOFD_IX(g.guard, S::u(r, xdir ? hi + 1 : hi, xdir ? hj : hj + 1), S::kU)];
      }
      const int s0 = row * sw + col;
      const T *fp = Fp + WENOFD_SPAN(g.guard, s0, s0 + 4 * ss + 3 * scount, S::kSplit);
      const T *fm = Fm + WENOFD_SPAN(g.guard, s0 + ss, s0 + 5 * ss + 3 * scount, S::kSplit);
      if (plain || !face_flux_f64<SCHEME>(dir, pair, gamma, zpl, um, u0, fp, fm, ss, scount, out)) {
        const Flux4 o = xdir ? face_flux_plain<0, SCHEME>(gamma, zpl, um[0], um[1], um[2], um[3], u0[0], u0[1], u0[2],
                                                          u0[3], fp, fm, ss, scount)
                             : face_flux_plain<1, SCHEME>(gamma, zpl, um[0], um[1], um[2], um[3], u0[0], u0[1], u0[2],
                                                          u0[3], fp, fm, ss, scount);
#pragma unroll
        for (int r = 0; r < 4; ++r) out[r] = o.v[r];
      }
      if (inside && w % lanes == 0) {
#pragma unroll
        for (int r = 0; r < 4; ++r) Hf[WENOFD_IX(g.guard, r * fcount + t, S::kFace)] = out[r];
      }
    }
    __syncthreads();
    // rhs = 0 + x term, then + y term (rhs zeroed in assembleRHS, += in the sweeps)
    const T h = xdir ? g.dx : g.dy;
    const IntDivisor by_h(h);
    const bool h_ok = in_range<-200, 200>(h);
#pragma unroll
    for (int k = 0; k < PPT; ++k) {
      const int t = threadIdx.x + k * NT;
      const int i = t / TJ, j = t - (t / TJ) * TJ;
      if (t < rows * TJ) {
        const int left = i * fw + j, right = xdir ? left + TJ : left + 1;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const T hr = Hf[WENOFD_IX(g.guard, r * fcount + right, S::kFace)],
                  hl = Hf[WENOFD_IX(g.guard, r * fcount + left, S::kFace)];
          const T d = -(hr - hl);
          rhs[k][r] = rhs[k][r] + (h_ok && in_range<-700, 300>(d) ? by_h.quotient(d) : tdiv(d, h));
        }
      }
    }
    __syncthreads();
  }

  // --- source, RK combination, store
  if constexpr (!COH) chain_release();
  const double dt = COH ? __ldcg(a.dt) : *a.dt;
#pragma unroll
  for (int k = 0; k < PPT; ++k) {
    const int t = threadIdx.x + k * NT;
    if (t >= rows * TJ) continue;
    const int i = t / TJ, j = t - i * TJ;
    if (i0 + i >= g.nx || j0 + j >= g.ny) continue;
    T rr[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) rr[r] = rhs[k][r];
    const long long gidx = WENOFD_NODE(g, i0 + i, j0 + j);
    if (g.gravity) {  // RTI, g = 1 (src/WENOFD.cpp:807-813)
      const T g_g0 = T(1.0);
      rr[3] += Us[WENOFD_IX(g.guard, S::u(2, i + 3, j + 3), S::kU)] * g_g0;
      rr[2] += Us[WENOFD_IX(g.guard, S::u(0, i + 3, j + 3), S::kU)] * g_g0;
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const long long ix = r * g.plane + gidx;
      if (a.mode == kModeRHS) {
        a.uout[ix] = rr[r];
      } else {
        const double un = COH ? __ldcg(&a.un[ix]) : a.un[ix], ui = COH ? __ldcg(&a.uin[ix]) : a.uin[ix];
        a.uout[ix] = a.a * un + a.b * ui + a.c * dt * rr[r];
      }
    }
  }
  if constexpr (COH) store_tile_ghosts<TJ, NT>(g, a, i0, j0, rows);
}

// Residency: the FP32 tiles read their FP64 inputs back in the epilogue
// instead of staging them, and ask for four (routed) or three resident
// 256-thread blocks per SM: the stage is issue-bound and latency-bound, and
// trading registers for resident warps pays.  The FP64 tile runs two blocks
// (shared memory's limit), so that one block's sums on the FP64 pipe overlap
// another's products on the integer pipes.
template <typename T, bool ROUTE, int NT>
__host__ __device__ constexpr int stage_blocks_per_sm() {
  if constexpr (sizeof(T) == 8) return 2;
  else return NT <= 256 ? (ROUTE ? 4 : 3) : (ROUTE ? 2 : 1);
}
// FP32 tiles stage their FP64 inputs in shared memory only at one block per SM.
template <typename T, bool ROUTE, int NT>
__host__ __device__ constexpr bool stage_keeps_inputs() {
  return stage_blocks_per_sm<T, ROUTE, NT>() == 1;
}

// The FP32 tiles take their halo (and flags) by TMA through the maps in
// `tma`; the FP64 tile ignores them.
template <typename T, int SCHEME, int TI, int TJ, int NT, bool ROUTE>
__global__ void __launch_bounds__(NT, stage_blocks_per_sm<T, ROUTE, NT>())
    k_stage(Geom g, StageArgs a, const __grid_constant__ StageTma tma) {
  chain_wait();
  if (*a.active == 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // first interior node of the tile (0-based)
  if constexpr (sizeof(T) == 4) {
    stage_tile_f32<SCHEME, TI, TJ, NT, ROUTE, false, stage_keeps_inputs<T, ROUTE, NT>(), true>(
        g, a, int(blockIdx.y) * TI, int(blockIdx.x) * TJ, smem_raw, int(blockIdx.y * gridDim.x + blockIdx.x),
        &tma);
  } else {
    stage_tile_f64<SCHEME, TI, TJ, NT, false, true>(g, a, int(blockIdx.y) * a.rows, int(blockIdx.x) * TJ, a.rows,
                                                    a.pair != 0, smem_raw, &tma);
  }
}

// Dynamic shared memory of one stage tile.
template <typename T, int TI, int TJ, bool ROUTE = false, int NT = 256>
constexpr size_t stage_smem_bytes() {
  if constexpr (sizeof(T) == 4) return StageSmem32<TI, TJ, stage_keeps_inputs<T, ROUTE, NT>()>::bytes;
  else return StageSmem<TI, TJ>::bytes;
}

// Host-side launcher for one precision: picks the kernel instance for the
// scheme and tile height, sets its shared-memory size, launches it.
template <typename T, int TI, int NT, bool ROUTE = false>
cudaError_t launch_stage_tile(const Geom &g, const StageArgs &args, const StageTma &tma, int scheme, cudaStream_t s,
                              int rows = TI, int pair = 0) {
  constexpr int TJ = 32;
  constexpr size_t smem = stage_smem_bytes<T, TI, TJ, ROUTE, NT>();
  StageArgs a = args;
  a.rows = rows;
  a.pair = pair;
  const dim3 grid((g.ny + TJ - 1) / TJ, (g.nx + rows - 1) / rows);
  void (*fn)(Geom, StageArgs, StageTma) = nullptr;
  switch (scheme) {
    case kWenoJS: fn = k_stage<T, kWenoJS, TI, TJ, NT, ROUTE>; break;
    case kWenoZ: fn = k_stage<T, kWenoZ, TI, TJ, NT, ROUTE>; break;
    case kWenoZP: fn = k_stage<T, kWenoZP, TI, TJ, NT, ROUTE>; break;
    case kWenoZPI: fn = k_stage<T, kWenoZPI, TI, TJ, NT, ROUTE>; break;
    default: return cudaErrorInvalidValue;
  }
  // The dynamic shared-memory limit is a per-device function attribute: set
  // it on the first launch per device (before any stream capture; the C ABI
  // runs one plain step before it captures a graph).
  static unsigned long long configured[4] = {0, 0, 0, 0};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(configured[scheme & 3] & bit)) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return e;
    configured[scheme & 3] |= bit;
  }
  return launch_chained(fn, grid, NT, smem, s, g, a, tma);
}

}  // namespace dev
}  // namespace wenofd
