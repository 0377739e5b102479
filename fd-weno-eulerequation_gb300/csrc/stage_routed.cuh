// One RK stage of the learned form on grids of many tiles: a 16 x 32 tile made
// for the faces that take the linear flux, nearly all of them.
//
// Phases of a block (256 threads, four blocks per SM):
//   halo box (TMA) -> a thread's three or four nodes to FP32 registers
//   -> x split of them to shared memory -> x march (lane = column, warp = two
//   rows): three faces, two differences -> y split -> y march (lane = row, two
//   columns) -> the differences to the lanes that own the columns -> RK
//   combination in FP64, coalesced.
// A march loads a stencil node once for its faces (7 128-bit shared loads a node
// and direction instead of 10 and the face array's 3), a tile without a flag
// forms its flux differences in registers (no face array, no barrier around
// it), and the state stays in registers between the two splits.
// A tile with a flag on or around it (block-uniform) also stores the faces,
// recomputes the listed ones with characteristic WENO (weno_face_lane, four
// lanes a face, the faces' nodes from the state it keeps) and takes the
// differences from the stored faces.
//
// What bounds it, 4096^2, mean of the three stages, without the time-step
// screen: the copies, barriers and stores alone 268 us (HBM's part 211), with
// the conversion and the splits 279, with the marches 327, with the FP64
// combination 424: the FP64 pipe (262 us of it) and the copies' latency, partly
// overlapped.  Stages 1 / 2 / 3 in the time loop: 444 / 497 / 587 us with the 15 x
// 32 tile of stage_f32.cuh, 339 / 408 / 526 here with no flag in the interior; 487
// / 550 / 638 and 441 / 522 / 637 with 0.7 % of the nodes flagged one by one.  Those
// with the listed faces' nodes loaded from global memory; kept in shared memory, a
// step at 2400^2 with 10 / 28 / 100 % of the nodes flagged takes 0.89 / 1.20 / 1.49
// ms instead of 1.08 / 1.55 / 2.01 (15 x 32: 0.94 / 1.24 / 1.52), and 4096^2 with
// few flags 1.68 instead of 1.73; placed behind the box instead of over its end,
// 12 % less L1 for the spills cost the batched kernel 5 %.
// Other shapes (rows, threads, blocks per SM): (32, 256, 3) 319 / 440 / 541, (32,
// 512, 2) 375 / 483 / 640, (16, 256, 5) 390 / 482 / 557, (16, 128, 5) 332 / 449 /
// 553; the next tile's copies under this one's combination (persistent blocks)
// 397 / 588 / 687; the RHS-independent sums in integers 346 / 472 / 603.
#pragma once

#include "stage_f32.cuh"

namespace wenofd {
namespace dev {

struct RoutedTile {
  static constexpr int TI = 16, TJ = 32, HI = TI + 6, NT = 256, kBlocks = 4;
  static constexpr int kWarps = NT / 32;
  static constexpr int kRows = TI / kWarps;   // rows of a warp in the x march and the combination
  static constexpr int kCols = TI * TJ / NT;  // columns of a thread in the y march (a lane a row)
  static constexpr int kBoxJ = 40, kFlagBoxJ = 48;
  static constexpr unsigned kBoxBytes = 4u * HI * kBoxJ * 8u;
  static constexpr unsigned kFlagBoxBytes = unsigned(kFlagBoxJ) * (TI + 4);
  static constexpr int kX = HI * TJ;           // split fluxes of the x sweep [HI][TJ], one of F+, F-
  static constexpr int kYS = TJ + 7;           // row stride of the y sweep's [TI][TJ + 6] (odd: no bank conflicts)
  static constexpr int kY = TI * kYS;
  static constexpr int kHS = TJ + 1;           // row stride of the y faces and differences
  static constexpr int kFace = (TI + 1) * TJ > TI * kHS ? (TI + 1) * TJ : TI * kHS;
  // shared memory: F+ and F- of a sweep, the state of a tile with a flag, the
  // faces; the box lies over the first two and is in registers before either is
  // written.  (The L1 cache has what four blocks leave: spills live there.)
  static constexpr size_t kSplits = 2 * sizeof(float4) * (kX > kY ? kX : kY);
  static constexpr int kUS = TJ + 6, kU = HI * kUS;  // FP32 state with halo [HI][TJ + 6], kept by tiles with a flag
  static constexpr size_t kFaces = kSplits + sizeof(float4) * kU;  // offset of the faces
  static_assert(kBoxBytes <= kFaces && kSplits % 16 == 0, "the box ends before the faces");
  static constexpr size_t bytes = 128 + kFaces + sizeof(float4) * kFace;
};

// N + 1 consecutive faces of one line of nodes: faces f0 .. f0 + N from F+ at
// nodes f0 .. f0 + N + 4 and F- at f0 + 1 .. f0 + N + 5 (`ss` apart), each the
// linear fifth-order upwind flux, summed node by node as linear_face4 does.
template <int N>
__device__ __forceinline__ void linear_march(const float4 *P, const float4 *M, int ss, float4 h[N + 1]) {
  float2 lo[N + 1], hi[N + 1];
#pragma unroll
  for (int n = 0; n < N + 6; ++n) {
    if (n < N + 5) {
      const float4 p = P[n * ss];
#pragma unroll
      for (int k = 0; k <= N; ++k) {
        const int s = n - k;  // F+ of the face's node s
        if (s == 0) {
          lo[k] = __fmul2_rn(splat2(lin_coef(0)), lo2(p));
          hi[k] = __fmul2_rn(splat2(lin_coef(0)), hi2(p));
        } else if (s > 0 && s < 5) {
          lo[k] = __ffma2_rn(splat2(lin_coef(s)), lo2(p), lo[k]);
          hi[k] = __ffma2_rn(splat2(lin_coef(s)), hi2(p), hi[k]);
        }
      }
    }
    if (n > 0) {
      const float4 m = M[(n - 1) * ss];
#pragma unroll
      for (int k = 0; k <= N; ++k) {
        const int s = n - 1 - k;  // F- of the face's node s, mirrored
        if (s >= 0 && s < 5) {
          lo[k] = __ffma2_rn(splat2(lin_coef(4 - s)), lo2(m), lo[k]);
          hi[k] = __ffma2_rn(splat2(lin_coef(4 - s)), hi2(m), hi[k]);
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k <= N; ++k) h[k] = join2(lo[k], hi[k]);
}

// The FP32 state of ghosted node (ei, ej), as the tile's conversion gives it.
__device__ __forceinline__ float4 node_f32(const Geom &g, const double *U, int ei, int ej) {
  const double *p = U + WENOFD_GNODE(g, ei, ej);
  return f64x4_to_f32(__ldcg(p), __ldcg(p + g.plane), __ldcg(p + 2 * g.plane), __ldcg(p + 3 * g.plane));
}

// The tile of interior nodes from (i0, j0), number `tile` of its grid; all
// threads of the block.  COH (batched kernel): a thread loads its halo nodes from
// L2 straight into registers and the flag rows by 16-byte loads, without the
// boxes and their TMA maps.
template <int SCHEME, bool COH>
__device__ __forceinline__ void routed_tile(const Geom &g, const StageArgs &a, const int i0, const int j0,
                                            unsigned char *smem_raw, const int tile, const StageTma *tma) {
  using S = RoutedTile;
  constexpr int TI = S::TI, TJ = S::TJ, HI = S::HI, NT = S::NT, W = S::kWarps, RW = S::kRows, CW = S::kCols;
  unsigned char *base = smem_raw + (((tma_smem_addr(smem_raw) + 127u) & ~127u) - tma_smem_addr(smem_raw));
  float4 *Us = reinterpret_cast<float4 *>(base + S::kSplits), *Hf = reinterpret_cast<float4 *>(base + S::kFaces);
  __shared__ __align__(128) unsigned char sflag[S::kFlagBoxBytes];
  __shared__ short slist[S::kFace];
  __shared__ int scount_x, scount_y;
  __shared__ __align__(8) unsigned long long tma_bar;
  const int lane = int(threadIdx.x) & 31, warp = int(threadIdx.x) >> 5;
  const bool stage1 = a.form == kFormStage1;

  if (threadIdx.x == 0) {
    scount_x = scount_y = 0;
    if constexpr (!COH) {
      tma_bar_init(tma_smem_addr(&tma_bar), 1);
      const unsigned bar = tma_smem_addr(&tma_bar);
      tma_fence_proxy();
      tma_bar_expect(bar, S::kBoxBytes + S::kFlagBoxBytes);
      // first coordinates x * element size a multiple of 16 bytes: j0 is a
      // multiple of 32 (an unissued copy leaves the wait below to give up)
      if (WENOFD_REQUIRE(g.guard, (j0 & 1) == 0, j0, 2)) tma_load_3d(tma_smem_addr(base), &tma->u, j0, 1 + i0, 0, bar);
      if (WENOFD_REQUIRE(g.guard, (j0 & 15) == 0, j0, 16))
        tma_load_2d(tma_smem_addr(sflag), &tma->flags, j0, 2 + i0, bar);
    }
  }
  // stages 2 and 3: ask L2 for this warp's rows of U^n (stage_tile_f32): lane =
  // component, row, and the line of column 0, 16 or 28
  if (a.mode == kModeRK && !stage1) {
#pragma unroll
    for (int t = lane; t < 12 * RW; t += 32) {
      const int ii = min(i0 + RW * warp + (t >> 2) % RW, g.nx - 1), l = (t >> 2) / RW;
      prefetch_l2(a.un + (t & 3) * g.plane + WENOFD_NODE(g, ii, min(j0 + (l == 2 ? 28 : 16 * l), g.ny - 1)));
    }
  }
  if constexpr (!COH) {
    __syncthreads();  // the barrier is initialised
    if (threadIdx.x == 0) finish_step(a);
    const bool landed = tma_bar_wait(tma_smem_addr(&tma_bar), 0, kTmaWaitLimit);
    if (__syncthreads_or(!landed)) {
      if (threadIdx.x == 0) {
        if (a.wait_error) atomicExch(a.wait_error, 1);
        tma_bar_wait(tma_smem_addr(&tma_bar), 0, kTmaWaitLimit);
      }
      __syncthreads();
      return;
    }
  }

  // this thread's nodes: column `lane` of halo rows warp, warp + W, ..; and of
  // the 6 x TI nodes beside the tile's columns one (halo column 0..2 or 35..37)
  static_assert(NT >= 6 * TI, "a thread for each node beside the tile's columns");
  constexpr int NR = (HI + W - 1) / W;
  float4 q[NR + 1];
  const int side = int(threadIdx.x) % 6, side_row = int(threadIdx.x) / 6;  // rows below TI only
  const int side_col = side < 3 ? side : TJ + side;                          // halo column
  // flag node (fi, fj) is byte fi * 48 + fj + 2 of sflag, a row three 16-byte parts
  const int flag_row = int(threadIdx.x) / 3, flag_part = int(threadIdx.x) % 3;
  const bool has_flags = flag_row < TI + 4;
  uint4 fv = make_uint4(0u, 0u, 0u, 0u);
  if constexpr (COH) {
    if (has_flags && 2 + i0 + flag_row < g.nxt && j0 + 16 * flag_part < g.pitch) {  // (rows are a multiple of 32)
      const long long o = (long long)(2 + i0 + flag_row) * g.pitch + j0 + 16 * flag_part;
      fv = __ldg(reinterpret_cast<const uint4 *>(a.flags + WENOFD_SPAN(g.guard, o, o + 15, (long long)g.nxt * g.pitch)));
    }
    auto node = [&](int hi, int hj) {  // beyond the last ghosts: a node of the last row or column, not used
      return node_f32(g, a.uin, min(1 + i0 + hi, g.nxt - 1), min(1 + j0 + hj, g.nyt - 1));
    };
#pragma unroll
    for (int m = 0; m < NR; ++m) q[m] = node(min(warp + W * m, HI - 1), lane + 3);
    q[NR] = node(min(side_row, TI - 1) + 3, side_col);
    if (has_flags) reinterpret_cast<uint4 *>(sflag)[WENOFD_IX(g.guard, int(threadIdx.x), S::kFlagBoxBytes / 16)] = fv;
  } else {
    const double *box = reinterpret_cast<const double *>(base);
    auto node = [&](int hi, int hj) {  // box column = halo column + 1
      const int o = hi * S::kBoxJ + hj + 1;
      constexpr int plane = HI * S::kBoxJ;
      return f64x4_to_f32(box[WENOFD_IX(g.guard, o, S::kBoxBytes / 8)], box[WENOFD_IX(g.guard, plane + o, S::kBoxBytes / 8)],
                          box[WENOFD_IX(g.guard, 2 * plane + o, S::kBoxBytes / 8)],
                          box[WENOFD_IX(g.guard, 3 * plane + o, S::kBoxBytes / 8)]);
    };
#pragma unroll
    for (int m = 0; m < NR; ++m) q[m] = node(min(warp + W * m, HI - 1), lane + 3);
    q[NR] = node(min(side_row, TI - 1) + 3, side_col);
    if (has_flags) fv = reinterpret_cast<const uint4 *>(sflag)[WENOFD_IX(g.guard, int(threadIdx.x), S::kFlagBoxBytes / 16)];
  }
  // any flag on the tile or within two nodes of it: the row's first two and last
  // ten bytes do not count
  const unsigned seen = flag_part == 0 ? (fv.x & 0xffff0000u) | fv.y | fv.z | fv.w
                                       : (flag_part == 1 ? fv.x | fv.y | fv.z | fv.w : fv.x | (fv.y & 0x0000ffffu));
  const bool routed = __syncthreads_or(seen != 0u);
  if (routed) {  // the listed faces' nodes
#pragma unroll
    for (int m = 0; m < NR; ++m)
      if (warp + W * m < HI) Us[WENOFD_IX(g.guard, (warp + W * m) * S::kUS + lane + 3, S::kU)] = q[m];
    if (side_row < TI) Us[WENOFD_IX(g.guard, (side_row + 3) * S::kUS + side_col, S::kU)] = q[NR];
  }

  const float gamma = g.gamma32, zpl = g.zpl32;
  float4 *Fp = reinterpret_cast<float4 *>(base), *Fm = Fp + S::kX;
#pragma unroll
  for (int m = 0; m < NR; ++m) {
    const int hi = warp + W * m;
    if (hi < HI) {
      const int o = WENOFD_IX(g.guard, hi * TJ + lane, S::kX);
      split4<0>(gamma, q[m], Fm[o], Fp[o]);
    }
  }
  __syncthreads();

  // --- x march: column `lane`, rows RW warp .. + RW - 1, faces RW warp .. + RW
  float4 rhs[RW];
  {
    const int o = WENOFD_SPAN(g.guard, RW * warp * TJ + lane, (RW * warp + RW + 5) * TJ + lane, S::kX);
    float4 h[RW + 1];
    linear_march<RW>(Fp + o, Fm + o + TJ, TJ, h);
    if (routed) {
#pragma unroll
      for (int k = 0; k <= RW; ++k) {
        const int f = RW * warp + k, t = f * TJ + lane;
        if (k == RW && warp != W - 1) continue;  // the next warp's first
        Hf[WENOFD_IX(g.guard, t, S::kFace)] = h[k];
        if (i0 + f > g.nx || j0 + lane >= g.ny) continue;
        const unsigned char *fl =
            sflag + WENOFD_SPAN(g.guard, f * S::kFlagBoxJ + lane + 4, (f + 3) * S::kFlagBoxJ + lane + 4, S::kFlagBoxBytes);
        if (fl[0] | fl[S::kFlagBoxJ] | fl[2 * S::kFlagBoxJ] | fl[3 * S::kFlagBoxJ])
          slist[WENOFD_IX(g.guard, atomicAdd(&scount_x, 1), S::kFace)] = short(t);
      }
      __syncthreads();
      const int nw = scount_x;
      for (int b = threadIdx.x & ~31; b < 4 * nw; b += NT) {  // 4 lanes per face, whole warps
        const int q4 = b + lane;
        const int t = slist[WENOFD_IX(g.guard, q4 < 4 * nw ? q4 >> 2 : 0, S::kFace)];
        const int f = t / TJ, j = t - f * TJ;
        const float w = weno_face_lane<0, SCHEME>(
            gamma, zpl, Us[WENOFD_IX(g.guard, (f + 2) * S::kUS + j + 3, S::kU)],
            Us[WENOFD_IX(g.guard, (f + 3) * S::kUS + j + 3, S::kU)],
            Fp + WENOFD_SPAN(g.guard, t, t + 4 * TJ, S::kX), Fm + WENOFD_SPAN(g.guard, t + TJ, t + 5 * TJ, S::kX), TJ,
            q4 & 3);
        if (q4 < 4 * nw) reinterpret_cast<float *>(&Hf[WENOFD_IX(g.guard, t, S::kFace)])[q4 & 3] = w;
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k <= RW; ++k) h[k] = Hf[WENOFD_IX(g.guard, (RW * warp + k) * TJ + lane, S::kFace)];
    }
    const float2 mi = splat2(-g.inv_dx32);
#pragma unroll
    for (int k = 0; k < RW; ++k)
      rhs[k] = join2(__fmul2_rn(sub2(lo2(h[k + 1]), lo2(h[k])), mi), __fmul2_rn(sub2(hi2(h[k + 1]), hi2(h[k])), mi));
  }
  __syncthreads();

  // --- y split over the same region
  Fm = Fp + S::kY;
#pragma unroll
  for (int m = 0; m < NR; ++m) {
    const int i = warp + W * m - 3;  // tile row
    if (unsigned(i) < unsigned(TI)) {
      const int o = WENOFD_IX(g.guard, i * S::kYS + lane + 3, S::kY);
      split4<1>(gamma, q[m], Fm[o], Fp[o]);
    }
  }
  if (side_row < TI) {
    const int o = WENOFD_IX(g.guard, side_row * S::kYS + side_col, S::kY);
    split4<1>(gamma, q[NR], Fm[o], Fp[o]);
  }
  __syncthreads();

  // --- y march: row yi, columns y0 .. y0 + CW - 1 (a lane a row)
  {
    const int yi = int(threadIdx.x) % TI, y0 = int(threadIdx.x) / TI * CW;
    const int o = WENOFD_SPAN(g.guard, yi * S::kYS + y0, yi * S::kYS + y0 + CW + 5, S::kY);
    float4 h[CW + 1];
    linear_march<CW>(Fp + o, Fm + o + 1, 1, h);
    if (!routed) {
#pragma unroll
      for (int k = 0; k < CW; ++k)
        Hf[WENOFD_IX(g.guard, yi * S::kHS + y0 + k, S::kFace)] =
            join2(sub2(lo2(h[k + 1]), lo2(h[k])), sub2(hi2(h[k + 1]), hi2(h[k])));
    } else {
#pragma unroll
      for (int k = 0; k <= CW; ++k) {
        const int f = y0 + k, t = yi * S::kHS + f;
        if (k == CW && f != TJ) continue;  // the next thread's first
        Hf[WENOFD_IX(g.guard, t, S::kFace)] = h[k];
        if (i0 + yi >= g.nx || j0 + f > g.ny) continue;
        const unsigned char *fl = sflag + WENOFD_SPAN(g.guard, (yi + 2) * S::kFlagBoxJ + f + 2,
                                                      (yi + 2) * S::kFlagBoxJ + f + 5, S::kFlagBoxBytes);
        if (fl[0] | fl[1] | fl[2] | fl[3]) slist[WENOFD_IX(g.guard, atomicAdd(&scount_y, 1), S::kFace)] = short(t);
      }
      __syncthreads();
      const int nw = scount_y;
      for (int b = threadIdx.x & ~31; b < 4 * nw; b += NT) {
        const int q4 = b + lane;
        const int t = slist[WENOFD_IX(g.guard, q4 < 4 * nw ? q4 >> 2 : 0, S::kFace)];
        const int i = t / S::kHS, f = t - i * S::kHS, s = i * S::kYS + f;
        const float w = weno_face_lane<1, SCHEME>(
            gamma, zpl, Us[WENOFD_IX(g.guard, (i + 3) * S::kUS + f + 2, S::kU)],
            Us[WENOFD_IX(g.guard, (i + 3) * S::kUS + f + 3, S::kU)],
            Fp + WENOFD_SPAN(g.guard, s, s + 4, S::kY), Fm + WENOFD_SPAN(g.guard, s + 1, s + 5, S::kY), 1, q4 & 3);
        if (q4 < 4 * nw) reinterpret_cast<float *>(&Hf[WENOFD_IX(g.guard, t, S::kFace)])[q4 & 3] = w;
      }
    }
  }
  // --- y term, source, RK combination in FP64, store (rows RW warp .. + RW - 1);
  // a row's inputs are loaded while the row before it is worked on, the first
  // row's across the barrier (block-uniform bases and 32-bit offsets)
  const long long origin = (long long)(kGhost + i0) * g.pitch + (kGhost + j0);
  const double *in = a.uin + origin, *un0 = a.un + origin;
  double *out = a.uout + origin;
  double ui[2][4], un[2][4];
  auto load_row = [&](int k, int b) {
    const int i = RW * warp + k;
    const bool ok = i0 + i < g.nx && j0 + lane < g.ny;
    const unsigned at = ok ? unsigned(WENOFD_NODE(g, i0 + i, j0 + lane) - origin) : 0u;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      ui[b][r] = __ldcg(in + r * g.plane + at);
      un[b][r] = stage1 ? 0.0 : __ldcg(un0 + r * g.plane + at);
    }
  };
  load_row(0, 0);
  __syncthreads();
  if constexpr (!COH) chain_release();
  const double dt = COH ? __ldcg(a.dt) : *a.dt;
  float lo = 0.0f, hi = 0.0f;  // screen bounds of this thread's nodes
  const float2 mi = splat2(-g.inv_dy32);
#pragma unroll
  for (int k = 0; k < RW; ++k) {
    if (k < RW - 1) load_row(k + 1, (k + 1) & 1);
    const int i = RW * warp + k, j = lane, b = k & 1;
    if (i0 + i >= g.nx || j0 + j >= g.ny) continue;
    float4 d = Hf[WENOFD_IX(g.guard, i * S::kHS + j, S::kFace)];
    if (routed) {
      const float4 r = Hf[WENOFD_IX(g.guard, i * S::kHS + j + 1, S::kFace)];
      d = join2(sub2(lo2(r), lo2(d)), sub2(hi2(r), hi2(d)));
    }
    const float2 r01 = __ffma2_rn(lo2(d), mi, lo2(rhs[k])), r23 = __ffma2_rn(hi2(d), mi, hi2(rhs[k]));
    float rr[4] = {r01.x, r01.y, r23.x, r23.y};
    if (g.gravity) {  // RTI, g = 1 (src/WENOFD.cpp:807-813)
      rr[3] += f64_to_f32(ui[b][2]) * 1.0f;
      rr[2] += f64_to_f32(ui[b][0]) * 1.0f;
    }
    double w[4];
    rk_combine(a, dt, rr, ui[b], un[b], w);
    const unsigned at = unsigned(WENOFD_NODE(g, i0 + i, j0 + j) - origin);
#pragma unroll
    for (int r = 0; r < 4; ++r) out[r * g.plane + at] = w[r];
    if (a.bounds) {
      float s32, e;
      screen_speed(g, w[0], w[1], w[2], w[3], s32, e);
      lo = fmaxf(lo, s32 - e);
      hi = fmaxf(hi, s32 + e);
    }
  }
  if (a.bounds) store_tile_bounds<NT>(g, a, lo, hi, tile);
  store_tile_ghosts<TJ, NT>(g, a, i0, j0, TI);
}

template <int SCHEME>
__global__ void __launch_bounds__(RoutedTile::NT, RoutedTile::kBlocks)
    k_stage_routed(Geom g, StageArgs a, const __grid_constant__ StageTma tma) {
  chain_wait();
  if (*a.active == 0) return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  routed_tile<SCHEME, false>(g, a, int(blockIdx.y) * RoutedTile::TI, int(blockIdx.x) * RoutedTile::TJ, smem_raw,
                             int(blockIdx.y * gridDim.x + blockIdx.x), &tma);
}

}  // namespace dev
}  // namespace wenofd
