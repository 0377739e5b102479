// Device bodies shared by the per-solve kernels (aux_kernels.cu) and the
// persistent batched kernel (batch_kernel.cuh): the boundary fill of one
// ghost entry and a node's wave-speed sum for the time step.
#pragma once

#include "approx.cuh"
#include "chain.cuh"
#include "convert.cuh"
#include "guard.cuh"
#include "int_f64.cuh"
#include "wenofd_internal.h"

namespace wenofd {
namespace dev {

// Member owning work item `item` of a batch's prefix array (n+1 entries).
// The prefix arrays and the member table are read-only for the whole launch.
__device__ __forceinline__ int owner(const int *prefix, int n, int item) {
  int lo = 0, hi = n;  // prefix[lo] <= item < prefix[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(&prefix[mid]) <= item) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ long long at(const Geom &g, int r, int ei, int ej) {
  return WENOFD_IXC(g.guard, unsigned(r) < 4u && unsigned(ei) < unsigned(g.nxt) && unsigned(ej) < unsigned(g.pitch),
                    r * g.plane + (long long)ei * g.pitch + ej, 4 * g.plane);
}

// exchangeGhostCellsValue (src/WENOFD.cpp:850-929, one rank) + setBoundary
// (998-1159).  Every ghost node a stencil reads -- x ghosts on interior
// rows, y ghosts on interior columns -- is a function of interior nodes
// only, so all of them are filled in one pass:
//   x, periodic  : ghost[sx-k] = U[ex-1-k], ghost[ex-1+k] = U[sx+k]
//                  (node-based: the duplicated end node is skipped)
//   SYMMETRIC    : mirror about the boundary node, ghost[sx-k] = U[sx+k]
//   SLIP         : mirror and negate the normal momentum
//   SPECIAL      : initial-condition value at the boundary node (table)
// The y direction uses the bottom condition on both sides (line 1009).
// Corner ghosts (x ghost and y ghost at once) are never read by the sweeps
// (lines 513-797) but are read by the indicator's 5x5 windows; they get the
// reference's values: its y fill runs over every column, ghost columns
// included, after the x exchange, and its x conditions then run over every
// row, ghost rows included.  So a corner is the y rule applied to the
// x-periodic source column (x periodic) or the x rule applied to the y ghost
// of the interior source column (x not periodic).
// Number of ghost entries (each covers the 4 conserved variables).
__host__ __device__ __forceinline__ int bc_entries(const Geom &g) { return 8 * g.nx + 8 * g.ny + 64; }

// Ghost entry t in [0, bc_entries(g)).  Reads go through L2 only: in the
// persistent batched kernel the sources were written by other blocks.
__device__ __forceinline__ void bc_fill_entry(const Geom &g, double *U, const double *special, const int t) {
  const int nxg = 4 * g.nx, nyg = 4 * g.ny;
  const int sx = kGhost, ex = kGhost + g.nx, sy = kGhost, ey = kGhost + g.ny;
  {
    if (t < 2 * nyg) {  // x ghosts on interior rows
      const int side = t / nyg, rem = t - side * nyg;
      const int e1 = rem / g.ny + 1, ej = sy + (rem - (e1 - 1) * g.ny);
      const int bc = side == 0 ? g.bc_left : g.bc_right;
      const int dst = side == 0 ? sx - e1 : ex - 1 + e1;
      int src;
      if (bc == kPeriod) src = side == 0 ? ex - 1 - e1 : sx + e1;
      else src = side == 0 ? sx + e1 : ex - 1 - e1;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        double v;
        if (bc == kSpecial) v = special[WENOFD_SPECIAL(g, 8 * g.nxt + (side * 4 + r) * g.nyt + ej)];
        else v = __ldcg(&U[at(g, r, src, ej)]);
        if (bc == kSlip && r == 1) v *= -1;
        U[at(g, r, dst, ej)] = v;
      }
    } else if (t >= 2 * nyg + 2 * nxg) {  // the 4 x 16 corner ghosts
      const int c = t - 2 * nyg - 2 * nxg;
      const int sidex = c >> 5, sidey = (c >> 4) & 1;
      const int kx = ((c >> 2) & 3) + 1, ky = (c & 3) + 1;
      const int ei = sidex == 0 ? sx - kx : ex - 1 + kx;
      const int ej = sidey == 0 ? sy - ky : ey - 1 + ky;
      const int bcx = sidex == 0 ? g.bc_left : g.bc_right;
      const int srcy = g.bc_y == kPeriod ? (sidey == 0 ? ey - 1 - ky : sy + ky) : (sidey == 0 ? sy + ky : ey - 1 - ky);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        double v;
        if (bcx == kSpecial) {
          v = special[WENOFD_SPECIAL(g, 8 * g.nxt + (sidex * 4 + r) * g.nyt + ej)];
        } else {
          const int col = bcx == kPeriod ? (sidex == 0 ? ex - 1 - kx : sx + kx) : (sidex == 0 ? sx + kx : ex - 1 - kx);
          // y rule at ghost column ei (x periodic: its interior rows hold
          // column col) or at interior column col (x not periodic)
          if (g.bc_y == kSpecial) v = special[WENOFD_SPECIAL(g, (sidey * 4 + r) * g.nxt + (bcx == kPeriod ? ei : col))];
          else v = __ldcg(&U[at(g, r, col, srcy)]);
          if (g.bc_y == kSlip && r == 2) v *= -1;
          if (bcx == kSlip && r == 1) v *= -1;
        }
        U[at(g, r, ei, ej)] = v;
      }
    } else {  // y ghosts on interior columns
      const int u = t - 2 * nyg;
      const int side = u / nxg, rem = u - side * nxg;
      const int e1 = rem / g.nx + 1, ei = sx + (rem - (e1 - 1) * g.nx);
      const int bc = g.bc_y;
      const int dst = side == 0 ? sy - e1 : ey - 1 + e1;
      int src;
      if (bc == kPeriod) src = side == 0 ? ey - 1 - e1 : sy + e1;
      else src = side == 0 ? sy + e1 : ey - 1 - e1;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        double v;
        if (bc == kSpecial) v = special[WENOFD_SPECIAL(g, (side * 4 + r) * g.nxt + ei)];
        else v = __ldcg(&U[at(g, r, ei, src)]);
        if (bc == kSlip && r == 2) v *= -1;
        U[at(g, r, ei, dst)] = v;
      }
    }
  }
}

// The ghost nodes whose value interior node (i, j) determines (bc_fill_entry's
// rules the other way round: its images across x, across y and in the corners).
// SPECIAL ghosts are constants and stay as filled.
__device__ __forceinline__ void store_images(const Geom &g, double *U, int i, int j) {
  auto ghost = [](int k) { return unsigned(k - 1) < unsigned(kGhost); };
  // image across the low (side 0) and the high edge: the node's distance k from
  // the edge that the rule reads, ghost node k of that side
  const int xl = g.bc_left == kPeriod ? g.nx - 1 - i : i, xr = g.bc_right == kPeriod ? i : g.nx - 1 - i;
  const int yl = g.bc_y == kPeriod ? g.ny - 1 - j : j, yr = g.bc_y == kPeriod ? j : g.ny - 1 - j;
  const bool hx[2] = {g.bc_left != kSpecial && ghost(xl), g.bc_right != kSpecial && ghost(xr)};
  const bool hy[2] = {g.bc_y != kSpecial && ghost(yl), g.bc_y != kSpecial && ghost(yr)};
  if (!(hx[0] || hx[1] || hy[0] || hy[1])) return;
  const int ei[2] = {kGhost - xl, kGhost + g.nx - 1 + xr}, ej[2] = {kGhost - yl, kGhost + g.ny - 1 + yr};
  const bool sx[2] = {g.bc_left == kSlip, g.bc_right == kSlip}, sy = g.bc_y == kSlip;
  double w[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) w[r] = __ldcg(&U[at(g, r, kGhost + i, kGhost + j)]);
  auto put = [&](int di, int dj, bool x, bool y) {
    U[at(g, 0, di, dj)] = w[0];
    U[at(g, 1, di, dj)] = x ? -w[1] : w[1];
    U[at(g, 2, di, dj)] = y ? -w[2] : w[2];
    U[at(g, 3, di, dj)] = w[3];
  };
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    if (hx[a]) put(ei[a], kGhost + j, sx[a], false);
    if (hy[a]) put(kGhost + i, ej[a], false, sy);
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
      if (hx[a] && hy[b]) put(ei[a], ej[b], sx[a], sy);
}

// End of a stage tile in the time loop (all NT threads): the ghosts that the
// tile's nodes determine, so that the loop needs no boundary launch (batched
// kernel: phase) per stage.
// Read back from the nodes just stored, in the tiles at the grid's edge only:
// done at each node's store it cost the grids of many tiles 4 to 12 % (a call and
// the grid's description on the stack of every thread).
template <int TJ, int NT>
__device__ __forceinline__ void store_tile_ghosts(const Geom &g, const StageArgs &a, int i0, int j0, int rows) {
  if (!a.ghosts || (i0 > kGhost && j0 > kGhost && i0 + rows + kGhost < g.nx && j0 + TJ + kGhost < g.ny)) return;
  __syncthreads();  // the tile's nodes are stored
  for (int t = threadIdx.x; t < rows * TJ; t += NT) {
    const int i = i0 + t / TJ, j = j0 + t % TJ;
    if (i < g.nx && j < g.ny) store_images(g, a.uout, i, j);
  }
}

// Whether the next graph-driven step runs: while |now - t_end| > 1e-9 (the loop
// condition of src/WENOFD.cpp:213), no error, and under the step cap.
__device__ __forceinline__ void gate_step(Ctrl *c) {
  c->active = (!c->done && !c->error && c->steps < c->max_steps) ? 1 : 0;
}

// m_now += dt; count++ (src/WENOFD.cpp:238-239), then the loop condition.
// fused: the step's last stage wrote the screen bounds of the new U^n.
__device__ __forceinline__ void end_step(Ctrl *c, int fused) {
  c->now += c->dt;
  c->steps += 1;
  c->done = !(fabs(c->now - c->t_end) > 1e-9);
  c->bounds_valid = fused;
}

// True in the thread whose arrival is the launch's last; one thread of each
// block calls it.
__device__ __forceinline__ bool arrive_last(Ctrl *c) {
  if (atomicAdd(&c->arrivals, 1u) != gridDim.x * gridDim.y - 1u) return false;
  c->arrivals = 0u;
  return true;
}

// In the last stage of a step: the last block to come here ends the step.  Of
// what that writes a stage reads only the gate, so one thread of each block calls
// it once its block has passed the gate (a barrier after it), beside the wait for
// the tile's copy; the stage itself need not have ended.
__device__ __forceinline__ void finish_step(const StageArgs &a) {
  if (a.end && arrive_last(a.end)) {
    end_step(a.end, 1);
    gate_step(a.end);
  }
}

// A node's s depends only on its four state values.  In uniform regions
// (the quadrants of a Riemann problem) every node ties for the maximum and
// the FP64 evaluation (five divisions and a square root on a pipe at 1/73 of
// the FP32 rate) would run for each of them: a thread skips a node whose
// values are bit for bit those of the last node it evaluated, which leaves
// the maximum and the NaN flag unchanged.
struct SpeedMemo {
  long long k[4] = {0, 0, 0, 0};
  bool valid = false;
  __device__ __forceinline__ bool repeat(double rho, double mu, double mv, double E) {
    const long long a = __double_as_longlong(rho), b = __double_as_longlong(mu), c = __double_as_longlong(mv),
                    d = __double_as_longlong(E);
    const bool same = valid && a == k[0] && b == k[1] && c == k[2] && d == k[3];
    k[0] = a;
    k[1] = b;
    k[2] = c;
    k[3] = d;
    valid = true;
    return same;
  }
};

// One node's s = lx/dx + ly/dy exactly as calculateDeltaT forms it
// (src/WENOFD.cpp:419-423 with utils/equations.hpp:137-147): products,
// quotients and the root on the integer pipes where their domain allows (the
// same bits; the FP64 pipe takes 19 cycles of an SM per warp instruction, and
// five divisions and a root are some 65 of them), FP64 arithmetic elsewhere.  Where
// every node ties, the refinement at 257 x 193 takes 8.6 us instead of 13.3.  Out
// of line: few nodes get here.
template <int = 0>
__device__ __noinline__ double exact_speed(double gamma, double dx, double dy, double rho, double mu, double mv,
                                           double E) {
  if (positive_in_range<-60, 60>(rho) && in_range<-200, 60>(mu) && in_range<-200, 60>(mv) &&
      positive_in_range<-60, 60>(E) && positive_in_range<-200, 200>(dx) && positive_in_range<-200, 200>(dy)) {
    const IntDivisor by_rho(rho);
    const double u = by_rho.quotient(mu), v = by_rho.quotient(mv);
    const double p = int_mul(gamma - 1.0, fma(-0.5, int_mul(rho, int_mul(u, u) + int_mul(v, v)), E));
    if (positive_in_range<-60, 60>(p)) {
      const double c = int_sqrt(by_rho.quotient(int_mul(gamma, p)));
      return IntDivisor(dx).quotient(fabs(u) + c) + IntDivisor(dy).quotient(fabs(v) + c);
    }
  }
  // Rounded operation by operation: the FP32 batches are compiled with contraction.
  const double u = __ddiv_rn(mu, rho), v = __ddiv_rn(mv, rho);
  const double K = __dadd_rn(__dmul_rn(u, u), __dmul_rn(v, v));
  const double p = __dmul_rn(gamma - 1.0, __dsub_rn(E, __dmul_rn(__dmul_rn(0.5, rho), K)));
  const double cs = __dsqrt_rn(__ddiv_rn(__dmul_rn(gamma, p), rho));
  const double lx = __dadd_rn(fabs(__dadd_rn(u, __dmul_rn(v, 0.0))), cs);
  const double ly = __dadd_rn(fabs(__dadd_rn(__dmul_rn(u, 0.0), v)), cs);
  return __dadd_rn(__ddiv_rn(lx, dx), __ddiv_rn(ly, dy));
}

// FP32 estimate s32 of a node's s and a bound e with |s32 - s| <= e.  Error
// budget (eps = 2^-23, each operation and the hardware's reciprocal and root at
// most eps): inputs truncated to FP32 (eps each), u and v 4 eps, kinetic energy
// ke 7 eps, so p = (gamma-1)(E - ke) carries at most rp = 12 eps (|E| + ke) /
// (E - ke) relative error (the cancellation term); c^2 that plus 5 eps, c half
// of it plus eps; s = (|u| + c)/dx + (|v| + c)/dy then 7 eps of itself plus rp/2
// of c/dx + c/dy.  The bound takes 4x that.  Nodes with a non-positive or
// non-finite FP32 pressure or sound speed get e = inf.  (About 30 instructions:
// the last stage of every step runs it on every node; IEEE divisions and root
// here took some 100.)
__device__ __forceinline__ void screen_speed(const Geom &g, double rho_d, double mu_d, double mv_d, double E_d,
                                             float &s, float &e) {
  // Explicit round-to-nearest operations: no multiply-add contraction, so
  // every translation unit (the stage kernels' fused screen, the reduction
  // kernels, the batched kernel) computes the same s and e.
  const float eps = 1.1920929e-07f;
  const float4 q = f64x4_to_f32(rho_d, mu_d, mv_d, E_d);
  const float ir = rcp_ftz(q.x), u = __fmul_rn(q.y, ir), v = __fmul_rn(q.z, ir);
  const float ke = __fmul_rn(0.5f, __fmaf_rn(q.y, u, __fmul_rn(q.z, v)));
  const float pp = __fadd_rn(q.w, -ke);
  const float c2 = __fmul_rn(__fmul_rn(g.gg32, pp), ir);
  if (!(pp > 0.0f) || !(c2 > 0.0f) || !(c2 < 3.0e38f)) {
    s = 0.0f;
    e = __int_as_float(0x7f800000);
    return;
  }
  const float c = sqrt_ftz(c2);
  const float cs = __fmaf_rn(c, g.inv_dx32, __fmul_rn(c, g.inv_dy32));
  s = __fmaf_rn(fabsf(u), g.inv_dx32, __fmaf_rn(fabsf(v), g.inv_dy32, cs));
  // 4 (7 eps s + (rp / 2) cs)
  const float rp = __fmul_rn(__fadd_rn(fabsf(q.w), ke), rcp_ftz(pp));
  e = __fmul_rn(eps, __fmaf_rn(28.0f, s, __fmul_rn(24.0f, __fmul_rn(rp, cs))));
}

// The largest s of the nodes first, first + stride, .. below end of this
// thread, FP64 form: a first pass screens them in FP32 and raises *screen, the
// greatest lower bound that any warp has found so far, a second one evaluates
// exactly where the upper bound still reaches it.  Whatever value it has when it
// is read, the node of the maximum reaches it, so the maximum is that of the
// exact pass over every node; only how many others are evaluated depends on the
// order.  All lanes of the warp call it.  State outside the range in which the
// FP32 bound holds (values FP32 cannot hold, or flushes) is always evaluated.
// Warm, a launch: 4096^2 1952 us with every node exact on the FP64 pipe, 191 now
// (two loads of the state where candidates lie, else one); 800^2 89 -> 16, 100^2
// 8.8 -> 5.9.
template <class Node, class Offer>
__device__ __forceinline__ void screened_max(const Geom &g, unsigned *screen, long long first, long long end,
                                             long long stride, Node node, Offer offer) {
  auto bounds = [&](long long t, double &rho, double &mu, double &mv, double &E, float &s, float &e) {
    node(t, rho, mu, mv, E);
    screen_speed(g, rho, mu, mv, E, s, e);
    if (!(positive_in_range<-30, 30>(rho) && positive_in_range<-30, 30>(E) && e < 3.0e38f)) {
      s = 0.0f;
      e = __int_as_float(0x7f800000);
    }
  };
  double rho, mu, mv, E;
  float s, e, lo = 0.0f, hi = 0.0f;
  for (long long t = first; t < end; t += stride) {
    bounds(t, rho, mu, mv, E, s, e);
    lo = fmaxf(lo, s - e);
    hi = fmaxf(hi, s + e);
  }
  for (int o = 16; o > 0; o >>= 1) lo = fmaxf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
  unsigned L = __float_as_uint(lo);  // (positive floats order as their bits)
  if ((threadIdx.x & 31) == 0) L = max(L, atomicMax(screen, L));
  lo = __uint_as_float(__shfl_sync(0xffffffffu, L, 0));
  if (hi < lo) return;
  SpeedMemo memo;
  for (long long t = first; t < end; t += stride) {
    bounds(t, rho, mu, mv, E, s, e);
    if (s + e >= lo && !memo.repeat(rho, mu, mv, E)) offer(exact_speed(g.gamma, g.dx, g.dy, rho, mu, mv, E));
  }
}

}  // namespace dev
}  // namespace wenofd
