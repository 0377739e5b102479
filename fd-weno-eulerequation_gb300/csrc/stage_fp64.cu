// FP64 stage kernels: the parity path.  This translation unit is compiled
// with -fmad=false so that no multiply-add is contracted into an FMA; with
// IEEE division and square root every operation then rounds as in the
// reference built with -ffp-contract=off.
#include "stage_kernel.cuh"

namespace wenofd {

// A stage's time on the SM with the most tiles, in microseconds, is the larger
// of two sums over them: warps of faces times the throughput of two resident
// blocks (5.4 a warp; a pair of lanes repeats the face's eigenvectors: 3.0), and
// rounds of a block's eight warps times the latency of one round (45; two lanes
// a face: 24).  Few tiles: the latency counts, and short tiles on more SMs with
// two lanes a face win; many: the tallest tiles share the most.
// Measured (rows, lanes a face): 100^2 WENO-JS, a step: (15, 1) 586 us, (7, 1)
// 324, (3, 1) 255, (3, 2) 208; 121x481 SSP-RK2: (15, 1) 418, (7, 1) 358, (7, 2)
// 394; 800^2: (15, 1) 4.77 ms, (7, 1) 5.00, (15, 2) 5.28.
Fp64Split fp64_split(const int *nx, const int *ny, int n, int sms, int most) {
  Fp64Split best{most, 0};
  double best_cost = 0.0;
  for (int pair = 0; pair < 2; ++pair)
    for (int rows = most; rows >= 1; --rows) {
      long long tiles = 0;
      for (int m = 0; m < n; ++m) tiles += (long long)((nx[m] + rows - 1) / rows) * ((ny[m] + 31) / 32);
      const int wx = (rows + 1) << pair, wy = ((rows * 33 + 31) / 32) << pair;  // warps of faces
      const double each = pair ? 3.0 : 5.4, alone = (pair ? 18.0 : 33.0) + (pair ? 0.8 : 1.5) * 8;
      const long long per_sm = (tiles + sms - 1) / sms;
      const double busy = double(per_sm) * (wx + wy) * each;
      const double chain = double((per_sm + 1) / 2) * ((wx + 7) / 8 + (wy + 7) / 8) * alone;
      const double cost = busy > chain ? busy : chain;
      if ((rows == most && !pair) || cost < 0.97 * best_cost) {
        best = Fp64Split{rows, pair};
        best_cost = cost;
      }
    }
  return best;
}

// The tile's halo arrives by TMA through the map in `tma` (make_stage_tma
// for this tile height).
cudaError_t launch_stage_fp64(const Geom &g, const StageArgs &a, const StageTma &tma, int scheme, int tile_i,
                              cudaStream_t s) {
  switch (tile_i) {
    case 0: {
      static int sms_of[64] = {0};
      int device = 0;
      cudaError_t e = cudaGetDevice(&device);
      if (e != cudaSuccess) return e;
      int &sms = sms_of[device & 63];
      if (sms == 0 && (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)) != cudaSuccess) return e;
      const Fp64Split x = fp64_split(&g.nx, &g.ny, 1, sms, 15);
      return dev::launch_stage_tile<double, 15, 256>(g, a, tma, scheme, s, x.rows, x.pair);
    }
    case 15: return dev::launch_stage_tile<double, 15, 256>(g, a, tma, scheme, s);
    case 7: return dev::launch_stage_tile<double, 7, 256>(g, a, tma, scheme, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace wenofd
