// FP32-arithmetic stage kernels (the precision form): split fluxes,
// eigenvectors, projection, WENO reconstruction and flux differences in
// FP32; the state is read and written as FP64 and the RK combination
// a*Un + b*U + c*dt*rhs is evaluated in FP64.
#include <cudaTypedefs.h>

#include <mutex>

#include "stage_kernel.cuh"
#include "stage_routed.cuh"

namespace wenofd {

namespace {

template <int SCHEME>
cudaError_t launch_routed(const Geom &g, const StageArgs &a, const StageTma &tma, cudaStream_t s) {
  using T = dev::RoutedTile;
  static unsigned long long configured = 0;  // one bit per device (launch_stage_tile)
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (device & 63);
  if (!(configured & bit)) {
    e = cudaFuncSetAttribute(dev::k_stage_routed<SCHEME>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(T::bytes));
    if (e != cudaSuccess) return e;
    configured |= bit;
  }
  const dim3 grid((g.ny + T::TJ - 1) / T::TJ, (g.nx + T::TI - 1) / T::TI);
  return launch_chained(dev::k_stage_routed<SCHEME>, grid, T::NT, T::bytes, s, g, a, tma);
}

}  // namespace

// The learned form's default tile: k_stage_routed's where its tiles fill the
// resident blocks (four on each of 152 SMs) one and a half times, else 15 x 32,
// whose block is done sooner.  Measured, 8 steps (k_stage_routed / 15 x 32): 512^2
// 920 / 911 us, 700^2 1,133 / 1,145, 1024^2 1,694 / 1,764, 2048^2 4,538 / 4,801.
// Grids whose tiles of 7 rows fit the resident blocks at once (three on each SM in
// the FP32 form, four in the learned form) take those: a tile's time is the
// latency of its rounds of faces, and a short tile has two instead of four.  A step,
// 7 rows / 15: FP32 100^2 25 / 36 us, 257 x 193 31 / 38, 300^2 (430 tiles of 456) 34
// / 44; learned 100^2 33 / 44, 257 x 193 39 / 49, 350^2 (550 of 608) 52 / 63.
int stage_rows(const Geom &g, int precision, int tile_i) {
  using T = dev::RoutedTile;
  if (precision != 0 && tile_i == 0) {
    const long long tiles = (long long)((g.nx + 6) / 7) * ((g.ny + 31) / 32);
    if (tiles <= (precision == 2 ? 4 : 3) * 152LL) return 7;
  }
  if (precision == 2 && tile_i == 0) {
    const long long tiles = (long long)((g.nx + T::TI - 1) / T::TI) * ((g.ny + T::TJ - 1) / T::TJ);
    if (tiles > 3LL * T::kBlocks * 152 / 2) return T::TI;
  }
  return tile_i > 0 ? tile_i : 15;
}

// With a.flags set the kernel routes each face: linear upwind flux unless a
// node around it is flagged, characteristic WENO otherwise.
cudaError_t launch_stage_fp32(const Geom &g, const StageArgs &a, const StageTma &tma, int scheme, int tile_i, int rows,
                              cudaStream_t s) {
  if (a.flags && rows == dev::RoutedTile::TI && tile_i == 0) {
    switch (scheme) {
      case kWenoJS: return launch_routed<kWenoJS>(g, a, tma, s);
      case kWenoZ: return launch_routed<kWenoZ>(g, a, tma, s);
      case kWenoZP: return launch_routed<kWenoZP>(g, a, tma, s);
      case kWenoZPI: return launch_routed<kWenoZPI>(g, a, tma, s);
    }
    return cudaErrorInvalidValue;
  }
  if (rows == 7 && tile_i == 0)
    return a.flags ? dev::launch_stage_tile<float, 7, 256, true>(g, a, tma, scheme, s)
                   : dev::launch_stage_tile<float, 7, 256>(g, a, tma, scheme, s);
  if (a.flags) {
    switch (tile_i) {
      case 0:
      case 15: return dev::launch_stage_tile<float, 15, 256, true>(g, a, tma, scheme, s);
      case 31: return dev::launch_stage_tile<float, 31, 512, true>(g, a, tma, scheme, s);
    }
    return cudaErrorInvalidValue;
  }
  switch (tile_i) {
    case 0:
    case 15: return dev::launch_stage_tile<float, 15, 256>(g, a, tma, scheme, s);
    case 31: return dev::launch_stage_tile<float, 31, 512>(g, a, tma, scheme, s);
  }
  return cudaErrorInvalidValue;
}

namespace {

// cuTensorMapEncodeTiled, reached through the runtime (the library does
// not link the driver library itself).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static std::once_flag once;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

}  // namespace

cudaError_t make_stage_tma(const Geom &g, const double *state, const unsigned char *flags, int rows,
                           StageTma *out) {
  PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
  if (!encode || !out || !state) return cudaErrorInvalidValue;
  const int ti = (rows == 31 || rows == 7 || rows == dev::RoutedTile::TI) ? rows : 15;
  *out = StageTma{};
  {
    using S = dev::StageSmem32<15, 32>;
    const cuuint64_t dims[3] = {cuuint64_t(g.pitch), cuuint64_t(g.nxt), 4};
    const cuuint64_t strides[2] = {cuuint64_t(g.pitch) * sizeof(double), cuuint64_t(g.plane) * sizeof(double)};
    const cuuint32_t box[3] = {cuuint32_t(S::kBoxJ), cuuint32_t(ti + 6), 4}, step[3] = {1, 1, 1};
    if (encode(&out->u, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, const_cast<double *>(state), dims, strides, box, step,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
  }
  if (flags) {
    using S = dev::StageSmem32<15, 32>;
    const cuuint64_t dims[2] = {cuuint64_t(g.pitch), cuuint64_t(g.nxt)};
    const cuuint64_t strides[1] = {cuuint64_t(g.pitch)};
    const cuuint32_t box[2] = {cuuint32_t(S::kFlagBoxJ), cuuint32_t(ti + 4)}, step[2] = {1, 1};
    if (encode(&out->flags, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<unsigned char *>(flags), dims, strides, box,
               step, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return cudaErrorInvalidValue;
  }
  return cudaSuccess;
}

}  // namespace wenofd
