// Launch dispatch of the block-sparse products over (dtype, operand majorness); the kernel lives
// in bsmm_kernel.cuh.
#include "bsmm_kernel.cuh"

namespace mb {
namespace bsmm {

namespace {
template <typename T, int BN>
cudaError_t launch_t(bool a_mn, bool b_mn, const CUtensorMap& ta, const CUtensorMap& tb, const BsmmParams& p, int grid,
                     cudaStream_t stream) {
  if (a_mn) return b_mn ? launch_one<T, true, true, BN>(ta, tb, p, grid, stream)
                        : launch_one<T, true, false, BN>(ta, tb, p, grid, stream);
  return b_mn ? launch_one<T, false, true, BN>(ta, tb, p, grid, stream)
              : launch_one<T, false, false, BN>(ta, tb, p, grid, stream);
}
}  // namespace

cudaError_t launch(bool bf16, bool a_mn_major, bool b_mn_major, const CUtensorMap& ta, const CUtensorMap& tb,
                   const BsmmParams& p, int grid, cudaStream_t stream) {
  if (p.mode != kSdd && p.mode != kDsd && p.mode != kDds) return cudaErrorInvalidValue;
  if (p.num_tiles <= 0) return cudaSuccess;
  if (p.tile_cols != 128 && !(p.tile_cols == 256 && p.mode == kDsd)) return cudaErrorInvalidValue;
  if (p.tile_cols == 256)
    return bf16 ? launch_t<__nv_bfloat16, 256>(a_mn_major, b_mn_major, ta, tb, p, grid, stream)
                : launch_t<__half, 256>(a_mn_major, b_mn_major, ta, tb, p, grid, stream);
  return bf16 ? launch_t<__nv_bfloat16, 128>(a_mn_major, b_mn_major, ta, tb, p, grid, stream)
              : launch_t<__half, 128>(a_mn_major, b_mn_major, ta, tb, p, grid, stream);
}

}  // namespace bsmm
}  // namespace mb
