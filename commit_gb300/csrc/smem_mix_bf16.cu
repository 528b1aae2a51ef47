// The shared-memory reduced-precision kernels with a BF16 table (smem_mix.cuh).
#include "smem_mix.cuh"

namespace cgb {

int launch_mix_smem_bf16(int adjoint, int nq, int grid, size_t smem, cudaStream_t st, const detail::SmMixArgs &a, int cs) {
    return launch_mix_smem<__nv_bfloat16>(adjoint, nq, grid, smem, st, a, cs);
}

}  // namespace cgb
