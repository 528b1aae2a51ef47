// The shared-memory reduced-precision kernels with an FP16 table (smem_mix.cuh).
#include "smem_mix.cuh"

namespace cgb {

int launch_mix_smem_fp16(int adjoint, int nq, int grid, size_t smem, cudaStream_t st, const detail::SmMixArgs &a, int cs) {
    return launch_mix_smem<__half>(adjoint, nq, grid, smem, st, a, cs);
}

}  // namespace cgb
