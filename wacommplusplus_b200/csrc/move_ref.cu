// Move kernels in reference arithmetic (compiled with -fmad=false: every product and sum is
// rounded on its own, as in the reference's x86-64 Release build).
#include "engine.h"
#include "move_kernels.cuh"

namespace wb {

cudaError_t move_ref_dispatch(int semantics, const wacomm_b200_config &cfg,
                              const IntervalParams &P, const PackedArgs &A, const ParticleSoA &S,
                              const MoveLaunch &L, int blockSize, cudaStream_t stream) {
    const PackedView V = packed_view(A);
    if (semantics == SEM_HOST)
        return launch_move_soa<SEM_HOST>(cfg, P, V, S, L, blockSize, stream);
    return launch_move_soa<SEM_DEVICE>(cfg, P, V, S, L, blockSize, stream);
}

}  // namespace wb
