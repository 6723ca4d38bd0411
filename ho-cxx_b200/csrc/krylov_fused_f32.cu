// krylov_fused_f32.cu -- instances of the one-kernel solve (krylov_fused.cuh): FP32 with exact and BF16 blocks.
#include "krylov_fused.cuh"

namespace ho2d {

cudaError_t fused_f32_exact(const MfOp<float>& op, const BicgVectors<float>& v, const FusedScratch& fs, int max_iter,
                     const Precond<float>& pc, KrylovScalars* sc, cudaStream_t s, bool* fits) {
    HO2D_FUSED_SWITCH(op.K, (fused_launch<KK, float, 0, false>(op, v, fs, max_iter, pc, sc, s, fits)));
}

cudaError_t fused_f32_bf16(const MfOp<float>& op, const BicgVectors<float>& v, const FusedScratch& fs, int max_iter,
                     const Precond<float>& pc, KrylovScalars* sc, cudaStream_t s, bool* fits) {
    HO2D_FUSED_SWITCH(op.K, (fused_launch<KK, float, 1, false>(op, v, fs, max_iter, pc, sc, s, fits)));
}

}  // namespace ho2d
