// krylov_fused_tr.cu -- instances of the one-kernel solve (krylov_fused.cuh): the transposed operator, FP64 and FP32.
#include "krylov_fused.cuh"

namespace ho2d {

cudaError_t fused_tr64(const MfOp<double>& op, const BicgVectors<double>& v, const FusedScratch& fs, int max_iter,
                     const Precond<double>& pc, KrylovScalars* sc, cudaStream_t s, bool* fits) {
    HO2D_FUSED_SWITCH(op.K, (fused_launch<KK, double, 0, true>(op, v, fs, max_iter, pc, sc, s, fits)));
}

cudaError_t fused_tr32(const MfOp<float>& op, const BicgVectors<float>& v, const FusedScratch& fs, int max_iter,
                     const Precond<float>& pc, KrylovScalars* sc, cudaStream_t s, bool* fits) {
    HO2D_FUSED_SWITCH(op.K, (fused_launch<KK, float, 0, true>(op, v, fs, max_iter, pc, sc, s, fits)));
}

}  // namespace ho2d
