// krylov_fused_f64k.cu -- instances of the one-kernel solve (krylov_fused.cuh): FP64 with Kronecker-sum factors.
#include "krylov_fused.cuh"

namespace ho2d {

cudaError_t fused_f64_kron(const MfOp<double>& op, const BicgVectors<double>& v, const FusedScratch& fs, int max_iter,
                     const Precond<double>& pc, KrylovScalars* sc, cudaStream_t s, bool* fits) {
    HO2D_FUSED_SWITCH(op.K, (fused_launch<KK, double, 2, false>(op, v, fs, max_iter, pc, sc, s, fits)));
}

}  // namespace ho2d
