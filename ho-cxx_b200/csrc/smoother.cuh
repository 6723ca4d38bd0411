// smoother.cuh -- the fine smoother's element inverse on the row-parallel mapping (rows.cuh):
// exact blocks (or their transposes), BF16 blocks or Kronecker-sum factors, applied to one
// element vector.
#pragma once

#include <type_traits>

#include "rows.cuh"

namespace ho2d {

// The smoother's element data (BS): 0 = inverse blocks in T; 1 = inverse blocks as BF16 bit
// patterns (FP32 smoother); 2 = Kronecker-sum factors, with the exact blocks only for the
// elements the fit does not approximate well; 3 = the blocks of 0 applied transposed, read where
// they lie (the adjoint's solve without a transposed copy). Each element's data starts on a
// 16-byte boundary (padded_count). A warp's EPW blocks (or factor sets) are one
// contiguous span, copied into shared memory by one bulk copy when the span is at most
// 26 KB (so a CTA's four spans leave room for two CTAs per SM); larger blocks are read
// from global memory directly.
template <int K, typename T, int BS>
struct PostRows {
    using DT = typename std::conditional<BS == 1, unsigned short, T>::type;
    static constexpr int K2 = K * K, K4 = K2 * K2;
    static constexpr int STRIDE = padded_count(K4, (int)sizeof(DT));  // values of DT per element
    static constexpr int KF = 4 * K2 + 2 * K;                      // Kronecker factors per element
    static constexpr int KFS = padded_count(KF, (int)sizeof(T));
    static constexpr int XSTRIDE = padded_count(K4, (int)sizeof(T));  // compact exact blocks (BS 2)
    // bytes of one element's staged data: its inverse block, or (BS 2) its factors
    static constexpr int ELEM = BS == 2 ? KFS * (int)sizeof(T) : STRIDE * (int)sizeof(DT);
    static constexpr int SPAN = Rows<K>::EPW * ELEM;  // bytes per warp
    static constexpr bool kStage = SPAN <= 26 * 1024;
    static constexpr int SMEM = kStage ? Rows<K>::WARPS * SPAN : 0;  // dynamic shared memory
};

__device__ __forceinline__ float block_value(unsigned short b) { return __uint_as_float((unsigned)b << 16); }
template <typename T>
__device__ __forceinline__ T block_value(T v) {
    return v;
}

// K consecutive block values (row t of one r-slice of an element block, [rs][ij] layout),
// widened to T; vector loads as wide as the slice's alignment allows (its offset is a
// multiple of K values from a 16-byte-aligned block start).
template <int K, typename T, typename DT>
__device__ __forceinline__ void load_slice(const DT* p, T (&v)[K]) {
    constexpr int AL = (K * (int)sizeof(DT)) % 16 == 0 ? 16 : ((K * (int)sizeof(DT)) % 8 == 0 ? 8 : ((K * (int)sizeof(DT)) % 4 == 0 ? 4 : (int)sizeof(DT)));
    if constexpr (sizeof(DT) == 2) {
        if constexpr (AL >= 4) {
#pragma unroll
            for (int i = 0; i < K; i += 2) {
                const unsigned w = *reinterpret_cast<const unsigned*>(p + i);
                v[i] = __uint_as_float(w << 16);
                v[i + 1] = __uint_as_float(w & 0xffff0000u);
            }
        } else {
#pragma unroll
            for (int i = 0; i < K; ++i) v[i] = block_value(p[i]);
        }
    } else if constexpr (AL == 16 && sizeof(DT) == 4) {
#pragma unroll
        for (int i = 0; i < K; i += 4) {
            const float4 q = *reinterpret_cast<const float4*>(p + i);
            v[i] = q.x;
            v[i + 1] = q.y;
            v[i + 2] = q.z;
            v[i + 3] = q.w;
        }
    } else if constexpr (AL >= 8 && sizeof(DT) == 4) {
#pragma unroll
        for (int i = 0; i < K; i += 2) {
            const float2 q = *reinterpret_cast<const float2*>(p + i);
            v[i] = q.x;
            v[i + 1] = q.y;
        }
    } else if constexpr (AL == 16 && sizeof(DT) == 8) {
#pragma unroll
        for (int i = 0; i < K; i += 2) {
            const double2 q = *reinterpret_cast<const double2*>(p + i);
            v[i] = q.x;
            v[i + 1] = q.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < K; ++i) v[i] = T(p[i]);
    }
}

// acc[i] = sum_r blk[r][t K + i] sr[r] over the K^2 values r of the element's residual sr
// (shared memory): row t of D^-1 sr.
template <int K, typename T, typename DT>
__device__ __forceinline__ void block_rows(const DT* blk, const T* sr, int t, T (&acc)[K]) {
    constexpr int K2 = K * K;
#pragma unroll
    for (int i = 0; i < K; ++i) acc[i] = T(0);
#pragma unroll 4
    for (int r = 0; r < K2; ++r) {
        T m[K];
        load_slice<K, T, DT>(blk + r * K2 + t * K, m);
        const T s = sr[r];
#pragma unroll
        for (int i = 0; i < K; ++i) acc[i] += m[i] * s;
    }
}

// The same with the block's transpose: acc[i] = sum_r blk[t K + i][r] sr[r], r in the same order, so
// the result has the bits that block_rows gives on a transposed copy. Each thread streams K rows of
// the block, its neighbours the next K, so a warp's loads fall into many lines at once (the cost
// stands at Solver::adjoint_blocks).
template <int K, typename T>
__device__ __forceinline__ void block_rows_transposed(const T* blk, const T* sr, int t, T (&acc)[K]) {
    constexpr int K2 = K * K;
#pragma unroll
    for (int i = 0; i < K; ++i) acc[i] = T(0);
#pragma unroll 4
    for (int r = 0; r < K2; ++r) {
        const T s = sr[r];
#pragma unroll
        for (int i = 0; i < K; ++i) acc[i] += blk[(t * K + i) * K2 + r] * s;
    }
}

// The smoother's element inverse M (exact block, BF16 block or Kronecker-sum factors)
// applied to one element vector held in shared memory (srow, K^2 values, [j][i]): row t of
// M srow into acc. For BS 2 the transposes are warp-collective, so every lane runs them;
// zb is a K x K scratch of the element. Warp-collective.
template <int K, typename T, int BS>
__device__ __forceinline__ void smoother_rows(const MfOp<T>& op, const typename PostRows<K, T, BS>::DT* blk,
                                              const T* fk, int kx, const T* srow, T (&zb)[K][K], int t, bool act,
                                              T (&acc)[K]) {
    using PS = PostRows<K, T, BS>;
    constexpr int K2 = K * K;
    if constexpr (BS == 2) {
        // exact block where the fit falls back, Kronecker-sum step (fast diagonalisation,
        // the element body of kron_apply.cuh by rows) for the others
        const bool kr = act && kx < 0;
        if (act && kx >= 0) block_rows<K, T, T>(op.kron_exact + (size_t)kx * PS::XSTRIDE, srow, t, acc);
        const T *vx = fk, *vxi = fk + K2, *vy = fk + 2 * K2, *vyi = fk + 3 * K2, *lx = fk + 4 * K2, *ly = lx + K;
        T c1[K], r1[K], r2[K], c2[K], c3[K], r3[K];
        // column t of Vy^-1 R
#pragma unroll
        for (int j = 0; j < K; ++j) {
            T s = T(0);
            if (kr) {
#pragma unroll
                for (int l = 0; l < K; ++l) s += vyi[j * K + l] * srow[l * K + t];
            }
            c1[j] = s;
        }
        col_to_row<K, T>(zb, c1, r1, t, kr);
        // row t of (Vy^-1 R Vx^-T) ./ (ly_t + lx_i)
#pragma unroll
        for (int i = 0; i < K; ++i) {
            T s = T(0);
            if (kr) {
#pragma unroll
                for (int k = 0; k < K; ++k) s += r1[k] * vxi[i * K + k];
                s = s / (ly[t] + lx[i]);
            }
            r2[i] = s;
        }
        __syncwarp();  // zb is rewritten next
        rows_to_col<K, T>(zb, r2, c2, t, kr);
        // column t of Vy (that), then row t of the product with Vx^T
#pragma unroll
        for (int j = 0; j < K; ++j) {
            T s = T(0);
            if (kr) {
#pragma unroll
                for (int l = 0; l < K; ++l) s += vy[j * K + l] * c2[l];
            }
            c3[j] = s;
        }
        __syncwarp();
        col_to_row<K, T>(zb, c3, r3, t, kr);
        if (kr) {
#pragma unroll
            for (int i = 0; i < K; ++i) {
                T s = T(0);
#pragma unroll
                for (int k = 0; k < K; ++k) s += r3[k] * vx[i * K + k];
                acc[i] = s;
            }
        }
        __syncwarp();  // zb may be reused by the caller
    } else if constexpr (BS == 3) {
        if (act) block_rows_transposed<K, T>(blk, srow, t, acc);
    } else {
        if (act) block_rows<K, T, typename PS::DT>(blk, srow, t, acc);
    }
}

}  // namespace ho2d
