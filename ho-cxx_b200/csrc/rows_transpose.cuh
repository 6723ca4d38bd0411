// rows_transpose.cuh -- the transposed Poisson operator y = A^T x on the row-parallel mapping
// (rows.cuh): the reverse of row_apply_core, phase by phase.
//
// Reversed, an element's map ends in adjoints of its neighbours' face traces. They go into
// the neighbours' incoming slots ([N][K][4], the scatter table of the forward traces: the
// neighbour's point that meets this face point), one writer each, and a second launch adds
// an element's slots through the transposed trace map. So y = A^T x takes two launches:
// row_transpose_own (own part + slots), then row_transpose_gather.
//
// Boundary slots are never written and must be zero.
#pragma once

#include "rows.cuh"

namespace ho2d {

// Own part of A^T z, row t of element `el` (`z` = row t of the operand), into `own`; the
// adjoints of the neighbours' traces into sv (values) and sg (normal derivatives).
// Warp-collective.
template <int K, typename T>
__device__ __forceinline__ void row_transpose_own(const MfOp<T>& op, const T (&z)[K], RowScratch<K, T>& sm,
                                                  const RowIdx<K>& ix, T* __restrict__ sv, T* __restrict__ sg,
                                                  T (&own)[K]) {
    const PoisGeom<T>& g = op.g;
    const DevBases<T>& b = op.b;
    const int t = ix.t, lw = ix.lw;
    const bool act = ix.active;
    T g11[K], g12r[K], g22[K], g12c[K], fa[4], fb[4], nfa[4], nfb[4];
    int code[4], dst[4];
    if (act) {
        const size_t e2 = (size_t)ix.el * K * K, q4 = ((size_t)ix.el * K + t) * 4;
        load_row<K, T>(g.G11 + e2 + t * K, g11);
        load_row<K, T>(g.G12 + e2 + t * K, g12r);
        load_col<K, T>(g.G22 + e2 + t, g22);
        load_col<K, T>(g.G12 + e2 + t, g12c);
        load4<T>(g.fa + q4, fa);
        load4<T>(g.fb + q4, fb);
        load4<T>(g.nfa + q4, nfa);
        load4<T>(g.nfb + q4, nfb);
        load4i(g.code + ix.el * 4, code);
        load4i(g.scat + q4, dst);
    } else {
#pragma unroll
        for (int i = 0; i < K; ++i) g11[i] = g12r[i] = g22[i] = g12c[i] = T(0);
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            fa[f] = fb[f] = nfa[f] = nfb[f] = T(0);
            code[f] = dst[f] = -1;
        }
    }
    T zc[K];
    rows_to_col<K, T>(sm.tr[0][lw], z, zc, t, act);
    if (!act) {
#pragma unroll
        for (int j = 0; j < K; ++j) zc[j] = T(0);
    }
    // divergence reversed: adjoints of the flux jumps (face point t) and of the contravariant
    // gradient, a along row t and b down column t
    T lc[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int i = 0; i < K; ++i) {
        lc[0] += z[i] * b.gR[i * 2 + 0];
        lc[1] += z[i] * b.gR[i * 2 + 1];
        lc[2] += zc[i] * b.gR[i * 2 + 0];
        lc[3] += zc[i] * b.gR[i * 2 + 1];
    }
    T la[K], lb[K];
#pragma unroll
    for (int d = 0; d < K; ++d) {
        T sa = T(0), sb = T(0);
#pragma unroll
        for (int i = 0; i < K; ++i) {
            sa += z[i] * b.D[d * K + i];
            sb += zc[i] * b.D[d * K + i];
        }
        la[d] = sa - lc[0] * b.sbb[d * 2 + 0] - lc[1] * b.sbb[d * 2 + 1];
        lb[d] = sb - lc[2] * b.sbb[d * 2 + 0] - lc[3] * b.sbb[d * 2 + 1];
    }
    T lbr[K], lac[K], ldx[K], lde[K];
    col_to_row<K, T>(sm.tr[1][lw], lb, lbr, t, act);  // (its barrier also frees tr[0])
    rows_to_col<K, T>(sm.tr[0][lw], la, lac, t, act);
#pragma unroll
    for (int i = 0; i < K; ++i) {
        ldx[i] = act ? la[i] * g11[i] + lbr[i] * g12r[i] : T(0);
        lde[i] = act ? lb[i] * g22[i] + lac[i] * g12c[i] : T(0);
    }
    // common values and fluxes of face point t reversed
    T lcom[4] = {T(0), T(0), T(0), T(0)};
#pragma unroll
    for (int i = 0; i < K; ++i) {
        lcom[0] += ldx[i] * b.gR[i * 2 + 0];
        lcom[1] += ldx[i] * b.gR[i * 2 + 1];
        lcom[2] += lde[i] * b.gR[i * 2 + 0];
        lcom[3] += lde[i] * b.gR[i * 2 + 1];
    }
    T tv[4], tg[4], nv[4], ng[4];  // adjoints of the own and of the neighbour's traces
    bool any_rev = false;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        tv[f] = -lcom[f];
        tg[f] = nv[f] = ng[f] = T(0);
        if (!act) continue;
        if (code[f] <= -2) {  // Neumann: zero common flux; the common-value system below
            sm.com[lw][f][t] = lcom[f];
            continue;
        }
        const bool in = code[f] >= 0;
        const T lfl = in ? T(0.5) * lc[f] : lc[f];
        const T ldv = lfl * fa[f];
        T cross = -lfl * fb[f];
        tg[f] = ldv;
        tv[f] -= ldv * b.gp[f & 1];
        lcom[f] += ldv * b.gp[f & 1];
        if (in) {
            const int nijp = code[f] & 3, rev = code[f] >> 2;
            const T lfn = T(0.5) * T(2 * ((f + nijp) % 2) - 1) * lc[f];
            const T ldn = lfn * nfa[f], crn = -lfn * nfb[f];
            const T gpn = (nijp & 1) ? b.gp[1] : b.gp[0];
            ng[f] = ldn;
            nv[f] = -ldn * gpn;
            lcom[f] += ldn * gpn;
            if (rev) {
                any_rev = true;
                sm.nr[lw][f][t] = crn;
            } else {
                cross += crn;
            }
        }
        sm.com[lw][f][t] = cross;
    }
    __syncwarp();
    // the face derivative of the common values reversed (entry m = t of each face), on both
    // sides of the face; the Neumann system's transpose
    if (act) {
        T Dr[K];
#pragma unroll
        for (int k = 0; k < K; ++k) Dr[k] = b.D[t * K + k];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            if (code[f] <= -2) {
                const T* mi = g.minv + (size_t)(-2 - code[f]) * K * K + t;
                T acc = T(0);
#pragma unroll
                for (int k = 0; k < K; ++k) acc += __ldg(mi + k * K) * sm.com[lw][f][k];
                tg[f] -= fa[f] * acc;
                tv[f] += fa[f] * acc * b.gp[f & 1];
                continue;
            }
            T acc = T(0);
#pragma unroll
            for (int k = 0; k < K; ++k) acc += sm.com[lw][f][k] * Dr[k];
            lcom[f] += acc;
        }
        if (any_rev) {
            T Dn[K];
#pragma unroll
            for (int k = 0; k < K; ++k) Dn[k] = b.D[(K - 1 - t) * K + (K - 1 - k)];
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                if (code[f] < 4) continue;  // interior face met in the reverse direction
                T acc = T(0);
#pragma unroll
                for (int k = 0; k < K; ++k) acc += sm.nr[lw][f][k] * Dn[k];
                lcom[f] += acc;
            }
        }
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            if (code[f] < 0) continue;  // interior: com = (own + neighbour's trace) / 2
            tv[f] += T(0.5) * lcom[f];
            nv[f] += T(0.5) * lcom[f];
            sv[dst[f]] = nv[f];
            sg[dst[f]] = ng[f];
        }
    }
    // derivatives and own traces -> the element's own values
    T oc[K], ocr[K];
#pragma unroll
    for (int d = 0; d < K; ++d) {
        T sr = T(0), sc = T(0);
#pragma unroll
        for (int i = 0; i < K; ++i) {
            sr += ldx[i] * b.D[d * K + i];
            sc += lde[i] * b.D[d * K + i];
        }
        own[d] = sr + tv[0] * b.sbb[d * 2 + 0] + tg[0] * b.sbgb[d * 2 + 0] + tv[1] * b.sbb[d * 2 + 1] +
                 tg[1] * b.sbgb[d * 2 + 1];
        oc[d] = sc + tv[2] * b.sbb[d * 2 + 0] + tg[2] * b.sbgb[d * 2 + 0] + tv[3] * b.sbb[d * 2 + 1] +
                tg[3] * b.sbgb[d * 2 + 1];
    }
    // (tr[1]'s rows were read before the barrier of the la transpose)
    col_to_row<K, T>(sm.tr[1][lw], oc, ocr, t, act);
    if (act) {
#pragma unroll
        for (int i = 0; i < K; ++i) own[i] += ocr[i];
    }
    __syncwarp();  // the scratch may be rewritten by the caller's next use
}

// Second half: y (row t of the own part) += the transposed traces of face point t's incoming
// slots, values v and normal derivatives d. Warp-collective.
template <int K, typename T>
__device__ __forceinline__ void transpose_traces(const DevBases<T>& b, const T (&v)[4], const T (&d)[4], T (&buf)[K][K],
                                                 const RowIdx<K>& ix, T (&y)[K]) {
    T c[K], r[K];
#pragma unroll
    for (int j = 0; j < K; ++j)
        c[j] = v[2] * b.sbb[j * 2 + 0] + d[2] * b.sbgb[j * 2 + 0] + v[3] * b.sbb[j * 2 + 1] + d[3] * b.sbgb[j * 2 + 1];
    col_to_row<K, T>(buf, c, r, ix.t, ix.active);
    if (ix.active) {
#pragma unroll
        for (int i = 0; i < K; ++i)
            y[i] += r[i] + (v[0] * b.sbb[i * 2 + 0] + d[0] * b.sbgb[i * 2 + 0] + v[1] * b.sbb[i * 2 + 1] +
                            d[1] * b.sbgb[i * 2 + 1]);
    }
    __syncwarp();  // buf may be rewritten by the caller's next use
}

// The second half with the own part and the slots from global memory.
template <int K, typename T>
__device__ __forceinline__ void row_transpose_gather(const DevBases<T>& b, const T* own, const T* sv, const T* sg,
                                                     T (&buf)[K][K], const RowIdx<K>& ix, T (&y)[K]) {
    T v[4] = {T(0), T(0), T(0), T(0)}, d[4] = {T(0), T(0), T(0), T(0)};
    if (ix.active) {
        const size_t q4 = ((size_t)ix.el * K + ix.t) * 4;
        load4<T>(sv + q4, v);
        load4<T>(sg + q4, d);
        load_row<K, T>(own + (size_t)ix.el * K * K + ix.t * K, y);
    }
    transpose_traces<K, T>(b, v, d, buf, ix, y);
}

}  // namespace ho2d
