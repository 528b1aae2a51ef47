// Second pass of A': every IC column is the FP64 sum of its fibre's per-segment terms.
//
// A column's terms are taken by 8 lanes (lane = list position mod 8, so a lane's terms and
// their order do not depend on where slabs cut the list) and the 8 sums are added by a fixed
// butterfly: deterministic, no atomics.  The lanes read the position list in whole 32-byte
// sectors and keep 4 gathers each in flight.  One thread per column walks its terms in a chain
// of dependent loads and leaves most of the chip idle below some 100k columns, but needs fewer
// instructions for many short lists.  Measured, us, 8 lanes / one thread: 300 columns of 24
// terms 4.2 / 10.7, 3000 of 14 3.9 / 10.7, 30k of 14 8.3 / 12.9, 300k of 14 49 / 37, of 20
// 55 / 53, of 40 79 / 116, 1M of 14 153 / 102; 5000 columns of 80 terms 9.7 / 36.
#pragma once
#include "operator_pair.cuh"

namespace cgb {

constexpr int kFibreLanes = 8;

// lanes per column of a handle (a property of the handle: sums carry over from slab to slab)
inline int fibre_lanes(const cgb_op *op) {
    const int64_t f = op->nF;
    return op->n >= 20 * f || (f * op->nIC < 100000 && op->n >= 4 * f) ? kFibreLanes : 1;
}

namespace detail {

__device__ __forceinline__ double fibre_widen(double t) { return t; }
__device__ __forceinline__ double fibre_widen(float t) { return widen(t); }

// a + lane `sub`'s terms of the list positions [beg, end), in order; perm null: terms in list order
template <int G, class T>
__device__ __forceinline__ double fibre_lane_sum(const uint32_t *__restrict__ perm, const T *__restrict__ terms,
                                                 uint32_t beg, uint32_t end, int sub, double a) {
    if constexpr (G == 1) {
        uint32_t k = beg;
        for (; k + 8 <= end; k += 8) {
            uint32_t i[8];
            T t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) i[u] = perm ? __ldg(perm + k + u) : k + u;
#pragma unroll
            for (int u = 0; u < 8; ++u) t[u] = __ldg(terms + i[u]);
#pragma unroll
            for (int u = 0; u < 8; ++u) a += fibre_widen(t[u]);
        }
        for (; k < end; ++k) a += fibre_widen(__ldg(terms + (perm ? __ldg(perm + k) : k)));
        return a;
    }
    constexpr int U = 4;
    uint32_t k = (beg & ~(uint32_t)(G - 1)) + sub;
    if (k < beg) k += G;
    while (k < end) {
        uint32_t i[U];
        T t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const uint32_t kk = min(k + u * G, end - 1);
            i[u] = perm ? __ldg(perm + kk) : kk;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) t[u] = __ldg(terms + i[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (k + u * G < end) a += fibre_widen(t[u]);
        k += U * G;
    }
    return a;
}

template <int G>
__device__ __forceinline__ double fibre_reduce(double a) {
#pragma unroll
    for (int d = G / 2; d >= 1; d >>= 1) a += __shfl_xor_sync(0xffffffffu, a, d, G);
    return a;
}

// Slab s of S of the pass over all columns, in pass order (fib_order); running sums between
// slabs in accb [column][lane].  S == 1: the whole lists.
template <int G, class T>
__global__ void __launch_bounds__(256) k_fibre_pass(const OpDev P, const T *__restrict__ terms,
                                                    double *__restrict__ xout, const uint32_t *__restrict__ fib_slab,
                                                    double *__restrict__ accb, int s, int S) {
    const int64_t total = (int64_t)P.nF * P.nIC;
    const int sub = threadIdx.x & (G - 1);
    const int64_t step = (int64_t)gridDim.x * (256 / G);
    // whole warps stay in the loop: the butterfly takes every lane
    for (int64_t q0 = blockIdx.x * (256ll / G) + (threadIdx.x & ~31) / G; q0 < total; q0 += step) {
        const int64_t q = q0 + (threadIdx.x & 31) / G;
        const bool on = q < total;
        const int i = on ? (int)(q / P.nF) : 0;
        const int64_t fq = on ? q - (int64_t)i * P.nF : 0;
        uint32_t f = 0, beg = 0, end = 0;
        if (on) {
            if (S == 1) {
                f = P.fib_order[fq];
                beg = P.fib_ptr[f];
                end = P.fib_ptr[f + 1];
            } else {
                beg = fib_slab[(size_t)s * P.nF + fq];
                end = fib_slab[(size_t)(s + 1) * P.nF + fq];
                if (s == S - 1) f = P.fib_order[fq];
            }
        }
        const bool idle = !on || (s > 0 && s < S - 1 && beg == end);
        double a = s == 0 || idle ? 0.0 : accb[q * G + sub];
        a = fibre_lane_sum<G>(P.fib_perm, terms + (size_t)i * P.n, beg, end, sub, a);
        if (s == S - 1) {
            a = fibre_reduce<G>(a);
            if (on && sub == 0) {
                const int64_t c = (int64_t)i * P.nF + f;
                xout[c] = a * (double)P.eval[c];
            }
        } else if (!idle) {
            accb[q * G + sub] = a;
        }
    }
}

}  // namespace detail

template <class T>
int launch_fibre_pass(cgb_op *op, const T *terms, double *xout, double *accb, int s, int S, cudaStream_t st) {
    if (op->nIC == 0 || op->nF == 0) return CGB_OK;
    const int G = fibre_lanes(op);
    const int64_t total = (int64_t)op->nF * op->nIC, per = 256 / G;
    int64_t gb = (total + per - 1) / per;
    if (gb > op->nsm * 64) gb = op->nsm * 64;
    if (G == 1) detail::k_fibre_pass<1, T><<<(int)gb, 256, 0, st>>>(op->dev(), terms, xout, op->fib_slab, accb, s, S);
    else
        detail::k_fibre_pass<kFibreLanes, T><<<(int)gb, 256, 0, st>>>(op->dev(), terms, xout, op->fib_slab, accb, s, S);
    CGB_CUDA(cudaGetLastError());
    return CGB_OK;
}

}  // namespace cgb
