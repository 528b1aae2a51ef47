// Reduced-precision A*x and A'*y of FP32 vectors with the IC table in shared memory.
//
// The gathering kernels (operator_mixed.cuh) spend most of their instructions on forming the
// coefficients of a batch (scans, shuffles) and on rows of two voxels per warp; keeping their
// structure and only moving the table to shared memory gained nothing (measured).  Here the
// runs (smem_ff.cuh) get their coefficients in one pass, a warp takes four voxels, 8 lanes and
// four samples per load each, and the table (BF16, FP16 or FP32) stays in shared memory for
// the launch, in chunks of the samples where it does not fit.  FP32 accumulation
// and FP16 lengths as in the gathering kernels; only the order of the sums differs, so the
// solvers (whose FP64 iterates would show it) stay on those, and FP32 products come here.
// The passes are bound by the conversions and FMAs of the runs (a quad of 16-bit values costs two
// conversions and two packed FMAs for its one load).  Measured on a tractogram of 15 M segments x
// 145 samples: FP16 A 693 -> 298 us and 78 for the coefficients, A' 842 -> 395 us; FP32 (two
// chunks) A 679 -> 559 us in all and A' 975 -> 764.
#pragma once
#include "operator_mixed.cuh"
#include "smem_ff.cuh"

namespace cgb {

struct MixPlan {
    int nq, nc, cs;      // quads of samples per lane, chunks of 32 * nq samples, row stride (elements)
    char *img;           // [nc][nIC * ndirs][cs] (null: no room for the buffers)
    float *coef;         // [nIC * nruns]
    float *part;         // [nIC * nruns][nc] (nc > 1)
    double *epart;       // [EC and ISO columns][nc] (nc > 1)
    StreamOrder order;   // of the products, which share the buffers
    size_t bytes;        // of the handle's, held here
};

constexpr int kMixThreads = 768;

namespace detail {

// four consecutive samples of a table row
template <class LT>
struct Quad {
    __device__ static __forceinline__ void conv(uint2 u, f2 &a, f2 &b) {
        a = LutPair<LT>::conv(u.x);
        b = LutPair<LT>::conv(u.y);
    }
    __device__ static __forceinline__ void lds(const LT *p, f2 &a, f2 &b) {
        conv(*reinterpret_cast<const uint2 *>(p), a, b);
    }
    __device__ static __forceinline__ void ldg(const LT *p, f2 &a, f2 &b) {
        conv(__ldg(reinterpret_cast<const uint2 *>(p)), a, b);
    }
};
template <>
struct Quad<float> {
    __device__ static __forceinline__ void lds(const float *p, f2 &a, f2 &b) {
        const ulonglong2 u = *reinterpret_cast<const ulonglong2 *>(p);
        a = u.x;
        b = u.y;
    }
    __device__ static __forceinline__ void ldg(const float *p, f2 &a, f2 &b) {
        const ulonglong2 u = __ldg(reinterpret_cast<const ulonglong2 *>(p));
        a = u.x;
        b = u.y;
    }
};

struct SmMixArgs {
    const uint32_t *vperm, *run_ptr, *run_seg;
    const uint16_t *run_o;
    int64_t n, nruns;
    const void *img;
    int nIC, ndirs, nS, nV, nc, p0, p1, v0, v1;
    const uint32_t *ec_ptr, *ec_col, *iso_ptr, *iso_col;
    const uint16_t *ec_o;
    const void *lutEC, *lutISO;  // rows of stride nSp
    int nSp, nEC, nISO;
    int64_t ec_base, iso_base, nE, nISOv;
    const float *x;              // A: columns
    float *y;                    // A: rows
    const float *z;              // A': rows
    double *xout;                // A': columns
    const __half *seg_l16;       // lengths times 1 / l_scale (FP32 table: null, and seg_l)
    const float *seg_l;
    float l_scale;
    float *coef, *part, *scratch;
    double *epart;
    int vec_ok;                  // rows are 16-byte aligned and a multiple of four samples
};

template <bool F32>
__device__ __forceinline__ float mix_length(const SmMixArgs &A, uint32_t j) {
    return F32 ? A.seg_l[j] : __half2float(A.seg_l16[j]) * A.l_scale;
}

// a + b in s with its rounding error in e (0 when the sum is not finite): with an FP32 table the
// last sums of a dot product are those that show, and the term l * (s + e) rounds once
__device__ __forceinline__ float sum_err(float a, float b, float &e) {
    const float s = a + b, bb = s - a;
    e = (a - (s - bb)) + (b - bb);
    if (!(fabsf(e) <= 3.0e38f)) e = 0.f;
    return s;
}

// quad of register k: odd groups take neighbouring quads swapped (16-bit rows are a multiple of 128
// bytes apart, and the two groups of a half-warp then read the two halves of a line)
template <class LT, int NQ>
__device__ __forceinline__ int quad_of(int k, int par) {
    return sizeof(LT) == 2 && (k ^ 1) < NQ ? k ^ par : k;
}

template <class LT, int NQ>
__global__ void __launch_bounds__(kMixThreads, 1) k_fwd_mix_smem(const __grid_constant__ SmMixArgs A, int cs) {
    extern __shared__ __align__(16) float smraw[];
    const LT *tab = reinterpret_cast<const LT *>(smraw);
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & 7, lg = lane >> 3, par = lg & 1;
    const int chunk = blockIdx.x % A.nc, cta = blockIdx.x / A.nc, ncta = gridDim.x / A.nc;
    const int rows = A.nIC * A.ndirs, words = rows * cs * (int)sizeof(LT) / 4;
    fill_table<kMixThreads>(smraw, reinterpret_cast<const float *>(A.img) + (size_t)chunk * words, words);
    const int s_base = chunk * 32 * NQ;
    const int last = A.p1 - A.p0, stride = ncta * (kMixThreads / 8);
    const int first = ((int)(threadIdx.x >> 5) * ncta + cta) * 4;
    auto voxel = [&](int pos) {
        int v = -1;
        if (pos < last) v = (int)A.vperm[A.p0 + pos];
        return v < A.v0 || v >= A.v1 ? -1 : v;
    };
    int v = voxel(first + lg), vn = voxel(first + lg + stride);
    uint32_t rb = v >= 0 ? A.run_ptr[v] : 0u, re = v >= 0 ? A.run_ptr[v + 1] : 0u;
    fill_wait();
    for (int w = first; w < last; w += stride) {
        const uint32_t rbn = vn >= 0 ? A.run_ptr[vn] : 0u, ren = vn >= 0 ? A.run_ptr[vn + 1] : 0u;
        const int vnn = voxel(w + lg + 2 * stride);
        const uint32_t eb = v >= 0 && A.nEC ? A.ec_ptr[v] : 0u, ee = v >= 0 && A.nEC ? A.ec_ptr[v + 1] : 0u;
        const uint32_t ib = v >= 0 && A.nISO ? A.iso_ptr[v] : 0u, ie = v >= 0 && A.nISO ? A.iso_ptr[v + 1] : 0u;
        for (uint32_t j = rbn + 32 * sub; j < ren; j += 256) prefetch_l2(A.coef + j);
        for (uint32_t j = rbn + 64 * sub; j < ren; j += 512) prefetch_l2(A.run_o + j);
        int nb = (int)(re - rb + 7) / 8;
        nb = max(nb, __shfl_xor_sync(full, nb, 8));
        nb = max(nb, __shfl_xor_sync(full, nb, 16));
        f2 a0[NQ], a1[NQ];
#pragma unroll
        for (int k = 0; k < NQ; ++k) a0[k] = a1[k] = 0ull;
        auto add = [&](float c, const LT *L) {
            const f2 c2 = f2_pack(c, c);
#pragma unroll
            for (int k = 0; k < NQ; ++k) {
                f2 u, t;
                Quad<LT>::lds(L + 32 * quad_of<LT, NQ>(k, par), u, t);
                a0[k] = f2_fma(c2, u, a0[k]);
                a1[k] = f2_fma(c2, t, a1[k]);
            }
        };
#pragma unroll 1
        for (int i = 0; i < A.nIC; ++i) {
            const float *cf = A.coef + (size_t)i * A.nruns;
            uint32_t j = rb + sub;
            float nc = j < re ? cf[j] : 0.f;
            uint32_t no = j < re ? A.run_o[j] : 0u;
#pragma unroll 1
            for (int it = 0; it < nb; ++it) {
                const float c = nc;
                const unsigned row = ((unsigned)(i * A.ndirs) + no) * (unsigned)cs;
                j += 8;
                nc = j < re ? cf[j] : 0.f;
                no = j < re ? A.run_o[j] : 0u;
                unsigned f = __ballot_sync(full, c != 0.f);
                f |= f >> 16;
                f = (f | f >> 8) & 0xffu;
                if (f == 0xffu) {
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const float ct = __shfl_sync(full, c, t, 8);
                        add(ct, tab + __shfl_sync(full, row, t, 8) + 4 * sub);
                    }
                } else {
#pragma unroll 1
                    while (f) {
                        const int t = __ffs(f) - 1;
                        f &= f - 1;
                        const float ct = __shfl_sync(full, c, t, 8);
                        add(ct, tab + __shfl_sync(full, row, t, 8) + 4 * sub);
                    }
                }
            }
        }
        // EC and ISO elements, (element, response) by (element, response); rows from L1 / L2
        const int te = (int)(ee - eb) * A.nEC, tt = te + (int)(ie - ib) * A.nISO;
        int m = max(tt, __shfl_xor_sync(full, tt, 8));
        m = max(m, __shfl_xor_sync(full, m, 16));
#pragma unroll 1
        for (int b = 0; b < m; b += 8) {
            const int q = b + sub;
            float c = 0.f;
            const LT *row = (const LT *)(A.nISO ? A.lutISO : A.lutEC);
            if (q < te) {
                const uint32_t j = eb + q / A.nEC;
                const int i = q % A.nEC;
                row = (const LT *)A.lutEC + (size_t)((unsigned)(i * A.ndirs) + A.ec_o[j]) * A.nSp;
                c = A.x[A.ec_base + i * A.nE + A.ec_col[j]];
            } else if (q < tt) {
                const int i = (q - te) % A.nISO;
                row = (const LT *)A.lutISO + (size_t)i * A.nSp;
                c = A.x[A.iso_base + i * A.nISOv + A.iso_col[ib + (q - te) / A.nISO]];
            }
            const int cnt = min(m - b, 8);
#pragma unroll 1
            for (int t = 0; t < cnt; ++t) {
                const float ct = __shfl_sync(full, c, t, 8);
                const LT *L = reinterpret_cast<const LT *>(
                                  __shfl_sync(full, reinterpret_cast<unsigned long long>(row), t, 8)) + s_base + 4 * sub;
                const f2 c2 = f2_pack(ct, ct);
#pragma unroll
                for (int k = 0; k < NQ; ++k) {
                    const int o = 32 * quad_of<LT, NQ>(k, par);
                    if (s_base + o + 4 * sub < A.nSp) {
                        f2 u, s;
                        Quad<LT>::ldg(L + o, u, s);
                        a0[k] = f2_fma(c2, u, a0[k]);
                        a1[k] = f2_fma(c2, s, a1[k]);
                    }
                }
            }
        }
        if (v >= 0) {
#pragma unroll
            for (int k = 0; k < NQ; ++k) {
                const int s = s_base + 4 * (sub + 8 * quad_of<LT, NQ>(k, par));
                if (s >= A.nS) continue;
                float o[4];
                f2_unpack(a0[k], o[0], o[1]);
                f2_unpack(a1[k], o[2], o[3]);
                float *p = A.y + (size_t)v * A.nS + s;
                if (A.vec_ok) {
                    *reinterpret_cast<float4 *>(p) = make_float4(o[0], o[1], o[2], o[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (s + e < A.nS) p[e] = o[e];
                }
            }
        }
        __syncwarp();
        v = vn;
        vn = vnn;
        rb = rbn;
        re = ren;
    }
}

// A' parts of the runs and of the EC / ISO elements; eight runs at a time as in k_adj_smem
template <class LT, int NQ>
__global__ void __launch_bounds__(kMixThreads, 1) k_adj_mix_smem(const __grid_constant__ SmMixArgs A, int cs) {
    extern __shared__ __align__(16) float smraw[];
    const LT *tab = reinterpret_cast<const LT *>(smraw);
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & 7, lg = lane >> 3, par = lg & 1;
    const int chunk = blockIdx.x % A.nc, cta = blockIdx.x / A.nc, ncta = gridDim.x / A.nc;
    const int rows = A.nIC * A.ndirs, words = rows * cs * (int)sizeof(LT) / 4;
    fill_table<kMixThreads>(smraw, reinterpret_cast<const float *>(A.img) + (size_t)chunk * words, words);
    const int s_base = chunk * 32 * NQ;
    const int last = A.p1 - A.p0, stride = ncta * (kMixThreads / 8);
    const int first = ((int)(threadIdx.x >> 5) * ncta + cta) * 4;
    auto voxel = [&](int pos) {
        int v = -1;
        if (pos < last) v = (int)A.vperm[A.p0 + pos];
        return v < A.v0 || v >= A.v1 ? -1 : v;
    };
    int v = voxel(first + lg), vn = voxel(first + lg + stride);
    uint32_t rb = v >= 0 ? A.run_ptr[v] : 0u, re = v >= 0 ? A.run_ptr[v + 1] : 0u;
    const uint32_t own = (uint32_t)((sub & 1) * 4 + (sub >> 1));  // this lane's run of a batch
    unsigned on = rb + own < re ? A.run_o[rb + own] : 0u;
    const bool whole = A.nc == 1;  // the dot products are complete: straight to the segments' terms
    uint32_t sn = 0, en = 0;
    auto segs = [&](uint32_t j, bool ok) {
        if (!whole) return;
        sn = ok ? __ldg(A.run_seg + j) : 0u;
        en = ok ? __ldg(A.run_seg + j + 1) : 0u;
    };
    segs(rb + own, rb + own < re);
    fill_wait();
    for (int w = first; w < last; w += stride) {
        const uint32_t rbn = vn >= 0 ? A.run_ptr[vn] : 0u, ren = vn >= 0 ? A.run_ptr[vn + 1] : 0u;
        const int vnn = voxel(w + lg + 2 * stride);
        f2 z0[NQ], z1[NQ];
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            const int s = s_base + 4 * (sub + 8 * quad_of<LT, NQ>(k, par));
            float o[4] = {0.f, 0.f, 0.f, 0.f};
            if (v >= 0 && s < A.nS) {
                const float *p = A.z + (size_t)v * A.nS + s;
                if (A.vec_ok) {
                    const float4 t = *reinterpret_cast<const float4 *>(p);
                    o[0] = t.x;
                    o[1] = t.y;
                    o[2] = t.z;
                    o[3] = t.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (s + e < A.nS) o[e] = p[e];
                }
            }
            z0[k] = f2_pack(o[0], o[1]);
            z1[k] = f2_pack(o[2], o[3]);
        }
        if (vn >= 0 && s_base + 32 * sub < A.nS && 32 * sub < 32 * NQ) prefetch_l2(A.z + (size_t)vn * A.nS + s_base + 32 * sub);
        for (uint32_t j = rbn + 64 * sub; j < ren; j += 512) prefetch_l2(A.run_o + j);
        int most = (int)(re - rb);
        most = max(most, __shfl_xor_sync(full, most, 8));
        most = max(most, __shfl_xor_sync(full, most, 16));
        if (most == 0) {
            on = rbn + own < ren ? __ldg(A.run_o + rbn + own) : 0u;
            segs(rbn + own, rbn + own < ren);
        }
#pragma unroll 1
        for (int b = 0; b < most; b += 8) {
            const uint32_t j = rb + b + own;
            const bool valid = j < re;
            const unsigned o = valid ? on : 0u;
            const uint32_t jn = b + 8 < most ? j + 8 : rbn + own;
            const bool okn = jn < (b + 8 < most ? re : ren);
            on = okn ? __ldg(A.run_o + jn) : 0u;
            const uint32_t sb = sn, se = en;
            const float l0 = whole && valid ? mix_length<sizeof(LT) == 4>(A, sb) : 0.f;
            segs(jn, okn);
#pragma unroll 1
            for (int i = 0; i < A.nIC; ++i) {
                const unsigned row = ((unsigned)(i * A.ndirs) + o) * (unsigned)cs;
                f2 M = 0ull, N = 0ull;  // N the first four, M the others (as k_adj_smem)
#pragma unroll 1
                for (int u = 0; u < 2; ++u) {
                    N = M;
                    M = 0ull;
                    if (u && b + 4 >= most) break;
                    f2 P[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const LT *L = tab + __shfl_sync(full, row, ((q ^ (sub >> 1)) << 1) + u, 8) + 4 * sub;
                        P[q] = 0ull;
                        f2 R = 0ull;  // FP32 table: two chains, the rounding of a chain grows with its length
#pragma unroll
                        for (int k = 0; k < NQ; ++k) {
                            f2 a, c;
                            Quad<LT>::lds(L + 32 * quad_of<LT, NQ>(k, par), a, c);
                            P[q] = f2_fma(a, z0[k], P[q]);
                            if (sizeof(LT) == 4) R = f2_fma(c, z1[k], R);
                            else P[q] = f2_fma(c, z1[k], P[q]);
                        }
                        if (sizeof(LT) == 4) P[q] = f2_add(P[q], R);
                    }
#pragma unroll
                    for (int h = 2, d = 4; h >= 1; h /= 2, d /= 2)
#pragma unroll
                        for (int g = 0; g < h; ++g) P[g] = f2_add(P[g], __shfl_xor_sync(full, P[g + h], d, 8));
                    M = P[0];
                }
                const bool odd = (sub & 1) != 0;
                const f2 got = __shfl_xor_sync(full, odd ? N : M, 1, 8);
                float t0, t1;
                f2_unpack(f2_add(odd ? M : N, got), t0, t1);
                if (!valid) continue;
                if (whole) {
                    float *out = A.scratch + (size_t)i * A.n;
                    float e = 0.f;
                    const float t = sizeof(LT) == 4 ? sum_err(t0, t1, e) : t0 + t1;
                    out[sb] = fmaf(l0, t, l0 * e);
                    for (uint32_t g = sb + 1; g < se; ++g) {
                        const float l = mix_length<sizeof(LT) == 4>(A, g);
                        out[g] = fmaf(l, t, l * e);
                    }
                } else {
                    A.part[((size_t)i * A.nruns + j) * A.nc + chunk] = t0 + t1;
                }
            }
        }
        uint32_t eb = 0, ib = 0;
        int te = 0, tt = 0;
        if (v >= 0) {
            if (A.nEC) {
                eb = A.ec_ptr[v];
                te = (int)(A.ec_ptr[v + 1] - eb) * A.nEC;
            }
            tt = te;
            if (A.nISO) {
                ib = A.iso_ptr[v];
                tt += (int)(A.iso_ptr[v + 1] - ib) * A.nISO;
            }
        }
        int m = max(tt, __shfl_xor_sync(full, tt, 8));
        m = max(m, __shfl_xor_sync(full, m, 16));
#pragma unroll 1
        for (int b = 0; b < m; b += 8) {
            const int q = b + sub;
            const LT *row = (const LT *)(A.nISO ? A.lutISO : A.lutEC);
            int64_t col = -1;  // from the first EC column on
            if (q < te) {
                const uint32_t j = eb + q / A.nEC;
                const int i = q % A.nEC;
                row = (const LT *)A.lutEC + (size_t)((unsigned)(i * A.ndirs) + A.ec_o[j]) * A.nSp;
                col = (int64_t)i * A.nE + A.ec_col[j];
            } else if (q < tt) {
                const int i = (q - te) % A.nISO;
                row = (const LT *)A.lutISO + (size_t)i * A.nSp;
                col = A.iso_base - A.ec_base + (int64_t)i * A.nISOv + A.iso_col[ib + (q - te) / A.nISO];
            }
            const int cnt = min(m - b, 8);
            double mine = 0.0;
#pragma unroll 1
            for (int t = 0; t < cnt; ++t) {
                const LT *L = reinterpret_cast<const LT *>(
                                  __shfl_sync(full, reinterpret_cast<unsigned long long>(row), t, 8)) + s_base + 4 * sub;
                f2 P = 0ull, R = 0ull;
#pragma unroll
                for (int k = 0; k < NQ; ++k) {
                    const int o = 32 * quad_of<LT, NQ>(k, par);
                    if (s_base + o + 4 * sub < A.nSp) {
                        f2 a, c;
                        Quad<LT>::ldg(L + o, a, c);
                        P = f2_fma(a, z0[k], P);
                        R = f2_fma(c, z1[k], R);
                    }
                }
                P = f2_add(P, R);
                float t0, t1, e = 0.f;
                if (sizeof(LT) == 4) {  // single dots: the last three sums keep their errors
                    P = f2_add(P, __shfl_xor_sync(full, P, 4, 8));
                    f2_unpack(P, t0, t1);
                    t0 = sum_err(t0, t1, e);
#pragma unroll
                    for (int d = 2; d >= 1; d >>= 1) {
                        float g;
                        t0 = sum_err(t0, __shfl_xor_sync(full, t0, d, 8), g);
                        e += __shfl_xor_sync(full, e, d, 8) + g;
                    }
                    t1 = 0.f;
                } else {
#pragma unroll
                    for (int d = 4; d >= 1; d >>= 1) P = f2_add(P, __shfl_xor_sync(full, P, d, 8));
                    f2_unpack(P, t0, t1);
                }
                if (sub == t) mine = sizeof(LT) == 4 ? (double)t0 + (double)e : (double)(t0 + t1);
            }
            if (col >= 0) {
                if (A.nc > 1) A.epart[col * A.nc + chunk] = mine;
                else A.xout[A.ec_base + col] = mine;
            }
        }
        __syncwarp();
        v = vn;
        vn = vnn;
        rb = rbn;
        re = ren;
    }
}

}  // namespace detail

// the two kernels of a table type; returns CGB_ERR_UNSUPPORTED for a shape without kernels
template <class LT>
int launch_mix_smem(int adjoint, int nq, int grid, size_t smem, cudaStream_t st, const detail::SmMixArgs &a, int cs) {
    using namespace detail;
#define CGB_MIX(N)                                                                                          \
    if (nq == N) {                                                                                          \
        auto kern = adjoint ? k_adj_mix_smem<LT, N> : k_fwd_mix_smem<LT, N>;                                \
        CGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));       \
        kern<<<grid, kMixThreads, smem, st>>>(a, cs);                                                       \
        CGB_CUDA(cudaGetLastError());                                                                       \
        return CGB_OK;                                                                                      \
    }
    CGB_MIX(1) CGB_MIX(2) CGB_MIX(3) CGB_MIX(4) CGB_MIX(5) CGB_MIX(6)
#undef CGB_MIX
    return fail(CGB_ERR_UNSUPPORTED, "no shared-memory kernel for this shape");
}

int launch_mix_smem_bf16(int adjoint, int nq, int grid, size_t smem, cudaStream_t st, const detail::SmMixArgs &a, int cs);
int launch_mix_smem_fp16(int adjoint, int nq, int grid, size_t smem, cudaStream_t st, const detail::SmMixArgs &a, int cs);
int launch_mix_smem_f32(int adjoint, int nq, int grid, size_t smem, cudaStream_t st, const detail::SmMixArgs &a, int cs);

}  // namespace cgb
