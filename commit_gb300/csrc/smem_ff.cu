// Run layout, table images, kernels and launches of the shared-memory float-float products
// (smem_ff.cuh).
#include <cub/cub.cuh>

#include <mutex>
#include <vector>

#include "operator_launch.cuh"
#include "smem_ff.cuh"

namespace cgb {
namespace {

using namespace detail;

// ------------------------------------------------------------------ layout
__global__ void k_run_heads(const uint16_t *__restrict__ o, int64_t n, uint32_t *__restrict__ head) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
        head[j] = j == 0 || o[j] != o[j - 1];
}

__global__ void k_voxel_heads(const uint32_t *__restrict__ vox_ptr, int nV, uint32_t *__restrict__ head) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < nV && vox_ptr[v] < vox_ptr[v + 1]) head[vox_ptr[v]] = 1u;
}

// id[j] = runs that begin before segment j (exclusive scan of head)
__global__ void k_run_fill(const uint32_t *__restrict__ head, const uint32_t *__restrict__ id,
                           const uint16_t *__restrict__ o, int64_t n, uint32_t nruns, uint16_t *__restrict__ run_o,
                           uint32_t *__restrict__ run_seg) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
        if (head[j]) {
            run_o[id[j]] = o[j];
            run_seg[id[j]] = (uint32_t)j;
        }
    if (blockIdx.x == 0 && threadIdx.x == 0) run_seg[nruns] = (uint32_t)n;
}

__global__ void k_run_ptr(const uint32_t *__restrict__ vox_ptr, const uint32_t *__restrict__ id, int nV, int64_t n,
                          uint32_t nruns, uint32_t *__restrict__ run_ptr) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v <= nV) run_ptr[v] = v < nV && vox_ptr[v] < n ? id[vox_ptr[v]] : nruns;
}

// sort key of a voxel: its window, then its run count falling
__global__ void k_perm_key(const uint32_t *__restrict__ run_ptr, int nV, uint64_t *__restrict__ key,
                           uint32_t *__restrict__ val) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nV) return;
    key[v] = ((uint64_t)(v / kVoxWindow) << 32) | (0xffffffffu - (run_ptr[v + 1] - run_ptr[v]));
    val[v] = (uint32_t)v;
}

// first run of each voxel whose orientation is in range b or beyond
__global__ void k_run_blk(const uint32_t *__restrict__ run_ptr, const uint16_t *__restrict__ run_o, int nV, int nb,
                          int no, uint32_t *__restrict__ run_blk) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= nV) return;
    uint32_t lo = run_ptr[v];
    const uint32_t end = run_ptr[v + 1];
    for (int b = 0; b <= nb; ++b) {
        uint32_t hi = end;
        while (lo < hi) {
            const uint32_t m = lo + (hi - lo) / 2;
            if ((int)run_o[m] < b * no) lo = m + 1;
            else hi = m;
        }
        run_blk[(size_t)b * nV + v] = b == nb ? end : lo;
    }
}

// table images: A [chunk][row][fcs], A' [chunk][range][response][orientation][acs]
__global__ void k_fwd_image(const float *__restrict__ lut, int rows, int nS, int nc, int width, int cs,
                            float *__restrict__ img) {
    const int64_t total = (int64_t)nc * rows * cs;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(q % cs);
        const int64_t t = q / cs;
        const int r = (int)(t % rows), c = (int)(t / rows);
        const int s = c * width + k;
        img[q] = k < width && s < nS ? lut[(size_t)r * nS + s] : 0.f;
    }
}

__global__ void k_adj_image(const float *__restrict__ lut, int nIC, int ndirs, int nS, int nc, int width, int nb, int no,
                            int cs, float *__restrict__ img) {
    const int64_t total = (int64_t)nc * nb * nIC * no * cs;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(q % cs);
        int64_t t = q / cs;
        const int o = (int)(t % no);
        t /= no;
        const int i = (int)(t % nIC);
        t /= nIC;
        const int b = (int)(t % nb), c = (int)(t / nb);
        const int d = b * no + o, s = c * width + k;
        img[q] = k < width && s < nS && d < ndirs ? lut[((size_t)i * ndirs + d) * nS + s] : 0.f;
    }
}

// Column maxima (zero beyond nS; 32 samples per block) and, in the blocks from kColPad / 32 on, the
// smallest sum of eight rows each; of a non-negative table
__global__ void __launch_bounds__(256) k_table_bounds(const float *__restrict__ lut, int rows, int nS,
                                                      float *__restrict__ colmax, float *__restrict__ rowmin) {
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int rb = (int)blockIdx.x - kColPad / 32;
    if (rb < 0) {
        const int s = blockIdx.x * 32 + lane;
        float m = 0.f;
        if (s < nS)
            for (int r = w; r < rows; r += 8) m = fmaxf(m, lut[(size_t)r * nS + s]);
        red[w][lane] = m;
        __syncthreads();
        if (w) return;
        for (int q = 1; q < 8; ++q) m = fmaxf(m, red[q][lane]);
        colmax[s] = m;
    } else {
        const int r = rb * 8 + w;
        float t = 0.f;
        if (r < rows)
            for (int s = lane; s < nS; s += 32) t += lut[(size_t)r * nS + s];
#pragma unroll
        for (int d = 16; d; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
        if (lane == 0) red[w][0] = r < rows ? t : 3.4e38f;
        __syncthreads();
        if (threadIdx.x) return;
        for (int q = 1; q < 8; ++q) t = fminf(t, red[q][0]);
        rowmin[rb] = t;
    }
}

__global__ void k_eval_flags(const uint32_t *__restrict__ eval, int64_t n, unsigned *__restrict__ flags) {
    bool bad = false;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        bad |= eval[i] != 1u;
    if (bad) atomicOr(flags, 1u);
}

int grid_n(int64_t n) {
    int64_t g = (n + 255) / 256;
    return (int)(g < 1 ? 1 : (g > 8192 ? 8192 : g));
}

// ------------------------------------------------------------------ run coefficients
// c[i][r] = sum over the run's segments of l * x[i*nF + f] * eval, in float-float; x scaled
// by the range guard's power of two.  A thread takes kCoefRuns runs at once: the chain run ->
// segment -> x is three dependent loads, and the x gathers hit L2.
constexpr int kCoefRuns = 4;

__device__ __forceinline__ void seg_coef(const OpDev &P, double xv, size_t q, float l, int ex, int eval_ones, float &h,
                                         float &e) {
    if (ex) xv = xv * pow2(-ex);
    if (!eval_ones) {
        const uint32_t ev = P.eval[q];
        if (ev != 1u) xv *= (double)ev;
    }
    float xh, xl;
    split_bits(xv, xh, xl);
    h = __fmul_rn(l, xh);
    e = __fmaf_rn(l, xl, __fmaf_rn(l, xh, -h));
}

__global__ void __launch_bounds__(256) k_run_coef(const OpDev P, const uint32_t *__restrict__ run_seg, int64_t nruns,
                                                  const double *__restrict__ x, int eval_ones,
                                                  float2 *__restrict__ coef) {
    const int ex = ff_exp_x(P);
    for (int64_t r0 = blockIdx.x * (256ll * kCoefRuns) + threadIdx.x; r0 < nruns;
         r0 += (int64_t)gridDim.x * (256 * kCoefRuns)) {
        uint32_t beg[kCoefRuns], end[kCoefRuns], f[kCoefRuns];
        float l[kCoefRuns];
#pragma unroll
        for (int u = 0; u < kCoefRuns; ++u) {
            const int64_t r = r0 + 256 * u < nruns ? r0 + 256 * u : nruns - 1;
            beg[u] = run_seg[r];
            end[u] = run_seg[r + 1];
        }
#pragma unroll
        for (int u = 0; u < kCoefRuns; ++u) {
            f[u] = P.seg_f[beg[u]];
            l[u] = P.seg_l[beg[u]];
        }
        for (int i = 0; i < P.nIC; ++i) {
            double xv[kCoefRuns];
#pragma unroll
            for (int u = 0; u < kCoefRuns; ++u) xv[u] = x[(size_t)i * P.nF + f[u]];
#pragma unroll
            for (int u = 0; u < kCoefRuns; ++u) {
                float ch, cl;
                seg_coef(P, xv[u], (size_t)i * P.nF + f[u], l[u], ex, eval_ones, ch, cl);
                for (uint32_t j = beg[u] + 1; j < end[u]; ++j) {
                    const size_t q = (size_t)i * P.nF + P.seg_f[j];
                    float h, e;
                    seg_coef(P, x[q], q, P.seg_l[j], ex, eval_ones, h, e);
                    ff_add(ch, cl, h, e);
                }
                const float h = __fadd_rn(ch, cl);
                if (r0 + 256 * u < nruns)
                    coef[(size_t)i * nruns + r0 + 256 * u] = make_float2(h, __fsub_rn(cl, __fsub_rn(h, ch)));
            }
        }
    }
}

// ------------------------------------------------------------------ A
// 8 lanes own a voxel, lane `sub` the sample pairs sub + 8k, k < NP, of the block's chunk
// (16 * NP samples).  Odd groups take the pairs of an even / odd k swapped, so the two groups
// of a half-warp read the two halves of a 128-byte line and their shared-memory loads do
// not conflict (rows are a multiple of 128 bytes apart).
template <int NP>
__global__ void __launch_bounds__(kFwdThreads, 1) k_fwd_smem(const __grid_constant__ SmFwdArgs A) {
    constexpr int NE = (NP + 1) & ~1, CS = 16 * NE, W = 16 * NP, GPB = kFwdThreads / 8;
    extern __shared__ __align__(16) float tab[];
    const unsigned full = 0xffffffffu;
    const int sub = threadIdx.x & 7, par = (threadIdx.x >> 3) & 1;
    const int chunk = blockIdx.x % A.nc, cta = blockIdx.x / A.nc, ncta = (gridDim.x - chunk + A.nc - 1) / A.nc;
    const int rows = A.nIC * A.ndirs;
    fill_table<kFwdThreads>(tab, A.img + (size_t)chunk * rows * CS, rows * CS);
    const int s_base = chunk * W;
    // pair of register k: kk(k); in a row, even and odd k have a base each
    auto kk = [&](int k) { return (k ^ 1) < NP ? k ^ par : k; };
    const float *tb = tab + 2 * sub, *tb0 = tb + 16 * par, *tb1 = tb - 16 * par;
    auto pair = [&](unsigned row, int k) {
        return *reinterpret_cast<const f2 *>(((k ^ 1) < NP ? (k & 1 ? tb1 : tb0) : tb) + row + 16 * k);
    };
    const int ex = A.xmax ? ff_exp_hi((unsigned)(*A.xmax >> 32), A.lut_exp) : 0;
    const bool even = (A.nS & 1) == 0 && A.vec_ok;
    double nrm = 0.0;
    // a warp takes four voxels at a time, neighbouring warps' fours going to different blocks (the
    // voxels are sorted by run count: every block gets long and short ones)
    const int last = A.p1 - A.p0, stride = ncta * GPB;
    const int lg = (int)((threadIdx.x & 31) >> 3), first = ((int)(threadIdx.x >> 5) * ncta + cta) * 4;
    // the voxel of the next step and its runs are fetched during this one
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
        // largest coefficient and whether all are finite and >= 0
        float cm = 0.f;
        bool ok = true;
        for (int i = 0; i < A.nIC; ++i)
            for (uint32_t j = rb + sub; j < re; j += 8) {
                const float h = A.coef[(size_t)i * A.nruns + j].x;
                ok = ok && h >= 0.f && h <= A.coef_max;
                cm = fmaxf(cm, h);
            }
        __syncwarp();
#pragma unroll
        for (int d = 4; d; d >>= 1) cm = fmaxf(cm, __shfl_xor_sync(full, cm, d, 8));
        ok = ((__ballot_sync(full, !ok) >> ((threadIdx.x & 31) & ~7)) & 0xffu) == 0u;
        for (uint32_t j = rbn + 16 * sub; j < ren; j += 128) prefetch_l2(A.coef + j);
        for (uint32_t j = rbn + 64 * sub; j < ren; j += 512) prefetch_l2(A.run_o + j);
        const int mine = (int)(re - rb + 7) / 8;  // this voxel's batches; the warp runs the most of its four
        int nb = max(mine, __shfl_xor_sync(full, mine, 8));
        nb = max(nb, __shfl_xor_sync(full, nb, 16));
        DD2 acc[NP];
#pragma unroll
        for (int k = 0; k < NP; ++k) dd2_zero(acc[k]);
        unsigned biased = 0u;  // halves that carry the bias cm * colmax
#pragma unroll 1
        for (int i = 0; i < A.nIC; ++i) {
            const float2 *cf = A.coef + (size_t)i * A.nruns;
            uint32_t j = rb + sub;
            float2 nc = make_float2(0.f, 0.f);
            uint32_t no = 0;
            if (j < re) {
                nc = cf[j];
                no = A.run_o[j];
            }
#pragma unroll 1
            for (int it = 0; it < nb; ++it) {
                const float2 c = nc;
                const unsigned row = ((unsigned)(i * A.ndirs) + no) * (unsigned)CS;
                j += 8;
                nc = make_float2(0.f, 0.f);
                no = 0;
                if (j < re) {
                    nc = cf[j];
                    no = A.run_o[j];
                }
                const bool gen = !ok || (it == 0 && i == 0);  // general sum for this group's batch
                const bool nz = c.x != 0.f || c.y != 0.f;
                unsigned g = __ballot_sync(full, nz && gen), f = __ballot_sync(full, nz && !gen);
                g |= g >> 16;
                g = (g | g >> 8) & 0xffu;
                f |= f >> 16;
                f = (f | f >> 8) & 0xffu;
                // zero coefficients add exactly nothing, so a group may sit out a step
                if (g) {
                    const float gx = gen ? c.x : 0.f, gy = gen ? c.y : 0.f;
#pragma unroll 2
                    for (int t = 0; t < 8; ++t) {
                        if (!(g >> t & 1u)) continue;
                        const float h = __shfl_sync(full, gx, t, 8), l = __shfl_sync(full, gy, t, 8);
                        const unsigned r = __shfl_sync(full, row, t, 8);
                        const f2 h2 = f2_pack(h, h), l2 = f2_pack(l, l);
#pragma unroll
                        for (int k = 0; k < NP; ++k)
                            dd2_fma_any(acc[k], h2, l2, pair(r, k), A.zero);
                    }
                }
                const float fx = gen ? 0.f : c.x, fy = gen ? 0.f : c.y;
                if (f == 0xffu) {
#pragma unroll 4
                    for (int t = 0; t < 8; ++t) {
                        const float h = __shfl_sync(full, fx, t, 8), l = __shfl_sync(full, fy, t, 8);
                        const unsigned r = __shfl_sync(full, row, t, 8);
                        const f2 h2 = f2_pack(h, h), l2 = f2_pack(l, l);
#pragma unroll
                        for (int k = 0; k < NP; ++k)
                            dd2_fma_same(acc[k], h2, l2, pair(r, k));
                    }
                } else {
                    while (f) {
                        const int t = __ffs(f) - 1;
                        f &= f - 1;
                        const float h = __shfl_sync(full, fx, t, 8), l = __shfl_sync(full, fy, t, 8);
                        const unsigned r = __shfl_sync(full, row, t, 8);
                        const f2 h2 = f2_pack(h, h), l2 = f2_pack(l, l);
#pragma unroll
                        for (int k = 0; k < NP; ++k)
                            dd2_fma_same(acc[k], h2, l2, pair(r, k));
                    }
                }
                if (ok && i == 0 && it == 0 && (mine > 1 || A.nIC > 1)) {
                    // from here on the sums must not be below a term: add the bound where they may be
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        float m0, m1, a0, a1;
                        f2_unpack(f2_ldg(A.colmax + s_base + 2 * (sub + 8 * kk(k))), m0, m1);
                        f2_unpack(acc[k].s, a0, a1);
                        m0 = __fmul_rn(cm, m0);
                        m1 = __fmul_rn(cm, m1);
                        const bool b0 = a0 < m0, b1 = a1 < m1;
                        biased |= (b0 ? 1u << (2 * k) : 0u) | (b1 ? 2u << (2 * k) : 0u);
                        dd2_addf(acc[k], f2_pack(b0 ? m0 : 0.f, b1 ? m1 : 0.f));
                    }
                } else if (ok && it < mine) {
#pragma unroll
                    for (int k = 0; k < NP; ++k) {
                        const f2 s = f2_add(acc[k].s, acc[k].e);
                        acc[k].e = f2_add(acc[k].e, f2_sub(acc[k].s, s));
                        acc[k].s = s;
                    }
                }
            }
        }
        if (biased) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                float m0, m1;
                f2_unpack(f2_ldg(A.colmax + s_base + 2 * (sub + 8 * kk(k))), m0, m1);
                dd2_addf(acc[k], f2_pack(biased >> (2 * k) & 1u ? -__fmul_rn(cm, m0) : 0.f,
                                         biased >> (2 * k) & 2u ? -__fmul_rn(cm, m1) : 0.f));
            }
        }
        __syncwarp();
        // EC and ISO elements, (element, response) by (element, response); rows from L1 / L2
        {
            const int te = (int)(ee - eb) * A.nEC, tt = te + (int)(ie - ib) * A.nISO;
            int m = max(tt, __shfl_xor_sync(full, tt, 8));
            m = max(m, __shfl_xor_sync(full, m, 16));
#pragma unroll 1
            for (int b = 0; b < m; b += 8) {
                const int q = b + sub;
                float h = 0.f, l = 0.f;
                const float *row = A.nISO ? A.lutISO : A.lutEC;  // lanes past the end read (and drop) a row that exists
                if (q < tt) {
                    double xv;
                    if (q < te) {
                        const uint32_t j = eb + q / A.nEC;
                        const int i = q % A.nEC;
                        row = A.lutEC + (size_t)((unsigned)(i * A.ndirs) + A.ec_o[j]) * A.nSp;
                        xv = A.x[A.ec_base + i * A.nE + A.ec_col[j]];
                    } else {
                        const int i = (q - te) % A.nISO;
                        row = A.lutISO + (size_t)i * A.nSp;
                        xv = A.x[A.iso_base + i * A.nISOv + A.iso_col[ib + (q - te) / A.nISO]];
                    }
                    if (ex) xv = xv * pow2(-ex);
                    split_bits(xv, h, l);
                }
                unsigned g = __ballot_sync(full, h != 0.f || l != 0.f);
                g |= g >> 16;
                g = (g | g >> 8) & 0xffu;
#pragma unroll
                for (int k = 0; k < NP; ++k) {
                    const f2 s = f2_add(acc[k].s, acc[k].e);
                    acc[k].e = f2_add(acc[k].e, f2_sub(acc[k].s, s));
                    acc[k].s = s;
                }
                while (g) {
                    const int t = __ffs(g) - 1;
                    g &= g - 1;
                    const Coef2 q = coef2(__shfl_sync(full, h, t, 8), __shfl_sync(full, l, t, 8));
                    const float *L = reinterpret_cast<const float *>(
                                         __shfl_sync(full, reinterpret_cast<unsigned long long>(row), t, 8)) +
                                     s_base + 2 * sub;
#pragma unroll
                    for (int k = 0; k < NP; ++k)
                        dd2_fma(acc[k], q, s_base + 2 * (sub + 8 * kk(k)) < A.nSp ? f2_ldg(L + 16 * kk(k)) : 0ull);
                }
            }
        }
        if (v >= 0) {
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                const int s = s_base + 2 * (sub + 8 * kk(k));
                if (s >= A.nS) continue;
                float s0, s1, e0, e1;
                f2_unpack(acc[k].s, s0, s1);
                f2_unpack(acc[k].e, e0, e1);
                double a0 = ff_join(s0, e0), a1 = ff_join(s1, e1);
                if (ex) {
                    a0 = a0 * pow2(ex);
                    a1 = a1 * pow2(ex);
                }
                const size_t idx = (size_t)v * A.nS + s;
                const bool two = s + 1 < A.nS;
                if (A.yout) {
                    if (two && even) *reinterpret_cast<double2 *>(A.yout + idx) = make_double2(a0, a1);
                    else { A.yout[idx] = a0; if (two) A.yout[idx + 1] = a1; }
                }
                if (A.axout) {
                    if (two && even) *reinterpret_cast<double2 *>(A.axout + idx) = make_double2(a0, a1);
                    else { A.axout[idx] = a0; if (two) A.axout[idx + 1] = a1; }
                }
                if (A.partials) {
                    double r0 = A.yobs ? a0 - A.yobs[idx] : a0;
                    if (A.sqw) r0 *= A.sqw[idx];
                    nrm = fma(r0, r0, nrm);
                    if (two) {
                        double r1 = A.yobs ? a1 - A.yobs[idx + 1] : a1;
                        if (A.sqw) r1 *= A.sqw[idx + 1];
                        nrm = fma(r1, r1, nrm);
                    }
                }
            }
        }
        __syncwarp();
        v = vn;
        vn = vnn;
        rb = rbn;
        re = ren;
    }
    if (A.partials) {
        __shared__ double red[kFwdThreads / 32];
#pragma unroll
        for (int o = 16; o; o >>= 1) nrm += __shfl_xor_sync(full, nrm, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = nrm;
        __syncthreads();
        if (threadIdx.x == 0) {
            double t = 0.0;
            for (int q = 0; q < kFwdThreads / 32; ++q) t += red[q];
            A.partials[(size_t)blockIdx.x * kRedSlots] = t;
        }
    }
}

// ------------------------------------------------------------------ A'
// 8 lanes own a voxel and hold the block's chunk of its input row as float-float pairs (pairs
// laid out as in A); a batch of 8 runs is taken four at a time (butterfly reduce-scatter as
// batch_dots_p).  The runs' parts go to `part`; k_adj_join adds them and writes the terms
// l * <L, z> of their segments (also with one chunk: the segment loads would be waited for in
// the voxel pass).  EC / ISO elements of four voxels are taken
// by the blocks of one of the orientation ranges in turn.

// First two levels of a butterfly reduce-scatter over four items: P[q] of lane sub is item
// q ^ (sub >> 1) (each lane takes the items in its own order, so what it keeps is always in
// front and no value is selected by lane); item sub >> 1, summed over the lanes of one parity,
// is left in P[0].
__device__ __forceinline__ void scatter4(DD2 (&P)[4]) {
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int h = 2, m = 4; h >= 1; h /= 2, m /= 2)
#pragma unroll
        for (int j = 0; j < h; ++j) dd2_add(P[j], dd2_shfl_xor(full, P[j + h], m, 8));
}

template <int NP>
__global__ void __launch_bounds__(adj_threads(NP), 1) k_adj_smem(const __grid_constant__ SmAdjArgs A) {
    constexpr int NE = (NP + 1) & ~1, CS = 16 * NE, W = 16 * NP, GPB = adj_threads(NP) / 8;
    extern __shared__ __align__(16) float tab[];
    const unsigned full = 0xffffffffu;
    const int sub = threadIdx.x & 7, par = (threadIdx.x >> 3) & 1;
    const int parts = A.nc * A.nb, part = blockIdx.x % parts, chunk = part / A.nb, blk = part % A.nb;
    const int s_base = chunk * W;
    fill_table<adj_threads(NP)>(tab, A.img + (size_t)part * A.nIC * A.no * CS, A.nIC * A.no * CS);
    auto kk = [&](int k) { return (k ^ 1) < NP ? k ^ par : k; };
    const float *tb = tab + 2 * sub, *tb0 = tb + 16 * par, *tb1 = tb - 16 * par;
    auto pair = [&](unsigned row, int k) {
        return *reinterpret_cast<const f2 *>(((k ^ 1) < NP ? (k & 1 ? tb1 : tb0) : tb) + row + 16 * k);
    };
    const bool even = (A.nS & 1) == 0 && A.vec_ok;
    const int last = A.p1 - A.p0, ncta = (int)(gridDim.x / parts), stride = ncta * GPB;
    // the voxel of the next step, its first runs and its row are fetched during this one
    auto voxel = [&](int pos) {
        int v = -1;
        if (pos < last) v = (int)A.vperm[A.p0 + pos];
        return v < A.v0 || v >= A.v1 ? -1 : v;
    };
    const uint32_t *rb_of = A.run_blk + (size_t)blk * A.nV, *re_of = rb_of + A.nV;
    // fours of voxels interleaved over the blocks as in A
    const int lg = (int)((threadIdx.x & 31) >> 3);
    const int first = ((int)(threadIdx.x >> 5) * ncta + (int)(blockIdx.x / parts)) * 4;
    int v = voxel(first + lg), vn = voxel(first + lg + stride);
    uint32_t rb = v >= 0 ? rb_of[v] : 0u, re = v >= 0 ? re_of[v] : 0u;
    const uint32_t own = (uint32_t)((sub & 1) * 4 + (sub >> 1));  // this lane's run of a batch
    unsigned on = rb + own < re ? A.run_o[rb + own] : 0u;         // its orientation, of the next batch
    fill_wait();
    for (int w = first; w < last; w += stride) {  // w: the warp's first position
        const uint32_t rbn = vn >= 0 ? rb_of[vn] : 0u, ren = vn >= 0 ? re_of[vn] : 0u;
        const int vnn = voxel(w + lg + 2 * stride);
        f2 zh[NP], zl[NP];
        unsigned zmax = 0, neg = A.general;
        auto load = [&](int k, double &z0, double &z1) {
            const int s = s_base + 2 * (sub + 8 * kk(k));
            z0 = z1 = 0.0;
            if (v >= 0 && s < A.nS) {
                const double *p = A.z + (size_t)v * A.nS + s;
                if (even) {
                    const double2 t = *reinterpret_cast<const double2 *>(p);
                    z0 = t.x;
                    z1 = t.y;
                } else {
                    z0 = p[0];
                    if (s + 1 < A.nS) z1 = p[1];
                }
            }
        };
#pragma unroll
        for (int k = 0; k < NP; ++k) {
            double z0, z1;
            load(k, z0, z1);
            zmax = max(zmax, max(abs_hi(z0), abs_hi(z1)));
            neg |= (unsigned)(__double2hiint(z0) | __double2hiint(z1));
            float h0, l0, h1, l1;
            split_bits(z0, h0, l0);
            split_bits(z1, h1, l1);
            zh[k] = f2_pack(h0, h1);
            zl[k] = f2_pack(l0, l1);
        }
        if (vn >= 0) {
            const char *p = reinterpret_cast<const char *>(A.z + (size_t)vn * A.nS + s_base);
            if (128 * sub < 8 * W && s_base + 16 * sub < A.nS) prefetch_l2(p + 128 * sub);
            for (uint32_t j = rbn + 32 * sub; j < ren; j += 256) prefetch_l2(A.run_seg + j);
            for (uint32_t j = rbn + 64 * sub; j < ren; j += 512) prefetch_l2(A.run_o + j);
        }
        // range guard: a chunk of a row outside float-float's range is split again, scaled (exact)
        const int ez = ff_exp_hi(group_max_u<8>(zmax, full), A.lut_exp);
        if (ez) {
#pragma unroll 1
            for (int k = 0; k < NP; ++k) {
                double z0, z1;
                load(k, z0, z1);
                f2 h, l, unused;
                split2(z0 * pow2(-ez), z1 * pow2(-ez), h, l, unused);
#pragma unroll
                for (int q = 0; q < NP; ++q)
                    if (q == k) {
                        zh[q] = h;
                        zl[q] = l;
                    }
            }
        }
        // rows without a negative entry take the five-operation sums (file comment of
        // smem_ff.cuh): the bias is a power of two just below this lane's largest term bound
        bool pos = ((__ballot_sync(full, (neg >> 31) != 0u) >> ((threadIdx.x & 31) & ~7)) & 0xffu) == 0u;
        f2 bias = 0ull;
        float low = 0.f;  // smallest dot product that the lanes' biases do not dwarf
        if (__any_sync(full, pos)) {
            float x0 = 0.f, x1 = 0.f;
#pragma unroll
            for (int k = 0; k < NP; ++k) {
                float a0, a1;
                f2_unpack(f2_mul(zh[k], f2_ldg(A.colmax + s_base + 2 * (sub + 8 * kk(k)))), a0, a1);
                x0 = fmaxf(x0, a0);
                x1 = fmaxf(x1, a1);
            }
            auto down = [](float b) { return __uint_as_float(__float_as_uint(b * 1.001f) & 0x7f800000u); };
            x0 = down(x0);
            x1 = down(x1);
            bias = f2_pack(x0, x1);
            low = x0 + x1;
#pragma unroll
            for (int d = 4; d; d >>= 1) low += __shfl_xor_sync(full, low, d, 8);
            low *= 1.f / kBiasAdj;
        }
        int most = (int)(re - rb);
        most = max(most, __shfl_xor_sync(full, most, 8));
        most = max(most, __shfl_xor_sync(full, most, 16));
        if (most == 0) on = rbn + own < ren ? __ldg(A.run_o + rbn + own) : 0u;
        // once more with the general sums where the biased ones gave a dot product that the bias dwarfs
#pragma unroll 1
        for (;;) {
            const bool any_pos = __any_sync(full, pos), any_mix = __any_sync(full, !pos);
            bool small = false;
            // Eight runs at a time, four by four: run t of the batch belongs to lane (t & 3) * 2 + (t >> 2),
            // which is where the butterfly leaves its dot product.
#pragma unroll 1
            for (int b = 0; b < most; b += 8) {
                const uint32_t j = rb + b + own;
                const bool valid = j < re;
                const unsigned o = valid ? on - (unsigned)(blk * A.no) : 0u;
                const uint32_t jn = b + 8 < most ? j + 8 : rbn + own;
                on = jn < (b + 8 < most ? re : ren) ? __ldg(A.run_o + jn) : 0u;
#pragma unroll 1
                for (int i = 0; i < A.nIC; ++i) {
                    const unsigned row = ((unsigned)(i * A.no) + o) * (unsigned)CS;
                    // four dot products' partial sums, of one sign (the bias is a power of two not above
                    // the sums: the difference is exact) or of any
                    auto four_pos = [&](int u) {
                        DD2 P[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const unsigned r = __shfl_sync(full, row, ((q ^ (sub >> 1)) << 1) + u, 8);
                            const f2 L0 = pair(r, 0);
                            const f2 s = f2_fma(zh[0], L0, bias);
                            P[q].e = f2_fma(zl[0], L0, f2_fma(zh[0], L0, f2_sub(bias, s)));
                            P[q].s = s;
#pragma unroll
                            for (int k = 1; k < NP; ++k) dd2_fma_same(P[q], zh[k], zl[k], pair(r, k));
                            P[q].s = f2_sub(P[q].s, bias);
                        }
                        scatter4(P);
                        return P[0];
                    };
                    auto four_any = [&](int u) {
                        DD2 P[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const unsigned r = __shfl_sync(full, row, ((q ^ (sub >> 1)) << 1) + u, 8);
                            const f2 L0 = pair(r, 0);
                            const f2 s = f2_fma(zh[0], L0, A.zero);
                            P[q].e = f2_fma(zl[0], L0, f2_fma(zh[0], L0, f2_neg(s)));
                            P[q].s = s;
#pragma unroll
                            for (int k = 1; k < NP; ++k) dd2_fma_any(P[q], zh[k], zl[k], pair(r, k), A.zero);
                        }
                        scatter4(P);
                        return P[0];
                    };
                    // the lanes of even parity finish the first four, those of odd parity the others
                    DD2 M, N;
                    dd2_zero(M);
#pragma unroll 1
                    for (int u = 0; u < 2; ++u) {
                        N = M;
                        if (u && b + 4 >= most) {
                            dd2_zero(M);
                            break;
                        }
                        if (any_pos) M = four_pos(u);
                        if (any_mix) {
                            const DD2 Q = four_any(u);
                            if (any_pos) M.s = pos ? M.s : Q.s, M.e = pos ? M.e : Q.e;
                            else M = Q;
                        }
                    }
                    const bool odd = (sub & 1) != 0;
                    DD2 send, keep;
                    send.s = odd ? N.s : M.s;  // N the first four, M the others
                    send.e = odd ? N.e : M.e;
                    keep.s = odd ? M.s : N.s;
                    keep.e = odd ? M.e : N.e;
                    dd2_add(keep, dd2_shfl_xor(full, send, 1, 8));
                    if (valid) {
                        float ds, de, s1, e1;
                        f2_unpack(keep.s, ds, s1);
                        f2_unpack(keep.e, de, e1);
                        ff_add(ds, de, s1, e1);
                        small = small || !(ds >= low);
                        double t = ff_join(ds, de);
                        if (ez) t = t * pow2(ez);
                        A.part[((size_t)i * A.nruns + j) * A.nc + chunk] = t;
                    }
                    __syncwarp();
                }
            }
            const unsigned bad = __ballot_sync(full, pos && small);
            if (!bad) break;
            pos = pos && !(bad >> ((threadIdx.x & 31) & ~7) & 0xffu);
            on = rb + own < re ? __ldg(A.run_o + rb + own) : 0u;
        }
        const unsigned tile = (unsigned)(A.p0 + w) / 4u;
        const bool ends = tile % (unsigned)A.nb == (unsigned)blk;  // this range takes the voxels' EC / ISO elements
        uint32_t eb = 0, ib = 0;
        int te = 0, tt = 0;
        if (ends && v >= 0) {
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
        // column of (element, response) q, from the first EC column on; its table row
        auto column = [&](int q) -> int64_t {
            if (q < te) return (int64_t)(q % A.nEC) * A.nE + A.ec_col[eb + q / A.nEC];
            q -= te;
            return A.iso_base - A.ec_base + (int64_t)(q % A.nISO) * A.nISOv + A.iso_col[ib + q / A.nISO];
        };
        int m = max(tt, __shfl_xor_sync(full, tt, 8));
        m = max(m, __shfl_xor_sync(full, m, 16));
#pragma unroll 1
        for (int b = 0; b < m; b += 8) {
            const int q0 = b + sub;
            const float *row = A.nISO ? A.lutISO : A.lutEC;
            int64_t col = -1;
            if (q0 < tt) {
                col = column(q0);
                row = q0 < te ? A.lutEC + (size_t)((unsigned)(q0 % A.nEC * A.ndirs) + A.ec_o[eb + q0 / A.nEC]) * A.nSp
                              : A.lutISO + (size_t)((q0 - te) % A.nISO) * A.nSp;
            }
            const int cnt = min(m - b, 8);
            double mine = 0.0;
#pragma unroll 1
            for (int u = 0; u < cnt; ++u) {
                const float *L = reinterpret_cast<const float *>(
                                     __shfl_sync(full, reinterpret_cast<unsigned long long>(row), u, 8)) +
                                 s_base + 2 * sub;
                DD2 P;
                dd2_zero(P);
#pragma unroll
                for (int k = 0; k < NP; ++k)
                    dd2_fma_any(P, zh[k], zl[k], s_base + 2 * (sub + 8 * kk(k)) < A.nSp ? f2_ldg(L + 16 * kk(k)) : 0ull,
                                A.zero);
                dd2_add(P, dd2_shfl_xor(full, P, 4, 8));
                dd2_add(P, dd2_shfl_xor(full, P, 2, 8));
                // the last sum rounds at the size of the result: in FP64 for these single dots
                float s0, s1, e0, e1;
                f2_unpack(P.s, s0, s1);
                f2_unpack(P.e, e0, e1);
                ff_add(s0, e0, s1, e1);
                double t = ff_join(s0, e0);
                t += __shfl_xor_sync(full, t, 1, 8);
                if (sub == u) mine = t;
            }
            if (ez) mine = mine * pow2(ez);
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

// Adds the chunks' parts for the voxels [v0, v1): terms l * <L, z> of the runs' segments, EC and
// ISO columns.  A pass of its own streams the parts (1M streamlines: 2.4 GB, 0.7 ms); letting
// the warp that finished a voxel last add them up cost 2.6 ms of latency in the voxel pass.
__global__ void __launch_bounds__(256) k_adj_join(const SmAdjArgs A, const uint32_t *__restrict__ run_ptr) {
    const int64_t first = blockIdx.x * 256ll + threadIdx.x, step = gridDim.x * 256ll;
    const int64_t r0 = run_ptr[A.v0], r1 = run_ptr[A.v1];
    for (int64_t r = r0 + first; r < r1; r += step) {
        const uint32_t sb = A.run_seg[r], se = A.run_seg[r + 1];
        const float l0 = A.seg_l[sb];
        for (int i = 0; i < A.nIC; ++i) {
            const double *q = A.part + ((size_t)i * A.nruns + r) * A.nc;
            double t = q[0];
            for (int c = 1; c < A.nc; ++c) t += q[c];
            double *out = A.scratch + (size_t)i * A.n;
            out[sb] = widen(l0) * t;
            for (uint32_t g = sb + 1; g < se; ++g) out[g] = widen(A.seg_l[g]) * t;
        }
    }
    auto column = [&](int64_t col) {
        double t = A.epart[col * A.nc];
        for (int c = 1; c < A.nc; ++c) t += A.epart[col * A.nc + c];
        A.xout[A.ec_base + col] = t;
    };
    if (A.nc == 1) return;  // EC and ISO columns are written by the voxel pass
    if (A.nEC) {
        const int64_t e0 = A.ec_ptr[A.v0], e1 = A.ec_ptr[A.v1];
        for (int64_t j = e0 + first; j < e1; j += step)
            for (int i = 0; i < A.nEC; ++i) column((int64_t)i * A.nE + A.ec_col[j]);
    }
    if (A.nISO) {
        const int64_t e0 = A.iso_ptr[A.v0], e1 = A.iso_ptr[A.v1];
        for (int64_t j = e0 + first; j < e1; j += step)
            for (int i = 0; i < A.nISO; ++i) column(A.iso_base - A.ec_base + (int64_t)i * A.nISOv + A.iso_col[j]);
    }
}

// weighted residual z = sqw * r, r = sqw * (A x - yobs) with A x = ax_a (mode 1) or
// ca*ax_a + cb*ax_b (mode 2), and the block sums of r^2 (ax_a may be z)
__global__ void __launch_bounds__(kBlock) k_residual(int64_t n, int mode, const double *ax_a,
                                                     const double *__restrict__ ax_b, double ca, double cb,
                                                     const double *__restrict__ yobs, const double *__restrict__ sqw,
                                                     double *z, double *__restrict__ partials) {
    double nrm = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x; i < n; i += (int64_t)gridDim.x * kBlock) {
        const double av = mode == 1 ? ax_a[i] : ax_combine(ca, ax_a[i], cb, ax_b[i]);
        double r = av - yobs[i];
        if (sqw) r *= sqw[i];
        nrm = fma(r, r, nrm);
        z[i] = sqw ? sqw[i] * r : r;
    }
    if (partials) block_sum_store(nrm, partials + (size_t)blockIdx.x * kRedSlots);
}

struct Buf {
    void *p = nullptr;
    ~Buf() {
        if (p) cudaFree(p);
    }
    template <class T>
    int get(T **out, size_t count) {
        CGB_CUDA(cudaMalloc(&p, (count ? count : 1) * sizeof(T)));
        *out = (T *)p;
        return CGB_OK;
    }
};

constexpr size_t kTableBytes = 224 << 10;  // of the 227 KB a block may have

// sample chunks of A: the fewest whose table part fits, at most 6 pairs per lane
bool fwd_shape(int rows, int nS, FfPlan *f) {
    for (int nc = (nS + 95) / 96; nc <= 64; ++nc) {
        const int np = (nS + 16 * nc - 1) / (16 * nc), ne = (np + 1) & ~1;
        if ((size_t)rows * 16 * ne * sizeof(float) > kTableBytes) {
            if (np <= 2) return false;
            continue;
        }
        if (np < 2 || np * 16 * (nc - 1) >= nS) return false;  // no kernel for one pair, no empty last chunk
        f->fnp = np;
        f->fnc = nc;
        f->fcs = 16 * ne;
        return true;
    }
    return false;
}

// sample chunks and orientation ranges of A': the fewest parts, then the fewest chunks
bool adj_shape(int nIC, int ndirs, int nS, FfPlan *f) {
    int best = 17;
    for (int nc = (nS + 95) / 96; nc <= 16; ++nc) {
        const int np = (nS + 16 * nc - 1) / (16 * nc), cs = 16 * ((np + 1) & ~1);
        if (np < 2 || np * 16 * (nc - 1) >= nS) break;
        const int per = (int)(kTableBytes / sizeof(float)) / cs / nIC;  // orientations that fit
        if (per < 1) continue;
        const int nb = (ndirs + per - 1) / per;
        if (nc * nb >= best) continue;
        best = nc * nb;
        f->anc = nc;
        f->anp = np;
        f->anb = nb;
        f->ano = (ndirs + nb - 1) / nb;
        f->acs = cs;
    }
    return best <= 16;
}

void drop_runs(cgb_op *op, RunLayout *R) {
    void *p[] = {R->run_ptr, R->run_o, R->run_seg, R->vperm};
    for (void *q : p)
        if (q) cudaFree(q);
    op->bytes -= R->bytes;
    delete R;
}

// table images, column maxima and row sums, queued on the legacy stream
int queue_images(cgb_op *op, FfPlan *f) {
    const int rows = op->nIC * op->ndirs;
    if (f->fimg)
        k_fwd_image<<<grid_n((int64_t)f->fnc * rows * f->fcs), 256>>>(op->lutIC, rows, op->nS, f->fnc, 16 * f->fnp,
                                                                     f->fcs, f->fimg);
    if (f->aimg)
        k_adj_image<<<grid_n((int64_t)f->anc * f->anb * op->nIC * f->ano * f->acs), 256>>>(
            op->lutIC, op->nIC, op->ndirs, op->nS, f->anc, 16 * f->anp, f->anb, f->ano, f->acs, f->aimg);
    k_table_bounds<<<kColPad / 32 + (rows + 7) / 8, 256>>>(op->lutIC, rows, op->nS, f->colmax, f->colmax + kColPad);
    CGB_CUDA(cudaGetLastError());
    return CGB_OK;
}

// whether the table's rows are uneven; waits for the images (the next product may be on a stream
// that the legacy one does not order)
int finish_images(cgb_op *op, FfPlan *f) {
    const int nb = (op->nIC * op->ndirs + 7) / 8;
    std::vector<float> b((size_t)kColPad + nb);
    CGB_CUDA(cudaMemcpy(b.data(), f->colmax, b.size() * sizeof(float), cudaMemcpyDeviceToHost));
    double sum = 0.0, low = b[kColPad];
    for (int s = 0; s < op->nS; ++s) sum += b[s];
    for (int r = 1; r < nb; ++r) low = b[kColPad + r] < low ? b[kColPad + r] : low;
    f->uneven = !(sum <= kBiasA * low);
    return CGB_OK;
}

int build_runs(cgb_op *op, RunLayout *R) {
    const int64_t n = op->n;
    const int nV = op->nV;
    Buf bh, bi, bt, bk, bk2, bv, bf;
    uint32_t *head, *id;
    CGB_TRY(bh.get(&head, (size_t)n));
    CGB_TRY(bi.get(&id, (size_t)n));
    k_run_heads<<<grid_n(n), 256>>>(op->seg_o, n, head);
    k_voxel_heads<<<(nV + 255) / 256, 256>>>(op->vox_ptr, nV, head);
    uint64_t *key, *key2;
    uint32_t *val;
    unsigned *flags;
    CGB_TRY(bk.get(&key, (size_t)nV));
    CGB_TRY(bk2.get(&key2, (size_t)nV));
    CGB_TRY(bv.get(&val, (size_t)nV));
    CGB_TRY(bf.get(&flags, 1));
    size_t b1 = 0, b2 = 0;
    CGB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b1, head, id, (int)n));
    CGB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b2, key, key2, val, val, nV, 0, 64));
    char *tmp;
    CGB_TRY(bt.get(&tmp, b1 > b2 ? b1 : b2));
    CGB_CUDA(cub::DeviceScan::ExclusiveSum(tmp, b1, head, id, (int)n));
    CGB_CUDA(cudaMemset(flags, 0, sizeof(unsigned)));
    k_eval_flags<<<grid_n((int64_t)op->nF * op->nIC), 256>>>(op->eval, (int64_t)op->nF * op->nIC, flags);
    uint32_t lastid[2];
    unsigned hf = 0;
    CGB_CUDA(cudaMemcpy(&lastid[0], id + (n - 1), 4, cudaMemcpyDeviceToHost));
    CGB_CUDA(cudaMemcpy(&lastid[1], head + (n - 1), 4, cudaMemcpyDeviceToHost));
    CGB_CUDA(cudaMemcpy(&hf, flags, 4, cudaMemcpyDeviceToHost));
    R->nruns = (int64_t)lastid[0] + lastid[1];
    R->eval_ones = hf == 0u;
    CGB_TRY(keep_buffer(op, &R->bytes, &R->run_ptr, (size_t)nV + 1));
    CGB_TRY(keep_buffer(op, &R->bytes, &R->run_o, (size_t)R->nruns));
    CGB_TRY(keep_buffer(op, &R->bytes, &R->run_seg, (size_t)R->nruns + 1));
    CGB_TRY(keep_buffer(op, &R->bytes, &R->vperm, (size_t)nV));
    k_run_fill<<<grid_n(n), 256>>>(head, id, op->seg_o, n, (uint32_t)R->nruns, R->run_o, R->run_seg);
    k_run_ptr<<<(nV + 256) / 256, 256>>>(op->vox_ptr, id, nV, n, (uint32_t)R->nruns, R->run_ptr);
    k_perm_key<<<(nV + 255) / 256, 256>>>(R->run_ptr, nV, key, val);
    CGB_CUDA(cub::DeviceRadixSort::SortPairs(tmp, b2, key, key2, val, R->vperm, nV, 0, 64));
    CGB_CUDA(cudaDeviceSynchronize());
    return CGB_OK;
}

bool dense(const cgb_op *op, double items) { return (double)op->n * op->nIC >= items * op->nV; }

// the directions whose shape and density suit these kernels, and nothing for the others
int build_plan(cgb_op *op, FfPlan *f) {
    const int nV = op->nV;
    if (op->lut_signed) return CGB_OK;  // the pair kernels skip zero coefficients, these may multiply by one
    const bool fs = fwd_shape(op->nIC * op->ndirs, op->nS, f) && dense(op, smem_min_items(op->nS, f->fnc));
    const bool as = adj_shape(op->nIC, op->ndirs, op->nS, f) && dense(op, smem_min_items(op->nS, f->anc * f->anb));
    if (!fs && !as) return CGB_OK;
    CGB_TRY(ensure_runs(op));
    const RunLayout *R = op->runs;
    CGB_TRY(keep_buffer(op, &f->bytes, &f->colmax, (size_t)kColPad + (op->nIC * op->ndirs + 7) / 8));
    if (fs) {
        CGB_TRY(keep_buffer(op, &f->bytes, &f->fimg, (size_t)f->fnc * op->nIC * op->ndirs * f->fcs));
        CGB_TRY(keep_buffer(op, &f->bytes, &f->coef, (size_t)op->nIC * R->nruns));
        CGB_TRY(order_create(&f->order));
    }
    if (as) {
        CGB_TRY(keep_buffer(op, &f->bytes, &f->aimg, (size_t)f->anc * f->anb * op->nIC * f->ano * f->acs));
        CGB_TRY(keep_buffer(op, &f->bytes, &f->part, (size_t)op->nIC * R->nruns * f->anc));
        if (f->anc > 1)
            CGB_TRY(keep_buffer(op, &f->bytes, &f->epart, ((size_t)op->nE * op->nEC + (size_t)op->nISOv * op->nISO) * f->anc));
        CGB_TRY(keep_buffer(op, &f->bytes, &f->run_blk, (size_t)(f->anb + 1) * nV));
        k_run_blk<<<(nV + 255) / 256, 256>>>(R->run_ptr, R->run_o, nV, f->anb, f->ano, f->run_blk);
    }
    CGB_TRY(queue_images(op, f));
    CGB_TRY(finish_images(op, f));
    CGB_CUDA(cudaDeviceSynchronize());
    f->fwd_ok = fs;
    f->adj_ok = as;
    return CGB_OK;
}

bool capturing(cudaStream_t st) {
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
}

// perm positions that hold the voxels [v0, v1): whole windows
void perm_range(const cgb_op *op, int &v0, int &v1, int &p0, int &p1) {
    v0 = op->vr1 > 0 ? op->vr0 : 0;
    v1 = op->vr1 > 0 ? op->vr1 : op->nV;
    p0 = v0 / kVoxWindow * kVoxWindow;
    p1 = (v1 + kVoxWindow - 1) / kVoxWindow * kVoxWindow;
    if (p1 > op->nV) p1 = op->nV;
}

// blocks of a launch: one per SM, a whole number for every part of the table
int sm_grid(const cgb_op *op, int parts, int voxels, int per_block) {
    int g = op->nsm / parts;
    const int need = (voxels + per_block - 1) / per_block;
    if (need < g) g = need;
    return parts * (g < 1 ? 1 : g);
}

template <class F, class A>
int launch_sm(F kern, int grid, int threads, size_t smem, cudaStream_t st, const A &a) {
    CGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kern<<<grid, threads, smem, st>>>(a);
    CGB_CUDA(cudaGetLastError());
    return CGB_OK;
}

}  // namespace

static thread_local bool in_place = false;
InPlaceScope::InPlaceScope(cudaStream_t st) : was(in_place) { in_place = in_place || capturing(st); }
InPlaceScope::~InPlaceScope() { in_place = was; }
bool in_place_only() { return in_place; }

// the handle's runs, laid out on first use (not under stream capture: the callers see to it)
int ensure_runs(cgb_op *op) {
    static std::mutex m;
    std::lock_guard<std::mutex> g(m);
    if (op->runs) return CGB_OK;
    RunLayout *R = new RunLayout();
    memset((void *)R, 0, sizeof(RunLayout));
    const int rc = build_runs(op, R);
    if (rc != CGB_OK) {
        drop_runs(op, R);
        return rc;
    }
    op->runs = R;
    return CGB_OK;
}

void free_runs(cgb_op *op) {
    if (op->runs) drop_runs(op, op->runs);
    op->runs = nullptr;
}

static void drop_plan(cgb_op *op, FfPlan *f) {
    void *p[] = {f->coef, f->fimg, f->colmax, f->aimg, f->run_blk, f->part, f->epart, f->zrow};
    for (void *q : p)
        if (q) cudaFree(q);
    if (f->order.done) cudaEventDestroy(f->order.done);
    op->bytes -= f->bytes;
    memset((void *)f, 0, sizeof(*f));
}

void free_ff_plan(cgb_op *op) {
    if (!op->ffp) return;
    drop_plan(op, op->ffp);
    delete op->ffp;
    op->ffp = nullptr;
}

// the handle's plan if the shared-memory kernels are to run this product, else null; `slots`: the pair
// kernels that would run it otherwise
static int plan_for(cgb_op *op, cudaStream_t st, unsigned slots, FfPlan **out) {
    *out = nullptr;
    if (in_place_only() || op->ff_variant != 1 || op->ff_pinned || (op->occ_set & slots)) return CGB_OK;
    if (op->nolut || op->nIC == 0 || op->n == 0 || op->nF == 0) return CGB_OK;
    if (op->nS < 17 || (double)op->n * op->nIC * op->nS < kSmemMinWork) return CGB_OK;
    if (!op->ffp) {
        if (capturing(st)) return CGB_OK;
        static std::mutex m;
        std::lock_guard<std::mutex> g(m);
        if (!op->ffp) {
            FfPlan *f = new FfPlan();
            memset((void *)f, 0, sizeof(*f));
            const bool had_runs = op->runs != nullptr;
            const int rc = build_plan(op, f);
            if (rc != CGB_OK) {
                drop_plan(op, f);
                if (!had_runs) free_runs(op);
                if (rc != CGB_ERR_NOMEM) {
                    delete f;
                    return rc;
                }
                f->no_room = 1;  // the plan stays empty and the pair kernels run
            }
            op->ffp = f;
        }
    }
    *out = op->ffp;
    return CGB_OK;
}

int queue_ff_images(cgb_op *op) { return op->ffp && op->ffp->colmax ? queue_images(op, op->ffp) : CGB_OK; }

int refresh_ff_plan(cgb_op *op) {
    if (!op->ffp) return CGB_OK;
    FfPlan *f = op->ffp;
    if (f->no_room) return CGB_OK;
    if (op->lut_signed || !f->colmax) {  // the choice of kernels changed: laid out anew
        free_ff_plan(op);
        return CGB_OK;
    }
    return finish_images(op, f);
}

// A x with the table in shared memory; *ran = 0 when the pair kernels are to do it
int forward_smem(cgb_op *op, const double *x, double *y, double *ax, const double *yobs, const double *sqw,
                 double *partials, cudaStream_t st, int *grid, int *ran) {
    *ran = 0;
    FfPlan *f;
    CGB_TRY(plan_for(op, st, kOccOfFwdFF, &f));
    if (!f || !f->fwd_ok) return CGB_OK;
    const OpDev P = op->dev();
    SmFwdArgs a;
    memset(&a, 0, sizeof(a));
    const RunLayout &R = *op->runs;
    a.vperm = R.vperm; a.run_ptr = R.run_ptr; a.run_o = R.run_o; a.coef = f->coef; a.nruns = R.nruns;
    a.img = f->fimg; a.colmax = f->colmax;
    a.coef_max = f->uneven ? -1.f : 3.0e38f;
    a.nIC = op->nIC; a.ndirs = op->ndirs; a.nS = op->nS; a.nc = f->fnc;
    perm_range(op, a.v0, a.v1, a.p0, a.p1);
    a.ec_ptr = op->ec_ptr; a.ec_col = op->ec_col; a.ec_o = op->ec_o; a.iso_ptr = op->iso_ptr; a.iso_col = op->iso_col;
    a.lutEC = op->lutEC_p; a.lutISO = op->lutISO_p; a.nSp = op->nSp;
    a.nEC = op->nE > 0 ? op->nEC : 0; a.nISO = op->nISOv > 0 ? op->nISO : 0;
    a.ec_base = P.ec_base; a.iso_base = P.iso_base; a.nE = op->nE; a.nISOv = op->nISOv;
    a.x = x; a.xmax = P.xmax; a.lut_exp = P.lut_exp_fwd;
    a.yout = y; a.axout = ax; a.yobs = yobs; a.sqw = sqw; a.partials = partials;
    a.vec_ok = ((uintptr_t)y % 16 == 0) && ((uintptr_t)ax % 16 == 0);
    // the coefficients belong to the handle: a product on another stream waits for the last
    // one (under capture the graph's own order applies)
    const bool cap = capturing(st);
    if (!cap) CGB_TRY(order_enter(&f->order, st));
    if (op->vr1 <= 0 || op->vr0 == 0)
        k_run_coef<<<grid_n((R.nruns + kCoefRuns - 1) / kCoefRuns), 256, 0, st>>>(P, R.run_seg, R.nruns, x, R.eval_ones,
                                                                                  f->coef);
    CGB_CUDA(cudaGetLastError());
    const int g = sm_grid(op, f->fnc, a.p1 - a.p0, kFwdThreads / 8);
    const size_t smem = (size_t)op->nIC * op->ndirs * f->fcs * sizeof(float);
    int rc = CGB_ERR_UNSUPPORTED;
    switch (f->fnp) {
        case 2: rc = launch_sm(k_fwd_smem<2>, g, kFwdThreads, smem, st, a); break;
        case 3: rc = launch_sm(k_fwd_smem<3>, g, kFwdThreads, smem, st, a); break;
        case 4: rc = launch_sm(k_fwd_smem<4>, g, kFwdThreads, smem, st, a); break;
        case 5: rc = launch_sm(k_fwd_smem<5>, g, kFwdThreads, smem, st, a); break;
        case 6: rc = launch_sm(k_fwd_smem<6>, g, kFwdThreads, smem, st, a); break;
    }
    CGB_TRY(rc);
    if (!cap) CGB_TRY(order_leave(&f->order, st));
    if (grid) *grid = g;
    *ran = 1;
    return CGB_OK;
}

// voxel pass of A' with the table in shared memory over the current voxel range
int adjoint_smem(cgb_op *op, const double *z, double *xout, cudaStream_t st, int *ran) {
    *ran = 0;
    FfPlan *f;
    CGB_TRY(plan_for(op, st, kOccOfAdjFF, &f));
    if (!f || !f->adj_ok) return CGB_OK;
    const OpDev P = op->dev();
    SmAdjArgs a;
    memset(&a, 0, sizeof(a));
    const RunLayout &R = *op->runs;
    a.vperm = R.vperm; a.run_blk = f->run_blk; a.run_seg = R.run_seg; a.run_o = R.run_o; a.seg_l = op->seg_l;
    a.n = op->n; a.nruns = R.nruns; a.img = f->aimg; a.colmax = f->colmax;
    a.general = f->uneven ? 0x80000000u : 0u;
    a.nIC = op->nIC; a.nS = op->nS; a.nV = op->nV; a.nc = f->anc; a.nb = f->anb; a.no = f->ano;
    perm_range(op, a.v0, a.v1, a.p0, a.p1);
    a.ec_ptr = op->ec_ptr; a.ec_col = op->ec_col; a.ec_o = op->ec_o; a.iso_ptr = op->iso_ptr; a.iso_col = op->iso_col;
    a.lutEC = op->lutEC_p; a.lutISO = op->lutISO_p; a.nSp = op->nSp; a.ndirs = op->ndirs;
    a.nEC = op->nE > 0 ? op->nEC : 0; a.nISO = op->nISOv > 0 ? op->nISO : 0;
    a.ec_base = P.ec_base; a.iso_base = P.iso_base; a.nE = op->nE; a.nISOv = op->nISOv;
    a.z = z; a.lut_exp = P.lut_exp_adj; a.vec_ok = (uintptr_t)z % 16 == 0;
    a.scratch = op->scratch; a.xout = xout; a.part = f->part; a.epart = f->epart;
    const int g = sm_grid(op, f->anc * f->anb, a.p1 - a.p0, adj_threads(f->anp) / 8);
    const size_t smem = (size_t)op->nIC * f->ano * f->acs * sizeof(float);
    int rc = CGB_ERR_UNSUPPORTED;
    switch (f->anp) {
        case 2: rc = launch_sm(k_adj_smem<2>, g, adj_threads(2), smem, st, a); break;
        case 3: rc = launch_sm(k_adj_smem<3>, g, adj_threads(3), smem, st, a); break;
        case 4: rc = launch_sm(k_adj_smem<4>, g, adj_threads(4), smem, st, a); break;
        case 5: rc = launch_sm(k_adj_smem<5>, g, adj_threads(5), smem, st, a); break;
        case 6: rc = launch_sm(k_adj_smem<6>, g, adj_threads(6), smem, st, a); break;
    }
    CGB_TRY(rc);
    {
        const int64_t runs = R.nruns * (a.v1 - a.v0) / op->nV + 1;
        const int64_t blocks = (runs + 255) / 256, cap = (int64_t)op->nsm * 32;
        k_adj_join<<<(int)(blocks < cap ? blocks : cap), 256, 0, st>>>(a, R.run_ptr);
        CGB_CUDA(cudaGetLastError());
    }
    *ran = 1;
    return CGB_OK;
}

// z = the weighted residual of a gradient pass in the plan's row buffer (in_mode 1 computes
// A x first); *z stays null when the pair kernels are to do the gradient
int residual_smem(cgb_op *op, int in_mode, const double *x, const double *yobs, const double *sqw, const double *ax_a,
                  const double *ax_b, double ca, double cb, double *partials, cudaStream_t st, int *grid,
                  const double **z) {
    *z = nullptr;
    FfPlan *f;
    CGB_TRY(plan_for(op, st, kOccOfGradFF, &f));
    if (!f || !f->adj_ok || !f->fwd_ok) return CGB_OK;
    if (!f->zrow) {
        if (capturing(st)) return CGB_OK;
        const int rc = keep_buffer(op, &f->bytes, &f->zrow, (size_t)op->nrows);
        if (rc == CGB_ERR_NOMEM) return CGB_OK;
        CGB_TRY(rc);
    }
    if (in_mode == 1) {
        int ran = 0;
        CGB_TRY(forward_smem(op, x, f->zrow, nullptr, nullptr, nullptr, nullptr, st, nullptr, &ran));
        if (!ran) return CGB_OK;
        ax_a = f->zrow;
    }
    int g = (int)((op->nrows + kBlock - 1) / kBlock);
    if (g > op->nsm * 8) g = op->nsm * 8;
    k_residual<<<g, kBlock, 0, st>>>(op->nrows, in_mode, ax_a, ax_b, ca, cb, yobs, sqw, f->zrow, partials);
    CGB_CUDA(cudaGetLastError());
    if (grid) *grid = g;
    *z = f->zrow;
    return CGB_OK;
}

}  // namespace cgb
