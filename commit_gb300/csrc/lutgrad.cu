// Gradient of a loss with respect to the response-function LUTs, and LUT updates.
//
// y[v,s] depends linearly on the LUT entries: y[v,s] = sum over items of the voxel of
// c * LUT[row(item), s] with c = l*x*eval (IC), x (EC, ISO).  For an upstream gradient
// g = dLoss/dy the LUT gradient is therefore
//   G_IC[i,o,s]  = sum over IC segments j with orientation o of c_{j,i} * g[v_j, s]
//   G_EC[i,o,s]  = sum over EC elements e with orientation o of x_{EC,i,e} * g[v_e, s]
//   G_ISO[i,s]   = sum over ISO elements j of x_{ISO,i,j} * g[v_j, s].
// The items of a voxel with one orientation are adjacent (voxel-order arrays) and share g[v]:
// they are one run, whose coefficient is formed first.  The runs are visited in an
// orientation-sorted order (built once, on first use), split into chunks that never straddle
// an orientation; a warp reduces one chunk (FP64) into a partial row, and a second pass adds the
// partial rows of each orientation in chunk order -- deterministic, no atomics.
//
// Bound: the FP64 pipe (2 lanes / clock / SM).  A warp takes 32 runs at a time, a lane per run
// for the coefficients, then as many runs side by side as lanes-per-run leaves room for, so that
// the lanes of the FP64 multiply-adds are filled (66 samples: 4 runs of 8 lanes x 9 samples,
// 92 % of the slots, instead of 32 lanes x 3, 69 %).  50k streamlines in 12k voxels, nS = 66:
// 4.7 -> 0.53 ms for the IC rows (one warp walked 1024 segments in a chain of dependent loads);
// 2.9 M runs x 66 multiply-adds are 0.44 ms of that pipe.
#include <cub/cub.cuh>

#include <memory>
#include <vector>

#include "cgb_internal.cuh"

namespace cgb {
namespace {

struct GradStream {
    // runs of one compartment in orientation order: voxel, items [beg, end) (voxel-order positions)
    uint32_t *run_v = nullptr, *run_b = nullptr, *run_e = nullptr;
    uint32_t *chunk_beg = nullptr;  // per chunk: first run
    uint32_t *row_chunk = nullptr;  // [nrow+1] chunks of row o
    int nchunks = 0;
    ~GradStream() {
        void *p[] = {run_v, run_b, run_e, chunk_beg, row_chunk};
        for (void *q : p)
            if (q) cudaFree(q);
    }
};

// device buffers of the set-up, released on every way out
struct Temps {
    std::vector<void *> p;
    ~Temps() {
        for (void *q : p) cudaFree(q);
    }
    template <class T>
    int get(T **out, size_t n) {
        void *q = nullptr;
        CGB_CUDA(cudaMalloc(&q, (n ? n : 1) * sizeof(T)));
        p.push_back(q);
        *out = (T *)q;
        return CGB_OK;
    }
};

int grid_n(int64_t n) {
    int64_t g = (n + 255) / 256;
    if (g > 4096) g = 4096;
    if (g < 1) g = 1;
    return (int)g;
}

__global__ void k_run_head(const uint16_t *__restrict__ o, int64_t n, uint32_t *__restrict__ head) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
        head[j] = j == 0 || o[j] != o[j - 1];
}

__global__ void k_voxel_head(const uint32_t *__restrict__ ptr, int nV, uint32_t *__restrict__ head) {
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v < nV && ptr[v] < ptr[v + 1]) head[ptr[v]] = 1u;
}

// run number, orientation and first item of every run, in voxel order
__global__ void k_run_list(const uint32_t *__restrict__ head, const uint32_t *__restrict__ id,
                           const uint16_t *__restrict__ o, int64_t n, uint32_t *__restrict__ key,
                           uint32_t *__restrict__ num, uint32_t *__restrict__ first) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x)
        if (head[j]) {
            key[id[j]] = o[j];
            num[id[j]] = id[j];
            first[id[j]] = (uint32_t)j;
        }
}

__global__ void k_run_voxel(const uint32_t *__restrict__ ptr, const uint32_t *__restrict__ head,
                            const uint32_t *__restrict__ id, int nV, uint32_t *__restrict__ vox) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < nV; v += gridDim.x * blockDim.x)
        for (uint32_t j = ptr[v]; j < ptr[v + 1]; ++j)
            if (head[j]) vox[id[j]] = (uint32_t)v;
}

__global__ void k_run_gather(const uint32_t *__restrict__ num, const uint32_t *__restrict__ first,
                             const uint32_t *__restrict__ vox, int64_t nr, uint32_t n, uint32_t *__restrict__ run_v,
                             uint32_t *__restrict__ run_b, uint32_t *__restrict__ run_e) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < nr; q += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t r = num[q];
        run_v[q] = vox[r];
        run_b[q] = first[r];
        run_e[q] = r + 1 < nr ? first[r + 1] : n;
    }
}

// first run of each orientation (the sorted keys' lower bounds)
__global__ void k_row_first(const uint32_t *__restrict__ key, int64_t nr, int nrows, uint32_t *__restrict__ off) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r > nrows) return;
    int64_t lo = 0, hi = nr;
    while (lo < hi) {
        const int64_t m = (lo + hi) / 2;
        if (key[m] < (uint32_t)r) lo = m + 1;
        else hi = m;
    }
    off[r] = (uint32_t)lo;
}

// Runs of `n` voxel-ordered items with orientations o[] and voxel offsets ptr[], in orientation
// order and chunked.
int build_stream(const uint16_t *o, const uint32_t *ptr, int nV, int64_t n, int nrows, int nsm, GradStream &S) {
    std::vector<uint32_t> h_off(nrows + 1, 0);
    int64_t nr = 0;
    if (n > 0) {
        Temps T;
        uint32_t *head, *id, *key, *key2, *num, *num2, *first, *vox, *off;
        char *tmp;
        CGB_TRY(T.get(&head, n));
        CGB_TRY(T.get(&id, n));
        k_run_head<<<grid_n(n), 256>>>(o, n, head);
        k_voxel_head<<<(nV + 255) / 256, 256>>>(ptr, nV, head);
        size_t b1 = 0, b2 = 0;
        CGB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, b1, head, id, (int)n));
        CGB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, b2, head, head, head, head, (int)n, 0, 16));
        CGB_TRY(T.get(&tmp, b1 > b2 ? b1 : b2));
        CGB_CUDA(cub::DeviceScan::ExclusiveSum(tmp, b1, head, id, (int)n));
        uint32_t last[2];
        CGB_CUDA(cudaMemcpy(&last[0], id + n - 1, 4, cudaMemcpyDeviceToHost));
        CGB_CUDA(cudaMemcpy(&last[1], head + n - 1, 4, cudaMemcpyDeviceToHost));
        nr = (int64_t)last[0] + last[1];
        CGB_TRY(T.get(&key, nr));
        CGB_TRY(T.get(&key2, nr));
        CGB_TRY(T.get(&num, nr));
        CGB_TRY(T.get(&num2, nr));
        CGB_TRY(T.get(&first, nr));
        CGB_TRY(T.get(&vox, nr));
        CGB_TRY(T.get(&off, nrows + 1));
        k_run_list<<<grid_n(n), 256>>>(head, id, o, n, key, num, first);
        k_run_voxel<<<grid_n(nV), 256>>>(ptr, head, id, nV, vox);
        CGB_CUDA(cub::DeviceRadixSort::SortPairs(tmp, b2, key, key2, num, num2, (int)nr, 0, 16));
        CGB_CUDA(cudaMalloc((void **)&S.run_v, nr * sizeof(uint32_t)));
        CGB_CUDA(cudaMalloc((void **)&S.run_b, nr * sizeof(uint32_t)));
        CGB_CUDA(cudaMalloc((void **)&S.run_e, nr * sizeof(uint32_t)));
        k_run_gather<<<grid_n(nr), 256>>>(num2, first, vox, nr, (uint32_t)n, S.run_v, S.run_b, S.run_e);
        k_row_first<<<(nrows + 256) / 256, 256>>>(key2, nr, nrows, off);
        CGB_CUDA(cudaMemcpy(h_off.data(), off, h_off.size() * sizeof(uint32_t), cudaMemcpyDeviceToHost));
    }
    // chunks: enough for several warps per scheduler, 1024 runs at most
    int64_t chunk = (nr / ((int64_t)nsm * 96) + 31) / 32 * 32;
    chunk = chunk < 32 ? 32 : (chunk > 1024 ? 1024 : chunk);
    std::vector<uint32_t> cb, rc(nrows + 1, 0);
    for (int r = 0; r < nrows; ++r) {
        rc[r] = (uint32_t)cb.size();
        for (int64_t p = h_off[r]; p < h_off[r + 1]; p += chunk) cb.push_back((uint32_t)p);
    }
    rc[nrows] = (uint32_t)cb.size();
    S.nchunks = (int)cb.size();
    cb.push_back((uint32_t)nr);  // sentinel: end of the last chunk
    CGB_CUDA(cudaMalloc((void **)&S.chunk_beg, cb.size() * sizeof(uint32_t)));
    CGB_CUDA(cudaMalloc((void **)&S.row_chunk, rc.size() * sizeof(uint32_t)));
    CGB_CUDA(cudaMemcpy(S.chunk_beg, cb.data(), cb.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    CGB_CUDA(cudaMemcpy(S.row_chunk, rc.data(), rc.size() * sizeof(uint32_t), cudaMemcpyHostToDevice));
    return CGB_OK;
}

// one warp per chunk: partial[chunk, s] = sum over the chunk's runs of c * g[v, s], LG lanes a
// run and K samples a lane (samples beyond LG * K in further rounds)
// kind 0: IC (c = sum of l * x[i*nF + f] * eval), kind 1: EC (c = sum of x[ec_base + i*nE + col])
template <int LG, int K>
__global__ void __launch_bounds__(256) k_grad_chunks(const OpDev P, int kind, int rf, const uint32_t *__restrict__ run_v,
                                                     const uint32_t *__restrict__ run_b,
                                                     const uint32_t *__restrict__ run_e,
                                                     const uint32_t *__restrict__ chunk_beg, int nchunks,
                                                     const double *__restrict__ x, const double *__restrict__ g,
                                                     double *__restrict__ partial) {
    constexpr int W = 32 / LG;  // runs side by side
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & (LG - 1), grp = lane / LG;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int nS = P.nS;
    for (int c = warp; c < nchunks; c += nw) {
        const uint32_t b = chunk_beg[c], e = chunk_beg[c + 1];
        for (int s0 = 0; s0 < nS; s0 += LG * K) {
            double acc[K];
#pragma unroll
            for (int k = 0; k < K; ++k) acc[k] = 0.0;
            for (uint32_t p = b; p < e; p += 32) {
                const uint32_t r = p + lane;
                double coef = 0.0;
                uint32_t v = 0;
                if (r < e) {
                    v = run_v[r];
                    for (uint32_t j = run_b[r]; j < run_e[r]; ++j) {
                        if (kind == 0) {
                            const size_t col = (size_t)rf * P.nF + P.seg_f[j];
                            coef += (double)P.seg_l[j] * (x[col] * (double)P.eval[col]);
                        } else {
                            coef += x[P.ec_base + (size_t)rf * P.nE + P.ec_col[j]];
                        }
                    }
                }
                const int cnt = (int)min(32u, e - p);
                __syncwarp();
                for (int t = 0; t < cnt; t += W) {
                    const double ct = __shfl_sync(full, coef, t + grp);
                    const uint32_t vt = __shfl_sync(full, v, t + grp);
                    if (__any_sync(full, ct != 0.0)) {
                        const double *gr = g + (size_t)vt * nS + s0 + sub;
                        double z[K];
#pragma unroll
                        for (int k = 0; k < K; ++k) z[k] = ct != 0.0 && s0 + sub + LG * k < nS ? __ldg(gr + LG * k) : 0.0;
#pragma unroll
                        for (int k = 0; k < K; ++k) acc[k] = fma(ct, z[k], acc[k]);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < K; ++k) {
#pragma unroll
                for (int d = LG; d < 32; d <<= 1) acc[k] += __shfl_xor_sync(full, acc[k], d);
                const int s = s0 + sub + LG * k;
                if (grp == 0 && s < nS) partial[(size_t)c * nS + s] = acc[k];
            }
        }
    }
}

// lanes per run and samples per lane: the fewest FP64 slots per run
int launch_chunks(const cgb_op *op, int kind, int rf, const GradStream &S, const double *x, const double *g,
                  double *partial, cudaStream_t st) {
    const OpDev P = op->dev();
    int best = 0, cost = 1 << 30;
    const int lg[5] = {8, 8, 16, 16, 32}, kk[5] = {9, 12, 9, 12, 9};
    for (int i = 0; i < 5; ++i) {
        const int rounds = (op->nS + lg[i] * kk[i] - 1) / (lg[i] * kk[i]);
        const int slots = rounds * (lg[i] * kk[i] + 16);  // a round reads the runs again
        if (slots < cost) {
            cost = slots;
            best = i;
        }
    }
    const int blocks = op->nsm * 8;
#define CGB_GRAD(I, L, K)                                                                                        \
    if (best == I)                                                                                               \
        k_grad_chunks<L, K><<<blocks, 256, 0, st>>>(P, kind, rf, S.run_v, S.run_b, S.run_e, S.chunk_beg, S.nchunks, \
                                                    x, g, partial);
    CGB_GRAD(0, 8, 9) CGB_GRAD(1, 8, 12) CGB_GRAD(2, 16, 9) CGB_GRAD(3, 16, 12) CGB_GRAD(4, 32, 9)
#undef CGB_GRAD
    CGB_CUDA(cudaGetLastError());
    return CGB_OK;
}

// out[row, s] = sum of the row's chunk partials in chunk order
__global__ void k_grad_rows(const double *__restrict__ partial, const uint32_t *__restrict__ row_chunk, int nrows,
                            int nS, double *__restrict__ out) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < (int64_t)nrows * nS;
         q += (int64_t)gridDim.x * blockDim.x) {
        const int r = (int)(q / nS), s = (int)(q - (int64_t)r * nS);
        double t = 0.0;
        for (uint32_t c = row_chunk[r]; c < row_chunk[r + 1]; ++c) t += partial[(size_t)c * nS + s];
        out[q] = t;
    }
}

// ISO: one warp per voxel block partial over voxels, then a fixed-order sum
__global__ void k_grad_iso(const OpDev P, int rf, const double *__restrict__ x, const double *__restrict__ g,
                           double *__restrict__ partial) {
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const int nS = P.nS;
    for (int s0 = 0; s0 < nS; s0 += 32) {
        const int s = s0 + lane;
        double acc = 0.0;
        for (int v = warp; v < P.nV; v += nw)
            for (uint32_t j = P.iso_ptr[v]; j < P.iso_ptr[v + 1]; ++j) {
                const double c = x[P.iso_base + (size_t)rf * P.nISOv + P.iso_col[j]];
                if (s < nS) acc = fma(c, g[(size_t)v * nS + s], acc);
            }
        if (s < nS) partial[(size_t)warp * nS + s] = acc;
    }
}

// one block per sample: the column sum of the partial rows, fixed order
__global__ void __launch_bounds__(256) k_sum_rows(const double *__restrict__ partial, int nparts, int nS,
                                                  double *__restrict__ out) {
    __shared__ double red[8];
    double t = 0.0;
    for (int w = threadIdx.x; w < nparts; w += 256) t += partial[(size_t)w * nS + blockIdx.x];
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w];
        out[blockIdx.x] = t;
    }
}

}  // namespace

struct LutGradState {
    GradStream ic, ec;
    double *partial = nullptr;
    size_t partial_len = 0;
    ~LutGradState() {
        if (partial) cudaFree(partial);
    }
};

static int ensure_grad_state(cgb_op *op) {
    if (op->gstate) return CGB_OK;
    std::unique_ptr<LutGradState> G(new LutGradState());
    if (op->nIC > 0 && op->n > 0)
        CGB_TRY(build_stream(op->seg_o, op->vox_ptr, op->nV, op->n, op->ndirs, op->nsm, G->ic));
    if (op->nEC > 0 && op->nE > 0)
        CGB_TRY(build_stream(op->ec_o, op->ec_ptr, op->nV, op->nE, op->ndirs, op->nsm, G->ec));
    const int nwarps_iso = op->nsm * 32;
    size_t need = (size_t)std::max(std::max(G->ic.nchunks, G->ec.nchunks), nwarps_iso) * op->nS;
    CGB_CUDA(cudaMalloc((void **)&G->partial, (need ? need : 1) * sizeof(double)));
    G->partial_len = need;
    CGB_CUDA(cudaDeviceSynchronize());
    op->gstate = G.release();  // complete: a call that failed on the way leaves none
    return CGB_OK;
}

void free_grad_state(cgb_op *op) {
    if (op->gstate) {
        delete (LutGradState *)op->gstate;
        op->gstate = nullptr;
    }
}

}  // namespace cgb

using namespace cgb;

extern "C" {

int cgb_op_lut_grad(cgb_op *op, const double *x, const double *g, double *g_ic, double *g_ec, double *g_iso,
                    void *stream) {
    if (!op || !x || !g) return fail(CGB_ERR_INVALID, "null argument");
    if (op->nolut) return fail(CGB_ERR_UNSUPPORTED, "the LUT-free operator has no LUT");
    CGB_TRY(ensure_grad_state(op));
    LutGradState *G = (LutGradState *)op->gstate;
    cudaStream_t st = (cudaStream_t)stream;
    const OpDev P = op->dev();
    const int nS = op->nS;
    const size_t rowlen = (size_t)op->ndirs * nS;
    if (g_ic && op->nIC > 0) {
        for (int i = 0; i < op->nIC; ++i) {
            double *out = g_ic + (size_t)i * rowlen;
            if (G->ic.nchunks == 0) {
                CGB_CUDA(cudaMemsetAsync(out, 0, rowlen * sizeof(double), st));
                continue;
            }
            CGB_TRY(launch_chunks(op, 0, i, G->ic, x, g, G->partial, st));
            k_grad_rows<<<grid_n((int64_t)op->ndirs * nS), 256, 0, st>>>(G->partial, G->ic.row_chunk, op->ndirs, nS,
                                                                        out);
            CGB_CUDA(cudaGetLastError());
        }
    }
    if (g_ec && op->nEC > 0) {
        for (int i = 0; i < op->nEC; ++i) {
            double *out = g_ec + (size_t)i * rowlen;
            if (G->ec.nchunks == 0) {
                CGB_CUDA(cudaMemsetAsync(out, 0, rowlen * sizeof(double), st));
                continue;
            }
            CGB_TRY(launch_chunks(op, 1, i, G->ec, x, g, G->partial, st));
            k_grad_rows<<<grid_n((int64_t)op->ndirs * nS), 256, 0, st>>>(G->partial, G->ec.row_chunk, op->ndirs, nS,
                                                                        out);
            CGB_CUDA(cudaGetLastError());
        }
    }
    if (g_iso && op->nISO > 0) {
        const int blocks = op->nsm * 4;  // 32 warps per SM-block set -> nsm*32 partial rows
        for (int i = 0; i < op->nISO; ++i) {
            k_grad_iso<<<blocks, 256, 0, st>>>(P, i, x, g, G->partial);
            k_sum_rows<<<nS, 256, 0, st>>>(G->partial, blocks * 8, nS, g_iso + (size_t)i * nS);
            CGB_CUDA(cudaGetLastError());
        }
    }
    return CGB_OK;
}

}  // extern "C"
