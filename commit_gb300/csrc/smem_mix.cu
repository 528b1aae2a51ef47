// Plan, coefficient and join passes and launches of the shared-memory reduced-precision
// products (smem_mix.cuh).
#include <mutex>

#include "smem_mix.cuh"

namespace cgb {
namespace {

using namespace detail;

// table image [chunk][row][cs] from rows of stride nSp, zero beyond the chunk's samples
template <class T>
__global__ void k_mix_image(const T *__restrict__ lut, int rows, int nS, int nSp, int nc, int width, int cs,
                            T *__restrict__ img) {
    const int64_t total = (int64_t)nc * rows * cs;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total; q += (int64_t)gridDim.x * blockDim.x) {
        const int k = (int)(q % cs);
        const int64_t t = q / cs;
        const int r = (int)(t % rows), s = (int)(t / rows) * width + k;
        img[q] = k < width && s < nS ? lut[(size_t)r * nSp + s] : T(0);
    }
}

// run coefficients sum(l * x * eval) in FP32, four runs in flight per thread (as k_run_coef)
template <bool F32>
__global__ void __launch_bounds__(256) k_mix_coef(const __grid_constant__ SmMixArgs A, const uint32_t *__restrict__ seg_f,
                                                  const uint32_t *__restrict__ eval, int nF) {
    constexpr int U = 4;
    for (int64_t r0 = blockIdx.x * (256ll * U) + threadIdx.x; r0 < A.nruns; r0 += (int64_t)gridDim.x * (256 * U)) {
        uint32_t beg[U], end[U], f[U];
        float l[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int64_t r = r0 + 256 * u < A.nruns ? r0 + 256 * u : A.nruns - 1;
            beg[u] = A.run_seg[r];
            end[u] = A.run_seg[r + 1];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            f[u] = seg_f[beg[u]];
            l[u] = mix_length<F32>(A, beg[u]);
        }
        for (int i = 0; i < A.nIC; ++i) {
            const float *x = A.x + (size_t)i * nF;
            const uint32_t *ev = eval ? eval + (size_t)i * nF : nullptr;
            float c[U];
#pragma unroll
            for (int u = 0; u < U; ++u) c[u] = l[u] * x[f[u]] * (ev ? (float)ev[f[u]] : 1.f);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                for (uint32_t j = beg[u] + 1; j < end[u]; ++j)
                    c[u] += mix_length<F32>(A, j) * x[seg_f[j]] * (ev ? (float)ev[seg_f[j]] : 1.f);
                if (r0 + 256 * u < A.nruns) A.coef[(size_t)i * A.nruns + r0 + 256 * u] = c[u];
            }
        }
    }
}

// several chunks: terms l * <L, z> of the segments of the voxels [v0, v1) from the runs' parts, and
// their EC / ISO columns
template <bool F32>
__global__ void __launch_bounds__(256) k_mix_join(const __grid_constant__ SmMixArgs A) {
    const int64_t first = blockIdx.x * 256ll + threadIdx.x, step = gridDim.x * 256ll;
    const int64_t r0 = A.run_ptr[A.v0], r1 = A.run_ptr[A.v1];
    for (int64_t r = r0 + first; r < r1; r += step) {
        const uint32_t sb = A.run_seg[r], se = A.run_seg[r + 1];
        const float l0 = mix_length<F32>(A, sb);
        for (int i = 0; i < A.nIC; ++i) {
            const float *q = A.part + ((size_t)i * A.nruns + r) * A.nc;
            float t = q[0], e = 0.f;
            for (int c = 1; c < A.nc; ++c) {
                float d;
                t = sum_err(t, q[c], d);
                e += d;
            }
            float *out = A.scratch + (size_t)i * A.n;
            out[sb] = fmaf(l0, t, l0 * e);
            for (uint32_t g = sb + 1; g < se; ++g) {
                const float l = mix_length<F32>(A, g);
                out[g] = fmaf(l, t, l * e);
            }
        }
    }
    auto column = [&](int64_t col) {
        double t = A.epart[col * A.nc];
        for (int c = 1; c < A.nc; ++c) t += A.epart[col * A.nc + c];
        A.xout[A.ec_base + col] = t;
    };
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

int grid_of(int64_t n, int cap) {
    int64_t g = (n + 255) / 256;
    if (g > cap) g = cap;
    return (int)(g < 1 ? 1 : g);
}

// chunks of at most 192 samples whose table fits in a block's shared memory
bool mix_shape(const cgb_op *op, int word, MixPlan *m) {
    const int64_t rows = (int64_t)op->nIC * op->ndirs;
    for (int nc = (op->nS + 191) / 192; nc <= 8; ++nc) {
        const int nq = (op->nS + 32 * nc - 1) / (32 * nc), cs = word == 2 ? (32 * nq + 63) / 64 * 64 : 32 * nq;
        if (32 * nq * (nc - 1) >= op->nS) continue;  // the last chunk would be empty
        if (rows * cs * word <= (224 << 10)) {
            m->nq = nq;
            m->nc = nc;
            m->cs = cs;
            return true;
        }
    }
    return false;
}

void drop(cgb_op *op, MixPlan *m) {
    void *p[] = {m->img, m->coef, m->part, m->epart};
    for (void *q : p)
        if (q) cudaFree(q);
    op->bytes -= m->bytes;
    m->bytes = 0;
    m->img = nullptr;
    m->coef = m->part = nullptr;
    m->epart = nullptr;
}

int build_mix(cgb_op *op, int word, MixPlan *m) {
    CGB_TRY(ensure_runs(op));
    const int64_t runs = op->runs->nruns * op->nIC;
    CGB_TRY(keep_buffer(op, &m->bytes, &m->coef, (size_t)runs));
    if (m->nc > 1) CGB_TRY(keep_buffer(op, &m->bytes, &m->part, (size_t)runs * m->nc));
    if (m->nc > 1) CGB_TRY(keep_buffer(op, &m->bytes, &m->epart, ((size_t)op->nE * op->nEC + (size_t)op->nISOv * op->nISO) * m->nc));
    CGB_TRY(keep_buffer(op, &m->bytes, &m->img, (size_t)m->nc * op->nIC * op->ndirs * m->cs * word));
    CGB_TRY(order_create(&m->order));
    return CGB_OK;
}

// Where these kernels take over: the size from which FP64 vectors build the same run layout, and
// 0.5 segments x responses per voxel, or 3 per chunk where there are several (each reads the runs
// again).  Measured, us, here / gathering kernels: one chunk (FP16), 0.8 per voxel A 44 / 61 and A'
// 51 / 73, 48 per voxel 30 / 50 and 45 / 55, 27 per voxel 68 / 122 and 99 / 155; two chunks (FP32,
// 145 samples), 3.3 per voxel A 55 / 50, 13 per voxel 68 / 73 and 89 / 113; two responses (five
// chunks) 152 / 169 and 231 / 249.  Below, the layout costs more than a few products.
inline double mix_min_items(int nc) { return nc == 1 ? 0.5 : 3.0 * nc; }
// Against the tensor-core kernels (BF16), whose time hardly depends on the samples but grows with
// every segment, where this one follows the runs and the quads of samples: A here up to 6 quads x
// responses, A' up to 4, and up to 6 from 300 segments per voxel on.  Measured (us, here / tensor
// cores): 10 M segments, 200 per voxel: 145 samples (5 quads) A 204 / 249 and A' 297 / 304, 280
// samples (10) 314 / 255 and 467 / 367; 184 per voxel, 145 samples A 977 / 1188 and A'
// 1503 / 1420; 598 per voxel 406 / 541 and 693 / 950; 176 per voxel, 99 samples (4) 1396 / 1830
// and 2211 / 2348; three responses (15) 415 / 383 and 599 / 441.
constexpr int64_t kTcAdjDense = 300;

// the handle's plan with the image of `arith`, or null where the gathering kernels are to run.
// Its buffers stay where they are for the handle's life: the shape does not depend on `arith`.
int mix_plan(cgb_op *op, cudaStream_t st, int arith, int adjoint, MixPlan **out) {
    *out = nullptr;
    if (in_place_only() || op->ff_pinned || (op->occ_set & occ_of_mix(arith, adjoint))) return CGB_OK;
    if (op->nolut || op->nIC == 0 || op->n == 0 || op->nF == 0) return CGB_OK;
    const int f32 = arith == CGB_ARITH_F32, word = f32 ? 4 : 2;
    const bool tc = arith == CGB_ARITH_BF16 && tc_forward_enabled(op);
    if (tc && op->tc_mode == 2) return CGB_OK;
    // an entry that is not finite, as it stands or in FP16: a zero coefficient must skip its row
    if ((op->lut_signed & 2) || op->lut_exp_adj > (arith == CGB_ARITH_FP16 ? 14 : 126)) return CGB_OK;
    if (op->nS < 17 || (double)op->n * op->nIC * op->nS < kSmemMinWork) return CGB_OK;
    MixPlan shape{};
    if (!mix_shape(op, word, &shape) || (double)op->n * op->nIC < mix_min_items(shape.nc) * op->nV) return CGB_OK;
    if (tc && op->nIC * shape.nc * shape.nq > (adjoint && op->n < kTcAdjDense * op->nV ? 4 : 6)) return CGB_OK;
    if (op->mixp[f32] && !op->mixp[f32]->img) return CGB_OK;  // there was no room
    // only now: a product that ends on other kernels prepares the reduced tables itself, and the
    // preparation waits for the device
    CGB_TRY(ensure_reduced(op, arith));
    static std::mutex mu;
    std::lock_guard<std::mutex> g(mu);
    if (!op->mixp[f32] || (op->mixp[f32]->img && op->mixp_kind[f32] != arith)) {
        CGB_CUDA(cudaDeviceSynchronize());
        if (!op->mixp[f32]) {
            MixPlan *m = new MixPlan(shape);
            const bool had_runs = op->runs != nullptr;
            const int rc = build_mix(op, word, m);
            if (rc != CGB_OK) {
                drop(op, m);
                if (!had_runs) free_runs(op);
                if (rc != CGB_ERR_NOMEM) {
                    delete m;
                    return rc;
                }
                // no room: the plan stays empty and the gathering kernels run
            }
            op->mixp[f32] = m;
        }
        MixPlan *m = op->mixp[f32];
        if (m->img) {
            const int rows = op->nIC * op->ndirs;
            const int g = grid_of((int64_t)m->nc * rows * m->cs, 4096);
            if (f32)
                k_mix_image<<<g, 256>>>(op->lutIC_p, rows, op->nS, op->nSp, m->nc, 32 * m->nq, m->cs, (float *)m->img);
            else
                k_mix_image<<<g, 256>>>((const uint16_t *)op->lut_r_ic(arith), rows, op->nS, op->nSp_r, m->nc,
                                        32 * m->nq, m->cs, (uint16_t *)m->img);
            CGB_CUDA(cudaGetLastError());
            CGB_CUDA(cudaDeviceSynchronize());
            op->mixp_kind[f32] = arith;
        }
    }
    if (op->mixp[f32]->img) *out = op->mixp[f32];
    return CGB_OK;
}

SmMixArgs mix_args(const cgb_op *op, const MixPlan *m, int arith) {
    const RunLayout &R = *op->runs;
    const OpDev P = op->dev();
    SmMixArgs a{};
    a.vperm = R.vperm; a.run_ptr = R.run_ptr; a.run_seg = R.run_seg; a.run_o = R.run_o;
    a.n = op->n; a.nruns = R.nruns; a.img = m->img;
    a.nIC = op->nIC; a.ndirs = op->ndirs; a.nS = op->nS; a.nV = op->nV; a.nc = m->nc;
    a.v0 = op->vr1 > 0 ? op->vr0 : 0;
    a.v1 = op->vr1 > 0 ? op->vr1 : op->nV;
    a.p0 = a.v0 / kVoxWindow * kVoxWindow;
    a.p1 = (a.v1 + kVoxWindow - 1) / kVoxWindow * kVoxWindow;
    if (a.p1 > op->nV) a.p1 = op->nV;
    a.ec_ptr = op->ec_ptr; a.ec_col = op->ec_col; a.ec_o = op->ec_o; a.iso_ptr = op->iso_ptr; a.iso_col = op->iso_col;
    a.lutEC = op->lut_r_ec(arith); a.lutISO = op->lut_r_iso(arith);
    a.nSp = arith == CGB_ARITH_F32 ? op->nSp : op->nSp_r;
    a.nEC = op->nE > 0 ? op->nEC : 0; a.nISO = op->nISOv > 0 ? op->nISO : 0;
    a.ec_base = P.ec_base; a.iso_base = P.iso_base; a.nE = op->nE; a.nISOv = op->nISOv;
    a.seg_l = op->seg_l; a.seg_l16 = arith == CGB_ARITH_F32 ? nullptr : op->seg_l16; a.l_scale = op->len16_inv_scale;
    a.coef = m->coef; a.part = m->part; a.epart = m->epart; a.scratch = op->scratch32;
    return a;
}

int launch(const cgb_op *op, const MixPlan *m, int arith, int adjoint, const SmMixArgs &a, cudaStream_t st) {
    const int need = (a.p1 - a.p0 + kMixThreads / 8 - 1) / (kMixThreads / 8);
    int g = op->nsm / m->nc;
    if (need < g) g = need;
    g = m->nc * (g < 1 ? 1 : g);
    const size_t smem = (size_t)op->nIC * op->ndirs * m->cs * (arith == CGB_ARITH_F32 ? 4 : 2);
    if (arith == CGB_ARITH_BF16) return launch_mix_smem_bf16(adjoint, m->nq, g, smem, st, a, m->cs);
    if (arith == CGB_ARITH_F32) return launch_mix_smem_f32(adjoint, m->nq, g, smem, st, a, m->cs);
    return launch_mix_smem_fp16(adjoint, m->nq, g, smem, st, a, m->cs);
}

}  // namespace

void free_mix_plan(cgb_op *op) {
    for (MixPlan *&m : op->mixp) {
        if (!m) continue;
        drop(op, m);
        if (m->order.done) cudaEventDestroy(m->order.done);
        delete m;
        m = nullptr;
    }
}

int forward_smem_mix(cgb_op *op, const float *x, float *y, cudaStream_t st, int arith, int *ran) {
    *ran = 0;
    MixPlan *m;
    CGB_TRY(mix_plan(op, st, arith, 0, &m));
    if (!m) return CGB_OK;
    SmMixArgs a = mix_args(op, m, arith);
    a.x = x;
    a.y = y;
    a.vec_ok = op->nS % 4 == 0 && (uintptr_t)y % 16 == 0;
    CGB_TRY(order_enter(&m->order, st));
    auto coef = arith == CGB_ARITH_F32 ? k_mix_coef<true> : k_mix_coef<false>;
    coef<<<grid_of((a.nruns + 3) / 4, 8192), 256, 0, st>>>(a, op->seg_f, op->runs->eval_ones ? nullptr : op->eval, op->nF);
    CGB_CUDA(cudaGetLastError());
    CGB_TRY(launch(op, m, arith, 0, a, st));
    CGB_TRY(order_leave(&m->order, st));
    *ran = 1;
    return CGB_OK;
}

int adjoint_smem_mix(cgb_op *op, const float *y, double *x, cudaStream_t st, int arith, int *ran) {
    *ran = 0;
    MixPlan *m;
    CGB_TRY(mix_plan(op, st, arith, 1, &m));
    if (!m) return CGB_OK;
    CGB_TRY(order_enter(&m->order, st));
    auto pass = [&](cudaStream_t q) -> int {
        SmMixArgs a = mix_args(op, m, arith);
        a.z = y;
        a.xout = x;
        a.vec_ok = op->nS % 4 == 0 && (uintptr_t)y % 16 == 0;
        CGB_TRY(launch(op, m, arith, 1, a, q));
        if (m->nc == 1) return CGB_OK;
        auto join = arith == CGB_ARITH_F32 ? k_mix_join<true> : k_mix_join<false>;
        join<<<grid_of(a.nruns * (a.v1 - a.v0) / op->nV + 1, op->nsm * 32), 256, 0, q>>>(a);
        CGB_CUDA(cudaGetLastError());
        return CGB_OK;
    };
    if (op->nslab <= 1) {
        CGB_TRY(pass(st));
        CGB_TRY(fibre_sum32_from(op, op->scratch32, x, st));
    } else {
        CGB_TRY(slab_schedule(
            op, st,
            [&](int s, cudaStream_t q) {
                VoxelRange vr(op, op->slab_v[s], op->slab_v[s + 1]);
                return pass(q);
            },
            [&](int s, cudaStream_t q) { return fibre_sum32_slab(op, op->scratch32, x, s, q); }));
    }
    CGB_TRY(order_leave(&m->order, st));
    *ran = 1;
    return CGB_OK;
}

}  // namespace cgb
