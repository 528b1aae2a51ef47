// Float-float A*x and A'*y with the IC response table resident in shared memory.
//
// The pair kernels of operator_pair.cuh gather a table row per (voxel, orientation) run from
// L1 / L2: 0.6 MB of FP32 rows at 500 orientations and 288 samples do not fit one SM's L1, so
// at 1M streamlines the gathers (115 GB per product) bound them together with the 11 FP32
// operations per term.  Here a block keeps a part of the table in shared memory for the
// whole launch and walks every voxel:
//   A   the block holds a chunk of the samples for every orientation and computes these
//       samples of every row (no partial results leave the block);
//   A'  the block holds a chunk of the samples for a range of orientations (all of them when
//       they fit) and computes these samples' part of the runs' dot products; a streaming pass
//       adds the parts up.
// The runs (segments of a voxel with one orientation) are laid out once per handle
// (FfPlan); A first forms each run's coefficient sum(l * x * eval) in one pass.
//
// Arithmetic.  A term is added to a float-float accumulator (s, e) as
//   s' = fma(c.h, L, s);  d = s - s';  r = fma(c.h, L, d);  r = fma(c.l, L, r);  e += r
// five FP32 operations instead of eleven: d is exact and r is the term's rounding error
// whenever |c.h * L| <= |s| and s does not cancel.  Both hold when every term has the
// sign of s and s starts at a bound of the terms (the bias), which is removed afterwards:
//   A   x >= 0 and table >= 0 (checked per voxel / per handle): the first 8 runs are added
//       with the general two-sum, the bias tops s up to max(c) * max(column) where it is
//       below, and s, e are renormalised every 8 terms;
//   A'  row and table >= 0: the bias is the power of two just below the lane's largest term bound,
//       so that the sums neither cancel nor let the bias take their last bits.
// Voxels with a negative or non-finite coefficient and rows with a negative entry use the general
// two-sum throughout.
// The error is relative to sum + bias, and the bias follows the largest table value of each sample,
// whether the voxel has that row or not.  So it may be at most kBiasA times a voxel's own sum (A: a
// rule on the table, FfPlan::uneven, since the sum is at least the largest coefficient times the
// smallest row) and kBiasAdj times a dot product (A': the same rule, and every dot product is looked
// at), else the general sums are taken.  120 runs a voxel and an unused row 10^6 times as large: A was
// off by 2e-9 of a voxel's norm with the bias.  Rows that are rotations of one response have column
// maxima of 1.6 (b = 1000) to 3.8 (b = 10000 s/mm^2) times a row and biases up to 1.5 times a dot
// product for measured signals.  Cost, us a pair: 288 samples, 122 M segments 20580 / 20580,
// 15 M 4870 / 4850, three responses x 99 samples 901 / 908.
#pragma once
#include "operator_pair.cuh"

namespace cgb {

// Runs (segments of a voxel with one orientation) of a handle, built on its first large product
struct RunLayout {
    int64_t nruns;
    uint32_t *run_ptr;           // [nV+1] runs of voxel v
    uint16_t *run_o;             // [nruns] orientation
    uint32_t *run_seg;           // [nruns+1] first segment
    uint32_t *vperm;             // [nV] voxels, by falling run count within windows of kVoxWindow
    int eval_ones;               // eval is 1 everywhere
    size_t bytes;                // of the handle's, held here
};

// Products on different streams take turns with buffers of the handle: each waits for the last one's
// end, unless that ran on the same stream.  Streams are told apart by their id: the handle of a
// destroyed stream is given to new ones, and cudaStreamPerThread is one handle for many streams.
struct StreamOrder {
    cudaEvent_t done;            // the last product has finished
    unsigned long long last;     // ... its stream
    int used;
};
inline int order_create(StreamOrder *o) {
    CGB_CUDA(cudaEventCreateWithFlags(&o->done, cudaEventDisableTiming));
    return CGB_OK;
}
inline int order_enter(const StreamOrder *o, cudaStream_t st) {
    unsigned long long id = 0;
    CGB_CUDA(cudaStreamGetId(st, &id));
    if (o->used && o->last != id) CGB_CUDA(cudaStreamWaitEvent(st, o->done, 0));
    return CGB_OK;
}
inline int order_leave(StreamOrder *o, cudaStream_t st) {
    CGB_CUDA(cudaEventRecord(o->done, st));
    CGB_CUDA(cudaStreamGetId(st, &o->last));
    o->used = 1;
    return CGB_OK;
}

// Table images and buffers of the shared-memory float-float products
struct FfPlan {
    int fwd_ok, adj_ok;          // kernels usable for this handle's shape and table
    float2 *coef;                // [nIC * nruns] run coefficients (high, low word) of the current A
    // A: samples in fnc chunks of 16 * fnp, row stride fcs floats
    int fnp, fnc, fcs;
    float *fimg;                 // [fnc][nIC * ndirs][fcs]
    float *colmax;               // [kColPad] largest table value per sample, zero beyond nS; then
                                 // the smallest row sum of every eight rows
    int uneven;                  // sum(colmax) > kBiasA * the smallest row sum: no biased sums
    // A': samples in anc chunks of 16 * anp, orientations in anb ranges of ano, row stride acs
    int anp, anc, anb, ano, acs;
    float *aimg;                 // [anc][anb][nIC * ano][acs]
    uint32_t *run_blk;           // [anb + 1][nV] first run of the voxel in a range
    double *part;                // [nIC * nruns][anc] parts of the runs' dot products
    double *epart;               // [EC and ISO columns][anc] (anc > 1)
    double *zrow;                // [nrows] weighted residual (FISTA gradient)
    StreamOrder order;           // of the products that use coef
    int no_room;                 // the buffers did not fit: not tried again
    size_t bytes;                // of the handle's, held here
};

constexpr int kVoxWindow = 4096;
constexpr int kColPad = kMaxSamples + 128;
constexpr float kBiasA = 4.f, kBiasAdj = 8.f;  // largest bias against the sums it joins (file comment)
// threads of the one block per SM: 80 registers a thread, and 96 where A' needs them (measured at 5
// and 6 pairs per lane: 45 and 1900 us with 640 threads, 49 and 1940 with 768; at 4: 616 and 571)
constexpr int kFwdThreads = 768;
constexpr int adj_threads(int np) { return np <= 4 ? 768 : 640; }
// Where the shared-memory kernels take over from the pair kernels of operator_pair.cuh: a
// product of at least kSmemMinWork terms (segments x responses x samples) with at least
// smem_min_items() segments x responses per voxel: 4 for every chunk the sample count asks for,
// 8 for every further part that the table's size adds.  Measured, us, here / pair kernels:
//   terms      A 36 / 28 and A' 35 / 32 at 8 M, 39 / 41 and 40 / 46 at 12 M, 45 / 58 and 46 / 65 at 26 M;
//   per voxel  66 samples A 48 / 52, A' 48 / 59 at 5; 145 samples (2 chunks) 191 / 230, 209 / 275 at
//              8; 288 samples (3 chunks) 1096 / 1241, 1030 / 1556 at 13 and 1575 / 2251, 1534 / 2515 at 33;
//              2 responses x 66 samples (A 3 chunks for 1, A' 2 ranges) 345 / 319, 371 / 370 at 10.
// Below the lines the table fill (160-190 KB per SM) and the per-voxel steps, repeated for
// every part, cost more than the gathers from L2.
constexpr double kSmemMinWork = 1e7;
inline double smem_min_items(int nS, int parts) {
    const int chunks = (nS + 95) / 96;
    return 4.0 * chunks + 8.0 * (parts - chunks);
}

// device buffers that the handle keeps, counted in its bytes and in `held`
template <class T>
int keep_buffer(cgb_op *op, size_t *held, T **p, size_t count) {
    const size_t b = (count ? count : 1) * sizeof(T);
    CGB_CUDA(cudaMalloc((void **)p, b));
    op->bytes += b;
    *held += b;
    return CGB_OK;
}

namespace detail {

// a += b (exact two-sum into the error word)
__device__ __forceinline__ void dd2_addf(DD2 &a, f2 b) {
    const f2 s = f2_add(a.s, b);
    const f2 bb = f2_sub(s, a.s);
    const f2 err = f2_add(f2_sub(a.s, f2_sub(s, bb)), f2_sub(b, bb));
    a.e = f2_add(a.e, err);
    a.s = s;
}

// a += (h + l) * L for any terms: the two-sum of dd2_fma on the rounded product, whose last
// difference takes the product itself, so its rounding error comes along (9 operations).
// `zero` is 0 from a kernel argument: ptxas fuses a packed mul.rn whose only use is an add.rn
// (measured, also with -fmad=false), which would leave the product unrounded.
__device__ __forceinline__ void dd2_fma_any(DD2 &a, f2 h, f2 l, f2 L, f2 zero) {
    const f2 s = f2_add(a.s, f2_fma(h, L, zero));
    const f2 nb = f2_sub(a.s, s);
    f2 r = f2_fma(h, L, nb);
    r = f2_fma(l, L, r);
    const f2 q = f2_sub(a.s, f2_add(s, nb));
    a.e = f2_add(a.e, f2_add(r, q));
    a.s = s;
}

// a += (h + l) * L for terms that neither exceed nor cancel a.s (file comment)
__device__ __forceinline__ void dd2_fma_same(DD2 &a, f2 h, f2 l, f2 L) {
    const f2 s = f2_fma(h, L, a.s);
    const f2 d = f2_sub(a.s, s);
    f2 r = f2_fma(h, L, d);
    r = f2_fma(l, L, r);
    a.e = f2_add(a.e, r);
    a.s = s;
}

__device__ __forceinline__ f2 f2_neg(f2 a) { return a ^ 0x8000000080000000ull; }

// copies n floats (a multiple of 4, 16-byte aligned) to shared memory with all threads
template <int THREADS>
__device__ __forceinline__ void fill_table(float *dst, const float *__restrict__ src, int n) {
    const unsigned d0 = (unsigned)__cvta_generic_to_shared(dst);
    for (int i = threadIdx.x * 4; i < n; i += THREADS * 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d0 + 4u * i), "l"(src + i));
    asm volatile("cp.async.commit_group;");
}
__device__ __forceinline__ void fill_wait() {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

struct SmFwdArgs {
    const uint32_t *vperm, *run_ptr;
    const uint16_t *run_o;
    const float2 *coef;
    int64_t nruns;
    const float *img, *colmax;
    float coef_max;                           // largest coefficient of the fast sums (uneven table: none)
    int nIC, ndirs, nS, nc, p0, p1, v0, v1;   // perm positions [p0, p1), voxels [v0, v1)
    const uint32_t *ec_ptr, *ec_col, *iso_ptr, *iso_col;
    const uint16_t *ec_o;
    const float *lutEC, *lutISO;              // padded rows of stride nSp
    int nSp, nEC, nISO;
    int64_t ec_base, iso_base, nE, nISOv;
    const double *x;
    const unsigned long long *xmax;
    int lut_exp;
    double *yout, *axout;
    const double *yobs, *sqw;
    double *partials;
    int vec_ok;
    f2 zero;                                  // 0 (dd2_fma_any)
};

struct SmAdjArgs {
    const uint32_t *vperm, *run_blk, *run_seg;
    const uint16_t *run_o;
    const float *seg_l;
    int64_t n, nruns;
    const float *img, *colmax;
    unsigned general;                         // sign bit: general sums for every row (uneven table)
    int nIC, nS, nV, nc, nb, no, p0, p1, v0, v1;
    const uint32_t *ec_ptr, *ec_col, *iso_ptr, *iso_col;
    const uint16_t *ec_o;
    const float *lutEC, *lutISO;
    int nSp, ndirs, nEC, nISO;
    int64_t ec_base, iso_base, nE, nISOv;
    const double *z;
    int lut_exp, vec_ok;
    double *scratch, *xout;
    double *part, *epart;
    f2 zero;                                  // 0 (dd2_fma_any)
};

}  // namespace detail
}  // namespace cgb
