// Kinship operator K = Z Z^T / M over a sample / variant selection
// (src/kinship_operator.h:53-95, src/kinship_operator.cpp:29-374).
//
// Layout: the operator reads one packed matrix `view` whose rows are the selected
// variants and whose samples are the selected samples, padded to kRowAlign bytes with the
// missing code.  With the identity selection it is the resident genotype matrix itself;
// otherwise the selection is materialised once at construction by a repack kernel, so
// every apply streams contiguous rows (a keep list becomes a gather only once, not on
// every apply as in kinship_operator.cpp:127-134).  Selected variants with 1/sd == 0
// contribute nothing and are dropped from the copy, while the 1/M scaling still counts
// them, as the reference does (kinship_operator.cpp:63-64, 96).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "cs_internal.h"
#include "slices_internal.h"

namespace cs {

// Per view row t (SNP rows[t] of the matrix, or t): mean, 1 / sd, decode values and their squares,
// and, where counts are given, its code counts.  One launch instead of four copies of tables that
// a host loop filled (88 bytes a SNP): an operator on 100k SNPs is made in 0.9 ms instead of 1.6.
__global__ void __launch_bounds__(256)
k_operator_tables(const int32_t* __restrict__ rows, int64_t R, const double* __restrict__ g_mean,
                  const double* __restrict__ g_inv_std, const int32_t* __restrict__ g_counts,
                  double* __restrict__ mean, double* __restrict__ inv_std, int32_t* __restrict__ counts,
                  double* __restrict__ lut, double* __restrict__ lut_sq) {
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (t >= R) return;
    const int64_t j = rows ? rows[t] : t;
    const double mu = g_mean[j], is = g_inv_std[j];
    mean[t] = mu;
    inv_std[t] = is;
    // kinship_operator.cpp:276-277 decode values; code 01 (missing) -> 0
    const double z[4] = {(2.0 - mu) * is, 0.0, (1.0 - mu) * is, -mu * is};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        lut[4 * t + q] = z[q];
        lut_sq[4 * t + q] = z[q] * z[q];
        if (g_counts) counts[4 * t + q] = g_counts[4 * j + q];
    }
}

cs_kinship* kinship_create(const cs_genotypes* g, const int32_t* keep, int64_t n_keep,
                           const int32_t* variants, int64_t n_var) {
    prof::HostScope hs("kinship_create");
    if (g == nullptr) fail(CS_ERR_INVALID_ARGUMENT, "PlinkKinshipOperator: null reader");
    const int64_t N = g->n_samples, M = g->n_snps;
    bool identity = true;
    if (keep && n_keep > 0) {
        for (int64_t i = 0; i < n_keep; ++i)
            if (keep[i] < 0 || keep[i] >= N)
                fail(CS_ERR_INVALID_ARGUMENT, "PlinkKinshipOperator: sample index out of range");
        identity = (n_keep == N);
        for (int64_t i = 0; identity && i < N; ++i) identity = keep[i] == i;
    } else {
        keep = nullptr;
        n_keep = 0;
    }
    if (variants && n_var > 0) {
        bool all = (n_var == M);
        for (int64_t j = 0; j < n_var; ++j) {
            if (variants[j] < 0 || variants[j] >= M)
                fail(CS_ERR_INVALID_ARGUMENT, "PlinkKinshipOperator: variant index out of range");
            all = all && variants[j] == j;
        }
        if (all) {  // every SNP in file order: the resident matrix serves as is
            variants = nullptr;
            n_var = 0;
        }
    } else {
        variants = nullptr;
        n_var = 0;
    }
    auto* op = new cs_kinship();
    try {
        op->g = g;
        op->rows = keep ? n_keep : N;
        op->num_variants = variants ? n_var : M;
        if (op->num_variants == 0) fail(CS_ERR_INVALID_ARGUMENT, "PlinkKinshipOperator: no variants selected");
        cudaStream_t s = 0;
        std::vector<int32_t> active;
        DeviceBuffer<int32_t> d_rows;  // view rows -> SNPs of g, when they differ
        op->keep_identity = identity;
        if (!variants && identity) {
            op->view = cs_packed_view{g->packed.get(), M, N, g->stride};
            op->n_active = M;
            op->mean = g->mean;
            op->inv_std = g->inv_std;
            op->view_snp.resize(M);
            for (int64_t t = 0; t < M; ++t) op->view_snp[t] = (int32_t)t;
            op->view_pos = op->view_snp;
        } else {
            active.reserve(op->num_variants);
            for (int64_t t = 0; t < op->num_variants; ++t) {
                const int32_t j = variants ? variants[t] : (int32_t)t;
                if (g->inv_std[j] != 0.0) {
                    active.push_back(j);
                    op->view_pos.push_back((int32_t)t);
                }
            }
            op->n_active = (int64_t)active.size();
            const int64_t stride = round_up((op->rows + 3) / 4, kRowAlign);
            op->own_packed.resize(std::max<int64_t>(1, op->n_active * stride));
            DeviceBuffer<int32_t> d_keep;
            d_rows.resize(std::max<int64_t>(1, op->n_active));
            if (op->n_active)
                CS_CUDA(cudaMemcpyAsync(d_rows.get(), active.data(), op->n_active * 4,
                                        cudaMemcpyHostToDevice, s));
            if (!identity) {
                d_keep.resize(n_keep);
                CS_CUDA(cudaMemcpyAsync(d_keep.get(), keep, n_keep * 4, cudaMemcpyHostToDevice, s));
            }
            repack(g->packed.get(), g->stride, d_rows.get(), op->n_active,
                   identity ? nullptr : d_keep.get(), op->rows, op->own_packed.get(), stride, s);
            CS_CUDA(cudaStreamSynchronize(s));
            op->view = cs_packed_view{op->own_packed.get(), op->n_active, op->rows, stride};
            op->mean.resize(op->n_active);
            op->inv_std.resize(op->n_active);
            for (int64_t t = 0; t < op->n_active; ++t) {
                op->mean[t] = g->mean[active[t]];
                op->inv_std[t] = g->inv_std[active[t]];
            }
            op->view_snp = active;
        }
        const int64_t R = op->n_active;
        if (identity && (int64_t)g->code_counts.size() != 4 * g->n_snps)
            fail(CS_ERR_INVALID_ARGUMENT, "PlinkKinshipOperator: genotype statistics missing");
        // code counts over the operator's samples (trace, mixed-form corrections)
        op->counts.assign(4 * R, 0);
        if (identity) {
            // every sample: the counts the statistics pass kept
            for (int64_t t = 0; t < R; ++t)
                std::copy_n(&g->code_counts[4 * (int64_t)op->view_snp[t]], 4, &op->counts[4 * t]);
        } else if (R) {
            op->d_counts.resize(std::max<int64_t>(1, 4 * R));
            row_code_counts(op->view, op->d_counts.get(), s);
            CS_CUDA(cudaMemcpyAsync(op->counts.data(), op->d_counts.get(), 16 * R,
                                    cudaMemcpyDeviceToHost, s));
        }
        double total = 0.0;
        CS_CUDA(cudaStreamSynchronize(s));
        for (int64_t t = 0; t < R; ++t) {
            // trace(): sum over observed calls of z^2 (kinship_operator.cpp:306-344), of the decode
            // values of kinship_operator.cpp:276-277
            const double mu = op->mean[t], is = op->inv_std[t];
            const double z2 = (2.0 - mu) * is, z1 = (1.0 - mu) * is, z0 = -mu * is;
            total += op->counts[4 * t + 0] * (z2 * z2) + op->counts[4 * t + 2] * (z1 * z1) +
                     op->counts[4 * t + 3] * (z0 * z0);
        }
        op->trace = total / (double)op->num_variants;
        op->d_view_pos.resize(std::max<int64_t>(1, R));
        if (R)
            CS_CUDA(cudaMemcpy(op->d_view_pos.get(), op->view_pos.data(), 4 * R,
                               cudaMemcpyHostToDevice));
        op->d_lut.resize(std::max<int64_t>(1, 4 * R));
        op->d_lut_sq.resize(std::max<int64_t>(1, 4 * R));
        op->d_mean.resize(std::max<int64_t>(1, R));
        op->d_inv_std.resize(std::max<int64_t>(1, R));
        if (identity) op->d_counts.resize(std::max<int64_t>(1, 4 * R));
        if (R) {
            prof::Scope ps("operator_tables", s, 0.0, 112.0 * R);
            k_operator_tables<<<(unsigned)((R + 255) / 256), 256, 0, s>>>(
                d_rows.get(), R, g->d_mean.get(), g->d_inv_std.get(), identity ? g->d_code_counts.get() : nullptr,
                op->d_mean.get(), op->d_inv_std.get(), op->d_counts.get(), op->d_lut.get(), op->d_lut_sq.get());
            CS_LAUNCH("operator_tables");
            CS_CUDA(cudaStreamSynchronize(s));
        }
    } catch (...) {
        delete op;
        throw;
    }
    return op;
}

// FP64 form on the FP64 pipe: U = Z^T X (pass over rows), Y = Z U / M (pass over samples).
static void kinship_apply_pipe(cs_kinship* op, const double* X, int64_t ldx, int64_t k, double* Y,
                               int64_t ldy, cudaStream_t s) {
    const int64_t R = op->n_active;
    const double scale = 1.0 / (double)op->num_variants;
    if (R == 0) {
        // every selected variant is monomorphic: K = 0
        CS_CUDA(cudaMemset2DAsync(Y, ldy * 8, 0, k * 8, op->rows, s));
        return;
    }
    op->buf_u.resize(R * k);
    decode_gemm_rows_fp64(op->view, op->d_lut.get(), X, ldx, k, op->buf_u.get(), k, op->ws, s);
    decode_gemm_samples_fp64(op->view, op->d_lut.get(), op->buf_u.get(), k, k, Y, ldy, scale,
                             op->ws, s);
}

void kinship_apply_rowmajor(cs_kinship* op, const double* X, int64_t ldx, int64_t k, double* Y,
                            int64_t ldy, int precision, cudaStream_t s) {
    if (k <= 0) return;
    if (precision == CS_PRECISION_MIXED)
        kinship_apply_mixed(op, StridedIn{X, ldx, 1}, k, StridedOut{Y, ldy, 1}, s);
    else if (precision != CS_PRECISION_FP64)
        fail(CS_ERR_INVALID_ARGUMENT, "unknown precision mode");
    else if (!kinship_apply_slices(op, StridedIn{X, ldx, 1}, k, StridedOut{Y, ldy, 1}, s))
        kinship_apply_pipe(op, X, ldx, k, Y, ldy, s);
}

// FP32 column-major (ld) <-> FP64 row-major (n x k) around the FP32 entry point.
__global__ void k_f32col_to_f64row(const float* __restrict__ src, int64_t ld, int64_t n,
                                   int64_t k, double* __restrict__ dst) {
    const int64_t total = n * k;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = idx / k, c = idx - i * k;
        dst[idx] = (double)src[i + c * ld];
    }
}

__global__ void k_f64row_to_f32col(const double* __restrict__ src, int64_t n, int64_t k,
                                   float* __restrict__ dst, int64_t ld) {
    const int64_t total = n * k;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = idx / n, i = idx - c * n;
        dst[i + c * ld] = (float)src[i * k + c];
    }
}

// Whether two column-major blocks (ld, rows x k) share memory.
template <class T>
static bool overlap(const T* a, int64_t lda, int64_t rows_a, const T* b, int64_t ldb, int64_t rows_b,
                    int64_t k) {
    return a < b + (k - 1) * ldb + rows_b && b < a + (k - 1) * lda + rows_a;
}

// FP32 apply (device pointers): the inputs widened to FP64, the FP64 or mixed apply, the
// result rounded to FP32.  Y may alias X.
void kinship_apply_f32(cs_kinship* op, const float* X, int64_t ldx, int64_t k, float* Y,
                       int64_t ldy, int precision, cudaStream_t s) {
    if (k < 0) fail(CS_ERR_INVALID_ARGUMENT, "negative column count");
    if (k == 0) return;
    if (ldx < op->rows || ldy < op->rows)
        fail(CS_ERR_INVALID_ARGUMENT, "PlinkKinshipOperator::apply: dimension mismatch");
    const int64_t n = op->rows;
    // the tensor-core form reads and writes float columns itself
    if (precision == CS_PRECISION_MIXED &&
        ((X == Y && ldx == ldy) || !overlap(X, ldx, n, Y, ldy, n, k))) {
        kinship_apply_mixed(op, Strided<const float>{X, 1, ldx}, k, Strided<float>{Y, 1, ldy}, s);
        return;
    }
    op->buf_x.resize(n * k);
    op->buf_y.resize(n * k);
    const unsigned blocks = (unsigned)std::max<int64_t>(1, std::min<int64_t>((n * k + 255) / 256, 32LL * num_sms()));
    {
        prof::Scope ps("f32_to_f64", s, 0.0, 12.0 * n * k);
        k_f32col_to_f64row<<<blocks, 256, 0, s>>>(X, ldx, n, k, op->buf_x.get());
        CS_LAUNCH("f32_to_f64");
    }
    kinship_apply_rowmajor(op, op->buf_x.get(), k, k, op->buf_y.get(), k, precision, s);
    {
        prof::Scope ps("f64_to_f32", s, 0.0, 12.0 * n * k);
        k_f64row_to_f32col<<<blocks, 256, 0, s>>>(op->buf_y.get(), n, k, Y, ldy);
        CS_LAUNCH("f64_to_f32");
    }
}

// A column-major input as the kernels read it: as it is, or, where the output overlaps it (other
// than in its place, with `in_place`), from a copy.
static StridedIn apart(cs_kinship* op, const double* X, int64_t ldx, int64_t rows_x, const double* Y,
                       int64_t ldy, int64_t rows_y, int64_t k, bool in_place, cudaStream_t s) {
    if ((in_place && X == Y && ldx == ldy) || !overlap(X, ldx, rows_x, Y, ldy, rows_y, k))
        return StridedIn{X, 1, ldx};
    op->buf_x.resize(rows_x * k);
    colmajor_to_rowmajor(X, ldx, rows_x, k, op->buf_x.get(), k, s);
    return StridedIn{op->buf_x.get(), k, 1};
}

// Public column-major apply (device pointers).  The tensor-core kernels read and write column-major
// blocks themselves; the FP64-pipe kernels work between transposes.
void kinship_apply_colmajor(cs_kinship* op, const double* X, int64_t ldx, int64_t k, double* Y,
                            int64_t ldy, int precision, cudaStream_t s) {
    if (k < 0) fail(CS_ERR_INVALID_ARGUMENT, "negative column count");
    if (k == 0) return;
    if (ldx < op->rows || ldy < op->rows)
        fail(CS_ERR_INVALID_ARGUMENT, "PlinkKinshipOperator::apply: dimension mismatch");
    const int64_t n = op->rows;
    if (precision != CS_PRECISION_MIXED && precision != CS_PRECISION_FP64)
        fail(CS_ERR_INVALID_ARGUMENT, "unknown precision mode");
    const StridedIn x = apart(op, X, ldx, n, Y, ldy, n, k, true, s);
    if (precision == CS_PRECISION_MIXED) {
        kinship_apply_mixed(op, x, k, StridedOut{Y, 1, ldy}, s);
        return;
    }
    if (kinship_apply_slices(op, x, k, StridedOut{Y, 1, ldy}, s)) return;
    op->buf_x.resize(n * k);
    op->buf_y.resize(n * k);
    colmajor_to_rowmajor(X, ldx, n, k, op->buf_x.get(), k, s);
    kinship_apply_pipe(op, op->buf_x.get(), k, k, op->buf_y.get(), k, s);
    rowmajor_to_colmajor(op->buf_y.get(), k, n, k, Y, ldy, s);
}

// ---------------------------------------------------------------- GenotypeMatrix half-passes
// PlinkReader::multiply_Zt_v / multiply_Z_v (libCosmicCore/src/plink_reader.cpp:241-438, the
// GenotypeMatrix interface of libCosmicCore/src/matrix_adapter.h:40-53) over the operator's
// selection: Z is rows() x numVariants(), standardised with the all-sample statistics, missing
// calls 0, variants with 1/sd == 0 all zero; no 1/M scaling.

// out[pos[t] * ldo + c] = in[t * ldi + c] (view row t -> its selection position), c < k.
__global__ void k_scatter_rows(const double* __restrict__ in, int64_t ldi, int64_t R, int64_t k,
                               const int32_t* __restrict__ pos, double* __restrict__ out,
                               int64_t ldo) {
    const int64_t total = R * k;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = idx / k, c = idx - t * k;
        out[(int64_t)pos[t] * ldo + c] = in[t * ldi + c];
    }
}

// W[t * k + c] = V[pos[t] * ldv + c].
__global__ void k_gather_rows(const double* __restrict__ V, int64_t ldv, int64_t R, int64_t k,
                              const int32_t* __restrict__ pos, double* __restrict__ W) {
    const int64_t total = R * k;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = idx / k, c = idx - t * k;
        W[idx] = V[(int64_t)pos[t] * ldv + c];
    }
}

static unsigned grid_for(int64_t work) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((work + 255) / 256, 32LL * num_sms()));
}

// Column-major public forms (device pointers), on the tensor cores or, where those kernels are not
// available, the FP64 pipe between transposes.
static void require_precision(int precision) {
    if (precision != CS_PRECISION_MIXED && precision != CS_PRECISION_FP64)
        fail(CS_ERR_INVALID_ARGUMENT, "unknown precision mode");
}

// U (numVariants x k) = Z^T X.
void genotype_multiply_zt(cs_kinship* op, const double* X, int64_t ldx, int64_t k, double* U,
                          int64_t ldu, int precision, cudaStream_t s) {
    if (k < 0) fail(CS_ERR_INVALID_ARGUMENT, "negative column count");
    if (ldx < op->rows || ldu < op->num_variants)
        fail(CS_ERR_INVALID_ARGUMENT, "Dimension mismatch in multiply_Zt_v");
    if (k == 0) return;
    const int64_t n = op->rows, nv = op->num_variants, R = op->n_active;
    // rows of variants the view dropped (1/sd == 0) are zero
    auto clear = [&] { CS_CUDA(cudaMemset2DAsync(U, ldu * 8, 0, nv * 8, k, s)); };
    if (R == 0) {
        clear();
        return;
    }
    require_precision(precision);
    const StridedIn x = apart(op, X, ldx, n, U, ldu, nv, k, false, s);
    if (R < nv) clear();
    if (precision == CS_PRECISION_MIXED) {
        mixed_multiply_zt(op, x, k, StridedOut{U, 1, ldu}, s);
        return;
    }
    if (multiply_zt_slices(op, x, k, StridedOut{U, 1, ldu}, s)) return;
    if (x.p == X) {
        op->buf_x.resize(n * k);
        colmajor_to_rowmajor(X, ldx, n, k, op->buf_x.get(), k, s);
    }
    op->buf_u.resize(R * k);
    op->buf_y.resize(nv * k);
    decode_gemm_rows_fp64(op->view, op->d_lut.get(), op->buf_x.get(), k, k, op->buf_u.get(), k, op->ws, s);
    CS_CUDA(cudaMemsetAsync(op->buf_y.get(), 0, 8 * nv * k, s));
    {
        prof::Scope ps("scatter_rows", s, 0.0, 16.0 * R * k);
        k_scatter_rows<<<grid_for(R * k), 256, 0, s>>>(op->buf_u.get(), k, R, k, op->d_view_pos.get(),
                                                       op->buf_y.get(), k);
        CS_LAUNCH("scatter_rows");
    }
    rowmajor_to_colmajor(op->buf_y.get(), k, nv, k, U, ldu, s);
}

// Y (rows x k) = Z V.
void genotype_multiply_z(cs_kinship* op, const double* V, int64_t ldv, int64_t k, double* Y,
                         int64_t ldy, int precision, cudaStream_t s) {
    if (k < 0) fail(CS_ERR_INVALID_ARGUMENT, "negative column count");
    if (ldv < op->num_variants || ldy < op->rows)
        fail(CS_ERR_INVALID_ARGUMENT, "Dimension mismatch in multiply_Z_v");
    if (k == 0) return;
    const int64_t n = op->rows, nv = op->num_variants, R = op->n_active;
    if (R == 0) {
        CS_CUDA(cudaMemset2DAsync(Y, ldy * 8, 0, n * 8, k, s));
        return;
    }
    require_precision(precision);
    const StridedIn v = apart(op, V, ldv, nv, Y, ldy, n, k, false, s);
    if (precision == CS_PRECISION_MIXED) {
        mixed_multiply_z(op, v, k, StridedOut{Y, 1, ldy}, s);
        return;
    }
    if (multiply_z_slices(op, v, k, StridedOut{Y, 1, ldy}, s)) return;
    if (v.p == V) {
        op->buf_x.resize(nv * k);
        colmajor_to_rowmajor(V, ldv, nv, k, op->buf_x.get(), k, s);
    }
    op->buf_u.resize(R * k);
    op->buf_y.resize(n * k);
    {
        prof::Scope ps("gather_rows", s, 0.0, 16.0 * R * k);
        k_gather_rows<<<grid_for(R * k), 256, 0, s>>>(op->buf_x.get(), k, R, k, op->d_view_pos.get(),
                                                      op->buf_u.get());
        CS_LAUNCH("gather_rows");
    }
    decode_gemm_samples_fp64(op->view, op->d_lut.get(), op->buf_u.get(), k, k, op->buf_y.get(), k, 1.0,
                             op->ws, s);
    rowmajor_to_colmajor(op->buf_y.get(), k, n, k, Y, ldy, s);
}

// Diagonal of K before the scaling: sums over the view's rows of the squared decode values.  A thread
// sums one word (16 samples) of a chunk of rows, two rows at a time: the 16 sums that a pair of
// codes can give are tabulated per pair of rows in shared memory (32 banks: any mix of codes reads
// without conflicts), which halves the additions and look-ups, the bound here (half a look-up and
// addition a genotype; the packed bytes are a fifth of the time).  18,010 samples x 27,006 rows
// 124 us; the FP64 decode-GEMV with a vector of ones took 435.
constexpr int kDiagPairs = 32, kDiagThreads = 128;
__global__ void __launch_bounds__(kDiagThreads)
k_diagonal(const uint8_t* __restrict__ rows, int64_t R, int64_t stride, const double* __restrict__ lut_sq,
           int64_t chunk, double* __restrict__ part) {
    __shared__ double tab[kDiagPairs][16];
    const int64_t words = stride / 4, w = (int64_t)blockIdx.x * kDiagThreads + threadIdx.x;
    const int64_t t0 = blockIdx.y * chunk, t1 = min(R, t0 + chunk);
    double acc[16] = {};
    for (int64_t r0 = t0; r0 < t1; r0 += 2 * kDiagPairs) {
        __syncthreads();
        for (int e = threadIdx.x; e < kDiagPairs * 16; e += kDiagThreads) {
            const int64_t t = r0 + 2 * (e >> 4);
            tab[e >> 4][e & 15] = (t < t1 ? lut_sq[4 * t + (e & 3)] : 0.0) +
                                  (t + 1 < t1 ? lut_sq[4 * t + 4 + (e >> 2 & 3)] : 0.0);
        }
        __syncthreads();
        if (w >= words) continue;
        const uint32_t* p = reinterpret_cast<const uint32_t*>(rows + r0 * stride) + w;
#pragma unroll 4
        for (int q = 0; q < kDiagPairs; ++q, p += 2 * words) {
            const int64_t t = r0 + 2 * q;
            const uint32_t a = t < t1 ? __ldg(p) : 0u, b = t + 1 < t1 ? __ldg(p + words) : 0u;
            const uint32_t even = (a & 0x33333333u) | ((b & 0x33333333u) << 2);
            const uint32_t odd = ((a >> 2) & 0x33333333u) | (b & 0xCCCCCCCCu);
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                acc[2 * j] += tab[q][(even >> (4 * j)) & 15u];
                acc[2 * j + 1] += tab[q][(odd >> (4 * j)) & 15u];
            }
        }
    }
    if (w >= words) return;
#pragma unroll
    for (int j = 0; j < 16; ++j) part[((int64_t)blockIdx.y * 16 + j) * words + w] = acc[j];
}

__global__ void __launch_bounds__(256)
k_diagonal_sum(const double* __restrict__ part, int64_t words, int splits, int64_t n, double scale,
               double* __restrict__ diag) {
    const int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (e >= 16 * words) return;
    const int64_t i = e % words * 16 + e / words;
    if (i >= n) return;
    double sm = 0.0;
#pragma unroll 8
    for (int z = 0; z < splits; ++z) sm += part[(int64_t)z * 16 * words + e];
    diag[i] = sm * scale;
}

void kinship_diagonal(cs_kinship* op, double* diag_host) {
    const int64_t n = op->rows, R = op->n_active;
    if (R == 0) {
        std::fill(diag_host, diag_host + n, 0.0);
        return;
    }
    cudaStream_t s = 0;
    // chunks of rows for about six blocks an SM
    const int64_t words = op->view.stride / 4, across = (words + kDiagThreads - 1) / kDiagThreads;
    const int64_t want = std::max<int64_t>(1, (6LL * num_sms() + across - 1) / across);
    const int64_t chunk = round_up((R + want - 1) / want, 2 * kDiagPairs);
    const int splits = (int)((R + chunk - 1) / chunk);
    DeviceBuffer<double> part, d;
    part.resize(splits * 16 * words);
    d.resize(n);
    {
        prof::Scope ps("kinship_diagonal", s, (double)n * (double)R, (double)R * (double)op->view.stride);
        k_diagonal<<<dim3((unsigned)across, (unsigned)splits), kDiagThreads, 0, s>>>(
            op->view.rows, R, op->view.stride, op->d_lut_sq.get(), chunk, part.get());
        k_diagonal_sum<<<(unsigned)((16 * words + 255) / 256), 256, 0, s>>>(
            part.get(), words, splits, n, 1.0 / (double)op->num_variants, d.get());
        CS_LAUNCH("kinship_diagonal");
    }
    CS_CUDA(cudaMemcpy(diag_host, d.get(), 8 * n, cudaMemcpyDeviceToHost));
}

}  // namespace cs
