// Multi-right-hand-side preconditioned CG on the mixed-model covariance
// V = vg * Zr K Zr^T + vpe * Zr Zr^T + ve * I, and the record <-> genotype-row maps around
// the kinship operator.
//
// The reference solves one right-hand side at a time (libCosmicCore/src/matrix_free_pcg.h:
// 20-68, driven by libCosmicCore/src/stcg_vce.cpp:117-126), so every CG iteration streams
// the whole packed genotype matrix for one vector.  Here all right-hand sides that share a
// V advance together: one kinship apply per iteration carries every active column (the
// tensor-core operator needs width to be efficient), each column keeps its own alpha/beta
// recurrence, and columns whose residual meets the tolerance are compacted out of the
// block so later applies only carry live columns.  Reductions use a fixed row chunking, so
// a column's arithmetic does not depend on which other columns share the block.
#include <algorithm>
#include <cmath>
#include <utility>

#include "chain.cuh"
#include "vce_internal.h"

namespace cs {

// out = vg * fac * KU[row(r)] + vpe * U[row(r)] + ve * V[r]   (stcg_vce.cpp:103-115)
struct Covariance {
    const double *V, *KU, *U;
    int64_t ldv, ldk, ldu;
    const int32_t* rec_to_row;
    double vg, fac, vpe, ve;
    int with_pe;
    struct In {
        double g, pe, v;
    };
    __device__ In load(int64_t r, int64_t c) const {
        const int64_t i = rec_to_row ? rec_to_row[r] : r;
        return {i >= 0 ? KU[i * ldk + c] : 0.0, i >= 0 && with_pe ? U[i * ldu + c] : 0.0, V[r * ldv + c]};
    }
    __device__ double value(const In& in) const {
        double g = in.g;
        if (fac != 1.0) g *= fac;
        double o = vg * g;
        if (with_pe) o += vpe * in.pe;
        return o + ve * in.v;
    }
};

namespace {

// ---------------------------------------------------------------- column sums
// Sums over the rows of n x k blocks, NV per column, in an order that depends on n alone: chunks of
// `chunk` rows, eight interleaved lanes in each, lanes added in order, then the chunks by 32 lanes'
// strided sums and a tree (more than two sums a column: the chunks in order).  A block covers kc
// columns (a power of two up to 32) x 32 / kc chunks; the last block of a column tile finishes its
// columns, so that what follows from the sums (a step length, a coefficient) needs no kernel of its
// own.  What bounds it is the chain of dependent loads: a lane reads its rows' operands together
// before it uses them, and the last block reads the partials in the order of memory, several at
// once.  CG's update (n=20000, 34 columns) takes 23 us, 31 with one row at a time and a warp to a
// column; n=2000 9.3 us against 12.5.
constexpr int kChunkRows = 16, kMaxChunks = 512;
int64_t chunk_rows(int64_t n) {
    return kChunkRows * std::max<int64_t>(1, (n + (int64_t)kChunkRows * kMaxChunks - 1) /
                                                 ((int64_t)kChunkRows * kMaxChunks));
}
int64_t chunk_count(int64_t n) { return std::max<int64_t>(1, (n + chunk_rows(n) - 1) / chunk_rows(n)); }

// Elem: In load(r, c) reads what element (r, c) needs, use(in, r, c, v) adds it to the sums (and may
// write the element); Batch rows are loaded at once.
template <int NV, int Batch, class Elem, class Finish>
__global__ void __launch_bounds__(256)
k_column_reduce(int64_t n, int64_t k, int64_t chunk, int64_t nb, int kc, double* __restrict__ part,
                unsigned* __restrict__ counter, const Elem elem, const Finish finish) {
    chain_enter();
    constexpr int kScratch = NV <= 2 ? NV * 32 * 33 : NV * 256;
    __shared__ double sh[kScratch];  // lanes' sums [NV][256], then the finish
    __shared__ int last;
    const int chunks = 32 / kc;
    const int tc = threadIdx.x % kc, tl = threadIdx.x / kc;
    const int lane = tl & 7, ch = tl >> 3;
    const int64_t c0 = (int64_t)blockIdx.y * kc, c = c0 + tc;
    const int64_t b = (int64_t)blockIdx.x * chunks + ch;
    double v[NV] = {};
    if (c < k && b < nb) {
        const int64_t r1 = min(n, (b + 1) * chunk);
        for (int64_t r = b * chunk + lane; r < r1; r += 8 * Batch) {
            typename Elem::In in[Batch];
#pragma unroll
            for (int q = 0; q < Batch; ++q)
                if (r + 8 * q < r1) in[q] = elem.load(r + 8 * q, c);
#pragma unroll
            for (int q = 0; q < Batch; ++q)
                if (r + 8 * q < r1) elem.use(in[q], r + 8 * q, c, v);
        }
    }
    const int slot = (tc * chunks + ch) * 8 + lane;
#pragma unroll
    for (int q = 0; q < NV; ++q) sh[q * 256 + slot] = v[q];
    __syncthreads();
    // one thread per (column, chunk)
    const int oc = threadIdx.x & 31;
    const int64_t pc = c0 + oc / chunks, ob = (int64_t)blockIdx.x * chunks + oc % chunks;
    for (int q = threadIdx.x >> 5; q < NV; q += 8)
        if (pc < k && ob < nb) {
            double t = sh[q * 256 + oc * 8];
            for (int j = 1; j < 8; ++j) t += sh[q * 256 + oc * 8 + j];
            part[((int64_t)q * nb + ob) * k + pc] = t;
        }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(counter + blockIdx.y, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    if constexpr (NV <= 2) {
        const int slots = min(32, 256 / kc);
        if (tl < slots && c < k)
#pragma unroll
            for (int q = 0; q < NV; ++q)
                for (int l = tl; l < 32; l += slots) {
                    double t = 0.0;
#pragma unroll 8
                    for (int64_t i = l; i < nb; i += 32) t += __ldcg(part + ((int64_t)q * nb + i) * k + c);
                    sh[(q * 32 + l) * 33 + tc] = t;
                }
        __syncthreads();
        const int wl = threadIdx.x & 31;
        for (int j = threadIdx.x >> 5; j < kc && c0 + j < k; j += 8) {
            double tot[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                tot[q] = sh[(q * 32 + wl) * 33 + j];
                for (int off = 16; off; off >>= 1) tot[q] += __shfl_xor_sync(0xffffffffu, tot[q], off);
            }
            if (wl == 0) finish(c0 + j, tot);
        }
    } else {
        for (int p = threadIdx.x; p < NV * kc; p += 256) {
            const int q = p / kc, j = p % kc;
            double t = 0.0;
            if (c0 + j < k) {
#pragma unroll 16
                for (int64_t i = 0; i < nb; ++i) t += __ldcg(part + ((int64_t)q * nb + i) * k + c0 + j);
            }
            sh[q * 32 + j] = t;
        }
        __syncthreads();
        if (threadIdx.x < kc && c0 + threadIdx.x < k) {
            double tot[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) tot[q] = sh[q * 32 + threadIdx.x];
            finish(c0 + threadIdx.x, tot);
        }
    }
}

template <int NV, int Batch = 8, class Elem, class Finish>
void column_reduce(int64_t n, int64_t k, const Elem& elem, const Finish& finish, PcgWorkspace& ws,
                   cudaStream_t s) {
    ws.reserve_reduction(n, k, NV, s);
    int kc = 1;
    while (kc < k && kc < 32) kc *= 2;
    const int64_t nb = chunk_count(n), chunks = 32 / kc;
    launch_chained(k_column_reduce<NV, Batch, Elem, Finish>,
                   dim3((unsigned)((nb + chunks - 1) / chunks), (unsigned)((k + kc - 1) / kc)), 256, 0, s, n,
                   k, chunk_rows(n), nb, kc, ws.partial.get(), ws.counter.get(), elem, finish);
    CS_LAUNCH("column_reduce");
}

struct StoreSum {
    double* out;
    __device__ void operator()(int64_t c, const double (&t)[1]) const { out[c] = t[0]; }
};
struct StoreTwo {
    double *a, *b;
    __device__ void operator()(int64_t c, const double (&t)[2]) const {
        a[c] = t[0];
        b[c] = t[1];
    }
};
struct Dot {
    const double* A;
    int64_t lda;
    const double* B;
    int64_t ldb;
    struct In {
        double a, b;
    };
    __device__ In load(int64_t r, int64_t c) const { return {A[r * lda + c], B[r * ldb + c]}; }
    __device__ void use(const In& in, int64_t, int64_t, double (&v)[1]) const { v[0] += in.a * in.b; }
};
// R = B (columns idx), P = B / diag; r . r and r . p
struct CgInit {
    const double* B;
    int64_t ldb;
    const int32_t* idx;
    double *R, *P;
    int64_t ld;
    double diag;
    struct In {
        double b;
    };
    __device__ In load(int64_t r, int64_t c) const { return {B[r * ldb + idx[c]]}; }
    __device__ void use(const In& in, int64_t r, int64_t c, double (&v)[2]) const {
        const double b = in.b, p = b / diag;
        R[r * ld + c] = b;
        P[r * ld + c] = p;
        v[0] += b * b;
        v[1] += b * p;
    }
};
// AP = V p and p . AP
struct CgProduct {
    Covariance cov;
    double* out;
    int64_t ldo;
    using In = Covariance::In;
    __device__ In load(int64_t r, int64_t c) const { return cov.load(r, c); }
    __device__ void use(const In& in, int64_t r, int64_t c, double (&v)[1]) const {
        const double o = cov.value(in);
        out[r * ldo + c] = o;
        v[0] += in.v * o;
    }
};
// alpha = rsold / (p . Ap)
struct CgAlpha {
    const double* rsold;
    double* alpha;
    __device__ void operator()(int64_t c, const double (&t)[1]) const { alpha[c] = rsold[c] / t[0]; }
};
// x += alpha p, r -= alpha Ap; r . r and r . z with z = r / diag
struct CgUpdate {
    double* X;
    int64_t ldx;
    const int32_t* map;
    const double *P, *AP;
    double* R;
    int64_t ld;
    const double* alpha;
    double diag;
    struct In {
        double x, p, r, ap;
    };
    __device__ In load(int64_t r, int64_t c) const {
        return {X[r * ldx + map[c]], P[r * ld + c], R[r * ld + c], AP[r * ld + c]};
    }
    __device__ void use(const In& in, int64_t r, int64_t c, double (&v)[2]) const {
        const double a = alpha[c];
        X[r * ldx + map[c]] = in.x + a * in.p;
        const double rv = in.r - a * in.ap;
        R[r * ld + c] = rv;
        v[0] += rv * rv;
        v[1] += rv * (rv / diag);
    }
};
// beta = rz / rsold, rsold = rz; the squared residual (and rz) to the host
struct CgBeta {
    double *rsold, *beta, *rr_host, *rz_host;
    __device__ void operator()(int64_t c, const double (&t)[2]) const {
        rr_host[c] = t[0];
        rz_host[c] = t[1];
        beta[c] = t[1] / rsold[c];
        rsold[c] = t[1];
    }
};
struct CgBetaZ {
    double *rsold, *beta, *rz_host;
    __device__ void operator()(int64_t c, const double (&t)[1]) const {
        rz_host[c] = t[0];
        beta[c] = t[0] / rsold[c];
        rsold[c] = t[0];
    }
};
// w -= sum_q coef[q] o sub[q] (blocks of n x k), then NV sums: w . dot[q], or w . w without dot
constexpr int kLanczosGroup = kLanczosCoef;
template <int NV>
struct LanczosElem {
    double* w;
    const double *sub, *dot, *coef;
    int n_sub, n_dot;
    int64_t ld, block;
    struct In {
        double x, d[NV];
    };
    __device__ In load(int64_t r, int64_t c) const {
        In in;
        in.x = w[r * ld + c];
        double s[8];
        for (int q0 = 0; q0 < n_sub; q0 += 8) {
#pragma unroll
            for (int q = 0; q < 8; ++q) s[q] = q0 + q < n_sub ? sub[(q0 + q) * block + r * ld + c] : 0.0;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q0 + q < n_sub) in.x -= coef[(q0 + q) * ld + c] * s[q];
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) in.d[q] = q < n_dot ? dot[q * block + r * ld + c] : 0.0;
        return in;
    }
    __device__ void use(const In& in, int64_t r, int64_t c, double (&v)[NV]) const {
        if (n_sub) w[r * ld + c] = in.x;
        if (n_dot == 0) v[0] += in.x * in.x;
        else
#pragma unroll
            for (int q = 0; q < NV; ++q) v[q] += in.x * in.d[q];
    }
};
// w = V v_j - beta_{j-1} v_{j-1}; w . v_j  (V v_j from the product's parts)
struct LanczosFirst {
    Covariance cov;
    double* w;
    const double *prev, *coef;
    struct In {
        Covariance::In cov;
        double prev;
    };
    __device__ In load(int64_t r, int64_t c) const {
        return {cov.load(r, c), prev ? prev[r * cov.ldv + c] : 0.0};
    }
    __device__ void use(const In& in, int64_t r, int64_t c, double (&v)[1]) const {
        double x = cov.value(in.cov);
        if (prev) x -= coef[c] * in.prev;
        w[r * cov.ldv + c] = x;
        v[0] += x * in.cov.v;
    }
};
enum class LanczosMode { kAlpha, kBeta };
struct LanczosFinish {
    LanczosState st;
    LanczosMode mode;
    int step;
    __device__ void operator()(int64_t c, const double (&t)[1]) const {
        const bool done = st.done[c] != 0;
        double coef = done ? 0.0 : t[0];
        if (!done && mode == LanczosMode::kAlpha) st.alpha[c] = t[0];
        if (!done && mode == LanczosMode::kBeta) {
            coef = sqrt(t[0]);
            st.beta[c] = coef;
            if (coef < 1e-12) {
                st.steps[c] = step + 1;
                st.done[c] = 1;
                coef = 0.0;
            }
        }
        st.coef[c] = coef;
    }
};
struct LanczosGroup {
    LanczosState st;
    int64_t k;
    __device__ void operator()(int64_t c, const double (&t)[kLanczosGroup]) const {
        const bool done = st.done[c] != 0;
#pragma unroll
        for (int q = 0; q < kLanczosGroup; ++q) st.coef[q * k + c] = done ? 0.0 : t[q];
    }
};

// p = z + beta p
__global__ void k_direction_z(double* __restrict__ P, const double* __restrict__ Z, int64_t ld,
                              int64_t n, int64_t k, const double* __restrict__ beta) {
    chain_enter();
    const int64_t total = n * k;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / k, c = e - r * k;
        P[r * ld + c] = Z[r * ld + c] + beta[c] * P[r * ld + c];
    }
}

// p = r / diag + beta p
__global__ void k_direction(double* __restrict__ P, const double* __restrict__ R, int64_t ld,
                            int64_t n, int64_t k, double diag, const double* __restrict__ beta) {
    chain_enter();
    const int64_t total = n * k;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / k, c = e - r * k;
        P[r * ld + c] = R[r * ld + c] / diag + beta[c] * P[r * ld + c];
    }
}

__global__ void k_gather_cols(const double* __restrict__ src, int64_t lds, int64_t n,
                              const int32_t* __restrict__ idx, int64_t k, double* __restrict__ dst,
                              int64_t ldd) {
    const int64_t total = n * k;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / k, c = e - r * k;
        dst[r * ldd + c] = src[r * lds + idx[c]];
    }
}

// U[i, c] = sum of the records of row i, in record order (stcg_vce.cpp:64-70)
__global__ void k_records_to_rows(const double* __restrict__ V, int64_t ldv, int64_t k,
                                  const int32_t* __restrict__ row_ptr,
                                  const int32_t* __restrict__ row_recs, int64_t n_rows,
                                  double* __restrict__ U, int64_t ldu) {
    const int64_t total = n_rows * k;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / k, c = e - i * k;
        double s = 0.0;
        for (int32_t q = row_ptr[i]; q < row_ptr[i + 1]; ++q) s += V[(int64_t)row_recs[q] * ldv + c];
        U[i * ldu + c] = s;
    }
}

// g_out = fac * KU[row(r)], pe_out = U[row(r)]   (stcg_vce.cpp:89-101)
__global__ void k_scatter_rows(double* __restrict__ g_out, int64_t ldg, double* __restrict__ pe_out,
                               int64_t ldp, const double* __restrict__ KU, int64_t ldk,
                               const double* __restrict__ U, int64_t ldu,
                               const int32_t* __restrict__ rec_to_row, int64_t n_rec, int64_t k,
                               double fac) {
    const int64_t total = n_rec * k;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / k, c = e - r * k;
        const int64_t i = rec_to_row ? rec_to_row[r] : r;
        double g = 0.0, pe = 0.0;
        if (i >= 0) {
            g = KU[i * ldk + c];
            if (fac != 1.0) g *= fac;
            pe = U[i * ldu + c];
        }
        g_out[r * ldg + c] = g;
        if (pe_out) pe_out[r * ldp + c] = pe;
    }
}

__global__ void k_scale_copy(const double* __restrict__ src, int64_t lds, int64_t n, int64_t k,
                             double fac, double* __restrict__ dst, int64_t ldd) {
    const int64_t total = n * k;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = e / k, c = e - r * k;
        dst[r * ldd + c] = fac != 1.0 ? src[r * lds + c] * fac : src[r * lds + c];
    }
}

unsigned grid_for(int64_t total) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((total + 255) / 256, 16LL * num_sms()));
}

void swap_buffers(DeviceBuffer<double>& a, DeviceBuffer<double>& b) {
    std::swap(a.ptr, b.ptr);
    std::swap(a.count, b.count);
}

}  // namespace

// ---------------------------------------------------------------- record map
void RecordMap::build(const int32_t* rec_to_row_host, int64_t nrec, int64_t nrows) {
    n_rec = nrec;
    n_rows = nrows;
    identity = rec_to_row_host == nullptr;
    rec_to_row.clear();
    if (identity) {
        if (nrec != nrows)
            fail(CS_ERR_INVALID_ARGUMENT, "records without a record map must equal the operator rows");
        return;
    }
    rec_to_row.assign(rec_to_row_host, rec_to_row_host + nrec);
    std::vector<int32_t> ptr(nrows + 1, 0), recs;
    for (int64_t r = 0; r < nrec; ++r) {
        const int32_t i = rec_to_row[r];
        if (i < -1 || i >= nrows)
            fail(CS_ERR_INVALID_ARGUMENT, "record maps to a genotype row out of range");
        if (i >= 0) ++ptr[i + 1];
    }
    for (int64_t i = 0; i < nrows; ++i) ptr[i + 1] += ptr[i];
    recs.resize(ptr[nrows]);
    std::vector<int32_t> fill(ptr.begin(), ptr.end() - 1);
    for (int64_t r = 0; r < nrec; ++r)
        if (rec_to_row[r] >= 0) recs[fill[rec_to_row[r]]++] = (int32_t)r;
    d_rec_to_row.resize(std::max<int64_t>(1, nrec));
    d_row_ptr.resize(nrows + 1);
    d_row_recs.resize(std::max<size_t>(1, recs.size()));
    CS_CUDA(cudaMemcpy(d_rec_to_row.get(), rec_to_row.data(), 4 * nrec, cudaMemcpyHostToDevice));
    CS_CUDA(cudaMemcpy(d_row_ptr.get(), ptr.data(), 4 * (nrows + 1), cudaMemcpyHostToDevice));
    if (!recs.empty())
        CS_CUDA(cudaMemcpy(d_row_recs.get(), recs.data(), 4 * recs.size(), cudaMemcpyHostToDevice));
}

// ---------------------------------------------------------------- V operator
const double* VOperator::gather(const double* in, int64_t ldi, int64_t k, cudaStream_t s) {
    if (rm->identity) return in;
    u.resize(std::max<int64_t>(1, rm->n_rows * k));
    prof::Scope ps("records_to_rows", s, 0.0, 8.0 * (double)(rm->n_rec + rm->n_rows) * k);
    k_records_to_rows<<<grid_for(rm->n_rows * k), 256, 0, s>>>(
        in, ldi, k, rm->d_row_ptr.get(), rm->d_row_recs.get(), rm->n_rows, u.get(), k);
    CS_LAUNCH("records_to_rows");
    return u.get();
}

const double* VOperator::kinship(const double* in, int64_t ldi, int64_t k, int64_t& ldu, cudaStream_t s) {
    const double* U = gather(in, ldi, k, s);
    ldu = rm->identity ? ldi : k;
    ku.resize(std::max<int64_t>(1, rm->n_rows * k));
    kinship_apply_checked(op, U, ldu, k, ku.get(), k, precision, s);
    ++applies;
    apply_cols += k;
    return U;
}

Covariance VOperator::covariance(const double* in, int64_t ldi, const double* U, int64_t ldu, int64_t k) const {
    return Covariance{in, ku.get(), U, ldi, k, ldu, rm->identity ? nullptr : rm->d_rec_to_row.get(),
                      vg, fac, vpe, ve, with_pe ? 1 : 0};
}

void VOperator::apply_alpha(const double* p, int64_t k, double* out, const double* rsold, double* alpha,
                            PcgWorkspace& ws, cudaStream_t s) {
    int64_t ldu = 0;
    const double* U = kinship(p, k, k, ldu, s);
    const Covariance cov = covariance(p, k, U, ldu, k);
    prof::Scope ps("covariance_combine", s, 2.0 * (double)rm->n_rec * k, 8.0 * 3.0 * (double)rm->n_rec * k);
    column_reduce<1>(rm->n_rec, k, CgProduct{cov, out, k}, CgAlpha{rsold, alpha}, ws, s);
}

void VOperator::derivatives(const double* in, int64_t ldi, int64_t k, double* g_out, int64_t ldg,
                            double* pe_out, int64_t ldp, cudaStream_t s) {
    if (k <= 0) return;
    const double* U = gather(in, ldi, k, s);
    const int64_t ldu = rm->identity ? ldi : k;
    ku.resize(std::max<int64_t>(1, rm->n_rows * k));
    kinship_apply_checked(op, U, ldu, k, ku.get(), k, precision, s);
    ++applies;
    apply_cols += k;
    prof::Scope ps("records_scatter", s, 0.0, 8.0 * 2.0 * (double)rm->n_rec * k);
    k_scatter_rows<<<grid_for(rm->n_rec * k), 256, 0, s>>>(
        g_out, ldg, pe_out, ldp, ku.get(), k, U, ldu,
        rm->identity ? nullptr : rm->d_rec_to_row.get(), rm->n_rec, k, fac);
    CS_LAUNCH("records_scatter");
}

void VOperator::genetic_rows(const double* in, int64_t ldi, int64_t k, double* rows_out,
                             int64_t ldo, double* zt_out, int64_t ldz, cudaStream_t s) {
    if (k <= 0) return;
    const double* U = gather(in, ldi, k, s);
    const int64_t ldu = rm->identity ? ldi : k;
    ku.resize(std::max<int64_t>(1, rm->n_rows * k));
    kinship_apply_checked(op, U, ldu, k, ku.get(), k, precision, s);
    ++applies;
    apply_cols += k;
    k_scale_copy<<<grid_for(rm->n_rows * k), 256, 0, s>>>(ku.get(), k, rm->n_rows, k, fac,
                                                          rows_out, ldo);
    CS_LAUNCH("scale_copy");
    if (zt_out) {
        k_scale_copy<<<grid_for(rm->n_rows * k), 256, 0, s>>>(U, ldu, rm->n_rows, k, 1.0, zt_out, ldz);
        CS_LAUNCH("scale_copy");
    }
}

// ---------------------------------------------------------------- dots
void PcgWorkspace::reserve_reduction(int64_t n, int64_t k, int sums, cudaStream_t s) {
    partial.resize(std::max(2, sums) * chunk_count(n) * std::max<int64_t>(1, k));
    host.resize(2 * std::max<int64_t>(1, k));
    if (counter.count < (size_t)k) {
        counter.resize(k);
        CS_CUDA(cudaMemsetAsync(counter.get(), 0, sizeof(unsigned) * counter.count, s));
    }
}

void destroy_pcg(PcgWorkspace* w) { delete w; }

void column_dots(const double* A, int64_t lda, const double* B, int64_t ldb, int64_t n, int64_t k,
                 double* out_host, PcgWorkspace& ws, cudaStream_t s) {
    if (k <= 0) return;
    ws.reserve_reduction(n, k, 2, s);
    {
        prof::Scope ps("column_dots", s, 2.0 * n * k, 16.0 * n * k);
        column_reduce<1>(n, k, Dot{A, lda, B, ldb}, StoreSum{ws.host.ptr}, ws, s);
    }
    CS_CUDA(cudaStreamSynchronize(s));
    std::copy(ws.host.ptr, ws.host.ptr + k, out_host);
}

void lanczos_step(VOperator& V, const double* basis, int64_t k, double* w, const LanczosState& st, int step,
                  PcgWorkspace& ws, cudaStream_t s) {
    const int64_t n = V.rm->n_rec, block = n * k;
    const double* const vj = basis + step * block;
    int64_t ldu = 0;
    const double* U = V.kinship(vj, k, k, ldu, s);
    prof::Scope ps("lanczos_step", s, 4.0 * (step + 2) * block, 8.0 * (2 * step + 10) * block);
    column_reduce<1>(n, k, LanczosFirst{V.covariance(vj, k, U, ldu, k), w, step ? vj - block : nullptr, st.coef},
                     LanczosFinish{st, LanczosMode::kAlpha, step}, ws, s);
    // full reorthogonalisation against v_0 .. v_j, sixteen at a time; each kernel subtracts what the
    // one before it measured (first alpha v_j)
    const double* sub = vj;
    int n_sub = 1;
    for (int q = 0; q <= step; q += kLanczosGroup) {
        const int here = std::min(kLanczosGroup, step + 1 - q);
        column_reduce<kLanczosGroup, 2>(
            n, k, LanczosElem<kLanczosGroup>{w, sub, basis + q * block, st.coef, n_sub, here, k, block},
            LanczosGroup{st, k}, ws, s);
        sub = basis + q * block;
        n_sub = here;
    }
    column_reduce<1, 4>(n, k, LanczosElem<1>{w, sub, nullptr, st.coef, n_sub, 0, k, block},
                        LanczosFinish{st, LanczosMode::kBeta, step}, ws, s);
}

// ---------------------------------------------------------------- low-rank preconditioner
void LowRankPreconditioner::set_components(double vg, double ve, cudaStream_t s) {
    base = 1.0 / std::max(1e-300, vg * r0 + ve);
    std::vector<double> h(std::max<int64_t>(1, r));
    for (int64_t j = 0; j < r; ++j) h[j] = 1.0 / (vg * lambda[j] + ve) - base;
    c.resize(std::max<int64_t>(1, r));
    CS_CUDA(cudaMemcpyAsync(c.get(), h.data(), 8 * r, cudaMemcpyHostToDevice, s));
    CS_CUDA(cudaStreamSynchronize(s));  // h is a local
}

void LowRankPreconditioner::apply(const double* R, int64_t ldr, int64_t k, double* Z, int64_t ldz,
                                  cudaStream_t s) {
    if (k <= 0) return;
    cublasHandle_t blas = shared_blas();
    CS_BLAS(cublasSetStream(blas, s));
    T.resize(std::max<int64_t>(1, r * k));
    prof::Scope ps("lowrank_precondition", s, 4.0 * (double)n * r * k, 8.0 * (2.0 * n * k + n * r));
    // column-major views: R^T (k x n, ld ldr), U^T (r x n, ld r)
    const double one = 1.0, zero = 0.0;
    // T^T (k x r) = R^T U
    CS_BLAS(cublasDgemm(blas, CUBLAS_OP_N, CUBLAS_OP_T, (int)k, (int)r, (int)n, &one, R, (int)ldr,
                        U.get(), (int)r, &zero, T.get(), (int)k));
    // T^T[:, j] *= c_j
    CS_BLAS(cublasDdgmm(blas, CUBLAS_SIDE_RIGHT, (int)k, (int)r, T.get(), (int)k, c.get(), 1,
                        T.get(), (int)k));
    // Z^T = base R^T + T^T U^T
    CS_CUDA(cudaMemcpy2DAsync(Z, 8 * ldz, R, 8 * ldr, 8 * k, n, cudaMemcpyDeviceToDevice, s));
    CS_BLAS(cublasDgemm(blas, CUBLAS_OP_N, CUBLAS_OP_N, (int)k, (int)n, (int)r, &one, T.get(),
                        (int)k, U.get(), (int)r, &base, Z, (int)ldz));
}

// ---------------------------------------------------------------- block PCG
void pcg_solve_block(VOperator& A, double diag, const double* B, int64_t ldb, int64_t k,
                     double* X, int64_t ldx, double tol, bool relative, int max_iter,
                     PcgWorkspace& ws, PcgStats& st, cudaStream_t s, LowRankPreconditioner* M) {
    st.iterations.assign(k, 0);
    st.sweeps = 0;  // counts of this solve only
    st.column_iterations = 0;
    if (k <= 0) return;
    const int64_t n = A.rm->n_rec;
    const DeferChecks defer(A.op, s);
    CS_CUDA(cudaMemset2DAsync(X, ldx * 8, 0, k * 8, n, s));
    ws.R.resize(n * k);
    ws.P.resize(n * k);
    ws.AP.resize(n * k);
    ws.T.resize(n * k);
    ws.reserve_reduction(n, k, 2, s);
    for (auto* b : {&ws.alpha, &ws.beta, &ws.rsold}) b->resize(k);
    ws.map.resize(k);
    ws.idx.resize(k);
    double* const rr_h = ws.host.ptr;      // squared residuals and r . z of the live columns, written
    double* const rz_h = ws.host.ptr + k;  // by the kernels, read after a synchronisation
    std::vector<int32_t> map(k);
    for (int64_t c = 0; c < k; ++c) map[c] = (int32_t)c;
    CS_CUDA(cudaMemcpyAsync(ws.idx.get(), map.data(), 4 * k, cudaMemcpyHostToDevice, s));
    column_reduce<2>(n, k, CgInit{B, ldb, ws.idx.get(), ws.R.get(), ws.P.get(), k, diag},
                     StoreTwo{rr_h, rz_h}, ws, s);
    if (M) {
        ws.Zp.resize(n * k);
        M->apply(ws.R.get(), k, k, ws.P.get(), k, s);  // p0 = z0 = M^-1 r0
        column_reduce<1>(n, k, Dot{ws.R.get(), k, ws.P.get(), k}, StoreSum{rz_h}, ws, s);
    }
    // ||b||^2 and rsold = r . z
    CS_CUDA(cudaStreamSynchronize(s));
    std::vector<double> rr(rr_h, rr_h + k), rs(rz_h, rz_h + k);
    std::vector<double> tol_c(k);
    for (int64_t c = 0; c < k; ++c) tol_c[c] = relative ? tol * std::sqrt(rr[c]) : tol;
    // columns already solved by x = 0 (matrix_free_pcg.h:32)
    std::vector<int32_t> live;
    for (int64_t c = 0; c < k; ++c)
        if (!(std::sqrt(rr[c]) < 1e-20)) live.push_back((int32_t)c);
    int64_t ka = k;
    auto compact = [&](const std::vector<int32_t>& keep_pos, std::vector<double>& rs_host) {
        const int64_t kn = (int64_t)keep_pos.size();
        if (kn == 0) return;
        CS_CUDA(cudaMemcpyAsync(ws.idx.get(), keep_pos.data(), 4 * kn, cudaMemcpyHostToDevice, s));
        k_gather_cols<<<grid_for(n * kn), 256, 0, s>>>(ws.R.get(), ka, n, ws.idx.get(), kn, ws.T.get(), kn);
        CS_LAUNCH("gather_cols");
        swap_buffers(ws.R, ws.T);
        k_gather_cols<<<grid_for(n * kn), 256, 0, s>>>(ws.P.get(), ka, n, ws.idx.get(), kn, ws.T.get(), kn);
        CS_LAUNCH("gather_cols");
        swap_buffers(ws.P, ws.T);
        std::vector<double> r2(kn);
        for (int64_t j = 0; j < kn; ++j) r2[j] = rs_host[keep_pos[j]];
        rs_host = r2;
        CS_CUDA(cudaMemcpyAsync(ws.rsold.get(), rs_host.data(), 8 * kn, cudaMemcpyHostToDevice, s));
        std::vector<int32_t> m2(kn);
        for (int64_t j = 0; j < kn; ++j) m2[j] = map[keep_pos[j]];
        map = m2;
        ka = kn;
    };
    if ((int64_t)live.size() < k) {
        if (live.empty()) return;
        compact(live, rs);
    } else {
        CS_CUDA(cudaMemcpyAsync(ws.rsold.get(), rs.data(), 8 * k, cudaMemcpyHostToDevice, s));
    }
    CS_CUDA(cudaMemcpyAsync(ws.map.get(), map.data(), 4 * ka, cudaMemcpyHostToDevice, s));
    for (int it = 0; it < max_iter && ka > 0; ++it) {
        A.apply_alpha(ws.P.get(), ka, ws.AP.get(), ws.rsold.get(), ws.alpha.get(), ws, s);
        ++st.sweeps;
        st.column_iterations += ka;
        const CgUpdate update{X, ldx, ws.map.get(), ws.P.get(), ws.AP.get(), ws.R.get(), ka, ws.alpha.get(), diag};
        {
            prof::Scope ps("cg_step", s, 6.0 * n * ka, 8.0 * 6.0 * n * ka);
            if (M) {
                // z = M^-1 r and r . z in place of the scalar form's r . r / diag
                column_reduce<2>(n, ka, update, StoreTwo{rr_h, rz_h}, ws, s);
                M->apply(ws.R.get(), ka, ka, ws.Zp.get(), ka, s);
                column_reduce<1>(n, ka, Dot{ws.R.get(), ka, ws.Zp.get(), ka},
                                 CgBetaZ{ws.rsold.get(), ws.beta.get(), rz_h}, ws, s);
            } else {
                column_reduce<2>(n, ka, update, CgBeta{ws.rsold.get(), ws.beta.get(), rr_h, rz_h}, ws, s);
            }
        }
        // the next direction of every column (also of those that turn out to be done), so that the
        // device has it under way while the host looks at the residuals
        {
            prof::Scope ps("cg_direction", s, 2.0 * n * ka, 24.0 * n * ka);
            if (M)
                launch_chained(k_direction_z, grid_for(n * ka), 256, 0, s, ws.P.get(), ws.Zp.get(), ka, n, ka,
                               ws.beta.get());
            else
                launch_chained(k_direction, grid_for(n * ka), 256, 0, s, ws.P.get(), ws.R.get(), ka, n, ka,
                               diag, ws.beta.get());
            CS_LAUNCH("cg_direction");
        }
        CS_CUDA(cudaStreamSynchronize(s));
        for (int64_t c = 0; c < ka; ++c)
            if (std::isnan(rr_h[c])) {  // an FP64 apply that gave up leaves NaN (a mixed one may not)
                kinship_check(A.op, s);
                break;
            }
        std::vector<int32_t> keep_pos;
        for (int64_t c = 0; c < ka; ++c) {
            st.iterations[map[c]] = it + 1;
            if (!(std::sqrt(rr_h[c]) < tol_c[map[c]])) keep_pos.push_back((int32_t)c);
        }
        if (keep_pos.empty()) break;
        if ((int64_t)keep_pos.size() < ka) {
            std::vector<double> rs_h(rz_h, rz_h + ka);
            compact(keep_pos, rs_h);
            CS_CUDA(cudaMemcpyAsync(ws.map.get(), map.data(), 4 * ka, cudaMemcpyHostToDevice, s));
        }
    }
    kinship_check(A.op, s);
    CS_CUDA(cudaStreamSynchronize(s));
}

}  // namespace cs
