// Resident packed genotypes: upload, per-SNP statistics, code counts, repacking.
//
// Reference behaviour restated here:
//   libCosmicCore/src/plink_reader.cpp:67-92   openBed (magic 6C 1B 01, SNP-major only)
//   libCosmicCore/src/plink_reader.cpp:187-239 computeStats (mean, 1/sqrt(2p(1-p)))
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <fstream>
#include <string>
#include <thread>
#include <vector>

#include "cs_internal.h"

namespace cs {

namespace {

// Counts of the four 2-bit codes in a 32-bit word (16 samples).
__device__ __forceinline__ void count_codes(uint32_t w, int& c00, int& c01, int& c10, int& c11) {
    const uint32_t lo = w & 0x55555555u;
    const uint32_t hi = (w >> 1) & 0x55555555u;
    c01 += __popc(lo & ~hi);
    c10 += __popc(hi & ~lo);
    c11 += __popc(hi & lo);
    c00 += __popc(~(lo | hi) & 0x55555555u);
}

// One warp per row: counts of codes 00 (two A1), 01 (missing), 10 (het), 11 (zero A1).
__global__ void k_row_code_counts(const uint8_t* __restrict__ rows, int64_t n_rows,
                                  int64_t stride, int32_t* __restrict__ counts) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t n_warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = warp; t < n_rows; t += n_warps) {
        const uint4* row = reinterpret_cast<const uint4*>(rows + t * stride);
        int c00 = 0, c01 = 0, c10 = 0, c11 = 0;
        for (int64_t q = lane; q < stride / 16; q += 32) {
            const uint4 v = __ldg(row + q);
            count_codes(v.x, c00, c01, c10, c11);
            count_codes(v.y, c00, c01, c10, c11);
            count_codes(v.z, c00, c01, c10, c11);
            count_codes(v.w, c00, c01, c10, c11);
        }
        c00 = __reduce_add_sync(0xffffffffu, c00);
        c01 = __reduce_add_sync(0xffffffffu, c01);
        c10 = __reduce_add_sync(0xffffffffu, c10);
        c11 = __reduce_add_sync(0xffffffffu, c11);
        if (lane == 0) {
            counts[4 * t + 0] = c00;
            counts[4 * t + 1] = c01;
            counts[4 * t + 2] = c10;
            counts[4 * t + 3] = c11;
        }
    }
}

// plink_reader.cpp:213-233 with the same operation order and no contraction:
// mean = sum / count; p = mean / 2; var = 2 * p * (1 - p); inv_std = 1 / sqrt(var).
__global__ void k_stats_from_counts(const int32_t* __restrict__ counts, int64_t n,
                                    double* __restrict__ mean, double* __restrict__ inv_std,
                                    int32_t* __restrict__ count_out, double* __restrict__ sum_out) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int32_t c00 = counts[4 * j + 0], c10 = counts[4 * j + 2], c11 = counts[4 * j + 3];
    const int32_t count = c00 + c10 + c11;
    const double sum = (double)(2 * (int64_t)c00 + c10);
    count_out[j] = count;
    sum_out[j] = sum;
    if (count > 0) {
        const double m = __ddiv_rn(sum, (double)count);
        const double p = __ddiv_rn(m, 2.0);
        const double var = __dmul_rn(__dmul_rn(2.0, p), __dsub_rn(1.0, p));
        mean[j] = m;
        inv_std[j] = (var < 1e-9) ? 0.0 : __ddiv_rn(1.0, __dsqrt_rn(var));
    } else {
        mean[j] = 0.0;
        inv_std[j] = 0.0;
    }
}

// Samples at or beyond n_samples in the last byte of each row become "missing".
__global__ void k_sanitize_tail(uint8_t* rows, int64_t n_rows, int64_t stride, int64_t last_byte,
                                int used_codes) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n_rows) return;
    uint8_t b = rows[t * stride + last_byte];
    for (int q = used_codes; q < 4; ++q) b = (uint8_t)((b & ~(3u << (2 * q))) | (1u << (2 * q)));
    rows[t * stride + last_byte] = b;
}

// dst row t = src row rows[t] (or t) restricted to the samples keep (or the first n_keep), packed and
// padded with the missing code.  A block takes kRows rows: they go through shared memory whole
// (a keep list may name samples anywhere in the row, in any order), and a thread makes 16 output
// codes of each from one reading of its 16 indices.
// 20,011 samples x 30,007 variants to 18,010 x 27,006: 284 us (a shared-memory look-up and three
// operations a code), 623 with a byte at a time from global memory.
template <int kRows>
__global__ void __launch_bounds__(256)
k_repack(const uint8_t* __restrict__ src, int64_t src_stride, const int32_t* __restrict__ rows,
         int64_t n_rows, const int32_t* __restrict__ keep, int64_t n_keep,
         uint8_t* __restrict__ dst, int64_t dst_stride) {
    extern __shared__ __align__(16) uint8_t packed[];  // [kRows][src_stride]
    const int64_t t0 = (int64_t)blockIdx.x * kRows;
    const int here = (int)min((int64_t)kRows, n_rows - t0);
    for (int r = 0; r < kRows; ++r) {  // a part full block reads its last row again: no tests below
        const int64_t t = t0 + min(r, here - 1);
        const uint4* s = reinterpret_cast<const uint4*>(src + (int64_t)(rows ? rows[t] : t) * src_stride);
        for (int64_t q = threadIdx.x; q < src_stride / 16; q += 256)
            reinterpret_cast<uint4*>(packed + r * src_stride)[q] = __ldg(s + q);
    }
    __syncthreads();
    const int row_bytes = (int)src_stride;
    for (int64_t w = threadIdx.x; w < dst_stride / 4; w += 256) {
        uint32_t out[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) out[r] = 0u;
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int64_t i = 16 * w + j;
            if (i < n_keep) {
                const int32_t k = keep ? __ldg(keep + i) : (int32_t)i;
                const uint8_t* const p = packed + (k >> 2);
                const int sh = (k & 3) * 2;
#pragma unroll
                for (int r = 0; r < kRows; ++r) out[r] += ((p[r * row_bytes] >> sh) & 3u) * (1u << (2 * j));
            } else {
#pragma unroll
                for (int r = 0; r < kRows; ++r) out[r] += 1u << (2 * j);
            }
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r)
            if (r < here) reinterpret_cast<uint32_t*>(dst + (t0 + r) * dst_stride)[w] = out[r];
    }
}

// The same a byte at a time from global memory, for rows that do not fit shared memory.
__global__ void k_repack_long(const uint8_t* __restrict__ src, int64_t src_stride,
                              const int32_t* __restrict__ rows, int64_t n_rows,
                              const int32_t* __restrict__ keep, int64_t n_keep,
                              uint8_t* __restrict__ dst, int64_t dst_stride) {
    const int64_t total = n_rows * dst_stride;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t t = idx / dst_stride;
        const int64_t b = idx - t * dst_stride;
        const uint8_t* srow = src + (int64_t)(rows ? rows[t] : t) * src_stride;
        uint32_t out = 0;
        for (int q = 0; q < 4; ++q) {
            const int64_t r = 4 * b + q;
            uint32_t code = 1;
            if (r < n_keep) {
                const int64_t s = keep ? keep[r] : r;
                code = (srow[s >> 2] >> ((s & 3) * 2)) & 3u;
            }
            out |= code << (2 * q);
        }
        dst[idx] = (uint8_t)out;
    }
}

__global__ void k_col_to_row(const double* __restrict__ src, int64_t ld, int64_t n, int64_t k,
                             double* __restrict__ dst, int64_t kp) {
    const int64_t total = n * kp;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = idx / kp, c = idx - i * kp;
        dst[idx] = c < k ? src[i + c * ld] : 0.0;
    }
}

__global__ void k_row_to_col(const double* __restrict__ src, int64_t kp, int64_t n, int64_t k,
                             double* __restrict__ dst, int64_t ld) {
    const int64_t total = n * k;
    for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = idx / n, i = idx - c * n;
        dst[i + c * ld] = src[i * kp + c];
    }
}

int grid_for(int64_t work, int threads) {
    const int64_t blocks = (work + threads - 1) / threads;
    const int64_t cap = (int64_t)num_sms() * 32;
    return (int)std::max<int64_t>(1, std::min(blocks, cap));
}

}  // namespace

int num_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    return sms;
}

void row_code_counts(const cs_packed_view& v, int32_t* d_counts, cudaStream_t s) {
    if (v.n_rows == 0) return;
    const int threads = 256;
    prof::Scope ps("row_code_counts", s, 0.0, (double)v.n_rows * ((v.n_samples + 3) / 4));
    k_row_code_counts<<<grid_for(v.n_rows * 32, threads), threads, 0, s>>>(v.rows, v.n_rows,
                                                                          v.stride, d_counts);
    CS_LAUNCH("row_code_counts");
}

void repack(const uint8_t* src, int64_t src_stride, const int32_t* d_rows, int64_t n_rows,
            const int32_t* d_keep, int64_t n_keep, uint8_t* dst, int64_t dst_stride,
            cudaStream_t s) {
    if (n_rows == 0) return;
    prof::Scope ps("repack", s, 0.0, (double)n_rows * dst_stride);
    // as many rows a block as keep two blocks on an SM, four where one block must do (every row then
    // still shares the indices with three others)
    constexpr int64_t kHalf = 110 * 1024, kWhole = 220 * 1024;
    static PerDeviceOnce configured;
    once_per_device(configured, [] {
        cudaError_t e = cudaFuncSetAttribute(k_repack<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHalf);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_repack<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWhole);
        return e;
    }, "configure repack kernels");
    if (8 * src_stride <= kHalf)
        k_repack<8><<<(unsigned)((n_rows + 7) / 8), 256, 8 * src_stride, s>>>(
            src, src_stride, d_rows, n_rows, d_keep, n_keep, dst, dst_stride);
    else if (4 * src_stride <= kWhole)
        k_repack<4><<<(unsigned)((n_rows + 3) / 4), 256, 4 * src_stride, s>>>(
            src, src_stride, d_rows, n_rows, d_keep, n_keep, dst, dst_stride);
    else
        k_repack_long<<<grid_for(n_rows * dst_stride, 256), 256, 0, s>>>(
            src, src_stride, d_rows, n_rows, d_keep, n_keep, dst, dst_stride);
    CS_LAUNCH("repack");
}

void colmajor_to_rowmajor(const double* src, int64_t ld, int64_t n, int64_t k, double* dst,
                          int64_t kp, cudaStream_t s) {
    if (n * kp == 0) return;
    prof::Scope ps("colmajor_to_rowmajor", s, 0.0, 16.0 * n * kp);
    k_col_to_row<<<grid_for(n * kp, 256), 256, 0, s>>>(src, ld, n, k, dst, kp);
    CS_LAUNCH("colmajor_to_rowmajor");
}

void rowmajor_to_colmajor(const double* src, int64_t kp, int64_t n, int64_t k, double* dst,
                          int64_t ld, cudaStream_t s) {
    if (n * k == 0) return;
    prof::Scope ps("rowmajor_to_colmajor", s, 0.0, 16.0 * n * k);
    k_row_to_col<<<grid_for(n * k, 256), 256, 0, s>>>(src, kp, n, k, dst, ld);
    CS_LAUNCH("rowmajor_to_colmajor");
}

// The staged copy of upload_rows: whole rows, padded on the way, a megabyte at a time through
// page-locked memory, by as many threads as the copy to it takes (a core moves 10 to 15 GB/s, the
// link 50).  cudaMemcpy2D from pageable memory, which stages on one thread and row by row, took
// 20.8 ms for 150 MB (20,011 samples), and opening that matrix 22.5 ms; it is 4.3 ms this way (50,000
// samples, 1.25 GB: 147 to 28.6; 203 samples, 15 MB: 79 to 3.4).  False: no page-locked memory.
static bool upload_staged(const uint8_t* src, int64_t M, int64_t bps, int spare, uint8_t* dst,
                          int64_t stride, cudaStream_t s) {
    constexpr int64_t kPiece = 1 << 20;
    constexpr int kSlots = 2, kMaxThreads = 4;
    const int64_t rows = kPiece / stride, pieces = (M + rows - 1) / rows;
    const int threads = (int)std::min<int64_t>(
        {kMaxThreads, pieces, std::max<int64_t>(1, std::thread::hardware_concurrency())});
    const size_t bytes = (size_t)threads * kSlots * kPiece;
    uint8_t* staging = nullptr;
    try {
        staging = static_cast<uint8_t*>(pinned_alloc(bytes));
    } catch (const std::exception&) {
        return false;
    }
    int device = 0;
    cudaGetDevice(&device);
    std::atomic<int64_t> next{0};
    std::atomic<int> error{(int)cudaSuccess};
    auto work = [&](int w) {
        cudaError_t e = cudaSetDevice(device);
        cudaEvent_t done[kSlots] = {};
        bool used[kSlots] = {};
        for (int q = 0; q < kSlots && e == cudaSuccess; ++q)
            e = cudaEventCreateWithFlags(&done[q], cudaEventDisableTiming);
        for (int q = 0; e == cudaSuccess && error.load() == (int)cudaSuccess; q = (q + 1) % kSlots) {
            const int64_t i = next.fetch_add(1);
            if (i >= pieces) break;
            if (used[q]) e = cudaEventSynchronize(done[q]);
            if (e != cudaSuccess) break;
            uint8_t* const slot = staging + ((int64_t)w * kSlots + q) * kPiece;
            const int64_t r0 = i * rows, r1 = std::min(M, r0 + rows);
            for (int64_t r = r0; r < r1; ++r) {
                uint8_t* const row = slot + (r - r0) * stride;
                std::memcpy(row, src + r * bps, (size_t)bps);
                if (spare) {
                    const uint8_t mask = (uint8_t)((1 << (2 * spare)) - 1);
                    row[bps - 1] = (uint8_t)((row[bps - 1] & mask) | (kMissingByte & ~mask));
                }
                std::memset(row + bps, kMissingByte, (size_t)(stride - bps));
            }
            e = cudaMemcpyAsync(dst + r0 * stride, slot, (size_t)((r1 - r0) * stride), cudaMemcpyHostToDevice, s);
            if (e == cudaSuccess) e = cudaEventRecord(done[q], s);
            used[q] = e == cudaSuccess;
        }
        // the slots are free again when their copies have ended
        for (int q = 0; q < kSlots; ++q) {
            if (used[q]) {
                const cudaError_t e2 = cudaEventSynchronize(done[q]);
                if (e == cudaSuccess) e = e2;
            }
            if (done[q]) cudaEventDestroy(done[q]);
        }
        if (e != cudaSuccess) error.store((int)e);
    };
    std::vector<std::thread> helpers;
    try {
        helpers.reserve(threads);
        for (int w = 1; w < threads; ++w) helpers.emplace_back(work, w);
    } catch (const std::exception&) {  // fewer threads then: pieces go to whoever asks
    }
    work(0);
    for (auto& t : helpers) t.join();
    const cudaError_t e = (cudaError_t)error.load();
    if (e != cudaSuccess) cudaStreamSynchronize(s);  // whatever was queued from the staging memory
    pinned_free(staging, bytes);
    CS_CUDA(e);
    return true;
}

static bool pageable(const void* p) {
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// .bed rows (bps bytes each) to device rows of `stride` bytes; padding bytes and the last byte's
// spare codes become the missing code.  One copy takes matrices below 2 MiB, where a piece or two leave
// threads nothing to share (at 2.1 MB staged 0.40 ms against 1.31), rows too long for the pieces, and
// sources that are page-locked already, which the link reads where they are (50,000 samples, 1.25 GB
// 24.9 ms, staged 30 to 37), unless their rows are short (a strided copy pays 40 to 130 ns a row: 203
// samples x 300,000 variants 12.7 ms, staged 3.5).
static void upload_rows(const uint8_t* src, int64_t M, int64_t bps, int64_t n_samples, uint8_t* dst,
                        int64_t stride, cudaStream_t s) {
    const int spare = (int)(n_samples % 4);  // codes in use in the last byte, 0: all four
    if (M * stride >= (2 << 20) && stride <= (1 << 18) &&
        (bps < 4096 || (pageable(src) && pageable(src + M * bps - 1))) &&
        upload_staged(src, M, bps, spare, dst, stride, s))
        return;
    CS_CUDA(cudaMemsetAsync(dst, kMissingByte, M * stride, s));
    CS_CUDA(cudaMemcpy2DAsync(dst, stride, src, bps, bps, M, cudaMemcpyHostToDevice, s));
    if (spare) {
        prof::Scope ps("sanitize_tail", s);
        k_sanitize_tail<<<(unsigned)((M + 255) / 256), 256, 0, s>>>(dst, M, stride, bps - 1, spare);
        CS_LAUNCH("sanitize_tail");
    }
}

// Builds the device-resident matrix from the .bed bytes (magic included).
cs_genotypes* genotypes_from_bed(const uint8_t* bed, size_t n_bytes, int64_t n_samples,
                                 int64_t n_snps) {
    if (n_samples <= 0) fail(CS_ERR_INVALID_ARGUMENT, "No samples found in .fam file");
    if (n_snps < 0) fail(CS_ERR_INVALID_ARGUMENT, "negative SNP count");
    if (bed == nullptr || n_bytes < 3) fail(CS_ERR_FORMAT, "Invalid .bed file (too small)");
    if (bed[0] != 0x6C || bed[1] != 0x1B) fail(CS_ERR_FORMAT, "Invalid .bed file magic number");
    if (bed[2] != 0x01)
        fail(CS_ERR_FORMAT, "Only SNP-major mode (0x01) .bed files are supported");
    const int64_t bps = (n_samples + 3) / 4;
    if ((int64_t)n_bytes < 3 + n_snps * bps)
        fail(CS_ERR_FORMAT, "Invalid .bed file: " + std::to_string(n_bytes) +
                                " bytes < expected " + std::to_string(3 + n_snps * bps));
    prof::HostScope hs("genotypes_upload_stats");
    auto* g = new cs_genotypes();
    static std::atomic<uint64_t> next_uid{1};
    g->uid = next_uid.fetch_add(1);
    try {
        CS_CUDA(cudaGetDevice(&g->device));
        g->n_samples = n_samples;
        g->n_snps = n_snps;
        g->bytes_per_snp = bps;
        g->stride = round_up(bps, kRowAlign);
        const int64_t M = n_snps;
        g->packed.resize(std::max<int64_t>(1, M * g->stride));
        cudaStream_t s = 0;
        if (M > 0) upload_rows(bed + 3, M, bps, n_samples, g->packed.get(), g->stride, s);
        g->d_mean.resize(std::max<int64_t>(1, M));
        g->d_inv_std.resize(std::max<int64_t>(1, M));
        g->mean.assign(M, 0.0);
        g->inv_std.assign(M, 0.0);
        g->count.assign(M, 0);
        g->sum.assign(M, 0.0);
        g->code_counts.assign(4 * M, 0);
        if (M > 0) {
            DeviceBuffer<int32_t>& counts = g->d_code_counts;
            DeviceBuffer<int32_t> cnt;
            DeviceBuffer<double> sum;
            counts.resize(4 * M);
            cnt.resize(M);
            sum.resize(M);
            cs_packed_view v{g->packed.get(), M, n_samples, g->stride};
            row_code_counts(v, counts.get(), s);
            prof::Scope ps("stats_from_counts", s);
            k_stats_from_counts<<<(unsigned)((M + 255) / 256), 256, 0, s>>>(
                counts.get(), M, g->d_mean.get(), g->d_inv_std.get(), cnt.get(), sum.get());
            CS_LAUNCH("stats_from_counts");
            CS_CUDA(cudaMemcpyAsync(g->mean.data(), g->d_mean.get(), M * 8, cudaMemcpyDeviceToHost, s));
            CS_CUDA(cudaMemcpyAsync(g->inv_std.data(), g->d_inv_std.get(), M * 8,
                                    cudaMemcpyDeviceToHost, s));
            CS_CUDA(cudaMemcpyAsync(g->count.data(), cnt.get(), M * 4, cudaMemcpyDeviceToHost, s));
            CS_CUDA(cudaMemcpyAsync(g->sum.data(), sum.get(), M * 8, cudaMemcpyDeviceToHost, s));
            CS_CUDA(cudaMemcpyAsync(g->code_counts.data(), counts.get(), M * 16,
                                    cudaMemcpyDeviceToHost, s));
            CS_CUDA(cudaStreamSynchronize(s));
        }
    } catch (...) {
        delete g;
        throw;
    }
    return g;
}

static int64_t count_lines(const std::string& path) {
    std::ifstream ifs(path);
    if (!ifs) fail(CS_ERR_IO, "Cannot open file: " + path);
    std::string line;
    int64_t n = 0;
    while (std::getline(ifs, line))
        if (!line.empty()) ++n;
    return n;
}

cs_genotypes* genotypes_open_plink(const std::string& prefix) {
    const int64_t n = count_lines(prefix + ".fam");
    if (n == 0) fail(CS_ERR_INVALID_ARGUMENT, "No samples found in .fam file");
    const int64_t m = count_lines(prefix + ".bim");
    std::ifstream bed(prefix + ".bed", std::ios::binary);
    if (!bed) fail(CS_ERR_IO, "Could not open file for mmap: " + prefix + ".bed");
    bed.seekg(0, std::ios::end);
    const std::streamoff size = bed.tellg();
    bed.seekg(0);
    std::vector<uint8_t> bytes(static_cast<size_t>(size));
    if (size > 0) bed.read(reinterpret_cast<char*>(bytes.data()), size);
    return genotypes_from_bed(bytes.data(), bytes.size(), n, m);
}

}  // namespace cs
