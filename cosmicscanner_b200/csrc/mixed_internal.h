// What the tensor-core passes over the packed genotypes share (kinship_mixed.cu and
// kinship_slices.cu): the per-row tables of a packed view, its sample-major copy, tensor maps.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include "cs_internal.h"

namespace cs {

constexpr int kTcTile = 128;  // MMA M, and SNP rows / samples per decoded tile
constexpr int kTcQ = 63;      // dosage scale of the imputed-code tile

// A packed view with its per-row tables.
struct MixedRows {
    int64_t R = 0, n = 0, r_pad = 0, n_pad = 0;
    DeviceBuffer<double> mu, exc, s, resid;
    DeviceBuffer<uint32_t> lut;  // imputed code of each 2-bit code, one byte per code
    // q_t (byte 1 of lut[t]) at K position (t & ~15) + position_of(t & 15): the samples pass
    // over the sample-major copy reads the imputed codes of 16 SNPs per uint4
    DeviceBuffer<uint4> qperm;
    CUtensorMap tm{};
    const uint8_t* rows = nullptr;  // the view's packed rows (owned by the operator)
    int64_t stride = 0;
    // sample-major copy for the samples passes with A in TMEM (made on first use)
    DeviceBuffer<uint8_t> packed_t;
    CUtensorMap tm_t{};
};

// The sample-major copy of the view (once per context): n_pad rows of r_pad / 4 bytes.
void ensure_transposed(MixedRows& r, cudaStream_t s);
// The operator's tables (made on first use).
MixedRows& mixed_rows_for(cs_kinship* op);

// The mixed passes of at most 48 columns on the kernel of the FP64 form (kinship_slices.cu), which
// decodes four K-blocks at a time: kp columns (a multiple of 8) in one tile, operands and partial sums
// as the passes here lay them out, the six-set form in the samples pass.
bool mixed_narrow_fits(bool rows, int64_t kp);
void mixed_narrow_pass(bool rows, MixedRows& r, const int8_t* b, int64_t kp, int splits, int kbs,
                       const double* inv_f, double* part, int* status, uint32_t poll_ns, cudaStream_t s);

// T = Z_c^T X (rows of r, k columns) in the FP64 form on the int8 digits, with the state's buffers (made
// on first use); false, and nothing done, without device memory for them.
bool scan_project_slices(SliceOperator*& state, MixedRows& r, StridedIn X, int64_t k, StridedOut T,
                         cudaStream_t s);

// 2D uint8 tensor map: inner extent `inner` bytes, `outer` rows of `row_bytes`.
CUtensorMap make_map_u8(const void* base, uint64_t inner, uint64_t outer, uint64_t row_bytes,
                        uint32_t box_inner, uint32_t box_outer, bool swizzle);

// 16 codes (one 32-bit word, code j in bits 2j..2j+1) -> 16 int8 imputed codes (byte c of
// the row's table `lut` for code c) and 16 missing indicators in the interleaved sample order
// 0 2 4 .. 14 1 3 .. 15 within the group: the even codes, masked in place, are already
// byte-permute selectors (one nibble each), and so are the odd codes after one shift.
// sample_at(p) / position_of(s) convert.
__device__ __forceinline__ void decode_word_interleaved(uint32_t w, uint32_t lut, uint4& dos, uint4& mis) {
    const uint32_t se = w & 0x33333333u, so = (w >> 2) & 0x33333333u;
    dos.x = __byte_perm(lut, 0u, se);
    dos.y = __byte_perm(lut, 0u, se >> 16);
    dos.z = __byte_perm(lut, 0u, so);
    dos.w = __byte_perm(lut, 0u, so >> 16);
    mis.x = __byte_perm(0x00000100u, 0u, se);
    mis.y = __byte_perm(0x00000100u, 0u, se >> 16);
    mis.z = __byte_perm(0x00000100u, 0u, so);
    mis.w = __byte_perm(0x00000100u, 0u, so >> 16);
}
// position p (0..15) of the interleaved order -> sample offset in the group, and back
__host__ __device__ __forceinline__ int sample_at(int p) { return p < 8 ? 2 * p : 2 * (p - 8) + 1; }
__host__ __device__ __forceinline__ int position_of(int s) { return (s & 1) ? 8 + (s >> 1) : s >> 1; }

}  // namespace cs
