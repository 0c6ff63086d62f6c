// The FP64 kinship products on the int8 tensor cores (kinship_slices.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "cs_internal.h"

namespace cs {

// Range of a column's values: the bits of max |x| (NaN and infinity compare above every finite
// value) and the exponents of the nonzero |x|, summed and counted.  All integers, so the
// atomics that gather them are order independent.
struct ColumnRange {
    unsigned long long max_bits;
    long long exp_sum;
    unsigned long long count;
    unsigned long long pad;
};

// A fixed-point column holds every element to 2^-63 of its maximum.  A column whose nonzero elements
// lie on (geometric) average more than 2^kSliceRange below that maximum is summed in FP64 (direct_rows):
// up to there the average element has the 53 bits of an FP64 value, so that also what depends on the
// small elements alone (a row whose large ones all meet missing calls) is as good as FP64 sums.  So is
// a column with a non-finite value or a maximum near the ends of the exponent range (the scales and
// the scaled results stay normal numbers).  A normal sample of 50,000 lies 2^3 below its maximum;
// W = s^2 o Z^T X 2^4 more with minor allele frequencies down to 0.01, and 2^7 with 1 % of the variants at
// allele counts of 1 to 20 among 200,000 samples.
constexpr int kSliceRange = 10;
// An even column, whose elements lie on average at most 2^kSliceEven below its maximum, is held in 55 bits: K x of
// normal columns is then off by 1.3e-16 with W 2^4.3 below its maximum (6,000 x 3,000, minor allele
// frequencies from 0.01), and the error doubles with each binade: 6.4e-16 between 2^5 and 2^6 below (9,001 x
// 1,300, 2 % of the variants at counts of 1 to 20), 0.8e-15 to 1.5e-15 at 2^7.5 (singletons), where FP64 sums are
// off by 1.1e-15.
constexpr int kSliceEven = 5;
constexpr int kSliceMaxExp = 940;

__device__ __forceinline__ bool range_excluded(const ColumnRange& r) {
    const int ex = (int)(r.max_bits >> 52) - 1023;
    if (ex > kSliceMaxExp) return true;                       // NaN, infinity, huge
    if (r.count == 0) return false;                           // all zero
    if (ex < -kSliceMaxExp) return true;
    return (long long)ex * (long long)r.count - r.exp_sum > (long long)kSliceRange * (long long)r.count;
}

__device__ __forceinline__ bool range_uneven(const ColumnRange& r) {
    const int ex = (int)(r.max_bits >> 52) - 1023;
    return (long long)ex * (long long)r.count - r.exp_sum > (long long)kSliceEven * (long long)r.count &&
           !range_excluded(r);
}

struct SliceOperator;
void destroy_slices(SliceOperator* s);

// FP64 products through the slices where the operator has (or may have) a sample-major copy and there
// is device memory for it and the operands; false when the FP64-pipe kernels are to be used.  Results may
// overwrite the input.
// Y (rows x k) = K X.
bool kinship_apply_slices(cs_kinship* op, StridedIn X, int64_t k, StridedOut Y, cudaStream_t s);
// U (selected variants x k; rows of inactive variants are left alone) = Z^T X.
bool multiply_zt_slices(cs_kinship* op, StridedIn X, int64_t k, StridedOut U, cudaStream_t s);
// Y (rows x k) = Z V, V (selected variants x k).
bool multiply_z_slices(cs_kinship* op, StridedIn V, int64_t k, StridedOut Y, cudaStream_t s);

}  // namespace cs
