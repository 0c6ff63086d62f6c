// Tensor-core (mixed-precision) form of the kinship operator Y = Z Z^T X / M.
//
// Arithmetic.  Both passes run on tcgen05.mma kind::i8 with exact int32 accumulation:
//  * the genotype tile enters as int8 imputed codes e = Q G in {0, Q, 2Q} (Q = 63) for
//    observed calls and e = q_t = rint(Q mu_t) for missing ones, so that e / Q is the
//    mean-imputed dosage up to the row's residual r_t = mu_t - q_t / Q (|r_t| <= 1 / 2Q),
//    together with an int8 missing-indicator tile, both decoded from the packed 2-bit rows in
//    shared memory (a 128-SNP x 128-sample tile, 128-byte swizzled) through a per-row
//    byte-permute table;
//  * right-hand sides are quantised per column into three int8 pieces (base 254) after
//    centring: x' = (x - mean) * 127 / max|x - mean| ~ q1 + q2/254 + q3/254^2, i.e. about
//    23 significant bits, so the only rounding is this quantisation (~6e-8 of the column
//    maximum per element); products and sums are exact while a K slice holds at most
//    kMaxKbPerAccum K-blocks (|e q| <= 126 * 127 per element, plus 127 for the residual).
// With G_ti + mu_t miss_ti = e_ti / Q + r_t miss_ti, the residual term carries the factor
// |r_t| <= 1/126, so two pieces of its operand match the precision of the main term's three:
// per missing call the residual's rounding is at most 1.6e-5 (rows pass) / 3.1e-5 (samples
// pass) of a first-piece step, against up to 1.55e-5 per element for the main term's own.
// Five operand sets per K-block instead of the six of a separate dosage and missing-call
// product.
// Rows pass (U = Z^T X): with S_t, n_t the exact allele sum and observed count of row t,
//   u_t / s_t = mean * (S_t - mu_t n_t) + ( sum_i e_ti x'_i / Q + r_t sum_{i missing} x'_i
//               - mu_t sum_i x'_i ) / scale
// (the centring identity of src/kinship_operator.cpp:135 with the missing-call terms split
// out).  Samples pass (Y = Z W / M, W = s o U):
//   y_i = ( sum_t e_ti w_t / Q + sum_t miss_ti r_t w_t - sum_t mu_t w_t ) / M
// with W f and (Q r o W) f quantised with one factor f = 127 / max|w| (|Q r_t| <= 1/2 keeps
// the second operand's first piece within 64), three pieces of the first and two of the
// second accumulating into the same TMEM columns.  Each pass is one MMA of the imputed-code
// tile against three pieces (N = 3 kc) plus one of the missing-indicator tile against two
// (N = 2 kc): the first two pieces of the same operand in the rows pass (own accumulator,
// scaled by r_t in the epilogue), the residual pieces in the samples pass.
//
// Kernel structure (one CTA per SM, 15 warps): warp 14 issues TMA loads of the packed
// tiles (from HBM) into a deep ring of their own, warp 0 those of the quantised pieces (L2
// resident) into a ring of stages; warps 2-9 decode (with A in TMEM as two groups of four
// that take alternate K-blocks); warp 1 issues the MMAs from one thread
// into a TMEM accumulator; warps 10-13 drain it (tcgen05.ld) and write FP64 slice partials.
// The decoded tile (SNP rows x samples) serves as a K-major A operand in the rows pass and
// as an MN-major A operand in the samples pass.  The TMEMA layouts decode into tensor memory
// instead (tcgen05.st) and the MMAs read A from there; the samples pass then reads a
// sample-major copy of the packed matrix, where A is K-major too, either with the fixed
// dosage table and W / mu o W in six operand sets, or (TMEMA = 5) with each SNP's imputed
// code put in along K under a per-byte missing-call mask (the five sets, and the int32 sums,
// of the shared-memory form).  Wide blocks run on CTA pairs
// (cta_group::2): the partner CTA's MMA warp forwards each of its landed B stages to the
// leader.  Every wait is bounded; a timeout leaves a status code that the host reports as an
// error.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "chain.cuh"
#include "cs_internal.h"
#include "mixed_internal.h"
#include "sm100.cuh"

namespace cs {

namespace {

using namespace sm100;

constexpr int kTile = kTcTile;
constexpr int kKBlock = 128;      // K elements (int8) per stage: one 128-byte swizzle row
constexpr int kMaxKc = 80;        // column-tile width cap (MMA N = 3 kc <= 256)
constexpr int kWarps = 15;
constexpr int kThreads = kWarps * 32;
constexpr int kDecodeWarp0 = 2, kDecodeWarps = 8;
constexpr int kEpiWarp0 = 10;
constexpr int kPackedWarp = 14;
constexpr uint32_t kTmemCols = 512;
constexpr double kBase = 254.0;
constexpr int kImputeQ = kTcQ;
constexpr int kMaxKbPerAccum = 1024;  // K-blocks one int32 accumulation may hold:
                                      // 1024 * 128 * (126 * 127 + 127) < 2^31

constexpr int kATileBytes = kTile * kKBlock;     // 16 KB
constexpr int kPackedBytes = kTile * 32;         // 128 rows x 32 B

// Shared memory: a ring of decoded tiles {imputed codes, missing indicators}, a deep ring of
// packed tiles (HBM latency is the longest, so they are requested furthest ahead) and a ring
// of B stages (the quantised pieces, re-read by every CTA from L2).  The rows pass has 3 B
// pieces and accumulators of 3 kc + 2 kc TMEM columns (main and missing-call sums kept
// apart); the samples pass has 5 B pieces (W and Q r o W with one scale) and one accumulator
// of 3 kc columns, double-buffered.
//
// CTA pairs (cta_group::2): a cluster of two CTAs shares each MMA, M = 256 rows (128 from
// each CTA's decoded tile) by N = 3 kc, and each CTA holds only half of the B pieces (rows
// [1.5 kc r, 1.5 kc (r + 1)) of the 3 kc-row set, r = CTA rank).  The tensor core then
// reads half the B bytes per MAC from each SM's shared memory, which is what bounds the
// single-CTA MMAs (about 68 bytes of operands per clock per SM); the smaller B stages leave
// room for wider column tiles and a deeper decode ring, which covers the extra hop of the
// cross-CTA handshakes.
// Narrow single-CTA layouts (column tiles of at most 32): the small B stages leave room for
// a decode ring twice as deep and, in the rows pass, a second accumulator, for widths where the
// MMAs are short and the per-K-block handshakes set the pace.
// Pipeline depths {column-tile width cap, B stages, packed stages, decode stages}:
constexpr int kRowsW = 80, kRowsST = 4, kRowsSP = 8, kRowsSD = 2;
constexpr int kSamplesW = 48, kSamplesST = 3, kSamplesSP = 12, kSamplesSD = 2;
constexpr int kPairRowsW = 80, kPairRowsST = 4, kPairRowsSP = 8, kPairRowsSD = 4;
constexpr int kPairSamplesW = 80, kPairSamplesST = 3, kPairSamplesSP = 6, kPairSamplesSD = 3;
constexpr int kNarrowRowsW = 32, kNarrowRowsST = 4, kNarrowRowsSP = 8, kNarrowRowsSD = 4;
static_assert(kNarrowRowsW == 32, "the plans use one narrow width for both passes");
constexpr int kNarrowSamplesW = 32, kNarrowSamplesST = 3, kNarrowSamplesSP = 8, kNarrowSamplesSD = 4;
// Narrow passes with their A operand in tensor memory (TMEMA): the decoders store the two
// genotype tiles into TMEM (tcgen05.st) and the MMAs read them there, so shared memory
// carries only the packed tiles and the B pieces.  A TMEM operand must be K-major, so the
// samples pass then reads a sample-major copy of the packed matrix (rows = samples, four
// SNPs per byte).  Along its K the SNPs change every two bits, so one byte-permute table
// cannot carry the per-SNP imputed codes: these passes decode with the fixed dosage table and
// carry the missing calls with W and mu o W, three pieces each (the six-set form), except
// TMEMA = 5 below.  TMEMA = 1: column tiles of at most 32, two
// accumulators (5 x 32 columns rows, 3 x 32 samples); TMEMA = 2: tiles of at most 64, one
// accumulator (5 x 64 / 3 x 64), for 33 to 64 right-hand sides.  Then A stages of 64 TMEM
// columns (32 per tile: 128 int8 K elements per lane).
constexpr int kTmemARowsST = 8, kTmemARowsSP = 16, kTmemARowsSD = 3;
constexpr int kTmemASamplesST = 4, kTmemASamplesSP = 16, kTmemASamplesSD = 4;
constexpr int kTmemA64W = 64;
constexpr int kTmemA64RowsST = 6, kTmemA64RowsSP = 12, kTmemA64RowsSD = 3;
constexpr int kTmemA64SamplesST = 3, kTmemA64SamplesSP = 12, kTmemA64SamplesSD = 4;
// TMEMA = 3: the rows pass on CTA pairs with A in TMEM, column tiles of at most 64 (each CTA
// holds half of the B pieces, as in the shared-memory pair form).
constexpr int kTmemAPairRowsST = 8, kTmemAPairRowsSP = 16, kTmemAPairRowsSD = 3;
// TMEMA = 4: the samples pass on CTA pairs over the sample-major copy (six operand sets, each
// CTA holding half of each set).  TMEMA = 5: the same in the five-set form: the decoder
// permutes with the observed-call table (missing -> 0) and a missing-call mask table and ORs
// in q_t from a per-SNP byte array in the decoded K order (a third operation per four codes,
// and the K-block's 128 codes staged with each packed tile); B as in the shared-memory pair
// form.
constexpr int kTmemAPairSamplesST = 4, kTmemAPairSamplesSP = 16, kTmemAPairSamplesSD = 4;
constexpr uint32_t kTmemAStage = 64;

template <bool ROWS, bool PAIR, bool NARROW = false, int TMEMA = 0>
struct Layout {
    static_assert(!(PAIR && NARROW), "narrow layouts are single-CTA");
    static_assert(!TMEMA || (TMEMA == 3 ? (ROWS && PAIR && !NARROW)
                             : TMEMA >= 4 ? (!ROWS && PAIR && !NARROW) : (NARROW && !PAIR)),
                  "A in TMEM: the narrow single-CTA passes, or the passes on CTA pairs");
    // samples passes over the sample-major copy with the fixed dosage table: W and mu o W
    static constexpr bool kSixSets = !ROWS && (TMEMA == 1 || TMEMA == 2 || TMEMA == 4);
    static constexpr int kPieces = ROWS ? 3 : (kSixSets ? 6 : 5);  // per column tile, over the pair
    static constexpr int kMaxW = TMEMA >= 2 ? kTmemA64W
                                 : NARROW ? (ROWS ? kNarrowRowsW : kNarrowSamplesW)
                                 : PAIR ? (ROWS ? kPairRowsW : kPairSamplesW) : (ROWS ? kRowsW : kSamplesW);
    static constexpr int kTmaStages = TMEMA >= 4 ? kTmemAPairSamplesST
                                      : TMEMA == 3 ? kTmemAPairRowsST
                                      : TMEMA == 2 ? (ROWS ? kTmemA64RowsST : kTmemA64SamplesST)
                                      : TMEMA ? (ROWS ? kTmemARowsST : kTmemASamplesST)
                                      : NARROW ? (ROWS ? kNarrowRowsST : kNarrowSamplesST)
                                      : PAIR ? (ROWS ? kPairRowsST : kPairSamplesST) : (ROWS ? kRowsST : kSamplesST);
    static constexpr int kPackedStages = TMEMA >= 4 ? kTmemAPairSamplesSP
                                         : TMEMA == 3 ? kTmemAPairRowsSP
                                         : TMEMA == 2 ? (ROWS ? kTmemA64RowsSP : kTmemA64SamplesSP)
                                         : TMEMA ? (ROWS ? kTmemARowsSP : kTmemASamplesSP)
                                         : NARROW ? (ROWS ? kNarrowRowsSP : kNarrowSamplesSP)
                                         : PAIR ? (ROWS ? kPairRowsSP : kPairSamplesSP) : (ROWS ? kRowsSP : kSamplesSP);
    static constexpr int kDecodeStages = TMEMA >= 4 ? kTmemAPairSamplesSD
                                         : TMEMA == 3 ? kTmemAPairRowsSD
                                         : TMEMA == 2 ? (ROWS ? kTmemA64RowsSD : kTmemA64SamplesSD)
                                         : TMEMA ? (ROWS ? kTmemARowsSD : kTmemASamplesSD)
                                         : NARROW ? (ROWS ? kNarrowRowsSD : kNarrowSamplesSD)
                                         : PAIR ? (ROWS ? kPairRowsSD : kPairSamplesSD) : (ROWS ? kRowsSD : kSamplesSD);
    static constexpr int kAccCols = ROWS ? 5 * kMaxW : 3 * kMaxW;
    static constexpr int kAccBufs = ((ROWS && !NARROW) || TMEMA >= 2) ? 1 : 2;
    static constexpr uint32_t kAccStride = TMEMA ? (uint32_t)kAccCols : 256;
    // TMEM columns of decode stage d's imputed-code / missing-indicator tiles (TMEMA)
    static constexpr uint32_t kTmemA0 = kAccBufs * kAccStride;
    static __host__ __device__ constexpr uint32_t ta(int d) { return kTmemA0 + d * kTmemAStage; }
    static __host__ __device__ constexpr uint32_t tam(int d) { return ta(d) + kTmemAStage / 2; }
    static constexpr int kBBytes = kPieces * kMaxW * 128 / (PAIR ? 2 : 1);  // this CTA's share
    static constexpr int kTmaBytes = kBBytes;
    static constexpr int kDecBytes = 2 * kATileBytes;
    static constexpr int kDecodeRegion = TMEMA ? 0 : kDecodeStages * kDecBytes;
    // samples pass over the sample-major copy: the K-block's 128 imputed codes (P.qperm) ride
    // in each packed stage, so the decoders read them from shared memory
    static constexpr int kQBytes = TMEMA == 5 ? kKBlock : 0;
    // barriers: full / empty per B, packed and decode stage, full / empty per accumulator,
    // `drained`, then the TMEM slot
    static constexpr int kBarBytes =
        (2 * (kTmaStages + kPackedStages + kDecodeStages + kAccBufs) + 1) * 8 + 8;
    static constexpr int kSmem = kDecodeRegion + kTmaStages * kTmaBytes +
                                 kPackedStages * (kPackedBytes + kQBytes) + 1024 + kBarBytes;
    static __host__ __device__ constexpr int a(int d) { return d * kDecBytes; }
    static __host__ __device__ constexpr int am(int d) { return d * kDecBytes + kATileBytes; }
    static __host__ __device__ constexpr int b(int s) { return kDecodeRegion + s * kTmaBytes; }
    static __host__ __device__ constexpr int p(int s) {
        return kDecodeRegion + kTmaStages * kTmaBytes + s * kPackedBytes;
    }
    static __host__ __device__ constexpr int q(int s) {
        return kDecodeRegion + kTmaStages * kTmaBytes + kPackedStages * kPackedBytes + s * kQBytes;
    }
    static __host__ __device__ constexpr int bars() {
        return kDecodeRegion + kTmaStages * kTmaBytes + kPackedStages * (kPackedBytes + kQBytes);
    }
    static_assert(kSmem <= 227 * 1024, "mixed pass exceeds shared memory");
    static_assert(kTmaBytes % 1024 == 0, "TMA stages must keep 1024-byte alignment");
    static_assert(kAccBufs == 1 ? kAccCols <= (int)kTmemCols : kAccCols <= (int)kAccStride,
                  "accumulators exceed TMEM");
    static_assert(!TMEMA || ta(kDecodeStages) <= kTmemCols, "A stages exceed TMEM");
    static_assert(kMaxW % 16 == 0 && kMaxW <= kMaxKc, "column tiles are multiples of 16, at most 80");
};

struct PassArgs {
    int n_tiles, n_ctiles, n_splits;
    int kb_total, kb_per_split;  // K-blocks of the contraction, per slice
    int kc, kp;                  // column tile width, padded column count
    int kc_last;                 // width of the last column tile (a multiple of 16, <= kc)
    const uint32_t* lut;         // per SNP row: imputed code of each 2-bit code (byte-permute table)
    const uint4* qperm;          // samples pass over the sample-major copy: q_t of each SNP at
                                 // its position in the decoded K order, 16 SNPs per uint4
    const double* resid;         // rows pass: r_t = mu_t - q_t / Q per SNP row (epilogue)
    const double* inv_f;         // samples pass: 1 / (Q f) per column
    double* part;                // [n_splits][kp][ld] FP64 slice partials
    int64_t ld;                  // padded output rows
    int* status;
    uint32_t poll_ns;            // pairs: pause between polls of the long, off-critical-path waits
    uint32_t poll_dec_ns;        // pairs: pause between the decoders' polls for a free stage
};

// decode_word_interleaved for 16 codes of 16 different SNPs (a word of the sample-major copy): the observed
// calls through the fixed table 2Q / 0 / Q / 0, a 0xFF byte per missing call, and the SNPs'
// imputed codes q (four per word, in the interleaved order) put in under that mask.  The mask
// itself is the missing-indicator tile, as int8 -1: the samples operand of this form carries
// the residual pieces negated, so the products are those of the +1 tile.
constexpr uint32_t kObservedCodes = (uint32_t)(2 * kImputeQ) | ((uint32_t)kImputeQ << 16);
__device__ __forceinline__ void decode_word_imputed(uint32_t w, const uint4& q, uint4& dos, uint4& mis) {
    const uint32_t se = w & 0x33333333u, so = (w >> 2) & 0x33333333u;
    mis.x = __byte_perm(0x0000FF00u, 0u, se);
    mis.y = __byte_perm(0x0000FF00u, 0u, se >> 16);
    mis.z = __byte_perm(0x0000FF00u, 0u, so);
    mis.w = __byte_perm(0x0000FF00u, 0u, so >> 16);
    dos.x = __byte_perm(kObservedCodes, 0u, se) | (mis.x & q.x);
    dos.y = __byte_perm(kObservedCodes, 0u, se >> 16) | (mis.y & q.y);
    dos.z = __byte_perm(kObservedCodes, 0u, so) | (mis.z & q.z);
    dos.w = __byte_perm(kObservedCodes, 0u, so >> 16) | (mis.w & q.w);
}
// ALT (A in TMEM): the decoder warps in two groups that take alternate K-blocks whole.  Known at
// compile time: as an argument it cost the rows pass of 96 columns at 31,001 x 52,003 4 % (517 us for 495).
template <bool ROWS, bool PAIR, bool NARROW, int TMEMA, bool ALT>
__global__ void __launch_bounds__(kThreads, 1)
k_mixed_pass(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
             const __grid_constant__ CUtensorMap tm_bt, PassArgs P) {
    using L = Layout<ROWS, PAIR, NARROW, TMEMA>;
    // K-major A tiles decoded from rows of K elements: the rows pass, and the samples pass over
    // the sample-major copy
    constexpr bool KMAJOR = ROWS || TMEMA != 0;
    constexpr int ST = L::kTmaStages, SP = L::kPackedStages, SD = L::kDecodeStages, NB = L::kAccBufs;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::bars());
    uint64_t* full_t = bars;              // B stage landed (1 arrival + tx bytes)
    uint64_t* empty_t = full_t + ST;      // MMAs reading the B stage done (commit)
    uint64_t* full_p = empty_t + ST;      // packed tile landed (1 arrival + tx bytes)
    uint64_t* empty_p = full_p + SP;      // packed tile decoded (one arrival per decode warp)
    uint64_t* full_d = empty_p + SP;      // decoded (one arrival per decode warp; pair: the
                                          // leader's counts both CTAs' warps and the other
                                          // CTA's B-stage-landed arrival)
    uint64_t* empty_d = full_d + SD;      // MMAs reading the decoded tile done (commit)
    uint64_t* acc_full = empty_d + SD;    // accumulator ready for the epilogue (commit)
    uint64_t* acc_empty = acc_full + NB;  // accumulator drained (one arrival per epilogue warp)
    uint64_t* drained = acc_empty + NB;   // MMA thread's own work complete at exit
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kc = P.kc, kp = P.kp;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
    // TMEMA: the decoder warps either share every K-block (each its lane quarter and one half of
    // K) or split into two groups of four that take alternate K-blocks whole, so that two
    // K-blocks are in decode at once
    constexpr bool alt = TMEMA != 0 && ALT;
    const uint32_t dec_arrivals = alt ? 4u : (uint32_t)kDecodeWarps;
    if (threadIdx.x == 0) {
        for (int s = 0; s < ST; ++s) {
            mbar_init(&full_t[s], 1);
            mbar_init(&empty_t[s], 1);
        }
        for (int s = 0; s < SP; ++s) {
            mbar_init(&full_p[s], 1);
            mbar_init(&empty_p[s], dec_arrivals);
        }
        for (int d = 0; d < SD; ++d) {
            mbar_init(&full_d[d], PAIR ? 2 * dec_arrivals + 1 : dec_arrivals);
            mbar_init(&empty_d[d], 1);
        }
        for (int b = 0; b < NB; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], PAIR ? 8 : 4);
        }
        mbar_init(drained, 1);
        fence_mbar_init();
    }
    if (warp == 1) {
        if (PAIR)
            tmem_alloc_pair(tmem_slot, kTmemCols);
        else
            tmem_alloc(tmem_slot, kTmemCols);
    }
    chain_wait();
    tc_fence_before();
    if (PAIR)
        cluster_sync_all();
    else
        __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // A unit is one M tile (pair: two, one per CTA) x one column tile x one K slice; both
    // CTAs of a pair walk the same units.  The column tile varies fastest, so the CTAs that
    // run at the same time share each packed tile through L2 instead of re-reading the packed
    // matrix from HBM once per column tile.
    const int groups = PAIR ? P.n_tiles / 2 : P.n_tiles;
    const int units = groups * P.n_ctiles * P.n_splits;
    const int u0 = PAIR ? (int)cluster_id_x() : (int)blockIdx.x;
    const int ustep = PAIR ? (int)cluster_count_x() : (int)gridDim.x;
    auto unit_coords = [&](int u, int& tile, int& ct, int& split, int& kb0, int& kb1) {
        ct = u % P.n_ctiles;
        const int rest = u / P.n_ctiles;
        const int g = rest % groups;
        tile = PAIR ? 2 * g + (int)rank : g;
        split = rest / groups;
        kb0 = split * P.kb_per_split;
        kb1 = min(P.kb_total, kb0 + P.kb_per_split);
    };
    // columns [ct kc, ct kc + w) of the padded kp; only the last tile may be narrower
    auto width = [&](int ct) { return ct == P.n_ctiles - 1 ? P.kc_last : kc; };
    // Waits on barriers that the MMA commits arrive on (pair: multicast from the leader) or
    // that the other CTA arrives on: pairs poll without suspending (see mbar_poll); the
    // cluster form also acquires what the other CTA released.
    auto wait_commit = [&](uint64_t* bar, uint32_t parity, int code) {
        return PAIR ? mbar_poll(bar, parity, P.status, code) : mbar_wait(bar, parity, P.status, code);
    };
    auto wait_peer = [&](uint64_t* bar, uint32_t parity, int code) {
        return PAIR ? mbar_poll_cluster(bar, parity, P.status, code)
                    : mbar_wait(bar, parity, P.status, code);
    };
    // commit barriers that a warp waits on long and off the critical path (the epilogue's
    // accumulator, the B producer's free stage, the partner CTA's forwarding)
    auto wait_idle = [&](uint64_t* bar, uint32_t parity, int code) {
        return PAIR ? mbar_poll_sleep(bar, parity, P.status, code, P.poll_ns)
                    : mbar_wait(bar, parity, P.status, code);
    };

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (B)
        if (elect_one()) {
            prefetch_tensormap(&tm_b);
            prefetch_tensormap(&tm_bt);
            uint32_t j = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                const int w = width(ct);
                // the narrower last tile has its own map (box of kc_last rows, pair: half)
                const CUtensorMap* mb = ct == P.n_ctiles - 1 ? &tm_bt : &tm_b;
                const uint32_t bytes = (uint32_t)(L::kPieces * w * 128 / (PAIR ? 2 : 1));
                for (int kb = kb0; kb < kb1; ++kb, ++j) {
                    const int s = j % ST;
                    if (!(ok = wait_idle(&empty_t[s], ((j / ST) & 1) ^ 1, kTimeoutTma))) break;
                    mbar_arrive_expect_tx(&full_t[s], bytes);
                    if (PAIR) {
                        const int hw = w / 2;  // rows of one half-piece
                        if (ROWS) {
                            // half r of each piece, [p0(r) p1(r) p2(r)]: the missing-call MMA
                            // (N = 2 w) then finds [p0(r) p1(r)] at the start of each CTA's stage
#pragma unroll
                            for (int c = 0; c < 3; ++c)
                                tma_load_2d(smem + L::b(s) + c * hw * 128, mb, kb * kKBlock,
                                            c * kp + ct * kc + (int)rank * hw, &full_t[s]);
                        } else {
                            // main set: half-pieces [p0a p0b p1a p1b p2a p2b], this CTA loads
                            // 3 r .. 3 r + 2; residual set: piece 3 + r whole (six sets: the
                            // mu o W set split like the main one)
#pragma unroll
                            for (int c = 0; c < 3; ++c) {
                                const int h = 3 * (int)rank + c, q = h >> 1;
                                tma_load_2d(smem + L::b(s) + c * hw * 128, mb, kb * kKBlock,
                                            q * kp + ct * kc + (h & 1) * hw, &full_t[s]);
                            }
                            if constexpr (L::kSixSets) {
#pragma unroll
                                for (int c = 0; c < 3; ++c) {
                                    const int h = 3 * (int)rank + c, q = h >> 1;
                                    tma_load_2d(smem + L::b(s) + (3 + c) * hw * 128, mb, kb * kKBlock,
                                                (3 + q) * kp + ct * kc + (h & 1) * hw, &full_t[s]);
                                }
                            } else {
#pragma unroll
                                for (int c = 0; c < 2; ++c)
                                    tma_load_2d(smem + L::b(s) + (3 + c) * hw * 128, mb, kb * kKBlock,
                                                (3 + (int)rank) * kp + ct * kc + c * hw, &full_t[s]);
                            }
                        }
                    } else {
                        for (int q = 0; q < L::kPieces; ++q)
                            tma_load_2d(smem + L::b(s) + q * w * 128, mb, kb * kKBlock,
                                        q * kp + ct * kc, &full_t[s]);
                    }
                }
            }
            // leave no copy in flight
            for (uint32_t q = (j >= (uint32_t)ST ? j - ST : 0); q < j; ++q)
                mbar_wait(&full_t[q % ST], (q / ST) & 1, P.status, kTimeoutTma, 1u << 20);
            chain_next();
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (pair: leader)
        if ((!PAIR || rank == 0) && elect_one()) {
            // s8 x s8 -> s32; rows pass: K-major A (SNP rows x samples); samples pass:
            // MN-major A (the same tile read as samples x SNPs); N = 3 w (the three pieces
            // of a column tile side by side) for the imputed codes and 2 w for the missing
            // indicators, M = 128 (pair: 256)
            const uint32_t idesc0 = (2u << 4) | (1u << 7) | (1u << 10) | ((KMAJOR ? 0u : 1u) << 15) |
                                    ((uint32_t)((PAIR ? 2 : 1) * kTile >> 4) << 24);
            uint32_t j = 0;
            int ui = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep, ++ui) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                const int w = width(ct);
                const uint32_t idesc = idesc0 | ((uint32_t)((3 * w) >> 3) << 17);
                // the missing-indicator MMA: two pieces, or the three of mu o W (six sets)
                const uint32_t idesc_m = idesc0 | ((uint32_t)(((L::kSixSets ? 3 : 2) * w) >> 3) << 17);
                const int buf = ui % NB;
                if (!(ok = wait_peer(&acc_empty[buf], ((ui / NB) & 1) ^ 1, kTimeoutMma))) break;
                tc_fence_after();
                const uint32_t acc_main = tmem_base + buf * L::kAccStride;
                const uint32_t acc_miss = ROWS ? acc_main + 3 * w : acc_main;
                for (int kb = kb0; kb < kb1; ++kb, ++j) {
                    const int s = j % ST, d = j % SD;
                    if (!(ok = mbar_wait(&full_t[s], (j / ST) & 1, P.status, kTimeoutMma))) break;
                    if (!(ok = wait_peer(&full_d[d], (j / SD) & 1, kTimeoutMma))) break;
                    tc_fence_after();
                    const uint32_t a = smem_addr(smem + L::a(d));
                    const uint32_t am = smem_addr(smem + L::am(d));
                    const uint32_t b = smem_addr(smem + L::b(s));
                    // rows pass: the first two pieces (this CTA's halves of them); samples
                    // pass: the residual set after the W set (this CTA's share)
                    const uint32_t bm = ROWS ? b : b + 3 * w * 128 / (PAIR ? 2 : 1);
#pragma unroll
                    for (int ks = 0; ks < kKBlock / 32; ++ks) {
                        const uint32_t first = (kb == kb0 && ks == 0) ? 0u : 1u;
                        const uint64_t db = smem_desc_sw128(b + ks * 32, 16, 1024);
                        const uint64_t dbm = smem_desc_sw128(bm + ks * 32, 16, 1024);
                        if constexpr (TMEMA != 0) {
                            // A from TMEM: 32 K elements = 8 columns per MMA
                            if constexpr (PAIR) {
                                mma_i8_pair_tmem_a(acc_main, tmem_base + L::ta(d) + ks * 8, db, idesc, first);
                                mma_i8_pair_tmem_a(acc_miss, tmem_base + L::tam(d) + ks * 8, dbm, idesc_m,
                                                   ROWS ? first : 1u);
                            } else {
                                mma_i8_tmem_a(acc_main, tmem_base + L::ta(d) + ks * 8, db, idesc, first);
                                mma_i8_tmem_a(acc_miss, tmem_base + L::tam(d) + ks * 8, dbm, idesc_m,
                                              ROWS ? first : 1u);
                            }
                            continue;
                        }
                        const uint32_t aoff = ROWS ? ks * 32 : ks * 4096;  // 32 K elements
                        const uint64_t da = smem_desc_sw128(a + aoff, 16, 1024);
                        const uint64_t dm = smem_desc_sw128(am + aoff, 16, 1024);
                        // rows pass: separate missing-call sums; samples pass: the first two
                        // piece columns of the same accumulator
                        if (PAIR) {
                            mma_i8_pair(acc_main, da, db, idesc, first);
                            mma_i8_pair(acc_miss, dm, dbm, idesc_m, ROWS ? first : 1u);
                        } else {
                            mma_i8(acc_main, da, db, idesc, first);
                            mma_i8(acc_miss, dm, dbm, idesc_m, ROWS ? first : 1u);
                        }
                    }
                    if (PAIR) {
                        mma_commit_pair(&empty_t[s], 3);
                        mma_commit_pair(&empty_d[d], 3);
                    } else {
                        mma_commit(&empty_t[s]);
                        mma_commit(&empty_d[d]);
                    }
                }
                if (ok) {
                    if (PAIR)
                        mma_commit_pair(&acc_full[buf], 3);
                    else
                        mma_commit(&acc_full[buf]);
                }
            }
            if (PAIR)
                mma_commit_pair(drained, 1);
            else
                mma_commit(drained);
            mbar_wait(drained, 0, P.status, kTimeoutMma, 1u << 20);
        } else if (PAIR && rank == 1 && elect_one()) {
            // The leader's MMA also reads this CTA's half of each B stage: once the stage has
            // landed here, tell the leader (one arrival on its full_d, after the decoders'),
            // so that no decoder waits for the B copy of the K-block it has just decoded.
            // Like a decoder, wait until the decode stage is free so that the arrival counts
            // toward that stage's next phase.
            uint32_t j = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb, ++j) {
                    const int s = j % ST, d = j % SD;
                    if (!(ok = wait_idle(&empty_d[d], ((j / SD) & 1) ^ 1, kTimeoutDecode))) break;
                    if (!(ok = mbar_wait(&full_t[s], (j / ST) & 1, P.status, kTimeoutDecode))) break;
                    mbar_arrive_remote(mapa_shared(&full_d[d], 0));
                }
            }
        }
    } else if (warp < kEpiWarp0) {
        // ------------------------------------------------------------ decoders
        // thread dt: SNP row dt % 128, 64 samples (16 packed bytes) starting at 64 * (dt / 128);
        // TMEMA: row 32 (warp % 4) + lane, the TMEM lane quarter this warp may access
        const int dt = threadIdx.x - kDecodeWarp0 * 32;
        const int r = TMEMA ? 32 * (warp & 3) + lane : dt & 127;
        const int h = TMEMA ? (warp - kDecodeWarp0) >> 2 : dt >> 7;  // alt: the warp's group
        const int rbase = (r >> 3) * 1024 + (r & 7) * 128;
        uint32_t j = 0;
        bool ok = true;
        for (int u = u0; u < units && ok; u += ustep) {
            int tile, ct, split, kb0, kb1;
            unit_coords(u, tile, ct, split, kb0, kb1);
            // the row's imputed-code table: rows pass SNP tile * 128 + r, samples pass
            // kb * 128 + r (the packed tile's row); over the sample-major copy the fixed dosage
            // table 2 / 0 / 1 / 0 (six sets) or the K-block's imputed codes staged with the
            // packed tile (TMEMA = 5)
            uint32_t lut = ROWS ? __ldg(P.lut + (int64_t)tile * kTile + r) : 0x00010002u;
            for (int kb = kb0; kb < kb1; ++kb, ++j) {
                if (alt && (int)(j & 1u) != h) continue;  // the other group's K-block
                const int sp = j % SP, d = j % SD;
                if (!KMAJOR) lut = __ldg(P.lut + (int64_t)kb * kKBlock + r);
                if (!(ok = PAIR ? mbar_poll_sleep(&empty_d[d], ((j / SD) & 1) ^ 1, P.status,
                                                  kTimeoutDecode, P.poll_dec_ns)
                                : mbar_wait(&empty_d[d], ((j / SD) & 1) ^ 1, P.status, kTimeoutDecode)))
                    break;
                if (!(ok = mbar_wait(&full_p[sp], (j / SP) & 1, P.status, kTimeoutDecode))) break;
                if constexpr (TMEMA) {
                    tc_fence_after();  // after the MMA's release of this stage (empty_d)
                    // one K half of this lane: 64 K elements = 16 TMEM columns of each tile
                    auto decode_half = [&](int hq) {
                        const uint4 packed = *reinterpret_cast<const uint4*>(smem + L::p(sp) + r * 32 + hq * 16);
                        const uint32_t words[4] = {packed.x, packed.y, packed.z, packed.w};
                        // imputed codes of these 64 SNPs (the same for every lane of the warp:
                        // shared-memory broadcasts)
                        uint4 qv[4];
                        if constexpr (TMEMA == 5) {
#pragma unroll
                            for (int cj = 0; cj < 4; ++cj)
                                qv[cj] = *reinterpret_cast<const uint4*>(smem + L::q(sp) + hq * 64 + cj * 16);
                        }
                        uint32_t ev[16], mv[16];
#pragma unroll
                        for (int cj = 0; cj < 4; ++cj) {
                            uint4 dos, mis;
                            if constexpr (TMEMA == 5)
                                decode_word_imputed(words[cj], qv[cj], dos, mis);
                            else
                                decode_word_interleaved(words[cj], lut, dos, mis);
                            ev[4 * cj] = dos.x; ev[4 * cj + 1] = dos.y; ev[4 * cj + 2] = dos.z; ev[4 * cj + 3] = dos.w;
                            mv[4 * cj] = mis.x; mv[4 * cj + 1] = mis.y; mv[4 * cj + 2] = mis.z; mv[4 * cj + 3] = mis.w;
                        }
                        const uint32_t lane_base = tmem_base + ((uint32_t)(32 * (warp & 3)) << 16) + 16 * hq;
                        tmem_st16(lane_base + L::ta(d), ev);
                        tmem_st16(lane_base + L::tam(d), mv);
                    };
                    if (alt) {  // both halves of the K-block (this group's K-blocks only)
                        decode_half(0);
                        decode_half(1);
                    } else {
                        decode_half(h);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                } else {
                    const uint4 packed = *reinterpret_cast<const uint4*>(smem + L::p(sp) + r * 32 + h * 16);
                    const uint32_t words[4] = {packed.x, packed.y, packed.z, packed.w};
                    unsigned char* a = smem + L::a(d);
                    unsigned char* am = smem + L::am(d);
#pragma unroll
                    for (int cj = 0; cj < 4; ++cj) {
                        uint4 dos, mis;
                        decode_word_interleaved(words[cj], lut, dos, mis);
                        const int chunk = 4 * h + cj;  // 16 samples per 16-byte chunk
                        const int off = rbase + ((chunk ^ (r & 7)) << 4);
                        *reinterpret_cast<uint4*>(a + off) = dos;
                        *reinterpret_cast<uint4*>(am + off) = mis;
                    }
                    fence_proxy_async_smem();
                }
                __syncwarp();
                if (lane == 0) {
                    if (PAIR)
                        mbar_arrive_remote(mapa_shared(&full_d[d], 0));
                    else
                        mbar_arrive(&full_d[d]);
                    mbar_arrive(&empty_p[sp]);  // the packed tile has been read
                }
            }
        }
    } else if (warp == kPackedWarp) {
        // ------------------------------------------------------------ TMA producer (packed)
        if (elect_one()) {
            prefetch_tensormap(&tm_a);
            uint32_t j = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb, ++j) {
                    const int sp = j % SP;
                    if (!(ok = mbar_wait(&empty_p[sp], ((j / SP) & 1) ^ 1, P.status, kTimeoutTma))) break;
                    mbar_arrive_expect_tx(&full_p[sp], (uint32_t)(kPackedBytes + L::kQBytes));
                    // packed tile: 128 rows x 32 bytes (128 K elements)
                    if (KMAJOR)
                        tma_load_2d(smem + L::p(sp), &tm_a, kb * 32, tile * kTile, &full_p[sp]);
                    else
                        tma_load_2d(smem + L::p(sp), &tm_a, tile * 32, kb * kKBlock, &full_p[sp]);
                    if constexpr (L::kQBytes != 0)
                        bulk_load_1d(smem + L::q(sp), reinterpret_cast<const unsigned char*>(P.qperm) +
                                                          (int64_t)kb * kKBlock,
                                     (uint32_t)L::kQBytes, &full_p[sp]);
                }
            }
            // leave no copy in flight
            for (uint32_t q = (j >= (uint32_t)SP ? j - SP : 0); q < j; ++q)
                mbar_wait(&full_p[q % SP], (q / SP) & 1, P.status, kTimeoutTma, 1u << 20);
        }
    } else {
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3;  // TMEM lane quarter this warp may access
        int ui = 0;
        bool ok = true;
        const double ib = 1.0 / kBase, ib2 = 1.0 / (kBase * kBase);
        for (int u = u0; u < units && ok; u += ustep, ++ui) {
            int tile, ct, split, kb0, kb1;
            unit_coords(u, tile, ct, split, kb0, kb1);
            const int buf = ui % NB;
            if (!(ok = wait_idle(&acc_full[buf], (ui / NB) & 1, kTimeoutEpilogue))) break;
            tc_fence_after();
            // rows pass: TMEM lane = SNP row; samples pass: lane = position in the decoded
            // tile, whose samples are interleaved within each group of 16
            const int lp = 32 * q + lane;
            const int64_t row = (int64_t)tile * kTile + (KMAJOR ? lp : (lp & ~15) + sample_at(lp & 15));
            const uint32_t tb = tmem_base + buf * L::kAccStride + ((uint32_t)(32 * q) << 16);
            const int w = width(ct);
            double* dst = P.part + ((int64_t)split * kp + (int64_t)ct * kc) * P.ld + row;
            if (ROWS) {
                // TMEM columns: single CTA [p0 p1 p2 | m0 m1] (w each); pair, w / 2 = hw each,
                // [p0a p1a p2a p0b p1b p2b | m0a m1a m0b m1b] (half a from the leader's B)
                constexpr int CH = PAIR ? 8 : 16;
                const double rt = P.resid[row];
                const double inv_q = 1.0 / (double)kImputeQ;
                const int hw = w / 2;
                for (int c0 = 0; c0 < w; c0 += CH) {
                    const bool hb = PAIR && c0 >= hw;
                    const int cc = hb ? c0 - hw : c0;
                    const int step = PAIR ? hw : w;
                    const uint32_t cm = PAIR ? (hb ? 3 * hw : 0) + cc : c0;
                    const uint32_t cx = 3 * w + (PAIR ? (hb ? 2 * hw : 0) + cc : c0);
                    int32_t m1[CH], m2[CH], m3[CH];
                    tmem_ld_cols<CH>(tb + cm, m1);
                    tmem_ld_cols<CH>(tb + cm + step, m2);
                    tmem_ld_cols<CH>(tb + cm + 2 * step, m3);
                    // main sums first, then the missing-call sums (fewer live registers)
                    double mv[CH];
#pragma unroll
                    for (int i = 0; i < CH; ++i)
                        mv[i] = (double)m1[i] + (double)m2[i] * ib + (double)m3[i] * ib2;
                    tmem_ld_cols<CH>(tb + cx, m1);
                    tmem_ld_cols<CH>(tb + cx + step, m2);
#pragma unroll
                    for (int i = 0; i < CH; ++i) {
                        const double xv = (double)m1[i] + (double)m2[i] * ib;
                        dst[(int64_t)(c0 + i) * P.ld] = mv[i] * inv_q + rt * xv;
                    }
                }
            } else {
                for (int c0 = 0; c0 < w; c0 += 16) {
                    int32_t m1[16], m2[16], m3[16];
                    tmem_ld16i(tb + c0, m1);
                    tmem_ld16i(tb + w + c0, m2);
                    tmem_ld16i(tb + 2 * w + c0, m3);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const double mv = (double)m1[i] + (double)m2[i] * ib + (double)m3[i] * ib2;
                        dst[(int64_t)(c0 + i) * P.ld] = mv * P.inv_f[ct * kc + c0 + i];
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR)
                    mbar_arrive_remote(mapa_shared(&acc_empty[buf], 0));
                else
                    mbar_arrive(&acc_empty[buf]);
            }
        }
    }
    tc_fence_before();
    if (PAIR)
        cluster_sync_all();
    else
        __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        if (PAIR)
            tmem_dealloc_pair(tmem_base, kTmemCols);
        else
            tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---------------------------------------------------------------- operand preparation
// All reductions here are deterministic: FP64 sums over fixed tiles in a fixed order (whatever the
// column count and layout, so that a column's bits do not depend on its neighbours) and maxima of
// non-negative doubles' bits through atomics (order independent).  The order matters beyond that:
// a quantised digit flips where a sum's last bit moves it over a half, so that an iteration on the
// mixed form (the low-rank sketch) moves by 1e-8 when the order of one of these sums changes.
// Every kernel moves each element once, 16 bytes at a time where the layout allows: at 266 columns,
// N=50k, M=100k the operand and reduction kernels around the two passes take 0.39 ms of a 9.9 ms apply.

// Round to nearest even of |v| < 2^31 by adding 1.5 * 2^52: the sum's low word is the integer, two
// additions give it back as a double.  rint and a conversion are both quarter-rate instructions.
__device__ __forceinline__ double round_to(double v, int& q) {
    constexpr double kMagic = 6755399441055744.0;
    const double t = __dadd_rn(v, kMagic);
    q = __double2loint(t);
    return __dadd_rn(t, -kMagic);
}
// Quantises v (centred and multiplied by 127 / max) into three pieces of base 254, of which the low
// bytes are the int8 digits; the products round before the differences (no contraction), whichever
// kernel this is inlined in.
__device__ __forceinline__ void quantise3(double v, double& a, double& b, double& c, int& q1, int& q2, int& q3) {
    a = round_to(v, q1);
    const double r1 = __dmul_rn(__dsub_rn(v, a), kBase);
    b = round_to(r1, q2);
    c = round_to(__dmul_rn(__dsub_rn(r1, b), kBase), q3);
}
__device__ __forceinline__ void quantise3(double v, int& q1, int& q2, int& q3) {
    double a, b, c;
    quantise3(v, a, b, c, q1, q2, q3);
}

// Two pieces of base 254 (the residual operand of the samples pass, |v| <= 63.5).
__device__ __forceinline__ void quantise2(double v, int& q1, int& q2) {
    const double a = round_to(v, q1);
    round_to(__dmul_rn(__dsub_rn(v, a), kBase), q2);
}

// x / d for an integer |x| <= 128 and d = 254 or 254^2: one correction of x (1 / d) by its remainder
// (Markstein 1990) gives the correctly rounded quotient, as tests/test_small_quotient.py checks for each of
// these x.
template <int D>
__device__ __forceinline__ double small_quotient(double x) {
    constexpr double r = 1.0 / D;
    const double q = x * r;
    return fma(fma(-(double)D, q, x), r, q);
}

__device__ __forceinline__ double quant_factor(unsigned long long bits) {
    const double m = __longlong_as_double((long long)bits);
    return m > 0.0 ? 127.0 / m : 0.0;
}

// Whether this block is the last of `n` to arrive at the counter (which wraps back to zero).
// Every thread of the block calls it, after its own writes.
__device__ __forceinline__ bool last_block(unsigned* counter, unsigned n) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(counter, n - 1) == n - 1;
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// What the operand kernels of a call hand on: per column the mean and the bits of max |x - mean|
// (rows operand), the sum of the quantised values, the bits of max |W| and max(|W|, |mu W|) (samples
// operand), and the counters of last_block.
struct MixedColumns {
    double* mean;
    unsigned long long* max1;
    double* qsum;
    unsigned long long* max_w;
    unsigned long long* max_wmu;
    unsigned* counter;
};

// Sums over tiles in the order every column sum of these kernels has: part[t * ld + c] for tiles
// t = l, l + 32, ... by lane l, then the 32 lanes in a shuffle tree.  A block sums `cols` columns (a
// power of two up to 32) from c0 on; a warp calls out(j, sum) for column c0 + j; sh: 32 x 33 doubles.
// Columns are the fastest thread index, so that the partials are read in the order of memory.
template <int THREADS, class Out>
__device__ __forceinline__ void sum_tiles(const double* __restrict__ part, int64_t nt, int64_t ld, int64_t c0,
                                          int cols, int64_t k, double* sh, Out&& out) {
    const int cc = threadIdx.x % cols, slot = threadIdx.x / cols, slots = min(32, THREADS / cols);
    if (slot < slots)
        for (int l = slot; l < 32; l += slots) {
            double sm = 0.0;
            if (c0 + cc < k) {
#pragma unroll 8
                for (int64_t t = l; t < nt; t += 32) sm += __ldcg(part + t * ld + c0 + cc);
            }
            sh[l * 33 + cc] = sm;
        }
    __syncthreads();
    const int wl = threadIdx.x & 31;
    for (int j = threadIdx.x >> 5; j < cols; j += THREADS / 32) {
        double sm = sh[wl * 33 + j];
        for (int off = 16; off; off >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, off);
        if (c0 + j < k) out(j, sm);
    }
}

// Per-column sums over tiles of 64 rows (8 interleaved lanes each, added in lane order) and minima
// and maxima over chunks of two tiles, then, in the last block of a column tile, mean[c] = (sum over
// tiles) / n and max1[c] = the bits of max |x - mean| = max(max x - mean, mean - min x) (rounding is
// monotonic, so this equals the maximum of the rounded differences); the column's maxima of W are
// cleared.  A block covers kc columns (a power of two up to 32) x 32 / kc chunks.
constexpr int kStatTile = 64, kStatTiles = 2, kStatRows = kStatTiles * kStatTile;
template <class T>
__global__ void __launch_bounds__(256)
k_col_stats(const Strided<const T> X, int64_t n, int64_t k, int kc, int64_t nb,
            double* __restrict__ part, const MixedColumns C) {
    chain_enter();
    // the tiles' sums, minima, maxima; 8 lanes and a pad per (column, chunk); then the last block's sums
    __shared__ double red[6][32 * 9];
    static_assert(kStatTiles + 2 <= 6 && 6 * 32 * 9 >= 32 * 33 + 2 * 256);
    // threads in the order of memory: columns fastest in row-major input, lanes in column-major
    const int per = 256 / kc;  // 8 lanes x chunks
    const int tc = X.rs == 1 ? threadIdx.x / per : threadIdx.x % kc;
    const int tl = X.rs == 1 ? threadIdx.x % per : threadIdx.x / kc;
    const int lane = tl & 7, ch = tl >> 3;
    const int64_t c = (int64_t)blockIdx.y * kc + tc;
    const int64_t b = (int64_t)blockIdx.x * (per >> 3) + ch;
    const int64_t nt = (n + kStatTile - 1) / kStatTile;
    const int slot = (tc * (per >> 3) + ch) * 9 + lane;
    double mn = INFINITY, mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < kStatTiles; ++j) {
        double sm = 0.0;
        if (c < k && b < nb) {
            const int64_t r0 = b * kStatRows + j * kStatTile + lane;
#pragma unroll
            for (int q = 0; q < kStatTile; q += 8)
                if (r0 + q < n) {
                    const double v = (double)X.p[(r0 + q) * X.rs + c * X.cs];
                    sm += v;
                    mn = fmin(mn, v);
                    mx = fmax(mx, v);
                }
        }
        red[j][slot] = sm;
    }
    red[kStatTiles][slot] = mn;
    red[kStatTiles + 1][slot] = mx;
    __syncthreads();
    if (threadIdx.x < 32 * kStatTiles) {  // one thread per (column, chunk) and tile
        const int pair = threadIdx.x & 31, j = threadIdx.x >> 5;
        const int oc = pair / (per >> 3), och = pair % (per >> 3);
        const int64_t cc = (int64_t)blockIdx.y * kc + oc, bb = (int64_t)blockIdx.x * (per >> 3) + och;
        if (cc < k && bb < nb) {
            double sm = red[j][9 * pair];
            for (int q = 1; q < 8; ++q) sm += red[j][9 * pair + q];
            if (kStatTiles * bb + j < nt) part[(kStatTiles * bb + j) * k + cc] = sm;
            if (j == 0) {
                mn = INFINITY;
                mx = -INFINITY;
                for (int q = 0; q < 8; ++q) {
                    mn = fmin(mn, red[kStatTiles][9 * pair + q]);
                    mx = fmax(mx, red[kStatTiles + 1][9 * pair + q]);
                }
                part[(nt + bb) * k + cc] = mn;
                part[(nt + nb + bb) * k + cc] = mx;
            }
        }
    }
    if (!last_block(C.counter + blockIdx.y, gridDim.x)) return;
    double* const sh = &red[0][0];
    double *const smn = sh + 32 * 33, *const smx = smn + 256;
    const int64_t c0 = (int64_t)blockIdx.y * kc;
    const int cc = threadIdx.x % kc, sl = threadIdx.x / kc, slots = min(32, 256 / kc);
    if (sl < slots) {
        mn = INFINITY;
        mx = -INFINITY;
        if (c0 + cc < k) {
#pragma unroll 4
            for (int64_t q = sl; q < nb; q += slots) {
                mn = fmin(mn, __ldcg(part + (nt + q) * k + c0 + cc));
                mx = fmax(mx, __ldcg(part + (nt + nb + q) * k + c0 + cc));
            }
        }
        smn[sl * kc + cc] = mn;
        smx[sl * kc + cc] = mx;
    }
    sum_tiles<256>(part, nt, k, c0, kc, k, sh, [&](int j, double sm) {
        const int wl = threadIdx.x & 31;
        double lo = wl < slots ? smn[wl * kc + j] : INFINITY, hi = wl < slots ? smx[wl * kc + j] : -INFINITY;
        for (int off = 16; off; off >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, off));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, off));
        }
        if (wl == 0) {
            const double m = sm / (double)n;
            C.mean[c0 + j] = m;
            const double a = fmax(fmax(hi - m, m - lo), 0.0);
            C.max1[c0 + j] = (unsigned long long)__double_as_longlong(a);
            C.max_w[c0 + j] = 0;
            C.max_wmu[c0 + j] = 0;
        }
    });
}

// 16 int8 values (by K element) -> the 16 bytes of their K positions: interleaved as the decoded
// tiles are, or in order.
template <bool INTERLEAVE>
__device__ __forceinline__ uint4 pack16(const int (&q)[16]) {
    uint32_t w[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        const int e0 = INTERLEAVE ? sample_at(4 * g) : 4 * g, e1 = INTERLEAVE ? sample_at(4 * g + 1) : 4 * g + 1;
        const int e2 = INTERLEAVE ? sample_at(4 * g + 2) : 4 * g + 2, e3 = INTERLEAVE ? sample_at(4 * g + 3) : 4 * g + 3;
        w[g] = __byte_perm(__byte_perm((uint32_t)q[e0], (uint32_t)q[e1], 0x0040),
                           __byte_perm((uint32_t)q[e2], (uint32_t)q[e3], 0x0040), 0x5410);
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}

// Byte p of w = the low byte of q (p known at compile time).
__device__ __forceinline__ void put_byte(uint32_t (&w)[4], int p, int q) {
    w[p >> 2] = __byte_perm(w[p >> 2], (uint32_t)q, 0x3210 ^ (((p & 3) ^ 4) << (4 * (p & 3))));
}

// Rows 16 g .. 16 g + 15 of a tile of 64 (`rows` of them live, g = grp % 4 the thread's place among
// the tile's four, which are neighbours in a warp): the pieces' bytes at their K positions, and the
// sum over the tile of the represented values in the order rows i and i + 32, then + 16, + 8, + 4,
// + 2, + 1; each thread keeps a quarter of the pairs (j = 4 m + 2 lo + hi) as the values come.
__device__ __forceinline__ double split16(const double* x, int rows, double mean, double f, int grp,
                                          uint32_t (&w1)[4], uint32_t (&w2)[4], uint32_t (&w3)[4]) {
    const bool hi = grp & 2, lo = grp & 1;
    double val[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int j = 4 * m + q;
            double a, b, d;
            int q1, q2, q3;
            quantise3(j < rows ? __dmul_rn(x[j] - mean, f) : 0.0, a, b, d, q1, q2, q3);
            put_byte(w1, position_of(j), q1);
            put_byte(w2, position_of(j), q2);
            put_byte(w3, position_of(j), q3);
            v[q] = a + small_quotient<254>(b) + small_quotient<64516>(d);
        }
        const double x0 = (hi ? v[1] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[1], 2);
        const double x1 = (hi ? v[3] : v[2]) + __shfl_xor_sync(0xffffffffu, hi ? v[2] : v[3], 2);
        val[m] = (lo ? x1 : x0) + __shfl_xor_sync(0xffffffffu, lo ? x0 : x1, 1);
    }
    double sum = (val[0] + val[2]) + (val[1] + val[3]);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    return sum;
}

// Both of the above for n <= kWholeRows: a block per column holds it in shared memory, and a thread
// quantises 16 rows.  The same sums in the same order as k_col_stats and k_split_rows_operand, without
// a second kernel, the counters and the reading of the partial sums, which is what those two spend 22 us
// on at n=2000 and 34 columns: an AI-REML of 453 such products takes 45.5 ms with it and 48.8 without
// (of which the shorter chains of k_col_stats, k_reduce_samples and the solver's sums are a part).
constexpr int kWholeRows = 8192;
template <class T>
__global__ void __launch_bounds__(kWholeRows / 16)
k_rows_operand_whole(const Strided<const T> X, int64_t n, int64_t k, int64_t kp, int64_t n_pad,
                     const MixedColumns C, int8_t* __restrict__ B) {
    chain_enter();
    extern __shared__ double col[];  // [n_pad], one pad every 16
    __shared__ double sums[kWholeRows / 64], lo[16], hi[16], stat[2];
    const int64_t c = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    const int rows = (int)n, nt = (rows + 63) / 64;
    const bool live = c < k;
    double mn = INFINITY, mx = -INFINITY;
#pragma unroll 4
    for (int r = threadIdx.x; r < (int)n_pad; r += blockDim.x) {
        double v = 0.0;
        if (live && r < rows) {
            v = (double)X.p[r * X.rs + c * X.cs];
            mn = fmin(mn, v);
            mx = fmax(mx, v);
        }
        col[r + (r >> 4)] = v;
    }
    for (int off = 16; off; off >>= 1) {
        mn = fmin(mn, __shfl_xor_sync(0xffffffffu, mn, off));
        mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, off));
    }
    if (lane == 0) {
        lo[warp] = mn;
        hi[warp] = mx;
    }
    __syncthreads();
    // tiles of 64 rows, eight interleaved lanes added in lane order
    for (int t = threadIdx.x >> 3; t < (int)n_pad / 64; t += blockDim.x >> 3) {
        double sm = 0.0;
#pragma unroll
        for (int q = 0; q < 64; q += 8) {
            const int r = 64 * t + q + (threadIdx.x & 7);
            if (r < rows) sm += col[r + (r >> 4)];
        }
        double tot = __shfl_sync(0xffffffffu, sm, lane & 24);
#pragma unroll
        for (int j = 1; j < 8; ++j) tot += __shfl_sync(0xffffffffu, sm, (lane & 24) + j);
        if ((threadIdx.x & 7) == 0) sums[t] = tot;
    }
    __syncthreads();
    auto column_sum = [&]() {  // by one warp, as sum_tiles adds
        double sm = 0.0;
        for (int t = lane; t < nt; t += 32) sm += sums[t];
        for (int off = 16; off; off >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, off);
        return sm;
    };
    if (warp == 0) {
        const double m = column_sum() / (double)n;
        double a = lane < warps ? lo[lane & 15] : INFINITY, b = lane < warps ? hi[lane & 15] : -INFINITY;
        for (int off = 16; off; off >>= 1) {
            a = fmin(a, __shfl_xor_sync(0xffffffffu, a, off));
            b = fmax(b, __shfl_xor_sync(0xffffffffu, b, off));
        }
        if (lane == 0) {
            stat[0] = m;
            stat[1] = fmax(fmax(b - m, m - a), 0.0);
        }
    }
    __syncthreads();
    const double mean = stat[0];
    const unsigned long long max1 = (unsigned long long)__double_as_longlong(stat[1]);
    const int i0 = 16 * threadIdx.x;  // blockDim.x * 16 == n_pad rounded up to 512
    uint32_t w1[4] = {}, w2[4] = {}, w3[4] = {};
    const double sum = split16(col + 17 * threadIdx.x, live && i0 < rows ? min(16, rows - i0) : 0, mean,
                               live ? quant_factor(max1) : 0.0, threadIdx.x, w1, w2, w3);
    if (i0 < (int)n_pad) {
        *reinterpret_cast<uint4*>(B + c * n_pad + i0) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
        *reinterpret_cast<uint4*>(B + (kp + c) * n_pad + i0) = make_uint4(w2[0], w2[1], w2[2], w2[3]);
        *reinterpret_cast<uint4*>(B + (2 * kp + c) * n_pad + i0) = make_uint4(w3[0], w3[1], w3[2], w3[3]);
        if ((threadIdx.x & 3) == 0) sums[threadIdx.x >> 2] = sum;
    }
    __syncthreads();
    if (warp == 0 && live) {
        const double q = column_sum();
        if (lane == 0) {
            C.mean[c] = mean;
            C.max1[c] = max1;
            C.qsum[c] = q;
            C.max_w[c] = 0;
            C.max_wmu[c] = 0;
        }
    }
}

// Rows-pass operand: B1[q*kp + c][pos(i)] (int8 pieces of (x_ic - mean_c) 127 / max_c, i < n_pad;
// pos interleaves each group of 16 samples as the decoded tiles do) and the sums Q_c of the
// represented values: in tiles of 64 rows (rows i and i + 32, then the 32 pairs in a tree), the
// tiles by the last block of a column group.  A block takes COLS columns x ROWS rows through shared
// memory; a thread takes 16 rows of a column, four threads a tile.  Loads and arithmetic overlap only
// between blocks, so the registers are held to 64 for 1024 threads an SM: 79 us at 266 columns, N=50k,
// against 160 with 128 registers.
template <class T, int COLS, int ROWS>
__global__ void __launch_bounds__(ROWS / 16 * COLS, 1024 / (ROWS / 16 * COLS))
k_split_rows_operand(const Strided<const T> X, int64_t n, int64_t k, int64_t kp, int64_t n_pad,
                     const MixedColumns C, int8_t* __restrict__ B, double* __restrict__ part) {
    chain_enter();
    constexpr int TH = ROWS / 16 * COLS;
    constexpr int kPitch = ROWS + ROWS / 16 + 1;  // one pad every 16 rows and one per column
    static_assert(COLS * kPitch >= 32 * 33, "sum_tiles's scratch");
    __shared__ double tile[COLS * kPitch];
    const int64_t r0 = (int64_t)blockIdx.x * ROWS, c0 = (int64_t)blockIdx.y * COLS;
    for (int e = threadIdx.x; e < ROWS * COLS; e += TH) {
        const int rr = X.rs == 1 ? e % ROWS : e / COLS, cc = X.rs == 1 ? e / ROWS : e % COLS;
        const int64_t r = r0 + rr, c = c0 + cc;
        tile[cc * kPitch + rr + (rr >> 4)] = (r < n && c < k) ? (double)X.p[r * X.rs + c * X.cs] : 0.0;
    }
    __syncthreads();
    const int grp = threadIdx.x % (ROWS / 16), cc = threadIdx.x / (ROWS / 16);
    const int64_t c = c0 + cc, i0 = r0 + 16 * grp;
    const double f = c < k ? quant_factor(C.max1[c]) : 0.0;
    const double mc = c < k ? C.mean[c] : 0.0;
    uint32_t w1[4] = {}, w2[4] = {}, w3[4] = {};
    const double sum = split16(tile + cc * kPitch + 17 * grp, c < k ? (int)min((int64_t)16, n - i0) : 0, mc, f, grp,
                               w1, w2, w3);
    if (c < kp && i0 < n_pad) {
        *reinterpret_cast<uint4*>(B + c * n_pad + i0) = make_uint4(w1[0], w1[1], w1[2], w1[3]);
        *reinterpret_cast<uint4*>(B + (kp + c) * n_pad + i0) = make_uint4(w2[0], w2[1], w2[2], w2[3]);
        *reinterpret_cast<uint4*>(B + (2 * kp + c) * n_pad + i0) = make_uint4(w3[0], w3[1], w3[2], w3[3]);
    }
    const int64_t nt = (n + 63) / 64;
    if ((grp & 3) == 0 && c < k && i0 < n) part[(i0 >> 6) * k + c] = sum;
    if (c0 >= k || !last_block(C.counter + blockIdx.y, gridDim.x)) return;
    sum_tiles<TH>(part, nt, k, c0, COLS, k, tile, [&](int j, double sm) {
        if ((threadIdx.x & 31) == 0) C.qsum[c0 + j] = sm;
    });
}

// (sum_z part[z][c][t] - mu_t Q_c) / f_c + mean_c exc_t, the rows pass's centred product.
struct RowsColumn {
    double inv_f, mean, qsum;
    __device__ __forceinline__ RowsColumn(const MixedColumns& C, int64_t c) {
        const double f = quant_factor(C.max1[c]);
        inv_f = f > 0.0 ? 1.0 / f : 0.0;
        mean = C.mean[c];
        qsum = C.qsum[c];
    }
    __device__ __forceinline__ double value(double acc, double mu, double exc) const {
        return fma(mean, exc, __dmul_rn(fma(-mu, qsum, acc), inv_f));
    }
};

// Rows-pass reduction for an apply: W^T (column-major, R per column) = s^2 o the product, with the
// maxima of |W| and of max(|W|, |mu W|).  1024 SNPs per block, one column per blockIdx.y.
__global__ void __launch_bounds__(256)
k_reduce_rows(const double* __restrict__ part, int splits, int64_t kp, int64_t ld, int64_t R,
              const double* __restrict__ s_row, const double* __restrict__ exc_row,
              const double* __restrict__ mu, const MixedColumns C, double* __restrict__ out) {
    chain_enter();
    __shared__ double red[2][8];
    const int64_t c = blockIdx.y;
    const RowsColumn col(C, c);
    double mw = 0.0, mm = 0.0;
    const int64_t t0 = (int64_t)blockIdx.x * 1024 + threadIdx.x;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
    for (int z = 0; z < splits; ++z) {
        const double* p = part + ((int64_t)z * kp + c) * ld + t0;  // ld >= R rounded up to 256
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (t0 + 256 * j < R) acc[j] += p[256 * j];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int64_t t = t0 + 256 * j;
        if (t < R) {
            const double m = mu[t], s = s_row[t];
            const double v = col.value(acc[j], m, exc_row[t]) * s * s;
            out[c * R + t] = v;
            mw = fmax(mw, fabs(v));
            mm = fmax(mm, fmax(fabs(v), m * fabs(v)));
        }
    }
    for (int off = 16; off; off >>= 1) {
        mw = fmax(mw, __shfl_xor_sync(0xffffffffu, mw, off));
        mm = fmax(mm, __shfl_xor_sync(0xffffffffu, mm, off));
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = mw;
        red[1][threadIdx.x >> 5] = mm;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < 8; ++j) {
            mw = fmax(mw, red[0][j]);
            mm = fmax(mm, red[1][j]);
        }
        atomicMax(C.max_w + c, (unsigned long long)__double_as_longlong(mw));
        atomicMax(C.max_wmu + c, (unsigned long long)__double_as_longlong(mm));
    }
}

// Rows-pass reduction for a half-pass or a scan: out(row, c) = s_t o the product, row = pos[t] (or
// t).  Tiles of 32 SNPs x 32 columns; a row-major result goes through shared memory, so that both
// sides are coalesced.
__global__ void __launch_bounds__(256)
k_reduce_rows_out(const double* __restrict__ part, int splits, int64_t kp, int64_t ld, int64_t R,
                  int64_t k, const double* __restrict__ s_row, const double* __restrict__ exc_row,
                  const double* __restrict__ mu, const int32_t* __restrict__ pos, const MixedColumns C,
                  StridedOut out) {
    chain_enter();
    __shared__ double tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t t0 = (int64_t)blockIdx.x * 32, c0 = (int64_t)blockIdx.y * 32;
    const int64_t t = t0 + tx;
#pragma unroll
    for (int cc = ty; cc < 32; cc += 8) {
        const int64_t c = c0 + cc;
        if (c >= k || t >= R) continue;
        const RowsColumn col(C, c);
        double acc = 0.0;
        for (int z = 0; z < splits; ++z) acc += part[((int64_t)z * kp + c) * ld + t];
        const double v = col.value(acc, mu[t], exc_row[t]) * s_row[t];
        if (out.rs == 1) out.p[(pos ? (int64_t)pos[t] : t) + c * out.cs] = v;
        else tile[cc][tx] = v;
    }
    if (out.rs == 1) return;
    __syncthreads();
    for (int tt = ty; tt < 32; tt += 8) {
        const int64_t r = t0 + tt, c = c0 + tx;
        if (r < R && c < k) out.p[(pos ? (int64_t)pos[r] : r) * out.rs + c * out.cs] = tile[tx][tt];
    }
}

// Samples-pass operand from W^T (column-major, k x R), and the sums c0_c of mu_t W[t][c] (the
// centring term): chunks of 2048 SNPs, added in chunk order by the last block of the column.
//   SIX: pieces of W f (rows q kp + c) and of (mu o W) f (rows (3 + q) kp + c), f = 127 /
//        max(|W|, |mu W|), at interleaved K positions;
//   otherwise three pieces of W f and two of (Q r o W) f, f = 127 / max|W| (|Q r_t| <= 1/2), so
//        that both MMAs accumulate into the same TMEM columns; INTERLEAVE (over the sample-major
//        copy) also negates the residual pieces (that decoder's missing-indicator tile holds -1).
// inv_f[c] scales the sums back.  A thread takes 16 SNPs of a column.  Grid: (chunks, kp).
template <bool SIX, bool INTERLEAVE>
__global__ void __launch_bounds__(128)
k_split_samples_operand(const double* __restrict__ Wt, int64_t R, int64_t k, int64_t kp,
                        int64_t r_pad, const double* __restrict__ mu,
                        const double* __restrict__ resid, const MixedColumns C,
                        int8_t* __restrict__ B, double* __restrict__ inv_f,
                        double* __restrict__ cpart, double* __restrict__ c0) {
    chain_enter();
    __shared__ double red[8];
    // W and the second operand of 2048 SNPs, one pad every 16, read in the order of memory
    __shared__ double sw[128 * 17], sb[128 * 17];
    const int64_t c = blockIdx.y;
    const double f = c < k ? quant_factor(SIX ? C.max_wmu[c] : C.max_w[c]) : 0.0;
    if (blockIdx.x == 0 && threadIdx.x == 0) inv_f[c] = f > 0.0 ? 1.0 / (SIX ? f : f * kImputeQ) : 0.0;
    double cs[2] = {0.0, 0.0};  // a chunk is summed by 256 lanes, two to a thread
    const int64_t base = (int64_t)blockIdx.x * 2048;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int e = threadIdx.x + 128 * q;
        const int64_t t = base + e;
        double w = 0.0, b = 0.0;
        if (c < k && t < R) {
            const double m = mu[t];
            w = Wt[c * R + t];
            b = SIX ? __dmul_rn(m, w) : (INTERLEAVE ? -kImputeQ : kImputeQ) * resid[t] * w;
            cs[q & 1] = SIX ? __dadd_rn(cs[q & 1], b) : fma(m, w, cs[q & 1]);
        }
        sw[e + (e >> 4)] = w;
        sb[e + (e >> 4)] = b;
    }
    __syncthreads();
    const int64_t t0 = base + 16 * threadIdx.x;
    if (t0 < r_pad) {
        int8_t* dst = B + c * r_pad + t0;
        const int64_t step = kp * r_pad;
        int q1[16], q2[16], q3[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) quantise3(__dmul_rn(sw[17 * threadIdx.x + j], f), q1[j], q2[j], q3[j]);
        *reinterpret_cast<uint4*>(dst) = pack16<INTERLEAVE>(q1);
        *reinterpret_cast<uint4*>(dst + step) = pack16<INTERLEAVE>(q2);
        *reinterpret_cast<uint4*>(dst + 2 * step) = pack16<INTERLEAVE>(q3);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const double v = __dmul_rn(sb[17 * threadIdx.x + j], f);
            if (SIX) quantise3(v, q1[j], q2[j], q3[j]);
            else quantise2(v, q1[j], q2[j]);
        }
        *reinterpret_cast<uint4*>(dst + 3 * step) = pack16<INTERLEAVE>(q1);
        *reinterpret_cast<uint4*>(dst + 4 * step) = pack16<INTERLEAVE>(q2);
        if (SIX) *reinterpret_cast<uint4*>(dst + 5 * step) = pack16<INTERLEAVE>(q3);
    }
    if (c >= k) return;
    for (int off = 16; off; off >>= 1) {
        cs[0] += __shfl_xor_sync(0xffffffffu, cs[0], off);
        cs[1] += __shfl_xor_sync(0xffffffffu, cs[1], off);
    }
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = cs[0];
        red[4 + (threadIdx.x >> 5)] = cs[1];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double sm = red[0];
        for (int j = 1; j < 8; ++j) sm += red[j];
        cpart[(int64_t)blockIdx.x * k + c] = sm;
    }
    if (!last_block(C.counter + c, gridDim.x)) return;
    if (threadIdx.x < 32) {
        double sm = 0.0;
        for (int64_t b = threadIdx.x; b < gridDim.x; b += 32) sm += __ldcg(cpart + b * k + c);
        for (int off = 16; off; off >>= 1) sm += __shfl_xor_sync(0xffffffffu, sm, off);
        if (threadIdx.x == 0) c0[c] = sm;
    }
}

// Sample-major copy of a packed view for the samples pass with A in TMEM: dst row i (sample,
// i < n_pad) holds the 2-bit codes of SNPs 0..r_pad-1, four per byte (SNP t at bits
// 2 (t % 4) of byte t / 4), stride r_pad / 4.  SNP rows past R read as code 0 (they meet zero
// B rows); samples past the analysed ones keep the rows' missing-code padding.
// One CTA per 256 SNPs x 256 samples, a thread per 16 x 16 codes: sixteen words in registers,
// exchanged in four steps of halving block size (the first two byte permutes), then through
// shared memory so that reads and writes are 64-byte runs.  A byte-at-a-time form of 128 x 128
// tiles took 2.33 ms for N=50k, M=100k; this one takes 0.54 ms
// (two passes over 1.25 GB: 0.38).
constexpr int kTransposeTile = 256;
__global__ void __launch_bounds__(256)
k_transpose_packed(const uint8_t* __restrict__ src, int64_t R, int64_t stride,
                   uint8_t* __restrict__ dst, int64_t stride_t) {
    __shared__ uint32_t tile[kTransposeTile][17];
    const int64_t t0 = (int64_t)blockIdx.x * kTransposeTile, b0 = (int64_t)blockIdx.y * (kTransposeTile / 4);
    const int bj = threadIdx.x & 15, bi = threadIdx.x >> 4;  // sample block, SNP block
    uint32_t w[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int64_t t = t0 + 16 * bi + r;
        w[r] = t < R ? __ldg(reinterpret_cast<const uint32_t*>(src + t * stride + b0) + bj) : 0u;
    }
    // w[r] holds codes (r, 0..15); exchange the off-diagonal blocks of 8, 4, 2 and 1 codes
#pragma unroll
    for (int r = 0; r < 16; ++r)
        if (!(r & 8)) {
            const uint32_t a = w[r], c = w[r | 8];
            w[r] = __byte_perm(a, c, 0x5410);
            w[r | 8] = __byte_perm(a, c, 0x7632);
        }
#pragma unroll
    for (int r = 0; r < 16; ++r)
        if (!(r & 4)) {
            const uint32_t a = w[r], c = w[r | 4];
            w[r] = __byte_perm(a, c, 0x6240);
            w[r | 4] = __byte_perm(a, c, 0x7351);
        }
#pragma unroll
    for (int r = 0; r < 16; ++r)
        if (!(r & 2)) {
            const uint32_t x = ((w[r] >> 4) ^ w[r | 2]) & 0x0F0F0F0Fu;
            w[r | 2] ^= x;
            w[r] ^= x << 4;
        }
#pragma unroll
    for (int r = 0; r < 16; ++r)
        if (!(r & 1)) {
            const uint32_t x = ((w[r] >> 2) ^ w[r | 1]) & 0x33333333u;
            w[r | 1] ^= x;
            w[r] ^= x << 2;
        }
#pragma unroll
    for (int r = 0; r < 16; ++r) tile[16 * bj + r][bi] = w[r];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        const int i = q * 16 + (threadIdx.x >> 4);
        *(reinterpret_cast<uint32_t*>(dst + (b0 * 4 + i) * stride_t + t0 / 4) + bj) = tile[i][bj];
    }
}

// The samples operand's W of a half-pass, W^T[c][t] = s_t V[pos[t]][c], and its maxima (cleared
// before).  1024 SNPs per block, one column per blockIdx.y.
__global__ void __launch_bounds__(256)
k_gather_operand(const StridedIn V, int64_t R, const int32_t* __restrict__ pos,
                 const double* __restrict__ s_row, const double* __restrict__ mu, const MixedColumns C,
                 double* __restrict__ Wt) {
    chain_enter();
    const int64_t c = blockIdx.y;
    double mw = 0.0, mm = 0.0;
    const int64_t t0 = (int64_t)blockIdx.x * 1024;
    for (int64_t t = t0 + threadIdx.x; t < min(R, t0 + 1024); t += 256) {
        const double w = s_row[t] * V.p[(int64_t)pos[t] * V.rs + c * V.cs];
        Wt[c * R + t] = w;
        mw = fmax(mw, fabs(w));
        mm = fmax(mm, fmax(fabs(w), mu[t] * fabs(w)));
    }
    for (int off = 16; off; off >>= 1) {
        mw = fmax(mw, __shfl_xor_sync(0xffffffffu, mw, off));
        mm = fmax(mm, __shfl_xor_sync(0xffffffffu, mm, off));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(C.max_w + c, (unsigned long long)__double_as_longlong(mw));
        atomicMax(C.max_wmu + c, (unsigned long long)__double_as_longlong(mm));
    }
}

// Samples-pass reduction: Y[i][c] = (sum_z part[z][c][i] - c0_c) / M.  Tiles of 32 samples x 32
// columns; a row-major result goes through shared memory, so that both sides are coalesced.
template <class T>
__global__ void __launch_bounds__(256)
k_reduce_samples(const double* __restrict__ part, int splits, int64_t kp, int64_t ld, int64_t n,
                 int64_t k, const double* __restrict__ c0v, double inv_m, const Strided<T> Y) {
    chain_enter();
    __shared__ double tile[32][33];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * 32, c0 = (int64_t)blockIdx.y * 32;
    const int64_t i = i0 + tx;
    // four columns a thread, slices in order, four slices' loads at a time
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const double* p = part + (c0 + ty) * ld + i;  // i < n <= ld
#pragma unroll 4
    for (int z = 0; z < splits; ++z, p += kp * ld) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (c0 + ty + 8 * j < k && i < n) acc[j] += p[8 * j * ld];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int64_t c = c0 + ty + 8 * j;
        if (c >= k || i >= n) continue;
        const double v = (acc[j] - c0v[c]) * inv_m;
        if (Y.rs == 1) Y.p[i + c * Y.cs] = (T)v;
        else tile[ty + 8 * j][tx] = v;
    }
    if (Y.rs == 1) return;
    __syncthreads();
    for (int ii = ty; ii < 32; ii += 8) {
        const int64_t r = i0 + ii, c = c0 + tx;
        if (r < n && c < k) Y.p[r * Y.rs + c * Y.cs] = (T)tile[tx][ii];
    }
}

// ---------------------------------------------------------------- tensor maps
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                 const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    });
    if (!fn) fail(CS_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
    return fn;
}

}  // namespace

CUtensorMap make_map_u8(const void* base, uint64_t inner, uint64_t outer, uint64_t row_bytes,
                        uint32_t box_inner, uint32_t box_outer, bool swizzle) {
    CUtensorMap m;
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {row_bytes};
    const cuuint32_t box[2] = {box_inner, box_outer};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode_fn()(&m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base),
                                   dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                   swizzle ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        fail(CS_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
    return m;
}

namespace {

// Both passes run on CTA pairs (cta_group::2) for more than 32 right-hand sides unless
// CS_B200_CTA_PAIRS=0 selects the single-CTA kernels (=1: pairs for every width).  Measured
// on B200 at N=50k, M=100k: k=266 rows 5.4 vs 5.8 ms, samples 5.7 vs 7.7 ms (pair vs
// single); k=32 1.30 vs 1.14 ms per pass, the pair's cross-CTA handshakes per K-block
// outweighing its narrow MMAs.
constexpr int64_t kPairMinColumns = 33;
int pair_mode() {
    static const int mode = [] {
        const char* v = std::getenv("CS_B200_CTA_PAIRS");
        if (v && std::strcmp(v, "0") == 0) return 0;
        if (v && std::strcmp(v, "1") == 0) return 2;
        return 1;
    }();
    return mode;
}
// The narrow passes with A in TMEM, and the 64-wide form of them for 33 to 64 right-hand sides
// instead of CTA pairs (CS_B200_TMEM_A=0: A in shared memory; =1: the 32-wide form only).
// Measured at N=50k, M=100k, per pass (rows / samples): k <= 16 0.70 / 0.80 ms against
// 1.03 / 1.14 with A in shared memory; k = 34 0.90 / 1.07 against 1.15 / 1.24 on CTA pairs;
// k = 64 1.02 / 1.21 against 1.22 / 1.25.
int tmem_a_mode() {
    static const int mode = [] {
        const char* v = std::getenv("CS_B200_TMEM_A");
        if (v && std::strcmp(v, "0") == 0) return 0;
        if (v && std::strcmp(v, "1") == 0) return 1;
        return 2;
    }();
    return mode;
}
bool tmem_a_default() { return tmem_a_mode() != 0; }
// The passes on CTA pairs with A in TMEM (column tiles of at most 64; the samples pass over the
// sample-major copy, six operand sets) as the default pair plans (CS_B200_TMEM_A_PAIRS=0: A in
// shared memory; =1: the rows pass only; =3: the samples pass in the five-set form, TMEMA = 5).
// Measured at N=50k, M=100k, rows / samples per pass against A in shared memory: k = 96
// 1.75 / 1.93 vs 2.31 / 2.48 ms, k = 128 1.89 / 2.12 vs 2.33 / 2.52, k = 192 2.81 / 3.15 vs
// 3.41 / 3.70, k = 266 4.62 / 5.28 vs 4.92 / 5.47.
int tmem_a_pairs_mode() {
    static const int mode = [] {
        const char* v = std::getenv("CS_B200_TMEM_A_PAIRS");
        if (v && std::strcmp(v, "0") == 0) return 0;
        if (v && std::strcmp(v, "1") == 0) return 1;
        if (v && std::strcmp(v, "3") == 0) return 3;
        return 2;
    }();
    return mode;
}
// Pauses between polls in the pair kernels, in nanoseconds: the long waits (the epilogue's
// accumulator, the B producer's free stage, the partner CTA's forwarding;
// CS_B200_POLL_SLEEP_NS, default 128) and the decoders' waits for a free stage
// (CS_B200_POLL_SLEEP_DEC_NS, default 32).  A warp that polls without pause takes issue slots
// from the decoders and the MMA thread on its scheduler.  Measured per pass (rows / samples)
// at N=50k, M=100k, k=266 against no pauses: 4.46 / 5.24 vs 4.76-4.91 / 5.48-5.63 ms; k=96
// 1.67 / 1.88 vs 1.82 / 2.02; 512 ns pauses are slower than none.
// At most 1 us: a wait gives up after 2^26 polls, so the pause sets how long a stalled pass
// takes to report its timeout (about 12 s at the 128 ns default, 70 s at the cap).
uint32_t env_ns(const char* name, uint32_t def) {
    const char* v = std::getenv(name);
    if (!v || !*v) return def;
    const long x = std::strtol(v, nullptr, 10);
    return (uint32_t)std::max(0L, std::min(x, 1000L));
}
uint32_t poll_sleep_ns() {
    static const uint32_t ns = env_ns("CS_B200_POLL_SLEEP_NS", 128u);
    return ns;
}
uint32_t poll_dec_sleep_ns() {
    static const uint32_t ns = env_ns("CS_B200_POLL_SLEEP_DEC_NS", 32u);
    return ns;
}
// Passes with A in TMEM: the decoder warps in two groups of four taking alternate K-blocks
// whole (default), or all eight on every K-block, each one half of K for its lane quarter
// (CS_B200_DECODE_ALT=0).  With one K-block per warp at a time, a K-block's decode latency
// (the packed-tile read, the byte permutes, two tcgen05.st and their wait) set the pace of the
// TMEM passes; two groups keep two K-blocks in decode.  Measured at N=50k, M=100k, rows /
// samples per pass (ms), alternate vs shared, same box: k=16 0.70 / 0.73 vs 1.00 / 1.07; k=48
// 0.93 / 1.06 vs 1.01 / 1.09; k=96 1.66 / 1.97 vs 2.09 / 2.25; k=266 4.23 / 5.06 vs 5.24 / 5.75.
int decode_alt_mode() {
    static const int mode = [] {
        const char* v = std::getenv("CS_B200_DECODE_ALT");
        return (v && std::strcmp(v, "0") == 0) ? 0 : 1;
    }();
    return mode;
}
bool tmem_a_pairs_default() { return tmem_a_pairs_mode() != 0; }
// The narrow single-CTA layout for 32 or fewer right-hand sides (CS_B200_NARROW=0: never).
bool narrow_layouts() {
    static const bool on = [] {
        const char* v = std::getenv("CS_B200_NARROW");
        return !(v && std::strcmp(v, "0") == 0);
    }();
    return on;
}
bool use_cta_pairs(int64_t k) {
    const int mode = pair_mode();
    return mode != 0 && (mode == 2 || k >= kPairMinColumns) && num_sms() >= 2;
}

// Number of K slices so that about `target` work units cover the GPU, and at least enough that
// no slice holds more than kMaxKbPerAccum K-blocks (the int32 accumulators' exact range).
int choose_splits(int64_t units_per_split, int kb_total, int64_t target) {
    int64_t s = (target + units_per_split - 1) / units_per_split;
    s = std::max<int64_t>(1, std::min<int64_t>(s, std::max(1, kb_total / 8)));
    s = std::max<int64_t>(s, (kb_total + kMaxKbPerAccum - 1) / kMaxKbPerAccum);
    return (int)s;
}

}  // namespace

struct MixedWorkspace {
    DeviceBuffer<int8_t> b1, b2;
    DeviceBuffer<double> part, colpart, mean1, qsum, c0, W, inv_f;
    DeviceBuffer<unsigned long long> max1, max_w, max_wmu;
    DeviceBuffer<unsigned> counter;
    // the column words of a call on k columns (new counters start at zero)
    MixedColumns columns(int64_t k, cudaStream_t s) {
        mean1.resize(k);
        max1.resize(k);
        qsum.resize(k);
        max_w.resize(k);
        max_wmu.resize(k);
        if (counter.count < (size_t)k) {
            counter.resize(k);
            CS_CUDA(cudaMemsetAsync(counter.get(), 0, 4 * counter.count, s));
        }
        return MixedColumns{mean1.get(), max1.get(), qsum.get(), max_w.get(), max_wmu.get(), counter.get()};
    }
    CUtensorMap tm_b1{}, tm_b2{};
    CUtensorMap tm_b1t{}, tm_b2t{};  // boxes of the last column tile's width
    const void* tm_b1_base = nullptr;
    const void* tm_b2_base = nullptr;
    int64_t tm_b1_key = -1, tm_b2_key = -1;
    DeviceBuffer<int> status;
};

struct MixedOperator {
    MixedRows rows;
    MixedWorkspace ws;
    int64_t last_k = 0;  // columns of ws.W from the last apply (0: none yet)
};

void destroy_mixed(MixedOperator* m) { delete m; }

namespace {

template <bool ROWS, bool PAIR, bool NARROW = false, int TMEMA = 0>
cudaError_t allow_smem() {
    constexpr int bytes = Layout<ROWS, PAIR, NARROW, TMEMA>::kSmem;
    cudaError_t e = cudaFuncSetAttribute(k_mixed_pass<ROWS, PAIR, NARROW, TMEMA, false>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if constexpr (TMEMA != 0)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_mixed_pass<ROWS, PAIR, NARROW, TMEMA, true>,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    return e;
}

void configure_kernels() {
    static PerDeviceOnce configured;
    once_per_device(configured, [] {
        cudaError_t err = allow_smem<true, false>();
        constexpr int kWholeBytes = 8 * (kWholeRows + kWholeRows / 16 + 16);
        if (err == cudaSuccess)
            err = cudaFuncSetAttribute(k_rows_operand_whole<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeBytes);
        if (err == cudaSuccess)
            err = cudaFuncSetAttribute(k_rows_operand_whole<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWholeBytes);
        if (err == cudaSuccess) err = allow_smem<false, false>();
        if (err == cudaSuccess) err = allow_smem<true, true>();
        if (err == cudaSuccess) err = allow_smem<false, true>();
        if (err == cudaSuccess) err = allow_smem<true, false, true>();
        if (err == cudaSuccess) err = allow_smem<false, false, true>();
        if (err == cudaSuccess) err = allow_smem<true, false, true, 1>();
        if (err == cudaSuccess) err = allow_smem<false, false, true, 1>();
        if (err == cudaSuccess) err = allow_smem<true, false, true, 2>();
        if (err == cudaSuccess) err = allow_smem<false, false, true, 2>();
        if (err == cudaSuccess) err = allow_smem<true, true, false, 3>();
        if (err == cudaSuccess) err = allow_smem<false, true, false, 4>();
        if (err == cudaSuccess) err = allow_smem<false, true, false, 5>();
        return err;
    }, "configure tensor-core kernels");
}

// Clusters of two CTAs that can be resident at once (an SM without a partner in its GPC
// stays idle): the persistent pair kernels launch exactly that many, since clusters beyond
// it would run as a second wave after the first has finished all its units.
template <bool ROWS>
int resident_pairs() {
    static int cached[64] = {};  // per device ordinal
    int dev = 0;
    CS_CUDA(cudaGetDevice(&dev));
    int& n = cached[dev < 64 ? dev : 0];
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(num_sms() & ~1));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = Layout<ROWS, true>::kSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        CS_CUDA(cudaOccupancyMaxActiveClusters(&clusters, k_mixed_pass<ROWS, true, false, 0, false>, &cfg));
        n = std::max(1, std::min(clusters, num_sms() / 2));
    }
    return n;
}

// One CTA per SM, or (PAIR) as many clusters of two CTAs as are resident together.
template <bool ROWS, bool PAIR, bool NARROW, int TMEMA, bool ALT>
void launch_form(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tbt,
                 const PassArgs& P, cudaStream_t s) {
    if constexpr (PAIR) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(2 * resident_pairs<ROWS>()));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = Layout<ROWS, true, false, TMEMA>::kSmem;
        cfg.stream = s;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.numAttrs = 1;
        chain(cfg, attr);
        CS_CUDA(cudaLaunchKernelEx(&cfg, k_mixed_pass<ROWS, true, false, TMEMA, ALT>, ta, tb, tbt, P));
    } else {
        launch_chained(k_mixed_pass<ROWS, false, NARROW, TMEMA, ALT>, num_sms(), kThreads,
                       Layout<ROWS, false, NARROW, TMEMA>::kSmem, s, ta, tb, tbt, P);
    }
}

template <bool ROWS, bool PAIR, bool NARROW = false, int TMEMA = 0>
void launch_pass(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tbt,
                 const PassArgs& P, cudaStream_t s) {
    if constexpr (TMEMA == 0)
        launch_form<ROWS, PAIR, NARROW, 0, false>(ta, tb, tbt, P, s);
    else if (decode_alt_mode())
        launch_form<ROWS, PAIR, NARROW, TMEMA, true>(ta, tb, tbt, P, s);
    else
        launch_form<ROWS, PAIR, NARROW, TMEMA, false>(ta, tb, tbt, P, s);
}

// Per-row statistics: mu_t, exc_t = S_t - mu_t n_t (from code counts c00, c01, c10, c11),
// optional multiplier s_t, and the imputed-code table: codes 00 / 01 (missing) / 10 / 11 ->
// 2Q / q_t / Q / 0 with q_t = rint(Q mu_t), and the residual r_t = mu_t - q_t / Q.  Padding
// rows decode to zeros.
__global__ void __launch_bounds__(256)
k_row_tables(int64_t R, const double* __restrict__ mean, const int32_t* __restrict__ counts,
             const double* __restrict__ s, double* __restrict__ mu, double* __restrict__ exc,
             double* __restrict__ sv, double* __restrict__ resid, uint32_t* __restrict__ lut,
             uint8_t* __restrict__ qperm) {
    const int64_t t = (int64_t)blockIdx.x * 256 + threadIdx.x;  // r_pad is a multiple of 256
    double mt = 0.0, ex = 0.0, sc = 0.0, rs = 0.0;
    uint32_t q = 0, l = 0;
    if (t < R) {
        mt = mean[t];
        const bool ok = isfinite(mt);
        q = (uint32_t)fmin(fmax(ok ? rint(kImputeQ * mt) : 0.0, 0.0), 2.0 * kImputeQ);
        l = (uint32_t)(2 * kImputeQ) | (q << 8) | ((uint32_t)kImputeQ << 16);
        rs = ok ? __dsub_rn(mt, (double)q / kImputeQ) : 0.0;
        const int64_t c00 = counts[4 * t], c10 = counts[4 * t + 2], c11 = counts[4 * t + 3];
        ex = __dsub_rn((double)(2 * c00 + c10), __dmul_rn(mt, (double)(c00 + c10 + c11)));
        sc = s ? s[t] : 1.0;
    }
    mu[t] = mt;
    exc[t] = ex;
    sv[t] = sc;
    resid[t] = rs;
    lut[t] = l;
    qperm[(t & ~(int64_t)15) + position_of((int)(t & 15))] = (uint8_t)q;
}

// mean, counts and s on the device
void init_rows(MixedRows& r, const cs_packed_view& v, const double* mean, const int32_t* counts,
               const double* s_or_null) {
    const cudaStream_t st = 0;
    configure_kernels();
    r.R = v.n_rows;
    r.n = v.n_samples;
    // SNP rows padded to 256 as well: the rows pass runs on pairs of 128-row tiles
    r.r_pad = round_up(std::max<int64_t>(r.R, 1), 2 * kTile);
    // samples padded to 256: the samples pass runs on pairs of 128-sample tiles (packed rows
    // hold a multiple of 256 samples, so the padding tiles read missing codes)
    r.n_pad = round_up(std::max<int64_t>(r.n, 1), 2 * kTile);
    r.mu.resize(r.r_pad);
    r.exc.resize(r.r_pad);
    r.s.resize(r.r_pad);
    r.resid.resize(r.r_pad);
    r.lut.resize(r.r_pad);
    r.qperm.resize(r.r_pad / 16);
    k_row_tables<<<(unsigned)(r.r_pad / 256), 256, 0, st>>>(
        r.R, mean, counts, s_or_null, r.mu.get(), r.exc.get(), r.s.get(), r.resid.get(), r.lut.get(),
        reinterpret_cast<uint8_t*>(r.qperm.get()));
    CS_LAUNCH("row_tables");
    CS_CUDA(cudaStreamSynchronize(st));  // ready for whichever stream applies first
    // packed tiles: 32 bytes (128 samples) x 128 SNP rows; rows past R read as zeros and
    // either land in discarded output rows (rows pass) or meet zero B rows (samples pass)
    r.tm = make_map_u8(v.rows, v.stride, std::max<int64_t>(r.R, 1), v.stride, 32, kTile, false);
    r.rows = v.rows;
    r.stride = v.stride;
}

}  // namespace

// The sample-major copy of the view (once per context): n_pad rows of r_pad / 4 bytes.
void ensure_transposed(MixedRows& r, cudaStream_t s) {
    if (r.packed_t.get()) return;
    const int64_t stride_t = r.r_pad / 4;
    r.packed_t.resize((size_t)(r.n_pad * stride_t));
    {
        prof::Scope ps("transpose_packed", s, 0.0, 2.0 * (double)r.n_pad * (double)stride_t);
        const dim3 g((unsigned)(r.r_pad / kTransposeTile), (unsigned)(r.n_pad / kTransposeTile));
        k_transpose_packed<<<g, 256, 0, s>>>(r.rows, r.R, r.stride, r.packed_t.get(), stride_t);
        CS_LAUNCH("transpose_packed");
    }
    r.tm_t = make_map_u8(r.packed_t.get(), stride_t, r.n_pad, stride_t, 32, kTile, false);
}

namespace {

struct Tiling {
    int n_ctiles, kc, kc_last;
    int64_t kp;
};

// Column tiles of max_w columns and a last tile of the remainder rounded up to 16 (the MMA's
// N granularity), so that k = 266 runs 80 + 80 + 80 + 32 columns in the rows pass.  `uniform`
// (the CTA-pair kernel) gives every tile the same width instead.
Tiling tiling_for(int64_t k, int max_w, bool uniform = false) {
    Tiling t;
    t.n_ctiles = (int)((k + max_w - 1) / max_w);
    if (uniform || t.n_ctiles == 1) {
        t.kc = (int)round_up((k + t.n_ctiles - 1) / t.n_ctiles, 16);
        t.kc_last = t.kc;
    } else {
        t.kc = max_w;
        t.kc_last = (int)round_up(k - (int64_t)(t.n_ctiles - 1) * max_w, 16);
    }
    t.kp = (int64_t)t.kc * (t.n_ctiles - 1) + t.kc_last;
    return t;
}

void check_status(MixedWorkspace& ws, cudaStream_t s) {
    int status = 0;
    CS_CUDA(cudaMemcpyAsync(&status, ws.status.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    CS_CUDA(cudaStreamSynchronize(s));
    if (status != 0) {
        // cleared on the caller's stream: a non-blocking stream does not wait for the legacy one
        cudaMemsetAsync(ws.status.get(), 0, sizeof(int), s);
        cudaStreamSynchronize(s);
        fail(CS_ERR_CUDA, "tensor-core kinship kernel gave up waiting (status " +
                              std::to_string(status) + ")");
    }
}

// ---------------------------------------------------------------- pass plans and the autotuner
// A pass runs with a plan: CTA pairs or single CTAs, the layout (A in shared memory or in TMEM),
// the column-tile width cap and the number of K slices.  The default plan is the heuristic: up
// to 32 right-hand sides the four-K-block kernel (mixed_narrow_pass) or, in short slices, the narrow
// single-CTA layout with A in TMEM, 33 to 64 its 64-wide form, above that CTA pairs with A in TMEM (tiles of at most 64); slices so that about 8
// units per CTA cover the GPU.  The autotuner times the layout x width candidates of a shape
// once (shapes bucketed: rows and samples by factors of 1.25, columns to multiples of 16) and
// keeps the fastest.  It never changes the slice count (the order of the slice sums) nor, in
// the samples pass, the arithmetic form (five or six operand sets), so a tuned pass returns
// the same bits as the default one.  CS_B200_AUTOTUNE=0 turns it off.
struct PassPlan {
    bool pairs = false;
    bool narrow = false;  // single-CTA layout for column tiles of at most 32
    int tmem_a = 0;       // A operand in TMEM: 1 / 2 single CTA (tiles <= 32 / 64), 3 / 4 CTA
                          // pairs (rows / samples, tiles <= 64), 5 the five-set samples pairs,
                          // 6 mixed_narrow_pass
    int max_w = 0;
    int splits = 1;
    bool same_kernel(const PassPlan& o) const {
        return pairs == o.pairs && narrow == o.narrow && tmem_a == o.tmem_a && max_w == o.max_w;
    }
};

// the samples-pass form of a plan: six operand sets over the sample-major copy with the fixed
// dosage table (TMEMA 1, 2, 4, and 6), five otherwise
bool six_set_samples(const PassPlan& p) {
    return p.tmem_a == 1 || p.tmem_a == 2 || p.tmem_a == 4 || p.tmem_a == 6;
}

Tiling plan_tiling(const PassPlan& p, int64_t k) {
    if (p.tmem_a != 6) return tiling_for(k, p.max_w);
    const int w = (int)round_up(k, 8);
    return Tiling{1, w, w, w};
}

// Whether mixed_narrow_pass takes k columns in slices of kbs K-blocks.  Up to 24 columns it is the
// faster one at every slice length measured (us a pass, rows / samples, with it and with the 32-wide
// form: 2,000 x 10,000, k = 1 12.7 / 12.8 and 14.7 / 14.8; 10,000 x 20,000, k = 24 41.4 / 41.8 and
// 49.6 / 53.5; 40,000 x 40,000, k = 1 169 / 170 and 239 / 248, k = 24 187 / 190 and 278 / 300); with 25 to 32
// there is room for one accumulator only, which short slices (10 K-blocks: no difference) wait for,
// long ones do not (40,000 x 40,000, k = 30 212 / 205 and 279 / 300).  33 to 48 are left to the tuner (34 at
// N=50k, M=100k: pairs in the rows pass, 728 us, and this in the samples pass, 736 us).
bool narrow_pass(bool rows, int64_t k, int kb, int splits) {
    const int kbs = (kb + splits - 1) / splits;
    return mixed_narrow_fits(rows, round_up(k, 8)) && kbs >= (k <= 24 ? 2 : 16);
}

PassPlan default_plan(bool rows, int64_t tiles, int kb, int64_t k) {
    PassPlan p;
    p.pairs = use_cta_pairs(k) && tiles % 2 == 0;
    p.narrow = !p.pairs && k <= kNarrowRowsW && narrow_layouts();
    p.tmem_a = p.narrow && tmem_a_default() ? 1 : 0;
    if (tmem_a_mode() == 2 && narrow_layouts() && k > kNarrowRowsW && k <= kTmemA64W &&
        pair_mode() != 2) {
        p.pairs = false;
        p.narrow = true;
        p.tmem_a = 2;
    }
    if (rows && p.pairs && tmem_a_default() && tmem_a_pairs_default()) p.tmem_a = 3;
    if (!rows && p.pairs && tmem_a_default() && tmem_a_pairs_mode() >= 2)
        p.tmem_a = tmem_a_pairs_mode() == 3 ? 5 : 4;
    p.max_w = p.tmem_a >= 2 ? kTmemA64W
              : p.narrow ? kNarrowRowsW
                       : rows ? (p.pairs ? kPairRowsW : kRowsW) : (p.pairs ? kPairSamplesW : kSamplesW);
    const Tiling tl = tiling_for(k, p.max_w);
    p.splits = p.pairs ? choose_splits(tiles / 2 * tl.n_ctiles, kb, 4LL * num_sms())
                       : choose_splits(tiles * tl.n_ctiles, kb, 8LL * num_sms());
    if (p.tmem_a == 1 && narrow_pass(rows, k, kb, p.splits)) p.tmem_a = 6;
    return p;
}

bool autotune_env() {
    static const bool on = [] {
        const char* v = std::getenv("CS_B200_AUTOTUNE");
        return !(v && std::strcmp(v, "0") == 0);
    }();
    return on;
}

struct TuneKey {
    int rows;
    int64_t rb, nb, kb16;
    bool operator<(const TuneKey& o) const {
        return std::tie(rows, rb, nb, kb16) < std::tie(o.rows, o.rb, o.nb, o.kb16);
    }
};
struct TuneEntry {
    PassPlan plan;
    double ms_best = 0.0, ms_default = 0.0;
    int64_t R = 0, n = 0, k = 0;  // the shape it was tuned on
    int candidates = 0;
};
std::mutex g_tune_mu;
std::map<TuneKey, TuneEntry> g_tuned;

int64_t bucket(int64_t x) { return (int64_t)std::floor(std::log((double)std::max<int64_t>(x, 1)) / std::log(1.25)); }

// The plan for a pass of this shape: the tuned one (tuning it now when the shape is new and the
// pass may be timed: autotuning on, the stream not capturing, the work large enough to matter),
// or the default.  `run` executes the pass with a plan.
template <class Run>
PassPlan choose_plan(bool rows, bool allow, int64_t R, int64_t n, int64_t k, int64_t tiles, int kb,
                     cudaStream_t s, Run&& run) {
    const PassPlan def = default_plan(rows, tiles, kb, k);
    if (!allow || !autotune_env() || 2.0 * (double)R * (double)n * (double)k < 2e10) return def;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return def;
    const TuneKey key{rows ? 1 : 0, bucket(R), bucket(n), (k + 15) / 16};
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = g_tuned.find(key);
        if (it != g_tuned.end()) {
            PassPlan p = it->second.plan;
            p.splits = def.splits;
            return p;
        }
    }
    std::vector<PassPlan> cands;
    const int mode = pair_mode();
    if (mode != 2 && narrow_layouts())
        for (int w = 16; w <= kNarrowRowsW; w += 16)
            for (int t = 0; t < (tmem_a_default() ? 2 : 1); ++t) {
                PassPlan p;
                p.narrow = true;
                p.tmem_a = t;
                p.max_w = w;
                p.splits = def.splits;
                cands.push_back(p);
            }
    if (mode != 0 && tiles % 2 == 0 && num_sms() >= 2 && tmem_a_default())
        for (int w = 48; w <= kTmemA64W; w += 16) {
            PassPlan p;
            p.pairs = true;
            p.tmem_a = rows ? 3 : (def.tmem_a == 5 ? 5 : 4);
            p.max_w = w;
            p.splits = def.splits;
            cands.push_back(p);
        }
    if (mode != 2 && narrow_layouts() && tmem_a_default() && narrow_pass(rows, k, kb, def.splits)) {
        PassPlan p;
        p.narrow = true;
        p.tmem_a = 6;
        p.max_w = k <= kNarrowRowsW ? kNarrowRowsW : kTmemA64W;
        p.splits = def.splits;
        cands.push_back(p);
    }
    if (mode != 2 && narrow_layouts() && tmem_a_default() && k > kNarrowRowsW)
        for (int w = 48; w <= kTmemA64W; w += 16) {
            PassPlan p;
            p.narrow = true;
            p.tmem_a = 2;
            p.max_w = w;
            p.splits = def.splits;
            cands.push_back(p);
        }
    for (int pr = 0; pr < 2; ++pr) {
        if (pr == 1 && (mode == 0 || tiles % 2 != 0 || num_sms() < 2)) continue;
        if (pr == 0 && mode == 2) continue;
        const int cap_w = rows ? (pr ? kPairRowsW : kRowsW) : (pr ? kPairSamplesW : kSamplesW);
        int last_kc = -1, last_kl = -1, last_ct = -1;
        for (int w = 32; w <= cap_w; w += 16) {
            const Tiling tl = tiling_for(k, w);
            // a wider cap that gives the same tiling as a narrower one is the same plan
            if (tl.kc == last_kc && tl.kc_last == last_kl && tl.n_ctiles == last_ct &&
                !(pr == (def.pairs ? 1 : 0) && !def.narrow && w == def.max_w))
                continue;
            last_kc = tl.kc;
            last_kl = tl.kc_last;
            last_ct = tl.n_ctiles;
            PassPlan p;
            p.pairs = pr == 1;
            p.max_w = w;
            p.splits = def.splits;
            cands.push_back(p);
        }
    }
    // Samples-pass plans over the sample-major copy with the fixed dosage table compute the
    // six-set form (W and mu o W), the others the five-set form: only plans of the default's
    // form are candidates, so a tuned pass returns the same bits as the default one.
    if (!rows) {
        const bool six = six_set_samples(def);
        cands.erase(std::remove_if(cands.begin(), cands.end(),
                                   [six](const PassPlan& p) { return six_set_samples(p) != six; }),
                    cands.end());
    }
    cudaEvent_t e0, e1;
    CS_CUDA(cudaEventCreate(&e0));
    CS_CUDA(cudaEventCreate(&e1));
    TuneEntry best;
    best.plan = def;
    best.ms_best = 1e30;
    try {
        run(def);  // warm: maps, function attributes, operand buffers
        bool have_default = false;
        for (const PassPlan& p : cands) have_default = have_default || p.same_kernel(def);
        if (!have_default) cands.insert(cands.begin(), def);
        for (const PassPlan& p : cands) {
            CS_CUDA(cudaEventRecord(e0, s));
            run(p);
            CS_CUDA(cudaEventRecord(e1, s));
            CS_CUDA(cudaEventSynchronize(e1));
            float ms = 0.f;
            CS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
            if (p.same_kernel(def)) best.ms_default = ms;
            if (ms < best.ms_best) {
                best.ms_best = ms;
                best.plan = p;
            }
        }
    } catch (...) {
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    best.R = R;
    best.n = n;
    best.k = k;
    best.candidates = (int)cands.size();
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tuned.emplace(key, best);
    }
    return best.plan;
}

// Rows pass over a MixedRows context on X (n x k):
//   u_tc = sum_i (G_ti - mu_t)[obs] x_ic  (mean-imputed centred dosages)
// With Wt: W^T (column-major, R per column) = s_t^2 u and its maxima for the samples operand;
// otherwise out(pos[t] or t, c) = s_t u.
template <class T>
void rows_pass_plan(const PassPlan& plan, MixedRows& r, MixedWorkspace& ws, Strided<const T> X,
                    int64_t k, double* Wt, const int32_t* pos, StridedOut out, cudaStream_t s) {
    const int64_t tiles = r.r_pad / kTile;
    const bool pairs = plan.pairs;
    const Tiling tl = plan_tiling(plan, k);
    const int64_t n = r.n, R = r.R, n_pad = r.n_pad, r_pad = r.r_pad, kp = tl.kp;
    const int kb = (int)(n_pad / kKBlock);
    const int kbs = (kb + plan.splits - 1) / plan.splits;
    const int splits = (kb + kbs - 1) / kbs;  // no empty slice
    if (kbs > kMaxKbPerAccum) fail(CS_ERR_UNSUPPORTED, "rows pass: K slice exceeds the exact int32 range");
    const int64_t nst = (n + kStatRows - 1) / kStatRows;  // chunks of the column stats
    ws.b1.resize(3 * kp * n_pad);
    ws.part.resize((int64_t)splits * kp * r_pad);
    ws.colpart.resize(((n + kStatTile - 1) / kStatTile + 2 * nst) * k);
    const MixedColumns C = ws.columns(k, s);
    if (!ws.status.get()) {
        ws.status.resize(1);
        // on the pass's own stream, so the kernel never reads the pool's previous contents
        CS_CUDA(cudaMemsetAsync(ws.status.get(), 0, sizeof(int), s));
    }
    // boxes of one column tile's rows (pairs: half of them)
    const int box = pairs ? tl.kc / 2 : tl.kc, box_last = pairs ? tl.kc_last / 2 : tl.kc_last;
    const int64_t key = ((kp * 1000003 + n_pad) * 131 + box_last) * 131 + box;
    if (ws.tm_b1_base != ws.b1.get() || ws.tm_b1_key != key) {
        ws.tm_b1 = make_map_u8(ws.b1.get(), n_pad, 3 * kp, n_pad, kKBlock, box, true);
        ws.tm_b1t = make_map_u8(ws.b1.get(), n_pad, 3 * kp, n_pad, kKBlock, box_last, true);
        ws.tm_b1_base = ws.b1.get();
        ws.tm_b1_key = key;
    }
    {
        prof::Scope ps("mixed_prep_rows_operand", s, 0.0, 24.0 * n * k + 3.0 * kp * n_pad);
        if (n <= kWholeRows) {
            const unsigned threads = (unsigned)round_up(n_pad / 16, 32);
            launch_chained(k_rows_operand_whole<T>, (unsigned)kp, threads, 8 * (n_pad + n_pad / 16 + 16), s, X, n,
                           k, kp, n_pad, C, ws.b1.get());
        } else {
            int kc = 1;
            while (X.rs != 1 && kc < k && kc < 32) kc *= 2;
            const int64_t per = 32 / kc;  // chunks per block
            launch_chained(k_col_stats<T>, dim3((unsigned)((nst + per - 1) / per), (unsigned)((k + kc - 1) / kc)),
                           256, 0, s, X, n, k, kc, nst, ws.colpart.get(), C);
            if (kp <= 16)
                launch_chained(k_split_rows_operand<T, 4, 512>,
                               dim3((unsigned)((n_pad + 511) / 512), (unsigned)((kp + 3) / 4)), 128, 0, s, X, n, k,
                               kp, n_pad, C, ws.b1.get(), ws.colpart.get());
            else
                launch_chained(k_split_rows_operand<T, 16, 256>,
                               dim3((unsigned)(n_pad / 256), (unsigned)((kp + 15) / 16)), 256, 0, s, X, n, k, kp,
                               n_pad, C, ws.b1.get(), ws.colpart.get());
        }
        CS_LAUNCH("mixed rows operand");
    }
    PassArgs P{};
    P.n_tiles = (int)tiles;
    P.n_ctiles = tl.n_ctiles;
    P.n_splits = splits;
    P.kb_total = kb;
    P.kb_per_split = kbs;
    P.kc = tl.kc;
    P.kc_last = tl.kc_last;
    P.kp = (int)kp;
    P.lut = r.lut.get();
    P.resid = r.resid.get();
    P.part = ws.part.get();
    P.ld = r_pad;
    P.status = ws.status.get();
    P.poll_ns = poll_sleep_ns();
    P.poll_dec_ns = poll_dec_sleep_ns();
    {
        // algorithmic work: 2 n R k flops, one pass over the packed rows
        prof::Scope ps("kinship_rows_tc", s, 2.0 * (double)n * (double)R * (double)k,
                       (double)R * (double)((n + 3) / 4));
        if (plan.tmem_a == 6)
            mixed_narrow_pass(true, r, ws.b1.get(), kp, splits, kbs, nullptr, ws.part.get(), ws.status.get(),
                              poll_sleep_ns(), s);
        else if (pairs && plan.tmem_a == 3)
            launch_pass<true, true, false, 3>(r.tm, ws.tm_b1, ws.tm_b1t, P, s);
        else if (pairs)
            launch_pass<true, true>(r.tm, ws.tm_b1, ws.tm_b1t, P, s);
        else if (plan.narrow && plan.tmem_a == 2)
            launch_pass<true, false, true, 2>(r.tm, ws.tm_b1, ws.tm_b1t, P, s);
        else if (plan.narrow && plan.tmem_a)
            launch_pass<true, false, true, 1>(r.tm, ws.tm_b1, ws.tm_b1t, P, s);
        else if (plan.narrow)
            launch_pass<true, false, true>(r.tm, ws.tm_b1, ws.tm_b1t, P, s);
        else
            launch_pass<true, false>(r.tm, ws.tm_b1, ws.tm_b1t, P, s);
        CS_LAUNCH("kinship_rows_tc");
    }
    {
        prof::Scope ps("mixed_reduce_rows", s, 0.0, 8.0 * splits * kp * R + 8.0 * R * k);
        if (Wt)
            launch_chained(k_reduce_rows, dim3((unsigned)((R + 1023) / 1024), (unsigned)k), 256, 0, s,
                           ws.part.get(), splits, kp, r_pad, R, r.s.get(), r.exc.get(), r.mu.get(), C, Wt);
        else
            launch_chained(k_reduce_rows_out, dim3((unsigned)((R + 31) / 32), (unsigned)((k + 31) / 32)), 256,
                           0, s, ws.part.get(), splits, kp, r_pad, R, k, r.s.get(), r.exc.get(), r.mu.get(),
                           pos, C, out);
        CS_LAUNCH("reduce_rows");
    }
}

// Samples pass: Y (n x k) = (Z W) / M for W^T (k x R, column-major) with the per-column maxima that
// the rows pass (or the gather) left.
template <class T>
void samples_pass_plan(const PassPlan& plan, MixedRows& r, MixedWorkspace& ws, const double* Wt,
                       int64_t k, double inv_m, Strided<T> Y, cudaStream_t s) {
    const int64_t tiles = r.n_pad / kTile;
    const bool pairs = plan.pairs;
    const Tiling tl = plan_tiling(plan, k);
    const int64_t n = r.n, R = r.R, n_pad = r.n_pad, r_pad = r.r_pad, kp = tl.kp;
    const int kb = (int)(r_pad / kKBlock);
    const int kbs = (kb + plan.splits - 1) / plan.splits;
    const int splits = (kb + kbs - 1) / kbs;  // no empty slice
    if (kbs > kMaxKbPerAccum) fail(CS_ERR_UNSUPPORTED, "samples pass: K slice exceeds the exact int32 range");
    const int nrb = (int)((r_pad + 2047) / 2048);
    // A in TMEM: over the sample-major copy, B in the decoded K order; six sets with the fixed
    // dosage table, five with the imputed codes (TMEMA = 5)
    const bool tmem_a = plan.tmem_a != 0;  // narrow single-CTA forms, or 4 / 5 on CTA pairs
    const bool six = six_set_samples(plan);
    const int pieces = six ? 6 : 5;
    if (tmem_a) ensure_transposed(r, s);
    ws.b2.resize(pieces * kp * r_pad);
    ws.part.resize((int64_t)splits * kp * n_pad);
    ws.colpart.resize((int64_t)nrb * k);
    ws.inv_f.resize(kp);
    ws.c0.resize(k);
    // boxes of one column tile's rows (pairs: half of them)
    const int box = pairs ? tl.kc / 2 : tl.kc, box_last = pairs ? tl.kc_last / 2 : tl.kc_last;
    const int64_t key = (((kp * 1000003 + r_pad) * 131 + box_last) * 131 + box) * 7 + pieces;
    if (ws.tm_b2_base != ws.b2.get() || ws.tm_b2_key != key) {
        ws.tm_b2 = make_map_u8(ws.b2.get(), r_pad, pieces * kp, r_pad, kKBlock, box, true);
        ws.tm_b2t = make_map_u8(ws.b2.get(), r_pad, pieces * kp, r_pad, kKBlock, box_last, true);
        ws.tm_b2_base = ws.b2.get();
        ws.tm_b2_key = key;
    }
    {
        prof::Scope ps("mixed_prep_samples_operand", s, 0.0, 8.0 * R * k + pieces * kp * r_pad);
        const dim3 g((unsigned)nrb, (unsigned)kp);
        const MixedColumns C = ws.columns(k, s);
        auto split = [&](auto kern) {
            launch_chained(kern, g, 128, 0, s, Wt, R, k, kp, r_pad, r.mu.get(), r.resid.get(), C, ws.b2.get(),
                           ws.inv_f.get(), ws.colpart.get(), ws.c0.get());
        };
        if (six) split(k_split_samples_operand<true, true>);
        else if (tmem_a) split(k_split_samples_operand<false, true>);
        else split(k_split_samples_operand<false, false>);
        CS_LAUNCH("mixed samples operand");
    }
    PassArgs P{};
    P.n_tiles = (int)tiles;
    P.n_ctiles = tl.n_ctiles;
    P.n_splits = splits;
    P.kb_total = kb;
    P.kb_per_split = kbs;
    P.kc = tl.kc;
    P.kc_last = tl.kc_last;
    P.kp = (int)kp;
    P.lut = r.lut.get();
    P.qperm = r.qperm.get();
    P.inv_f = ws.inv_f.get();
    P.part = ws.part.get();
    P.ld = n_pad;
    P.status = ws.status.get();
    P.poll_ns = poll_sleep_ns();
    P.poll_dec_ns = poll_dec_sleep_ns();
    {
        prof::Scope ps("kinship_samples_tc", s, 2.0 * (double)n * (double)R * (double)k,
                       (double)R * (double)((n + 3) / 4));
        if (plan.tmem_a == 6)
            mixed_narrow_pass(false, r, ws.b2.get(), kp, splits, kbs, ws.inv_f.get(), ws.part.get(),
                              ws.status.get(), poll_sleep_ns(), s);
        else if (pairs && plan.tmem_a == 5)
            launch_pass<false, true, false, 5>(r.tm_t, ws.tm_b2, ws.tm_b2t, P, s);
        else if (pairs && tmem_a)
            launch_pass<false, true, false, 4>(r.tm_t, ws.tm_b2, ws.tm_b2t, P, s);
        else if (pairs)
            launch_pass<false, true>(r.tm, ws.tm_b2, ws.tm_b2t, P, s);
        else if (tmem_a && plan.tmem_a == 2)
            launch_pass<false, false, true, 2>(r.tm_t, ws.tm_b2, ws.tm_b2t, P, s);
        else if (tmem_a)
            launch_pass<false, false, true, 1>(r.tm_t, ws.tm_b2, ws.tm_b2t, P, s);
        else if (plan.narrow)
            launch_pass<false, false, true>(r.tm, ws.tm_b2, ws.tm_b2t, P, s);
        else
            launch_pass<false, false>(r.tm, ws.tm_b2, ws.tm_b2t, P, s);
        CS_LAUNCH("kinship_samples_tc");
    }
    {
        prof::Scope ps("mixed_reduce_samples", s, 0.0, 8.0 * splits * kp * n + 8.0 * n * k);
        launch_chained(k_reduce_samples<T>, dim3((unsigned)((n + 31) / 32), (unsigned)((k + 31) / 32)), 256, 0,
                       s, ws.part.get(), splits, kp, n_pad, n, k, ws.c0.get(), inv_m, Y);
        CS_LAUNCH("reduce_samples");
    }
}

template <class T>
void rows_pass(MixedRows& r, MixedWorkspace& ws, Strided<const T> X, int64_t k, double* Wt,
               const int32_t* pos, StridedOut out, cudaStream_t s, bool allow_tune) {
    const int64_t tiles = r.r_pad / kTile;
    const int kb = (int)(r.n_pad / kKBlock);
    const PassPlan plan = choose_plan(true, allow_tune, r.R, r.n, k, tiles, kb, s, [&](const PassPlan& p) {
        rows_pass_plan(p, r, ws, X, k, Wt, pos, out, s);
    });
    rows_pass_plan(plan, r, ws, X, k, Wt, pos, out, s);
}

template <class T>
void samples_pass(MixedRows& r, MixedWorkspace& ws, const double* Wt, int64_t k, double inv_m,
                  Strided<T> Y, cudaStream_t s, bool allow_tune, bool sample_major_copy) {
    const int64_t tiles = r.n_pad / kTile;
    const int kb = (int)(r.r_pad / kKBlock);
    PassPlan plan = choose_plan(false, allow_tune && sample_major_copy, r.R, r.n, k, tiles, kb, s,
                                [&](const PassPlan& p) {
                                    samples_pass_plan(p, r, ws, Wt, k, inv_m, Y, s);
                                });
    if (!sample_major_copy && plan.tmem_a) {
        // A in shared memory (narrow up to 32 columns, otherwise the general layouts): the same
        // int32 sums without the copy; the slice count stays the default plan's
        plan.tmem_a = 0;
        if (plan.max_w > kNarrowSamplesW) {
            plan.narrow = false;
            plan.pairs = use_cta_pairs(k) && tiles % 2 == 0;
            plan.max_w = plan.pairs ? kPairSamplesW : kSamplesW;
        }
    }
    samples_pass_plan(plan, r, ws, Wt, k, inv_m, Y, s);
}

}  // namespace

static MixedOperator* mixed_for(cs_kinship* op) {
    if (op->mixed) return op->mixed;
    auto* m = new MixedOperator();
    try {
        init_rows(m->rows, op->view, op->d_mean.get(), op->d_counts.get(), op->d_inv_std.get());
    } catch (...) {
        delete m;
        throw;
    }
    op->mixed = m;
    return m;
}

MixedRows& mixed_rows_for(cs_kinship* op) { return mixed_for(op)->rows; }

template <class T>
void kinship_apply_mixed(cs_kinship* op, Strided<const T> X, int64_t k, Strided<T> Y, cudaStream_t s) {
    if (k <= 0) return;
    const int64_t n = op->rows, R = op->n_active;
    if (R == 0) {
        const bool cm = Y.rs == 1;
        CS_CUDA(cudaMemset2DAsync(Y.p, sizeof(T) * (cm ? Y.cs : Y.rs), 0, sizeof(T) * (cm ? n : k),
                                  cm ? k : n, s));
        return;
    }
    MixedOperator* m = mixed_for(op);
    m->ws.W.resize(R * k);
    // W^T = s o s o (Z-centred)^T X: the rows pass output already scaled for the samples pass
    m->last_k = 0;
    rows_pass(m->rows, m->ws, X, k, m->ws.W.get(), nullptr, StridedOut{}, s, op->autotune);
    samples_pass(m->rows, m->ws, m->ws.W.get(), k, 1.0 / (double)op->num_variants, Y, s, op->autotune,
                 op->sample_major_copy);
    if (!op->defer_checks) check_status(m->ws, s);
    m->last_k = k;
}
void check_mixed(cs_kinship* op, cudaStream_t s) {
    if (op->mixed && op->mixed->ws.status.get()) check_status(op->mixed->ws, s);
}
void clear_mixed(cs_kinship* op, cudaStream_t s) {
    if (op->mixed && op->mixed->ws.status.get())
        CS_CUDA(cudaMemsetAsync(op->mixed->ws.status.get(), 0, sizeof(int), s));
}

template void kinship_apply_mixed<double>(cs_kinship*, Strided<const double>, int64_t, Strided<double>,
                                          cudaStream_t);
template void kinship_apply_mixed<float>(cs_kinship*, Strided<const float>, int64_t, Strided<float>,
                                         cudaStream_t);

// GenotypeMatrix::multiply_Zt_v on tensor cores.
void mixed_multiply_zt(cs_kinship* op, StridedIn X, int64_t k, StridedOut U, cudaStream_t s) {
    if (k <= 0 || op->n_active == 0) return;
    MixedOperator* m = mixed_for(op);
    m->last_k = 0;
    rows_pass(m->rows, m->ws, X, k, nullptr, op->d_view_pos.get(), U, s, op->autotune);
    check_status(m->ws, s);
}

// GenotypeMatrix::multiply_Z_v on tensor cores.
void mixed_multiply_z(cs_kinship* op, StridedIn V, int64_t k, StridedOut Y, cudaStream_t s) {
    if (k <= 0) return;
    const int64_t R = op->n_active;
    MixedOperator* m = mixed_for(op);
    m->last_k = 0;
    MixedWorkspace& ws = m->ws;
    if (!ws.status.get()) {
        ws.status.resize(1);
        CS_CUDA(cudaMemsetAsync(ws.status.get(), 0, sizeof(int), s));
    }
    ws.W.resize(R * k);
    const MixedColumns C = ws.columns(k, s);
    CS_CUDA(cudaMemsetAsync(C.max_w, 0, 8 * k, s));
    CS_CUDA(cudaMemsetAsync(C.max_wmu, 0, 8 * k, s));
    {
        prof::Scope ps("mixed_gather_operand", s, 0.0, 16.0 * R * k);
        launch_chained(k_gather_operand, dim3((unsigned)((R + 1023) / 1024), (unsigned)k), 256, 0, s, V, R,
                       op->d_view_pos.get(), m->rows.s.get(), m->rows.mu.get(), C, ws.W.get());
        CS_LAUNCH("gather_operand");
    }
    samples_pass(m->rows, ws, ws.W.get(), k, 1.0, Y, s, op->autotune, op->sample_major_copy);
    check_status(ws, s);
}

// The autotuner's table as JSON (reported with the profile summary).
std::string autotune_json() {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    std::string out = "[";
    char buf[384];
    bool first = true;
    for (const auto& kv : g_tuned) {
        const TuneEntry& e = kv.second;
        std::snprintf(buf, sizeof buf,
                      "%s{\"pass\": \"%s\", \"R\": %lld, \"n\": %lld, \"k\": %lld, "
                      "\"pairs\": %s, \"narrow\": %s, \"tmem_a\": %s, \"max_width\": %d, \"slices\": %d, "
                      "\"candidates\": %d, \"ms_best\": %.4f, \"ms_default\": %.4f}",
                      first ? "" : ", ", kv.first.rows ? "rows" : "samples", (long long)e.R,
                      (long long)e.n, (long long)e.k, e.plan.pairs ? "true" : "false",
                      e.plan.narrow ? "true" : "false",
                      e.plan.tmem_a == 6   ? "\"48\""
                      : e.plan.tmem_a == 5 ? "\"pair64_five\"" : e.plan.tmem_a >= 3 ? "\"pair64\""
                      : e.plan.tmem_a == 2 ? "64" : e.plan.tmem_a ? "32" : "false",
                      e.plan.max_w,
                      e.plan.splits, e.candidates,
                      e.ms_best, e.ms_default);
        out += buf;
        first = false;
    }
    return out + "]";
}

const double* mixed_rows_output(const cs_kinship* op, int64_t* R, int64_t* k) {
    if (!op->mixed || op->mixed->last_k == 0) return nullptr;
    *R = op->n_active;
    *k = op->mixed->last_k;
    return op->mixed->ws.W.get();
}

// Scan projection on tensor cores: T[t][c] = sum_i (g_ti - m_t)[observed] B[i][c] for every row
// of a packed view (the analysed samples), m_t = per-row mean of the observed dosages.
struct MixedScan {
    MixedRows rows;
    MixedWorkspace ws;
    SliceOperator* slices = nullptr;  // scan_project_fp64's
    ~MixedScan() { destroy_slices(slices); }
};

MixedScan* mixed_scan_create(const cs_packed_view& v, const double* row_mean, const int32_t* counts) {
    auto* m = new MixedScan();
    try {
        DeviceBuffer<double> d_mean;
        DeviceBuffer<int32_t> d_counts;
        d_mean.resize(std::max<int64_t>(1, v.n_rows));
        d_counts.resize(std::max<int64_t>(1, 4 * v.n_rows));
        CS_CUDA(cudaMemcpy(d_mean.get(), row_mean, 8 * v.n_rows, cudaMemcpyHostToDevice));
        CS_CUDA(cudaMemcpy(d_counts.get(), counts, 16 * v.n_rows, cudaMemcpyHostToDevice));
        init_rows(m->rows, v, d_mean.get(), d_counts.get(), nullptr);
    } catch (...) {
        delete m;
        throw;
    }
    return m;
}

void mixed_scan_destroy(MixedScan* m) { delete m; }

void mixed_scan_project(MixedScan* m, const double* B, int64_t ldb, int64_t k, double* T,
                        int64_t ldt, cudaStream_t s) {
    rows_pass(m->rows, m->ws, StridedIn{B, ldb, 1}, k, nullptr, nullptr, StridedOut{T, ldt, 1}, s, true);
    check_status(m->ws, s);
}

bool scan_project_fp64(MixedScan* m, const double* B, int64_t ldb, int64_t k, double* T, int64_t ldt,
                       cudaStream_t s) {
    return scan_project_slices(m->slices, m->rows, StridedIn{B, ldb, 1}, k, StridedOut{T, ldt, 1}, s);
}

}  // namespace cs
