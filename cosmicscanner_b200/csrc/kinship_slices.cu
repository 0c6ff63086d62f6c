// The FP64 form of the kinship products on the int8 tensor cores.
//
// Arithmetic.  Each right-hand side column becomes a 63-bit fixed-point column (one power of two
// per column, the largest element just below 2^63), split into eight int8 digits of base 256
// (balanced, -128..127): x = 2^-e sum_p d_p 256^(7-p) with an error of at most 2^-63 of the
// column's maximum.  Genotype codes are small integers, so every product and every sum of the
// int8 MMAs is exact in int32, the eight sums of an output are put together in two 64-bit
// integers (three digits and five), and the centring by the SNP means is done on those before the
// single conversion to FP64.  (Splitting a floating-point operand into slices whose products
// accumulate exactly: Ozaki, Ogita, Oishi, Rump 2012; on integer matrix units: Ootomo, Ozaki,
// Yokota 2024.)  An FP64 sum of K products carries a rounding error of the order of 2^-53 sqrt(K)
// of the result at best; here only the operand's own rounding remains.
//   Eight digits and not seven: an element 2^-b of its column's maximum keeps 63 - b bits, and b
// is large where a column is uneven.  W = s^2 o Z^T x of the samples pass is: a variant that one
// sample carries has s^2 = n.  With 5 % of such variants among 3,000 at 6,000 samples K x was off by
// 1.5e-15 to 2.9e-15 with seven digits, 1.1e-15 as FP64 sums, 8e-17 with eight.  An even column (range_uneven)
// needs no more than seven; its last digit is zero, whatever its neighbours are, and its results are those of
// seven digits.  A product of 266 columns at 18,009 x 27,006 takes 2.76 ms where all are even, 2.90 otherwise, and took
// 2.73 with seven digits.
//
//   rows pass     63 u_t / s_t = sum_obs 63 G x + sum_miss q_t x + (63 mu_t - q_t) sum_miss x
//                                - 63 mu_t sum x
//     with the imputed-code tile (63 G, or q_t = rint(63 mu_t) for a missing call) against the
//     digits and the missing-indicator tile against all but the column's last (|63 mu_t - q_t| <= 1/2
//     takes its place); 63 mu_t and the sums are carried in two doubles each, so the
//     difference of the large terms does not round.
//   samples pass  M y_i = sum_t G w + sum_miss (mu w) - sum_t (mu w),  w = s o U
//     with w and mu o w split at one scale (eight digits each) into the same accumulators; the
//     last sum is taken over the same digits, so that a missing call cancels exactly.
//
// Kernel.  The passes keep the genotype tiles in tensor memory (A, K-major: the packed rows in
// the rows pass, the operator's sample-major copy in the samples pass) and stream the digits (B)
// through shared memory; kinship_mixed.cu has the same structure at three digits.  Warp 0 loads
// B, warp 2 the packed tiles (both TMA), warps 8.. decode in groups of four that take K-blocks
// in turn (a warp may touch only its own quarter of the TMEM lanes), warp 1 issues the MMAs from
// one thread, warps 4-7 drain the accumulators.  The MMA thread's own instructions set the pace of
// narrow blocks, so a K-block's B rows and its decoded tile share one ring stage (one wait, one commit),
// and a packed tile spans four K-blocks.  What bounds them now is the decode: 13 integer
// operations per 16 genotypes at half rate are 208 of the 400 clocks a K-block takes, the ring and
// wait instructions of all warps about 120 more (ncu: ALU pipe 70 % busy, tensor pipe 14 %, DRAM a
// third of its rate).  Wide blocks come nearer to the MMAs (N / 2 clocks each): 512 of the 660 clocks that
// a K-block of a 16-column rows tile takes, and a 32-column samples tile is at theirs, 896 or 1024.  Wide blocks run
// on CTA pairs (cta_group::2): each CTA holds half of the B rows, which halves the L2 reads of B that would
// otherwise bound a wide block (64 bytes per clock and SM at the full MMA rate).
//
// Column tiles.  Up to 4 columns a column's digits sit in eight adjacent B rows (N = 8 w);
// wider tiles are digit-major in widths of 8 per CTA.  TMEM (512 columns) holds the
// accumulators (rows: main and missing-call sums apart, 15 per column; samples: 8) and the
// A stages (64 columns each).
//
// The mixed form's passes of up to 48 columns run on the same kernel with three digits (mixed_narrow_pass):
// it decodes a packed tile of four K-blocks at a time where kinship_mixed.cu's kernels take one, which
// is what bounds few columns.  At N=40k, M=40k, 24 columns a pass takes 187 us (rows) and 190 (samples)
// instead of 278 and 300.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <string>

#include "chain.cuh"
#include "cs_internal.h"
#include "mixed_internal.h"
#include "slices_internal.h"
#include "sm100.cuh"

namespace cs {

namespace {

using namespace sm100;

constexpr int kTile = kTcTile;
constexpr int kKBlock = 128;
constexpr int kDigits = 8;
constexpr int kEpiWarp0 = 4, kDecWarp0 = 8;
// decoder groups of four warps: G, by kernel
constexpr int threads_for(int groups) { return (kDecWarp0 + 4 * groups) * 32; }
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kAStage = 64;              // TMEM columns of a decoded K-block
constexpr int kMaxStages = 16;
constexpr int kPackedKb = 4;                  // K-blocks of a packed tile: one 128-byte row each
constexpr int kPackedBytes = kTile * 32 * kPackedKb;
constexpr int kMaxKbPerAccum = 1024;          // 1024 * 128 * 126 * 128 < 2^31
constexpr int kBarBytes = (4 * kMaxStages + 2 * 2 + 1) * 8 + 8;
constexpr int kSmemMax = 227 * 1024;
constexpr int kPassStatusOk = kOk;

// The mixed form uses hw for the global B rows from one set to the next, and mu for mu - q / 63 (rows
// pass, per SNP row) or 1 / f (samples pass, per column): three fields more, at the end, made the passes
// of one column 7 and 12 % longer (482 and 502 us for 449 at N=50k, M=100k) with the same kernel code.
struct SliceArgs {
    int n_tiles, n_ctiles, n_splits;
    int kb_total, kb_per_split;
    int k, w, hw;           // columns, columns per tile, per CTA
    int cmajor;             // digits of a column adjacent (eight B rows per column)
    int nm, nx;             // MMA N: main (and samples' second) product, rows' missing product
    int set_rows;           // B rows of one set in this CTA's shared memory
    int sd, sp, nb;         // ring depths: stages (B rows + decoded tile), packed tiles, accumulators
    uint32_t acc_stride, a0;
    const uint32_t* lut;    // rows pass: imputed code of each 2-bit code, per SNP row
    const double* mu;       // rows pass: per SNP row
    const longlong2* ksum;  // [n_splits][k]: sum of the fixed-point values (hi, lo) per slice
    double* part;           // [n_splits][k][ld]
    int64_t ld;
    int* status;
    uint32_t poll_ns, poll_dec_ns;
};

// hi 2^40 + lo of the eight digit sums of one output: hi of three digits, below 2^47, so that its
// conversion is exact and a difference of large terms does not round; lo of five, at most
// 126 * 2^17 (K) * 2^39.006 < 2^63.
constexpr double kLowDigits = 1099511627776.0;  // 2^40
__device__ __forceinline__ void join_digits(const int32_t (&m)[8], int64_t& hi, int64_t& lo) {
    hi = lo = 0;
#pragma unroll
    for (int p = 0; p < kDigits; ++p) {
        if (p < 3) hi = hi * 256 + m[p];
        else lo = lo * 256 + m[p];
    }
}

// Per SNP row: 63 mu in two doubles and 63 mu - q.
struct RowCentre {
    double ah, al, b;
};

// 63 u 2^e of one rows-pass output: M and X the joined main and missing-call sums, S the sum
// of the slice's fixed-point values.
__device__ __forceinline__ double rows_value(const RowCentre& c, int64_t mh, int64_t ml, int64_t xh,
                                             int64_t xl, double sh, double sl) {
    const double m1 = (double)mh * kLowDigits, m0 = (double)ml;
    const double x = fma((double)xh, kLowDigits, (double)xl);
    const double p = c.ah * sh, pe = fma(c.ah, sh, -p);
    const double d = m1 - p;
    return d + (((m0 - c.ah * sl) - pe) + fma(c.b, x, c.al * (x - (sh + sl))));
}

// DIGITS = 8: the FP64 form.  DIGITS = 3: the mixed form of kinship_mixed.cu (pieces of base 254,
// one column tile on single CTAs), with that file's operands, K slices (any number of K-blocks)
// and epilogue arithmetic, so that the bits are those of its own kernels.
template <bool ROWS, bool PAIR, int G, int DIGITS>
__global__ void __launch_bounds__(threads_for(G), 1)
k_slice_pass(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
             const SliceArgs P) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    constexpr int kSets = ROWS ? 1 : 2;
    const int b_bytes = kSets * P.set_rows * 128;  // a multiple of 1024
    unsigned char* smem_b = smem;
    unsigned char* smem_p = smem + P.sd * b_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_p + P.sp * kPackedBytes);
    uint64_t* full = bars;                    // stage ready: B rows landed (1 arrival + tx bytes) and
                                              // tile decoded (one arrival per warp of a group); pair:
                                              // the leader's also counts the other CTA's decoders and
                                              // its landed B rows, the other CTA's only its B rows
    uint64_t* empty = full + kMaxStages;      // MMAs reading the stage done (commit)
    uint64_t* full_p = empty + kMaxStages;    // packed tile landed
    uint64_t* empty_p = full_p + kMaxStages;  // packed tile read (one arrival per decoder warp)
    uint64_t* acc_full = empty_p + kMaxStages;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* drained = acc_empty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;
    const int SD = P.sd, SP = P.sp, NB = P.nb;
    if (threadIdx.x == 0) {
        for (int d = 0; d < SD; ++d) {
            mbar_init(&full[d], PAIR ? (rank == 0 ? 10 : 1) : 5);
            mbar_init(&empty[d], 1);
        }
        for (int s = 0; s < SP; ++s) {
            mbar_init(&full_p[s], 1);
            mbar_init(&empty_p[s], 4 * G);
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
    // Pairs, whose time is the MMAs': nothing to do where no column is inside the fixed-point range, no MMAs for
    // an eighth digit that no column has (the ranges stand in front of the sums: SliceCall).  A product of 266
    // even columns at 18,009 x 27,006 takes 2.76 ms with that and 2.90 without.  In the single-CTA kernels, at
    // their limit of 80 registers, the same cost a pass of one column 2 % (459 us for 450).
    int live = 1, eighth = 1;
    if constexpr (PAIR) {
        const ColumnRange* const range = reinterpret_cast<const ColumnRange*>(P.ksum) - P.k;
        int in = 0, uneven = 0;
        for (int c = threadIdx.x; c < P.k; c += (int)blockDim.x) {
            in |= !range_excluded(range[c]);
            uneven |= range_uneven(range[c]);
        }
        cluster_sync_all();
        live = __syncthreads_or(in);
        eighth = __syncthreads_or(uneven);
    } else {
        __syncthreads();
    }
    const int nm = eighth ? P.nm : 2 * (((kDigits - 1) * P.hw + 15) / 16 * 16);
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    // A unit is one M tile (pair: two) x one column tile x one K slice, column tiles fastest so
    // that the CTAs running at one time share packed tiles through L2.
    const int groups = PAIR ? P.n_tiles / 2 : P.n_tiles;
    const int units = live ? groups * P.n_ctiles * P.n_splits : 0;
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
    // barriers that MMA commits or the other CTA arrive on: pairs poll (a suspended try_wait can
    // sleep through a remote arrival); long waits off the critical path pause between polls
    auto wait_peer = [&](uint64_t* bar, uint32_t parity, int code) {
        return PAIR ? mbar_poll_cluster_look(bar, parity, P.status, code)
                    : mbar_wait_look(bar, parity, P.status, code);
    };
    auto wait_idle = [&](uint64_t* bar, uint32_t parity, int code, uint32_t ns) {
        return PAIR ? mbar_poll_sleep_look(bar, parity, P.status, code, ns)
                    : mbar_wait_look(bar, parity, P.status, code);
    };

    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer (B)
        if (elect_one()) {
            prefetch_tensormap(&tm_b);
            // a third of a deep ring at a time: stages come free in order, so the last one's
            // barrier stands for all
            const int batch = SD >= 6 ? SD / 3 : 1;
            int d = 0, loaded = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                const int row0 = (ct * (PAIR ? 2 : 1) + (int)rank) * kSets * P.set_rows;
                for (int kb = kb0; kb < kb1;) {
                    const int n = min(batch, kb1 - kb);
                    const int last = d + n - 1;
                    ok = wait_idle(&empty[last >= SD ? last - SD : last], last >= SD ? ph : ph ^ 1,
                                   kTimeoutTma, P.poll_ns);
                    if (!ok) break;
                    for (int i = 0; i < n; ++i, ++kb) {
                        mbar_arrive_expect_tx(&full[d], (uint32_t)b_bytes);
#pragma unroll
                        for (int q = 0; q < kSets; ++q)
                            tma_load_2d(smem_b + d * b_bytes + q * P.set_rows * 128, &tm_b, kb * kKBlock,
                                        row0 + q * (DIGITS == kDigits ? P.set_rows : P.hw), &full[d]);
                        ++loaded;
                        if (++d == SD) { d = 0; ph ^= 1; }
                    }
                }
            }
            // leave no copy in flight (in a pass that ran through, the MMAs have waited for them all)
            for (int q = min(loaded, SD); q > 0; --q) {
                if (--d < 0) { d = SD - 1; ph ^= 1; }
                mbar_wait_look(&full[d], ph, P.status, kTimeoutTma, 1u << 20);
            }
            chain_next();
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ TMA producer (packed)
        if (elect_one()) {
            prefetch_tensormap(&tm_a);
            int s = 0, loaded = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                for (int kb = kb0; kb < kb1; kb += kPackedKb) {
                    if (!(ok = mbar_wait_look(&empty_p[s], ph ^ 1, P.status, kTimeoutTma))) break;
                    mbar_arrive_expect_tx(&full_p[s], (uint32_t)kPackedBytes);
                    // 128 rows x 128 bytes (zeros past the row's end)
                    tma_load_2d(smem_p + s * kPackedBytes, &tm_a, kb * 32, tile * kTile, &full_p[s]);
                    ++loaded;
                    if (++s == SP) { s = 0; ph ^= 1; }
                }
            }
            for (int q = min(loaded, SP); q > 0; --q) {
                if (--s < 0) { s = SP - 1; ph ^= 1; }
                mbar_wait_look(&full_p[s], ph, P.status, kTimeoutTma, 1u << 20);
            }
        }
    } else if (warp == 1 && (!PAIR || rank == 0)) {
        // ------------------------------------------------------------ MMA issuer (pair: leader)
        // The whole role under elect: tcgen05 operands are uniform registers, and where the compiler
        // cannot see that one lane runs, it issues lane by lane (700 clocks a K-block, not 100).
        if (elect_one()) {
            // s8 x s8 -> s32, both operands K-major, M = 128 (pair: 256)
            const uint32_t idesc0 = (2u << 4) | (1u << 7) | (1u << 10) |
                                    ((uint32_t)((PAIR ? 2 : 1) * kTile >> 4) << 24);
            const uint32_t idesc = idesc0 | ((uint32_t)(nm >> 3) << 17);
            const uint32_t idesc_x = idesc0 | ((uint32_t)((ROWS ? P.nx : nm) >> 3) << 17);
            int d = 0, buf = 0;
            uint32_t ph = 0, ph_a = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                if (!(ok = wait_peer(&acc_empty[buf], ph_a ^ 1, kTimeoutMma))) break;
                tc_fence_after();
                const uint32_t acc = tmem_base + buf * P.acc_stride;
                // rows: the missing-call sums beside the main ones; samples: the same columns
                const uint32_t acc_x = ROWS ? acc + P.nm : acc;
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!(ok = wait_peer(&full[d], ph, kTimeoutMma))) break;
                    tc_fence_after();
                    const uint32_t ta = tmem_base + P.a0 + d * kAStage;
                    const uint64_t db = smem_desc_sw128(smem_addr(smem_b + d * b_bytes), 16, 1024);
                    const uint64_t dbx = ROWS ? db : db + (uint64_t)(P.set_rows * 128 >> 4);
#pragma unroll
                    for (int ks = 0; ks < kKBlock / 32; ++ks) {
                        const uint32_t first = (kb == kb0 && ks == 0) ? 0u : 1u;
                        if constexpr (PAIR) {
                            mma_i8_pair_tmem_a(acc, ta + ks * 8, db + 2 * ks, idesc, first);
                            mma_i8_pair_tmem_a(acc_x, ta + kAStage / 2 + ks * 8, dbx + 2 * ks, idesc_x,
                                               ROWS ? first : 1u);
                        } else {
                            mma_i8_tmem_a(acc, ta + ks * 8, db + 2 * ks, idesc, first);
                            mma_i8_tmem_a(acc_x, ta + kAStage / 2 + ks * 8, dbx + 2 * ks, idesc_x,
                                          ROWS ? first : 1u);
                        }
                    }
                    if (PAIR)
                        mma_commit_pair(&empty[d], 3);
                    else
                        mma_commit(&empty[d]);
                    if (++d == SD) { d = 0; ph ^= 1; }
                }
                if (ok) {
                    if (PAIR)
                        mma_commit_pair(&acc_full[buf], 3);
                    else
                        mma_commit(&acc_full[buf]);
                }
                if (++buf == NB) { buf = 0; ph_a ^= 1; }
            }
            if (PAIR)
                mma_commit_pair(drained, 1);
            else
                mma_commit(drained);
            mbar_wait_look(drained, 0, P.status, kTimeoutMma, 1u << 20);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            // the leader's MMA also reads this CTA's half of each stage's B rows: tell it (one
            // arrival on its full) once they have landed here
            int d = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int u = u0; u < units && ok; u += ustep) {
                int tile, ct, split, kb0, kb1;
                unit_coords(u, tile, ct, split, kb0, kb1);
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (!(ok = mbar_wait_look(&full[d], ph, P.status, kTimeoutDecode))) break;
                    mbar_arrive_remote(mapa_shared(&full[d], 0));
                    if (++d == SD) { d = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp >= kDecWarp0) {
        // ------------------------------------------------------------ decoders
        // lane = TMEM lane (row of A) 32 (warp % 4) + lane; group g = (warp - 8) / 4 takes K-blocks
        // g, g + G, .. of every packed tile whole: 128 codes per lane, 32 TMEM columns of each tile
        static_assert(kPackedKb % G == 0, "a packed tile holds the same number of K-blocks per group");
        constexpr int kOwn = kPackedKb / G;
        const int q = warp & 3, grp = (warp - kDecWarp0) >> 2;
        const int r = 32 * q + lane;
        // Stage of this group's next K-block.  Every unit holds a multiple of four K-blocks and the
        // ring has at least four stages, so that a group is never more than a lap ahead of the
        // MMAs on the stage that it waits for (a parity tells one lap from the next, no more).
        // (Units of any length, DIGITS = 3: groups take K-blocks in turn across units, j0 counts them,
        // so that a group's K-blocks are four apart all the same.)
        static_assert(DIGITS == kDigits || (!PAIR && kOwn == 1));
        int sp = 0, d = grp;
        uint32_t ph_p = 0, ph_d = 0, j0 = 0;
        bool ok = true;
        for (int u = u0; u < units && ok; u += ustep) {
            int tile, ct, split, kb0, kb1;
            unit_coords(u, tile, ct, split, kb0, kb1);
            const uint32_t lut = ROWS ? __ldg(P.lut + (int64_t)tile * kTile + r) : 0x00010002u;
            for (int kb = kb0; kb < kb1 && ok; kb += kPackedKb) {
                // (votes keep the warp together when a wait gives up)
                ok = __all_sync(0xffffffffu, mbar_wait_look(&full_p[sp], ph_p, P.status, kTimeoutDecode));
                if (!ok) break;
                const unsigned char* src = smem_p + sp * kPackedBytes + r * 128;
                int mine = 0;
                if constexpr (DIGITS != kDigits) {
                    const int here = min(kPackedKb, kb1 - kb);
                    mine = (int)((uint32_t)grp - j0) & (kPackedKb - 1);
                    j0 += (uint32_t)here;
                    if (mine >= here) {  // none of this tile's
                        if (lane == 0) mbar_arrive(&empty_p[sp]);
                        if (++sp == SP) { sp = 0; ph_p ^= 1; }
                        continue;
                    }
                }
                uint32_t words[kOwn][8];
#pragma unroll
                for (int o = 0; o < kOwn; ++o) {
                    const int c = 2 * ((DIGITS == kDigits ? grp : mine) + o * G);  // 16-byte chunk of the row, 128-byte swizzle
                    const uint4 p0 = *reinterpret_cast<const uint4*>(src + ((c ^ (r & 7)) << 4));
                    const uint4 p1 = *reinterpret_cast<const uint4*>(src + (((c + 1) ^ (r & 7)) << 4));
                    words[o][0] = p0.x; words[o][1] = p0.y; words[o][2] = p0.z; words[o][3] = p0.w;
                    words[o][4] = p1.x; words[o][5] = p1.y; words[o][6] = p1.z; words[o][7] = p1.w;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty_p[sp]);  // the packed tile has been read
                if (++sp == SP) { sp = 0; ph_p ^= 1; }
#pragma unroll
                for (int o = 0; o < kOwn; ++o) {
                    // half a K-block (64 codes of this lane) at a time: 16 TMEM columns of each tile;
                    // the first half is decoded before the wait for a free stage
                    uint32_t ev[16], mv[16];
                    auto decode_half = [&](int h) {
#pragma unroll
                        for (int cj = 0; cj < 4; ++cj) {
                            uint4 dos, mis;
                            decode_word_interleaved(words[o][4 * h + cj], lut, dos, mis);
                            ev[4 * cj] = dos.x; ev[4 * cj + 1] = dos.y; ev[4 * cj + 2] = dos.z; ev[4 * cj + 3] = dos.w;
                            mv[4 * cj] = mis.x; mv[4 * cj + 1] = mis.y; mv[4 * cj + 2] = mis.z; mv[4 * cj + 3] = mis.w;
                        }
                    };
                    decode_half(0);
                    ok = __all_sync(0xffffffffu, wait_idle(&empty[d], ph_d ^ 1, kTimeoutDecode, P.poll_dec_ns));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t ta = tmem_base + ((uint32_t)(32 * q) << 16) + P.a0 + d * kAStage;
                    tmem_st16(ta, ev);
                    tmem_st16(ta + kAStage / 2, mv);
                    decode_half(1);
                    tmem_st16(ta + 16, ev);
                    tmem_st16(ta + kAStage / 2 + 16, mv);
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (PAIR)
                            mbar_arrive_remote(mapa_shared(&full[d], 0));
                        else
                            mbar_arrive(&full[d]);
                    }
                    d += G;
                    if (d >= SD) { d -= SD; ph_d ^= 1; }
                }
            }
        }
    } else if (warp >= kEpiWarp0) {
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3;  // TMEM lane quarter this warp may access
        int buf = 0;
        uint32_t ph_a = 0;
        bool ok = true;
        for (int u = u0; u < units && ok; u += ustep) {
            int tile, ct, split, kb0, kb1;
            unit_coords(u, tile, ct, split, kb0, kb1);
            const int64_t row = (int64_t)tile * kTile + 32 * q + lane;
            RowCentre rc{0.0, 0.0, 0.0};
            if (ROWS && DIGITS == kDigits) {
                const double m = P.mu[row];
                rc.ah = (double)kTcQ * m;
                rc.al = fma((double)kTcQ, m, -rc.ah);
                rc.b = rc.ah - (double)((P.lut[row] >> 8) & 0xFFu);
            }
            ok = __all_sync(0xffffffffu, wait_idle(&acc_full[buf], ph_a, kTimeoutEpilogue, P.poll_ns));
            if (!ok) break;
            tc_fence_after();
            const uint32_t tb = tmem_base + buf * P.acc_stride + ((uint32_t)(32 * q) << 16);
            const int c_base = ct * P.w;
            const int cols = min(P.w, P.k - c_base);
            double* dst = P.part + ((int64_t)split * P.k + c_base) * P.ld + row;
            if constexpr (DIGITS == 3) {
                const double ib = 1.0 / 254.0, ib2 = 1.0 / (254.0 * 254.0), inv_q = 1.0 / (double)kTcQ;
                const double rt = ROWS ? P.mu[row] : 0.0;
                for (int c0 = 0; c0 < P.w; c0 += 8) {
                    int32_t m1[8], m2[8], m3[8];
                    double v[8];
                    tmem_ld8i(tb + c0, m1);
                    tmem_ld8i(tb + P.w + c0, m2);
                    tmem_ld8i(tb + 2 * P.w + c0, m3);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        v[i] = fma((double)m3[i], ib2, fma((double)m2[i], ib, (double)m1[i]));
                    if (ROWS) {
                        tmem_ld8i(tb + P.nm + c0, m1);
                        tmem_ld8i(tb + P.nm + P.w + c0, m2);
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        dst[(int64_t)(c0 + i) * P.ld] =
                            ROWS ? fma(v[i], inv_q, __dmul_rn(rt, fma((double)m2[i], ib, (double)m1[i])))
                                 : __dmul_rn(v[i], P.mu[c0 + i]);
                }
            }
            const longlong2* ks = P.ksum + (int64_t)split * P.k + c_base;
            // the missing-call sums leave out a column's last digit (the ranges stand in front of the sums:
            // SliceCall)
            const ColumnRange* const range = reinterpret_cast<const ColumnRange*>(P.ksum) - P.k + c_base;
            const unsigned uneven = ROWS && DIGITS == kDigits
                ? __ballot_sync(0xffffffffu, lane < cols && range_uneven(range[lane])) : 0u;
            auto emit = [&](int c, int64_t mh, int64_t ml, int64_t xh, int64_t xl) {
                const longlong2 sum = ks[c];
                double v;
                if (ROWS)
                    v = rows_value(rc, mh, ml, xh, xl, (double)sum.x * kLowDigits, (double)sum.y);
                else
                    v = fma((double)(mh - sum.x), kLowDigits, (double)(ml - sum.y));
                dst[(int64_t)c * P.ld] = v;
            };
            if (DIGITS == 3) {
                // written above
            } else if (P.cmajor) {
                for (int c = 0; c < cols; ++c) {
                    int32_t m[8];
                    int64_t mh, ml, xh = 0, xl = 0;
                    tmem_ld8i(tb + 8 * c, m);
                    join_digits(m, mh, ml);
                    if (ROWS) {
                        tmem_ld8i(tb + P.nm + 8 * c, m);
                        m[kDigits - 1] = 0;
                        if (!(uneven >> c & 1u)) m[kDigits - 2] = 0;
                        join_digits(m, xh, xl);
                    }
                    emit(c, mh, ml, xh, xl);
                }
            } else {
                // D columns: half h of the tile's columns (pair: from CTA h's B rows), then digit,
                // then column; eight columns at a time
                for (int c0 = 0; c0 < cols; c0 += 8) {
                    const int h = c0 >= P.hw ? 1 : 0;  // single CTA: hw = w
                    const int cl = c0 - h * P.hw;
                    const uint32_t cm = tb + h * (nm / 2) + cl;
                    int64_t mh[8], ml[8], xh[8], xl[8];
                    int32_t m[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) mh[i] = ml[i] = xh[i] = xl[i] = 0;
#pragma unroll
                    for (int p = 0; p < kDigits; ++p) {
                        const bool none = PAIR && p == kDigits - 1 && !eighth;
                        if (!none) tmem_ld8i(cm + p * P.hw, m);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            if (none) ml[i] *= 256;
                            else if (p < 3) mh[i] = mh[i] * 256 + m[i];
                            else ml[i] = ml[i] * 256 + m[i];
                        }
                    }
                    if (ROWS) {
                        const uint32_t cx = tb + P.nm + h * (P.nx / 2) + cl;
#pragma unroll
                        for (int p = 0; p < kDigits - 1; ++p) {
                            tmem_ld8i(cx + p * P.hw, m);
#pragma unroll
                            for (int i = 0; i < 8; ++i) {
                                if (p == kDigits - 2 && !(uneven >> (c0 + i) & 1u)) m[i] = 0;
                                if (p < 3) xh[i] = xh[i] * 256 + m[i];
                                else xl[i] = xl[i] * 256 + m[i];
                            }
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (c0 + i < cols) emit(c0 + i, mh[i], ml[i], xh[i], xl[i] * 256);
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
            if (++buf == NB) { buf = 0; ph_a ^= 1; }
        }
    }
    __syncwarp();
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

// Exponent e of the column's scale: |x| 2^e <= 127 2^56 for every element, 2^62 <= max 2^e or the
// half of it.
__device__ __forceinline__ int slice_exponent(unsigned long long max_bits) {
    if (max_bits == 0) return 0;
    const int ex = (int)(max_bits >> 52) - 1023;
    // mantissa above 127/64 would round up to 128 2^56
    const bool top = (max_bits & 0xFFFFFFFFFFFFFull) > 0xFC00000000000ull;
    return max(-kSliceMaxExp, min(kSliceMaxExp + 62, (top ? 61 : 62) - ex));
}
__device__ __forceinline__ double pow2(int e) {
    return __longlong_as_double((long long)(e + 1023) << 52);
}

__device__ __forceinline__ void range_of(double v, unsigned long long& mx, long long& es, unsigned& n) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7FFFFFFFFFFFFFFFull;
    mx = b > mx ? b : mx;
    if (b) {
        es += (int)(b >> 52) - 1023;
        ++n;
    }
}

__device__ __forceinline__ unsigned long long shfl_max(unsigned long long v, int width) {
    for (int off = width / 2; off; off >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, off);
        v = o > v ? o : v;
    }
    return v;
}
__device__ __forceinline__ long long shfl_sum(long long v, int width) {
    for (int off = width / 2; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

__device__ __forceinline__ void add_range(ColumnRange* out, unsigned long long mx, long long es,
                                          unsigned long long n) {
    atomicMax(&out->max_bits, mx);
    atomicAdd(reinterpret_cast<unsigned long long*>(&out->exp_sum), (unsigned long long)es);
    atomicAdd(&out->count, n);
}

// The words a chunk clears before its kernels add to them (see SliceCall), and the status that its
// passes report to: they only ever set it, and the first kernel of a call clears it (`clear`), not of
// a chunk, nor of a call whose caller looks at it after several (DeferChecks).
struct SliceSums {
    int* status;
    int clear;
    ColumnRange* range;        // of X, per column
    ColumnRange* range_w;      // of the samples operand
    unsigned long long* sum;   // [slices][k][2]: (hi, lo) sums of the fixed-point values, rows pass
    unsigned long long* sum_w; // the same of mu o w, samples pass
    int splits, splits_w;
};

__device__ __forceinline__ void clear_status(const SliceSums& S, bool first_block) {
    if (first_block && S.clear && threadIdx.x == 0) *S.status = kPassStatusOk;
}

// Ranges of X's columns: a block covers kc columns x rows_per_block rows, kc a power of two: one for
// column-major input, otherwise up to 32, so that a warp reads adjacent elements either way.
__global__ void __launch_bounds__(256)
k_slice_ranges(const StridedIn X, int64_t n, int64_t k, int kc, int64_t rows_per_block,
               const SliceSums S) {
    chain_enter();
    clear_status(S, blockIdx.x == 0 && blockIdx.y == 0);
    __shared__ unsigned long long s_mx[256];
    __shared__ long long s_es[256];
    __shared__ unsigned s_n[256];
    const int tc = threadIdx.x % kc, tr = threadIdx.x / kc, nr = 256 / kc;
    const int64_t c = (int64_t)blockIdx.y * kc + tc;
    const int64_t r0 = (int64_t)blockIdx.x * rows_per_block;
    const int64_t r1 = min(n, r0 + rows_per_block);
    unsigned long long mx = 0;
    long long es = 0;
    unsigned cnt = 0;
    if (c < k) {
#pragma unroll 4
        for (int64_t r = r0 + tr; r < r1; r += nr) range_of(X.p[r * X.rs + c * X.cs], mx, es, cnt);
    }
    s_mx[threadIdx.x] = mx;
    s_es[threadIdx.x] = es;
    s_n[threadIdx.x] = cnt;
    __syncthreads();
    for (int off = nr / 2; off > 0; off >>= 1) {
        if (tr < off) {
            const int o = threadIdx.x + off * kc;
            s_mx[threadIdx.x] = max(s_mx[threadIdx.x], s_mx[o]);
            s_es[threadIdx.x] += s_es[o];
            s_n[threadIdx.x] += s_n[o];
        }
        __syncthreads();
    }
    if (tr == 0 && c < k) add_range(&S.range[c], s_mx[threadIdx.x], s_es[threadIdx.x], s_n[threadIdx.x]);
}

// The scale of a column: its fixed-point values are rint(x f) << shift, the low digit zero in an even one.
struct SliceScale {
    double f;
    int shift;
    __device__ __forceinline__ explicit SliceScale(const ColumnRange& r)
        : f(pow2(slice_exponent(r.max_bits) - (range_uneven(r) ? 0 : 8))), shift(range_uneven(r) ? 0 : 8) {}
    __device__ __forceinline__ int64_t value(double x) const {
        return (int64_t)((uint64_t)__double2ll_rn(x * f) << shift);
    }
};

// Transposes 4 x 4 bytes: out[j] = byte j of in[0..3].
__device__ __forceinline__ void transpose4(const uint32_t (&in)[4], uint32_t (&out)[4]) {
    const uint32_t a = __byte_perm(in[0], in[1], 0x5140), b = __byte_perm(in[2], in[3], 0x5140);
    const uint32_t c = __byte_perm(in[0], in[1], 0x7362), d = __byte_perm(in[2], in[3], 0x7362);
    out[0] = __byte_perm(a, b, 0x5410);
    out[1] = __byte_perm(a, b, 0x7632);
    out[2] = __byte_perm(c, d, 0x5410);
    out[3] = __byte_perm(c, d, 0x7632);
}

// The eight digits of 16 fixed-point values, each digit's 16 bytes in the interleaved order of
// the decoded tiles: dig[p] for digit p (0 the most significant).
__device__ __forceinline__ void digits16(const int64_t (&v)[16], uint4 (&dig)[kDigits]) {
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        // positions 4g .. 4g + 3 hold samples sample_at(4g) ..
        uint32_t lo[4], hi[4], tl[4], th[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            // adding 128 to each of the lower seven digits makes the plain bytes the balanced
            // digits plus 128
            const uint64_t u = (uint64_t)v[sample_at(4 * g + j)] + 0x0080808080808080ull;
            lo[j] = (uint32_t)u ^ 0x80808080u;
            hi[j] = (uint32_t)(u >> 32) ^ 0x00808080u;
        }
        transpose4(lo, tl);
        transpose4(hi, th);
        uint32_t* w = reinterpret_cast<uint32_t*>(dig);
        w[0 * 4 + g] = th[3];
        w[1 * 4 + g] = th[2];
        w[2 * 4 + g] = th[1];
        w[3 * 4 + g] = th[0];
        w[4 * 4 + g] = tl[3];
        w[5 * 4 + g] = tl[2];
        w[6 * 4 + g] = tl[1];
        w[7 * 4 + g] = tl[0];
    }
}

// (hi, lo) of v = hi 2^40 + lo with lo the value of the five lower digits
__device__ __forceinline__ void split_value(int64_t v, int64_t& hi, int64_t& lo) {
    hi = (v + 0x8080808080ll) >> 40;
    lo = v - (hi << 40);
}

struct BLayout {
    int w, hw, cmajor, halves, sets, set_rows;
    // row of B that holds digit p of column c (set q)
    __device__ __forceinline__ int64_t row(int64_t c, int q, int p) const {
        const int64_t ct = c / w;
        const int cw = (int)(c - ct * w);
        const int h = cw / hw, cl = cw - h * hw;
        const int in = cmajor ? 8 * cl + p : p * hw + cl;
        return ((ct * halves + h) * sets + q) * set_rows + in;
    }
};

__device__ __forceinline__ void add_sums(unsigned long long* dst, int64_t hi, int64_t lo) {
    atomicAdd(dst, (unsigned long long)hi);
    atomicAdd(dst + 1, (unsigned long long)lo);
}

// 16 fixed-point values of column c -> their digits' bytes at rows B.row(c, set, p), from K
// position i0 on; their sums are added to (hi, lo).
__device__ __forceinline__ void emit_digits(const int64_t (&v)[16], const BLayout& B, int64_t c, int set,
                                            int64_t i0, int64_t pitch, int8_t* out) {
    uint4 dig[kDigits];
    digits16(v, dig);
#pragma unroll
    for (int p = 0; p < kDigits; ++p)
        *reinterpret_cast<uint4*>(out + B.row(c, set, p) * pitch + i0) = dig[p];
}

// Rows-pass operand: B rows of X's columns (columns k .. k_pad with zeros), and the sums of the
// fixed-point values per K slice.  A block takes COLS columns x ROWS rows through shared memory; a
// thread takes 16 rows of a column.
template <int COLS, int ROWS>
__global__ void __launch_bounds__(ROWS / 16 * COLS)
k_slice_rows_operand(const StridedIn X, int64_t n, int64_t k, int64_t k_pad, int64_t n_pad,
                     int slice_rows, const SliceSums S, BLayout B, int8_t* __restrict__ out) {
    chain_enter();
    constexpr int T = ROWS / 16 * COLS;
    static_assert(ROWS % 256 == 0 && (ROWS / 16) % 16 == 0, "a half warp covers 256 rows of a column");
    // one pad every 16 rows and one per column: conflict-free both ways
    __shared__ double tile[COLS][ROWS + ROWS / 16 + 1];
    const int64_t r0 = (int64_t)blockIdx.x * ROWS, c0 = (int64_t)blockIdx.y * COLS;
    for (int e = threadIdx.x; e < ROWS * COLS; e += T) {
        const int rr = X.rs == 1 ? e % ROWS : e / COLS, cc = X.rs == 1 ? e / ROWS : e % COLS;
        const int64_t r = r0 + rr, c = c0 + cc;
        tile[cc][rr + (rr >> 4)] = (r < n && c < k) ? X.p[r * X.rs + c * X.cs] : 0.0;
    }
    __syncthreads();
    const int grp = threadIdx.x % (ROWS / 16), cc = threadIdx.x / (ROWS / 16);
    const int64_t c = c0 + cc, i0 = r0 + 16 * grp;
    const bool live = c < k_pad && i0 < n_pad;
    int64_t sh = 0, sl = 0;
    if (live) {
        const SliceScale sc(c < k ? S.range[c] : ColumnRange{0, 0, 0, 0});
        int64_t v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            v[j] = sc.value(tile[cc][17 * grp + j]);
            int64_t h, l;
            split_value(v[j], h, l);
            sh += h;
            sl += l;
        }
        emit_digits(v, B, c, 0, i0, n_pad, out);
    }
    // 16 threads hold 256 rows, which lie in one slice
    sh = shfl_sum(sh, 16);
    sl = shfl_sum(sl, 16);
    if ((threadIdx.x & 15) == 0 && live && c < k) add_sums(S.sum + 2 * ((i0 / slice_rows) * k + c), sh, sl);
}

// The same for a short X, one block per column and 16 rows a thread, held in registers from the range
// to the digits; the call's other words are cleared here, so that a small call needs neither the
// memset nor the range kernel (a launch costs such a call more than the work in it).
constexpr int64_t kWholeRows = 8192;
__global__ void __launch_bounds__(kWholeRows / 16)
k_slice_rows_operand_whole(const StridedIn X, int64_t n, int64_t k, int64_t n_pad, int slice_rows,
                           const SliceSums S, BLayout B, int8_t* __restrict__ out) {
    chain_enter();
    __shared__ unsigned long long s_mx[16], s_sum[64][2];
    __shared__ long long s_es[16];
    __shared__ unsigned s_n[16];
    const int64_t c = blockIdx.x, i0 = 16 * (int64_t)threadIdx.x;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = (blockDim.x + 31) >> 5;
    double x[16];
    unsigned long long mx = 0;
    long long es = 0;
    unsigned cnt = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = (c < k && i0 + j < n) ? X.p[(i0 + j) * X.rs + c * X.cs] : 0.0;
#pragma unroll
    for (int j = 0; j < 16; ++j) range_of(x[j], mx, es, cnt);
    mx = shfl_max(mx, 32);
    es = shfl_sum(es, 32);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) {
        s_mx[warp] = mx;
        s_es[warp] = es;
        s_n[warp] = cnt;
    }
    for (int z = threadIdx.x; z < 2 * S.splits; z += blockDim.x) s_sum[z >> 1][z & 1] = 0;
    clear_status(S, c == 0);
    if (c < k) {
        if (threadIdx.x == 0) S.range_w[c] = ColumnRange{0, 0, 0, 0};
        for (int z = threadIdx.x; z < 2 * S.splits_w; z += blockDim.x)
            S.sum_w[2 * ((z >> 1) * k + c) + (z & 1)] = 0;
    }
    __syncthreads();
    unsigned long long n_all = 0;
    mx = 0;
    es = 0;
    for (int w = 0; w < warps; ++w) {
        mx = max(mx, s_mx[w]);
        es += s_es[w];
        n_all += s_n[w];
    }
    const ColumnRange rg{mx, es, n_all, 0};
    if (threadIdx.x == 0 && c < k) S.range[c] = rg;
    const SliceScale sc(rg);
    int64_t v[16], sh = 0, sl = 0;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        v[j] = sc.value(x[j]);
        int64_t h, l;
        split_value(v[j], h, l);
        sh += h;
        sl += l;
    }
    if (i0 < n_pad) emit_digits(v, B, c, 0, i0, n_pad, out);
    sh = shfl_sum(sh, 16);
    sl = shfl_sum(sl, 16);
    if ((threadIdx.x & 15) == 0 && i0 < n_pad) {
        atomicAdd(&s_sum[i0 / slice_rows][0], (unsigned long long)sh);
        atomicAdd(&s_sum[i0 / slice_rows][1], (unsigned long long)sl);
    }
    __syncthreads();
    if (c < k)
        for (int z = threadIdx.x; z < 2 * S.splits; z += blockDim.x)
            S.sum[2 * ((z >> 1) * k + c) + (z & 1)] = s_sum[z >> 1][z & 1];
}

// Samples-pass operand from W^T (column-major, R per column): the digits of w and of mu o w at
// one scale per column, and the sums of mu o w per K slice.  One column per blockIdx.y, 2048 SNPs
// per block.
__global__ void __launch_bounds__(128)
k_slice_samples_operand(const double* __restrict__ Wt, int64_t R, int64_t k, int64_t r_pad,
                        int slice_rows, const double* __restrict__ mu, const SliceSums S, BLayout B,
                        int8_t* __restrict__ out) {
    chain_enter();
    // w and mu o w of 2048 SNPs, one pad every 16, read in the order of memory
    __shared__ double sw[128 * 17], sb[128 * 17];
    const int64_t c = blockIdx.y, base = (int64_t)blockIdx.x * 2048;
#pragma unroll 8
    for (int e = threadIdx.x; e < 2048; e += 128) {
        const int64_t t = base + e;
        const double w = (c < k && t < R) ? Wt[c * R + t] : 0.0;
        sw[e + (e >> 4)] = w;
        sb[e + (e >> 4)] = t < R ? mu[t] * w : 0.0;
    }
    __syncthreads();
    const int64_t t0 = base + 16 * threadIdx.x;
    const bool live = t0 < r_pad;
    int64_t sh = 0, sl = 0;
    if (live) {
        const SliceScale sc(c < k ? S.range_w[c] : ColumnRange{0, 0, 0, 0});
        int64_t v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = sc.value(sw[17 * threadIdx.x + j]);
        emit_digits(v, B, c, 0, t0, r_pad, out);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            v[j] = sc.value(sb[17 * threadIdx.x + j]);
            int64_t h, l;
            split_value(v[j], h, l);
            sh += h;
            sl += l;
        }
        emit_digits(v, B, c, 1, t0, r_pad, out);
    }
    // 16 threads hold 256 SNPs, which lie in one slice
    sh = shfl_sum(sh, 16);
    sl = shfl_sum(sl, 16);
    if ((threadIdx.x & 15) == 0 && live && c < k) add_sums(S.sum_w + 2 * ((t0 / slice_rows) * k + c), sh, sl);
}

// A pass that gave up waiting leaves NaN, so that the failure shows wherever the caller looks.
__device__ __forceinline__ double checked(double v, const int* status) {
    return *status == kPassStatusOk ? v : __longlong_as_double(0x7FF8000000000000ll);
}

// (G - mu) of a 2-bit code, 0 for a missing call
__device__ __forceinline__ double centred(uint32_t code, double mu) {
    return code == 0u ? 2.0 - mu : code == 1u ? 0.0 : code == 2u ? 1.0 - mu : -mu;
}

struct PackedRows {
    const uint8_t* rows;
    int64_t stride;
};

// ---------------------------------------------------------------- columns outside the fixed-point range
// Plain FP64 sums of (G - mu) times the operand for up to kDirectCols columns at a time, by the blocks that
// reduce the other columns: which columns these are is known on the device only, and a kernel of
// their own would cost every small product its launch.  A decode value comes from a table in
// shared memory laid out so that no mix of codes conflicts (two wavefronts a value) and serves four
// columns; a block whose outputs are too few for its threads splits the sum over them.  Missing calls
// multiply by zero, so a non-finite value reaches every output, as it does in the FP64-pipe kernels.
// FP64 K x where every column of x is outside, ms (a value of -9999 left among normals), with the FP64-pipe kernels
// that took such columns before, with a warp to a SNP row and a thread to a sample, and so: 50,000 x 100,000, one
// column 7.2, 42.4, 3.7, 34 columns 58.7, 634, 30.4; 18,009 x 27,006, 34 columns 5.6, 76, 3.3, 266 columns 23.5, 462,
// 21.4; 2,000 x 10,000, one column 0.163, 1.59, 0.065.  One of 34 columns at 50,000 x 100,000: 58.7, 59.5, 11.8.
// What bounds them is the shared-memory pipe (twelve wavefronts for 16 multiply-adds a lane).
constexpr int kDirectCols = 4;
constexpr int kDirectRows = 1024;  // SNPs of a table: of direct_rows at most, of direct_samples
constexpr int kDirectSnps = 512;

// The columns that a block of column c takes: c and the next excluded ones where c is the first, fifth, ..
// excluded column, none otherwise.  Every thread of the block calls it.
__device__ __forceinline__ int direct_group(const ColumnRange* range, int64_t k, int64_t c, int* cols, int* count) {
    if (threadIdx.x < 32) {
        int before = 0, here = 0;
        for (int64_t j0 = 0; j0 < k && here < kDirectCols; j0 += 32) {
            const int64_t j = j0 + threadIdx.x;
            unsigned m = __ballot_sync(0xffffffffu, j < k && range_excluded(range[j]));
            const unsigned low = c >= j0 + 32 ? 0xffffffffu : c > j0 ? (1u << (int)(c - j0)) - 1u : 0u;
            before += __popc(m & low);
            for (m &= ~low; m && here < kDirectCols; m &= m - 1u, ++here)
                if (threadIdx.x == 0) cols[here] = (int)(j0 + __ffs(m) - 1);
        }
        if (threadIdx.x == 0) *count = before % kDirectCols == 0 ? here : 0;
    }
    __syncthreads();
    return *count;
}

// Whether a thread's sums have all become NaN, which nothing that follows changes.
template <int NG>
__device__ __forceinline__ int all_nan(const double (&acc)[4][NG], int ng) {
    bool lost = true;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int g = 0; g < NG; ++g) lost = lost && (g >= ng || acc[i][g] != acc[i][g]);
    return lost;
}

template <int NG>
__device__ __forceinline__ void load_values(const double* p, double (&v)[NG]) {
    if constexpr (NG == 4) {
        const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
        v[0] = a.x;
        v[1] = a.y;
        v[2] = b.x;
        v[3] = b.y;
    } else {
        v[0] = *p;
    }
}

// buf[g * rpb + row] = sum_i (G - mu) x_i,cols[g] of `rows` SNPs from t0 on and NG columns; rpb (64, 256 or
// 1024) rows a block, four of them a thread, 1024 / rpb threads to a row.
template <int NG>
__device__ __forceinline__ void direct_rows(const PackedRows& G, int64_t t0, int rows, int rpb,
                                            const double* __restrict__ mu, const StridedIn& X, const int* cols,
                                            int ng, int64_t n, double* buf) {
    const int groups = rpb / 4, parts = 256 / groups, grp = threadIdx.x % groups, part = threadIdx.x / groups;
    // [code][row]: a warp's lanes read neighbouring rows, whatever their codes
    for (int e = threadIdx.x; e < 4 * rpb; e += 256)
        buf[e] = e % rpb < rows ? centred((uint32_t)(e / rpb), mu[t0 + e % rpb]) : 0.0;
    __syncthreads();
    const uint8_t* const src = G.rows + t0 * G.stride;
    uint32_t row_at[4];  // below 2^32: finish_rows
#pragma unroll
    for (int i = 0; i < 4; ++i) row_at[i] = (uint32_t)min(grp + groups * i, rows - 1) * (uint32_t)G.stride;
    // 256 samples at a time, `here` of them to a part: x read by one thread a sample while the ones before
    // are used (past the last it is zero)
    const int here = 256 / parts, pitch = here * NG + 4;
    double* const xs = buf + 4 * rpb;
    double* const mine = xs + (threadIdx.x / here) * pitch + (threadIdx.x % here) * NG;
    double next[NG];
    auto fetch = [&](int64_t i) {
#pragma unroll
        for (int g = 0; g < NG; ++g) next[g] = i < n && g < ng ? X.p[i * X.rs + cols[g] * X.cs] : 0.0;
    };
    fetch(threadIdx.x);
    const double* const lut = buf + grp;
    double acc[4][NG] = {};
    int lost = 0;
    for (int64_t base = 0; base < n; base += 256) {
        if (__syncthreads_and(lost)) break;
#pragma unroll
        for (int g = 0; g < NG; ++g) mine[g] = next[g];
        __syncthreads();
        fetch(base + 256 + threadIdx.x);
        const int64_t i0 = base + part * here;
        const double* x = xs + part * pitch;
#pragma unroll 1
        for (int64_t at = i0; at < min(n, i0 + here); at += 16) {
            uint32_t word[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) word[i] = *reinterpret_cast<const uint32_t*>(src + row_at[i] + (at >> 2));
#pragma unroll 4
            for (int j = 0; j < 16; ++j, x += NG) {
                double xv[NG];
                load_values<NG>(x, xv);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const double z = lut[(int)((word[i] >> (2 * j)) & 3u) * rpb + groups * i];
#pragma unroll
                    for (int g = 0; g < NG; ++g) acc[i][g] = fma(z, xv[g], acc[i][g]);
                }
            }
        }
        lost = all_nan(acc, ng);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int g = 0; g < NG; ++g) buf[(part * NG + g) * rpb + grp + groups * i] = acc[i][g];
    __syncthreads();
    for (int e = threadIdx.x; e < NG * rpb; e += 256) {
        double v = buf[e];
        for (int p = 1; p < parts; ++p) v += buf[p * NG * rpb + e];
        buf[e] = v;
    }
    __syncthreads();
}

// sum_t (G - mu) W_t,cols[g] of samples i0 .. i0 + 31: thread g * 32 + sample (< 32 NG) returns its own.
// Four samples of a SNP a thread, 32 SNPs at a time, tables of 512 SNPs.
template <int NG>
__device__ __forceinline__ double direct_samples(const PackedRows& G, int64_t i0, const double* __restrict__ mu,
                                                 const double* __restrict__ Wt, int64_t R,
                                                 const int64_t (&cols)[kDirectCols], int ng, double* buf) {
    const int bc = threadIdx.x & 7, part = threadIdx.x >> 3;
    const uint8_t* src = G.rows + (i0 >> 2) + bc;
    double* const wv = buf + 4 * kDirectSnps;
    double acc[4][NG] = {};
    int lost = 0;
    for (int64_t base = 0; base < R; base += kDirectSnps) {
        const int here = (int)min((int64_t)kDirectSnps, R - base);
        if (__syncthreads_and(lost)) break;
        for (int e = threadIdx.x; e < here; e += 256) {
            const double m = mu[base + e];
#pragma unroll
            for (int q = 0; q < 4; ++q) buf[4 * e + q] = centred((uint32_t)q, m);
#pragma unroll
            for (int g = 0; g < NG; ++g) wv[NG * e + g] = g < ng ? Wt[cols[g] * R + base + e] : 0.0;
        }
        __syncthreads();
        for (int r0 = part; r0 < here; r0 += 8 * 32) {
            uint32_t codes[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) codes[j] = r0 + 32 * j < here ? src[(base + r0 + 32 * j) * G.stride] : 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int row = r0 + 32 * j;
                if (row >= here) break;
                double w[NG];
                load_values<NG>(wv + NG * row, w);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const double z = buf[4 * row + (int)((codes[j] >> (2 * i)) & 3u)];
#pragma unroll
                    for (int g = 0; g < NG; ++g) acc[i][g] = fma(z, w[g], acc[i][g]);
                }
            }
        }
        lost = all_nan(acc, ng);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            double v = acc[i][g];
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if ((threadIdx.x & 31) < 8) buf[((threadIdx.x >> 5) * NG + g) * 32 + 4 * bc + i] = v;
        }
    __syncthreads();
    double v = 0.0;
    if (threadIdx.x < 32 * NG)
        for (int p = 0; p < 8; ++p) v += buf[p * 32 * NG + threadIdx.x];
    __syncthreads();
    return v;
}

// Rows-pass result u / s = 2^-e / 63 sum_z part (or the direct sum).  rpb SNPs per block, one column
// per blockIdx.y.  With Wt: W^T (column-major, R per column) = s^2 (u / s) and the ranges of
// max(|W|, |mu W|) for the samples operand; with out: s (u / s) at row pos[t] (or t).
__global__ void __launch_bounds__(256, 3)
k_slice_reduce_rows(const double* __restrict__ part, int64_t ld, int64_t R, int64_t k, int rpb,
                    const double* __restrict__ s_row, const double* __restrict__ mu,
                    const PackedRows G, const StridedIn X, int64_t n, const SliceSums S,
                    double* __restrict__ Wt, const int32_t* __restrict__ pos, StridedOut out) {
    chain_enter();
    __shared__ __align__(16) double buf[4 * kDirectRows + 256 * kDirectCols + 64];
    __shared__ unsigned long long s_mx[8];
    __shared__ long long s_es[8];
    __shared__ unsigned s_n[8];
    __shared__ int s_cols[kDirectCols], s_count;
    const int64_t c = blockIdx.y;
    const ColumnRange rg = S.range[c];
    unsigned long long mx = 0;
    long long es = 0;
    unsigned cnt = 0;
    const int64_t t0 = (int64_t)blockIdx.x * rpb;
    const int rows = (int)min((int64_t)rpb, R - t0);
    auto finish = [&](int64_t col, int64_t t, double v) {
        const double s = s_row[t];
        if (Wt) {
            const double w = v * s * s;
            Wt[col * R + t] = w;
            range_of(mu[t] > 1.0 ? mu[t] * w : w, mx, es, cnt);
        } else {
            out.p[(pos ? (int64_t)pos[t] : t) * out.rs + col * out.cs] = v * s;
        }
    };
    auto close = [&](int64_t col) {  // the block's range, one atomic each
        if (!Wt) return;
        mx = shfl_max(mx, 32);
        es = shfl_sum(es, 32);
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if ((threadIdx.x & 31) == 0) {
            s_mx[threadIdx.x >> 5] = mx;
            s_es[threadIdx.x >> 5] = es;
            s_n[threadIdx.x >> 5] = cnt;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; ++w) {
                mx = max(mx, s_mx[w]);
                es += s_es[w];
                cnt += s_n[w];
            }
            add_range(&S.range_w[col], mx, es, cnt);
        }
        __syncthreads();
    };
    if (!range_excluded(rg)) {
        const double f = pow2(-slice_exponent(rg.max_bits));
        // four rows a thread at a time: few blocks are resident beside the direct sums' registers
        double acc[4] = {};
        const double* p = part + c * ld + t0 + threadIdx.x;
        for (int z = 0; z < S.splits; ++z, p += k * ld) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if ((int)threadIdx.x + 256 * j < rows) acc[j] += p[256 * j];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int e = threadIdx.x + 256 * j;
            if (e < rows) finish(c, t0 + e, checked(acc[j] * f * (1.0 / (double)kTcQ), S.status));
        }
        close(c);
        return;
    }
    const int ng = direct_group(S.range, k, c, s_cols, &s_count);
    if (ng == 0) return;
    if (ng == 1) direct_rows<1>(G, t0, rows, rpb, mu, X, s_cols, ng, n, buf);
    else direct_rows<kDirectCols>(G, t0, rows, rpb, mu, X, s_cols, ng, n, buf);
    for (int g = 0; g < ng; ++g) {
        mx = 0;
        es = 0;
        cnt = 0;
        for (int e = threadIdx.x; e < rows; e += 256) finish(s_cols[g], t0 + e, buf[g * rpb + e]);
        close(s_cols[g]);
    }
}

// The samples operand of a half-pass: W^T[c][t] = s_t V[pos[t]][c] and its ranges (1024 SNPs per
// block, one column per blockIdx.y).
__global__ void __launch_bounds__(256)
k_slice_gather(const StridedIn V, int64_t R, const int32_t* __restrict__ pos,
               const double* __restrict__ s_row, const double* __restrict__ mu, const SliceSums S,
               double* __restrict__ Wt) {
    chain_enter();
    clear_status(S, blockIdx.x == 0 && blockIdx.y == 0);
    const int64_t c = blockIdx.y;
    unsigned long long mx = 0;
    long long es = 0;
    unsigned cnt = 0;
    const int64_t t0 = (int64_t)blockIdx.x * 1024;
    for (int64_t t = t0 + threadIdx.x; t < min(R, t0 + 1024); t += 256) {
        const double w = s_row[t] * V.p[(int64_t)pos[t] * V.rs + c * V.cs];
        Wt[c * R + t] = w;
        range_of(mu[t] > 1.0 ? mu[t] * w : w, mx, es, cnt);
    }
    mx = shfl_max(mx, 32);
    es = shfl_sum(es, 32);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if ((threadIdx.x & 31) == 0) add_range(&S.range_w[c], mx, es, cnt);
}

// Samples-pass result: Y[i][c] = scale 2^-e sum_z part[z][c][i] (or the direct sum over the column's
// W).  Column-major output: a warp's lanes are samples; row-major: tiles of 32 samples x 32 columns
// through shared memory, so that both sides are coalesced.
__global__ void __launch_bounds__(256, 3)
k_slice_reduce_samples(const double* __restrict__ part, int64_t ld, int64_t n, int64_t k,
                       const double* __restrict__ Wt, int64_t R, const double* __restrict__ mu,
                       const PackedRows G, const SliceSums S, double scale, StridedOut Y) {
    chain_enter();
    __shared__ double tile[32][33];
    __shared__ __align__(16) double buf[(4 + kDirectCols) * kDirectSnps];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int64_t i0 = (int64_t)blockIdx.x * 32, c0 = (int64_t)blockIdx.y * 32;
    const int64_t i = i0 + tx;
    const unsigned direct = __ballot_sync(0xffffffffu, c0 + tx < k && range_excluded(S.range_w[c0 + tx]));
    auto store = [&](int cc, double v) {
        if (Y.rs == 1) Y.p[i + (c0 + cc) * Y.cs] = v;
        else tile[cc][tx] = v;
    };
    // four columns a thread at a time, as above
    double acc[4] = {};
    const double* p = part + (c0 + ty) * ld + i;
    for (int z = 0; z < S.splits_w; ++z, p += k * ld) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (c0 + ty + 8 * j < k && i < n) acc[j] += p[8 * j * ld];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int cc = ty + 8 * j;
        if (c0 + cc >= k || i >= n || (direct >> cc & 1u)) continue;
        store(cc, checked(acc[j] * pow2(-slice_exponent(S.range_w[c0 + cc].max_bits)) * scale, S.status));
    }
    for (unsigned m = direct; m;) {
        int64_t cols[kDirectCols] = {};
        int ng = 0, mine = 0;
#pragma unroll
        for (int g = 0; g < kDirectCols; ++g)
            if (m) {
                const int cc = __ffs(m) - 1;
                cols[g] = c0 + cc;
                if (ty == g) mine = cc;
                m &= m - 1u;
                ++ng;
            }
        const double v = ng == 1 ? direct_samples<1>(G, i0, mu, Wt, R, cols, ng, buf)
                                 : direct_samples<kDirectCols>(G, i0, mu, Wt, R, cols, ng, buf);
        if (ty < ng && i < n) store(mine, v * scale);
    }
    if (Y.rs == 1) return;
    __syncthreads();
    for (int ii = ty; ii < 32; ii += 8) {
        const int64_t r = i0 + ii, c = c0 + tx;
        if (r < n && c < k) Y.p[r * Y.rs + c * Y.cs] = tile[tx][ii];
    }
}

// ---------------------------------------------------------------- plans

struct SlicePlan {
    bool pair = false;
    int w = 0, hw = 0, cmajor = 0, n_ctiles = 0;
    int nm = 0, nx = 0, set_rows = 0;
    int sd = 0, sp = 0, nb = 0;
    uint32_t acc_stride = 0, a0 = 0;
    int splits = 1, kbs = 0;
    size_t smem = 0;
    double cost = 0.0;
    BLayout blayout(bool rows) const {
        return BLayout{w, hw, cmajor, pair ? 2 : 1, rows ? 1 : 2, set_rows};
    }
    int64_t b_rows(bool rows) const {
        return (int64_t)n_ctiles * (pair ? 2 : 1) * (rows ? 1 : 2) * set_rows;
    }
};

// Layout of column tiles of w columns, with two accumulators where they leave room for `stages2`
// stages; false when it does not fit.
bool lay_out(bool rows, bool pair, int w, int64_t k, SlicePlan& p, int digits = kDigits, int stages2 = 4) {
    const int halves = pair ? 2 : 1;
    p.pair = pair;
    p.w = w;
    p.hw = w / halves;
    p.cmajor = w <= 4 && digits == kDigits ? 1 : 0;
    p.n_ctiles = (int)((k + w - 1) / w);
    auto up16 = [](int x) { return (x + 15) / 16 * 16; };
    const int half_m = p.cmajor ? up16(8 * w) : up16(digits * p.hw);
    const int half_x = p.cmajor ? half_m : up16((digits - 1) * p.hw);
    p.nm = halves * half_m;
    p.nx = halves * half_x;
    p.set_rows = half_m;
    if (p.nm > 256) return false;
    p.acc_stride = (uint32_t)(rows ? p.nm + p.nx : p.nm);
    p.nb = 2 * p.acc_stride + stages2 * kAStage <= kTmemCols ? 2 : 1;
    p.a0 = (p.nb * p.acc_stride + 31) / 32 * 32;
    p.sp = 4;
    const int b_bytes = (rows ? 1 : 2) * p.set_rows * 128;
    const int room = (kSmemMax - 1024 - kBarBytes - p.sp * kPackedBytes) / b_bytes;
    p.sd = std::min(std::min(8, room), ((int)kTmemCols - (int)p.a0) / (int)kAStage);
    if (p.sd < 4) return false;
    p.smem = (size_t)p.sd * b_bytes + (size_t)p.sp * kPackedBytes + kBarBytes + 1024;
    return true;
}

// K slices: the count (at most 1024 K-blocks and a multiple of four in each) with the shortest
// last finisher, a unit costing its K-blocks plus the fill and drain of its pipeline.
void choose_slices(SlicePlan& p, int64_t units, int kb, int ctas) {
    double best = 1e300;
    for (int s = 1; s <= 64; ++s) {
        int kbs = (kb + s - 1) / s;
        kbs = (kbs + kPackedKb - 1) / kPackedKb * kPackedKb;
        if (kbs > kMaxKbPerAccum) continue;
        const int real = (kb + kbs - 1) / kbs;
        if (real != s) continue;
        const double waves = std::ceil((double)units * real / ctas);
        const double cost = waves * (kbs + 6.0) + 0.25 * real;
        if (cost < best) {
            best = cost;
            p.splits = real;
            p.kbs = kbs;
        }
    }
    if (best >= 1e300) {  // more than 64 slices of 1024
        p.kbs = kMaxKbPerAccum;
        p.splits = (kb + p.kbs - 1) / p.kbs;
        best = std::ceil((double)units * p.splits / ctas) * (p.kbs + 6.0);
    }
    p.cost = best;
}

// The plan with the least estimated time.  A K-block costs its MMAs (N / 2 clocks for each of
// 4 + 4 instructions on a CTA) or its decode, whichever is longer.  The costs are those of seven
// digits: with them the plans were measured, the eighth digit's MMAs do not show (1.28 and 1.30 ms a rows pass,
// 1.04 and 1.04 a samples pass of 266 columns at 18,009 x 27,006), and the K slices, whose sums are added in
// FP64, stay where they were.
SlicePlan choose_slice_plan(bool rows, int64_t tiles, int kb, int64_t k) {
    SlicePlan best;
    best.cost = 1e300;
    auto consider = [&](bool pair, int w) {
        SlicePlan p, seven;
        if (!lay_out(rows, pair, w, k, p) || !lay_out(rows, pair, w, k, seven, kDigits - 1)) return;
        const int ctas = pair ? num_sms() / 2 : num_sms();
        choose_slices(p, (pair ? tiles / 2 : tiles) * p.n_ctiles, kb, ctas);
        const double mma = 2.0 * (rows ? seven.nm + seven.nx : 2 * seven.nm);
        // a single CTA streams all B rows from L2 itself
        const double l2 = (pair ? 0.5 : 1.0) * (rows ? 1 : 2) * seven.nm * 128.0 / 28.0;
        p.cost *= std::max(std::max(mma, l2), pair ? 420.0 : 380.0);
        if (p.cost < best.cost) best = p;
    };
    if (k <= 4) {
        consider(false, (int)k);
    } else {
        for (int w = 8; w <= 32; w += 8) consider(false, w);
        if (num_sms() >= 2)
            for (int w = 16; w <= 32; w += 16) consider(true, w);
    }
    return best;
}

// Decoder groups: single CTAs are bound by the decode, pairs by the MMAs.
constexpr int kSingleGroups = 4, kPairGroups = 2;
template <bool PAIR>
constexpr int groups_of() { return PAIR ? kPairGroups : kSingleGroups; }

template <bool ROWS, bool PAIR, int DIGITS = kDigits>
cudaError_t allow_smem() {
    return cudaFuncSetAttribute(k_slice_pass<ROWS, PAIR, groups_of<PAIR>(), DIGITS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSmemMax);
}

void configure_slices() {
    static PerDeviceOnce configured;
    once_per_device(configured, [] {
        cudaError_t e = allow_smem<true, false>();
        if (e == cudaSuccess) e = allow_smem<false, false>();
        if (e == cudaSuccess) e = allow_smem<true, true>();
        if (e == cudaSuccess) e = allow_smem<false, true>();
        if (e == cudaSuccess) e = allow_smem<true, false, 3>();
        if (e == cudaSuccess) e = allow_smem<false, false, 3>();
        return e;
    }, "configure slice kernels");
}

// CS_B200_GIVE_UP=i: the process's FP64 pass number i (from 0) is reported as one that gave up waiting
// (the word is set behind it on the stream), so that tests can see what each caller makes of that.
void report_as_given_up(int* status, cudaStream_t s) {
    static const long long which = [] {
        const char* v = std::getenv("CS_B200_GIVE_UP");
        return v ? std::atoll(v) : -1LL;
    }();
    if (which < 0) return;
    static std::atomic<long long> passes{0};
    if (passes.fetch_add(1) == which) CS_CUDA(cudaMemsetAsync(status, 1, sizeof(int), s));
}

template <bool ROWS, bool PAIR, int DIGITS = kDigits>
void launch_slice_pass(const SlicePlan& p, const CUtensorMap& ta, const CUtensorMap& tb,
                       const SliceArgs& A, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(threads_for(groups_of<PAIR>()));
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    if constexpr (PAIR) {
        cfg.gridDim = dim3((unsigned)(num_sms() & ~1));
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        // as many pairs as are resident together (an SM without a partner in its GPC stays idle)
        static int resident[PerDeviceOnce::kMaxDevices] = {};
        int dev = 0;
        CS_CUDA(cudaGetDevice(&dev));
        int& pairs = resident[dev];
        if (pairs == 0) {
            cudaLaunchConfig_t probe = cfg;
            probe.dynamicSmemBytes = kSmemMax;
            int c = 0;
            CS_CUDA(cudaOccupancyMaxActiveClusters(&c, k_slice_pass<ROWS, true, kPairGroups, DIGITS>, &probe));
            pairs = std::max(1, std::min(c, num_sms() / 2));
        }
        cfg.gridDim = dim3((unsigned)(2 * pairs));
    } else {
        cfg.gridDim = dim3((unsigned)std::min<int64_t>(
            num_sms(), std::max<int64_t>(1, (int64_t)A.n_tiles * A.n_ctiles * A.n_splits)));
    }
    chain(cfg, attr);
    CS_CUDA(cudaLaunchKernelEx(&cfg, k_slice_pass<ROWS, PAIR, groups_of<PAIR>(), DIGITS>, ta, tb, A));
    if (DIGITS == kDigits) report_as_given_up(A.status, s);
}

}  // namespace

struct SliceOperator {
    DeviceBuffer<int8_t> b;
    DeviceBuffer<double> part, W;
    DeviceBuffer<unsigned long long> words;  // SliceCall's
    DeviceBuffer<int> status;                // a word of its own: the chunks of a call share it
    // packed rows and their sample-major copy, 128 rows x 128 bytes at a time (both belong to the
    // operator and keep their place for its lifetime)
    CUtensorMap tm_packed{}, tm_packed_t{};
    bool map_rows = false, map_samples = false;
    void release_operands() {
        b.release();
        part.release();
        W.release();
        words.release();
    }
};

void destroy_slices(SliceOperator* s) { delete s; }

namespace {

// Columns per call of the passes: bounds the operand buffers (16 bytes per row and column) and
// keeps a K slice's digits in L2.
constexpr int64_t kChunkColumns = 288;

// One chunk of columns: the plans of the passes it runs and its cleared words: the ranges of X (4 a column)
// and behind them the slice sums of the rows pass (2 a column and slice), then the same of W.
struct SliceCall {
    SlicePlan rows, samples;
    int64_t k = 0, range = 0, range_w = 0, sum = 0, sum_w = 0, words = 0;
};

SliceCall plan_call(const MixedRows& r, int64_t k) {
    SliceCall c;
    c.k = k;
    c.rows = choose_slice_plan(true, r.r_pad / kTile, (int)(r.n_pad / kKBlock), k);
    c.samples = choose_slice_plan(false, r.n_pad / kTile, (int)(r.r_pad / kKBlock), k);
    c.range = 0;
    c.sum = c.range + 4 * k;
    c.range_w = c.sum + 2 * k * c.rows.splits;
    c.sum_w = c.range_w + 4 * k;
    c.words = c.sum_w + 2 * k * c.samples.splits;
    return c;
}

SliceSums sums_of(SliceOperator& so, const SliceCall& c, bool clear) {
    unsigned long long* z = so.words.get();
    SliceSums S;
    S.status = so.status.get();
    S.clear = clear ? 1 : 0;
    S.range = reinterpret_cast<ColumnRange*>(z + c.range);
    S.range_w = reinterpret_cast<ColumnRange*>(z + c.range_w);
    S.sum = z + c.sum;
    S.sum_w = z + c.sum_w;
    S.splits = c.rows.splits;
    S.splits_w = c.samples.splits;
    return S;
}

int64_t digit_bytes(const MixedRows& r, const SliceCall& c) {
    return std::max(c.rows.b_rows(true) * r.n_pad, c.samples.b_rows(false) * r.r_pad);
}
int64_t part_values(const MixedRows& r, const SliceCall& c) {
    return c.k * std::max(c.rows.splits * r.r_pad, c.samples.splits * r.n_pad);
}
size_t operand_bytes(const MixedRows& r, const SliceCall& c) {
    return (size_t)(digit_bytes(r, c) + 8 * (part_values(r, c) + r.R * c.k + c.words));
}
void reserve(SliceOperator& so, const MixedRows& r, const SliceCall& c) {
    so.b.resize(digit_bytes(r, c));
    so.part.resize(part_values(r, c));
    so.W.resize(r.R * c.k);
    so.words.resize(c.words);
}

// The status word, clear when it is new.
void make_status(SliceOperator& so, cudaStream_t s) {
    if (so.status.get()) return;
    so.status.resize(1);
    CS_CUDA(cudaMemsetAsync(so.status.get(), 0, sizeof(int), s));
}

SliceArgs slice_args(const SlicePlan& p, bool rows, int64_t tiles, int kb, int64_t k) {
    SliceArgs A{};
    A.n_tiles = (int)tiles;
    A.n_ctiles = p.n_ctiles;
    A.n_splits = p.splits;
    A.kb_total = (kb + kPackedKb - 1) / kPackedKb * kPackedKb;  // past the operand's end: zeros
    A.kb_per_split = p.kbs;
    A.k = (int)k;
    A.w = p.w;
    A.hw = p.hw;
    A.cmajor = p.cmajor;
    A.nm = p.nm;
    A.nx = rows ? p.nx : p.nm;
    A.set_rows = p.set_rows;
    A.sp = p.sp;
    A.sd = p.sd;
    A.nb = p.nb;
    A.acc_stride = p.acc_stride;
    A.a0 = p.a0;
    A.poll_ns = 128;
    A.poll_dec_ns = 32;
    return A;
}

// The sums of the rows pass of one chunk (X's digits, then the pass) into so.part.
void run_rows(SliceOperator& so, MixedRows& r, const SliceCall& c, const SliceSums& S, StridedIn X,
              cudaStream_t s) {
    const int64_t n = r.n, R = r.R, k = c.k;
    const SlicePlan& p = c.rows;
    const int64_t k_pad = (int64_t)p.n_ctiles * p.w;
    const BLayout B = p.blayout(true);
    const int slice_rows = p.kbs * kKBlock;
    if (n <= kWholeRows && p.splits <= 64) {
        prof::Scope ps("slice_prep_rows_operand", s, 0.0, 16.0 * n * k + 8.0 * k_pad * r.n_pad);
        const unsigned threads = (unsigned)round_up(r.n_pad / 16, 32);
        launch_chained(k_slice_rows_operand_whole, (unsigned)k_pad, threads, 0, s, X, n, k, r.n_pad,
                       slice_rows, S, B, so.b.get());
        CS_LAUNCH("slice rows operand");
    } else {
        CS_CUDA(cudaMemsetAsync(so.words.get(), 0, 8 * c.words, s));
        prof::Scope ps("slice_prep_rows_operand", s, 0.0, 16.0 * n * k + 8.0 * k_pad * r.n_pad);
        int kc = 1;
        while (X.rs != 1 && kc < k && kc < 32) kc *= 2;
        const int64_t rpb = std::max<int64_t>(256, 4096 / kc);
        launch_chained(k_slice_ranges, dim3((unsigned)((n + rpb - 1) / rpb), (unsigned)((k + kc - 1) / kc)),
                       256, 0, s, X, n, k, kc, rpb, S);
        if (k_pad <= 1)
            launch_chained(k_slice_rows_operand<1, 1024>, dim3((unsigned)((r.n_pad + 1023) / 1024), 1), 64, 0,
                           s, X, n, k, k_pad, r.n_pad, slice_rows, S, B, so.b.get());
        else if (k_pad <= 4)
            launch_chained(k_slice_rows_operand<4, 512>, dim3((unsigned)((r.n_pad + 511) / 512), 1), 128, 0, s,
                           X, n, k, k_pad, r.n_pad, slice_rows, S, B, so.b.get());
        else
            launch_chained(k_slice_rows_operand<16, 256>,
                           dim3((unsigned)(r.n_pad / 256), (unsigned)((k_pad + 15) / 16)), 256, 0, s, X, n, k,
                           k_pad, r.n_pad, slice_rows, S, B, so.b.get());
        CS_LAUNCH("slice rows operand");
    }
    const CUtensorMap tb = make_map_u8(so.b.get(), (uint64_t)r.n_pad, (uint64_t)p.b_rows(true),
                                       (uint64_t)r.n_pad, kKBlock, (uint32_t)p.set_rows, true);
    SliceArgs A = slice_args(p, true, r.r_pad / kTile, (int)(r.n_pad / kKBlock), k);
    A.lut = r.lut.get();
    A.mu = r.mu.get();
    A.ksum = reinterpret_cast<const longlong2*>(S.sum);
    A.part = so.part.get();
    A.ld = r.r_pad;
    A.status = S.status;
    prof::Scope ps("kinship_rows_slices", s, 2.0 * (double)n * (double)R * (double)k,
                   (double)R * (double)((n + 3) / 4));
    if (p.pair)
        launch_slice_pass<true, true>(p, so.tm_packed, tb, A, s);
    else
        launch_slice_pass<true, false>(p, so.tm_packed, tb, A, s);
    CS_LAUNCH("kinship_rows_slices");
}

// Y (n x k) = scale Z_c W of one chunk, from so.W and its ranges.
void run_samples(SliceOperator& so, MixedRows& r, const SliceCall& c, const SliceSums& S, double scale,
                 StridedOut Y, cudaStream_t s) {
    const int64_t n = r.n, R = r.R, k = c.k;
    const SlicePlan& p = c.samples;
    const int64_t k_pad = (int64_t)p.n_ctiles * p.w;
    {
        prof::Scope ps("slice_prep_samples_operand", s, 0.0, 8.0 * R * k + 16.0 * k_pad * r.r_pad);
        launch_chained(k_slice_samples_operand, dim3((unsigned)((r.r_pad + 2047) / 2048), (unsigned)k_pad),
                       128, 0, s, so.W.get(), R, k, r.r_pad, p.kbs * kKBlock, r.mu.get(), S, p.blayout(false),
                       so.b.get());
        CS_LAUNCH("slice samples operand");
    }
    const CUtensorMap tb = make_map_u8(so.b.get(), (uint64_t)r.r_pad, (uint64_t)p.b_rows(false),
                                       (uint64_t)r.r_pad, kKBlock, (uint32_t)p.set_rows, true);
    SliceArgs A = slice_args(p, false, r.n_pad / kTile, (int)(r.r_pad / kKBlock), k);
    A.ksum = reinterpret_cast<const longlong2*>(S.sum_w);
    A.part = so.part.get();
    A.ld = r.n_pad;
    A.status = S.status;
    {
        prof::Scope ps("kinship_samples_slices", s, 2.0 * (double)n * (double)R * (double)k,
                       (double)R * (double)((n + 3) / 4));
        if (p.pair)
            launch_slice_pass<false, true>(p, so.tm_packed_t, tb, A, s);
        else
            launch_slice_pass<false, false>(p, so.tm_packed_t, tb, A, s);
        CS_LAUNCH("kinship_samples_slices");
    }
    prof::Scope ps("slice_reduce_samples", s, 0.0, 8.0 * (p.splits + 1) * (double)k * n);
    launch_chained(k_slice_reduce_samples, dim3((unsigned)((n + 31) / 32), (unsigned)((k + 31) / 32)), 256, 0,
                   s, so.part.get(), r.n_pad, n, k, so.W.get(), R, r.mu.get(), PackedRows{r.rows, r.stride}, S,
                   scale, Y);
    CS_LAUNCH("slice_reduce_samples");
}

// W (Wt) or s o u at the rows' positions (out) from the sums of run_rows.
void finish_rows(SliceOperator& so, MixedRows& r, const SliceCall& c, const SliceSums& S, StridedIn X,
                 double* Wt, const int32_t* pos, StridedOut out, cudaStream_t s) {
    prof::Scope ps("slice_reduce_rows", s, 0.0, 8.0 * (c.rows.splits + 1) * (double)c.k * r.R);
    // as many rows a block as leave two blocks for every SM if all columns are summed directly, and within
    // 32-bit offsets (four million bytes a row, sixteen million samples, before that binds)
    const int64_t groups = (c.k + kDirectCols - 1) / kDirectCols;
    int rpb = kDirectRows;
    while (rpb > 64 && ((r.R + rpb - 1) / rpb * groups < 2 * num_sms() || rpb * r.stride >> 32)) rpb /= 4;
    launch_chained(k_slice_reduce_rows, dim3((unsigned)((r.R + rpb - 1) / rpb), (unsigned)c.k), 256, 0, s,
                   so.part.get(), r.r_pad, r.R, c.k, rpb, r.s.get(), r.mu.get(), PackedRows{r.rows, r.stride}, X,
                   r.n, S, Wt, pos, out);
    CS_LAUNCH("slice_reduce_rows");
}

// CS_B200_FP64_DMMA or CS_B200_FP64_NARROW, which choose among the FP64-pipe kernels, keep these.
bool pipe_kernels_chosen() {
    static const bool on = std::getenv("CS_B200_FP64_DMMA") || std::getenv("CS_B200_FP64_NARROW");
    return on;
}

// Columns per call of the passes, at most kChunkColumns, whose operands `reserve(columns)` finds device memory
// for: half as many after each failure (`release` gives back what was had), until it throws for eight.
template <class Reserve, class Release>
int64_t widest_chunk(int64_t k, Reserve&& reserve, Release&& release) {
    for (int64_t w = kChunkColumns;; w = std::min(w, k) / 2) {
        try {
            if (k >= w) reserve(w);
            if (k % w) reserve(k % w);
            return w;
        } catch (const OutOfMemory&) {
            release();
            if (std::min(w, k) / 2 < 8) throw;
        }
    }
}

// The operator's slice state with room for chunks of `columns` of the k columns; null without a
// sample-major copy where that is needed and not allowed, or without device memory for it or for the
// operands.  In that case it gives back what it had taken and is tried again by the first call that
// finds the memory.  The slices are taken at every shape: against the
// FP64-pipe kernels an apply took (us) 27 / 99 at n=40, M=1000 and one column, 31 / 152 at n=2000,
// M=10000, 930 / 7210 at n=50000, M=100000; 35 / 187, 86 / 470 and 168 / 954 at n=2000, M=10000 and
// 8, 80 and 200 columns; 2900 / 23480 at n=18009, M=27006 and 266.
struct SliceRoom {
    SliceOperator* so = nullptr;
    int64_t columns = 0;
    explicit operator bool() const { return so != nullptr; }
};

SliceRoom slices_for(cs_kinship* op, int64_t k, bool samples, cudaStream_t s) {
    const int64_t R = op->n_active;
    if (!op->sample_major_copy || R == 0 || k <= 0 || pipe_kernels_chosen()) return {};
    if (op->slices_need && device_room() < op->slices_need) return {};
    MixedRows* r = nullptr;
    bool new_copy = false;
    try {
        r = &mixed_rows_for(op);
        configure_slices();
        new_copy = samples && !r->packed_t.get();
        if (!op->slices) op->slices = new SliceOperator();
        SliceOperator& so = *op->slices;
        make_status(so, s);
        if (!so.map_rows) {
            so.tm_packed = make_map_u8(r->rows, r->stride, R, r->stride, 128, kTile, true);
            so.map_rows = true;
        }
        if (samples) ensure_transposed(*r, s);
        if (samples && !so.map_samples) {
            so.tm_packed_t = make_map_u8(r->packed_t.get(), r->r_pad / 4, r->n_pad, r->r_pad / 4, 128, kTile, true);
            so.map_samples = true;
        }
        const int64_t columns = widest_chunk(
            k, [&](int64_t w) { reserve(so, *r, plan_call(*r, w)); }, [&] { so.release_operands(); });
        op->slices_need = 0;
        return {&so, columns};
    } catch (const OutOfMemory&) {
        // the FP64-pipe kernels need neither the copy nor the operands
        destroy_slices(op->slices);
        op->slices = nullptr;
        op->slices_need = 1;
        if (r) op->slices_need += operand_bytes(*r, plan_call(*r, std::min<int64_t>(k, 8)));
        if (new_copy) {
            r->packed_t.release();
            op->slices_need += (size_t)(r->n_pad * r->r_pad / 4);
        }
        return {};
    }
}

template <class Chunk>
void for_chunks(const MixedRows& r, int64_t k, int64_t columns, Chunk&& chunk) {
    for (int64_t c0 = 0; c0 < k; c0 += columns)
        chunk(c0, plan_call(r, std::min(columns, k - c0)));
}

StridedIn from_column(StridedIn m, int64_t c) { return StridedIn{m.p + c * m.cs, m.rs, m.cs}; }
StridedOut from_column(StridedOut m, int64_t c) { return StridedOut{m.p + c * m.cs, m.rs, m.cs}; }

}  // namespace

bool kinship_apply_slices(cs_kinship* op, StridedIn X, int64_t k, StridedOut Y, cudaStream_t s) {
    const SliceRoom room = slices_for(op, k, true, s);
    if (!room) return false;
    SliceOperator* const so = room.so;
    MixedRows& r = mixed_rows_for(op);
    for_chunks(r, k, room.columns, [&](int64_t c0, const SliceCall& c) {
        const SliceSums S = sums_of(*so, c, c0 == 0 && !op->defer_checks);
        const StridedIn x = from_column(X, c0);
        run_rows(*so, r, c, S, x, s);
        finish_rows(*so, r, c, S, x, so->W.get(), nullptr, StridedOut{}, s);
        run_samples(*so, r, c, S, 1.0 / (double)op->num_variants, from_column(Y, c0), s);
    });
    return true;
}

bool multiply_zt_slices(cs_kinship* op, StridedIn X, int64_t k, StridedOut U, cudaStream_t s) {
    const SliceRoom room = slices_for(op, k, false, s);
    if (!room) return false;
    SliceOperator* const so = room.so;
    MixedRows& r = mixed_rows_for(op);
    for_chunks(r, k, room.columns, [&](int64_t c0, const SliceCall& c) {
        const SliceSums S = sums_of(*so, c, c0 == 0 && !op->defer_checks);
        const StridedIn x = from_column(X, c0);
        run_rows(*so, r, c, S, x, s);
        finish_rows(*so, r, c, S, x, nullptr, op->d_view_pos.get(), from_column(U, c0), s);
    });
    return true;
}

bool multiply_z_slices(cs_kinship* op, StridedIn V, int64_t k, StridedOut Y, cudaStream_t s) {
    const SliceRoom room = slices_for(op, k, true, s);
    if (!room) return false;
    SliceOperator* const so = room.so;
    MixedRows& r = mixed_rows_for(op);
    for_chunks(r, k, room.columns, [&](int64_t c0, const SliceCall& c) {
        const SliceSums S = sums_of(*so, c, c0 == 0 && !op->defer_checks);
        CS_CUDA(cudaMemsetAsync(so->words.get(), 0, 8 * c.words, s));
        {
            prof::Scope ps("slice_gather", s, 0.0, 16.0 * r.R * c.k);
            launch_chained(k_slice_gather, dim3((unsigned)((r.R + 1023) / 1024), (unsigned)c.k), 256, 0, s,
                           from_column(V, c0), r.R, op->d_view_pos.get(), r.s.get(), r.mu.get(), S, so->W.get());
            CS_LAUNCH("slice_gather");
        }
        run_samples(*so, r, c, S, 1.0, from_column(Y, c0), s);
    });
    return true;
}

static void check_slices(SliceOperator* so, cudaStream_t s) {
    if (!so || !so->status.get()) return;
    int status = 0;
    CS_CUDA(cudaMemcpyAsync(&status, so->status.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    CS_CUDA(cudaStreamSynchronize(s));
    if (status != kPassStatusOk) {
        cudaMemsetAsync(so->status.get(), 0, sizeof(int), s);
        cudaStreamSynchronize(s);
        fail(CS_ERR_CUDA, "tensor-core kinship kernel gave up waiting (status " + std::to_string(status) + ")");
    }
}

void check_slices(cs_kinship* op, cudaStream_t s) { check_slices(op->slices, s); }

void clear_slices(cs_kinship* op, cudaStream_t s) {
    if (op->slices && op->slices->status.get())
        CS_CUDA(cudaMemsetAsync(op->slices->status.get(), 0, sizeof(int), s));
}

bool scan_project_slices(SliceOperator*& state, MixedRows& r, StridedIn X, int64_t k, StridedOut T,
                         cudaStream_t s) {
    if (r.R == 0 || k <= 0 || pipe_kernels_chosen()) return false;
    int64_t columns = 0;
    try {
        configure_slices();
        if (!state) state = new SliceOperator();
        SliceOperator& so = *state;
        make_status(so, s);
        if (!so.map_rows) {
            so.tm_packed = make_map_u8(r.rows, r.stride, r.R, r.stride, 128, kTile, true);
            so.map_rows = true;
        }
        auto reserve_rows = [&](const SliceCall& c) {
            so.b.resize(c.rows.b_rows(true) * r.n_pad);
            so.part.resize(c.k * c.rows.splits * r.r_pad);
            so.words.resize(c.words);
        };
        columns = widest_chunk(
            k, [&](int64_t w) { reserve_rows(plan_call(r, w)); }, [&] { so.release_operands(); });
    } catch (const OutOfMemory&) {
        destroy_slices(state);
        state = nullptr;
        return false;
    }
    SliceOperator& so = *state;
    for_chunks(r, k, columns, [&](int64_t c0, const SliceCall& c) {
        const SliceSums S = sums_of(so, c, c0 == 0);
        const StridedIn x = from_column(X, c0);
        run_rows(so, r, c, S, x, s);
        finish_rows(so, r, c, S, x, nullptr, nullptr, from_column(T, c0), s);
    });
    check_slices(&so, s);
    return true;
}

// ---------------------------------------------------------------- the mixed form's narrow passes
bool mixed_narrow_fits(bool rows, int64_t kp) {
    SlicePlan p;
    return kp > 0 && kp <= 256 && lay_out(rows, false, (int)kp, kp, p, 3);
}

void mixed_narrow_pass(bool rows, MixedRows& r, const int8_t* b, int64_t kp, int splits, int kbs,
                       const double* inv_f, double* part, int* status, uint32_t poll_ns, cudaStream_t s) {
    configure_slices();
    SlicePlan p;
    // long slices: two more stages are worth more than an epilogue beside the next unit's MMAs
    // (N=50k, M=100k, a product of 20 columns 1.22 ms against 1.38)
    if (!lay_out(rows, false, (int)kp, kp, p, 3, kbs >= 64 ? 6 : 4)) fail(CS_ERR_UNSUPPORTED, "narrow pass: too many columns");
    p.splits = splits;
    p.kbs = kbs;
    const int64_t m = rows ? r.r_pad : r.n_pad, kk = rows ? r.n_pad : r.r_pad;
    const int kb = (int)(kk / kKBlock);
    SliceArgs A = slice_args(p, rows, m / kTile, kb, kp);
    A.kb_total = kb;
    A.hw = (int)(3 * kp);
    A.lut = r.lut.get();
    A.mu = rows ? r.resid.get() : inv_f;
    A.part = part;
    A.ld = m;
    A.status = status;
    A.poll_ns = poll_ns;
    const int64_t stride = rows ? r.stride : r.r_pad / 4, packed_rows = rows ? std::max<int64_t>(r.R, 1) : r.n_pad;
    const CUtensorMap ta = make_map_u8(rows ? r.rows : r.packed_t.get(), stride, packed_rows, stride, 128, kTile, true);
    const CUtensorMap tb = make_map_u8(b, kk, (rows ? 3 : 6) * kp, kk, kKBlock, p.set_rows, true);
    if (rows)
        launch_slice_pass<true, false, 3>(p, ta, tb, A, s);
    else
        launch_slice_pass<false, false, 3>(p, ta, tb, A, s);
}

}  // namespace cs
