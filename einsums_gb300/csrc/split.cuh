// Split-BF16 ("Ozaki") form of the canonical contraction.
//
// Every FP64 operand row (a fixed (batch, m) of A, or (batch, n) of B, over
// all summed modes k) is scaled by its own power of two 2^e, |x| < 2^e, and
// cut into S balanced base-256 digits:
//     x = 2^(e-7) * sum_{s<S} a_s 2^(-8 s),   a_s integer in [-128, 128]
// so each digit ("slice") is exact in BF16 and a slice product is an integer
// below 2^14.  The product of two rows is
//     sum_k A B = 2^(eA+eB-14) * sum_d 2^(-8 d) G_d,   G_d = sum_{s+t=d} sum_k a_s b_t
// and the triangular truncation keeps d < S (S(S+1)/2 slice pairs).  The
// tensor cores accumulate G_d in FP32 over chunks of at most 1024 products,
// which keeps every partial sum an integer of at most 2^24 and therefore
// exact; the epilogue converts each chunk to an integer and accumulates
//     R = sum_d 2^(8 (S-1-d)) G_d
// exactly in int64 in registers.  The only roundings of the whole
// product are the digit truncation and the final int64 -> FP64 conversion.
// This is the scheme of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59,
// 2012) as mapped to integer-exact tensor-core products by Ootomo, Ozaki and
// Yokota (IJHPCA 2024), with BF16 digits and FP32 accumulation.
#pragma once

#include <climits>

#include <cuda.h>

#include "common.cuh"

namespace eg::split {

constexpr int kBits = 8;        // digit width
constexpr int kTopBits = 7;     // magnitude bits of the leading digit
constexpr int kMaxSlices = 6;   // keeps the scaled digits and the int64 accumulator in range
constexpr int kBM = 128, kBN = 128, kBK = 64;
// The FP64 form: eight slices (63 bits below each row's power of two) and the
// accuracy check of launch_f64_tensor.
constexpr int kF64Slices = 8, kF64High = 4;
// The check of one output over its N products that are not zero, M the sum of their leading
// magnitudes' products (p_a p_b): it passes when N = 0, or N >= 8 and M >= 20 N, or N >= 2 and
// M >= 20 N + 256.  A product that stands alone is left to the FMA kernel, which rounds it once.
constexpr float kTriedMean = 32.0f; // of p_a p_b, see left_out in tc_gemm.cu
constexpr int kCheckPer = 20, kCheckFew = 8, kCheckMore = 256;
__host__ __device__ constexpr bool check_fails(int products, int excess) { // excess: M - 20 N
    return products == 1 || (products > 1 && excess < (products < kCheckFew ? kCheckMore : 0));
}
// The check of one K slice of a tile, to be added up: the excess, below a bound that no sum
// over the slices falls back from (the least is -20 65536), and N, where 8 stands for more.
__host__ __device__ constexpr int pack_check(int products, int excess) {
    return (excess < (1 << 22) ? excess : 1 << 22) * 16 + (products < kCheckFew ? products : kCheckFew);
}
constexpr int kTileRegions = 8; // parts of a tile, one per epilogue warp: 32 rows by 64 columns in turns of 16
constexpr int kChunkKB = 16;    // 16 x 64 = 1024 products per exact FP32 chunk
constexpr int kKStep = 2 * kBK;  // granularity of the longest exact pass (K itself is padded to kBK)

struct TcGemmParams {
    int S;
    int planes; // planes per batch index of each operand: S, or S + 2 in the FP64 form
    int nkb;  // K blocks in this pass
    int kb0;  // first K block of this pass
    int mtiles, ntiles, nbatch;
    int64_t M, N;
    int Mp, Np;
    ModeGroup bg, mg, ng; // output offsets in C (component 2)
    double *C;
    double cp, ab;
    int ab_pow2; // ab = +-2^k: folded into the exponent (ab_neg gives the sign)
    int ab_neg;
    int zero;
    const int *eA; // [nbatch][Mp] row exponents; INT_MIN marks a non-finite row
    const int *eB; // [nbatch][Np]
    int shift_const; // -14 - 8 (S-1), plus k when ab = +-2^k
    // Where a wait that gives up is recorded: the executing stream's word -- *status_at when set
    // (lists, which do not know the stream before they run) -- and this call's own, which the
    // launches that follow look at.
    int *status;
    int *const *status_at;
    int *lost;
    unsigned long long timeout_ns;
    // Optional per-CTA cycle counters (null in normal runs): see kProf* in tc_gemm.cu.
    unsigned long long *prof;
    // Per-CTA scratch of gridDim.x * 128 * 128 int64, where a finished tile's sums wait
    // (in the FP64 form three such planes: the low sums, and the high sums of two tiles).
    long long *rbuf;
    // The first t0 schedule entries are whole tiles.  The tiles left for the last,
    // partly filled round of the CTAs (all of them when there are fewer tiles than
    // CTAs) are cut along K so that the round is full: entry t >= t0 is K slice
    // (t - t0) % ksplit (kslice K blocks; the last slice takes the rest) of
    // tile t0 + (t - t0) / ksplit.  A slice's exact int64 sums go to parts ([t - t0]
    // [128 columns][128 rows], two planes in the FP64 form; with CTA pairs an entry is
    // two tiles, one after the other) and its outputs' checks (pack_check) to parts_check
    // ([t - t0][128][128]); k_tc_finish_slices adds them up.  Unused when t0 is the number of tiles.
    int t0;
    int ksplit, kslice;
    long long *parts;
    int *parts_check;
    // Launch as CTA pairs (cta_group::2, 256x128 tiles): single contractions only.
    int pair;
    // Slice groups d0 <= d < d1 (anti-diagonals s + t = d of the digit pairs)
    // summed by this launch: all of them (0, S) unless a long K is split into
    // group ranges whose exact sums each fit int64 (finished into C one by one).
    int d0, d1;
    // First batch index, row and column of the panel of C this launch computes (0 when
    // it computes all of it): mt, nt and the exponents count from there.
    int64_t b0, m0, n0;
    // FP64 form (redo set): the exact sums do not fit 64 bits, so the slice groups
    // below hid form one int64 sum and the others a second; a region of
    // a tile whose accuracy check fails is left alone and listed in redo ({batch, row,
    // column}, in grouped launches {item, batch, row, column}; redo_count entries) for
    // the FMA kernel.
    int hid;
    int4 *redo;
    int *redo_count;
    // Grouped launches: two tensor maps per item (A, B) over the item's own digit
    // planes with its own row and K extents, so that TMA fills the tile's rows
    // past M (N) and K blocks past K with zeros instead of reading the padding.
    const CUtensorMap *item_maps;
    const int *ranges; // each CTA's work entries
    // FP64 form: the sums of the leading magnitudes (p_a of the check) over all of A and all of B.
    // Grouped launches: [item][2].  Else, may be null, of a sample of rows: A's sum, the number of
    // its elements that are not zero, and the same of B.
    const unsigned long long *magnitudes;
};

// Records a wait that gave up in the executing stream's word.
__device__ __forceinline__ void report_lost(int *const *status_at, int *status, int code) {
    atomicCAS(status_at ? *status_at : status, 0, code);
}

// One item of a grouped launch: an independent contraction whose digit planes have
// tensor maps of their own (TcGemmParams::item_maps) and whose exponents start at
// eAoff / eBoff.  Work entries (int4) are {item, batch index, mt, nt}.
struct TcItem {
    double *C;
    int64_t M, N;
    int nkb;
    float tried; // the product of its two magnitudes from which on the item is tried (left_out)
    int eAoff, eBoff;
    int Mp, Np;
    ModeGroup bg, mg, ng;
};

// The bits of x, by way of an instruction the compiler does not look into: it turns
// tests on the fields of a double's bits into FP64 comparisons, which run on this
// GPU's slow FP64 pipe (a third of the splitting kernels' time).
__device__ __forceinline__ unsigned long long bits_of(double x) {
    unsigned long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
}

// IEEE bit pattern of |x|: for non-negative doubles (and NaN above Inf) the
// unsigned order of the patterns is the numeric order.
__device__ __forceinline__ unsigned long long abs_bits(double x) { return bits_of(x) & 0x7FFFFFFFFFFFFFFFull; }

// The exponent of a row whose largest |x| has the given bits: |x| < 2^e (INT_MIN for
// a row holding an infinity or NaN, 0 for a row of zeros).
__device__ __forceinline__ int row_exponent(unsigned long long bits) {
    const int field = (int)(bits >> 52);
    if (field == 0x7ff) return INT_MIN;
    if (field) return field - 1022;
    return bits ? -1010 - __clzll((long long)bits) : 0; // subnormal: 2^-1074 times the bits
}

// For row_exponent: the largest |x|'s bits among n values of a row in shared memory
// (16-byte aligned, readable and zero up to an even count), found by a warp.  The
// exponent field decides, so the upper words do, at two instructions a value and with a
// lower word of zero, unless all are subnormal.
__device__ __forceinline__ unsigned long long row_max_bits(const double *row, int n, int lane) {
    uint32_t mx = 0;
    for (int k = 2 * lane; k < n; k += 64) {
        const uint4 v = *(const uint4 *)&row[k];
        mx = max(mx, max(v.y & 0x7FFFFFFFu, v.w & 0x7FFFFFFFu));
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (mx >= 0x00100000u) return (unsigned long long)mx << 32;
    unsigned long long m = 0;
    for (int k = lane; k < n; k += 32) m = max(m, abs_bits(row[k]));
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    return m;
}

// round(x * 2^sh) to nearest, ties to even, for |x| 2^sh < 2^63, built from the
// IEEE fields with integer operations (the FP64 pipe of this GPU runs about two
// operations per clock per SM; this is the splitting kernels' inner loop).
// SHRINKS: |x| 2^sh < 2^48, so that there is always a bit to drop.
template <bool SHRINKS = false>
__device__ __forceinline__ long long scaled_round(double x, int sh) {
    const unsigned long long bits = bits_of(x);
    const uint32_t hi = (uint32_t)(bits >> 32);
    const int ex = (int)((hi >> 20) & 0x7ff);
    const uint32_t top = (hi & 0xFFFFFu) | (ex != 0 ? 0x100000u : 0u);
    const unsigned long long mant = ((unsigned long long)top << 32) | (uint32_t)bits;
    const int r = 1075 - max(ex, 1) - sh; // |x| 2^sh = mant 2^-r
    unsigned long long q;
    if (!SHRINKS && r <= 0) {
        q = mant << (-r < 63 ? -r : 63); // a whole number already
    } else if (r > 62) {
        q = 0; // below 1/2
    } else {
        // round half to even in one add: the carry out of the r low bits happens
        // exactly when they exceed half, or equal half with an odd quotient
        q = (mant + ((1ull << (r - 1)) - 1ull) + ((mant >> r) & 1ull)) >> r;
    }
    return (int)hi < 0 ? -(long long)q : (long long)q;
}

// |sum| * 2^e rounded to nearest (ties to even), built with integer operations so the
// FP64 pipe -- about 1.75 operations per clock per SM on this GPU -- is left for
// the one fused multiply-add with C.  x holds the leading one at bit 63 (or is 0),
// its value x 2^(e - lz); the bits below its lowest are known to be zero or only
// break ties (they are or-ed into bit 0).
//   FAST: e lies in [kFastMin, kFastMax], so the result is a normal number;
//   otherwise one rounding also where the result is subnormal, and infinity beyond
//   the largest number -- with no floating-point fallback, which the compiler would
//   run for every element beside the integer path.
constexpr int kFastMin = -1000, kFastMax = 900; // sums have up to 96 bits
template <bool FAST>
__device__ __forceinline__ double pack_rn(unsigned long long x, int lz, bool neg, int e) {
    const int biased = 1086 - lz + e; // exponent field of the leading one
    const unsigned long long sign = neg ? 0x8000000000000000ull : 0ull;
    unsigned long long bits;
    if constexpr (FAST) {
        const uint32_t low = (uint32_t)x;
        const uint32_t up = (low & 0x7FFu) + ((low >> 11) & 1u) > 0x400u ? 1u : 0u;
        // the leading one of the 53-bit mantissa carries into the exponent field
        bits = ((unsigned long long)(uint32_t)(biased - 1) << 52) + (x >> 11) + up;
    } else {
        const int drop = 11 + (biased > 0 ? 0 : min(1 - biased, 54)); // fewer bits below the smallest normal number
        const int r = min(drop, 63);
        unsigned long long mant = x >> r;
        const unsigned long long rem = x << (64 - r); // the dropped bits, the half at bit 63
        const unsigned long long half = 0x8000000000000000ull;
        mant += (rem > half || (rem == half && (mant & 1ull))) ? 1ull : 0ull;
        if (drop > 63) mant = drop == 64 && x > half ? 1ull : 0ull; // at most half of the smallest subnormal
        bits = ((unsigned long long)(biased > 0 ? biased - 1 : 0) << 52) + mant;
        if (biased > 2047) bits = 0x7FF0000000000000ull;
        bits = min(bits, 0x7FF0000000000000ull);
    }
    return x ? __longlong_as_double((long long)(bits | sign)) : 0.0;
}

template <bool FAST = false>
__device__ __forceinline__ double int_times_pow2_rn(long long R, int e) {
    const unsigned long long a = R < 0 ? (unsigned long long)(-R) : (unsigned long long)R;
    const int lz = __clzll((long long)a);
    return pack_rn<FAST>(a << (lz & 63), lz, R < 0, e);
}

// The same for the exact sum (hi 2^32 + lo), negated if neg; |hi| < 2^62.
template <bool FAST>
__device__ __forceinline__ double words_times_pow2_rn(long long hi, long long lo, bool neg, int e) {
    hi += lo >> 32;
    uint32_t w = (uint32_t)lo; // the sum is hi 2^32 + w
    const bool minus = hi < 0;
    if (minus) {
        hi = ~hi + (w == 0 ? 1 : 0);
        w = 0u - w;
    }
    if (hi == 0) {
        hi = w;
        w = 0;
        e -= 32;
    }
    const int lz = __clzll(hi);
    const unsigned long long below = (unsigned long long)w << 32;
    const unsigned long long x = ((unsigned long long)hi << (lz & 63)) | (lz > 0 && lz < 64 ? below >> (64 - lz) : 0ull) |
                                 ((below << (lz & 63)) != 0 ? 1ull : 0ull);
    return pack_rn<FAST>(x, lz, minus != neg, e + 32);
}

// The leading digit: G >> 8(S-1), except that with eight slices G = F + bias may
// leave 64 bits, so there the carry out of the low bytes is added to F's own top.
template <int S>
__device__ __forceinline__ int top_digit(long long F, unsigned long long G, long long bias) {
    if constexpr (S < 8) {
        return (int)((long long)G >> (8 * (S - 1)));
    } else {
        constexpr unsigned long long low = (1ull << 56) - 1;
        return (int)(F >> 56) + (int)((((unsigned long long)F & low) + (unsigned long long)bias) >> 56);
    }
}

// The digits of two values as BF16 pairs: out[s] holds digit s of x0 in its low
// half and digit s of x1 in its high half — the same digits as to_digits.  With
// B = 127 (256^(S-2) + ... + 256 + 1), G = F + B has the ordinary base-256
// digits d_s + 127 in [0, 255] for s >= 1 and G >> 8(S-1) = d_0, so one 64-bit
// add replaces the subtract-and-shift chain.  A byte u becomes the float u - 127
// exactly as (2^23 + u) - (2^23 + 127) (bit OR, then an FP32 add), and d_0 as
// (1.5 * 2^23 + d_0) - 1.5 * 2^23; every digit has at most 8 significant bits,
// so its BF16 is the float's upper half, and one byte permute packs the pair.
template <int S>
__device__ __forceinline__ void digits_bf16x2(double x0, double x1, int e, uint32_t *out) {
    constexpr long long bias = [] {
        long long b = 0;
        for (int s = 1; s < S; s++) b = b * 256 + 127;
        return b;
    }();
    const int sh = kTopBits + kBits * (S - 1) - e;
    constexpr bool SHRINKS = S <= 6; // below 2^(7 + 8 (S - 1)), at most 2^47
    const long long F0 = scaled_round<SHRINKS>(x0, sh), F1 = scaled_round<SHRINKS>(x1, sh);
    const unsigned long long G0 = (unsigned long long)F0 + bias, G1 = (unsigned long long)F1 + bias;
    const uint32_t g0[2] = {(uint32_t)G0, (uint32_t)(G0 >> 32)};
    const uint32_t g1[2] = {(uint32_t)G1, (uint32_t)(G1 >> 32)};
#pragma unroll
    for (int s = 1; s < S; s++) {
        // byte S-1-s of G next to the bytes 00 00 4B: the float 2^23 + u in one permute
        const int byte = S - 1 - s, w = byte >> 2;
        const uint32_t sel = 0x7440u | (uint32_t)(byte & 3);
        const float f0 = __uint_as_float(__byte_perm(g0[w], 0x4B000000u, sel)) - 8388735.0f;
        const float f1 = __uint_as_float(__byte_perm(g1[w], 0x4B000000u, sel)) - 8388735.0f;
        out[s] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
    }
    const int t0 = top_digit<S>(F0, G0, bias), t1 = top_digit<S>(F1, G1, bias);
    const float f0 = __int_as_float(0x4B400000 + t0) - 12582912.0f;
    const float f1 = __int_as_float(0x4B400000 + t1) - 12582912.0f;
    out[0] = __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}

// The two check planes of the FP64 form for the pair whose leading digits are
// d0 (as floats in the halves of `lead`): max(|a_0| - 1, 0), at most 128 |x| 2^-e,
// and 1 where x is not zero.
__device__ __forceinline__ uint32_t check_magnitude(uint32_t lead) {
    const float f0 = fmaxf(fabsf(__uint_as_float(lead << 16)) - 1.0f, 0.0f);
    const float f1 = fmaxf(fabsf(__uint_as_float(lead & 0xFFFF0000u)) - 1.0f, 0.0f);
    return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}
__device__ __forceinline__ float pair_sum(uint32_t pair) { // of BF16 numbers
    return __uint_as_float(pair << 16) + __uint_as_float(pair & 0xFFFF0000u);
}
__device__ __forceinline__ uint32_t check_mark(double x0, double x1) {
    return (abs_bits(x0) ? 0x3F80u : 0u) | (abs_bits(x1) ? 0x3F800000u : 0u);
}

// Sets the kernels' shared-memory attribute, once for a device (call outside stream capture).
eg_status ensure_tc_attributes();
// Clusters of two k_tc_split_gemm CTAs that fit on the GPU at once (0 when CTA pairs
// are switched off with EINSUMS_GB300_TC_PAIRS=0), and whether they are asked for
// wherever they can run (EINSUMS_GB300_TC_PAIRS=1).
int tc_pair_clusters();
bool tc_pairs_forced();
// tmBh: B's planes in boxes of 64 rows (half a tile), read by CTA pairs.
eg_status launch_tc_gemm(const CUtensorMap &tmA, const CUtensorMap &tmB, const CUtensorMap &tmBh, const TcGemmParams &p,
                         cudaStream_t s);
// Grouped form: CTA c of `grid` runs the work entries of TcGemmParams::ranges[c] ..
// ranges[c + 1], per-tile parameters from `items`.
eg_status launch_tc_gemm_grouped(const CUtensorMap &tmA, const CUtensorMap &tmB, const TcGemmParams &p,
                                 const TcItem *items, const int4 *work, int grid, cudaStream_t s);

// Bytes of the per-CTA sum scratch a tensor launch needs (TcGemmParams::rbuf).
inline size_t rbuf_bytes(int planes = 1) { return (size_t)num_sms() * planes * kBM * kBN * sizeof(long long); }

// Largest K (a multiple of kKStep) one pass may sum without the int64
// accumulator overflowing 2^62 for S slices.
// Largest K (a multiple of kKStep) for which the exact sum over slice groups
// d0 <= d < d1, R = sum_d 2^(8 (d1-1-d)) G_d, stays below 2^62 in magnitude:
// |G_d| <= (d+1) K 2^14.
inline int64_t max_k_per_pass_groups(int d0, int d1) {
    double w = 0.0;
    for (int d = d0; d < d1; d++) w += (d + 1) * std::ldexp(1.0, 8 * (d1 - 1 - d));
    double kmax = std::ldexp(1.0, 62) / (std::ldexp(1.0, 14) * w);
    int64_t k = kmax > 9.0e18 ? INT64_MAX : (int64_t)kmax;
    return (k / kKStep) * kKStep;
}

inline int64_t max_k_per_pass(int S) { return max_k_per_pass_groups(0, S); }

// A-priori bound on the relative error of one product, relative to
// sum_k |A_row| |B_col| scaled to the row maxima: the dropped digit tail of
// both operands plus the dropped cross terms with s + t >= S.
inline double error_bound(int S) {
    const double u = std::ldexp(1.0, -(kTopBits + kBits * (S - 1))); // one unit of the last digit, relative
    return (S + 2) * u;
}

} // namespace eg::split
