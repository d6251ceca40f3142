// ozaki.cuh -- exact-digit BF16 products on the tcgen05 tensor cores.
//
// An FP64 operand row (a grid line, a spinor chunk, a point's spinor values,
// a matrix row) is scaled by a power of two chosen from its largest exponent
// and rounded to a signed integer of 47 bits, then written as six balanced
// base-256 digits (|d| <= 128), each exact in BF16.  Digit a is stored
// pre-scaled by 2^(-8a), so the product of digit a of one row and digit b of
// another carries its weight 2^(-8(a+b)) by itself.  Products are exact in
// FP32; sums of up to 2^8 products of one weight stay below 2^22 and are
// exact too.  Pairs of weight 0, 1 and 2 go to three accumulators that stay
// exact; all pairs of weight 3..5 share a fourth, whose FP32 rounding sits
// near 2^-48 of the result; pairs of weight 6 and above (below 2^-48) are
// dropped.  The epilogue adds the four accumulators as a double-float and
// multiplies by the two powers of two: 2^(E_row + E_col - 12), E being the
// exponent of each row's largest entry (2^E <= max < 2^(E+1)).
//
// After Ozaki, Ogita, Oishi, Rump, "Error-free transformations of matrix
// multiplication by using fast routines of matrix multiplication", Numer.
// Algorithms 59 (2012), with integer digits as in Ootomo, Ozaki, Yokota,
// "DGEMM on integer matrix multiplication unit", IJHPCA 2024.
#pragma once

#include <stdint.h>

#include <cmath>
#include <cstring>

#include "df.cuh"
#include "tc.cuh"

namespace mg {
namespace oz {

constexpr int kDigits = 6;                       // digits per operand entry
constexpr long long kDigitBias = 0x8080808080LL; // 128 in each of the five lower digits
constexpr uint32_t kAccs = 4;                    // accumulators per output

// float bit pattern of (u - 128) * 2^(-8A) for byte u of w, selected by sel
template <int A>
__device__ __forceinline__ uint32_t low_digit(uint32_t w, uint32_t sel) {
    constexpr uint32_t ebits = (uint32_t)(150 - 8 * A) << 23;   // 2^(23-8A), even exponent
    constexpr float off = (float)(8388608.0 + 128.0) * (1.0f / (float)(1ull << (8 * A)));
    const float f = __uint_as_float(__byte_perm(w, ebits, sel)) - off;
    return __float_as_uint(f);
}

// Biased exponent field of an FP64 value (0 for zero and subnormals).
__device__ __forceinline__ int bexp(double v) {
    return (int)(((unsigned long long)__double_as_longlong(v) >> 52) & 0x7FF);
}

// A row's entries become signed integers round(v * 2^f), f = 8 kDigits - 2 -
// (emax - 1023) for its largest biased exponent emax: |result| <= 2^47 (FixedRow).
// The fixed-point value of a float (part of a double-float), exact when
// the float's bits lie above 2^-f, rounded otherwise.
__device__ __forceinline__ long long fixed_f(float v, int emax) {
    const uint32_t u = __float_as_uint(v);
    const int ef = (int)((u >> 23) & 0xFFu);
    if (ef == 0) return 0;
    const long long m = (long long)((u & 0x7FFFFFu) | 0x800000u);
    // v * 2^f = m * 2^sh with f = 8 kDigits - 2 - (emax - 1023)
    const int sh = ef - 150 + (8 * kDigits - 2) - (emax - 1023);
    long long X;
    if (sh >= 0) X = sh < 39 ? (m << sh) : 0;   // above the row bound: not reached
    else if (sh > -40) X = (m + (1ll << (-sh - 1))) >> (-sh);
    else X = 0;
    return (u >> 31) ? -X : X;
}

// The pre-scaled digits (top digit first) of a fixed-point value X
// (|X| <= 2^47), as FP32 bit patterns whose upper halves are the exact BF16
// values.
__device__ __forceinline__ void digits_fixed(long long X, uint32_t (&d)[kDigits]) {
    const unsigned long long Y = (unsigned long long)(X + kDigitBias);
    const uint32_t ylo = (uint32_t)Y, yhi = (uint32_t)(Y >> 32);
    const int top = (int)yhi >> 8;   // Y >> 40 (arithmetic), in [-128, 128]
    d[0] = __float_as_uint(__int_as_float(0x4B400000 + top) - 12582912.0f);
    // digit a (a = 1..5) is byte (5 - a) of Y, biased by 128
    d[1] = low_digit<1>(yhi, 0x7540);
    d[2] = low_digit<2>(ylo, 0x7543);
    d[3] = low_digit<3>(ylo, 0x7542);
    d[4] = low_digit<4>(ylo, 0x7541);
    d[5] = low_digit<5>(ylo, 0x7540);
}

// Digits of 4 fixed-point values of a row as one 8-byte half of a core-matrix row
// per digit plane.
__device__ __forceinline__ void digits4_fixed(const long long (&X)[4], uint2 (&w)[kDigits]) {
    uint32_t x[kDigits][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t d0[kDigits], d1[kDigits];
        digits_fixed(X[2 * h], d0);
        digits_fixed(X[2 * h + 1], d1);
#pragma unroll
        for (int a = 0; a < kDigits; ++a) x[a][h] = __byte_perm(d0[a], d1[a], 0x7632);
    }
#pragma unroll
    for (int a = 0; a < kDigits; ++a) w[a] = make_uint2(x[a][0], x[a][1]);
}

// ---- eight digits: operands of 62 bits, results rounded once to FP64 -----------
//
// The FP64 form of a contraction over at most 128 terms.  Every entry is rounded to
// 62 bits of its row's largest (FP64 carries 53 of its own) and the 36 digit pairs of
// weight 0..7 are kept, each weight in an accumulator of its own, whose sums are exact
// (8 pairs x 128 terms x 2^14 = 2^24).  The epilogue adds weights 6 and 7 in FP32
// (rounded at 2^-61 of the largest product of the two rows, which is 2^12 in these
// units), takes all to a 64-bit integer in units of 2^-56 of it, and rounds that to
// FP64.  A chain of FP64 FMAs rounds every partial sum.  Norm-wise errors against
// extended-precision sums on Lagrange lines (5 to 32 points, folded and full):
// first derivatives 0.5e-16 to 1.1e-16 (the chain: 1.3e-16 to 2.8e-16),
// Laplacians 0.8e-16 to 2.4e-16 (1.5e-16 to 3.0e-16).
// (Seven digits, 55 bits, were not enough: second derivatives are small
// differences of large products, and 2.6e-15 came out where the chain has
// 2.6e-16.)

constexpr int kDigits64 = 8;
constexpr int kAccs64 = 8;
// product units: 2^(E_row + E_col - kUnit64), E as above
constexpr int kUnit64 = 10;

// power g of the fixed-point form round(v * 2^g) of a row with exponent E:
// one bit fewer than ND digits hold with eight, so that 64-bit integers do
template <int ND>
__host__ __device__ constexpr int fixed_power(int E) {
    return 8 * ND - (ND == kDigits64 ? 3 : 2) - E;
}

// What turns the values of a row into fixed-point words: per row, from the
// largest biased exponent emax of the row (rows with emax of 0 or near 2046
// are for the caller to leave out).
template <int ND>
struct FixedRow;

// Six digits: 47-bit integers, rounded half away from zero
// (one variable shift: floor((m + 2^(s-1)) / 2^s) = floor((floor(m / 2^(s-1)) + 1) / 2)).
template <>
struct FixedRow<kDigits> {
    int emax;
    __device__ __forceinline__ explicit FixedRow(int e) : emax(e) {}
    __device__ __forceinline__ unsigned long long biased(double v) const {
        const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
        const int e = (int)((hi >> 20) & 0x7FFu);
        const unsigned long long m = ((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo;
        const long long t = (long long)(((m >> min(53 - 8 * kDigits + emax - e, 63)) + 1) >> 1);
        const long long X = e == 0 ? 0 : t;
        return (unsigned long long)(((int)hi < 0 ? -X : X) + kDigitBias);
    }
};

// Eight digits: 53 bits shifted up by 9, down by the exponent's distance from
// the row's largest, in two's complement (so that what the shift drops, below
// 2^-61 of the largest, is rounded down).
template <>
struct FixedRow<kDigits64> {
    int emax;
    __device__ __forceinline__ explicit FixedRow(int e) : emax(e) {}
    __device__ __forceinline__ unsigned long long biased(double v) const {
        const uint32_t hi = (uint32_t)__double2hiint(v), lo = (uint32_t)__double2loint(v);
        const int e = (int)((hi >> 20) & 0x7FFu);
        const long long sgn = (long long)((int)hi >> 31);
        const long long m = (long long)((((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo) << 9);
        const long long X = (m ^ sgn) >> min(emax - e, 63);
        return (unsigned long long)(e == 0 ? 0 : X) + 0x80808080808080ULL;
    }
};

// The pre-scaled digits (top digit first) of a fixed-point value plus the
// digit bias.
template <int ND>
__device__ __forceinline__ void digits_of(unsigned long long Y, uint32_t (&d)[ND]) {
    static_assert(ND == kDigits || ND == kDigits64, "six or eight digits");
    const uint32_t ylo = (uint32_t)Y, yhi = (uint32_t)(Y >> 32);
    // the top digit is Y >> 8 (ND - 1) (arithmetic)
    const int top = (int)yhi >> (ND == kDigits ? 8 : 24);
    d[0] = __float_as_uint(__int_as_float(0x4B400000 + top) - 12582912.0f);
    if constexpr (ND == kDigits) {
        // digit a (a = 1..5) is byte (5 - a) of Y, biased by 128
        d[1] = low_digit<1>(yhi, 0x7540);
        d[2] = low_digit<2>(ylo, 0x7543);
        d[3] = low_digit<3>(ylo, 0x7542);
        d[4] = low_digit<4>(ylo, 0x7541);
        d[5] = low_digit<5>(ylo, 0x7540);
    } else {
        // digit a (a = 1..7) is byte (7 - a) of Y
        d[1] = low_digit<1>(yhi, 0x7542);
        d[2] = low_digit<2>(yhi, 0x7541);
        d[3] = low_digit<3>(yhi, 0x7540);
        d[4] = low_digit<4>(ylo, 0x7543);
        d[5] = low_digit<5>(ylo, 0x7542);
        d[6] = low_digit<6>(ylo, 0x7541);
        d[7] = low_digit<7>(ylo, 0x7540);
    }
}

// Digits of 4 values of a row as one 8-byte half of a core-matrix row per
// digit plane.
template <int ND>
__device__ __forceinline__ void digits4(const double (&v)[4], const FixedRow<ND>& row,
                                        uint2 (&w)[ND]) {
    uint32_t x[ND][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t d0[ND], d1[ND];
        digits_of<ND>(row.biased(v[2 * h]), d0);
        digits_of<ND>(row.biased(v[2 * h + 1]), d1);
#pragma unroll
        for (int a = 0; a < ND; ++a) x[a][h] = __byte_perm(d0[a], d1[a], 0x7632);
    }
#pragma unroll
    for (int a = 0; a < ND; ++a) w[a] = make_uint2(x[a][0], x[a][1]);
}

// A float that is a multiple of 2^-P below 2^(22 - P) (or any smaller value,
// rounded to one) plus the magic number 1.5 * 2^(23 - P): its bits are the
// integer multiple plus magic_bits(P).
template <int P>
__device__ __forceinline__ uint32_t units(uint32_t bits) {
    constexpr float magic = 12582912.0f / (float)(1ull << P);
    return __float_as_uint(__fadd_rn(__uint_as_float(bits), magic));
}
__host__ __device__ constexpr uint32_t magic_bits(int P) { return 0x4B400000u - ((uint32_t)P << 23); }

// I 2^(x - 44) as FP64, rounded once with integer instructions (an FP64
// instruction holds a warp's slot of the FP64 pipe for 16 clocks).  The caller keeps
// x between -900 and 900.
__device__ __forceinline__ double round64(unsigned long long I, int x) {
    const uint32_t sgn = (uint32_t)((int)(uint32_t)(I >> 32) >> 31);
    const unsigned long long s64 = ((unsigned long long)sgn << 32) | sgn;
    const unsigned long long u = (I ^ s64) - s64;
    uint32_t h = (uint32_t)(u >> 32), l = (uint32_t)u;
    int e = 1023 + 63 - 44 + x;
    if (h == 0) {
        h = l;
        l = 0;
        e -= 32;
    }
    const int lz = __clz((int)h);
    if (h == 0) return 0.0;
    h = __funnelshift_l(l, h, lz);
    l <<= lz;
    // 53 bits with the hidden one, rounded to nearest
    const unsigned long long r = ((((unsigned long long)h << 32) | l) >> 11) + ((l >> 10) & 1u);
    const uint32_t rh = (uint32_t)(r >> 32) + ((uint32_t)(e - lz - 1) << 20);
    return __hiloint2double((int)(rh | (sgn & 0x80000000u)), (int)(uint32_t)r);
}

// The eight accumulators' sum times 2^x as FP64: a 64-bit integer in units
// of 2^-44 (top digits are at most 64, so 32 products stay below 2^18 and the
// integer below 2^62), rounded once.  The accumulators' magic numbers are carried
// along and taken off once.
__device__ __forceinline__ double combine64(const uint32_t (&a)[kAccs64], int x) {
    const uint32_t hi = units<0>(a[0]) * 256u + units<8>(a[1]);     // 2^-8
    const uint32_t mid = units<16>(a[2]) * 256u + units<24>(a[3]);  // 2^-24, with its magic >= 0
    const uint32_t low = units<32>(a[4]) * 256u + units<40>(a[5]);  // 2^-40, with its magic >= 0
    const uint32_t tail = units<44>(__float_as_uint(__fadd_rn(__uint_as_float(a[6]), __uint_as_float(a[7]))));
    constexpr uint32_t mhi = magic_bits(0) * 256u + magic_bits(8);
    constexpr uint32_t mmid = magic_bits(16) * 256u + magic_bits(24);
    constexpr uint32_t mlow = magic_bits(32) * 256u + magic_bits(40);
    constexpr unsigned long long off = ((unsigned long long)mhi << 36) +
                                       ((unsigned long long)mmid << 20) +
                                       ((unsigned long long)mlow << 4) + magic_bits(44);
    const unsigned long long I = (unsigned long long)mid * (1ull << 20) +
                                 ((unsigned long long)low * 16u + tail) +
                                 ((unsigned long long)(hi << 4) << 32) - off;
    return round64(I, x);
}

// The same for sums of up to 128 products (6 pairs x 128 x 2^14 < 2^24 are exact in
// FP32 but past the magic numbers' range; the whole sum is below 2^63 units), and for
// any x.
__device__ __forceinline__ double combine64_any(const uint32_t (&a)[kAccs64], int x) {
    const auto part = [](float x, int up, int shift) {
        // a multiple of 2^-up below 2^(31 - up) as an integer, shifted
        const float f = x * __int_as_float((up + 127) << 23);
        return (unsigned long long)(long long)__float2int_rn(f) << shift;
    };
    const auto acc = [&a](int g) { return __uint_as_float(a[g]); };
    const unsigned long long I = part(acc(0), 0, 44) + part(acc(1), 8, 36) +
                                 part(acc(2), 16, 28) + part(acc(3), 24, 20) +
                                 part(acc(4), 32, 12) + part(acc(5), 40, 4) +
                                 part(__fadd_rn(acc(6), acc(7)), 44, 0);
    if (x >= -900 && x <= 900) return round64(I, x);
    // past the exponent range of one step: two exact ones and a rounding
    const int first = x < 0 ? max(x, -1960) / 2 : min(x, 1960) / 2;
    const int rest = (x < 0 ? max(x, -1960) : min(x, 1960)) - first;
    return round64(I, 0) * __longlong_as_double((long long)(first + 1023) << 52) *
           __longlong_as_double((long long)(rest + 1023) << 52);
}

// a0 + a1 + a2 + a3 as a normalised double-float.  a0 is an integer below
// 2^22, a1 a multiple of 2^-8 below 2^15, a2 a multiple of 2^-16 below 2^8
// (all exact); a3 is the small rounded remainder.  With a1 = i1 + f1
// (integer and fractional parts), a0 + i1 and f1 + a2 are exact float sums;
// one TwoSum of those two is exact, and a3 joins the low part before the
// final renormalisation (it is far below the high part).
__device__ __forceinline__ dfl combine4(float a0, float a1, float a2, float a3) {
    const float i1 = truncf(a1);
    const float f1 = __fsub_rn(a1, i1);
    const dfl s = df_two_sum(__fadd_rn(a0, i1), __fadd_rn(f1, a2));
    return df_norm(dfl{s.h, __fadd_rn(s.l, a3)});
}

// 2^x as a float for -126 <= x <= 127, 0 below (values under 2^-126 are
// dropped; they are far below the grid values)
__device__ __forceinline__ float pow2f(int x) {
    return x < -126 ? 0.0f : __int_as_float((min(x, 127) + 127) << 23);
}

// ---- digit-pair MMAs ------------------------------------------------------------
//
// The pairs of a block of `cols` columns with nd digits go into accumulators side by
// side, `cols` columns each: a weight a + b its own one, in the mixed form the weights
// from 3 on the last one together.  The B planes of the block are stacked row below
// row, so that plane a times planes b, b + 1, ... is one MMA of up to 256 columns over
// accumulators a + b, a + b + 1, ...: an MMA of 32 columns holds the tensor pipe for
// as long as one of 256 (~130 clocks), and with a pair per MMA the issue of 84 to 144
// of them per tile bound the derivative kernel.
//
// The order of two MMAs into one accumulator is only given where both have the same
// accumulator columns and the same shape.  So the accumulators come in groups of
// `width`, and every MMA into a group covers all of it: for the accumulators before a,
// which have no pair of digit a, the stack begins with planes of zeros.
__host__ __device__ constexpr int own_accs(int nd) {   // accumulators of one weight
    return nd == kDigits64 ? kAccs64 : (int)kAccs - 1;
}
constexpr int kStackCols = 192;
// the fewest groups that this allows, of even width (what is left over: the first)
__host__ __device__ constexpr int stack_width(int nd, int cols) {
    const int own = own_accs(nd), most = kStackCols / cols < own ? kStackCols / cols : own;
    const int groups = (own + most - 1) / most;
    return (own + groups - 1) / groups;
}
__host__ __device__ constexpr int stack_zeros(int nd, int cols) { return stack_width(nd, cols) - 1; }
// planes of a block with its zeros
__host__ __device__ constexpr int stack_planes(int nd, int cols) { return stack_zeros(nd, cols) + nd; }

// mma(a, b, ks, acc, count, first): plane a times planes b .. b + count - 1 (zeros where
// negative), K step ks, into accumulators acc .. acc + count - 1; `first`: the first MMA
// into them.
template <int ND, int COLS, int KSTEPS, class Mma>
__host__ __device__ __forceinline__ void stacked_pairs(Mma mma) {
    constexpr int own = own_accs(ND), width = stack_width(ND, COLS);
    constexpr int rest = (own - 1) % width + 1;   // the first group: as many MMAs as its end
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ++ks)
#pragma unroll
        for (int a = 0; a < own; ++a)
#pragma unroll
            for (int end = rest; end <= own; end += width) {
                const int count = end == rest ? rest : width;
                if (end > a) mma(a, end - count - a, ks, end - count, count, ks == 0 && a == 0);
            }
    // the weights that share the last accumulator, one pair at a time in order of weight and a
#pragma unroll
    for (int c = own; c < ND; ++c)
#pragma unroll
        for (int a = 0; a <= c; ++a)
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks)
                mma(a, c - a, ks, own, 1, c == own && a == 0 && ks == 0);
}

// A planes at aBase + a aPlane, the stacked B planes at bBase, behind stack_zeros(ND,
// COLS) planes of zeros.  accumulate: the accumulators hold an earlier K stage's sums.
template <int ND, int COLS, int KSTEPS>
__device__ __forceinline__ void issue_stacked(uint32_t tmem, uint32_t aBase, uint32_t aPlane,
                                              uint32_t bBase, uint32_t sbo,
                                              bool accumulate = false) {
    constexpr uint32_t bPlane = COLS * KSTEPS * 32;
    constexpr int zeros = stack_zeros(ND, COLS);
    const uint64_t da = tc::desc_sbo(aBase, sbo), db = tc::desc_sbo(bBase - zeros * bPlane, sbo);
    // the descriptors' address field counts 16 bytes
    stacked_pairs<ND, COLS, KSTEPS>([&](int a, int b, int ks, int acc, int count, bool first) {
        tc::mma_bf16(tmem + (uint32_t)(acc * COLS), da + ((a * aPlane + ks * tc::kKStep) >> 4),
                     db + (((b + zeros) * bPlane + ks * tc::kKStep) >> 4),
                     tc::idesc_bf16(128, count * COLS), first && !accumulate ? 0u : 1u);
    });
}

// Host form of the digits: BF16 bit patterns of the pre-scaled digits of
// round(x * scale), scale a power of two, top first.
inline void host_digits(double x, double scale, uint16_t* out, int nd = kDigits) {
    const long long X = std::llrint(x * scale);
    long long bias = 0;
    for (int b = 1; b < nd; ++b) bias = bias * 256 + 128;
    const long long Y = X + bias;
    float weight = 1.0f;   // 2^(-8 b)
    for (int b = 0; b < nd; ++b, weight *= 1.0f / 256.0f) {
        const int j = nd - 1 - b;   // byte position
        const float d = b == 0 ? (float)(Y >> (8 * j)) : (float)((int)((Y >> (8 * j)) & 0xFF) - 128);
        const float f = d * weight;
        uint32_t u;
        std::memcpy(&u, &f, 4);
        out[b] = (uint16_t)(u >> 16);
    }
}

// The power g = 8 kDigits - 2 - E used for a row whose largest |entry| is mx,
// and E itself (0 for an all-zero row).
inline int host_row_exponent(double mx) {
    if (!(mx > 0.0)) return 0;
    int fe;
    std::frexp(mx, &fe);   // mx = f * 2^fe, 0.5 <= f < 1
    return fe - 1;
}

}  // namespace oz
}  // namespace mg
