/*
 * scft_pass_tc.cu — one axis pass of the contour step on the tensor cores, with
 * the rounding of the value type: y = K x for every line of one grid axis, K the
 * dense diffusion operator of that axis (funPDESolver_periodic and
 * funPDESolver_DirichletBC, SCFT.c:2474-2631, apply the same factor by FFTs).
 *
 * GB300 issues FP64 at 1/58 of its FP32 rate and a double-float product costs
 * 8-12 FP32 instructions, so a pass in either arithmetic is bound by its
 * multiply-adds (192x96 film: 85 % of the FP64 rate in the dense z pass at
 * large batches, 3 % of the copy bandwidth). Here the contraction runs on the
 * fp16 tensor cores without rounding, by the splitting scheme of Ozaki, Ogita,
 * Oishi and Rump ("Error-free transformations of matrix multiplication by using
 * fast routines of matrix multiplication and its applications", Numer. Algor.
 * 59, 2012):
 *   - a line becomes integers X = x 2^e with one exponent per line (58 bits
 *     for FP64 and FP32x2 values, 28 for FP32);
 *   - the operator commutes with the reversal of the axis and, on a periodic
 *     axis of length 4k, with the shift by half its length: integer sums and
 *     differences split it into NB = 2 or 4 blocks of size n/NB, exactly;
 *   - block operands and operators are cut into balanced digits of 10 bits,
 *     which fp16 holds exactly, |digit| <= 512. Digit pairs (i, j) with i + j = l
 *     share the FP32 accumulator of level l; the levels kept (6 of FP64's, 4 of
 *     FP32's) leave out terms of 2^-56 (2^-27) of the line's largest value;
 *   - a level's sum is an integer, which the accumulator holds exactly up to 2^24.
 *     Its bound, 512 times the sum of the operator's digits up to that level over a
 *     row, is taken from the digits when the table is made (tc_table). Where it stays
 *     below, the sums are taken as they are; where it does not, what is above 2^9 is
 *     carried to the level above after every 16 points: on every level for operators
 *     that reach over many points, whose digits and those of a flat line add up with
 *     one sign, so that all levels are exact; on levels 1 to 3 of FP64 and FP32x2 for
 *     the others (long axes, 1.05 times 2^24 on level 3 of 192 points). Their last two
 *     levels, and FP32's, then rest on the digits' mixed signs: twelve standard
 *     deviations away, and a unit that is lost is below 2^-56 (FP32: 2^-27);
 *   - the levels are joined in 64-bit integers (FP32: three multiply-adds), and
 *     each output is rounded once to the value type.
 * Results do not depend on the tile, the number of output parts, the carries or what
 * shares the launch: every line is computed by the same integer arithmetic.
 *
 * A CTA takes `tile` lines and a range of output chunks. Data digits and
 * operator digits sit in shared memory as 8 x 16-byte cells, which ldmatrix
 * reads without conflicts; a warp multiplies 16 lines x 8 outputs with
 * mma.sync and joins the levels in its own registers. The same products by
 * tcgen05.mma (accumulators in tensor memory, 64 or 128 lines) measured slower
 * at every size tried: the MMAs of a chunk of 16 outputs took 1100-2000 clocks
 * from issue to completion, the accumulators (24 words for 4 outputs) had to
 * pass through shared memory to reach all warps (1200 clocks), and a tile fills
 * 8-48 of the 64 rows. 192x96 film, FP64, 32 instances: 16.3 ms an iteration
 * against 12.7; 64^3 blend: 18.4 against 14.3. The passes are bound by the
 * integer pipe (splitting, joining: ~100 operations per value, 2 issue slots
 * each) and by the rate of mma.sync (~13 clocks each on an SM quarter).
 * Measured against the FP64 and double-float passes (FFT along periodic axes,
 * dense products along the others), ms per iteration, contour steps and all:
 * 192x96 film, one FP64 instance 4.36 -> 1.15, 32 FP64 instances 46.5 -> 10.9,
 * 16 FP32x2 instances 11.4 -> 5.8; 64^3 four-diblock blend, FP64, 56.0 -> 14.1;
 * 150x75 film, FP32, 4 instances 2.65 -> 1.22. Errors against 64-bit references
 * are no larger than before in every form.
 *
 * A line with a NaN or an infinity comes out as NaN.
 */
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "scft_dfloat.cuh"
#include "scft_internal.h"
#include "scft_mbar.cuh"
#include "scft_pdl.cuh"

/* Set when a tensor-core wait of a pass gave up (the tile is then written as NaN). */
__device__ int g_scft_pass_fault;

namespace {

constexpr int W = 8;      /* block outputs of a chunk (the N of an MMA) */
constexpr int ROWS = 128; /* lines of the largest tile */
constexpr int GROUPS = 2; /* groups of warps of k_chain_tc, each with its own tiles */

/* digits of the data, of the operator, and levels kept */
template <typename P>
struct Dig {
    static constexpr int S = 6, SK = 6, L = 6;
};
template <>
struct Dig<float> {
    static constexpr int S = 3, SK = 4, L = 4;
};

template <typename P>
struct FixT {
    using T = long long;
};
template <>
struct FixT<float> {
    using T = int;
};

/* biased exponent of a value (0: zero or subnormal, taken as zero) */
__device__ __forceinline__ int expo(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ int expo(dfloat x) { return (__float_as_int(x.hi) >> 23) & 0xff; }
__device__ __forceinline__ int expo(float x) { return (__float_as_int(x) >> 23) & 0xff; }
template <typename P>
struct ExpoMax {
    static constexpr int v = std::is_same<P, double>::value ? 2047 : 255; /* infinities and NaN */
};

/* x 2^s as an integer, s such that values below 2^(emax + 1 - bias) stay below
 * 2^(58 - NB/4) (FP32: 2^(28 - NB/4), rounded to nearest; the others drop bits
 * below that, of which a value within 2^-5 of the line's largest has none).
 * Subnormals count as zero, and in FP64 both as 2^-1023, which lines above 2^-965
 * shift out: the range is that of the normal numbers, with an error of the smallest.
 * (Taking such lines up by a power of two first keeps subnormals too, but the test for
 * it in the digits cost 1-3 % of a whole solve, 192x96 in FP64 6.83 -> 6.87-7.06 ms.) */
template <int NB>
__device__ __forceinline__ long long fix(double x, int emax)
{
    const int hi = __double2hiint(x);
    const unsigned lo = (unsigned)__double2loint(x), h = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const long long m = (long long)(((unsigned long long)__funnelshift_l(lo, h, 10) << 32) | (lo << 10)); /* leading bit 62 */
    const long long v = m >> min(emax - ((hi >> 20) & 0x7ff) + (NB == 4 ? 6 : 5), 63);
    return hi < 0 ? -v : v;
}
template <int NB>
__device__ __forceinline__ long long fix_part(float x, int emax)
{
    const int b = __float_as_int(x), e = (b >> 23) & 0xff;
    const unsigned long long m = (unsigned long long)(((unsigned)b & 0x7fffffu) | 0x800000u) << (NB == 4 ? 33 : 34);
    const int d = min(emax - e, 63); /* lo's exponent is never above hi's */
    const long long v = e ? (long long)(m >> d) : 0;
    return b < 0 ? -v : v;
}
template <int NB>
__device__ __forceinline__ long long fix(dfloat x, int emax)
{
    return fix_part<NB>(x.hi, emax) + fix_part<NB>(x.lo, emax);
}
template <int NB>
__device__ __forceinline__ int fix(float x, int emax)
{
    const int b = __float_as_int(x), e = (b >> 23) & 0xff;
    const unsigned m = (((unsigned)b & 0x7fffffu) | 0x800000u) << (NB == 4 ? 3 : 4);
    const int d = min(emax - e, 30);
    const int v = e ? (int)((m + ((1u << d) >> 1)) >> d) : 0;
    return b < 0 ? -v : v;
}

/* Digit i (0 = top) of two biased integers as a half2 of balanced digits: the
 * fields' 16-bit windows side by side, masked, made 1024 + f in fp16, less 1536
 * (the top field reaches 1024, so it has a mask of its own and is added). */
template <int S, typename U>
__device__ __forceinline__ uint32_t digit2(U ya, U yb, int i)
{
    const int bit = 10 * (S - 1 - i);
    uint32_t t;
    if (sizeof(U) == 8 && bit / 8 == 3) { /* the window straddles the words */
        t = __byte_perm((uint32_t)(ya >> 24), (uint32_t)(yb >> 24), 0x5410);
    } else {
        const int word = sizeof(U) == 8 && bit >= 32 ? 1 : 0, byte = bit / 8 - 4 * word;
        const uint32_t wa = word ? (uint32_t)((unsigned long long)ya >> 32) : (uint32_t)ya;
        const uint32_t wb = word ? (uint32_t)((unsigned long long)yb >> 32) : (uint32_t)yb;
        t = __byte_perm(wa, wb, byte == 0 ? 0x5410 : byte == 1 ? 0x6521 : 0x7632);
    }
    t >>= bit % 8;
    t = i == 0 ? (t & 0x07ff07ffu) + 0x64006400u : (t & 0x03ff03ffu) | 0x64006400u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&t), __half2half2(__ushort_as_half(0x6600))); /* 1536 */
    return *reinterpret_cast<const uint32_t *>(&h);
}

/* the block operands of two points from the points' NB images, and their digits into the item's cells */
template <typename P, int NB, typename Fix>
__device__ __forceinline__ void put_digits(Fix (&X)[NB][2], unsigned char *cell)
{
    constexpr int S = Dig<P>::S;
    using UFix = typename std::make_unsigned<Fix>::type;
    constexpr UFix BIAS = S == 6 ? (UFix)0x0802008020080200ull : (UFix)0x20080200u; /* 512 in every field */
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        if constexpr (NB == 4) { /* half-axis sums, then mirror sums */
            const Fix a0 = X[0][q] + X[2][q], a1 = X[1][q] + X[3][q], b0 = X[0][q] - X[2][q], b1 = X[1][q] - X[3][q];
            X[0][q] = a0 + a1;
            X[1][q] = a0 - a1;
            X[2][q] = b0 + b1;
            X[3][q] = b0 - b1;
        } else {
            const Fix s = X[0][q] + X[1][q];
            X[1][q] = X[0][q] - X[1][q];
            X[0][q] = s;
        }
    }
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        const UFix ya = (UFix)X[b][0] + BIAS, yb = (UFix)X[b][1] + BIAS;
#pragma unroll
        for (int i = 0; i < S; ++i)
            *reinterpret_cast<uint32_t *>(cell + (i * NB + b) * 128) = digit2<S, UFix>(ya, yb, i);
    }
}

/* two consecutive values of a row, 16-byte aligned (FP32: 8) */
__device__ __forceinline__ void ld2(const double *p, double (&v)[2])
{
    const double2 t = __ldcg(reinterpret_cast<const double2 *>(p));
    v[0] = t.x;
    v[1] = t.y;
}
__device__ __forceinline__ void ld2(const dfloat *p, dfloat (&v)[2])
{
    const float4 t = __ldcg(reinterpret_cast<const float4 *>(p));
    v[0] = dfloat(t.x, t.y);
    v[1] = dfloat(t.z, t.w);
}
__device__ __forceinline__ void ld2(const float *p, float (&v)[2])
{
    const float2 t = __ldcg(reinterpret_cast<const float2 *>(p));
    v[0] = t.x;
    v[1] = t.y;
}
/* the same from shared memory */
__device__ __forceinline__ void lds2(const double *p, double &a, double &b)
{
    const double2 t = *reinterpret_cast<const double2 *>(p);
    a = t.x;
    b = t.y;
}
__device__ __forceinline__ void lds2(const dfloat *p, dfloat &a, dfloat &b)
{
    const float4 t = *reinterpret_cast<const float4 *>(p);
    a = dfloat(t.x, t.y);
    b = dfloat(t.z, t.w);
}
__device__ __forceinline__ void lds2(const float *p, float &a, float &b)
{
    const float2 t = *reinterpret_cast<const float2 *>(p);
    a = t.x;
    b = t.y;
}
__device__ __forceinline__ void st2(double *p, double a, double b) { *reinterpret_cast<double2 *>(p) = make_double2(a, b); }
__device__ __forceinline__ void st2(dfloat *p, dfloat a, dfloat b)
{
    *reinterpret_cast<float4 *>(p) = make_float4(a.hi, a.lo, b.hi, b.lo);
}
__device__ __forceinline__ void st2(float *p, float a, float b) { *reinterpret_cast<float2 *>(p) = make_float2(a, b); }
__device__ __forceinline__ double ld1(const double *p) { return __ldcg(p); }
__device__ __forceinline__ float ld1(const float *p) { return __ldcg(p); }
__device__ __forceinline__ dfloat ld1(const dfloat *p)
{
    const float2 t = __ldcg(reinterpret_cast<const float2 *>(p));
    return dfloat(t.x, t.y);
}

/* factors that no one writes after pdl_wait(): they may stay in L1. Ordinary loads, as the
 * kernel can have started while the one before it wrote them: the read-only path
 * (ld.global.nc, __ldg) wants data that no one writes from a kernel's start on, and neither
 * the wait nor the compiler orders it */
__device__ __forceinline__ double ldc(const double *p) { return *p; }
__device__ __forceinline__ float ldc(const float *p) { return *p; }
__device__ __forceinline__ dfloat ldc(const dfloat *p)
{
    const float2 t = *reinterpret_cast<const float2 *>(p);
    return dfloat(t.x, t.y);
}

/* four 8 x 8 matrices of 16-bit values from shared memory, rows of 16 bytes at each lane's address */
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
/* c += a b: 16 rows x 8 columns x 16 points */
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

/* What is above 2^9 in the sums of levels FROM to TO, an integer, moved to the level above,
 * so that the next 16 points add to sums of at most 2^15: exact, two sums at a time.
 * Upwards, so that no step waits for the one before it. Always done it costs 2-6 % of a whole
 * solve (192x96, FP64 6.83 -> 6.97-7.12 ms, 150x75 FP32 4.84 -> 5.16), hence only where an
 * operator needs it, in kernels of their own, as the test for it alone costs 2 %. */
template <int FROM, int TO, int L>
__device__ __forceinline__ void carry_sums(float (&d)[L][4])
{
#pragma unroll
    for (int l = FROM; l <= TO; ++l)
#pragma unroll
        for (int v = 0; v < 4; v += 2)
            asm("{\n\t.reg .b64 x, u, t, c;\n\t"
                "mov.b64 x, {%0, %1};\n\tmov.b64 u, {%2, %3};\n\t"
                "mov.b64 t, {0f4B400000, 0f4B400000};\n\tmov.b64 c, {0f3A800000, 0f3A800000};\n\t"
                "fma.rn.f32x2 t, x, c, t;\n\t" /* 1.5 2^23 + x / 1024: its unit is 1 */
                "mov.b64 c, {0fCB400000, 0fCB400000};\n\tadd.rn.f32x2 t, t, c;\n\t"
                "add.rn.f32x2 u, u, t;\n\t"
                "mov.b64 c, {0fC4800000, 0fC4800000};\n\tfma.rn.f32x2 x, t, c, x;\n\t"
                "mov.b64 {%0, %1}, x;\n\tmov.b64 {%2, %3}, u;\n\t}"
                : "+f"(d[l][v]), "+f"(d[l][v + 1]), "+f"(d[l - 1][v]), "+f"(d[l - 1][v + 1]));
}
/* Before the next 16 points, and after half of the digit pairs of 16 points, where five or six
 * of them alone could pass 2^24. how: InstOps::tc_carry of the axis. */
template <int L>
__device__ __forceinline__ void carry_step(float (&d)[L][4], int how)
{
    if (how) carry_sums<1, 3>(d);
    if (L > 4 && how > 1) carry_sums<4, L - 1>(d);
}
template <int L>
__device__ __forceinline__ void carry_half(float (&d)[L][4], int how)
{
    if (L > 4 && how > 1) carry_sums<4, L - 1>(d);
}
/* In the end, so that the last level rounds into the one above alike whichever pairs came first. */
template <int L>
__device__ __forceinline__ void carry_end(float (&d)[L][4], int how)
{
    if (L > 4 && how > 1) {
        carry_sums<L - 1, L - 1>(d);
        carry_sums<L - 2, L - 2>(d);
    }
}

__device__ __forceinline__ long long mad_wide(int a, int b, long long c)
{
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
/* Levels of one block output joined: 64-bit integer in units of 2^60 of the
 * digit products (level 5 rounds into level 4), FP32: a float in units of 2^50. */
__device__ __forceinline__ long long join(const float (&d)[6][4], int v)
{
    long long y = __float2int_rn(fmaf(d[5][v], 0x1p-10f, d[4][v]));
    y = mad_wide(__float2int_rn(d[3][v]), 1 << 10, y);
    y = mad_wide(__float2int_rn(d[2][v]), 1 << 20, y);
    y = mad_wide(__float2int_rn(d[1][v]), 1 << 30, y);
    return y + ((long long)(__float2int_rn(d[0][v]) << 8) << 32);
}
__device__ __forceinline__ float join(const float (&d)[4][4], int v)
{
    return fmaf(fmaf(fmaf(d[3][v], 0x1p-10f, d[2][v]), 0x1p-10f, d[1][v]), 0x1p-10f, d[0][v]);
}

/* The joined value back in the value type, rounded once; the scales of fix() and
 * of the operator table are folded into the exponents.
 * FP64, the rare cases: a value below 2^-25 of its line's largest, exponents
 * near the ends of the range, lines of zeros (or subnormals, which come out as zeros). */
__device__ __noinline__ double from_fix_slow(long long acc, int emax)
{
    const unsigned long long u = acc < 0 ? (unsigned long long)-acc : (unsigned long long)acc;
    if (emax == 0 || u == 0) return 0.0;
    const int lz = __clzll((long long)u), eb = emax + 7 - lz; /* biased exponent */
    const unsigned long long m = u << lz;
    if (eb < -51) return 0.0;
    const int sh = eb > 0 ? 11 : 12 - eb; /* a subnormal's units are 2^-1074 */
    unsigned long long r = (m >> sh) + ((m >> (sh - 1)) & 1);
    if (eb > 0) r += (unsigned long long)(eb - 1) << 52;
    if (eb >= 2047) r = 0x7ff0000000000000ull;
    return __longlong_as_double((long long)(r | ((unsigned long long)acc & 0x8000000000000000ull)));
}
__device__ __forceinline__ void from_fix(long long acc, int emax, double &y)
{
    /* |acc| < 2^58; the integer pipe bounds this phase, so in 32-bit steps */
    const unsigned long long u = (unsigned long long)(acc < 0 ? -acc : acc);
    const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
    if ((unsigned)(emax - 300) > 1400u || hi == 0) {
        y = from_fix_slow(acc, emax);
        return;
    }
    const int top = 31 - __clz((int)hi), k = 25 - top; /* leading bit to 57, then 53 bits */
    unsigned h = __funnelshift_l(lo, hi, k), l = lo << k;
    asm("add.cc.u32 %0, %0, 16;\n\taddc.u32 %1, %1, 0;" : "+r"(l), "+r"(h));
    l = __funnelshift_r(l, h, 5);
    h = (h >> 5) + (unsigned)(emax - 25 + top) * (1u << 20); /* the leading bit adds one to the exponent */
    y = __hiloint2double((int)(h | ((unsigned)((unsigned long long)acc >> 32) & 0x80000000u)), (int)l);
}
__device__ __forceinline__ void from_fix(long long acc, int emax, dfloat &y)
{
    /* three signed pieces of 20 bits and what is above, exact in FP32 */
    const int p0 = ((int)acc << 12) >> 12;
    const long long a1 = (acc - p0) >> 20;
    const int p1 = ((int)a1 << 12) >> 12;
    const int p2 = (int)((a1 - p1) >> 20);
    const dfloat s = dfo::fast_two_sum((float)p2 * 0x1p-16f, (float)p1 * 0x1p-36f);
    const dfloat t = dfo::fast_two_sum(s.hi, dfo::f_add(s.lo, (float)p0 * 0x1p-56f));
    const float sc = __int_as_float(emax << 23);
    y = dfloat(t.hi * sc, t.lo * sc);
}
__device__ __forceinline__ void from_fix(float acc, int emax, float &y)
{
    y = (acc * 0x1p-16f) * __int_as_float(emax << 23);
}

__device__ __forceinline__ void set_nan(double &y) { y = __longlong_as_double(0x7ff8000000000000ll); }
__device__ __forceinline__ void set_nan(dfloat &y) { y = dfloat(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000)); }
__device__ __forceinline__ void set_nan(float &y) { y = __int_as_float(0x7fc00000); }

/* Shared memory (byte offsets): one barrier per axis, four sets of line
 * exponents (two for each group of warps, see k_chain2d_tc for its own), operator
 * digits (one region per axis), then the digits of a tile's lines. */
constexpr uint32_t SM_BAR = 0, SM_FAIL = 32, SM_ELINE = 64, SM_OP = SM_ELINE + 4 * ROWS * 4;
/* k_chain2d_tc: what peers send for an axis, and what the tile in hand keeps of it */
__host__ __device__ constexpr uint32_t sm_received(int ax) { return SM_ELINE + ax * ROWS * 4; }
__host__ __device__ constexpr uint32_t sm_kept(int set) { return SM_ELINE + (2 + set) * ROWS * 4; }

/* bytes of a tile's digits (an MMA of a pass reads 16 lines, of the loops 8) */
__host__ __device__ inline uint32_t tile_bytes(const TcGeom &g, int digits, int lines)
{
    return (uint32_t)((g.tile + lines - 1) / lines * lines) * g.hp * g.nb * digits * 2;
}

/* bytes of the exchange of block sums in the loops, for a part of the outputs */
__host__ __device__ inline uint32_t exchange_bytes(const TcGeom &g, int value)
{
    return (uint32_t)g.tile * (g.cpp * W * g.nb + 4) * value;
}

/* Level sums of 16 outputs (chunks 2 cp, 2 cp + 1) x 8 lines (group rg) of block b: tiles of 8
 * lines fill the MMA. ldmatrix rows: operator (8 outputs, 8 points) cells at (output half, point
 * half) = (lane >> 3 & 1, lane >> 4), line cells at (digit, point half) = (lane >> 4, lane >> 3 & 1).
 * d[.][v]: output (lane >> 2) + 8 (v >> 1), line 2 (lane & 3) + (v & 1). */
template <typename P, int NB, bool CARRY>
__device__ __forceinline__ void products16x8(float (&d)[Dig<P>::L][4], uint32_t op, uint32_t lines, int nk8, int ks, int nc, int rg, int cp, int b, int carry)
{
    constexpr int S = Dig<P>::S, SK = Dig<P>::SK, L = Dig<P>::L, CELL = S * NB * 128;
    const int lane = threadIdx.x & 31;
    const int cc = min(2 * cp + ((lane >> 3) & 1), nc - 1); /* an odd last chunk is read twice */
    const uint32_t a0 = op + (uint32_t)((cc * NB + b) * ks * SK * 256 + (lane >> 4) * 128 + (lane & 7) * 16);
    const uint32_t b0 = lines + (uint32_t)((rg * nk8 + ((lane >> 3) & 1)) * CELL + b * 128 + (lane & 7) * 16);
#pragma unroll
    for (int l = 0; l < L; ++l)
#pragma unroll
        for (int v = 0; v < 4; ++v) d[l][v] = 0.0f;
#pragma unroll 1
    for (int k = 0; k < ks; ++k) {
        if (CARRY && k > 0) carry_step(d, carry);
        uint32_t bf[(S + 1) / 2][4]; /* line digits 2i, 2i + 1 */
#pragma unroll
        for (int i = 0; i < (S + 1) / 2; ++i)
            ldsm4(bf[i], b0 + (uint32_t)(2 * k * CELL + min(2 * i + (lane >> 4), S - 1) * NB * 128));
#pragma unroll
        for (int j = 0; j < SK; ++j) {
            if (CARRY && j == SK / 2) carry_half(d, carry);
            uint32_t af[4];
            ldsm4(af, a0 + (uint32_t)((k * SK + j) * 256));
#pragma unroll
            for (int i = 0; i < S; ++i)
                if (i + j < L) mma16816(d[i + j], af, bf[i / 2][2 * (i & 1)], bf[i / 2][2 * (i & 1) + 1]);
        }
    }
    if (CARRY) carry_end(d, carry);
}

/* Where a CTA (or a group of its warps) is. */
struct TcPhase {
    uint32_t tile; /* tiles done */
    bool ok;       /* no wait has given up */
};

/* ---- lines that pass between the CTAs of a cluster through shared memory (k_chain2d_tc) */

/* Lines of one axis in this CTA's shared memory, and where its outputs go: lines of the other axis. */
template <typename P>
struct Exchange {
    const P *in;       /* the tile's lines, `pitch` values apart */
    const int *eline;  /* their largest exponents, below the step's number; peers write here */
    int *kept;         /* the tile's copy of them, for its outputs */
    int pitch, tag;    /* tag: the number the receiver expects, in place */
    uint32_t out, out_eline, bar; /* offsets in every CTA's shared memory */
    int out_pitch, out_tile;
    unsigned out_mag;  /* ceil(2^32 / out_tile) */
    bool send;
    const P *bz, *bnext; /* after the last axis: this and the next step's factors */
    P *dst;              /* then q_{s+1} */
};
__device__ __forceinline__ uint32_t at_rank(uint32_t addr, uint32_t rank)
{
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
/* two neighbouring values into another CTA's shared memory, counted by its barrier (one store
 * costs the same ~2 clocks a lane whatever its width) */
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, unsigned long long a, unsigned long long b)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr), "l"(a), "l"(b), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, double a, double b)
{
    send(addr, bar, (unsigned long long)__double_as_longlong(a), (unsigned long long)__double_as_longlong(b));
}
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, dfloat a, dfloat b)
{
    send(addr, bar, (unsigned long long)__float_as_uint(a.lo) << 32 | __float_as_uint(a.hi),
         (unsigned long long)__float_as_uint(b.lo) << 32 | __float_as_uint(b.hi));
}
__device__ __forceinline__ void send(uint32_t addr, uint32_t bar, float a, float b)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr), "r"(__float_as_uint(a)),
                 "r"(__float_as_uint(b)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ double swap_rows(double v) { return __shfl_xor_sync(0xffffffffu, v, 4); }
__device__ __forceinline__ float swap_rows(float v) { return __shfl_xor_sync(0xffffffffu, v, 4); }
__device__ __forceinline__ dfloat swap_rows(dfloat v) { return dfloat(swap_rows(v.hi), swap_rows(v.lo)); }
/* the largest of the values sent, counted by the barrier like them */
__device__ __forceinline__ void send_max(uint32_t addr, uint32_t bar, uint32_t v)
{
    asm volatile("red.async.relaxed.cluster.mbarrier::complete_tx::bytes.shared::cluster.max.u32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar)
                 : "memory");
}
constexpr int EBITS = 11; /* bits of an exponent */

/* The tile of k_chain2d_tc: like tc_tile, from lines with their exponents in
 * shared memory to lines of the other axis in their CTAs' shared memory. */
template <typename P, int NB, int NT, bool CARRY>
__device__ __forceinline__ void tc_tile2d(const TcGeom &g, const Exchange<P> &xc, bool last, int tile_i, unsigned char *smem,
                                          uint32_t sm_op, uint32_t sm_a, uint32_t sm_ex, uint32_t bar_op, bool wait_op,
                                          int carry, bool &ok)
{
    constexpr int S = Dig<P>::S, L = Dig<P>::L, CELL = S * NB * 128;
    using Fix = typename FixT<P>::T;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0); /* uniform */
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    const int n = g.n, hb = g.hb, m = n / 2, nk8 = g.hp / 8, nc = g.nchunks;
    const int L0 = tile_i * g.tile, nlines = (int)min((long)g.tile, g.lines - L0);
    auto pos = [&](int p, int k) { /* as in tc_tile */
        if (NB == 2) return p == 0 ? k : n - 1 - k;
        return p == 0 ? k : p == 1 ? m - 1 - k : p == 2 ? k + m : n - 1 - k;
    };

    /* a CTA that has its points may send the next lines while other warps are at this tile's outputs */
    if (tid < g.tile) xc.kept[tid] = xc.eline[tid] & ((1 << EBITS) - 1);
    /* ---- digits: an item is two neighbouring points and their images of one line */
#pragma unroll 1
    for (int idx = tid; idx < g.tile * nk8 * 4; idx += NT) {
        const int u = idx >> 5, rg = nk8 == 1 ? u : (int)__umulhi((unsigned)u, g.mag_nk8), k8 = u - rg * nk8;
        const int r = rg * 8 + ((idx >> 2) & 7), k = k8 * 8 + 2 * (idx & 3);
        const int em = xc.eline[r] & ((1 << EBITS) - 1);
        const P *in = xc.in + r * xc.pitch;
        Fix X[NB][2];
#pragma unroll
        for (int p = 0; p < NB; ++p) {
            P v[2] = {P(0), P(0)};
            if (r < nlines) {
                if (n % 2 == 0 && k + 1 < hb) { /* pairs of an even axis are aligned */
                    lds2(in + ((p & 1) ? pos(p, k + 1) : pos(p, k)), v[p & 1], v[1 - (p & 1)]);
                } else {
#pragma unroll
                    for (int q = 0; q < 2; ++q)
                        if (k + q < hb) v[q] = in[pos(p, k + q)];
                }
            }
            X[p][0] = fix<NB>(v[0], em);
            X[p][1] = fix<NB>(v[1], em);
        }
        put_digits<P, NB>(X, smem + sm_a + u * CELL + (idx & 31) * 4);
    }
    if (wait_op && tid == 0 && !(ok && mbar_wait(bar_op, 0))) *reinterpret_cast<volatile int *>(smem + SM_FAIL) = 1;
    __syncthreads();
    ok = *reinterpret_cast<volatile int *>(smem + SM_FAIL) == 0;

    /* ---- products, 16 outputs x 8 lines of one block at a time */
    using Acc = typename std::conditional<std::is_same<P, float>::value, float, long long>::type;
    Acc *ex = reinterpret_cast<Acc *>(smem + sm_ex);
    const int pitch = nc * W * NB + 4; /* values of a line: block by block, shifted by four from line to line */
    const int nr = (nlines + 7) / 8, np = (nc + 1) / 2, ks = g.hp / 16;
#pragma unroll 1
    for (int u = warp; u < nr * np * NB; u += NT / 32) {
        const int b = u % NB, v = u / NB, rg = nr == 1 ? 0 : v / np, cp = v - rg * np;
        float d[L][4];
        products16x8<P, NB, CARRY>(d, sbase + sm_op, sbase + sm_a, nk8, ks, nc, rg, cp, b, carry);
        Acc *at = ex + (rg * 8 + 2 * (lane & 3)) * pitch + (b * nc + 2 * cp) * W + (lane >> 2);
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < 2 || 2 * cp + 1 < nc) at[(i & 1) * pitch + (i >> 1) * W] = join(d, i);
    }
    __syncthreads();

    /* ---- outputs: a warp takes 8 lines x 4 block outputs, and of these all images, or a pair or one
     * of them where there are too few to go round. Two neighbouring lines' values go in one store:
     * of a pair of images the even line's thread sends the first, the odd one's the second. */
    constexpr int NH = NB / 2; /* pairs of images */
    const int og = nc * (W / 4), units = nr * og;
    const int parts = units * NB <= NT / 32 ? NB : units * NH <= NT / 32 ? NH : 1;
#pragma unroll 1
    for (int w = warp; w < units * parts; w += NT / 32) {
        const int u = parts == 1 ? w : parts == NB ? w / NB : w / NH, part = parts == 1 ? 0 : w - u * parts;
        const int rg = nr == 1 ? 0 : (int)__umulhi((unsigned)u, g.mag_og), k = (u - rg * og) * 4 + (lane & 3), r = rg * 8 + (lane >> 2);
        const bool in = r < nlines && k < hb;
        const int em = xc.kept[r];
        const bool bad = em == ExpoMax<P>::v || !ok;
        const int base = g.ls == 1 ? (L0 + r) * n : L0 + r;
        const int odd = (lane >> 2) & 1;
        const Acc *s = ex + r * pitch + k;
        const Acc sm[2] = {s[0] + s[nc * W], s[0] - s[nc * W]};
        Acc sp[2] = {0, 0};
        if constexpr (NB == 4) {
            sp[0] = s[2 * nc * W] + s[3 * nc * W];
            sp[1] = s[2 * nc * W] - s[3 * nc * W];
        }
        /* image q of pair h: y = q_{s+1} (or the next axis' input) and z, what is sent */
        auto point = [&](int h, int q, int x, bool on, P &y, P &z) {
            P f = P(0);
            if (last && on) f = ldc(xc.bz + base + g.ls * x);
            from_fix(NB == 2 ? sm[q] : h ? sm[q] - sp[q] : sm[q] + sp[q], em, y);
            if (bad) set_nan(y);
            if (last) y = y * f;
            z = y;
            if (last && xc.send) z = y * (xc.bnext == xc.bz ? f : on ? ldc(xc.bnext + base + g.ls * x) : P(0));
        };
        auto put = [&](int x, P a, P b, unsigned e) {
            const int to = xc.out_tile == 1 ? x : (int)__umulhi((unsigned)x, xc.out_mag), row = x - to * xc.out_tile;
            const uint32_t there = at_rank(sbase, to);
            send(there + xc.out + (uint32_t)((row * xc.out_pitch + L0 + r - odd) * sizeof(P)), there + xc.bar, a, b);
            if (lane < 8) send_max(there + xc.out_eline + (uint32_t)row * 4, there + xc.bar, (uint32_t)xc.tag | e);
        };
        if (parts == NB) {
            const int x = pos(part, k);
            const bool line = k < hb && !(NB == 2 && part == 1 && x == k); /* odd n: one middle point */
            P y, z;
            if (part & 1)
                point(part >> 1, 1, x, in && line, y, z);
            else
                point(part >> 1, 0, x, in && line, y, z);
            if (xc.send && ok) { /* nothing is sent after a wait that ran out */
                unsigned e = in ? (unsigned)expo(z) : 0u;
                e = max(e, __shfl_xor_sync(0xffffffffu, e, 4));
                e = max(e, __shfl_xor_sync(0xffffffffu, e, 8));
                e = max(e, __shfl_xor_sync(0xffffffffu, e, 16));
                const P got = swap_rows(z);
                if (line && in && !odd) put(x, z, got, e);
            }
            if (last && in && line) xc.dst[base + g.ls * x] = y;
        } else {
#pragma unroll 1
            for (int h = part; h < NH; h += parts) {
                const int x0 = pos(2 * h, k), x1 = pos(2 * h + 1, k), x = odd ? x1 : x0;
                const bool line1 = !(NB == 2 && x1 == k);
                P y0, y1, z0, z1;
                point(h, 0, x0, in, y0, z0);
                point(h, 1, x1, in && line1, y1, z1);
                if (xc.send && ok) {
                    unsigned e = in ? (unsigned)expo(z0) | (unsigned)expo(z1) << 16 : 0u;
                    e = __vmaxu2(e, __shfl_xor_sync(0xffffffffu, e, 4));
                    e = __vmaxu2(e, __shfl_xor_sync(0xffffffffu, e, 8));
                    e = __vmaxu2(e, __shfl_xor_sync(0xffffffffu, e, 16));
                    const P got = swap_rows(odd ? z0 : z1);
                    if (k < hb && r - odd < nlines && (!odd || line1)) put(x, odd ? got : z0, odd ? z1 : got, odd ? e >> 16 : e & 0xffffu);
                }
                if (last && in) {
                    xc.dst[base + g.ls * x0] = y0;
                    if (line1) xc.dst[base + g.ls * x1] = y1;
                }
            }
        }
    }
}

/* One tile of lines and one part of its outputs: y = K x (times b before the
 * first axis, after the last). Ends with every thread of the CTA past the digits. */
template <typename P, int NB, int NT, bool SPLIT, bool CARRY>
__device__ __forceinline__ void tc_tile(const TcGeom &g, const P *src, P *dst, const P *bz,
                                        bool first, bool last, int tile_i, int part, unsigned char *smem,
                                        uint32_t sm_op, uint32_t sm_a, uint32_t bar_op, bool wait_op, int carry, TcPhase &ph)
{
    constexpr int S = Dig<P>::S, SK = Dig<P>::SK, L = Dig<P>::L;
    using Fix = typename FixT<P>::T;
    using UFix = typename std::make_unsigned<Fix>::type;
    /* SPLIT: a group of NT threads with its own barrier */
    const int tid = SPLIT ? threadIdx.x % NT : threadIdx.x, lane = tid & 31, group = SPLIT ? threadIdx.x / NT : 0;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0); /* uniform */
    auto sync = [&]() {
        if (SPLIT)
            asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(NT) : "memory");
        else
            __syncthreads();
    };
    /* line exponents: one set in use, the other zeroed for the next tile */
    int *eline = reinterpret_cast<int *>(smem + SM_ELINE) + (2 * group + (ph.tile & 1)) * ROWS;
    int *enext = reinterpret_cast<int *>(smem + SM_ELINE) + (2 * group + (~ph.tile & 1)) * ROWS;
    ++ph.tile;
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    const int c0 = part * g.cpp, c1 = min(c0 + g.cpp, g.nchunks);
    const int n = g.n, hb = g.hb, m = n / 2, ls = g.ls, nk8 = g.hp / 8;
    const int L0 = tile_i * g.tile, nlines = (int)min((long)g.tile, g.lines - L0);
    const bool vec = ls == 1 && n % 2 == 0; /* rows of whole pairs (n = 4 j for NB = 4) */
    const int items = g.tile * nk8 * 4;
    constexpr int CELL = S * NB * 128; /* one 8-line, 8-point core matrix of every digit and block */

    /* first element of line r of the tile: rows (the axis is contiguous), columns of
     * one plane (the slowest axis), or the general case */
    auto line_base = [&](int r) {
        const int line = L0 + r;
        if (ls == 1) return line * n;
        if (g.lines == g.inner) return line;
        const int o = line / g.inner;
        return o * n * ls + (line - o * g.inner);
    };

    /* position of point k of side p: 0 k, 1 its mirror; 2, 3 the same half an axis on (NB = 4) */
    auto pos = [&](int p, int k) {
        if (NB == 2) return p == 0 ? k : n - 1 - k;
        return p == 0 ? k : p == 1 ? m - 1 - k : p == 2 ? k + m : n - 1 - k;
    };

    /* ---- load. An item is two neighbouring points (and their images) of one
     * line; the warp's 32 items fill one 8-line core matrix of every digit. The
     * values wait for the line's exponent in the words their digits will take. */
#pragma unroll 1
    for (int idx = tid; idx < items; idx += NT) {
        const int u = idx >> 5, rg = nk8 == 1 ? u : (int)__umulhi((unsigned)u, g.mag_nk8), k8 = u - rg * nk8;
        const int r = rg * 8 + ((idx >> 2) & 7), k = k8 * 8 + 2 * (idx & 3);
        unsigned char *cell = smem + sm_a + u * CELL + (idx & 31) * 4;
        P v[NB][2], bb[NB][2];
        int em = 0;
        const bool on = r < nlines && k < hb;
        const int base = line_base(min(r, nlines - 1));
        if (on && vec && k + 1 < hb) {
#pragma unroll
            for (int p = 0; p < NB; ++p) ld2(src + base + ((p & 1) ? pos(p, k + 1) : pos(p, k)), v[p]);
            if (first) {
#pragma unroll
                for (int p = 0; p < NB; ++p) ld2(bz + base + ((p & 1) ? pos(p, k + 1) : pos(p, k)), bb[p]);
            }
#pragma unroll
            for (int p = 1; p < NB; p += 2) {
                P t = v[p][0];
                v[p][0] = v[p][1];
                v[p][1] = t;
                t = bb[p][0];
                bb[p][0] = bb[p][1];
                bb[p][1] = t;
            }
        } else {
#pragma unroll
            for (int p = 0; p < NB; ++p)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const bool in = on && k + q < hb;
                    v[p][q] = bb[p][q] = P(0);
                    if (in) v[p][q] = ld1(src + base + ls * pos(p, k + q));
                    if (in && first) bb[p][q] = ld1(bz + base + ls * pos(p, k + q));
                }
        }
#pragma unroll
        for (int p = 0; p < NB; ++p)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                constexpr int PW = sizeof(P) / 4;
                const P x = first ? v[p][q] * bb[p][q] : v[p][q];
                em = max(em, expo(x));
                uint32_t w[PW];
                memcpy(w, &x, sizeof(P));
#pragma unroll
                for (int i = 0; i < PW; ++i) *reinterpret_cast<uint32_t *>(cell + ((p * 2 + q) * PW + i) * 128) = w[i];
            }
        atomicMax(&eline[r], em);
    }
    sync();

    if (tid < ROWS) enext[tid] = 0;
    /* ---- digits of the block operands, over the item's own words */
#pragma unroll 1
    for (int idx = tid; idx < items; idx += NT) {
        const int u = idx >> 5, rg = nk8 == 1 ? u : (int)__umulhi((unsigned)u, g.mag_nk8);
        const int em = eline[rg * 8 + ((idx >> 2) & 7)];
        unsigned char *cell = smem + sm_a + u * CELL + (idx & 31) * 4;
        Fix X[NB][2];
#pragma unroll
        for (int p = 0; p < NB; ++p)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                constexpr int PW = sizeof(P) / 4;
                uint32_t w[PW];
#pragma unroll
                for (int i = 0; i < PW; ++i)
                    w[i] = *reinterpret_cast<const uint32_t *>(cell + ((p * 2 + q) * PW + i) * 128);
                P x;
                memcpy(&x, w, sizeof(P));
                X[p][q] = fix<NB>(x, em);
            }
        put_digits<P, NB>(X, cell);
    }
    /* the operator digits, loaded once: one thread waits for all */
    if (wait_op && tid == 0 && !(ph.ok && mbar_wait(bar_op, 0))) *reinterpret_cast<volatile int *>(smem + SM_FAIL) = 1;
    sync();
    ph.ok = *reinterpret_cast<volatile int *>(smem + SM_FAIL) == 0;

    if (!SPLIT) pdl_trigger(); /* the next pass' CTAs may set themselves up where there is room */

    /* ---- products, and the levels joined in registers */
    using Acc = typename std::conditional<std::is_same<P, float>::value, float, long long>::type;
    const int nc = min(c1, (hb + W - 1) / W) - c0, ks = g.hp / 16;
    /* block sums back to the NB points of an output */
    auto points = [&](const Acc (&s)[NB], int em, P (&y)[NB]) {
        Acc t[NB];
        if constexpr (NB == 4) {
            const Acc s0 = s[0] + s[1], s1 = s[0] - s[1], s2 = s[2] + s[3], s3 = s[2] - s[3];
            t[0] = s0 + s2;
            t[1] = s1 + s3;
            t[2] = s0 - s2;
            t[3] = s1 - s3;
        } else {
            t[0] = s[0] + s[1];
            t[1] = s[0] - s[1];
        }
#pragma unroll
        for (int p = 0; p < NB; ++p) {
            from_fix(t[p], em, y[p]);
            if (em == ExpoMax<P>::v || !ph.ok) set_nan(y[p]);
        }
    };
    if constexpr (SPLIT) {
        /* a warp takes one block of 16 outputs x 8 lines, and the sums meet in shared memory: four
         * (two) times as many, shorter pieces of work as with all blocks in one warp */
        Acc *ex = reinterpret_cast<Acc *>(smem + sm_a + tile_bytes(g, S, 8));
        const int pitch = nc * W * NB + 4; /* values of a line: block by block, shifted by four from line to line */
        const int nr = (nlines + 7) / 8, np = (nc + 1) / 2;
#pragma unroll 1
        for (int u = warp; u < nr * np * NB; u += NT / 32) {
            const int b = u % NB, v = u / NB, rg = nr == 1 ? 0 : v / np, cp = v - rg * np;
            float d[L][4];
            products16x8<P, NB, CARRY>(d, sbase + sm_op, sbase + sm_a, nk8, ks, nc, rg, cp, b, carry);
            Acc *at = ex + (rg * 8 + 2 * (lane & 3)) * pitch + (b * nc + 2 * cp) * W + (lane >> 2);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < 2 || 2 * cp + 1 < nc) at[(i & 1) * pitch + (i >> 1) * W] = join(d, i);
        }
        sync();
        /* a warp takes 8 lines x 4 outputs: whole sectors along either direction */
        const int og = g.cpp * (W / 4);
#pragma unroll 1
        for (int u = warp; u < nr * og; u += NT / 32) {
            const int rg = nr == 1 ? 0 : (int)__umulhi((unsigned)u, g.mag_og), o = (u - rg * og) * 4 + (lane & 3);
            const int r = rg * 8 + (lane >> 2), k = c0 * W + o;
            if (r >= nlines || k >= hb) continue;
            const int base = line_base(r);
            P f[NB], y[NB];
            if (last) {
#pragma unroll
                for (int p = 0; p < NB; ++p) f[p] = ld1(bz + base + ls * pos(p, k));
            }
            Acc s[NB];
#pragma unroll
            for (int b = 0; b < NB; ++b) s[b] = ex[r * pitch + b * nc * W + o];
            points(s, eline[r], y);
#pragma unroll
            for (int p = 0; p < NB; ++p) dst[base + ls * pos(p, k)] = last ? y[p] * f[p] : y[p];
        }
    } else {
        /* 16 lines x 8 outputs at a time */
        const int lt = (nlines + 15) / 16;
        /* ldmatrix rows: A (8 lines, 8 points) cells at (line half, point half) = (lane >> 3 & 1, lane >> 4),
         * B (8 outputs, 8 points) cells at (digit, point half) = (lane >> 4, lane >> 3 & 1) */
        const uint32_t a_lane = sbase + sm_a + (uint32_t)((((lane >> 3) & 1) * nk8 + (lane >> 4)) * CELL + (lane & 7) * 16);
        const uint32_t b_lane = sbase + sm_op + (uint32_t)((lane >> 4) * 256 + ((lane >> 3) & 1) * 128 + (lane & 7) * 16);
        /* accumulator v: line (lane >> 2) + 8 (v >> 1), output 2 (lane & 3) + (v & 1) */
        auto products = [&](int l16, int cc, int b, Acc (&acc)[4]) {
            const uint32_t a0 = a_lane + (uint32_t)(l16 * 2 * nk8 * CELL + b * 128);
            const uint32_t b0 = b_lane + (uint32_t)((cc * NB + b) * ks * SK * 256);
            float d[L][4];
#pragma unroll
            for (int l = 0; l < L; ++l)
#pragma unroll
                for (int v = 0; v < 4; ++v) d[l][v] = 0.0f;
#pragma unroll 1
            for (int k = 0; k < ks; ++k) {
                if (CARRY && k > 0) carry_step(d, carry);
                uint32_t bf[SK / 2][4]; /* digits 2j, 2j + 1 */
#pragma unroll
                for (int j = 0; j < SK / 2; ++j) ldsm4(bf[j], b0 + (uint32_t)(k * SK * 256 + j * 512));
#pragma unroll
                for (int i = 0; i < S; ++i) {
                    if (CARRY && i == S / 2) carry_half(d, carry);
                    uint32_t af[4];
                    ldsm4(af, a0 + (uint32_t)(2 * k * CELL + i * NB * 128));
#pragma unroll
                    for (int j = 0; j < SK; ++j)
                        if (i + j < L) mma16816(d[i + j], af, bf[j / 2][2 * (j & 1)], bf[j / 2][2 * (j & 1) + 1]);
                }
            }
            if (CARRY) carry_end(d, carry);
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[v] = join(d, v);
        };
        /* a warp takes all blocks of them and writes the outputs from its registers */
#pragma unroll 1
        for (int u = warp; u < lt * nc; u += NT / 32) {
            const int cc = u / lt, l16 = u - cc * lt, k0 = (c0 + cc) * W + 2 * (lane & 3);
            Acc acc[NB][4];
#pragma unroll
            for (int b = 0; b < NB; ++b) products(l16, cc, b, acc[b]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = l16 * 16 + 8 * h + (lane >> 2);
                if (r >= nlines) continue;
                const int em = eline[r], base = line_base(r);
                P y[2][NB];
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    Acc s[NB];
#pragma unroll
                    for (int b = 0; b < NB; ++b) s[b] = acc[b][2 * h + q];
                    points(s, em, y[q]);
                }
                if (vec && k0 + 1 < hb) {
#pragma unroll
                    for (int p = 0; p < NB; ++p) {
                        const int at = base + ((p & 1) ? pos(p, k0 + 1) : pos(p, k0));
                        P o[2] = {y[p & 1][p], y[1 - (p & 1)][p]};
                        if (last) {
                            P f[2];
                            ld2(bz + at, f);
                            o[0] = o[0] * f[0];
                            o[1] = o[1] * f[1];
                        }
                        st2(dst + at, o[0], o[1]);
                    }
                } else {
#pragma unroll
                    for (int p = 0; p < NB; ++p)
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            if (k0 + q >= hb) continue;
                            const int at = base + ls * pos(p, k0 + q);
                            P o = y[q][p];
                            if (last) o = o * ld1(bz + at);
                            dst[at] = o;
                        }
                }
            }
        }
    }
    sync();
}

/* This part's operator digits. */
template <typename P, int NB>
__device__ __forceinline__ void tc_start_op(const TcGeom &g, const void *table, int part, uint32_t dst, uint32_t bar)
{
    /* consecutive chunks of the table; one thread */
    constexpr int SK = Dig<P>::SK;
    const int c0 = part * g.cpp, c1 = min(c0 + g.cpp, g.nchunks);
    const uint32_t per = (uint32_t)(NB * g.hp * SK * 2); /* bytes per output */
    const uint32_t bytes = per * (min(c1 * W, g.hp) - c0 * W);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(reinterpret_cast<const unsigned char *>(table) + per * (c0 * W)), "r"(bytes), "r"(bar)
                 : "memory");
}

/* Barriers and line exponents; ends with a CTA barrier. */
__device__ __forceinline__ void tc_begin(unsigned char *smem, int nax)
{
    for (int i = threadIdx.x; i < 4 * ROWS; i += blockDim.x) reinterpret_cast<int *>(smem + SM_ELINE)[i] = 0;
    if (threadIdx.x == 32) {
        *reinterpret_cast<volatile int *>(smem + SM_FAIL) = 0;
        for (int i = 0; i < nax; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(smem) + SM_BAR + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

} // namespace

/* One pass: a CTA per (tile, part) and chain. */
template <typename P, int NB, bool CARRY>
__global__ void __launch_bounds__(256, 2) k_pass_tc(TcGeom g, PassArgs a)
{
    const ChainDesc cd = a.chains[blockIdx.y];
    const bool active = a.s < cd.len - 1; /* uniform over the CTA */

    extern __shared__ __align__(128) unsigned char smem[];
    const int part = blockIdx.x % g.parts, tile_i = blockIdx.x / g.parts;
    tc_begin(smem, 1);
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem), bar_op = sbase + SM_BAR;
    if (active && threadIdx.x == 32) /* in flight until the products need them */
        tc_start_op<P, NB>(g, cd.ops->tc[a.axis], part, sbase + SM_OP, bar_op);
    /* what is read up to here no kernel writes. Every CTA waits, so that a pass ends after the
     * one before it */
    pdl_wait();
    if (!active) return;
    if (a.state && a.state[cd.instance].done) {
        mbar_wait(bar_op, 0); /* for its own copy */
        return;
    }
    const P *src = a.first ? reinterpret_cast<const P *>(cd.q) + (long)a.s * a.sstride
                           : reinterpret_cast<const P *>(cd.tmp);
    P *dst = a.last ? reinterpret_cast<P *>(cd.q) + (long)(a.s + 1) * a.sstride : reinterpret_cast<P *>(cd.tmp);
    const P *bz = reinterpret_cast<const P *>(a.s < cd.seg_end ? cd.b0 : cd.b1);
    TcPhase ph = {0, true};
    const int carry = CARRY ? cd.ops->tc_carry >> 2 * a.axis & 3 : 0;
    tc_tile<P, NB, 256, false, CARRY>(g, src, dst, bz, a.first, a.last, tile_i, part, smem, SM_OP, SM_OP + g.op_part, bar_op, true, carry, ph);
    if (!ph.ok && threadIdx.x == 0) atomicExch(&g_scft_pass_fault, 1);
}

/* The whole contour loop of a chain in one cluster. Each CTA keeps its part of
 * every axis' operator digits in shared memory and takes the same tiles at every
 * step; the slices pass between the CTAs through L2 (the intermediate slice of
 * one axis, then q_{s+1}), ordered by a cluster barrier after each axis. A step
 * thus costs two or three short phases per CTA, without the launches, the
 * set-up and the cold instruction cache that a pass of its own has (~4 of 8 us
 * on a 192x96 slice). Two groups of warps with a barrier each take their own
 * tiles, so that one splits or writes while the other multiplies: 46.5 -> 43.2 us a
 * step for 192x96 chains of two CTAs with the GPU full, against one tile of all
 * 512 threads at a time (three groups, or groups of 384 threads, do not fit or
 * gain nothing: issue slots are ~45 % busy, shared memory 50 %, and neither more
 * warps nor more overlap moves that). Control flow is uniform over the cluster. */
template <typename P, bool CARRY>
__global__ void __launch_bounds__(512, 1) k_chain_tc(const __grid_constant__ TcLoop lp, Step2DArgs a)
{
    const int rank = blockIdx.x % lp.cluster, slot = blockIdx.x / lp.cluster; /* clusters are consecutive blocks */
    const StepRange run = step_range(a, slot);
    const ChainDesc cd = a.chains[run.chain];
    const int s_end = run.s_end < cd.len - 1 ? run.s_end : cd.len - 1;
    const bool any = run.s < s_end; /* uniform over the cluster */

    extern __shared__ __align__(128) unsigned char smem[];
    tc_begin(smem, lp.nax);
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem);
    if (any && threadIdx.x == 32)
        for (int ax = 0; ax < lp.nax; ++ax) {
            const TcGeom &g = lp.g[ax];
            if (rank / g.parts >= lp.slots[ax] || (long)(rank / g.parts) * g.tile >= g.lines) continue;
            if (g.nb == 4)
                tc_start_op<P, 4>(g, cd.ops->tc[ax], rank % g.parts, sbase + lp.op_at[ax], sbase + SM_BAR + 8 * ax);
            else
                tc_start_op<P, 2>(g, cd.ops->tc[ax], rank % g.parts, sbase + lp.op_at[ax], sbase + SM_BAR + 8 * ax);
        }
    pdl_wait();
    if (!any) return;
    if (a.state && a.state[cd.instance].done) { /* uniform over the cluster */
        for (int ax = 0; ax < lp.nax; ++ax) /* its own copies */
            if (rank / lp.g[ax].parts < lp.slots[ax] && (long)(rank / lp.g[ax].parts) * lp.g[ax].tile < lp.g[ax].lines)
                mbar_wait(sbase + SM_BAR + 8 * ax, 0);
        return;
    }
    TcPhase ph = {0, true};
    const int carry = CARRY ? cd.ops->tc_carry : 0;
    const int group = threadIdx.x / (512 / GROUPS);
    const uint32_t tile_at = lp.tile_at + (uint32_t)group * lp.tile_bytes;
#pragma unroll 1
    for (int s = run.s; s < s_end; ++s) {
        if (s + 1 == s_end) pdl_trigger();
        const P *bz = reinterpret_cast<const P *>(s < cd.seg_end ? cd.b0 : cd.b1);
#pragma unroll 1
        for (int ax = 0; ax < lp.nax; ++ax) {
            const TcGeom &g = lp.g[ax];
            const bool first = ax == 0, last = ax == lp.nax - 1;
            const P *src = first ? reinterpret_cast<const P *>(cd.q) + (long)s * a.sstride : reinterpret_cast<const P *>(cd.tmp);
            P *dst = last ? reinterpret_cast<P *>(cd.q) + (long)(s + 1) * a.sstride : reinterpret_cast<P *>(cd.tmp);
            const int t0 = rank / g.parts + group * lp.slots[ax], part = rank % g.parts;
            if (rank / g.parts < lp.slots[ax])
#pragma unroll 1
                for (int t = t0; (long)t * g.tile < g.lines; t += GROUPS * lp.slots[ax]) {
                    if (g.nb == 4)
                        tc_tile<P, 4, 512 / GROUPS, true, CARRY>(g, src, dst, bz, first, last, t, part, smem, lp.op_at[ax], tile_at,
                                                 sbase + SM_BAR + 8 * ax, s == run.s && t == t0, carry >> 2 * ax & 3, ph);
                    else
                        tc_tile<P, 2, 512 / GROUPS, true, CARRY>(g, src, dst, bz, first, last, t, part, smem, lp.op_at[ax], tile_at,
                                                 sbase + SM_BAR + 8 * ax, s == run.s && t == t0, carry >> 2 * ax & 3, ph);
                }
            /* this axis' slice is complete before the next one reads it */
            asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
    }
    if (!ph.ok && threadIdx.x % (512 / GROUPS) == 0) atomicExch(&g_scft_pass_fault, 1);
}

/* The same loop on a 2D grid with one tile per CTA and axis, whose lines never
 * leave shared memory: each output goes straight to the CTA whose line of the
 * other axis it belongs to (st.async), with the largest exponent of the 8 lines a
 * warp sends, and that CTA waits for its bytes on its own barrier. No CTA waits
 * for stores to reach L2, for a cluster barrier and for the loads after it, nor
 * looks for a line's largest value. Only q_{s+1} goes to global memory, for the densities; what is sent
 * after the last axis is b q_{s+1} already.
 *
 * A CTA's lines of an axis are complete when every CTA has sent the points of them;
 * warps whose outputs go elsewhere may still be at work, there and in the CTA
 * itself. What orders each write to a buffer after the last read of what it held:
 *   - lines of an axis are read into digits before the tile's first CTA barrier; a CTA
 *     sends points of the next ones only after it has received its lines of the other
 *     axis whole, a point of each of these lines among them, sent after that barrier;
 *   - digits are read by the products, before the tile's second CTA barrier, and
 *     written again for the next tile, after it;
 *   - block sums are read by the outputs and written again by the next tile's products,
 *     after its first CTA barrier; they lie behind the digits of either axis, which
 *     warps that have already gone on may be writing;
 *   - the largest exponents sent with the lines are read before the tile's first CTA
 *     barrier, like the lines; the outputs read a copy of them, of which there are two
 *     in turn, so that one is written again two tiles on, after the CTA barriers between.
 *
 * A step is two serial phases of digits, products and outputs, each bounded by
 * the latency of its own instructions on small grids (one item a thread) and on
 * 192x96 by the integer pipe (digits ~1300 + 900 clocks, outputs 2700 + 3000)
 * and the rate of mma.sync (2500 + 2500), with ~600 between them. FP64, a step:
 * 32x16 7.0 -> 4.0 us, 64x64 6.9 -> 5.2, 192x96 10.8 -> 8.4 against the loop
 * above, which stays for 3D grids and for slices that do not fit one tile a CTA. */
template <typename P, bool CARRY>
__global__ void __launch_bounds__(512, 1) k_chain2d_tc(const __grid_constant__ TcLoop lp, Step2DArgs a)
{
    const int rank = blockIdx.x % lp.cluster, slot = blockIdx.x / lp.cluster; /* clusters are consecutive blocks */
    const StepRange run = step_range(a, slot);
    const ChainDesc cd = a.chains[run.chain];
    const int s_end = run.s_end < cd.len - 1 ? run.s_end : cd.len - 1;
    const bool any = run.s < s_end; /* uniform over the cluster */

    extern __shared__ __align__(128) unsigned char smem[];
    tc_begin(smem, 4); /* operator digits of the two axes, lines of the two axes */
    const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(smem), bars = sbase + SM_BAR;
    bool mine[2], ok = true;
    uint32_t bytes[2];
    int tiles = 0; /* tiles done */
    const int carry = CARRY ? cd.ops->tc_carry : 0;
#pragma unroll
    for (int ax = 0; ax < 2; ++ax) {
        const TcGeom &g = lp.g[ax];
        mine[ax] = any && (long)rank * g.tile < g.lines;
        /* a line's values, in pairs, and the largest exponent of each 8 of them that one warp sends */
        bytes[ax] = mine[ax] ? (uint32_t)(min((long)g.tile, g.lines - (long)rank * g.tile) * ((g.n + 1) / 2 * 2 * sizeof(P) + (g.n + 7) / 8 * 4)) : 0u;
        if (mine[ax] && threadIdx.x == 32) {
            if (g.nb == 4)
                tc_start_op<P, 4>(g, cd.ops->tc[ax], 0, sbase + lp.op_at[ax], bars + 8 * ax);
            else
                tc_start_op<P, 2>(g, cd.ops->tc[ax], 0, sbase + lp.op_at[ax], bars + 8 * ax);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bars + 16 + 8 * ax), "r"(bytes[ax]) : "memory");
        }
    }
    pdl_wait();
    if (!any) return;
    if (a.state && a.state[cd.instance].done) { /* uniform over the cluster */
        for (int ax = 0; ax < 2; ++ax)
            if (mine[ax]) mbar_wait(bars + 8 * ax, 0); /* its own copies */
        return;
    }
    /* the first lines: b q_s from global memory */
    if (mine[0]) {
        const TcGeom &g = lp.g[0];
        const P *src = reinterpret_cast<const P *>(cd.q) + (long)run.s * a.sstride;
        const P *bz = reinterpret_cast<const P *>(run.s < cd.seg_end ? cd.b0 : cd.b1);
        P *in = reinterpret_cast<P *>(smem + lp.buf_at[0]);
        int *eline = reinterpret_cast<int *>(smem + sm_received(0));
        const int L0 = rank * g.tile, nlines = (int)min((long)g.tile, g.lines - L0);
        for (int i = threadIdx.x; i < nlines * g.n; i += 512) {
            const int x = i / nlines, r = i - x * nlines; /* lines of the slowest axis: neighbours in memory */
            const long at = g.ls == 1 ? (long)(L0 + r) * g.n + x : (long)x * g.ls + L0 + r;
            const P v = ld1(src + at) * ld1(bz + at);
            in[r * lp.pitch[0] + x] = v;
            atomicMax(&eline[r], expo(v));
        }
    }
    /* every CTA's barriers are set up before anyone sends */
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll 1
    for (int s = run.s; s < s_end; ++s) {
        if (s + 1 == s_end) pdl_trigger();
        const P *bz = reinterpret_cast<const P *>(s < cd.seg_end ? cd.b0 : cd.b1);
#pragma unroll 1
        for (int ax = 0; ax < 2; ++ax) {
            if (!mine[ax]) continue;
            const TcGeom &g = lp.g[ax], &o = lp.g[1 - ax];
            const int t = s - run.s;
            if (t > 0 || ax == 1) {
                /* the lines are there; one thread re-arms the barrier for the next step */
                const uint32_t bar = bars + 16 + 8 * ax;
                const bool got = ok && mbar_wait<true>(bar, (uint32_t)(t - 1 + ax) & 1u);
                if (!got) *reinterpret_cast<volatile int *>(smem + SM_FAIL) = 1;
                if (got && s + 1 < s_end && threadIdx.x == 0)
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes[ax]) : "memory");
            }
            const Exchange<P> xc = {reinterpret_cast<const P *>(smem + lp.buf_at[ax]),
                                    reinterpret_cast<const int *>(smem + sm_received(ax)),
                                    reinterpret_cast<int *>(smem + sm_kept(tiles++ & 1)),
                                    lp.pitch[ax],
                                    (t + 1 + ax) << EBITS, /* larger than all before: the maxima need no reset */
                                    lp.buf_at[1 - ax],
                                    sm_received(1 - ax),
                                    SM_BAR + 16 + 8 * (1 - ax),
                                    lp.pitch[1 - ax],
                                    o.tile,
                                    lp.mag_tile[1 - ax],
                                    ax == 0 || s + 1 < s_end,
                                    bz,
                                    reinterpret_cast<const P *>(s + 1 < cd.seg_end ? cd.b0 : cd.b1),
                                    reinterpret_cast<P *>(cd.q) + (long)(s + 1) * a.sstride};
            if (g.nb == 4)
                tc_tile2d<P, 4, 512, CARRY>(g, xc, ax == 1, rank, smem, lp.op_at[ax], lp.tile_at, lp.ex_at, bars + 8 * ax, t == 0, carry >> 2 * ax & 3, ok);
            else
                tc_tile2d<P, 2, 512, CARRY>(g, xc, ax == 1, rank, smem, lp.op_at[ax], lp.tile_at, lp.ex_at, bars + 8 * ax, t == 0, carry >> 2 * ax & 3, ok);
        }
    }
    if (!ok && threadIdx.x == 0) atomicExch(&g_scft_pass_fault, 1);
    /* no CTA leaves while another could still send to it */
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

/* ------------------------------------------------------------- launchers */
size_t scft_pass_tc_smem(int prec, const TcGeom &g)
{
    return SM_OP + g.op_part + (prec == SCFT_PREC_FP32 ? tile_bytes(g, Dig<float>::S, 16)
                                                      : tile_bytes(g, Dig<double>::S, 16));
}

template <typename P, bool CARRY>
static cudaError_t launch_tc(const TcGeom &g, const PassArgs &a, cudaStream_t st)
{
    const size_t smem = SM_OP + g.op_part + tile_bytes(g, Dig<P>::S, 16);
    const dim3 grid((unsigned)((g.lines + g.tile - 1) / g.tile * g.parts), a.nchains);
    if (g.tile < 8 || g.tile % 8 || g.tile > ROWS) return cudaErrorInvalidValue;
    return g.nb == 4 ? pdl_launch(k_pass_tc<P, 4, CARRY>, grid, 256, smem, st, g, a)
                     : pdl_launch(k_pass_tc<P, 2, CARRY>, grid, 256, smem, st, g, a);
}

int scft_pass_tc_fits(int prec, const TcGeom &g, int smem_limit)
{
    return scft_pass_tc_smem(prec, g) <= (size_t)smem_limit;
}

/* carry: some operator of the context needs the carries of carry_sums. */
cudaError_t scft_launch_pass_tc(int prec, int carry, const TcGeom &g, const PassArgs &a, cudaStream_t st)
{
    if (prec == SCFT_PREC_FP64) return carry ? launch_tc<double, true>(g, a, st) : launch_tc<double, false>(g, a, st);
    if (prec == SCFT_PREC_FP32X2) return carry ? launch_tc<dfloat, true>(g, a, st) : launch_tc<dfloat, false>(g, a, st);
    return carry ? launch_tc<float, true>(g, a, st) : launch_tc<float, false>(g, a, st);
}

/* Shared-memory layout of the cluster loop, from the axes' tiles and parts;
 * returns its bytes. */
size_t scft_chain_tc_layout(int prec, TcLoop &lp)
{
    uint32_t at = SM_OP, tile = 0, digits = 0, sums = 0;
    for (int ax = 0; ax < lp.nax; ++ax) {
        lp.op_at[ax] = at;
        at += (lp.g[ax].op_part + 127) / 128 * 128;
        const int S = prec == SCFT_PREC_FP32 ? Dig<float>::S : Dig<double>::S, value = prec == SCFT_PREC_FP32 ? 4 : 8;
        const uint32_t d = (tile_bytes(lp.g[ax], S, 8) + 127) / 128 * 128, e = exchange_bytes(lp.g[ax], value);
        if (d > digits) digits = d;
        if (e > sums) sums = e;
        if (d + e > tile) tile = d + e;
        lp.slots[ax] = lp.cluster / lp.g[ax].parts;
        if (lp.exchange) { /* lines, shifted by half the banks from one to the next */
            lp.pitch[ax] = (lp.g[ax].n + 15) / 16 * 16 + 8;
            lp.buf_at[ax] = at;
            lp.mag_tile[ax] = (unsigned)((0xFFFFFFFFull + lp.g[ax].tile) / lp.g[ax].tile);
            at += (uint32_t)(lp.g[ax].tile * lp.pitch[ax] * value + 127) / 128 * 128;
        }
    }
    lp.tile_at = at;
    lp.ex_at = at + digits;
    lp.tile_bytes = ((lp.exchange ? digits + sums : tile) + 127) / 128 * 128;
    return (size_t)at + (lp.exchange ? 1 : GROUPS) * lp.tile_bytes;
}

/* First byte and end of an axis' digits and of its block sums in the exchange form. */
void scft_chain_tc_regions(int prec, const TcLoop &lp, int ax, long at[4])
{
    at[0] = lp.tile_at;
    at[1] = at[0] + tile_bytes(lp.g[ax], prec == SCFT_PREC_FP32 ? Dig<float>::S : Dig<double>::S, 8);
    at[2] = lp.ex_at;
    at[3] = at[2] + exchange_bytes(lp.g[ax], prec == SCFT_PREC_FP32 ? 4 : 8);
}

/* Test hook: first byte and end of the line exponents in k_chain2d_tc: sent by peers for
 * either axis, then the two sets that the outputs read. */
extern "C" void scft_tc_exchange_exponents(long at[4][2])
{
    for (int k = 0; k < 4; ++k) {
        at[k][0] = k < 2 ? sm_received(k) : sm_kept(k - 2);
        at[k][1] = at[k][0] + ROWS * 4;
    }
}

template <typename P, bool CARRY>
static cudaError_t launch_chain(const TcLoop &lp, const Step2DArgs &a, int nchains, cudaStream_t st, int *clusters)
{
    TcLoop l = lp;
    const int prec = std::is_same<P, double>::value ? SCFT_PREC_FP64 : std::is_same<P, float>::value ? SCFT_PREC_FP32 : SCFT_PREC_FP32X2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(nchains * lp.cluster), 1, 1);
    cfg.blockDim = dim3(512, 1, 1);
    cfg.dynamicSmemBytes = scft_chain_tc_layout(prec, l);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = lp.cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (lp.exchange) {
        if (clusters) return cudaOccupancyMaxActiveClusters(clusters, k_chain2d_tc<P, CARRY>, &cfg);
        return cudaLaunchKernelEx(&cfg, k_chain2d_tc<P, CARRY>, l, a);
    }
    if (clusters) return cudaOccupancyMaxActiveClusters(clusters, k_chain_tc<P, CARRY>, &cfg);
    return cudaLaunchKernelEx(&cfg, k_chain_tc<P, CARRY>, l, a);
}

/* Launches the contour loops of nchains chains; with clusters != NULL only asks
 * how many clusters can be resident. */
cudaError_t scft_launch_chain_tc(int prec, int carry, const TcLoop &lp, const Step2DArgs &a, int nchains, cudaStream_t st,
                                 int *clusters)
{
    if (prec == SCFT_PREC_FP64)
        return carry ? launch_chain<double, true>(lp, a, nchains, st, clusters) : launch_chain<double, false>(lp, a, nchains, st, clusters);
    if (prec == SCFT_PREC_FP32X2)
        return carry ? launch_chain<dfloat, true>(lp, a, nchains, st, clusters) : launch_chain<dfloat, false>(lp, a, nchains, st, clusters);
    return carry ? launch_chain<float, true>(lp, a, nchains, st, clusters) : launch_chain<float, false>(lp, a, nchains, st, clusters);
}

template <typename P, bool CARRY>
static cudaError_t configure_tc(int smem_bytes)
{
    /* one carve-out for every pass, so the SMs keep their split between launches */
    const void *k[] = {(const void *)k_pass_tc<P, 4, CARRY>, (const void *)k_pass_tc<P, 2, CARRY>, (const void *)k_chain_tc<P, CARRY>,
                       (const void *)k_chain2d_tc<P, CARRY>};
    cudaError_t e = cudaSuccess;
    for (const void *f : k) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    }
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_chain_tc<P, CARRY>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_chain2d_tc<P, CARRY>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e;
}

/* Raise the dynamic shared-memory limit of a form's kernels once, outside any stream capture. */
cudaError_t scft_pass_tc_configure(int prec, int smem_bytes)
{
    cudaError_t e;
    if (prec == SCFT_PREC_FP64) {
        e = configure_tc<double, false>(smem_bytes);
        if (e == cudaSuccess) e = configure_tc<double, true>(smem_bytes);
    } else if (prec == SCFT_PREC_FP32X2) {
        e = configure_tc<dfloat, false>(smem_bytes);
        if (e == cudaSuccess) e = configure_tc<dfloat, true>(smem_bytes);
    } else {
        e = configure_tc<float, false>(smem_bytes);
        if (e == cudaSuccess) e = configure_tc<float, true>(smem_bytes);
    }
    return e;
}

int scft_pass_tc_take_fault(void)
{
    int v = 0;
    const int zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_scft_pass_fault, sizeof(int)) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (v) cudaMemcpyToSymbol(g_scft_pass_fault, &zero, sizeof(int));
    return v;
}
