// wg_soft64.h — the Laplacian's sums of doubles on the integer pipes, rounded as the FP64 pipe
// rounds them.
//
// The FP64 pipe of this GPU retires 1.68 additions, multiplications or fused multiply-adds a
// clock and SM (measured; the integer pipes 64 to 93 operations), so a leapfrog update is
// bound by its 7 to 12 FP64 operations.  The four of them that form the Laplacian,
//     RN(RN(RN(RN(n + s) + e) + w) - 4x)
// (RN: round to nearest, ties to even, as each operation of the reference), and x - y, are
// done here on 64-bit integers instead, beside the FP64 pipe's other work.
//
// A value is an integer of its 53 significand bits times 2^G and an exponent.  The operands
// are shifted to the largest exponent among them; that loses nothing while the exponents
// differ by at most G, and G = 7 leaves |n| + |s| + |e| + |w| + 4|x| below 2^63.  Each partial
// sum is then rounded to 53 significant bits where it stands (s64_round53), which is the FP64
// operation's rounding, since the integer holds the exact sum.  +0 is taken with any
// exponents.  Operands further apart, -0, subnormals, infinities, NaN and results of less than
// 2^-28 of the largest operand are refused: the caller takes the FP64 pipe for that cell.
//
// Host and device code, so that the rounding is tested on the host against the machine's own
// additions.
#pragma once
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define WG_HD __host__ __device__ __forceinline__
#else
#define WG_HD inline
#endif

namespace wg {

constexpr int S64_G = 7;        // guard bits below the last significand bit of the largest operand
constexpr int S64_ZERO = 4095;  // S64::z of +0

struct S64 {
    long long m;  // signed significand x 2^G (of a zero: 2^(52 + G), shifted out by its z)
    int e;        // biased exponent; 0 for zeros and subnormals
    int z;        // the same, but S64_ZERO for +0
};

WG_HD int s64_max3(int a, int b, int c)
{
#ifdef __CUDA_ARCH__
    return __vimax3_s32(a, b, c);
#else
    return a > b ? (a > c ? a : c) : (b > c ? b : c);
#endif
}
WG_HD int s64_min3(int a, int b, int c)
{
#ifdef __CUDA_ARCH__
    return __vimin3_s32(a, b, c);
#else
    return a < b ? (a < c ? a : c) : (b < c ? b : c);
#endif
}
// arithmetic shift right; 63 for any larger (unsigned) count
WG_HD long long s64_shr(long long m, int k)
{
#ifdef __CUDA_ARCH__
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(k));
    return r;
#else
    return m >> ((unsigned)k > 63u ? 63 : k);
#endif
}

WG_HD S64 s64_unpack(double v)
{
    unsigned hi, lo;
#ifdef __CUDA_ARCH__
    hi = (unsigned)__double2hiint(v);
    lo = (unsigned)__double2loint(v);
#else
    uint64_t b;
    memcpy(&b, &v, 8);
    hi = (unsigned)(b >> 32);
    lo = (unsigned)b;
#endif
    S64 r;
    r.e = (int)((hi >> 20) & 0x7FFu);
    r.z = (hi | lo) == 0u ? S64_ZERO : r.e;
    const unsigned long long mag = (((unsigned long long)((hi & 0xFFFFFu) | 0x100000u) << 32) | lo) << S64_G;
    const long long s = (long long)((int)hi >> 31);
    r.m = ((long long)mag ^ s) - s;
    return r;
}

// s rounded to 53 significant bits (nearest, ties to even); s is below 2^63 in magnitude and
// stays so.  Two's complement: adding half - 1 + (the last kept bit) and clearing the low bits
// rounds either sign the same way.
WG_HD long long s64_round53(long long s)
{
    const int hi = (int)(s >> 32);
    int top;  // index of the highest bit of the high word that differs from the sign, -1: none
    unsigned mask;
#ifdef __CUDA_ARCH__
    asm("bfind.s32 %0, %1;" : "=r"(top) : "r"(hi));
    const int k = max(top - 20, 0);
    asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(mask) : "r"(k));
#else
    const unsigned h = (unsigned)(hi ^ (hi >> 31));
    top = h ? 31 - __builtin_clz(h) : -1;
    const int k = top > 20 ? top - 20 : 0;
    mask = (1u << k) - 1u;
#endif
    const unsigned odd = ((unsigned)s >> k) & mask & 1u;
    s += (long long)((mask >> 1) + odd);
    const unsigned lo = (unsigned)s & ~mask;
    return (long long)(((unsigned long long)s & 0xFFFFFFFF00000000ull) | lo);
}

// The double t x 2^(emax - 1075 - G) of a sum of at most 53 significant bits whose high word is
// not zero (its magnitude at least 2^-28 of 2^(emax - 1022)); +0 when every operand is (zero).
WG_HD double s64_pack(long long t, int emax, bool zero, bool &high)
{
    const long long g = t >> 63;
    const unsigned long long mag = (unsigned long long)((t ^ g) - g);
    const unsigned mh = (unsigned)(mag >> 32), ml = (unsigned)mag;
    unsigned z;  // left shift that brings the leading bit to bit 63
#ifdef __CUDA_ARCH__
    asm("bfind.shiftamt.u32 %0, %1;" : "=r"(z) : "r"(mh));
    const unsigned th = __funnelshift_l(ml, mh, z), tl = ml << (z & 31u);
    const unsigned bl = __funnelshift_r(tl, th, 11);
#else
    z = mh ? (unsigned)__builtin_clz(mh) : 0xFFFFFFFFu;
    const unsigned long long tt = mag << (z & 31u);
    const unsigned th = (unsigned)(tt >> 32), tl = (unsigned)tt;
    const unsigned bl = (tl >> 11) | (th << 21);
#endif
    // adding the exponent less one turns the leading bit, now 2^52, into the hidden bit
    unsigned bh = (th >> 11) + ((unsigned)(emax + 3 - (int)z) << 20);
    bh |= (unsigned)(g >> 32) & 0x80000000u;
    high = mh != 0u;
    bh = zero ? 0u : bh;
    const unsigned rl = zero ? 0u : bl;
#ifdef __CUDA_ARCH__
    return __hiloint2double((int)bh, (int)rl);
#else
    const uint64_t bits = ((uint64_t)bh << 32) | rl;
    double v;
    memcpy(&v, &bits, 8);
    return v;
#endif
}

// Exponents that may be summed: the spread within G, every operand and the result normal.
WG_HD bool s64_reach(int emax, int emin) { return emax - emin <= S64_G && (unsigned)(emax - 64) <= 1936u; }

// RN(RN(RN(RN(n + s) + e) + w) - 4x); ok: the operands are within reach of one another.
WG_HD double s64_laplacian(const S64 &n, const S64 &s, const S64 &e, const S64 &w, const S64 &x, bool &ok)
{
    const int emax = s64_max3(s64_max3(n.e, s.e, x.e), e.e, w.e), emin = s64_min3(s64_min3(n.z, s.z, x.z), e.z, w.z);
    long long t = s64_round53(s64_shr(n.m, emax - n.z) + s64_shr(s.m, emax - s.z));
    t = s64_round53(t + s64_shr(e.m, emax - e.z));
    t = s64_round53(t + s64_shr(w.m, emax - w.z));
    t = s64_round53(t - (s64_shr(x.m, emax - x.z) << 2));
    bool high;
    const bool zero = emin == S64_ZERO;
    const double d = s64_pack(t, emax, zero, high);
    ok = zero || (s64_reach(emax, emin) && high);
    return d;
}

// RN(x - y); ok as above.
WG_HD double s64_sub(const S64 &x, const S64 &y, bool &ok)
{
    const int emax = x.e > y.e ? x.e : y.e, emin = x.z < y.z ? x.z : y.z;
    bool high;
    const bool zero = emin == S64_ZERO;
    const double d = s64_pack(s64_round53(s64_shr(x.m, emax - x.z) - s64_shr(y.m, emax - y.z)), emax, zero, high);
    ok = zero || (s64_reach(emax, emin) && high);
    return d;
}

}  // namespace wg
