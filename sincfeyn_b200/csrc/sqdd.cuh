/* sqdd.cuh -- double-double numbers for the precision fallback, usable in device and host code.
 *
 * A value is hi + lo with |lo| <= ulp(hi)/2, about 32 significant digits.  The operations are the
 * error-free transformations of Dekker and Knuth (two-sum, quick-two-sum) and the fma two-product, as
 * published for the QD library by Hida, Li and Bailey ("Algorithms for quad-double precision floating
 * point arithmetic", 2001).  The reference evaluator fixes which variant of each operation its
 * fallback uses (driver/dd.h:18-75), and the fallback test assumes that error model, so the same
 * variants are used here:
 *   - addition is the "sloppy" form (absolute error ~2^-104 (|a|+|b|), driver/dd.h:30-32);
 *   - dd op double does not promote the double (driver/dd.h:35-36);
 *   - multiplication adds both cross terms to the low part (driver/dd.h:39-41);
 *   - division takes three quotient digits (driver/dd.h:42-47).
 * Every rounding step is an explicit round-to-nearest intrinsic on the device (and plain IEEE
 * operations on the host, compiled without contraction), so no compiler contraction can change a
 * result: the values agree bit for bit with the reference's double-double built with
 * -ffp-contract=off. */
#pragma once
#include <math.h>

#if defined(__CUDACC__)
#define SQDD_HD __host__ __device__ __forceinline__
#define SQDD_M __host__ __device__ __forceinline__
#else
#define SQDD_HD static inline
#define SQDD_M inline
#endif

#if defined(__CUDA_ARCH__)
#define SQ_ADD(a, b) __dadd_rn((a), (b))
#define SQ_SUB(a, b) __dsub_rn((a), (b))
#define SQ_MUL(a, b) __dmul_rn((a), (b))
#define SQ_DIV(a, b) __ddiv_rn((a), (b))
#define SQ_FMA(a, b, c) __fma_rn((a), (b), (c))
#else
#define SQ_ADD(a, b) ((a) + (b))
#define SQ_SUB(a, b) ((a) - (b))
#define SQ_MUL(a, b) ((a) * (b))
#define SQ_DIV(a, b) ((a) / (b))
#define SQ_FMA(a, b, c) fma((a), (b), (c))
#endif

struct sqdd {
    double hi, lo;
    SQDD_M sqdd() : hi(0), lo(0) {}
    SQDD_M sqdd(double x) : hi(x), lo(0) {}
    SQDD_M sqdd(int x) : hi((double)x), lo(0) {}
    SQDD_M sqdd(double h, double l) : hi(h), lo(l) {}
    SQDD_M double value() const { return SQ_ADD(hi, lo); }
};

/* s + e = a + b exactly (Knuth) */
SQDD_HD sqdd sqdd_two_sum(double a, double b){
    double s = SQ_ADD(a, b), bb = SQ_SUB(s, a);
    double e = SQ_ADD(SQ_SUB(a, SQ_SUB(s, bb)), SQ_SUB(b, bb));
    return sqdd(s, e);
}
/* s + e = a + b exactly, given |a| >= |b| (Dekker) */
SQDD_HD sqdd sqdd_quick_two_sum(double a, double b){
    double s = SQ_ADD(a, b);
    return sqdd(s, SQ_SUB(b, SQ_SUB(s, a)));
}
/* p + e = a * b exactly (fma) */
SQDD_HD sqdd sqdd_two_prod(double a, double b){
    double p = SQ_MUL(a, b);
    return sqdd(p, SQ_FMA(a, b, -p));
}

SQDD_HD sqdd operator+(const sqdd &a, const sqdd &b){
    sqdd s = sqdd_two_sum(a.hi, b.hi);
    s.lo = SQ_ADD(s.lo, SQ_ADD(a.lo, b.lo));
    return sqdd_quick_two_sum(s.hi, s.lo);
}
SQDD_HD sqdd sqdd_add_d(const sqdd &a, double b){
    sqdd s = sqdd_two_sum(a.hi, b);
    s.lo = SQ_ADD(s.lo, a.lo);
    return sqdd_quick_two_sum(s.hi, s.lo);
}
SQDD_HD sqdd sqdd_mul_d(const sqdd &a, double b){
    sqdd p = sqdd_two_prod(a.hi, b);
    p.lo = SQ_ADD(p.lo, SQ_MUL(a.lo, b));
    return sqdd_quick_two_sum(p.hi, p.lo);
}
SQDD_HD sqdd operator-(const sqdd &a){ return sqdd(-a.hi, -a.lo); }
SQDD_HD sqdd operator-(const sqdd &a, const sqdd &b){ return a + (-b); }
SQDD_HD sqdd operator*(const sqdd &a, const sqdd &b){
    sqdd p = sqdd_two_prod(a.hi, b.hi);
    p.lo = SQ_ADD(p.lo, SQ_ADD(SQ_MUL(a.hi, b.lo), SQ_MUL(a.lo, b.hi)));
    return sqdd_quick_two_sum(p.hi, p.lo);
}
#if !defined(__CUDA_ARCH__)
SQDD_HD sqdd operator/(const sqdd &a, const sqdd &b){
    double q1 = SQ_DIV(a.hi, b.hi);
    sqdd r = a - b*sqdd(q1);
    double q2 = SQ_DIV(r.hi, b.hi);
    r = r - b*sqdd(q2);
    double q3 = SQ_DIV(r.hi, b.hi);
    sqdd q = sqdd_quick_two_sum(q1, q2);
    return q + sqdd(q3);
}
#endif

/* a / b with r = sqdd_rcp(b) at hand (a table column and its reciprocal): the rounded quotient in five
 * operations instead of a division's ten or more.  a r is within two ulp of a / b; one correction brings it
 * within one ulp, and a second, from its exact remainder, to RN(a / b) (Markstein's theorem: P. Markstein,
 * IBM J. Res. Dev. 34, 1990, 111), as long as nothing leaves the normal range.  One test sees to that: r is NaN unless b lies
 * within 2^+-SQDD_DIVR, and the quotient is checked to lie there too, so that a lies within 2^+-900 and the remainders,
 * 2^-106 a at the least, are normal; any other operands (zeros, infinities, NaN) divide. */
#define SQDD_DIVR 450
SQDD_HD bool sqdd_within(double x, int bits){
#if defined(__CUDA_ARCH__)
    return (((unsigned)__double2hiint(x) >> 20) & 0x7ff) - (1023u - bits) < 2u*bits;
#else
    return fabs(x) >= ldexp(1.0, -bits) && fabs(x) < ldexp(1.0, bits);
#endif
}
#if defined(__CUDACC__)
static __host__ __device__ __noinline__ double sqdd_div_any(double a, double b){ return SQ_DIV(a, b); }
#else
static inline double sqdd_div_any(double a, double b){ return SQ_DIV(a, b); }
#endif
SQDD_HD double sq_divu(double a, double b, double r){
    const double q0 = SQ_MUL(a, r), q1 = SQ_FMA(SQ_FMA(-q0, b, a), r, q0), q2 = SQ_FMA(SQ_FMA(-q1, b, a), r, q1);
    return sqdd_within(q1, SQDD_DIVR) ? q2 : sqdd_div_any(a, b);
}
/* what a table keeps of a divisor: RN(1/b), of the high part; NaN if sq_divu is not to use it */
SQDD_HD double sqdd_rcp(double b){ return sqdd_within(b, SQDD_DIVR) ? SQ_DIV(1.0, b) : NAN; }
/* a / b in double-double (operator/) with r = sqdd_rcp(b): its three quotient digits by sq_divu */
SQDD_HD sqdd sq_divu(const sqdd &a, const sqdd &b, double r){
    double q1 = sq_divu(a.hi, b.hi, r);
    sqdd t = a - b*sqdd(q1);
    double q2 = sq_divu(t.hi, b.hi, r);
    t = t - b*sqdd(q2);
    double q3 = sq_divu(t.hi, b.hi, r);
    sqdd q = sqdd_quick_two_sum(q1, q2);
    return q + sqdd(q3);
}
SQDD_HD double sqdd_rcp(const sqdd &b){ return sqdd_rcp(b.hi); }
/* sq_divu and sqdd_rcp with the tests put off (CK = 0): several quotients in a row raise *bad, and one test of it, by
 * sqdd_bad, tells whether any lay outside the window; the caller then computes the whole again with CK = 1, which
 * divides where it must.  In double-double every quotient is tested. */
#define SQDD_DIVLIM ((2u*SQDD_DIVR) << 21)
SQDD_HD void sqdd_flag(unsigned *bad, double x){
#if defined(__CUDA_ARCH__)
    *bad = max(*bad, 2u*(unsigned)__double2hiint(x) - ((1023u - SQDD_DIVR) << 21));     /* without the sign; wraps below */
#else
    if(!sqdd_within(x, SQDD_DIVR)) *bad = ~0u;
#endif
}
SQDD_HD bool sqdd_bad(unsigned bad){ return bad >= SQDD_DIVLIM; }
template<int CK> SQDD_HD double sq_divc(double a, double b, double r, unsigned *bad){
    if(CK) return sq_divu(a, b, r);
    const double q0 = SQ_MUL(a, r), q1 = SQ_FMA(SQ_FMA(-q0, b, a), r, q0);
    sqdd_flag(bad, q1);
    return SQ_FMA(SQ_FMA(-q1, b, a), r, q1);
}
template<int CK> SQDD_HD double sq_rcpc(double b, unsigned *bad){
    if(CK) return sqdd_rcp(b);
    sqdd_flag(bad, b);
    return SQ_DIV(1.0, b);
}
template<int CK> SQDD_HD sqdd sq_divc(const sqdd &a, const sqdd &b, double r, unsigned *){ return sq_divu(a, b, r); }
template<int CK> SQDD_HD double sq_rcpc(const sqdd &b, unsigned *){ return sqdd_rcp(b); }
#if defined(__CUDA_ARCH__)
/* the three quotient digits share one reciprocal: the same rounded quotients (sq_divu) for one division and fifteen
 * operations instead of three divisions */
SQDD_HD sqdd operator/(const sqdd &a, const sqdd &b){ return sq_divu(a, b, sqdd_rcp(b)); }
#endif
SQDD_HD sqdd &operator+=(sqdd &a, const sqdd &b){ a = a + b; return a; }
SQDD_HD sqdd &operator-=(sqdd &a, const sqdd &b){ a = a - b; return a; }
SQDD_HD sqdd &operator*=(sqdd &a, const sqdd &b){ a = a * b; return a; }
SQDD_HD sqdd &operator/=(sqdd &a, const sqdd &b){ a = a / b; return a; }
SQDD_HD bool operator<(const sqdd &a, const sqdd &b){ return a.hi < b.hi || (a.hi == b.hi && a.lo < b.lo); }
SQDD_HD bool operator>(const sqdd &a, const sqdd &b){ return b < a; }
SQDD_HD bool operator<=(const sqdd &a, const sqdd &b){ return !(b < a); }
SQDD_HD bool operator>=(const sqdd &a, const sqdd &b){ return !(a < b); }
SQDD_HD bool operator==(const sqdd &a, const sqdd &b){ return a.hi == b.hi && a.lo == b.lo; }
SQDD_HD bool operator!=(const sqdd &a, const sqdd &b){ return !(a == b); }
/* mixed forms with int and double operands: the scalar is not promoted to a double-double */
SQDD_HD sqdd operator+(int a, const sqdd &b){ return sqdd_add_d(b, (double)a); }
SQDD_HD sqdd operator+(const sqdd &a, int b){ return sqdd_add_d(a, (double)b); }
SQDD_HD sqdd operator-(int a, const sqdd &b){ return sqdd_add_d(-b, (double)a); }
SQDD_HD sqdd operator-(const sqdd &a, int b){ return sqdd_add_d(a, -(double)b); }
SQDD_HD sqdd operator*(int a, const sqdd &b){ return sqdd_mul_d(b, (double)a); }
SQDD_HD sqdd operator*(const sqdd &a, int b){ return sqdd_mul_d(a, (double)b); }
SQDD_HD sqdd operator/(int a, const sqdd &b){ return sqdd((double)a) / b; }
SQDD_HD sqdd operator/(const sqdd &a, int b){ return a / sqdd((double)b); }
SQDD_HD sqdd operator+(double a, const sqdd &b){ return sqdd_add_d(b, a); }
SQDD_HD sqdd operator+(const sqdd &a, double b){ return sqdd_add_d(a, b); }
SQDD_HD sqdd operator-(double a, const sqdd &b){ return sqdd_add_d(-b, a); }
SQDD_HD sqdd operator-(const sqdd &a, double b){ return sqdd_add_d(a, -b); }
SQDD_HD sqdd operator*(double a, const sqdd &b){ return sqdd_mul_d(b, a); }
SQDD_HD sqdd operator*(const sqdd &a, double b){ return sqdd_mul_d(a, b); }
SQDD_HD bool operator<(const sqdd &a, int b){ return a < sqdd((double)b); }
SQDD_HD bool operator>(const sqdd &a, int b){ return a > sqdd((double)b); }
SQDD_HD bool operator!=(const sqdd &a, int b){ return a != sqdd((double)b); }
SQDD_HD bool operator==(const sqdd &a, int b){ return a == sqdd((double)b); }

/* |x| with the reference's RABS semantics (x < 0 ? -x : x, driver/common.h:23) */
SQDD_HD sqdd sq_rabs(const sqdd &x){ return x < sqdd(0.0) ? -x : x; }
/* in double the sign of a zero never reaches a result (every |.| value is only added and multiplied
 * into non-negative sums), so the single sign-clearing instruction is used */
SQDD_HD double sq_rabs(double x){ return fabs(x); }

/* e^a in double-double: a = (128 m + j) ln2/128 + r with |r| <= 0.0028, e^a = 2^m 2^(j/128) e^r, by a table of 2^(j/128)
 * (three parts, from 100-digit values) and the Taylor series of e^r to degree 10 (truncation below 2e-36), its terms
 * from r^6/6! on summed in double (they are below 6e-19) and the others in double-double.  ln 2 comes in three
 * parts whose products with k are exact, so that r is accurate for every m.  About 170 operations; the reduction by
 * 2^-10 with ten doublings that this replaces took 410, its roundings amplified by the doublings: largest relative
 * error over 2e4 arguments |a| < 0.01, 1, 35, 600 against 60-digit values: 1.2e-32, 1.1e-32, 8.7e-33, 7.9e-33, before
 * 1.2e-32, 2.9e-32, 5.5e-31, 1.4e-29.  Every step is a double-double operation of this file or an fma, so host
 * and device results agree bit for bit. */
#define SQDD_EXP2_128 { \
    0x1.0000000000000p+0, 0x0.0p+0, 0x0.0p+0, \
    0x1.0163da9fb3335p+0, 0x1.b61299ab8cdb7p-54, 0x1.bf48007d80987p-109, \
    0x1.02c9a3e778061p+0, -0x1.19083535b085dp-56, -0x1.9085b0a3d74d5p-110, \
    0x1.04315e86e7f85p+0, -0x1.0a31c1977c96ep-54, -0x1.912fbf44b4040p-112, \
    0x1.059b0d3158574p+0, 0x1.d73e2a475b465p-55, 0x1.05ff94f8d257ep-110, \
    0x1.0706b29ddf6dep+0, -0x1.c91dfe2b13c27p-55, 0x1.fb41f2e2c24abp-110, \
    0x1.0874518759bc8p+0, 0x1.186be4bb284ffp-57, 0x1.15820d96b414fp-111, \
    0x1.09e3ecac6f383p+0, 0x1.1487818316136p-54, -0x1.48b45d1fdc259p-108, \
    0x1.0b5586cf9890fp+0, 0x1.8a62e4adc610bp-54, -0x1.67c9bd6ebf74cp-108, \
    0x1.0cc922b7247f7p+0, 0x1.01edc16e24f71p-54, 0x1.e8aac564e6fe3p-108, \
    0x1.0e3ec32d3d1a2p+0, 0x1.03a1727c57b53p-59, -0x1.5aa76994e9ddbp-113, \
    0x1.0fb66affed31bp+0, -0x1.b9bedc44ebd7bp-57, -0x1.aeb1f49d84259p-112, \
    0x1.11301d0125b51p+0, -0x1.6c51039449b3ap-54, 0x1.9d58b988f562dp-109, \
    0x1.12abdc06c31ccp+0, -0x1.1b514b36ca5c7p-58, -0x1.08d8f42083120p-112, \
    0x1.1429aaea92de0p+0, -0x1.32fbf9af1369ep-54, -0x1.2fe7bb4c76416p-108, \
    0x1.15a98c8a58e51p+0, 0x1.2406ab9eeab0ap-55, -0x1.01b575279c474p-110, \
    0x1.172b83c7d517bp+0, -0x1.19041b9d78a76p-55, 0x1.4f2406aa13ff0p-109, \
    0x1.18af9388c8deap+0, -0x1.11023d1970f6cp-54, 0x1.725f0040b97c5p-110, \
    0x1.1a35beb6fcb75p+0, 0x1.e5b4c7b4968e4p-55, 0x1.ad36183926ae8p-111, \
    0x1.1bbe084045cd4p+0, -0x1.95386352ef607p-54, -0x1.40ca69503718ep-109, \
    0x1.1d4873168b9aap+0, 0x1.e016e00a2643cp-54, 0x1.ea62d0881b918p-110, \
    0x1.1ed5022fcd91dp+0, -0x1.1df98027bb78cp-54, 0x1.e504d36c47475p-108, \
    0x1.2063b88628cd6p+0, 0x1.dc775814a8495p-55, -0x1.781dbc16f1ea4p-111, \
    0x1.21f49917ddc96p+0, 0x1.2a97e9494a5eep-55, -0x1.693c2b3b7106bp-109, \
    0x1.2387a6e756238p+0, 0x1.9b07eb6c70573p-54, -0x1.4d89f9af532e0p-109, \
    0x1.251ce4fb2a63fp+0, 0x1.ac155bef4f4a4p-55, 0x1.1a9c8afdcf797p-112, \
    0x1.26b4565e27cddp+0, 0x1.2bd339940e9d9p-55, 0x1.277393a461b77p-110, \
    0x1.284dfe1f56381p+0, -0x1.a4c3a8c3f0d7ep-54, 0x1.67fdaa2e52d7dp-108, \
    0x1.29e9df51fdee1p+0, 0x1.612e8afad1255p-55, 0x1.de54485604690p-111, \
    0x1.2b87fd0dad990p+0, -0x1.10adcd6381aa4p-59, 0x1.0885fb8796dbdp-113, \
    0x1.2d285a6e4030bp+0, 0x1.0024754db41d5p-54, -0x1.ee9d8f8cb9307p-110, \
    0x1.2ecafa93e2f56p+0, 0x1.1ca0f45d52383p-56, 0x1.d7b08dee6d12ap-111, \
    0x1.306fe0a31b715p+0, 0x1.6f46ad23182e4p-55, 0x1.7b7b2f09cd0d9p-110, \
    0x1.32170fc4cd831p+0, 0x1.a9ce78e18047cp-55, 0x1.b778c882b85e8p-110, \
    0x1.33c08b26416ffp+0, 0x1.32721843659a6p-54, -0x1.406a2ea6cfc6bp-108, \
    0x1.356c55f929ff1p+0, -0x1.b5cee5c4e4628p-55, -0x1.8e524e520d5f2p-109, \
    0x1.371a7373aa9cbp+0, -0x1.63aeabf42eae2p-54, 0x1.87e3e12516bfap-108, \
    0x1.38cae6d05d866p+0, -0x1.e958d3c9904bdp-54, 0x1.0a77a61404f21p-109, \
    0x1.3a7db34e59ff7p+0, -0x1.5e436d661f5e3p-56, 0x1.9b0b1ff17c296p-111, \
    0x1.3c32dc313a8e5p+0, -0x1.efff8375d29c3p-54, -0x1.1143f2a93395ap-109, \
    0x1.3dea64c123422p+0, 0x1.ada0911f09ebcp-55, -0x1.808ba68fa8fb7p-109, \
    0x1.3fa4504ac801cp+0, -0x1.7d023f956f9f3p-54, -0x1.0473e3724200dp-108, \
    0x1.4160a21f72e2ap+0, -0x1.ef3691c309278p-58, -0x1.32b43eafc6518p-114, \
    0x1.431f5d950a897p+0, -0x1.1c7dde35f7999p-55, 0x1.903c496195fefp-109, \
    0x1.44e086061892dp+0, 0x1.89b7a04ef80d0p-59, -0x1.0ac312de3d922p-114, \
    0x1.46a41ed1d0057p+0, 0x1.c944bd1648a76p-54, 0x1.7df404ff21f3ap-108, \
    0x1.486a2b5c13cd0p+0, 0x1.3c1a3b69062f0p-56, 0x1.e1eebae743ac0p-111, \
    0x1.4a32af0d7d3dep+0, 0x1.9cb62f3d1be56p-54, 0x1.91876c761e2c7p-110, \
    0x1.4bfdad5362a27p+0, 0x1.d4397afec42e2p-56, 0x1.c06c7745c2b39p-113, \
    0x1.4dcb299fddd0dp+0, 0x1.8ecdbbc6a7833p-54, 0x1.212c969559b43p-110, \
    0x1.4f9b2769d2ca7p+0, -0x1.4b309d25957e3p-54, -0x1.1aa1fd7b685cdp-112, \
    0x1.516daa2cf6642p+0, -0x1.f768569bd93efp-55, 0x1.90e718226177dp-112, \
    0x1.5342b569d4f82p+0, -0x1.07abe1db13cadp-55, 0x1.fa733951f214cp-111, \
    0x1.551a4ca5d920fp+0, -0x1.d689cefede59bp-55, 0x1.9c991771b0493p-110, \
    0x1.56f4736b527dap+0, 0x1.9bb2c011d93adp-54, -0x1.ff86852a613ffp-111, \
    0x1.58d12d497c7fdp+0, 0x1.295e15b9a1de8p-55, -0x1.a26d92ad1e4c6p-109, \
    0x1.5ab07dd485429p+0, 0x1.6324c054647adp-54, -0x1.744ee506fdafep-109, \
    0x1.5c9268a5946b7p+0, 0x1.c4b1b816986a2p-60, 0x1.ec2735254978cp-119, \
    0x1.5e76f15ad2148p+0, 0x1.ba6f93080e65ep-54, -0x1.95f9ab75fa7d6p-108, \
    0x1.605e1b976dc09p+0, -0x1.3e2429b56de47p-54, -0x1.32c54b92e2588p-110, \
    0x1.6247eb03a5585p+0, -0x1.383c17e40b497p-54, 0x1.5d8e757cfb991p-111, \
    0x1.6434634ccc320p+0, -0x1.c483c759d8933p-55, 0x1.3904000c1c40fp-110, \
    0x1.6623882552225p+0, -0x1.bb60987591c34p-54, 0x1.4a337f4dc0a3bp-108, \
    0x1.68155d44ca973p+0, 0x1.038ae44f73e65p-57, -0x1.f2803633b04ffp-113, \
    0x1.6a09e667f3bcdp+0, -0x1.bdd3413b26456p-54, 0x1.57d3e3adec175p-108, \
    0x1.6c012750bdabfp+0, -0x1.2895667ff0b0dp-56, 0x1.fef5c58766c19p-111, \
    0x1.6dfb23c651a2fp+0, -0x1.bbe3a683c88abp-57, 0x1.a59f88abbe778p-115, \
    0x1.6ff7df9519484p+0, -0x1.83c0f25860ef6p-55, -0x1.001923f4a956ep-110, \
    0x1.71f75e8ec5f74p+0, -0x1.16e4786887a99p-55, -0x1.269796953a4c3p-109, \
    0x1.73f9a48a58174p+0, -0x1.0a8d96c65d53cp-54, 0x1.82ae217f3a768p-108, \
    0x1.75feb564267c9p+0, -0x1.0245957316dd3p-54, -0x1.8f8e7fa19e5e8p-108, \
    0x1.780694fde5d3fp+0, 0x1.866b80a02162dp-54, -0x1.44d42307932f7p-108, \
    0x1.7a11473eb0187p+0, -0x1.41577ee04992fp-55, -0x1.4217a932d10d4p-113, \
    0x1.7c1ed0130c132p+0, 0x1.f124cd1164dd6p-54, -0x1.d4d236cc2bb03p-108, \
    0x1.7e2f336cf4e62p+0, 0x1.05d02ba15797ep-56, 0x1.70a1427f8fcdfp-112, \
    0x1.80427543e1a12p+0, -0x1.27c86626d972bp-54, 0x1.d4e0d71c9b16ep-109, \
    0x1.82589994cce13p+0, -0x1.d4c1dd41532d8p-54, 0x1.0f6ad65cbbac1p-112, \
    0x1.8471a4623c7adp+0, -0x1.8d684a341cdfbp-55, -0x1.591e15c16efd1p-109, \
    0x1.868d99b4492edp+0, -0x1.fc6f89bd4f6bap-54, -0x1.f16f65181d921p-109, \
    0x1.88ac7d98a6699p+0, 0x1.994c2f37cb53ap-54, 0x1.d61283ef385dep-108, \
    0x1.8ace5422aa0dbp+0, 0x1.6e9f156864b27p-54, -0x1.30644a7836333p-110, \
    0x1.8cf3216b5448cp+0, -0x1.0d55e32e9e3aap-56, -0x1.3dab3db839dd6p-111, \
    0x1.8f1ae99157736p+0, 0x1.5cc13a2e3976cp-55, 0x1.3bf26d2b85163p-114, \
    0x1.9145b0b91ffc6p+0, -0x1.dd6792e582524p-54, 0x1.c03855204534ap-109, \
    0x1.93737b0cdc5e5p+0, -0x1.75fc781b57ebcp-57, 0x1.697e257ac0db2p-111, \
    0x1.95a44cbc8520fp+0, -0x1.64b7c96a5f039p-56, -0x1.07053c9a98bbbp-113, \
    0x1.97d829fde4e50p+0, -0x1.d185b7c1b85d1p-54, 0x1.7edb9d7144b6fp-108, \
    0x1.9a0f170ca07bap+0, -0x1.173bd91cee632p-54, -0x1.053987854965fp-110, \
    0x1.9c49182a3f090p+0, 0x1.c7c46b071f2bep-56, 0x1.6376b7943085cp-110, \
    0x1.9e86319e32323p+0, 0x1.824ca78e64c6ep-56, 0x1.0f92c082bbae0p-116, \
    0x1.a0c667b5de565p+0, -0x1.359495d1cd533p-54, 0x1.354084551b4fbp-109, \
    0x1.a309bec4a2d33p+0, 0x1.6305c7ddc36abp-54, 0x1.547fa22c26d17p-108, \
    0x1.a5503b23e255dp+0, -0x1.d2f6edb8d41e1p-54, -0x1.bfd7adfd63f48p-111, \
    0x1.a799e1330b358p+0, 0x1.bcb7ecac563c7p-54, -0x1.678693176f751p-108, \
    0x1.a9e6b5579fdbfp+0, 0x1.0fac90ef7fd31p-54, 0x1.8b16ae39e8cb9p-109, \
    0x1.ac36bbfd3f37ap+0, -0x1.f9234cae76cd0p-55, -0x1.c60dbfc7696f8p-111, \
    0x1.ae89f995ad3adp+0, 0x1.7a1cd345dcc81p-54, 0x1.a7fbc3ae675eap-108, \
    0x1.b0e07298db666p+0, -0x1.bdef54c80e425p-54, 0x1.41cbb95c55600p-109, \
    0x1.b33a2b84f15fbp+0, -0x1.2805e3084d708p-57, 0x1.2babc0edda4d9p-111, \
    0x1.b59728de5593ap+0, -0x1.c71dfbbba6de3p-54, -0x1.c7470081df7dfp-111, \
    0x1.b7f76f2fb5e47p+0, -0x1.5584f7e54ac3bp-56, 0x1.aa64481e1ab72p-111, \
    0x1.ba5b030a1064ap+0, -0x1.efcd30e54292ep-54, -0x1.ad1bf91503c67p-113, \
    0x1.bcc1e904bc1d2p+0, 0x1.23dd07a2d9e84p-55, 0x1.9a164050e1258p-109, \
    0x1.bf2c25bd71e09p+0, -0x1.efdca3f6b9c73p-54, 0x1.27e81cecd59dap-110, \
    0x1.c199bdd85529cp+0, 0x1.11065895048ddp-55, 0x1.99e51125928dap-110, \
    0x1.c40ab5fffd07ap+0, 0x1.b4537e083c60ap-54, 0x1.4a6cdfa70f4f8p-109, \
    0x1.c67f12e57d14bp+0, 0x1.2884dff483cadp-54, -0x1.fc44c329d5cb2p-109, \
    0x1.c8f6d9406e7b5p+0, 0x1.1acbc48805c44p-56, 0x1.6edaac100b8fap-111, \
    0x1.cb720dcef9069p+0, 0x1.503cbd1e949dbp-56, 0x1.d8765566b032ep-110, \
    0x1.cdf0b555dc3fap+0, -0x1.dd83b53829d72p-55, -0x1.aea073a742049p-112, \
    0x1.d072d4a07897cp+0, -0x1.cbc3743797a9cp-54, -0x1.e7044039da0f6p-108, \
    0x1.d2f87080d89f2p+0, -0x1.d487b719d8578p-54, 0x1.2da62b2a9fae7p-111, \
    0x1.d5818dcfba487p+0, 0x1.2ed02d75b3707p-55, -0x1.ab053b05531fcp-111, \
    0x1.d80e316c98398p+0, -0x1.11ec18beddfe8p-54, -0x1.ed04e7ac8765ap-110, \
    0x1.da9e603db3285p+0, 0x1.c2300696db532p-54, 0x1.7f6246f0ec615p-108, \
    0x1.dd321f301b460p+0, 0x1.2da5778f018c3p-54, -0x1.c6cdead661cf3p-108, \
    0x1.dfc97337b9b5fp+0, -0x1.1a5cd4f184b5cp-54, 0x1.b7225a944efd6p-108, \
    0x1.e264614f5a129p+0, -0x1.7b627817a1496p-54, -0x1.b9818808c409ap-108, \
    0x1.e502ee78b3ff6p+0, 0x1.39e8980a9cc8fp-55, 0x1.1e92cb3c2d278p-109, \
    0x1.e7a51fbc74c83p+0, 0x1.2d522ca0c8de2p-54, -0x1.8a757b0b6a9cbp-108, \
    0x1.ea4afa2a490dap+0, -0x1.e9c23179c2893p-54, -0x1.fc0f242bbf3dep-109, \
    0x1.ecf482d8e67f1p+0, -0x1.c93f3b411ad8cp-54, -0x1.0b9dfef44b43bp-108, \
    0x1.efa1bee615a27p+0, 0x1.dc7f486a4b6b0p-54, 0x1.f6dd5d229ff69p-108, \
    0x1.f252b376bba97p+0, 0x1.3a1a5bf0d8e43p-54, 0x1.4c6ad5476b516p-108, \
    0x1.f50765b6e4540p+0, 0x1.9d3e12dd8a18bp-54, -0x1.4019bffc80ef3p-110, \
    0x1.f7bfdad9cbe14p+0, -0x1.dbb12d006350ap-54, 0x1.5c5ce7280fa4dp-108, \
    0x1.fa7c1819e90d8p+0, 0x1.74853f3a5931ep-55, 0x1.dc060c36f7651p-112, \
    0x1.fd3c22b8f71f1p+0, 0x1.2eb74966579e7p-57, 0x1.2f096934ec56cp-111 \
    }
#if defined(__CUDACC__)
static __device__ const double sqdd_exp2_dev[384] = SQDD_EXP2_128;
#endif
static const double sqdd_exp2_host[384] = SQDD_EXP2_128;
/* a + b for |a| > |b| */
SQDD_HD sqdd sqdd_add_less(const sqdd &a, const sqdd &b){
    sqdd s = sqdd_quick_two_sum(a.hi, b.hi);
    s.lo = SQ_ADD(s.lo, SQ_ADD(a.lo, b.lo));
    return sqdd_quick_two_sum(s.hi, s.lo);
}
SQDD_HD sqdd sqdd_exp(const sqdd &a){
    if(a.hi > 709.0) return sqdd(exp(a.hi));          /* overflow: +inf */
    if(a.hi < -745.0) return sqdd(0.0);
    if(!(a.hi == a.hi)) return a;
    const double kd = rint(SQ_MUL(a.hi, 184.66496523378731));  /* 128/ln2 */
    const int k = (int)kd, j = k & 127, m = (k - j)/128;
    /* ln2/128 in parts of 35, 35 and 53 bits: |k| < 2^18, so a.hi - k L1 and k L2 are exact */
    const sqdd d = sqdd_two_sum(SQ_FMA(-kd, 0x1.62e42fef80000p-8, a.hi), -SQ_MUL(kd, 0x1.1cf79abc80000p-43)), e = sqdd_two_sum(d.hi, a.lo);
    const sqdd r = sqdd_quick_two_sum(e.hi, SQ_FMA(-kd, 0x1.e3b39803f2f6bp-79, SQ_ADD(d.lo, e.lo)));
    /* 1/6! .. 1/10! in double, 1/5!, 1/4!, 1/3! in double-double */
    const double x = r.hi;
    const double t = SQ_MUL(x, SQ_FMA(x, SQ_FMA(x, SQ_FMA(x, SQ_FMA(x, 2.755731922398589e-07, 2.7557319223985893e-06),
                     2.48015873015873e-05), 0.0001984126984126984), 0.001388888888888889));
    sqdd s = sqdd_quick_two_sum(0.008333333333333333, t);
    s.lo = SQ_ADD(s.lo, 1.1564823173178714e-19);
    s = sqdd_add_less(sqdd(0.041666666666666664, 2.3129646346357427e-18), s*r);
    s = sqdd_add_less(sqdd(0.16666666666666666, 9.25185853854297e-18), s*r);
    s = sqdd_add_less(sqdd(0.5), s*r);
    s = sqdd_add_less(sqdd(1.0), s*r);
    s = s*r;                                                   /* e^r - 1 */
#if defined(__CUDA_ARCH__)
    const sqdd E(__ldg(sqdd_exp2_dev + 3*j), __ldg(sqdd_exp2_dev + 3*j + 1));
    const double E3 = __ldg(sqdd_exp2_dev + 3*j + 2);
#else
    const sqdd E(sqdd_exp2_host[3*j], sqdd_exp2_host[3*j + 1]);
    const double E3 = sqdd_exp2_host[3*j + 2];
#endif
    /* E + E s with one rounding of the low part */
    s = E*s;
    const sqdd h = sqdd_quick_two_sum(E.hi, s.hi), l = sqdd_two_sum(h.lo, E.lo);
    const sqdd u = sqdd_quick_two_sum(h.hi, l.hi);
    s = sqdd_quick_two_sum(u.hi, SQ_ADD(u.lo, SQ_ADD(l.lo, SQ_ADD(s.lo, E3))));
#if defined(__CUDA_ARCH__)
    if(m > -960 && m < 1000){                                  /* 2^m and the product are normal numbers */
        const double p = __hiloint2double((m + 1023) << 20, 0);
        return sqdd(SQ_MUL(s.hi, p), SQ_MUL(s.lo, p));
    }
#endif
    return sqdd(ldexp(s.hi, m), ldexp(s.lo, m));
}
/* log a in double-double: with x the double logarithm of the high part, log a = x + log(1 + e), e = a e^{-x} - 1 at most an
 * ulp of x: the first two terms of its series (without the second, |log a| = 600 came out at 9e-31 relative) */
SQDD_HD sqdd sqdd_log(const sqdd &a){
    if(!(a.hi > 0)) return sqdd(log(a.hi));
    const sqdd x(log(a.hi)), y = sqdd_exp(-x), p = sqdd_two_prod(a.hi, y.hi);
    const sqdd e = sqdd_two_sum(SQ_SUB(p.hi, 1.0), SQ_FMA(a.hi, y.lo, SQ_FMA(a.lo, y.hi, p.lo)));
    return x + sqdd_add_d(e, SQ_MUL(-0.5, SQ_MUL(e.hi, e.hi)));
}
/* exp and log for the integrands that need them (SQ_EXP, SQ_LOG): the double versions are the math
 * library's, the double-double versions the ones above */
SQDD_HD double sq_exp(double x){ return exp(x); }
SQDD_HD double sq_log(double x){ return log(x); }
SQDD_HD sqdd sq_exp(const sqdd &x){ return sqdd_exp(x); }
SQDD_HD sqdd sq_log(const sqdd &x){ return sqdd_log(x); }
