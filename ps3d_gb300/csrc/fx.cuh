// Fixed-point FFTs for the FP64 transforms.
//
// GB300 issues FP64 at 1/64 of the FP32 rate (2 results per clock and SM),
// and 32-bit integer multiply-adds at 64: an FP64 FFT is bound by the FP64
// pipe at 10-15 times the time its bytes take.  Here a real line is turned
// into 64-bit integers on one scale per line (its largest magnitude), the
// FFT runs on the integer pipes, and the outputs go back to FP64.  Sums are
// exact; a product with a twiddle keeps 63 bits, so the rounding of a whole
// transform stays below that of the FP64 Stockham transforms it stands for, at
// every length they serve (mean over random lines of the error relative to the
// line's norm, 0.1 to 0.85 of theirs: tests/test_fx_accuracy.py).  A unit is
// common to a line, so single lines can be above: entries far below its largest
// hold fewer bits than FP64.
//
// Everything here is plain integer arithmetic, compiled for host and device:
// the host build of the same functions is what the CPU test runs.
#pragma once
#include <limits.h>
#include <math.h>
#include <stdint.h>

#include <cuda_runtime.h>

namespace ps3d {
namespace fx {

using I2 = longlong2;
#define FX_FN __host__ __device__ __forceinline__

FX_FN I2 mk2(long long x, long long y)
{
    I2 r;
    r.x = x;
    r.y = y;
    return r;
}
FX_FN I2 add(I2 a, I2 b) { return mk2(a.x + b.x, a.y + b.y); }
FX_FN I2 sub(I2 a, I2 b) { return mk2(a.x - b.x, a.y - b.y); }

// a 64-bit value as hi 2^32 + lo with both halves signed 32-bit
struct Half {
    int h, l;
};
FX_FN Half split(long long x)
{
    Half r;
    r.l = (int)(unsigned)x;
    r.h = (int)(unsigned)((uint64_t)x >> 32) + (int)(((unsigned)x) >> 31);
    return r;
}
// a b + c, 32 x 32 + 64 bits.  The device form is spelled out: from the C
// expression the compiler makes separate 64-bit sums (a complex product took
// 71 instructions, 29 here), and these products at 32 per clock and SM are
// what the transforms' arithmetic costs most.
FX_FN long long wide(int a, int b, long long c)
{
#ifdef __CUDA_ARCH__
    long long r;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
    return r;
#else
    return (long long)a * (long long)b + c;
#endif
}
// the upper word, sign extended
FX_FN long long high(long long m)
{
#ifdef __CUDA_ARCH__
    return (long long)(int)__double2hiint(__longlong_as_double(m));
#else
    return m >> 32;
#endif
}
constexpr long long ROUND = 0x80000000ll;

// c + round(x w / 2^64), the product within one unit; |x| < 2^63 - 2^31
FX_FN long long mulh(Half x, Half w, long long c = 0)
{
    return wide(x.h, w.h, c + high(wide(x.l, w.h, wide(x.h, w.l, ROUND))));
}
// x c for a constant 0 < c < 1: c 2^64 where c < 1/2, else x + x (c - 1)
template <long long CM> FX_FN long long mulc(long long x)
{
    constexpr int l = (int)(unsigned)CM, h = (int)((CM >> 32) + (((unsigned)CM) >> 31));
    return mulh(split(x), Half{h, l}, CM < 0 ? x : 0);
}

// complex product with a twiddle w = (cos, sin) 2^62 (halves already split,
// no lower half is -2^31): z w / 4
struct Tw {
    int ch, cl, sh, sl;
};
FX_FN I2 cmulw(I2 z, Tw w, bool conj)
{
    const Half a = split(z.x), b = split(z.y);
    const int mh = -w.sh, ml = -w.sl;
    const int ph = conj ? mh : w.sh, pl = conj ? ml : w.sl;  // w.y
    const int nh = conj ? w.sh : mh, nl = conj ? w.sl : ml;  // -w.y
    const long long mr = wide(b.l, nh, wide(b.h, nl, wide(a.l, w.ch, wide(a.h, w.cl, ROUND))));
    const long long mi = wide(a.l, ph, wide(a.h, pl, wide(b.l, w.ch, wide(b.h, w.cl, ROUND))));
    return mk2(wide(b.h, nh, wide(a.h, w.ch, high(mr))), wide(a.h, ph, wide(b.h, w.ch, high(mi))));
}
// z / 4, rounded
FX_FN I2 quarter(I2 z) { return mk2((z.x + 2) >> 2, (z.y + 2) >> 2); }

template <bool INV> FX_FN I2 mul_mi(I2 a) { return INV ? mk2(-a.y, a.x) : mk2(a.y, -a.x); }

FX_FN void dft2(I2 &a, I2 &b)
{
    const I2 t = a;
    a = add(t, b);
    b = sub(t, b);
}
template <bool INV> FX_FN void dft4(I2 &a0, I2 &a1, I2 &a2, I2 &a3)
{
    const I2 t0 = add(a0, a2), t1 = sub(a0, a2), t2 = add(a1, a3), u = sub(a1, a3);
    a0 = add(t0, t2);
    a2 = sub(t0, t2);
    // t1 + (-i u) and t1 - (-i u) (forward), without forming -u
    a1 = INV ? mk2(t1.x - u.y, t1.y + u.x) : mk2(t1.x + u.y, t1.y - u.x);
    a3 = INV ? mk2(t1.x + u.y, t1.y - u.x) : mk2(t1.x - u.y, t1.y + u.x);
}
// c 2^64, or (c - 1) 2^64 where c >= 1/2
constexpr long long C_R2 = -5402926248376769404ll;  // 1 / sqrt 2
constexpr long long C_S3 = -2471395088767036514ll;  // sqrt 3 / 2
constexpr long long C_C1 = 5700357409661599243ll;  // cos(2 pi / 5)
constexpr long long C_C2 = -3523014627193176565ll;  // -cos(4 pi / 5)
constexpr long long C_S1 = -902847917979075853ll;  // sin(2 pi / 5)
constexpr long long C_S2 = -7604019954369499282ll;  // sin(4 pi / 5)
template <bool INV> FX_FN void dft8(I2 *v)
{
    dft4<INV>(v[0], v[2], v[4], v[6]);
    dft4<INV>(v[1], v[3], v[5], v[7]);
    const I2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    const I2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = add(e0, o0);
    v[4] = sub(e0, o0);
    if (!INV) {
        // o1 (1 - i)/sqrt2, -i o2, o3 (-1 - i)/sqrt2
        const long long p = mulc<C_R2>(o1.x + o1.y), q = mulc<C_R2>(o1.y - o1.x);
        const long long r = mulc<C_R2>(o3.y - o3.x), s = mulc<C_R2>(o3.x + o3.y);
        v[1] = mk2(e1.x + p, e1.y + q);
        v[5] = mk2(e1.x - p, e1.y - q);
        v[2] = mk2(e2.x + o2.y, e2.y - o2.x);
        v[6] = mk2(e2.x - o2.y, e2.y + o2.x);
        v[3] = mk2(e3.x + r, e3.y - s);
        v[7] = mk2(e3.x - r, e3.y + s);
    } else {
        const long long p = mulc<C_R2>(o1.x - o1.y), q = mulc<C_R2>(o1.x + o1.y);
        const long long r = mulc<C_R2>(o3.x + o3.y), s = mulc<C_R2>(o3.x - o3.y);
        v[1] = mk2(e1.x + p, e1.y + q);
        v[5] = mk2(e1.x - p, e1.y - q);
        v[2] = mk2(e2.x - o2.y, e2.y + o2.x);
        v[6] = mk2(e2.x + o2.y, e2.y - o2.x);
        v[3] = mk2(e3.x - r, e3.y + s);
        v[7] = mk2(e3.x + r, e3.y - s);
    }
}
template <bool INV> FX_FN void dft3(I2 *v)
{
    const I2 t1 = add(v[1], v[2]), t2 = sub(v[1], v[2]);
    const I2 m = mk2(v[0].x - (t1.x >> 1), v[0].y - (t1.y >> 1));
    const long long a = mulc<C_S3>(t2.y), b = mulc<C_S3>(t2.x);
    const I2 s = INV ? mk2(-a, b) : mk2(a, -b);
    v[0] = add(v[0], t1);
    v[1] = add(m, s);
    v[2] = sub(m, s);
}
template <bool INV> FX_FN void dft5(I2 *v)
{
    const I2 t1 = add(v[1], v[4]), t2 = add(v[2], v[3]), t3 = sub(v[1], v[4]), t4 = sub(v[2], v[3]);
    const I2 m1 = mk2(v[0].x + mulc<C_C1>(t1.x) - mulc<C_C2>(t2.x), v[0].y + mulc<C_C1>(t1.y) - mulc<C_C2>(t2.y));
    const I2 m2 = mk2(v[0].x - mulc<C_C2>(t1.x) + mulc<C_C1>(t2.x), v[0].y - mulc<C_C2>(t1.y) + mulc<C_C1>(t2.y));
    const I2 n1 = mk2(mulc<C_S1>(t3.x) + mulc<C_S2>(t4.x), mulc<C_S1>(t3.y) + mulc<C_S2>(t4.y));
    const I2 n2 = mk2(mulc<C_S2>(t3.x) - mulc<C_S1>(t4.x), mulc<C_S2>(t3.y) - mulc<C_S1>(t4.y));
    const I2 j1 = INV ? mk2(-n1.y, n1.x) : mk2(n1.y, -n1.x);
    const I2 j2 = INV ? mk2(-n2.y, n2.x) : mk2(n2.y, -n2.x);
    v[0] = add(v[0], add(t1, t2));
    v[1] = add(m1, j1);
    v[4] = sub(m1, j1);
    v[2] = add(m2, j2);
    v[3] = sub(m2, j2);
}
template <int R, bool INV> FX_FN void dft(I2 *v)
{
    if (R == 2) dft2(v[0], v[1]);
    else if (R == 3) dft3<INV>(v);
    else if (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
    else if (R == 5) dft5<INV>(v);
    else dft8<INV>(v);
}

// The passes of a length: radix 8 while 8 divides what is left, one radix 4
// or 2, then 3s and 5s.  Every pass after the first divides by 4 (its
// twiddles are held at 2^62 and products keep the upper 64 bits), or by 2
// (its input is doubled) where the radix is below 8.  A line of length
// 2 odd starts with a 5 or 3 and takes the 2 later.
FX_FN int next_radix(int rem)
{
    return rem % 8 == 0 ? 8 : rem % 4 == 0 ? 4 : rem % 2 == 0 ? 2 : rem % 3 == 0 ? 3 : rem % 5 == 0 ? 5 : 1;
}
FX_FN int first_radix(int n)
{
    return n % 8 == 0 ? 8 : n % 4 == 0 ? 4 : n % 5 == 0 ? 5 : n % 3 == 0 ? 3 : 2;
}
FX_FN constexpr int up_shift(int r) { return r <= 5 ? 1 : 0; }

// Bits of the fixed-point form.  A line is held in units of 2^(e + 1 - E),
// 2^e <= its largest magnitude < 2^(e+1): magnitudes up to 2^E.  E is the
// largest that keeps every modulus of the transform at 2^61.5 or less, which
// leaves one bit for the sum of two outputs that separates a forward pair
// and for the doubled input of a small radix.  A modulus after the passes of product p
// is bounded by p times the largest input and by the sum over the line's
// inputs: l, the least with sum < 2^(l + e + 1), is measured per line, so that
// a line with a few large entries (a decaying spectrum) keeps more bits.  It
// counts from 2^(e+1) as the unit does: counted from the largest magnitude
// it allows for up to a bit that is not there, in the lines whose largest
// value lies just above 2^e and whose unit is coarsest as it is.
// Two real lines go as a + i b: moduli up to 2^(E+1/2), sums 2^(E+1+l); a
// pair of Hermitian spectra one bit more of each; a column pair is folded
// first: sums of four terms, then a quarter of them.  Every input enters two
// terms of a folded sequence (the middle one a doubled term), so a sequence
// sums to at most half of what the columns do: 2^(E+l).
constexpr int MAXL = 13;
struct Plan {
    signed char E[MAXL];  // bits for l = 0..MAXL-1
    int lcap;             // ceil(log2 of the number of inputs)
    int up;               // power of two the passes divided by, and the last product's
    Half c;               // the scale: c 2^up' with c in [1/2, 1), held as c 2^63
};
// mode 0 forward lines, 1 inverse lines, 2 columns (n: the FFTs' length)
inline Plan make_plan(int n, int mode, int inputs, double scale2)
{
    Plan pl;
    pl.lcap = 0;
    while ((1 << pl.lcap) < inputs) ++pl.lcap;
    const double m = mode == 1 ? 1.5 : 0.5, sm = mode == 1 ? 2.0 : 1.0;
    int passes = 0;
    double down = 0.0;
    for (int l = 0; l < MAXL; ++l) {
        double top = mode == 2 ? fmin(2.5, l + sm) : fmin(m, l + sm), lp = 0.0;
        down = 0.0;
        passes = 0;
        for (int rem = n; rem > 1; ++passes) {
            const int r = (mode < 2 && !passes) ? first_radix(n) : next_radix(rem);
            rem /= r;
            lp += log2((double)r);
            if (passes) down += 2.0 - up_shift(r);
            top = fmax(top, fmin(lp + m, mode == 2 ? l : l + sm) - down);
        }
        pl.E[l] = (signed char)(int)floor(61.5 - top + 1e-9);
    }
    pl.up = (int)down + (mode == 2 ? 2 : 0);
    // 1/sqrt(scale2) = c 2^-k, c in [1/2, 1)
    long double c = 1.0L / sqrtl((long double)scale2);
    while (c < 0.5L) {
        c *= 2.0L;
        pl.up -= 1;
    }
    while (c >= 1.0L) {
        c *= 0.5L;
        pl.up += 1;
    }
    pl.c = split(llrintl(c * 9223372036854775808.0L));
    pl.up += 1;  // mulh with c 2^63 halves
    return pl;
}
// forward lines carry a factor 1/2 (two outputs are added)
inline Plan line_plan(int n, bool inverse) { return make_plan(n, inverse ? 1 : 0, n, inverse ? n : 4.0 * n); }
inline Plan col_plan(int nz) { return make_plan(nz / 2, 2, nz + 1, 2.0 * nz); }
// t[k] = exp(-2 pi i k / n) 2^62 with its halves split, k < n
inline void fill_twiddles(Tw *t, int n)
{
    const long double pi = acosl(-1.0L), one = 4611686018427387904.0L;
    for (int k = 0; k < n; ++k) {
        // the angle reduced to an eighth of the circle (8 k / n exact)
        const int oct = (int)(8LL * k / n);
        const long long r = 8LL * k - (long long)oct * n;  // eighths beyond the octant, over n
        const long long f = (oct & 1) ? n - r : r;
        const long double a = pi / 4.0L * (long double)f / (long double)n;
        const long double ca = cosl(a), sa = sinl(a);
        const bool swap = ((oct + 1) >> 1) & 1;
        long double co = swap ? sa : ca, si = swap ? ca : sa;
        if (oct >= 2 && oct < 6) co = -co;
        if (oct >= 4) si = -si;
        Half c = split(llrintl(co * one)), s = split(llrintl(-si * one));
        if (c.l == INT_MIN) c.l += 1;  // its negative has to fit
        if (s.l == INT_MIN) s.l += 1;
        t[k] = Tw{c.h, c.l, s.h, s.l};
    }
}

// ----- conversion
// magnitude order of x: the upper word without its sign (monotone in |x|;
// >= 0x7ff00000 for infinities and NaN)
FX_FN unsigned mag(double x)
{
#ifdef __CUDA_ARCH__
    return (unsigned)__double2hiint(x) & 0x7fffffffu;
#else
    union { double d; uint64_t u; } c;
    c.d = x;
    return (unsigned)(c.u >> 32) & 0x7fffffffu;
#endif
}
FX_FN uint64_t bits(double x)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    union { double d; uint64_t u; } c;
    c.d = x;
    return c.u;
#endif
}
FX_FN double from_bits(uint64_t u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    union { double d; uint64_t u; } c;
    c.u = u;
    return c.d;
#endif
}
// biased exponent of a line's largest magnitude word; subnormal lines count
// as exponent 1 (their significands have no implicit bit)
FX_FN int line_exp(unsigned m)
{
    const int e = (int)(m >> 20);
    return e < 1 ? 1 : e;
}
// x in units of 2^(e + 1 - E), e the line's exponent (lexp its biased form):
// the significand at the top of 64 bits, shifted right by 64 - E and the
// distance to the line's exponent, the rest dropped.  A subnormal x counts
// as zero except in lines within 2^-64 of the subnormal range.
FX_FN long long to_fixed(double x, int lexp, int E)
{
    const uint64_t u = bits(x);
    const int e = (int)(u >> 52) & 0x7ff;
    uint64_t m = (u << 11) | 0x8000000000000000ull;
    unsigned k = (unsigned)(63 - E + lexp - e) + 1u;
    if (lexp < 70 && e == 0) {
        m = u << 11;
        k -= 1u;
    }
#ifdef __CUDA_ARCH__
    uint64_t v;
    asm("shr.u64 %0, %1, %2;" : "=l"(v) : "l"(m), "r"(k));  // amounts above 63 give 0
#else
    const uint64_t v = k > 63 ? 0 : m >> k;
#endif
    const long long s = (long long)u >> 63;
    return ((long long)v ^ s) - s;
}
// a magnitude word as FP32, 0 below FP32's normal range (above it: not a
// magnitude; spread looks at the line's largest word first)
FX_FN float magf(unsigned m)
{
    int t = (int)m - (896 << 20);
    t = t < 0 ? 0 : t;
#ifdef __CUDA_ARCH__
    return __int_as_float((int)((unsigned)t << 3));
#else
    union { float f; int i; } c;
    c.i = (int)((unsigned)t << 3);
    return c.f;
#endif
}
// l of a line from the FP32 sum of its magnitudes (rounded, of truncated
// words: raised by 1/1000) and its largest word; the bound lcap where FP32
// does not reach
FX_FN int spread(float sum, unsigned m, int lcap)
{
    if (m < (933u << 20) || m > (1123u << 20)) return lcap;
    const float r = sum * 1.001f;
#ifdef __CUDA_ARCH__
    const int q = __float_as_int(r);
#else
    union { float f; int i; } c;
    c.f = r;
    const int q = c.i;
#endif
    const int l = (q >> 23) + 896 - (int)(m >> 20);  // floor(log2 r) - e
    return l < 0 ? 0 : l > lcap ? lcap : l;
}
// how a line's fixed-point outputs go back: v c 2^k
struct Scale {
    Half c;
    int add;   // k << 20 for the upper word, where that stays in range
    bool far;  // else: exponent k (or a non-finite line)
    int k;
};
FX_FN Scale scale_of(unsigned m, int E, const Plan &pl)
{
    Scale r;
    r.c = pl.c;
    r.k = line_exp(m) - 1022 - E + pl.up;
    r.add = (int)((unsigned)r.k << 20);
    r.far = r.k < -1000 || r.k > 950 || m >= 0x7ff00000u;
    if (m >= 0x7ff00000u) r.k = 1 << 20;
    return r;
}
FX_FN double pow2(int k) { return from_bits((uint64_t)(1023 + k) << 52); }
FX_FN double far_double(double d, int k)
{
    if (k == 1 << 20) return from_bits(0x7ff8000000000000ull);  // a non-finite line gives NaN throughout
    const int a = k / 2;
    return d * pow2(a) * pow2(k - a);
}
// one rounding: the product with c is exact to the last unit of v
FX_FN double to_double(long long v, const Scale &s)
{
    const long long u = mulh(split(v), s.c);
#ifdef __CUDA_ARCH__
    const double d = __ll2double_rn(u);
    if (s.far) return far_double(d, s.k);
    const int hi = __double2hiint(d);
    return __hiloint2double(u == 0 ? hi : hi + s.add, __double2loint(d));
#else
    const double d = (double)u;
    if (s.far) return far_double(d, s.k);
    return u == 0 ? d : from_bits(bits(d) + ((uint64_t)(unsigned)s.add << 32));
#endif
}

// ----- passes
// Stockham autosort passes over nseq groups of B = 2^LB interleaved
// sequences of length n; element j of lane b at (j << LB) + (b ^ sw(j)): the
// XOR keeps accesses along j and along b free of bank conflicts.
template <int LB> FX_FN int at(int j, int b)
{
    constexpr int B = 1 << LB;
    return (j << LB) + (b ^ ((LB >= 3 ? j : j >> (3 - LB)) & (B - 1)));
}
// One pass of radix R.  Ns: product of the radices already applied;
// tw[k tws] = exp(-2 pi i k / n) 2^62, halves split.
template <int R, bool INV, int LB>
FX_FN void pass(const I2 *src, I2 *dst, int n, int nseq, int Ns, const Tw *__restrict__ tw, int tws, int tid,
                int nthreads)
{
    const int B = 1 << LB;
    const int nR = n / R;
    const int nbf = nR << LB;
    const int twstride = nR / Ns * tws;
    for (int g = tid; g < nbf * nseq; g += nthreads) {
        int h = g, off = 0;
        while (h >= nbf) {
            h -= nbf;
            off += n << LB;
        }
        const I2 *in = src + off;
        I2 *out = dst + off;
        const int b = h & (B - 1);
        const int j = h >> LB;
        const int k = ((Ns & (Ns - 1)) == 0) ? (j & (Ns - 1)) : (j % Ns);
        I2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = in[at<LB>(j + r * nR, b)];
        // a radix below 8: doubled first, so the product divides by 2
        v[0] = up_shift(R) ? mk2((v[0].x + 1) >> 1, (v[0].y + 1) >> 1) : quarter(v[0]);
        const Tw *t = tw;
#pragma unroll
        for (int r = 1; r < R; ++r) {
            t += k * twstride;
            if (up_shift(R)) v[r] = add(v[r], v[r]);
            v[r] = cmulw(v[r], *t, INV);
        }
        dft<R, INV>(v);
        const int o = (j - k) * R + k;
#pragma unroll
        for (int r = 0; r < R; ++r) out[at<LB>(o + r * Ns, b)] = v[r];
    }
}
// the complex spectrum C_k = A_k + i B_k of two packed Hermitian lines from
// row k and its partner row n - k: A_k = (lo.x, hi.x), B_k = (lo.y, hi.y),
// lo the row <= n/2
FX_FN I2 join(I2 own, I2 other, int k, int h)
{
    if (k == 0 || k == h) return own;
    return k < h ? mk2(own.x - other.y, other.x + own.y) : mk2(other.x + own.y, other.y - own.x);
}
// the first pass (no twiddles): butterfly (j, b) of v, row j + r n / R
template <int R, bool INV, int LB> FX_FN void first_pass(I2 *v, I2 *dst, int j, int b)
{
    dft<R, INV>(v);
#pragma unroll
    for (int r = 0; r < R; ++r) dst[at<LB>(j * R + r, b)] = v[r];
}

// the passes from Ns = ns on (s: buffer that holds the data, d the other);
// BAR is the block barrier.  Returns the buffer that holds the result.
template <bool INV, int LB, typename BAR>
FX_FN I2 *passes(I2 *s, I2 *d, int n, int nseq, int ns, const Tw *__restrict__ tw, int tws, int tid, int nthreads,
                 BAR bar)
{
    int Ns = ns;
    for (int rem = n / ns; rem > 1;) {
        const int r = next_radix(rem);
        if (r == 8) pass<8, INV, LB>(s, d, n, nseq, Ns, tw, tws, tid, nthreads);
        else if (r == 4) pass<4, INV, LB>(s, d, n, nseq, Ns, tw, tws, tid, nthreads);
        else if (r == 2) pass<2, INV, LB>(s, d, n, nseq, Ns, tw, tws, tid, nthreads);
        else if (r == 3) pass<3, INV, LB>(s, d, n, nseq, Ns, tw, tws, tid, nthreads);
        else pass<5, INV, LB>(s, d, n, nseq, Ns, tw, tws, tid, nthreads);
        bar();
        I2 *t = s;
        s = d;
        d = t;
        Ns *= r;
        rem /= r;
    }
    return s;
}
// A pass in place: thread tid of nthreads reads and transforms all its
// butterflies (at most ceil(R1 / R): there are n B / R1 threads), then, when
// every thread has read, writes them.  nthreads is a multiple of B.
template <int R1, int R, bool INV, int LB> struct PassRegs {
    static constexpr int NB = (R1 + R - 1) / R, B = 1 << LB;
    I2 v[NB][R];
    int o[NB];
    FX_FN void read(const I2 *buf, int n, int Ns, const Tw *__restrict__ tw, int tid, int nthreads)
    {
        const int nR = n / R, nbf = nR << LB, twstride = nR / Ns, b = tid & (B - 1);
#pragma unroll
        for (int q = 0; q < NB; ++q) {
            const int h = tid + q * nthreads;
            o[q] = -1;
            if (h < nbf) {
                const int j = h >> LB;
                const int k = ((Ns & (Ns - 1)) == 0) ? (j & (Ns - 1)) : (j % Ns);
#pragma unroll
                for (int r = 0; r < R; ++r) v[q][r] = buf[at<LB>(j + r * nR, b)];
                // a radix below 8: doubled first, so the product divides by 2
                v[q][0] = up_shift(R) ? mk2((v[q][0].x + 1) >> 1, (v[q][0].y + 1) >> 1) : quarter(v[q][0]);
                const Tw *t = tw;
#pragma unroll
                for (int r = 1; r < R; ++r) {
                    t += k * twstride;
                    if (up_shift(R)) v[q][r] = add(v[q][r], v[q][r]);
                    v[q][r] = cmulw(v[q][r], *t, INV);
                }
                dft<R, INV>(v[q]);
                o[q] = (j - k) * R + k;
            }
        }
    }
    FX_FN void write(I2 *buf, int Ns, int tid) const
    {
#pragma unroll
        for (int q = 0; q < NB; ++q)
            if (o[q] >= 0) {
#pragma unroll
                for (int r = 0; r < R; ++r) buf[at<LB>(o[q] + r * Ns, tid & (B - 1))] = v[q][r];
            }
    }
};
// the passes of a line after its first, of radix R1, in place; run(pass, Ns)
// carries out one (pass: a PassRegs type's empty value)
template <int R1, bool INV, int LB, typename RUN> FX_FN void later_passes(int n, RUN run)
{
    int Ns = R1;
    for (int rem = n / R1; rem > 1;) {
        const int r = next_radix(rem);
        if (R1 == 8 && r == 8) run(PassRegs<R1, 8, INV, LB>(), Ns);
        else if (R1 == 8 && r == 4) run(PassRegs<R1, 4, INV, LB>(), Ns);
        else if (r == 2) run(PassRegs<R1, 2, INV, LB>(), Ns);
        else if (r == 3) run(PassRegs<R1, 3, INV, LB>(), Ns);
        else run(PassRegs<R1, 5, INV, LB>(), Ns);
        Ns *= r;
        rem /= r;
    }
}
// the first pass from shared memory (column sequences)
template <int R, bool INV, int LB>
FX_FN void pass1(const I2 *src, I2 *dst, int n, int nseq, int tid, int nthreads)
{
    const int nR = n / R, nbf = nR << LB;
    for (int g = tid; g < nbf * nseq; g += nthreads) {
        int h = g, off = 0;
        while (h >= nbf) {
            h -= nbf;
            off += n << LB;
        }
        const int b = h & ((1 << LB) - 1), j = h >> LB;
        I2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) v[r] = src[off + at<LB>(j + r * nR, b)];
        first_pass<R, INV, LB>(v, dst + off, j, b);
    }
}
template <bool INV, int LB, typename BAR>
FX_FN I2 *fft(I2 *s, I2 *d, int n, int nseq, const Tw *__restrict__ tw, int tws, int tid, int nthreads, BAR bar)
{
    const int r = next_radix(n);
    if (r == 8) pass1<8, INV, LB>(s, d, n, nseq, tid, nthreads);
    else if (r == 4) pass1<4, INV, LB>(s, d, n, nseq, tid, nthreads);
    else if (r == 2) pass1<2, INV, LB>(s, d, n, nseq, tid, nthreads);
    else if (r == 3) pass1<3, INV, LB>(s, d, n, nseq, tid, nthreads);
    else pass1<5, INV, LB>(s, d, n, nseq, tid, nthreads);
    bar();
    return passes<INV, LB>(d, s, n, nseq, r, tw, tws, tid, nthreads, bar);
}

// ----- column transforms
// The transform of a column's odd (DST) or even (DCT) extension of length
// 2n, n = 2N, for two columns packed as one complex sequence z_0..z_n
// (Z_m = sum over the extension of z_j exp(-i pi j m / n)), from three FFTs
// of length N instead of one of length 4N.  With a sign s = -1 (DST) or +1
// (DCT), u_j = z_j + s z_{n-j}, g_j = z_j - s z_{n-j}, w = exp(-i pi / n):
//   Z_{4k}   = FFT_N(u_j + s u_{N-j})
//   Z_{4k+2} = FFT_N((u_j - s u_{N-j}) w^{2j})
//   Z_{4k+1} = FFT_N((g_j + s i g_{N-j}) w^j),   Z_{2n-m} = s Z_m
// (decimation in frequency of the extension; the values at N + j follow
// from those at N - j).  No division by sines and no running sums, so no
// error of a low index reaches the others.  fold forms the inputs of the
// three FFTs, a quarter each (the factor cmulw brings); W[k] = w^k 2^62.
// Z at (j << LB) + (p ^ sw(j)); sequence q at seq + q (N << LB).
template <bool DCT, int LB>
FX_FN void fold(const I2 *Z, I2 *seq, int N, int p, int j, const Tw *__restrict__ W)
{
    const int n = 2 * N;
    I2 *s0 = seq, *s1 = seq + ((size_t)N << LB), *s2 = s1 + ((size_t)N << LB);
    const int q = at<LB>(j, p);
    if (j == 0) {
        const I2 zN = Z[at<LB>(N, p)];
        if (DCT) {
            const I2 a = Z[q], b = Z[at<LB>(n, p)];
            const I2 u = add(a, b), v = add(zN, zN);
            s0[q] = quarter(add(u, v));
            s1[q] = quarter(sub(u, v));
            s2[q] = quarter(sub(a, b));
        } else {
            s0[q] = s1[q] = mk2(0, 0);
            const I2 v = add(zN, zN);
            s2[q] = quarter(mk2(v.y, -v.x));
        }
        return;
    }
    const int qn = at<LB>(N - j, p);
    const I2 a = Z[q], b = Z[at<LB>(n - j, p)], c = Z[qn], d = Z[at<LB>(N + j, p)];
    const I2 ap = add(a, b), am = sub(a, b), cp = add(c, d), cm = sub(c, d);
    if (DCT) {
        const I2 e0 = quarter(add(ap, cp)), e1 = sub(ap, cp);
        s0[q] = e0;
        s0[qn] = e0;
        s1[q] = cmulw(e1, W[2 * j], false);
        s1[qn] = cmulw(mk2(-e1.x, -e1.y), W[2 * (N - j)], false);
        s2[q] = cmulw(mk2(am.x - cm.y, am.y + cm.x), W[j], false);
        s2[qn] = cmulw(mk2(cm.x - am.y, cm.y + am.x), W[N - j], false);
    } else {
        const I2 e0 = quarter(sub(am, cm)), e1 = add(am, cm);
        s0[q] = e0;
        s0[qn] = mk2(-e0.x, -e0.y);
        s1[q] = cmulw(e1, W[2 * j], false);
        s1[qn] = cmulw(e1, W[2 * (N - j)], false);
        s2[q] = cmulw(mk2(ap.x + cp.y, ap.y - cp.x), W[j], false);
        s2[qn] = cmulw(mk2(cp.x + ap.y, cp.y - ap.x), W[N - j], false);
    }
}
// where Z_m (0 <= m <= n) lies in the transformed sequences: index into the
// sequences' buffer; *neg where the symmetry changes its sign
template <bool DCT, int LB> FX_FN int unfold(int m, int N, int p, bool *neg)
{
    const int r = m & 3;
    *neg = !DCT && r == 3;
    const int k = r == 3 ? (4 * N - m - 1) >> 2 : m >> 2;
    const int s = r == 0 ? 0 : r == 2 ? 1 : 2;
    return ((s * N) << LB) + at<LB>(k, p);
}

}  // namespace fx
}  // namespace ps3d
