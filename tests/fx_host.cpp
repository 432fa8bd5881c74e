// Host build of the fixed-point transforms (ps3d_gb300/csrc/fx.cuh): the
// same conversion, passes, folds and scales as the device kernels, one
// sequence pair at a time.
#include <math.h>

#include <vector>

#include "fx.cuh"

using namespace ps3d::fx;
using std::vector;

static vector<Tw> table(int n)
{
    vector<Tw> t(n);
    fill_twiddles(t.data(), n);
    return t;
}
static unsigned top(const double *a, int n)
{
    unsigned m = 0;
    for (int i = 0; i < n; ++i) m = mag(a[i]) > m ? mag(a[i]) : m;
    return m;
}
static int bits_of(const double *a, int n, unsigned m, const Plan &pl)
{
    float s = 0.0f;
    for (int i = 0; i < n; ++i) s += magf(mag(a[i]));
    return pl.E[spread(s, m, pl.lcap)];
}

// lines a, b of length n (n even), the pair in every one of 2^LB lanes; the
// first pass on values in hand, as the kernel's threads hold them
template <int R, int LB>
static void line(int n, int inverse, const double *a, const double *b, double *oa, double *ob)
{
    const Plan pl = line_plan(n, inverse != 0);
    const vector<Tw> tw = table(n);
    vector<I2> b0((size_t)n << LB);
    const unsigned ma = top(a, n), mb = top(b, n);
    const int ea = line_exp(ma), eb = line_exp(mb), h = n / 2;
    const int Ea = bits_of(a, n, ma, pl), Eb = bits_of(b, n, mb, pl);
    for (int p = 0; p < 1 << LB; ++p)
        for (int j = 0; j < n / R; ++j) {
            I2 v[R];
            for (int r = 0; r < R; ++r) {
                const int k = j + r * (n / R), kn = k ? n - k : 0;
                v[r] = mk2(to_fixed(a[k], ea, Ea), to_fixed(b[k], eb, Eb));
                if (inverse) v[r] = join(v[r], mk2(to_fixed(a[kn], ea, Ea), to_fixed(b[kn], eb, Eb)), k, h);
            }
            if (inverse) first_pass<R, true, LB>(v, b0.data(), j, p);
            else first_pass<R, false, LB>(v, b0.data(), j, p);
        }
    // the later passes in place, all threads of a block reading before any writes
    const int nt = (((n / R) << LB) + 31) / 32 * 32;
    const auto run = [&](auto pass, int Ns) {
        vector<decltype(pass)> regs(nt);
        for (int t = 0; t < nt; ++t) regs[t].read(b0.data(), n, Ns, tw.data(), t, nt);
        for (int t = 0; t < nt; ++t) regs[t].write(b0.data(), Ns, t);
    };
    if (inverse) later_passes<R, true, LB>(n, run);
    else later_passes<R, false, LB>(n, run);
    const I2 *q = b0.data();
    const Scale sa = scale_of(ma, Ea, pl), sb = scale_of(mb, Eb, pl);
    const int p = (1 << LB) - 1;
    for (int k = 0; k < n; ++k) {
        const I2 ck = q[at<LB>(k, p)];
        if (inverse) {
            oa[k] = to_double(ck.x, sa);
            ob[k] = to_double(ck.y, sb);
        } else if (k <= h) {
            const I2 cn = q[at<LB>(k == 0 ? 0 : n - k, p)];
            oa[k] = to_double(ck.x + cn.x, sa);
            ob[k] = to_double(ck.y + cn.y, sb);
            if (k > 0 && k < h) {
                oa[n - k] = to_double(ck.y - cn.y, sa);
                ob[n - k] = to_double(cn.x - ck.x, sb);
            }
        }
    }
}
extern "C" void fx_line(int n, int inverse, int, const double *a, const double *b, double *oa, double *ob)
{
    const int r = first_radix(n);
    if (r == 8) line<8, 2>(n, inverse, a, b, oa, ob);
    else if (r == 4) line<4, 2>(n, inverse, a, b, oa, ob);
    else if (r == 5) line<5, 2>(n, inverse, a, b, oa, ob);
    else line<3, 1>(n, inverse, a, b, oa, ob);
}

// plain dst (rows 1..nz-1) or dct (rows 0..nz) of columns a, b
template <bool DCT, int LB>
static void column(int nz, const double *a, const double *b, double *oa, double *ob)
{
    const Plan pl = col_plan(nz);
    const vector<Tw> W = table(2 * nz);
    const int N = nz / 2;
    vector<I2> Z((size_t)(nz + 1) << LB), seq((size_t)3 * N << LB), seq2(seq.size());
    const int lo = DCT ? 0 : 1, cnt = DCT ? nz + 1 : nz - 1;
    const unsigned ma = top(a + lo, cnt), mb = top(b + lo, cnt);
    const int ea = line_exp(ma), eb = line_exp(mb);
    const int Ea = bits_of(a + lo, cnt, ma, pl), Eb = bits_of(b + lo, cnt, mb, pl);
    for (int p = 0; p < 1 << LB; ++p) {
        for (int j = 0; j <= nz; ++j)
            Z[at<LB>(j, p)] = (!DCT && (j == 0 || j == nz)) ? mk2(0, 0)
                                                            : mk2(to_fixed(a[j], ea, Ea), to_fixed(b[j], eb, Eb));
        for (int j = 0; j <= N / 2; ++j) fold<DCT, LB>(Z.data(), seq.data(), N, p, j, W.data());
    }
    const I2 *r = fft<false, LB>(seq.data(), seq2.data(), N, 3, W.data(), 4, 0, 1, [] {});
    const Scale sa = scale_of(ma, Ea, pl), sb = scale_of(mb, Eb, pl);
    const int p = (1 << LB) - 1;
    for (int m = 0; m <= nz; ++m) {
        bool neg;
        const I2 c = r[unfold<DCT, LB>(m, N, p, &neg)];
        long long x = DCT ? c.x : -c.y, y = DCT ? c.y : c.x;
        if (neg) {
            x = -x;
            y = -y;
        }
        oa[m] = to_double(x, sa);
        ob[m] = to_double(y, sb);
    }
}
extern "C" void fx_column(int nz, int dct, int wide, const double *a, const double *b, double *oa, double *ob)
{
    if (dct) wide ? column<true, 3>(nz, a, b, oa, ob) : column<true, 2>(nz, a, b, oa, ob);
    else wide ? column<false, 3>(nz, a, b, oa, ob) : column<false, 2>(nz, a, b, oa, ob);
}
