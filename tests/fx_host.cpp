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

// lines a, b of length n (n_even), in the layout of `lanes` = 2^logB lanes
// with the pair in every lane
extern "C" void fx_line(int n, int inverse, int logB, const double *a, const double *b, double *oa, double *ob)
{
    const Plan pl = line_plan(n, inverse != 0);
    const vector<Tw> tw = table(n);
    vector<I2> b0((size_t)n << logB), b1(b0.size());
    const unsigned ma = top(a, n), mb = top(b, n);
    const int ea = line_exp(ma), eb = line_exp(mb), h = n / 2;
    const int Ea = bits_of(a, n, ma, pl), Eb = bits_of(b, n, mb, pl);
    for (int p = 0; p < 1 << logB; ++p)
        for (int k = 0; k < n; ++k) {
            I2 v = mk2(to_fixed(a[k], ea, Ea), to_fixed(b[k], eb, Eb));
            if (inverse && k > 0 && k != h) {
                const int kn = n - k;
                const I2 u = mk2(to_fixed(a[kn], ea, Ea), to_fixed(b[kn], eb, Eb));
                v = k < h ? mk2(v.x - u.y, u.x + v.y) : mk2(u.x + v.y, u.y - v.x);
            }
            b0[at(k, p, logB)] = v;
        }
    auto nobar = [] {};
    const I2 *r = inverse ? fft<true>(b0.data(), b1.data(), n, logB, 1, tw.data(), 1, 0, 1, nobar)
                          : fft<false>(b0.data(), b1.data(), n, logB, 1, tw.data(), 1, 0, 1, nobar);
    const Scale sa = scale_of(ma, Ea, pl), sb = scale_of(mb, Eb, pl);
    const int p = (1 << logB) - 1;
    for (int k = 0; k < n; ++k) {
        const I2 ck = r[at(k, p, logB)];
        if (inverse) {
            oa[k] = to_double(ck.x, sa);
            ob[k] = to_double(ck.y, sb);
        } else if (k <= h) {
            const I2 cn = r[at(k == 0 ? 0 : n - k, p, logB)];
            oa[k] = to_double(ck.x + cn.x, sa);
            ob[k] = to_double(ck.y + cn.y, sb);
            if (k > 0 && k < h) {
                oa[n - k] = to_double(ck.y - cn.y, sa);
                ob[n - k] = to_double(cn.x - ck.x, sb);
            }
        }
    }
}

// plain dst (rows 1..nz-1) or dct (rows 0..nz) of columns a, b
extern "C" void fx_column(int nz, int dct, int logB, const double *a, const double *b, double *oa, double *ob)
{
    const Plan pl = col_plan(nz);
    const vector<Tw> W = table(2 * nz);
    const int N = nz / 2;
    vector<I2> Z((size_t)(nz + 1) << logB), seq((size_t)3 * N << logB), seq2(seq.size());
    const int lo = dct ? 0 : 1, cnt = dct ? nz + 1 : nz - 1;
    const unsigned ma = top(a + lo, cnt), mb = top(b + lo, cnt);
    const int ea = line_exp(ma), eb = line_exp(mb);
    const int Ea = bits_of(a + lo, cnt, ma, pl), Eb = bits_of(b + lo, cnt, mb, pl);
    for (int p = 0; p < 1 << logB; ++p) {
        for (int j = 0; j <= nz; ++j)
            Z[at(j, p, logB)] = (!dct && (j == 0 || j == nz)) ? mk2(0, 0)
                                                              : mk2(to_fixed(a[j], ea, Ea), to_fixed(b[j], eb, Eb));
        for (int j = 0; j <= N / 2; ++j) {
            if (dct) fold<true>(Z.data(), seq.data(), N, logB, p, j, W.data());
            else fold<false>(Z.data(), seq.data(), N, logB, p, j, W.data());
        }
    }
    const I2 *r = fft<false>(seq.data(), seq2.data(), N, logB, 3, W.data(), 4, 0, 1, [] {});
    const Scale sa = scale_of(ma, Ea, pl), sb = scale_of(mb, Eb, pl);
    const int p = (1 << logB) - 1;
    for (int m = 0; m <= nz; ++m) {
        bool neg;
        const I2 c = r[dct ? unfold<true>(m, N, logB, p, &neg) : unfold<false>(m, N, logB, p, &neg)];
        long long x = dct ? c.x : -c.y, y = dct ? c.y : c.x;
        if (neg) {
            x = -x;
            y = -y;
        }
        oa[m] = to_double(x, sa);
        ob[m] = to_double(y, sb);
    }
}
