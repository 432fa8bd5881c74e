// Host build of the FP64 Stockham transforms (ps3d_gb300/csrc/common.cuh) in
// the layout of k_lines and k_columns (transforms.cu), one sequence pair at a
// time and one thread: what the fixed-point transforms' error is held against.
#include <math.h>

#include <utility>
#include <vector>

#include <cuda_runtime.h>

// the twiddle product as the device rounds it (found by argument-dependent
// lookup before the template of common.cuh)
inline double2 cmul(double2 a, double2 b)
{
    return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
// what common.cuh takes from the device
static struct { int x; } threadIdx{0}, blockDim{1};
static inline void __syncthreads() {}
long long __double_as_longlong(double);
double __longlong_as_double(long long);
float __uint_as_float(unsigned);
unsigned __float_as_uint(float);
#include "common.cuh"

using ps3d::smem_fft;
using std::vector;

static vector<double2> table(int n)
{
    vector<double2> t(n);
    const long double pi = acosl(-1.0L);
    for (int k = 0; k < n; ++k) t[k] = make_double2((double)cosl(2 * pi * k / n), (double)-sinl(2 * pi * k / n));
    return t;
}

extern "C" void fp64_line(int n, int inverse, int, const double *a, const double *b, double *oa, double *ob)
{
    const vector<double2> tw = table(n);
    vector<double2> b0(n), b1(n);
    const int h = n / 2;
    const double s = 1.0 / sqrt((double)n);
    if (inverse) {
        for (int k = 0; k <= h; ++k) {
            const bool two = k > 0 && k < h;
            const double ha = two ? a[n - k] : 0.0, hb = two ? b[n - k] : 0.0;
            b0[k] = make_double2(a[k] - hb, ha + b[k]);
            if (two) b0[n - k] = make_double2(a[k] + hb, b[k] - ha);
        }
        const double2 *r = smem_fft<true>(b0.data(), b1.data(), n, 0, tw.data());
        for (int i = 0; i < n; ++i) {
            oa[i] = r[i].x * s;
            ob[i] = r[i].y * s;
        }
        return;
    }
    for (int i = 0; i < n; ++i) b0[i] = make_double2(a[i], b[i]);
    const double2 *r = smem_fft<false>(b0.data(), b1.data(), n, 0, tw.data());
    for (int k = 0; k <= h; ++k) {
        const double2 c = r[k], d = r[k ? n - k : 0];
        oa[k] = 0.5 * (c.x + d.x) * s;
        ob[k] = 0.5 * (c.y + d.y) * s;
        if (k > 0 && k < h) {
            oa[n - k] = 0.5 * (c.y - d.y) * s;
            ob[n - k] = -0.5 * (c.x - d.x) * s;
        }
    }
}

// plain dst (rows 1..nz-1) or dct (rows 0..nz)
extern "C" void fp64_column(int nz, int dct, int, const double *a, const double *b, double *oa, double *ob)
{
    const int L = 2 * nz;
    const vector<double2> tw = table(L);
    vector<double2> b0(L), b1(L);
    for (int j = 0; j <= nz; ++j) {
        const bool end = j == 0 || j == nz;
        b0[j] = end && !dct ? make_double2(0.0, 0.0) : make_double2(a[j], b[j]);
        if (!end) b0[L - j] = dct ? b0[j] : make_double2(-a[j], -b[j]);
    }
    const double2 *r = smem_fft<false>(b0.data(), b1.data(), L, 0, tw.data());
    const double s = 1.0 / sqrt(2.0 * (double)nz);
    for (int j = 0; j <= nz; ++j) {
        oa[j] = (dct ? r[j].x : -r[j].y) * s;
        ob[j] = (dct ? r[j].y : r[j].x) * s;
    }
}
