// FP64 column transforms on the integer pipes (fx.cuh): dst / dct along z of
// src/fft/stafft.f90:410-550, with the harmonic parts of
// field_decompose_semi_spectral / field_combine_semi_spectral
// (inversion_utils.f90:563-647) in FP64, and the column work of vor2vel and
// source fused around them.
//
// A block of 8 warps owns 2B columns, B = 2^LB packed pairs; G = 8 / B warps
// share a pair, lanes along z (coalesced).  Both columns' values stay in
// registers (NIT levels each per lane) until their scales are known, go to
// shared memory as one 16-byte complex value per level (no bank conflicts:
// 8-byte halves of it took twice the wavefronts), are folded into the three
// half-length sequences and transformed by the whole block, and come back
// the same way.  Two buffers of 3 nz / 2 complex values per pair alternate.
//
// Integer issue bounds all of them (about 300 M warp instructions for two
// fields at 256^3).  256^3, us: combine 255 -> 215 per field; combine, z
// difference and decomposition of one component 647 (three kernels) -> 456;
// w and dw/dz 823 (five kernels) -> 708; the three tendency components 915
// (assembly and decomposition) -> 774.
#include "kernels.h"

#include "fx.cuh"

namespace ps3d {

using fx::I2;
using fx::Tw;

template <int LB> struct ColState {
    unsigned mag[2 << LB];
    int bits[2 << LB];
    unsigned pm[8][2];  // per warp, where two warps share a pair
    float ps[8][2];
};

// the pair and levels of a thread: level(i) = lane + 32 (i G + part)
template <int NIT, int LB> struct ColThread {
    static constexpr int B = 1 << LB, G = 8 / B;
    int lane, warp, p, part;
    long long col;  // first column of the pair
    bool on;
    __device__ ColThread(long long ncol)
    {
        lane = threadIdx.x & 31;
        warp = threadIdx.x >> 5;
        p = warp & (B - 1);
        part = warp >> LB;
        col = ((long long)blockIdx.x * B + p) * 2;
        on = col < ncol;  // ncol is even
    }
    __device__ int level(int i) const { return lane + 32 * (i * G + part); }
};

// values a, b of the pair's levels 1..nz-1 (0 elsewhere; levels 0 and nz too
// where ends is set: za, zb hold level nz, on the lane that has level 0)
// to fixed point in Z
template <int NIT, int LB>
__device__ __forceinline__ void col_stage(I2 *Z, ColState<LB> &sh, const ColThread<NIT, LB> &t, int nz,
                                          const fx::Plan &pl, const double (&a)[NIT], const double (&b)[NIT],
                                          bool ends = false, double za = 0.0, double zb = 0.0)
{
    unsigned ma = fx::mag(za), mb = fx::mag(zb);
    float ta = fx::magf(ma), tb = fx::magf(mb);
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const unsigned xa = fx::mag(a[i]), xb = fx::mag(b[i]);
        ma = max(ma, xa);
        mb = max(mb, xb);
        ta += fx::magf(xa);
        tb += fx::magf(xb);
    }
    ma = __reduce_max_sync(0xffffffffu, ma);
    mb = __reduce_max_sync(0xffffffffu, mb);
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) {
        ta += __shfl_xor_sync(0xffffffffu, ta, q);
        tb += __shfl_xor_sync(0xffffffffu, tb, q);
    }
    if (t.G == 2) {
        if (t.lane == 0) {
            sh.pm[t.warp][0] = ma;
            sh.pm[t.warp][1] = mb;
            sh.ps[t.warp][0] = ta;
            sh.ps[t.warp][1] = tb;
        }
        __syncthreads();
        const int w = t.warp & (t.B - 1), v = w + t.B;  // both warps sum in the same order
        ma = max(sh.pm[w][0], sh.pm[v][0]);
        mb = max(sh.pm[w][1], sh.pm[v][1]);
        ta = sh.ps[w][0] + sh.ps[v][0];
        tb = sh.ps[w][1] + sh.ps[v][1];
    }
    const int Ea = pl.E[fx::spread(ta, ma, pl.lcap)], Eb = pl.E[fx::spread(tb, mb, pl.lcap)];
    const int ea = fx::line_exp(ma), eb = fx::line_exp(mb);
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        if (iz < nz) Z[fx::at<LB>(iz, t.p)] = fx::mk2(fx::to_fixed(a[i], ea, Ea), fx::to_fixed(b[i], eb, Eb));
    }
    if (ends && t.lane == 0 && t.part == 0)
        Z[fx::at<LB>(nz, t.p)] = fx::mk2(fx::to_fixed(za, ea, Ea), fx::to_fixed(zb, eb, Eb));
    if (t.lane == 0 && t.part == 0) {
        sh.mag[2 * t.p] = ma;
        sh.mag[2 * t.p + 1] = mb;
        sh.bits[2 * t.p] = Ea;
        sh.bits[2 * t.p + 1] = Eb;
    }
}

// fold Z into seq and transform; returns the buffer with the result, *other
// the free one (after its last reader's barrier)
template <bool DCT, int LB>
__device__ __forceinline__ const I2 *col_transform(I2 *Z, I2 *seq, int nz, const Tw *__restrict__ W, I2 **other)
{
    const int N = nz / 2;
    __syncthreads();
    for (int g = threadIdx.x; g < (N / 2 + 1) << LB; g += 256)
        fx::fold<DCT, LB>(Z, seq, N, g & ((1 << LB) - 1), g >> LB, W);
    __syncthreads();
    I2 *res = fx::fft<false, LB>(seq, Z, N, 3, W, 4, threadIdx.x, 256, [] { __syncthreads(); });
    *other = res == seq ? Z : seq;
    return res;
}

// f(level, a, b, i) for the transformed values of the thread's levels below
// nz, and with last set, level nz on the lane that has level 0 (i = NIT)
template <bool DCT, int NIT, int LB, typename F>
__device__ __forceinline__ void col_values(const I2 *res, const ColState<LB> &sh, const ColThread<NIT, LB> &t, int nz,
                                           const fx::Plan &pl, bool last, F f)
{
    const fx::Scale sa = fx::scale_of(sh.mag[2 * t.p], sh.bits[2 * t.p], pl),
                    sb = fx::scale_of(sh.mag[2 * t.p + 1], sh.bits[2 * t.p + 1], pl);
    const auto one = [&](int iz, int i) {
        bool neg;
        const I2 c = res[fx::unfold<DCT, LB>(iz, nz / 2, t.p, &neg)];
        // the dst is -Im Z of the first column and, i times it being the
        // packed second one, Re Z
        const long long x = DCT ? c.x : neg ? c.y : -c.y, y = DCT ? c.y : neg ? -c.x : c.x;
        f(iz, fx::to_double(x, sa), fx::to_double(y, sb), i);
    };
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        if (iz < nz) one(iz, i);
    }
    if (last && t.lane == 0 && t.part == 0) one(nz, NIT);
}

#define COL_SHARED                                             \
    extern __shared__ __align__(16) unsigned char smem_raw[];  \
    __shared__ ColState<LB> sh;                                \
    I2 *buf0 = reinterpret_cast<I2 *>(smem_raw);               \
    I2 *buf1 = buf0 + ((3 * (nz / 2)) << LB); /* 3 nz / 2 >= nz + 1 */ \
    const ColThread<NIT, LB> t(ncol);                          \
    I2 *other;

// the modes of columns() (kernels.h)
template <int MODE, int NIT, int LB>
__global__ void __launch_bounds__(256) k_fx_columns(const double *in, double *out, int nz,
                                                    int P, long long ncol, long long fs,
                                                    const double *__restrict__ phim, const double *__restrict__ phip,
                                                    const __grid_constant__ fx::Plan pl, const Tw *__restrict__ W)
{
    constexpr bool DCT = MODE == COL_DCT;
    COL_SHARED
    const long long oa = t.col * P, ob = oa + P;
    in += blockIdx.y * fs;
    out += blockIdx.y * fs;
    double fa = 0.0, fb = 0.0, ga = 0.0, gb = 0.0;  // levels 0 and nz
    if (t.on) {
        fa = in[oa];
        fb = in[ob];
        ga = in[oa + nz];
        gb = in[ob + nz];
    }
    double a[NIT], b[NIT];
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        a[i] = b[i] = 0.0;
        if (t.on && iz < nz && (DCT || iz > 0)) {
            a[i] = in[oa + iz];
            b[i] = in[ob + iz];
            if (MODE == COL_DECOMP) {
                a[i] = a[i] - (fa * phim[oa + iz] + ga * phip[oa + iz]);
                b[i] = b[i] - (fb * phim[ob + iz] + gb * phip[ob + iz]);
            }
        }
    }
    col_stage<NIT, LB>(buf1, sh, t, nz, pl, a, b, DCT, DCT && t.lane == 0 && t.part == 0 ? ga : 0.0,
                       DCT && t.lane == 0 && t.part == 0 ? gb : 0.0);
    const I2 *res = col_transform<DCT, LB>(buf1, buf0, nz, W, &other);
    if (!t.on) return;
    col_values<DCT, NIT, LB>(res, sh, t, nz, pl, DCT, [&](int iz, double x, double y, int) {
        if (MODE == COL_COMBINE) {
            x = x + fa * phim[oa + iz] + ga * phip[oa + iz];
            y = y + fb * phim[ob + iz] + gb * phip[ob + iz];
        }
        if (!DCT && iz == 0) {
            x = fa;
            y = fb;
        }
        out[oa + iz] = x;
        out[ob + iz] = y;
    });
    if (!DCT && t.lane == 0 && t.part == 0) {
        out[oa + nz] = MODE == COL_DST ? 0.0 : ga;
        out[ob + nz] = MODE == COL_DST ? 0.0 : gb;
    }
}

// cs = combine(c), es = decompose(central_diffz(cs)) (inversion.f90:41-47):
// the combined column stays on chip for its difference
template <int NIT, int LB>
__global__ void __launch_bounds__(256) k_fx_comdec(const double *__restrict__ c, double *__restrict__ cs,
                                                   double *__restrict__ es, int nz, int P, long long ncol, double dzi,
                                                   const double *__restrict__ phim, const double *__restrict__ phip,
                                                   const __grid_constant__ fx::Plan pl, const Tw *__restrict__ W)
{
    COL_SHARED
    const long long oa = t.col * P, ob = oa + P;
    double fa = 0.0, fb = 0.0, ga = 0.0, gb = 0.0;
    if (t.on) {
        fa = c[oa];
        fb = c[ob];
        ga = c[oa + nz];
        gb = c[ob + nz];
    }
    double a[NIT], b[NIT];
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        const bool in = t.on && iz > 0 && iz < nz;
        a[i] = in ? c[oa + iz] : 0.0;
        b[i] = in ? c[ob + iz] : 0.0;
    }
    col_stage<NIT, LB>(buf1, sh, t, nz, pl, a, b);
    I2 *res = const_cast<I2 *>(col_transform<false, LB>(buf1, buf0, nz, W, &other));
    double2 *raw = reinterpret_cast<double2 *>(other);
    col_values<false, NIT, LB>(res, sh, t, nz, pl, false, [&](int iz, double x, double y, int) {
        if (t.on) {
            x = x + fa * phim[oa + iz] + ga * phip[oa + iz];
            y = y + fb * phim[ob + iz] + gb * phip[ob + iz];
        }
        if (iz == 0) {
            x = fa;
            y = fb;
        }
        raw[fx::at<LB>(iz, t.p)] = make_double2(x, y);
        if (t.on) {
            cs[oa + iz] = x;
            cs[ob + iz] = y;
        }
    });
    if (t.lane == 0 && t.part == 0) {
        raw[fx::at<LB>(nz, t.p)] = make_double2(ga, gb);
        if (t.on) {
            cs[oa + nz] = ga;
            cs[ob + nz] = gb;
        }
    }
    __syncthreads();
    // central_diffz (inversion_utils.f90:653-673)
    const double hdzi = 0.5 * dzi;
    const auto at = [&](int iz) { return raw[fx::at<LB>(iz, t.p)]; };
    const double2 r0 = at(0), r1 = at(1), rm = at(nz - 1), rn = at(nz);
    const double ea0 = dzi * (r1.x - r0.x), eb0 = dzi * (r1.y - r0.y), ean = dzi * (rn.x - rm.x),
                 ebn = dzi * (rn.y - rm.y);
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        a[i] = b[i] = 0.0;
        if (t.on && iz > 0 && iz < nz) {
            const double2 lo = at(iz - 1), hi = at(iz + 1);
            a[i] = (hi.x - lo.x) * hdzi - (ea0 * phim[oa + iz] + ean * phip[oa + iz]);
            b[i] = (hi.y - lo.y) * hdzi - (eb0 * phim[ob + iz] + ebn * phip[ob + iz]);
        }
    }
    col_stage<NIT, LB>(res, sh, t, nz, pl, a, b);
    const I2 *res2 = col_transform<false, LB>(res, other, nz, W, &other);
    if (!t.on) return;
    col_values<false, NIT, LB>(res2, sh, t, nz, pl, false, [&](int iz, double x, double y, int) {
        es[oa + iz] = iz == 0 ? ea0 : x;
        es[ob + iz] = iz == 0 ? eb0 : y;
    });
    if (t.lane == 0 && t.part == 0) {
        es[oa + nz] = ean;
        es[ob + nz] = ebn;
    }
}

// the vertical velocity of vor2vel (inversion.f90:86-139) from the state
// components A, B: ds = D_y A - D_x B, g = green ds,
// w = [0, dst(g) + ds_0 thetam + ds_nz thetap, 0],
// es = dw/dz = dct(rkz g) + ds_0 dthetam + ds_nz dthetap.
// ds is formed from the partner columns and stays on chip.
struct WTables {
    const double *thetam, *thetap, *dthetam, *dthetap, *green, *rkz;
};
template <int NIT, int LB>
__global__ void __launch_bounds__(256, 3) k_fx_w(const double *__restrict__ A, const double *__restrict__ Bc,
                                              double *__restrict__ w, double *__restrict__ es, int nx, int ny, int nz,
                                              int P, long long ncol, Deriv D, WTables tb,
                                              const __grid_constant__ fx::Plan pl, const Tw *__restrict__ W)
{
    COL_SHARED
    const long long oa = t.col * P, ob = oa + P;
    long long xa = 0, ya = 0, xb = 0, yb = 0;  // partner columns
    double cxa = 0.0, cya = 0.0, cxb = 0.0, cyb = 0.0;
    if (t.on) {
        const auto partners = [&](long long col, long long &x, long long &y, double &cx, double &cy) {
            const int kx = (int)(col / ny), ky = (int)(col - (long long)kx * ny);
            x = ((long long)(kx ? nx - kx : 0) * ny + ky) * P;
            y = ((long long)kx * ny + (ky ? ny - ky : 0)) * P;
            cx = D.cx[kx];
            cy = D.cy[ky];
        };
        partners(t.col, xa, ya, cxa, cya);
        partners(t.col + 1, xb, yb, cxb, cyb);
    }
    const auto dsa = [&](int iz) { return cya * A[ya + iz] - cxa * Bc[xa + iz]; };
    const auto dsb = [&](int iz) { return cyb * A[yb + iz] - cxb * Bc[xb + iz]; };
    double fa = 0.0, fb = 0.0, ga = 0.0, gb = 0.0;
    if (t.on) {
        fa = dsa(0);
        fb = dsb(0);
        ga = dsa(nz);
        gb = dsb(nz);
    }
    double a[NIT], b[NIT];
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        const bool in = t.on && iz > 0 && iz < nz;
        a[i] = in ? tb.green[oa + iz] * dsa(iz) : 0.0;
        b[i] = in ? tb.green[ob + iz] * dsb(iz) : 0.0;
    }
    col_stage<NIT, LB>(buf1, sh, t, nz, pl, a, b);
    I2 *res = const_cast<I2 *>(col_transform<false, LB>(buf1, buf0, nz, W, &other));
    if (t.on) {
        col_values<false, NIT, LB>(res, sh, t, nz, pl, false, [&](int iz, double x, double y, int) {
            w[oa + iz] = iz ? x + (fa * tb.thetam[oa + iz] + ga * tb.thetap[oa + iz]) : 0.0;
            w[ob + iz] = iz ? y + (fb * tb.thetam[ob + iz] + gb * tb.thetap[ob + iz]) : 0.0;
        });
        if (t.lane == 0 && t.part == 0) w[oa + nz] = w[ob + nz] = 0.0;
    }
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        const double k = iz < nz ? tb.rkz[iz] : 0.0;
        a[i] *= k;
        b[i] *= k;
    }
    __syncthreads();  // every pair has read its first result (and its scale)
    col_stage<NIT, LB>(res, sh, t, nz, pl, a, b, true);
    const I2 *res2 = col_transform<true, LB>(res, other, nz, W, &other);
    if (!t.on) return;
    col_values<true, NIT, LB>(res2, sh, t, nz, pl, true, [&](int iz, double x, double y, int) {
        es[oa + iz] = (fa * tb.dthetam[oa + iz] + ga * tb.dthetap[oa + iz]) + x;
        es[ob + iz] = (fb * tb.dthetam[ob + iz] + gb * tb.dthetap[ob + iz]) + y;
    });
}

// the tendency components (inversion.f90:341-367) formed from the
// transformed products (fs apart: r, q, p, dq/dz, dp/dz) and decomposed;
// component blockIdx.y of D_y r - dq/dz, dp/dz - D_x r, D_x q - D_y p
template <int NIT, int LB>
__global__ void __launch_bounds__(256) k_fx_src(const double *__restrict__ f, double *__restrict__ out, int nx, int ny,
                                                int nz, int P, long long ncol, long long fs, Deriv D,
                                                const double *__restrict__ phim, const double *__restrict__ phip,
                                                const __grid_constant__ fx::Plan pl, const Tw *__restrict__ W)
{
    COL_SHARED
    const long long oa = t.col * P, ob = oa + P;
    const int k = blockIdx.y;
    out += k * fs;
    // value = u c1 - v c2, u and v from these columns
    const double *ua = f, *va = f, *ub = f, *vb = f;
    double c1a = 0.0, c2a = 0.0, c1b = 0.0, c2b = 0.0;
    if (t.on) {
        const auto set = [&](long long col, const double *&u, const double *&v, double &c1, double &c2) {
            const int kx = (int)(col / ny), ky = (int)(col - (long long)kx * ny);
            const long long o = col * P, ox = ((long long)(kx ? nx - kx : 0) * ny + ky) * P,
                            oy = ((long long)kx * ny + (ky ? ny - ky : 0)) * P;
            if (k == 0) {
                u = f + oy;
                c1 = D.cy[ky];
                v = f + 3 * fs + o;
                c2 = 1.0;
            } else if (k == 1) {
                u = f + 4 * fs + o;
                c1 = 1.0;
                v = f + ox;
                c2 = D.cx[kx];
            } else {
                u = f + fs + ox;
                c1 = D.cx[kx];
                v = f + 2 * fs + oy;
                c2 = D.cy[ky];
            }
        };
        set(t.col, ua, va, c1a, c2a);
        set(t.col + 1, ub, vb, c1b, c2b);
    }
    const auto sa = [&](int iz) { return c1a * ua[iz] - c2a * va[iz]; };
    const auto sb = [&](int iz) { return c1b * ub[iz] - c2b * vb[iz]; };
    double fa = 0.0, fb = 0.0, ga = 0.0, gb = 0.0;
    if (t.on) {
        fa = sa(0);
        fb = sb(0);
        ga = sa(nz);
        gb = sb(nz);
    }
    double a[NIT], b[NIT];
#pragma unroll
    for (int i = 0; i < NIT; ++i) {
        const int iz = t.level(i);
        a[i] = b[i] = 0.0;
        if (t.on && iz > 0 && iz < nz) {
            a[i] = sa(iz) - (fa * phim[oa + iz] + ga * phip[oa + iz]);
            b[i] = sb(iz) - (fb * phim[ob + iz] + gb * phip[ob + iz]);
        }
    }
    col_stage<NIT, LB>(buf1, sh, t, nz, pl, a, b);
    const I2 *res = col_transform<false, LB>(buf1, buf0, nz, W, &other);
    if (!t.on) return;
    col_values<false, NIT, LB>(res, sh, t, nz, pl, false, [&](int iz, double x, double y, int) {
        out[oa + iz] = iz ? x : fa;
        out[ob + iz] = iz ? y : fb;
    });
    if (t.lane == 0 && t.part == 0) {
        out[oa + nz] = ga;
        out[ob + nz] = gb;
    }
}

// levels per lane and pairs per block of a column length: 8 pairs (one warp
// each) up to 128 levels, 4 pairs of two warps above (48 nz bytes of shared
// memory per pair: four blocks per SM up to 256) and where 8 pairs would make
// fewer than two blocks per SM (32^3: w and dw/dz 18.7 us with 8 pairs, 17.0
// with 4)
template <typename F> static void col_shape(int nz, long long ncol, F f)
{
    using std::integral_constant;
    const bool few = ncol < 2 * 152 * 16;
    if (nz <= 64 && few) f(integral_constant<int, 1>(), integral_constant<int, 2>());
    else if (nz <= 64) f(integral_constant<int, 2>(), integral_constant<int, 3>());
    else if (nz <= 128 && few) f(integral_constant<int, 2>(), integral_constant<int, 2>());
    else if (nz <= 128) f(integral_constant<int, 4>(), integral_constant<int, 3>());
    else if (nz <= 256) f(integral_constant<int, 4>(), integral_constant<int, 2>());
    else f(integral_constant<int, 8>(), integral_constant<int, 2>());
}
static dim3 col_grid(const Dims &d, int LB, int nf)
{
    return dim3((unsigned)((d.ncol + (2 << LB) - 1) / (2 << LB)), (unsigned)nf);
}

void fx_columns(const Dims &d, cudaStream_t st, int mode, const double *in, double *out, const double *phim,
                const double *phip, const void *tw, int nf)
{
    const Tw *W = reinterpret_cast<const Tw *>(tw);
    const fx::Plan pl = fx::col_plan(d.nz);
    col_shape(d.nz, d.ncol, [&](auto nit, auto lb) {
        constexpr int NIT = decltype(nit)::value, LB = decltype(lb)::value;
        const auto go = [&](auto kern) {
            kern<<<col_grid(d, LB, nf), 256, (size_t)d.nz * 48 << LB, st>>>(in, out, d.nz, d.P, d.ncol, d.nfield, phim,
                                                                            phip, pl, W);
        };
        if (mode == COL_DST) go(k_fx_columns<COL_DST, NIT, LB>);
        else if (mode == COL_DCT) go(k_fx_columns<COL_DCT, NIT, LB>);
        else if (mode == COL_DECOMP) go(k_fx_columns<COL_DECOMP, NIT, LB>);
        else go(k_fx_columns<COL_COMBINE, NIT, LB>);
    });
}
// bytes of nf fields, for the probe
static double field_bytes(const Dims &d, int nf)
{
    return (double)nf * (double)d.ncol * (double)(d.nz + 1) * sizeof(double);
}

void fx_comdec(const Dims &d, cudaStream_t st, const double *c, double *cs, double *es, double dzi,
               const double *phim, const double *phip, const void *tw, Probe *pr)
{
    const fx::Plan pl = fx::col_plan(d.nz);
    if (pr) pr->begin(PROBE_COLUMNS, st);
    col_shape(d.nz, d.ncol, [&](auto nit, auto lb) {
        constexpr int NIT = decltype(nit)::value, LB = decltype(lb)::value;
        k_fx_comdec<NIT, LB><<<col_grid(d, LB, 1), 256, (size_t)d.nz * 48 << LB, st>>>(
            c, cs, es, d.nz, d.P, d.ncol, dzi, phim, phip, pl, reinterpret_cast<const Tw *>(tw));
    });
    if (pr) pr->end(PROBE_COLUMNS, st, field_bytes(d, 3));
}
void fx_w(const Dims &d, cudaStream_t st, const double *A, const double *B, double *w, double *es, const Deriv &D,
          const double *thetam, const double *thetap, const double *dthetam, const double *dthetap,
          const double *green, const double *rkz, const void *tw, Probe *pr)
{
    const fx::Plan pl = fx::col_plan(d.nz);
    if (pr) pr->begin(PROBE_COLUMNS, st);
    const WTables tb{thetam, thetap, dthetam, dthetap, green, rkz};
    col_shape(d.nz, d.ncol, [&](auto nit, auto lb) {
        constexpr int NIT = decltype(nit)::value, LB = decltype(lb)::value;
        k_fx_w<NIT, LB><<<col_grid(d, LB, 1), 256, (size_t)d.nz * 48 << LB, st>>>(
            A, B, w, es, d.nx, d.ny, d.nz, d.P, d.ncol, D, tb, pl, reinterpret_cast<const Tw *>(tw));
    });
    if (pr) pr->end(PROBE_COLUMNS, st, field_bytes(d, 4));
}
void fx_src(const Dims &d, cudaStream_t st, const double *f, double *out, const Deriv &D, const double *phim,
            const double *phip, const void *tw, Probe *pr)
{
    const fx::Plan pl = fx::col_plan(d.nz);
    if (pr) pr->begin(PROBE_COLUMNS, st);
    col_shape(d.nz, d.ncol, [&](auto nit, auto lb) {
        constexpr int NIT = decltype(nit)::value, LB = decltype(lb)::value;
        k_fx_src<NIT, LB><<<col_grid(d, LB, 3), 256, (size_t)d.nz * 48 << LB, st>>>(
            f, out, d.nx, d.ny, d.nz, d.P, d.ncol, d.nfield, D, phim, phip, pl, reinterpret_cast<const Tw *>(tw));
    });
    if (pr) pr->end(PROBE_COLUMNS, st, field_bytes(d, 8));
}

void fx_columns_init()
{
    for (int nz : {64, 128, 256, 512, -64, -128})
        col_shape(nz < 0 ? -nz : nz, nz < 0 ? 0 : 1 << 20, [&](auto nit, auto lb) {
            constexpr int NIT = decltype(nit)::value, LB = decltype(lb)::value;
            const auto set = [](auto kern) {
                cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024);
            };
            set(k_fx_columns<COL_DST, NIT, LB>);
            set(k_fx_columns<COL_DCT, NIT, LB>);
            set(k_fx_columns<COL_DECOMP, NIT, LB>);
            set(k_fx_columns<COL_COMBINE, NIT, LB>);
            set(k_fx_comdec<NIT, LB>);
            set(k_fx_w<NIT, LB>);
            set(k_fx_src<NIT, LB>);
        });
}

}  // namespace ps3d
