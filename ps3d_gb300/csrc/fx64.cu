// FP64 line and column transforms on the integer pipes (fx.cuh).
//
// Measured per field at 128^3 (one launch): line passes 81-90 us with the
// FP64 Stockham kernels, which the FP64 pipe bounds, 33-36 us here; column
// transforms 118-136 us before, 36-46 us here.
#include "kernels.h"

#include "fx.cuh"

namespace ps3d {

using fx::I2;
using fx::Tw;

// ------------------------------------------------------------------------
// y / x line transforms (fftxyp2s / fftxys2p of src/fft/sta3dfft.f90:136-260)
// ------------------------------------------------------------------------
// A block owns 2B consecutive z values of one line set, packed in pairs as
// one complex sequence each; layout, padding rows and Hermitian storage as
// in k_lines (transforms.cu).  Each real line has its own fixed-point scale:
// one pass keeps the raw values in shared memory and finds the largest
// magnitude word per line, the next converts them in place.
template <bool INV>
__global__ void __launch_bounds__(256) k_fx_lines(const double *__restrict__ in, double *__restrict__ out, int n,
                                                  int logB, int P, int zv, long long line_stride,
                                                  long long batch_stride, long long fs_in, long long fs_out, const __grid_constant__ fx::Plan pl,
                                                  const Tw *__restrict__ tw)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned smax[16];
    __shared__ float ssum[8][16];
    I2 *buf0 = reinterpret_cast<I2 *>(smem_raw);
    double2 *raw = reinterpret_cast<double2 *>(smem_raw);
    const int B = 1 << logB;
    I2 *buf1 = buf0 + ((size_t)n << logB);
    const int z0 = blockIdx.x * 2 * B;
    const long long base = (long long)blockIdx.y * batch_stride + z0;
    const double2 *inC = reinterpret_cast<const double2 *>(in + blockIdx.z * fs_in);
    double2 *outC = reinterpret_cast<double2 *>(out + blockIdx.z * fs_out);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int p = tid & (B - 1);  // nt is a multiple of B
    const int z = z0 + 2 * p;
    const int h = n / 2;

    if (tid < 16) smax[tid] = 0u;
    __syncthreads();
    unsigned mx = 0u, my = 0u;
    float tx = 0.0f, ty = 0.0f;
    for (int i = tid >> logB; i < n; i += nt >> logB) {
        double2 v = make_double2(0.0, 0.0);
        if (z < P) v = inC[(base + i * line_stride + 2 * p) >> 1];
        // padding rows (z >= zv) enter as zero
        if (z + 1 >= zv) v.y = 0.0;
        if (z >= zv) v.x = 0.0;
        raw[fx::at(i, p, logB)] = v;
        const unsigned ax = fx::mag(v.x), ay = fx::mag(v.y);
        mx = max(mx, ax);
        my = max(my, ay);
        tx += fx::magf(ax);
        ty += fx::magf(ay);
    }
    for (int o = 16; o >= B; o >>= 1) {
        mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        my = max(my, __shfl_xor_sync(0xffffffffu, my, o));
        tx += __shfl_xor_sync(0xffffffffu, tx, o);
        ty += __shfl_xor_sync(0xffffffffu, ty, o);
    }
    if ((tid & 31) < B) {
        atomicMax(&smax[2 * p], mx);
        atomicMax(&smax[2 * p + 1], my);
        ssum[tid >> 5][2 * p] = tx;
        ssum[tid >> 5][2 * p + 1] = ty;
    }
    __syncthreads();
    mx = smax[2 * p];
    my = smax[2 * p + 1];
    tx = ty = 0.0f;
    for (int w = 0; w < nt >> 5; ++w) {  // in a fixed order: every thread of a line gets the same sum
        tx += ssum[w][2 * p];
        ty += ssum[w][2 * p + 1];
    }
    const int ex = fx::line_exp(mx), ey = fx::line_exp(my);
    const int Ex = pl.E[fx::spread(tx, mx, pl.lcap)], Ey = pl.E[fx::spread(ty, my, pl.lcap)];
    if (!INV) {
        for (int i = tid >> logB; i < n; i += nt >> logB) {
            const int q = fx::at(i, p, logB);
            const double2 v = raw[q];
            buf0[q] = fx::mk2(fx::to_fixed(v.x, ex, Ex), fx::to_fixed(v.y, ey, Ey));
        }
    } else {
        // the complex spectrum C_k = A_k + i B_k of the two packed real
        // sequences: A_k = (lo.x, hi.x), B_k = (lo.y, hi.y)
        for (int k = tid >> logB; k <= h; k += nt >> logB) {
            const int q = fx::at(k, p, logB);
            const double2 lo = raw[q];
            const I2 l = fx::mk2(fx::to_fixed(lo.x, ex, Ex), fx::to_fixed(lo.y, ey, Ey));
            if (k > 0 && k < h) {
                const int qn = fx::at(n - k, p, logB);
                const double2 hi = raw[qn];
                const I2 u = fx::mk2(fx::to_fixed(hi.x, ex, Ex), fx::to_fixed(hi.y, ey, Ey));
                buf0[q] = fx::mk2(l.x - u.y, u.x + l.y);
                buf0[qn] = fx::mk2(l.x + u.y, l.y - u.x);
            } else {
                buf0[q] = l;
            }
        }
    }
    __syncthreads();
    const I2 *res = fx::fft<INV>(buf0, buf1, n, logB, 1, tw, 1, tid, nt, [] { __syncthreads(); });
    if (z >= P) return;
    const fx::Scale sx = fx::scale_of(mx, Ex, pl), sy = fx::scale_of(my, Ey, pl);
    if (!INV) {
        for (int k = tid >> logB; k <= h; k += nt >> logB) {
            const I2 ck = res[fx::at(k, p, logB)];
            const I2 cn = res[fx::at(k == 0 ? 0 : n - k, p, logB)];
            // twice A_k and B_k (the factor 1/2 is in the plan's scale)
            outC[(base + k * line_stride + 2 * p) >> 1] =
                make_double2(fx::to_double(ck.x + cn.x, sx), fx::to_double(ck.y + cn.y, sy));
            if (k > 0 && k < h)
                outC[(base + (n - k) * line_stride + 2 * p) >> 1] =
                    make_double2(fx::to_double(ck.y - cn.y, sx), fx::to_double(cn.x - ck.x, sy));
        }
    } else {
        for (int i = tid >> logB; i < n; i += nt >> logB) {
            const I2 v = res[fx::at(i, p, logB)];
            outC[(base + i * line_stride + 2 * p) >> 1] =
                make_double2(fx::to_double(v.x, sx), fx::to_double(v.y, sy));
        }
    }
}

// z pairs per block: 8 (128-byte rows), or 4 where the last tile of 16
// levels would be mostly padding; both buffers within 128 KiB
static int fx_line_lanes(int n, int zv)
{
    int logB = 3;
    const int w16 = (zv + 15) / 16 * 16, w8 = (zv + 7) / 8 * 8;
    if (w16 * 8 > w8 * 9) logB = 2;
    while (logB > 0 && (size_t)n * 32 << logB > 128 * 1024) --logB;
    return logB;
}

void fx_lines(cudaStream_t st, const double *in, double *out, int n, int P, int zv, long long line_stride,
              long long nbatch, long long batch_stride, bool inverse, const void *tw, int nf, long long fs_in,
              long long fs_out)
{
    const int logB = fx_line_lanes(n, zv), B = 1 << logB;
    const fx::Plan pl = fx::line_plan(n, inverse);
    int nt = (n << logB) / 8;
    nt = nt < 64 ? 64 : nt > 256 ? 256 : (nt + 31) / 32 * 32;
    const dim3 grid((zv + 2 * B - 1) / (2 * B), (unsigned)nbatch, (unsigned)nf);
    const size_t sm = (size_t)n * 32 << logB;
    if (inverse)
        k_fx_lines<true><<<grid, nt, sm, st>>>(in, out, n, logB, P, zv, line_stride, batch_stride, fs_in, fs_out,
                                               pl, reinterpret_cast<const Tw *>(tw));
    else
        k_fx_lines<false><<<grid, nt, sm, st>>>(in, out, n, logB, P, zv, line_stride, batch_stride, fs_in, fs_out,
                                                pl, reinterpret_cast<const Tw *>(tw));
}

// ------------------------------------------------------------------------
// z column transforms (dst / dct of src/fft/stafft.f90:410-550), with the
// harmonic parts of field_decompose_semi_spectral / field_combine_semi_spectral
// (inversion_utils.f90:563-647) in FP64 as in k_columns (transforms.cu)
// ------------------------------------------------------------------------
// A block owns 2B columns (B packed pairs).  A warp takes one column at a
// time (lanes along z: coalesced) and finds that column's scale by shuffles
// alone; the pairs are then folded into the three half-length sequences
// (fx.cuh), transformed together and unfolded by the same warps.
template <int MODE>
__global__ void __launch_bounds__(256) k_fx_columns(const double *__restrict__ in, double *__restrict__ out, int nz,
                                                    int P, long long ncol, int logB, const double *__restrict__ phim,
                                                    const double *__restrict__ phip, const __grid_constant__ fx::Plan pl,
                                                    const Tw *__restrict__ W)
{
    constexpr bool DCT = MODE == COL_DCT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double bnd[16][2];
    __shared__ unsigned smag[16];
    __shared__ int sbits[16];
    const int B = 1 << logB, N = nz / 2;
    I2 *seq = reinterpret_cast<I2 *>(smem_raw);
    I2 *Z = seq + ((size_t)3 * N << logB);  // 3N >= nz + 1
    long long *Zs = reinterpret_cast<long long *>(Z);
    double *raw = reinterpret_cast<double *>(Z);
    const long long col0 = (long long)blockIdx.x * 2 * B;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5;

    for (int cl = warp; cl < 2 * B; cl += nt >> 5) {
        const int p = cl >> 1, comp = cl & 1;
        const long long o = (col0 + cl) * P;
        const bool on = col0 + cl < ncol;
        const double f0 = on ? in[o] : 0.0, fn = on ? in[o + nz] : 0.0;
        unsigned m = 0u;
        float t = 0.0f;
        for (int iz = lane; iz <= nz; iz += 32) {
            double v = 0.0;
            if (on && (DCT || (iz > 0 && iz < nz))) {
                v = in[o + iz];
                if (MODE == COL_DECOMP) v = v - (f0 * phim[o + iz] + fn * phip[o + iz]);
            }
            raw[2 * fx::at(iz, p, logB) + comp] = v;
            const unsigned a = fx::mag(v);
            m = max(m, a);
            t += fx::magf(a);
        }
        m = __reduce_max_sync(0xffffffffu, m);
        for (int q = 16; q > 0; q >>= 1) t += __shfl_xor_sync(0xffffffffu, t, q);
        const int E = pl.E[fx::spread(t, m, pl.lcap)], e = fx::line_exp(m);
        for (int iz = lane; iz <= nz; iz += 32) {
            const int q = 2 * fx::at(iz, p, logB) + comp;
            Zs[q] = fx::to_fixed(raw[q], e, E);
        }
        if (lane == 0) {
            bnd[cl][0] = f0;
            bnd[cl][1] = fn;
            smag[cl] = m;
            sbits[cl] = E;
        }
    }
    __syncthreads();
    for (int g = tid; g < (N / 2 + 1) << logB; g += nt) fx::fold<DCT>(Z, seq, N, logB, g & (B - 1), g >> logB, W);
    __syncthreads();
    const I2 *res = fx::fft<false>(seq, Z, N, logB, 3, W, 4, tid, nt, [] { __syncthreads(); });
    const long long *rs = reinterpret_cast<const long long *>(res);
    for (int cl = warp; cl < 2 * B; cl += nt >> 5) {
        if (col0 + cl >= ncol) return;
        const int p = cl >> 1, comp = cl & 1;
        const long long o = (col0 + cl) * P;
        const double f0 = bnd[cl][0], fn = bnd[cl][1];
        const fx::Scale s = fx::scale_of(smag[cl], sbits[cl], pl);
        for (int iz = lane; iz <= nz; iz += 32) {
            bool neg;
            const int q = fx::unfold<DCT>(iz, N, logB, p, &neg);
            // the dst is -Im Z of the first column and, i times it being
            // the packed second one, Re Z
            long long x = rs[2 * q + (DCT ? comp : 1 - comp)];
            if (!DCT && (comp == 0) != neg) x = -x;
            double v = fx::to_double(x, s);
            if (MODE == COL_COMBINE) v = v + f0 * phim[o + iz] + fn * phip[o + iz];
            if (!DCT) {
                if (iz == 0) v = f0;
                if (iz == nz) v = MODE == COL_DST ? 0.0 : fn;
            }
            out[o + iz] = v;
        }
    }
}

// pairs per block: 8, fewer where the buffers would pass 64 KiB (three
// blocks per SM)
static int fx_col_lanes(int nz)
{
    int logB = 3;
    while (logB > 0 && (size_t)nz * 48 << logB > 64 * 1024) --logB;
    return logB;
}

void fx_columns(const Dims &d, cudaStream_t st, int mode, const double *in, double *out, const double *phim,
                const double *phip, const void *tw)
{
    const int logB = fx_col_lanes(d.nz), B = 1 << logB;
    const fx::Plan pl = fx::col_plan(d.nz);
    const unsigned grid = (unsigned)((d.ncol + 2 * B - 1) / (2 * B));
    const size_t sm = (size_t)d.nz * 48 << logB;
    const Tw *W = reinterpret_cast<const Tw *>(tw);
    switch (mode) {
    case COL_DST:
        k_fx_columns<COL_DST><<<grid, 256, sm, st>>>(in, out, d.nz, d.P, d.ncol, logB, phim, phip, pl, W);
        break;
    case COL_DCT:
        k_fx_columns<COL_DCT><<<grid, 256, sm, st>>>(in, out, d.nz, d.P, d.ncol, logB, phim, phip, pl, W);
        break;
    case COL_DECOMP:
        k_fx_columns<COL_DECOMP><<<grid, 256, sm, st>>>(in, out, d.nz, d.P, d.ncol, logB, phim, phip, pl, W);
        break;
    default:
        k_fx_columns<COL_COMBINE><<<grid, 256, sm, st>>>(in, out, d.nz, d.P, d.ncol, logB, phim, phip, pl, W);
        break;
    }
}

bool fx_serves(int n) { return n <= 512; }
void fx_twiddles(void *host, int n) { fx::fill_twiddles(reinterpret_cast<Tw *>(host), n); }

void fx_init()
{
    cudaFuncSetAttribute(k_fx_lines<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    cudaFuncSetAttribute(k_fx_lines<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    cudaFuncSetAttribute(k_fx_columns<COL_DST>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(k_fx_columns<COL_DCT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(k_fx_columns<COL_DECOMP>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
    cudaFuncSetAttribute(k_fx_columns<COL_COMBINE>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 * 1024);
}

}  // namespace ps3d
