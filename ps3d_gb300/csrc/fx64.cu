// FP64 line transforms on the integer pipes (fx.cuh).
//
// Measured per field, one launch.  128^3: line passes 81-90 us with the FP64
// Stockham kernels, which the FP64 pipe bounds, 33-36 us in the first
// fixed-point form; column transforms 118-136 and 36-46 us.  256^3: line
// passes 195 us with every pass in shared memory and the products left to
// the compiler, 136-157 us with the first pass on registers and mad.wide
// spelled out; column transforms 314 and 200-257 us.
#include "kernels.h"

#include "fx.cuh"

namespace ps3d {

using fx::I2;
using fx::Tw;

// ------------------------------------------------------------------------
// y / x line transforms (fftxyp2s / fftxys2p of src/fft/sta3dfft.f90:136-260)
// ------------------------------------------------------------------------
// A block owns 2B consecutive z values of one line set (B = 2^LB), packed in
// pairs as one complex sequence each; layout, padding rows and Hermitian
// storage as in k_lines (transforms.cu).  A thread holds the R1 rows of one
// butterfly of the first pass in registers from the load on; the largest
// magnitude and the magnitude sum of each real line meet in shared memory,
// then every line is converted on its own scale.  Integer issue bounds it:
// the pair exchange of the inverse and of the forward output and the later
// passes go through shared memory, 16 bytes per complex value each way.
template <int R1, bool INV, int LB>
__global__ void __launch_bounds__(R1 == 8 ? 256 : 512)
    k_fx_lines(const double *in, double *out, int n, int P, int zv, long long line_stride,
               long long batch_stride, long long fs_in, long long fs_out, const __grid_constant__ fx::Plan pl,
               const Tw *__restrict__ tw)
{
    constexpr int B = 1 << LB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned smax[16];
    __shared__ float ssum[16][16];
    I2 *buf0 = reinterpret_cast<I2 *>(smem_raw);
    I2 *buf1 = buf0 + (n << LB);
    const int tid = threadIdx.x, nt = blockDim.x;
    const int p = tid & (B - 1), j = tid >> LB;
    const int z = blockIdx.x * 2 * B + 2 * p;
    const int nR = n / R1, h = n / 2;
    const bool work = j < nR, zin = z < P;
    const long long base = (long long)blockIdx.y * batch_stride + z;
    in += blockIdx.z * fs_in + base;
    out += blockIdx.z * fs_out + base;

    if (tid < 16) smax[tid] = 0u;
    __syncthreads();
    double2 raw[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) {
        raw[r] = make_double2(0.0, 0.0);
        if (work && zin) raw[r] = *reinterpret_cast<const double2 *>(in + (j + r * nR) * line_stride);
    }
    // padding rows (z >= zv) enter as zero
    if (z + 1 >= zv) {
#pragma unroll
        for (int r = 0; r < R1; ++r) {
            raw[r].y = 0.0;
            if (z >= zv) raw[r].x = 0.0;
        }
    }
    unsigned mx = 0u, my = 0u;
    float tx = 0.0f, ty = 0.0f;
#pragma unroll
    for (int r = 0; r < R1; ++r) {
        const unsigned ax = fx::mag(raw[r].x), ay = fx::mag(raw[r].y);
        mx = max(mx, ax);
        my = max(my, ay);
        tx += fx::magf(ax);
        ty += fx::magf(ay);
    }
#pragma unroll
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
    const int Ex = pl.E[fx::spread(tx, mx, pl.lcap)], Ey = pl.E[fx::spread(ty, my, pl.lcap)];
    I2 v[R1];
    {
        const int ex = fx::line_exp(mx), ey = fx::line_exp(my);
#pragma unroll
        for (int r = 0; r < R1; ++r) v[r] = fx::mk2(fx::to_fixed(raw[r].x, ex, Ex), fx::to_fixed(raw[r].y, ey, Ey));
    }
    if (INV) {
        if (work) {
#pragma unroll
            for (int r = 0; r < R1; ++r) buf1[fx::at<LB>(j + r * nR, p)] = v[r];
        }
        __syncthreads();
        if (work) {
#pragma unroll
            for (int r = 0; r < R1; ++r) {
                const int k = j + r * nR;
                v[r] = fx::join(v[r], buf1[fx::at<LB>(k ? n - k : 0, p)], k, h);
            }
        }
    }
    if (work) fx::first_pass<R1, INV, LB>(v, buf0, j, p);
    __syncthreads();
    const I2 *res = fx::passes<INV, LB>(buf0, buf1, n, 1, R1, tw, 1, tid, nt, [] { __syncthreads(); });
    if (!zin) return;
    const fx::Scale sx = fx::scale_of(mx, Ex, pl), sy = fx::scale_of(my, Ey, pl);
    if (!INV) {
        for (int k = j; k <= h; k += nt >> LB) {
            const I2 ck = res[fx::at<LB>(k, p)];
            const I2 cn = res[fx::at<LB>(k == 0 ? 0 : n - k, p)];
            // twice A_k and B_k (the factor 1/2 is in the plan's scale)
            *reinterpret_cast<double2 *>(out + k * line_stride) =
                make_double2(fx::to_double(ck.x + cn.x, sx), fx::to_double(ck.y + cn.y, sy));
            if (k > 0 && k < h)
                *reinterpret_cast<double2 *>(out + (n - k) * line_stride) =
                    make_double2(fx::to_double(ck.y - cn.y, sx), fx::to_double(cn.x - ck.x, sy));
        }
    } else {
        for (int i = j; i < n; i += nt >> LB) {
            const I2 u = res[fx::at<LB>(i, p)];
            *reinterpret_cast<double2 *>(out + i * line_stride) =
                make_double2(fx::to_double(u.x, sx), fx::to_double(u.y, sy));
        }
    }
}

template <int R1, int LB>
static void launch_fx_lines(cudaStream_t st, const double *in, double *out, int n, int P, int zv,
                            long long line_stride, long long nbatch, long long batch_stride, bool inverse,
                            const Tw *tw, int nf, long long fs_in, long long fs_out)
{
    const fx::Plan pl = fx::line_plan(n, inverse);
    const int nt = (((n / R1) << LB) + 31) / 32 * 32;
    const dim3 grid((zv + (2 << LB) - 1) / (2 << LB), (unsigned)nbatch, (unsigned)nf);
    const size_t sm = (size_t)n * 32 << LB;
    if (inverse)
        k_fx_lines<R1, true, LB><<<grid, nt, sm, st>>>(in, out, n, P, zv, line_stride, batch_stride, fs_in, fs_out,
                                                       pl, tw);
    else
        k_fx_lines<R1, false, LB><<<grid, nt, sm, st>>>(in, out, n, P, zv, line_stride, batch_stride, fs_in, fs_out,
                                                        pl, tw);
}

void fx_lines(cudaStream_t st, const double *in, double *out, int n, int P, int zv, long long line_stride,
              long long nbatch, long long batch_stride, bool inverse, const void *tw, int nf, long long fs_in,
              long long fs_out)
{
    // z pairs per block: 8 (128-byte rows); 4 where the last tile of 16
    // levels would be mostly padding, or where 8 would take more threads
    // than a block of the kernel has (one butterfly per thread).  2 odd
    // lengths of 3s only (18, 54, 162, 486): 2.
    const int r = fx::first_radix(n);
    const int w16 = (zv + 15) / 16 * 16, w8 = (zv + 7) / 8 * 8;
    const bool wide = w16 * 8 <= w8 * 9 && (n / r) * 8 <= (r == 8 ? 256 : 512);
    auto go = [&](auto f) {
        f(st, in, out, n, P, zv, line_stride, nbatch, batch_stride, inverse, reinterpret_cast<const Tw *>(tw), nf,
          fs_in, fs_out);
    };
    if (r == 8) wide ? go(launch_fx_lines<8, 3>) : go(launch_fx_lines<8, 2>);
    else if (r == 4) wide ? go(launch_fx_lines<4, 3>) : go(launch_fx_lines<4, 2>);
    else if (r == 5) wide ? go(launch_fx_lines<5, 3>) : go(launch_fx_lines<5, 2>);
    else go(launch_fx_lines<3, 1>);
}

bool fx_serves(int n) { return n <= 512; }
void fx_twiddles(void *host, int n) { fx::fill_twiddles(reinterpret_cast<Tw *>(host), n); }

template <int R1, int LB> static void fx_line_attrs()
{
    cudaFuncSetAttribute(k_fx_lines<R1, true, LB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
    cudaFuncSetAttribute(k_fx_lines<R1, false, LB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 128 * 1024);
}
void fx_init()
{
    fx_line_attrs<8, 3>();
    fx_line_attrs<8, 2>();
    fx_line_attrs<4, 3>();
    fx_line_attrs<4, 2>();
    fx_line_attrs<5, 3>();
    fx_line_attrs<5, 2>();
    fx_line_attrs<3, 1>();
    fx_columns_init();
}

}  // namespace ps3d
