// FP64 line transforms on the integer pipes (fx.cuh).
//
// Per field, one launch: at 128^3 81-90 us with the FP64 Stockham kernels,
// which the FP64 pipe bounds, 33-36 us in the first fixed-point form; at
// 256^3 that one took 195 us, the ones below in the kernel's comment.
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
// then every line is converted on its own scale.  The pair exchange of the
// inverse, the later passes and the forward output go through one shared
// buffer, written in place after a barrier, or through two (BUFS) below 128
// points, where both are small and a block's few warps wait for barriers
// most (32^3 run 13.95 ms with one, 13.66 with two).
//
// Neither the integer work (without its passes the kernel still took 100 of
// 150 us at 256^3) nor DRAM (40 us) bounds it but the chain load, barrier,
// convert, passes, store of a block: what helps is more and smaller blocks
// per SM.  T is the largest block, 1024 / T of them fit an SM at 64
// registers.  256^3, one field forward / inverse, us: two buffers and 8 pairs
// (three 256-thread blocks per SM) 151 / 156, 4 pairs 139 / 144, one buffer
// and 8 pairs 131 / 134, one buffer and 4 pairs (eight 128-thread blocks,
// the form here) 126 / 132.
template <int R1, int T, bool INV, int LB, int BUFS>
__global__ void __launch_bounds__(T, 1024 / T)
    k_fx_lines(const double *in, double *out, int n, int P, int zv, long long line_stride,
               long long batch_stride, long long fs_in, long long fs_out, const __grid_constant__ fx::Plan pl,
               const Tw *__restrict__ tw)
{
    constexpr int B = 1 << LB;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ unsigned smax[16];
    __shared__ float ssum[16][16];
    I2 *buf = reinterpret_cast<I2 *>(smem_raw), *buf1 = BUFS == 2 ? buf + (n << LB) : buf;
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
    if (INV && BUFS == 1) __syncthreads();
    if (work) fx::first_pass<R1, INV, LB>(v, buf, j, p);
    __syncthreads();
    fx::later_passes<R1, INV, LB>(n, [&](auto pass, int Ns) {
        pass.read(buf, n, Ns, tw, tid, nt);
        if (BUFS == 1) __syncthreads();
        pass.write(buf1, Ns, tid);
        __syncthreads();
        I2 *x = buf;
        buf = buf1;
        buf1 = x;
    });
    if (!zin) return;
    const fx::Scale sx = fx::scale_of(mx, Ex, pl), sy = fx::scale_of(my, Ey, pl);
    if (!INV) {
        for (int k = j; k <= h; k += nt >> LB) {
            const I2 ck = buf[fx::at<LB>(k, p)];
            const I2 cn = buf[fx::at<LB>(k == 0 ? 0 : n - k, p)];
            // twice A_k and B_k (the factor 1/2 is in the plan's scale)
            *reinterpret_cast<double2 *>(out + k * line_stride) =
                make_double2(fx::to_double(ck.x + cn.x, sx), fx::to_double(ck.y + cn.y, sy));
            if (k > 0 && k < h)
                *reinterpret_cast<double2 *>(out + (n - k) * line_stride) =
                    make_double2(fx::to_double(ck.y - cn.y, sx), fx::to_double(cn.x - ck.x, sy));
        }
    } else {
        for (int i = j; i < n; i += nt >> LB) {
            const I2 u = buf[fx::at<LB>(i, p)];
            *reinterpret_cast<double2 *>(out + i * line_stride) =
                make_double2(fx::to_double(u.x, sx), fx::to_double(u.y, sy));
        }
    }
}

template <int R1, int T, int LB, int BUFS = 1>
static void launch_fx_lines(cudaStream_t st, const double *in, double *out, int n, int P, int zv,
                            long long line_stride, long long nbatch, long long batch_stride, bool inverse,
                            const Tw *tw, int nf, long long fs_in, long long fs_out)
{
    const fx::Plan pl = fx::line_plan(n, inverse);
    const int nt = (((n / R1) << LB) + 31) / 32 * 32;
    const dim3 grid((zv + (2 << LB) - 1) / (2 << LB), (unsigned)nbatch, (unsigned)nf);
    const size_t sm = (size_t)n * 16 * BUFS << LB;  // at most 32 KB
    if (inverse)
        k_fx_lines<R1, T, true, LB, BUFS><<<grid, nt, sm, st>>>(in, out, n, P, zv, line_stride, batch_stride, fs_in,
                                                                fs_out, pl, tw);
    else
        k_fx_lines<R1, T, false, LB, BUFS><<<grid, nt, sm, st>>>(in, out, n, P, zv, line_stride, batch_stride, fs_in,
                                                                 fs_out, pl, tw);
}

void fx_lines(cudaStream_t st, const double *in, double *out, int n, int P, int zv, long long line_stride,
              long long nbatch, long long batch_stride, bool inverse, const void *tw, int nf, long long fs_in,
              long long fs_out)
{
    // 4 z pairs per block (64-byte rows), one butterfly of the first pass per
    // thread; 8 pairs where those fill their warps and the levels so much
    // better that a tenth of the threads is saved and two blocks per SM are
    // left (96x160x60 run: 10.32 ms with 8 pairs, 10.42 with 4; 32^3: 13.70
    // and 12.95); 2 pairs for the lengths 2 3^b (18, 54, 162, 486), whose
    // first radix is 3
    const int r = fx::first_radix(n), t = n / r * 4;
    const auto cost = [&](int pairs) {
        return (long long)((zv + 2 * pairs - 1) / (2 * pairs)) * ((n / r * pairs + 31) / 32);
    };
    const bool wide = 2 * t <= 256 && 10 * cost(8) < 9 * cost(4) && (zv + 15) / 16 * nbatch * nf >= 2 * 152;
    const bool two = n < 128;
    auto go = [&](auto f) {
        f(st, in, out, n, P, zv, line_stride, nbatch, batch_stride, inverse, reinterpret_cast<const Tw *>(tw), nf,
          fs_in, fs_out);
    };
    if (r == 8 && wide) two ? go(launch_fx_lines<8, 256, 3, 2>) : go(launch_fx_lines<8, 256, 3, 1>);
    else if (r == 8 && two) go(launch_fx_lines<8, 128, 2, 2>);
    else if (r == 8 && t <= 128) go(launch_fx_lines<8, 128, 2>);
    else if (r == 8) go(launch_fx_lines<8, 256, 2>);
    else if (r == 4 && wide) go(launch_fx_lines<4, 256, 3, 2>);  // at most 124 points
    else if (r == 4 && two) go(launch_fx_lines<4, 128, 2, 2>);
    else if (r == 4 && t <= 256) go(launch_fx_lines<4, 256, 2>);
    else if (r == 4) go(launch_fx_lines<4, 512, 2>);
    else if (r == 5 && two) go(launch_fx_lines<5, 128, 2, 2>);
    else if (r == 5 && t <= 256) go(launch_fx_lines<5, 256, 2>);
    else if (r == 5) go(launch_fx_lines<5, 512, 2>);
    else go(launch_fx_lines<3, 512, 1>);
}

bool fx_serves(int n) { return n <= 512; }
void fx_twiddles(void *host, int n) { fx::fill_twiddles(reinterpret_cast<Tw *>(host), n); }

void fx_init() { fx_columns_init(); }

}  // namespace ps3d
