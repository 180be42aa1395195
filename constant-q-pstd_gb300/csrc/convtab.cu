// convtab.cu -- multipliers of the per-kz convolutions (XconvArgs), built in FP64 on the device.
//
// A stationary symbol's column at kz acts along x as a circular convolution with
// h = DFT_n(symbol column) / (nxx nzz), real and even; its multiplier on the padded length m is the
// transform of h wrapped to m.  Both transforms run in double (the first by Bluestein's identity on
// m), so that a multiplier's error is its one rounding, relative to itself.  In FP32 the error was
// relative to the column's largest multiplier: operators came out 1.3 - 1.9 times further from 64
// bits at widths that transform directly, where the symbol itself would have been the multiplier.
//
// A CTA takes two columns as the real and imaginary parts of one line in shared memory.  The
// transforms are decimation in frequency in place, the inverse its mirror image, so nothing is
// sorted: the spectra are met at their digit-reversed positions.  Bound by FP64 arithmetic (2
// fused multiply-adds per clock and SM), about 250 operations per point of a line.
#include <cuda_runtime.h>

#include "qpstd_internal.h"

namespace qp {
namespace {

__device__ __forceinline__ double2 mul(double2 a, double2 b) {
    return make_double2(fma(a.x, b.x, -a.y * b.y), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 mulc(double2 a, double2 b) {  // a conj(b)
    return make_double2(fma(a.x, b.x, a.y * b.y), fma(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// DFT of R values, S = -1 forward, +1 inverse; root[q * step] = e^{-2 pi i q / R}
template <int R, int S> __device__ __forceinline__ void dft(double2 (&v)[R], const double2* __restrict__ root, int step) {
    if constexpr (R == 2) {
        const double2 a = v[0], b = v[1];
        v[0] = a + b;
        v[1] = a - b;
    } else if constexpr (R == 4) {
        const double2 a = v[0] + v[2], b = v[0] - v[2], c = v[1] + v[3], d = v[1] - v[3];
        const double2 up = make_double2(b.x - d.y, b.y + d.x), dn = make_double2(b.x + d.y, b.y - d.x);
        v[0] = a + c;
        v[2] = a - c;
        v[1] = S > 0 ? up : dn;
        v[3] = S > 0 ? dn : up;
    } else {
        constexpr int H = (R - 1) / 2;
        double2 a[H], b[H], w[H + 1];
        double2 s0 = v[0];
#pragma unroll
        for (int r = 1; r <= H; r++) {
            a[r - 1] = v[r] + v[R - r];
            b[r - 1] = v[r] - v[R - r];
            s0 = s0 + a[r - 1];
            w[r] = root[r * step];
        }
#pragma unroll
        for (int q = 1; q <= H; q++) {
            double2 re = v[0], im = make_double2(0.0, 0.0);
#pragma unroll
            for (int r = 1; r <= H; r++) {
                const int m = (r * q) % R;
                const int k = m <= H ? m : R - m;
                const double c = w[k].x, s = m <= H ? -w[k].y : w[k].y;
                re.x = fma(a[r - 1].x, c, re.x);
                re.y = fma(a[r - 1].y, c, re.y);
                im.x = fma(b[r - 1].x, s, im.x);
                im.y = fma(b[r - 1].y, s, im.y);
            }
            const double2 up = make_double2(re.x - im.y, re.y + im.x), dn = make_double2(re.x + im.y, re.y - im.x);
            v[q] = S > 0 ? up : dn;
            v[R - q] = S > 0 ? dn : up;
        }
        v[0] = s0;
    }
}

// One pass in place over blocks of len: butterflies of R values len / R apart.  Forward: the DFT,
// then the twiddles; inverse: the mirror image.
template <int R, int S> __device__ __forceinline__ void pass(double2* x, const ConvTabArgs& a, int len) {
    const int q = len / R, step = a.m / len;
    for (int i = threadIdx.x; i < a.m / R; i += blockDim.x) {
        const int blk = i / q, j = i - blk * q, o = blk * len + j;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
            v[r] = x[o + r * q];
            if (S > 0 && r > 0) v[r] = mulc(v[r], a.w[j * r * step]);
        }
        dft<R, S>(v, a.w, a.m / R);
#pragma unroll
        for (int r = 0; r < R; r++) {
            if (S < 0 && r > 0) v[r] = mul(v[r], a.w[j * r * step]);
            x[o + r * q] = v[r];
        }
    }
    __syncthreads();
}
template <int S> __device__ __forceinline__ void pass_any(double2* x, const ConvTabArgs& a, int r, int len) {
    if (r == 2) pass<2, S>(x, a, len);
    else if (r == 3) pass<3, S>(x, a, len);
    else if (r == 4) pass<4, S>(x, a, len);
    else if (r == 5) pass<5, S>(x, a, len);
    else pass<7, S>(x, a, len);
}
// natural order -> digit-reversed, and back
__device__ void forward(double2* x, const ConvTabArgs& a) {
    int len = a.m;
    for (int p = 0; p < a.nrad; p++) {
        pass_any<-1>(x, a, a.rad[p], len);
        len /= a.rad[p];
    }
}
__device__ void inverse(double2* x, const ConvTabArgs& a) {
    int len = 1;
    for (int p = a.nrad - 1; p >= 0; p--) {
        len *= a.rad[p];
        pass_any<1>(x, a, a.rad[p], len);
    }
}
// frequency at position i of a forward transform
__device__ __forceinline__ int freq(int i, const ConvTabArgs& a) {
    int f = 0, len = a.m, mult = 1;
    for (int p = 0; p < a.nrad; p++) {
        len /= a.rad[p];
        const int s = i / len;
        i -= s * len;
        f += s * mult;
        mult *= a.rad[p];
    }
    return f;
}

// The symbol at (kx, kz) of table t: 0 (k^2)^(1/32), 1 k^2, 2 (k^2)^(33/32), 3 (k^2)^0.505; with V
// the low-rank factor t (half grid, mirrored).
__device__ __forceinline__ double symbol(const ConvTabArgs& a, int t, int kx, int kz) {
    const int hz = min(kz, a.nzz - kz);
    if (a.V) return a.V[((size_t)t * (a.nxx / 2 + 1) + kx) * (a.nzz / 2 + 1) + hz];
    const double x = kx * a.dkx, z = hz * a.dkz, k2 = x * x + z * z;
    if (t == 1) return k2;
    if (t == 0) return pow(k2, 1.0 / 32.0);
    if (t == 2) return pow(k2, 33.0 / 32.0);
    return pow(k2, 0.505);
}

__global__ void convtab_kernel(ConvTabArgs a) {
    extern __shared__ double2 x[];
    const int n = a.nxx, m = a.m, kz = 2 * blockIdx.x, t = blockIdx.y;
    for (int i = threadIdx.x; i < m; i += blockDim.x)
        if (i >= n) x[i] = make_double2(0.0, 0.0);
    for (int i = threadIdx.x; i <= n / 2; i += blockDim.x) {
        const double2 v = make_double2(symbol(a, t, i, kz), symbol(a, t, i, kz + 1));
        x[i] = mul(v, a.chirp[i]);
        if (i > 0) x[n - i] = mul(v, a.chirp[n - i]);
    }
    __syncthreads();
    forward(x, a);
    for (int i = threadIdx.x; i < m; i += blockDim.x) x[i] = mul(x[i], a.bhat[freq(i, a)]);
    __syncthreads();
    inverse(x, a);
    // h at the lags 0 .. n-1 and, wrapped, -(n-1) .. -1 (m >= 2n-1: distinct slots)
    for (int i = threadIdx.x; i <= m - n; i += blockDim.x)
        if (i >= n) x[i] = make_double2(0.0, 0.0);
    for (int d = threadIdx.x; d < n; d += blockDim.x) {
        const double2 h = mul(x[d], a.chirp[d]), v = make_double2(h.x * a.scale, h.y * a.scale);
        x[d] = v;
        if (d > 0) x[m - d] = v;
    }
    __syncthreads();
    forward(x, a);
    const int mh = m / 2 + 1;
    float* out = a.out + ((size_t)t * a.nzh + kz) * mh;
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const int f = freq(i, a);
        if (f < mh) {
            out[f] = (float)x[i].x;
            out[mh + f] = (float)x[i].y;
        }
    }
}

}  // namespace

cudaError_t launch_convtab(const ConvTabArgs& a, int ntab, cudaStream_t s) {
    convtab_kernel<<<dim3(a.nzh / 2, ntab), a.m < 2048 ? 256 : 512, sizeof(double2) * (size_t)a.m, s>>>(a);
    return cudaGetLastError();
}
int convtab_set_smem_limits() {
    return cudaFuncSetAttribute(convtab_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, QP_SMEM_DYN_MAX) != cudaSuccess;
}

}  // namespace qp
