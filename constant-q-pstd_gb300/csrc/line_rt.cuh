// line_rt.cuh -- line transforms that start and end in registers.
//
// The pass kernels apply operators y = F^-1[H . F x] to lines of the grid.  A
// Stockham transform (fft_reg.cuh) sorts its output, and every pass of it goes
// through shared memory with two barriers.  An operator does not need the
// spectrum sorted: here the forward transform is decimation in frequency in
// place, its last pass, the multiplier and the first pass of the inverse
// (decimation in time, the same positions backwards) are one pass, the first
// pass takes its inputs from registers and the last one leaves its outputs in
// the same registers of the same thread.  Against the Stockham roundtrip of a
// three-radix length this is 8 sweeps over shared memory instead of 14 and 4
// barriers instead of 14, and the loads and epilogues around it work on
// registers.
//
// A thread runs the same butterflies of W complex lines at once: W = 2 holds
// them as pairs for the packed FP32 instructions (fma.rn.f32x2 and the like),
// which run at the FP32 pipe's rate on half the issue slots (measured 117 - 127
// lane operations per clock and SM against 86 - 126 for the scalar forms), and
// shares twiddles and addresses between the lines.
//
// Measured (batches that fill the SMs, clocks of one SM per point and roundtrip): 3360 points
// 1.07 with two lines per thread and 1.22 with one, against 2.7 of the Stockham roundtrip;
// 256 points 0.50, 1024 0.73, 4096 0.93.
//
// Twiddles come from a table of M + R2 R3 factors in the order the passes read them
// (rt_twiddles, host_setup.cpp): w_M^(a j) at a M/R1 + j, then w_(R2 R3)^(b c) at M + b R3 + c.
//
// Lengths are M = R1 R2 R3 (R2 = 1: two passes).  Element (a, b, c) of a line,
// input index a M/R1 + b R3 + c or, transformed in place, frequency
// a + R1 b + R1 R2 c, sits at a P1 + b R3 + c.  P1 is R2 R3 padded so that both
// the middle pass (threads c fastest) and the merged pass (threads a fastest,
// which reads the multiplier in its natural order) touch distinct banks.
#pragma once
#include <cuda_runtime.h>

#include "fft_reg.cuh"

namespace qp {

// ---- values of W lines: T = float (W = 1) or float2 (W = 2, packed) ---------------
// The packed forms work on 64-bit register pairs.
__device__ __forceinline__ unsigned long long u64(float2 a) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 f2(unsigned long long a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
__device__ __forceinline__ float vadd(float a, float b) { return a + b; }
__device__ __forceinline__ float vsub(float a, float b) { return a - b; }
__device__ __forceinline__ float vmul(float a, float b) { return a * b; }
__device__ __forceinline__ float vfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ float2 vadd(float2 a, float2 b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(u64(a)), "l"(u64(b)));
    return f2(r);
}
__device__ __forceinline__ float2 vsub(float2 a, float2 b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(u64(a)), "l"(u64(b)));
    return f2(r);
}
__device__ __forceinline__ float2 vmul(float2 a, float2 b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(u64(a)), "l"(u64(b)));
    return f2(r);
}
__device__ __forceinline__ float2 vfma(float2 a, float2 b, float2 c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(u64(a)), "l"(u64(b)), "l"(u64(c)));
    return f2(r);
}
template <class T> __device__ __forceinline__ T bcast(float s);
template <> __device__ __forceinline__ float bcast<float>(float s) { return s; }
template <> __device__ __forceinline__ float2 bcast<float2>(float s) { return make_float2(s, s); }

template <int W> struct LineVal;
template <> struct LineVal<1> {
    using T = float;
};
template <> struct LineVal<2> {
    using T = float2;
};
// one complex value of each of the W lines
template <class T> struct Cx {
    T x, y;
};
template <class T> __device__ __forceinline__ Cx<T> czero() { return {bcast<T>(0.f), bcast<T>(0.f)}; }
template <class T> __device__ __forceinline__ Cx<T> operator+(Cx<T> a, Cx<T> b) { return {vadd(a.x, b.x), vadd(a.y, b.y)}; }
template <class T> __device__ __forceinline__ Cx<T> operator-(Cx<T> a, Cx<T> b) { return {vsub(a.x, b.x), vsub(a.y, b.y)}; }
// a * (wr + i wi), the same factor for every line
template <class T> __device__ __forceinline__ Cx<T> cmulw(Cx<T> a, float wr, float wi) {
    const T r = bcast<T>(wr), i = bcast<T>(wi), ni = bcast<T>(-wi);
    return {vfma(a.y, ni, vmul(a.x, r)), vfma(a.y, r, vmul(a.x, i))};
}
template <class T> __device__ __forceinline__ Cx<T> cmuls(Cx<T> a, T s) { return {vmul(a.x, s), vmul(a.y, s)}; }

// ---- in-register DFTs of size R, S = -1 forward, +1 inverse; the first NZ inputs
// may be non-zero, the others are not read -------------------------------------------
template <int P, int S, int NZ, class T> __device__ __forceinline__ void rdft_prime(Cx<T> (&v)[P]) {
    constexpr int H = (P - 1) / 2;
    constexpr Roots<P> rt{};
    Cx<T> a[H], b[H];
#pragma unroll
    for (int r = 1; r <= H; r++) {
        if (P - r < NZ) {
            a[r - 1] = v[r] + v[P - r];
            b[r - 1] = v[r] - v[P - r];
        } else if (r < NZ) {
            a[r - 1] = b[r - 1] = v[r];
        }
    }
    const Cx<T> x0 = v[0];
    Cx<T> s0 = x0;
#pragma unroll
    for (int r = 1; r <= H; r++)
        if (r < NZ) s0 = s0 + a[r - 1];
#pragma unroll
    for (int q = 1; q <= H; q++) {
        Cx<T> re = x0, im;
#pragma unroll
        for (int r = 1; r <= H; r++) {
            if (r >= NZ) continue;
            const int m = (r * q) % P;
            const T c = bcast<T>(rt.c[m]), s = bcast<T>(rt.s[m]);
            re.x = vfma(a[r - 1].x, c, re.x);
            re.y = vfma(a[r - 1].y, c, re.y);
            if (r == 1) {
                im.x = vmul(b[r - 1].x, s);
                im.y = vmul(b[r - 1].y, s);
            } else {
                im.x = vfma(b[r - 1].x, s, im.x);
                im.y = vfma(b[r - 1].y, s, im.y);
            }
        }
        if (NZ < 2) {
            v[q] = v[P - q] = x0;
            continue;
        }
        // re + S i im and its mirror
        const Cx<T> up{vsub(re.x, im.y), vadd(re.y, im.x)}, dn{vadd(re.x, im.y), vsub(re.y, im.x)};
        v[q] = S > 0 ? up : dn;
        v[P - q] = S > 0 ? dn : up;
    }
    v[0] = s0;
}

template <int R, int S, int NZ, class T> __device__ __forceinline__ void rdft(Cx<T> (&v)[R]) {
    if constexpr (R == 1) {
        return;
    } else if constexpr (NZ <= 1) {
#pragma unroll
        for (int r = 1; r < R; r++) v[r] = v[0];
    } else if constexpr (R == 2) {
        const Cx<T> a = v[0], b = v[1];
        v[0] = a + b;
        v[1] = a - b;
    } else if constexpr (R == 4) {
        Cx<T> t0, t1, t2, d;
        if constexpr (NZ > 2) {
            t0 = v[0] + v[2];
            t1 = v[0] - v[2];
        } else {
            t0 = t1 = v[0];
        }
        if constexpr (NZ > 3) {
            t2 = v[1] + v[3];
            d = v[1] - v[3];
        } else {
            t2 = d = v[1];
        }
        v[0] = t0 + t2;
        v[2] = t0 - t2;
        const Cx<T> up{vsub(t1.x, d.y), vadd(t1.y, d.x)}, dn{vadd(t1.x, d.y), vsub(t1.y, d.x)};
        v[1] = S > 0 ? up : dn;
        v[3] = S > 0 ? dn : up;
    } else if constexpr (small_factor<R>() == R) {
        rdft_prime<R, S, NZ>(v);
    } else {
        constexpr int A0 = small_factor<R>();
        constexpr int A = (A0 == 2 && R % 4 == 0 && R > 4) ? 4 : A0;
        constexpr int B = R / A;
        constexpr Roots<R> rt{};
        Cx<T> u[A][B];
        auto inner = [&]<int I>() {
            constexpr int nz = NZ > I ? (NZ - I + A - 1) / A : 0;  // inputs I, I + A, ... below NZ
#pragma unroll
            for (int b = 0; b < B; b++)
                if (b < nz) u[I][b] = v[I + A * b];
            if constexpr (nz > 0) rdft<B, S, nz>(u[I]);
#pragma unroll
            for (int q = 1; q < B; q++) {
                if (I == 0 || nz == 0) continue;
                const int m = (I * q) % R;
                if (4 * m == R) u[I][q] = S > 0 ? Cx<T>{vsub(bcast<T>(0.f), u[I][q].y), u[I][q].x}
                                                : Cx<T>{u[I][q].y, vsub(bcast<T>(0.f), u[I][q].x)};
                else u[I][q] = cmulw(u[I][q], rt.c[m], (float)S * rt.s[m]);
            }
        };
        inner.template operator()<0>();
        inner.template operator()<1>();
        if constexpr (A > 2) inner.template operator()<2>();
        if constexpr (A > 3) inner.template operator()<3>();
        if constexpr (A > 4) inner.template operator()<4>();
        static_assert(A <= 5 || A0 == R, "inner DFTs written out for A <= 5");
        constexpr int NA = NZ < A ? NZ : A;
#pragma unroll
        for (int q = 0; q < B; q++) {
            Cx<T> t[A];
#pragma unroll
            for (int a = 0; a < A; a++)
                if (a < NA) t[a] = u[a][q];
            rdft<A, S, NA>(t);
#pragma unroll
            for (int p = 0; p < A; p++) v[q + B * p] = t[p];
        }
    }
}

// v[r] *= w_r (S > 0: conjugate), r = 1 .. R-1, w_r = t[r * step]: every factor from a table,
// correctly rounded.  (Powers of one loaded factor, by repeated products or by squaring, have
// up to R times its rounding error, and the inverse passes repeat the forward ones' factors:
// over tens of steps the images came out 2 - 3 times further from 64 bits.  Products of w, w^2,
// w^4 and w^8 cost more than the loads they save: the 64-shot batch 10.4 -> 9.8 Gpts/s.)
template <int R, int S, class T> __device__ __forceinline__ void twiddle(Cx<T> (&v)[R], const float2* t, int step) {
#pragma unroll
    for (int r = 1; r < R; r++) {
        const float2 w = t[r * step];
        v[r] = cmulw(v[r], w.x, S > 0 ? -w.y : w.y);
    }
}

// ---- overlap with the kernels before and after on the stream -------------------------------
// A launch with a programmatic dependency (launch_rt) may start while the kernel before it
// still runs: everything that kernel writes is read after rt_wait.  rt_release lets the next
// one start; it then waits beside this kernel's last pass with its tables copied.
__device__ __forceinline__ void rt_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void rt_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Launches kernel k; pdl: with the programmatic dependency.
template <class K, class A>
void launch_rt(K k, unsigned grid, int threads, size_t smem, cudaStream_t s, int pdl, const A& a) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&c, k, a);  // the callers check cudaGetLastError
}

// ---- the engine ------------------------------------------------------------------------
// PAD: a zero-padded line, inputs and outputs [0, M/2]; else all M.
// G: line groups (of W lines) per CTA; GF: consecutive threads are consecutive groups (the
// z passes: neighbouring rows), else consecutive butterflies of a group.  MB: resident
// CTAs per SM the kernels are compiled for (their register cap).  EPI: registers an epilogue
// loop's loads in flight may take.
template <int W_, bool PAD, bool GF, int G_, int MB, int R1_, int R2_, int R3_, int EPI> struct LineRT {
    static constexpr int W = W_, G = G_, kMinB = MB, R1 = R1_, R2 = R2_, R3 = R3_;
    static constexpr bool kPad = PAD;
    static constexpr int kEpiRegs = EPI;
    using T = typename LineVal<W>::T;
    using C = Cx<T>;
    static constexpr int M = R1 * R2 * R3;
    static constexpr int B1 = M / R1, B2 = (R2 > 1) ? M / R2 : 0, B3 = M / R3;
    // threads per group: a butterfly of the first and of the merged pass each; the middle pass,
    // whose values stay in shared memory, takes its butterflies in kTurns turns
    static constexpr int kMaxB = B1 > B3 ? B1 : B3;
    static constexpr int kTurns = (B2 + kMaxB - 1) / kMaxB;
    static constexpr int kThreads = (G * kMaxB + 31) / 32 * 32;
    static constexpr int NZ = PAD ? (R1 + 1) / 2 : R1;  // values of a thread: indices j + r B1, r < NZ
    // bank period of one element: 16 8-byte or 8 16-byte elements per wavefront
    static constexpr int kPeriod = W == 1 ? 16 : 8;
    static constexpr int P1 = [] {
        int p = R2 * R3;
        if (R3 % 2) {
            while (p % kPeriod != R3 % kPeriod) p++;
        } else {
            p |= 1;
        }
        return p;
    }();
    // elements of one group; with GF the threads of a wavefront spread over the groups,
    // whose buffers then start kPeriod / G banks apart
    static constexpr int kElems = [] {
        int e = R1 * P1;
        if (GF && G > 1)
            while (e % kPeriod != (kPeriod / G) % kPeriod) e++;
        return e;
    }();
    static constexpr size_t kLines = ((size_t)G * kElems * 8 * W + 15) / 16 * 16;  // bytes of a CTA's lines
    // Behind the lines, the CTA's copy of the twiddle table: read through L1 its factors cost
    // the passes an L2 latency each whenever shots with tables of their own share an SM.
    static constexpr int kTab = (M + R2 * R3 + 1) / 2 * 2;        // (padded to 16 bytes)
    static constexpr size_t kSmem = kLines + (size_t)kTab * 8;

    using E = typename std::conditional<W == 1, float2, float4>::type;
    __device__ __forceinline__ static C ld(const E* s) {
        if constexpr (W == 1) {
            const float2 e = *s;
            return {e.x, e.y};
        } else {
            const float4 e = *s;
            return {make_float2(e.x, e.y), make_float2(e.z, e.w)};
        }
    }
    __device__ __forceinline__ static void st(E* s, C c) {
        if constexpr (W == 1) *s = make_float2(c.x, c.y);
        else *s = make_float4(c.x.x, c.x.y, c.y.x, c.y.y);
    }
    // This thread's group and butterfly.
    __device__ __forceinline__ static int group() { return G == 1 ? 0 : GF ? threadIdx.x % G : threadIdx.x / kMaxB; }
    __device__ __forceinline__ static int bfly() { return G == 1 ? threadIdx.x : GF ? threadIdx.x / G : threadIdx.x % kMaxB; }
    __device__ __forceinline__ static E* base(void* smem) { return reinterpret_cast<E*>(smem) + (G == 1 ? 0 : group() * kElems); }
    __device__ __forceinline__ static bool live() { return G * kMaxB == kThreads || threadIdx.x < G * kMaxB; }
    // Starts the copy of the table and returns where it will be; complete after tables_ready().
    __device__ __forceinline__ static const float2* tables(void* smem, const float2* __restrict__ tw) {
        char* d = reinterpret_cast<char*>(smem) + kLines;
        const unsigned sd = (unsigned)__cvta_generic_to_shared(d);
        for (int i = threadIdx.x; i < kTab / 2; i += kThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sd + i * 16), "l"(tw + i * 2) : "memory");
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        return reinterpret_cast<const float2*>(d);
    }
    __device__ __forceinline__ static void tables_ready() {
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
    }
    // Natural index of value r of the register side, and frequency of value r of the merged pass.
    __device__ __forceinline__ static int index(int r) { return bfly() + r * B1; }
    __device__ __forceinline__ static int freq(int r) { return bfly() + r * (R1 * R2); }
    __device__ __forceinline__ static bool act1() { return live() && bfly() < B1; }
    __device__ __forceinline__ static bool act3() { return live() && bfly() < B3; }

    // The middle pass, in place, and the barrier after it.
    template <int S> __device__ __forceinline__ static void middle(E* s, const float2* tw, int j0) {
        if constexpr (R2 > 1) {
#pragma unroll
            for (int t = 0; t < kTurns; t++) {
                const int j = j0 + t * kMaxB;
                if (live() && j < B2) {
                    const int c = j % R3, o = (j / R3) * P1 + c;
                    C v[R2];
#pragma unroll
                    for (int r = 0; r < R2; r++) v[r] = ld(&s[o + r * R3]);
                    if (S > 0) twiddle<R2, 1>(v, tw + M + c, R3);
                    rdft<R2, S, R2>(v);
                    if (S < 0) twiddle<R2, -1>(v, tw + M + c, R3);
#pragma unroll
                    for (int r = 0; r < R2; r++) st(&s[o + r * R3], v[r]);
                }
            }
            __syncthreads();
        }
    }
    // Values in registers -> the R3 spectrum values of the merged pass, x[r] at freq(r).  Starts
    // without and ends without a barrier: the caller's threads may still read only what they
    // wrote themselves (the values of the last inverse pass).
    __device__ __forceinline__ static void forward(const C (&in)[NZ], E* s, const float2* tw, C (&x)[R3]) {
        const int j = bfly();
        if (act1()) {
            C v[R1];
#pragma unroll
            for (int r = 0; r < NZ; r++) v[r] = in[r];
            rdft<R1, -1, NZ>(v);
            twiddle<R1, -1>(v, tw + j, B1);
#pragma unroll
            for (int r = 0; r < R1; r++) st(&s[j + r * P1], v[r]);
        }
        __syncthreads();
        middle<-1>(s, tw, j);
        if (act3()) {
            const int o = (j % R1) * P1 + (j / R1) * R3;
#pragma unroll
            for (int r = 0; r < R3; r++) x[r] = ld(&s[o + r]);
            rdft<R3, -1, R3>(x);
        }
    }
    // The spectrum values x[r] at freq(r) (of the threads act3()) -> values in registers.
    __device__ __forceinline__ static void inverse(C (&x)[R3], E* s, const float2* tw, C (&out)[NZ]) {
        const int j = bfly();
        if (act3()) {
            const int o = (j % R1) * P1 + (j / R1) * R3;
            rdft<R3, 1, R3>(x);
#pragma unroll
            for (int r = 0; r < R3; r++) st(&s[o + r], x[r]);
        }
        __syncthreads();
        middle<1>(s, tw, j);
        if (act1()) {
            C v[R1];
#pragma unroll
            for (int r = 0; r < R1; r++) v[r] = ld(&s[j + r * P1]);
            twiddle<R1, 1>(v, tw + j, B1);
            rdft<R1, 1, R1>(v);
#pragma unroll
            for (int r = 0; r < NZ; r++) out[r] = v[r];
        }
    }
    // v <- F^-1[H . F v] with a complex multiplier H of length M (1/M folded in).
    __device__ __forceinline__ static void roundtrip(C (&v)[NZ], E* s, const float2* tw,
                                                     const float2* __restrict__ H) {
        C x[R3];
        forward(v, s, tw, x);
        if (act3()) {
#pragma unroll
            for (int r = 0; r < R3; r++) {
                const float2 h = __ldg(&H[freq(r)]);
                x[r] = cmulw(x[r], h.x, h.y);
            }
        }
        inverse(x, s, tw, v);
    }
};

}  // namespace qp
