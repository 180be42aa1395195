// rt_kernels.cuh -- the x passes on the register-to-register line transforms
// (line_rt.cuh): the same steps as ac_xpass_kernel (ac_kernels.cuh) and the
// x-spectral convolution passes (vz_kernels.cuh), with the fields going from HBM
// straight into the first pass's registers and from the last pass's registers
// through the update back to HBM.  Only the transforms themselves touch shared
// memory, and consecutive operators chain in registers.
#pragma once
#include "line_rt.cuh"
#include "pass_common.cuh"

namespace qp {

// The value of a thread of an x pass is one row of its 2W columns: W = 2 packs
// columns (0, 1) and (2, 3) as the real and imaginary parts of its two lines.
// V: the rows are aligned for one vector access (nzz a multiple of 2W, aligned
// buffers); else the columns below nc are accessed one by one.
template <bool V> __device__ __forceinline__ Cx<float> ld_cols(const float* __restrict__ f, unsigned i, int nc, Cx<float>*) {
    if (V) {
        const float2 t = *reinterpret_cast<const float2*>(f + i);
        return {t.x, t.y};
    }
    return {f[i], nc > 1 ? f[i + 1] : 0.f};
}
template <bool V> __device__ __forceinline__ Cx<float2> ld_cols(const float* __restrict__ f, unsigned i, int nc, Cx<float2>*) {
    if (V) {
        const float4 t = *reinterpret_cast<const float4*>(f + i);
        return {make_float2(t.x, t.y), make_float2(t.z, t.w)};
    }
    return {make_float2(f[i], nc > 1 ? f[i + 1] : 0.f), make_float2(nc > 2 ? f[i + 2] : 0.f, nc > 3 ? f[i + 3] : 0.f)};
}
template <bool V> __device__ __forceinline__ void st_cols(float* f, unsigned i, int nc, Cx<float> c) {
    if (V) {
        *reinterpret_cast<float2*>(f + i) = make_float2(c.x, c.y);
    } else {
        f[i] = c.x;
        if (nc > 1) f[i + 1] = c.y;
    }
}
template <bool V> __device__ __forceinline__ void st_cols(float* f, unsigned i, int nc, Cx<float2> c) {
    if (V) {
        *reinterpret_cast<float4*>(f + i) = make_float4(c.x.x, c.x.y, c.y.x, c.y.y);
    } else {
        f[i] = c.x.x;
        if (nc > 1) f[i + 1] = c.x.y;
        if (nc > 2) f[i + 2] = c.y.x;
        if (nc > 3) f[i + 3] = c.y.y;
    }
}
// column c of a row value
__device__ __forceinline__ float& col(Cx<float>& v, int c) { return c ? v.y : v.x; }
__device__ __forceinline__ float& col(Cx<float2>& v, int c) { return c == 0 ? v.x.x : c == 1 ? v.x.y : c == 2 ? v.y.x : v.y.y; }
// a b + c and a s + b t over the columns
template <class T> __device__ __forceinline__ Cx<T> rfma(Cx<T> a, Cx<T> b, Cx<T> c) {
    return {vfma(a.x, b.x, c.x), vfma(a.y, b.y, c.y)};
}
template <class T> __device__ __forceinline__ Cx<T> rmix(float s, Cx<T> a, float t, Cx<T> b) {
    const T vs = bcast<T>(s), vt = bcast<T>(t);
    return {vfma(vs, a.x, vmul(vt, b.x)), vfma(vs, a.y, vmul(vt, b.y))};
}
__device__ __forceinline__ float vneg(float a) { return -a; }
__device__ __forceinline__ float2 vneg(float2 a) { return make_float2(-a.x, -a.y); }

// Points of an epilogue loop whose loads are in flight together: as many as LR::kEpiRegs
// registers hold of F fields' values.
template <class LR> constexpr int rt_batch(int F) {
    const int u = LR::kEpiRegs / (F * 2 * LR::W);
    return u < 1 ? 1 : u > LR::NZ ? LR::NZ : u;
}
// use(r, ix, i, load(i, ix)) for this thread's rows r (ix = index(r) < n), the loads of U
// rows in flight before the first use.  Offsets are 32 bits: the windows these passes run (up to
// 4608 points wide and, with z on a Stockham plan, up to 6561 deep) stay far below 2^32 elements.
template <class LR, int U, class LoadF, class UseF>
__device__ __forceinline__ void rt_rows(int n, unsigned pitch, unsigned off, bool on, LoadF&& load, UseF&& use) {
    using In = decltype(load(off, 0));
#pragma unroll
    for (int r0 = 0; r0 < LR::NZ; r0 += U) {
        In t[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int ix = LR::index(r0 + u);
            if (r0 + u < LR::NZ && on && ix < n) t[u] = load((unsigned)ix * pitch + off, ix);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int ix = LR::index(r0 + u);
            if (r0 + u < LR::NZ && on && ix < n) use(r0 + u, ix, (unsigned)ix * pitch + off, t[u]);
        }
    }
}

// ---- x pass -----------------------------------------------------------------------------
// Bound by the transforms' FP32 and shared-memory work.  Rows of the
// blocked fields are contiguous over the tile's threads.
template <bool P, bool V, class LR>
__device__ __forceinline__ void rt_xpass(const AcXArgs& a, float4* smem) {
    using C = typename LR::C;
    using T = typename LR::T;
    constexpr int NC = 2 * LR::W, NZ = LR::NZ;
    constexpr C* kC = nullptr;
    typename LR::E* s = LR::base(smem);
    const int nxx = a.nxx, nzz = a.nzz;
    const unsigned rs = a.rs;
    const int iz0 = (blockIdx.x * LR::G + LR::group()) * NC;
    const int nc = min(nzz - iz0, NC);
    const unsigned o0 = (unsigned)(iz0 >> 2) * a.sb + (iz0 & 3);  // point (0, iz0)
    const bool on = LR::act1() && nc > 0;
    const float2* tw = LR::tables(smem, a.pl.w);
    rt_wait();
    C v[NZ];
#pragma unroll
    for (int r = 0; r < NZ; r++) v[r] = czero<T>();
    // the padding of the next operator's input (a roundtrip leaves the tail of its
    // convolution there)
    auto clip = [&]() {
#pragma unroll
        for (int r = 0; r < NZ; r++)
            if (LR::index(r) >= nxx) v[r] = czero<T>();
    };
    auto fill = [&](const float* f) {
        rt_rows<LR, NZ>(nxx, rs, o0, on, [&](unsigned i, int) { return ld_cols<V>(f, i, nc, kC); },
                        [&](int r, int, unsigned, const C& c) { v[r] = c; });
    };
    if (P) {
        fill(a.div);
        LR::tables_ready();
        LR::roundtrip(v, s, tw, a.kx2);
        struct In {
            C lz, p0, c1, c2, dv;
        };
        const int cs = a.zs - iz0;
        rt_rows<LR, rt_batch<LR>(5)>(
            nxx, rs, o0, on,
            [&](unsigned i, int) {
                return In{ld_cols<V>(a.Lz, i, nc, kC), ld_cols<V>(a.p, i, nc, kC), ld_cols<V>(a.c1, i, nc, kC),
                          ld_cols<V>(a.c2, i, nc, kC), ld_cols<V>(a.div, i, nc, kC)};
            },
            [&](int r, int ix, unsigned i, const In& t) {
                const C lap = v[r] + t.lz;
                const C w{vfma(vneg(t.c2.x), lap.x, t.dv.x), vfma(vneg(t.c2.y), lap.y, t.dv.y)};
                C pn = rfma(t.c1, w, t.p0);
                if (ix == a.xs) {
#pragma unroll
                    for (int c = 0; c < NC; c++)
                        if (c == cs) col(pn, c) += a.src;
                }
                v[r] = pn;
            });
        clip();
        // receivers of this tile: record (source side) or inject (receiver side), through the
        // line buffer (which the other threads may still be reading)
        if (a.rec_off) {
            const int q0 = a.rec_off[blockIdx.x], q1 = a.rec_off[blockIdx.x + 1];
            if (q1 > q0) {
                __syncthreads();
                if (on)
#pragma unroll
                    for (int r = 0; r < NZ; r++)
                        if (LR::index(r) < nxx) LR::st(&s[LR::index(r)], v[r]);
                __syncthreads();
                float* sf = reinterpret_cast<float*>(smem);
                const int it0 = blockIdx.x * LR::G * NC;
                for (int q = q0 + threadIdx.x; q < q1; q += LR::kThreads) {
                    const RecEntry e = a.rec[q];
                    const int rel = e.gz - it0;
                    float* at = sf + ((size_t)(rel / NC) * LR::kElems + e.gx) * NC + rel % NC;
                    if (a.gather_row) a.gather_row[e.ir] = *at;
                    if (a.obs_row && e.inject) *at = a.obs_row[e.ir];
                }
                __syncthreads();
                if (on)
#pragma unroll
                    for (int r = 0; r < NZ; r++)
                        if (LR::index(r) < nxx) v[r] = LR::ld(&s[LR::index(r)]);
                __syncthreads();
            }
        }
#pragma unroll
        for (int r = 0; r < NZ; r++)
            if (on && LR::index(r) < nxx) st_cols<V>(a.p, (unsigned)LR::index(r) * rs + o0, nc, v[r]);
        if (a.ssg || a.img) {
            // illumination or image (a step has one of them): Kahan pairs over the grid's layout,
            // of which the interior is read in the end
            float* sum = a.ssg ? a.ssg : a.img;
            float* cmp = a.ssg ? a.ssg_c : a.img_c;
            struct Acc {
                C s, sc, ps;
            };
            rt_rows<LR, rt_batch<LR>(3)>(
                nxx, rs, o0, on,
                [&](unsigned i, int) {
                    return Acc{ld_cols<V>(sum, i, nc, kC), ld_cols<V>(cmp, i, nc, kC), a.img ? ld_cols<V>(a.ps, i, nc, kC) : czero<T>()};
                },
                [&](int r, int, unsigned i, const Acc& t) {
                    const C w = a.img ? t.ps : v[r];
                    const C y{vfma(w.x, v[r].x, vneg(t.sc.x)), vfma(w.y, v[r].y, vneg(t.sc.y))};
                    const C sm = t.s + y;
                    st_cols<V>(sum, i, nc, sm);
                    st_cols<V>(cmp, i, nc, (sm - t.s) - y);
                });
        }
    } else if (a.do_v) {
        fill(a.p);
        LR::tables_ready();
    } else {
        fill(a.vx);
        LR::tables_ready();
    }
    if (a.do_v) {
        if (!a.do_dx) rt_release();
        LR::roundtrip(v, s, tw, a.HxP);
        struct In {
            C pp, v0, bb;
            float hb, ha;
        };
        rt_rows<LR, rt_batch<LR>(3)>(
            nxx, rs, o0, on,
            [&](unsigned i, int ix) {
                return In{ld_cols<V>(a.psi_px, i, nc, kC), ld_cols<V>(a.vx, i, nc, kC), ld_cols<V>(a.bbx, i, nc, kC),
                          __ldg(&a.h_bx[ix]), __ldg(&a.h_ax[ix])};
            },
            [&](int r, int, unsigned i, const In& t) {
                const C ps = rmix(t.hb, t.pp, t.ha, v[r]);
                st_cols<V>(a.psi_px, i, nc, ps);
                const T dt = bcast<T>(a.dt);
                v[r] = rfma(C{vmul(dt, t.bb.x), vmul(dt, t.bb.y)}, v[r] + ps, t.v0);
                st_cols<V>(a.vx, i, nc, v[r]);
            });
        clip();
    } else if (P && a.do_dx) {
        fill(a.vx);
    }
    if (a.do_dx) {
        rt_release();
        LR::roundtrip(v, s, tw, a.HxM);
        struct In {
            C pv;
            float ib, ia;
        };
        rt_rows<LR, rt_batch<LR>(1)>(
            nxx, rs, o0, on,
            [&](unsigned i, int ix) {
                return In{ld_cols<V>(a.psi_vx, i, nc, kC), __ldg(&a.i_bx[ix]), __ldg(&a.i_ax[ix])};
            },
            [&](int r, int, unsigned i, const In& t) {
                const C ps = rmix(t.ib, t.pv, t.ia, v[r]);
                st_cols<V>(a.psi_vx, i, nc, ps);
                st_cols<V>(a.Dx, i, nc, v[r] + ps);
            });
    }
}
template <bool P, class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_xpass_kernel(AcXArgs a) {
    extern __shared__ float4 rt_smem[];
    if (a.vec) rt_xpass<P, true, LR>(a, rt_smem);
    else rt_xpass<P, false, LR>(a, rt_smem);
}

// ---- x-spectral passes: stationary symbols as per-kz convolutions --------------------------
// W kz columns per group (the pitch of the half spectra is even, so a pair is one
// 16-byte access); out_b = F^-1[tab_b . F in] for NOUT outputs.  With more than one
// output the spectrum waits in a second buffer, each thread reading back its own values.
template <int W> __device__ __forceinline__ Cx<typename LineVal<W>::T> ld_spec(const float2* __restrict__ f);
template <> __device__ __forceinline__ Cx<float> ld_spec<1>(const float2* __restrict__ f) {
    const float2 t = *f;
    return {t.x, t.y};
}
template <> __device__ __forceinline__ Cx<float2> ld_spec<2>(const float2* __restrict__ f) {
    const float4 t = *reinterpret_cast<const float4*>(f);
    return {make_float2(t.x, t.z), make_float2(t.y, t.w)};
}
__device__ __forceinline__ void st_spec(float2* f, Cx<float> c) { *f = make_float2(c.x, c.y); }
__device__ __forceinline__ void st_spec(float2* f, Cx<float2> c) {
    *reinterpret_cast<float4*>(f) = make_float4(c.x.x, c.y.x, c.x.y, c.y.y);
}
template <int W> __device__ __forceinline__ typename LineVal<W>::T ld_tab(const float* __restrict__ t, int mh2) {
    if constexpr (W == 1) return __ldg(t);
    else return make_float2(__ldg(t), __ldg(t + mh2));
}

// MANY: more than one output (the spectrum is kept).
template <bool MANY, class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_xconv_kernel(XconvArgs a) {
    extern __shared__ float4 rt_smem[];
    using C = typename LR::C;
    typename LR::E* s = LR::base(rt_smem);
    const float2* tw = LR::tables(rt_smem, a.pl.w);
    rt_wait();
    typename LR::E* X = reinterpret_cast<typename LR::E*>(reinterpret_cast<char*>(rt_smem) + LR::kSmem) + LR::group() * LR::M;
    const int nxx = a.nxx, nzh = a.nzh;
    const int kz0 = (blockIdx.x * LR::G + LR::group()) * LR::W;
    const unsigned o0 = (unsigned)(kz0 >> 1) * a.ssb + (kz0 & 1);
    const bool on = LR::act1() && kz0 < nzh;
    // rows of the even halves of the multipliers; past the last column the last one's
    constexpr int mh = LR::M / 2 + 1;
    const int kt = min(kz0, nzh - 1), d2 = (kz0 + 1 < nzh) ? mh : 0;
    C v[LR::NZ], x[LR::R3];
#pragma unroll
    for (int r = 0; r < LR::NZ; r++) v[r] = czero<typename LR::T>();
    rt_rows<LR, LR::NZ>(nxx, a.srs, o0, on, [&](unsigned i, int) { return ld_spec<LR::W>(a.in + i); },
                        [&](int r, int, unsigned, const C& c) { v[r] = c; });
    LR::tables_ready();
    LR::forward(v, s, tw, x);
    if (MANY && LR::act3()) {
#pragma unroll
        for (int r = 0; r < LR::R3; r++) LR::st(&X[LR::freq(r)], x[r]);
    }
#pragma unroll 1
    for (int b = 0; b < (MANY ? a.nout : 1); b++) {
        // a zero the compiler does not know: keeps it from holding the loop's offsets (rows and
        // multiplier entries) in registers across the transforms
        unsigned z = 0;
        if (MANY) asm volatile("mov.u32 %0, 0;" : "=r"(z));
        const float* tk = a.tab + b * a.tab_step + (size_t)kt * mh;
        if (LR::act3()) {
#pragma unroll
            for (int r = 0; r < LR::R3; r++) {
                const int f = LR::freq(r) + z;
                if (MANY) x[r] = LR::ld(&X[f]);
                x[r] = cmuls(x[r], ld_tab<LR::W>(tk + min(f, LR::M - f), d2));
            }
        }
        if (MANY && b > 0) __syncthreads();  // the last output's values have been read
        if (b + 1 == (MANY ? a.nout : 1)) rt_release();
        LR::inverse(x, s, tw, v);
        float2* out = a.out + b * a.out_step;
        rt_rows<LR, LR::NZ>(nxx + z, a.srs + z, o0, on, [&](unsigned, int) { return 0; },
                            [&](int r, int, unsigned i, int) { st_spec(out + i, v[r]); });
    }
}

// ---- exact DFTs of a length n on the entry's padded length (Bluestein) ------------------------
// The DFT is chirp . conv(chirp . x): one roundtrip with the transform of the wrapped
// conjugate chirp (a.bhat) as the multiplier.  Values stay at index(r), here frequencies.
template <int S, class LR>
__device__ __forceinline__ void rt_blue(typename LR::C (&v)[LR::NZ], typename LR::E* s, const FFTPlanDev& pl, const float2* tw) {
    auto chirp = [&]() {
#pragma unroll
        for (int r = 0; r < LR::NZ; r++)
            if (LR::act1() && LR::index(r) < pl.n) {
                const float2 c = __ldg(&pl.chirp[LR::index(r)]);
                v[r] = cmulw(v[r], c.x, c.y);
            } else {
                v[r] = czero<typename LR::T>();
            }
    };
    // inverse = conj(DFT(conj(x)))
    if (S > 0)
#pragma unroll
        for (int r = 0; r < LR::NZ; r++) v[r].y = vneg(v[r].y);
    chirp();
    LR::roundtrip(v, s, tw, pl.bhat);
    chirp();
    if (S > 0)
#pragma unroll
        for (int r = 0; r < LR::NZ; r++) v[r].y = vneg(v[r].y);
}

// One output with a symbol that changes in time (the stabilised Q-RTM filter).
template <class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_xexact_kernel(VxsArgs a) {
    extern __shared__ float4 rt_smem[];
    using T = typename LR::T;
    const float2* tw = LR::tables(rt_smem, a.pl.w);
    rt_wait();
    typename LR::E* s = LR::base(rt_smem);
    const int kz0 = (blockIdx.x * LR::G + LR::group()) * LR::W;
    const unsigned o0 = (unsigned)(kz0 >> 1) * a.ssb + (kz0 & 1);
    const bool on = LR::act1() && kz0 < a.nzh;
    typename LR::C v[LR::NZ];
#pragma unroll
    for (int r = 0; r < LR::NZ; r++) v[r] = czero<T>();
    rt_rows<LR, LR::NZ>(a.nxx, a.srs, o0, on, [&](unsigned i, int) { return ld_spec<LR::W>(a.in + i); },
                        [&](int r, int, unsigned, const typename LR::C& c) { v[r] = c; });
    LR::tables_ready();
    rt_blue<-1, LR>(v, s, a.pl, tw);
    rt_rows<LR, 1>(a.nxx, a.srs, o0, on, [&](unsigned, int ix) { return __ldg(&a.kx2[ix]); },
                   [&](int r, int, unsigned, float kx2) {
                       T sy = bcast<T>(spec_symbol(a, 0, kx2 + a.kz2[kz0]) * a.norm);
                       if constexpr (LR::W == 2)
                           sy.y = spec_symbol(a, 0, kx2 + a.kz2[min(kz0 + 1, a.nzz - 1)]) * a.norm;
                       v[r] = cmuls(v[r], sy);
                   });
    rt_release();
    rt_blue<1, LR>(v, s, a.pl, tw);
    rt_rows<LR, LR::NZ>(a.nxx, a.srs, o0, on, [&](unsigned, int) { return 0; },
                        [&](int r, int, unsigned i, int) { st_spec(a.out0 + i, v[r]); });
}

}  // namespace qp
