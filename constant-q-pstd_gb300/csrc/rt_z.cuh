// rt_z.cuh -- the z passes on the register-to-register line transforms (line_rt.cuh): the
// same steps as ac_zpass_kernel (ac_kernels.cuh) and the z passes of the constant-Q step
// (vz_kernels.cuh).
//
// A line packs the two x rows of its group's pair as real and imaginary parts.  Point (ix, iz)
// of a field that both directions touch (p, Dx; acoustic also div, Lz) sits at (iz / 4) sb +
// iz % 4 + ix rs: blocked (rs = 4, sb = 4 nxx), where an x pass's rows are contiguous and a CTA
// of 4 z rows touches 64-byte pieces, or row by row (rs = nzz, sb = 4).  The fields of one
// direction lie its way: the x pass's blocked, the z passes' row by row (rz = nzz).  Measured
// with every field row by row: the x passes of a 1678 x 660 shot 45 against 32 us, 2461 x 860
// 161 against 94; with every field blocked the z passes lose more than that.  Half spectra:
// (ix, kz) at (kz / 2) ssb + kz % 2 + ix srs, blocked likewise.
#pragma once
#include "rt_kernels.cuh"

namespace qp {

// Two rows of a field at address i of the first, nr of them on the grid.  Loads take rs = 0 when
// the second is not (it then repeats the first one, which keeps its line finite).
__device__ __forceinline__ Cx<float> ld_rows(const float* __restrict__ f, unsigned i, unsigned rs) {
    return {f[i], f[i + rs]};
}
__device__ __forceinline__ void st_rows(float* f, unsigned i, unsigned rs, int nr, Cx<float> c) {
    f[i] = c.x;
    if (nr > 1) f[i + rs] = c.y;
}

// A thread's share of a z pass: its rows, and the loops over its points.
template <class LR> struct ZRows {
    static_assert(LR::W == 1, "a group's line holds one pair of rows");
    using C = typename LR::C;
    static constexpr int NR = 2, NZ = LR::NZ;
    int n, x0, nr;
    unsigned rs, sb, rz;   // strides
    unsigned ls, lz;       // row strides of loads (0 when rows are missing)
    unsigned a0, o0;       // this thread's point 0: in the shared fields, in the z passes' own
    bool on;               // this thread holds points of rows on the grid
    __device__ __forceinline__ ZRows(int nxx, int nzz, unsigned rs_, unsigned sb_, unsigned rz_) {
        n = nzz;
        x0 = (blockIdx.x * LR::G + LR::group()) * NR;
        nr = min(nxx - x0, NR);
        rs = rs_;
        sb = sb_;
        rz = rz_;
        ls = nr == NR ? rs : 0;
        lz = nr == NR ? rz : 0;
        on = LR::act1() && nr > 0;
        const unsigned j = LR::bfly();
        a0 = (j >> 2) * sb + (j & 3) + (unsigned)x0 * rs;
        o0 = j + (unsigned)x0 * rz;
    }
    // does point r lie on the line?
    __device__ __forceinline__ bool has(int r) const { return on && (!LR::kPad || LR::index(r) < n); }
    // its address in the shared fields (steps of whole blocks: B1 a multiple of 4), in the own ones
    __device__ __forceinline__ unsigned at(int r) const {
        if constexpr (LR::B1 % 4 == 0) return a0 + (unsigned)(r * (LR::B1 / 4)) * sb;
        const unsigned q = LR::index(r);
        return (q >> 2) * sb + (q & 3) + (unsigned)x0 * rs;
    }
    __device__ __forceinline__ unsigned own(int r) const { return o0 + r * LR::B1; }
    __device__ __forceinline__ C ld(const float* f, unsigned i) const { return ld_rows(f, i, ls); }
    __device__ __forceinline__ void st(float* f, unsigned i, C c) const { st_rows(f, i, rs, nr, c); }
    __device__ __forceinline__ C ldo(const float* f, unsigned i) const { return ld_rows(f, i, lz); }
    __device__ __forceinline__ void sto(float* f, unsigned i, C c) const { st_rows(f, i, rz, nr, c); }
    // use(r, q, i, o, load(i, o, q)) for this thread's points q = index(r), their addresses i in the
    // shared fields and o in the z passes' own; F: fields load reads
    template <int F, class LoadF, class UseF> __device__ __forceinline__ void each(LoadF&& load, UseF&& use) const {
        using In = decltype(load(0u, 0u, 0));
        constexpr int U = rt_batch<LR>(F);
#pragma unroll
        for (int r0 = 0; r0 < NZ; r0 += U) {
            In t[U];
#pragma unroll
            for (int u = 0; u < U; u++)
                if (r0 + u < NZ && has(r0 + u)) t[u] = load(at(r0 + u), own(r0 + u), LR::index(r0 + u));
#pragma unroll
            for (int u = 0; u < U; u++)
                if (r0 + u < NZ && has(r0 + u)) use(r0 + u, LR::index(r0 + u), at(r0 + u), own(r0 + u), t[u]);
        }
    }
    // O: the z passes' own field
    template <bool O> __device__ __forceinline__ void fill(C (&v)[NZ], const float* f) const {
#pragma unroll
        for (int r = 0; r < NZ; r++)
            v[r] = has(r) ? (O ? ldo(f, own(r)) : ld(f, at(r))) : czero<typename LR::T>();
    }
    template <bool O> __device__ __forceinline__ void put(const C (&v)[NZ], float* f) const {
#pragma unroll
        for (int r = 0; r < NZ; r++)
            if (has(r)) {
                if (O) sto(f, own(r), v[r]);
                else st(f, at(r), v[r]);
            }
    }
    // zeros in the padding (a roundtrip leaves the tail of its convolution there)
    __device__ __forceinline__ void clip(C (&v)[NZ]) const {
        if constexpr (LR::kPad) {
#pragma unroll
            for (int r = 0; r < NZ; r++)
                if (LR::index(r) >= n) v[r] = czero<typename LR::T>();
        }
    }
};

// Exact length-n DFTs of the rows' lines: spectrum values x[r] at freq(r), on the entry's own
// length or by Bluestein's identity on a padded one (values then stay where the points are).
template <class LR> struct ZDft {
    using C = typename LR::C;
    static constexpr int NS = LR::kPad ? LR::NZ : LR::R3;
    __device__ __forceinline__ static int freq(int r) { return LR::kPad ? LR::index(r) : LR::freq(r); }
    __device__ __forceinline__ static bool act(int r, int n) { return LR::kPad ? LR::act1() && LR::index(r) < n : LR::act3(); }
    __device__ __forceinline__ static void forward(C (&v)[LR::NZ], typename LR::E* s, const FFTPlanDev& pl, const float2* tw, C (&x)[NS]) {
        if constexpr (LR::kPad) {
#pragma unroll
            for (int r = 0; r < NS; r++) x[r] = v[r];
            rt_blue<-1, LR>(x, s, pl, tw);
        } else {
            LR::forward(v, s, tw, x);
        }
    }
    __device__ __forceinline__ static void inverse(C (&x)[NS], typename LR::E* s, const FFTPlanDev& pl, const float2* tw, C (&v)[LR::NZ]) {
        if constexpr (LR::kPad) {
#pragma unroll
            for (int r = 0; r < NS; r++) v[r] = x[r];
            rt_blue<1, LR>(v, s, pl, tw);
        } else {
            LR::inverse(x, s, tw, v);
        }
    }
    // Two real rows a, b share a line z = a + ib: A(k) = (Z(k) + conj Z(n-k))/2,
    // B(k) = (Z(k) - conj Z(n-k))/(2i), and back Z(k) = A(k) + iB(k).
    // x <- half spectra of the rows
    __device__ __forceinline__ static void load(C (&x)[NS], const ZRows<LR>& z, const float2* __restrict__ S, int nzh,
                                                unsigned srs, unsigned ssb) {
#pragma unroll
        for (int r = 0; r < NS; r++) {
            x[r] = czero<typename LR::T>();
            if (!act(r, z.n) || z.nr <= 0) continue;
            const int f = freq(r), k = f < nzh ? f : z.n - f;
            const float sg = f < nzh ? 1.f : -1.f;
            const unsigned i = (unsigned)(k >> 1) * ssb + (k & 1) + (unsigned)z.x0 * srs;
            const unsigned rs = z.nr == ZRows<LR>::NR ? srs : 0;  // a missing row repeats the first
            const float2 a = S[i], b = S[i + rs];
            x[r] = {fmaf(-sg, b.y, a.x), fmaf(sg, a.y, b.x)};
        }
    }
    // half spectra of the rows <- x, through the line buffer (barriers before, between and after)
    __device__ __forceinline__ static void store(const C (&x)[NS], typename LR::E* s, const ZRows<LR>& z, float2* S, int nzh,
                                                 unsigned srs, unsigned ssb) {
        __syncthreads();
#pragma unroll
        for (int r = 0; r < NS; r++)
            if (act(r, z.n)) LR::st(&s[freq(r)], x[r]);
        __syncthreads();
        if (LR::live() && z.nr > 0)
            for (int k = 2 * LR::bfly(); k < nzh; k += 2 * LR::kMaxB) {
                // columns k and k + 1 of every row, one 16-byte store each
                const C p0 = LR::ld(&s[k]), p1 = LR::ld(&s[k + 1]);
                const C q0 = LR::ld(&s[k ? z.n - k : 0]), q1 = LR::ld(&s[z.n - k - 1]);
                const typename LR::T h = bcast<typename LR::T>(0.5f);
                const C a0{vmul(vadd(p0.x, q0.x), h), vmul(vsub(p0.y, q0.y), h)}, b0{vmul(vadd(p0.y, q0.y), h), vmul(vsub(q0.x, p0.x), h)};
                const C a1{vmul(vadd(p1.x, q1.x), h), vmul(vsub(p1.y, q1.y), h)}, b1{vmul(vadd(p1.y, q1.y), h), vmul(vsub(q1.x, p1.x), h)};
                float2* o = S + ((unsigned)(k >> 1) * ssb + (unsigned)z.x0 * srs);
                auto put = [&](int row, float e0, float e1, float e2, float e3) {
                    if (row < z.nr) *reinterpret_cast<float4*>(o + row * srs) = make_float4(e0, e1, e2, e3);
                };
                put(0, a0.x, a0.y, a1.x, a1.y);
                put(1, b0.x, b0.y, b1.x, b1.y);
            }
        __syncthreads();
    }
};

// dt b (d + psi) with the memory variable psi <- hb psi + ha d: the velocity updates
#define RT_Z_SETUP                                                          \
    extern __shared__ float4 rt_smem[];                                     \
    using C = typename LR::C;                                               \
    using T = typename LR::T;                                               \
    typename LR::E* s = LR::base(rt_smem);                                  \
    const ZRows<LR> z(a.nxx, a.nzz, a.rs, a.sb, a.rz);                            \
    const float2* tw = LR::tables(rt_smem, a.pl.w);                         \
    rt_wait();                                                              \
    C v[LR::NZ];

// vz <- vz + dt bbz (d + psi), v <- the new vz
template <class LR, class A>
__device__ __forceinline__ void rt_z_vupdate(const A& a, const ZRows<LR>& z, typename LR::C (&v)[LR::NZ]) {
    using C = typename LR::C;
    using T = typename LR::T;
    struct In {
        C pp, v0, bb;
        float hb, ha;
    };
    z.template each<3>([&](unsigned, unsigned o, int q) { return In{z.ldo(a.psi_pz, o), z.ldo(a.vz, o), z.ldo(a.bbz, o), __ldg(&a.h_bz[q]), __ldg(&a.h_az[q])}; },
           [&](int r, int, unsigned, unsigned o, const In& t) {
               const C ps = rmix(t.hb, t.pp, t.ha, v[r]);
               z.sto(a.psi_pz, o, ps);
               const T dt = bcast<T>(a.dt);
               v[r] = rfma(C{vmul(dt, t.bb.x), vmul(dt, t.bb.y)}, v[r] + ps, t.v0);
               z.sto(a.vz, o, v[r]);
           });
}
// div <- Dx + d + psi, v <- div (O: div is the z passes' own)
template <bool O, class LR, class A>
__device__ __forceinline__ void rt_z_div(const A& a, const ZRows<LR>& z, typename LR::C (&v)[LR::NZ]) {
    using C = typename LR::C;
    struct In {
        C pv, dx;
        float ib, ia;
    };
    z.template each<2>([&](unsigned i, unsigned o, int q) { return In{z.ldo(a.psi_vz, o), z.ld(a.Dx, i), __ldg(&a.i_bz[q]), __ldg(&a.i_az[q])}; },
           [&](int r, int, unsigned i, unsigned o, const In& t) {
               const C ps = rmix(t.ib, t.pv, t.ia, v[r]);
               z.sto(a.psi_vz, o, ps);
               v[r] = t.dx + (v[r] + ps);
               if (O) z.sto(a.div, o, v[r]);
               else z.st(a.div, i, v[r]);
           });
}

// ---- acoustic z pass -----------------------------------------------------------------------
template <class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_zpass_kernel(AcZArgs a) {
    RT_Z_SETUP
    (void)sizeof(T);
    if (a.do_v) {
        z.template fill<false>(v, a.p);
        LR::tables_ready();
        LR::roundtrip(v, s, tw, a.HzP);
        rt_z_vupdate<LR>(a, z, v);
        z.clip(v);
    } else {
        z.template fill<true>(v, a.vz);
        LR::tables_ready();
    }
    if (!a.do_div) return;
    LR::roundtrip(v, s, tw, a.HzM);
    rt_z_div<false, LR>(a, z, v);
    z.clip(v);
    rt_release();
    LR::roundtrip(v, s, tw, a.kz2);
    z.template put<false>(v, a.Lz);
}

// ---- constant-Q z passes --------------------------------------------------------------------
template <class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_passA_kernel(VzArgsA a) {
    RT_Z_SETUP
    (void)sizeof(T);
    using D = ZDft<LR>;
    C x[D::NS];
    if (a.aux_spec) {
        D::load(x, z, a.aux_spec, a.nzh, a.srs, a.ssb);
        LR::tables_ready();
        D::inverse(x, s, a.pl, tw, v);
        z.template put<true>(v, a.aux);
    }
    z.template fill<true>(v, a.vz);
    if (!a.aux_spec) LR::tables_ready();
    LR::roundtrip(v, s, tw, a.HzM);
    rt_z_div<true, LR>(a, z, v);
    z.clip(v);
    rt_release();
    D::forward(v, s, a.pl, tw, x);
    D::store(x, s, z, a.G, a.nzh, a.srs, a.ssb);
}

// The running total waits in a second buffer, where each thread reads back its own values.
template <class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_passB_kernel(VzArgsB a) {
    RT_Z_SETUP
    using D = ZDft<LR>;
    typename LR::E* acc = reinterpret_cast<typename LR::E*>(reinterpret_cast<char*>(rt_smem) + LR::kSmem) + LR::group() * LR::kElems;
    C x[D::NS];
#pragma unroll 1
    for (int b = 0; b < 3; b++) {
        if (b == 0) LR::tables_ready();
        else __syncthreads();  // the last term's values have been read
        D::load(x, z, b == 0 ? a.Y2 : b == 1 ? a.Y3 : a.Y4, a.nzh, a.srs, a.ssb);
        D::inverse(x, s, a.pl, tw, v);
        const float* cf = b == 0 ? a.y2 : b == 1 ? a.y3c : a.y4c;
        const T sg = bcast<T>(b == 0 ? 1.f : -1.f);
        z.template each<1>([&](unsigned, unsigned o, int) { return z.ldo(cf, o); },
               [&](int r, int q, unsigned, unsigned, const C& c) {
                   const C t = b == 0 ? czero<T>() : LR::ld(&acc[q]);
                   LR::st(&acc[q], rfma(C{vmul(sg, c.x), vmul(sg, c.y)}, v[r], t));
               });
    }
    struct In {
        C y1, dv;
    };
    z.template each<2>([&](unsigned, unsigned o, int) { return In{z.ldo(a.y1, o), z.ldo(a.div, o)}; },
           [&](int r, int q, unsigned, unsigned o, const In& t) {
               v[r] = rfma(t.y1, t.dv, LR::ld(&acc[q]));
               z.sto(a.total, o, v[r]);
           });
    z.clip(v);
    rt_release();
    D::forward(v, s, a.pl, tw, x);
    D::store(x, s, z, a.T, a.nzh, a.srs, a.ssb);
}

template <class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_passC_kernel(VzArgsC a) {
    RT_Z_SETUP
    using D = ZDft<LR>;
    constexpr int NR = ZRows<LR>::NR;
    C x[D::NS];
    if (a.Dspec) {
        D::load(x, z, a.Dspec, a.nzh, a.srs, a.ssb);
        LR::tables_ready();
        D::inverse(x, s, a.pl, tw, v);
    } else {
        LR::tables_ready();
#pragma unroll
        for (int r = 0; r < LR::NZ; r++) v[r] = czero<T>();
    }
    struct In {
        C p, e1, tot, e2, e3, aux;
    };
    const T sgn = bcast<T>(a.sgn);
    const int xs = a.xs - z.x0;
    z.template each<6>([&](unsigned i, unsigned o, int) { return In{z.ld(a.p, i), z.ldo(a.e1, o), z.ldo(a.total, o), z.ldo(a.e2, o), z.ldo(a.e3, o), z.ldo(a.aux, o)}; },
           [&](int r, int q, unsigned, unsigned, const In& t) {
               // p + e1 (total +- e2 D) +- e3 aux
               const C D1 = rfma(C{vmul(sgn, t.e2.x), vmul(sgn, t.e2.y)}, v[r], t.tot);
               C pn = rfma(C{vmul(sgn, t.e3.x), vmul(sgn, t.e3.y)}, t.aux, rfma(t.e1, D1, t.p));
               if (a.xs >= 0 && q == a.zs) {
#pragma unroll
                   for (int c = 0; c < NR; c++)
                       if (c == xs) col(pn, c) += a.src;
               }
               v[r] = pn;
           });
    z.clip(v);
    // receivers of this CTA's rows: record or inject, through the line buffer
    if (a.rec_off) {
        const int q0 = a.rec_off[blockIdx.x], q1 = a.rec_off[blockIdx.x + 1];
        if (q1 > q0) {
            __syncthreads();
#pragma unroll
            for (int r = 0; r < LR::NZ; r++)
                if (z.on && LR::index(r) < z.n) LR::st(&s[LR::index(r)], v[r]);
            __syncthreads();
            float* sf = reinterpret_cast<float*>(rt_smem);
            const int xt = blockIdx.x * LR::G * NR;
            for (int q = q0 + threadIdx.x; q < q1; q += LR::kThreads) {
                const RecEntry e = a.rec[q];
                const int rel = e.gx - xt;
                float* at = sf + ((size_t)(rel / NR) * LR::kElems + e.gz) * NR + rel % NR;
                if (a.gather_row) a.gather_row[e.ir] = *at;
                if (a.obs_row && e.inject) *at = a.obs_row[e.ir];
            }
            __syncthreads();
#pragma unroll
            for (int r = 0; r < LR::NZ; r++)
                if (z.on && LR::index(r) < z.n) v[r] = LR::ld(&s[LR::index(r)]);
            __syncthreads();
        }
    }
    z.template put<false>(v, a.p);
    if (a.ssg || a.img) {
        // illumination and image of the interior (Kahan pairs over the grid, row by row)
        float* sum = a.ssg ? a.ssg : a.img;
        float* cmp = a.ssg ? a.ssg_c : a.img_c;
        struct Acc {
            C s, sc, ps;
        };
        z.template each<3>([&](unsigned i, unsigned o, int) { return Acc{z.ldo(sum, o), z.ldo(cmp, o), a.img ? z.ld(a.ps, i) : czero<T>()}; },
               [&](int r, int q, unsigned, unsigned o, const Acc& t) {
                   if (q < a.pml || q >= z.n - a.pml) return;
                   const C w = a.img ? t.ps : v[r];
                   const C y{vfma(w.x, v[r].x, vneg(t.sc.x)), vfma(w.y, v[r].y, vneg(t.sc.y))};
                   const C sm = t.s + y;
                   z.sto(sum, o, sm);
                   z.sto(cmp, o, (sm - t.s) - y);
               });
    }
    rt_release();
    // half spectrum of the new p for the aux operator, and its staggered z derivative
    if constexpr (LR::kPad) {
        C w[LR::NZ];
#pragma unroll
        for (int r = 0; r < LR::NZ; r++) w[r] = v[r];
        LR::roundtrip(w, s, tw, a.HzP);
        rt_z_vupdate<LR>(a, z, w);
        D::forward(v, s, a.pl, tw, x);
        D::store(x, s, z, a.P, a.nzh, a.srs, a.ssb);
    } else {
        D::forward(v, s, a.pl, tw, x);
        D::store(x, s, z, a.P, a.nzh, a.srs, a.ssb);
        if (LR::act3()) {
#pragma unroll
            for (int r = 0; r < LR::R3; r++) {
                const float2 h = __ldg(&a.HzP[LR::freq(r)]);
                x[r] = cmulw(x[r], h.x, h.y);
            }
        }
        LR::inverse(x, s, tw, v);
        rt_z_vupdate<LR>(a, z, v);
    }
}

// psc = sum_b c_b(x) q_b(x) over row half spectra Q_b, q_b their inverse z transforms; without
// coefficients (c null) the one real field of the one spectrum.
template <class LR> __global__ void __launch_bounds__(LR::kThreads, LR::kMinB) rt_zsum_kernel(LrsArgs a) {
    RT_Z_SETUP
    using D = ZDft<LR>;
    typename LR::E* acc = reinterpret_cast<typename LR::E*>(reinterpret_cast<char*>(rt_smem) + LR::kSmem) + LR::group() * LR::kElems;
    C x[D::NS];
#pragma unroll 1
    for (int b = 0; b < a.row; b++) {
        if (b == 0) LR::tables_ready();
        else __syncthreads();  // the last factor's values have been read
        D::load(x, z, a.Q + (size_t)b * a.nxx * a.nzh, a.nzh, a.srs, a.ssb);
        D::inverse(x, s, a.pl, tw, v);
        if (!a.c) {
            z.template put<true>(v, a.psc);
            return;
        }
        const float* cb = a.c + (size_t)b * a.npts;
        z.template each<1>([&](unsigned, unsigned o, int) { return z.ldo(cb, o); },
               [&](int r, int q, unsigned, unsigned o, const C& c) {
                   const C t = rfma(c, v[r], b == 0 ? czero<T>() : LR::ld(&acc[q]));
                   if (b + 1 < a.row) LR::st(&acc[q], t);
                   else z.sto(a.psc, o, t);
               });
    }
}

}  // namespace qp
