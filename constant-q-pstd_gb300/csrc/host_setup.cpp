// host_setup.cpp -- one-time FP64 coefficient setup and line-FFT plans.
//
// The reference computes its coefficient tables on the host in float
// (sgpstd-qmodeling/funca.c, func.c); here every table is evaluated in double
// and rounded once to float.  The formulas are the reference's:
//   CPML profiles            funca.c:223-340  (get_pml_parameters)
//   half-cell shift symbols  funca.c:342-432  (cal_shift_parameters)
//   wavenumbers              funca.c:366-381 / func.c:550-585 (cal_k2d)
// including the reference's pi = 3.1415926 and its mirror index n/2*2-i for the
// negative-frequency shift phases.
#include "host_setup.h"

#include <initializer_list>
#include <memory>

#include "rt_list.h"

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstring>
#include <vector>

namespace qp {

static const double REF_PI = 3.1415926;  // funca.c:6

void pml_coeffs(int pml, double fm, int nxx, int nzz, double dx, double dz, double dt, std::vector<double>* out8) {
    const double alpha_max = REF_PI * fm, R = 1e-5, vmax = 5000.0;
    const int n1 = 2, n2 = 1, n3 = 1;
    std::vector<double> idx(nxx), idz(nzz), iax(nxx), iaz(nzz), hdx(nxx), hdz(nzz), hax(nxx), haz(nzz);
    const double dmaxx = (1 + n1 + n2) * vmax * std::log(1.0 / R) / (2.0 * pml * dx);
    const double dmaxz = (1 + n1 + n2) * vmax * std::log(1.0 / R) / (2.0 * pml * dz);
    for (int i = 0; i < pml; i++) {
        const double t1 = std::pow((double)(pml - 1 - i) / pml, n1 + n2);
        const double t3 = std::pow((double)i / (pml - 1), n3);
        idx[i] = dmaxx * t1;
        idz[i] = dmaxz * t1;
        iax[i] = alpha_max * t3;
        iaz[i] = iax[i];
        idx[nxx - 1 - i] = idx[i];
        idz[nzz - 1 - i] = idz[i];
        iax[nxx - 1 - i] = iax[i];
        iaz[nzz - 1 - i] = iaz[i];
    }
    for (int i = pml; i < nxx - pml; i++) { idx[i] = 0; iax[i] = iax[pml - 1]; }
    for (int j = pml; j < nzz - pml; j++) { idz[j] = 0; iaz[j] = iaz[pml - 1]; }
    for (int i = 0; i < pml - 1; i++) {
        const double t2 = std::pow((pml - 1.5 - i) / pml, n1 + n2);
        const double t4 = std::pow((i + 0.5) / (pml - 1), n3);
        hdx[i] = dmaxx * t2;
        hdz[i] = dmaxz * t2;
        hdx[nxx - 2 - i] = hdx[i];
        hdz[nzz - 2 - i] = hdz[i];
        hax[i] = alpha_max * t4;
        haz[i] = hax[i];
        hax[nxx - 2 - i] = hax[i];
        haz[nzz - 2 - i] = haz[i];
    }
    for (int i = pml - 1; i < nxx - pml; i++) { hdx[i] = 0; hax[i] = hax[pml - 2]; }
    hdx[nxx - 1] = 0;
    hax[nxx - 1] = hax[nxx - 2];
    for (int j = pml - 1; j < nzz - pml; j++) { hdz[j] = 0; haz[j] = haz[pml - 2]; }
    hdz[nzz - 1] = 0;
    haz[nzz - 1] = haz[nzz - 2];
    // order: i_ax, i_bx, i_az, i_bz, h_ax, h_bx, h_az, h_bz
    for (int k = 0; k < 8; k++) out8[k].assign((k % 4 < 2) ? nxx : nzz, 0.0);
    for (int i = 0; i < nxx; i++) {
        double t = idx[i] + iax[i];
        out8[1][i] = std::exp(-dt * t);
        out8[0][i] = idx[i] / t * (out8[1][i] - 1.0);
        t = hdx[i] + hax[i];
        out8[5][i] = std::exp(-dt * t);
        out8[4][i] = hdx[i] / t * (out8[5][i] - 1.0);
    }
    for (int j = 0; j < nzz; j++) {
        double t = idz[j] + iaz[j];
        out8[3][j] = std::exp(-dt * t);
        out8[2][j] = idz[j] / t * (out8[3][j] - 1.0);
        t = hdz[j] + haz[j];
        out8[7][j] = std::exp(-dt * t);
        out8[6][j] = hdz[j] / t * (out8[7][j] - 1.0);
    }
}

double wavenumber(int i, int n, double d) {
    const double dk = 2.0 * REF_PI / (n * d);
    return (i < n / 2 + 1) ? i * dk : (n - i) * dk;
}

// Reference symbol of shift_vxz_kernel / shift_pxz_kernel at index i
// (acps4.cu:1047-1108): the kernels form H = -b + i a for i < n/2+1 and
// H = b - i a above, from the table pair (a, b).
static std::complex<double> ref_symbol(double a, double b, int i, int n) {
    return (i < n / 2 + 1) ? std::complex<double>(-b, a) : std::complex<double>(b, -a);
}

void shift_symbols(int n, double d, int which, std::vector<std::complex<double>>& H, bool raw) {
    // which: 0 = "m" tables used for the velocity derivative along x
    //            (kxsmr, kxsmi) ; 1 = "c" tables used for the pressure
    //            derivative along x (kxscr, kxsci) ; 2 = z velocity derivative
    //            (kzscr, kzsci) ; 3 = z pressure derivative (kzsmr, kzsmi)
    std::vector<double> sr(n), si(n), a(n), b(n);
    const int nh = n / 2 + 1;
    for (int i = 0; i < n; i++) {
        if (i < nh) {
            const double t = i * REF_PI / n;
            sr[i] = std::cos(t);
            si[i] = std::sin(t);
        } else {
            sr[i] = sr[n / 2 * 2 - i];
            si[i] = -si[n / 2 * 2 - i];
        }
        const double k = wavenumber(i, n, d);
        switch (which) {
            case 0: a[i] = k * sr[i]; b[i] = -k * si[i]; break;  // kxsmr, kxsmi
            case 1: a[i] = k * sr[i]; b[i] = k * si[i]; break;   // kxscr, kxsci
            case 2: a[i] = k * sr[i]; b[i] = -k * si[i]; break;  // kzscr, kzsci
            default: a[i] = k * sr[i]; b[i] = k * si[i]; break;  // kzsmr, kzsmi
        }
    }
    if (raw) {
        // the reference's own symbol, as multiplied inside its 2-D C2C path
        H.assign(n, 0.0);
        for (int i = 0; i < n; i++) H[i] = ref_symbol(a[i], b[i], i, n);
        return;
    }
    // The reference keeps Re of a C2C inverse of real data, i.e. it applies the
    // Hermitian part (H(k) + conj(H(-k)))/2 of its symbol.  For odd n the
    // mirrored phases make H itself non-Hermitian, so the effective symbol is
    // formed explicitly; the 1/n of the line transform is folded in.
    H.assign(n, 0.0);
    for (int i = 0; i < n; i++) {
        const std::complex<double> h = ref_symbol(a[i], b[i], i, n);
        const int j = (n - i) % n;
        const std::complex<double> hm = ref_symbol(a[j], b[j], j, n);
        H[i] = 0.5 * (h + std::conj(hm)) / (double)n;
    }
}

// ---- FFT plans --------------------------------------------------------------
static bool smooth7(int v) {
    for (int f : {2, 3, 5, 7})
        while (v % f == 0) v /= f;
    return v == 1;
}

// Radices of the register passes (each 2..16): fewest passes first, then the
// largest smallest radix, since a pass of radix R keeps m/R threads per line
// busy (5184 -> 9,9,8,8 runs on 648 threads; 1728 -> 12,12,12 on 144), then
// the smaller largest radix (a plan with radices up to 12 runs the kernels'
// 12-entry register array, in fewer registers).
static void factor_search(int v, int maxr, std::vector<int>& cur, std::vector<int>& best) {
    if (v == 1) {
        if (best.empty() || cur.size() < best.size()) {
            best = cur;
        } else if (cur.size() == best.size()) {
            const int cmin = *std::min_element(cur.begin(), cur.end());
            const int bmin = *std::min_element(best.begin(), best.end());
            const int cmax = *std::max_element(cur.begin(), cur.end());
            const int bmax = *std::max_element(best.begin(), best.end());
            if (cmin > bmin || (cmin == bmin && cmax < bmax)) best = cur;
        }
        return;
    }
    if (!best.empty() && cur.size() + 1 > best.size()) return;
    for (int r = std::min(maxr, 16); r >= 2; r--) {
        if (v % r) continue;
        cur.push_back(r);
        factor_search(v / r, r, cur, best);  // non-increasing radices: each multiset once
        cur.pop_back();
    }
}

// Relative cost of a length whose plan has radices up to 12: the pass kernels
// then run at 48 instead of 56 registers per thread (qpstd_internal.h), which
// is worth a slightly longer transform when several lengths are admissible.
static double radix_weight(const std::vector<int>& rad) {
    return (*std::max_element(rad.begin(), rad.end()) <= 12) ? 0.85 : 1.0;
}

static bool factor_direct(int n, std::vector<int>& rad) {
    rad.clear();
    if (n > 65535) return false;
    std::vector<int> cur;
    factor_search(n, 16, cur, rad);
    if (rad.empty() || (int)rad.size() > QP_MAXST) return false;
    // odd radices first: the first pass writes at stride R, which is free of
    // shared-memory bank conflicts only for odd R (measured: -12 % step time on a
    // 1678-wide Q-RTM shot, whose 3360 = 16*15*14 convolution length runs 15,16,14)
    std::stable_partition(rad.begin(), rad.end(), [](int r) { return r % 2 == 1; });
    const int rmin = *std::min_element(rad.begin(), rad.end());
    return n / rmin <= QP_MAXTHREADS;
}

// ---- FP64 transforms of the table setup ------------------------------------------
// Stockham passes of small radices on a table of roots: the multipliers of a shot take about
// twenty transforms of the convolution lengths, which evaluated root by root (and the sums over
// the window's own DFT term by term) were most of a shot's creation.
namespace {
struct Cd {
    double x, y;
};
inline Cd mul(Cd a, Cd b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }

struct HostFFT {
    int n;
    std::vector<int> rad;
    std::vector<Cd> w, tmp;  // w[k] = e^{-2 pi i k / n}
    explicit HostFFT(int n_) : n(n_), w(n_), tmp(n_) {
        int v = n;
        for (int f : {4, 3, 5, 7, 11, 13, 2})
            for (; v % f == 0; v /= f) rad.push_back(f);
        for (int k = 0; k < n; k++) w[k] = {std::cos(2.0 * M_PI * k / n), -std::sin(2.0 * M_PI * k / n)};
    }
    // sgn -1: forward, +1: inverse, unnormalised
    void run(std::vector<Cd>& x, int sgn) {
        Cd *src = x.data(), *dst = tmp.data();
        int ns = 1;
        for (int r : rad) {
            const int nb = n / r, step = n / (ns * r), rs = n / r;
            for (int j = 0; j < nb; j++) {
                const int k = j % ns;
                Cd v[13];
                v[0] = src[j];
                for (int q = 1; q < r; q++) {
                    Cd t = w[q * k * step];
                    if (sgn > 0) t.y = -t.y;
                    v[q] = mul(src[j + q * nb], t);
                }
                Cd* o = dst + (j - k) * r + k;
                if (r == 4) {
                    const Cd a{v[0].x + v[2].x, v[0].y + v[2].y}, b{v[0].x - v[2].x, v[0].y - v[2].y};
                    const Cd c{v[1].x + v[3].x, v[1].y + v[3].y}, d{v[1].x - v[3].x, v[1].y - v[3].y};
                    o[0] = {a.x + c.x, a.y + c.y};
                    o[2 * ns] = {a.x - c.x, a.y - c.y};
                    o[ns] = {b.x - sgn * d.y, b.y + sgn * d.x};
                    o[3 * ns] = {b.x + sgn * d.y, b.y - sgn * d.x};
                    continue;
                }
                for (int q = 0; q < r; q++) {
                    Cd acc = v[0];
                    for (int u = 1; u < r; u++) {
                        Cd t = w[(u * q % r) * rs];
                        if (sgn > 0) t.y = -t.y;
                        const Cd p = mul(v[u], t);
                        acc.x += p.x;
                        acc.y += p.y;
                    }
                    o[q * ns] = acc;
                }
            }
            std::swap(src, dst);
            ns *= r;
        }
        if (src != x.data()) x.swap(tmp);
    }
};

// e^{-i pi k^2 / n} and the transform of the wrapped conjugate chirp, over m
struct Chirp {
    std::vector<Cd> c, b;
    Chirp(int n, HostFFT& f) : c(n), b(f.n, Cd{0.0, 0.0}) {
        for (long long k = 0; k < n; k++) {
            const double a = M_PI * (double)((k * k) % (2LL * n)) / (double)n;
            c[k] = {std::cos(a), -std::sin(a)};
        }
        for (int k = 0; k < n; k++) b[k] = {c[k].x, -c[k].y};
        for (int k = 1; k < n; k++) b[f.n - k] = b[k];
        f.run(b, -1);
        for (Cd& v : b) v = {v.x / f.n, v.y / f.n};
    }
};
}  // namespace

// What the tables of one plan share.
struct TableMaker {
    HostFFT f;
    Chirp ch;
    TableMaker(int n, int m) : f(m), ch(n, f) {}
};
static TableMaker& maker(const HostPlan& hp) {
    if (!hp.maker) hp.maker = std::make_shared<TableMaker>(hp.n, hp.m);
    return *hp.maker;
}

// ---- the gain of a roundtrip ------------------------------------------------------------
// The line transforms of line_rt.cuh apply the same rounded constants w forward and, conjugated,
// inverse, so that a roundtrip multiplies by |w|^2 where it should multiply by 1, the same way at
// every step: a line came out scaled by 1 - 8e-8 .. 1 + 6e-8, derivatives that much off, waves that
// much slow, with amplitudes and arrival times drifting steadily (illuminations 2e-7 - 4e-7 high
// where rounding alone leaves 1e-7).  The multipliers take the mean of it back: to first order it is
// the sum over the stages of the mean of |w|^2 - 1, each stage being unitary but for its rounding.

// |w|^2 - 1 of the float constants cos, sin(2 pi m / R)
static double root_excess(int m, int R) {
    const double c = (float)std::cos(2.0 * M_PI * m / R), s = (float)std::sin(2.0 * M_PI * m / R);
    return c * c + s * s - 1.0;
}
// of an in-register DFT of size R and its inverse (rdft, line_rt.cuh)
static double radix_gain(int R) {
    if (R <= 2 || R == 4) return 0.0;
    int p = 2;
    while (R % p) p++;
    double g = 0.0;
    if (p == R) {  // every product of the sums over q, r > 0 has a rounded root
        for (int q = 1; q < R; q++)
            for (int r = 1; r < R; r++) g += root_excess(r * q % R, R);
        return g / ((double)R * R);
    }
    const int A = (p == 2 && R % 4 == 0) ? 4 : p, B = R / A;
    for (int i = 1; i < A; i++)
        for (int q = 1; q < B; q++)
            if (4 * i * q != R) g += root_excess(i * q, R);
    return g / R + radix_gain(A) + radix_gain(B);
}
// mean of |w|^2 - 1 of n complex factors in float
static double mean_excess(const std::complex<double>* w, int n) {
    double g = 0.0;
    for (int k = 0; k < n; k++) {
        const double c = (float)w[k].real(), s = (float)w[k].imag();
        g += c * c + s * s - 1.0;
    }
    return n ? g / n : 0.0;
}

static RtEntry entry(int id, RtAxis axis, bool quick) {
    if (axis == kRtX) return rt_entry(id, quick);
    return axis == kRtZQ || (axis == kRtZ && id < kRtzVisco) ? rtz_entry(id, quick) : RtEntry{};
}

int rt_choose(int n, RtAxis axis) {
    int best = 0;
    double cost = 1e300;
    for (int id = 1; id <= std::max(kRtIds, kRtzIds); id++) {
        const RtEntry e = entry(id, axis, false);
        if (e.m && (e.pad ? e.m >= 2 * n - 1 : e.m == n) && (double)e.m * e.cost < cost) {
            cost = (double)e.m * e.cost;
            best = id;
        }
    }
    return best;
}

int rt_lines(int id, RtAxis axis, int quick) { return entry(id, axis, quick != 0).lines; }
int rt_length(int id, RtAxis axis) { return entry(id, axis, false).m; }

// The quick form where the wide one would leave SMs without a CTA (one of several lines then
// bounds the pass): fewer CTAs than the 152 SMs of the chip this is written for.  By the shot
// alone, also in a batch or server.  With the line at two CTAs per SM the 64-shot batch fell from 5.4 to 6.3 ms a
// step and the 1678 x 660 shot from 138.8 to 141.7 us; at half a CTA small grids lose up to 30 %.
int rt_quick(int id, RtAxis axis, int lines) {
    const RtEntry w = entry(id, axis, false), q = entry(id, axis, true);
    return q.m > 0 && (lines + w.lines - 1) / w.lines < 152;
}

// The smooth lengths m in [2n-1, 2.3n+8] a zero-padded convolution or a
// Bluestein transform of an n-point line can use, with their radices: the
// cheapest by pass work (extra_pass: 1 for Bluestein's two transforms per
// DFT).
static bool choose_inner_length(int n, int extra_pass, HostPlan& hp) {
    double best = 1e300;
    for (int m = 2 * n - 1; m <= (int)(2.3 * n) + 8; m++) {
        if (!smooth7(m)) continue;
        std::vector<int> r;
        if (!factor_direct(m, r)) continue;
        double cost = (double)m * (r.size() + extra_pass) * radix_weight(r);
        if (cost < best) {
            best = cost;
            hp.m = m;
            hp.rad = r;
        }
    }
    return best < 1e300;
}

static void plan_twiddles(HostPlan& hp) {
    hp.w.resize(hp.m);
    for (int k = 0; k < hp.m; k++) {
        const double a = -2.0 * M_PI * (double)k / (double)hp.m;
        hp.w[k] = std::complex<double>(std::cos(a), std::sin(a));
    }
}

void add_bluestein(HostPlan& hp, int quick) {
    const Chirp& ch = maker(hp).ch;
    hp.chirp.clear();
    hp.bhat.clear();
    for (const Cd& v : ch.c) hp.chirp.emplace_back(v.x, v.y);
    // rt: bhat takes back the gain of its roundtrip and of the chirps, of which a DFT applies two
    // and its inverse their conjugates
    const double f = hp.rt ? 1.0 - hp.gain[quick] - mean_excess(hp.chirp.data(), hp.n) : 1.0;
    for (const Cd& v : ch.b) hp.bhat.emplace_back(v.x * f, v.y * f);
}

int build_plan_host(int n, HostPlan& hp) {
    hp = HostPlan();
    hp.n = n;
    if (n == 1) {
        hp.m = 1;
    } else if (factor_direct(n, hp.rad)) {
        hp.m = n;
    } else {
        // Bluestein: the {2,3,5,7}-smooth inner length in [2n-1, 2.3n] with the
        // lowest pass work, m * (passes + 1), weighted by radix_weight
        hp.blue = 1;
        if (!choose_inner_length(n, 1, hp)) return -1;
    }
    plan_twiddles(hp);
    if (hp.blue) add_bluestein(hp);
    return 0;
}

// A separable spectral operator y = IDFT_n(H . DFT_n(x)) is the circular
// convolution of x with h = IDFT_n(H).  Any length m >= 2n-1 computes it with
// one zero-padded forward and one inverse length-m FFT (every lag i-j in
// (-n, n) lands on a distinct slot of the length-m wrap), so a window length
// with a large prime factor costs two smooth FFTs instead of Bluestein's four.
bool stockham_line(int n) {
    HostPlan hp;
    return n == 1 || factor_direct(n, hp.rad) || choose_inner_length(n, 0, hp);
}

int build_conv_plan_host(int n, HostPlan& hp, RtAxis axis) {
    hp = HostPlan();
    hp.n = n;
    if ((hp.rt = rt_choose(n, axis)) > 0) {
        const RtEntry e = entry(hp.rt, axis, false);
        hp.m = e.m;
        for (int r : {e.r1, e.r2, e.r3})
            if (r > 1) hp.rad.push_back(r);
    } else if (n == 1) {
        hp.m = 1;
    } else if (factor_direct(n, hp.rad)) {
        hp.m = n;
    } else if (!choose_inner_length(n, 0, hp)) {
        return -1;
    }
    if (!hp.rt) {
        plan_twiddles(hp);
        return 0;
    }
    // the tables of the entry's two forms (line_rt.cuh)
    for (bool quick : {false, true}) {
        const RtEntry e = entry(hp.rt, axis, quick);
        if (!e.m) continue;
        auto put = [&](long long k, int n) {
            const double a = -2.0 * M_PI * (double)(k % n) / (double)n;
            hp.w.push_back(std::complex<double>(std::cos(a), std::sin(a)));
        };
        for (int r = 0; r < e.r1; r++)
            for (int j = 0; j < e.m / e.r1; j++) put((long long)r * j, e.m);
        for (int b = 0; b < e.r2; b++)
            for (int c = 0; c < e.r3; c++) put((long long)b * c, e.r2 * e.r3);
        if (hp.w.size() % 2) hp.w.push_back(0.0);  // the kernels copy it in 16-byte pieces
        const size_t at = quick ? hp.wq : 0;
        hp.gain[quick] = radix_gain(e.r1) + radix_gain(e.r2) + radix_gain(e.r3) + mean_excess(&hp.w[at], e.m) +
                         mean_excess(&hp.w[at + e.m], e.r2 * e.r3);
        if (!quick) hp.wq = (int)hp.w.size();
    }
    return 0;
}

// Spectrum (length m, 1/m folded in) of the zero-padded, wrapped kernel of the
// operator whose length-n symbol is Hn (1/n already folded in).
void conv_table(const HostPlan& hp, const std::vector<std::complex<double>>& Hn,
                std::vector<std::complex<double>>& out, int quick) {
    const int n = hp.n, m = hp.m;
    const double f = 1.0 - hp.gain[quick];
    if (m == n) {
        out = Hn;
        for (auto& c : out) c *= f;
        return;
    }
    // h[d] = sum_k Hn[k] e^{+2 pi i k d / n} = conj(DFT_n(conj Hn)), by Bluestein's identity on m
    TableMaker& t = maker(hp);
    std::vector<Cd> x(m, Cd{0.0, 0.0}), hm(m, Cd{0.0, 0.0});
    for (int k = 0; k < n; k++) x[k] = mul({Hn[k].real(), -Hn[k].imag()}, t.ch.c[k]);
    t.f.run(x, -1);
    for (int k = 0; k < m; k++) x[k] = mul(x[k], t.ch.b[k]);
    t.f.run(x, +1);
    for (int d = 0; d < n; d++) {
        const Cd v = mul(x[d], t.ch.c[d]);
        const Cd h{v.x, -v.y};
        hm[d] = h;                          // lags 0 .. n-1
        if (d > 0) hm[m - n + d] = h;       // lags -(n-1) .. -1: slot m - (n - d)
    }
    t.f.run(hm, -1);
    out.resize(m);
    for (int k = 0; k < m; k++) out[k] = std::complex<double>(hm[k].x / m * f, hm[k].y / m * f);
}

void convtab_tables(const HostPlan& hp, std::vector<double2>& out, ConvTabArgs& a) {
    const TableMaker& t = maker(hp);
    out.clear();
    for (const std::vector<Cd>* v : {&t.f.w, &t.ch.c, &t.ch.b})
        for (const Cd& c : *v) out.push_back(make_double2(c.x, c.y));
    a.m = hp.m;
    a.nrad = (int)t.f.rad.size();
    std::copy(t.f.rad.begin(), t.f.rad.end(), a.rad);
}

int fill_plan_dev(const HostPlan& hp, FFTPlanDev& d) {
    d.n = hp.n;
    d.m = hp.m;
    d.blue = hp.blue;
    d.nst = (int)hp.rad.size();
    int ns = 1, maxb = 1;
    for (int i = 0; i < d.nst; i++) {
        FFTPass& p = d.pass[i];
        p.R = hp.rad[i];
        p.ns = ns;
        p.B = hp.m / p.R;
        p.twstride = hp.m / (ns * p.R);
        p.ns_magic = (ns > 1) ? (unsigned)(((1ull << 32) + ns - 1) / ns) : 0u;
        maxb = std::max(maxb, p.B);
        ns *= p.R;
    }
    d.w = d.chirp = d.bhat = nullptr;
    d.rt = hp.rt;
    d.quick = 0;
    d.pdl = 0;
    if (hp.rt) {  // the entry's own thread count
        d.tx = 32;
        return 0;
    }
    d.tx = std::min(QP_MAXTHREADS, (maxb + 31) / 32 * 32);
    return (maxb > QP_MAXTHREADS) ? -1 : 0;
}

void plan_tables(const HostPlan& hp, std::vector<float2>& out) {
    out.clear();
    out.reserve(hp.w.size() + hp.chirp.size() + hp.bhat.size());
    for (auto& c : hp.w) out.push_back(make_float2((float)c.real(), (float)c.imag()));
    for (auto& c : hp.chirp) out.push_back(make_float2((float)c.real(), (float)c.imag()));
    for (auto& c : hp.bhat) out.push_back(make_float2((float)c.real(), (float)c.imag()));
}

int choose_L(int nlines, int m, int tx, int nbuf, bool pow2, size_t extra_per_line, size_t budget) {
    const size_t per_line = (size_t)8 * m * nbuf + extra_per_line;
    const int lmax = std::max(1, std::min(QP_MAXTHREADS / tx, (int)(budget / per_line)));
    int L = (nlines + 2 * 152 - 1) / (2 * 152);
    L = std::max(1, std::min(L, lmax));
    if (pow2) {
        int p = 1;
        while (p * 2 <= L) p *= 2;
        L = p;
    }
    return L;
}

}  // namespace qp
