// host_setup.h -- FP64 coefficient setup and line-FFT plan construction.
#pragma once
#include <complex>
#include <memory>
#include <vector>

#include "qpstd_internal.h"

namespace qp {

// CPML coefficients; out8 = i_ax, i_bx, i_az, i_bz, h_ax, h_bx, h_az, h_bz.
void pml_coeffs(int pml, double fm, int nxx, int nzz, double dx, double dz, double dt, std::vector<double>* out8);

// |k| on an n-point grid as the reference builds it (kkx / kkz).
double wavenumber(int i, int n, double d);

// Effective (Hermitian) staggered-derivative symbol divided by n, or with
// raw=true the reference's own (unnormalised, possibly non-Hermitian) symbol.
// which: 0 = x velocity derivative, 1 = x pressure derivative,
//        2 = z velocity derivative, 3 = z pressure derivative.
void shift_symbols(int n, double d, int which, std::vector<std::complex<double>>& H, bool raw = false);

struct TableMaker;
struct HostPlan {
    int n = 0, m = 0, blue = 0;
    int rt = 0;  // entry of rt_list.h (0: a Stockham plan of fft_reg.cuh, one butterfly per thread)
    int wq = 0;  // rt: where the twiddles of the entry's quick form start in w
    double gain[2] = {0.0, 0.0};  // rt: what a roundtrip of the wide, the quick form scales a line by, less 1
    std::vector<int> rad;
    std::vector<std::complex<double>> w, chirp, bhat;
    mutable std::shared_ptr<TableMaker> maker;  // FP64 transforms of the tables, made when first needed
};
// Exact DFT plan of a Stockham pass: n itself when it factors into radices <= 16,
// else Bluestein on a smooth m >= 2n-1.
int build_plan_host(int n, HostPlan& hp);
// Length-m FFT plan for separable operators applied as zero-padded circular
// convolutions.  On an entry of rt_list.h's x or z passes (axis), where one is long
// enough; else (or for kStockham) a Stockham plan, m = n when n factors into radices
// <= 16, else a smooth m >= 2n-1.
// kRtZQ: the z lines of the constant-Q step, which has entries of its own
enum RtAxis { kStockham, kRtX, kRtZ, kRtZQ };
inline RtAxis rt_zaxis(bool visco) { return visco ? kRtZQ : kRtZ; }
int build_conv_plan_host(int n, HostPlan& hp, RtAxis axis = kStockham);
// Is there a Stockham plan for an n-point line?
bool stockham_line(int n);
// Adds the tables of the exact length-n DFT by Bluestein's identity on hp.m; rt: for its wide or
// quick form.
void add_bluestein(HostPlan& hp, int quick = 0);
// The entry of rt_list.h an n-point line runs on (0: none is long enough), whether
// it runs the entry's quick form for this number of lines, and its lines per CTA.
int rt_choose(int n, RtAxis axis);
int rt_quick(int id, RtAxis axis, int lines);
int rt_lines(int id, RtAxis axis, int quick);
int rt_length(int id, RtAxis axis);
// Length-m multiplier of the convolution form of the symbol Hn (1/n folded in); rt: for the
// entry's wide or quick form.
void conv_table(const HostPlan& hp, const std::vector<std::complex<double>>& Hn,
                std::vector<std::complex<double>>& out, int quick = 0);

// FP64 tables of Bluestein's identity on hp.m for convtab.cu: m roots, n chirp values, m of the
// chirp's transform; a.m and the radices.
void convtab_tables(const HostPlan& hp, std::vector<double2>& out, ConvTabArgs& a);

// Device view of a plan without its tables: passes, thread count per line.
// Returns -1 when a pass needs more threads per line than a CTA holds.
int fill_plan_dev(const HostPlan& hp, FFTPlanDev& d);
// The plan's tables in device order: twiddles, then (Bluestein) chirp and bhat.
void plan_tables(const HostPlan& hp, std::vector<float2>& out);

// Complex lines per CTA: bounded by the CTA's threads (tx per line), by shared
// memory (nbuf line buffers of m float2, plus extra_per_line bytes), and small
// enough that the grid covers the 152 SMs about twice.  pow2: a power of two.
int choose_L(int nlines, int m, int tx, int nbuf, bool pow2, size_t extra_per_line = 0,
             size_t budget = 160 * 1024);

}  // namespace qp
