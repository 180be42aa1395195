// rt_list.h -- the line lengths compiled into the register-to-register passes
// (line_rt.cuh), host and device view.
//
// x entries are X(ID, W, G, MB, R1, R2, R3, COST): W complex lines per thread, G groups of W
// lines per CTA, MB CTAs per SM the kernels are compiled for, the radices, and the measured
// clocks x 1000 per point and roundtrip of one SM (loops of roundtrips on full SMs).  All of
// them serve zero-padded lines: an n-point line runs on the entry of length M >= 2n - 1 with the
// least M x COST.  Radices of powers of two cost least, so the ladder is dense around them:
// lengths between two entries would cost as much as the next one (3840: 0.99, 4096: 0.93).
// Short lines take three passes of radices up to 16: two of radices up to 32 measured 0.74
// clocks against 0.82 at 1024 points but leave too few threads a line.  Two packed lines per
// thread beat one up to 4096 points (3360: 1.07 against 1.22); beyond 4608 they leave no
// registers for a second CTA (5120: 1.19 against 1.14).
//
// z entries are X(ID, W, PAD, GF, G, MB, R1, R2, R3, COST): PAD 0 transforms lines of exactly
// M points, PAD 1 serves n <= (M + 1) / 2 (operators as padded convolutions, exact DFTs by
// Bluestein's identity).  GF 1: a warp's threads are neighbouring rows, whose points are
// neighbours in the blocked fields.  The COSTs of the z entries decide nothing: at every depth the
// shortest entry that fits has the least M x COST.
//
// The exact lengths up to entry 9 are the depths of the programs' standard models (160 + 2 x 10,
// 160 + 2 x 20, 600 + 2 x 30) and a ladder of smooth depths from 256 to 800.  Those from entry 25 on
// serve the constant-Q step alone: they are smooth depths where its batches ran slower padded (ten
// roundtrips of more than 2n points a step) than on a direct Stockham transform.  16 shots 1300 to
// 1855 wide, us a step, Stockham / padded / exact: 600 deep 1986 / 2354 / 1379, 768 2284 / 2575 /
// 1652, 900 2717 / 2851 / 2026, 1728 5530 / 5714 / 3657.  Up to 384 points padded is faster than
// Stockham, and at the smooth depths left out (490, 504, 972, 1152, 1400, 1500) within 8 % of it.
// They have no quick form: lone shots 150 to 1000 wide take 0.54 to 1.03 of the padded forms' time.
// An acoustic step (three roundtrips along z) is faster padded than Stockham at all of them, and a
// lone one 1000 x 480 faster than exact too (23.6 against 29.2 us).
//
// The wide forms fill the chip with many lines; the quick forms have the same lengths with
// fewer lines per CTA on more threads, for grids whose wide form has fewer CTAs than the
// chip has SMs (there the latency of one line counts).
#pragma once

// Each group is compiled by itself (rt_group.cu), to keep the build parallel.
#define QP_RT_G0(X) X(1, 2, 8, 4, 10, 1, 16, 650) X(2, 2, 8, 3, 16, 1, 16, 500) X(3, 2, 2, 5, 8, 6, 8, 800)
#define QP_RT_G1(X) X(4, 2, 2, 4, 8, 8, 8, 760) X(5, 2, 1, 5, 8, 12, 8, 850)
#define QP_RT_G2(X) X(6, 2, 1, 4, 8, 16, 8, 820) X(7, 2, 1, 4, 16, 8, 10, 980)
#define QP_RT_G3(X) X(8, 2, 1, 3, 16, 8, 12, 1000) X(9, 2, 1, 4, 16, 8, 16, 950)
#define QP_RT_G4(X) X(10, 2, 1, 2, 16, 12, 12, 1060) X(11, 2, 1, 3, 16, 10, 16, 1080)
#define QP_RT_G5(X) X(12, 2, 1, 2, 16, 12, 16, 1050) X(13, 2, 1, 2, 16, 14, 15, 1070)
#define QP_RT_G6(X) X(14, 2, 1, 2, 16, 16, 16, 930) X(15, 1, 1, 2, 16, 20, 16, 1140)
#define QP_RT_G7(X) X(16, 1, 1, 1, 24, 16, 16, 1400) X(17, 1, 1, 1, 20, 18, 20, 1470)
#define QP_RT_G8(X) X(18, 1, 1, 1, 24, 18, 20, 1460) X(19, 1, 1, 1, 24, 16, 24, 1460)
#define QP_RT_G9(X) X(1, 1, 1, 8, 8, 4, 5, 0) X(2, 1, 1, 8, 8, 4, 8, 0) X(3, 1, 1, 8, 8, 6, 8, 0) X(4, 1, 1, 8, 8, 8, 8, 0) X(5, 1, 1, 5, 8, 12, 8, 0)
#define QP_RT_G10(X) X(6, 1, 1, 4, 8, 16, 8, 0) X(7, 1, 1, 3, 8, 16, 10, 0) X(8, 1, 1, 2, 8, 16, 12, 0)
#define QP_RT_G11(X) X(9, 1, 1, 2, 8, 16, 16, 0) X(10, 1, 1, 2, 12, 12, 16, 0) X(11, 1, 1, 2, 16, 10, 16, 0)
#define QP_RT_G12(X) X(12, 1, 1, 2, 16, 12, 16, 0) X(13, 1, 1, 2, 16, 14, 15, 0) X(14, 1, 1, 2, 16, 16, 16, 0)
#define QP_RTZ_G0(X) X(1, 1, 0, 1, 8, 4, 15, 1, 12, 1000) X(2, 1, 0, 1, 8, 3, 10, 1, 20, 1110) X(3, 1, 0, 1, 8, 4, 16, 1, 16, 700)
#define QP_RTZ_G1(X) X(4, 1, 0, 1, 4, 4, 8, 5, 8, 1100) X(5, 1, 0, 1, 4, 3, 10, 5, 8, 1200) X(6, 1, 0, 1, 2, 5, 8, 8, 8, 1050)
#define QP_RTZ_G2(X) X(7, 1, 0, 1, 2, 4, 8, 8, 10, 1150) X(8, 1, 0, 1, 2, 4, 11, 6, 10, 1600)
#define QP_RTZ_G3(X) X(9, 1, 0, 1, 2, 4, 10, 8, 10, 1250) X(15, 1, 1, 1, 2, 2, 8, 16, 8, 1000)
#define QP_RTZ_G4(X) X(10, 1, 1, 1, 8, 4, 10, 1, 16, 800) X(11, 1, 1, 1, 8, 4, 16, 1, 16, 600) X(12, 1, 1, 1, 4, 3, 8, 6, 8, 1000)
#define QP_RTZ_G5(X) X(13, 1, 1, 1, 2, 5, 8, 8, 8, 950) X(14, 1, 1, 1, 2, 3, 8, 12, 8, 1050)
#define QP_RTZ_G6(X) X(16, 1, 1, 1, 2, 2, 16, 8, 10, 1200) X(17, 1, 1, 1, 2, 2, 16, 8, 12, 1200)
#define QP_RTZ_G7(X) X(18, 1, 1, 1, 2, 2, 16, 8, 16, 1150) X(19, 1, 1, 0, 1, 3, 16, 12, 12, 1250)
#define QP_RTZ_G8(X) X(20, 1, 1, 0, 1, 4, 16, 10, 16, 1250) X(21, 1, 1, 0, 1, 3, 16, 12, 16, 1250)
#define QP_RTZ_G9(X) X(22, 1, 1, 0, 1, 2, 16, 16, 16, 1150) X(23, 1, 1, 0, 1, 2, 16, 20, 16, 1140)
#define QP_RTZ_G10(X) X(24, 1, 1, 0, 1, 1, 24, 16, 16, 1400)
#define QP_RTZ_G11(X) X(25, 1, 0, 1, 2, 5, 8, 6, 10, 1200) X(26, 1, 0, 1, 2, 5, 10, 5, 10, 1200) X(27, 1, 0, 1, 2, 5, 9, 6, 10, 1200)
#define QP_RTZ_G12(X) X(28, 1, 0, 1, 2, 4, 8, 7, 10, 1200) X(29, 1, 0, 1, 2, 5, 10, 6, 10, 1200) X(30, 1, 0, 1, 2, 4, 10, 7, 10, 1200)
#define QP_RTZ_G13(X) X(31, 1, 0, 1, 2, 4, 9, 8, 10, 1200) X(32, 1, 0, 1, 2, 3, 8, 12, 8, 1200) X(33, 1, 0, 1, 2, 3, 10, 7, 12, 1200)
#define QP_RTZ_G14(X) X(34, 1, 0, 1, 2, 3, 10, 9, 10, 1200) X(35, 1, 0, 1, 2, 3, 10, 8, 12, 1200)
#define QP_RTZ_G15(X) X(36, 1, 0, 1, 2, 2, 10, 7, 14, 1200) X(37, 1, 0, 1, 2, 2, 10, 10, 10, 1200) X(38, 1, 0, 1, 2, 2, 8, 16, 8, 1200)
#define QP_RTZ_G16(X) X(39, 1, 0, 1, 2, 5, 7, 7, 8, 1200) X(40, 1, 0, 1, 2, 5, 10, 6, 7, 1200) X(41, 1, 0, 1, 2, 5, 8, 6, 9, 1200) X(42, 1, 0, 1, 2, 5, 8, 7, 8, 1200) X(43, 1, 0, 1, 2, 5, 10, 5, 9, 1200)
#define QP_RTZ_G17(X) X(44, 1, 0, 1, 2, 4, 8, 8, 9, 1200) X(45, 1, 0, 1, 2, 3, 7, 7, 12, 1200) X(46, 1, 0, 1, 2, 4, 10, 7, 9, 1200) X(47, 1, 0, 1, 2, 4, 9, 8, 9, 1200) X(48, 1, 0, 1, 2, 3, 8, 7, 12, 1200)
#define QP_RTZ_G18(X) X(49, 1, 0, 1, 2, 2, 8, 7, 14, 1200) X(50, 1, 0, 1, 2, 3, 9, 9, 10, 1200) X(51, 1, 0, 1, 2, 3, 9, 8, 12, 1200) X(52, 1, 0, 1, 2, 2, 9, 7, 14, 1200) X(53, 1, 0, 1, 2, 2, 8, 8, 14, 1200)
#define QP_RTZ_G19(X) X(54, 1, 0, 1, 2, 2, 10, 7, 15, 1200) X(55, 1, 0, 1, 2, 2, 10, 9, 12, 1200) X(56, 1, 0, 1, 2, 2, 10, 8, 14, 1200) X(57, 1, 0, 1, 2, 2, 12, 9, 12, 1200) X(58, 1, 0, 1, 2, 2, 12, 8, 14, 1200)
#define QP_RTZ_G20(X) X(59, 1, 0, 0, 1, 4, 10, 10, 16, 1200) X(60, 1, 0, 0, 1, 4, 12, 10, 14, 1200) X(61, 1, 0, 0, 1, 4, 12, 12, 12, 1200) X(62, 1, 0, 0, 1, 4, 16, 8, 14, 1200) X(63, 1, 0, 0, 1, 4, 12, 10, 15, 1200)
#define QP_RTZ_G21(X) X(1, 1, 0, 0, 1, 4, 5, 6, 6, 0) X(2, 1, 0, 0, 1, 4, 5, 5, 8, 0) X(3, 1, 0, 0, 1, 4, 8, 4, 8, 0) X(4, 1, 0, 0, 1, 4, 8, 5, 8, 0) X(5, 1, 0, 0, 1, 4, 10, 5, 8, 0)
#define QP_RTZ_G22(X) X(6, 1, 0, 0, 1, 4, 8, 8, 8, 0) X(7, 1, 0, 0, 1, 4, 8, 8, 10, 0) X(8, 1, 0, 0, 1, 4, 11, 6, 10, 0) X(9, 1, 0, 0, 1, 4, 10, 8, 10, 0)
#define QP_RTZ_G23(X) X(10, 1, 1, 0, 1, 4, 8, 4, 5, 0) X(11, 1, 1, 0, 1, 4, 8, 4, 8, 0) X(12, 1, 1, 0, 1, 4, 8, 6, 8, 0) X(13, 1, 1, 0, 1, 4, 8, 8, 8, 0)
#define QP_RTZ_G24(X) X(14, 1, 1, 0, 1, 4, 8, 12, 8, 0) X(15, 1, 1, 0, 1, 4, 8, 16, 8, 0)
#define QP_RT_WIDE_ALL(X) \
    QP_RT_G0(X) QP_RT_G1(X) QP_RT_G2(X) QP_RT_G3(X) QP_RT_G4(X) QP_RT_G5(X) QP_RT_G6(X) QP_RT_G7(X) QP_RT_G8(X)
#define QP_RT_QUICK_ALL(X) \
    QP_RT_G9(X) QP_RT_G10(X) QP_RT_G11(X) QP_RT_G12(X)
#define QP_RTZ_WIDE_ALL(X) \
    QP_RTZ_G0(X) QP_RTZ_G1(X) QP_RTZ_G2(X) QP_RTZ_G3(X) QP_RTZ_G4(X) QP_RTZ_G5(X) QP_RTZ_G6(X) QP_RTZ_G7(X) QP_RTZ_G8(X) QP_RTZ_G9(X) QP_RTZ_G10(X) \
    QP_RTZ_G11(X) QP_RTZ_G12(X) QP_RTZ_G13(X) QP_RTZ_G14(X) QP_RTZ_G15(X) QP_RTZ_G16(X) QP_RTZ_G17(X) QP_RTZ_G18(X) QP_RTZ_G19(X) QP_RTZ_G20(X)
#define QP_RTZ_QUICK_ALL(X) \
    QP_RTZ_G21(X) QP_RTZ_G22(X) QP_RTZ_G23(X) QP_RTZ_G24(X)
// groups of the wide forms come first
#define QP_RT_NWIDE 9
#define QP_RT_NGROUPS 13
#define QP_RTZ_NWIDE 21
// of which those from here on serve the constant-Q step alone
#define QP_RTZ_NBOTH 11
#define QP_RTZ_NGROUPS 25

// Registers that an epilogue loop's loads in flight may take.  Wide z passes: 36 at 96 registers a
// thread, four CTAs per SM (z passes of a 4100 x 660 constant-Q shot 119 us; 24: 121; three CTAs of
// 128 registers 132, which a lone 1678 x 660 shot would like better, 62 against 64.5, and the
// 64-shot batch worse, 5.68 against 5.36 ms).  Acoustic z passes of 1700- and 2500-wide shots, us at
// 36 and at 24: 512 points 18.0 and 18.4, 600 39.6 and 41.5, 661 42.3 and 44.3, 768 47.9 and 49.6,
// 1024 58.0 and 59.5, 2000 104.9 and 107; slower at 400 (18.0 and 16.8), 660 (31.4 and 30.3), both
// of which spill at 36, and at 1200 (74.6 and 70.5).  Wide x passes: 24 (36 spills on the longest
// lines: x pass of 4100 x 660 91 -> 99 us).  Quick: registers are plenty and each round of loads is a wait.
constexpr int kEpiWide = 24, kEpiWideZ = 36, kEpiQuick = 96;

// An entry's complex lines per CTA, length and radices (m = 0: no such entry).
struct RtEntry {
    int lines, m, pad, cost, r1, r2, r3;
};
inline RtEntry rt_entry(int id, bool quick) {
#define QP_RT_CASE(ID, W, G, MB, R1, R2, R3, COST) \
    if (id == ID) return {W * G, R1 * R2 * R3, 1, COST, R1, R2, R3};
    if (quick) {
        QP_RT_QUICK_ALL(QP_RT_CASE)
    } else {
        QP_RT_WIDE_ALL(QP_RT_CASE)
    }
#undef QP_RT_CASE
    return {0, 0, 0, 0, 0, 0, 0};
}
inline RtEntry rtz_entry(int id, bool quick) {
#define QP_RT_CASE(ID, W, PAD, GF, G, MB, R1, R2, R3, COST) \
    if (id == ID) return {W * G, R1 * R2 * R3, PAD, COST, R1, R2, R3};
    if (quick) {
        QP_RTZ_QUICK_ALL(QP_RT_CASE)
    } else {
        QP_RTZ_WIDE_ALL(QP_RT_CASE)
    }
#undef QP_RT_CASE
    return {0, 0, 0, 0, 0, 0, 0};
}
constexpr int kRtIds = 19, kRtzIds = 63;
constexpr int kRtzVisco = 25;  // z entries from here on serve the constant-Q step alone
