// vz_kernels.cu -- launchers of the constant-Q pass kernels (vz_kernels.cuh).
#include "vz_kernels.cuh"
#include "rt.cuh"

namespace qp {
int convtab_set_smem_limits();

// ---- launchers -------------------------------------------------------------------
static size_t lsm(int L, int m, int nbuf) { return sizeof(float2) * (size_t)nbuf * L * m; }
static int zgrid(int nxx, int L) { return (nxx + 2 * L - 1) / (2 * L); }

// launches kernel template K for a plan with radices up to 12 (r12) or 16
#define QP_BY_RADIX(r12, K, ...)                                            \
    do {                                                                    \
        if (r12) K<RtFFT<12>><<<__VA_ARGS__, s>>>(a);                       \
        else K<RtFFT<16>><<<__VA_ARGS__, s>>>(a);                           \
    } while (0)

void launch_vz_passA(const VzArgsA& a, cudaStream_t s) {
    if (a.pl.rt) {
        rtz_any(a.pl.quick, [&](const RtzGroup& g) { return g.passA(a, s); });
        return;
    }
    const dim3 blk(max(a.pl.tx, a.plc.tx), a.L);
    const size_t sm = lsm(a.L, max(a.pl.m, a.plc.m), 1);
    const bool r12 = plan_max_radix(a.pl) <= 12 && plan_max_radix(a.plc) <= 12;
    QP_BY_RADIX(r12, vz_passA_kernel, zgrid(a.nxx, a.L), blk, sm);
}
void launch_vz_xspec(const VxsArgs& a, cudaStream_t s) {
    if (a.pl.rt) {
        rt_any(false, [&](const RtGroup& g) { return g.xexact(a, s); });
        return;
    }
    const int grid = (a.nzh + a.L - 1) / a.L;
    const size_t sm = lsm(a.L, a.pl.m, a.mode == 0 ? 2 : 1);
    if (plan_max_radix(a.pl) <= 12) vz_xspec_kernel<RtFFT<12>><<<grid, dim3(a.pl.tx, a.L), sm, s>>>(a);
    else vz_xspec_kernel<RtFFT<16>><<<grid, dim3(a.pl.tx, a.L), sm, s>>>(a);
}
void launch_rt_xconv(const XconvArgs& a, cudaStream_t s) {
    rt_any(a.pl.quick, [&](const RtGroup& g) { return g.xconv(a, s); });
}
void launch_vz_convtab(const VtabArgs& a, cudaStream_t s) {
    const int grid = (a.nzh + a.L - 1) / a.L;
    const dim3 blk(max(a.pl.tx, a.plc.tx), a.L);
    const size_t sm = lsm(a.L, max(a.pl.m, a.plc.m), 1);
    vz_convtab_kernel<RtFFT<16>><<<grid, blk, sm, s>>>(a);
}
void launch_lr_xconv(const LrxArgs& a, cudaStream_t s) {
    const int grid = (a.nzh + a.L - 1) / a.L;
    const dim3 blk(a.plc.tx, a.L);
    const size_t sm = lsm(a.L, a.plc.m, 2);
    if (plan_max_radix(a.plc) <= 12) lr_xconv_kernel<RtFFT<12>><<<grid, blk, sm, s>>>(a);
    else lr_xconv_kernel<RtFFT<16>><<<grid, blk, sm, s>>>(a);
}
void launch_lr_zsum(const LrsArgs& a, cudaStream_t s) {
    if (a.pl.rt) {
        rtz_any(a.pl.quick, [&](const RtzGroup& g) { return g.zsum(a, s); });
        return;
    }
    const dim3 blk(a.pl.tx, a.L);
    const size_t sm = lsm(a.L, a.pl.m, 1);
    for (int b = 0; b < a.row; b++) {
        if (plan_max_radix(a.pl) <= 12) lr_zsum_kernel<RtFFT<12>><<<zgrid(a.nxx, a.L), blk, sm, s>>>(a, b);
        else lr_zsum_kernel<RtFFT<16>><<<zgrid(a.nxx, a.L), blk, sm, s>>>(a, b);
    }
}

void launch_vz_passB(const VzArgsB& a, cudaStream_t s) {
    if (a.pl.rt) {
        rtz_any(a.pl.quick, [&](const RtzGroup& g) { return g.passB(a, s); });
        return;
    }
    const dim3 blk(a.pl.tx, a.L);
    const size_t sm = lsm(a.L, a.pl.m, 2);
    QP_BY_RADIX(plan_max_radix(a.pl) <= 12, vz_passB_kernel, zgrid(a.nxx, a.L), blk, sm);
}
void launch_vz_passC(const VzArgsC& a, cudaStream_t s) {
    if (a.pl.rt) {
        rtz_any(a.pl.quick, [&](const RtzGroup& g) { return g.passC(a, s); });
        return;
    }
    const dim3 blk(a.pl.tx, a.L);
    const size_t sm = lsm(a.L, a.pl.m, 1);
    QP_BY_RADIX(plan_max_radix(a.pl) <= 12, vz_passC_kernel, zgrid(a.nxx, a.L), blk, sm);
}
void launch_vz_zinv(const VzArgsI& a, cudaStream_t s) {
    const dim3 blk(a.pl.tx, a.L);
    const size_t sm = lsm(a.L, a.pl.m, 1);
    QP_BY_RADIX(plan_max_radix(a.pl) <= 12, vz_zinv_kernel, zgrid(a.nxx, a.L), blk, sm);
}

template <class FP> static int vz_set_limits_one() {
    const int lim = 200 * 1024;
    int bad = 0;
    bad |= cudaFuncSetAttribute(vz_passA_kernel<FP>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(vz_passB_kernel<FP>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(vz_passC_kernel<FP>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(vz_zinv_kernel<FP>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(lr_zsum_kernel<FP>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    return bad;
}

int vz_set_smem_limits() {
    const int lim = 200 * 1024;
    int bad = vz_set_limits_one<RtFFT<12>>() | vz_set_limits_one<RtFFT<16>>() | convtab_set_smem_limits();
    bad |= cudaFuncSetAttribute(vz_xspec_kernel<RtFFT<12>>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(vz_xspec_kernel<RtFFT<16>>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(vz_convtab_kernel<RtFFT<16>>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(lr_xconv_kernel<RtFFT<12>>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    bad |= cudaFuncSetAttribute(lr_xconv_kernel<RtFFT<16>>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) != cudaSuccess;
    return bad ? -1 : 0;
}

}  // namespace qp
