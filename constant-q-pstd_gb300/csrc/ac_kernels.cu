// ac_kernels.cu -- launchers of the acoustic pass kernels (ac_kernels.cuh).
#include <cstdint>

#include "ac_kernels.cuh"
#include "rt.cuh"

namespace qp {

size_t ac_zpass_smem(int L, int m, int nzz, bool stage) {
    return sizeof(float2) * (size_t)L * m + (stage ? sizeof(float) * 5 * (size_t)L * 2 * nzz : 0);
}
size_t ac_xpass_smem(int L, int m, int nxx, int nstaged) {
    return sizeof(float2) * (size_t)L * m + sizeof(float) * (size_t)nstaged * nxx * 2 * L;
}

void launch_ac_zpass(const AcZArgs& a, cudaStream_t s) {
    if (a.pl.rt) {
        rtz_any(a.pl.quick, [&](const RtzGroup& g) { return g.zpass && g.zpass(a, s); });
        return;
    }
    const int grid = (a.nxx + 2 * a.L - 1) / (2 * a.L);
    const size_t sm = ac_zpass_smem(a.L, a.pl.m, a.nzz, a.stage);
    const dim3 blk(a.pl.tx, a.L);
    if (plan_max_radix(a.pl) <= 12) ac_zpass_kernel<RtFFT<12>><<<grid, blk, sm, s>>>(a);
    else ac_zpass_kernel<RtFFT<16>><<<grid, blk, sm, s>>>(a);
}

// Every buffer of the pass at 16 bytes (the library's own are; a caller's state may not be).
static bool aligned16(const AcXArgs& a) {
    uintptr_t v = 0;
    for (const void* p : {(const void*)a.p, (const void*)a.vx, (const void*)a.psi_px, (const void*)a.psi_vx, (const void*)a.Dx,
                          (const void*)a.div, (const void*)a.Lz, (const void*)a.bbx, (const void*)a.c1, (const void*)a.c2})
        v |= (uintptr_t)p;
    return (v & 15) == 0;
}

void launch_ac_xpass(const AcXArgs& a0, cudaStream_t s) {
    AcXArgs a = a0;
    if (a.pl.rt) {
        a.vec = a.rs == 4 || (a.nzz % 4 == 0 && aligned16(a));  // blocked fields are aligned by construction
        rt_any(a.pl.quick, [&](const RtGroup& g) { return g.xpass(a, s); });
        return;
    }
    const int grid = (a.nzz + 2 * a.L - 1) / (2 * a.L);
    const int nst = a.stage ? xstage_count(xstage_fields(a.do_p, a.do_v, a.do_dx)) : 0;
    const size_t sm = ac_xpass_smem(a.L, a.pl.m, a.nxx, nst);
    // the instance without the p update carries only the transforms it runs
    const dim3 blk(a.pl.tx, a.L);
    const bool r12 = plan_max_radix(a.pl) <= 12;
    if (a.do_p && r12) ac_xpass_kernel<true, RtFFT<12>><<<grid, blk, sm, s>>>(a);
    else if (a.do_p) ac_xpass_kernel<true, RtFFT<16>><<<grid, blk, sm, s>>>(a);
    else if (r12) ac_xpass_kernel<false, RtFFT<12>><<<grid, blk, sm, s>>>(a);
    else ac_xpass_kernel<false, RtFFT<16>><<<grid, blk, sm, s>>>(a);
}

int ac_set_smem_limits() {
    const int lim = QP_SMEM_DYN_MAX;
    int bad = 0;
    auto z = [&](auto fp) {
        bad |= cudaFuncSetAttribute(ac_zpass_kernel<decltype(fp)>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) !=
               cudaSuccess;
    };
    z(RtFFT<12>{});
    z(RtFFT<16>{});
    auto x = [&](auto fp) {
        using F = decltype(fp);
        bad |= cudaFuncSetAttribute(ac_xpass_kernel<true, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) !=
               cudaSuccess;
        bad |= cudaFuncSetAttribute(ac_xpass_kernel<false, F>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim) !=
               cudaSuccess;
    };
    x(RtFFT<12>{});
    x(RtFFT<16>{});
    for (const RtGroup* g : rt_groups) bad |= g->limits() != 0;
    for (const RtzGroup* g : rtz_groups) bad |= g->limits() != 0;
    return bad ? -1 : 0;
}

}  // namespace qp
