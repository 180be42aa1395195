// rt.cuh -- launchers of the register-to-register passes (rt_kernels.cuh, rt_z.cuh) by group
// of entries (rt_list.h); each group is a translation unit of its own (rt_group.cu,
// rtz_group.cu).
#pragma once
#include <cuda_runtime.h>

#include "qpstd_internal.h"
#include "rt_list.h"

namespace qp {

// Each launches the kernel on the entry plan.rt and returns true, or launches nothing and
// returns false when the entry is not in the group; the quick groups have no xexact.  limits raises the dynamic shared-memory limits (non-zero: failed).
struct RtGroup {
    bool (*xpass)(const AcXArgs& a, cudaStream_t s);
    bool (*xconv)(const XconvArgs& a, cudaStream_t s);
    bool (*xexact)(const VxsArgs& a, cudaStream_t s);
    int (*limits)();
};
// (zpass: null in the groups of the constant-Q step alone)
struct RtzGroup {
    bool (*zpass)(const AcZArgs& a, cudaStream_t s);
    bool (*passA)(const VzArgsA& a, cudaStream_t s);
    bool (*passB)(const VzArgsB& a, cudaStream_t s);
    bool (*passC)(const VzArgsC& a, cudaStream_t s);
    bool (*zsum)(const LrsArgs& a, cudaStream_t s);
    int (*limits)();
};
// the groups in the order of rt_list.h, the wide forms' first
extern const RtGroup* const rt_groups[QP_RT_NGROUPS];
extern const RtzGroup* const rtz_groups[QP_RTZ_NGROUPS];

template <class Fn> bool rt_any(bool quick, Fn&& fn) {
    for (int g = quick ? QP_RT_NWIDE : 0; g < (quick ? QP_RT_NGROUPS : QP_RT_NWIDE); g++)
        if (fn(*rt_groups[g])) return true;
    return false;
}
template <class Fn> bool rtz_any(bool quick, Fn&& fn) {
    for (int g = quick ? QP_RTZ_NWIDE : 0; g < (quick ? QP_RTZ_NGROUPS : QP_RTZ_NWIDE); g++)
        if (fn(*rtz_groups[g])) return true;
    return false;
}

}  // namespace qp
