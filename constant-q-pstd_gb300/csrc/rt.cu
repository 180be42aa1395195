// rt.cu -- the groups of register-to-register passes, in the order of rt_list.h.
#include "rt.cuh"

namespace qp {

extern const RtGroup rt_group_0, rt_group_1, rt_group_2, rt_group_3, rt_group_4, rt_group_5, rt_group_6, rt_group_7, rt_group_8, rt_group_9, rt_group_10, rt_group_11, rt_group_12;
extern const RtzGroup rtz_group_0, rtz_group_1, rtz_group_2, rtz_group_3, rtz_group_4, rtz_group_5, rtz_group_6, rtz_group_7, rtz_group_8, rtz_group_9, rtz_group_10, rtz_group_11, rtz_group_12, rtz_group_13, rtz_group_14, rtz_group_15, rtz_group_16, rtz_group_17, rtz_group_18, rtz_group_19, rtz_group_20, rtz_group_21, rtz_group_22, rtz_group_23, rtz_group_24;

const RtGroup* const rt_groups[QP_RT_NGROUPS] = {&rt_group_0, &rt_group_1, &rt_group_2, &rt_group_3, &rt_group_4, &rt_group_5, &rt_group_6, &rt_group_7, &rt_group_8, &rt_group_9, &rt_group_10, &rt_group_11, &rt_group_12};
const RtzGroup* const rtz_groups[QP_RTZ_NGROUPS] = {&rtz_group_0, &rtz_group_1, &rtz_group_2, &rtz_group_3, &rtz_group_4, &rtz_group_5, &rtz_group_6, &rtz_group_7, &rtz_group_8, &rtz_group_9, &rtz_group_10, &rtz_group_11, &rtz_group_12, &rtz_group_13, &rtz_group_14, &rtz_group_15, &rtz_group_16, &rtz_group_17, &rtz_group_18, &rtz_group_19, &rtz_group_20, &rtz_group_21, &rtz_group_22, &rtz_group_23, &rtz_group_24};

}  // namespace qp
