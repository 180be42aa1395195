// rtz_group.cu -- the z passes of one group of entries, QP_RTZ_G<k> of rt_list.h; compiled once
// per group with -DQP_RTZ_GROUP=<k>.
#include "rt.cuh"
#include "rt_z.cuh"

#define QP_RT_CAT(a, b) a##b
#define QP_RT_CAT2(a, b) QP_RT_CAT(a, b)
#define QP_RTZ_ENTRIES QP_RT_CAT2(QP_RTZ_G, QP_RTZ_GROUP)

namespace qp {
namespace {

template <class LR> unsigned z_grid(int nxx) { return (nxx + 2 * LR::G * LR::W - 1) / (2 * LR::G * LR::W); }
// passes with a second buffer (running sums)
template <class LR> constexpr size_t smem_sum() { return LR::kSmem + LR::kLines; }

// entries of the constant-Q step alone have no acoustic pass
#define QP_RTZ_VISCO (QP_RTZ_GROUP >= QP_RTZ_NBOTH && QP_RTZ_GROUP < QP_RTZ_NWIDE)

#define QP_RTZ_SWITCH(ID_OF, CASE) \
    switch (ID_OF) {               \
        QP_RTZ_ENTRIES(CASE)       \
        default: return false;     \
    }                              \
    return true;
// the launcher of kernel K with SMEM bytes, and its dispatch by entry
#define QP_RTZ_LAUNCH(NAME, ARGS, K, SMEM)                                                                            \
    template <int W, bool PAD, bool GF, int G, int MB, int R1, int R2, int R3>                             \
    void l_##NAME(const ARGS& a, cudaStream_t s) {                                                                    \
        using LR = LineRT<W, PAD, GF, G, MB, R1, R2, R3, (QP_RTZ_GROUP < QP_RTZ_NWIDE ? kEpiWideZ : kEpiQuick)>;                                                              \
        launch_rt(K<LR>, z_grid<LR>(a.nxx), LR::kThreads, SMEM, s, a.pl.pdl, a);                                                       \
    }
#if !QP_RTZ_VISCO
QP_RTZ_LAUNCH(zpass, AcZArgs, rt_zpass_kernel, LR::kSmem)
#endif
QP_RTZ_LAUNCH(passA, VzArgsA, rt_passA_kernel, LR::kSmem)
QP_RTZ_LAUNCH(passB, VzArgsB, rt_passB_kernel, smem_sum<LR>())
QP_RTZ_LAUNCH(passC, VzArgsC, rt_passC_kernel, LR::kSmem)
QP_RTZ_LAUNCH(zsum, LrsArgs, rt_zsum_kernel, smem_sum<LR>())

template <class K> bool up(K k, size_t bytes) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess;
}
template <int W, bool PAD, bool GF, int G, int MB, int R1, int R2, int R3> int l_limits() {
    using LR = LineRT<W, PAD, GF, G, MB, R1, R2, R3, (QP_RTZ_GROUP < QP_RTZ_NWIDE ? kEpiWideZ : kEpiQuick)>;
    static_assert(smem_sum<LR>() <= QP_SMEM_DYN_MAX, "lines of an entry fit a CTA's shared memory");
    bool bad = up(rt_passA_kernel<LR>, LR::kSmem) | up(rt_passB_kernel<LR>, smem_sum<LR>()) |
               up(rt_passC_kernel<LR>, LR::kSmem) | up(rt_zsum_kernel<LR>, smem_sum<LR>());
#if !QP_RTZ_VISCO
    bad |= up(rt_zpass_kernel<LR>, LR::kSmem);
#endif
    return bad;
}

#if QP_RTZ_VISCO
constexpr bool (*g_zpass)(const AcZArgs&, cudaStream_t) = nullptr;
#else
bool g_zpass(const AcZArgs& a, cudaStream_t s) {
#define C_(ID, W, PAD, GF, G, MB, R1, R2, R3, COST) \
    case ID: l_zpass<W, PAD, GF, G, MB, R1, R2, R3>(a, s); break;
    QP_RTZ_SWITCH(a.pl.rt, C_)
#undef C_
}
#endif
bool g_passA(const VzArgsA& a, cudaStream_t s) {
#define C_(ID, W, PAD, GF, G, MB, R1, R2, R3, COST) \
    case ID: l_passA<W, PAD, GF, G, MB, R1, R2, R3>(a, s); break;
    QP_RTZ_SWITCH(a.pl.rt, C_)
#undef C_
}
bool g_passB(const VzArgsB& a, cudaStream_t s) {
#define C_(ID, W, PAD, GF, G, MB, R1, R2, R3, COST) \
    case ID: l_passB<W, PAD, GF, G, MB, R1, R2, R3>(a, s); break;
    QP_RTZ_SWITCH(a.pl.rt, C_)
#undef C_
}
bool g_passC(const VzArgsC& a, cudaStream_t s) {
#define C_(ID, W, PAD, GF, G, MB, R1, R2, R3, COST) \
    case ID: l_passC<W, PAD, GF, G, MB, R1, R2, R3>(a, s); break;
    QP_RTZ_SWITCH(a.pl.rt, C_)
#undef C_
}
bool g_zsum(const LrsArgs& a, cudaStream_t s) {
#define C_(ID, W, PAD, GF, G, MB, R1, R2, R3, COST) \
    case ID: l_zsum<W, PAD, GF, G, MB, R1, R2, R3>(a, s); break;
    QP_RTZ_SWITCH(a.pl.rt, C_)
#undef C_
}
int g_limits() {
    int bad = 0;
#define C_(ID, W, PAD, GF, G, MB, R1, R2, R3, COST) bad |= l_limits<W, PAD, GF, G, MB, R1, R2, R3>();
    QP_RTZ_ENTRIES(C_)
#undef C_
    return bad;
}

}  // namespace

extern const RtzGroup QP_RT_CAT2(rtz_group_, QP_RTZ_GROUP);
const RtzGroup QP_RT_CAT2(rtz_group_, QP_RTZ_GROUP) = {g_zpass, g_passA, g_passB, g_passC, g_zsum, g_limits};

}  // namespace qp
