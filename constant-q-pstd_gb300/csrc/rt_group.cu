// rt_group.cu -- the x passes of one group of entries, QP_RT_G<k> of rt_list.h; compiled once
// per group with -DQP_RT_GROUP=<k>.
#include "rt.cuh"
#include "rt_kernels.cuh"

#define QP_RT_CAT(a, b) a##b
#define QP_RT_CAT2(a, b) QP_RT_CAT(a, b)
#define QP_RT_ENTRIES QP_RT_CAT2(QP_RT_G, QP_RT_GROUP)

namespace qp {
namespace {

// a CTA takes G W pairs of z columns (G W kz columns)
template <class LR> unsigned x_grid(int cols) { return (cols + LR::G * LR::W - 1) / (LR::G * LR::W); }
// the lines, and beside them the kept spectra
template <class LR> constexpr size_t smem_many() { return LR::kSmem + (size_t)LR::G * LR::M * 8 * LR::W; }

// case ID: BODY on the entry's line type LR
#define QP_RT_SWITCH(ID_OF, CASE) \
    switch (ID_OF) {              \
        QP_RT_ENTRIES(CASE)       \
        default: return false;    \
    }                             \
    return true;
#define QP_RT_LR using LR = LineRT<W, true, false, G, MB, R1, R2, R3, (QP_RT_GROUP < QP_RT_NWIDE ? kEpiWide : kEpiQuick)>;

template <int W, int G, int MB, int R1, int R2, int R3> void l_xpass(const AcXArgs& a, cudaStream_t s) {
    QP_RT_LR
    const unsigned grid = x_grid<LR>((a.nzz + 1) / 2);
    if (a.do_p) launch_rt(rt_xpass_kernel<true, LR>, grid, LR::kThreads, LR::kSmem, s, a.pl.pdl, a);
    else launch_rt(rt_xpass_kernel<false, LR>, grid, LR::kThreads, LR::kSmem, s, a.pl.pdl, a);
}
template <int W, int G, int MB, int R1, int R2, int R3> void l_xconv(const XconvArgs& a, cudaStream_t s) {
    QP_RT_LR
    if (a.nout > 1) launch_rt(rt_xconv_kernel<true, LR>, x_grid<LR>(a.nzh), LR::kThreads, smem_many<LR>(), s, a.pl.pdl, a);
    else launch_rt(rt_xconv_kernel<false, LR>, x_grid<LR>(a.nzh), LR::kThreads, LR::kSmem, s, a.pl.pdl, a);
}
template <class K> bool up(K k, size_t bytes) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) != cudaSuccess;
}
template <int W, int G, int MB, int R1, int R2, int R3> int l_limits() {
    QP_RT_LR
    static_assert(smem_many<LR>() <= QP_SMEM_DYN_MAX, "lines of an entry fit a CTA's shared memory");
    bool bad = up(rt_xpass_kernel<true, LR>, LR::kSmem) | up(rt_xpass_kernel<false, LR>, LR::kSmem) |
               up(rt_xconv_kernel<false, LR>, LR::kSmem) | up(rt_xconv_kernel<true, LR>, smem_many<LR>());
#if QP_RT_GROUP < QP_RT_NWIDE
    bad |= up(rt_xexact_kernel<LR>, LR::kSmem);
#endif
    return bad;
}

bool g_xpass(const AcXArgs& a, cudaStream_t s) {
#define C_(ID, W, G, MB, R1, R2, R3, COST) \
    case ID: l_xpass<W, G, MB, R1, R2, R3>(a, s); break;
    QP_RT_SWITCH(a.pl.rt, C_)
#undef C_
}
bool g_xconv(const XconvArgs& a, cudaStream_t s) {
#define C_(ID, W, G, MB, R1, R2, R3, COST) \
    case ID: l_xconv<W, G, MB, R1, R2, R3>(a, s); break;
    QP_RT_SWITCH(a.pl.rt, C_)
#undef C_
}
#if QP_RT_GROUP < QP_RT_NWIDE
template <int W, int G, int MB, int R1, int R2, int R3> void l_xexact(const VxsArgs& a, cudaStream_t s) {
    QP_RT_LR
    launch_rt(rt_xexact_kernel<LR>, x_grid<LR>(a.nzh), LR::kThreads, LR::kSmem, s, a.pl.pdl, a);
}
bool g_xexact(const VxsArgs& a, cudaStream_t s) {
#define C_(ID, W, G, MB, R1, R2, R3, COST) \
    case ID: l_xexact<W, G, MB, R1, R2, R3>(a, s); break;
    QP_RT_SWITCH(a.pl.rt, C_)
#undef C_
}
#else
constexpr bool (*g_xexact)(const VxsArgs&, cudaStream_t) = nullptr;
#endif
int g_limits() {
    int bad = 0;
#define C_(ID, W, G, MB, R1, R2, R3, COST) bad |= l_limits<W, G, MB, R1, R2, R3>();
    QP_RT_ENTRIES(C_)
#undef C_
    return bad;
}

}  // namespace

extern const RtGroup QP_RT_CAT2(rt_group_, QP_RT_GROUP);
const RtGroup QP_RT_CAT2(rt_group_, QP_RT_GROUP) = {g_xpass, g_xconv, g_xexact, g_limits};

}  // namespace qp
