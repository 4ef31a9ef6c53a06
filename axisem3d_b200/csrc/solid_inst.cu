// The solid stiffness kernels of one precision and rheology: compiled once per pair with
// -DAXG_INST_T, -DAXG_INST_AT (arithmetic and SLS-state types) and -DAXG_INST_RHEO.
#include "solid_pick.cuh"

namespace axg {

// NS: the register-resident SLS recursions are built for 3 and 5 SLS (3-D slices and
// 1-D Fourier slots); other counts take the generic path
template <class T, class AT, int RHEO, int ATT, bool RTZ>
static SolidKernel<T, AT> pick3(int nsls, bool fft) {
#ifndef AXG_GENERIC_SLS_ONLY
    if constexpr (ATT != ATT_NONE) {
        if (fft && nsls == 3) return solid_stiffness_kernel<T, AT, RHEO, ATT, RTZ, 3, true>;
        if (fft && nsls == 5) return solid_stiffness_kernel<T, AT, RHEO, ATT, RTZ, 5, true>;
        if (nsls == 3) return solid_stiffness_kernel<T, AT, RHEO, ATT, RTZ, 3>;
        if (nsls == 5) return solid_stiffness_kernel<T, AT, RHEO, ATT, RTZ, 5>;
    }
#endif
    if constexpr (ATT == ATT_NONE) {
        if (fft) return solid_stiffness_kernel<T, AT, RHEO, ATT, RTZ, 0, true>;
    }
    return solid_stiffness_kernel<T, AT, RHEO, ATT, RTZ, 0>;
}
template <class T, class AT, int RHEO, int ATT, bool RTZ>
static Solid1DKernel<T, AT> pick3_1d(int nsls) {
#ifndef AXG_GENERIC_SLS_ONLY
    if constexpr (ATT != ATT_NONE) {
        if (nsls == 3) return solid_1d_kernel<T, AT, RHEO, ATT, RTZ, 3>;
        if (nsls == 5) return solid_1d_kernel<T, AT, RHEO, ATT, RTZ, 5>;
    }
#endif
    return solid_1d_kernel<T, AT, RHEO, ATT, RTZ, 0>;
}
// isotropic stress is the same in both frames: no RTZ instantiation
template <class T, class AT, int RHEO, int ATT>
static SolidKernel<T, AT> pick2(bool rtz, int nsls, bool fft) {
    if constexpr (RHEO != RHEO_ISO)
        if (rtz) return pick3<T, AT, RHEO, ATT, true>(nsls, fft);
    return pick3<T, AT, RHEO, ATT, false>(nsls, fft);
}
template <class T, class AT, int RHEO, int ATT>
static Solid1DKernel<T, AT> pick2_1d(bool rtz, int nsls) {
    if constexpr (RHEO != RHEO_ISO)
        if (rtz) return pick3_1d<T, AT, RHEO, ATT, true>(nsls);
    return pick3_1d<T, AT, RHEO, ATT, false>(nsls);
}
template <class T, class AT, int RHEO>
SolidKernel<T, AT> pick_solid_of(int att, bool rtz, int nsls, bool fft) {
    switch (att) {
        case ATT_NONE: return pick2<T, AT, RHEO, ATT_NONE>(rtz, nsls, fft);
        case ATT_FULL: return pick2<T, AT, RHEO, ATT_FULL>(rtz, nsls, fft);
        default: return pick2<T, AT, RHEO, ATT_CG4>(rtz, nsls, fft);
    }
}
template <class T, class AT, int RHEO>
Solid1DKernel<T, AT> pick_solid_1d_of(int att, bool rtz, int nsls) {
    switch (att) {
        case ATT_NONE: return pick2_1d<T, AT, RHEO, ATT_NONE>(rtz, nsls);
        case ATT_FULL: return pick2_1d<T, AT, RHEO, ATT_FULL>(rtz, nsls);
        default: return pick2_1d<T, AT, RHEO, ATT_CG4>(rtz, nsls);
    }
}

template <class T, class AT, int RHEO, int ATT>
static PrtKernel<T, AT> pick_prt2(bool is3d, bool rtz) {
    if (is3d) return rtz ? solid_prt_kernel<T, AT, RHEO, ATT, true, true> : solid_prt_kernel<T, AT, RHEO, ATT, true, false>;
    return rtz ? solid_prt_kernel<T, AT, RHEO, ATT, false, true> : solid_prt_kernel<T, AT, RHEO, ATT, false, false>;
}
template <class T, class AT, int RHEO>
PrtKernel<T, AT> pick_prt_of(int att, bool is3d, bool rtz) {
    switch (att) {
        case ATT_NONE: return pick_prt2<T, AT, RHEO, ATT_NONE>(is3d, rtz);
        case ATT_FULL: return pick_prt2<T, AT, RHEO, ATT_FULL>(is3d, rtz);
        default: return pick_prt2<T, AT, RHEO, ATT_CG4>(is3d, rtz);
    }
}

template SolidKernel<AXG_INST_T, AXG_INST_AT> pick_solid_of<AXG_INST_T, AXG_INST_AT, AXG_INST_RHEO>(int, bool, int,
                                                                                                   bool);
template Solid1DKernel<AXG_INST_T, AXG_INST_AT> pick_solid_1d_of<AXG_INST_T, AXG_INST_AT, AXG_INST_RHEO>(int, bool,
                                                                                                        int);
template PrtKernel<AXG_INST_T, AXG_INST_AT> pick_prt_of<AXG_INST_T, AXG_INST_AT, AXG_INST_RHEO>(int, bool, bool);

}  // namespace axg
