// solid_pick.cuh -- the instantiations of the solid stiffness kernels and their choice by
// element kind. Each (precision, rheology) pair is compiled in a translation unit of its own
// (solid_inst.cu, once per pair), so that the kernels of one library build side by side; the
// engine only takes the function pointers.
#pragma once

#include "prt_kernel.cuh"
#include "solid1d_kernel.cuh"
#include "solid_kernel.cuh"

namespace axg {

template <class T, class AT>
using SolidKernel = void (*)(const SolidArgs<T, AT>, int, int, int, int, size_t);
template <class T, class AT>
using Solid1DKernel = void (*)(const SolidArgs<T, AT>, int);
template <class T, class AT>
using PrtKernel = void (*)(const PrtArgs<T, AT>, int, int, int, size_t);

// one rheology's kernels (defined in solid_inst.cu)
template <class T, class AT, int RHEO>
SolidKernel<T, AT> pick_solid_of(int att, bool rtz, int nsls, bool fft);
template <class T, class AT, int RHEO>
Solid1DKernel<T, AT> pick_solid_1d_of(int att, bool rtz, int nsls);
template <class T, class AT, int RHEO>
PrtKernel<T, AT> pick_prt_of(int att, bool is3d, bool rtz);

template <class T, class AT>
SolidKernel<T, AT> pick_solid(int rheo, int att, bool rtz, int nsls, bool fft) {
    switch (rheo) {
        case RHEO_ISO: return pick_solid_of<T, AT, RHEO_ISO>(att, rtz, nsls, fft);
        case RHEO_TISO: return pick_solid_of<T, AT, RHEO_TISO>(att, rtz, nsls, fft);
        default: return pick_solid_of<T, AT, RHEO_ANISO>(att, rtz, nsls, fft);
    }
}
template <class T, class AT>
Solid1DKernel<T, AT> pick_solid_1d(int rheo, int att, bool rtz, int nsls) {
    switch (rheo) {
        case RHEO_ISO: return pick_solid_1d_of<T, AT, RHEO_ISO>(att, rtz, nsls);
        case RHEO_TISO: return pick_solid_1d_of<T, AT, RHEO_TISO>(att, rtz, nsls);
        default: return pick_solid_1d_of<T, AT, RHEO_ANISO>(att, rtz, nsls);
    }
}
template <class T, class AT>
PrtKernel<T, AT> pick_prt(int rheo, int att, bool is3d, bool rtz) {
    switch (rheo) {
        case RHEO_ISO: return pick_prt_of<T, AT, RHEO_ISO>(att, is3d, rtz);
        case RHEO_TISO: return pick_prt_of<T, AT, RHEO_TISO>(att, is3d, rtz);
        default: return pick_prt_of<T, AT, RHEO_ANISO>(att, is3d, rtz);
    }
}

}  // namespace axg
