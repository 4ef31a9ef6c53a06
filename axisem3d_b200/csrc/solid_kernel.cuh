// solid_kernel.cuh -- fused stiffness of solid spectral elements (nPol = 4) with properties per
// azimuthal slice (3-D elements; those without are in solid1d_kernel.cuh).
//
// One team of threads evaluates one element at a time, entirely on chip:
//   gather u from the points (zero-padded above each point's nu)
//     SolidPoint::scatterDisplToElement   (SOLVER/src/core/point/SolidPoint.hpp:82-98)
//   GLL gradient + analytic d/dphi, axial L'Hopital rows
//     GradientQuadrature::computeGrad6    (SOLVER/src/core/element/grad/GradientQuadrature.hpp:207-231)
//   [RTZ] CoordTransformSpherical::transformSPZ_RTZ6 (crd/CoordTransformSpherical.hpp:186-216)
//   Fourier -> phi slices (direct DFT in shared memory, FFTW conventions,
//     SOLVER/src/core/fft/SolverFFTW.hpp:101-172), strainToStress_CD per slice,
//     slices -> Fourier
//   Isotropic / TransverselyIsotropic / Anisotropic::strainToStress
//     (material/elastic/anisotropy/*.hpp)
//   AttenuationFull / AttenuationCG4::apply (material/elastic/attenuation/*.hpp)
//   [RTZ] transformRTZ_SPZ6
//   GradientQuadrature::computeQuad6 (GradientQuadrature.hpp:294-324)
//   scatter-add: point.stiff -= f   SolidPoint::gatherStiffFromElement (SolidPoint.hpp:101-109)
//
// Shared memory per team (T = float or double, C = complex T):
//   geometry 10 x 25 T, trig 4 x 25 T, twiddles 2 x nr T,
//   region A: 6 x nu x 25 C  (strain E, then stress S, then quadrature X/Y)
//   region B: max(3 x mt x 25 C, nr x 6 x qc T)  (u, then stress slices, then A terms)
// The gather + gradient and the two quadrature passes run over tiles of mt modes (each
// Fourier mode is independent there), so region B holds one tile of u and of the A terms;
// mt = nu unless the element's nr is too large for that (one tile, the common case).
#pragma once

#include "common.cuh"
#include "slice_fft.cuh"

namespace axg {

constexpr int RHEO_ISO = 0, RHEO_TISO = 1, RHEO_ANISO = 2;
constexpr int ATT_NONE = 0, ATT_FULL = 1, ATT_CG4 = 2;
// register blocking of the two phi transforms and the occupancy target of the
// solid kernel (build-time tuning knobs)
#ifndef AXG_KB
#define AXG_KB 2
#endif
#ifndef AXG_AB
#define AXG_AB 2
#endif
#ifndef AXG_SOLID_MIN_BLOCKS
#define AXG_SOLID_MIN_BLOCKS 2
#endif
#ifndef AXG_KP
#define AXG_KP 2
#endif
// the same two blockings for elements without attenuation, whose slice pass holds no SLS
// state in registers and can afford wider blocks
#ifndef AXG_KP_ELASTIC
#define AXG_KP_ELASTIC 4
#endif
#ifndef AXG_AB_ELASTIC
#define AXG_AB_ELASTIC 4
#endif
// 1 = L2 prefetch of an element's slice operands (moduli, attenuation moduli, SLS state)
// at the start of its slice phase
#ifndef AXG_PREFETCH_SLICES
#define AXG_PREFETCH_SLICES 1
#endif
// 1 = when a chunk holds all 25 points (and, for the slice -> Fourier pass, outside RTZ
// elements), the two direct-sum passes give each thread 6 consecutive columns of the
// (component, point) block instead of the 6 components of one point, read and written as
// 16- / 8-byte vectors, and order the threads 5 column groups by pair (or mode) groups, so
// that a warp touches few distinct words of region A, region B and the twiddle table per step
#ifndef AXG_COLUMN_TILES
#define AXG_COLUMN_TILES 1
#endif
// unrolling of the mode loop (Fourier -> slice) and of the slice loop (slice -> Fourier) of
// the column-tiled passes
#ifndef AXG_DFT_UNROLL
#define AXG_DFT_UNROLL 1
#endif
constexpr int KP = AXG_KP;   // slice pairs per thread in the paired Fourier -> slice pass
constexpr int KB = AXG_KB;   // slices per thread in the Fourier -> slice transform
constexpr int AB = AXG_AB;   // modes per thread in the slice -> Fourier transform
constexpr int DFT_UNROLL = AXG_DFT_UNROLL;

template <class T, class AT>
struct SolidArgs {
    int n_elem;
    const int *nr;             // [n]
    const int *pts;            // [n*25]
    const uint8_t *axial;      // [n]
    const T *geom;             // [n][10][25]
    const T *trig;             // [n][4][25] sin t, cos t, sin 2t, cos 2t (RTZ only)
    const T *mod;              // moduli pool
    const int64_t *mod_off;    // [n]
    const T *attmod;           // dlambda, dmu pool
    const int64_t *att_off;    // [n]
    AT *state;                 // attenuation state pool
    const int64_t *state_off;  // [n] in AT units
    const int *pt_off;         // [npoints] first mode of each point
    const int *pt_nu;          // [npoints]
    const cx_t<T> *displ;      // [sum nu][3]
    cx_t<T> *stiff;            // [sum nu][3]
    const T *tw;               // twiddle pool: for each nr, nr cos then nr sin
    const int *tw_off;         // [nr_max + 1]
    int nsls;
    AT alpha[8], beta[8], gamma[8];
    const T *gmat;             // [2][25]: G_GLL, G_GLJ (row-major, G(j,i) = l_j'(x_i))
    int nwave;                 // wavefields sharing the mesh (independent sources)
    size_t fstride;            // complex values between wavefields in displ / stiff
    size_t sstride;            // AT values between wavefields in the state pool
    const unsigned *fft_plan;  // [nr_max + 1] radices of every nr that takes the FFT (fft_factors), 0 = direct sums
    const int2 *tab;           // [n][25] first mode and number of modes of the element's points
    const int4 *tiles;         // 1-D elements: (element, first mode, modes, nu | axial << 30) per block
};

// shared memory layout of one team
struct TeamLayout {
    int nr_max, nu_max, qc;
    size_t geom, trig, ipt, tw, regA, regB, total;
};

template <class T>
__host__ __device__ inline TeamLayout team_layout(int nr_max, int qc, int mt) {
    TeamLayout L;
    L.nr_max = nr_max;
    L.nu_max = nr_max / 2 + 1;
    L.qc = qc;
    mt = mt < L.nu_max ? mt : L.nu_max;
    size_t o = 0;
    auto al = [](size_t x) { return (x + 15) & ~(size_t)15; };
    L.geom = o; o = al(o + 10 * 25 * sizeof(T));
    L.trig = o; o = al(o + 4 * 25 * sizeof(T));
    L.tw = o;   o = al(o + 2 * (size_t)nr_max * sizeof(T));
    L.regA = o; o = al(o + 6 * (size_t)L.nu_max * 25 * 2 * sizeof(T));
    size_t b1 = 3 * (size_t)mt * 25 * 2 * sizeof(T);
    size_t b2 = (size_t)nr_max * 6 * qc * sizeof(T);
    L.regB = o; o = al(o + (b1 > b2 ? b1 : b2));
    L.total = o;
    return L;
}

// six consecutive complex / real values of a team's shared buffers as 16- or 8-byte vectors;
// complex groups start on 16 bytes, real groups on 2 T (the callers' column groups start at
// even offsets of 16-byte aligned regions)
template <class T>
__device__ __forceinline__ void ld6c(const cx_t<T> *p, cx_t<T> (&v)[6]) {
    if constexpr (sizeof(T) == 4) {
        const float4 *q = reinterpret_cast<const float4 *>(p);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const float4 t = q[i];
            v[2 * i] = mk<T>(t.x, t.y);
            v[2 * i + 1] = mk<T>(t.z, t.w);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 6; i++) v[i] = p[i];
    }
}
template <class T>
__device__ __forceinline__ void st6c(cx_t<T> *p, const cx_t<T> (&v)[6]) {
    if constexpr (sizeof(T) == 4) {
        float4 *q = reinterpret_cast<float4 *>(p);
#pragma unroll
        for (int i = 0; i < 3; i++) q[i] = make_float4(v[2 * i].x, v[2 * i].y, v[2 * i + 1].x, v[2 * i + 1].y);
    } else {
#pragma unroll
        for (int i = 0; i < 6; i++) p[i] = v[i];
    }
}
template <class T>
__device__ __forceinline__ void ld6r(const T *p, T (&v)[6]) {
    const cx_t<T> *q = reinterpret_cast<const cx_t<T> *>(p);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const cx_t<T> t = q[i];
        v[2 * i] = t.x;
        v[2 * i + 1] = t.y;
    }
}
template <class T>
__device__ __forceinline__ void st6r(T *p, const T (&v)[6]) {
    cx_t<T> *q = reinterpret_cast<cx_t<T> *>(p);
#pragma unroll
    for (int i = 0; i < 3; i++) q[i] = mk<T>(v[2 * i], v[2 * i + 1]);
}

// ------------------------------------------------------------ rheology ---
// Isotropic::strainToStress (Isotropic.hpp:154-170); 2 mu is exact as mu + mu
template <class V, class R>
__device__ __forceinline__ void stress_iso(const V e[6], V s[6], R lam, R mu) {
    R mu2 = mu + mu;
    V sii = cscale(cadd(cadd(e[0], e[1]), e[2]), lam);
    s[0] = cmac(sii, e[0], mu2);
    s[1] = cmac(sii, e[1], mu2);
    s[2] = cmac(sii, e[2], mu2);
    s[3] = cscale(e[3], mu);
    s[4] = cscale(e[4], mu);
    s[5] = cscale(e[5], mu);
}
// TransverselyIsotropic::strainToStress (TransverselyIsotropic.hpp:160-180)
template <class V, class R>
__device__ __forceinline__ void stress_tiso(const V e[6], V s[6], R A, R C, R F, R L, R Nn) {
    R mN2 = -(Nn + Nn);
    V t3 = cadd(e[0], e[1]);
    V t4 = cmac(cscale(e[2], F), t3, A);
    s[0] = cmac(t4, e[1], mN2);
    s[1] = cmac(t4, e[0], mN2);
    s[2] = cmac(cscale(e[2], C), t3, F);
    s[3] = cscale(e[3], L);
    s[4] = cscale(e[4], L);
    s[5] = cscale(e[5], Nn);
}
// Anisotropic::strainToStress (Anisotropic.hpp:202-274); c = upper triangle row-major
template <class V, class R>
__device__ __forceinline__ void stress_aniso(const V e[6], V s[6], const R c[21]) {
    const int idx[6][6] = {{0, 1, 2, 3, 4, 5},      {1, 6, 7, 8, 9, 10},
                           {2, 7, 11, 12, 13, 14},  {3, 8, 12, 15, 16, 17},
                           {4, 9, 13, 16, 18, 19},  {5, 10, 14, 17, 19, 20}};
#pragma unroll
    for (int i = 0; i < 6; i++) {
        V acc = cscale(e[0], c[idx[i][0]]);
#pragma unroll
        for (int j = 1; j < 6; j++) acc = cmac(acc, e[j], c[idx[i][j]]);
        s[i] = acc;
    }
}

// scalar "complex" wrapper so that the rheology templates serve real slices too
template <class T> struct re1 { T x; };
template <class T> __device__ __forceinline__ re1<T> cadd(re1<T> a, re1<T> b) { return {a.x + b.x}; }
template <class T> __device__ __forceinline__ re1<T> csub(re1<T> a, re1<T> b) { return {a.x - b.x}; }
template <class T, class R> __device__ __forceinline__ re1<T> cscale(re1<T> a, R s) { return {a.x * (T)s}; }
template <class T, class R> __device__ __forceinline__ re1<T> cmac(re1<T> acc, re1<T> a, R s) { return {acc.x + a.x * (T)s}; }

template <int RHEO, class T, class V>
__device__ __forceinline__ void elastic_at(const T *mod, int nslice, int slice, int q,
                                           const V e[6], V s[6]) {
    const size_t ns = (size_t)nslice * 25, o = (size_t)slice * 25 + q;
    if constexpr (RHEO == RHEO_ISO) {
        stress_iso(e, s, __ldg(mod + o), __ldg(mod + ns + o));
    } else if constexpr (RHEO == RHEO_TISO) {
        stress_tiso(e, s, __ldg(mod + o), __ldg(mod + ns + o), __ldg(mod + 2 * ns + o),
                    __ldg(mod + 3 * ns + o), __ldg(mod + 4 * ns + o));
    } else {
        T c[21];
#pragma unroll
        for (int k = 0; k < 21; k++) c[k] = __ldg(mod + k * ns + o);
        stress_aniso(e, s, c);
    }
}

// CoordTransformSpherical::transformSPZ_RTZ6 / transformRTZ_SPZ6 (one point of one mode)
template <class V, class T>
__device__ __forceinline__ void spz_to_rtz6(V e[6], T s1, T c1, T s2, T c2) {
    const T half = (T)0.5;
    V s02 = cadd(e[0], e[2]), d02 = csub(e[0], e[2]);
    e[0] = cscale(csub(cmac(s02, d02, c2), cscale(e[4], s2)), half);
    e[2] = csub(s02, e[0]);
    e[4] = cmac(cscale(e[4], c2), d02, s2);
    V t3 = e[3];
    e[3] = cmac(cscale(t3, c1), e[5], s1);
    e[5] = csub(cscale(e[5], c1), cscale(t3, s1));
}
template <class V, class T>
__device__ __forceinline__ void rtz_to_spz6(V s[6], T s1, T c1, T s2, T c2) {
    const T half = (T)0.5;
    V s02 = cadd(s[0], s[2]), d02 = csub(s[0], s[2]);
    s[0] = cmac(cscale(cmac(s02, d02, c2), half), s[4], s2);
    s[2] = csub(s02, s[0]);
    s[4] = csub(cscale(s[4], c2), cscale(cscale(d02, s2), half));
    V t3 = s[3];
    s[3] = csub(cscale(t3, c1), cscale(s[5], s1));
    s[5] = cmac(cscale(s[5], c1), t3, s1);
}

// ----------------------------------------------------------- attenuation ---
// One point of one mode (complex) or slice (real):
//   stress -= sum_l mem_l; mem_l = alpha_l mem_l + beta_l dstress;
//   dstress = iso(dlambda, dmu)(strain); mem_l += gamma_l dstress
// (AttenuationFull.hpp:189-207, Attenuation.hpp:92-134). The state (dstress,
// mem) lives in AT (double in the mixed-precision mode) and is streamed from
// and to HBM once per step.
template <bool CPLX, class AT, class V>
__device__ __forceinline__ AT part(const V &v, int w) {
    if constexpr (CPLX) return (AT)(w ? v.y : v.x);
    else return (AT)v.x;
}

template <class T, class AT, bool CPLX, class V>
__device__ __forceinline__ void attenuate(const SolidArgs<T, AT> &a, AT *state, size_t nslot,
                                          size_t slot, const V e[6], V s[6], T dl, T dm) {
    constexpr int W = CPLX ? 2 : 1;
    AT *dst = state;                             // [6][nslot] (x W)
    AT *mem = state + 6 * nslot * W;             // [nsls][6][nslot] (x W)
    const size_t sls = 6 * nslot * W;
    AT ds[6][W], sv[6][W];
#pragma unroll
    for (int d = 0; d < 6; d++)
#pragma unroll
        for (int w = 0; w < W; w++) {
            ds[d][w] = dst[(d * nslot + slot) * W + w];
            sv[d][w] = part<CPLX, AT>(s[d], w);
        }
    for (int l = 0; l < a.nsls; l++) {
        AT *m = mem + l * sls;
        const AT al = a.alpha[l], be = a.beta[l];
#pragma unroll
        for (int d = 0; d < 6; d++)
#pragma unroll
            for (int w = 0; w < W; w++) {
                AT mv = m[(d * nslot + slot) * W + w];
                sv[d][w] -= mv;
                m[(d * nslot + slot) * W + w] = al * mv + be * ds[d][w];
            }
    }
    // new dstress from the strain (Isotropic::strainToStress with dlambda, dmu)
    const AT lam = (AT)dl, mu = (AT)dm, mu2 = mu + mu;
#pragma unroll
    for (int w = 0; w < W; w++) {
        const AT e0 = part<CPLX, AT>(e[0], w), e1 = part<CPLX, AT>(e[1], w),
                 e2 = part<CPLX, AT>(e[2], w);
        const AT sii = (e0 + e1 + e2) * lam;
        ds[0][w] = sii + e0 * mu2;
        ds[1][w] = sii + e1 * mu2;
        ds[2][w] = sii + e2 * mu2;
        ds[3][w] = part<CPLX, AT>(e[3], w) * mu;
        ds[4][w] = part<CPLX, AT>(e[4], w) * mu;
        ds[5][w] = part<CPLX, AT>(e[5], w) * mu;
    }
#pragma unroll
    for (int d = 0; d < 6; d++)
#pragma unroll
        for (int w = 0; w < W; w++) dst[(d * nslot + slot) * W + w] = ds[d][w];
    for (int l = 0; l < a.nsls; l++) {
        AT *m = mem + l * sls;
        const AT ga = a.gamma[l];
#pragma unroll
        for (int d = 0; d < 6; d++)
#pragma unroll
            for (int w = 0; w < W; w++) m[(d * nslot + slot) * W + w] += ga * ds[d][w];
    }
#pragma unroll
    for (int d = 0; d < 6; d++) {
        if constexpr (CPLX) { s[d].x = (T)sv[d][0]; s[d].y = (T)sv[d][1]; }
        else s[d].x = (T)sv[d][0];
    }
}

// L2 prefetch of [p, p + bytes), 128-byte lines spread over the team; every
// address issued lies inside the region (lines are aligned down only at the start,
// and pools are 256-byte aligned allocations)
__device__ __forceinline__ void prefetch_l2(const void *p, size_t bytes, int lane, int team) {
    const uintptr_t a1 = (uintptr_t)p + bytes;
    uintptr_t a = ((uintptr_t)p & ~(uintptr_t)127) + (uintptr_t)lane * 128;
    for (; a < a1; a += (uintptr_t)team * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
}

// SLS recursion on one real slice point with the state already in registers
// (same steps and order as attenuate<>; NS = number of SLS, a compile-time size)
template <int NS, class T, class AT>
__device__ __forceinline__ void attenuate_regs(const AT *alpha, const AT *beta, const AT *gamma, AT ds[6],
                                               AT mem[NS][6], const T e[6], T s[6], T dl, T dm) {
    AT sv[6];
#pragma unroll
    for (int d = 0; d < 6; d++) sv[d] = (AT)s[d];
#pragma unroll
    for (int l = 0; l < NS; l++)
#pragma unroll
        for (int d = 0; d < 6; d++) {
            sv[d] -= mem[l][d];
            mem[l][d] = alpha[l] * mem[l][d] + beta[l] * ds[d];
        }
    const AT lam = (AT)dl, mu = (AT)dm, mu2 = mu + mu;
    const AT e0 = (AT)e[0], e1 = (AT)e[1], e2 = (AT)e[2];
    const AT sii = (e0 + e1 + e2) * lam;
    ds[0] = sii + e0 * mu2;
    ds[1] = sii + e1 * mu2;
    ds[2] = sii + e2 * mu2;
    ds[3] = (AT)e[3] * mu;
    ds[4] = (AT)e[4] * mu;
    ds[5] = (AT)e[5] * mu;
#pragma unroll
    for (int l = 0; l < NS; l++)
#pragma unroll
        for (int d = 0; d < 6; d++) mem[l][d] += gamma[l] * ds[d];
#pragma unroll
    for (int d = 0; d < 6; d++) s[d] = (T)sv[d];
}

__device__ __forceinline__ int cg4_slot(int q) {
    // (1,1) (1,3) (3,1) (3,3) -> 0..3, else -1
    return q == 6 ? 0 : q == 8 ? 1 : q == 16 ? 2 : q == 18 ? 3 : -1;
}

// ----------------------------------------------------------------- kernel ---
// Largest block: 512 threads where an element can be too large for two blocks per SM (FP64, and
// the large nr of the FFT instantiations), so that the one block still fills the register file.
template <class T, bool FFT>
constexpr int solid_threads() { return FFT || sizeof(T) == 8 ? 512 : 256; }

// NS: compile-time number of SLS for the register-resident recursion; 0 = the generic path with
// the count read at run time
// FFT: the instantiation that holds the slice FFTs (buckets with large nr); the others
// keep only the direct sums, so the FFT code costs them no registers
template <class T, class AT, int RHEO, int ATT, bool RTZ, int NS, bool FFT = false>
__global__ void __launch_bounds__(solid_threads<T, FFT>(), solid_threads<T, FFT>() == 512 ? 1 : AXG_SOLID_MIN_BLOCKS)
solid_stiffness_kernel(const SolidArgs<T, AT> a, const int nr_max, const int qc_max, const int mt_max,
                       const int teams_per_cta, const size_t team_bytes) {
    using C = cx_t<T>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // register blocking of the paired Fourier -> slice pass and of the slice -> Fourier pass
    constexpr int KPc = ATT == ATT_NONE ? AXG_KP_ELASTIC : KP;
    constexpr int ABc = ATT == ATT_NONE ? AXG_AB_ELASTIC : AB;
    const int TEAM = blockDim.x / teams_per_cta;
    const int team = threadIdx.x / TEAM;
    const int lane = threadIdx.x % TEAM;
    // G tables, once per CTA
    __shared__ T sGll[25], sGlj[25];
    for (int i = threadIdx.x; i < 25; i += blockDim.x) {
        sGll[i] = a.gmat[i];
        sGlj[i] = a.gmat[25 + i];
    }
    __syncthreads();
    if (team >= teams_per_cta) return;

    const TeamLayout L = team_layout<T>(nr_max, qc_max, mt_max);
    unsigned char *base = smem_raw + (size_t)team * team_bytes;
    T *sGeo = reinterpret_cast<T *>(base + L.geom);
    T *sTrig = reinterpret_cast<T *>(base + L.trig);
    T *sTw = reinterpret_cast<T *>(base + L.tw);
    C *rA = reinterpret_cast<C *>(base + L.regA);
    C *rBc = reinterpret_cast<C *>(base + L.regB);
    T *rBr = reinterpret_cast<T *>(base + L.regB);

    // geometry aliases
    const T *dsdxii = sGeo, *dsdeta = sGeo + 25, *dzdxii = sGeo + 50, *dzdeta = sGeo + 75,
            *invs = sGeo + 100;
    const T *dsdxii_if = sGeo + 125, *dsdeta_if = sGeo + 150, *dzdxii_if = sGeo + 175,
            *dzdeta_if = sGeo + 200, *invs_if = sGeo + 225;

    const int stride = gridDim.x * teams_per_cta;
    for (int e = blockIdx.x * teams_per_cta + team; e < a.n_elem; e += stride) {
        const int nr = a.nr[e];
        const int nu = nr / 2 + 1;
        const bool axial = a.axial[e] != 0;
        const T *Gxi = axial ? sGlj : sGll;
        // ---------------- element header -> shared memory ----------------
        for (int i = lane; i < 250; i += TEAM) sGeo[i] = a.geom[(size_t)e * 250 + i];
        if constexpr (RTZ)
            for (int i = lane; i < 100; i += TEAM) sTrig[i] = a.trig[(size_t)e * 100 + i];
        const int2 *tab = a.tab + (size_t)e * 25;
        {
            const T *tw = a.tw + a.tw_off[nr];
            // interleaved (cos, sin) pairs: one 2-word shared load per twiddle
            for (int i = lane; i < 2 * nr; i += TEAM) sTw[i] = (i & 1) ? tw[nr + (i >> 1)] : tw[i >> 1];
        }
        // every wavefield of the batch reuses the element header; the barrier after the first gather
        // covers it
        for (int w = blockIdx.y; w < a.nwave; w += gridDim.y) {
        const C *displw = a.displ + (size_t)w * a.fstride;
        C *stiffw = a.stiff + (size_t)w * a.fstride;
        AT *statew = a.state + (size_t)w * a.sstride;
        const int64_t moff = a.mod_off[e];
        const int nslice = nr;
        for (int t0 = 0; t0 < nu; t0 += mt_max) {
        const int mt = min(mt_max, nu - t0);
        // ---------------- gather displacement: U[a - t0][c][q] in region B ----------------
        const float rmt = 1.f / (float)mt;
        for (int i = lane; i < mt * 25; i += TEAM) {
            const int q = div_n(i, mt, rmt), la = i - q * mt, al = t0 + la;
            const int2 on = __ldg(tab + q);
            C u0 = mk<T>(0, 0), u1 = u0, u2 = u0;
            if (al < on.y) {
                const C *src = displw + ((size_t)on.x + al) * 3;
                u0 = src[0]; u1 = src[1]; u2 = src[2];
            }
            rBc[(la * 3 + 0) * 25 + q] = u0;
            rBc[(la * 3 + 1) * 25 + q] = u1;
            rBc[(la * 3 + 2) * 25 + q] = u2;
        }
        team_sync(team, TEAM);

        // ---------------- gradient (computeGrad6) ----------------
        for (int i = lane; i < mt * 25; i += TEAM) {
            const int la = i / 25, q = i - la * 25, al = t0 + la;
            const int ii = q / 5, jj = q - ii * 5;
            const C *U = rBc + la * 75;
            C X[3], Y[3];
#pragma unroll
            for (int c = 0; c < 3; c++) { X[c] = mk<T>(0, 0); Y[c] = mk<T>(0, 0); }
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const T gx = Gxi[k * 5 + ii];        // GT_xi(ii, k)
                const T gy = sGll[k * 5 + jj];       // G_GLL(k, jj)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    X[c] = cmac(X[c], U[c * 25 + k * 5 + jj], gx);
                    Y[c] = cmac(Y[c], U[c * 25 + ii * 5 + k], gy);
                }
            }
            const T ze = dzdeta[q], zx = dzdxii[q], se = dsdeta[q], sx = dsdxii[q];
            C eps[6], S[3];
#pragma unroll
            for (int c = 0; c < 3; c++) S[c] = cmac(cscale(Y[c], zx), X[c], ze);
            eps[0] = S[0];
            eps[4] = cadd(cmac(cscale(Y[0], sx), X[0], se), S[2]);
            eps[3] = cmac(cscale(Y[1], sx), X[1], se);
            eps[2] = cmac(cscale(Y[2], sx), X[2], se);
            // lower-order terms A / s; on the axis (L'Hopital) dA / ds, the same combination of
            // the derivatives
            const T alf = (T)al;
            const bool lim = axial && ii == 0;
            const C b0 = lim ? S[0] : U[q], b1 = lim ? S[1] : U[25 + q], b2 = lim ? S[2] : U[50 + q];
            const T is = lim ? (T)1 : invs[q];
            eps[5] = cadd(S[1], cscale(csub(cia(alf, b0), b1), is));
            eps[1] = cscale(cadd(cia(alf, b1), b0), is);
            eps[3] = cadd(eps[3], cscale(cia(alf, b2), is));
            if constexpr (RTZ) {
                spz_to_rtz6(eps, sTrig[q], sTrig[25 + q], sTrig[50 + q], sTrig[75 + q]);
            }
#pragma unroll
            for (int d = 0; d < 6; d++) rA[(al * 6 + d) * 25 + q] = eps[d];
        }
        team_sync(team, TEAM);
        }   // mode tiles of the gather + gradient

        // ---------------- 3-D material: slices ----------------
        {
            using T2 = cx_t<T>;
            const T2 *tw2 = reinterpret_cast<const T2 *>(sTw);
            const T inv_nr = (T)1 / (T)nr;
            const int nkb = (nr + KB - 1) / KB;
            const int nab = (nu + ABc - 1) / ABc;
#if AXG_PREFETCH_SLICES
            if constexpr (NS > 0 || ATT == ATT_NONE) {
                // the slice operands of this element start moving into L2 now, so that the
                // stress pass finds them there after the Fourier -> slice pass
                constexpr int NM_ = RHEO == RHEO_ISO ? 2 : RHEO == RHEO_TISO ? 5 : 21;
                prefetch_l2(a.mod + moff, (size_t)NM_ * nr * 25 * sizeof(T), lane, TEAM);
                if constexpr (ATT != ATT_NONE) {
                    constexpr int NPA_ = ATT == ATT_CG4 ? 4 : 25;
                    const size_t slots = (size_t)nr * NPA_;
                    prefetch_l2(a.attmod + a.att_off[e], 2 * slots * sizeof(T), lane, TEAM);
                    prefetch_l2(statew + a.state_off[e], (size_t)(6 + 6 * NS) * slots * sizeof(AT), lane, TEAM);
                }
            }
#endif
            // the FFT path (register-resident slice path only): an nr the plan covers
            unsigned plan = 0;
            if constexpr (FFT && (NS > 0 || ATT == ATT_NONE)) {
                if (a.fft_plan) plan = __ldg(a.fft_plan + nr);
            }
            const bool use_fft = FFT && plan != 0;
            for (int q0 = 0; q0 < 25; q0 += qc_max) {
                const int qcnt = min(qc_max, 25 - q0);
                // slices of this chunk: [k][d][qq] reals in region B (direct sums) or, on the
                // FFT path, x_2p + i x_2p+1 of sample k in whichever view the C2R left them
                const FftView<T> vB{rBc, 3 * qcnt, qcnt}, vA{rA + q0, 75, 25};
                FftView<T> vs = vB, vo = vB;   // strain slices, stress slices
                if constexpr (NS > 0 || ATT == ATT_NONE) {
                constexpr int NM = RHEO == RHEO_ISO ? 2 : RHEO == RHEO_TISO ? 5 : 21;
                constexpr int NSR = NS > 0 ? NS : 1;
                constexpr int NPA = ATT == ATT_CG4 ? 4 : 25;
                const T *modp = a.mod + moff;
                const size_t nsl = (size_t)nslice * 25;
                if (FFT && use_fft) {
                    // from here on the chunk's columns of region A are free until the unpacking; the
                    // stress goes to the view the strain is not in, from which the passes back end
                    // in region B
                    vs = fft_run<T>(rA + q0, vA, vB, nr, qcnt, plan, tw2, team, lane, TEAM);
                    vo = vs.p == rBc ? vA : vB;
                } else {
                {
                // Register-resident slice path. Two passes:
                //  1. computeC2R, one thread per (slice pair, point): slices k and nr - k
                //     share their twiddles (cos equal, sin opposite), so one pass over the
                //     modes gives both, x_k = c0 + 2 (A - B) and x_{nr-k} = c0 + 2 (A + B)
                //     with A = sum Re(c) cos, B = sum Im(c) sin; the slice strains go to the
                //     slots of region B that the slice stresses later overwrite;
                //  2. one thread per (slice, point): the global operands of the point-slice
                //     (moduli, attenuation moduli, SLS state) are loaded into registers,
                //     stress and attenuation applied, the state stored back.
                // KPc slice pairs per thread: each mode value read from shared memory feeds
                // 2 KPc products
                const int npair = nr / 2 + 1;
                const int npb = (npair + KPc - 1) / KPc;
#if AXG_COLUMN_TILES
                if (qcnt == 25) {
                    // column n = d * 25 + q of the block: mode a at rA[a * 150 + n], slice k
                    // at rBr[k * 150 + n]; a thread takes KPc pairs x 6 columns
                    for (int i = lane; i < 25 * npb; i += TEAM) {
                        const int pb = (i / 5) % npb, n0 = 6 * ((i / (5 * npb)) * 5 + i % 5);
                        const int k0 = pb * KPc;
                        C AB[KPc][6];   // sums of Re cos and of Im sin, side by side
                        int j[KPc], kst[KPc];
#pragma unroll
                        for (int kk = 0; kk < KPc; kk++) {
                            j[kk] = 0;
                            kst[kk] = k0 + kk < npair ? k0 + kk : 0;
#pragma unroll
                            for (int c = 0; c < 6; c++) AB[kk][c] = mk<T>(0, 0);
                        }
#pragma unroll DFT_UNROLL
                        for (int al = 1; al < nu; al++) {
                            C ev[6];
                            ld6c<T>(rA + al * 150 + n0, ev);
#pragma unroll
                            for (int kk = 0; kk < KPc; kk++) {
                                j[kk] += kst[kk];
                                j[kk] = j[kk] >= nr ? j[kk] - nr : j[kk];
                                const T2 w2 = tw2[j[kk]];
#pragma unroll
                                for (int c = 0; c < 6; c++) AB[kk][c] = cmacv(AB[kk][c], ev[c], w2);
                            }
                        }
                        C c0[6];
                        ld6c<T>(rA + n0, c0);
#pragma unroll
                        for (int kk = 0; kk < KPc; kk++) {
                            const int k = k0 + kk;
                            if (k >= npair) break;
                            T x[6];
#pragma unroll
                            for (int c = 0; c < 6; c++) x[c] = c0[c].x + (T)2 * (AB[kk][c].x - AB[kk][c].y);
                            st6r<T>(rBr + (size_t)k * 150 + n0, x);
                            if (k != 0 && 2 * k != nr) {
#pragma unroll
                                for (int c = 0; c < 6; c++) x[c] = c0[c].x + (T)2 * (AB[kk][c].x + AB[kk][c].y);
                                st6r<T>(rBr + (size_t)(nr - k) * 150 + n0, x);
                            }
                        }
                    }
                } else
#endif
                for (int i = lane; i < npb * qcnt; i += TEAM) {
                    const int pb = i / qcnt, qq = i - pb * qcnt, q = q0 + qq;
                    const int k0 = pb * KPc;
                    C AB[KPc][6];
                    int j[KPc], kst[KPc];
#pragma unroll
                    for (int kk = 0; kk < KPc; kk++) {
                        j[kk] = 0;
                        kst[kk] = k0 + kk < npair ? k0 + kk : 0;
#pragma unroll
                        for (int d = 0; d < 6; d++) AB[kk][d] = mk<T>(0, 0);
                    }
                    for (int al = 1; al < nu; al++) {
                        C ev[6];
#pragma unroll
                        for (int d = 0; d < 6; d++) ev[d] = rA[(al * 6 + d) * 25 + q];
#pragma unroll
                        for (int kk = 0; kk < KPc; kk++) {
                            j[kk] += kst[kk];
                            j[kk] = j[kk] >= nr ? j[kk] - nr : j[kk];
                            const T2 w2 = tw2[j[kk]];
#pragma unroll
                            for (int d = 0; d < 6; d++) AB[kk][d] = cmacv(AB[kk][d], ev[d], w2);
                        }
                    }
#pragma unroll
                    for (int kk = 0; kk < KPc; kk++) {
                        const int k = k0 + kk;
                        if (k >= npair) break;
                        const bool two = k != 0 && 2 * k != nr;
#pragma unroll
                        for (int d = 0; d < 6; d++) {
                            const T c0 = rA[d * 25 + q].x;
                            rBr[((size_t)k * 6 + d) * qcnt + qq] = c0 + (T)2 * (AB[kk][d].x - AB[kk][d].y);
                            if (two) rBr[((size_t)(nr - k) * 6 + d) * qcnt + qq] = c0 + (T)2 * (AB[kk][d].x + AB[kk][d].y);
                        }
                    }
                }
                team_sync(team, TEAM);
                }
                }   // direct Fourier -> slice sums
                // component d of slice k at point qq: in + (d >> 1) sp + (d & 1) sq, and the stress at
                // out + (d >> 1) op + (d & 1) oq (the FFT takes its pairs with the parts exchanged)
                const int sp = use_fft ? 2 * vs.ps : 2 * qcnt, sq = use_fft ? 1 : qcnt;
                const int op = use_fft ? 2 * vo.ps : 2 * qcnt, oq = use_fft ? -1 : qcnt;
                auto stress_at = [&](int k, int qq, auto with_att) {
                    constexpr bool ATTEN = decltype(with_att)::value;
                    const int q = q0 + qq;
                    const T *in = use_fft ? reinterpret_cast<const T *>(&vs.at(k, 0, qq)) : rBr + (size_t)k * 6 * qcnt + qq;
                    T *out = use_fft ? reinterpret_cast<T *>(&vo.at(k, 0, qq)) + 1 : rBr + (size_t)k * 6 * qcnt + qq;
                    T md[NM];
#pragma unroll
                    for (int mm = 0; mm < NM; mm++) md[mm] = __ldg(modp + mm * nsl + (size_t)k * 25 + q);
                    AT ds[6], mem[NSR][6];
                    T dl = 0, dmu = 0;
                    AT *st = nullptr;
                    size_t slot = 0, nslot = 0;
                    if constexpr (ATTEN) {
                        nslot = (size_t)nr * NPA;
                        slot = (size_t)k * NPA + (ATT == ATT_CG4 ? cg4_slot(q) : q);
                        st = statew + a.state_off[e];
                        const T *am = a.attmod + a.att_off[e];
                        dl = __ldg(am + slot);
                        dmu = __ldg(am + nslot + slot);
#pragma unroll
                        for (int d = 0; d < 6; d++) ds[d] = st[d * nslot + slot];
#pragma unroll
                        for (int l = 0; l < NSR; l++)
#pragma unroll
                            for (int d = 0; d < 6; d++) mem[l][d] = st[(6 + l * 6 + d) * nslot + slot];
                    }
                    re1<T> ev[6], sg[6];
#pragma unroll
                    for (int d = 0; d < 6; d++) ev[d].x = in[(d >> 1) * sp + (d & 1) * sq];
                    if constexpr (RHEO == RHEO_ISO) {
                        stress_iso(ev, sg, md[0], md[1]);
                    } else if constexpr (RHEO == RHEO_TISO) {
                        stress_tiso(ev, sg, md[0], md[1], md[2], md[3], md[4]);
                    } else {
                        stress_aniso(ev, sg, md);
                    }
                    if constexpr (ATTEN) {
                        T e6[6], s6[6];
#pragma unroll
                        for (int d = 0; d < 6; d++) { e6[d] = ev[d].x; s6[d] = sg[d].x; }
                        attenuate_regs<NSR, T, AT>(a.alpha, a.beta, a.gamma, ds, mem, e6, s6, dl, dmu);
#pragma unroll
                        for (int d = 0; d < 6; d++) sg[d].x = s6[d];
#pragma unroll
                        for (int d = 0; d < 6; d++) st[d * nslot + slot] = ds[d];
#pragma unroll
                        for (int l = 0; l < NSR; l++)
#pragma unroll
                            for (int d = 0; d < 6; d++) st[(6 + l * 6 + d) * nslot + slot] = mem[l][d];
                    }
#pragma unroll
                    for (int d = 0; d < 6; d++) out[(d >> 1) * op + (d & 1) * oq] = sg[d].x;
                };
                if constexpr (ATT == ATT_CG4) {
                    // the four attenuating points apart from the elastic ones, so that no warp
                    // runs the recursion for a few of its lanes: c0 of them lie before the chunk
                    auto before = [](int q) { return (q > 6) + (q > 8) + (q > 16) + (q > 18); };
                    const int c0 = before(q0), nc = before(q0 + qcnt) - c0, ne = qcnt - nc;
                    const float rne = 1.f / (float)max(ne, 1);
                    for (int i = lane; i < nr * nc; i += TEAM) {
                        const int k = nc == 4 ? i >> 2 : i / nc, k4 = c0 + i - k * nc;
                        stress_at(k, 6 + 2 * (k4 & 1) + 10 * (k4 >> 1) - q0, std::true_type{});
                    }
                    for (int i = lane; i < nr * ne; i += TEAM) {
                        const int k = div_n(i, ne, rne), j = q0 - c0 + i - k * ne;
                        stress_at(k, j + (j >= 6) + (j >= 7) + (j >= 14) + (j >= 15) - q0, std::false_type{});
                    }
                } else {
                    for (int i = lane; i < nr * qcnt; i += TEAM) {
                        const int k = i / qcnt;
                        stress_at(k, i - k * qcnt, std::integral_constant<bool, ATT != ATT_NONE>{});
                    }
                }
                } else
                // Fourier -> slices (computeC2R), stress, attenuation -> rBr[k][d][qq]
                for (int i = lane; i < nkb * qcnt; i += TEAM) {
                    const int kb = i / qcnt, qq = i - kb * qcnt, q = q0 + qq;
                    const int k0 = kb * KB;
                    T acc[KB][6];
                    int j[KB];
#pragma unroll
                    for (int d = 0; d < 6; d++) {
                        const T r0 = rA[d * 25 + q].x;
#pragma unroll
                        for (int kk = 0; kk < KB; kk++) acc[kk][d] = r0;
                    }
                    int kstep[KB];
#pragma unroll
                    for (int kk = 0; kk < KB; kk++) {
                        j[kk] = 0;
                        kstep[kk] = (k0 + kk < nr) ? k0 + kk : 0;
                    }
                    for (int al = 1; al < nu; al++) {
                        C ev[6];
#pragma unroll
                        for (int d = 0; d < 6; d++) ev[d] = rA[(al * 6 + d) * 25 + q];
#pragma unroll
                        for (int kk = 0; kk < KB; kk++) {
                            j[kk] += kstep[kk];
                            j[kk] = j[kk] >= nr ? j[kk] - nr : j[kk];
                            const T2 w2 = tw2[j[kk]];
                            const T c = w2.x, s = w2.y;
#pragma unroll
                            for (int d = 0; d < 6; d++)
                                acc[kk][d] += (T)2 * (ev[d].x * c - ev[d].y * s);
                        }
                    }
#pragma unroll
                    for (int kk = 0; kk < KB; kk++) {
                        const int k = k0 + kk;
                        if (k >= nr) break;
                        re1<T> ev[6], sg[6];
#pragma unroll
                        for (int d = 0; d < 6; d++) ev[d].x = acc[kk][d];
                        elastic_at<RHEO>(a.mod + moff, nslice, k, q, ev, sg);
                        if constexpr (ATT == ATT_FULL) {
                            const int64_t ao = a.att_off[e];
                            AT *st = statew + a.state_off[e];
                            const size_t ns = (size_t)nr * 25;
                            attenuate<T, AT, false>(a, st, ns, (size_t)k * 25 + q, ev, sg,
                                                    a.attmod[ao + (size_t)k * 25 + q],
                                                    a.attmod[ao + ns + (size_t)k * 25 + q]);
                        } else if constexpr (ATT == ATT_CG4) {
                            const int k4 = cg4_slot(q);
                            if (k4 >= 0) {
                                const int64_t ao = a.att_off[e];
                                AT *st = statew + a.state_off[e];
                                const size_t ns = (size_t)nr * 4;
                                attenuate<T, AT, false>(a, st, ns, (size_t)k * 4 + k4, ev, sg,
                                                        a.attmod[ao + (size_t)k * 4 + k4],
                                                        a.attmod[ao + ns + (size_t)k * 4 + k4]);
                            }
                        }
#pragma unroll
                        for (int d = 0; d < 6; d++) rBr[((size_t)k * 6 + d) * qcnt + qq] = sg[d].x;
                    }
                }
                team_sync(team, TEAM);
                if (FFT && use_fft) {
                    // forward FFT of the stress pairs, then each pair's two spectra:
                    // S_2p = (Z_a + conj Z_nr-a) / 2, S_2p+1 = (Z_a - conj Z_nr-a) / 2i, scaled by 1/nr
                    const FftView<T> Z = fft_run<T>(nullptr, vo, vs, nr, qcnt, plan, tw2, team, lane, TEAM);
                    const T h = (T)0.5 * inv_nr;
                    for (int i = lane; i < nu * qcnt; i += TEAM) {
                        const int al = i / qcnt, qq = i - al * qcnt, q = q0 + qq;
                        const int bl = al == 0 ? 0 : nr - al;
                        C sg[6];
#pragma unroll
                        for (int pp = 0; pp < 3; pp++) {
                            const C ya = Z.at(al, pp, qq), yb = Z.at(bl, pp, qq);
                            const C za = mk<T>(ya.y, ya.x), zb = mk<T>(yb.y, yb.x);   // parts back in place
                            T r1 = (za.x + zb.x) * h, m1 = (za.y - zb.y) * h;
                            T r2 = (za.y + zb.y) * h, m2 = (zb.x - za.x) * h;
                            if (al == 0) { m1 = 0; m2 = 0; }
                            if ((nr & 1) == 0 && 2 * al == nr) { r1 *= (T)0.5; r2 *= (T)0.5; m1 = 0; m2 = 0; }
                            sg[2 * pp] = mk<T>(r1, m1);
                            sg[2 * pp + 1] = mk<T>(r2, m2);
                        }
                        if constexpr (RTZ) {
                            rtz_to_spz6(sg, sTrig[q], sTrig[25 + q], sTrig[50 + q], sTrig[75 + q]);
                        }
#pragma unroll
                        for (int d = 0; d < 6; d++) rA[(al * 6 + d) * 25 + q] = sg[d];
                    }
                    team_sync(team, TEAM);
                    continue;
                }
                // slices -> Fourier (computeR2C) into region A for these points
#if AXG_COLUMN_TILES
                if (!RTZ && qcnt == 25) {
                    // ABc modes x 6 columns per thread (the column layout of the Fourier ->
                    // slice pass); the 1/nr scaling applied once to the sums
                    for (int i = lane; i < 25 * nab; i += TEAM) {
                        const int ab = (i / 5) % nab, n0 = 6 * ((i / (5 * nab)) * 5 + i % 5);
                        const int a0 = ab * ABc;
                        C ri[ABc][6];
                        int j[ABc], astep[ABc];
#pragma unroll
                        for (int aa = 0; aa < ABc; aa++) {
                            j[aa] = 0;
                            astep[aa] = (a0 + aa) % nr;
#pragma unroll
                            for (int c = 0; c < 6; c++) ri[aa][c] = mk<T>(0, 0);
                        }
#pragma unroll DFT_UNROLL
                        for (int k = 0; k <= nr / 2; k++) {
                            // (x_k + x_nr-k, x_nr-k - x_k) against (cos, sin)
                            T xs[6];
                            C p[6];
                            ld6r<T>(rBr + (size_t)k * 150 + n0, xs);
                            if (k != 0 && 2 * k != nr) {
                                T x2[6];
                                ld6r<T>(rBr + (size_t)(nr - k) * 150 + n0, x2);
#pragma unroll
                                for (int c = 0; c < 6; c++) p[c] = mk<T>(xs[c] + x2[c], x2[c] - xs[c]);
                            } else {
#pragma unroll
                                for (int c = 0; c < 6; c++) p[c] = mk<T>(xs[c], -xs[c]);
                            }
#pragma unroll
                            for (int aa = 0; aa < ABc; aa++) {
                                const T2 w2 = tw2[j[aa]];
#pragma unroll
                                for (int c = 0; c < 6; c++) ri[aa][c] = cmacv(ri[aa][c], p[c], w2);
                                j[aa] += astep[aa];
                                j[aa] = j[aa] >= nr ? j[aa] - nr : j[aa];
                            }
                        }
#pragma unroll
                        for (int aa = 0; aa < ABc; aa++) {
                            const int al = a0 + aa;
                            if (al >= nu) break;
                            const bool nyq = (nr & 1) == 0 && al == nr / 2;
                            const T sr = nyq ? (T)0.5 * inv_nr : inv_nr;
                            const bool noim = al == 0 || nyq;
                            C sg[6];
#pragma unroll
                            for (int c = 0; c < 6; c++) sg[c] = mk<T>(ri[aa][c].x * sr, noim ? (T)0 : ri[aa][c].y * inv_nr);
                            st6c<T>(rA + al * 150 + n0, sg);
                        }
                    }
                } else
#endif
                for (int i = lane; i < nab * qcnt; i += TEAM) {
                    const int ab = i / qcnt, qq = i - ab * qcnt, q = q0 + qq;
                    const int a0 = ab * ABc;
                    T re[ABc][6], im[ABc][6];
                    int j[ABc], astep[ABc];
#pragma unroll
                    for (int aa = 0; aa < ABc; aa++) {
                        j[aa] = 0;
                        astep[aa] = (a0 + aa) % nr;
#pragma unroll
                        for (int d = 0; d < 6; d++) { re[aa][d] = 0; im[aa][d] = 0; }
                    }
                    // slices k and nr - k in one pass: cos(a phi) is even and sin(a phi) odd
                    // in k, so they enter as x_k + x_{nr-k} and x_k - x_{nr-k}
                    for (int k = 0; k <= nr / 2; k++) {
                        const bool two = k != 0 && 2 * k != nr;
                        T xs[6], xd[6];
#pragma unroll
                        for (int d = 0; d < 6; d++) {
                            const T x1 = rBr[((size_t)k * 6 + d) * qcnt + qq];
                            const T x2 = two ? rBr[((size_t)(nr - k) * 6 + d) * qcnt + qq] : (T)0;
                            xs[d] = (x1 + x2) * inv_nr;
                            xd[d] = (x1 - x2) * inv_nr;
                        }
#pragma unroll
                        for (int aa = 0; aa < ABc; aa++) {
                            const T2 w2 = tw2[j[aa]];
                            const T c = w2.x, s = w2.y;
#pragma unroll
                            for (int d = 0; d < 6; d++) {
                                re[aa][d] += xs[d] * c;
                                im[aa][d] -= xd[d] * s;
                            }
                            j[aa] += astep[aa];
                            j[aa] = j[aa] >= nr ? j[aa] - nr : j[aa];
                        }
                    }
#pragma unroll
                    for (int aa = 0; aa < ABc; aa++) {
                        const int al = a0 + aa;
                        if (al >= nu) break;
                        C sg[6];
#pragma unroll
                        for (int d = 0; d < 6; d++) {
                            T r = re[aa][d], m = im[aa][d];
                            if (al == 0) m = 0;
                            if ((nr & 1) == 0 && al == nr / 2) { r *= (T)0.5; m = 0; }
                            sg[d] = mk<T>(r, m);
                        }
                        if constexpr (RTZ) {
                            rtz_to_spz6(sg, sTrig[q], sTrig[25 + q], sTrig[50 + q], sTrig[75 + q]);
                        }
#pragma unroll
                        for (int d = 0; d < 6; d++) rA[(al * 6 + d) * 25 + q] = sg[d];
                    }
                }
                team_sync(team, TEAM);
            }
        }

        for (int t0 = 0; t0 < nu; t0 += mt_max) {
        const int mt = min(mt_max, nu - t0);
        // ---------------- quadrature (computeQuad6), pass 1: X, Y, A ----------------
        // the axial terms (the transpose of dA / ds) join X and Y at the axial row
        for (int i = lane; i < mt * 25; i += TEAM) {
            const int la = i / 25, q = i - la * 25, al = t0 + la;
            C s[6];
#pragma unroll
            for (int d = 0; d < 6; d++) s[d] = rA[(al * 6 + d) * 25 + q];
            const T ze = dzdeta_if[q], zx = dzdxii_if[q], se = dsdeta_if[q], sx = dsdxii_if[q];
            const T alf = (T)al, is = invs_if[q];
            C A[3], x[6];
            A[0] = csub(cia(alf, s[5]), s[1]);
            A[1] = cadd(cia(alf, s[1]), s[5]);
            A[2] = cia(alf, s[3]);
            x[0] = cmac(cscale(s[4], se), s[0], ze);
            x[1] = cmac(cscale(s[4], sx), s[0], zx);
            x[2] = cmac(cscale(s[3], se), s[5], ze);
            x[3] = cmac(cscale(s[3], sx), s[5], zx);
            x[4] = cmac(cscale(s[2], se), s[4], ze);
            x[5] = cmac(cscale(s[2], sx), s[4], zx);
            if (axial && q < 5) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    x[2 * c] = csub(x[2 * c], cscale(A[c], ze));
                    x[2 * c + 1] = csub(x[2 * c + 1], cscale(A[c], zx));
                }
            }
            C *xy = rA + al * 150;
#pragma unroll
            for (int d = 0; d < 6; d++) xy[d * 25 + q] = x[d];
#pragma unroll
            for (int c = 0; c < 3; c++) rBc[(la * 3 + c) * 25 + q] = cscale(A[c], is);
        }
        team_sync(team, TEAM);

        // ---------------- quadrature pass 2: the forces, in the place of A ----------------
        for (int i = lane; i < mt * 25; i += TEAM) {
            const int la = i / 25, q = i - la * 25, al = t0 + la;
            const int ii = q / 5, jj = q - ii * 5;
            const C *xy = rA + al * 150;
            C *A = rBc + la * 75 + q;
            C f[3];
#pragma unroll
            for (int c = 0; c < 3; c++) f[c] = mk<T>(-A[c * 25].x, -A[c * 25].y);
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const T gx = Gxi[ii * 5 + k];      // G_xi(ii, k)
                const T gt = sGll[jj * 5 + k];     // GT_GLL(k, jj) = G_GLL(jj, k)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const C xv = xy[(2 * c) * 25 + k * 5 + jj];
                    const C yv = xy[(2 * c + 1) * 25 + ii * 5 + k];
                    f[c] = cmac(f[c], xv, gx);
                    f[c] = cmac(f[c], yv, gt);
                }
            }
            if constexpr (sizeof(T) == 4) {
                // scatter-add, one vector reduction per component
                const int2 on = __ldg(tab + q);
                if (al < on.y) {
                    C *dst = stiffw + ((size_t)on.x + al) * 3;
#pragma unroll
                    for (int c = 0; c < 3; c++) atomic_add_cx(dst + c, mk<T>(-f[c].x, -f[c].y));
                }
            } else {
#pragma unroll
                for (int c = 0; c < 3; c++) A[c * 25] = f[c];
            }
        }
        if constexpr (sizeof(T) == 8) {
            // FP64 has no vector reduction: the forces go through shared memory, so that a warp's
            // lanes cover consecutive words of the field (point, mode, component, part)
            team_sync(team, TEAM);
            const int run = 6 * mt;
            const float rrun = 1.f / (float)run;
            for (int j = lane; j < 25 * run; j += TEAM) {
                const int p = div_n(j, run, rrun), r = j - p * run;
                const int2 on = __ldg(tab + p);
                const T f = reinterpret_cast<const T *>(rBc + (r >> 1) * 25 + p)[r & 1];
                if (t0 + r / 6 < on.y)
                    atomicAdd(reinterpret_cast<T *>(stiffw + ((size_t)on.x + t0) * 3) + r, -f);
            }
        }
        team_sync(team, TEAM);
        }   // mode tiles of the quadrature
        }   // wavefields
    }
}

}  // namespace axg
