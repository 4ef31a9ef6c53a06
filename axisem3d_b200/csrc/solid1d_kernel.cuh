// solid1d_kernel.cuh -- fused stiffness of solid elements whose properties do not vary with phi.
//
// Every Fourier mode of such an element is on its own, so the unit of work of a block is a tile
// of at most blockDim / 25 modes of one element, one thread per (mode, point):
//   gather (SolidPoint::scatterDisplToElement), computeGrad6, strainToStress_FR, the SLS
//   recursion per mode (AttenuationFull / AttenuationCG4::apply), computeQuad6, scatter-add
//   (SolidPoint::gatherStiffFromElement); SOLVER/src/core/element/SolidElement.cpp:112-222.
//
// What bounds it: latency. An element has a few hundred operations per (mode, point) and, without
// attenuation, a few KB of operands, so the time is the chain tile -> points -> displacement ->
// barrier -> strain -> barrier -> force -> barrier -> scatter. Hence small blocks (at most five
// modes, 128 threads, by default), many of them per SM in different phases; geometry, moduli and
// derivative rows in registers; the offsets of the 25 points in one table per element instead of
// point ids to follow; and the lower-order terms folded into the strain's and the quadrature's
// local values, so that two reads of shared memory per (component, neighbour) are all there is:
//   - on the axis A / s becomes dA / ds of A = (i a u0 - u1, i a u1 + u0, i a u2), which is the
//     same combination of the derivatives already formed;
//   - its transpose subtracts A_c dz/deta and A_c dz/dxi from the terms under the xi and eta
//     derivatives at the axial row.
// The gather and the scatter run over (point, mode, component) with the components fastest, the
// order of the point fields, so that loads and reductions cover consecutive words.
#pragma once

#include "solid_kernel.cuh"

namespace axg {

// shared memory of a block: gathered displacement (then the forces, point-major with an odd
// stride), the terms under the two derivatives and A; with CG4 the corrections and strains of the
// four attenuating points
template <class T, class AT>
struct Tile1D {
    int u, xy, a, geo, corr, e4, total;
};
template <class T, class AT, int ATT>
__host__ __device__ inline Tile1D<T, AT> tile_1d(int mt) {
    Tile1D<T, AT> L;
    const int c = 2 * (int)sizeof(T);
    auto al = [](int x) { return (x + 15) & ~15; };
    L.u = 0;
    L.xy = al(25 * ((3 * mt) | 1) * c);
    L.a = al(L.xy + mt * 150 * c);
    L.geo = al(L.a + mt * 75 * c);
    L.corr = al(L.geo + 125 * (int)sizeof(T));
    L.e4 = L.corr + (ATT == ATT_CG4 ? al(mt * 24 * 2 * (int)sizeof(AT)) : 0);
    L.total = L.e4 + (ATT == ATT_CG4 ? al(mt * 24 * c) : 0);
    return L;
}

// SLS recursion of one (mode, point) with full attenuation, the steps of attenuate<>: groups of G
// stress components, the G (1 + NS) state words of a group as complex loads in flight together. Two
// components with five SLS hold as many words as three with three; three of them spilled 480 B in
// FP32. Measured, 12 000 elements of nr up to 64 per step, G = 3 / 2 / 1: five SLS FP32 687 / 493 /
// 715 us, FP64 state in FP32 elements 836 / 704 / 829 (FP64 985 / 817); three SLS FP32 371 / 404 /
// 647, 553 / 559 / 756.
template <int NS, class T, class AT>
__device__ __forceinline__ void attenuate_full_1d(const SolidArgs<T, AT> &a, cx_t<AT> *st, size_t nslot,
                                                  const cx_t<T> (&e)[6], cx_t<T> (&s)[6], T dl, T dm) {
    using CA = cx_t<AT>;
    constexpr int G = NS > 3 ? 2 : 3;
    const AT lam = (AT)dl, mu = (AT)dm, mu2 = mu + mu;
    const CA tr = mk<AT>(((AT)e[0].x + (AT)e[1].x + (AT)e[2].x) * lam, ((AT)e[0].y + (AT)e[1].y + (AT)e[2].y) * lam);
#pragma unroll
    for (int g = 0; g < 6 / G; g++) {
        CA ds[G], mem[NS][G];
#pragma unroll
        for (int c = 0; c < G; c++) ds[c] = st[(G * g + c) * nslot];
#pragma unroll
        for (int l = 0; l < NS; l++)
#pragma unroll
            for (int c = 0; c < G; c++) mem[l][c] = st[(6 + l * 6 + G * g + c) * nslot];
#pragma unroll
        for (int c = 0; c < G; c++) {
            const int d = G * g + c;
            const CA ed = mk<AT>((AT)e[d].x, (AT)e[d].y);
            const CA dn = d < 3 ? mk<AT>(tr.x + ed.x * mu2, tr.y + ed.y * mu2) : mk<AT>(ed.x * mu, ed.y * mu);
            CA sv = mk<AT>((AT)s[d].x, (AT)s[d].y);
            st[d * nslot] = dn;
#pragma unroll
            for (int l = 0; l < NS; l++) {
                CA m = mem[l][c];
                sv.x -= m.x;
                sv.y -= m.y;
                m.x = a.alpha[l] * m.x + a.beta[l] * ds[c].x;
                m.y = a.alpha[l] * m.y + a.beta[l] * ds[c].y;
                m.x += a.gamma[l] * dn.x;
                m.y += a.gamma[l] * dn.y;
                st[(6 + l * 6 + d) * nslot] = m;
            }
            s[d] = mk<T>((T)sv.x, (T)sv.y);
        }
    }
}

// registers: 1024 threads per SM for elastic elements, 768 with the state in FP32, else 512. Measured
// (per pass): FP64 elastic at 128 / 80 / 64 registers 37.1 / 37.4 / 33.5 ms (adjoint of a 100 x 100
// box), FP32 with full attenuation at 80 / 64 0.96 / 1.20 ms (hook loop), FP64 state in FP32 elements
// at 128 / 80 / 64 18.5 / 28.1 / 31.6 ms.
template <class T, class AT, int ATT>
constexpr int blocks_1d() { return ATT == ATT_NONE ? 4 : sizeof(T) == 8 ? 2 : sizeof(AT) == 4 ? 3 : 2; }

// whether the quadrature's operators are staged in shared memory (FP32 elastic elements have the
// registers, and staging cost the 40 x 40 box 1.7 us per step there)
template <class T, int ATT>
__host__ __device__ constexpr bool stage_1d() { return sizeof(T) == 8 || ATT != ATT_NONE; }

template <class T, class AT, int RHEO, int ATT, bool RTZ, int NS>
__global__ void __launch_bounds__(256, blocks_1d<T, AT, ATT>())
solid_1d_kernel(const SolidArgs<T, AT> a, const int mt_max) {
    using C = cx_t<T>;
    using CA = cx_t<AT>;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Tile1D<T, AT> L = tile_1d<T, AT, ATT>(mt_max);
    C *sU = reinterpret_cast<C *>(smem_raw + L.u);
    C *sXY = reinterpret_cast<C *>(smem_raw + L.xy);
    C *sA = reinterpret_cast<C *>(smem_raw + L.a);
    T *sGeo = reinterpret_cast<T *>(smem_raw + L.geo);
    CA *sCorr = reinterpret_cast<CA *>(smem_raw + L.corr);
    C *sE4 = reinterpret_cast<C *>(smem_raw + L.e4);
    const int tid = threadIdx.x, nt = blockDim.x;

    const int4 tile = __ldg(a.tiles + blockIdx.x);
    const int e = tile.x, t0 = tile.y, mt = tile.z, nu = tile.w & 0xffffff;
    const bool axial = (tile.w >> 30) != 0;
    const int run = 3 * mt, frow = run | 1;
    const float rrun = 1.f / (float)run;
    const int2 *tab = a.tab + (size_t)e * 25;

    // this thread's (mode, point) and its operands
    const int la = tid / 25, q = tid - la * 25, al = t0 + la;
    const bool on = la < mt;
    const int ii = q / 5, jj = q - ii * 5;
    const T *geo = a.geom + (size_t)e * 250 + q;
    T dsx = 0, dse = 0, dzx = 0, dze = 0, is = 0;
    constexpr int NM = RHEO == RHEO_ISO ? 2 : RHEO == RHEO_TISO ? 5 : 21;
    T md[NM], dl = 0, dm = 0;
    T s1 = 0, c1 = 0, s2 = 0, c2 = 0;
    if (on) {
        dsx = __ldg(geo); dse = __ldg(geo + 25); dzx = __ldg(geo + 50); dze = __ldg(geo + 75); is = __ldg(geo + 100);
        if constexpr (NM <= 5) {
            const T *mod = a.mod + a.mod_off[e] + q;
#pragma unroll
            for (int k = 0; k < NM; k++) md[k] = __ldg(mod + k * 25);
        }
        if constexpr (ATT == ATT_FULL) {
            const T *am = a.attmod + a.att_off[e] + q;
            dl = __ldg(am);
            dm = __ldg(am + 25);
        }
        if constexpr (RTZ) {
            const T *tr = a.trig + (size_t)e * 100 + q;
            s1 = __ldg(tr); c1 = __ldg(tr + 25); s2 = __ldg(tr + 50); c2 = __ldg(tr + 75);
        }
    }
    // the operators of the quadrature: in registers from the start where there is room, else they
    // wait in shared memory, out of the stress's registers
    T quad[5] = {0, 0, 0, 0, 0};
    if constexpr (stage_1d<T, ATT>()) {
        for (int i = tid; i < 125; i += nt) sGeo[i] = __ldg(a.geom + (size_t)e * 250 + 125 + i);
    } else if (on) {
#pragma unroll
        for (int k = 0; k < 5; k++) quad[k] = __ldg(geo + 125 + 25 * k);
    }
    const T *Gl = a.gmat, *Gx = a.gmat + (axial ? 25 : 0);

    for (int w = blockIdx.y; w < a.nwave; w += gridDim.y) {
        const C *displw = a.displ + (size_t)w * a.fstride;
        C *stiffw = a.stiff + (size_t)w * a.fstride;
        AT *st = ATT == ATT_NONE ? nullptr : a.state + (size_t)w * a.sstride + a.state_off[e];

        // ---------------- SLS state on its way ----------------
        // full: into L2 (24 words per slot are too many to hold across the strain); CG4: the
        // recursion's items (component, slot) in registers, and the sum of the memory variables,
        // which the stress needs and which does not depend on the strain (a count known at run time
        // only is read again for the recursion: the whole recursion on the four points' own threads
        // took 674 us per step of 12 000 elements with two SLS, mixed, this way 387)
        CA ds4, mem4[NS > 0 ? NS : 1];
        const int n4 = 4 * mt, d4 = tid / n4, k4 = tid - d4 * n4;
        const bool item4 = ATT == ATT_CG4 && tid < 6 * n4;
        const int nsls = NS > 0 ? NS : a.nsls;
        if constexpr (ATT == ATT_FULL && NS > 0) {
            // the 128-byte lines that the tile's part of each row touches, in one walk of the block: a
            // warp per row leaves most lanes idle where rows are short (100 000 TI elements of nr = 1 / 2
            // / 8, mixed, per step: 762 / 1309 / 2707 us that way, 651 / 1194 / 2675 this way)
            const size_t row = (size_t)nu * 25 * 2, bytes = (size_t)mt * 50 * sizeof(AT);
            const int per = (int)((bytes + 127) / 128) + 1;
            const float rper = 1.f / (float)per;
            for (int i = tid; i < per * (6 + 6 * NS); i += nt) {
                const int r = div_n(i, per, rper);
                const uintptr_t p0 = (uintptr_t)(st + r * row + (size_t)t0 * 50);
                const uintptr_t line = (p0 & ~(uintptr_t)127) + (uintptr_t)(i - r * per) * 128;
                if (line < p0 + bytes) asm volatile("prefetch.global.L2 [%0];" ::"l"(line));
            }
        }
        if constexpr (ATT == ATT_CG4) {
            if (item4) {
                const CA *s0 = reinterpret_cast<const CA *>(st) + (size_t)d4 * nu * 4 + t0 * 4 + k4;
                const size_t row = (size_t)6 * nu * 4;
                ds4 = s0[0];
                CA sum = mk<AT>(0, 0);
#pragma unroll
                for (int l = 0; l < nsls; l++) {
                    const CA m = s0[(l + 1) * row];
                    if constexpr (NS > 0) mem4[l] = m;
                    sum = cadd(sum, m);
                }
                sCorr[d4 * n4 + k4] = sum;
            }
        }

        // ---------------- gather: U[mode][c][point] ----------------
        for (int j = tid; j < 25 * run; j += nt) {
            const int p = div_n(j, run, rrun), r = j - p * run;
            const int2 on_ = __ldg(tab + p);
            const int m = r / 3;
            sU[r * 25 + p] = t0 + m < on_.y ? displw[((size_t)on_.x + t0) * 3 + r] : mk<T>(0, 0);
        }
        __syncthreads();

        // ---------------- strain, stress, terms of the quadrature ----------------
        if (on) {
            const C *U = sU + la * 75;
            C X[3], Y[3];
#pragma unroll
            for (int c = 0; c < 3; c++) { X[c] = mk<T>(0, 0); Y[c] = mk<T>(0, 0); }
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const T gx = __ldg(Gx + k * 5 + ii), gy = __ldg(Gl + k * 5 + jj);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const C uc = U[c * 25 + k * 5 + jj], ur = U[c * 25 + ii * 5 + k];
                    X[c] = cmac(X[c], uc, gx);
                    Y[c] = cmac(Y[c], ur, gy);
                }
            }
            const T alf = (T)al;
            C eps[6], sig[6];
            {
                // ds, dz of the components, then A / s (on the axis dA / ds)
                C S[3], o[3];
#pragma unroll
                for (int c = 0; c < 3; c++) S[c] = cmac(cscale(Y[c], dzx), X[c], dze);
                eps[0] = S[0];
                eps[4] = cadd(cmac(cscale(Y[0], dsx), X[0], dse), S[2]);
                eps[3] = cmac(cscale(Y[1], dsx), X[1], dse);
                eps[2] = cmac(cscale(Y[2], dsx), X[2], dse);
                eps[5] = S[1];
                const bool lim = axial && ii == 0;
                const C b0 = lim ? S[0] : U[q], b1 = lim ? S[1] : U[25 + q], b2 = lim ? S[2] : U[50 + q];
                const T f = lim ? (T)1 : is;
                o[0] = cscale(csub(cia(alf, b0), b1), f);
                o[1] = cscale(cadd(cia(alf, b1), b0), f);
                o[2] = cscale(cia(alf, b2), f);
                eps[5] = cadd(eps[5], o[0]);
                eps[1] = o[1];
                eps[3] = cadd(eps[3], o[2]);
            }
            if constexpr (RTZ) spz_to_rtz6(eps, s1, c1, s2, c2);
            if constexpr (RHEO == RHEO_ISO) stress_iso(eps, sig, md[0], md[1]);
            else if constexpr (RHEO == RHEO_TISO) stress_tiso(eps, sig, md[0], md[1], md[2], md[3], md[4]);
            else elastic_at<RHEO>(a.mod + a.mod_off[e], 1, 0, q, eps, sig);
            if constexpr (ATT == ATT_FULL) {
                if constexpr (NS > 0)
                    attenuate_full_1d<NS, T, AT>(a, reinterpret_cast<CA *>(st) + (size_t)al * 25 + q, (size_t)nu * 25, eps,
                                                 sig, dl, dm);
                else
                    attenuate<T, AT, true>(a, st, (size_t)nu * 25, (size_t)al * 25 + q, eps, sig, dl, dm);
            } else if constexpr (ATT == ATT_CG4) {
                const int s4 = cg4_slot(q);
                if (s4 >= 0) {
#pragma unroll
                    for (int d = 0; d < 6; d++) {
                        const CA cr = sCorr[d * n4 + la * 4 + s4];
                        sig[d] = mk<T>((T)((AT)sig[d].x - cr.x), (T)((AT)sig[d].y - cr.y));
                        sE4[d * n4 + la * 4 + s4] = eps[d];
                    }
                }
            }
            if constexpr (RTZ) rtz_to_spz6(sig, s1, c1, s2, c2);
            if constexpr (stage_1d<T, ATT>()) {
#pragma unroll
                for (int k = 0; k < 5; k++) quad[k] = sGeo[25 * k + q];
            }
            const T dsx_i = quad[0], dse_i = quad[1], dzx_i = quad[2], dze_i = quad[3], is_i = quad[4];
            C A[3], x[6];
            A[0] = csub(cia(alf, sig[5]), sig[1]);
            A[1] = cadd(cia(alf, sig[1]), sig[5]);
            A[2] = cia(alf, sig[3]);
            x[0] = cmac(cscale(sig[4], dse_i), sig[0], dze_i);
            x[1] = cmac(cscale(sig[4], dsx_i), sig[0], dzx_i);
            x[2] = cmac(cscale(sig[3], dse_i), sig[5], dze_i);
            x[3] = cmac(cscale(sig[3], dsx_i), sig[5], dzx_i);
            x[4] = cmac(cscale(sig[2], dse_i), sig[4], dze_i);
            x[5] = cmac(cscale(sig[2], dsx_i), sig[4], dzx_i);
            if (axial && ii == 0) {
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    x[2 * c] = csub(x[2 * c], cscale(A[c], dze_i));
                    x[2 * c + 1] = csub(x[2 * c + 1], cscale(A[c], dzx_i));
                }
            }
#pragma unroll
            for (int d = 0; d < 6; d++) sXY[la * 150 + d * 25 + q] = x[d];
#pragma unroll
            for (int c = 0; c < 3; c++) sA[la * 75 + c * 25 + q] = cscale(A[c], is_i);
        }
        __syncthreads();

        // ---------------- forces, point-major over the displacement ----------------
        if (on) {
            const C *xy = sXY + la * 150, *A = sA + la * 75;
            C f[3];
#pragma unroll
            for (int c = 0; c < 3; c++) f[c] = mk<T>(-A[c * 25 + q].x, -A[c * 25 + q].y);
#pragma unroll
            for (int k = 0; k < 5; k++) {
                const T gx = __ldg(Gx + ii * 5 + k), gt = __ldg(Gl + jj * 5 + k);
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    const C xv = xy[(2 * c) * 25 + k * 5 + jj], yv = xy[(2 * c + 1) * 25 + ii * 5 + k];
                    f[c] = cmac(f[c], xv, gx);
                    f[c] = cmac(f[c], yv, gt);
                }
            }
#pragma unroll
            for (int c = 0; c < 3; c++) sU[q * frow + la * 3 + c] = f[c];
        }
        if constexpr (ATT == ATT_CG4) {
            // the recursion of this thread's (component, slot) with the strain of the slot
            if (item4) {
                const T *am = a.attmod + a.att_off[e] + (k4 & 3);
                const AT lam = (AT)__ldg(am), mu = (AT)__ldg(am + 4);
                const C ed = sE4[d4 * n4 + k4];
                CA dn = mk<AT>((AT)ed.x * mu, (AT)ed.y * mu);
                if (d4 < 3) {
                    const C e0 = sE4[k4], e1 = sE4[n4 + k4], e2 = sE4[2 * n4 + k4];
                    dn = mk<AT>(((AT)e0.x + (AT)e1.x + (AT)e2.x) * lam + (AT)ed.x * (mu + mu),
                                ((AT)e0.y + (AT)e1.y + (AT)e2.y) * lam + (AT)ed.y * (mu + mu));
                }
                CA *s0 = reinterpret_cast<CA *>(st) + (size_t)d4 * nu * 4 + t0 * 4 + k4;
                const size_t row = (size_t)6 * nu * 4;
                s0[0] = dn;
#pragma unroll
                for (int l = 0; l < nsls; l++) {
                    CA m;
                    if constexpr (NS > 0) m = mem4[l];
                    else m = s0[(l + 1) * row];
                    m.x = a.alpha[l] * m.x + a.beta[l] * ds4.x;
                    m.y = a.alpha[l] * m.y + a.beta[l] * ds4.y;
                    m.x += a.gamma[l] * dn.x;
                    m.y += a.gamma[l] * dn.y;
                    s0[(l + 1) * row] = m;
                }
            }
        }
        __syncthreads();

        // ---------------- scatter-add ----------------
        if constexpr (sizeof(T) == 4) {
            for (int j = tid; j < 25 * run; j += nt) {
                const int p = div_n(j, run, rrun), r = j - p * run;
                const int2 on_ = __ldg(tab + p);
                const C f = sU[p * frow + r];
                if (t0 + r / 3 < on_.y) atomic_add_cx(stiffw + ((size_t)on_.x + t0) * 3 + r, mk<T>(-f.x, -f.y));
            }
        } else {
            // one real per thread: consecutive lanes cover consecutive words
            for (int j = tid; j < 50 * run; j += nt) {
                const int p = div_n(j, 2 * run, 0.5f * rrun), r = j - p * 2 * run;
                const int2 on_ = __ldg(tab + p);
                const T f = reinterpret_cast<const T *>(sU + p * frow)[r];
                if (t0 + r / 6 < on_.y)
                    atomicAdd(reinterpret_cast<T *>(stiffw + ((size_t)on_.x + t0) * 3) + r, -f);
            }
        }
        if (a.nwave > 1) __syncthreads();
    }
}

}  // namespace axg
