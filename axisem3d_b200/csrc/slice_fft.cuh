// slice_fft.cuh -- the phi transforms of 3-D elements of large nr as FFTs in shared memory.
//
// SolverFFTW::computeC2R / computeR2C (SOLVER/src/core/fft/SolverFFTW.hpp:101-172: R2C scaled by
// 1/nr, the Nyquist mode halved, imaginary parts of modes 0 and nr/2 dropped; C2R with the Nyquist
// mode doubled) as complex FFTs of length nr over a batch of 3 qc signals: the six strain / stress
// components of a point go in pairs, x_2p + i x_2p+1, one complex signal per pair. Signal
// s = pair pp of point qq of the chunk (s = pp qc + qq), sample n.
//
// The transform is a mixed-radix Stockham FFT, one pass over shared memory per factor of nr, and a
// pass costs a barrier of the team, a read and a write of every sample and the index arithmetic,
// whatever its radix. So the factors are as few and as even as they go: radices up to 16 (FP64: 10, 11
// and 13), each a DFT in registers (of its prime factors, constants folded in). An nr of 26 .. 128
// without a prime factor above 13 takes two passes in FP32 (125 three) where prime radices took up to
// six; in FP64 75, 84, 96, 98, 105, 108, 112, 120, 126 and 128 take three as well. The transforms of
// both directions run with the positive sign: the spectrum of (x_2p+1, x_2p), real and imaginary part exchanged, is the exchanged
// spectrum of the negative sign.
#pragma once

#include "common.cuh"

#include <utility>

namespace axg {

// ---------------------------------------------------------- compile-time trigonometry ---
// cos and sin of pi a / n, by reduction to [0, pi / 4] and the Taylor series (to 1e-17)
__host__ __device__ constexpr double fft_series(double x, bool cosine) {
    double term = cosine ? 1.0 : x, sum = term;
    for (int k = cosine ? 1 : 2; k < 26; k += 2) {
        term *= -x * x / (k * (k + 1.0));
        sum += term;
    }
    return sum;
}
constexpr double fft_pi = 3.14159265358979323846;
__host__ __device__ constexpr double fft_cos(int a, int n) {
    a %= 2 * n;
    if (a > n) a = 2 * n - a;
    if (2 * a > n) return -fft_cos(n - a, n);
    if (4 * a > n) return fft_series(fft_pi * (n - 2 * a) / (2.0 * n), false);
    return fft_series(fft_pi * a / n, true);
}
__host__ __device__ constexpr double fft_sin(int a, int n) { return fft_cos(((n - 2 * a) % (4 * n) + 4 * n) % (4 * n), 2 * n); }

// f(0), f(1), ... with the index a compile-time constant
template <int I>
struct FftIndex {
    static constexpr int value = I;
    __device__ constexpr operator int() const { return I; }
};
template <class F, int... I>
__device__ __forceinline__ void fft_each(F f, std::integer_sequence<int, I...>) {
    (f(FftIndex<I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void fft_for(F f) {
    fft_each(f, std::make_integer_sequence<int, N>{});
}

template <class T>
__device__ __forceinline__ cx_t<T> cmul(cx_t<T> a, cx_t<T> b) {
    return mk<T>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// a exp(2 pi i K / N)
template <int K, int N, class T>
__device__ __forceinline__ cx_t<T> fft_rot(cx_t<T> a) {
    constexpr int k = K % N;
    if constexpr (k == 0) return a;
    else if constexpr (4 * k == N) return mk<T>(-a.y, a.x);
    else if constexpr (2 * k == N) return mk<T>(-a.x, -a.y);
    else if constexpr (4 * k == 3 * N) return mk<T>(a.y, -a.x);
    else {
        constexpr T c = (T)fft_cos(2 * k, N), s = (T)fft_sin(2 * k, N);
        return mk<T>(a.x * c - a.y * s, a.x * s + a.y * c);
    }
}

// ------------------------------------------------------------ DFTs in registers ---
// first factor of a composite radix
__host__ __device__ constexpr int fft_first(int r) {
    return r == 16 ? 4 : r % 2 == 0 && r > 4 ? 2 : r == 9 ? 3 : r == 15 ? 3 : r;
}

// v_t <- sum_r v_r exp(2 pi i r t / R)
template <int R, class T>
__device__ __forceinline__ void fft_dft(cx_t<T> (&v)[R]) {
    using C = cx_t<T>;
    if constexpr (R == 2) {
        const C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (R == 4) {
        const C s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
        const C s13 = cadd(v[1], v[3]), d13 = csub(v[1], v[3]);
        const C jd = mk<T>(-d13.y, d13.x);
        v[0] = cadd(s02, s13);
        v[2] = csub(s02, s13);
        v[1] = cadd(d02, jd);
        v[3] = csub(d02, jd);
    } else if constexpr (fft_first(R) == R) {
        // odd prime: r and R - r together, V_t and V_R-t = (v0 + sum c a) +- i (sum s b)
        constexpr int H = (R - 1) / 2;
        C a[H], b[H];
        C v0 = v[0], sum = v0;
        fft_for<H>([&](auto j) {
            a[j] = cadd(v[j + 1], v[R - 1 - j]);
            b[j] = csub(v[j + 1], v[R - 1 - j]);
            sum = cadd(sum, a[j]);
        });
        v[0] = sum;
        fft_for<H>([&](auto t) {
            C m = v0, n = mk<T>(0, 0);
            fft_for<H>([&](auto j) {
                constexpr int k = (decltype(j)::value + 1) * (decltype(t)::value + 1) % R;
                constexpr T c = (T)fft_cos(2 * k, R), s = (T)fft_sin(2 * k, R);
                m = cmac(m, a[j], c);
                n = cmac(n, b[j], s);
            });
            const C jn = mk<T>(-n.y, n.x);
            v[t + 1] = cadd(m, jn);
            v[R - 1 - t] = csub(m, jn);
        });
    } else {
        // R = A B: r = B a + b, t = t1 + A t2
        constexpr int A = fft_first(R), B = R / A;
        C y[R];
        fft_for<B>([&](auto b) {
            C u[A];
            fft_for<A>([&](auto a) { u[a] = v[B * a + b]; });
            fft_dft<A, T>(u);
            fft_for<A>([&](auto t) { y[B * t + b] = fft_rot<decltype(b)::value * decltype(t)::value, R, T>(u[t]); });
        });
        fft_for<A>([&](auto t) {
            C u[B];
            fft_for<B>([&](auto b) { u[b] = y[B * t + b]; });
            fft_dft<B, T>(u);
            fft_for<B>([&](auto t2) { v[t + A * t2] = u[t2]; });
        });
    }
}

// ------------------------------------------------------------------ passes ---
// largest radix of a plan: 16 samples in registers in FP32, 10 in FP64 (and the primes 11, 13)
template <class T>
__host__ __device__ constexpr int fft_max_radix() { return sizeof(T) == 4 ? 16 : 10; }

// The radices of n, 4 bits per pass (radix - 1), 0 if n has a prime factor above 13: the fewest
// factors, then the most even ones.
inline unsigned fft_factors(int n, int max_radix) {
    unsigned best = 0;
    int best_passes = 99, best_max = 99;
    auto walk = [&](auto &self, int left, int low, unsigned plan, int passes, int top) -> void {
        if (left == 1) {
            if (passes < best_passes || (passes == best_passes && top < best_max)) {
                best = plan;
                best_passes = passes;
                best_max = top;
            }
            return;
        }
        if (passes >= 8 || passes >= best_passes) return;
        for (int r = low; r <= 16; r++)
            if (left % r == 0 && (r <= max_radix || r == 11 || r == 13))
                self(self, left / r, r, plan << 4 | (unsigned)(r - 1), passes + 1, r > top ? r : top);
    };
    if (n > 1) walk(walk, n, 2, 0u, 0, 0);
    return best;
}

// quotient of 0 <= x < 2^22 by d > 0, rd = 1 / d (the float quotient is off by at most one and
// corrected): index splits without integer division
__device__ __forceinline__ int div_n(int x, int d, float rd) {
    int q = (int)((float)x * rd);
    const int r = x - q * d;
    q -= r < 0 ? 1 : 0;
    q += r >= d ? 1 : 0;
    return q;
}

// a batch of signals in shared memory: sample n of signal (pp, qq) at p[n rs + pp ps + qq]
template <class T>
struct FftView {
    cx_t<T> *p;
    int rs, ps;
    __device__ __forceinline__ cx_t<T> &at(int n, int pp, int qq) const { return p[n * rs + pp * ps + qq]; }
};

// One pass of radix R over 3 qc signals of N samples; Ns = product of the earlier radices. With
// modes != null the samples are the Hermitian spectra of the component pairs, formed from the
// modes c[a][6][25] at the chunk's columns: Z = Y_2p + i Y_2p+1, Y_0 = Re c_0, Y_a = c_a,
// Y_N-a = conj c_a, Y_N/2 = 2 Re c_N/2.
template <int R, class T>
__device__ __forceinline__ void fft_pass_r(const cx_t<T> *modes, const FftView<T> in, const FftView<T> out, int N,
                                           int qc, int Ns, const cx_t<T> *tw2, int lane, int TEAM) {
    using C = cx_t<T>;
    const int S = 3 * qc, NR = N / R, span = NR / Ns;
    const float rS = 1.f / (float)S, rNs = 1.f / (float)Ns;
    for (int i = lane; i < NR * S; i += TEAM) {
        const int j = div_n(i, S, rS), s = i - j * S;
        const int pp = (s >= qc) + (s >= 2 * qc), qq = s - pp * qc;
        const int jn = div_n(j, Ns, rNs), k = j - jn * Ns;
        C v[R];
        if (modes) {
            const C *m = modes + 50 * pp + qq;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int n = j + r * NR, al = 2 * n > N ? N - n : n;
                const C c1 = m[al * 150], c2 = m[al * 150 + 25];
                // c2's and the conjugate's signs; at 0 and N/2 only the real parts count
                const T f = (n == 0 || 2 * n == N) ? (T)0 : 2 * n > N ? (T)-1 : (T)1;
                const T g = 2 * n == N ? (T)2 : (T)1;
                v[r] = mk<T>(g * c1.x - f * c2.y, g * c2.x + f * c1.y);
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; r++) v[r] = in.at(j + r * NR, pp, qq);
            if (k) {
                int m = 0;
#pragma unroll
                for (int r = 1; r < R; r++) {
                    m += k * span;
                    v[r] = cmul<T>(v[r], tw2[m]);
                }
            }
        }
        fft_dft<R, T>(v);
        const int d = jn * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) out.at(d + r * Ns, pp, qq) = v[r];
    }
}

// the whole transform by the plan, from the modes or from view b0 into b1 and back in turn;
// returns the view that holds the result (natural order); the team synchronises after every pass
template <class T>
__device__ __forceinline__ FftView<T> fft_run(const cx_t<T> *modes, FftView<T> b0, FftView<T> b1, int N, int qc,
                                              unsigned plan, const cx_t<T> *tw2, int team, int lane, int TEAM) {
    FftView<T> in = b0, out = b1;
    int Ns = 1;
    for (; plan; plan >>= 4) {
        const int R = (int)(plan & 15u) + 1;
#define AXG_FFT_PASS(r) \
    case r: fft_pass_r<r, T>(modes, in, out, N, qc, Ns, tw2, lane, TEAM); break;
        switch (R) {
            AXG_FFT_PASS(2) AXG_FFT_PASS(3) AXG_FFT_PASS(4) AXG_FFT_PASS(5) AXG_FFT_PASS(6) AXG_FFT_PASS(7)
            AXG_FFT_PASS(8) AXG_FFT_PASS(9) AXG_FFT_PASS(10) AXG_FFT_PASS(11) AXG_FFT_PASS(13)
            default:
                if constexpr (fft_max_radix<T>() > 10) {
                    switch (R) {
                        AXG_FFT_PASS(12) AXG_FFT_PASS(14) AXG_FFT_PASS(15) AXG_FFT_PASS(16)
                    }
                }
        }
#undef AXG_FFT_PASS
        team_sync(team, TEAM);
        modes = nullptr;
        Ns *= R;
        const FftView<T> t = in; in = out; out = t;
    }
    return in;
}

}  // namespace axg
