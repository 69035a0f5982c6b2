// Half-full line transforms for the fused FFT chain: a line of P points of
// which the first P/2 at most are non-zero going in (forward) or wanted
// coming out (inverse), by T threads of one warp, FFTW sign convention
// (forward exp(-i)), unnormalised.
//
// P = T * N1, PER = N1 / T.  x[n], n = t + T k (t < T, k < N1):
//   X[a + N1 b] = sum_t w_T^(t b) [ w_P^(t a) sum_k x[t + T k] w_N1^(k a) ]
// forward: thread t holds x[t + T k], k < N1/2, in registers (the other half
// is zero), forms the N1-point DFT as two DFTs of half the length (even and
// odd a), multiplies by w_P^(t a); the line's threads exchange through shared
// memory; thread t then forms the T-point DFTs of its PER values of a and
// holds X[t PER + p + N1 b] as u[p][b].  The inverse runs the same steps
// backwards from u[p][b] and ends with x[t + T k], k < N1/2, so that between
// the two a spectrum can be multiplied in registers, and each transform costs
// one exchange instead of a store, two exchanges and a load.
//
// The twiddles inside a thread's DFTs are compile-time constants; w_P^(t a)
// comes from the line's table tw[i] = exp(-2 pi i i / P).  Every step is a
// host function too, so that a host program can run the threads of a line in
// turn.
#pragma once
#include <utility>

#include "common.cuh"

// exp(2 pi i e / N) at compile time: octant reduction, then Taylor series on
// [0, pi/4] (terms below 1e-19 dropped)
constexpr double CT_PI = 3.14159265358979323846264338327950288;
SCD_HD constexpr double ct_sin(double x) {
    double s = 0, t = x;
    for (int k = 1; k < 24; k += 2) { s += t; t *= -x * x / ((k + 1) * (k + 2)); }
    return s;
}
SCD_HD constexpr double ct_cos(double x) {
    double s = 0, t = 1;
    for (int k = 0; k < 24; k += 2) { s += t; t *= -x * x / ((k + 1) * (k + 2)); }
    return s;
}
SCD_HD constexpr double ct_cos2pi(int e, int N) {
    const int r = ((e % N) + N) % N, o = 8 * r / N;
    const double x = (o & 1) ? 2 * CT_PI * ((o + 1) * N - 8 * r) / (8.0 * N) : 2 * CT_PI * (8 * r - o * N) / (8.0 * N);
    const double c = ct_cos(x), s = ct_sin(x);
    return o == 0 || o == 7 ? c : o == 1 ? s : o == 2 ? -s : o == 3 || o == 4 ? -c : o == 5 ? -s : s;
}
SCD_HD constexpr double ct_sin2pi(int e, int N) { return ct_cos2pi(4 * e - N, 4 * N); }

template <typename F, int... I> SCD_HD void ct_each(F f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, typename F> SCD_HD void ct_for(F f) { ct_each(f, std::make_integer_sequence<int, N>{}); }

template <typename C> SCD_HD C cscale_r(C v, double s);
template <> SCD_HD cd cscale_r<cd>(cd v, double s) { return make_double2(SCD_MUL(v.x, s), SCD_MUL(v.y, s)); }
template <> SCD_HD cf cscale_r<cf>(cf v, double s) { return make_float2(SCD_MULF(v.x, (float)s), SCD_MULF(v.y, (float)s)); }
// a + s b
template <typename C> SCD_HD C cadd_r(C a, double s, C b);
template <> SCD_HD cd cadd_r<cd>(cd a, double s, cd b) { return make_double2(SCD_FMA(s, b.x, a.x), SCD_FMA(s, b.y, a.y)); }
template <> SCD_HD cf cadd_r<cf>(cf a, double s, cf b) {
    return make_float2(SCD_FMAF((float)s, b.x, a.x), SCD_FMAF((float)s, b.y, a.y));
}
// -i v (forward) or +i v (inverse)
template <bool INV, typename C> SCD_HD C crot(C v) {
    C r;
    r.x = INV ? -v.y : v.y;
    r.y = INV ? v.x : -v.x;
    return r;
}

// v * exp(-/+ 2 pi i E / N)
template <int E, int N, bool INV, typename C> SCD_HD C ct_twiddle(C v) {
    constexpr int e = ((E % N) + N) % N;
    if constexpr (e == 0) return v;
    else if constexpr (4 * e == N) return crot<INV>(v);
    else if constexpr (2 * e == N) return cscale_r<C>(v, -1.0);
    else if constexpr (4 * e == 3 * N) return crot<!INV>(v);
    else {
        constexpr double c = ct_cos2pi(e, N), s = INV ? ct_sin2pi(e, N) : -ct_sin2pi(e, N);
        return cmul(cmake<C>(c, s), v);
    }
}

// in-place DFT of prime length R = 3, 5, 7: pairs x_j +- x_(R-j)
template <int R, bool INV, typename C> SCD_HD void dft_prime(C (&x)[R]) {
    constexpr int H = R / 2;
    C p[H], m[H], y0 = x[0];
    ct_for<H>([&](auto j) {
        p[j] = cadd(x[j + 1], x[R - 1 - j]);
        m[j] = crot<INV>(csub(x[j + 1], x[R - 1 - j]));
        y0 = cadd(y0, p[j]);
    });
    C a[H], b[H];
    ct_for<H>([&](auto k) {
        a[k] = x[0];
        ct_for<H>([&](auto j) {
            constexpr int e = (decltype(j)::value + 1) * (decltype(k)::value + 1);
            a[k] = cadd_r<C>(a[k], ct_cos2pi(e, R), p[j]);
            if constexpr (decltype(j)::value == 0) b[k] = cscale_r<C>(m[j], ct_sin2pi(e, R));
            else b[k] = cadd_r<C>(b[k], ct_sin2pi(e, R), m[j]);
        });
    });
    x[0] = y0;
    ct_for<H>([&](auto k) {
        x[k + 1] = cadd(a[k], b[k]);
        x[R - 1 - k] = csub(a[k], b[k]);
    });
}

// in-place DFT of length N (natural order), N = 2^a 3^b 5^c 7^d
template <int N, bool INV, typename C> SCD_HD void ct_dft(C (&v)[N]) {
    if constexpr (N == 1) {
    } else if constexpr (N == 2) {
        const C a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (N == 4) {
        const C a0 = cadd(v[0], v[2]), a1 = csub(v[0], v[2]), a2 = cadd(v[1], v[3]), a3 = crot<INV>(csub(v[1], v[3]));
        v[0] = cadd(a0, a2);
        v[2] = csub(a0, a2);
        v[1] = cadd(a1, a3);
        v[3] = csub(a1, a3);
    } else if constexpr (N == 3 || N == 5 || N == 7) {
        dft_prime<N, INV>(v);
    } else {
        constexpr int R = N % 4 == 0 && N != 8 ? 4 : N % 2 == 0 ? 2 : N % 3 == 0 ? 3 : N % 5 == 0 ? 5 : 7, M = N / R;
        C t[R][M];
        ct_for<R>([&](auto j) {
            ct_for<M>([&](auto m) { t[j][m] = v[j + R * m]; });
            ct_dft<M, INV>(t[j]);
        });
        ct_for<M>([&](auto k1) {
            C u[R];
            ct_for<R>([&](auto j) { u[j] = ct_twiddle<decltype(j)::value * decltype(k1)::value, N, INV>(t[j][k1]); });
            ct_dft<R, INV>(u);
            ct_for<R>([&](auto k2) { v[k1 + M * k2] = u[k2]; });
        });
    }
}

// The lengths the fused chain takes, the threads of a line and the exchange
// buffer: value a of thread t at t * ROW + a, lines ES apart.  A half-warp
// holds four threads of four lines (eight of two for T = 2): with ROW = 4 or
// 12 mod 16 (8 for T = 2) and ES = 1 mod 16 its stores fall in distinct
// 8-byte banks.
constexpr bool half_len(int P) {
    return P == 16 || P == 32 || P == 40 || P == 48 || P == 64 || P == 80 || P == 96 || P == 112 || P == 128 || P == 192;
}
constexpr int half_row(int n1, int T) {
    int r = n1;
    while (T == 2 ? r % 16 != 8 : (r % 16 != 4 && r % 16 != 12)) ++r;
    return r;
}
constexpr int half_threads(int P) { return P == 40 ? 2 : P % 64 == 0 ? 8 : 4; }
constexpr int half_es(int P) { return half_threads(P) * half_row(P / half_threads(P), half_threads(P)) + 1; }
constexpr int half_ew(int P) { return 32 / half_threads(P) * half_es(P); }
template <int P> struct HalfLine {
    static_assert(half_len(P), "length");
    static constexpr int T = half_threads(P);
    static constexpr int N1 = P / T, M = N1 / 2, PER = N1 / T;
    static_assert(N1 * T == P && PER * T == N1 && 2 * M == N1, "P = T T PER");
    static constexpr int ROW = half_row(N1, T), ES = half_es(P);
    static constexpr int LW = 32 / T;                // lines of a warp
    static constexpr int EW = half_ew(P);             // exchange elements of a warp
};
// thread and line of a lane: four consecutive lanes are threads 0..3
template <int P> SCD_HD int half_t(int lane) {
    constexpr int T = HalfLine<P>::T;
    return T == 8 ? (lane & 3) | ((lane >> 4) << 2) : lane % T;
}
template <int P> SCD_HD int half_l(int lane) {
    constexpr int T = HalfLine<P>::T;
    return T == 8 ? (lane >> 2) & 3 : lane / T;
}

// w_P^(t a), conjugated for the inverse
template <bool INV, typename C> SCD_HD C half_tw(const C *tw, int i) {
    C w = tw[i];
    if (INV) w.y = -w.y;
    return w;
}
// forward, before the exchange: x[k] = x(t + T k) -> line buffer e
template <int P, typename C> SCD_HD void half_fwd_a(const C (&x)[HalfLine<P>::M], C *e, const C *tw, int t) {
    using H = HalfLine<P>;
    C ev[H::M], od[H::M];
    ct_for<H::M>([&](auto k) {
        ev[k] = x[k];
        od[k] = ct_twiddle<decltype(k)::value, H::N1, false>(x[k]);
    });
    ct_dft<H::M, false>(ev);
    ct_dft<H::M, false>(od);
    C *row = e + t * H::ROW;
    ct_for<H::M>([&](auto q) {
        constexpr int a = 2 * decltype(q)::value;
        row[a] = a ? cmul(half_tw<false>(tw, t * a), ev[q]) : ev[q];
        row[a + 1] = cmul(half_tw<false>(tw, t * (a + 1)), od[q]);
    });
}
// forward, after the exchange: u[p][b] = X(t PER + p + N1 b)
template <int P, typename C>
SCD_HD void half_fwd_b(const C *e, C (&u)[HalfLine<P>::PER][HalfLine<P>::T], int t) {
    using H = HalfLine<P>;
    ct_for<H::PER>([&](auto p) {
        ct_for<H::T>([&](auto m) { u[p][m] = e[m * H::ROW + t * H::PER + p]; });
        ct_dft<H::T, false>(u[p]);
    });
}
// inverse, before the exchange
template <int P, typename C> SCD_HD void half_inv_b(C (&u)[HalfLine<P>::PER][HalfLine<P>::T], C *e, int t) {
    using H = HalfLine<P>;
    ct_for<H::PER>([&](auto p) {
        ct_dft<H::T, true>(u[p]);
        ct_for<H::T>([&](auto m) { e[m * H::ROW + t * H::PER + p] = u[p][m]; });
    });
}
// inverse, after the exchange: x[k] = x(t + T k), k < N1/2
template <int P, typename C> SCD_HD void half_inv_a(const C *e, const C *tw, C (&x)[HalfLine<P>::M], int t) {
    using H = HalfLine<P>;
    C ev[H::M], od[H::M];
    const C *row = e + t * H::ROW;
    ct_for<H::M>([&](auto q) {
        constexpr int a = 2 * decltype(q)::value;
        ev[q] = a ? cmul(half_tw<true>(tw, t * a), row[a]) : row[a];
        od[q] = cmul(half_tw<true>(tw, t * (a + 1)), row[a + 1]);
    });
    ct_dft<H::M, true>(ev);
    ct_dft<H::M, true>(od);
    ct_for<H::M>([&](auto k) { x[k] = cadd(ev[k], ct_twiddle<decltype(k)::value, H::N1, true>(od[k])); });
}
