// Block-level mixed-radix FFTs of batched lines, for transforms whose loads and stores are part
// of the kernel (filters, masks, products, band limits).
//
// A line of n points (n = R0 R1 or R0 R1 R2 with radices up to 16) takes two or three Stockham
// passes: the first reads its operands through a functor (global memory, transformed on the way),
// the last hands its results to a functor, and only the exchange between passes goes through
// shared memory.  A butterfly of 8 - 16 points per thread in registers keeps that to one exchange
// for most lengths up to 256, and that many independent loads in flight per thread.  A kernel instantiated for a length
// N > 0 has that length's radices, strides and counts in its code (AxisUse); its form for N = 0 takes the plan at run
// time and serves every length (the branch on the radix is uniform).
//   pass q (Ns = product of the earlier radices, nb = n / R): butterfly j < nb takes elements
//   j + r nb, twiddled by e^{+-2 pi i r (j mod Ns) / (Ns R)}, to (j / Ns) Ns R + j mod Ns + r Ns.
#pragma once
#include <cmath>
#include <type_traits>
#include "pb_common.cuh"

namespace pb {
namespace fft {

constexpr int MAX_RADIX = 16;

// ---- complex arithmetic -------------------------------------------------------------
template <typename C> __device__ __forceinline__ C add(C a, C b) { a.x += b.x; a.y += b.y; return a; }
template <typename C> __device__ __forceinline__ C sub(C a, C b) { a.x -= b.x; a.y -= b.y; return a; }
template <typename C> __device__ __forceinline__ C mul(C a, C b) {
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
template <int SIGN, typename C> __device__ __forceinline__ C mul_tw(C a, C w) {  // w conjugated for SIGN < 0
    if (SIGN < 0) w.y = -w.y;
    return mul(a, w);
}
template <int SIGN, typename C> __device__ __forceinline__ C rot90(C a) {  // SIGN i a
    C r;
    r.x = SIGN > 0 ? -a.y : a.y;
    r.y = SIGN > 0 ? a.x : -a.x;
    return r;
}

// cos and sin of 2 pi p / q by their Taylor series about the nearest multiple of pi / 4 turns
// (|argument| <= pi / 4), at compile time
constexpr double taylor_sin(double x) {
    double t = x, s = x;
    for (int k = 1; k < 12; ++k) {
        t *= -x * x / ((2.0 * k) * (2.0 * k + 1.0));
        s += t;
    }
    return s;
}
constexpr double taylor_cos(double x) {
    double t = 1.0, s = 1.0;
    for (int k = 1; k < 12; ++k) {
        t *= -x * x / ((2.0 * k - 1.0) * (2.0 * k));
        s += t;
    }
    return s;
}
constexpr double PI = 3.14159265358979323846;
constexpr double cos_turn(int p, int q) {
    p %= q;
    if (p < 0) p += q;
    if (2 * p > q) p = q - p;                          // cos(2 pi - x) = cos x
    if (4 * p > q) return -cos_turn(q - 2 * p, 2 * q);  // cos(pi - x) = -cos x
    if (8 * p > q) return taylor_sin(PI * (q - 4 * p) / (2.0 * q));
    return taylor_cos(2.0 * PI * p / q);
}
constexpr double sin_turn(int p, int q) { return cos_turn(4 * p - q, 4 * q); }  // sin x = cos(x - pi / 2)
// cos and sin of 2 pi p / N, p < N, evaluated by the compiler
template <int N> struct Turns {
    double c[N], s[N];
    constexpr Turns() : c(), s() {
        for (int p = 0; p < N; ++p) {
            c[p] = cos_turn(p, N);
            s[p] = sin_turn(p, N);
        }
    }
};

// ---- DFTs in registers --------------------------------------------------------------
template <int R, int SIGN, typename T, typename C> struct Dft;

template <int SIGN, typename T, typename C> struct Dft<1, SIGN, T, C> {
    static __device__ __forceinline__ void run(C (&)[1]) {}
};
template <int SIGN, typename T, typename C> struct Dft<2, SIGN, T, C> {
    static __device__ __forceinline__ void run(C (&v)[2]) {
        const C t = v[0];
        v[0] = add(t, v[1]);
        v[1] = sub(t, v[1]);
    }
};
template <int SIGN, typename T, typename C> struct Dft<4, SIGN, T, C> {
    static __device__ __forceinline__ void run(C (&v)[4]) {
        const C a = add(v[0], v[2]), b = sub(v[0], v[2]), c = add(v[1], v[3]), d = rot90<SIGN>(sub(v[1], v[3]));
        v[0] = add(a, c);
        v[2] = sub(a, c);
        v[1] = add(b, d);
        v[3] = sub(b, d);
    }
};
// odd primes: X[k], X[R - k] = x0 + sum_m cos(2 pi k m / R) (x_m + x_{R-m}) +- i sum_m sin(..) (x_m - x_{R-m})
template <int R, int SIGN, typename T, typename C> struct DftOdd {
    static __device__ __forceinline__ void run(C (&v)[R]) {
        constexpr int H = R / 2;
        constexpr Turns<R> W{};
        C s[H], d[H], x0 = v[0];
#pragma unroll
        for (int m = 1; m <= H; ++m) {
            s[m - 1] = add(v[m], v[R - m]);
            d[m - 1] = sub(v[m], v[R - m]);
            v[0] = add(v[0], s[m - 1]);
        }
#pragma unroll
        for (int k = 1; k <= H; ++k) {
            C a = x0, b;
            b.x = b.y = (T)0;
#pragma unroll
            for (int m = 1; m <= H; ++m) {
                const T c = (T)W.c[k * m % R], n = (T)W.s[k * m % R];
                a.x += c * s[m - 1].x;
                a.y += c * s[m - 1].y;
                b.x += n * d[m - 1].x;
                b.y += n * d[m - 1].y;
            }
            b = rot90<SIGN>(b);
            v[k] = add(a, b);
            v[R - k] = sub(a, b);
        }
    }
};
template <int SIGN, typename T, typename C> struct Dft<3, SIGN, T, C> : DftOdd<3, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<5, SIGN, T, C> : DftOdd<5, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<7, SIGN, T, C> : DftOdd<7, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<11, SIGN, T, C> : DftOdd<11, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<13, SIGN, T, C> : DftOdd<13, SIGN, T, C> {};

// R = A B: A-point transforms of the stride-B subsequences, constant twiddles, B-point transforms
template <int A, int B, int SIGN, typename T, typename C> struct DftPair {
    static __device__ __forceinline__ void run(C (&v)[A * B]) {
        constexpr Turns<A * B> W{};
        C t[B][A];
#pragma unroll
        for (int b = 0; b < B; ++b) {
#pragma unroll
            for (int a = 0; a < A; ++a) t[b][a] = v[a * B + b];
            Dft<A, SIGN, T, C>::run(t[b]);
        }
#pragma unroll
        for (int a = 0; a < A; ++a) {
            C u[B];
#pragma unroll
            for (int b = 0; b < B; ++b) {
                const int p = a * b;
                if (p == 0) u[b] = t[b][a];
                else if (4 * p == A * B) u[b] = rot90<SIGN>(t[b][a]);
                else {
                    C w;
                    w.x = (T)W.c[p];
                    w.y = (T)W.s[p];
                    u[b] = mul_tw<SIGN>(t[b][a], w);
                }
            }
            Dft<B, SIGN, T, C>::run(u);
#pragma unroll
            for (int b = 0; b < B; ++b) v[a + A * b] = u[b];
        }
    }
};
template <int SIGN, typename T, typename C> struct Dft<6, SIGN, T, C> : DftPair<2, 3, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<8, SIGN, T, C> : DftPair<2, 4, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<9, SIGN, T, C> : DftPair<3, 3, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<10, SIGN, T, C> : DftPair<2, 5, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<12, SIGN, T, C> : DftPair<4, 3, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<14, SIGN, T, C> : DftPair<2, 7, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<15, SIGN, T, C> : DftPair<3, 5, SIGN, T, C> {};
template <int SIGN, typename T, typename C> struct Dft<16, SIGN, T, C> : DftPair<4, 4, SIGN, T, C> {};

// f(std::integral_constant<int, R>) for the run-time radix R
#define PB_RADIX_CASE(K) case K: f(std::integral_constant<int, K>()); break;
template <typename F> __device__ __forceinline__ void with_radix(int R, F &&f) {
    switch (R) {
        PB_RADIX_CASE(2) PB_RADIX_CASE(3) PB_RADIX_CASE(4) PB_RADIX_CASE(5) PB_RADIX_CASE(6) PB_RADIX_CASE(7)
        PB_RADIX_CASE(8) PB_RADIX_CASE(9) PB_RADIX_CASE(10) PB_RADIX_CASE(11) PB_RADIX_CASE(12) PB_RADIX_CASE(13)
        PB_RADIX_CASE(14) PB_RADIX_CASE(15) PB_RADIX_CASE(16)
    }
}
#undef PB_RADIX_CASE

// f(radix of pass Q) for the plan AX (AxisUse below): the one radix of a compile-time length, or a switch.  (Left
// to the optimiser, the switches took the compiler ten times as long.)
template <int Q, typename AX, typename F> __device__ __forceinline__ void with_pass_radix(const AX &use, F &&f) {
    if constexpr (AX::FIXED) {
        if constexpr (Q < AX::PASSES) f(std::integral_constant<int, AX::PLAN.R[Q]>());
    } else {
        with_radix(use.v.R[Q], f);
    }
}
template <typename AX, typename F> __device__ __forceinline__ void with_last_radix(const AX &use, F &&f) {
    if constexpr (AX::FIXED) f(std::integral_constant<int, AX::PLAN.R[AX::PASSES - 1]>());
    else with_radix(use.v.R[use.v.np - 1], f);
}

// ---- plan of an axis ----------------------------------------------------------------
struct Axis {
    int n, np;            // length, passes (1 - 3)
    int R[3], nb[3], ns[3];
    uint32_t div_ns1;     // ceil(2^20 / R0): j / R0 = j div_ns1 >> 20 for j < 4096
    int pad;              // rows in shared memory get one element of padding per 2^pad (0: none, R0 odd)
    int tw[3];            // offset of pass q's twiddles [r - 1][j mod Ns] in the axis's table
    int tw_len;
};

__device__ __forceinline__ int div_r0(const Axis &ax, int e) { return (int)(((uint32_t)e * ax.div_ns1) >> 20); }
// element e of a padded row: a first pass writes runs of R0 from neighbouring lanes, which the padding
// puts on distinct banks
__device__ __forceinline__ int row_at(const Axis &ax, int e) { return ax.pad ? e + (e >> ax.pad) : e; }
__host__ __device__ __forceinline__ constexpr int row_len(const Axis &ax) {
    return ax.pad ? ax.n + ((ax.n - 1) >> ax.pad) : ax.n;
}

// Half of the line that element e = j + r n / R lies in, known from r when R is even: -1 below n / 2, 1 from
// n / 2 on, 0 not known.  The functors of the outer passes get it with the element, so that the frequency's
// sign costs nothing where the compiler knows r.
__device__ __forceinline__ int abs_label(int e, int n, int side) {  // |frequency| of element e
    if (side == 0) return e < (n >> 1) ? e : n - e;
    return side < 0 ? e : n - e;
}

// functor of line_pass that leaves the loaded elements as they are
struct Keep {
    template <typename C> __device__ __forceinline__ C operator()(int, C v) const { return v; }
};

// One pass (number Q) of the lines of a block.  ld(e, side) gives element e, fix(e, v) finishes it once all of
// a butterfly's loads are on their way, st(e, v, side) takes a result; `t` of `nt` threads share the line.
template <typename T, int SIGN, int Q, typename AX, typename LD, typename ST, typename FX = Keep>
__device__ __forceinline__ void line_pass(const AX &use, int t, int nt, const typename cplx<T>::type *tw, LD &&ld,
                                          ST &&st, FX &&fix = FX()) {
    using C = typename cplx<T>::type;
    const Axis &ax = use.v;
    with_pass_radix<Q>(use, [&](auto RC) {
        constexpr int R = decltype(RC)::value;
        const int nb = ax.nb[Q], ns = Q == 0 ? 1 : ax.ns[Q];
        for (int j = t; j < nb; j += nt) {
            const int jq = Q == 0 ? j : (Q == ax.np - 1 ? 0 : div_r0(ax, j));
            const int jm = Q == 0 ? 0 : j - jq * ns;
            C v[R];
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = ld(j + r * nb, R % 2 ? 0 : (2 * r >= R ? 1 : -1));
#pragma unroll
            for (int r = 0; r < R; ++r) v[r] = fix(j + r * nb, v[r]);
            if (Q > 0) {
                const C *w = tw + ax.tw[Q] + jm;
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = mul_tw<SIGN>(v[r], w[(r - 1) * ns]);
            }
            Dft<R, SIGN, T, C>::run(v);
            const int o = jq * ns * R + jm;
#pragma unroll
            for (int r = 0; r < R; ++r)
                st(o + r * ns, v[r], R % 2 || Q != ax.np - 1 ? 0 : (2 * r >= R ? 1 : -1));
        }
    });
}

// All passes of a line: operands from ld, results to st, exchanges through sm (element e of this
// line at sm[at(e)]) and, for three passes, sm2.  Every thread of the block calls it; `on`: the
// line exists (threads of other lines only join the barriers).
template <typename T, int SIGN, typename AX, typename AT, typename LD, typename ST, typename FX = Keep>
__device__ __forceinline__ void line_fft(const AX &use, int t, int nt, bool on, typename cplx<T>::type *sm,
                                         typename cplx<T>::type *sm2, const typename cplx<T>::type *tw, AT &&at,
                                         LD &&ld, ST &&st, FX &&fix = FX()) {
    using C = typename cplx<T>::type;
    const Axis &ax = use.v;
    if (ax.np == 1) {
        if (on) line_pass<T, SIGN, 0>(use, t, nt, tw, ld, st, fix);
        return;
    }
    if (on) line_pass<T, SIGN, 0>(use, t, nt, tw, ld, [&](int e, C v, int) { sm[at(e)] = v; }, fix);
    __syncthreads();
    if (ax.np == 2) {
        if (on) line_pass<T, SIGN, 1>(use, t, nt, tw, [&](int e, int) { return sm[at(e)]; }, st);
        return;
    }
    if (on)
        line_pass<T, SIGN, 1>(use, t, nt, tw, [&](int e, int) { return sm[at(e)]; }, [&](int e, C v, int) { sm2[at(e)] = v; });
    __syncthreads();
    if (on) line_pass<T, SIGN, 2>(use, t, nt, tw, [&](int e, int) { return sm2[at(e)]; }, st);
}

// ---- planning -----------------------------------------------------------------------
// n = R0 R1 with both radices at most 16 and R0 <= R1 as large as possible; 0 when impossible
__host__ __device__ constexpr int balanced_radix(int n) {
    for (int r = 16; r >= 2; --r)
        if (n % r == 0 && n / r <= MAX_RADIX && n / r >= r) return r;
    return 0;
}

// Radices of n: two passes where possible (the larger radix last), else three, the largest last radix
// whose cofactor splits in two; np = 0 when n has another prime factor than 2, 3, 5, 7, 11, 13 or needs
// more passes.  `reversed`: the same radices in the opposite order.
__host__ __device__ constexpr Axis make_axis(int n, bool reversed) {
    Axis ax{};
    int r[3] = {n, 0, 0};
    if (n < 2 || n > 4096) return ax;
    int np = 0;
    if (n <= MAX_RADIX) {
        np = 1;
    } else if (balanced_radix(n)) {
        np = 2;
        r[0] = balanced_radix(n);
        r[1] = n / r[0];
    } else {
        for (int c = MAX_RADIX; c >= 2 && !np; --c) {
            if (n % c) continue;
            const int b = balanced_radix(n / c);
            if (b && n / c / b <= c) {
                np = 3;
                r[0] = b;
                r[1] = n / c / b;
                r[2] = c;
            }
        }
        if (!np) return ax;
    }
    if (reversed && np > 1) {
        const int t = r[0];
        r[0] = r[np - 1];
        r[np - 1] = t;
    }
    ax.n = n;
    ax.np = np;
    int ns = 1;
    for (int q = 0; q < np; ++q) {
        ax.R[q] = r[q];
        ax.nb[q] = n / r[q];
        ax.ns[q] = ns;
        ax.tw[q] = ax.tw_len;
        if (q > 0) ax.tw_len += (r[q] - 1) * ns;
        ns *= r[q];
    }
    ax.div_ns1 = ((1u << 20) + (uint32_t)r[0] - 1) / (uint32_t)r[0];
    ax.pad = r[0] % 2 ? 0 : r[0] <= 2 ? 1 : r[0] <= 4 ? 2 : r[0] <= 8 ? 3 : 4;
    return ax;
}

// The axis a kernel works with: the plan of a compile-time length N (radices, strides and counts fold
// into the code), or for N = 0 the run-time plan.
template <int N, bool REV> struct AxisUse {
    static constexpr bool FIXED = true;
    static constexpr Axis PLAN = make_axis(N, REV);
    static constexpr int PASSES = PLAN.np;
    Axis v;
    __device__ __forceinline__ AxisUse(const Axis &) {
        constexpr Axis c = make_axis(N, REV);
        v = c;
    }
};
template <bool REV> struct AxisUse<0, REV> {
    static constexpr bool FIXED = false;
    const Axis &v;
    __device__ __forceinline__ AxisUse(const Axis &a) : v(a) {}
};

// e^{2 pi i r jm / (Ns R)} of every pass into out[tw_len] (re, im pairs)
void fill_twiddles(const Axis &ax, double *out);

}  // namespace fft
}  // namespace pb
