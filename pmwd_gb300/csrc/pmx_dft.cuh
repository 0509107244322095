// In-register DFTs shared by the FFT kernels.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace pmx {

constexpr double kPi = 3.141592653589793238462643383279502884;

// cos/sin by their Taylor series on [-pi, pi], evaluated at compile time;
// used only for the exact small-radix twiddles exp(-2 pi i k / R), R <= 32.
constexpr double taylor_cos(double x) {
    double term = 1.0, sum = 1.0;
    for (int i = 1; i < 24; ++i) {
        term *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
        sum += term;
    }
    return sum;
}
constexpr double taylor_sin(double x) {
    double term = x, sum = x;
    for (int i = 1; i < 24; ++i) {
        term *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
        sum += term;
    }
    return sum;
}

struct Twiddle32 {
    float c[32], s[32];  // cos / sin of 2 pi k / 32
    constexpr Twiddle32() : c(), s() {
        for (int k = 0; k < 32; ++k) {
            double a = 2.0 * kPi * k / 32.0;
            if (a > kPi) a -= 2.0 * kPi;
            c[k] = (float)taylor_cos(a);
            s[k] = (float)taylor_sin(a);
        }
    }
};

template <int R>
struct Log2 {
    static constexpr int v = R <= 1 ? 0 : 1 + Log2<R / 2>::v;
};
template <>
struct Log2<1> {
    static constexpr int v = 0;
};

// In-register DFT of length R (power of two, <= 32): natural-order input,
// output in bit-reversed order (element k holds frequency brev(k)); radix-2
// decimation in frequency.  The butterflies are generated by fold
// expressions so every register index is a compile-time constant (the
// arrays stay in registers).  INV selects exp(+2 pi i ...) (unnormalised).
constexpr Twiddle32 kTw32 = Twiddle32();

template <int R, bool INV, int S, int J>
__device__ __forceinline__ void bfly(float (&re)[R], float (&im)[R]) {
    constexpr int half = 1 << (S - 1), len = 1 << S;
    constexpr int g = J / half, k = J % half;
    constexpr int a = g * len + k, b = a + half, ti = k * (32 >> S);
    const float ur = re[a], ui = im[a], vr = re[b], vi = im[b];
    re[a] = ur + vr;
    im[a] = ui + vi;
    const float dr = ur - vr, di = ui - vi;
    // twiddle exp(-+2 pi i ti / 32), a compile-time constant; 1 and -+i exactly
    if constexpr (ti == 0) {
        re[b] = dr;
        im[b] = di;
    } else if constexpr (ti == 8) {
        re[b] = INV ? -di : di;
        im[b] = INV ? dr : -dr;
    } else {
        constexpr float wc = kTw32.c[ti];
        constexpr float ws = INV ? kTw32.s[ti] : -kTw32.s[ti];
        re[b] = dr * wc - di * ws;
        im[b] = dr * ws + di * wc;
    }
}

template <int R, bool INV, int S, int... Js>
__device__ __forceinline__ void dft_stage(float (&re)[R], float (&im)[R],
                                          std::integer_sequence<int, Js...>) {
    (bfly<R, INV, S, Js>(re, im), ...);
}

template <int R, bool INV, int... Ss>
__device__ __forceinline__ void dft_stages(float (&re)[R], float (&im)[R],
                                           std::integer_sequence<int, Ss...>) {
    (dft_stage<R, INV, Log2<R>::v - Ss>(re, im, std::make_integer_sequence<int, R / 2>{}), ...);
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float (&re)[R], float (&im)[R]) {
    dft_stages<R, INV>(re, im, std::make_integer_sequence<int, Log2<R>::v>{});
}

// bit reversal of the low `bits` bits
__device__ __forceinline__ int brev(int k, int bits) { return (int)(__brev((unsigned)k) >> (32 - bits)); }


constexpr int cbrev(int k, int bits) {
    int r = 0;
    for (int b = 0; b < bits; ++b) r |= ((k >> b) & 1) << (bits - 1 - b);
    return r;
}

// out[i] = in[brev(i)]: bit-reversed register order -> natural order, with
// compile-time indices (fold expression).
template <int R, int... Is>
__device__ __forceinline__ void unbrev_impl(const float2 (&in)[R], float2 (&out)[R],
                                            std::integer_sequence<int, Is...>) {
    ((out[Is] = in[cbrev(Is, Log2<R>::v)]), ...);
}
template <int R>
__device__ __forceinline__ void unbrev(const float2 (&in)[R], float2 (&out)[R]) {
    unbrev_impl<R>(in, out, std::make_integer_sequence<int, R>{});
}

// float2 wrappers of the split-array register DFT
template <int R, bool INV, int... Is>
__device__ __forceinline__ void dft2_impl(float2 (&v)[R], std::integer_sequence<int, Is...>) {
    float re[R], im[R];
    ((re[Is] = v[Is].x, im[Is] = v[Is].y), ...);
    dft<R, INV>(re, im);
    ((v[Is] = make_float2(re[Is], im[Is])), ...);
}
template <int R, bool INV>
__device__ __forceinline__ void dft2(float2 (&v)[R]) {
    dft2_impl<R, INV>(v, std::make_integer_sequence<int, R>{});
}

// f(integral_constant<int, 0>{}), ..., f(integral_constant<int, N - 1>{}):
// an unrolled loop whose index is a constant expression.
template <class F, int... Is>
__device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, Is...>) {
    (f(std::integral_constant<int, Is>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F &&f) {
    static_for_impl(static_cast<F &&>(f), std::make_integer_sequence<int, N>{});
}

constexpr double circle(double a) {  // a - 2 pi round(a / 2 pi) for a in (-4 pi, 4 pi)
    while (a > kPi) a -= 2.0 * kPi;
    while (a < -kPi) a += 2.0 * kPi;
    return a;
}

// Frequency of element e after reg_dft<R> (R = 2^k or 3 * 2^k).
template <int R>
constexpr int reg_freq(int e) {
    if constexpr (R % 3 == 0) {
        constexpr int Q = R / 3;
        return 3 * cbrev(e % Q, Log2<Q>::v) + e / Q;
    } else {
        return cbrev(e, Log2<R>::v);
    }
}

// In-register DFT of length R = 2^k or 3 * 2^k (<= 32): natural-order input,
// element e of the output holds frequency reg_freq<R>(e).  3 * 2^k: one
// radix-3 decimation-in-frequency stage, then three power-of-two DFTs.
template <int R, bool INV>
__device__ __forceinline__ void reg_dft(float2 (&v)[R]) {
    if constexpr (R % 3 == 0) {
        constexpr int Q = R / 3;
        constexpr float s3 = (float)0.86602540378443864676372317075294;
        static_for<Q>([&](auto J) {
            constexpr int j = J;
            const float2 a = v[j], b = v[j + Q], c = v[j + 2 * Q];
            const float2 s = make_float2(b.x + c.x, b.y + c.y);
            const float2 d = make_float2(s3 * (b.x - c.x), s3 * (b.y - c.y));
            const float2 m = make_float2(a.x - 0.5f * s.x, a.y - 0.5f * s.y);
            v[j] = make_float2(a.x + s.x, a.y + s.y);
            // y1 = m -+ i d, y2 = m +- i d (forward: upper signs)
            float2 y1 = INV ? make_float2(m.x - d.y, m.y + d.x) : make_float2(m.x + d.y, m.y - d.x);
            float2 y2 = INV ? make_float2(m.x + d.y, m.y - d.x) : make_float2(m.x - d.y, m.y + d.x);
            if constexpr (j > 0) {
                constexpr double a1 = circle((INV ? 2.0 : -2.0) * kPi * j / R);
                constexpr double a2 = circle((INV ? 4.0 : -4.0) * kPi * j / R);
                constexpr float c1 = (float)taylor_cos(a1), s1 = (float)taylor_sin(a1);
                constexpr float c2 = (float)taylor_cos(a2), s2 = (float)taylor_sin(a2);
                y1 = make_float2(y1.x * c1 - y1.y * s1, y1.x * s1 + y1.y * c1);
                y2 = make_float2(y2.x * c2 - y2.y * s2, y2.x * s2 + y2.y * c2);
            }
            v[j + Q] = y1;
            v[j + 2 * Q] = y2;
        });
        static_for<3>([&](auto K) {
            constexpr int o = K * Q;
            float2 u[Q];
            static_for<Q>([&](auto J) { u[J] = v[o + J]; });
            dft2<Q, INV>(u);
            static_for<Q>([&](auto J) { v[o + J] = u[J]; });
        });
    } else {
        dft2<R, INV>(v);
    }
}

// out[frequency] = in[element]: the register order of reg_dft back to the
// natural order, by compile-time renaming.
template <int R>
__device__ __forceinline__ void reg_natural(const float2 (&in)[R], float2 (&out)[R]) {
    static_for<R>([&](auto E) { out[reg_freq<R>(E)] = in[E]; });
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cmulc(float2 a, float2 b) {  // a * conj(b)
    return make_float2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

}  // namespace pmx
