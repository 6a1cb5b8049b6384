// In-register DFTs of up to 16 points and the switch over their lengths, used
// by the line transforms, and their copies into shared memory.
#pragma once

#include "mpm_common.cuh"
#include "mpm_fft_consts.cuh"

#include <type_traits>

namespace mpm {

namespace {

// -i v (forward rotation) or +i v (inverse)
template <typename R, bool INV>
__device__ __forceinline__ cplx<R> rot(cplx<R> v) {
    return INV ? mk<R>(-v.y, v.x) : mk<R>(v.y, -v.x);
}

template <typename R, bool INV, int RAD>
__device__ __forceinline__ void dft_small(cplx<R> (&x)[RAD]);

// W_N^j = exp(-2 pi i j / N) (conjugated for INV) from the constant tables
template <typename R, bool INV, int N>
__device__ __forceinline__ cplx<R> wconst(int j) {
    cplx<R> w;
    static_assert(N == 7 || (N >= 9 && N <= 16), "no constant table for this radix");
    if constexpr (sizeof(R) == 8) {
        if constexpr (N == 7) w = kW7d[j];
        else if constexpr (N == 9) w = kW9d[j];
        else if constexpr (N == 10) w = kW10d[j];
        else if constexpr (N == 11) w = kW11d[j];
        else if constexpr (N == 12) w = kW12d[j];
        else if constexpr (N == 13) w = kW13d[j];
        else if constexpr (N == 14) w = kW14d[j];
        else if constexpr (N == 15) w = kW15d[j];
        else w = kW16d[j];
    } else {
        if constexpr (N == 7) w = kW7f[j];
        else if constexpr (N == 9) w = kW9f[j];
        else if constexpr (N == 10) w = kW10f[j];
        else if constexpr (N == 11) w = kW11f[j];
        else if constexpr (N == 12) w = kW12f[j];
        else if constexpr (N == 13) w = kW13f[j];
        else if constexpr (N == 14) w = kW14f[j];
        else if constexpr (N == 15) w = kW15f[j];
        else w = kW16f[j];
    }
    if (INV) w.y = -w.y;
    return w;
}

// Composite DFT of A*B points in registers (Cooley-Tukey, decimation in
// time): input m = B m1 + m2, output k = k1 + A k2,
//   y_k = sum_m2 W_B^(m2 k2) [ W_N^(m2 k1) sum_m1 x_(B m1 + m2) W_A^(m1 k1) ].
template <typename R, bool INV, int A, int B>
__device__ __forceinline__ void dft_ct(cplx<R> (&x)[A * B]) {
    constexpr int N = A * B;
    cplx<R> z[B][A];
#pragma unroll
    for (int m2 = 0; m2 < B; ++m2) {
        cplx<R> t[A];
#pragma unroll
        for (int m1 = 0; m1 < A; ++m1) t[m1] = x[B * m1 + m2];
        dft_small<R, INV, A>(t);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) z[m2][k1] = m2 * k1 == 0 ? t[k1] : t[k1] * wconst<R, INV, N>(m2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
        cplx<R> t[B];
#pragma unroll
        for (int m2 = 0; m2 < B; ++m2) t[m2] = z[m2][k1];
        dft_small<R, INV, B>(t);
#pragma unroll
        for (int k2 = 0; k2 < B; ++k2) x[k1 + A * k2] = t[k2];
    }
}

// Odd prime P in registers: with a_q = x_q + x_(P-q), b_q = x_q - x_(P-q),
// y_p = x_0 + sum_q a_q cos(2 pi p q / P) -+ i sum_q b_q sin(2 pi p q / P)
// and y_(P-p) the same with the sine term negated.
template <typename R, bool INV, int P>
__device__ __forceinline__ void dft_odd(cplx<R> (&x)[P]) {
    constexpr int H = (P - 1) / 2;
    cplx<R> a[H], b[H];
#pragma unroll
    for (int q = 1; q <= H; ++q) {
        a[q - 1] = x[q] + x[P - q];
        b[q - 1] = x[q] - x[P - q];
    }
    cplx<R> y0 = x[0];
#pragma unroll
    for (int q = 0; q < H; ++q) y0 += a[q];
#pragma unroll
    for (int p = 1; p <= H; ++p) {
        cplx<R> t = x[0], u = mk<R>(R(0), R(0));
#pragma unroll
        for (int q = 1; q <= H; ++q) {
            const cplx<R> w = wconst<R, false, P>((p * q) % P);   // (cos, -sin)
            t = t + a[q - 1] * w.x;
            u = u + b[q - 1] * (-w.y);
        }
        // -i u (forward) or +i u (inverse)
        const cplx<R> ru = rot<R, INV>(u);
        x[p] = t + ru;
        x[P - p] = t - ru;
    }
    x[0] = y0;
}

// In-register DFT of RAD points, y_p = sum_q x_q W^(p q), W = exp(-+2 pi i/RAD),
// written out for 2, 3, 4, 5, 6, 8, tabulated primes 7, 11, 13 and composed
// 9, 10, 12, 14, 15, 16.
template <typename R, bool INV, int RAD>
__device__ __forceinline__ void dft_small(cplx<R> (&x)[RAD]) {
    if constexpr (RAD == 1) {
    } else if constexpr (RAD == 7) {
        dft_odd<R, INV, 7>(x);
    } else if constexpr (RAD == 9) {
        dft_ct<R, INV, 3, 3>(x);
    } else if constexpr (RAD == 10) {
        dft_ct<R, INV, 2, 5>(x);
    } else if constexpr (RAD == 11) {
        dft_odd<R, INV, 11>(x);
    } else if constexpr (RAD == 12) {
        dft_ct<R, INV, 4, 3>(x);
    } else if constexpr (RAD == 13) {
        dft_odd<R, INV, 13>(x);
    } else if constexpr (RAD == 14) {
        dft_ct<R, INV, 2, 7>(x);
    } else if constexpr (RAD == 15) {
        dft_ct<R, INV, 3, 5>(x);
    } else if constexpr (RAD == 16) {
        dft_ct<R, INV, 4, 4>(x);
    } else if constexpr (RAD == 2) {
        const cplx<R> a = x[0], b = x[1];
        x[0] = a + b;
        x[1] = a - b;
    } else if constexpr (RAD == 3) {
        const R h = R(0.86602540378443864676);   // sin(2 pi / 3)
        const cplx<R> s = x[1] + x[2];
        const cplx<R> t = x[0] - s * R(0.5);
        const cplx<R> d = (x[1] - x[2]) * h;
        x[0] = x[0] + s;
        x[1] = t + rot<R, INV>(d);
        x[2] = t - rot<R, INV>(d);
    } else if constexpr (RAD == 4) {
        const cplx<R> a = x[0] + x[2], b = x[0] - x[2], c = x[1] + x[3], d = rot<R, INV>(x[1] - x[3]);
        x[0] = a + c;
        x[2] = a - c;
        x[1] = b + d;
        x[3] = b - d;
    } else if constexpr (RAD == 5) {
        const R c1 = R(0.30901699437494742410), c2 = R(-0.80901699437494742410);
        const R s1 = R(0.95105651629515357212), s2 = R(0.58778525229247312917);
        const cplx<R> a1 = x[1] + x[4], b1 = x[1] - x[4], a2 = x[2] + x[3], b2 = x[2] - x[3];
        const cplx<R> t1 = x[0] + a1 * c1 + a2 * c2, t2 = x[0] + a1 * c2 + a2 * c1;
        const cplx<R> u1 = rot<R, INV>(b1 * s1 + b2 * s2), u2 = rot<R, INV>(b1 * s2 - b2 * s1);
        x[0] = x[0] + a1 + a2;
        x[1] = t1 + u1;
        x[4] = t1 - u1;
        x[2] = t2 + u2;
        x[3] = t2 - u2;
    } else if constexpr (RAD == 6) {
        // even / odd halves as two 3-point DFTs, then W6^p between them
        cplx<R> e[3] = {x[0], x[2], x[4]}, o[3] = {x[1], x[3], x[5]};
        dft_small<R, INV, 3>(e);
        dft_small<R, INV, 3>(o);
        const R h = R(0.86602540378443864676);
        const cplx<R> w1 = mk<R>(R(0.5), INV ? h : -h), w2 = mk<R>(R(-0.5), INV ? h : -h);
        const cplx<R> o1 = o[1] * w1, o2 = o[2] * w2;
        x[0] = e[0] + o[0];
        x[3] = e[0] - o[0];
        x[1] = e[1] + o1;
        x[4] = e[1] - o1;
        x[2] = e[2] + o2;
        x[5] = e[2] - o2;
    } else if constexpr (RAD == 8) {
        const R q = R(0.70710678118654752440);
        cplx<R> u[4], v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            u[k] = x[k] + x[k + 4];
            v[k] = x[k] - x[k + 4];
        }
        // v_k *= W8^k
        v[1] = (v[1] + rot<R, INV>(v[1])) * q;
        v[2] = rot<R, INV>(v[2]);
        v[3] = (rot<R, INV>(v[3]) - v[3]) * q;
        dft_small<R, INV, 4>(u);
        dft_small<R, INV, 4>(v);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[2 * k] = u[k];
            x[2 * k + 1] = v[k];
        }
    }
}

template <int CLS, typename Fn>
__device__ __forceinline__ void radix_dispatch(int r, Fn&& fn) {
    switch (r) {
        case 1: fn(std::integral_constant<int, 1>{}); break;
        case 2: fn(std::integral_constant<int, 2>{}); break;
        case 3: fn(std::integral_constant<int, 3>{}); break;
        case 4: fn(std::integral_constant<int, 4>{}); break;
        case 5: fn(std::integral_constant<int, 5>{}); break;
        case 6: fn(std::integral_constant<int, 6>{}); break;
        case 7: fn(std::integral_constant<int, 7>{}); break;
        case 8: fn(std::integral_constant<int, 8>{}); break;
        default:
            // register classes: radices up to CLS only (8, 12 or 16)
            if constexpr (CLS > 8) {
                switch (r) {
                    case 9: fn(std::integral_constant<int, 9>{}); break;
                    case 10: fn(std::integral_constant<int, 10>{}); break;
                    case 11: fn(std::integral_constant<int, 11>{}); break;
                    case 12: fn(std::integral_constant<int, 12>{}); break;
                    default: break;
                }
            }
            if constexpr (CLS > 12) {
                switch (r) {
                    case 13: fn(std::integral_constant<int, 13>{}); break;
                    case 14: fn(std::integral_constant<int, 14>{}); break;
                    case 15: fn(std::integral_constant<int, 15>{}); break;
                    case 16: fn(std::integral_constant<int, 16>{}); break;
                    default: break;
                }
            }
            break;
    }
}

// global -> shared copy of one element without a register round trip, so a
// thread's whole share of the line is in flight at once (src_bytes = 0 fills
// the element with zeros and reads nothing)
template <typename R>
__device__ __forceinline__ void copy_async(cplx<R>* dst, const cplx<R>* src, bool live) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    const int bytes = live ? int(sizeof(cplx<R>)) : 0;
    if constexpr (sizeof(cplx<R>) == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

}  // namespace

}  // namespace mpm
