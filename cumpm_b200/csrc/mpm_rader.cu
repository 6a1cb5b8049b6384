// Line transform n = r1 * p with an in-register radix r1 <= 16 and the prime
// pass by Rader's algorithm (see mpm_fft.h): with g a primitive root mod p,
// a_q = x[g^-q], b_s = W_p^(g^s),
//   y[0] = x[0] + sum_q a_q,   y[g^m] = x[0] + (a (*) b)_m   (cyclic, length N = p-1)
// and the cyclic convolution is IDFT_N(DFT_N(a) . Bh) with Bh = DFT_N(b) / N
// precomputed.  N = A * B with both in-register radices, so DFT_N is one
// Cooley-Tukey step through shared memory: R1 (thread per (j, q2)) an A-point
// DFT over q1 of a[B q1 + q2] and the twiddles W_N^(q2 k1); R2 (thread per
// (j, k1)) the B-point DFT over q2, the product with Bh, the B-point inverse
// DFT and the twiddles W_N^(-m1 k1) in registers; R4 (thread per (j, m1)) the
// A-point inverse DFT giving c[m1 + B m2], written to global memory at row
// g^(m1 + B m2).  Bound by its shared round trips and barriers, whatever p,
// where the product's arithmetic grows with p: AxisFFT::path takes it above
// the lengths at which the two cross.
#include "mpm_butterfly.cuh"
#include "mpm_chain.cuh"
#include "mpm_fft.h"

#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

namespace mpm {

namespace {

constexpr int kRaderMaxThreads = 384;
constexpr int kRaderLanes = 24;                 // threads per column
constexpr size_t kRaderSmem = 110 * 1024;       // two CTAs per SM (228 KB per SM)

template <typename R, int CW, bool INV, int CLS>
__global__ void __launch_bounds__(kRaderMaxThreads) k_rader(cplx<R>* __restrict__ data, const cplx<R>* __restrict__ tw,
                                                            const cplx<R>* __restrict__ rtab,
                                                            const int* __restrict__ rperm, int r1, int p, int A,
                                                            int B, size_t es, int ncols, size_t os, int ngroups) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = r1 * p;
    const int N = p - 1;
    const int L = blockDim.x / CW;
    cplx<R>* S = reinterpret_cast<cplx<R>*>(smem_raw);   // [n][CW] pass-1 output
    cplx<R>* Tt = S + size_t(n) * CW;                      // [r1 * N][CW] Rader work rows
    cplx<R>* T = Tt + size_t(r1) * N * CW;                 // [n] line twiddles
    cplx<R>* WN = T + n;                                   // [N] W_N^t
    cplx<R>* Bh = WN + N;                                  // [N] this direction's Bh
    int* pin = reinterpret_cast<int*>(Bh + N);             // [N] g^-q
    int* pout = pin + N;                                   // [N] g^m
    const int o = blockIdx.x / ngroups;
    const int g = blockIdx.x - o * ngroups;
    const int c = threadIdx.x & (CW - 1);
    const int lane = threadIdx.x / CW;
    const int c0 = g * CW;
    const bool live = c0 + c < ncols;
    cplx<R>* line = data + size_t(o) * os + c0 + c;
    chain_enter();
    for (int t = threadIdx.x; t < n; t += blockDim.x) {
        cplx<R> w = tw[t];
        if (INV) w.y = -w.y;
        T[t] = w;
    }
    for (int t = threadIdx.x; t < N; t += blockDim.x) {
        WN[t] = rtab[t];
        Bh[t] = rtab[(INV ? 2 : 1) * N + t];
        pin[t] = rperm[t];
        pout[t] = rperm[N + t];
    }
    __syncthreads();
    // pass 1: radix r1, global -> shared with pass 2's twiddles applied
    radix_dispatch<CLS>(r1, [&](auto rc) {
        constexpr int RAD = decltype(rc)::value;
#pragma unroll 2
        for (int j1 = lane; j1 < p; j1 += L) {
            cplx<R> x[RAD];
#pragma unroll
            for (int q = 0; q < RAD; ++q) x[q] = live ? line[size_t(j1 + q * p) * es] : mk<R>(R(0), R(0));
            dft_small<R, INV, RAD>(x);
            S[(j1 * RAD) * CW + c] = x[0];
#pragma unroll
            for (int p1 = 1; p1 < RAD; ++p1) S[(j1 * RAD + p1) * CW + c] = x[p1] * T[j1 * p1];
        }
    });
    __syncthreads();
    // R1: A-point DFTs over q1 of a[B q1 + q2], twiddled by W_N^(q2 k1)
    radix_dispatch<CLS>(A, [&](auto rc) {
        constexpr int RA = decltype(rc)::value;
        for (int u = lane; u < r1 * B; u += L) {
            const int q2 = u / r1;
            const int j = u - q2 * r1;
            cplx<R> z[RA];
#pragma unroll
            for (int q1 = 0; q1 < RA; ++q1) z[q1] = S[(j + pin[B * q1 + q2] * r1) * CW + c];
            dft_small<R, false, RA>(z);
            cplx<R>* trow = Tt + (size_t(j) * N + q2 * RA) * CW + c;
            trow[0] = z[0];
#pragma unroll
            for (int k1 = 1; k1 < RA; ++k1) trow[k1 * CW] = q2 ? z[k1] * WN[q2 * k1] : z[k1];
        }
    });
    __syncthreads();
    // R2: B-point DFT over q2 (-> DFT_N(a) at k1 + A k2), times Bh, B-point
    // inverse DFT over k2, twiddles W_N^(-m1 k1); the thread rewrites the
    // same Tt slots it read
    radix_dispatch<CLS>(B, [&](auto rc) {
        constexpr int RB = decltype(rc)::value;
        for (int u = lane; u < r1 * A; u += L) {
            const int k1 = u / r1;
            const int j = u - k1 * r1;
            cplx<R>* tcol = Tt + (size_t(j) * N + k1) * CW + c;
            cplx<R> v[RB];
#pragma unroll
            for (int q2 = 0; q2 < RB; ++q2) v[q2] = tcol[q2 * A * CW];
            dft_small<R, false, RB>(v);
            if (k1 == 0 && live) {
                const cplx<R> x0 = S[j * CW + c];
                line[size_t(j) * es] = x0 + v[0];   // y[0] = x[0] + sum a
            }
#pragma unroll
            for (int k2 = 0; k2 < RB; ++k2) v[k2] = v[k2] * Bh[k1 + A * k2];
            dft_small<R, true, RB>(v);
            tcol[0] = v[0];
#pragma unroll
            for (int m1 = 1; m1 < RB; ++m1) {
                cplx<R> w = WN[m1 * k1];
                w.y = -w.y;
                tcol[m1 * A * CW] = k1 ? v[m1] * w : v[m1];
            }
        }
    });
    __syncthreads();
    // R4: A-point inverse DFT over k1 -> c[m1 + B m2]; y[g^m] = x[0] + c[m]
    radix_dispatch<CLS>(A, [&](auto rc) {
        constexpr int RA = decltype(rc)::value;
        for (int u = lane; u < r1 * B; u += L) {
            const int m1 = u / r1;
            const int j = u - m1 * r1;
            const cplx<R>* trow = Tt + (size_t(j) * N + m1 * RA) * CW + c;
            cplx<R> d[RA];
#pragma unroll
            for (int k1 = 0; k1 < RA; ++k1) d[k1] = trow[k1 * CW];
            dft_small<R, true, RA>(d);
            if (!live) continue;
            const cplx<R> x0 = S[j * CW + c];
#pragma unroll
            for (int m2 = 0; m2 < RA; ++m2) line[size_t(pout[m1 + B * m2] * r1 + j) * es] = x0 + d[m2];
        }
    });
}

int rader_class(int r) { return r <= 8 ? 8 : (r <= 12 ? 12 : 16); }

size_t rader_smem(int n, int r1, int N, int cw, size_t elem) {
    return (size_t(n) * cw + size_t(r1) * N * cw + n + 2 * size_t(N)) * elem + 2 * sizeof(int) * N;
}

// smallest primitive root of the prime p
int primitive_root(int p) {
    for (int g = 2; g < p; ++g) {
        int order = 1;
        for (long long v = g; v != 1; v = v * g % p) ++order;
        if (order == p - 1) return g;
    }
    return 0;
}

}  // namespace

void RaderDFT::init(int n, int r1, int p, int A, int B) {
    n_ = 0;
    if (!A || p < 3 || rader_smem(n, r1, p - 1, 4, sizeof(double2)) > kRaderSmem) return;
    const int N = p - 1, g = primitive_root(p);
    std::vector<int> perm(2 * N);
    std::vector<int> gp(N);   // g^s mod p
    long long v = 1;
    for (int t = 0; t < N; ++t, v = v * g % p) gp[t] = int(v);
    for (int q = 0; q < N; ++q) perm[q] = gp[(N - q) % N];   // a_q = x[g^-q]
    for (int m = 0; m < N; ++m) perm[N + m] = gp[m];         // y[g^m]
    // (angles and sums in more than 64 bits: rounded ones cost the fp64
    // transform a third of its rms error)
    using lc = std::complex<long double>;
    auto roots = [](int m) {
        std::vector<lc> w(m);
        for (int t = 0; t < m; ++t) w[t] = std::polar(1.0L, -2.0L * kPiL * t / m);
        return w;
    };
    const std::vector<lc> wn = roots(N), wp = roots(p);
    std::vector<double2> t64(3 * size_t(N));
    auto d2 = [](lc z) { return make_double2(double(z.real()), double(z.imag())); };
    for (int k = 0; k < N; ++k) {
        t64[k] = d2(wn[k]);
        // Bh = DFT_N(b) / N, b_s = W_p^(g^s) (forward) or its conjugate (inverse)
        lc f = 0, i = 0;
        for (int t = 0; t < N; ++t) {
            const lc e = wn[size_t(t) * k % N];
            f += wp[gp[t]] * e;
            i += std::conj(wp[gp[t]]) * e;
        }
        t64[N + k] = d2(f / (long double)N);
        t64[2 * N + k] = d2(i / (long double)N);
    }
    std::vector<float2> t32(t64.size());
    for (size_t k = 0; k < t64.size(); ++k) t32[k] = make_float2(float(t64[k].x), float(t64[k].y));
    t64_.ensure(sizeof(double2) * t64.size());
    t32_.ensure(sizeof(float2) * t32.size());
    perm_.ensure(sizeof(int) * perm.size());
    upload(t64_.p, t64.data(), sizeof(double2) * t64.size());
    upload(t32_.p, t32.data(), sizeof(float2) * t32.size());
    upload(perm_.p, perm.data(), sizeof(int) * perm.size());
    n_ = n; r1_ = r1; p_ = p; a_ = A; b_ = B;
}

template <typename R>
void RaderDFT::run(cplx<R>* data, const cplx<R>* tw, size_t es, int ncols, size_t os, int nouter, bool inverse,
                   cudaStream_t s) const {
    const int N = p_ - 1, cls = rader_class(std::max(r1_, a_));
    // wide butterfly classes hold more registers: smaller CTAs
    int cw = cls > 8 ? 8 : 16;
    while (cw > 4 && (cw * kRaderLanes > (sizeof(R) == 8 ? 192 : kRaderMaxThreads) ||
                      rader_smem(n_, r1_, N, cw, sizeof(cplx<R>)) > kRaderSmem))
        cw /= 2;
    const size_t shm = rader_smem(n_, r1_, N, cw, sizeof(cplx<R>));
    const int ngroups = (ncols + cw - 1) / cw;
    const cplx<R>* rt = sizeof(R) == 4 ? reinterpret_cast<const cplx<R>*>(t32_.p)
                                       : reinterpret_cast<const cplx<R>*>(t64_.p);
    auto go = [&](auto kern) {
        set_smem_limit(kern, shm);
        launch_chained(kern, nouter * ngroups, cw * kRaderLanes, shm, s, data, tw, rt, perm_.as<int>(), r1_, p_, a_,
                       b_, es, ncols, os, ngroups);
    };
    auto width = [&](auto invc, auto clsc) {
        constexpr bool INV = decltype(invc)::value;
        constexpr int CLS = decltype(clsc)::value;
        if (cw == 16) go(k_rader<R, 16, INV, CLS>);
        else if (cw == 8) go(k_rader<R, 8, INV, CLS>);
        else go(k_rader<R, 4, INV, CLS>);
    };
    auto dir = [&](auto invc) {
        if (cls == 8) width(invc, std::integral_constant<int, 8>{});
        else if (cls == 12) width(invc, std::integral_constant<int, 12>{});
        else width(invc, std::integral_constant<int, 16>{});
    };
    if (inverse) dir(std::true_type{});
    else dir(std::false_type{});
}

template void RaderDFT::run<float>(float2*, const float2*, size_t, int, size_t, int, bool, cudaStream_t) const;
template void RaderDFT::run<double>(double2*, const double2*, size_t, int, size_t, int, bool, cudaStream_t) const;

}  // namespace mpm
