// Line transform n = r1 * m with an in-register radix r1 <= 16 and the m-point
// DFTs evaluated as register-tiled products with their cosine and sine tables
// (AxisFFT::run_dense; see mpm_fft.h).
//
// The grid lengths follow from the Ewald rule, so primes (109, 53, 61) are as
// common as smooth lengths.  An m-point DFT with m odd or even is the pair of
// real products, over q = 1 .. H = m / 2 and p = 0 .. H,
//   A_p = sum_q (x_q + x_(m-q)) cos(2 pi p q / m),
//   B_p = sum_q (x_q - x_(m-q)) sin(2 pi p q / m),
//   y_p = x_0 + A_p - i B_p,  y_(m-p) = x_0 + A_p + i B_p,
// m real FMAs per element.  A thread holds eight p of two fp32 columns (one
// fp64 column) in registers, so a step over q costs 64 (32) FMAs against 8
// (10) shared loads: at one FMA per lane and clock an element of m = 109 costs 3 ps
// of this GPU, against the 2.5 ps that its trip through HBM takes, and m = 53
// is bound by that trip.  (Packed fp32 pairs, fma.rn.f32x2, halve the FMA
// instructions but took more to arrange their operands: slower.)  The
// alternative for primes, Rader's convolution through two (p-1)-point
// transforms, needs a quarter of the arithmetic but three more shared round
// trips and gathers by g^q: it ran at 12 ps per element where this kernel
// takes 8.9 (109^3 x 48 columns, fp32).
//
// Columns are enumerated over lines and columns together (f = line * ncols +
// column), so a transform of few columns per line (the z axis of a solve's
// three right-hand sides) still fills its tiles.
#include "mpm_butterfly.cuh"
#include "mpm_chain.cuh"
#include "mpm_fft.h"

#include <algorithm>
#include <cmath>
#include <vector>

namespace mpm {

namespace {

constexpr int kDenseMaxThreads = 256;
constexpr int kPC = 8;    // output pairs per thread
// CTAs per SM that the registers allow: the product's accumulators take 128 a
// thread, two fp32 butterflies half of them
template <typename R> __host__ __device__ constexpr int dense_ctas(bool radix2) { return radix2 && sizeof(R) == 4 ? 4 : 2; }

template <typename R> constexpr int dense_ct() { return sizeof(R) == 4 ? 2 : 1; }   // columns per thread

template <typename R>
struct DenseArgs {
    cplx<R>* data;
    const cplx<R>* tw;    // W_n^t, t < n
    const R* tab;         // [H][2][ld]: cos, sin of 2 pi p q / m (row q = m/2 of an even m holds halves)
    int n, r1, m, H, ld, nch;
    size_t es, os;
    int ncols, ntiles, cwl, inv;
    long long ntot;
    const R* sc;          // SCALED: output element e of line o, column c times sc[(e nouter + o) sz + c / sb]
    size_t estep;         // nouter * sz
    int sz, sb;
};

// One work item: the output pairs p0 .. p0 + 7 of the m-point DFT of CT
// columns whose inputs are S[q * CW + t * half]; A and B above per pair.
template <typename R, int CT> struct DenseAcc { cplx<R> a[CT][kPC], b[CT][kPC]; };

// eight table entries as 16-byte words
__device__ __forceinline__ void load8(const float* t, float (&v)[8]) {
    const float4 x = *reinterpret_cast<const float4*>(t), y = *reinterpret_cast<const float4*>(t + 4);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
}
__device__ __forceinline__ void load8(const double* t, double (&v)[8]) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double2 x = *reinterpret_cast<const double2*>(t + 2 * k);
        v[2 * k] = x.x;
        v[2 * k + 1] = x.y;
    }
}

template <typename R, int CT>
__device__ __forceinline__ void dense_dot(const cplx<R>* S, int CW, int half, int m, int H, const R* tab, int ld,
                                          DenseAcc<R, CT>& o) {
#pragma unroll
    for (int t = 0; t < CT; ++t)
#pragma unroll
        for (int k = 0; k < kPC; ++k) o.a[t][k] = o.b[t][k] = mk<R>(R(0), R(0));
    const cplx<R>* lo = S + CW;
    const cplx<R>* hi = S + (m - 1) * CW;
#pragma unroll 1
    for (int q = 1; q <= H; ++q, lo += CW, hi -= CW, tab += 2 * ld) {
        cplx<R> p[CT], d[CT];
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            const cplx<R> u = lo[t * half], v = hi[t * half];
            p[t] = u + v;
            d[t] = u - v;
        }
        R w[kPC];
        load8(tab, w);
#pragma unroll
        for (int t = 0; t < CT; ++t)
#pragma unroll
            for (int k = 0; k < kPC; ++k) fma_rc(o.a[t][k], w[k], p[t]);
        load8(tab + ld, w);
#pragma unroll
        for (int t = 0; t < CT; ++t)
#pragma unroll
            for (int k = 0; k < kPC; ++k) fma_rc(o.b[t][k], w[k], d[t]);
    }
}

// The m-point DFTs of every sub-line p1 < r1 of the tile S ([r1][m][CW]);
// put(t, p1, output index, value) takes each output once, t the thread's
// column (threadIdx mod half + t half).
template <typename R, typename Put>
__device__ __forceinline__ void dense_pass(const cplx<R>* S, const DenseArgs<R>& a, const R* tab, bool inv, Put&& put) {
    constexpr int CT = dense_ct<R>();
    const int CW = 1 << a.cwl, half = CW / CT;
    const int lgh = a.cwl - (CT == 2 ? 1 : 0);
    const int items = (a.r1 * a.nch) << lgh;
    for (int u = threadIdx.x; u < items; u += blockDim.x) {
        const int c = u & (half - 1);
        const int w = u >> lgh;
        const int p1 = w / a.nch, p0 = (w - p1 * a.nch) * kPC;
        const cplx<R>* Sp = S + p1 * a.m * CW + c;
        DenseAcc<R, CT> o;
        dense_dot<R, CT>(Sp, CW, half, a.m, a.H, tab + p0, a.ld, o);
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            const cplx<R> x0 = Sp[t * half];
#pragma unroll
            for (int k = 0; k < kPC; ++k) {
                const int p = p0 + k;
                if (p > a.H) continue;
                const cplx<R> e = x0 + o.a[t][k], f = o.b[t][k];
                const cplx<R> y = mk<R>(e.x + f.y, e.y - f.x), z = mk<R>(e.x - f.y, e.y + f.x);
                const int pr = p == 0 ? 0 : a.m - p;     // the mirrored output (itself for p = 0 and p = m / 2)
                put(t, p1, inv ? pr : p, y);
                if (pr != p) put(t, p1, inv ? p : pr, z);
            }
        }
    }
}

__device__ __forceinline__ int imax(int a, int b) { return a > b ? a : b; }

// line and column of flattened column f
__device__ __forceinline__ void line_of(long long f, long long ntot, int ncols, int& o, int& c) {
    if (ntot <= 0x7fffffffLL) {
        o = int(unsigned(f) / unsigned(ncols));
        c = int(unsigned(f) - unsigned(o) * unsigned(ncols));
    } else {
        o = int(f / ncols);
        c = int(f - (long long)o * ncols);
    }
}

// TS: the tables are staged in shared memory once per CTA, which then stays
// for several tiles.  KIND 0: r1 = 1; 1: r1 > 1; 2: m is an in-register radix
// too, and takes the product's place (84 = 12 * 7 points of 9 columns, 43 MB:
// 38 us with the product, 26).  A tile is copied in with all its loads in
// flight (cp.async; loads of four at a time spent two thirds of the kernel
// waiting), transformed in place by the radix pass, and read by the product
// whose outputs go straight to global memory; the SM's other CTAs compute
// meanwhile.  (Two buffers per CTA, the next tile copied in during this one's
// product, left half the warps: 601 us against 555 for a 109-point pass
// of 497 MB.  Forward, scale and inverse in one launch needs the outputs of a
// whole tile in registers or a second tile: 2010 us at 109 points where two
// launches take 1245.)
template <typename R, bool SCALED, bool TS, int KIND>
__global__ void __launch_bounds__(kDenseMaxThreads, dense_ctas<R>(KIND == 2)) k_dense(DenseArgs<R> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int CW = 1 << a.cwl;
    cplx<R>* S = reinterpret_cast<cplx<R>*>(smem_raw);                   // [n][CW]
    R* tabS = reinterpret_cast<R*>(S + size_t(a.n) * CW);
    cplx<R>* T = reinterpret_cast<cplx<R>*>(tabS + (TS ? imax(1, a.H) * 2 * a.ld : 0));   // [n], r1 > 1
    const int c = threadIdx.x & (CW - 1);
    const int lane = threadIdx.x >> a.cwl, lanes = blockDim.x >> a.cwl;
    constexpr int CT = dense_ct<R>();
    const int half = CW / CT;
    const bool inv = a.inv != 0;
    // (the tables are older than any launch of this stream)
    if (TS && KIND != 2) {
        const int nt = imax(1, a.H) * 2 * a.ld * int(sizeof(R)) / 16;
        const double2* g = reinterpret_cast<const double2*>(a.tab);
        for (int t = threadIdx.x; t < nt; t += blockDim.x) copy_async<double>(reinterpret_cast<double2*>(tabS) + t, g + t, true);
    }
    if (KIND != 0)
        for (int t = threadIdx.x; t < a.n; t += blockDim.x) copy_async<R>(T + t, a.tw + t, true);
    const R* tab = TS ? tabS : a.tab;
    chain_wait();
    for (int tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x) {
        const long long f0 = (long long)tile << a.cwl;
        {
            const bool live = f0 + c < a.ntot;       // dead columns: zeros, the address is a placeholder
            int o = 0, cc = 0;
            if (live) line_of(f0 + c, a.ntot, a.ncols, o, cc);
            const cplx<R>* line = a.data + size_t(o) * a.os + cc;
            const size_t es = live ? a.es : 0;
            for (int e = lane; e < a.n; e += lanes) copy_async<R>(S + e * CW + c, line + size_t(e) * es, live);
        }
        // a successor that is scheduled earlier takes slots from work on other
        // streams for as long as this CTA's tiles last
        if (tile + gridDim.x >= a.ntiles) chain_release();
        copy_async_wait();
        __syncthreads();
        if constexpr (KIND != 0) {
            // radix-r1 butterflies over x[j + q m], times W_n^(j p), in place: S[p][j]
            radix_dispatch<16>(a.r1, [&](auto rc) {
                constexpr int RAD = decltype(rc)::value;
                if constexpr (RAD > 1) {
                    for (int j = lane; j < a.m; j += lanes) {
                        cplx<R> x[RAD];
#pragma unroll
                        for (int q = 0; q < RAD; ++q) x[q] = S[(j + q * a.m) * CW + c];
                        dft_small<R, false, RAD>(x);
#pragma unroll
                        for (int k = 0; k < RAD; ++k) {
                            // the inverse butterfly is the forward one with its outputs mirrored
                            const int p = inv && k ? RAD - k : k;
                            cplx<R> w = T[j * p];
                            if (inv) w.y = -w.y;
                            S[(p * a.m + j) * CW + c] = k == 0 ? x[k] : x[k] * w;
                        }
                    }
                }
            });
            __syncthreads();
        }
        if constexpr (KIND == 2) {
            // radix-m butterflies over S[p1][j]: outputs p1 + r1 p (mirrored for the inverse)
            const bool live = f0 + c < a.ntot;
            int o = 0, cc = 0;
            if (live) line_of(f0 + c, a.ntot, a.ncols, o, cc);
            cplx<R>* line = a.data + size_t(o) * a.os + cc;
            const R* sc = SCALED ? a.sc + size_t(o) * a.sz + cc / a.sb : nullptr;
            if (live)
                radix_dispatch<16>(a.m, [&](auto rc) {
                    constexpr int RAD = decltype(rc)::value;
                    for (int p1 = lane; p1 < a.r1; p1 += lanes) {
                        cplx<R> x[RAD];
#pragma unroll
                        for (int q = 0; q < RAD; ++q) x[q] = S[(p1 * RAD + q) * CW + c];
                        dft_small<R, false, RAD>(x);
#pragma unroll
                        for (int k = 0; k < RAD; ++k) {
                            const int e = p1 + a.r1 * (inv && k ? RAD - k : k);
                            line[size_t(e) * a.es] = SCALED ? x[k] * sc[size_t(e) * a.estep] : x[k];
                        }
                    }
                });
        } else {
            // the columns of this thread's work items
            cplx<R>* oline[CT];
            bool olive[CT];
            const R* osc[CT];
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                const long long g = f0 + (threadIdx.x & (half - 1)) + t * half;
                olive[t] = g < a.ntot;
                int go = 0, gc = 0;
                if (olive[t]) line_of(g, a.ntot, a.ncols, go, gc);
                oline[t] = a.data + size_t(go) * a.os + gc;
                osc[t] = SCALED ? a.sc + size_t(go) * a.sz + gc / a.sb : nullptr;
            }
            dense_pass<R>(S, a, tab, inv, [&](int t, int p1, int p, cplx<R> v) {
                if (!olive[t]) return;
                const int e = p1 + a.r1 * p;
                if constexpr (SCALED) v = v * osc[t][size_t(e) * a.estep];
                oline[t][size_t(e) * a.es] = v;
            });
        }
        __syncthreads();   // the tile's buffer is free
    }
}

int sm_count() {
    static const int sms = [] {
        int d = 0, v = 148;
        if (cudaGetDevice(&d) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d) != cudaSuccess)
            v = 148;
        return v;
    }();
    return sms;
}

constexpr size_t kDenseSmemMax = 220 * 1024;

}  // namespace

// Tables longer than this stay in global memory (L1): m above 131.
constexpr size_t kDenseTableSmem = 72 * 1024;

void DenseDFT::init(int n, int r1) {
    r1_ = r1;
    m_ = r1 ? n / r1 : 0;
    n_ = n;
    if (!r1) return;
    H_ = m_ / 2;
    ld_ = (H_ + 1 + kPC - 1) / kPC * kPC;
    std::vector<double> t(size_t(std::max(1, H_)) * 2 * ld_, 0.0);
    for (int q = 1; q <= H_; ++q) {
        const double f = 2 * q == m_ ? 0.5 : 1.0;     // x_q + x_(m-q) counts the middle input twice
        for (int p = 0; p <= H_; ++p) {
            const double w = 2.0 * kPi * double((long long)p * q % m_) / m_;
            t[(size_t(q - 1) * 2) * ld_ + p] = f * std::cos(w);
            t[(size_t(q - 1) * 2 + 1) * ld_ + p] = 2 * q == m_ ? 0.0 : std::sin(w);
        }
    }
    std::vector<float> tf(t.begin(), t.end());
    t64_.ensure(sizeof(double) * t.size());
    t32_.ensure(sizeof(float) * tf.size());
    upload(t64_.p, t.data(), sizeof(double) * t.size());
    upload(t32_.p, tf.data(), sizeof(float) * tf.size());
}

bool DenseDFT::fits(bool fp64) const {
    const size_t elem = fp64 ? sizeof(double2) : sizeof(float2);
    return r1_ && elem * (size_t(n_) * 4 + (r1_ > 1 ? n_ : 0)) <= kDenseSmemMax;
}

template <typename R>
void DenseDFT::run(cplx<R>* data, const cplx<R>* tw, size_t es, int ncols, size_t os, int nouter, int mode,
                   const R* scale, int sz, int sb, cudaStream_t s) const {
    if (mode == 2) {
        launch<R>(data, tw, es, ncols, os, nouter, false, scale, sz, sb, s);
        launch<R>(data, tw, es, ncols, os, nouter, true, nullptr, 1, 1, s);
        return;
    }
    launch<R>(data, tw, es, ncols, os, nouter, mode == 1, nullptr, 1, 1, s);
}

template <typename R>
void DenseDFT::launch(cplx<R>* data, const cplx<R>* tw, size_t es, int ncols, size_t os, int nouter, bool inverse,
                      const R* scale, int sz, int sb, cudaStream_t s) const {
    constexpr int CT = dense_ct<R>();
    DenseArgs<R> a{};
    a.data = data;
    a.tw = tw;
    a.tab = sizeof(R) == 4 ? reinterpret_cast<const R*>(t32_.p) : reinterpret_cast<const R*>(t64_.p);
    a.n = n_; a.r1 = r1_; a.m = m_; a.H = H_; a.ld = ld_; a.nch = ld_ / kPC;
    a.es = es; a.os = os; a.ncols = ncols; a.inv = inverse;
    a.ntot = (long long)nouter * ncols;
    a.sc = scale;
    a.estep = size_t(nouter) * sz;
    a.sz = sz;
    a.sb = sb;
    const size_t tabb = sizeof(R) * size_t(std::max(1, H_)) * 2 * ld_;
    const size_t twb = r1_ > 1 ? sizeof(cplx<R>) * size_t(n_) : 0;
    const size_t per_col = size_t(n_) * sizeof(cplx<R>);
    const bool radix2 = r1_ > 1 && m_ <= 16;       // no table
    const bool ts = !radix2 && tabb <= kDenseTableSmem && (per_col << 2) + tabb + twb <= kDenseSmemMax;
    auto smem = [&](int cwl) { return (per_col << cwl) + (ts ? tabb : 0) + twb; };
    auto items = [&](int cwl) { return a.r1 * a.nch * ((1 << cwl) / CT); };
    // columns per tile: 64 (fp64: 32), so that a warp's lanes are the columns
    // of one p range and read its table entries as one word; fewer while the
    // SM would not hold two CTAs, whose copies and products overlap, or the
    // tiles would not cover two per SM (few columns in all)
    int cwl = sizeof(R) == 4 ? 6 : 5;
    const int regs = 256 / dense_ctas<R>(radix2);
    while (cwl > 2 && (smem(cwl) > size_t(224 * 1024 / dense_ctas<R>(radix2)) || (a.ntot >> cwl) < 2 * sm_count())) --cwl;
    const size_t shm = smem(cwl);
    if (shm > kDenseSmemMax) throw std::runtime_error("FFT line does not fit in shared memory");
    a.cwl = cwl;
    a.ntiles = int((a.ntot + (1ll << cwl) - 1) >> cwl);
    // threads: the work items in equal rounds, a whole number of column rows
    const int it = radix2 ? r1_ << cwl : items(cwl), rounds = (it + kDenseMaxThreads - 1) / kDenseMaxThreads;
    const int unit = std::max(32, 1 << cwl);
    int nt = ((it + rounds - 1) / rounds + unit - 1) / unit * unit;
    nt = std::min(kDenseMaxThreads, std::max(nt, 128));   // the copies and radix pass use them all
    // resident CTAs; each stays for its share of the tiles
    const int per_sm = std::max(1, std::min({int(227 * 1024 / (shm + 1024)), 65536 / (regs * nt), 16}));
    const int grid = std::min(a.ntiles, per_sm * sm_count());
    auto go = [&](auto kern) {
        set_smem_limit(kern, shm);
        launch_chained(kern, grid, nt, shm, s, a);
    };
    auto pick = [&](auto scaled) {
        constexpr bool SC = decltype(scaled)::value;
        if (radix2) go(k_dense<R, SC, false, 2>);
        else if (r1_ == 1) ts ? go(k_dense<R, SC, true, 0>) : go(k_dense<R, SC, false, 0>);
        else ts ? go(k_dense<R, SC, true, 1>) : go(k_dense<R, SC, false, 1>);
    };
    if (scale) pick(std::true_type{});
    else pick(std::false_type{});
}

template void DenseDFT::run<float>(float2*, const float2*, size_t, int, size_t, int, int, const float*, int, int,
                                   cudaStream_t) const;
template void DenseDFT::run<double>(double2*, const double2*, size_t, int, size_t, int, int, const double*, int, int,
                                    cudaStream_t) const;

}  // namespace mpm
