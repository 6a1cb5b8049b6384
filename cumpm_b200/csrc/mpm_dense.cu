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
// m real FMAs per element.  A thread holds A and B (BLK: A or B) of eight p and
// two columns (fp64: one) in registers, so a step over q costs 64 (32) FMAs
// against 8 (4) shared loads: at one FMA per lane and clock an element of
// m = 109 costs 3 ps of this GPU, against the 2.5 ps that its trip through HBM
// takes, and m = 53 is bound by that trip.  (Packed fp32 pairs, fma.rn.f32x2,
// halve the FMA instructions but took more to arrange their operands: slower.)
// The alternative for primes, Rader's convolution (mpm_rader.cu), needs a
// quarter of the arithmetic but three more shared round trips and gathers by
// g^q: 736 us for a 109-point pass of 497 MB (48 fp32 columns) that takes 515
// here; see AxisFFT::path for where it is the faster one.
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

constexpr int kChunk = 2 * kPC;   // eight pairs' table entries: cosines, sines

// where row q - 1's entries of chunk ch begin (s = 0: cosines, 1: sines).  In
// blocks (BLK below) a warp reads both of one chunk, else one of up to four
// chunks: what it reads lies side by side and meets no bank twice (366 points,
// 90 columns, fp64: 54 us with a chunk's sines behind its cosines, 42 so)
template <bool BLK>
__host__ __device__ constexpr int tab_at(int nch, int ch, int s) {
    return BLK ? ch * kChunk + s * kPC : (s * nch + ch) * kPC;
}

template <typename R> __host__ __device__ constexpr int dense_ct() { return sizeof(R) == 4 ? 2 : 1; }   // columns per thread

template <typename R>
struct DenseArgs {
    cplx<R>* data;
    const cplx<R>* tw;    // W_n^t, t < n
    const R* tab;         // [H] rows of cos, sin of 2 pi p q / m (tab_at)
    int n, r1, m, H, nch;
    size_t es, os;
    int ncols, ntiles, cwl, inv;
    long long ntot;
    const R* sc;          // SCALED: output element e of line o, column c times sc[(e nouter + o) sz + c / sb]
    size_t estep;         // nouter * sz
    int sz, sb;
};

// BLK: bits of a thread's number within its work items: the low lhb (at most
// four) bits of its columns, the half (A or B), the rest of the columns.
struct ItemBits {
    int lgh, lhb;     // log2 of the columns per thread row, of those beside one another in a warp
    __device__ __forceinline__ explicit ItemBits(int cwl) : lgh(cwl - 1), lhb(lgh < 4 ? lgh : 4) {}
    __device__ __forceinline__ bool second(int u) const { return (u >> lhb) & 1; }
    // its t-th column in the tile (a B lane has them in the other order: of the
    // halves of a row that each kind reads, no bank twice)
    __device__ __forceinline__ int column(int u, int t) const {
        return ((u & ((1 << lhb) - 1)) | (((u >> (lhb + 1)) & ((1 << (lgh - lhb)) - 1)) << lhb)) +
               ((second(u) ? 1 - t : t) << lgh);
    }
};
template <typename R, bool BLK>
__device__ __forceinline__ int column_of(int cwl, int u, int t) {
    if constexpr (BLK) return ItemBits(cwl).column(u, t);
    const int half = (1 << cwl) / dense_ct<R>();
    return (u & (half - 1)) + t * half;
}

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

// One half of a blocked work item: x_0 + A_p (tab the cosines, S the sums x_q +
// x_(m-q), o = x_0) or -i B_p (the sines, S the differences times -i, o = 0)
// above for p = p0 .. p0 + 7 and the columns S, S + cs, added to o; rows of S
// and tab are rs and ts apart.  Sums of some 20 terms that are then added up:
// one running sum over m / 2 terms had up to 2.4 times the largest error of
// transforms in short radices (241 points) and 1.4 times their rms error; so
// both are 0.5 to 0.9 and 0.4 to 1.1 of theirs at the primes from 53 to 257.
constexpr int kSumBlock = 20;
// Shorter products are summed at once: up to 47 points the largest error was no
// larger than that of short radices either, and the split of the work items
// costs more (43 points, 46 MB: 37 us, 42 in blocks; 53 points, 229 MB: 87 and
// 92 us, but with 1.2 times the largest error).
constexpr int kPlainTerms = 24;
template <typename R> __host__ __device__ constexpr bool blocked(int H) { return sizeof(R) == 4 && H > kPlainTerms; }

__device__ __forceinline__ void dense_sums(const float2* S, int rs, int cs, int H, const float* tab, int ts,
                                           float2 (&o)[2][kPC]) {
    const float2* S1 = S + cs;
    const int len = H / ((H + kSumBlock - 1) / kSumBlock) + 1;    // blocks of about the same length
#pragma unroll 1
    for (int q = 0; q < H; q += len) {
        const int n = min(len, H - q);
        float2 a[2][kPC];
        auto term = [&](auto first) {
            float w[kPC];
            load8(tab, w);
            const float2 x[2] = {*S, *S1};
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int k = 0; k < kPC; ++k) {
                    if constexpr (decltype(first)::value) a[t][k] = x[t] * w[k];
                    else fma_rc(a[t][k], w[k], x[t]);
                }
            S += rs;
            S1 += rs;
            tab += ts;
        };
        term(std::true_type{});
// (unrolled by 3, 4 and 5: 515, 534 and 540 us for the 109-point pass)
#pragma unroll 3
        for (int e = 1; e < n; ++e) term(std::false_type{});
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int k = 0; k < kPC; ++k) o[t][k] += a[t][k];
    }
}

// The m-point DFTs of every sub-line p1 < r1 of the tile S ([r1][m][CW]; BLK:
// of each sub-line x_0, then x_q + x_(m-q) at q <= m / 2, -i (x_q - x_(m-q)) at
// m - q); put(t, p1, output index, value) takes each output once, t the
// thread's column (column_of).  (The block is a multiple of CW threads: a
// thread's columns, and its half, are the same in every round.)
//
// BLK: a work item is eight output pairs of two columns, its A and its B in
// two lanes of a warp (so that the sums and block sums of one of them fit in a
// thread's registers): they exchange their sums, and the A lane puts y_p, the
// B lane y_(m-p).
template <typename Put>
__device__ __forceinline__ void dense_pass(const float2* S, const DenseArgs<float>& a, const float* tab, bool inv,
                                           Put&& put, std::true_type) {
    const int CW = 1 << a.cwl, half = CW / 2;
    const ItemBits ib(a.cwl);
    const bool second = ib.second(threadIdx.x);
    const float sg = second ? -1.0f : 1.0f;
    const int items = (a.r1 * a.nch) << a.cwl;
    for (int u0 = 0; u0 < items; u0 += blockDim.x) {
        const int u = u0 + threadIdx.x;
        const bool act = u < items;
        const int w = act ? u >> a.cwl : 0;
        const int p1 = w / a.nch, ch = w - p1 * a.nch, p0 = ch * kPC;
        const float2* Sp = S + p1 * a.m * CW;
        float2 o[2][kPC];
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            const float2 x0 = second ? make_float2(0.0f, 0.0f) : Sp[ib.column(threadIdx.x, t)];
#pragma unroll
            for (int k = 0; k < kPC; ++k) o[t][k] = x0;
        }
        if (act)
            dense_sums(Sp + (second ? a.m - 1 : 1) * CW + ib.column(threadIdx.x, 0), second ? -CW : CW,
                       second ? -half : half, a.H, tab + tab_at<true>(a.nch, ch, second), a.nch * kChunk, o);
        __syncwarp();
#pragma unroll
        for (int t = 0; t < 2; ++t) {
#pragma unroll
            for (int k = 0; k < kPC; ++k) {
                const int p = p0 + k;
                // (1 - t: the other lane's number of this column)
                const float2 v = make_float2(__shfl_xor_sync(0xffffffffu, o[1 - t][k].x, 1 << ib.lhb),
                                             __shfl_xor_sync(0xffffffffu, o[1 - t][k].y, 1 << ib.lhb));
                const int pr = p == 0 ? 0 : a.m - p;     // the mirrored output (itself for p = 0 and p = m / 2)
                if (!act || p > a.H || (second && pr == p)) continue;
                // y_p = (x_0 + A) + (-i B), y_(m-p) = (x_0 + A) - (-i B)
                put(t, p1, inv == second ? p : pr, make_float2(fmaf(sg, o[t][k].x, v.x), fmaf(sg, o[t][k].y, v.y)));
            }
        }
    }
}

// One running sum: a work item is eight output pairs of the columns of
// dense_ct, A and B together.  fp64 (rms error 0.3 to 0.5 of that of transforms
// in short radices whose twiddles come from angles rounded to 64 bits), and fp32
// products of at most kPlainTerms terms.
template <typename R, typename Put>
__device__ __forceinline__ void dense_pass(const cplx<R>* S, const DenseArgs<R>& a, const R* tab, bool inv, Put&& put,
                                           std::false_type) {
    constexpr int CT = dense_ct<R>();
    const int CW = 1 << a.cwl, half = CW / CT, lgh = a.cwl - (CT == 2 ? 1 : 0);
    const int items = (a.r1 * a.nch) << lgh;
    const int sines = tab_at<false>(a.nch, 0, 1);
    for (int u = threadIdx.x; u < items; u += blockDim.x) {
        const int w = u >> lgh;
        const int p1 = w / a.nch, ch = w - p1 * a.nch, p0 = ch * kPC;
        const cplx<R>* Sp = S + p1 * a.m * CW + (u & (half - 1));
        cplx<R> A[CT][kPC], B[CT][kPC];
#pragma unroll
        for (int t = 0; t < CT; ++t)
#pragma unroll
            for (int k = 0; k < kPC; ++k) A[t][k] = B[t][k] = mk<R>(R(0), R(0));
        const cplx<R>* lo = Sp + CW;
        const cplx<R>* hi = Sp + (a.m - 1) * CW;
        const R* tq = tab + tab_at<false>(a.nch, ch, 0);
#pragma unroll 1
        for (int q = 1; q <= a.H; ++q, lo += CW, hi -= CW, tq += a.nch * kChunk) {
            cplx<R> x[CT], y[CT];
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                x[t] = lo[t * half] + hi[t * half];
                y[t] = lo[t * half] - hi[t * half];
            }
            R v[kPC];
            load8(tq, v);
#pragma unroll
            for (int t = 0; t < CT; ++t)
#pragma unroll
                for (int k = 0; k < kPC; ++k) fma_rc(A[t][k], v[k], x[t]);
            load8(tq + sines, v);
#pragma unroll
            for (int t = 0; t < CT; ++t)
#pragma unroll
                for (int k = 0; k < kPC; ++k) fma_rc(B[t][k], v[k], y[t]);
        }
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            const cplx<R> x0 = Sp[t * half];
#pragma unroll
            for (int k = 0; k < kPC; ++k) {
                const int p = p0 + k;
                if (p > a.H) continue;
                const cplx<R> e = x0 + A[t][k], f = B[t][k];
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
// launches take 1189.)
template <typename R, bool SCALED, bool TS, int KIND, bool BLK>
__global__ void __launch_bounds__(kDenseMaxThreads, dense_ctas<R>(KIND == 2)) k_dense(DenseArgs<R> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int CW = 1 << a.cwl;
    cplx<R>* S = reinterpret_cast<cplx<R>*>(smem_raw);                   // [n][CW]
    R* tabS = reinterpret_cast<R*>(S + size_t(a.n) * CW);
    cplx<R>* T = reinterpret_cast<cplx<R>*>(tabS + (TS ? imax(1, a.H) * a.nch * kChunk : 0));   // [n], r1 > 1
    const int c = threadIdx.x & (CW - 1);
    const int lane = threadIdx.x >> a.cwl, lanes = blockDim.x >> a.cwl;
    const bool inv = a.inv != 0;
    // (the tables are older than any launch of this stream)
    if (TS && KIND != 2) {
        const int nt = imax(1, a.H) * a.nch * kChunk * int(sizeof(R)) / 16;
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
            if (BLK && KIND == 0) {   // a thread copies the rows that it pairs
                for (int e = lane; e <= a.H; e += lanes) {
                    copy_async<R>(S + e * CW + c, line + size_t(e) * es, live);
                    if (e && 2 * e < a.m) copy_async<R>(S + (a.m - e) * CW + c, line + size_t(a.m - e) * es, live);
                }
            } else {
                for (int e = lane; e < a.n; e += lanes) copy_async<R>(S + e * CW + c, line + size_t(e) * es, live);
            }
        }
        // a successor that is scheduled earlier takes slots from work on other
        // streams for as long as this CTA's tiles last
        if (tile + gridDim.x >= a.ntiles) chain_release();
        copy_async_wait();
        // rows q and m - q of a column: their sum, and -i times their difference
        auto fold = [&](cplx<R>* col, int q) {
            cplx<R>&u = col[q * CW], &v = col[(a.m - q) * CW];
            const cplx<R> x = u, y = v;
            u = x + y;
            v = mk<R>(x.y - y.y, y.x - x.x);
        };
        if constexpr (BLK && KIND == 0)
            for (int e = lane ? lane : lanes; 2 * e < a.m; e += lanes) fold(S + c, e);
        __syncthreads();
        if constexpr (KIND != 0) {
            // radix-r1 butterflies over x[j + q m], times W_n^(j p), in place:
            // S[p][j] (BLK: of the pair j, m - j the sum and the difference)
            radix_dispatch<16>(a.r1, [&](auto rc) {
                constexpr int RAD = decltype(rc)::value;
                if constexpr (RAD > 1) {
                    auto butterfly = [&](int j) {
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
                    };
                    if constexpr (!BLK) {
                        for (int j = lane; j < a.m; j += lanes) butterfly(j);
                    } else {
                        for (int j = lane; j <= a.H; j += lanes) {
                            const bool pair = j && 2 * j < a.m;
#pragma unroll 1
                            for (int h = 0; h <= int(pair); ++h) butterfly(h ? a.m - j : j);
                            if (pair) {
#pragma unroll 2
                                for (int p = 0; p < RAD; ++p) fold(S + p * a.m * CW + c, j);
                            }
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
            cplx<R>* oline[dense_ct<R>()];
            bool olive[dense_ct<R>()];
            const R* osc[dense_ct<R>()];
#pragma unroll
            for (int t = 0; t < dense_ct<R>(); ++t) {
                const long long g = f0 + column_of<R, BLK>(a.cwl, threadIdx.x, t);
                olive[t] = g < a.ntot;
                int go = 0, gc = 0;
                if (olive[t]) line_of(g, a.ntot, a.ncols, go, gc);
                oline[t] = a.data + size_t(go) * a.os + gc;
                osc[t] = SCALED ? a.sc + size_t(go) * a.sz + gc / a.sb : nullptr;
            }
            dense_pass(S, a, tab, inv, [&](int t, int p1, int p, cplx<R> v) {
                if (!olive[t]) return;
                const int e = p1 + a.r1 * p;
                if constexpr (SCALED) v = v * osc[t][size_t(e) * a.estep];
                oline[t][size_t(e) * a.es] = v;
            }, std::bool_constant<BLK>{});
        }
        __syncthreads();   // the tile's buffer is free
    }
}

constexpr size_t kDenseSmemMax = 220 * 1024;

}  // namespace

int sm_count() {
    static const int sms = [] {
        int d = 0, v = 148;
        if (cudaGetDevice(&d) != cudaSuccess || cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, d) != cudaSuccess)
            v = 148;
        return v;
    }();
    return sms;
}

// Tables longer than this stay in global memory (L1): m above 191, in fp64 127.
constexpr size_t kDenseTableSmem = 72 * 1024;

void DenseDFT::init(int n, int r1) {
    r1_ = r1;
    m_ = r1 ? n / r1 : 0;
    n_ = n;
    if (!r1) return;
    H_ = m_ / 2;
    nch_ = (H_ + 1 + kPC - 1) / kPC;
    std::vector<double2> w(m_);
    for (int j = 0; j < m_; ++j) w[j] = unit_root(j, m_);
    auto fill = [&](auto zero, DevBuf& buf) {
        using R = decltype(zero);
        const bool blk = blocked<R>(H_);
        auto at = [&](int ch, int s) { return blk ? tab_at<true>(nch_, ch, s) : tab_at<false>(nch_, ch, s); };
        std::vector<R> t(size_t(std::max(1, H_)) * nch_ * kChunk, zero);
        for (int q = 1; q <= H_; ++q)
            for (int p = 0; p <= H_; ++p) {
                const size_t j = size_t(p) * q % m_;
                R* e = t.data() + size_t(q - 1) * nch_ * kChunk + p % kPC;
                // (without blocks the middle row of an even m meets itself as a pair)
                e[at(p / kPC, 0)] = R(!blk && 2 * q == m_ ? 0.5 * w[j].x : w[j].x);
                e[at(p / kPC, 1)] = 2 * q == m_ ? zero : R(w[j].y);
            }
        buf.ensure(sizeof(R) * t.size());
        upload(buf.p, t.data(), sizeof(R) * t.size());
    };
    fill(0.0, t64_);
    fill(0.0f, t32_);
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
    DenseArgs<R> a{};
    a.data = data;
    a.tw = tw;
    a.tab = sizeof(R) == 4 ? reinterpret_cast<const R*>(t32_.p) : reinterpret_cast<const R*>(t64_.p);
    a.n = n_; a.r1 = r1_; a.m = m_; a.H = H_; a.nch = nch_;
    a.es = es; a.os = os; a.ncols = ncols; a.inv = inverse;
    a.ntot = (long long)nouter * ncols;
    a.sc = scale;
    a.estep = size_t(nouter) * sz;
    a.sz = sz;
    a.sb = sb;
    const size_t tabb = sizeof(R) * size_t(std::max(1, H_)) * nch_ * kChunk;
    const size_t twb = r1_ > 1 ? sizeof(cplx<R>) * size_t(n_) : 0;
    const size_t per_col = size_t(n_) * sizeof(cplx<R>);
    const bool radix2 = r1_ > 1 && m_ <= 16;       // no table
    const bool ts = !radix2 && tabb <= kDenseTableSmem && (per_col << 2) + tabb + twb <= kDenseSmemMax;
    auto smem = [&](int cwl) { return (per_col << cwl) + (ts ? tabb : 0) + twb; };
    const bool blk = blocked<R>(H_) && !radix2;
    // threads: a work item (in blocks: the A or B of one) each
    auto items = [&](int cwl) { return (a.r1 * a.nch << cwl) / (blk ? 1 : dense_ct<R>()); };
    // columns per tile: 64 (fp64: 32), so that a warp's lanes are the columns
    // of one p range and read its table entries as one word; fewer while the
    // SM would not hold `ctas` CTAs, whose copies and products overlap, or the
    // tiles would not cover two per SM (few columns in all)
    auto widest = [&](int ctas) {
        int l = sizeof(R) == 4 ? 6 : 5;
        while (l > 2 && (smem(l) > size_t(224 * 1024 / ctas) || (a.ntot >> l) < 2 * sm_count())) --l;
        return l;
    };
    int maxthr = kDenseMaxThreads, cwl = widest(dense_ctas<R>(radix2));
    const int regs = 256 / dense_ctas<R>(radix2);
    // four CTAs of 128 threads instead of two of 256 where their tiles, of
    // eight columns at least, are no smaller than the tables beside them
    // (before the inner loop was unrolled by three: 109 points and 48 columns
    // 558 us against 597, 366 points and 90 columns 34 against 37; with four
    // columns per tile 151 points took 145 against 93)
    const int l4 = widest(4);
    if (blk && l4 > 2 && smem(l4) <= 56 * 1024 && (per_col << l4) >= (ts ? tabb : 0)) {
        cwl = l4;
        maxthr = 128;
    }
    const size_t shm = smem(cwl);
    if (shm > kDenseSmemMax) throw std::runtime_error("FFT line does not fit in shared memory");
    a.cwl = cwl;
    a.ntiles = int((a.ntot + (1ll << cwl) - 1) >> cwl);
    // threads: the work items in equal rounds, a whole number of column rows
    const int it = radix2 ? r1_ << cwl : items(cwl), rounds = (it + maxthr - 1) / maxthr;
    const int unit = std::max(32, 1 << cwl);
    int nt = ((it + rounds - 1) / rounds + unit - 1) / unit * unit;
    nt = std::min(maxthr, std::max(nt, 128));   // the copies and radix pass use them all
    // resident CTAs; each stays for its share of the tiles
    const int per_sm = std::max(1, std::min({int(227 * 1024 / (shm + 1024)), 65536 / (regs * nt), 16}));
    const int grid = std::min(a.ntiles, per_sm * sm_count());
    auto go = [&](auto kern) {
        set_smem_limit(kern, shm);
        launch_chained(kern, grid, nt, shm, s, a);
    };
    auto pick = [&](auto scaled, auto blkc) {
        constexpr bool SC = decltype(scaled)::value, BLK = decltype(blkc)::value;
        if (r1_ == 1) ts ? go(k_dense<R, SC, true, 0, BLK>) : go(k_dense<R, SC, false, 0, BLK>);
        else ts ? go(k_dense<R, SC, true, 1, BLK>) : go(k_dense<R, SC, false, 1, BLK>);
    };
    auto kind = [&](auto scaled) {
        if (radix2) {
            go(k_dense<R, decltype(scaled)::value, false, 2, false>);
            return;
        }
        if constexpr (sizeof(R) == 4) {
            if (blk) {
                pick(scaled, std::true_type{});
                return;
            }
        }
        pick(scaled, std::false_type{});
    };
    if (scale) kind(std::true_type{});
    else kind(std::false_type{});
}

template void DenseDFT::run<float>(float2*, const float2*, size_t, int, size_t, int, int, const float*, int, int,
                                   cudaStream_t) const;
template void DenseDFT::run<double>(double2*, const double2*, size_t, int, size_t, int, int, const double*, int, int,
                                    cudaStream_t) const;

}  // namespace mpm
