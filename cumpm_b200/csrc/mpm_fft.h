// Batched 1-D DFT along one axis of a grid whose batch index is innermost.
//
// The spectral-Ewald grids are stored [x][y][slot][b] with the right-hand
// sides innermost, so a transform along x or y sees, for every grid point,
// a contiguous row of independent columns.  Each CTA stages one line of a
// chunk of columns in shared memory and runs a mixed-radix Stockham
// autosort there (every radix pass computes each output as an r-term sum
// with table twiddles, so any prime factor works without Bluestein), then
// writes the line back in place.  Global loads and stores are row-coalesced.
// Unnormalised in both directions (the 1/V factor lives in the k-space
// scale, as in the reference's cuFFT use).
#pragma once

#include "mpm_common.cuh"

#include <vector>

namespace mpm {

constexpr int kFftMaxFactors = 16;

struct FftFactors {
    int n = 1;
    int nf = 0;
    int r[kFftMaxFactors] = {};
    // factors above 16 (streamed passes): offset and row length of their
    // W_r^(p q) table, rows q = 1..(r-1)/2, columns p = 1..(r-1)/2 (padded)
    int pt_off[kFftMaxFactors] = {};
    int pt_ld[kFftMaxFactors] = {};
    int pt_total = 0;     // entries of all tables together
};

// SMs of the first device used (the rules that share work between CTAs)
int sm_count();

// Line transform of n = r1 * m points by an in-register radix-r1 pass and
// m-point DFTs as products with their tables (mpm_dense.cu).  r1 = 0: off.
class DenseDFT {
public:
    void init(int n, int r1);     // (the caller waits for the uploads, uploads_done)
    // whether a tile of four columns fits in shared memory
    bool fits(bool fp64) const;
    int radix() const { return r1_; }
    int rest() const { return m_; }
    // as AxisFFT::run / run_scaled (mode 2: two launches); tw: W_n^t, t < n
    template <typename R>
    void run(cplx<R>* data, const cplx<R>* tw, size_t es, int ncols, size_t os, int nouter, int mode, const R* scale,
             int sz, int sb, cudaStream_t s) const;

private:
    template <typename R>
    void launch(cplx<R>* data, const cplx<R>* tw, size_t es, int ncols, size_t os, int nouter, bool inverse,
                const R* scale, int sz, int sb, cudaStream_t s) const;
    int n_ = 0, r1_ = 0, m_ = 0, H_ = 0, nch_ = 0;
    DevBuf t64_, t32_;   // cosines and sines of 2 pi p q / m, see mpm_dense.cu
};

// Line transform of n = r1 * p points, p a prime with p - 1 = A * B, by an
// in-register radix-r1 pass and Rader's convolution (mpm_rader.cu).
class RaderDFT {
public:
    void init(int n, int r1, int p, int A, int B);     // (likewise)
    // false: not set up (A = 0, or a tile does not fit in shared memory)
    bool usable() const { return n_ != 0; }
    // as AxisFFT::run
    template <typename R>
    void run(cplx<R>* data, const cplx<R>* tw, size_t es, int ncols, size_t os, int nouter, bool inverse,
             cudaStream_t s) const;

private:
    int n_ = 0, r1_ = 0, p_ = 0, a_ = 0, b_ = 0;
    DevBuf t64_, t32_;   // W_N^t, N = p - 1, then the forward and the inverse Bh
    DevBuf perm_;        // g^-q, then g^m
};

class AxisFFT {
public:
    void init(int n);
    int n() const { return f_.n; }
    // transform `nouter` lines: line o, column c, element e lives at
    // data[o*os + e*es + c], c in [0, ncols)
    template <typename R>
    void run(cplx<R>* data, size_t es, int ncols, size_t os, int nouter, bool inverse, cudaStream_t s) const;
    // forward transform, multiplication of element e of line o, column c by
    // scale[(e * nouter + o) * sz + c / sb], inverse transform: the k-space
    // step of a convolution fused into one pass over the lines
    template <typename R>
    void run_scaled(cplx<R>* data, size_t es, int ncols, size_t os, int nouter, const R* scale, int sz, int sb,
                    cudaStream_t s) const;
    // whether one line of this length fits in shared memory
    static bool fits(int n, bool fp64);
    // run every length through the general multi-pass kernel (tests)
    void set_force_general(bool v) { force_general_ = v; }
    // kernel a transform of ncols columns takes: 1 two-pass in registers (both
    // factors in-register radices, at least half a tile of columns per line),
    // 2 in-register radix times table product or a second one (mpm_dense.cu:
    // lengths with one prime above 16, two radices with few columns per line,
    // other lengths with a factor of 11 or 13 and none above),
    // 3 in-register radix and Rader's convolution (mpm_rader.cu: one prime too
    // long for the product, at least half a tile of columns per line, no
    // fused scale), 0 general multi-pass
    int path(int ncols, bool fp64, int mode) const {
        if (force_general_) return 0;
        if (kind_ == 1 && ncols >= 16) return 1;
        if (kind_ == 2 && ncols >= 16 && mode != 2 && rader_.usable() && rader_faster(fp64)) return 3;
        return dense_.fits(fp64) ? 2 : 0;
    }
    // the split of the kernel that such a transform takes, (0, 0) for the
    // general one
    std::pair<int, int> split(int ncols, bool fp64, int mode) const {
        const int p = path(ncols, fp64, mode);
        if (p == 2) return {dense_.radix(), dense_.rest()};
        return p ? std::pair<int, int>{r1_, r2_} : std::pair<int, int>{0, 0};
    }

    // The k-space step of the pruned (z-slab) monodisperse grid fused with
    // this axis's transforms, for the y axis: data is the grid
    // [x][y][slot][c][m] (Zs slots, 3 components, M right-hand sides), already
    // transformed along x.  For every (kx, chunk of right-hand sides) one CTA
    // loads its Ny x Zs x 3 x chunk values into shared memory, transforms
    // along y, applies the slab Green tensor of every (kx, ky) column as
    // three scalar Toeplitz kernels in z (taps [x][y][3][2 Zs - 1]:
    // t_n(d) = sum_kz kz^n S(k) / |k|^2 exp(2 pi i kz d / Nz), n = 0, 1, 2),
    //   a = kx E_x + ky E_y,  u = t0 * a + t1 * E_z,
    //   E_x <- kx u,  E_y <- ky u,  E_z <- t1 * a + t2 * E_z,
    // transforms back along y and stores: one HBM round trip for the y
    // transforms and the Green tensor.  kxu, kyu: the wavenumber of one
    // grid frequency along x and y (2 pi / L); nx: grid points along x.
    template <typename R>
    void run_slab(cplx<R>* data, int nx, int Zs, int M, const cplx<R>* taps, double kxu, double kyu,
                  cudaStream_t s) const;
    // whether run_slab handles this slab (two-pass in-register y transform,
    // Zs <= 16 slots, tile within the shared-memory budget)
    bool slab_ok(int Zs, bool fp64) const;

private:
    template <typename R>
    void launch_line(cplx<R>* data, size_t es, int ncols, size_t os, int nouter, int mode, const R* scale, int sz,
                     int sb, cudaStream_t s) const;
    static void upload_table(std::vector<double2> t64, DevBuf& d64, DevBuf& d32);
    FftFactors f_;
    // the length's own split n = r1 * r2: kind 1 both in-register radices (r1 >=
    // r2), kind 2 r1 in-register and r2 a prime above 16; (0, 0) if neither
    int kind_ = 0, r1_ = 0, r2_ = 0;
    bool force_general_ = false;
    DevBuf tw64_, tw32_;
    DevBuf pt64_, pt32_;   // prime-pass twiddle tables (see FftFactors)
    DenseDFT dense_;
    RaderDFT rader_;
    // The product's m FMAs per element against Rader's fixed cost (us per pass
    // of 46 MB, product and Rader: fp64 127 points 58 and 91, 131 113 and 89,
    // 257 211 and 84; fp32 181 points 88 and 139, 197 136 and 138, 211 160 and
    // 139, 257 177 and 131; 2 * 157 points 99 and 100, 2 * 181 104 and 98,
    // 2 * 193 142 and 93).  With the fused scale the product's two launches
    // are the faster ones (181 points, fp32: 200 and 2 x 139).
    bool rader_faster(bool fp64) const { return fp64 ? r2_ > 128 : r2_ > 200 || (r1_ > 1 && r2_ > 180); }
};

}  // namespace mpm
