// Batched device Krylov solvers (see mpm_krylov.h).
#include "mpm_krylov.h"
#include "mpm_chain.cuh"
#include "mpm_profile.h"

#include <algorithm>
#include <atomic>
#include <cmath>

namespace mpm {

namespace {

inline int nblk(long long n, int b) { return int((n + b - 1) / b); }

// ----------------------------------------------------------- reductions --

// out[i][m] = sum_row op(V_i[row][m]) * w[row][m], op = conj or identity.
// Stage 1 writes per-CTA partials; stage 2 sums them.  shift >= 0 (the
// GMRES step, w = V_{nvec-1} = A V_shift): the sums are taken with
// u = w - V_shift in place of w, and the last vector's entry is |u|^2.
__global__ void __launch_bounds__(256) k_dots1(const double2* __restrict__ V, size_t vstride, int nvec,
                                               const double2* __restrict__ w, int rows, int M, int conj,
                                               double2* __restrict__ partial, int shift) {
    __shared__ double2 red[8][8][32];
    const int m = blockIdx.y * 32 + threadIdx.x;
    const int i0 = blockIdx.z * 8;
    double2 acc[8];
    for (int k = 0; k < 8; ++k) acc[k] = make_double2(0, 0);
    const int nv = min(8, nvec - i0);
    if (m < M) {
#pragma unroll 4
        for (int row = blockIdx.x * 8 + threadIdx.y; row < rows; row += gridDim.x * 8) {
            double2 wv = w[size_t(row) * M + m];
            if (shift >= 0) wv -= V[size_t(shift) * vstride + size_t(row) * M + m];
            for (int k = 0; k < nv; ++k) {
                const double2 v = (shift >= 0 && i0 + k == nvec - 1) ? wv
                                                                       : V[size_t(i0 + k) * vstride + size_t(row) * M + m];
                if (conj) acc[k] += conjmul(v, wv);
                else acc[k] += v * wv;
            }
        }
    }
    for (int k = 0; k < 8; ++k) red[k][threadIdx.y][threadIdx.x] = acc[k];
    __syncthreads();
    if (threadIdx.y < nv && m < M) {
        double2 s = make_double2(0, 0);
        for (int r = 0; r < 8; ++r) s += red[threadIdx.y][r][threadIdx.x];
        partial[(size_t(blockIdx.x) * nvec + i0 + threadIdx.y) * M + m] = s;
    }
}

// Few columns (M < 16): threads run over the flat [row][M] elements, L =
// (256 / M) * M of them per CTA, so that each thread keeps one column for the
// whole grid-stride loop.

// The CTA's per-column sums of acc[0 .. nv) into out[k * M + m]: 2 to 8 lanes
// per sum (as many as the 256 threads give), a fixed shuffle tree.  One
// thread per sum walked up to 85 values in shared memory one after another.
__device__ __forceinline__ void cta_column_sums(const double2 (&acc)[8], int nv, int M, int L, double2 (*red)[256],
                                                double2* __restrict__ out) {
    const int j = threadIdx.x;
#pragma unroll
    for (int k = 0; k < 8; ++k) red[k][j] = acc[k];
    __syncthreads();
    const int n = nv * M;
    const int gs = n <= 32 ? 8 : n <= 64 ? 4 : 2;      // n <= 8 * 15
    const int o = j / gs, sl = j % gs;
    const bool live = o < n;
    const int k = live ? o / M : 0, m = live ? o - k * M : 0;
    double2 sum = make_double2(0, 0);
    if (live)
        for (int q = m + sl * M; q < L; q += gs * M) sum += red[k][q];
    for (int off = gs / 2; off > 0; off >>= 1) {
        sum.x += __shfl_xor_sync(0xffffffffu, sum.x, off);
        sum.y += __shfl_xor_sync(0xffffffffu, sum.y, off);
    }
    if (live && sl == 0) out[o] = sum;
    __syncthreads();
}

// true in every thread of the last CTA of `total` to get here (one counter,
// no waiting); everything the others wrote before is then visible
__device__ __forceinline__ bool last_cta(unsigned int* done, unsigned int total) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(done, 1u) == total - 1;
        if (last) *done = 0u;
    }
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// sums over the gx CTAs of partial[b][n] into out (shared or global): eight
// lanes per sum, a fixed shuffle tree
__device__ __forceinline__ void reduce_partials(const double2* __restrict__ partial, int gx, int n,
                                                double2* __restrict__ out) {
    const int g = threadIdx.x >> 3, sl = threadIdx.x & 7;
    for (int o0 = 0; o0 < n; o0 += 32) {
        const int o = o0 + g;
        double2 sum = make_double2(0, 0);
        if (o < n) {
#pragma unroll 8
            for (int b = sl; b < gx; b += 8) sum += __ldcg(&partial[size_t(b) * n + o]);
        }
        for (int off = 4; off > 0; off >>= 1) {
            sum.x += __shfl_xor_sync(0xffffffffu, sum.x, off);
            sum.y += __shfl_xor_sync(0xffffffffu, sum.y, off);
        }
        if (o < n && sl == 0) out[o] = sum;
    }
}

// k_dots1 + k_dots2 for few columns in one launch: the last CTA reduces the
// partials; nrm (may be null) takes the square roots of the sums' real parts
__global__ void __launch_bounds__(256) k_dots1s(const double2* __restrict__ V, size_t vstride, int nvec,
                                                const double2* __restrict__ w, int rows, int M, int conj,
                                                double2* __restrict__ partial, double2* __restrict__ out,
                                                double* __restrict__ nrm, unsigned int* __restrict__ done) {
    chain_enter();
    __shared__ double2 red[8][256];
    const int L = (256 / M) * M;
    const int j = threadIdx.x;
    const int i0 = blockIdx.z * 8;
    const int nv = min(8, nvec - i0);
    const size_t n = size_t(rows) * M;
    double2 acc[8];
    for (int k = 0; k < 8; ++k) acc[k] = make_double2(0, 0);
    if (j < L) {
        for (size_t t = size_t(blockIdx.x) * L + j; t < n; t += size_t(gridDim.x) * L) {
            const double2 wv = w[t];
            // a fixed trip count, so that the group's loads issue together
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                if (k >= nv) break;
                const double2 v = V[size_t(i0 + k) * vstride + t];
                if (conj) acc[k] += conjmul(v, wv);
                else acc[k] += v * wv;
            }
        }
    }
    cta_column_sums(acc, nv, M, L, red, partial + (size_t(blockIdx.x) * nvec + i0) * M);
    if (!last_cta(done, gridDim.x * gridDim.z)) return;
    reduce_partials(partial, gridDim.x, nvec * M, out);
    if (nrm) {
        __syncthreads();
        if (j < M) nrm[j] = sqrt(fmax(out[j].x, 0.0));
    }
}

// one warp per output: lanes stride over the per-CTA partials, then a fixed
// shuffle tree (deterministic order)
__global__ void k_dots2(const double2* __restrict__ partial, int gx, int nvec, int M, double2* __restrict__ out) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (t >= nvec * M) return;
    double2 s = make_double2(0, 0);
    for (int b = lane; b < gx; b += 32) s += partial[size_t(b) * nvec * M + t];
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    if (lane == 0) out[t] = s;
}

__global__ void k_sqrt_re(const double2* __restrict__ in, int M, double* __restrict__ out) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < M) out[m] = sqrt(fmax(in[m].x, 0.0));
}

// w[row][m] += sgn * sum_{i < n_m} V_i[row][m] h[i][m]
__global__ void k_vupdate(double2* __restrict__ w, const double2* __restrict__ V, size_t vstride, int nvec,
                          const double2* __restrict__ h, int rows, int M, double sgn, const int* __restrict__ nper) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= size_t(rows) * M) return;
    const int m = int(t % M);
    const int n = nper ? nper[m] : nvec;
    double2 acc = make_double2(0, 0);
    for (int i = 0; i < n; ++i) acc += V[size_t(i) * vstride + t] * h[size_t(i) * M + m];
    w[t] += acc * sgn;
}

// out = a - b
__global__ void k_sub(const double2* __restrict__ a, const double2* __restrict__ b, double2* __restrict__ out,
                      size_t n) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n) out[t] = a[t] - b[t];
}

// out = diag(self)^-1 in  over the unknown layout (jacobi_precond_kernel,
// numerical_solver.cu:250-285: per particle 1/s, quads use their particle).
__global__ void k_jacobi(const double2* __restrict__ in, double2* __restrict__ out, int N, int Nq, int M,
                         const int* __restrict__ quad_idx, const double2* __restrict__ sc) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const size_t rows = size_t(3 * N + 5 * Nq);
    if (t >= rows * M) return;
    const int row = int(t / M), m = int(t % M);
    int p;
    if (row < 3 * N) p = row / 3;
    else {
        p = quad_idx[(row - 3 * N) / 5];
        if (p < 0 || p >= N) p = 0;
    }
    const double2 s = sc[size_t(p) * M + m];
    const double den = s.x * s.x + s.y * s.y;
    const double2 inv = den > 1e-30 ? make_double2(s.x / den, -s.y / den) : make_double2(1.0, 0.0);
    out[t] = in[t] * inv;
}

// ------------------------------------------------------------ GMRES state --

struct GState {
    int active;      // still solving (outer)
    int cyc;         // in the current Arnoldi cycle
    int kcount;      // Arnoldi columns of the current cycle
    int iters;       // total Arnoldi steps
    int converged;
    int reorth;      // this Arnoldi step: 0 one projection, 1 second pass pending, 2 second pass done
    int pad[2];
};

__device__ __forceinline__ double col_tol(double tol, const double* tolv, int m) { return tolv ? tolv[m] : tol; }

// start of a restart cycle: residual norm test and V_0 = r / |r|.
// flag[0] counts the cycling columns, flag[1 + m] is column m's cycle flag.
__global__ void k_gm_begin(GState* __restrict__ st, const double* __restrict__ rn, const double* __restrict__ bn,
                           double tol, const double* __restrict__ tolv, int maxiter, int restart,
                           double2* __restrict__ g, int M, int* __restrict__ flag) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    GState s = st[m];
    s.cyc = 0;
    s.kcount = 0;
    if (s.active) {
        if (rn[m] < col_tol(tol, tolv, m) * bn[m]) {
            s.active = 0;
            s.converged = 1;
        } else if (s.iters >= maxiter) {
            s.active = 0;
        } else {
            s.cyc = 1;
            g[size_t(m) * (restart + 1)] = make_double2(rn[m], 0.0);
            for (int i = 1; i <= restart; ++i) g[size_t(m) * (restart + 1) + i] = make_double2(0, 0);
            atomicAdd(flag, 1);
        }
    }
    flag[1 + m] = s.cyc;
    st[m] = s;
}

// V_dst[row][m] = src[row][m] / nrm[m] for cycling RHS (0 otherwise)
__global__ void k_normalize(const double2* __restrict__ src, double2* __restrict__ dst,
                            const double* __restrict__ nrm, const GState* __restrict__ st, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int m = int(t % M);
    const double d = nrm[m];
    dst[t] = (st[m].cyc && d > 0.0) ? src[t] * (1.0 / d) : make_double2(0, 0);
}

// ------------------------------------------------- Arnoldi step kernels --
//
// The operator writes A V_k straight into V_{k+1}, so one pass of k_dots1 over
// the k+2 vectors V_0..V_{k+1} gives h_i = V_i^H u (i <= k) and |u|^2 (i =
// k+1) for u = w - V_k (then h_k(w) = h_k(u) + 1; u has the same projection
// remainder w' as w).  Every column takes two projections (CGS2); the norm of
// the second remainder follows by Pythagoras.  The Givens rotation of a column
// uses the final h and |w'|; the last launch projects and normalises V_{k+1}
// in place.

// Givens update of Hessenberg column k of one right-hand side (h[i * M + m],
// i <= k, plus `shift` on the diagonal; the previous rotations, a new rotation, the residual estimate; gmres_solver.cu:120-184)
__device__ void gm_givens(GState& s, const double2* __restrict__ h, double wn, double2* __restrict__ Hm,
                          double2* __restrict__ gm, double* __restrict__ csm, double2* __restrict__ snm, int k,
                          int ld, int M, int m, int restart, double tolm, double bnm, int maxiter,
                          double2 shift = make_double2(0.0, 0.0)) {
    double2* col = Hm + size_t(k) * ld;
    // the previous rotations applied down the column, the running entry in
    // a register (the column's inputs and the rotations are independent loads)
    double2 carry = h[m];
    if (k == 0) carry += shift;
    for (int i0 = 0; i0 < k; i0 += 8) {
        // eight rotations loaded before any is used
        double c8[8];
        double2 s8[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (i0 + u < k) {
                c8[u] = csm[i0 + u];
                s8[u] = snm[i0 + u];
            }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (i0 + u < k) {
                const int i = i0 + u;
                double2 h2 = h[size_t(i + 1) * M + m];
                if (i + 1 == k) h2 += shift;
                const double c = c8[u];
                const double2 sv = s8[u];
                const double2 cs_ = make_double2(sv.x, -sv.y);
                col[i] = carry * c + cs_ * h2;
                carry = (sv * carry) * -1.0 + h2 * c;
            }
    }
    const double2 h1 = carry, h2 = make_double2(wn, 0.0);
    double c = 1.0;
    double2 sv = make_double2(0, 0);
    if (h2.x != 0.0 || h2.y != 0.0) {
        const double a1 = hypot(h1.x, h1.y);
        if (a1 == 0.0) {
            c = 0.0;
            sv = make_double2(1.0, 0.0);
        } else {
            const double a2 = hypot(h2.x, h2.y);
            const double sc = a1 + a2;
            const double n1 = a1 / sc, n2 = a2 / sc;
            const double hh = sc * sqrt(n1 * n1 + n2 * n2);
            c = a1 / hh;
            // (conj(h1)/|h1|) * (h2/hh)
            const double2 u = make_double2(h1.x / a1, -h1.y / a1);
            sv = u * make_double2(h2.x / hh, h2.y / hh);
        }
    }
    csm[k] = c;
    snm[k] = sv;
    const double2 scj = make_double2(sv.x, -sv.y);
    col[k] = h1 * c + scj * h2;
    col[k + 1] = make_double2(0, 0);
    const double2 g1 = gm[k], g2 = gm[k + 1];
    gm[k] = g1 * c + scj * g2;
    gm[k + 1] = (sv * g1) * -1.0 + g2 * c;
    s.iters += 1;
    const double resid = hypot(gm[k + 1].x, gm[k + 1].y);
    if (resid < tolm * bnm || k + 1 >= restart || s.iters >= maxiter) {
        s.cyc = 0;
        s.kcount = k + 1;
    }
}

// What follows a projection's sums, by one CTA.  First, h = [V_0..V_k, u]^H u
// with u = w - V_k: h_k += 1 (the coefficients of w) and the cycling columns
// marked for their second projection.
__device__ __forceinline__ void arn_finish1_body(GState* __restrict__ st, double2* __restrict__ h, int k, int M) {
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        const int cyc = st[m].cyc;
        st[m].reorth = cyc ? 1 : 0;
        if (cyc) h[size_t(k) * M + m].x += 1.0;
    }
}

// Second, h2 = [V_0..V_k, w']^H w' after the first: h += h2, |w''| by
// Pythagoras, the Givens update (givens = 0, the seeds of a shifted solve:
// none, they are the members', shift_givens_body).  flag[0] = columns still
// cycling, flag[1 + m] = column m cycling.
__device__ __forceinline__ void arn_finish2_body(GState* __restrict__ st, double2* __restrict__ h,
                                                 const double2* __restrict__ h2, int givens,
                                                 double* __restrict__ nu_out, double* __restrict__ inv_nu,
                                                 double2* __restrict__ H, double2* __restrict__ g,
                                                 double* __restrict__ cs, double2* __restrict__ sn, int k, int restart,
                                                 int M, const double* __restrict__ bn, double tol,
                                                 const double* __restrict__ tolv, int maxiter,
                                                 int* __restrict__ flag) {
    __shared__ int ncyc;
    if (threadIdx.x == 0) ncyc = 0;
    // (columns not cycling have w' = 0, so h2 = 0)
    for (int t = threadIdx.x; t < (k + 1) * M; t += blockDim.x) h[t] += h2[t];
    __syncthreads();
    const int ld = restart + 1;
    int c_cyc = 0;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        GState s = st[m];
        if (s.cyc && s.reorth == 1) {
            const double wn2 = h2[size_t(k + 1) * M + m].x;
            double hs = 0.0;
#pragma unroll 8
            for (int i = 0; i <= k; ++i) {
                const double2 v = h2[size_t(i) * M + m];
                hs += v.x * v.x + v.y * v.y;
            }
            const double nu = sqrt(fmax(wn2 - hs, 0.0));
            inv_nu[m] = nu > 0.0 ? 1.0 / nu : 0.0;
            if (nu_out) nu_out[m] = nu;
            if (givens)
                gm_givens(s, h, nu, H + size_t(m) * ld * restart, g + size_t(m) * ld, cs + size_t(m) * restart,
                          sn + size_t(m) * restart, k, ld, M, m, restart, col_tol(tol, tolv, m), bn[m], maxiter);
            s.reorth = 2;
            st[m] = s;
        }
        c_cyc += s.cyc;
        flag[1 + m] = s.cyc;
    }
    if (c_cyc) atomicAdd(&ncyc, c_cyc);
    __syncthreads();
    if (threadIdx.x == 0) flag[0] = ncyc;
}

__global__ void __launch_bounds__(256) k_arn_finish1(GState* __restrict__ st, double2* __restrict__ h, int k, int M) {
    arn_finish1_body(st, h, k, M);
}

// V_{k+1} -= sum_{i <= k} V_i h_i for the columns of this pass (pass 1: the
// columns still cycling; pass 2: those whose second projection was just
// finished), then scaled by 1/|w'| unless a second pass is pending; the
// other columns of V_{k+1} (ended cycles, unused) are zeroed in pass 1.
__global__ void k_arn_update(double2* __restrict__ V, size_t vstride, int k, const double2* __restrict__ h,
                             const GState* __restrict__ st, const double* __restrict__ inv_nu, int rows, int M,
                             int pass) {
    chain_enter();
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= size_t(rows) * M) return;
    const int m = int(t % M);
    const GState s = st[m];
    double2* w = V + size_t(k + 1) * vstride + t;
    const bool mine = pass == 1 ? s.cyc != 0 : s.reorth == 2;
    if (!mine) {
        if (pass == 1) *w = make_double2(0, 0);
        return;
    }
    // four independent partial sums, so that a thread has four loads of V
    // in flight (the sum's order is fixed)
    double2 a0 = make_double2(0, 0), a1 = a0, a2 = a0, a3 = a0;
    int i = 0;
    for (; i + 3 <= k; i += 4) {
        a0 += V[size_t(i) * vstride + t] * h[size_t(i) * M + m];
        a1 += V[size_t(i + 1) * vstride + t] * h[size_t(i + 1) * M + m];
        a2 += V[size_t(i + 2) * vstride + t] * h[size_t(i + 2) * M + m];
        a3 += V[size_t(i + 3) * vstride + t] * h[size_t(i + 3) * M + m];
    }
    for (; i <= k; ++i) a0 += V[size_t(i) * vstride + t] * h[size_t(i) * M + m];
    const double2 acc = (a0 + a1) + (a2 + a3);
    double2 v = *w - acc;
    if (s.reorth != 1) v = v * inv_nu[m];
    *w = v;
}

// ---------------------------------------------------------- shifted solve --
//
// Columns m whose self coefficients are one particle profile c times a
// scalar, sc[:, m] = f_m c, have operators A_m = G + f_m diag(c) (G the
// interactions and the self value common to all columns); scaled by
// diag(c)^-1 they are the shifted family A0 + (f_m - 1) I with A0 = diag(c)^-1
// G + I, the operator apply gives with self coefficients c and Jacobi
// scaling.  Columns with the same right-hand side share one Krylov space of
// A0: one seed column per distinct right-hand side is iterated, and every
// member m of a seed's group runs its own Givens QR on the seed's Hessenberg
// column with sigma_m = f_m - 1 added to the diagonal (GMRES for shifted
// systems with x0 = 0, whose residuals stay collinear).

// f_m = sc[0][m] / sc[0][0]; bad[m] = 1 unless sc[i][m] = f_m sc[i][0] for
// every particle i (relative 1e-12)
__global__ void k_shift_ratio(const double2* __restrict__ sc, int N, int M, double2* __restrict__ f,
                              int* __restrict__ bad) {
    const int m = blockIdx.x;
    const double2 a = sc[m], c0 = sc[0];
    const double den = c0.x * c0.x + c0.y * c0.y;
    const double2 fm = den > 0.0 ? make_double2((a.x * c0.x + a.y * c0.y) / den, (a.y * c0.x - a.x * c0.y) / den)
                                 : make_double2(0, 0);
    int miss = den > 0.0 ? 0 : 1;
    for (int i = threadIdx.x; i < N && !miss; i += blockDim.x) {
        const double2 v = sc[size_t(i) * M + m], r = sc[size_t(i) * M] * fm;
        const double dx = v.x - r.x, dy = v.y - r.y;
        if (dx * dx + dy * dy > 1e-24 * (v.x * v.x + v.y * v.y) || (v.x == 0.0 && v.y == 0.0)) miss = 1;
    }
    miss = __syncthreads_or(miss);
    if (threadIdx.x == 0) {
        f[m] = fm;
        bad[m] = miss;
    }
}

// eq[m][m2] = 1 if right-hand-side columns m and m2 < m are equal
__global__ void k_col_equal(const double2* __restrict__ b, int rows, int M, int* __restrict__ eq) {
    const int m = blockIdx.x, m2 = blockIdx.y;
    if (m2 >= m) return;
    int diff = 0;
    for (int r = threadIdx.x; r < rows && !diff; r += blockDim.x) {
        const double2 u = b[size_t(r) * M + m], v = b[size_t(r) * M + m2];
        if (u.x != v.x || u.y != v.y) diff = 1;
    }
    diff = __syncthreads_or(diff);
    if (threadIdx.x == 0) eq[size_t(m) * M + m2] = !diff;
}

// member m of seed grp[m]: Hessenberg column k of the seed plus sigma_m on
// the diagonal, then its Givens update (gm_givens), once the seed's second
// projection is done (reorth 2).  A seed cycles while any member does
// (written back to its state).  One CTA: flag[0] = seeds cycling,
// flag[1 + g] = seed g cycling.
__device__ __forceinline__ void shift_givens_body(GState* __restrict__ mst, GState* __restrict__ sst,
                                                  const double2* __restrict__ hs, const double* __restrict__ nu,
                                                  const double2* __restrict__ sigma, const int* __restrict__ grp,
                                                  int G, double2* __restrict__ H,
                                                  double2* __restrict__ g, double* __restrict__ cs,
                                                  double2* __restrict__ sn, int k, int restart, int M,
                                                  const double* __restrict__ bs, const double* __restrict__ tolv,
                                                  int maxiter, int* __restrict__ seed_cyc, int* __restrict__ flag) {
    __shared__ int n;
    if (threadIdx.x == 0) n = 0;
    for (int t = threadIdx.x; t < G; t += blockDim.x) seed_cyc[t] = 0;
    __syncthreads();
    const int ld = restart + 1;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        GState s = mst[m];
        if (!s.cyc) continue;
        const int gi = grp[m];
        if (sst[gi].reorth == 2) {
            gm_givens(s, hs, nu[gi], H + size_t(m) * ld * restart, g + size_t(m) * ld, cs + size_t(m) * restart,
                      sn + size_t(m) * restart, k, ld, G, gi, restart, tolv[m], bs[gi], maxiter, sigma[m]);
            mst[m] = s;
        }
        if (s.cyc) atomicOr(&seed_cyc[gi], 1);
    }
    __syncthreads();
    for (int t = threadIdx.x; t < G; t += blockDim.x) {
        flag[1 + t] = seed_cyc[t];
        sst[t].cyc = seed_cyc[t];
        if (seed_cyc[t]) atomicAdd(&n, 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) flag[0] = n;
}

// The members of a shifted solve: their Givens updates (shift_givens_body)
// follow the seeds' second projection (arn_finish2_body without Givens) in the
// same CTA (finish2_body).  They read only the seeds' Hessenberg column and
// norm, so the seeds' normalisation of V_{k+1} can follow.
struct MemberArgs {
    GState* st;             // null: no members (plain GMRES)
    const double2* sigma;
    const int* grp;
    int M;
    const double* tolv;
    int* seed_cyc;
};

// The Hessenberg / Givens state a finish works on (plain GMRES: of the columns
// themselves; shifted solve: of the members)
struct HessArgs {
    double2* H;
    double2* g;
    double* cs;
    double2* sn;
    const double* bn;       // |b| per column (shifted: per seed)
    double tol;
    const double* tolv;
    int maxiter, restart;
    double* nu;             // |w'| per seed (shifted), or null
    double* inv_nu;
    int* flag;
    int* hflag;             // the same words for the host (page-locked): hflag[0] = seq once hflag[1 + t] = flag[t]
    int seq;
};

__device__ __forceinline__ void finish2_body(GState* st, double2* h, const double2* h2, const HessArgs& a,
                                             const MemberArgs& mb, int k, int M) {
    const bool seeds = mb.st != nullptr;
    arn_finish2_body(st, h, h2, seeds ? 0 : 1, a.nu, a.inv_nu, a.H, a.g, a.cs, a.sn, k, a.restart, M, a.bn, a.tol,
                    seeds ? nullptr : a.tolv, a.maxiter, a.flag);
    __syncthreads();
    if (seeds) {
        shift_givens_body(mb.st, st, h, a.nu, mb.sigma, mb.grp, M, a.H, a.g, a.cs, a.sn, k, a.restart, mb.M, a.bn,
                          mb.tolv, a.maxiter, mb.seed_cyc, a.flag);
        __syncthreads();
    }
    // the flags go straight to the host, which waits for them while the last
    // launch of the step still runs
    for (int t = threadIdx.x; t <= M; t += blockDim.x) a.hflag[1 + t] = a.flag[t];
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) *static_cast<volatile int*>(a.hflag) = a.seq;
}

// the second finish of many columns (M >= 16), with the members' updates when
// there are seeds
__global__ void __launch_bounds__(256) k_arn_finish2(GState* __restrict__ st, double2* __restrict__ h,
                                                      const double2* __restrict__ h2, HessArgs a, MemberArgs mb,
                                                      int k, int M) {
    finish2_body(st, h, h2, a, mb, k, M);
}

// ---- the Arnoldi step of few columns (M < 16) in three launches
//
// Each projection's sums, their reduction and the one-CTA kernel that follows
// are one launch: the last CTA to finish reduces the partials and does the
// finish.  The second launch also applies the first projection.  With the
// launches separate (dots, finish, update, twice) a step took 44 to 66 us of
// 5 to 15 us launches, all latency; 31 now (N = 4000, 3 columns, 5 steps).

// [V_0 .. V_k, u]^H u for u = w - V_k, then arn_finish1_body
__global__ void __launch_bounds__(256) k_arn_dots(const double2* __restrict__ V, size_t vstride, int k, int rows,
                                                  int M, double2* __restrict__ partial, GState* __restrict__ st,
                                                  double2* __restrict__ h, unsigned int* __restrict__ done) {
    chain_enter();
    __shared__ double2 red[8][256];
    const int nvec = k + 2;
    const int L = (256 / M) * M;
    const int j = threadIdx.x;
    const int i0 = blockIdx.z * 8;
    const int nv = min(8, nvec - i0);
    const size_t n = size_t(rows) * M;
    const double2* w = V + size_t(k + 1) * vstride;
    const double2* vk = V + size_t(k) * vstride;
    double2 acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = make_double2(0, 0);
    if (j < L) {
        for (size_t t = size_t(blockIdx.x) * L + j; t < n; t += size_t(gridDim.x) * L) {
            const double2 u = w[t] - vk[t];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (i >= nv) break;
                const double2 v = i0 + i == nvec - 1 ? u : V[size_t(i0 + i) * vstride + t];
                acc[i] += conjmul(v, u);
            }
        }
    }
    cta_column_sums(acc, nv, M, L, red, partial + (size_t(blockIdx.x) * nvec + i0) * M);
    if (!last_cta(done, gridDim.x * gridDim.z)) return;
    reduce_partials(partial, gridDim.x, nvec * M, h);
    __syncthreads();
    arn_finish1_body(st, h, k, M);
}

// w' = w - sum_{i <= k} V_i h_i (columns not cycling: 0), [V_0 .. V_k, w']^H w'
// into h2, then finish2_body
__global__ void __launch_bounds__(256) k_arn_project(double2* __restrict__ V, size_t vstride, int k, int rows, int M,
                                                     double2* __restrict__ partial, GState* __restrict__ st,
                                                     double2* __restrict__ h, double2* __restrict__ h2, HessArgs a,
                                                     MemberArgs mb, unsigned int* __restrict__ done) {
    chain_enter();
    __shared__ double2 red[8][256];
    const int nvec = k + 2;
    const int L = (256 / M) * M;
    const int j = threadIdx.x;
    const size_t n = size_t(rows) * M;
    double2* w = V + size_t(k + 1) * vstride;
    const size_t step = size_t(gridDim.x) * L;
    const size_t t0 = size_t(blockIdx.x) * L + j;
    const int m = j % M;
    if (j < L) {
        const bool mine = st[m].cyc != 0;
        for (size_t t = t0; t < n; t += step) {
            if (!mine) {
                w[t] = make_double2(0, 0);
                continue;
            }
            double2 a0 = make_double2(0, 0), a1 = a0, a2 = a0, a3 = a0;
            int i = 0;
            for (; i + 3 <= k; i += 4) {
                a0 += V[size_t(i) * vstride + t] * h[size_t(i) * M + m];
                a1 += V[size_t(i + 1) * vstride + t] * h[size_t(i + 1) * M + m];
                a2 += V[size_t(i + 2) * vstride + t] * h[size_t(i + 2) * M + m];
                a3 += V[size_t(i + 3) * vstride + t] * h[size_t(i + 3) * M + m];
            }
            for (; i <= k; ++i) a0 += V[size_t(i) * vstride + t] * h[size_t(i) * M + m];
            w[t] = w[t] - ((a0 + a1) + (a2 + a3));
        }
    }
    // (a thread reads back only what it wrote)
    for (int i0 = 0; i0 < nvec; i0 += 8) {
        const int nv = min(8, nvec - i0);
        double2 acc[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = make_double2(0, 0);
        if (j < L) {
            for (size_t t = t0; t < n; t += step) {
                const double2 u = w[t];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    if (i >= nv) break;
                    acc[i] += conjmul(V[size_t(i0 + i) * vstride + t], u);
                }
            }
        }
        cta_column_sums(acc, nv, M, L, red, partial + (size_t(blockIdx.x) * nvec + i0) * M);
    }
    if (!last_cta(done, gridDim.x)) return;
    // the finish on copies of h and h2 in shared memory (when they fit): it is
    // a chain of dependent reads by a few threads
    const int n2 = nvec * M;
    const bool fits = 2 * n2 <= 8 * 256;
    double2* hs = fits ? &red[0][0] : h;
    double2* h2s = fits ? hs + n2 : h2;
    reduce_partials(partial, gridDim.x, n2, h2s);
    if (fits)
        for (int t = j; t < n2 - M; t += 256) hs[t] = h[t];
    __syncthreads();
    if (fits)
        for (int t = j; t < n2; t += 256) h2[t] = h2s[t];      // for k_arn_update
    finish2_body(st, hs, h2s, a, mb, k, M);
}

// member states: active and cycling from the start, x0 = 0; g_m = (beta, 0..);
// members already converged (skip[m], may be null) take no part
__global__ void k_shift_init(GState* __restrict__ mst, const int* __restrict__ grp, const double* __restrict__ bs,
                             const int* __restrict__ skip, double2* __restrict__ g, int restart, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    GState s{};
    const double beta = (skip && skip[m]) ? 0.0 : bs[grp[m]];
    s.active = beta > 0.0;
    s.cyc = s.active;
    s.converged = !s.active;
    mst[m] = s;
    g[size_t(m) * (restart + 1)] = make_double2(beta, 0.0);
    for (int i = 1; i <= restart; ++i) g[size_t(m) * (restart + 1) + i] = make_double2(0, 0);
}

// x[row][m] = sum_{i < kper[m]} V_i[row][grp[m]] y[i][m] (columns skipped
// as converged keep their x)
__global__ void k_shift_x(double2* __restrict__ x, const double2* __restrict__ V, size_t vstride, int G,
                          const double2* __restrict__ y, const int* __restrict__ grp, const int* __restrict__ kper,
                          const int* __restrict__ skip, int rows, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= size_t(rows) * M) return;
    const size_t row = t / M;
    const int m = int(t - row * M);
    if (skip && skip[m]) return;
    const int gi = grp[m];
    double2 acc = make_double2(0, 0);
    for (int i = 0; i < kper[m]; ++i) acc += V[size_t(i) * vstride + row * G + gi] * y[size_t(i) * M + m];
    x[t] = acc;
}

// back substitution H y = g, y stored [i][m].  Warp per column, lanes over the
// rows still to solve (the running right-hand side in shared memory): a step
// divides one entry and subtracts its column of H, read contiguously and
// ahead of its use.  One thread per column took 112 us for 30 columns of 14
// steps.
constexpr int kBacksubWarps = 4;

__global__ void __launch_bounds__(kBacksubWarps * 32) k_gm_backsub(const GState* __restrict__ st,
                                                                   const double2* __restrict__ H,
                                                                   const double2* __restrict__ g,
                                                                   double2* y, int restart, int M,
                                                                   int* __restrict__ kper, int in_smem) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m = blockIdx.x * kBacksubWarps + warp;
    if (m >= M) return;   // whole warps leave together
    // the running right-hand side (in y itself when the restart is too long)
    double2* v = in_smem ? reinterpret_cast<double2*>(smem_raw) + size_t(warp) * restart : y + m;
    const size_t vs = in_smem ? 1 : size_t(M);
    const int k = st[m].kcount;
    if (lane == 0) kper[m] = k;
    const int ld = restart + 1;
    const double2* Hm = H + size_t(m) * ld * restart;
    for (int i = lane; i < k; i += 32) v[i * vs] = g[size_t(m) * ld + i];
    __syncwarp();
    double2 d = k > 0 ? Hm[size_t(k - 1) * ld + k - 1] : make_double2(1.0, 0.0);
    for (int i = k - 1; i >= 0; --i) {
        const double2* col = Hm + size_t(i) * ld;
        const double2 dn = i > 0 ? Hm[size_t(i - 1) * ld + i - 1] : d;
        const double2 c0 = lane < i ? col[lane] : make_double2(0, 0);
        const double2 vi = v[i * vs];
        const double den = d.x * d.x + d.y * d.y;
        const double2 yi = make_double2((vi.x * d.x + vi.y * d.y) / den, (vi.y * d.x - vi.x * d.y) / den);
        __syncwarp();      // every lane has read v[i]
        if (lane == 0) y[size_t(i) * M + m] = yi;
        if (lane < i) v[lane * vs] -= c0 * yi;
        for (int l = lane + 32; l < i; l += 32) v[l * vs] -= col[l] * yi;
        __syncwarp();
        d = dn;
    }
}

// seeds: cycling from the start unless their right-hand side is zero
__global__ void k_seed_init(GState* __restrict__ st, const double* __restrict__ bn, int G) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= G) return;
    GState s{};
    s.active = s.cyc = bn[m] > 0.0;
    st[m] = s;
}

__global__ void k_zero_rhs_cols(double2* __restrict__ x, const double* __restrict__ bn, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    if (bn[t % M] == 0.0) x[t] = make_double2(0, 0);
}

__global__ void k_gm_init(GState* __restrict__ st, const double* __restrict__ bn, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    GState s{};
    s.active = bn[m] > 0.0 ? 1 : 0;
    s.converged = bn[m] > 0.0 ? 0 : 1;
    st[m] = s;
}

// --------------------------------------------------------- BiCGSTAB state --

struct BState {
    double2 rho, alpha, omega, beta;
    int active, converged, iters, pad;
};

__global__ void k_bi_init(BState* __restrict__ st, const double* __restrict__ bn, const double* __restrict__ rn,
                          double tol, const double* __restrict__ tolv, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    BState s{};
    s.rho = s.alpha = s.omega = make_double2(1.0, 0.0);
    s.beta = make_double2(0, 0);
    s.active = 1;
    if (bn[m] == 0.0) { s.active = 0; s.converged = 1; }
    else if (rn[m] < col_tol(tol, tolv, m) * bn[m]) { s.active = 0; s.converged = 1; }
    st[m] = s;
}

__device__ __forceinline__ double2 cdiv(double2 a, double2 b) {
    const double den = b.x * b.x + b.y * b.y;
    return make_double2((a.x * b.x + a.y * b.y) / den, (a.y * b.x - a.x * b.y) / den);
}
__device__ __forceinline__ double cabs_(double2 a) { return hypot(a.x, a.y); }

// step A: rho_new test and beta (bicgstab_solver.cu:153-169)
__global__ void k_bi_a(BState* __restrict__ st, const double2* __restrict__ rho_new, int it, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    BState s = st[m];
    if (!s.active) return;
    const double2 rn = rho_new[m];
    if (cabs_(rn) < 1e-16) { s.active = 0; st[m] = s; return; }
    s.beta = it > 0 ? cdiv(rn, s.rho) * cdiv(s.alpha, s.omega) : make_double2(0, 0);
    s.rho = rn;
    s.iters += 1;
    st[m] = s;
}

// p = r + beta (p - omega v)  (it > 0), p unchanged at it == 0
__global__ void k_bi_p(double2* __restrict__ p, const double2* __restrict__ v, const double2* __restrict__ r,
                       const BState* __restrict__ st, int it, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n || it == 0) return;
    const BState& s = st[t % M];
    if (!s.active) return;
    p[t] = (p[t] - s.omega * v[t]) * s.beta + r[t];
}

// step B: alpha = rho / (r0 . v)
__global__ void k_bi_b(BState* __restrict__ st, const double2* __restrict__ rv, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    BState s = st[m];
    if (!s.active) return;
    if (cabs_(rv[m]) < 1e-16) { s.active = 0; st[m] = s; return; }
    s.alpha = cdiv(s.rho, rv[m]);
    st[m] = s;
}

// s = r - alpha v
__global__ void k_bi_s(double2* __restrict__ sv, const double2* __restrict__ r, const double2* __restrict__ v,
                       const BState* __restrict__ st, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const BState& s = st[t % M];
    if (!s.active) return;
    sv[t] = r[t] - s.alpha * v[t];
}

// step C: |s| < tol |b| => x += alpha p and stop (mode 1)
__global__ void k_bi_c(BState* __restrict__ st, const double* __restrict__ sn, const double* __restrict__ bn,
                       double tol, const double* __restrict__ tolv, int* __restrict__ mode, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    BState s = st[m];
    mode[m] = 0;
    if (!s.active) return;
    if (sn[m] < col_tol(tol, tolv, m) * bn[m]) {
        mode[m] = 1;
        s.active = 0;
        s.converged = 1;
        st[m] = s;
    }
}

__global__ void k_bi_xfinal(double2* __restrict__ x, const double2* __restrict__ p, const BState* __restrict__ st,
                            const int* __restrict__ mode, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int m = int(t % M);
    if (mode[m] == 1) x[t] += st[m].alpha * p[t];
}

// step D: omega = (t, s) / (t, t)
__global__ void k_bi_d(BState* __restrict__ st, const double2* __restrict__ ts, const double2* __restrict__ tt, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    BState s = st[m];
    if (!s.active) return;
    if (cabs_(tt[m]) < 1e-16) { s.active = 0; st[m] = s; return; }
    s.omega = ts[m] * (1.0 / tt[m].x);
    st[m] = s;
}

// x += alpha p + omega s ; r = s - omega t
__global__ void k_bi_xr(double2* __restrict__ x, double2* __restrict__ r, const double2* __restrict__ p,
                        const double2* __restrict__ sv, const double2* __restrict__ tv,
                        const BState* __restrict__ st, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const BState& s = st[t % M];
    if (!s.active) return;
    x[t] += s.alpha * p[t] + s.omega * sv[t];
    r[t] = sv[t] - s.omega * tv[t];
}

// step E: |r| < tol |b| or omega ~ 0 => stop; count still active
__global__ void k_bi_e(BState* __restrict__ st, const double* __restrict__ rn, const double* __restrict__ bn,
                       double tol, const double* __restrict__ tolv, int maxiter, int* __restrict__ flag, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    BState s = st[m];
    if (s.active) {
        if (rn[m] < col_tol(tol, tolv, m) * bn[m]) { s.active = 0; s.converged = 1; }
        else if (cabs_(s.omega) < 1e-16) s.active = 0;
        else if (s.iters >= maxiter) s.active = 0;
        if (s.active) atomicAdd(flag, 1);
        st[m] = s;
    }
    flag[1 + m] = s.active;
}

__global__ void k_bi_count(const BState* __restrict__ st, int* __restrict__ flag, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    flag[1 + m] = st[m].active;
    if (st[m].active) atomicAdd(flag, 1);
}

// refinement bookkeeping: a column stays converged once its true residual
// met the target (later rounds leave its x and its stale residual alone)
__global__ void k_conv_update(const double* __restrict__ rn, const double* __restrict__ bn, double tol,
                              int* __restrict__ conv, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m < M && !conv[m] && rn[m] <= tol * bn[m]) conv[m] = 1;
}

// zero the correction right-hand side of converged columns
__global__ void k_mask_conv(double2* __restrict__ r, const int* __restrict__ conv, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    if (conv[t % M]) r[t] = make_double2(0, 0);
}

// columns with sel[m] set take the fp64 residual (r, its norm) in place of
// the fp32 screen's
__global__ void k_take_cols(double2* __restrict__ r, const double2* __restrict__ r64, double* __restrict__ rn,
                            const double* __restrict__ rn64, const int* __restrict__ sel, size_t n, int M) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int m = int(t % M);
    if (!sel[m]) return;
    r[t] = r64[t];
    if (t < size_t(M)) rn[t] = rn64[t];
}

__global__ void k_axpy1(double2* __restrict__ x, const double2* __restrict__ d, size_t n) {
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n) x[t] += d[t];
}

// dst[row][j] = src[row][idx[j]]  (compact batch of the listed columns)
__global__ void k_gather_cols(const double2* __restrict__ src, int M, double2* __restrict__ dst, int Ma,
                              const int* __restrict__ idx, int rows) {
    chain_enter();
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= size_t(rows) * Ma) return;
    const size_t row = t / Ma;
    const int j = int(t - row * Ma);
    dst[t] = src[row * M + idx[j]];
}

// dst[row][idx[j]] = src[row][j]
__global__ void k_scatter_cols(const double2* __restrict__ src, int Ma, double2* __restrict__ dst, int M,
                               const int* __restrict__ idx, int rows) {
    chain_enter();
    const size_t t = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= size_t(rows) * Ma) return;
    const size_t row = t / Ma;
    const int j = int(t - row * Ma);
    dst[row * M + idx[j]] = src[t];
}

// inner tolerance of column m: stop once its residual is below 0.5 tol |b_m|,
// i.e. relative to its own right-hand side |r_m|: 0.5 tol |b_m| / |r_m|,
// but ask no inner solve for a reduction below `floor` (fp32 rounding of
// the operator limits what one inner solve can reach) nor above 0.5.
__global__ void k_inner_tol(const double* __restrict__ rn, const double* __restrict__ bn, double tol, double floor,
                            double* __restrict__ tolv, int M) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M) return;
    double t = rn[m] > 0.0 ? 0.5 * tol * bn[m] / rn[m] : 0.5;
    tolv[m] = fmin(0.5, fmax(floor, t));
}

}  // namespace

// ------------------------------------------------------------ host side --

BatchSolver::BatchSolver() = default;
BatchSolver::~BatchSolver() = default;

int BatchSolver::read_flags(const int* dflag, int M, cudaStream_t s) {
    // (no copy into the words is in flight: every read ends with a wait)
    flagbuf_.ensure(sizeof(int) * (size_t(M) + 1));
    flag_ = flagbuf_.as<int>();
    MPM_CUDA(cudaMemcpyAsync(flag_, dflag, sizeof(int) * (M + 1), cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaStreamSynchronize(s));
    return *flag_;
}

int* BatchSolver::poll_words(int M) {
    const size_t bytes = sizeof(int) * (size_t(M) + 2);
    if (!poll_.p || poll_.bytes < bytes) {
        poll_.ensure(bytes);
        poll_.as<int>()[0] = 0;        // no sequence number (they start at 1)
    }
    return poll_.as<int>();
}

// Waits for the flags of the Arnoldi step with the latest sequence number and
// returns the count.  The kernel that makes them writes them to page-locked
// memory, so the host need not wait for the step's last launch nor for a
// copy; the stream is queried now and then, so that a failed launch ends the
// wait with its error.
int BatchSolver::wait_flags(cudaStream_t s) {
    const volatile int* w = poll_.as<int>();
    for (unsigned it = 1; w[0] != poll_seq_; ++it) {
        if (it % 4096) continue;
        const cudaError_t e = cudaStreamQuery(s);
        if (e == cudaErrorNotReady) continue;
        MPM_CUDA(e);
        if (w[0] != poll_seq_) throw std::runtime_error("Krylov step ended without its flags");
    }
    std::atomic_thread_fence(std::memory_order_acquire);
    return w[1];
}

int BatchSolver::apply_cols(Field& F, const double2* X, double2* Y, int M, const double2* sc, bool jacobi,
                            bool r32, bool re32, const int* active, bool compact, cudaStream_t s) {
    if (!compact || !active) {
        F.apply(X, Y, M, sc, jacobi, r32, re32, s);
        return M;
    }
    std::vector<int> cols;
    cols.reserve(M);
    for (int m = 0; m < M; ++m)
        if (active[m]) cols.push_back(m);
    const int Ma = int(cols.size());
    if (Ma == 0) return 0;
    if (Ma == M) {
        F.apply(X, Y, M, sc, jacobi, r32, re32, s);
        return M;
    }
    const int rin = F.rows_in(), rout = F.rows_out(), N = F.num_particles();
    if (cols != cur_cols_) {
        StageScope scope(ST_KRYLOV, s);
        // the previous upload from hidx_ has completed: every change of the
        // column set follows flags that were made after it on this stream
        hidx_.ensure(sizeof(int) * M);
        std::copy(cols.begin(), cols.end(), hidx_.as<int>());
        cidx_.ensure(sizeof(int) * M);
        MPM_CUDA(cudaMemcpyAsync(cidx_.p, hidx_.p, sizeof(int) * Ma, cudaMemcpyHostToDevice, s));
        if (sc) {
            scc_.ensure(sizeof(double2) * size_t(N) * M);
            k_gather_cols<<<nblk((long long)N * Ma, 256), 256, 0, s>>>(sc, M, scc_.as<double2>(), Ma,
                                                                        cidx_.as<int>(), N);
            MPM_LAUNCH();
        }
        cur_cols_ = cols;
    }
    xc_.ensure(sizeof(double2) * size_t(rin) * M);
    yc_.ensure(sizeof(double2) * size_t(rout) * M);
    {
        StageScope scope(ST_KRYLOV, s);
        launch_chained(k_gather_cols, nblk((long long)rin * Ma, 256), 256, 0, s, X, M, xc_.as<double2>(), Ma,
                       cidx_.as<int>(), rin);
    }
    F.apply(xc_.as<double2>(), yc_.as<double2>(), Ma, sc ? scc_.as<double2>() : nullptr, jacobi, r32, re32, s);
    {
        StageScope scope(ST_KRYLOV, s);
        launch_chained(k_scatter_cols, nblk((long long)rout * Ma, 256), 256, 0, s, yc_.as<double2>(), Ma, Y, M,
                       cidx_.as<int>(), rout);
    }
    return Ma;
}

// CTAs of the few-column kernels over n elements: at most two per SM, so that
// the last one's reduction stays short
int BatchSolver::small_ctas(size_t n, int M) const {
    const size_t L = size_t(256 / M) * M;
    return int(std::max<size_t>(1, std::min<size_t>(296, (n + L - 1) / L)));
}

unsigned int* BatchSolver::done_counter(cudaStream_t s) {
    if (!dots_done_.p) {
        dots_done_.ensure(sizeof(unsigned int));
        MPM_CUDA(cudaMemsetAsync(dots_done_.p, 0, sizeof(unsigned int), s));
    }
    return dots_done_.as<unsigned int>();
}

void BatchSolver::dots(const double2* V, size_t vstride, int nvec, const double2* w, int rows, int M, int conj,
                       double2* out, cudaStream_t s, int shift, double* nrm) {
    StageScope scope(ST_KRYLOV, s);
    if (M < 16 && shift < 0) {
        const int gx = small_ctas(size_t(rows) * M, M);
        partial_.ensure(sizeof(double2) * size_t(gx) * nvec * M);
        k_dots1s<<<dim3(gx, 1, (nvec + 7) / 8), 256, 0, s>>>(V, vstride, nvec, w, rows, M, conj,
                                                             partial_.as<double2>(), out, nrm, done_counter(s));
        MPM_LAUNCH();
        return;
    }
    // four CTAs per SM: the sums are latency-bound, not bandwidth-bound
    const int gx = std::max(1, std::min(592, (rows + 7) / 8));
    partial_.ensure(sizeof(double2) * size_t(gx) * nvec * M);
    dim3 grd(gx, (M + 31) / 32, (nvec + 7) / 8);
    k_dots1<<<grd, dim3(32, 8), 0, s>>>(V, vstride, nvec, w, rows, M, conj, partial_.as<double2>(), shift);
    MPM_LAUNCH();
    k_dots2<<<nblk((long long)nvec * M * 32, 256), 256, 0, s>>>(partial_.as<double2>(), gx, nvec, M, out);
    MPM_LAUNCH();
    if (nrm) {
        k_sqrt_re<<<nblk(M, 128), 128, 0, s>>>(out, M, nrm);
        MPM_LAUNCH();
    }
}

void BatchSolver::norms(const double2* w, int rows, int M, double* out, cudaStream_t s) {
    h2_.ensure(sizeof(double2) * M);
    dots(w, 0, 1, w, rows, M, 1, h2_.as<double2>(), s, -1, out);
}

namespace {
void backsub(const GState* st, const double2* H, const double2* g, double2* y, int restart, int M, int* kper,
             cudaStream_t s) {
    size_t shm = sizeof(double2) * kBacksubWarps * size_t(restart);
    const int in_smem = shm <= 48 * 1024;
    if (!in_smem) shm = 0;
    k_gm_backsub<<<nblk(M, kBacksubWarps), kBacksubWarps * 32, shm, s>>>(st, H, g, y, restart, M, kper, in_smem);
    MPM_LAUNCH();
}
}  // namespace

// Orthogonalisation of V_{k+1} = A V_k against V_0 .. V_k, the Hessenberg
// column and the Givens updates: CGS2, [V_0..V_k, u]^H u with u = w - V_k (the
// preconditioned operator is close to the identity, so w is mostly V_k: the
// first projection then works on the part that is not), w -= V h; then
// [V_0..V_k, w']^H w', w' -= V h2, normalised.
template <typename Hess, typename Member>
void BatchSolver::arnoldi(double2* V, int k, int rows, int M, void* state, const Hess& a, const Member& mb,
                          cudaStream_t s) {
    GState* st = static_cast<GState*>(state);
    const size_t n = size_t(rows) * M;
    double2* h = h_.as<double2>();
    double2* h2 = h2_.as<double2>();
    const int vb = nblk((long long)n, 256);
    StageScope scope(ST_KRYLOV, s);
    if (M < 16) {
        const int gx = small_ctas(n, M);
        partial_.ensure(sizeof(double2) * size_t(gx) * (a.restart + 2) * M);
        double2* part = partial_.as<double2>();
        unsigned int* done = done_counter(s);
        launch_chained(k_arn_dots, dim3(gx, 1, (k + 2 + 7) / 8), 256, 0, s, V, n, k, rows, M, part, st, h, done);
        launch_chained(k_arn_project, gx, 256, 0, s, V, n, k, rows, M, part, st, h, h2, a, mb, done);
    } else {
        double2* w = V + size_t(k + 1) * n;
        const bool seeds = mb.st != nullptr;
        const int fthr = std::min(256, ((std::max(M, seeds ? mb.M : M) + 31) / 32) * 32);
        dots(V, n, k + 2, w, rows, M, 1, h, s, k);
        k_arn_finish1<<<1, fthr, 0, s>>>(st, h, k, M);
        MPM_LAUNCH();
        k_arn_update<<<vb, 256, 0, s>>>(V, n, k, h, st, a.inv_nu, rows, M, 1);
        MPM_LAUNCH();
        dots(V, n, k + 2, w, rows, M, 1, h2, s);
        k_arn_finish2<<<1, fthr, 0, s>>>(st, h, h2, a, mb, k, M);
        MPM_LAUNCH();
    }
    launch_chained(k_arn_update, vb, 256, 0, s, V, n, k, h2, st, a.inv_nu, rows, M, 2);
}

void BatchSolver::true_residual(Field& F, const double2* b, const double2* x, int M, const double2* sc,
                                std::vector<double>& out, cudaStream_t s) {
    const int rows = F.rows_in();
    const size_t n = size_t(rows) * M;
    w_.ensure(sizeof(double2) * n);
    rr_.ensure(sizeof(double2) * n);
    rnorm_.ensure(sizeof(double) * M * 2);
    F.apply(x, w_.as<double2>(), M, sc, false, false, false, s);
    k_sub<<<nblk((long long)n, 256), 256, 0, s>>>(b, w_.as<double2>(), rr_.as<double2>(), n);
    MPM_LAUNCH();
    norms(rr_.as<double2>(), rows, M, rnorm_.as<double>(), s);
    norms(b, rows, M, rnorm_.as<double>() + M, s);
    std::vector<double> h(2 * M);
    MPM_CUDA(cudaMemcpyAsync(h.data(), rnorm_.p, sizeof(double) * 2 * M, cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaStreamSynchronize(s));
    out.resize(M);
    for (int m = 0; m < M; ++m) out[m] = h[M + m] > 0 ? h[m] / h[M + m] : 0.0;
}

void BatchSolver::gmres(Field& F, const double2* b, double2* x, int M, const double2* sc, const SolveOptions& opt,
                        SolveStats& st, bool r32, bool re32, cudaStream_t s, bool x_zero, const double* tolv,
                        bool precond_rel) {
    const int rows = F.rows_in();
    const size_t n = size_t(rows) * M;
    const int restart = std::max(1, std::min(rows, opt.restart));
    V_.ensure(sizeof(double2) * n * (restart + 1));
    H_.ensure(sizeof(double2) * size_t(M) * (restart + 1) * restart);
    g_.ensure(sizeof(double2) * size_t(M) * (restart + 1));
    cs_.ensure(sizeof(double) * size_t(M) * restart);
    sn_.ensure(sizeof(double2) * size_t(M) * restart);
    y_.ensure(sizeof(double2) * size_t(M) * restart);
    h_.ensure(sizeof(double2) * size_t(M) * (restart + 1));
    h2_.ensure(sizeof(double2) * size_t(M) * (restart + 1));
    bnorm_.ensure(sizeof(double) * M);
    rnorm_.ensure(sizeof(double) * M * 2);
    state_.ensure(sizeof(GState) * M + sizeof(int) * M);
    w_.ensure(sizeof(double2) * n);
    r_.ensure(sizeof(double2) * n);
    bj_.ensure(sizeof(double2) * n);
    flagdev_.ensure(sizeof(int) * (M + 2));   // count, M column flags
    cur_cols_.clear();  // self coefficients may differ from the previous call
    double2* V = V_.as<double2>();
    GState* gs = state_.as<GState>();
    int* kper = reinterpret_cast<int*>(gs + M);
    int* dflag = flagdev_.as<int>();
    const int mb = nblk(M, 128);
    const int vb = nblk((long long)n, 256);

    norms(b, rows, M, bnorm_.as<double>(), s);
    k_gm_init<<<mb, 128, 0, s>>>(gs, bnorm_.as<double>(), M);
    MPM_LAUNCH();
    k_zero_rhs_cols<<<vb, 256, 0, s>>>(x, bnorm_.as<double>(), n, M);
    MPM_LAUNCH();
    const double2* bj = b;
    if (opt.jacobi) {
        k_jacobi<<<vb, 256, 0, s>>>(b, bj_.as<double2>(), F.num_particles(), F.num_quads(), M, F.quad_idx_dev(), sc);
        MPM_LAUNCH();
        bj = bj_.as<double2>();
        if (precond_rel) norms(bj, rows, M, bnorm_.as<double>(), s);
    }
    // columns cycling at the start of the current cycle (empty: all)
    std::vector<int> begin_cols;
    bool first = true;
    while (true) {
        // r = D^-1 (b - A x), for the columns that cycled last time
        if (first && x_zero) {
            MPM_CUDA(cudaMemcpyAsync(r_.p, bj, sizeof(double2) * n, cudaMemcpyDeviceToDevice, s));
        } else {
            st.column_matvecs += apply_cols(F, x, w_.as<double2>(), M, sc, opt.jacobi, r32, re32,
                                            begin_cols.empty() ? nullptr : begin_cols.data(), opt.compact, s);
            st.matvecs++;
            k_sub<<<vb, 256, 0, s>>>(bj, w_.as<double2>(), r_.as<double2>(), n);
            MPM_LAUNCH();
        }
        first = false;
        norms(r_.as<double2>(), rows, M, rnorm_.as<double>(), s);
        MPM_CUDA(cudaMemsetAsync(dflag, 0, sizeof(int), s));
        k_gm_begin<<<mb, 128, 0, s>>>(gs, rnorm_.as<double>(), bnorm_.as<double>(), opt.tol, tolv, opt.maxiter,
                                      restart, g_.as<double2>(), M, dflag);
        MPM_LAUNCH();
        k_normalize<<<vb, 256, 0, s>>>(r_.as<double2>(), V, rnorm_.as<double>(), gs, n, M);
        MPM_LAUNCH();
        if (read_flags(dflag, M, s) == 0) break;
        begin_cols.assign(flag_ + 1, flag_ + 1 + M);
        std::vector<int> cyc = begin_cols;
        for (int k = 0; k < restart; ++k) {
            double2* Vk = V + size_t(k) * n;
            double2* w = V + size_t(k + 1) * n;   // A V_k lands in V_{k+1}
            st.column_matvecs += apply_cols(F, Vk, w, M, sc, opt.jacobi, r32, re32, cyc.data(), opt.compact, s);
            st.matvecs++;
            HessArgs ha{H_.as<double2>(), g_.as<double2>(), cs_.as<double>(), sn_.as<double2>(), bnorm_.as<double>(),
                        opt.tol, tolv, opt.maxiter, restart, nullptr, rnorm_.as<double>(), dflag, poll_words(M), ++poll_seq_};
            arnoldi(V, k, rows, M, gs, ha, MemberArgs{}, s);
            st.reorth_steps++;
            // the count and the M column flags
            const int left = wait_flags(s);
            if (left == 0) break;
            cyc.assign(poll_.as<int>() + 2, poll_.as<int>() + 2 + M);
        }
        backsub(gs, H_.as<double2>(), g_.as<double2>(), y_.as<double2>(), restart, M, kper, s);
        k_vupdate<<<vb, 256, 0, s>>>(x, V, n, restart, y_.as<double2>(), rows, M, 1.0, kper);
        MPM_LAUNCH();
    }
    std::vector<GState> h(M);
    MPM_CUDA(cudaMemcpyAsync(h.data(), gs, sizeof(GState) * M, cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaStreamSynchronize(s));
    st.iters.resize(M);
    st.converged.resize(M);
    for (int m = 0; m < M; ++m) {
        st.iters[m] += h[m].iters;
        st.converged[m] = h[m].converged;
    }
}

bool BatchSolver::detect_shifts(const double2* b, const double2* sc, int rows, int N, int M, cudaStream_t s,
                                std::vector<int>& grp, std::vector<double2>& f) {
    if (M < 2 || M > 1024 || !sc) return false;
    shf_.ensure(sizeof(double2) * M);
    shflag_.ensure(sizeof(int) * (size_t(M) + size_t(M) * M));
    int* bad = shflag_.as<int>();
    int* eq = bad + M;
    MPM_CUDA(cudaMemsetAsync(eq, 0, sizeof(int) * size_t(M) * M, s));
    k_shift_ratio<<<M, 256, 0, s>>>(sc, N, M, shf_.as<double2>(), bad);
    MPM_LAUNCH();
    k_col_equal<<<dim3(M, M), 256, 0, s>>>(b, rows, M, eq);
    MPM_LAUNCH();
    std::vector<int> h(size_t(M) + size_t(M) * M);
    f.resize(M);
    MPM_CUDA(cudaMemcpyAsync(h.data(), bad, sizeof(int) * h.size(), cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaMemcpyAsync(f.data(), shf_.p, sizeof(double2) * M, cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaStreamSynchronize(s));
    for (int m = 0; m < M; ++m)
        if (h[m]) return false;
    grp.assign(M, -1);
    int G = 0;
    for (int m = 0; m < M; ++m) {
        for (int m2 = 0; m2 < m && grp[m] < 0; ++m2)
            if (h[M + size_t(m) * M + m2]) grp[m] = grp[m2];
        if (grp[m] < 0) grp[m] = G++;
    }
    return G < M;   // no shared right-hand side: nothing to gain
}

void BatchSolver::gmres_shifted(Field& F, const double2* b, double2* x, int M, const double2* sc,
                                const SolveOptions& opt, SolveStats& st, bool r32, bool re32, cudaStream_t s,
                                const double* tolv, const std::vector<int>& grp, const std::vector<double2>& f,
                                const int* skip, const int* live) {
    const int rows = F.rows_in(), N = F.num_particles();
    const int G = 1 + *std::max_element(grp.begin(), grp.end());
    const int restart = std::max(1, std::min(rows, opt.restart));
    const size_t ns = size_t(rows) * G;
    std::vector<int> seed(G, -1), zeros(G, 0);
    for (int m = 0; m < M; ++m)
        if (seed[grp[m]] < 0) seed[grp[m]] = m;
    std::vector<double2> sigma(M);
    for (int m = 0; m < M; ++m) sigma[m] = make_double2(f[m].x - 1.0, f[m].y);
    // device copies: member -> seed, seed columns, zero indices (ints), then
    // sigma (double2) at a 16-byte aligned offset
    const size_t sig_off = (sizeof(int) * (size_t(M) + 2 * G) + 15) & ~size_t(15);
    shmeta_.ensure(sig_off + sizeof(double2) * M);
    int* dgrp = shmeta_.as<int>();
    int* dseed = dgrp + M;
    int* dzero = dseed + G;
    double2* dsig = reinterpret_cast<double2*>(shmeta_.as<char>() + sig_off);
    MPM_CUDA(cudaMemcpyAsync(dgrp, grp.data(), sizeof(int) * M, cudaMemcpyHostToDevice, s));
    MPM_CUDA(cudaMemcpyAsync(dseed, seed.data(), sizeof(int) * G, cudaMemcpyHostToDevice, s));
    MPM_CUDA(cudaMemcpyAsync(dzero, zeros.data(), sizeof(int) * G, cudaMemcpyHostToDevice, s));
    MPM_CUDA(cudaMemcpyAsync(dsig, sigma.data(), sizeof(double2) * M, cudaMemcpyHostToDevice, s));
    // seed operator: self coefficients c = sc[:, 0] for every seed, Jacobi
    // scaling: A0 = diag(c)^-1 G + I; seed right-hand sides diag(c)^-1 b
    shsc_.ensure(sizeof(double2) * size_t(N) * G);
    shb_.ensure(sizeof(double2) * ns * 2);
    double2* scs = shsc_.as<double2>();
    double2* sb = shb_.as<double2>();
    double2* sbj = sb + ns;
    k_gather_cols<<<nblk((long long)N * G, 256), 256, 0, s>>>(sc, M, scs, G, dzero, N);
    MPM_LAUNCH();
    k_gather_cols<<<nblk((long long)ns, 256), 256, 0, s>>>(b, M, sb, G, dseed, rows);
    MPM_LAUNCH();
    k_jacobi<<<nblk((long long)ns, 256), 256, 0, s>>>(sb, sbj, N, F.num_quads(), G, F.quad_idx_dev(), scs);
    MPM_LAUNCH();
    V_.ensure(sizeof(double2) * ns * (restart + 1));
    H_.ensure(sizeof(double2) * size_t(M) * (restart + 1) * restart);
    g_.ensure(sizeof(double2) * size_t(M) * (restart + 1));
    cs_.ensure(sizeof(double) * size_t(M) * restart);
    sn_.ensure(sizeof(double2) * size_t(M) * restart);
    y_.ensure(sizeof(double2) * size_t(M) * restart);
    h_.ensure(sizeof(double2) * size_t(G) * (restart + 1));
    h2_.ensure(sizeof(double2) * size_t(G) * (restart + 1));
    state_.ensure(sizeof(GState) * M + sizeof(int) * M);
    // seed states, seed cycling flags, then |b~| and |w'| per seed (8-byte aligned)
    const size_t bs_off = (sizeof(GState) * G + sizeof(int) * G + 7) & ~size_t(7);
    shst_.ensure(bs_off + 2 * sizeof(double) * G);
    rnorm_.ensure(sizeof(double) * std::max(M, G) * 2);
    flagdev_.ensure(sizeof(int) * (G + 2));
    cur_cols_.clear();
    double2* V = V_.as<double2>();
    GState* mst = state_.as<GState>();
    int* kper = reinterpret_cast<int*>(mst + M);
    GState* sst = shst_.as<GState>();
    int* scyc = reinterpret_cast<int*>(sst + G);
    double* bs = reinterpret_cast<double*>(shst_.as<char>() + bs_off);
    double* nu = bs + G;
    int* dflag = flagdev_.as<int>();
    norms(sbj, rows, G, bs, s);
    k_seed_init<<<nblk(G, 128), 128, 0, s>>>(sst, bs, G);
    MPM_LAUNCH();
    k_shift_init<<<nblk(M, 128), 128, 0, s>>>(mst, dgrp, bs, skip, g_.as<double2>(), restart, M);
    MPM_LAUNCH();
    k_normalize<<<nblk((long long)ns, 256), 256, 0, s>>>(sbj, V, bs, sst, ns, G);
    MPM_LAUNCH();
    std::vector<double> hbs(G);
    MPM_CUDA(cudaMemcpyAsync(hbs.data(), bs, sizeof(double) * G, cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaStreamSynchronize(s));
    std::vector<int> cyc(G);
    std::vector<int> used(G, live ? 0 : 1);
    for (int m = 0; m < M && live; ++m) used[grp[m]] |= live[m] != 0;
    for (int gi = 0; gi < G; ++gi) cyc[gi] = hbs[gi] > 0.0 && used[gi];
    for (int k = 0; k < restart; ++k) {
        if (std::count(cyc.begin(), cyc.end(), 1) == 0) break;
        double2* Vk = V + size_t(k) * ns;
        double2* w = V + size_t(k + 1) * ns;
        st.column_matvecs += apply_cols(F, Vk, w, G, scs, true, r32, re32, cyc.data(), opt.compact, s);
        st.matvecs++;
        HessArgs ha{H_.as<double2>(), g_.as<double2>(), cs_.as<double>(), sn_.as<double2>(), bs, opt.tol, nullptr,
                    opt.maxiter, restart, nu, rnorm_.as<double>(), dflag, poll_words(G), ++poll_seq_};
        arnoldi(V, k, rows, G, sst, ha, MemberArgs{mst, dsig, dgrp, M, tolv, scyc}, s);
        st.reorth_steps++;
        const int left = wait_flags(s);
        if (left == 0) break;
        cyc.assign(poll_.as<int>() + 2, poll_.as<int>() + 2 + G);
    }
    backsub(mst, H_.as<double2>(), g_.as<double2>(), y_.as<double2>(), restart, M, kper, s);
    k_shift_x<<<nblk((long long)rows * M, 256), 256, 0, s>>>(x, V, ns, G, y_.as<double2>(), dgrp, kper, skip, rows,
                                                             M);
    MPM_LAUNCH();
    std::vector<GState> h(M);
    MPM_CUDA(cudaMemcpyAsync(h.data(), mst, sizeof(GState) * M, cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaStreamSynchronize(s));
    st.iters.resize(M);
    st.converged.resize(M);
    for (int m = 0; m < M; ++m) {
        st.iters[m] += h[m].iters;
        st.converged[m] = h[m].converged;
    }
    st.shift_seeds = G;
}

void BatchSolver::bicgstab(Field& F, const double2* b, double2* x, int M, const double2* sc, const SolveOptions& opt,
                           SolveStats& st, bool r32, bool re32, cudaStream_t s, bool x_zero, const double* tolv,
                        bool precond_rel) {
    const int rows = F.rows_in();
    const size_t n = size_t(rows) * M;
    for (DevBuf* d : {&r0_, &p_, &v_, &s_, &t_, &r_, &w_, &bj_}) d->ensure(sizeof(double2) * n);
    bnorm_.ensure(sizeof(double) * M);
    rnorm_.ensure(sizeof(double) * M * 2);
    scal_.ensure(sizeof(BState) * M + sizeof(int) * M);
    h_.ensure(sizeof(double2) * M * 2);
    flagdev_.ensure(sizeof(int) * (M + 1));
    cur_cols_.clear();
    BState* bs = scal_.as<BState>();
    int* mode = reinterpret_cast<int*>(bs + M);
    int* dflag = flagdev_.as<int>();
    double2* hv = h_.as<double2>();
    const int mb = nblk(M, 128);
    const int vb = nblk((long long)n, 256);

    norms(b, rows, M, bnorm_.as<double>(), s);
    k_zero_rhs_cols<<<vb, 256, 0, s>>>(x, bnorm_.as<double>(), n, M);
    MPM_LAUNCH();
    const double2* bj = b;
    if (opt.jacobi) {
        k_jacobi<<<vb, 256, 0, s>>>(b, bj_.as<double2>(), F.num_particles(), F.num_quads(), M, F.quad_idx_dev(), sc);
        MPM_LAUNCH();
        bj = bj_.as<double2>();
        if (precond_rel) norms(bj, rows, M, bnorm_.as<double>(), s);
    }
    double2* r = r_.as<double2>();
    if (x_zero) {
        MPM_CUDA(cudaMemcpyAsync(r, bj, sizeof(double2) * n, cudaMemcpyDeviceToDevice, s));
    } else {
        F.apply(x, w_.as<double2>(), M, sc, opt.jacobi, r32, re32, s);
        st.matvecs++;
        st.column_matvecs += M;
        k_sub<<<vb, 256, 0, s>>>(bj, w_.as<double2>(), r, n);
        MPM_LAUNCH();
    }
    norms(r, rows, M, rnorm_.as<double>(), s);
    k_bi_init<<<mb, 128, 0, s>>>(bs, bnorm_.as<double>(), rnorm_.as<double>(), opt.tol, tolv, M);
    MPM_LAUNCH();
    MPM_CUDA(cudaMemcpyAsync(r0_.p, r, sizeof(double2) * n, cudaMemcpyDeviceToDevice, s));
    MPM_CUDA(cudaMemcpyAsync(p_.p, r, sizeof(double2) * n, cudaMemcpyDeviceToDevice, s));
    MPM_CUDA(cudaMemsetAsync(v_.p, 0, sizeof(double2) * n, s));
    MPM_CUDA(cudaMemsetAsync(dflag, 0, sizeof(int), s));
    k_bi_count<<<mb, 128, 0, s>>>(bs, dflag, M);
    MPM_LAUNCH();
    if (read_flags(dflag, M, s) > 0) {
        std::vector<int> act(flag_ + 1, flag_ + 1 + M);
        for (int it = 0; it < opt.maxiter; ++it) {
            dots(r0_.as<double2>(), 0, 1, r, rows, M, 0, hv, s);
            k_bi_a<<<mb, 128, 0, s>>>(bs, hv, it, M);
            MPM_LAUNCH();
            k_bi_p<<<vb, 256, 0, s>>>(p_.as<double2>(), v_.as<double2>(), r, bs, it, n, M);
            MPM_LAUNCH();
            st.column_matvecs += apply_cols(F, p_.as<double2>(), v_.as<double2>(), M, sc, opt.jacobi, r32, re32,
                                            act.data(), opt.compact, s);
            st.matvecs++;
            dots(r0_.as<double2>(), 0, 1, v_.as<double2>(), rows, M, 0, hv, s);
            k_bi_b<<<mb, 128, 0, s>>>(bs, hv, M);
            MPM_LAUNCH();
            k_bi_s<<<vb, 256, 0, s>>>(s_.as<double2>(), r, v_.as<double2>(), bs, n, M);
            MPM_LAUNCH();
            norms(s_.as<double2>(), rows, M, rnorm_.as<double>(), s);
            k_bi_c<<<mb, 128, 0, s>>>(bs, rnorm_.as<double>(), bnorm_.as<double>(), opt.tol, tolv, mode, M);
            MPM_LAUNCH();
            k_bi_xfinal<<<vb, 256, 0, s>>>(x, p_.as<double2>(), bs, mode, n, M);
            MPM_LAUNCH();
            st.column_matvecs += apply_cols(F, s_.as<double2>(), t_.as<double2>(), M, sc, opt.jacobi, r32, re32,
                                            act.data(), opt.compact, s);
            st.matvecs++;
            dots(t_.as<double2>(), 0, 1, s_.as<double2>(), rows, M, 1, hv, s);
            dots(t_.as<double2>(), 0, 1, t_.as<double2>(), rows, M, 1, hv + M, s);
            k_bi_d<<<mb, 128, 0, s>>>(bs, hv, hv + M, M);
            MPM_LAUNCH();
            k_bi_xr<<<vb, 256, 0, s>>>(x, r, p_.as<double2>(), s_.as<double2>(), t_.as<double2>(), bs, n, M);
            MPM_LAUNCH();
            norms(r, rows, M, rnorm_.as<double>(), s);
            MPM_CUDA(cudaMemsetAsync(dflag, 0, sizeof(int), s));
            k_bi_e<<<mb, 128, 0, s>>>(bs, rnorm_.as<double>(), bnorm_.as<double>(), opt.tol, tolv, opt.maxiter, dflag,
                                      M);
            MPM_LAUNCH();
            if (read_flags(dflag, M, s) == 0) break;
            act.assign(flag_ + 1, flag_ + 1 + M);
        }
    }
    std::vector<BState> h(M);
    MPM_CUDA(cudaMemcpyAsync(h.data(), bs, sizeof(BState) * M, cudaMemcpyDeviceToHost, s));
    MPM_CUDA(cudaStreamSynchronize(s));
    st.iters.resize(M);
    st.converged.resize(M);
    for (int m = 0; m < M; ++m) {
        st.iters[m] += h[m].iters;
        st.converged[m] = h[m].converged;
    }
}

void BatchSolver::solve(Field& F, const double2* b, double2* x, int M, const double2* sc, const SolveOptions& opt,
                        SolveStats& st, cudaStream_t s) {
    st.iters.assign(M, 0);
    st.converged.assign(M, 0);
    st.matvecs = 0;
    st.column_matvecs = 0;
    st.refine_steps = 0;
    st.reorth_steps = 0;
    st.shift_seeds = 0;
    st.fp64_matvecs = 0;
    if (!opt.refine) {
        if (opt.method == SOLVER_BICGSTAB) bicgstab(F, b, x, M, sc, opt, st, opt.recip_fp32, opt.real_fp32, s);
        else gmres(F, b, x, M, sc, opt, st, opt.recip_fp32, opt.real_fp32, s);
        return;
    }
    // Mixed-precision iterative refinement: fp64 true residual outside,
    // fp32 operator inside.
    const int rows = F.rows_in();
    const size_t n = size_t(rows) * M;
    xr_.ensure(sizeof(double2) * n);
    d_.ensure(sizeof(double2) * n);
    bn2_.ensure(sizeof(double) * M);
    rn2_.ensure(sizeof(double) * M);
    convd_.ensure(sizeof(int) * M);
    double* bn2 = bn2_.as<double>();
    double* rn2 = rn2_.as<double>();
    int* convd = convd_.as<int>();
    const int vb = nblk((long long)n, 256);
    norms(b, rows, M, bn2, s);
    MPM_CUDA(cudaMemsetAsync(convd, 0, sizeof(int) * M, s));
    SolveOptions in = opt;
    in.refine = false;
    const double floor = opt.inner_tol > 0.0 ? opt.inner_tol : 1e-4;
    in.tol = 0.5;
    tolv_.ensure(sizeof(double) * M);
    std::vector<int> conv(M, 0), act(M, 1);
    st.rel_resid.assign(M, 0.0);
    cur_cols_.clear();
    // Shifted structure (one particle profile of self coefficients, shared
    // right-hand sides: a frequency sweep of one material): the first
    // correction is solved from x = 0 for all columns at once on the seeds'
    // Krylov spaces; later corrections are per column.
    std::vector<int> grp;
    std::vector<double2> fsh;
    // (quadrupole rows carry 2.5 s / a^2 + 0.5 g on the diagonal, which is
    // not a multiple of s: no shifted family with quadrupoles)
    const bool shifted = opt.shifted && opt.method == SOLVER_GMRES && F.num_quads() == 0 &&
                         detect_shifts(b, sc, rows, F.num_particles(), M, s, grp, fsh);
    bool reset = false;   // x replaced by the shifted solve from zero: every column active again
    std::vector<double> hb(M), hr(M);
    for (int step = 0; step < opt.max_refine; ++step) {
        // true residual of the columns not yet converged (a converged
        // column's x no longer changes).  The initial guess is screened with
        // the fp32 operator first: a column whose fp32 residual is above
        // 4 tol is not converged whatever the fp32 operator's error (about
        // 1e-7 relative), so only the columns below that take the fp64
        // residual; every later check is fp64 for all unconverged columns.
        const bool screen = step == 0 && !reset && opt.tol < 0.25;
        st.column_matvecs += apply_cols(F, x, xr_.as<double2>(), M, sc, false, screen, screen,
                                        step == 0 || reset ? nullptr : act.data(), opt.compact, s);
        reset = false;
        st.matvecs++;
        if (!screen) st.fp64_matvecs++;
        k_sub<<<vb, 256, 0, s>>>(b, xr_.as<double2>(), xr_.as<double2>(), n);
        MPM_LAUNCH();
        norms(xr_.as<double2>(), rows, M, rn2, s);
        if (screen) {
            MPM_CUDA(cudaMemcpyAsync(hb.data(), bn2, sizeof(double) * M, cudaMemcpyDeviceToHost, s));
            MPM_CUDA(cudaMemcpyAsync(hr.data(), rn2, sizeof(double) * M, cudaMemcpyDeviceToHost, s));
            MPM_CUDA(cudaStreamSynchronize(s));
            std::vector<int> near(M, 0);
            int nnear = 0;
            for (int m = 0; m < M; ++m) {
                near[m] = hr[m] <= 4.0 * opt.tol * hb[m];
                nnear += near[m];
            }
            if (nnear) {
                // fp64 residual of those columns into d_, swapped in
                st.column_matvecs += apply_cols(F, x, d_.as<double2>(), M, sc, false, false, false, near.data(),
                                                opt.compact, s);
                st.matvecs++;
                st.fp64_matvecs++;
                k_sub<<<vb, 256, 0, s>>>(b, d_.as<double2>(), d_.as<double2>(), n);
                MPM_LAUNCH();
                sel_.ensure(sizeof(int) * M);
                rn64_.ensure(sizeof(double) * M);
                norms(d_.as<double2>(), rows, M, rn64_.as<double>(), s);
                MPM_CUDA(cudaMemcpyAsync(sel_.p, near.data(), sizeof(int) * M, cudaMemcpyHostToDevice, s));
                k_take_cols<<<vb, 256, 0, s>>>(xr_.as<double2>(), d_.as<double2>(), rn2, rn64_.as<double>(),
                                               sel_.as<int>(), n, M);
                MPM_LAUNCH();
            }
        }
        k_conv_update<<<nblk(M, 128), 128, 0, s>>>(rn2, bn2, opt.tol, convd, M);
        MPM_LAUNCH();
        MPM_CUDA(cudaMemcpyAsync(hb.data(), bn2, sizeof(double) * M, cudaMemcpyDeviceToHost, s));
        MPM_CUDA(cudaMemcpyAsync(hr.data(), rn2, sizeof(double) * M, cudaMemcpyDeviceToHost, s));
        MPM_CUDA(cudaStreamSynchronize(s));
        int left = 0;
        for (int m = 0; m < M; ++m) {
            if (!act[m]) continue;  // converged in an earlier round
            st.rel_resid[m] = hb[m] > 0 ? hr[m] / hb[m] : 0.0;
            conv[m] = hr[m] <= opt.tol * hb[m];
            act[m] = !conv[m];
            left += act[m];
        }
        if (!left) break;
        double best = 1e300;
        int live_seeds = 0;
        if (shifted) {
            std::vector<char> seen(M, 0);
            for (int m = 0; m < M; ++m)
                if (act[m] && !seen[grp[m]]) {
                    seen[grp[m]] = 1;
                    ++live_seeds;
                }
        }
        for (int m = 0; m < M; ++m)
            if (act[m]) best = std::min(best, st.rel_resid[m]);
        if (step == 0 && shifted && (best >= 0.05 || left >= 8 * live_seeds)) {
            // a poor initial guess (every unconverged column's residual at
            // least 5% of |b|), or at least eight unconverged columns per
            // seed (the seeds' Krylov spaces cost a small part of per-column
            // solves even from x = 0): those columns start again from x = 0
            // and their first correction is solved on the seeds' Krylov
            // spaces; converged columns (a warm start) keep their x.  The
            // target is the outer one (half of it, no inner floor): the
            // seeds' GMRES works in fp64 on the fp32 operator, so its
            // residual estimate keeps falling below the fp32 operator error,
            // and a first correction this tight usually leaves nothing for
            // the per-column corrections but the fp64 check
            k_inner_tol<<<nblk(M, 128), 128, 0, s>>>(bn2, bn2, opt.tol, 0.0, tolv_.as<double>(), M);
            MPM_LAUNCH();
            SolveStats inner;
            inner.iters.assign(M, 0);
            gmres_shifted(F, b, x, M, sc, in, inner, true, true, s, tolv_.as<double>(), grp, fsh, convd,
                          act.data());
            for (int m = 0; m < M; ++m) st.iters[m] += inner.iters[m];
            st.matvecs += inner.matvecs;
            st.column_matvecs += inner.column_matvecs;
            st.reorth_steps += inner.reorth_steps;
            st.shift_seeds = inner.shift_seeds;
            st.refine_steps++;
            reset = true;
            continue;
        }
        k_mask_conv<<<vb, 256, 0, s>>>(xr_.as<double2>(), convd, n, M);
        MPM_LAUNCH();
        MPM_CUDA(cudaMemsetAsync(d_.p, 0, sizeof(double2) * n, s));
        k_inner_tol<<<nblk(M, 128), 128, 0, s>>>(rn2, bn2, opt.tol, floor, tolv_.as<double>(), M);
        MPM_LAUNCH();
        const double* tolv = tolv_.as<double>();
        SolveStats inner;
        inner.iters.assign(M, 0);
        if (opt.method == SOLVER_BICGSTAB)
            bicgstab(F, xr_.as<double2>(), d_.as<double2>(), M, sc, in, inner, true, true, s, true, tolv, true);
        else
            gmres(F, xr_.as<double2>(), d_.as<double2>(), M, sc, in, inner, true, true, s, true, tolv, true);
        k_axpy1<<<vb, 256, 0, s>>>(x, d_.as<double2>(), n);
        MPM_LAUNCH();
        for (int m = 0; m < M; ++m) st.iters[m] += inner.iters[m];
        st.matvecs += inner.matvecs;
        st.column_matvecs += inner.column_matvecs;
        st.reorth_steps += inner.reorth_steps;
        st.refine_steps++;
    }
    for (int m = 0; m < M; ++m) st.converged[m] = conv[m];
}

}  // namespace mpm
