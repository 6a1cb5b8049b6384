// Shared device/host helpers for the cuMPM-B200 operator and solvers.
//
// Complex numbers are float2/double2 (interleaved re/im) so that buffers can
// be handed to cuFFT without copies.  Every multi-right-hand-side buffer in
// this library uses the "RHS-innermost" layout [row][M]: the M right-hand
// sides of one unknown are contiguous, which makes every per-particle access
// a coalesced M-wide vector.
#pragma once

#include <cuda_runtime.h>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>

namespace mpm {

// ---------------------------------------------------------------- errors --

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

inline void cuda_check(cudaError_t e, const char* what, const char* file, int line) {
    if (e != cudaSuccess) {
        throw CudaError(std::string("CUDA error: ") + cudaGetErrorString(e) + " in " + what + " at " +
                        file + ":" + std::to_string(line));
    }
}
#define MPM_CUDA(x) ::mpm::cuda_check((x), #x, __FILE__, __LINE__)

// Raises a kernel's dynamic shared-memory limit to at least `bytes` and never
// lowers it.  The limit is one attribute per kernel for the whole process:
// fields solved at once from several host threads share it, and a lower
// value set for one would make another's larger launch fail.
void raise_smem_limit(const void* kernel, size_t bytes);
template <typename K>
inline void set_smem_limit(K* kernel, size_t bytes) {
    raise_smem_limit(reinterpret_cast<const void*>(kernel), bytes);
}
// count one of this library's kernel launches and check it
void note_launch();
#define MPM_LAUNCH() (::mpm::note_launch(), ::mpm::cuda_check(cudaGetLastError(), "kernel launch", __FILE__, __LINE__))

// Host data for kernels on any stream.  cudaMemcpy from pageable memory may
// return once the data are staged, and a stream made with
// cudaStreamNonBlocking does not wait for the legacy stream that carries them:
// uploads_done(), after the last of a set, waits for that stream.
inline void upload(void* dst, const void* src, size_t bytes) {
    MPM_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
}
inline void uploads_done() { MPM_CUDA(cudaStreamSynchronize(cudaStreamLegacy)); }

// --------------------------------------------------------------- complex --

template <typename R> struct CTraits;
template <> struct CTraits<float> { using T = float2; };
template <> struct CTraits<double> { using T = double2; };
template <typename R> using cplx = typename CTraits<R>::T;

template <typename R> __host__ __device__ __forceinline__ cplx<R> mk(R a, R b) {
    cplx<R> c; c.x = a; c.y = b; return c;
}
__host__ __device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ float2 operator*(float2 a, float s) { return make_float2(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ float2 operator*(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ void operator+=(float2& a, float2 b) { a.x += b.x; a.y += b.y; }
__host__ __device__ __forceinline__ void operator-=(float2& a, float2 b) { a.x -= b.x; a.y -= b.y; }
__host__ __device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__host__ __device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__host__ __device__ __forceinline__ double2 operator*(double2 a, double s) { return make_double2(a.x * s, a.y * s); }
__host__ __device__ __forceinline__ double2 operator*(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__host__ __device__ __forceinline__ void operator+=(double2& a, double2 b) { a.x += b.x; a.y += b.y; }
__host__ __device__ __forceinline__ void operator-=(double2& a, double2 b) { a.x -= b.x; a.y -= b.y; }

__host__ __device__ __forceinline__ double2 conjmul(double2 a, double2 b) {  // conj(a) * b
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

template <typename R> __device__ __forceinline__ cplx<R> to_r(double2 v);
template <> __device__ __forceinline__ float2 to_r<float>(double2 v) { return make_float2((float)v.x, (float)v.y); }
template <> __device__ __forceinline__ double2 to_r<double>(double2 v) { return v; }
__device__ __forceinline__ double2 to_d(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 to_d(double2 v) { return v; }

// fused multiply-add of a real weight into a complex accumulator
__device__ __forceinline__ void fma_rc(float2& acc, float w, float2 v) {
    acc.x = fmaf(w, v.x, acc.x); acc.y = fmaf(w, v.y, acc.y);
}
__device__ __forceinline__ void fma_rc(double2& acc, double w, double2 v) {
    acc.x = fma(w, v.x, acc.x); acc.y = fma(w, v.y, acc.y);
}

// positive modulo for grid indices
__host__ __device__ __forceinline__ int pmod(int a, int n) { int r = a % n; return r < 0 ? r + n : r; }

// signed cyclic distance a-b on a ring of n in (-n/2, n/2]
__host__ __device__ __forceinline__ int cyc_diff(int a, int b, int n) {
    int d = pmod(a - b, n);
    return (2 * d > n) ? d - n : d;
}

constexpr double kPi = 3.14159265358979323846;
constexpr long double kPiL = 3.14159265358979323846264338327950288L;   // (host)

// exp(2 pi i j / n), 0 <= j < n, to all digits of a double: from an angle of at
// most pi / 4 (one of up to 2 pi, rounded to a double, loses three bits)
inline double2 unit_root(long long j, long long n) {
    const long long q = 4 * j / n, r = 4 * j - q * n;     // quarters of a turn, and r / n of one
    const bool hi = 2 * r > n;
    const double x = double(kPiL / 2 * (hi ? n - r : r) / n);
    const double c = hi ? std::sin(x) : std::cos(x), s = hi ? std::cos(x) : std::sin(x);
    return q == 0 ? make_double2(c, s) : q == 1 ? make_double2(-s, c) : q == 2 ? make_double2(-c, -s)
                                                                               : make_double2(s, -c);
}

// --------------------------------------------------------------- buffers --

// device (or page-locked host) memory from / to the bounded cache of
// mpm_alloc.cpp; buf_free waits for the work that uses it, as cudaFree does
void* buf_alloc(size_t n, bool host);
void buf_free(void* p, bool host);

// Owning buffer; contents do not survive a growing ensure().
template <bool HOST>
struct Buffer {
    void* p = nullptr;
    size_t bytes = 0;
    Buffer() = default;
    Buffer(const Buffer&) = delete;
    Buffer& operator=(const Buffer&) = delete;
    ~Buffer() { release(); }
    void release() {
        if (p) buf_free(p, HOST);
        p = nullptr;
        bytes = 0;
    }
    void ensure(size_t n) {
        if (n <= bytes && p) return;
        release();
        if (n == 0) return;
        p = buf_alloc(n, HOST);
        bytes = n;
    }
    template <typename T> T* as() const { return static_cast<T*>(p); }
};
using DevBuf = Buffer<false>;
// Page-locked host buffer (reused across calls, so host<->device copies run
// at full PCIe/C2C speed and never fault fresh pages).
using HostBuf = Buffer<true>;

}  // namespace mpm
