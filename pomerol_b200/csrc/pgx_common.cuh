// Common device/host helpers for libpgx (B200, sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>

#include "../../include/pgx.h"

namespace pgx {

// ---------------------------------------------------------------- complex
struct cd {
    double x, y;
};

__host__ __device__ __forceinline__ cd mk(double x, double y = 0.0) { return cd{x, y}; }
__host__ __device__ __forceinline__ cd operator+(cd a, cd b) { return cd{a.x + b.x, a.y + b.y}; }
__host__ __device__ __forceinline__ cd operator-(cd a, cd b) { return cd{a.x - b.x, a.y - b.y}; }
__host__ __device__ __forceinline__ cd operator*(cd a, cd b) {
    return cd{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x};
}
__host__ __device__ __forceinline__ cd operator*(cd a, double s) { return cd{a.x * s, a.y * s}; }
__host__ __device__ __forceinline__ cd operator*(double s, cd a) { return cd{a.x * s, a.y * s}; }
__host__ __device__ __forceinline__ cd conj(cd a) { return cd{a.x, -a.y}; }
__host__ __device__ __forceinline__ double abs2(cd a) { return a.x * a.x + a.y * a.y; }
// 1/a as conj(a)/|a|^2 (one real division).
__host__ __device__ __forceinline__ cd inv(cd a) {
    double r = 1.0 / abs2(a);
    return cd{a.x * r, -a.y * r};
}
__host__ __device__ __forceinline__ cd div(cd a, cd b) { return a * inv(b); }

#ifdef __CUDACC__
// 1/x by one third-order step y <- y + y (e + e^2), e = 1 - x y, which triples
// the number of correct bits (the Householder iteration of order three; Muller
// et al., "Handbook of Floating-Point Arithmetic", 2nd ed., sec. 4.7 for the
// family), seeded with the hardware's approximation (PTX rcp.approx.ftz.f64,
// about 20 bits): the error left is at the double rounding level.  Three FP64
// operations and no conversion, against four and two for a single-precision
// seed with two Newton-Raphson steps.  Valid where x and 1/x are normal.
__device__ __forceinline__ double recip_iter(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
// |x| in [2^-1012, 2^1013), tested on the exponent field so that the FP64 pipe
// is left alone; the IEEE division covers the rest.
__device__ __forceinline__ bool recip_in_range(double x) {
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) - 0x00b00000u < 0x7e900000u;
}
__device__ __forceinline__ double recip_pos(double x) { return recip_in_range(x) ? recip_iter(x) : 1.0 / x; }
// 1/a = conj(a) / |a|^2 with recip_pos for the real reciprocal.
__device__ __forceinline__ cd inv_fast(cd a) {
    const double r = recip_pos(abs2(a));
    return cd{a.x * r, -a.y * r};
}
#endif

// Scalar-type helpers used by templated kernels (double or cd).
__host__ __device__ __forceinline__ cd tocd(double a) { return cd{a, 0.0}; }
__host__ __device__ __forceinline__ cd tocd(cd a) { return a; }
template <typename T> struct is_cd { static constexpr bool value = false; };
template <> struct is_cd<cd> { static constexpr bool value = true; };

// ------------------------------------------------------------ error plumbing
struct Error {
    int code;
    std::string msg;
};

#define PGX_CUDA(call)                                                                 \
    do {                                                                               \
        cudaError_t e_ = (call);                                                       \
        if (e_ != cudaSuccess)                                                         \
            throw ::pgx::Error{PGX_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)}; \
    } while (0)

#define PGX_CHECK(cond, code, text)                                 \
    do {                                                            \
        if (!(cond)) throw ::pgx::Error{(code), std::string(text)}; \
    } while (0)

// Kernel launches issued by this library (process-wide).
long long& launch_counter();

inline void check_launch(const char* what) {
    ++launch_counter();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error{PGX_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e)};
}

inline int ceil_div(long a, long b) { return int((a + b - 1) / b); }

}  // namespace pgx
