// CUDA device functions compiled by the host compiler, for tests that run them on the CPU: the qualifiers vanish, the
// integer and floating-point intrinsics are restated, and anything that needs other threads ends the program.  Include
// it before the header under test, and build with -ffp-contract=off: the device code states its own fused operations.
#pragma once
#include <cuda_runtime.h>
#include <algorithm>
#include <bit>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#define __CUDACC__ 1
#define __noinline__

using std::max;
using std::min;

inline uint3 threadIdx{0, 0, 0}, blockIdx{0, 0, 0};

inline int __double2hiint(double d) { return int(std::bit_cast<uint64_t>(d) >> 32); }
inline double __hiloint2double(int hi, int lo) { return std::bit_cast<double>(uint64_t(uint32_t(hi)) << 32 | uint32_t(lo)); }
inline double __longlong_as_double(long long v) { return std::bit_cast<double>(v); }
inline uint32_t __byte_perm(uint32_t x, uint32_t y, uint32_t s) {      // selector nibbles 0-7
    const uint64_t v = uint64_t(y) << 32 | x;
    uint32_t r = 0;
    for (int k = 0; k < 4; k++) r |= uint32_t(v >> (8 * (s >> (4 * k) & 7)) & 255) << (8 * k);
    return r;
}
template <class T> T __ldg(const T *p) { return *p; }
inline float __fadd_rn(float a, float b) { return a + b; }
inline float __fsub_rn(float a, float b) { return a - b; }
inline float __fmul_rn(float a, float b) { return a * b; }
inline float __fdiv_rn(float a, float b) { return a / b; }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __dmul_rn(double a, double b) { return a * b; }

[[noreturn]] inline void other_threads() { fprintf(stderr, "a warp operation was reached on the host\n"); abort(); }
template <class T> T __shfl_sync(unsigned, T, int) { other_threads(); }
template <class T> T __shfl_xor_sync(unsigned, T, int) { other_threads(); }
inline unsigned __ballot_sync(unsigned, int) { other_threads(); }
inline int __any_sync(unsigned, int) { other_threads(); }
inline void __syncwarp() { other_threads(); }
