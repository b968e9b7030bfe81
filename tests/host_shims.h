// The device functions' intrinsics for a host build of the headers (one ray,
// one lane), for the CPU tests of device code.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

static inline uint32_t __float_as_uint(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
static inline float __uint_as_float(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static inline int __float_as_int(float f) { return int(__float_as_uint(f)); }
static inline float __int_as_float(int i) { return __uint_as_float(uint32_t(i)); }
template <typename T> static inline T __ldg(const T* p) { return *p; }
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline int __popc(unsigned v) { return __builtin_popcount(v); }
static inline int __ffs(int v) { return __builtin_ffs(v); }
static inline int __clz(int v) { return v ? __builtin_clz(unsigned(v)) : 32; }
static inline bool __any_sync(unsigned, bool p) { return p; }
static inline uint32_t __byte_perm(uint32_t x, uint32_t y, uint32_t s) {
    uint64_t both = uint64_t(y) << 32 | x;
    uint32_t r = 0;
    for (int k = 0; k < 4; ++k) r |= uint32_t(both >> (8 * (s >> (4 * k) & 7u)) & 0xffu) << (8 * k);
    return r;
}
using std::isfinite;
using std::max;
using std::min;
