// What the FP32/FP16 cell headers (csrc/lbm_fast_*.cuh) need to compile as plain C++ for the host
// checks: the intrinsics in their IEEE meaning, and names of the execution model that the checked
// functions do not use.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

using std::min;
struct HostThread {
    unsigned x = 0, y = 0, z = 0;
};
static HostThread threadIdx, blockIdx, blockDim, gridDim;
static inline float __fmaf_rn(float a, float b, float c) { return std::fma(a, b, c); }
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __uint_as_float(unsigned u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
template <class T>
static inline T __ldg(const T* p) {
    return *p;
}
static inline bool __all_sync(unsigned, bool x) { return x; }
static inline void __syncthreads() {}
static inline unsigned atomicInc(unsigned*, unsigned) { return 0; }
