// log2 of x >= 0 in FP32 (-inf for 0) from the bits of x, without FP64
// arithmetic on normal numbers: exponent exact, the top 23 mantissa bits
// (truncation: relative error < 2^-23, i.e. < 1.8e-7 in log2) through
// log2f (1 ulp), then the FP32 sum (<= 2^-14 for |result| < 2048). Ranks
// FP64 values before an exact FP64 evaluation of the near-best ones.
#pragma once

#include <cuda_runtime.h>
#include <math.h>

namespace cafe {

__device__ __forceinline__ float flog2(double x) {
    long long b = __double_as_longlong(x);
    if (b <= 0) return -INFINITY;   // +0 (and negative values, which never occur)
    int e = (int)((b >> 52) & 0x7ff);
    int bias = 1023;
    if (e == 0) {                   // subnormal: scale into the normal range
        b = __double_as_longlong(x * 0x1p64);
        e = (int)((b >> 52) & 0x7ff);
        bias += 64;
    }
    const float m = __int_as_float(0x3f800000 | (int)((b >> 29) & 0x7fffff));
    return (float)(e - bias) + log2f(m);
}

}  // namespace cafe
