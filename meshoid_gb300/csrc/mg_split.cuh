// FP64 values as sums of FP32 values, without the FP64 pipe: conversions and
// subtractions in FP64 run at 1/64 of the FP32 rate on this GPU, and the staging
// kernels that split every field were bound by them.  The same
// bits as h = (float)v, m = (float)(v - h), l = (float)(v - h - m).  Host and
// device: the CPU tests compare the two forms.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace mg {

__host__ __device__ __forceinline__ float split_bits_float(uint32_t b) {
#ifdef __CUDA_ARCH__
    return __uint_as_float(b);
#else
    float f;
    memcpy(&f, &b, 4);
    return f;
#endif
}

// hi = v rounded to FP32 and the remainder v - hi = rem * unit, exact: hi takes
// the 24 leading bits of the significand, rounded to nearest even; rem is what
// that leaves of the lower 29, |rem| <= 2^28.  False where the exponent leaves
// no room for every part as a normal FP32 value (zero, |v| outside 2^-70 ..
// 2^126, infinities, NaN): the caller splits in FP64.
__host__ __device__ __forceinline__ bool split_f64(double v, float &hi, int32_t &rem, float &unit) {
#ifdef __CUDA_ARCH__
    const uint32_t bh = (uint32_t)__double2hiint(v), bl = (uint32_t)__double2loint(v);
#else
    uint64_t b64;
    memcpy(&b64, &v, 8);
    const uint32_t bh = (uint32_t)(b64 >> 32), bl = (uint32_t)b64;
#endif
    const int e = (int)(bh >> 20 & 0x7ffu) - 1023;
    if (e < -70 || e > 125) return false;
    const uint32_t sign = bh & 0x80000000u;
    const uint32_t q = (bh << 3 & 0x7fffffu) | bl >> 29;  // 23 bits below the leading one
    const uint32_t r = bl & 0x1fffffffu, half = 1u << 28;
    const uint32_t up = r > half || (r == half && (q & 1u)) ? 1u : 0u;
    // a carry out of q raises the exponent, as it should
    hi = split_bits_float(sign | (((uint32_t)(e + 127) << 23) + q + up));
    const int32_t d = (int32_t)(r - (up << 29));
    rem = sign ? -d : d;
    unit = split_bits_float((uint32_t)(e - 52 + 127) << 23);
    return true;
}

// hi + lo = v to ~2^-48 |v|.
__host__ __device__ __forceinline__ void split2_f64(double v, float &hi, float &lo) {
    int32_t rem;
    float unit;
    if (split_f64(v, hi, rem, unit)) {
        lo = (float)rem * unit;  // the product with a power of two is exact
    } else {
        hi = (float)v;
        lo = (float)(v - (double)hi);
    }
}

// hi + mid + lo = v to ~2^-72 |v|.
__host__ __device__ __forceinline__ void split3_f64(double v, float &hi, float &mid, float &lo) {
    int32_t rem;
    float unit;
    if (split_f64(v, hi, rem, unit)) {
        const float m = (float)rem;
        mid = m * unit;
        lo = (float)(rem - (int32_t)m) * unit;
    } else {
        hi = (float)v;
        const double r = v - (double)hi;
        mid = (float)r;
        lo = (float)(r - (double)mid);
    }
}

}  // namespace mg
