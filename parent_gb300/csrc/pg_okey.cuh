// MI values as order-preserving integers, shared by the MIST kernels.
#pragma once

namespace pg {

// order-preserving image of a double; 0 is below every value. NaN maps to 0:
// it never beats anything, as no strict '>' with a NaN holds in the reference.
__device__ __forceinline__ unsigned long long okey(double x) {
    unsigned long long b = (unsigned long long)__double_as_longlong(x);
    if ((b & 0x7fffffffffffffffull) > 0x7ff0000000000000ull) return 0ull;  // NaN
    if (b == 0x8000000000000000ull) b = 0ull;  // -0 == +0
    return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double okey_value(unsigned long long k) {
    const unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
    return __longlong_as_double((long long)b);
}

}  // namespace pg
