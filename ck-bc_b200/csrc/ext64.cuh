// Extended-range non-negative numbers in 64 bits, for shortest-path counts
// that overflow uint64 and double (a 2048 x 2048 grid has counts near 2^4088).
//
// Encoding: 0 is 0; otherwise bits 63..48 hold a biased exponent E (1..65535)
// and bits 47..0 the fraction f of a 49-bit significand M = 2^48 + f, value
// M * 2^(E - kExtBias) with kExtBias = 32768 + 48: values from about 2^-32815
// to 2^32816, 49 significant bits.  As unsigned integers the encodings order
// like the values, so 0 tests and comparisons need no decoding.  Every
// operation rounds to nearest, ties to even, on the 49-bit significand.
#pragma once
#include <stdint.h>

namespace bcg {

constexpr int kExtBias = 32768 + 48;
constexpr unsigned long long kExtOne = 0x8000000000000000ull;  // 1.0: E = 32768, f = 0
constexpr unsigned long long kExtFrac = (1ull << 48) - 1;

// s in [2^61, 2^63) stands for the value s * 2^(e - kExtBias - 13), its bit 0
// set where more bits follow below; rounds it to a 49-bit significand.  (No
// branch: the lanes of a warp round alike, and a chain of these operations is
// what a level of a deep search waits for.)
__host__ __device__ __forceinline__ unsigned long long ext_round(unsigned long long s, int e) {
    const int up = (int)(s >> 62), sh = 13 + up;
    const unsigned long long m = (s + ((1ull << (sh - 1)) - 1ull) + ((s >> sh) & 1ull)) >> sh;  // up to 2^49
    const int f = e + up + (int)(m >> 49);
    unsigned long long r = ((unsigned long long)(e + up) << 48) + (m - (1ull << 48));
    r = f > 65535 ? ~0ull : r;  // an exponent outside the encodable range saturates
    return f < 1 ? 0ull : r;
}

__host__ __device__ __forceinline__ unsigned long long ext_add(unsigned long long a, unsigned long long b) {
    const unsigned long long x = a < b ? b : a, y = a < b ? a : b;
    const int e = (int)(x >> 48), gap = e - (int)(y >> 48), d = gap < 63 ? gap : 63;
    const unsigned long long A = ((x & kExtFrac) | (1ull << 48)) << 13;
    const unsigned long long B = y ? ((y & kExtFrac) | (1ull << 48)) << 13 : 0ull;
    const unsigned long long t = B >> d;
    const unsigned long long r = ext_round((A + t) | ((t << d) != B ? 1ull : 0ull), e);
    return x ? r : 0ull;
}

__host__ __device__ __forceinline__ unsigned long long ext_mul(unsigned long long a, unsigned long long b) {
    const unsigned long long ma = (a & kExtFrac) | (1ull << 48), mb = (b & kExtFrac) | (1ull << 48);
#ifdef __CUDA_ARCH__
    const unsigned long long hi = __umul64hi(ma, mb), lo = ma * mb;
#else
    const unsigned __int128 p = (unsigned __int128)ma * mb;
    const unsigned long long hi = (unsigned long long)(p >> 64), lo = (unsigned long long)p;
#endif
    // p = ma * mb in [2^96, 2^98), value p * 2^(ea + eb - 2 bias); s = p >> 35 in
    // [2^61, 2^63) stands for s * 2^(e - bias - 13) (ext_round's scaling), so
    // e - bias - 13 = 35 + ea + eb - 2 bias, i.e. e = ea + eb - bias + 48
    const unsigned long long s = (hi << 29) | (lo >> 35) | ((lo & ((1ull << 35) - 1)) ? 1ull : 0ull);
    const unsigned long long r = ext_round(s, (int)(a >> 48) + (int)(b >> 48) - kExtBias + 48);
    return a && b ? r : 0ull;
}

// x > 0 finite double -> extended value x * 2^k.
__host__ __device__ __forceinline__ unsigned long long ext_from_double(double x, int k = 0) {
    if (!(x > 0.0)) return 0ull;
    int q;
#ifdef __CUDA_ARCH__
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    const int be = (int)(bits >> 52);
    if (be != 0) {  // a normal number: its fields are the significand and exponent
        q = be - 1022;
        return ext_round(((bits & ((1ull << 52) - 1)) | (1ull << 52)) << 9, q + k - 49 + kExtBias);
    }
#endif
    const double m = frexp(x, &q);  // x = m * 2^q, m in [0.5, 1)
    // 53-bit integer significand D = m * 2^53, x * 2^k = D * 2^(q - 53 + k);
    // s = D * 2^9 in [2^61, 2^62) stands for s * 2^(e - bias - 13), so
    // e = q + k - 49 + bias
    const unsigned long long D = (unsigned long long)ldexp(m, 53);
    return ext_round(D << 9, q + k - 49 + kExtBias);
}

// Extended value -> double (inf / 0 outside the double range).
__host__ __device__ __forceinline__ double ext_to_double(unsigned long long a) {
    if (!a) return 0.0;
    const unsigned long long m = (a & kExtFrac) | (1ull << 48);
#ifdef __CUDA_ARCH__
    // 49 bits fit a double's 53: inside its normal range the fields are moved over
    const int be = (int)(a >> 48) - kExtBias + 48 + 1023;
    if (be > 0 && be < 2047)
        return __longlong_as_double((long long)((unsigned long long)be << 52 | (a & kExtFrac) << 4));
#endif
    return ldexp((double)m, (int)(a >> 48) - kExtBias);
}

// num / value(a) for a double num > 0 and a != 0, as an extended value.
__host__ __device__ __forceinline__ unsigned long long ext_div(double num, unsigned long long a) {
    const unsigned long long m = (a & kExtFrac) | (1ull << 48);
    return ext_from_double(num / (double)m, kExtBias - (int)(a >> 48));
}

}  // namespace bcg
