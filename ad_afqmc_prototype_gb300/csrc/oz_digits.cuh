// Digits of binary64 values for exact products on the bf16 tensor cores, and
// the way back (k_ozgemm.cu describes the scheme; k_trotter_oz.cu uses it too).
#pragma once
#include "afq_internal.cuh"

namespace afq {

constexpr int OZ_S = 7;             // digits
constexpr int OZ_NAN = 0x7fffffff;  // scale of a row holding inf or nan
constexpr int OZ_KMAX = 65535;      // longest product: below 2^16 its integer sum stays below 2^62
constexpr int OZ_ZERO = -1022;      // scale of a row of zeros
constexpr int OZ_EMPTY = (int)0x80808080u;  // a maximum of nothing yet (bytes of one value: a memset makes it)

// a key that orders as |x| does (0 below 2^-1042)
__device__ __forceinline__ int oz_key(double x) { return __double2hiint(x) & 0x7fffffff; }
// scale of a row whose largest key is given: |x| < 2^E
__device__ __forceinline__ int oz_scale(int key) {
    return key >= 0x7ff00000 ? OZ_NAN : key == 0 ? OZ_ZERO : max(key >> 20, 1) - 1022;
}

// x 2^(55 - E) rounded to an integer, |.| <= 2^55, plus 0x808080808080, whose
// low six bytes are then the lower digits plus 128 (zero for subnormal x and
// in a row of scale OZ_NAN).
__device__ __forceinline__ long long oz_fix(double x, int E) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(x);
    const int eb = (int)((u >> 52) & 0x7ffu);
    long long y = 0;
    if (eb != 0 && E != OZ_NAN) {
        const unsigned long long m = (u & 0xfffffffffffffull) | (1ull << 52);
        const int r = E + 1020 - eb;  // right shift, >= -2
        if (r <= 0) y = (long long)(m << (-r));
        else if (r < 60) y = (long long)((m + (1ull << (r - 1))) >> r);
        if ((long long)u < 0) y = -y;
    }
    return y + 0x0000808080808080ll;
}
// digit s of y (from oz_fix) times 2^(-8 s), exact in fp32 and bf16
template <int S>
__device__ __forceinline__ float oz_dig(long long y) {
    constexpr float sc = 1.0f / (float)(1ull << (8 * S));
    if (S == 0) {  // the top digit, in [-128, 128]
        const uint32_t t = (uint32_t)((int)(y >> 48) + 256);
        return __uint_as_float(0x4B000000u | t) - 8388864.f;
    }
    const uint32_t t = (uint32_t)((unsigned long long)y >> (48 - 8 * S)) & 255u;
    return fmaf(__uint_as_float(0x4B000000u | t), sc, -8388736.f * sc);
}
__device__ __forceinline__ uint32_t oz_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *(const uint32_t*)&v;
}
template <int S>
__device__ __forceinline__ uint4 oz_pack8(const long long (&y)[8]) {
    return make_uint4(oz_pack(oz_dig<S>(y[0]), oz_dig<S>(y[1])), oz_pack(oz_dig<S>(y[2]), oz_dig<S>(y[3])),
                      oz_pack(oz_dig<S>(y[4]), oz_dig<S>(y[5])), oz_pack(oz_dig<S>(y[6]), oz_dig<S>(y[7])));
}

// What a product by digits may lose.  Its rows are held to 2^-55 of their largest entries, so its error scales with
// the largest entries of both operands, that of a binary64 chain with the terms: where large entries meet small ones
// only (rows graded in opposite directions, a sum that cancels) the chain is the better one.  Checked by its
// results, a walker (or a column) at a time: amax and bmax are the operands' largest scales there, and the product
// stands where some result reaches 2^-OZ_LOSS of 2^(amax + bmax), so that its error stays within about 2^-49 of
// the largest result, a chain's of a few hundred terms.  Otherwise, and with inf, nan or scales whose products come near
// the subnormals, the caller forms it again on the binary64 pipe.
constexpr int OZ_LOSS = 6;
// the larger part's key, and the exponent of a key
__device__ __forceinline__ int oz_key(double2 v) { return max(oz_key(v.x), oz_key(v.y)); }
__device__ __forceinline__ int oz_key_expo(int key) { return (key >> 20) - 1023; }
// the exponent that one result has to reach
__device__ __forceinline__ int oz_reach(int amax, int bmax) {
    return amax == OZ_NAN || bmax == OZ_NAN ? OZ_NAN : amax + bmax - OZ_LOSS;
}
__device__ __forceinline__ bool oz_lost(int amax, int bmax, bool reached) {
    if (amax == OZ_NAN || bmax == OZ_NAN) return true;
    if (amax <= OZ_ZERO || bmax <= OZ_ZERO) return false;  // zeros: so are the results
    return amax + bmax < -880 || !reached;
}
// whether one of n results, over the warp's lanes, reaches: mostly one of the first 32
__device__ __forceinline__ bool oz_scan(const double2* x, long long n, int reach) {
    for (long long i0 = 0; i0 < n; i0 += 32) {
        const long long i = i0 + (threadIdx.x & 31);
        if (__any_sync(0xffffffffu, i < n && oz_key_expo(oz_key(x[i])) >= reach)) return true;
    }
    return false;
}

// (acc 2^-32 + tail) 2^ex in binary64, rounded to nearest even, by integer
// operations (the binary64 pipe converts two a clock an SM): acc is shifted up
// until it or the tail's last bits fill 62 bits, and the tail added there.
__device__ __forceinline__ double oz_to_double(long long acc, float tail, int ex) {
    const unsigned long long am = acc < 0 ? 0ull - (unsigned long long)acc : (unsigned long long)acc;
    const int te = (int)((__float_as_uint(tail) >> 23) & 255u) - 127;  // |tail| < 2^(te + 1)
    const int sh = min(am ? __clzll((long long)am) - 2 : 62, 29 - te);
    const long long v = (long long)((unsigned long long)acc << sh) + __float2ll_rn(tail * __int_as_float((127 + 32 + sh) << 23));
    const unsigned long long sign = (unsigned long long)v & 0x8000000000000000ull;
    const unsigned long long mag = sign ? 0ull - (unsigned long long)v : (unsigned long long)v;
    if (mag == 0) return 0.0;
    const int lz = __clzll((long long)mag);
    const unsigned long long nrm = mag << lz;
    const unsigned long long m = (nrm >> 11) + (((nrm & 0x7ffull) + ((nrm >> 11) & 1ull)) > 0x400ull ? 1ull : 0ull);
    const int e = 63 - lz + ex - 32 - sh + 1023;
    if (e <= 0) return __longlong_as_double((long long)sign);
    const unsigned long long bits = ((unsigned long long)(e - 1) << 52) + m;  // m carries its leading bit
    if (e >= 2047) return __longlong_as_double((long long)(sign | 0x7ff0000000000000ull));
    return __longlong_as_double((long long)(sign | bits));
}

}  // namespace afq
