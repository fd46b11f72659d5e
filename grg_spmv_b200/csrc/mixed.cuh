// Mixed storage (GRG_B200_MIXED): a value in 6 bytes, as an FP32 word and 16 further mantissa bits.
//
// hi is the sign, the 8-bit exponent and the leading 23 mantissa bits of the value, lo the next 16
// bits: with the implicit one, 40 significant bits, rounded to nearest even, so a stored value is
// within 2^-40 of the exact one relative to it, and integers up to 2^40 are exact.  Below 2^-126
// the spacing is 2^-165; from 2^128 on, infinities and NaN, hi is that FP32 value and lo is 0.
//
// The words are laid out so that decoding is integer shifts and one multiply-add: the bits moved
// into place make the double x 2^-896 (FP32's exponent field read as FP64's), for normal and
// subnormal values and zero alike, and the walk's fma scales it back while it adds.
#ifndef GRG_B200_MIXED_CUH
#define GRG_B200_MIXED_CUH

#include "level_common.cuh"

namespace grg {

constexpr long long kMxUpBits = (1023LL + 896) << 52;    // 2^896
constexpr long long kMxDownBits = (1023LL - 896) << 52;  // 2^-896

// The value x 2^-896 of finite words, lo in the upper half of `lo16` (FUNNEL: the 64 bits hi:lo16
// moved right by 3, the sign kept in place) or moved up by 13 already.  The funnel shift is the
// shorter of the two and makes up walks 4 to 6% faster (1.5M nodes, k = 32: 605 -> 581 us); in down
// walks, whose 64 registers are full, it made them 1 to 4% slower (k = 8: 309 -> 321 us).
template <bool FUNNEL>
__device__ __forceinline__ double mx_scaled(uint32_t hi, uint32_t lo) {
    return __hiloint2double(static_cast<int>((static_cast<int32_t>(hi) >> 3) & 0x8fffffff),
                            static_cast<int>(FUNNEL ? __funnelshift_r(lo, hi, 3) : (hi << 29) | lo));
}

__device__ __forceinline__ double mx_decode(uint32_t hi, uint32_t lo) {
    if ((hi & 0x7f800000u) == 0x7f800000u) return static_cast<double>(__uint_as_float(hi));
    return __dmul_rn(mx_scaled<true>(hi, lo << 16), __longlong_as_double(kMxUpBits));
}

__device__ __forceinline__ void mx_encode(double v, uint32_t& hi, uint32_t& lo) {
    const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(__dmul_rn(v, __longlong_as_double(kMxDownBits))));
    const uint32_t sign = static_cast<uint32_t>(bits >> 32) & 0x80000000u;
    unsigned long long m = bits & 0x7fffffffffffffffull;
    m = (m + 0xfffull + ((m >> 13) & 1)) >> 13;  // 8 + 39 bits, nearest even
    if (m >= (255ull << 39)) m = (v != v ? (511ull << 38) : (255ull << 39));  // NaN or infinity
    hi = sign | static_cast<uint32_t>(m >> 16);
    lo = static_cast<uint32_t>(m) & 0xffffu;
}

struct Quad {
    double v[4];
};

__device__ __forceinline__ Quad zero_quad() { return Quad{{0.0, 0.0, 0.0, 0.0}}; }

__device__ __forceinline__ void add_quad(Quad& a, const Quad& b) {
#pragma unroll
    for (int i = 0; i < 4; ++i) a.v[i] = a.v[i] + b.v[i];
}

// Four columns as a 16-byte hi and an 8-byte lo load or store.
__device__ __forceinline__ Quad mx_load(const uint32_t* hi_row, const uint16_t* lo_row) {
    const uint4 h = ld_words4(hi_row);
    const uint2 l = ld_words2(lo_row);
    return Quad{{mx_decode(h.x, l.x & 0xffffu), mx_decode(h.y, l.x >> 16), mx_decode(h.z, l.y & 0xffffu), mx_decode(h.w, l.y >> 16)}};
}

__device__ __forceinline__ void mx_store(uint32_t* hi_row, uint16_t* lo_row, const Quad& q) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) mx_encode(q.v[i], h[i], l[i]);
    *reinterpret_cast<uint4*>(hi_row) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint2*>(lo_row) = make_uint2(l[0] | (l[1] << 16), l[2] | (l[3] << 16));
}

// Columns [c, c + 4) of an FP64 row, columns >= k read as zero and not written: two 16-byte accesses
// where `vec` says that k, the stride and the base allow them.
__device__ __forceinline__ Quad f64_load(const double* row, int64_t c, int64_t k, bool vec) {
    Quad q;
    if (vec) {
        const Pack<double, 2> lo = ld_row<double, 2>(row + c), hi = ld_row<double, 2>(row + c + 2);
        return Quad{{lo.v[0], lo.v[1], hi.v[0], hi.v[1]}};
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) q.v[i] = c + i < k ? ld_row<double, 1>(row + c + i).v[0] : 0.0;
    return q;
}

__device__ __forceinline__ void f64_store(double* row, int64_t c, int64_t k, bool vec, const Quad& q) {
    if (vec) {
        st_pack(row + c, Pack<double, 2>{{q.v[0], q.v[1]}});
        st_pack(row + c + 2, Pack<double, 2>{{q.v[2], q.v[3]}});
        return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if (c + i < k) row[c + i] = q.v[i];
}

// Columns [c, c + 4) of a node's init value.
__device__ __forceinline__ Quad mx_init(const LevelArgs& a, int init_mode, int64_t row, int64_t c) {
    if (init_mode == GRG_B200_INIT_VECTOR) return f64_load(static_cast<const double*>(a.init_vector), c, a.k, false);
    if (init_mode == GRG_B200_INIT_XTX) {
        const double x = __ldg(static_cast<const double*>(a.xtx_node) + row);
        return Quad{{x, x, x, x}};
    }
    if (init_mode == GRG_B200_INIT_MATRIX) {
        const int64_t orig = __ldg(a.node_perm + row);
        if (a.err && (orig < 0 || orig >= a.lim_state)) {
            report(a.err, kErrPerm);
            return zero_quad();
        }
        return f64_load(static_cast<const double*>(a.init_matrix) + orig * a.ld_init, c, a.k, false);
    }
    return zero_quad();
}

}  // namespace grg

#endif  // GRG_B200_MIXED_CUH
