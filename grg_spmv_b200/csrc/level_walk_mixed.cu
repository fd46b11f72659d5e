// The row walk over mixed storage (GRG_B200_MIXED, mixed.cuh): the kernels of walk_rows.cuh with
// rows of 6-byte values, FP64 sums, and any init.
//
// The walk is bound by instruction issue: a value costs four or five integer instructions (the words moved
// into a double's place), one FP32 fma (the test for infinities and NaN) and one FP64 fma, where the
// earlier format (a signed correction to a rounded FP32 value) took two conversions, the unit of
// the correction and a test, in kernels with per-segment sums and a second launch for heavy rows.
// 1.5M nodes, us: k = 32 up 1221 -> 605, down 1619 -> 647; k = 8 up 539 -> 329, down 748 -> 309.
#include "level_walk.h"
#include "mixed.cuh"
#include "walk_rows.cuh"

namespace {

// Four columns of a row as loaded (16-byte hi, 8-byte lo).  Eight columns a lane (32 and 16 bytes)
// spill at 64 registers: 1.5M nodes, k = 16, up 397 -> 440 us, down 418 -> 569.
constexpr int kMxCols = 4;

struct MxRaw {
    uint32_t hi[kMxCols];
    uint32_t lo[kMxCols / 2];  // two columns a word
};

__device__ __forceinline__ MxRaw mx_ld(const uint32_t* hi, const uint16_t* lo) {
    const uint4 h = ld_words4(hi);
    const uint2 l = ld_words2(lo);
    return MxRaw{{h.x, h.y, h.z, h.w}, {l.x, l.y}};
}

// Row named by a coded entry (hi and lo row starts); false when the entry is skipped.
template <bool UPONLY>
__device__ __forceinline__ bool mx_entry(const LevelArgs& a, uint32_t code, const uint32_t*& hi, const uint16_t*& lo) {
    const uint32_t src = (code >> GRG_B200_SRC_SHIFT) & GRG_B200_SRC_MASK;
    const uint32_t id = code & GRG_B200_ID_MASK;
    const void *h = a.state, *l = a.state_lo;
    int64_t lim = a.lim_state;
    int32_t bad = kErrStateId;
    if (src != GRG_B200_SRC_STATE) {
        if (UPONLY || src == GRG_B200_SRC_NULL || (src == GRG_B200_SRC_MISS && !a.use_miss)) return false;
        const bool miss = src == GRG_B200_SRC_MISS;
        h = miss ? a.miss : a.x;
        l = miss ? a.miss_lo : a.x_lo;
        lim = miss ? a.lim_miss : a.lim_x;
        bad = miss ? kErrMissId : kErrInputId;
    }
    if (a.err && id >= lim) {
        report(a.err, bad);
        return false;
    }
    const size_t off = static_cast<size_t>(id) * static_cast<uint32_t>(a.ld_state);  // encoded copies share the state's stride
    hi = static_cast<const uint32_t*>(h) + off;
    lo = static_cast<const uint16_t*>(l) + off;
    return true;
}

template <bool UPONLY>
struct MixedRows {
    using Value = double;
    using Acc = Pack<double, kMxCols>;
    static constexpr int kCols = kMxCols;
    static constexpr bool kUpOnly = UPONLY;
    static constexpr int kInFlight = 4;

    template <bool FAST, int N>
    static __device__ __forceinline__ void add_batch(const LevelArgs& a, const uint32_t (&code)[N], int c, Acc& acc) {
        MxRaw r[N];
        uint32_t any = 0;
#pragma unroll
        for (int u = 0; u < N; ++u) any |= code[u];
        if (FAST && a.err == nullptr && (any & (GRG_B200_SRC_MASK << GRG_B200_SRC_SHIFT)) == 0) {
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const size_t off = static_cast<size_t>(code[u] & GRG_B200_ID_MASK) * static_cast<uint32_t>(a.ld_state) + c;
                r[u] = mx_ld(static_cast<const uint32_t*>(a.state) + off, static_cast<const uint16_t*>(a.state_lo) + off);
            }
        } else {
#pragma unroll
            for (int u = 0; u < N; ++u) {
                const uint32_t* hi;
                const uint16_t* lo;
                r[u] = mx_entry<UPONLY>(a, code[u], hi, lo) ? mx_ld(hi + c, lo + c) : MxRaw{};
            }
        }
        // 0 unless a value is infinite or NaN, whose words are not the scaled double
        float special = 0.0f;
#pragma unroll
        for (int u = 0; u < N; ++u)
#pragma unroll
            for (int i = 0; i < kMxCols; ++i) special = __fmaf_rn(__uint_as_float(r[u].hi[i]), 0.0f, special);
        const double up = __longlong_as_double(kMxUpBits);
        if (special == 0.0f) {
#pragma unroll
            for (int u = 0; u < N; ++u)
#pragma unroll
                for (int i = 0; i < kMxCols; i += 2) {
                    const uint32_t l = r[u].lo[i / 2];
                    acc.v[i] = __fma_rn(mx_scaled<UPONLY>(r[u].hi[i], UPONLY ? l << 16 : (l << 13) & 0x1fffe000u), up, acc.v[i]);
                    acc.v[i + 1] = __fma_rn(mx_scaled<UPONLY>(r[u].hi[i + 1], UPONLY ? l & 0xffff0000u : (l >> 3) & 0x1fffe000u), up, acc.v[i + 1]);
                }
        } else {
#pragma unroll
            for (int u = 0; u < N; ++u)
#pragma unroll
                for (int i = 0; i < kMxCols; i += 2) {
                    const uint32_t l = r[u].lo[i / 2];
                    acc.v[i] = __dadd_rn(acc.v[i], mx_decode(r[u].hi[i], l & 0xffffu));
                    acc.v[i + 1] = __dadd_rn(acc.v[i + 1], mx_decode(r[u].hi[i + 1], l >> 16));
                }
        }
    }

    static __device__ __forceinline__ void store(const LevelArgs& a, int init_mode, int64_t row, int c, const Acc& acc) {
        const int64_t off = row * a.ld_state + c;
        Quad q{{acc.v[0], acc.v[1], acc.v[2], acc.v[3]}};
        if (init_mode != GRG_B200_INIT_NONE) {
            Quad init = mx_init(a, init_mode, row, c);
            add_quad(init, q);
            q = init;
        }
        mx_store(static_cast<uint32_t*>(a.state) + off, static_cast<uint16_t*>(a.state_lo) + off, q);
    }
};

}  // namespace

int launch_walk_mixed(const LevelArgs& la, int init_mode, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s) {
    // the walk's columns are 32-bit, and a lane may step one pass (up to 128 columns) past k
    if (la.ld_state >= (int64_t{1} << 32) || la.k > INT32_MAX - 256)
        return grg_fail(GRG_B200_ERR_UNSUPPORTED, "mixed storage: k = %lld or ld_state = %lld is too large", (long long)la.k, (long long)la.ld_state);
    return la.up ? launch_rows<MixedRows<true>, MixedRows<true>>(la, init_mode, num_entries, long_counts, pdl, s)
                 : launch_rows<MixedRows<false>, MixedRows<false>>(la, init_mode, num_entries, long_counts, pdl, s);
}
