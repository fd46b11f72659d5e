// The row walk of default-mode level launches: one kernel for every width k.
//
// A level is a gather-sum of random rows of k columns, bound by the latency of each row's chain
// (list extent, codes, rounds of row fetches) and by the L2 rate of the fetches, so lanes are
// handed out to keep independent fetches in flight:
//
//  * Columns: a row's k columns are cut into chunks of CW columns, 32 bytes where the buffers
//    allow it, and chunk lane w of the W chunks owns columns [w CW, w CW + CW).  W is any number
//    up to 32 (wider rows take several passes), not only a power of two: 32 / (W S) rows share a
//    warp and the lanes left over idle.
//  * Entries: a narrow row's lanes form S entry slots; slot e takes entries e (4 / S), ... of
//    every 4-entry quad and the slots' sums are added by shuffles in a fixed order.
//  * Heavy rows (the suffix) are walked by `heavy_warps` warps each, whose lane groups take
//    quads in turn; the partial sums are combined in a fixed order (shuffles, then shared
//    memory), so results are deterministic.
//  * Very long rows (a mutation hub can have 10^5 entries) are walked by a cluster of 8 CTAs each
//    (level_hub_kernel) and combined through distributed shared memory.
//
// Sums are reassociated against the reference's left-to-right order, as in every default-mode
// kernel: exact for integer-valued inputs.
#include "level_walk.h"
#include "walk_rows.cuh"

namespace {

// Columns [c, c + CW) of the row named by `code` (0 for padding and miss rows that are off).  XV:
// input and miss rows allow the vector load; otherwise their columns are loaded one by one.
template <typename T, bool UPONLY, int CW, bool XV>
__device__ __forceinline__ Pack<T, CW> fetch(const LevelArgs& a, uint32_t code, int c) {
    bool ok;
    const T* p = lean_source<T, UPONLY>(a, code, ok);
    if constexpr (!UPONLY && !XV && CW > 1) {
        if (ok && ((code >> GRG_B200_SRC_SHIFT) & GRG_B200_SRC_MASK) != GRG_B200_SRC_STATE) {
            Pack<T, CW> r;
#pragma unroll
            for (int i = 0; i < CW; ++i) r.v[i] = c + i < a.k ? ld_row<T, 1>(p + c + i).v[0] : T(0);
            return r;
        }
    }
    return ok ? ld_cols<T, CW>(p + c) : zero_pack<T, CW>();
}

// FP64 and FP32 rows.
template <typename T, bool UPONLY, int CW, bool XV>
struct PlainRows {
    using Value = T;
    using Acc = Pack<T, CW>;
    static constexpr int kCols = CW;
    static constexpr bool kUpOnly = UPONLY;
    static constexpr int kInFlight = CW * sizeof(T) == 32 ? 4 : 8;

    // The sum of N entries' columns, added to acc in order.  FAST: a batch that names state rows only
    // (most do) skips the choice of a source and the padding tests.  Down levels are bound by
    // instruction issue (82% of issue slots, 26% of L2 throughput on an all-heavy level at k = 8): the
    // traversal of 1.5M nodes went from 301 to 255 us.  Narrow up rows decode in two instructions
    // and go without (with it, 227 -> 253 us at k = 8).
    template <bool FAST, int N>
    static __device__ __forceinline__ void add_batch(const LevelArgs& a, const uint32_t (&code)[N], int c, Acc& acc) {
        Acc v[N];
        uint32_t any = 0;
#pragma unroll
        for (int u = 0; u < N; ++u) any |= code[u];
        if (FAST && (any & (GRG_B200_SRC_MASK << GRG_B200_SRC_SHIFT)) == 0) {
            const T* base = static_cast<const T*>(a.state) + c;
#pragma unroll
            for (int u = 0; u < N; ++u)
                v[u] = ld_cols<T, CW>(base + static_cast<size_t>(code[u] & GRG_B200_ID_MASK) * static_cast<uint32_t>(a.ld_state));
        } else {
#pragma unroll
            for (int u = 0; u < N; ++u) v[u] = fetch<T, UPONLY, CW, XV>(a, code[u], c);
        }
#pragma unroll
        for (int u = 0; u < N; ++u) add_into(acc, v[u]);
    }

    static __device__ __forceinline__ void store(const LevelArgs& a, int, int64_t row, int c, const Acc& acc) {
        st_pack(static_cast<T*>(a.state) + row * a.ld_state + c, acc);
    }
};

template <typename T, int CW, int HV>
int launch_dir(const LevelArgs& la, bool xv, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s) {
    constexpr int none = GRG_B200_INIT_NONE;
    if (la.up) return launch_rows<PlainRows<T, true, CW, true>, PlainRows<T, true, HV, true>>(la, none, num_entries, long_counts, pdl, s);
    if (CW == 1 || xv) return launch_rows<PlainRows<T, false, CW, true>, PlainRows<T, false, HV, true>>(la, none, num_entries, long_counts, pdl, s);
    return launch_rows<PlainRows<T, false, CW, false>, PlainRows<T, false, HV, false>>(la, none, num_entries, long_counts, pdl, s);
}

}  // namespace

bool walk_serves(const LevelArgs& la, int init_mode, bool exact) {
    return la.err == nullptr && !exact && init_mode == GRG_B200_INIT_NONE && la.list_align == 4 && la.k < (int64_t{1} << 24) &&
           la.ld_state < (int64_t{1} << 32) && la.ld_x < (int64_t{1} << 32) && la.ld_miss < (int64_t{1} << 32);
}

template <typename T>
int launch_walk(const LevelArgs& la, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s) {
    constexpr int C = Chunk32<T>::C;
    // the widest chunk that the call's state columns hold whole and that its rows align
    int cw = C;
    while (cw > 1 && (la.ld_state % cw != 0 || !aligned(la.state, cw * static_cast<int>(sizeof(T))) || la.k <= cw / 2 ||
                      (la.k + cw - 1) / cw * cw > la.state_cols))
        cw >>= 1;
    const int64_t cols = (la.k + cw - 1) / cw * cw;  // columns that whole chunks touch
    const bool xv = cols == la.k && la.ld_x % cw == 0 && aligned(la.x, cw * static_cast<int>(sizeof(T))) &&
                    (!la.use_miss || (la.ld_miss % cw == 0 && aligned(la.miss, cw * static_cast<int>(sizeof(T)))));
    if (cw == C) {
        // heavy rows: 16-byte lanes while a row fills few of them (down k = 8, 1.5M nodes: 244 us
        // against 253 with 32 bytes), 32-byte ones from four chunks (k = 16: 336 -> 330 us, k = 32: 562 -> 551)
        if (la.k > 3 * C) return launch_dir<T, C, C>(la, xv, num_entries, long_counts, pdl, s);
        return launch_dir<T, C, C / 2>(la, xv, num_entries, long_counts, pdl, s);
    }
    if (cw == C / 2) return launch_dir<T, C / 2, C / 2>(la, xv, num_entries, long_counts, pdl, s);
    if constexpr (C == 8) {
        if (cw == 2) return launch_dir<T, 2, 2>(la, xv, num_entries, long_counts, pdl, s);
    }
    return launch_dir<T, 1, 1>(la, xv, num_entries, long_counts, pdl, s);
}

template int launch_walk<double>(const LevelArgs&, int64_t, const int64_t*, bool, cudaStream_t);
template int launch_walk<float>(const LevelArgs&, int64_t, const int64_t*, bool, cudaStream_t);
