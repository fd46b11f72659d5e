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
#include <cooperative_groups.h>

#include "level_walk.h"

namespace cg = cooperative_groups;

namespace {

// Launch geometry of the walk (host-chosen, see launch_walk).
struct WalkShape {
    int32_t chunks;        // ceil(k / CW): chunk lanes of a row over all passes
    int32_t w;             // chunk lanes per pass
    int32_t slots;         // entry slots of a narrow row: 1, 2 or 4
    int32_t inv_group;     // 65536 / (w * slots), rounded up: lane / (w * slots) by multiplication
    int32_t inv_w;         // 65536 / w, rounded up
    int32_t rows_per_warp;
    int32_t short_rows_per_warp;  // 32 / w: rows of at most one quad take one slot
    int32_t heavy_blocks;  // CTAs [0, heavy_blocks) walk heavy rows
    int32_t long_blocks;   // the next long_blocks the narrow rows, the rest the short ones
    int32_t heavy_warps;   // warps per heavy row (divides the CTA's)
    int32_t hubs;          // leading heavy_rows left to level_hub_kernel
    int32_t hw;            // heavy rows: lanes of HV columns per pass
    int32_t inv_hw;
    int32_t groups;        // 32 / hw: lane groups of a warp
};

constexpr int kWalkWarps = 4;  // warps per CTA of level_walk_kernel

__device__ __forceinline__ int div_small(int x, int inv) { return (x * inv) >> 16; }  // x < 32

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
            for (int i = 0; i < CW; ++i) r.v[i] = c + i < a.k ? __ldg(p + c + i) : T(0);
            return r;
        }
    }
    return ok ? ld_cols<T, CW>(p + c) : zero_pack<T, CW>();
}

// The sum of N entries' columns, added to acc in order.  FAST: a batch that names state rows only
// (most do) skips the choice of a source and the padding tests.  Down levels are bound by
// instruction issue (82% of issue slots, 26% of L2 throughput on an all-heavy level at k = 8): the
// traversal of 1.5M nodes went from 301 to 255 us.  Narrow up rows decode in two instructions
// and go without (with it, 227 -> 253 us at k = 8).
template <typename T, bool UPONLY, int CW, bool XV, bool FAST, int N>
__device__ __forceinline__ void add_batch(const LevelArgs& a, const uint32_t (&code)[N], int c, Pack<T, CW>& acc) {
    Pack<T, CW> v[N];
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

template <typename T, int V>
__device__ __forceinline__ Pack<T, V> shfl_down_pack(const Pack<T, V>& x, int off) {
    Pack<T, V> r;
#pragma unroll
    for (int i = 0; i < V; ++i) r.v[i] = __shfl_down_sync(kFullMask, x.v[i], off);
    return r;
}

// This slot's 4 / S codes of a quad.
template <int S>
struct SlotCodes {
    uint32_t c[4 / S];
};

template <int S>
__device__ __forceinline__ SlotCodes<S> ld_codes(const uint32_t* entries, int32_t quad, int e) {
    SlotCodes<S> r;
    if constexpr (S == 1) {
        const uint4 q = __ldg(reinterpret_cast<const uint4*>(entries) + quad);
        r.c[0] = q.x;
        r.c[1] = q.y;
        r.c[2] = q.z;
        r.c[3] = q.w;
    } else if constexpr (S == 2) {
        const uint2 q = __ldg(reinterpret_cast<const uint2*>(entries) + 2 * quad + e);
        r.c[0] = q.x;
        r.c[1] = q.y;
    } else {
        r.c[0] = __ldg(entries + 4 * quad + e);
    }
    return r;
}

template <int S>
__device__ __forceinline__ SlotCodes<S> null_codes() {
    SlotCodes<S> r;
#pragma unroll
    for (int i = 0; i < 4 / S; ++i) r.c[i] = GRG_B200_SRC_NULL << GRG_B200_SRC_SHIFT;
    return r;
}

// Narrow rows with S entry slots.  The list is static, so its extent and the codes of its first
// 2 S quads (8 codes a lane) are loaded before the wait on the previous level.
template <typename T, bool UPONLY, int CW, bool XV, int NW, int S, int LB>
__device__ __forceinline__ void walk_rows(const LevelArgs& a, const WalkShape& ws, int64_t block, int64_t first, int64_t end,
                                          int rows_per_warp, int inv_group) {
    constexpr int PQ = 2 * S;      // quads whose codes are loaded up front
    constexpr int NC = 4 / S;      // codes of a quad per slot
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int r = div_small(lane, inv_group);
    const int in_row = lane - r * (ws.w * S);
    const int e = S == 1 ? 0 : div_small(in_row, ws.inv_w);
    const int w = in_row - e * ws.w;
    const int64_t pos = first + (block * NW + warp) * rows_per_warp + r;
    const bool live = r < rows_per_warp && pos < end;  // other lanes still join the shuffles
    int32_t q0 = 0, q1 = 0;
    int64_t row = 0;
    SlotCodes<S> pre[PQ];
#pragma unroll
    for (int j = 0; j < PQ; ++j) pre[j] = null_codes<S>();
    if (live) {
        q0 = __ldg(a.row_ptr + pos) >> 2;
        q1 = __ldg(a.row_ptr + pos + 1) >> 2;
        row = level_row(a, pos);
#pragma unroll
        for (int j = 0; j < PQ; ++j)
            if (q0 + j < q1) pre[j] = ld_codes<S>(a.entries, q0 + j, e);
    }
    pdl_wait();
    for (int c0 = 0; c0 < ws.chunks; c0 += ws.w) {  // one pass up to 32 chunks
        const bool on = c0 + w < ws.chunks;
        const int c = (c0 + w) * CW;
        Pack<T, CW> acc = zero_pack<T, CW>();
        if (on) {
#pragma unroll
            for (int t = 0; t < PQ * NC; t += LB) {  // LB fetches in flight
                if (q0 + t / NC < q1) {
                    uint32_t code[LB];
#pragma unroll
                    for (int u = 0; u < LB; ++u) code[u] = pre[(t + u) / NC].c[(t + u) % NC];
                    add_batch<T, UPONLY, CW, XV, !UPONLY>(a, code, c, acc);
                }
            }
            constexpr int LT = LB < 4 ? LB : 4;
            for (int32_t q = q0 + PQ; q < q1; q += S) {
                SlotCodes<S> cur[S];
#pragma unroll
                for (int j = 0; j < S; ++j) cur[j] = q + j < q1 ? ld_codes<S>(a.entries, q + j, e) : null_codes<S>();
#pragma unroll
                for (int t = 0; t < 4; t += LT) {
                    uint32_t code[LT];
#pragma unroll
                    for (int u = 0; u < LT; ++u) code[u] = cur[(t + u) / NC].c[(t + u) % NC];
                    add_batch<T, UPONLY, CW, XV, !UPONLY>(a, code, c, acc);
                }
            }
        }
        if constexpr (S == 4) add_into(acc, shfl_down_pack(acc, 2 * ws.w));
        if constexpr (S >= 2) add_into(acc, shfl_down_pack(acc, ws.w));
        if (live && e == 0 && on) st_pack(static_cast<T*>(a.state) + row * a.ld_state + c, acc);
    }
}

// This lane group's part of a heavy row: quads first, first + stride, ... of [.., q1), columns
// [c, c + HV), the next quad's codes loaded while the current one's rows are fetched.
template <typename T, bool UPONLY, int HV, bool XV>
__device__ __forceinline__ Pack<T, HV> heavy_part(const LevelArgs& a, int32_t first, int32_t q1, int32_t stride, int c, bool on) {
    const uint4* codes4 = reinterpret_cast<const uint4*>(a.entries);
    const uint32_t null_code = GRG_B200_SRC_NULL << GRG_B200_SRC_SHIFT;
    const uint4 null4 = make_uint4(null_code, null_code, null_code, null_code);
    Pack<T, HV> part = zero_pack<T, HV>();
    if (!on) return part;
    uint4 cur = first < q1 ? __ldg(codes4 + first) : null4;
    for (int32_t q = first; q < q1; q += stride) {
        const uint4 nxt = q + stride < q1 ? __ldg(codes4 + q + stride) : null4;
        const uint32_t code[4] = {cur.x, cur.y, cur.z, cur.w};
        add_batch<T, UPONLY, HV, XV, true>(a, code, c, part);
        cur = nxt;
    }
    return part;
}

// Adds the lane groups' parts (groups of hw lanes) into group 0, in a fixed order.
template <typename T, int HV>
__device__ __forceinline__ void reduce_groups(Pack<T, HV>& part, int grp, int groups, int hw) {
    for (int n = groups; n > 1;) {
        const int h = (n + 1) >> 1;
        const Pack<T, HV> other = shfl_down_pack(part, h * hw);
        if (grp + h < n) add_into(part, other);
        n = h;
    }
}

// Heavy rows, heavy_warps warps each.
template <typename T, bool UPONLY, int HV, bool XV, int NW>
__device__ __forceinline__ void walk_heavy(const LevelArgs& a, const WalkShape& ws, int64_t block) {
    extern __shared__ __align__(32) unsigned char heavy_smem[];  // with heavy_warps > 1: NW x 32 packs
    Pack<T, HV>(*red)[32] = reinterpret_cast<Pack<T, HV>(*)[32]>(heavy_smem);
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int rows_per_cta = NW / ws.heavy_warps;
    const int sub = warp % ws.heavy_warps;  // this warp's turn inside its row
    const int64_t h = ws.hubs + block * rows_per_cta + warp / ws.heavy_warps;
    const int grp = div_small(lane, ws.inv_hw);
    const int gl = lane - grp * ws.hw;
    const bool live = h < a.num_heavy && grp < ws.groups;
    int32_t qs = 0, q1 = 0;
    int64_t row = 0;
    if (live) {
        const int64_t pos = __ldg(a.heavy_rows + h);
        qs = __ldg(a.row_ptr + pos) >> 2;
        q1 = __ldg(a.row_ptr + pos + 1) >> 2;
        row = level_row(a, pos);
    }
    pdl_wait();
    const int k = static_cast<int>(a.k);
    for (int base = 0; base < k; base += HV * ws.hw) {  // one pass up to 32 lanes
        const int c = base + gl * HV;
        const bool on = live && c < k;
        Pack<T, HV> part = heavy_part<T, UPONLY, HV, XV>(a, qs + sub * ws.groups + grp, q1, ws.heavy_warps * ws.groups, c, on);
        reduce_groups(part, grp, ws.groups, ws.hw);
        if (ws.heavy_warps > 1) {  // uniform across the CTA
            if (grp == 0) red[warp][lane] = part;
            __syncthreads();
            if (sub == 0 && grp == 0)
                for (int i = 1; i < ws.heavy_warps; ++i) add_into(part, red[warp + i][lane]);
            __syncthreads();
        }
        if (on && sub == 0 && grp == 0) st_pack(static_cast<T*>(a.state) + row * a.ld_state + c, part);
    }
}

// A level's rows, hubs aside: narrow rows of more than one quad with S entry slots, LB fetches in
// flight per lane at 32 warps per SM (64 registers).  Against 2 in flight at 40 warps per SM:
// 1.5M nodes, k = 8: up 272 -> 242 us, down 312 -> 286; k = 1: up 214 -> 207, down 210 -> 197.
template <typename T, bool UPONLY, int CW, int HV, bool XV, int S, int LB>
__global__ void __launch_bounds__(32 * kWalkWarps, 32 / kWalkWarps) level_walk_kernel(LevelArgs a, WalkShape ws) {
    pdl_trigger();
    const int64_t narrow = a.num_rows - a.num_heavy;  // heavy positions form the suffix
    const int64_t long_end = narrow - a.short_rows;
    const int b = blockIdx.x;
    if (b < ws.heavy_blocks) walk_heavy<T, UPONLY, HV, XV, kWalkWarps>(a, ws, b);
    else if (b < ws.heavy_blocks + ws.long_blocks)
        walk_rows<T, UPONLY, CW, XV, kWalkWarps, S, LB>(a, ws, b - ws.heavy_blocks, 0, long_end, ws.rows_per_warp, ws.inv_group);
    else
        walk_rows<T, UPONLY, CW, XV, kWalkWarps, 1, LB>(a, ws, b - ws.heavy_blocks - ws.long_blocks, long_end, narrow, ws.short_rows_per_warp, ws.inv_w);
}

// Levels without narrow rows: 8 rows per CTA (neighbouring rows share an SM's L1).
template <typename T, bool UPONLY, int HV, bool XV>
__global__ void __launch_bounds__(256, HV * sizeof(T) > 16 ? 4 : 6) level_heavy_kernel(LevelArgs a, WalkShape ws) {
    pdl_trigger();
    walk_heavy<T, UPONLY, HV, XV, 8>(a, ws, blockIdx.x);
}

constexpr int kHubCtas = 8;    // CTAs of a cluster (portable size), one row each
constexpr int kHubWarps = 16;

// Very long rows, one cluster each: all 128 warps' lane groups take quads in turn, each CTA adds
// its warps' parts in warp order, and CTA 0 adds the CTAs' sums in rank order.
template <typename T, bool UPONLY, int HV, bool XV>
__global__ void __cluster_dims__(kHubCtas, 1, 1) __launch_bounds__(32 * kHubWarps) level_hub_kernel(LevelArgs a, WalkShape ws) {
    __shared__ Pack<T, HV> red[kHubWarps][32];
    __shared__ Pack<T, HV> total[32];
    pdl_trigger();
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = static_cast<int>(cluster.block_rank());
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int grp = div_small(lane, ws.inv_hw);
    const int gl = lane - grp * ws.hw;
    const int64_t pos = __ldg(a.heavy_rows + blockIdx.x / kHubCtas);
    const int32_t qs = __ldg(a.row_ptr + pos) >> 2;
    const int32_t q1 = __ldg(a.row_ptr + pos + 1) >> 2;
    const int64_t row = level_row(a, pos);
    pdl_wait();
    const int k = static_cast<int>(a.k);
    for (int base = 0; base < k; base += HV * ws.hw) {
        const int c = base + gl * HV;
        const bool on = grp < ws.groups && c < k;
        const int turn = (rank * kHubWarps + warp) * ws.groups + grp;
        Pack<T, HV> part = heavy_part<T, UPONLY, HV, XV>(a, qs + turn, q1, kHubCtas * kHubWarps * ws.groups, c, on);
        reduce_groups(part, grp, ws.groups, ws.hw);
        if (grp == 0) red[warp][lane] = part;
        __syncthreads();
        if (warp == 0 && grp == 0) {
            for (int i = 1; i < kHubWarps; ++i) add_into(part, red[i][lane]);
            total[lane] = part;
        }
        cluster.sync();
        if (rank == 0 && warp == 0 && grp == 0 && c < k) {
            for (int i = 1; i < kHubCtas; ++i) add_into(part, cluster.map_shared_rank(total, i)[lane]);
            st_pack(static_cast<T*>(a.state) + row * a.ld_state + c, part);
        }
        cluster.sync();  // the other CTAs' shared memory is read until here
    }
}

int ceil_div(int64_t a, int64_t b) { return static_cast<int>((a + b - 1) / b); }
int inverse16(int d) { return (65536 + d - 1) / d; }

constexpr int64_t kResidentWarps = 148 * 32;
constexpr int64_t kSlotWarps = 2 * kResidentWarps;

template <typename T, bool UPONLY, int CW, int HV, bool XV>
int launch_shape(const LevelArgs& la, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s) {
    WalkShape ws{};
    const int64_t narrow = la.num_rows - la.num_heavy;
    ws.chunks = ceil_div(la.k, CW);
    const int passes = ceil_div(ws.chunks, 32);
    ws.w = ceil_div(ws.chunks, passes);
    ws.inv_w = inverse16(ws.w);
    ws.short_rows_per_warp = 32 / ws.w;
    const int hlanes = ceil_div(la.k, HV);
    ws.hw = ceil_div(hlanes, ceil_div(hlanes, 32));
    ws.inv_hw = inverse16(ws.hw);
    ws.groups = 32 / ws.hw;
    const int64_t long_rows = narrow - la.short_rows;
    // Entry slots: as many as keep the level within two waves of resident warps.  More slots give
    // a row fewer rounds of fetches, which is what a level of one or two waves waits for; beyond
    // that they only cost instructions.  Whole traversals with 1 / 2 / 4 slots everywhere, us, FP64:
    //   1.5M nodes up k = 1: 250 / 207 / 160, k = 8: 382 / 242 / 267, k = 32: 517 / 549 / 791;
    //   5M nodes up k = 1: 419 / 303 / 371, k = 8: 617 / 617 / 802, k = 16: 945 / 1015 / 1407.
    ws.slots = 4;
    while (ws.slots > 1 && (ws.w * ws.slots > 32 || (long_rows * ws.slots + la.short_rows) * ws.w > 32 * kSlotWarps)) ws.slots >>= 1;
    ws.inv_group = inverse16(ws.w * ws.slots);
    ws.rows_per_warp = 32 / (ws.w * ws.slots);
    const bool only_heavy = narrow == 0;
    const int nw = only_heavy ? 8 : kWalkWarps;
    // Heavy rows: more warps a row while the rows alone leave the GPU idle.
    ws.heavy_warps = 1;
    while (ws.heavy_warps < nw && la.num_heavy * ws.heavy_warps * 2 <= kResidentWarps) ws.heavy_warps *= 2;
    // Rows left to one CTA must not outlast their level: those of 16 rounds of fetches and more, and
    // more than twice the level's own rounds per warp, go to clusters.  A 10,491-entry row at
    // k = 64 held one warp for 1477 us (the whole down traversal of 600k nodes: 2423 us, now 601).
    const int64_t level_rounds = num_entries / (4 * ws.groups) / kResidentWarps;
    for (int i = 0; i < GRG_B200_LONG_CLASSES && ws.hubs == 0; ++i) {
        const int64_t rounds = (int64_t{GRG_B200_LONG_ROW} << i) / (4 * ws.groups * ws.heavy_warps);
        if (rounds >= 16 && rounds > 2 * level_rounds) ws.hubs = static_cast<int>(long_counts[i]);
    }
    if (ws.hubs > 0)
        GRG_CUDA_TRY(launch_k(pdl, s, dim3(static_cast<unsigned>(ws.hubs * kHubCtas)), 32 * kHubWarps, level_hub_kernel<T, UPONLY, HV, XV>, la, ws));
    ws.heavy_blocks = ceil_div(la.num_heavy - ws.hubs, nw / ws.heavy_warps);
    if (only_heavy) {
        if (ws.heavy_blocks > 0)
            GRG_CUDA_TRY(launch_smem_k(pdl, s, dim3(static_cast<unsigned>(ws.heavy_blocks)), 256, ws.heavy_warps > 1 ? 8 * 32 * sizeof(Pack<T, HV>) : 0, level_heavy_kernel<T, UPONLY, HV, XV>, la, ws));
    } else {
        ws.long_blocks = ceil_div(ceil_div(long_rows, ws.rows_per_warp), nw);
        const int short_blocks = ceil_div(ceil_div(la.short_rows, ws.short_rows_per_warp), nw);
        const dim3 grid(static_cast<unsigned>(ws.heavy_blocks + ws.long_blocks + short_blocks));
        const size_t smem = ws.heavy_blocks > 0 && ws.heavy_warps > 1 ? kWalkWarps * 32 * sizeof(Pack<T, HV>) : 0;
        constexpr int LB = CW * sizeof(T) == 32 ? 4 : 8;
#define GRG_WALK(S) GRG_CUDA_TRY(launch_smem_k(pdl, s, grid, 32 * kWalkWarps, smem, level_walk_kernel<T, UPONLY, CW, HV, XV, S, LB>, la, ws))
        if (ws.slots == 4) GRG_WALK(4);
        else if (ws.slots == 2) GRG_WALK(2);
        else GRG_WALK(1);
#undef GRG_WALK
    }
    GRG_LAUNCH_CHECK("level_walk_kernel");
    return GRG_B200_OK;
}

template <typename T, int CW, int HV>
int launch_dir(const LevelArgs& la, bool xv, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s) {
    if (la.up) return launch_shape<T, true, CW, HV, true>(la, num_entries, long_counts, pdl, s);
    if constexpr (CW == 1) return launch_shape<T, false, CW, HV, true>(la, num_entries, long_counts, pdl, s);
    else return xv ? launch_shape<T, false, CW, HV, true>(la, num_entries, long_counts, pdl, s)
                   : launch_shape<T, false, CW, HV, false>(la, num_entries, long_counts, pdl, s);
}

}  // namespace

bool walk_serves(const LevelArgs& la, int init_mode, bool exact) {
    return la.err == nullptr && !exact && init_mode == GRG_B200_INIT_NONE && la.list_align == 4 && la.k < (int64_t{1} << 24) &&
           la.ld_state < (int64_t{1} << 32) && la.ld_x < (int64_t{1} << 32) && la.ld_miss < (int64_t{1} << 32);
}

template <typename T>
int launch_walk(const LevelArgs& la, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s) {
    constexpr int C = Chunk32<T>::C;
    // the widest chunk that the state rows hold whole (their padding columns are scratch) and align
    int cw = C;
    while (cw > 1 && (la.ld_state % cw != 0 || !aligned(la.state, cw * static_cast<int>(sizeof(T))) || (cw > 1 && la.k <= cw / 2))) cw >>= 1;
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
