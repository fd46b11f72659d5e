// The row walk's device code and launch, for any row storage.  A storage R has
//   Value, kCols, Acc = Pack<Value, kCols>   a lane's accumulator
//   kUpOnly                                  the lists name state rows and padding only
//   kInFlight                                fetches in flight per lane of a narrow row
//   add_batch<FAST>(a, codes, c, acc)        adds the columns [c, c + kCols) of each entry's row
//   store(a, init_mode, row, c, acc)         stores a row's sum (plus its init)
// The design is described in level_walk.cu.
#ifndef GRG_B200_WALK_ROWS_CUH
#define GRG_B200_WALK_ROWS_CUH

#include <cooperative_groups.h>

#include "level_common.cuh"

namespace {

namespace cg = cooperative_groups;

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
    int32_t init_mode;     // mixed storage: the init added to every row (grg_b200_init)
};

constexpr int kWalkWarps = 4;  // warps per CTA of level_walk_kernel

__device__ __forceinline__ int div_small(int x, int inv) { return (x * inv) >> 16; }  // x < 32

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

// The quads [q0, q1) of a narrow position: by arithmetic where the level's rows are in order of their
// quads, which takes the row pointers' latency off every CTA's way to its first fetch.
__device__ __forceinline__ void narrow_quads(const LevelArgs& a, int64_t pos, int32_t& q0, int32_t& q1) {
    if (a.quad_rows[0] > 0) {
        const int32_t p = static_cast<int32_t>(pos);
        q0 = 0;
        int32_t n = 0;
#pragma unroll
        for (int i = 0; i < GRG_B200_QUAD_CLASSES; ++i) {
            q0 += min(p, a.quad_rows[i]);
            n += p < a.quad_rows[i];
        }
        q1 = q0 + n;
    } else {
        q0 = __ldg(a.row_ptr + pos) >> 2;
        q1 = __ldg(a.row_ptr + pos + 1) >> 2;
    }
}

// Narrow rows with S entry slots.  The list is static, so its extent and the codes of its first
// 2 S quads (8 codes a lane) are loaded before the wait on the previous level.
template <class R, int NW, int S, int LB>
__device__ __forceinline__ void walk_rows(const LevelArgs& a, const WalkShape& ws, int64_t block, int64_t first, int64_t end,
                                          int rows_per_warp, int inv_group) {
    constexpr int PQ = 2 * S;      // quads whose codes are loaded up front
    constexpr int NC = 4 / S;      // codes of a quad per slot
    using Acc = typename R::Acc;
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
        narrow_quads(a, pos, q0, q1);
        row = level_row(a, pos);
#pragma unroll
        for (int j = 0; j < PQ; ++j)
            if (q0 + j < q1) pre[j] = ld_codes<S>(a.entries, q0 + j, e);
    }
    pdl_wait();
    for (int c0 = 0; c0 < ws.chunks; c0 += ws.w) {  // one pass up to 32 chunks
        const bool on = c0 + w < ws.chunks;
        const int c = (c0 + w) * R::kCols;
        Acc acc = zero_pack<typename R::Value, R::kCols>();
        if (on) {
#pragma unroll
            for (int t = 0; t < PQ * NC; t += LB) {  // LB fetches in flight
                if (q0 + t / NC < q1) {
                    uint32_t code[LB];
#pragma unroll
                    for (int u = 0; u < LB; ++u) code[u] = pre[(t + u) / NC].c[(t + u) % NC];
                    R::template add_batch<!R::kUpOnly>(a, code, c, acc);
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
                    R::template add_batch<!R::kUpOnly>(a, code, c, acc);
                }
            }
        }
        if constexpr (S == 4) add_into(acc, shfl_down_pack(acc, 2 * ws.w));
        if constexpr (S >= 2) add_into(acc, shfl_down_pack(acc, ws.w));
        if (live && e == 0 && on) R::store(a, ws.init_mode, row, c, acc);
    }
}

// This lane group's part of a heavy row: quads first, first + stride, ... of [.., q1), columns
// [c, c + kCols), the next quad's codes loaded while the current one's rows are fetched.
template <class R>
__device__ __forceinline__ typename R::Acc heavy_part(const LevelArgs& a, int32_t first, int32_t q1, int32_t stride, int c, bool on) {
    const uint4* codes4 = reinterpret_cast<const uint4*>(a.entries);
    const uint32_t null_code = GRG_B200_SRC_NULL << GRG_B200_SRC_SHIFT;
    const uint4 null4 = make_uint4(null_code, null_code, null_code, null_code);
    typename R::Acc part = zero_pack<typename R::Value, R::kCols>();
    if (!on) return part;
    uint4 cur = first < q1 ? __ldg(codes4 + first) : null4;
    for (int32_t q = first; q < q1; q += stride) {
        const uint4 nxt = q + stride < q1 ? __ldg(codes4 + q + stride) : null4;
        const uint32_t code[4] = {cur.x, cur.y, cur.z, cur.w};
        R::template add_batch<true>(a, code, c, part);
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
template <class R, int NW>
__device__ __forceinline__ void walk_heavy(const LevelArgs& a, const WalkShape& ws, int64_t block) {
    extern __shared__ __align__(32) unsigned char heavy_smem[];  // with heavy_warps > 1: NW x 32 packs
    using Acc = typename R::Acc;
    Acc(*red)[32] = reinterpret_cast<Acc(*)[32]>(heavy_smem);
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
    for (int base = 0; base < k; base += R::kCols * ws.hw) {  // one pass up to 32 lanes
        const int c = base + gl * R::kCols;
        const bool on = live && c < k;
        Acc part = heavy_part<R>(a, qs + sub * ws.groups + grp, q1, ws.heavy_warps * ws.groups, c, on);
        reduce_groups(part, grp, ws.groups, ws.hw);
        if (ws.heavy_warps > 1) {  // uniform across the CTA
            if (grp == 0) red[warp][lane] = part;
            __syncthreads();
            if (sub == 0 && grp == 0)
                for (int i = 1; i < ws.heavy_warps; ++i) add_into(part, red[warp + i][lane]);
            __syncthreads();
        }
        if (on && sub == 0 && grp == 0) R::store(a, ws.init_mode, row, c, part);
    }
}

// A level's rows, hubs aside: narrow rows of more than one quad with S entry slots, LB fetches in
// flight per lane at 32 warps per SM (64 registers).  Against 2 in flight at 40 warps per SM:
// 1.5M nodes, k = 8: up 272 -> 242 us, down 312 -> 286; k = 1: up 214 -> 207, down 210 -> 197.
template <class R, class H, int S, int LB>
__global__ void __launch_bounds__(32 * kWalkWarps, 32 / kWalkWarps) level_walk_kernel(LevelArgs a, WalkShape ws) {
    pdl_trigger();
    const int64_t narrow = a.num_rows - a.num_heavy;  // heavy positions form the suffix
    const int64_t long_end = narrow - a.short_rows;
    const int b = blockIdx.x;
    if (b < ws.heavy_blocks) walk_heavy<H, kWalkWarps>(a, ws, b);
    else if (b < ws.heavy_blocks + ws.long_blocks)
        walk_rows<R, kWalkWarps, S, LB>(a, ws, b - ws.heavy_blocks, 0, long_end, ws.rows_per_warp, ws.inv_group);
    else
        walk_rows<R, kWalkWarps, 1, LB>(a, ws, b - ws.heavy_blocks - ws.long_blocks, long_end, narrow, ws.short_rows_per_warp, ws.inv_w);
}

// Levels without narrow rows: 8 rows per CTA (neighbouring rows share an SM's L1).
template <class H>
__global__ void __launch_bounds__(256, sizeof(typename H::Acc) > 16 ? 4 : 6) level_heavy_kernel(LevelArgs a, WalkShape ws) {
    pdl_trigger();
    walk_heavy<H, 8>(a, ws, blockIdx.x);
}

constexpr int kHubCtas = 8;    // CTAs of a cluster (portable size), one row each
constexpr int kHubWarps = 16;

// Very long rows, one cluster each: all 128 warps' lane groups take quads in turn, each CTA adds
// its warps' parts in warp order, and CTA 0 adds the CTAs' sums in rank order.
template <class R>
__global__ void __cluster_dims__(kHubCtas, 1, 1) __launch_bounds__(32 * kHubWarps) level_hub_kernel(LevelArgs a, WalkShape ws) {
    using Acc = typename R::Acc;
    __shared__ Acc red[kHubWarps][32];
    __shared__ Acc total[32];
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
    for (int base = 0; base < k; base += R::kCols * ws.hw) {
        const int c = base + gl * R::kCols;
        const bool on = grp < ws.groups && c < k;
        const int turn = (rank * kHubWarps + warp) * ws.groups + grp;
        Acc part = heavy_part<R>(a, qs + turn, q1, kHubCtas * kHubWarps * ws.groups, c, on);
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
            R::store(a, ws.init_mode, row, c, part);
        }
        cluster.sync();  // the other CTAs' shared memory is read until here
    }
}

int ceil_div(int64_t a, int64_t b) { return static_cast<int>((a + b - 1) / b); }
int inverse16(int d) { return (65536 + d - 1) / d; }

constexpr int64_t kResidentWarps = 148 * 32;
constexpr int64_t kSlotWarps = 2 * kResidentWarps;

// Launches one level: its very long rows, if any, then every other row (R: narrow rows, H: heavy).
template <class R, class H>
int launch_rows(const LevelArgs& la, int init_mode, int64_t num_entries, const int64_t* long_counts, bool pdl, cudaStream_t s) {
    WalkShape ws{};
    ws.init_mode = init_mode;
    const int64_t narrow = la.num_rows - la.num_heavy;
    ws.chunks = ceil_div(la.k, R::kCols);
    const int passes = ceil_div(ws.chunks, 32);
    ws.w = ceil_div(ws.chunks, passes);
    ws.inv_w = inverse16(ws.w);
    ws.short_rows_per_warp = 32 / ws.w;
    const int hlanes = ceil_div(la.k, H::kCols);
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
    const auto level_warps = [&](int slots) {
        return (long_rows + 32 / (ws.w * slots) - 1) / (32 / (ws.w * slots)) + (la.short_rows + ws.short_rows_per_warp - 1) / ws.short_rows_per_warp;
    };
    while (ws.slots > 1 && (ws.w * ws.slots > 32 || level_warps(ws.slots) > kSlotWarps)) ws.slots >>= 1;
    ws.inv_group = inverse16(ws.w * ws.slots);
    ws.rows_per_warp = 32 / (ws.w * ws.slots);
    const bool only_heavy = narrow == 0;
    const int nw = only_heavy ? 8 : kWalkWarps;
    // Heavy rows: more warps a row while the rows alone leave the GPU idle.
    ws.heavy_warps = 1;
    while (ws.heavy_warps < nw && la.num_heavy * ws.heavy_warps * 2 <= kResidentWarps) ws.heavy_warps *= 2;
    // Rows left to one CTA must not outlast their level: those of 8 rounds of fetches and more, and
    // more than twice the level's own rounds per warp, go to clusters (at 16: 80k nodes down k = 1 35.1
    // us, at 8: 32.8; at 32: k = 4 47.1 against 36.9).  A 10,491-entry row at
    // k = 64 held one warp for 1477 us (the whole down traversal of 600k nodes: 2423 us, now 601).
    const int64_t level_rounds = num_entries / (4 * ws.groups) / kResidentWarps;
    for (int i = 0; i < GRG_B200_LONG_CLASSES && ws.hubs == 0; ++i) {
        const int64_t rounds = (int64_t{GRG_B200_LONG_ROW} << i) / (4 * ws.groups * ws.heavy_warps);
        if (rounds >= 8 && rounds > 2 * level_rounds) ws.hubs = static_cast<int>(long_counts[i]);
    }
    if (ws.hubs > 0)
        GRG_CUDA_TRY(launch_k(pdl, s, dim3(static_cast<unsigned>(ws.hubs * kHubCtas)), 32 * kHubWarps, level_hub_kernel<H>, la, ws));
    ws.heavy_blocks = ceil_div(la.num_heavy - ws.hubs, nw / ws.heavy_warps);
    if (only_heavy) {
        if (ws.heavy_blocks > 0)
            GRG_CUDA_TRY(launch_smem_k(pdl, s, dim3(static_cast<unsigned>(ws.heavy_blocks)), 256, ws.heavy_warps > 1 ? 8 * 32 * sizeof(typename H::Acc) : 0, level_heavy_kernel<H>, la, ws));
    } else {
        ws.long_blocks = ceil_div(ceil_div(long_rows, ws.rows_per_warp), nw);
        const int short_blocks = ceil_div(ceil_div(la.short_rows, ws.short_rows_per_warp), nw);
        const dim3 grid(static_cast<unsigned>(ws.heavy_blocks + ws.long_blocks + short_blocks));
        const size_t smem = ws.heavy_blocks > 0 && ws.heavy_warps > 1 ? kWalkWarps * 32 * sizeof(typename H::Acc) : 0;
#define GRG_WALK(S) GRG_CUDA_TRY(launch_smem_k(pdl, s, grid, 32 * kWalkWarps, smem, level_walk_kernel<R, H, S, R::kInFlight>, la, ws))
        if (ws.slots == 4) GRG_WALK(4);
        else if (ws.slots == 2) GRG_WALK(2);
        else GRG_WALK(1);
#undef GRG_WALK
    }
    GRG_LAUNCH_CHECK("level_walk_kernel");
    return GRG_B200_OK;
}

}  // namespace

#endif  // GRG_B200_WALK_ROWS_CUH
