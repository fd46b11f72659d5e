// Pieces shared by the kernel files of libgrg_b200: error reporting, launches, vector packs and
// loads, the parameters of a level launch and the decoding of gather entries.
#ifndef GRG_B200_LEVEL_COMMON_CUH
#define GRG_B200_LEVEL_COMMON_CUH

#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "grg_b200.h"

// Records the calling thread's error message (grg_b200_last_error) and returns `code`.
__attribute__((visibility("hidden"))) int grg_fail(int code, const char* fmt, ...);

namespace grg {

#define GRG_CUDA_TRY(...)                                                                   \
    do {                                                                                    \
        cudaError_t err__ = (__VA_ARGS__);                                                       \
        if (err__ != cudaSuccess)                                                           \
            return grg_fail(GRG_B200_ERR_CUDA, "%s failed: %s", #__VA_ARGS__, cudaGetErrorString(err__)); \
    } while (0)

#define GRG_LAUNCH_CHECK(name)                                                              \
    do {                                                                                    \
        cudaError_t err__ = cudaGetLastError();                                             \
        if (err__ != cudaSuccess)                                                           \
            return grg_fail(GRG_B200_ERR_CUDA, "launch of %s failed: %s", name, cudaGetErrorString(err__)); \
    } while (0)

// Launch with programmatic dependent launch when `pdl` (the kernel must call pdl_wait()
// before touching data that earlier kernels of the stream produce).
template <typename... KArgs, typename... Args>
cudaError_t launch_smem_k(bool pdl, cudaStream_t s, dim3 grid, int block, size_t smem, void (*kernel)(KArgs...), Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(static_cast<unsigned>(block));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = pdl ? attr : nullptr;
    cfg.numAttrs = pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename... KArgs, typename... Args>
cudaError_t launch_k(bool pdl, cudaStream_t s, dim3 grid, int block, void (*kernel)(KArgs...), Args... args) {
    return launch_smem_k(pdl, s, grid, block, 0, kernel, args...);
}

// ---------------------------------------------------------------------------------------
// Vector packs
// ---------------------------------------------------------------------------------------
template <typename T, int V>
struct alignas(sizeof(T) * V) Pack {
    T v[V];
};

template <typename T, int V>
__device__ __forceinline__ Pack<T, V> zero_pack() {
    Pack<T, V> r;
#pragma unroll
    for (int i = 0; i < V; ++i) r.v[i] = T(0);
    return r;
}

template <typename T, int V>
__device__ __forceinline__ Pack<T, V> splat(T x) {
    Pack<T, V> r;
#pragma unroll
    for (int i = 0; i < V; ++i) r.v[i] = x;
    return r;
}

template <typename T, int V>
__device__ __forceinline__ void add_into(Pack<T, V>& a, const Pack<T, V>& b) {
#pragma unroll
    for (int i = 0; i < V; ++i) a.v[i] = a.v[i] + b.v[i];
}

// Loads of what other kernels write (node rows, inputs, init values).  A kernel launched early is
// resident while the previous one still writes, so these are ordinary loads, in program order behind
// pdl_wait(): a read-only load (ld.global.nc, __ldg) promises that nothing writes the memory while
// the kernel lives, may be moved ahead of the wait, and rows narrower than a 32-byte sector share
// sectors with rows that the previous level writes.  Lists and other static arrays are read by __ldg.
// Ordinary loads cost nothing (1.5M nodes, up k = 1 169 us, down k = 3 219 us; 5M nodes, up k = 8 533 us:
// the same with either).
__device__ __forceinline__ uint4 ld_words4(const uint32_t* p) {
    uint4 r;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}

__device__ __forceinline__ uint2 ld_words2(const void* p) {
    uint2 r;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(r.x), "=r"(r.y) : "l"(p));
    return r;
}

template <typename T, int V>
__device__ __forceinline__ Pack<T, V> ld_row(const T* p) {
    Pack<T, V> r;
    if constexpr (std::is_same<T, double>::value && V == 1) {
        asm volatile("ld.global.f64 %0, [%1];" : "=d"(r.v[0]) : "l"(p));
    } else if constexpr (std::is_same<T, double>::value && V == 2) {
        asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(r.v[0]), "=d"(r.v[1]) : "l"(p));
    } else if constexpr (V == 1) {
        asm volatile("ld.global.f32 %0, [%1];" : "=f"(r.v[0]) : "l"(p));
    } else if constexpr (V == 2) {
        asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(r.v[0]), "=f"(r.v[1]) : "l"(p));
    } else {
        static_assert(std::is_same<T, float>::value && V == 4, "unsupported pack");
        asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]) : "l"(p));
    }
    return r;
}

// L2 load (rows written by other SMs during this launch must not come from a stale L1 line).
template <typename T, int V>
__device__ __forceinline__ Pack<T, V> ld_l2(const T* p) {
    Pack<T, V> r;
    if constexpr (V == 1) {
        r.v[0] = __ldcg(p);
    } else if constexpr (std::is_same<T, double>::value && V == 2) {
        const double2 d = __ldcg(reinterpret_cast<const double2*>(p));
        r.v[0] = d.x;
        r.v[1] = d.y;
    } else if constexpr (std::is_same<T, float>::value && V == 2) {
        const float2 d = __ldcg(reinterpret_cast<const float2*>(p));
        r.v[0] = d.x;
        r.v[1] = d.y;
    } else {
        const float4 d = __ldcg(reinterpret_cast<const float4*>(p));
        r.v[0] = d.x;
        r.v[1] = d.y;
        r.v[2] = d.z;
        r.v[3] = d.w;
    }
    return r;
}

// Source-row load of the level walkers: through L1, or L2 only (CG) where rows read
// here may have been written by other SMs earlier in the same launch.
template <typename T, int V, bool CG>
__device__ __forceinline__ Pack<T, V> ld_src(const T* p) {
    if constexpr (CG) return ld_l2<T, V>(p);
    else return ld_row<T, V>(p);
}

template <typename T, int V>
__device__ __forceinline__ void st_pack(T* p, const Pack<T, V>& x) {
    *reinterpret_cast<Pack<T, V>*>(p) = x;
}

__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }

// ---------------------------------------------------------------------------------------
// Kernel parameters
// ---------------------------------------------------------------------------------------
struct LevelArgs {
    int64_t row_begin;
    int64_t num_rows;
    const int32_t* row_ptr;
    const uint32_t* entries;
    const int32_t* heavy_rows;
    const int32_t* row_ids;
    int64_t num_heavy;
    int32_t heavy_threshold;
    int32_t list_align;
    int32_t use_miss;
    void* state;
    int64_t ld_state;
    int64_t state_cols;  // columns of a state row that belong to the call: k, or ld_state (GRG_B200_STATE_PADDING)
    const void* x;
    int64_t ld_x;
    const void* miss;
    int64_t ld_miss;
    const void* init_vector;
    const void* init_matrix;
    int64_t ld_init;
    const int32_t* node_perm;
    const void* xtx_node;
    int64_t k;
    int32_t log2g;
    int32_t* err;
    int64_t lim_state;
    int64_t lim_x;
    int64_t lim_miss;
    int32_t log2s;  // narrow rows split over 2^log2s lane groups (default mode, variant 6)
    int32_t num_slot_buckets;  // > 0: narrow lists located from the slot table, not row_ptr
    int32_t slot_width[GRG_B200_MAX_SLOT_BUCKETS];
    int64_t slot_pos[GRG_B200_MAX_SLOT_BUCKETS];
    int64_t slot_entry[GRG_B200_MAX_SLOT_BUCKETS];
    // mixed storage only: the 16-bit planes of state, x and miss (x/miss hold encoded copies)
    void* state_lo;
    const void* x_lo;
    const void* miss_lo;
    int32_t up;  // an up level: its lists name state rows (and null padding) only
    int64_t short_rows;  // entry kernels: the last short_rows narrow positions take one entry slot
    int32_t quad_rows[GRG_B200_QUAD_CLASSES];  // row walk: narrow positions of more than i quads; [0] = 0: read row_ptr
};

enum DeviceError : int32_t {
    kErrStateId = 1,
    kErrInputId = 2,
    kErrMissId = 3,
    kErrPerm = 4,
    kErrSelector = 5,
    kErrWaitTimeout = 6,  // dataflow: a source row never became ready within the spin limit
};

__device__ __forceinline__ void report(int32_t* err, int32_t code) {
    if (err) atomicCAS(err, 0, code);
}

// Programmatic dependent launch: a kernel launched with it may start while the previous
// kernel of the stream is finishing; it reads only static data (level lists) until
// pdl_wait(), which returns once the previous grid has completed and its writes are visible
// (immediately when the launch did not use the attribute).  pdl_trigger() lets the next
// kernel launch once every CTA of this grid has started.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" :::); }

template <typename T, int V, int INIT>
__device__ __forceinline__ Pack<T, V> init_value(const LevelArgs& a, int64_t row, int64_t c) {
    if constexpr (INIT == GRG_B200_INIT_VECTOR) {
        return ld_row<T, V>(static_cast<const T*>(a.init_vector) + c);
    } else if constexpr (INIT == GRG_B200_INIT_XTX) {
        return splat<T, V>(__ldg(static_cast<const T*>(a.xtx_node) + row));
    } else if constexpr (INIT == GRG_B200_INIT_MATRIX) {
        const int64_t orig = __ldg(a.node_perm + row);
        if (a.err && (orig < 0 || orig >= a.lim_state)) {
            report(a.err, kErrPerm);
            return zero_pack<T, V>();
        }
        return ld_row<T, V>(static_cast<const T*>(a.init_matrix) + orig * a.ld_init + c);
    } else {
        return zero_pack<T, V>();
    }
}

// Address of the row named by a coded entry; nullptr when the entry is skipped.
template <typename T>
__device__ __forceinline__ const T* entry_row(const LevelArgs& a, uint32_t code) {
    const uint32_t src = (code >> GRG_B200_SRC_SHIFT) & GRG_B200_SRC_MASK;
    const int64_t id = code & GRG_B200_ID_MASK;
    if (src == GRG_B200_SRC_STATE) {
        if (a.err && id >= a.lim_state) {
            report(a.err, kErrStateId);
            return nullptr;
        }
        return static_cast<const T*>(a.state) + id * a.ld_state;
    }
    if (src == GRG_B200_SRC_INPUT) {
        if (a.err && id >= a.lim_x) {
            report(a.err, kErrInputId);
            return nullptr;
        }
        return static_cast<const T*>(a.x) + id * a.ld_x;
    }
    if (src != GRG_B200_SRC_MISS || !a.use_miss) return nullptr;  // null padding, or miss rows off
    if (a.err && id >= a.lim_miss) {
        report(a.err, kErrMissId);
        return nullptr;
    }
    return static_cast<const T*>(a.miss) + id * a.ld_miss;
}

constexpr unsigned kFullMask = 0xffffffffu;

__device__ __forceinline__ int64_t level_row(const LevelArgs& a, int64_t pos) {
    return a.row_begin + (a.row_ids ? static_cast<int64_t>(__ldg(a.row_ids + pos)) : pos);
}

template <typename T, int V>
__device__ __forceinline__ Pack<T, V> shfl_xor_pack(const Pack<T, V>& x, int off) {
    Pack<T, V> r;
#pragma unroll
    for (int i = 0; i < V; ++i) r.v[i] = __shfl_xor_sync(kFullMask, x.v[i], off);
    return r;
}

// Source row of a coded entry for launches without bounds checks (ids and leading dimensions
// below 2^32: one 32 x 32 -> 64-bit multiply); ok is false for entries that are skipped.
template <typename T, bool UPONLY>
__device__ __forceinline__ const T* lean_source(const LevelArgs& a, uint32_t code, bool& ok) {
    const uint32_t id = code & GRG_B200_ID_MASK;
    const uint32_t src = (code >> GRG_B200_SRC_SHIFT) & GRG_B200_SRC_MASK;
    if constexpr (UPONLY) {
        ok = src == GRG_B200_SRC_STATE;
        return static_cast<const T*>(a.state) + static_cast<size_t>(id) * static_cast<uint32_t>(a.ld_state);
    } else {
        ok = src == GRG_B200_SRC_STATE || src == GRG_B200_SRC_INPUT || (src == GRG_B200_SRC_MISS && a.use_miss);
        const T* base = src == GRG_B200_SRC_STATE ? static_cast<const T*>(a.state)
                                                   : (src == GRG_B200_SRC_INPUT ? static_cast<const T*>(a.x) : static_cast<const T*>(a.miss));
        const uint32_t ld = static_cast<uint32_t>(src == GRG_B200_SRC_STATE ? a.ld_state : (src == GRG_B200_SRC_INPUT ? a.ld_x : a.ld_miss));
        return base + static_cast<size_t>(id) * ld;
    }
}

// 32-byte vector loads (sm_100): one chunk of 4 doubles or 8 floats, an ordinary load like ld_row.
template <typename T>
struct Chunk32 {
    static constexpr int C = 32 / static_cast<int>(sizeof(T));
    using type = Pack<T, C>;
};

template <typename T>
__device__ __forceinline__ typename Chunk32<T>::type ld_chunk(const T* p) {
    typename Chunk32<T>::type r;
    if constexpr (std::is_same<T, double>::value) {
        asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                     : "=d"(r.v[0]), "=d"(r.v[1]), "=d"(r.v[2]), "=d"(r.v[3]) : "l"(p));
    } else {
        asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=f"(r.v[0]), "=f"(r.v[1]), "=f"(r.v[2]), "=f"(r.v[3]), "=f"(r.v[4]), "=f"(r.v[5]), "=f"(r.v[6]), "=f"(r.v[7])
                     : "l"(p));
    }
    return r;
}

// One chunk lane's CW columns: a 32-byte load when CW fills a chunk, else the shape's vector
// load (k below a chunk: CW = k, one chunk lane per row).
template <typename T, int CW>
__device__ __forceinline__ Pack<T, CW> ld_cols(const T* p) {
    if constexpr (CW == Chunk32<T>::C) return ld_chunk<T>(p);
    else return ld_row<T, CW>(p);
}

inline bool aligned(const void* p, int bytes) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) % bytes) == 0; }

}  // namespace grg

using namespace grg;

#endif  // GRG_B200_LEVEL_COMMON_CUH
