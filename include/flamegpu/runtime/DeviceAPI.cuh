#ifndef INCLUDE_FLAMEGPU_RUNTIME_DEVICEAPI_CUH_
#define INCLUDE_FLAMEGPU_RUNTIME_DEVICEAPI_CUH_
// Header-only device API used inside FLAMEGPU_AGENT_FUNCTION bodies: agent
// variables, message input/output iterators (MessageNone, MessageBruteForce,
// MessageSpatial2D, MessageSpatial3D), agent output (birth), environment
// properties and random numbers. Mirrors the reference's device API
// (include/flamegpu/runtime/DeviceAPI.cuh:163-557,
// include/flamegpu/runtime/messaging/*/*Device.cuh) with the same names and
// iteration semantics; the storage behind it is the GB300 layout (sorted
// message records, per-function lookup tables).
#include <cstdint>
#include <type_traits>

#include "flamegpu/defines.h"
#include "flamegpu/detail/device_types.cuh"

#ifndef FLAMEGPU_SEATBELTS
#define FLAMEGPU_SEATBELTS 1
#endif

namespace flamegpu {

class MessageNone;
class MessageBruteForce;
class MessageSpatial2D;
class MessageSpatial3D;
class MessageArray;
class MessageArray2D;
class MessageArray3D;
class MessageBucket;

namespace detail {

#ifdef __CUDACC__
__device__ __forceinline__ void device_error(const LaunchParams& P, uint32_t code, uint32_t hash, uint32_t idx) {
    if (P.error) {
        if (atomicCAS(&P.error[0], 0u, code) == 0u) {
            P.error[1] = hash;
            P.error[2] = idx;
        }
        atomicAdd(&P.error[3], 1u);
    }
}

// Threads of the largest agent-function block.
constexpr unsigned int kAgentBlock = 128;

// The calling block's instance context (shared memory; batched launches only).
__device__ __forceinline__ InstanceCtx& ctx() {
    __shared__ InstanceCtx c;
    return c;
}

/** A launch as its agents' code sees it: the parameters, and which of the
 * kernel's variants runs. `batch` and `stage` are literals of the variant, so
 * once inlined every choice below folds away: a single simulation reads its
 * grid, PBM and environment straight from the parameter space (no context in
 * shared memory, no barrier before the first agent), and a launch without a
 * staged window reads records as global memory through 64-bit arithmetic on
 * launch constants. */
struct Launch {
    const LaunchParams& P;
    bool batch;  // ctx() holds the instance of the block's rows
    bool stage;  // the block may have a staged window
    bool& words_held;  // a wrapped search of this thread holds its range words (a local of the kernel)
    __device__ __forceinline__ operator const LaunchParams&() const { return P; }
    __device__ __forceinline__ const fg_spatial_grid& grid() const { return batch ? ctx().grid : P.in_grid; }
    __device__ __forceinline__ const uint32_t* pbm() const { return batch ? ctx().pbm : P.in_pbm; }
    __device__ __forceinline__ uint32_t pbm_alloc() const { return batch ? ctx().pbm_alloc : P.in_pbm_alloc; }
    __device__ __forceinline__ uint32_t step() const { return batch ? ctx().step : (P.d_step ? *P.d_step : 0u); }
    __device__ __forceinline__ const char* env() const { return batch ? ctx().env : P.env; }
    __device__ __forceinline__ uint64_t seed() const { return batch ? ctx().seed : P.seed; }
    // first row of the instance; in a single simulation, the rows before it failed the function's condition
    __device__ __forceinline__ uint32_t row_begin() const { return batch ? ctx().row_begin : (P.d_first ? *P.d_first : 0u); }
    // first row of the instance's sorted messages
    __device__ __forceinline__ uint32_t row_base() const { return batch ? ctx().row_begin : 0u; }
    __device__ __forceinline__ uint32_t inst() const { return batch ? ctx().inst : 0u; }
};

// A launch constant below 2^24 that stays in a register. What is computed from
// the launch's parameters alone, the compiler recomputes where it is used,
// inside a neighbour loop, in the uniform unit: four payload offsets (multiply,
// shift, multiply each) and the record size were a fifth of the instructions
// that a warp issued for a message. It does not repeat a conversion to float
// and back, which is exact here. 2D payload iterate of 4,194,304 agents 1,020
// -> 842 us, 3D of 8,388,608 366 -> 325 ms, Boids of 1,048,576 198 -> 188 us.
__device__ __forceinline__ uint32_t launch_constant(uint32_t v) {
    return static_cast<uint32_t>(static_cast<float>(v));
}

// Address of element `elem` of variable `hash` in row `row` of table `t`.
// Returns null (after recording a device error) when seatbelts are on and the
// name, the type size or the array index is wrong.
template <typename T>
__device__ __forceinline__ T* var_addr(const LaunchParams& P, const VarTable* __restrict__ t, uint32_t hash,
                                       uint32_t row, uint32_t elem) {
    // t points into the kernel's parameter space: plain loads, constant bank
    const uint32_t s = table_slot(t->mult, t->shift, hash);
    const VarSlot* vs = &t->slot[s];
    char* base = vs->ptr;
    const uint32_t stride = vs->stride;
#if FLAMEGPU_SEATBELTS
    if (vs->hash != hash) {
        device_error(P, kDevUnknownVariable, hash, row);
        return nullptr;
    }
    if (vs->elem_bytes != sizeof(T)) {
        device_error(P, kDevTypeMismatch, hash, row);
        return nullptr;
    }
    if (elem >= vs->elements) {
        device_error(P, kDevArrayIndex, hash, row);
        return nullptr;
    }
#endif
    return reinterpret_cast<T*>(base + static_cast<size_t>(row) * stride + static_cast<size_t>(elem) * sizeof(T));
}

template <typename T>
__device__ __forceinline__ T ldg_any(const T* p) {
    if constexpr (sizeof(T) == 4 || sizeof(T) == 8 || sizeof(T) == 2 || sizeof(T) == 1) {
        return __ldg(p);
    } else {
        return *p;
    }
}
template <>
__device__ __forceinline__ bool ldg_any<bool>(const bool* p) {
    return *p;
}

// Read-only read of a variable (messages, environment): non-coherent path.
template <typename T>
__device__ __forceinline__ T read_ro(const LaunchParams& P, const VarTable* t, uint32_t hash, uint32_t row,
                                     uint32_t elem = 0) {
    const T* a = var_addr<T>(P, t, hash, row, elem);
    return a ? ldg_any(a) : T{};
}
template <typename T>
__device__ __forceinline__ T read_rw(const LaunchParams& P, const VarTable* t, uint32_t hash, uint32_t row,
                                     uint32_t elem = 0) {
    const T* a = var_addr<T>(P, t, hash, row, elem);
    return a ? *a : T{};
}
template <typename T>
__device__ __forceinline__ void write_var(const LaunchParams& P, const VarTable* t, uint32_t hash, uint32_t row, T v,
                                          uint32_t elem = 0) {
    T* a = var_addr<T>(P, t, hash, row, elem);
    if (a) *a = v;
}

// SplitMix64 finaliser (Steele, Lea & Flood, OOPSLA 2014).
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
    return z ^ (z >> 31);
}

__device__ __forceinline__ int clamp_cell(int v, uint32_t dim) {
    const int d = static_cast<int>(dim);
    return v < 0 ? 0 : (v >= d ? d - 1 : v);
}
// getGridPosition3D / getGridPosition2D (MessageSpatial3DDevice.cuh:646-659)
__device__ __forceinline__ int grid_cell(const fg_spatial_grid& g, int axis, float p) {
    return clamp_cell(static_cast<int>(floorf((p - g.min[axis]) / g.radius)), g.gridDim[axis]);
}
// getHash3D / getHash2D (MessageSpatial3DDevice.cuh:660-672): x clamped
__device__ __forceinline__ uint32_t grid_hash(const fg_spatial_grid& g, int x, int y, int z) {
    const uint32_t ux = static_cast<uint32_t>(clamp_cell(x, g.gridDim[0]));
    return static_cast<uint32_t>(z) * g.gridDim[0] * g.gridDim[1] + static_cast<uint32_t>(y) * g.gridDim[0] + ux;
}
__device__ __forceinline__ float virtual_coord(float p1, float p2, float width) {
    // getVirtualX (MessageSpatial3DDevice.cuh:373-397): p2 - (d / |d|) * width
    // when |d| > width / 2. For the finite non-zero d of that branch, d / |d| is
    // exactly +-1 and width / 2 exactly width * 0.5, so the same value comes
    // from a sign copy, without the division.
    const float d = p2 - p1;
    return fabsf(d) > width * 0.5f ? p2 - copysignf(width, d) : p2;
}

// ---- shared-memory staging window of a block's spatial neighbourhood ----
// Layout of the dynamic shared memory: StageHeader (64 B) | PBM slice | records.
__device__ __forceinline__ char* dyn_smem() {
    extern __shared__ __align__(128) char fg_dyn_smem[];
    return fg_dyn_smem;
}
__device__ __forceinline__ StageHeader* stage_hdr() { return reinterpret_cast<StageHeader*>(dyn_smem()); }
__device__ __forceinline__ const uint32_t* stage_pbm() {
    return reinterpret_cast<const uint32_t*>(dyn_smem() + sizeof(StageHeader));
}
__device__ __forceinline__ const char* stage_records(const StageHeader* h) {
    return dyn_smem() + sizeof(StageHeader) + static_cast<size_t>(h->pbm_n) * 4u;
}

/** Column of a variable of an input message list, kept by a message view from
 * one message to the next: its address and stride, and the name and element
 * size they were looked up for (0: none yet). */
struct ColumnRef {
    const char* base = nullptr;
    uint32_t stride = 0;
    uint32_t name = 0, bytes = 0;
};

// Read of element `elem` of a variable of message `index` of an input list of
// columns. A name that the view has looked up (and, with device checks on,
// checked) for an earlier message is not looked up again: a loop over a
// brute-force list then spends a compare, an address and the load on a
// variable. With the lookup and its checks repeated for every message, 16,384
// agents reading 11,500 messages took 1,190 us instead of 574 (one warp a
// scheduler: 104 cycles a message). Reading the next message's element ahead
// made it 785 us.
template <typename T>
__device__ __forceinline__ T read_msg(const LaunchParams& P, ColumnRef (&refs)[4], uint32_t hash, uint32_t index,
                                      uint32_t elem) {
    if (elem == 0u) {
        ColumnRef& r = refs[hash & 3u];  // the name is a literal, so which one is known at compile time
        if (r.name != hash || r.bytes != sizeof(T)) {
            const T* a = var_addr<T>(P, &P.T.msg_in, hash, 0u, 0u);
            if (!a) return T{};
            r.base = reinterpret_cast<const char*>(a);
            r.stride = P.T.msg_in.slot[table_slot(P.T.msg_in.mult, P.T.msg_in.shift, hash)].stride;
            r.name = hash;
            r.bytes = sizeof(T);
        }
        return ldg_any(reinterpret_cast<const T*>(r.base + static_cast<size_t>(index) * r.stride));
    }
    const T* a = var_addr<T>(P, &P.T.msg_in, hash, index, elem);
    return a ? ldg_any(a) : T{};
}

// Byte offset of element `elem` of variable `hash` inside a sorted message
// record: a per-name constant of the launch (slot pointer minus records base).
template <typename T>
__device__ __forceinline__ size_t record_offset(const LaunchParams& P, uint32_t hash, uint32_t elem) {
    const VarTable* t = &P.T.msg_in;
    const VarSlot* vs = &t->slot[table_slot(t->mult, t->shift, hash)];
#if FLAMEGPU_SEATBELTS
    if (vs->hash != hash || vs->ptr == nullptr) {
        device_error(P, kDevUnknownVariable, hash, 0);
        return 0;
    }
    if (vs->elem_bytes != sizeof(T)) {
        device_error(P, kDevTypeMismatch, hash, 0);
        return 0;
    }
    if (elem >= vs->elements) {
        device_error(P, kDevArrayIndex, hash, 0);
        return 0;
    }
#endif
    return static_cast<size_t>(vs->ptr - P.in_records) + static_cast<size_t>(elem) * sizeof(T);
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Bounded wait on the staging mbarrier; false if it gave up.
__device__ __forceinline__ bool stage_wait(StageHeader* h, uint32_t phase) {
    const uint32_t mb = smem_addr(&h->mbar);
    for (uint32_t it = 0; it < (1u << 20); ++it) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(mb), "r"(phase)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Stage the window of sorted messages every agent of this block can see:
// the bins between (lowest agent bin - one z/y/x slab) and (highest + one),
// a contiguous range of the sorted records, copied with TMA bulk copies
// (cp.async.bulk) completing on an mbarrier. All threads of the block call it.
template <int DIMS>
__device__ void stage_window(const Launch& L, uint32_t idx, bool active, bool first) {
    const LaunchParams& P = L.P;
    __shared__ uint32_t s_min, s_max;
    StageHeader* h = stage_hdr();
    if (threadIdx.x == 0) {
        s_min = 0xFFFFFFFFu;
        s_max = 0u;
        if (first) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&h->mbar)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            h->phase = 0;
            h->off = 0;
        }
    }
    uint32_t key = 0xFFFFFFFFu, kmax = 0u;
    if (active) {
        const fg_spatial_grid& g = L.grid();
        const float x = read_rw<float>(P, &P.T.agent, VarName("x").hash, idx);
        const float y = read_rw<float>(P, &P.T.agent, VarName("y").hash, idx);
        const float z = DIMS == 3 ? read_rw<float>(P, &P.T.agent, VarName("z").hash, idx) : 0.0f;
        const int cx = clamp_cell(static_cast<int>(floorf((x - g.min[0]) / g.radius)), g.gridDim[0]);
        const int cy = clamp_cell(static_cast<int>(floorf((y - g.min[1]) / g.radius)), g.gridDim[1]);
        const int cz = DIMS == 3 ? clamp_cell(static_cast<int>(floorf((z - g.min[2]) / g.radius)), g.gridDim[2]) : 0;
        key = static_cast<uint32_t>(cz) * g.gridDim[0] * g.gridDim[1] + static_cast<uint32_t>(cy) * g.gridDim[0] +
              static_cast<uint32_t>(cx);
        kmax = key;
    }
    key = __reduce_min_sync(0xFFFFFFFFu, key);
    kmax = __reduce_max_sync(0xFFFFFFFFu, kmax);
    __syncthreads();  // everyone is done with the previous window; s_min/s_max initialised
    if ((threadIdx.x & 31u) == 0) {
        atomicMin(&s_min, key);
        atomicMax(&s_max, kmax);
    }
    __syncthreads();
    uint32_t tx = 0;
    if (threadIdx.x == 0) {
        h->rec_n = 0;
        h->pbm_n = 0;
        h->rec_lo = 0;
        h->pbm_lo = 0;
        // after a wait that gave up, copies of that window may still land on
        // the mbarrier and in the buffer: the block reads from HBM from then on
        if (s_min != 0xFFFFFFFFu && !h->off) {
            const fg_spatial_grid& g = L.grid();
            const uint32_t* pbm = L.pbm();
            const uint32_t B = g.binCount;
            const uint32_t span = DIMS == 3 ? g.gridDim[0] * g.gridDim[1] + g.gridDim[0] + 1u : g.gridDim[0] + 1u;
            const uint32_t hlo = s_min > span ? s_min - span : 0u;
            const uint32_t hhi = (s_max + span < B) ? s_max + span : B - 1u;
            const uint32_t plo = hlo & ~3u;
            uint32_t pend = (hhi + 2u + 3u) & ~3u;
            if (pend > L.pbm_alloc()) pend = L.pbm_alloc();
            const uint32_t pn = pend - plo;
            const uint32_t rlo = __ldg(pbm + hlo), rhi = __ldg(pbm + hhi + 1u);
            const size_t pbytes = static_cast<size_t>(pn) * 4u;
            const size_t rbytes = static_cast<size_t>(rhi - rlo) * P.in_record_bytes;
            // bulk copies need 16-byte aligned addresses and sizes; anything else
            // (a caller's layout mistake) is not staged: reads then go to HBM
            const bool aligned = ((pbytes | rbytes) & 15u) == 0 &&
                                 (reinterpret_cast<uintptr_t>(pbm + plo) & 15u) == 0 &&
                                 (reinterpret_cast<uintptr_t>(P.in_records) & 15u) == 0 &&
                                 (P.in_record_bytes & 15u) == 0;
            if (aligned && pbytes + rbytes <= P.stage_bytes && pn > 0) {
                h->pbm_lo = plo;
                h->pbm_n = pn;
                h->rec_lo = rlo;
                h->rec_n = rhi - rlo;
                tx = static_cast<uint32_t>(pbytes + rbytes);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                const uint32_t mb = smem_addr(&h->mbar);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(tx) : "memory");
                // PBM slice, then the records, in chunks of at most 32 KiB
                auto copy = [&](char* dst, const char* src, size_t bytes) {
                    while (bytes) {
                        const uint32_t c = bytes > 32768 ? 32768u : static_cast<uint32_t>(bytes);
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                smem_addr(dst)),
                            "l"(src), "r"(c), "r"(mb)
                            : "memory");
                        dst += c;
                        src += c;
                        bytes -= c;
                    }
                };
                char* base = dyn_smem() + sizeof(StageHeader);
                copy(base, reinterpret_cast<const char*>(pbm + plo), pbytes);
                if (rbytes) copy(base + pbytes, P.in_records + static_cast<size_t>(rlo) * P.in_record_bytes, rbytes);
            }
        }
        h->pad[0] = tx;
    }
    __syncthreads();
    if (h->pad[0]) {
        const uint32_t phase = h->phase;
        // a copy that has not landed after the bounded wait is waited for once
        // more (bounded), then the window is dropped and staging is switched
        // off for the rest of this block: reads fall back to HBM
        bool ok = stage_wait(h, phase);
        if (!ok) ok = stage_wait(h, phase);
        __syncthreads();
        if (threadIdx.x == 0) {
            h->phase = phase ^ 1u;
            if (!ok) {
                device_error(P, kDevStageTimeout, 0, idx);
                h->rec_n = 0;
                h->pbm_n = 0;
                h->off = 1;
            }
        }
    }
    __syncthreads();
}
#endif  // __CUDACC__

}  // namespace detail

#ifdef __CUDACC__

// ------------------------------------------------------------------ messages

/** No message input/output (include/flamegpu/runtime/messaging/MessageNone.h). */
class MessageNone {
 public:
    class Description;
    class In {
     public:
        __device__ explicit In(const detail::LaunchParams&) {}
    };
    class Out {
     public:
        __device__ Out(const detail::LaunchParams&, uint32_t) {}
        __device__ uint32_t written() const { return 0; }
    };
};

/** Output half shared by every message type (MessageBruteForceDevice.cuh:259-294). */
class MessageOutBase {
 public:
    __device__ MessageOutBase(const detail::LaunchParams& p, uint32_t idx) : P(p), index(idx) {}
    template <typename T>
    __device__ void setVariable(detail::VarName name, T value) const {
        if (!P.msg_out_enabled) {
            detail::device_error(P, detail::kDevMessageOutNotEnabled, name.hash, index);
            return;
        }
        detail::write_var<T>(P, &P.T.msg_out, name.hash, index, value);
        flag = 1;
        if constexpr (std::is_same<T, float>::value) {  // the location, kept for the launch's epilogue
            if (name.hash == detail::VarName("x").hash) loc[0] = value;
            if (name.hash == detail::VarName("y").hash) loc[1] = value;
            if (name.hash == detail::VarName("z").hash) loc[2] = value;
        }
    }
    template <typename T, flamegpu::size_type N>
    __device__ void setVariable(detail::VarName name, unsigned int i, T value) const {
        if (!P.msg_out_enabled) {
            detail::device_error(P, detail::kDevMessageOutNotEnabled, name.hash, index);
            return;
        }
        detail::write_var<T>(P, &P.T.msg_out, name.hash, index, value, i);
        flag = 1;
    }
    __device__ uint32_t written() const { return flag; }
    /** The message's x, y, z as last set (spatial messages). */
    __device__ float location(int a) const { return loc[a]; }

 protected:
    const detail::LaunchParams& P;
    uint32_t index;
    mutable uint32_t flag = 0;
    mutable float loc[3] = {0.0f, 0.0f, 0.0f};
};

/** Message in an input list, addressed by its (sorted) index. */
class MessageView {
 public:
    __device__ MessageView(const detail::LaunchParams& p, uint32_t i) : P(p), index(i) {}
    template <typename T>
    __device__ T getVariable(detail::VarName name) const {
        return detail::read_msg<T>(P, refs, name.hash, index, 0);
    }
    template <typename T, flamegpu::size_type N>
    __device__ T getVariable(detail::VarName name, unsigned int i) const {
        return detail::read_msg<T>(P, refs, name.hash, index, i);
    }
    __device__ uint32_t getIndex() const { return index; }

 protected:
    const detail::LaunchParams& P;
    mutable detail::ColumnRef refs[4];

 public:
    uint32_t index;
};

/** Every message of the list (MessageBruteForceDevice.cuh:19-172,222-257). */
class MessageBruteForce {
 public:
    class Description;
    class Out : public MessageOutBase {
     public:
        __device__ Out(const detail::LaunchParams& p, uint32_t idx) : MessageOutBase(p, idx) {}
    };
    class In {
     public:
        class Message : public MessageView {
         public:
            __device__ Message(const detail::LaunchParams& p, uint32_t i) : MessageView(p, i) {}
        };
        class iterator {
         public:
            __device__ iterator(const detail::LaunchParams& p, uint32_t i) : m(p, i) {}
            __device__ iterator& operator++() {
                ++m.index;
                return *this;
            }
            __device__ bool operator!=(const iterator& o) const { return m.index != o.m.index; }
            __device__ bool operator==(const iterator& o) const { return m.index == o.m.index; }
            __device__ const Message& operator*() const { return m; }
            __device__ const Message* operator->() const { return &m; }

         private:
            Message m;
        };
        __device__ explicit In(const detail::LaunchParams& p) : P(p), len(p.in_count ? *p.in_count : 0u) {}
        __device__ iterator begin() const { return iterator(P, 0); }
        __device__ iterator end() const { return iterator(P, len); }
        __device__ uint32_t size() const { return len; }

     private:
        const detail::LaunchParams& P;
        uint32_t len;
    };
};


/**
 * Array messages (MessageArrayDevice.cuh, MessageArray2DDevice.cuh,
 * MessageArray3DDevice.cuh): the input list is the array itself, index
 * x + dim_x * (y + dim_y * z), holding the message output to that index this
 * step or zeros. A search iterates the Moore (or von Neumann, |dx| + |dy| +
 * |dz| <= radius) neighbourhood of a cell, origin excluded, x offset outermost
 * and z innermost, clamped to the array or wrapped around it.
 */
template <int D>
class ArrayIn {
 public:
    /** A message of the array (at(), or a neighbour of a search; an index past
     *  the array is an invalid message whose variables read 0). */
    class Message : public MessageView {
     public:
        __device__ Message(const detail::LaunchParams& p, uint32_t i, int ox = 0, int oy = 0, int oz = 0)
            : MessageView(p, i), off{ox, oy, oz} {}
        template <typename T>
        __device__ T getVariable(detail::VarName name) const {
            if (index >= P.in_dims[0] * P.in_dims[1] * P.in_dims[2]) {
                detail::device_error(P, detail::kDevArrayMessage, name.hash, index);
                return T{};
            }
            return MessageView::getVariable<T>(name);
        }
        template <typename T, flamegpu::size_type N>
        __device__ T getVariable(detail::VarName name, unsigned int i) const {
            if (index >= P.in_dims[0] * P.in_dims[1] * P.in_dims[2]) {
                detail::device_error(P, detail::kDevArrayMessage, name.hash, index);
                return T{};
            }
            return MessageView::getVariable<T, N>(name, i);
        }
        __device__ uint32_t getX() const { return index % P.in_dims[0]; }
        __device__ uint32_t getY() const { return (index / P.in_dims[0]) % P.in_dims[1]; }
        __device__ uint32_t getZ() const { return index / (P.in_dims[0] * P.in_dims[1]); }
        __device__ int getOffsetX() const { return off[0]; }
        __device__ int getOffsetY() const { return off[1]; }
        __device__ int getOffsetZ() const { return off[2]; }

     private:
        int off[3];
    };

    /** The neighbourhood of loc within radius: clamped to the array (WRAP
     *  false) or wrapped around it, Moore (VN false) or von Neumann. */
    template <bool WRAP, bool VN>
    class Filter {
     public:
        class iterator {
         public:
            __device__ iterator(const Filter& f, bool at_end) : F(f) {
                for (int a = 0; a < 3; ++a) d[a] = F.lo[a];
                if (at_end || F.empty) {
                    d[0] = F.hi[0] + 1;
                    return;
                }
                skip();
            }
            __device__ iterator& operator++() {
                step();
                skip();
                return *this;
            }
            __device__ bool operator!=(const iterator& o) const { return d[0] != o.d[0] || d[1] != o.d[1] || d[2] != o.d[2]; }
            __device__ bool operator==(const iterator& o) const { return !(*this != o); }
            __device__ Message operator*() const {
                uint32_t idx = 0, mul = 1;
                for (int a = 0; a < D; ++a) {
                    const int dim = static_cast<int>(F.P.in_dims[a]);
                    int c = static_cast<int>(F.loc[a]) + d[a];
                    if (WRAP) c = (c % dim + dim) % dim;
                    idx += static_cast<uint32_t>(c) * mul;
                    mul *= static_cast<uint32_t>(dim);
                }
                return Message(F.P, idx, d[0], d[1], d[2]);
            }

         private:
            // next offset: the innermost axis first
            __device__ void step() {
                for (int a = D - 1; a >= 0; --a) {
                    if (d[a] < F.hi[a] || a == 0) {
                        ++d[a];
                        return;
                    }
                    d[a] = F.lo[a];
                }
            }
            // past the origin and, for von Neumann, the cells beyond the radius
            __device__ void skip() {
                while (d[0] <= F.hi[0]) {
                    const int manhattan = abs(d[0]) + abs(d[1]) + abs(d[2]);
                    if (manhattan != 0 && (!VN || manhattan <= F.radius)) return;
                    step();
                }
            }
            const Filter& F;
            int d[3];
        };
        __device__ Filter(const detail::LaunchParams& p, const uint32_t (&l)[3], uint32_t r, bool bad)
            : P(p), radius(static_cast<int>(r)), empty(bad) {
            for (int a = 0; a < 3; ++a) {
                loc[a] = l[a];
                if (a >= D) {
                    lo[a] = hi[a] = 0;
                } else if (WRAP) {
                    lo[a] = -radius;
                    hi[a] = radius;
                } else {
                    const int x = static_cast<int>(l[a]), dim = static_cast<int>(p.in_dims[a]);
                    lo[a] = x - radius < 0 ? -x : -radius;
                    hi[a] = x + radius >= dim ? dim - 1 - x : radius;
                }
            }
        }
        __device__ iterator begin() const { return iterator(*this, false); }
        __device__ iterator end() const { return iterator(*this, true); }

        const detail::LaunchParams& P;
        uint32_t loc[3];
        int lo[3], hi[3];
        int radius;
        bool empty;
    };

    __device__ explicit ArrayIn(const detail::LaunchParams& p) : P(p) {}
    __device__ uint32_t getDimX() const { return P.in_dims[0]; }
    __device__ uint32_t getDimY() const { return P.in_dims[1]; }
    __device__ uint32_t getDimZ() const { return P.in_dims[2]; }
    __device__ uint32_t size() const { return P.in_dims[0] * P.in_dims[1] * P.in_dims[2]; }

 protected:
    // The message at loc (an invalid one, reading 0, outside the array).
    __device__ Message at_loc(const uint32_t (&l)[3]) const {
        bool out = false;
        for (int a = 0; a < D; ++a) out = out || l[a] >= P.in_dims[a];
        if (out) {
#if FLAMEGPU_SEATBELTS
            detail::device_error(P, detail::kDevArrayMessage, 0, 0);
#endif
            return Message(P, size());
        }
        return Message(P, l[0] + P.in_dims[0] * (l[1] + P.in_dims[1] * l[2]));
    }
    // Whether a search at loc within radius is invalid (MessageArray2DDevice.cuh:1013-1025,
    // :1043-1058): radius 0, an origin outside the array, or for a wrapped
    // search a diameter wider than the array (cells would be read twice).
    __device__ bool bad_search(const uint32_t (&l)[3], uint32_t radius, bool wrap) const {
        bool bad = radius == 0;
        for (int a = 0; a < D; ++a) {
            bad = bad || l[a] >= P.in_dims[a];
            if (wrap) bad = bad || 2u * radius + 1u > P.in_dims[a];
        }
#if FLAMEGPU_SEATBELTS
        if (bad) detail::device_error(P, detail::kDevArrayMessage, 0, radius);
#endif
        return bad;
    }
    template <bool WRAP, bool VN>
    __device__ Filter<WRAP, VN> search(const uint32_t (&l)[3], uint32_t radius) const {
        return Filter<WRAP, VN>(P, l, radius, bad_search(l, radius, WRAP));
    }
    const detail::LaunchParams& P;
};

/** Output half of the array messages: setIndex places the message. */
template <int D>
class ArrayOut : public MessageOutBase {
 public:
    __device__ ArrayOut(const detail::LaunchParams& p, uint32_t idx) : MessageOutBase(p, idx) {}
    /** Whether setIndex was called: the message is output (MessageArray2DDevice.cuh:1360-1375). */
    __device__ uint32_t written() const { return index_set; }

 protected:
    __device__ void set_index(const uint32_t (&l)[3]) const {
        bool out = false;
        for (int a = 0; a < D; ++a) out = out || l[a] >= P.out_dims[a];
        if (out) {
            detail::device_error(P, detail::kDevArrayMessage, 0, index);
            return;
        }
        detail::write_var<uint32_t>(P, &P.T.msg_out, detail::VarName("___INDEX").hash, index,
                                    l[0] + P.out_dims[0] * (l[1] + P.out_dims[1] * l[2]));
        index_set = 1;
    }
    mutable uint32_t index_set = 0;
};

class MessageArray {
 public:
    class Description;
    class In : public ArrayIn<1> {
     public:
        __device__ explicit In(const detail::LaunchParams& p) : ArrayIn<1>(p) {}
        __device__ Message at(uint32_t x) const { return at_loc({x, 0u, 0u}); }
        __device__ Filter<false, false> operator()(uint32_t x, uint32_t radius = 1) const {
            return search<false, false>({x, 0u, 0u}, radius);
        }
        __device__ Filter<true, false> wrap(uint32_t x, uint32_t radius = 1) const {
            return search<true, false>({x, 0u, 0u}, radius);
        }
    };
    class Out : public ArrayOut<1> {
     public:
        __device__ Out(const detail::LaunchParams& p, uint32_t idx) : ArrayOut<1>(p, idx) {}
        __device__ void setIndex(uint32_t x) const { set_index({x, 0u, 0u}); }
    };
};

class MessageArray2D {
 public:
    class Description;
    class In : public ArrayIn<2> {
     public:
        __device__ explicit In(const detail::LaunchParams& p) : ArrayIn<2>(p) {}
        __device__ Message at(uint32_t x, uint32_t y) const { return at_loc({x, y, 0u}); }
        __device__ Filter<false, false> operator()(uint32_t x, uint32_t y, uint32_t radius = 1) const {
            return search<false, false>({x, y, 0u}, radius);
        }
        __device__ Filter<true, false> wrap(uint32_t x, uint32_t y, uint32_t radius = 1) const {
            return search<true, false>({x, y, 0u}, radius);
        }
        __device__ Filter<false, true> vn(uint32_t x, uint32_t y, uint32_t radius = 1) const {
            return search<false, true>({x, y, 0u}, radius);
        }
        __device__ Filter<true, true> vn_wrap(uint32_t x, uint32_t y, uint32_t radius = 1) const {
            return search<true, true>({x, y, 0u}, radius);
        }
    };
    class Out : public ArrayOut<2> {
     public:
        __device__ Out(const detail::LaunchParams& p, uint32_t idx) : ArrayOut<2>(p, idx) {}
        __device__ void setIndex(uint32_t x, uint32_t y) const { set_index({x, y, 0u}); }
    };
};

class MessageArray3D {
 public:
    class Description;
    class In : public ArrayIn<3> {
     public:
        __device__ explicit In(const detail::LaunchParams& p) : ArrayIn<3>(p) {}
        __device__ Message at(uint32_t x, uint32_t y, uint32_t z) const { return at_loc({x, y, z}); }
        __device__ Filter<false, false> operator()(uint32_t x, uint32_t y, uint32_t z, uint32_t radius = 1) const {
            return search<false, false>({x, y, z}, radius);
        }
        __device__ Filter<true, false> wrap(uint32_t x, uint32_t y, uint32_t z, uint32_t radius = 1) const {
            return search<true, false>({x, y, z}, radius);
        }
        __device__ Filter<false, true> vn(uint32_t x, uint32_t y, uint32_t z, uint32_t radius = 1) const {
            return search<false, true>({x, y, z}, radius);
        }
        __device__ Filter<true, true> vn_wrap(uint32_t x, uint32_t y, uint32_t z, uint32_t radius = 1) const {
            return search<true, true>({x, y, z}, radius);
        }
    };
    class Out : public ArrayOut<3> {
     public:
        __device__ Out(const detail::LaunchParams& p, uint32_t idx) : ArrayOut<3>(p, idx) {}
        __device__ void setIndex(uint32_t x, uint32_t y, uint32_t z) const { set_index({x, y, z}); }
    };
};

/**
 * Bucket messages (MessageBucketDevice.cuh): each message carries an integer
 * key in [lowerBound, upperBound]; the input iterates the messages of one key,
 * or of the keys [begin, end), in the order they were output.
 */
class MessageBucket {
 public:
    class Description;
    class In {
     public:
        class Message : public MessageView {
         public:
            __device__ Message(const detail::LaunchParams& p, uint32_t i) : MessageView(p, i) {}
        };
        class Filter {
         public:
            class iterator {
             public:
                __device__ iterator(const detail::LaunchParams& p, uint32_t i) : m(p, i) {}
                __device__ iterator& operator++() {
                    ++m.index;
                    return *this;
                }
                __device__ bool operator!=(const iterator& o) const { return m.index != o.m.index; }
                __device__ bool operator==(const iterator& o) const { return m.index == o.m.index; }
                __device__ const Message& operator*() const { return m; }
                __device__ const Message* operator->() const { return &m; }

             private:
                Message m;
            };
            __device__ Filter(const detail::LaunchParams& p, uint32_t b, uint32_t e) : P(p), first(b), last(e) {}
            __device__ iterator begin() const { return iterator(P, first); }
            __device__ iterator end() const { return iterator(P, last); }
            __device__ uint32_t size() const { return last - first; }

         private:
            const detail::LaunchParams& P;
            uint32_t first, last;
        };
        __device__ explicit In(const detail::LaunchParams& p) : P(p) {}
        /** The messages of one key (MessageBucketDevice.cuh:207-221). */
        __device__ Filter operator()(int32_t key) const {
            if (key < P.in_key_lo || key >= P.in_key_hi) {
                detail::device_error(P, detail::kDevBucketMessage, 0, static_cast<uint32_t>(key));
                return Filter(P, 0, 0);
            }
            const uint32_t k = static_cast<uint32_t>(key - P.in_key_lo);
            return Filter(P, __ldg(P.in_pbm + k), __ldg(P.in_pbm + k + 1));
        }
        /** The messages of the keys [beginKey, endKey) (:228-245). */
        __device__ Filter operator()(int32_t beginKey, int32_t endKey) const {
            if (beginKey < P.in_key_lo || endKey > P.in_key_hi || endKey <= beginKey) {
                detail::device_error(P, detail::kDevBucketMessage, 0, static_cast<uint32_t>(beginKey));
                return Filter(P, 0, 0);
            }
            return Filter(P, __ldg(P.in_pbm + (beginKey - P.in_key_lo)), __ldg(P.in_pbm + (endKey - P.in_key_lo)));
        }

     private:
        const detail::LaunchParams& P;
    };
    class Out : public MessageOutBase {
     public:
        __device__ Out(const detail::LaunchParams& p, uint32_t idx) : MessageOutBase(p, idx) {}
        /** The message's key (MessageBucketDevice.cuh:275-290); a key outside the bounds is a device error. */
        __device__ void setKey(int32_t key) const {
            if (key < P.out_key_lo || key >= P.out_key_hi) {
                detail::device_error(P, detail::kDevBucketMessage, 0, index);
                return;
            }
            detail::write_var<int32_t>(P, &P.T.msg_out, detail::VarName("___KEY").hash, index, key);
            key_set = 1;
        }
        /** Whether setKey was called: the message is output. */
        __device__ uint32_t written() const { return key_set; }

     private:
        mutable uint32_t key_set = 0;
    };
};

/** The staged window of the calling block, cached in registers by a filter. */
struct Window {
    uint32_t rec_lo = 0, rec_n = 0, pbm_lo = 0, pbm_n = 0;
    const char* rec = nullptr;
    const uint32_t* pbm = nullptr;
    const uint32_t* gpbm = nullptr;  // the instance's PBM in HBM
    __device__ explicit Window(const detail::Launch& L) {
        gpbm = L.pbm();
        if (!L.stage) return;
        const detail::StageHeader* h = detail::stage_hdr();
        rec_lo = h->rec_lo;
        rec_n = h->rec_n;
        pbm_lo = h->pbm_lo;
        pbm_n = h->pbm_n;
        pbm = detail::stage_pbm();
        rec = detail::stage_records(h);
    }
    __device__ uint32_t pbm_at(const detail::Launch& L, uint32_t h) const {
        if (!L.stage) return __ldg(gpbm + h);
        const uint32_t r = h - pbm_lo;
        return r < pbm_n ? pbm[r] : __ldg(gpbm + h);
    }
    __device__ const char* row(const detail::Launch& L, uint32_t index) const {
        const char* g = L.P.in_records + static_cast<size_t>(index) * L.P.in_record_bytes;
        if (!L.stage) return g;
        const uint32_t r = index - rec_lo;
        return r < rec_n ? rec + static_cast<size_t>(r) * L.P.in_record_bytes : g;
    }
};

/**
 * A message of a spatial input list: a view of its sorted record. `row` is
 * the record's address — in the block's shared-memory window when the
 * message is inside it, else in HBM — computed once per message by the
 * iterator; a field read is then one load at row + field offset, the offset
 * being a per-name constant of the launch. Every spatial record starts with
 * its location (x, y and, in 3D, z: the message type's first variables) and
 * is 16-byte aligned, so with device checks off those reads use constant
 * offsets from an aligned address, which the compiler can fold and merge;
 * every other field's offset is arithmetic on launch constants (its slot in
 * the record's own perfect hash), which the compiler hoists out of the loop.
 * With device checks on, reads go through the checked name table, whose
 * entries point at the same fields.
 */
template <int DIMS>
class RecordView {
 public:
    __device__ RecordView(const detail::LaunchParams& p, uint32_t i) : P(p), index(i), row(nullptr) {}
    template <typename T>
    __device__ T getVariable(detail::VarName name) const {
#if !FLAMEGPU_SEATBELTS
        const char* r = static_cast<const char*>(__builtin_assume_aligned(row, 16));
        if constexpr (sizeof(T) == 4) {
            if (name.hash == detail::VarName("x").hash) return *reinterpret_cast<const T*>(r);
            if (name.hash == detail::VarName("y").hash) return *reinterpret_cast<const T*>(r + 4);
            if (DIMS == 3 && name.hash == detail::VarName("z").hash) return *reinterpret_cast<const T*>(r + 8);
        }
        return *reinterpret_cast<const T*>(r + payload_offset(name.hash));
#else
        return *reinterpret_cast<const T*>(row + detail::record_offset<T>(P, name.hash, 0));
#endif
    }
    template <typename T, flamegpu::size_type N>
    __device__ T getVariable(detail::VarName name, unsigned int i) const {
#if !FLAMEGPU_SEATBELTS
        return *reinterpret_cast<const T*>(row + payload_offset(name.hash) + static_cast<size_t>(i) * sizeof(T));
#else
        return *reinterpret_cast<const T*>(row + detail::record_offset<T>(P, name.hash, i));
#endif
    }
    __device__ uint32_t getIndex() const { return index; }

 protected:
    // byte offset of a non-location field: arithmetic on launch constants only
    // (the slot of the name in the record's perfect hash), computed once
    // outside the neighbour loop
    __device__ __forceinline__ uint32_t payload_offset(uint32_t hash) const {
        return detail::launch_constant(4u * DIMS + detail::table_slot(P.in_pay_mult, P.in_pay_shift, hash) * P.in_pay_stride);
    }
    const detail::LaunchParams& P;

 public:
    uint32_t index;
    const char* row;
};

/*
 * Spatially partitioned messages; the iterators visit the reference's Moore
 * neighbourhood in the reference's order, with no radius test (user code
 * filters). A clamped search visits 3^(DIMS-1) x-strips, y-offset outer,
 * z-offset inner, each strip PBM[hash(x-1)] .. PBM[hash(x+1)+1] with x
 * clamped; a wrapped one 3^DIMS single bins, x offset outer, then y, z offset
 * inner, every axis taken modulo gridDim.
 *
 * What bounds it: in sparse neighbourhoods the lanes of a warp change range at
 * different messages, so nearly every message a warp visits pays for a change;
 * in dense ones the issue slots (the user's own arithmetic). So the cost of
 * entering the next range is what the cursors below keep small:
 *  - the wrapped search's 27 (9) bins: their bounds are read once and kept in
 *    shared memory, one word each. Recomputing the hash with its three wrapped
 *    axes and reading the bounds again took 7,000 warp instructions a warp and
 *    260 us for the Boids iterate of 1,048,576 agents, against 4,860 and 197
 *    us; the same words in local memory 278 us (their lines cost the records
 *    their place in L1, hit rate 84 -> 72%);
 *  - the clamped search's 9 (3) strips: the hash is two multiply-adds from the
 *    corner strip, so the strips are a bit mask and the bounds are read again.
 *    100,003 Boids: 37.3 -> 33.4 us. Words in shared memory as above would
 *    give 31.3 us there, but take 84 KB of L1 from the 12 resident blocks of
 *    the 8,388,608-agent Gaussian mixture, 371 -> 377 ms against 366 ms.
 * A range lies wholly inside or wholly outside the block's staged window, so
 * within a range the record address just advances by one record.
 */

/** The x strips of a clamped search (MessageSpatial3DDevice.cuh:693-719), the
 * non-empty ones in visit order. One bit per strip not yet entered; the next
 * one's bounds are read while the current one is walked. */
template <int DIMS>
class StripCursor {
    static constexpr int kStrips = DIMS == 3 ? 9 : 3;

 public:
    // a search keeps nothing but its origin: every walk reads the bounds itself
    struct Shared {
        __device__ __forceinline__ Shared(const detail::Launch&, const Window&, const float (&)[3]) {}
    };
    __device__ __forceinline__ StripCursor(const detail::Launch& l, const Window& w, const Shared&, const float (&p)[3],
                                           bool at_end)
        : L(l), win(w) {
        if (at_end) return;
        const fg_spatial_grid& g = L.grid();
        const int dx = static_cast<int>(g.gridDim[0]), dy = static_cast<int>(g.gridDim[1]), dz = static_cast<int>(g.gridDim[2]);
        const int cx = detail::grid_cell(g, 0, p[0]), cy = detail::grid_cell(g, 1, p[1]);
        const int cz = DIMS == 3 ? detail::grid_cell(g, 2, p[2]) : 0;
        const int x0 = cx > 0 ? cx - 1 : 0;
        width = static_cast<uint32_t>((cx + 1 < dx ? cx + 1 : dx - 1) - x0 + 1);
        // the first strip's first cell; outside the grid its hash wraps, and no bit selects it
        corner = static_cast<uint32_t>(x0 + (cy - 1) * dx + (DIMS == 3 ? (cz - 1) * dx * dy : 0));
#pragma unroll
        for (int t = 0; t < kStrips; ++t) {
            const int ay = cy + (DIMS == 3 ? t / 3 : t) - 1, az = cz + (DIMS == 3 ? t % 3 - 1 : 0);
            const bool inside = ay >= 0 && ay < dy && (DIMS == 2 || (az >= 0 && az < dz));
            if (inside) {
                const uint32_t h = hash(t);
                todo |= (win.pbm_at(L, h) < win.pbm_at(L, h + width) ? 1u : 0u) << t;
            }
        }
        read_ahead();
    }
    __device__ __forceinline__ void next(uint32_t& b, uint32_t& e) {
        b = nb;
        e = ne;
        read_ahead();
    }

 private:
    __device__ __forceinline__ uint32_t hash(uint32_t t) const {
        const fg_spatial_grid& g = L.grid();
        if (DIMS == 2) return corner + t * g.gridDim[0];
        const uint32_t q = (t * 11u) >> 5;  // t / 3, t < 9
        return corner + q * g.gridDim[0] + (t - 3u * q) * (g.gridDim[0] * g.gridDim[1]);
    }
    // an empty range when none is left
    __device__ __forceinline__ void read_ahead() {
        nb = ne = 0;
        if (todo) {
            const uint32_t h = hash(static_cast<uint32_t>(__ffs(todo) - 1));
            todo &= todo - 1u;
            nb = win.pbm_at(L, h);
            ne = win.pbm_at(L, h + width);
        }
    }
    const detail::Launch L;
    const Window win;
    uint32_t corner = 0, width = 0;  // strip t: cells hash(t) .. hash(t) + width - 1
    uint32_t todo = 0, nb = 0, ne = 0;
};

/** The single bins of a wrapped search (MessageSpatial3DDevice.cuh:264-276,
 * :727-749), the non-empty ones in visit order. Their bounds are read once,
 * when the search is made, and kept as one word each in shared memory (one
 * column per thread): the first message below, the length above bit
 * `in_index_bits`, then an end word; entering the next bin is one shared
 * load, issued one bin ahead. Where a length does not fit (more than
 * 2^(32 - in_index_bits) - 1 messages in one bin), or while another search of
 * the same thread (a nested loop) has its words there, or for a copied search,
 * the walk keeps a bit per non-empty bin and reads the next one's bounds ahead,
 * its hash two or three additions from the search's own bin (with the axes'
 * divisions again for every bin, the empty ones too: 200,000 agents at one a
 * bin searched around each neighbour 1,367 us a step, 1,160 so; the
 * 8,388,608-agent Gaussian mixture, wrapped, 440 ms and 425).
 * The listed walk keeps its speed: the state of the other one lies in its
 * registers where it can (a shared address kept as a pointer beside it took
 * 2,097,152 payload agents at 40 registers from 440 to 490 us; the staged
 * variant, which has the registers, keeps the pointer: ten steps of 16,384
 * Boids 304.1 us, 305.4 with the address), and the first look at the bins is a
 * call, but in a batch (inlined, 1,048,576 Boids 399.5 us instead of 396.7; a
 * call, 24 batched runs 17.03 ms instead of 16.85). All of it a call on local
 * memory: the listed walks 1.4 to 2.5 times as long. */
template <int DIMS>
class CellCursor {
    static constexpr int kCells = DIMS == 3 ? 27 : 9;
    // hash terms of the offsets -1, 0, +1 on each axis, modulo gridDim
    // (MessageSpatial3DDevice.cuh:736-738)
    struct Terms {
        uint32_t hx[3], hy[3], hz[3];
        __device__ __forceinline__ Terms(const fg_spatial_grid& g, const float (&p)[3]) {
            axis(hx, detail::grid_cell(g, 0, p[0]), g.gridDim[0], 1u);
            axis(hy, detail::grid_cell(g, 1, p[1]), g.gridDim[1], g.gridDim[0]);
            if (DIMS == 3) axis(hz, detail::grid_cell(g, 2, p[2]), g.gridDim[2], g.gridDim[0] * g.gridDim[1]);
        }
        __device__ __forceinline__ uint32_t hash(int t) const {
            return DIMS == 3 ? pick(hx, t / 9) + pick(hy, (t / 3) % 3) + pick(hz, t % 3) : pick(hx, t / 3) + pick(hy, t % 3);
        }
        __device__ __forceinline__ uint32_t hash_yz(int t) const { return DIMS == 3 ? hy[t / 3] + hz[t % 3] : hy[t]; }
        // a cell is its axis' first if its term is 0, its last if the next one's is
        __device__ __forceinline__ uint32_t edges() const {
            uint32_t e = (hx[1] == 0u ? 1u : 0u) | (hx[2] == 0u ? 2u : 0u) | (hy[1] == 0u ? 4u : 0u) | (hy[2] == 0u ? 8u : 0u);
            if (DIMS == 3) e |= (hz[1] == 0u ? 16u : 0u) | (hz[2] == 0u ? 32u : 0u);
            return e;
        }
        static __device__ __forceinline__ uint32_t pick(const uint32_t (&h)[3], int r) {
            return r == 0 ? h[0] : (r == 1 ? h[1] : h[2]);
        }
        // cell c is in [0, d), so c - 1 and c + 1 need at most one turn
        static __device__ __forceinline__ void axis(uint32_t (&h)[3], int c, uint32_t d, uint32_t scale) {
            const uint32_t u = static_cast<uint32_t>(c);
            h[0] = (u == 0u ? d - 1u : u - 1u) * scale;
            h[1] = u * scale;
            h[2] = (u + 1u == d ? 0u : u + 1u) * scale;
        }
    };
    static __device__ __forceinline__ uint32_t* column() {
        __shared__ uint32_t words[(kCells + 2) * detail::kAgentBlock];
        return words + threadIdx.x;
    }

 public:
    // holds the thread's words while it lives. The words are the thread's, so
    // the flag is too: every copy of the input list comes to the same one
    struct Shared {
        bool& held;
        const bool owner;
        bool listed = false;
        __device__ __forceinline__ Shared(const detail::Launch& L, const Window& win, const float (&p)[3])
            : held(L.words_held), owner(!L.words_held) {
            if (!owner) return;
            held = true;
            const Terms terms(L.grid(), p);
            uint32_t* w = column();
            const uint32_t bits = L.P.in_index_bits, base = L.row_base();
            listed = true;
#pragma unroll
            for (int t = 0; t < kCells; ++t) {
                const uint32_t h = terms.hash(t);
                const uint32_t b = win.pbm_at(L, h), e = win.pbm_at(L, h + 1u);
                const uint32_t len = b < e ? e - b : 0u;  // a PBM whose scan gave up may run backwards
                *w = (b - base) | (len << bits);
                w += len ? detail::kAgentBlock : 0u;
                listed = listed && (len >> 1) >> (31u - bits) == 0u;
            }
            w[0] = w[detail::kAgentBlock] = 0u;
        }
        __device__ __forceinline__ Shared(const Shared& o) : held(o.held), owner(false) {}
        __device__ __forceinline__ ~Shared() {
            if (owner) held = false;
        }
    };
    __device__ __forceinline__ CellCursor(const detail::Launch& l, const Window& w, const Shared& s, const float (&p)[3],
                                          bool at_end)
        : L(l), win(w), listed(s.listed) {
        if (at_end) return;
        if (listed) {
            if (L.stage)
                at = column();
            else
                place = static_cast<uint32_t>(__cvta_generic_to_shared(column()));
            ahead = word();
            return;
        }
        const Start start = L.batch ? look(L.grid(), win.gpbm, p[0], p[1], p[2])
                                    : look_call(L.grid(), win.gpbm, p[0], p[1], p[2]);
        centre = start.centre;
        place = start.place;
        edges = start.edges;
        read_ahead();
    }
    __device__ __forceinline__ void next(uint32_t& b, uint32_t& e) {
        if (listed) {
            const uint32_t bits = L.P.in_index_bits;
            b = L.row_base() + (ahead & ((1u << bits) - 1u));
            e = b + (ahead >> bits);
            if (L.stage)
                at += detail::kAgentBlock;
            else
                place += detail::kAgentBlock * 4u;
            ahead = word();  // in flight while this bin is read
            return;
        }
        b = ahead;
        e = last;
        read_ahead();
    }

 private:
    struct Start {
        uint32_t centre, place, edges;
    };
    // the search's own bin, and the non-empty ones among its neighbours
    static __device__ __forceinline__ Start look(const fg_spatial_grid& g, const uint32_t* pbm, float x, float y, float z) {
        const float p[3] = {x, y, z};
        const Terms terms(g, p);
        Start s{terms.hash(kCells / 2), DIMS == 3 ? 0u : terms.edges() << kCells, DIMS == 3 ? terms.edges() : 0u};
#pragma unroll 1
        for (int q = 0; q < 3; ++q) {
            const uint32_t hx = Terms::pick(terms.hx, q);
            uint32_t mask = 0;
#pragma unroll
            for (int t = 0; t < kCells / 3; ++t) {
                const uint32_t h = hx + terms.hash_yz(t);
                mask |= (__ldg(pbm + h) < __ldg(pbm + h + 1u) ? 1u : 0u) << t;
            }
            s.place |= mask << (q * (kCells / 3));
        }
        return s;
    }
    static __device__ __noinline__ Start look_call(const fg_spatial_grid& g, const uint32_t* pbm, float x, float y, float z) {
        return look(g, pbm, x, y, z);
    }
    __device__ __forceinline__ uint32_t word() const {
        return L.stage ? *at : *static_cast<const uint32_t*>(__cvta_shared_to_generic(place));
    }
    // bin t of the visit order, from the search's own bin: the neighbour on an
    // axis is one cell away, or the axis' length less one at the grid's edge
    __device__ __forceinline__ uint32_t hash(uint32_t t) const {
        const fg_spatial_grid& g = L.grid();
        const uint32_t q = (t * 11u) >> 5;  // t / 3, t < 27
        if (DIMS == 2) return centre + turn(q, 0, g.gridDim[0], 1u) + turn(t - 3u * q, 2, g.gridDim[1], g.gridDim[0]);
        const uint32_t x = (q * 11u) >> 5;
        return centre + turn(x, 0, g.gridDim[0], 1u) + turn(q - 3u * x, 2, g.gridDim[1], g.gridDim[0]) +
               turn(t - 3u * q, 4, g.gridDim[2], g.gridDim[0] * g.gridDim[1]);
    }
    __device__ __forceinline__ uint32_t turn(uint32_t r, int edge, uint32_t d, uint32_t scale) const {
        const uint32_t at = DIMS == 3 ? edges >> edge : place >> (kCells + edge);
        const uint32_t off = r == 0u ? (at & 1u ? d - 1u : ~0u) : (at & 2u ? 1u - d : 1u);
        return r == 1u ? 0u : off * scale;
    }
    // bounds of the next non-empty bin (an empty range when none is left)
    __device__ __forceinline__ void read_ahead() {
        ahead = last = 0;
        if (place & ((1u << kCells) - 1u)) {
            const uint32_t h = hash(static_cast<uint32_t>(__ffs(place) - 1));
            place &= place - 1u;
            ahead = win.pbm_at(L, h);
            last = win.pbm_at(L, h + 1u);
        }
    }
    const detail::Launch L;
    const Window win;
    const bool listed;
    const uint32_t* at = nullptr;  // listed, staged launches: the word read ahead
    uint32_t place = 0;  // listed: shared address of the word read ahead; else one bit per non-empty bin not yet entered
    uint32_t ahead = 0;  // that word; else the next bin's first message
    // not listed
    uint32_t last = 0;    // the next bin's end
    uint32_t centre = 0;  // hash of the search's own bin
    uint32_t edges = 0;   // per axis: the bin is the axis' first, its last (DIMS == 2: in place, above the bins)
};

/** A search's messages: the ranges its cursor gives, one after another. */
template <typename Cursor, typename MessageT>
class Search {
 public:
    class iterator {
     public:
        __device__ __forceinline__ iterator(const Search& s, bool at_end)
            : L(s.L), win(s.win), record_bytes(detail::launch_constant(s.L.P.in_record_bytes)),
              cursor(s.L, s.win, s.shared, s.loc, at_end), m(s.L, s.loc), end_(0) {
            if (!at_end) advance();
        }
        __device__ __forceinline__ iterator& operator++() {
            m.row += record_bytes;
            if (++m.index >= end_) advance();
            return *this;
        }
        __device__ __forceinline__ bool operator!=(const iterator&) const { return m.index < end_; }
        __device__ __forceinline__ bool operator==(const iterator& o) const { return !(*this != o); }
        __device__ __forceinline__ const MessageT& operator*() const { return m; }
        __device__ __forceinline__ const MessageT* operator->() const { return &m; }

     private:
        // enter the next range (past the last: an empty one, which ends the loop)
        __device__ __forceinline__ void advance() {
            cursor.next(m.index, end_);
            m.row = win.row(L, m.index);
        }
        const detail::Launch L;
        const Window win;
        const uint32_t record_bytes;
        Cursor cursor;
        MessageT m;
        uint32_t end_;
    };

    __device__ __forceinline__ Search(const detail::Launch& l, float x, float y, float z)
        : L(l), win(l), loc{x, y, z}, shared(l, win, loc) {}
    __device__ __forceinline__ iterator begin() const { return iterator(*this, false); }
    __device__ __forceinline__ iterator end() const { return iterator(*this, true); }

 private:
    const detail::Launch L;
    const Window win;
    const float loc[3];
    const typename Cursor::Shared shared;
};

template <int DIMS>
class SpatialIn {
 public:
    class ClampMessage : public RecordView<DIMS> {
     public:
        __device__ __forceinline__ ClampMessage(const detail::Launch& l, const float (&)[3]) : RecordView<DIMS>(l.P, 0) {}
    };
    class WrapMessage : public RecordView<DIMS> {
     public:
        __device__ __forceinline__ WrapMessage(const detail::Launch& l, const float (&p)[3])
            : RecordView<DIMS>(l.P, 0), L(l), x0(p[0]), y0(p[1]), z0(p[2]) {}
        __device__ float getVirtualX() const { return getVirtualX(x0); }
        __device__ float getVirtualY() const { return getVirtualY(y0); }
        __device__ float getVirtualZ() const { return getVirtualZ(z0); }
        __device__ float getVirtualX(float x1) const {
            return detail::virtual_coord(x1, this->template getVariable<float>("x"), L.grid().width[0]);
        }
        __device__ float getVirtualY(float y1) const {
            return detail::virtual_coord(y1, this->template getVariable<float>("y"), L.grid().width[1]);
        }
        __device__ float getVirtualZ(float z1) const {
            return detail::virtual_coord(z1, this->template getVariable<float>("z"), L.grid().width[2]);
        }

     private:
        const detail::Launch L;
        float x0, y0, z0;  // the search origin
    };
    class Filter : public Search<StripCursor<DIMS>, ClampMessage> {
     public:
        using Message = ClampMessage;
        using Search<StripCursor<DIMS>, ClampMessage>::Search;
    };
    class WrapFilter : public Search<CellCursor<DIMS>, WrapMessage> {
     public:
        using Message = WrapMessage;
        using Search<CellCursor<DIMS>, WrapMessage>::Search;
    };

    __device__ explicit SpatialIn(const detail::Launch& l) : L(l), P(l.P) {}
    __device__ float radius() const { return L.grid().radius; }

 protected:
    // MessageSpatial3D::In::wrap seatbelts (MessageSpatial3DDevice.cuh:527-549)
    __device__ bool wrap_ok(float x, float y, float z) const {
#if FLAMEGPU_SEATBELTS
        const fg_spatial_grid& g = L.grid();
        bool out = x > g.max[0] || y > g.max[1] || x < g.min[0] || y < g.min[1];
        if (DIMS == 3) out = out || z > g.max[2] || z < g.min[2];
        if (out) {
            detail::device_error(P, detail::kDevWrapOutOfBounds, 0, 0);
            return false;
        }
        if (!g.wrapCompatible) detail::device_error(P, detail::kDevWrapIncompatible, 0, 0);
#endif
        return true;
    }
    const detail::Launch L;
    const detail::LaunchParams& P;
};

/** MessageSpatial2D (include/flamegpu/runtime/messaging/MessageSpatial2D/MessageSpatial2DDevice.cuh). */
class MessageSpatial2D {
 public:
    class Description;
    class In : public SpatialIn<2> {
     public:
        __device__ explicit In(const detail::Launch& l) : SpatialIn<2>(l) {}
        __device__ Filter operator()(float x, float y) const { return Filter(L, x, y, 0.0f); }
        __device__ WrapFilter wrap(float x, float y) const {
            if (!wrap_ok(x, y, 0.0f)) return WrapFilter(L, L.grid().min[0], L.grid().min[1], 0.0f);
            return WrapFilter(L, x, y, 0.0f);
        }
    };
    class Out : public MessageOutBase {
     public:
        __device__ Out(const detail::LaunchParams& p, uint32_t idx) : MessageOutBase(p, idx) {}
        __device__ void setLocation(float x, float y) const {
            setVariable<float>("x", x);
            setVariable<float>("y", y);
        }
    };
};

/** MessageSpatial3D (include/flamegpu/runtime/messaging/MessageSpatial3D/MessageSpatial3DDevice.cuh). */
class MessageSpatial3D {
 public:
    class Description;
    class In : public SpatialIn<3> {
     public:
        __device__ explicit In(const detail::Launch& l) : SpatialIn<3>(l) {}
        __device__ Filter operator()(float x, float y, float z) const { return Filter(L, x, y, z); }
        __device__ WrapFilter wrap(float x, float y, float z) const {
            if (!wrap_ok(x, y, z)) return WrapFilter(L, L.grid().min[0], L.grid().min[1], L.grid().min[2]);
            return WrapFilter(L, x, y, z);
        }
    };
    class Out : public MessageOutBase {
     public:
        __device__ Out(const detail::LaunchParams& p, uint32_t idx) : MessageOutBase(p, idx) {}
        __device__ void setLocation(float x, float y, float z) const {
            setVariable<float>("x", x);
            setVariable<float>("y", y);
            setVariable<float>("z", z);
        }
    };
};

// ------------------------------------------------------- environment, random

namespace detail {
// Atomic operations on a 4- or 8-byte macro property element, through the
// native atomics where the type has them and a compare-and-swap loop on the
// element's bits otherwise.
template <typename T>
__device__ __forceinline__ auto as_word(T v) {
    static_assert(sizeof(T) == 4 || sizeof(T) == 8, "macro property atomics need 4- or 8-byte types");
    if constexpr (sizeof(T) == 4) {
        unsigned int u;
        memcpy(&u, &v, 4);
        return u;
    } else {
        unsigned long long u;
        memcpy(&u, &v, 8);
        return u;
    }
}
template <typename T, typename U>
__device__ __forceinline__ T from_word(U u) {
    T v;
    memcpy(&v, &u, sizeof(T));
    return v;
}
template <typename T>
__device__ __forceinline__ auto word_ptr(T* p) {
    if constexpr (sizeof(T) == 4) return reinterpret_cast<unsigned int*>(p);
    else return reinterpret_cast<unsigned long long*>(p);
}
// old value of *p, *p replaced by f(old)
template <typename T, typename F>
__device__ __forceinline__ T atomic_update(T* p, F f) {
    auto* w = word_ptr(p);
    auto old = *reinterpret_cast<volatile decltype(as_word(T{}))*>(w);
    while (true) {
        const auto seen = atomicCAS(w, old, as_word<T>(f(from_word<T>(old))));
        if (seen == old) return from_word<T>(old);
        old = seen;
    }
}
template <typename T>
__device__ __forceinline__ T atomic_add(T* p, T v) {
    if constexpr (std::is_same<T, float>::value || std::is_same<T, double>::value || std::is_same<T, int>::value ||
                  std::is_same<T, unsigned int>::value || std::is_same<T, unsigned long long>::value) {
        return atomicAdd(p, v);
    } else if constexpr (std::is_integral<T>::value && sizeof(T) == 8) {
        // two's complement: the unsigned sum has the same bits
        return static_cast<T>(atomicAdd(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(v)));
    } else if constexpr (std::is_integral<T>::value && sizeof(T) == 4) {
        return static_cast<T>(atomicAdd(reinterpret_cast<unsigned int*>(p), static_cast<unsigned int>(v)));
    } else {
        return atomic_update(p, [v](T o) { return o + v; });
    }
}
template <typename T>
__device__ __forceinline__ T atomic_sub(T* p, T v) {
    if constexpr (std::is_integral<T>::value) {
        using U = typename std::conditional<sizeof(T) == 8, unsigned long long, unsigned int>::type;
        return static_cast<T>(atomicAdd(reinterpret_cast<U*>(p), static_cast<U>(0) - static_cast<U>(v)));
    } else {
        return atomic_add(p, static_cast<T>(-v));
    }
}
template <typename T>
__device__ __forceinline__ T atomic_min(T* p, T v) {
    if constexpr (std::is_same<T, int>::value || std::is_same<T, unsigned int>::value ||
                  std::is_same<T, long long>::value || std::is_same<T, unsigned long long>::value) {
        return atomicMin(p, v);
    } else if constexpr (std::is_same<T, long>::value || std::is_same<T, unsigned long>::value) {
        using U = typename std::conditional<std::is_signed<T>::value, long long, unsigned long long>::type;
        return static_cast<T>(atomicMin(reinterpret_cast<U*>(p), static_cast<U>(v)));
    } else {
        return atomic_update(p, [v](T o) { return v < o ? v : o; });
    }
}
template <typename T>
__device__ __forceinline__ T atomic_max(T* p, T v) {
    if constexpr (std::is_same<T, int>::value || std::is_same<T, unsigned int>::value ||
                  std::is_same<T, long long>::value || std::is_same<T, unsigned long long>::value) {
        return atomicMax(p, v);
    } else if constexpr (std::is_same<T, long>::value || std::is_same<T, unsigned long>::value) {
        using U = typename std::conditional<std::is_signed<T>::value, long long, unsigned long long>::type;
        return static_cast<T>(atomicMax(reinterpret_cast<U*>(p), static_cast<U>(v)));
    } else {
        return atomic_update(p, [v](T o) { return v > o ? v : o; });
    }
}
}  // namespace detail

/**
 * DeviceMacroProperty<T, I, J, K, W> (include/flamegpu/runtime/environment/
 * DeviceMacroProperty.cuh:88-205): an agent function's view of an
 * environment macro property. operator[] selects along the first dimension
 * (an index past it is a device error, and the view stays at element 0); a
 * view of one element reads as T and updates atomically: +=, -=, addAtomic /
 * subAtomic (the new value), + and - (plain reads), ++ and -- (pre: the new
 * value, post: the old), min / max (the value left), CAS (the old value),
 * exchange (the old value). Within one agent function a property is either
 * read or updated (the reference's rule; not checked here).
 */
template <typename T, flamegpu::size_type I = 1, flamegpu::size_type J = 1, flamegpu::size_type K = 1,
          flamegpu::size_type W = 1>
class DeviceMacroProperty {
 public:
    __device__ DeviceMacroProperty(const detail::LaunchParams& p, T* at, uint32_t* f) : P(p), ptr(at), flag(f) {}
    __device__ DeviceMacroProperty<T, J, K, W, 1> operator[](unsigned int i) const {
        if (i >= I) {
            detail::device_error(P, detail::kDevArrayIndex, 0, i);
            return DeviceMacroProperty<T, J, K, W, 1>(P, nullptr, nullptr);
        }
        return DeviceMacroProperty<T, J, K, W, 1>(P, ptr ? ptr + static_cast<size_t>(i) * J * K * W : nullptr, flag);
    }
    __device__ operator T() const { return read() ? *reinterpret_cast<const volatile T*>(ptr) : T{}; }
    __device__ DeviceMacroProperty& operator+=(T v) {
        if (update()) detail::atomic_add(ptr, v);
        return *this;
    }
    __device__ DeviceMacroProperty& operator-=(T v) {
        if (update()) detail::atomic_sub(ptr, v);
        return *this;
    }
    __device__ T addAtomic(T v) { return update() ? detail::atomic_add(ptr, v) + v : T{}; }
    __device__ T subAtomic(T v) { return update() ? detail::atomic_sub(ptr, v) - v : T{}; }
    __device__ T operator+(T v) const { return static_cast<T>(*this) + v; }
    __device__ T operator-(T v) const { return static_cast<T>(*this) - v; }
    __device__ T operator++() { return update() ? detail::atomic_add(ptr, static_cast<T>(1)) + static_cast<T>(1) : T{}; }
    __device__ T operator--() { return update() ? detail::atomic_sub(ptr, static_cast<T>(1)) - static_cast<T>(1) : T{}; }
    __device__ T operator++(int) { return update() ? detail::atomic_add(ptr, static_cast<T>(1)) : T{}; }
    __device__ T operator--(int) { return update() ? detail::atomic_sub(ptr, static_cast<T>(1)) : T{}; }
    __device__ T min(T v) {
        if (!update()) return T{};
        const T old = detail::atomic_min(ptr, v);
        return v < old ? v : old;
    }
    __device__ T max(T v) {
        if (!update()) return T{};
        const T old = detail::atomic_max(ptr, v);
        return v > old ? v : old;
    }
    __device__ T CAS(T compare, T v) {
        if (!update()) return T{};
        return detail::from_word<T>(atomicCAS(detail::word_ptr(ptr), detail::as_word(compare), detail::as_word(v)));
    }
    __device__ T exchange(T v) {
        if (!update()) return T{};
        return detail::from_word<T>(atomicExch(detail::word_ptr(ptr), detail::as_word(v)));
    }

 private:
    // With device checks on, the property's flag word records a read (1) and
    // an update (2) in this agent function; both is a device error
    // (DeviceMacroProperty.cuh:219-235).
    __device__ bool read() const {
        if (!ptr) return false;
#if FLAMEGPU_SEATBELTS
        if ((atomicOr(flag, 1u) & 2u) != 0u) detail::device_error(P, detail::kDevMacroConflict, 0, 0);
#endif
        return true;
    }
    __device__ bool update() const {
        if (!ptr) return false;
#if FLAMEGPU_SEATBELTS
        if ((atomicOr(flag, 2u) & 1u) != 0u) detail::device_error(P, detail::kDevMacroConflict, 0, 0);
#endif
        return true;
    }
    const detail::LaunchParams& P;
    T* ptr;         // null after a device error: reads give 0, updates do nothing
    uint32_t* flag;  // read / update record of the whole property
};

/** Read-only environment properties (include/flamegpu/runtime/environment/DeviceEnvironment.cuh). */
class DeviceEnvironment {
 public:
    __device__ explicit DeviceEnvironment(const detail::Launch& l) : L(l), P(l.P) {}
    // env table pointers are offsets into the instance's environment buffer
    template <typename T>
    __device__ T getProperty(detail::VarName name) const {
        const T* off = detail::var_addr<T>(P, &P.T.env, name.hash, 0, 0);
        return detail::ldg_any(reinterpret_cast<const T*>(L.env() + reinterpret_cast<size_t>(off)));
    }
    template <typename T, flamegpu::size_type N>
    __device__ T getProperty(detail::VarName name, unsigned int i) const {
        const T* off = detail::var_addr<T>(P, &P.T.env, name.hash, 0, i);
        return detail::ldg_any(reinterpret_cast<const T*>(L.env() + reinterpret_cast<size_t>(off)));
    }
    /** DeviceEnvironment::getMacroProperty (DeviceEnvironment.cuh:95-112). A
     *  name that is not a macro property of this type and these dimensions is
     *  a device error, and the view then reads 0 and ignores updates. */
    template <typename T, flamegpu::size_type I = 1, flamegpu::size_type J = 1, flamegpu::size_type K = 1,
              flamegpu::size_type W = 1>
    __device__ DeviceMacroProperty<T, I, J, K, W> getMacroProperty(detail::VarName name) const {
        const detail::VarTable* t = &P.T.env;
        const detail::VarSlot* vs = &t->slot[detail::table_slot(t->mult, t->shift, name.hash)];
        // a macro property's slot holds the offset of its flag word as its stride (never 0)
        if (vs->hash != name.hash || vs->stride == 0 || vs->elem_bytes != sizeof(T) || vs->elements != I * J * K * W) {
            detail::device_error(P, vs->hash != name.hash ? detail::kDevUnknownVariable : detail::kDevTypeMismatch,
                                 name.hash, 0);
            return DeviceMacroProperty<T, I, J, K, W>(P, nullptr, nullptr);
        }
        char* env = const_cast<char*>(L.env());
        return DeviceMacroProperty<T, I, J, K, W>(P, reinterpret_cast<T*>(env + reinterpret_cast<size_t>(vs->ptr)),
                                                  reinterpret_cast<uint32_t*>(env + vs->stride));
    }

 private:
    const detail::Launch L;
    const detail::LaunchParams& P;
};

/**
 * Per-agent random numbers (include/flamegpu/runtime/random/AgentRandom.cuh).
 * Counter-based: draw k of agent index i in step s of function f is a
 * SplitMix64 hash of (seed, f, s, i, k); no per-thread generator state is
 * kept. The reference's curand Philox values are not reproduced; the
 * distributions and ranges are the reference's: uniform() in [0, 1),
 * uniform(min, max) in [min, max] for integers and min + (max - min) * [0, 1)
 * for floating point (min > max is a device error with seatbelts on),
 * normal() standard normal, logNormal(mean, stddev) = exp(mean + stddev *
 * normal()), poisson(mean) Poisson distributed.
 */
class AgentRandom {
 public:
    __device__ AgentRandom(const detail::Launch& l, uint32_t idx) : L(l), P(l.P), index(idx) {}
    template <typename T>
    __device__ T uniform() const;
    template <typename T>
    __device__ T uniform(T min, T max) const;
    template <typename T>
    __device__ T normal() const;
    template <typename T>
    __device__ T logNormal(T mean, T stddev) const;
    /** Poisson distributed count with the given mean (AgentRandom.cuh:50; 0 for mean <= 0). */
    __device__ unsigned int poisson(double mean = 1.0) const;

 private:
    __device__ uint64_t next() const {
        const uint64_t key = detail::mix64(L.seed() ^ (static_cast<uint64_t>(P.fn_uid) << 40) ^ L.step());
        return detail::mix64(detail::mix64(key + index) + (counter++));
    }
    const detail::Launch L;
    const detail::LaunchParams& P;
    uint32_t index;
    mutable uint32_t counter = 0;
};
template <>
__device__ inline float AgentRandom::uniform<float>() const {
    return static_cast<float>(next() >> 40) * (1.0f / 16777216.0f);
}
template <>
__device__ inline double AgentRandom::uniform<double>() const {
    return static_cast<double>(next() >> 11) * (1.0 / 9007199254740992.0);
}
template <>
__device__ inline float AgentRandom::normal<float>() const {
    const float u1 = 1.0f - uniform<float>(), u2 = uniform<float>();
    return sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2);
}
template <>
__device__ inline double AgentRandom::normal<double>() const {
    const double u1 = 1.0 - uniform<double>(), u2 = uniform<double>();
    return sqrt(-2.0 * log(u1)) * cospi(2.0 * u2);
}
template <>
__device__ inline float AgentRandom::logNormal<float>(float mean, float stddev) const {
    return expf(mean + stddev * normal<float>());
}
template <>
__device__ inline double AgentRandom::logNormal<double>(double mean, double stddev) const {
    return exp(mean + stddev * normal<double>());
}
// Means below kPoissonSmall: Knuth's product of uniforms (The Art of Computer
// Programming, vol. 2, 3.4.1): the count of factors before the running
// product falls to exp(-mean). Larger means: Hormann's transformed rejection
// with squeeze, PTRS ("The transformed rejection method for generating
// Poisson random variables", Insurance: Mathematics and Economics 12, 1993),
// which accepts about nine draws in ten. Both loops are bounded: past the
// bound (a probability far below 2^-60) the nearest integer to the mean is
// returned.
constexpr double kPoissonSmall = 10.0;
__device__ inline unsigned int AgentRandom::poisson(double mean) const {
    if (!(mean > 0.0)) return 0u;
    if (mean < kPoissonSmall) {
        const double limit = exp(-mean);
        double prod = 1.0;
        for (unsigned int k = 0; k < 1024u; ++k) {
            prod *= uniform<double>();
            if (prod <= limit) return k;
        }
        return static_cast<unsigned int>(floor(mean + 0.5));
    }
    const double slam = sqrt(mean), loglam = log(mean);
    const double b = 0.931 + 2.53 * slam;
    const double a = -0.059 + 0.02483 * b;
    const double inv_alpha = 1.1239 + 1.1328 / (b - 3.4);
    const double v_r = 0.9277 - 3.6224 / (b - 2.0);
    for (int it = 0; it < 64; ++it) {
        const double u = uniform<double>() - 0.5;
        const double v = uniform<double>();
        const double us = 0.5 - fabs(u);
        if (us <= 0.0) continue;
        const double k = floor((2.0 * a / us + b) * u + mean + 0.43);
        if (us >= 0.07 && v <= v_r) return static_cast<unsigned int>(k);
        if (k < 0.0 || (us < 0.013 && v > us)) continue;
        if (log(v) + log(inv_alpha) - log(a / (us * us) + b) <= -mean + k * loglam - lgamma(k + 1.0))
            return static_cast<unsigned int>(k);
    }
    return static_cast<unsigned int>(floor(mean + 0.5));
}
template <typename T>
__device__ inline T AgentRandom::uniform(T min, T max) const {
#if FLAMEGPU_SEATBELTS
    if (min > max) detail::device_error(P, detail::kDevRandomRange, 0, index);
#endif
    if constexpr (std::is_integral<T>::value) {
        const uint64_t span = static_cast<uint64_t>(static_cast<int64_t>(max) - static_cast<int64_t>(min)) + 1;
        return static_cast<T>(static_cast<int64_t>(min) + static_cast<int64_t>(next() % span));
    } else {
        return min + (max - min) * uniform<T>();
    }
}

// ------------------------------------------------------------------ DeviceAPI

/** The FLAMEGPU object of an agent function (DeviceAPI.cuh:163-401). */
template <typename MessageIn, typename MessageOut>
class DeviceAPI {
 public:
    /** agent_out: birth of at most one agent per agent function call (DeviceAPI.cuh:187-236). */
    class AgentOut {
     public:
        __device__ AgentOut(const detail::Launch& l, uint32_t idx) : L(l), P(l.P), index(idx) {}
        template <typename T>
        __device__ void setVariable(detail::VarName name, T value) const {
            if (!start(name)) return;
            detail::write_var<T>(P, &P.T.birth, name.hash, index, value);
        }
        template <typename T, flamegpu::size_type N>
        __device__ void setVariable(detail::VarName name, unsigned int i, T value) const {
            if (!start(name)) return;
            detail::write_var<T>(P, &P.T.birth, name.hash, index, value, i);
        }
        /** The new agent's id (DeviceAPI.cuh:546-557 of the reference: an atomic
         * increment of the output agent's next id). A birth whose id is never
         * asked for gets it when the step appends the new agents (next id +
         * birth rank, deterministic); one that asks claims it here, and keeps it. */
        __device__ id_t getID() const {
            if (!start_row(0u)) return ID_NOT_SET;
            if (is_born != 2u) {
                // a batch keeps one next id per instance
                claimed = atomicAdd(P.birth_next_id + L.inst(), 1u);
                detail::write_var<id_t>(P, &P.T.birth, detail::VarName("_id").hash, index, claimed);
                is_born = 2u;
            }
            return claimed;
        }
        /** Claims the new agent's id now (DeviceAPI.cuh:548-557 of the reference); getID() returns it. */
        __device__ void genID() const { (void)getID(); }
        __device__ uint32_t born() const { return is_born; }

     private:
        // First write of a birth: fill the staging row with the defaults.
        __device__ bool start(const detail::VarName& name) const {
            if (name.reserved && P.birth_flags) {
                detail::device_error(P, detail::kDevReservedName, name.hash, index);
                return false;
            }
            return start_row(name.hash);
        }
        __device__ bool start_row(uint32_t hash) const {
            if (!P.birth_flags) {
                detail::device_error(P, detail::kDevBirthNotEnabled, hash, index);
                return false;
            }
            if (!is_born) {
                is_born = 1;
                // few lanes of a warp give birth, so what it costs is the
                // instructions: one store per 4- or 8-byte variable, its value in
                // the launch's parameters (copied byte by byte over every slot of
                // a name table, ten steps of 1,048,576 agents with 14% births of
                // ten variables took 37.1 us a launch against 21.9)
                for (uint32_t v = 0; v < P.T.birth_defaults; ++v) {
                    const detail::BirthDefault& d = P.T.birth_default[v];
                    char* o = d.column + static_cast<size_t>(index) * d.bytes;
                    if (d.bytes == 4u) {
                        *reinterpret_cast<uint32_t*>(o) = static_cast<uint32_t>(d.value);
                    } else if (d.bytes == 8u) {
                        *reinterpret_cast<uint64_t*>(o) = d.value;
                    } else {
                        const char* src = reinterpret_cast<const char*>(d.value);
                        for (uint32_t b = 0; b < d.bytes; ++b) o[b] = src[b];
                    }
                }
            }
            return true;
        }
        const detail::Launch L;
        const detail::LaunchParams& P;
        uint32_t index;
        mutable uint32_t is_born = 0;  // 1: born, 2: born and its id claimed
        mutable id_t claimed = ID_NOT_SET;
    };

    /** msg_row: the row this agent's output message takes (the agent's index
     *  among those running the function). */
    __device__ DeviceAPI(const detail::Launch& l, uint32_t idx, uint32_t msg_row)
        : message_in(l), message_out(l, msg_row), agent_out(l, idx), environment(l), random(l, idx), L(l), P(l.P),
          index(idx) {}

    template <typename T>
    __device__ T getVariable(detail::VarName name) const {
        return detail::read_rw<T>(P, &P.T.agent, name.hash, index);
    }
    template <typename T, flamegpu::size_type N>
    __device__ T getVariable(detail::VarName name, unsigned int i) const {
        return detail::read_rw<T>(P, &P.T.agent, name.hash, index, i);
    }
    template <typename T>
    __device__ void setVariable(detail::VarName name, T value) {
#if FLAMEGPU_SEATBELTS
        if (name.reserved) {
            detail::device_error(P, detail::kDevReservedName, name.hash, index);
            return;
        }
#endif
        detail::write_var<T>(P, &P.T.agent, name.hash, index, value);
        if constexpr (std::is_same<T, float>::value) {  // the position, kept for the launch's epilogue
            if (name.hash == detail::VarName("x").hash) { pos[0] = value; pos_set |= 1u; }
            if (name.hash == detail::VarName("y").hash) { pos[1] = value; pos_set |= 2u; }
            if (name.hash == detail::VarName("z").hash) { pos[2] = value; pos_set |= 4u; }
        }
    }
    template <typename T, flamegpu::size_type N>
    __device__ void setVariable(detail::VarName name, unsigned int i, T value) {
        detail::write_var<T>(P, &P.T.agent, name.hash, index, value, i);
    }
    __device__ id_t getID() const { return detail::read_rw<id_t>(P, &P.T.agent, detail::VarName("_id").hash, index); }
    __device__ unsigned int getStepCounter() const { return L.step(); }
    __device__ unsigned int getIndex() const { return index - L.row_begin(); }
    /** Whether the function runs on agents of this name / in this state
     *  (DeviceAPI.cuh:366-380 of the reference; names compared by hash). */
    __device__ bool isAgent(const char* agent_name) const { return detail::fnv1a32(agent_name, ~0u) == P.agent_hash; }
    __device__ bool isState(const char* agent_state) const { return detail::fnv1a32(agent_state, ~0u) == P.state_hash; }

    typename MessageIn::In message_in;
    typename MessageOut::Out message_out;
    AgentOut agent_out;
    DeviceEnvironment environment;
    AgentRandom random;
    // float x, y, z this function set (bits 1, 2, 4 of pos_set), for the
    // launch's epilogue
    float pos[3] = {0.0f, 0.0f, 0.0f};
    uint32_t pos_set = 0;

 private:
    const detail::Launch L;
    const detail::LaunchParams& P;
    uint32_t index;
};

/** ReadOnlyDeviceAPI (DeviceAPI.cuh:42-142 of the reference): what an agent
 *  function condition may use — the agent's variables and id, the step
 *  counter, environment properties and random numbers; nothing is written. */
class ReadOnlyDeviceAPI {
 public:
    __device__ ReadOnlyDeviceAPI(const detail::Launch& l, uint32_t idx)
        : environment(l), random(l, idx), L(l), P(l.P), index(idx) {}
    template <typename T>
    __device__ T getVariable(detail::VarName name) const {
        return detail::read_rw<T>(P, &P.T.agent, name.hash, index);
    }
    template <typename T, flamegpu::size_type N>
    __device__ T getVariable(detail::VarName name, unsigned int i) const {
        return detail::read_rw<T>(P, &P.T.agent, name.hash, index, i);
    }
    __device__ id_t getID() const { return detail::read_rw<id_t>(P, &P.T.agent, detail::VarName("_id").hash, index); }
    __device__ unsigned int getStepCounter() const { return L.step(); }
    __device__ unsigned int getIndex() const { return index - L.row_begin(); }
    __device__ bool isAgent(const char* agent_name) const { return detail::fnv1a32(agent_name, ~0u) == P.agent_hash; }
    __device__ bool isState(const char* agent_state) const { return detail::fnv1a32(agent_state, ~0u) == P.state_hash; }

    DeviceEnvironment environment;
    AgentRandom random;

 private:
    const detail::Launch L;
    const detail::LaunchParams& P;
    uint32_t index;
};

#endif  // __CUDACC__

}  // namespace flamegpu

#endif  // INCLUDE_FLAMEGPU_RUNTIME_DEVICEAPI_CUH_
