// Fused, order-preserving birth/death compaction (one pass over the agents).
//
// Each block owns a tile of 1024 agents, read "striped" (item k of thread t is
// agent tile*1024 + k*256 + t) so that every flag load and column copy is
// coalesced. Survivor and birth ranks inside the tile come from warp ballots;
// the tile's offsets among all tiles come from a decoupled look-back on a
// packed (survivors, births) pair. Survivors land at their rank, births at
// S + birth rank where S = total survivors, so the reference's order —
// survivors in order, then children in parent order — falls out of one kernel.
// Tile statuses live in two arrays used on alternate calls; every call clears
// the array the next call will use, so nothing is reset from the host.
//
// What bounds it: below some millions of agents, the chain of dependent round
// trips to memory in one tile (its ticket, the flags, the look-back, the
// columns). So a tile loads four columns of all its items and births at once
// (the first four while its first warp looks back), the look-back reads 128
// predecessors a round, and tiles are small enough that 200,000 agents use
// every SM. Ten steps of 1,048,576 agents of 44
// bytes, 30% dying and 14% giving birth a step: 61.0 -> 27.2 us a call (in the
// step graph; with 2,048-row tiles, one row's four columns loaded before the
// next row's, and a serial prefix over the tile's ballots); 37,000 agents of
// four columns 20.1 -> 14.3 us.
#include <algorithm>

#include "common.cuh"

namespace fgk {

constexpr int kCompItems = 4;
constexpr uint32_t kCompTile = kThreads * kCompItems;  // 1024
constexpr int kCompWarps = kThreads / 32;
static_assert(kCompItems * kCompWarps == 32, "one lane per (item, warp) count");
constexpr uint64_t kPairMask = (1ull << 62) - 1ull;

struct CompactParams {
    fg_column col[FG_MAX_COLUMNS];
    fg_column bcol[FG_MAX_COLUMNS];
    uint32_t ncols;
    int32_t id_col;
};

// Look back over predecessor tiles; returns the exclusive packed (a << 31 | b).
// Each lane reads four neighbouring predecessors, so a round covers 128. At
// most `limit` polls per predecessor (a give-up is recorded in the header).
__device__ __forceinline__ uint64_t lookback_pair(const uint64_t* status, uint32_t tile, WsHeader* h,
                                                  uint32_t limit) {
    constexpr int kPer = 4;
    const uint32_t lane = lane_id();
    uint64_t excl = 0;
    int64_t pred = static_cast<int64_t>(tile) - 1;
    while (pred >= 0) {
        const int64_t t = pred - static_cast<int64_t>(lane) * kPer;  // this lane: t, t - 1, ...
        uint64_t s[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) s[j] = t >= j ? ld_status(status + (t - j)) : (2ull << 62);
        uint64_t sum = 0;     // this lane's tiles down to its nearest inclusive prefix
        bool prefix = false;  // one of them holds one
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            uint32_t spins = 0;
            while ((s[j] >> 62) == 0) {
                if (++spins > limit) {
                    record_status(h, FG_ERR_DEVICE_TIMEOUT);
                    s[j] = 2ull << 62;
                    break;
                }
                if (spins > 16) __nanosleep(spins > 1024 ? 256 : 32);
                s[j] = ld_status(status + (t - j));
            }
            if (!prefix) sum += s[j] & kPairMask;
            prefix = prefix || (s[j] >> 62) == 2;
        }
        const uint32_t pmask = __ballot_sync(0xFFFFFFFFu, prefix);
        // lanes past the nearest one with an inclusive prefix add nothing
        uint64_t contrib = (pmask && lane > static_cast<uint32_t>(__ffs(pmask) - 1)) ? 0ull : sum;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) contrib += __shfl_xor_sync(0xFFFFFFFFu, contrib, d);
        excl += contrib;
        if (pmask) break;
        pred -= 32 * kPer;
    }
    return excl;
}

__device__ __forceinline__ void copy_col(const fg_column& c, uint32_t src, uint32_t dst) {
    switch (c.elem_bytes) {
        case 4: reinterpret_cast<uint32_t*>(c.out)[dst] = reinterpret_cast<const uint32_t*>(c.in)[src]; break;
        case 8: reinterpret_cast<uint2*>(c.out)[dst] = reinterpret_cast<const uint2*>(c.in)[src]; break;
        case 16: reinterpret_cast<uint4*>(c.out)[dst] = reinterpret_cast<const uint4*>(c.in)[src]; break;
        case 1: reinterpret_cast<uint8_t*>(c.out)[dst] = reinterpret_cast<const uint8_t*>(c.in)[src]; break;
        case 2: reinterpret_cast<uint16_t*>(c.out)[dst] = reinterpret_cast<const uint16_t*>(c.in)[src]; break;
        default: {
            const uint8_t* a = reinterpret_cast<const uint8_t*>(c.in) + static_cast<size_t>(src) * c.elem_bytes;
            uint8_t* b = reinterpret_cast<uint8_t*>(c.out) + static_cast<size_t>(dst) * c.elem_bytes;
            for (uint32_t k = 0; k < c.elem_bytes; ++k) b[k] = a[k];
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_count_alive(uint32_t max_n, const uint32_t* d_n,
                                                          const uint32_t* __restrict__ alive, WsHeader* h) {
    flamegpu::detail::grid_dependency_enter();
    const uint32_t n = d_n ? min(*d_n, max_n) : max_n;
    uint32_t c = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        c += alive[i] != 0 ? 1u : 0u;
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if (lane_id() == 0 && c) atomicAdd(&h->alive_total, c);
}

__global__ void k_set_alive_total(uint32_t max_n, const uint32_t* d_n, WsHeader* h) {
    flamegpu::detail::grid_dependency_enter();
    h->alive_total = d_n ? min(*d_n, max_n) : max_n;
}

// Row i of columns [c0, c0 + nk) written at dst; the id column of births gets `id`.
__device__ __forceinline__ void copy_row_columns(const fg_column* cols, uint32_t c0, uint32_t nk, uint32_t i,
                                                 uint32_t dst, int id_col, uint32_t id) {
    for (uint32_t k = 0; k < nk; ++k) {
        if (static_cast<int32_t>(c0 + k) == id_col)
            reinterpret_cast<uint32_t*>(cols[c0 + k].out)[dst] = id;
        else
            copy_col(cols[c0 + k], i, dst);
    }
}

__device__ __forceinline__ bool four_byte_columns(const fg_column* cols, uint32_t c0, uint32_t nk) {
    bool words = true;
    for (uint32_t k = 0; k < nk; ++k) words = words && cols[c0 + k].elem_bytes == 4u;
    return words;
}

// A birth flagged 2 claimed its id during the function: it keeps the staging row's.
constexpr uint16_t kClaimed = 0x8000u;

// Shared memory of one tile.
struct CompSmem {
    uint32_t count[32];         // (item, warp): survivors | births << 16
    uint16_t birth[kCompTile];  // the tile's births, in row order: their place in the tile, kClaimed set if the id is kept
    uint64_t excl;              // survivors << 31 | births before the tile
};

// One tile of a list (or of a batch instance's segment), by the whole block.
struct CompTile {
    const uint32_t* alive;  // flags of the list's rows (null: every row survives)
    const uint32_t* born;   // (null: no births)
    int partition;          // 1: every row not in the first group is a "birth"; 2: no row survives
    uint32_t row0;          // first row of the list in every column
    uint32_t base;          // first row of the tile, from row0
    uint32_t n;             // rows of the list
    uint32_t S;             // survivors of the list
    uint32_t capacity;      // rows the list may hold
    uint32_t next_id;
    uint64_t* status;       // the list's tile statuses
    uint32_t tile;          // the tile's place among them
    bool withhold;          // test hook: do not publish
    uint32_t limit;         // look-back polls
};

// Compacts the tile; returns (in thread 0) survivors << 31 | births up to and including it.
__device__ __forceinline__ uint64_t compact_tile(const CompactParams& cp, const CompTile& t, CompSmem& sm, WsHeader* h) {
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5, lt = lanemask_lt();
    uint32_t fa[kCompItems], fb[kCompItems];
#pragma unroll
    for (int k = 0; k < kCompItems; ++k) {
        const uint32_t i = t.base + k * kThreads + tid;
        const bool in = i < t.n;
        fa[k] = in && t.partition != 2 ? (t.alive ? t.alive[t.row0 + i] : 1u) : 0u;
        fb[k] = in && t.partition != 1 && t.born ? t.born[t.row0 + i] : 0u;
    }
    uint32_t ba[kCompItems], bb[kCompItems];
#pragma unroll
    for (int k = 0; k < kCompItems; ++k) {
        ba[k] = __ballot_sync(0xFFFFFFFFu, fa[k] != 0u);
        if (t.partition == 1) fb[k] = (t.base + k * kThreads + tid < t.n && fa[k] == 0u) ? 1u : 0u;
        bb[k] = __ballot_sync(0xFFFFFFFFu, fb[k] != 0u);
        if (lane == 0) sm.count[k * kCompWarps + warp] = __popc(ba[k]) | (__popc(bb[k]) << 16);
    }
    __syncthreads();
    // every warp scans the 32 counts: its items' offsets in the tile, and the totals
    const uint32_t mine = sm.count[lane];
    uint32_t inc = mine;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, inc, d);
        if (lane >= static_cast<uint32_t>(d)) inc += v;
    }
    const uint32_t totals = __shfl_sync(0xFFFFFFFFu, inc, 31);
    const uint32_t nbirths = totals >> 16;
    const uint64_t agg = (static_cast<uint64_t>(totals & 0xFFFFu) << 31) | nbirths;
    uint32_t off[kCompItems];  // this thread's survivors' places in the tile
#pragma unroll
    for (int k = 0; k < kCompItems; ++k) {
        const uint32_t e = __shfl_sync(0xFFFFFFFFu, inc - mine, k * kCompWarps + warp);
        off[k] = (e & 0xFFFFu) + __popc(ba[k] & lt);
        if (fb[k]) 
            sm.birth[(e >> 16) + __popc(bb[k] & lt)] =
                static_cast<uint16_t>((k * kThreads + tid) | (fb[k] == 2u ? kClaimed : 0u));
    }
    uint64_t inclusive = 0;
    if (warp == 0) {
        uint64_t excl = 0;
        if (t.tile == 0) {
            if (lane == 0 && !t.withhold) st_status(t.status, (2ull << 62) | agg);
        } else {
            if (lane == 0) st_status(t.status + t.tile, (1ull << 62) | agg);
            excl = lookback_pair(t.status, t.tile, h, t.limit);
            if (lane == 0) st_status(t.status + t.tile, (2ull << 62) | ((excl + agg) & kPairMask));
        }
        if (lane == 0) sm.excl = excl;
        inclusive = excl + agg;
    }
    // four columns at a time: the survivors' and one birth's elements are all
    // loaded before any is stored; the first four are in flight while warp 0 looks back
    uint32_t ea = 0, eb = 0, src = 0, dst = 0;
    bool ready = false, birth = false, claimed = false;
    for (uint32_t c0 = 0; c0 < cp.ncols || !ready; c0 += 4) {
        const uint32_t nk = c0 < cp.ncols ? min(4u, cp.ncols - c0) : 0u;
        const bool words = four_byte_columns(cp.col, c0, nk);
        uint32_t v[4][kCompItems];
        if (words) {
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c)
#pragma unroll
                for (int k = 0; k < kCompItems; ++k)
                    if (c < nk && fa[k])
                        v[c][k] = static_cast<const uint32_t*>(cp.col[c0 + c].in)[t.row0 + t.base + k * kThreads + tid];
        }
        if (!ready) {
            __syncthreads();
            ready = true;
            ea = static_cast<uint32_t>((sm.excl >> 31) & 0x7FFFFFFFu);
            eb = static_cast<uint32_t>(sm.excl & 0x7FFFFFFFu);
            if (tid < nbirths) {
                const uint32_t w = sm.birth[tid];
                src = t.row0 + t.base + (w & (kCompTile - 1u));
                dst = t.S + eb + tid;
                birth = dst < t.capacity;
                claimed = (w & kClaimed) != 0u;
                if (!birth) record_status(h, FG_ERR_CAPACITY);
            }
        }
        const int32_t id_at = claimed ? -1 : cp.id_col;
        if (words) {
            uint32_t bv[4];
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c)
                if (c < nk && birth)
                    bv[c] = static_cast<int32_t>(c0 + c) == id_at ? t.next_id + eb + tid
                                                                   : static_cast<const uint32_t*>(cp.bcol[c0 + c].in)[src];
#pragma unroll
            for (uint32_t c = 0; c < 4; ++c) {
                if (c >= nk) break;
                uint32_t* out = static_cast<uint32_t*>(cp.col[c0 + c].out) + t.row0;
#pragma unroll
                for (int k = 0; k < kCompItems; ++k)
                    if (fa[k] && ea + off[k] < t.capacity) out[ea + off[k]] = v[c][k];
                if (birth) out[dst] = bv[c];
            }
        } else {
#pragma unroll
            for (int k = 0; k < kCompItems; ++k)
                if (fa[k] && ea + off[k] < t.capacity)
                    copy_row_columns(cp.col, c0, nk, t.row0 + t.base + k * kThreads + tid, t.row0 + ea + off[k], -1, 0u);
            if (birth) copy_row_columns(cp.bcol, c0, nk, src, t.row0 + dst, id_at, t.next_id + eb + tid);
        }
    }
    // births past the block's first 256
    for (uint32_t j = kThreads + tid; j < nbirths; j += kThreads) {
        const uint32_t w = sm.birth[j], d = t.S + eb + j;
        if (d < t.capacity)
            copy_row_columns(cp.bcol, 0, cp.ncols, t.row0 + t.base + (w & (kCompTile - 1u)), t.row0 + d,
                             (w & kClaimed) ? -1 : cp.id_col, t.next_id + eb + j);
        else
            record_status(h, FG_ERR_CAPACITY);
    }
    return inclusive;
}

// Persistent tiles: each block takes tiles of kCompTile rows by ticket (in
// launch order) until the rows [0, n) are covered, so the grid can be a few
// blocks per SM whatever the capacity, and a small population costs a few
// tiles rather than one block per tile of capacity. A tile waits only on
// lower tiles, taken earlier by running blocks that publish their aggregate
// before they look back themselves. Blocks past the tiles of this population
// take no ticket.
__global__ void __launch_bounds__(kThreads) k_compact(const __grid_constant__ CompactParams cp, uint32_t max_n,
                                                      const uint32_t* d_n, const uint32_t* __restrict__ alive,
                                                      const uint32_t* __restrict__ born, uint32_t* d_next_id,
                                                      const uint32_t* d_alive_total, uint32_t* d_n_out,
                                                      uint32_t out_capacity, uint64_t* status0, uint32_t stride_tiles,
                                                      WsHeader* h, int partition, uint32_t* d_s_out) {
    flamegpu::detail::grid_dependency_enter();
    __shared__ uint32_t s_tile;
    __shared__ CompSmem sm;
    const uint32_t tid = threadIdx.x;
    // written by earlier launches: plain loads, all in flight at once
    const uint32_t limit = spin_limit_of(h);
    const bool withhold = h->withhold != 0;
    const uint32_t parity = h->comp_parity & 1u;
    const uint32_t n = d_n ? min(*d_n, max_n) : max_n;
    const uint32_t S = d_alive_total ? *d_alive_total : h->alive_total;
    const uint32_t next_id = d_next_id ? *d_next_id : 0u;
    uint64_t* status = status0 + static_cast<size_t>(parity) * stride_tiles;
    // clear the whole status array the next call will use (its grid may differ)
    uint64_t* other = status0 + static_cast<size_t>(parity ^ 1u) * stride_tiles;
    for (uint32_t t = blockIdx.x * blockDim.x + tid; t < stride_tiles; t += gridDim.x * blockDim.x) other[t] = 0;
    const uint32_t tiles = (n + kCompTile - 1) / kCompTile;
    while (blockIdx.x < tiles) {
        if (tid == 0) s_tile = atomicAdd(&h->comp_ticket, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= tiles) break;  // the same in every thread: no rows left
        const CompTile t{alive, born, partition, 0u, tile * kCompTile, n, S, out_capacity, next_id, status, tile, withhold, limit};
        const uint64_t inc = compact_tile(cp, t, sm, h);
        if (tid == 0 && tile + 1u == tiles) {  // the last tile: publish the births, before this block counts as done
            h->pad[0] = static_cast<uint32_t>(inc & 0x7FFFFFFFu);
            __threadfence();
        }
        __syncthreads();  // s_tile and sm are reused by the next tile
    }
    // the last block to finish publishes the new count, flips the parity and
    // resets the tickets. A block counts as done once all its warps have read
    // the list's count, next id and the parity: the barrier, which a block past
    // the population's tiles (it skips the loop) has not met before
    __syncthreads();
    if (tid == 0) {
        if (atomicAdd(&h->comp_done, 1u) == gridDim.x - 1) {
            __threadfence();
            const uint32_t births = *static_cast<volatile uint32_t*>(&h->pad[0]);
            uint32_t total = S + births;
            if (total > out_capacity) total = out_capacity;
            if (d_n_out) *d_n_out = total;
            if (d_s_out) *d_s_out = S;
            if (d_next_id && cp.id_col >= 0) *d_next_id = next_id + births;
            h->pad[0] = 0;
            h->alive_total = 0;
            h->comp_ticket = 0;
            h->comp_done = 0;
            atomicExch(&h->comp_parity, parity ^ 1u);
            __threadfence();
        }
    }
}

}  // namespace fgk

using namespace fgk;

namespace {
int launch_err() {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FG_OK : FG_ERR_CUDA;
}
uint32_t comp_tiles(uint32_t max_n) { return std::max(1u, (max_n + kCompTile - 1) / kCompTile); }
uint32_t device_sms() {
    int dev = 0, sms = 132;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return static_cast<uint32_t>(sms);
}
// persistent compaction blocks: four per SM, or one per tile of capacity if fewer
uint32_t comp_grid(uint32_t max_n) { return std::min(comp_tiles(max_n), 4u * device_sms()); }
// survivor-count blocks (grid-stride over the flags): four per SM at most
uint32_t count_grid(uint32_t max_n) {
    return std::max(1u, std::min((max_n + kThreads - 1) / kThreads, 4u * device_sms()));
}
}  // namespace

uint32_t* fgi_compact_survivor_word(void* workspace) {
    return workspace ? &reinterpret_cast<WsHeader*>(workspace)->alive_total : nullptr;
}

extern "C" size_t fg_compact_workspace_size(uint32_t max_n) {
    return sizeof(WsHeader) + align_up(sizeof(uint64_t) * 2 * comp_tiles(max_n), 256);
}

extern "C" int fg_compact_agents(uint32_t max_n, const uint32_t* d_n, const uint32_t* alive, const uint32_t* born,
                                 const fg_column* cols, const fg_column* birth_cols, uint32_t ncols, int32_t id_col,
                                 uint32_t* d_next_id, const uint32_t* d_alive_total, uint32_t* d_n_out,
                                 uint32_t out_capacity, void* workspace, size_t workspace_bytes, void* stream) {
    if (!workspace || ncols > FG_MAX_COLUMNS || (ncols && !cols)) return FG_ERR_INVALID_ARGUMENT;
    if (born && ncols && !birth_cols) return FG_ERR_INVALID_ARGUMENT;
    if (id_col >= static_cast<int32_t>(ncols)) return FG_ERR_INVALID_ARGUMENT;
    if (id_col >= 0 && cols[id_col].elem_bytes != 4) return FG_ERR_INVALID_ARGUMENT;
    if (max_n >= (1u << 31)) return FG_ERR_UNSUPPORTED;
    if (workspace_bytes < fg_compact_workspace_size(max_n) || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return FG_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    WsHeader* h = reinterpret_cast<WsHeader*>(ws);
    uint64_t* status = reinterpret_cast<uint64_t*>(ws + sizeof(WsHeader));
    const uint32_t tiles = comp_grid(max_n);
    // h->alive_total is zero here: the workspace starts zeroed
    // (fg_workspace_init) and each compaction's last block resets it
    if (!d_alive_total && alive) {
        launch(k_count_alive, count_grid(max_n), kThreads, st, max_n, d_n, alive, h);
    } else if (!d_alive_total) {
        // every agent survives: S = n
        launch(k_set_alive_total, 1, 1, st, max_n, d_n, h);
    }
    CompactParams cp{};
    for (uint32_t c = 0; c < ncols; ++c) {
        cp.col[c] = cols[c];
        cp.bcol[c] = birth_cols ? birth_cols[c] : cols[c];
    }
    cp.ncols = ncols;
    cp.id_col = id_col;
    // both status arrays are strided by the workspace's tile capacity, so a
    // workspace keeps working when max_n changes between calls
    const uint32_t stride_tiles = static_cast<uint32_t>((workspace_bytes - sizeof(WsHeader)) / (2 * sizeof(uint64_t)));
    launch(k_compact, tiles, kThreads, st, cp, max_n, d_n, alive, born, d_next_id, d_alive_total, d_n_out, out_capacity,
           status, stride_tiles, h, 0, nullptr);
    return launch_err();
}

extern "C" int fg_partition_agents(uint32_t max_n, const uint32_t* d_n, const uint32_t* first_group,
                                   const fg_column* cols, uint32_t ncols, uint32_t* d_first_count,
                                   void* workspace, size_t workspace_bytes, void* stream) {
    if (!workspace || !first_group || ncols > FG_MAX_COLUMNS || (ncols && !cols)) return FG_ERR_INVALID_ARGUMENT;
    if (max_n >= (1u << 31)) return FG_ERR_UNSUPPORTED;
    if (workspace_bytes < fg_compact_workspace_size(max_n) || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return FG_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    WsHeader* h = reinterpret_cast<WsHeader*>(ws);
    uint64_t* status = reinterpret_cast<uint64_t*>(ws + sizeof(WsHeader));
    // the first group is the compaction's "survivors" (counted first, so the
    // second group knows where it starts), the rest its "births" in row order;
    // h->alive_total is zero here (see fg_compact_agents)
    launch(k_count_alive, count_grid(max_n), kThreads, st, max_n, d_n, first_group, h);
    CompactParams cp{};
    for (uint32_t c = 0; c < ncols; ++c) cp.col[c] = cp.bcol[c] = cols[c];
    cp.ncols = ncols;
    cp.id_col = -1;
    const uint32_t stride_tiles = static_cast<uint32_t>((workspace_bytes - sizeof(WsHeader)) / (2 * sizeof(uint64_t)));
    launch(k_compact, comp_grid(max_n), kThreads, st, cp, max_n, d_n, first_group, nullptr, nullptr, nullptr, nullptr,
           max_n, status, stride_tiles, h, 1, d_first_count);
    return launch_err();
}

extern "C" int fg_append_births(uint32_t max_n, const uint32_t* d_n, const uint32_t* born, const fg_column* cols,
                                uint32_t ncols, int32_t id_col, uint32_t* d_next_id, uint32_t* d_dst_count,
                                uint32_t dst_capacity, void* workspace, size_t workspace_bytes, void* stream) {
    if (!workspace || !born || !d_dst_count || ncols > FG_MAX_COLUMNS || (ncols && !cols))
        return FG_ERR_INVALID_ARGUMENT;
    if (id_col >= static_cast<int32_t>(ncols)) return FG_ERR_INVALID_ARGUMENT;
    if (id_col >= 0 && (cols[id_col].elem_bytes != 4 || !d_next_id)) return FG_ERR_INVALID_ARGUMENT;
    if (max_n >= (1u << 31)) return FG_ERR_UNSUPPORTED;
    if (workspace_bytes < fg_compact_workspace_size(max_n) || (reinterpret_cast<uintptr_t>(workspace) & 255))
        return FG_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    WsHeader* h = reinterpret_cast<WsHeader*>(ws);
    uint64_t* status = reinterpret_cast<uint64_t*>(ws + sizeof(WsHeader));
    // births-only compaction: no survivors, "S" = the destination's count, so
    // birth r lands at *d_dst_count + r and the count grows by the births
    CompactParams cp{};
    for (uint32_t c = 0; c < ncols; ++c) cp.col[c] = cp.bcol[c] = cols[c];
    cp.ncols = ncols;
    cp.id_col = id_col;
    const uint32_t stride_tiles = static_cast<uint32_t>((workspace_bytes - sizeof(WsHeader)) / (2 * sizeof(uint64_t)));
    launch(k_compact, comp_grid(max_n), kThreads, st, cp, max_n, d_n, nullptr, born, id_col >= 0 ? d_next_id : nullptr,
           static_cast<const uint32_t*>(d_dst_count), d_dst_count, dst_capacity, status, stride_tiles, h, 2,
           nullptr);
    return launch_err();
}

namespace fgk {

// rows [begin, end) of the source columns -> rows [dst0, dst0 + end - begin) of the destination
__global__ void __launch_bounds__(kThreads) k_append_rows(const __grid_constant__ CompactParams cp, uint32_t max_rows,
                                                          const uint32_t* d_begin, const uint32_t* d_end,
                                                          const uint32_t* d_dst_count, uint32_t dst_capacity,
                                                          WsHeader* h) {
    flamegpu::detail::grid_dependency_enter();
    const uint32_t begin = d_begin ? *d_begin : 0u;
    const uint32_t end = min(*d_end, max_rows);
    const uint32_t dst0 = *d_dst_count;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; begin + r < end; r += gridDim.x * blockDim.x) {
        const uint32_t dst = dst0 + r;
        if (dst >= dst_capacity) {
            record_status(h, FG_ERR_CAPACITY);
            return;
        }
        for (uint32_t c = 0; c < cp.ncols; ++c) copy_col(cp.col[c], begin + r, dst);
    }
}

__global__ void k_append_counts(uint32_t max_rows, const uint32_t* d_begin, uint32_t* d_src_count,
                                uint32_t* d_dst_count, uint32_t dst_capacity) {
    flamegpu::detail::grid_dependency_enter();
    const uint32_t begin = d_begin ? *d_begin : 0u;
    const uint32_t end = min(*d_src_count, max_rows);
    const uint32_t moved = end > begin ? end - begin : 0u;
    const uint32_t total = *d_dst_count + moved;
    *d_dst_count = total < dst_capacity ? total : dst_capacity;
    *d_src_count = begin < end ? begin : end;
}

}  // namespace fgk

extern "C" int fg_append_rows(const fg_column* cols, uint32_t ncols, uint32_t max_rows, const uint32_t* d_begin,
                              uint32_t* d_src_count, uint32_t* d_dst_count, uint32_t dst_capacity, void* workspace,
                              size_t workspace_bytes, void* stream) {
    if (!workspace || workspace_bytes < sizeof(WsHeader) || !d_src_count || !d_dst_count || ncols > FG_MAX_COLUMNS ||
        (ncols && !cols))
        return FG_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    WsHeader* h = reinterpret_cast<WsHeader*>(workspace);
    CompactParams cp{};
    for (uint32_t c = 0; c < ncols; ++c) cp.col[c] = cols[c];
    cp.ncols = ncols;
    cp.id_col = -1;
    int dev = 0, sms = 132;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const uint32_t grid = std::max(1u, std::min((max_rows + kThreads - 1) / kThreads, static_cast<uint32_t>(sms * 8)));
    launch(k_append_rows, grid, kThreads, st, cp, max_rows, d_begin, d_src_count, d_dst_count, dst_capacity, h);
    launch(k_append_counts, 1, 1, st, max_rows, d_begin, d_src_count, d_dst_count, dst_capacity);
    return launch_err();
}

// ------------------------------------------------------ segmented (batches)
//
// The same fused compaction over a batch of instances (fg_batch_instance):
// instance k owns rows [row_begin_k, row_begin_k + row_capacity_k) of every
// column and its first counts[k] rows are its agents. Its rows are cut into
// tiles of kCompTile rows that never cross into another instance (tile_begin
// maps instances to their first tile), so one launch compacts every instance
// in place of its own segment: a tile looks back only over the tiles of its
// instance, survivors of instance k land from row_begin_k, its births after
// its S_k survivors (counted first, per instance), with ids from next_ids[k].
// The last block to finish writes every instance's new count.
namespace fgk {

__device__ __forceinline__ uint32_t batch_instance_of_row(const fg_batch_instance* inst, uint32_t ninst, uint32_t row) {
    uint32_t lo = 0, hi = ninst - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (__ldg(&inst[mid].row_begin) <= row)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// survivors per instance: rows below the instance's count with alive != 0
// (alive == NULL: every agent survives)
__global__ void __launch_bounds__(kThreads) k_count_alive_batched(const fg_batch_instance* __restrict__ inst,
                                                                  uint32_t ninst, const uint32_t* __restrict__ counts,
                                                                  uint32_t total_rows, const uint32_t* __restrict__ alive,
                                                                  uint32_t* alive_total) {
    flamegpu::detail::grid_dependency_enter();
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < total_rows; base += stride) {
        const uint32_t i = base + threadIdx.x;
        bool a = false;
        uint32_t k = 0;
        if (i < total_rows) {
            k = batch_instance_of_row(inst, ninst, i);
            const uint32_t local = i - __ldg(&inst[k].row_begin);
            a = local < __ldg(counts + k) && (alive == nullptr || alive[i] != 0);
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, a);
        if (a) {
            const uint32_t peers = __match_any_sync(m, k);
            if (lane_id() == static_cast<uint32_t>(__ffs(peers) - 1)) atomicAdd(alive_total + k, __popc(peers));
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_compact_batched(
    const __grid_constant__ CompactParams cp, const fg_batch_instance* __restrict__ inst,
    const uint32_t* __restrict__ tile_begin, uint32_t ninst, uint32_t ntiles, uint32_t* counts,
    const uint32_t* __restrict__ alive, const uint32_t* __restrict__ born, uint32_t* next_ids, uint32_t* alive_total,
    uint32_t* birth_total, uint64_t* status0, uint32_t stride_tiles, WsHeader* h) {
    flamegpu::detail::grid_dependency_enter();
    __shared__ uint32_t s_tile, s_inst, s_last;
    __shared__ CompSmem sm;
    const uint32_t tid = threadIdx.x;
    // written by earlier launches: plain loads, all in flight at once
    const uint32_t limit = spin_limit_of(h);
    const bool withhold = h->withhold != 0;
    const uint32_t parity = h->comp_parity & 1u;
    uint64_t* status = status0 + static_cast<size_t>(parity) * stride_tiles;
    uint64_t* other = status0 + static_cast<size_t>(parity ^ 1u) * stride_tiles;
    for (uint32_t t = blockIdx.x * blockDim.x + tid; t < stride_tiles; t += gridDim.x * blockDim.x) other[t] = 0;
    for (;;) {
        if (tid == 0) {
            const uint32_t t = atomicAdd(&h->comp_ticket, 1u);
            s_tile = t;
            if (t < ntiles) {  // the instance whose tiles hold t
                uint32_t lo = 0, hi = ninst - 1;
                while (lo < hi) {
                    const uint32_t mid = (lo + hi + 1) >> 1;
                    if (__ldg(tile_begin + mid) <= t)
                        lo = mid;
                    else
                        hi = mid - 1;
                }
                s_inst = lo;
            }
        }
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= ntiles) break;  // the same in every thread
        const uint32_t k = s_inst;
        const uint32_t t0 = __ldg(tile_begin + k);
        const uint32_t local = tile - t0;
        const uint32_t rb = __ldg(&inst[k].row_begin), cap = __ldg(&inst[k].row_capacity);
        const uint32_t n = min(counts[k], cap);
        const uint32_t lbase = local * kCompTile;
        if (lbase >= n) {  // no agents in this tile (nor in the instance's later ones)
            __syncthreads();
            continue;
        }
        const CompTile t{alive, born, 0, rb, lbase, n, alive_total[k], cap, next_ids ? next_ids[k] : 0u, status + t0, local,
                         withhold && tile == 0, limit};
        const uint64_t inc = compact_tile(cp, t, sm, h);
        if (tid == 0 && lbase + kCompTile >= n)  // the instance's last tile with agents: its births
            birth_total[k] = static_cast<uint32_t>(inc & 0x7FFFFFFFu);
        __syncthreads();  // shared state is reused by the next tile
    }
    // the last block to finish writes the counts and resets the tickets
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        s_last = atomicAdd(&h->comp_done, 1u) == gridDim.x - 1 ? 1u : 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (uint32_t k = tid; k < ninst; k += blockDim.x) {
        const uint32_t births = *reinterpret_cast<volatile uint32_t*>(birth_total + k);
        const uint32_t S = *reinterpret_cast<volatile uint32_t*>(alive_total + k);
        const uint32_t cap = __ldg(&inst[k].row_capacity);
        const uint32_t total = S + births;
        counts[k] = total < cap ? total : cap;
        if (next_ids && cp.id_col >= 0) next_ids[k] += births;
        birth_total[k] = 0;
        alive_total[k] = 0;
    }
    __syncthreads();
    if (tid == 0) {
        h->comp_ticket = 0;
        h->comp_done = 0;
        atomicExch(&h->comp_parity, parity ^ 1u);
        __threadfence();
    }
}

__global__ void k_set_alive_total_batched(const uint32_t* counts, uint32_t ninst, uint32_t* alive_total) {
    flamegpu::detail::grid_dependency_enter();
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < ninst; k += gridDim.x * blockDim.x)
        alive_total[k] = counts[k];
}

struct BatchCompactLayout {
    size_t alive, births, status, total;
};
inline BatchCompactLayout batch_compact_layout(uint32_t ntiles, uint32_t ninst) {
    BatchCompactLayout L;
    L.alive = sizeof(WsHeader);
    L.births = L.alive + align_up(sizeof(uint32_t) * ninst, 256);
    L.status = L.births + align_up(sizeof(uint32_t) * ninst, 256);
    L.total = L.status + align_up(sizeof(uint64_t) * 2 * std::max(ntiles, 1u), 256);
    return L;
}

}  // namespace fgk

extern "C" uint32_t fg_batch_compact_tiles(const fg_batch_instance* instances, uint32_t ninst, uint32_t* tile_begin) {
    uint32_t t = 0;
    for (uint32_t k = 0; k < ninst; ++k) {
        if (tile_begin) tile_begin[k] = t;
        t += std::max(1u, (instances[k].row_capacity + kCompTile - 1) / kCompTile);
    }
    if (tile_begin) tile_begin[ninst] = t;
    return t;
}

extern "C" size_t fg_compact_batched_workspace_size(uint32_t ntiles, uint32_t ninst) {
    return batch_compact_layout(ntiles, ninst).total;
}

extern "C" int fg_compact_agents_batched(const fg_batch_instance* instances, const uint32_t* tile_begin, uint32_t ninst,
                                         uint32_t ntiles, uint32_t total_rows, uint32_t* counts, const uint32_t* alive,
                                         const uint32_t* born, const fg_column* cols, const fg_column* birth_cols,
                                         uint32_t ncols, int32_t id_col, uint32_t* next_ids, void* workspace,
                                         size_t workspace_bytes, void* stream) {
    if (!instances || !tile_begin || !ninst || !counts || !workspace || ncols > FG_MAX_COLUMNS || (ncols && !cols))
        return FG_ERR_INVALID_ARGUMENT;
    if (born && ncols && !birth_cols) return FG_ERR_INVALID_ARGUMENT;
    if (id_col >= static_cast<int32_t>(ncols)) return FG_ERR_INVALID_ARGUMENT;
    if (id_col >= 0 && (cols[id_col].elem_bytes != 4 || !next_ids)) return FG_ERR_INVALID_ARGUMENT;
    if (total_rows >= (1u << 31)) return FG_ERR_UNSUPPORTED;
    const BatchCompactLayout L = batch_compact_layout(ntiles, ninst);
    if (workspace_bytes < L.total || (reinterpret_cast<uintptr_t>(workspace) & 255)) return FG_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    WsHeader* h = reinterpret_cast<WsHeader*>(ws);
    uint32_t* alive_total = reinterpret_cast<uint32_t*>(ws + L.alive);
    uint32_t* birth_total = reinterpret_cast<uint32_t*>(ws + L.births);
    uint64_t* status = reinterpret_cast<uint64_t*>(ws + L.status);
    // alive_total / birth_total are zero here: the workspace starts zeroed and
    // every call's last block clears them
    if (alive)
        launch(k_count_alive_batched, count_grid(total_rows), kThreads, st, instances, ninst,
               static_cast<const uint32_t*>(counts), total_rows, alive, alive_total);
    else
        launch(k_set_alive_total_batched, std::max(1u, (ninst + kThreads - 1) / kThreads), kThreads, st,
               static_cast<const uint32_t*>(counts), ninst, alive_total);
    CompactParams cp{};
    for (uint32_t c = 0; c < ncols; ++c) {
        cp.col[c] = cols[c];
        cp.bcol[c] = birth_cols ? birth_cols[c] : cols[c];
    }
    cp.ncols = ncols;
    cp.id_col = id_col;
    const uint32_t stride_tiles =
        static_cast<uint32_t>((workspace_bytes - L.status) / (2 * sizeof(uint64_t)));
    launch(k_compact_batched, std::min(ntiles, 4u * device_sms()), kThreads, st, cp, instances, tile_begin, ninst,
           ntiles, counts, alive, born, next_ids, alive_total, birth_total, status, stride_tiles, h);
    return launch_err();
}
