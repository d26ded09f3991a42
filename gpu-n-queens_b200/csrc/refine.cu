// Splits the items of a launch that has too few of them, and builds the pools of small counts.
//
// A search kernel keeps its lanes busy only while it has several items a lane: with fewer,
// the time goes into handing pieces of long subtrees from lane to lane and from warp to warp.
// Before such a launch the items are split into their children, level by level, until there
// are kItemsPerLane a lane: a device pass over a few hundred thousand 16-byte items against a
// search of milliseconds.
//
// One level: an item with many free columns is replaced by its children, one per candidate
// of its next row that has a child itself (the step's leaf filter, search_step.cuh); the
// candidates are counted as nodes here, and the children are searched like any other item, so
// counts, nodes and unit nodes are those of the unsplit search.  Only items within
// kSplitSpread free columns of the largest are split, so the small boards of an uneven batch
// stay whole.  Children are appended behind an atomic count, one reservation a warp, so a level
// needs neither a scan nor a read-back; the order of the items is not kept (no result depends
// on it).  While a level writes its items it adds up how many the next level would make, so
// each level knows before it starts whether it fits the buffers, and hands its input on
// unchanged when it does not, when nothing would be split or when there are items enough.
//
// What bounds it: launch latency (a level is a few microseconds).  Batched form, whole calls:
// N=18 at pool depths 3 and 4 (1,710 and 18,132 items, split to 1.2M) 33.4 -> 19.0 ms, the time
// of the depth-6 pool; 8,192 uneven boards (n 16-20, split to 2.1M) 244 -> 215 ms.  Stopping
// at one item a lane leaves N=19 at depth 4 at 165 ms and the uneven boards at 239 ms, against
// 147.5 and 209 ms (same box) at two; at four, calls move within 4% either way.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "nqb_internal.h"
#include "search_step.cuh"

namespace nqb {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint32_t kItemsPerLane = 2;      // levels stop at this many items a resident lane
constexpr uint32_t kCapItems = 3200000;    // most room of each of the two buffers (51 MB)
constexpr uint32_t kMinSplitFree = 8;      // items with fewer free columns are a few hundred nodes
constexpr uint32_t kSplitSpread = 3;
constexpr unsigned kMaxLevels = 4;
constexpr unsigned kThreads = 256;
constexpr unsigned kMaxRecords = kMaxItemLevels;  // a pool's levels, then the split's
static_assert(kMaxRecords >= NQB_MAX_N + kMaxLevels, "one record a level");
// With fewer free columns at most, the host does not wait to learn how many items the split made:
// the search takes the number from the device.  Larger items are worth the wait (12 us), which also
// tells how deep a stack they need.
constexpr uint32_t kDeferFree = 12;
constexpr size_t kHeadBytes = 2048;
constexpr uint32_t kSeeds = 16;  // row-0 columns of the left half, at most
static_assert((NQB_MAX_N + 1) / 2 <= kSeeds, "seed_kernel writes them unasked");

using Level = ItemLevel;

__device__ __forceinline__ uint32_t free_columns(const uint4 s) {
    const uint32_t n = (s.w >> 8) & 0xFFu;
    return (n >= 32 ? 0xFFFFFFFFu : ((1u << n) - 1u)) & ~s.x;
}

// The candidates of an item's next row that have a child.
__device__ __forceinline__ uint32_t living(const uint4 s, uint32_t nc) {
    return drop_leaves(nc & ~(s.y | s.z), nc, s.y << 1, s.z);
}

// Items that `s` becomes in a level that splits from `cut` free columns on.
__device__ __forceinline__ uint32_t made_of(const uint4 s, uint32_t cut) {
    const uint32_t nc = free_columns(s);
    return (uint32_t)__popc(nc) >= cut ? __popc(living(s, nc)) : 1u;
}

__global__ void first_kernel(const uint4* __restrict__ items, const uint32_t* __restrict__ board, uint32_t n,
                             uint32_t cut, Level* __restrict__ out) {
    unsigned long long made = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        made += made_of(__ldg(items + i), cut);
    made = warp_sum_u64(made);
    if ((threadIdx.x & 31) == 0 && made) atomicAdd(&out->next, made);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        out->items = items;
        out->board = board;
        out->n = n;
    }
}

// One level: in -> out, or `in` handed on.  COUNT: the candidates of split items are counted as
// nodes (a level below the pool; the levels that build the pool split everything and count
// nothing).  UNIT: children whose row has exactly one candidate
// are counted as unit placements (a search kernel takes an item's first row for a start row).
template <bool COUNT, bool UNIT>
__global__ void __launch_bounds__(kThreads) level_kernel(const Level* __restrict__ in, Level* __restrict__ out,
                                                         uint4* __restrict__ to, uint32_t* __restrict__ to_board,
                                                         uint32_t cut, uint32_t next_cut, uint32_t room,
                                                         uint32_t enough, unsigned long long* __restrict__ totals,
                                                         unsigned long long* __restrict__ board_nodes) {
    const uint32_t n = in->n;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    if (in->next > room || (COUNT && (n >= enough || in->next == n))) {
        if (first) {
            out->items = in->items;
            out->board = in->board;
            out->n = n;
            out->next = COUNT ? n : ~0ull;  // the levels after this one hand it on too
            out->done = in->done;
        }
        return;
    }
    const uint4* const items = in->items;
    const uint32_t* const board = in->board;
    const uint32_t lane = threadIdx.x & 31;
    unsigned long long nodes = 0, made = 0;
    uint32_t units = 0;
    for (uint32_t i0 = (blockIdx.x * kThreads + threadIdx.x) & ~31u; i0 < n; i0 += gridDim.x * kThreads) {
        const uint32_t i = i0 + lane;
        const bool valid = i < n;
        const uint4 s = valid ? items[i] : make_uint4(0, 0, 0, 0);
        const uint32_t id = valid && to_board ? (board ? board[i] : i) : 0u;
        const uint32_t nc = free_columns(s);
        const bool split = valid && (uint32_t)__popc(nc) >= cut;
        const uint32_t kids = split ? living(s, nc) : 0u;
        if (COUNT && split) {
            const uint32_t placed = __popc(nc & ~(s.y | s.z));
            nodes += placed;
            if (board_nodes && placed) atomicAdd(board_nodes + id, (unsigned long long)placed);
        }
        const uint32_t c = split ? __popc(kids) : (uint32_t)valid;
        uint32_t p = c;  // inclusive prefix over the warp
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t v = __shfl_up_sync(kFull, p, d);
            if (lane >= (uint32_t)d) p += v;
        }
        const uint32_t total = __shfl_sync(kFull, p, 31);
        p -= c;
        uint32_t at = 0;
        if (lane == 0 && total) at = atomicAdd(&out->n, total);
        at = __shfl_sync(kFull, at, 0) + p;
        // total <= what `in` promised, so at + c stays inside the buffer
        uint32_t left = kids;
        for (uint32_t j = 0; j < c; ++j) {
            uint4 o = s;
            if (split) {
                const uint32_t b = left & (0u - left);
                left ^= b;
                o = make_uint4(s.x | b, (s.y | b) << 1, (s.z | b) >> 1, s.w);  // no kernel reads the row number
                if (UNIT) units += __popc(free_columns(o) & ~(o.y | o.z)) == 1;
            }
            to[at + j] = o;
            if (to_board) to_board[at + j] = id;
            made += made_of(o, next_cut);
        }
    }
    nodes = warp_sum_u64(nodes);
    made = warp_sum_u64(made);
    unsigned long long unit64 = units;
    if (UNIT) unit64 = warp_sum_u64(unit64);
    if (lane == 0) {
        if (nodes) atomicAdd(totals + 1, nodes);
        if (UNIT && unit64) atomicAdd(totals + 2, unit64);
        if (made) atomicAdd(&out->next, made);
    }
    if (first) {
        out->items = to;
        out->board = to_board;
        out->done = in->done + 1;
    }
}

// The first level of a pool: the row-0 placements of the left half whose next row has a
// candidate, weight 2 left of centre and 1 for the middle column of an odd board
// (GPU_NQueens.cu:354-357).  Also clears the level records.
__global__ void seed_kernel(uint32_t n, uint32_t next_cut, uint4* __restrict__ items, Level* __restrict__ lv) {
    const uint32_t lane = threadIdx.x;  // one warp; n <= 31
    for (uint32_t w = lane; w < kMaxRecords * sizeof(Level) / 4; w += 32) reinterpret_cast<uint32_t*>(lv)[w] = 0;
    __syncwarp();
    const uint32_t b = 1u << lane;
    const uint4 s = make_uint4(b, b << 1, b >> 1, 1u | (n << 8) | ((lane < (n >> 1) ? 2u : 1u) << 16));
    const bool kept = lane < (n + 1) / 2 && (free_columns(s) & ~(s.y | s.z));
    const uint32_t all = __ballot_sync(kFull, kept);
    if (kept) items[__popc(all & (b - 1u))] = s;
    const uint32_t made = (uint32_t)warp_sum_u64(kept ? made_of(s, next_cut) : 0);
    if (lane == 0) {
        lv->items = items;
        lv->n = __popc(all);
        lv->next = made;
    }
}

// Free columns from which level `level` of a split splits, of items that have max_free at most.
uint32_t cut_of(uint32_t max_free, unsigned level) {
    const uint32_t top = max_free - level;
    return std::max(kMinSplitFree, top > kSplitSpread ? top - kSplitSpread : 0u);
}

unsigned split_levels(uint32_t max_free) {
    return max_free <= kMinSplitFree ? 0 : std::min(kMaxLevels, max_free - kMinSplitFree);
}

// The buffers of a call's levels: the records, then two item buffers of `room` items, used in
// turn.  Room for no more than the levels can make: an N=8 count takes a few KB, only splits of
// hundreds of thousands of items take all of 2 x 51 MB (2 x 64 MB with output slots).
struct Levels {
    Level* records;
    uint4* items[2];
    uint32_t* board[2];
    uint32_t room;
    // *had = false (and NQB_OK) when the device has no memory to spare for them.
    int take(uint64_t want, bool boards, cudaStream_t s, Refined* out, bool* had) {
        static_assert(kMaxRecords * sizeof(Level) <= kHeadBytes, "the level records' room");
        room = (uint32_t)std::min<uint64_t>(want, kCapItems);
        room = (std::max(room, kSeeds) + 15u) & ~15u;  // keeps the buffers aligned
        size_t bytes = kHeadBytes + 2 * (size_t)room * (sizeof(uint4) + (boards ? sizeof(uint32_t) : 0));
#ifdef NQB_CHECKS  // tests: less room than the items need; 0: more memory than any device has
        if (const char* limit = std::getenv("NQB_SPLIT_ROOM")) {
            const uint32_t most = (uint32_t)std::strtoul(limit, nullptr, 10);
            if (most == 0) bytes = (size_t)1 << 50;
            else room = std::min(room, std::max(most, kSeeds) & ~15u);
        }
#endif
        NQB_TRY(dev_alloc_optional(&out->buf, bytes, s));
        *had = out->buf != nullptr;
        if (!*had) return NQB_OK;
        out->stream = s;
        char* at = static_cast<char*>(out->buf);
        records = reinterpret_cast<Level*>(at);
        at += kHeadBytes;
        for (int k = 0; k < 2; ++k) {
            items[k] = reinterpret_cast<uint4*>(at);
            at += (size_t)room * sizeof(uint4);
            board[k] = boards ? reinterpret_cast<uint32_t*>(at) : nullptr;
            if (boards) at += (size_t)room * sizeof(uint32_t);
        }
        return NQB_OK;
    }
};

// The most items that splitting n items of max_free free columns can make: one child a column.
uint64_t split_bound(uint32_t n, uint32_t max_free, unsigned levels) {
    uint64_t most = n;
    for (unsigned k = 0; k < levels && most < kCapItems; ++k) most *= max_free - k;
    return most;
}

}  // namespace

void Refined::release() {
    if (buf) dev_free(buf, stream);
    buf = nullptr;
}

int refine_items(const nqb_state* d_items, uint32_t n, const uint32_t* d_board, bool boards, bool unit,
                 unsigned stack_depth, int device, cudaStream_t s, unsigned long long* d_totals,
                 unsigned long long* d_board_nodes, unsigned* launches, Refined* out, bool may_defer) {
    out->items = d_items;
    out->board = d_board;
    out->n = n;
    out->stack_depth = stack_depth;
    int sms = 0;
    NQB_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)));
    const uint32_t enough = kItemsPerLane * (uint32_t)sms * 1152;  // 36 warps of an SM's stack memory
    const uint32_t max_free = stack_depth + 1;
    const unsigned levels = split_levels(max_free);
    if (n >= enough || levels == 0) return NQB_OK;
    Levels b;
    bool had = false;
    NQB_TRY(b.take(split_bound(n, max_free, levels), boards || d_board, s, out, &had));
    if (!had) return NQB_OK;  // no memory to spare: the items are searched as they are
    Level* const lv = b.records;
    NQB_TRY(cuda_status(cudaMemsetAsync(lv, 0, (levels + 1) * sizeof(Level), s)));
    const unsigned grid0 = std::max(1u, std::min((n + kThreads - 1) / kThreads, 4u * (unsigned)sms));
    first_kernel<<<grid0, kThreads, 0, s>>>(reinterpret_cast<const uint4*>(d_items), d_board, n, cut_of(max_free, 0),
                                            lv);
    for (unsigned k = 0; k < levels; ++k) {
        auto kern = unit ? level_kernel<true, true> : level_kernel<true, false>;
        kern<<<4 * sms, kThreads, 0, s>>>(lv + k, lv + k + 1, b.items[k & 1], b.board[k & 1], cut_of(max_free, k),
                                          cut_of(max_free, k + 1), b.room, enough, d_totals, d_board_nodes);
    }
    NQB_TRY(cuda_status(cudaGetLastError()));
    if (launches) *launches += 1 + levels;
    if (may_defer && max_free < kDeferFree) {
        out->level = lv + levels;
        out->n = (uint32_t)std::min<uint64_t>((uint64_t)n << (2 * levels), kCapItems);  // about 4 children a level
        return NQB_OK;
    }
    Level last;
    NQB_TRY(cuda_status(cudaMemcpyAsync(&last, lv + levels, sizeof(last), cudaMemcpyDeviceToHost, s)));
    NQB_TRY(cuda_status(cudaStreamSynchronize(s)));
    out->items = reinterpret_cast<const nqb_state*>(last.items);
    out->board = last.board;
    out->n = last.n;
    // Every item with more than max_free - done free columns has been split (a level's cut is
    // at most its largest).
    out->stack_depth = std::max(stack_depth > last.done ? stack_depth - last.done : 1u, 1u);
    return NQB_OK;
}

namespace {
// Estimated children per state of a level with `row` queens placed: 0.8 to 1.9 times the real
// ones over all levels to a depth of n / 2, n = 8..21.
double children_estimate(unsigned n, unsigned row) { return n * std::pow(1.0 - (double)row / n, 2.4); }
}  // namespace

bool small_pool(unsigned n, unsigned depth) {
    double size = (n + 1) / 2;
    for (unsigned r = 1; r < depth; ++r)
        if ((size *= children_estimate(n, r)) > 0.8 * kCapItems) return false;
    return true;
}

int small_pool_items(unsigned n, unsigned depth, bool unit, int device, cudaStream_t s, unsigned long long* d_totals,
                     unsigned* launches, Refined* out, const ItemLevel** all_levels, unsigned* n_levels,
                     cudaEvent_t pool_built) {
    int sms = 0;
    NQB_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device)));
    const uint32_t enough = kItemsPerLane * (uint32_t)sms * 1152;
    const uint32_t max_free = n - depth;
    const unsigned levels = split_levels(max_free), all = depth - 1 + levels;
    // Room for the largest level.  Over all (n, depth) that small_pool lets through the estimate is
    // 1.0 to 8 times what the levels make (replayed on the CPU); a split stops at `enough` items.
    double most = 0.0, level = (n + 1) / 2;
    for (unsigned k = 0; k <= all; ++k) {
        most = std::max(most, level);
        if (k >= depth - 1 && level >= 2.0 * enough) break;
        level *= children_estimate(n, k + 1);
    }
    Levels b;
    bool had = false;
    NQB_TRY(b.take((uint64_t)std::min<double>(most, kCapItems) + 64, false, s, out, &had));
    if (!had) return NQB_E_RANGE;  // no memory to spare: the caller builds the pool level by level
    Level* const lv = b.records;
    auto cut = [&](unsigned k) { return k < depth - 1 ? 0u : cut_of(max_free, k - (depth - 1)); };
    seed_kernel<<<1, 32, 0, s>>>(n, all ? cut(0) : 0u, b.items[1], lv);
    double size = (n + 1) / 2;  // of the level's input, for the grid
    for (unsigned k = 0; k < all; ++k) {
        if (k == depth - 1) NQB_TRY(cuda_status(cudaEventRecord(pool_built, s)));
        auto kern = k < depth - 1 ? level_kernel<false, false>
                                  : unit ? level_kernel<true, true> : level_kernel<true, false>;
        const unsigned grid = (unsigned)std::min(4.0 * sms, size / kThreads + 1.0);
        kern<<<grid, kThreads, 0, s>>>(lv + k, lv + k + 1, b.items[k & 1], nullptr, cut(k), cut(k + 1), b.room,
                                       enough, d_totals, nullptr);
        size *= children_estimate(n, k + 1);
    }
    if (all == depth - 1) NQB_TRY(cuda_status(cudaEventRecord(pool_built, s)));
    NQB_TRY(cuda_status(cudaGetLastError()));
    if (launches) *launches += 1 + all;
    *all_levels = lv;
    *n_levels = all + 1;
    out->stack_depth = max_free > 1 ? max_free - 1 : 1;
    if (max_free < kDeferFree) {
        out->level = lv + all;
        out->n = (uint32_t)std::min<double>(size * 1.25 + 1.0, kCapItems);
        return NQB_OK;
    }
    Level rec[kMaxRecords];
    NQB_TRY(cuda_status(cudaMemcpyAsync(rec, lv, (all + 1) * sizeof(Level), cudaMemcpyDeviceToHost, s)));
    NQB_TRY(cuda_status(cudaStreamSynchronize(s)));
    if (rec[depth - 1].done != depth - 1) return NQB_E_RANGE;  // a level of the pool did not fit
    const unsigned split = rec[all].done - (depth - 1);
    out->items = reinterpret_cast<const nqb_state*>(rec[all].items);
    out->n = rec[all].n;
    out->stack_depth = max_free > split + 1 ? max_free - split - 1 : 1;
    return NQB_OK;
}

}  // namespace nqb
