// Plain form: one thread per pool state, the drop-in for kern_doitall_v2_regld
// (GPU_NQueens.cu:338-452) and its launch in gpu_solver_driver (GPU_NQueens.cu:128-138).
//
// Each thread starts the depth-first search of search_step.cuh from its state.  States differ
// widely in size, so every kUnroll steps a warp looks at its idle lanes: lanes with pending
// rows hand them the shallowest one (share_rows), and the warp leaves once every lane is done
// (the reference's warps wait for their largest state; GPU_NQueens.cu:358-360).  What bounds
// the kernel is the step (search_step.cuh) in nearly all of its lanes: without the sharing
// 64% of the lane-steps placed a queen.  N=19 counts (pool depths 6 and 7, whole calls) take
// 153.6 ms against 241.1 ms without it.  The persistent queue of batched.cu is no faster on
// a fine pool (half of the N=19 depth-7 pool: 77.3 ms against 77.1 ms here); it adds stealing
// across warps, which pays where few items leave whole warps without work.
// Counters are 32-bit per lane and are folded into 64-bit totals every kEpoch rounds, so no
// lane counter can wrap.  Counts are reduced per warp with shuffles and per block through
// shared memory, then added with one uint64 atomic per block (the reference adds one atomic
// per thread, GPU_NQueens.cu:441-443).
#include <algorithm>

#include "nqb_internal.h"
#include "search_step.cuh"

namespace nqb {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;
constexpr uint32_t kNoItem = 0xFFFFFFFFu;
constexpr int kUnroll = 48;  // steps between looks at the idle lanes (24 and 72: 1.2% slower at N=19)
constexpr int kRefresh = 24;  // steps between refreshes of the lanes' sentinels
static_assert(kRefresh <= kMaxParkedSteps, "a parked lane would pop past its sentinel");
constexpr uint32_t kEpoch = (1u << 27) / kUnroll;  // rounds between folds: 31 nodes x kUnroll x kEpoch < 2^32

// Error flags written to out[3].
constexpr unsigned kErrStack = 1u;  // a state needed a deeper stack than provided
constexpr unsigned kErrBound = 2u;  // checked builds: a push would have passed a lane's last slot

// per_state (optional, zero at launch): weight x completions of each state, for per-board
// results.
// UNIT: also count placements made by unit-row propagation (the reference's split of
// nodes: the candidate of a row entered with exactly one candidate, other than the start
// row).  lane_stats (optional, LANES builds): {lane-steps that placed a queen, lane-step
// slots issued (32 per warp step)}: their ratio is the search loop's warp execution
// efficiency in active lanes.  LEVEL: states, count and board_of come from `level`, for
// launches whose host has not waited to learn them (N=14 counts 141 -> 128 us); an instance of
// its own, since the same branch in the others cost the N=19 counts 3%.
template <int BLOCK, bool UNIT, bool LANES, bool LEVEL>
__global__ void __launch_bounds__(BLOCK) plain_search_kernel(const uint4* states, uint32_t count,
                                                             unsigned long long* __restrict__ out,
                                                             unsigned long long* __restrict__ per_state,
                                                             const uint32_t* board_of, const ItemLevel* level,
                                                             unsigned long long* __restrict__ lane_stats,
                                                             uint32_t stack_depth) {
    extern __shared__ uint4 stack[];  // [stack_depth + 1][BLOCK]; row 0 holds the sentinels
    constexpr int kStride = BLOCK * 16;
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    if (LEVEL) {
        states = level->items;
        count = level->n;
        board_of = level->board;
        if (blockIdx.x * BLOCK >= count) return;
    }
    const uint32_t base0 = (uint32_t)__cvta_generic_to_shared(stack) + tid * 16;
    const uint32_t top = base0 + stack_depth * kStride;  // the lane's last slot
    uint32_t base = base0;
    write_sentinel(base0);

    Lane s;
    lane_park(s, base);
    s.sols = 0;
    s.nodes = 0;
    s.err = 0;
    s.placed = 0;
    uint32_t weight = 0, item = kNoItem;
    bool bad = false;
    auto take = [&](uint32_t i) {  // the lane's state: i, if there is one
        s.sols = 0;
        s.nodes = 0;
        if (i >= count) return;
        base = base0;
        write_sentinel(base0);
        const uint4 st = __ldg(states + i);
        if (lane_load(s, st, base) > stack_depth) {
            bad = true;  // skip the state: its search could overrun the stack
            lane_park(s, base);
            s.sols = 0;
            s.nodes = 0;
        } else {
            weight = (st.w >> 16) & 0xFFu;
            item = i;
        }
    };
    uint32_t gi = blockIdx.x * BLOCK + tid;
    take(gi);
    unsigned long long piece = 0, c = 0, nodes = 0, unit64 = 0, placed64 = 0, rounds = 0;
    uint32_t unit = 0;
    uint32_t epoch = kEpoch;
    for (;;) {
        const bool me_idle = s.avail == 0 && s.sp == base;
        const uint32_t idle = __ballot_sync(kFull, me_idle);
        if (idle) {
            if (me_idle && item != kNoItem) {  // the lane's piece of its state is complete
                const unsigned long long w = (piece + s.sols) * weight;
                c += w;
                if (per_state && w) atomicAdd(per_state + (board_of ? __ldg(board_of + item) : item), w);
                piece = 0;
                s.sols = 0;
                item = kNoItem;
            }
            if (idle == kFull) {
                if (!LEVEL) break;
                // a level may hold more states than the grid was sized for
                gi += gridDim.x * BLOCK;
                if (gi - lane >= count) break;
                nodes += s.nodes;
                take(gi);
            }
            const uint32_t donors = __ballot_sync(kFull, s.sp != base);
            if (donors) share_rows<kStride>(s, base, base0, weight, item, idle, donors, lane);
        }
        if (--epoch == 0) {  // fold lane counters before they can wrap
            piece += s.sols;
            nodes += s.nodes;
            s.sols = s.nodes = 0;
            unit64 += unit;
            placed64 += s.placed;
            unit = s.placed = 0;
            epoch = kEpoch;
        }
        if (LANES) ++rounds;
#pragma unroll
        for (int u = 0; u < kUnroll; u += 2) {
            if (u % kRefresh == 0) refresh_sentinel(base);
            const StepInfo si = search_two_steps<kStride, LANES>(s, base, top);
            if (UNIT) unit += (si.cand0 == 1u) + (si.cand1 == 1u);
        }
    }
    nodes += s.nodes;
    unit64 += unit;
    placed64 += s.placed;
    if (LANES) {
        const unsigned long long pw = warp_sum_u64(placed64);
        if (lane == 0) {
            atomicAdd(lane_stats + 0, pw);
            atomicAdd(lane_stats + 1, 32ull * kUnroll * rounds);
        }
    }

    unsigned long long un = unit64;
    c = warp_sum_u64(c);
    nodes = warp_sum_u64(nodes);
    if (UNIT) un = warp_sum_u64(un);
    const unsigned flags = (__any_sync(kFull, bad) ? kErrStack : 0u) | (__any_sync(kFull, s.err != 0) ? kErrBound : 0u);

    __syncthreads();  // the stack area is reused for the block reduction
    unsigned long long* red = reinterpret_cast<unsigned long long*>(stack);
    const uint32_t warp = tid >> 5;
    constexpr int kWarps = BLOCK / 32;
    if (lane == 0) {
        red[warp] = c;
        red[kWarps + warp] = nodes;
        red[2 * kWarps + warp] = un;
        red[3 * kWarps + warp] = flags;
    }
    __syncthreads();
    if (warp == 0) {
        c = lane < kWarps ? red[lane] : 0;
        nodes = lane < kWarps ? red[kWarps + lane] : 0;
        un = lane < kWarps ? red[2 * kWarps + lane] : 0;
        const unsigned of = warp_or(lane < kWarps ? (unsigned)red[3 * kWarps + lane] : 0u);
        c = warp_sum_u64(c);
        nodes = warp_sum_u64(nodes);
        un = warp_sum_u64(un);
        if (lane == 0) {
            if (c) atomicAdd(out + 0, c);
            atomicAdd(out + 1, nodes);
            if (UNIT && un) atomicAdd(out + 2, un);
            if (of) atomicOr(out + 3, (unsigned long long)of);
        }
    }
}

template <int BLOCK, bool UNIT, bool LANES, bool LEVEL>
int launch_t(const nqb_state* d_states, uint64_t count, unsigned long long* d_out,
             unsigned long long* d_per_state, const uint32_t* d_board_of, const ItemLevel* d_level,
             unsigned long long* d_lanes,
             unsigned stack_depth, cudaStream_t stream, unsigned* launches) {
    auto kern = plain_search_kernel<BLOCK, UNIT, LANES, LEVEL>;
    // Room for the stack (with its sentinel row), and for 4 x (BLOCK/32) reduction words.
    const size_t smem = std::max<size_t>((size_t)(stack_depth + 1) * BLOCK * sizeof(uint4),
                                         4 * (BLOCK / 32) * sizeof(unsigned long long));
    if (smem > kMaxDynamicSmem) return NQB_E_RANGE;
    NQB_TRY(allow_dynamic_smem(kern));
    const uint64_t kChunk = 1ull << 30;  // states per launch (grid.x stays < 2^31)
    const uint4* base = reinterpret_cast<const uint4*>(d_states);
    for (uint64_t off = 0; off < count; off += kChunk) {
        const uint32_t c = (uint32_t)std::min<uint64_t>(kChunk, count - off);
        const unsigned grid = (c + BLOCK - 1) / BLOCK;
        // without a slot map, a chunk's slots start at its first state
        kern<<<grid, BLOCK, smem, stream>>>(base + off, c, d_out,
                                            d_per_state && !d_board_of ? d_per_state + off : d_per_state,
                                            d_board_of ? d_board_of + off : nullptr, d_level, d_lanes, stack_depth);
        NQB_TRY(cuda_status(cudaGetLastError()));
        if (launches) (*launches)++;
    }
    return NQB_OK;
}

template <int BLOCK>
int launch_block(const nqb_state* d_states, uint64_t count, unsigned long long* d_out,
                 unsigned long long* d_per_state, const uint32_t* d_board_of, const ItemLevel* d_level,
             unsigned long long* d_lanes,
                 bool count_unit, unsigned stack_depth, cudaStream_t stream, unsigned* launches) {
    auto launch = d_level ? (d_lanes ? (count_unit ? launch_t<BLOCK, true, true, true> : launch_t<BLOCK, false, true, true>)
                                     : (count_unit ? launch_t<BLOCK, true, false, true>
                                                   : launch_t<BLOCK, false, false, true>))
                          : (d_lanes ? (count_unit ? launch_t<BLOCK, true, true, false>
                                                   : launch_t<BLOCK, false, true, false>)
                                     : (count_unit ? launch_t<BLOCK, true, false, false>
                                                   : launch_t<BLOCK, false, false, false>));
    return launch(d_states, count, d_out, d_per_state, d_board_of, d_level, d_lanes, stack_depth, stream, launches);
}

}  // namespace

int launch_plain(const nqb_state* d_states, uint64_t count, unsigned long long* d_out,
                 unsigned long long* d_per_state, int block_size, bool count_unit, unsigned stack_depth,
                 cudaStream_t stream, unsigned* launches, unsigned long long* d_lane_stats,
                 const uint32_t* d_board_of, const ItemLevel* d_level) {
    if (!d_out || (count && !d_states && !d_level)) return NQB_E_INVALID;
    if (count == 0) return NQB_OK;
    if (stack_depth == 0) stack_depth = NQB_MAX_N - 1;
    if (stack_depth > NQB_MAX_N) return NQB_E_INVALID;
    if (block_size == 0) block_size = 128;
    switch (block_size) {
        case 64:
            return launch_block<64>(d_states, count, d_out, d_per_state, d_board_of, d_level, d_lane_stats, count_unit, stack_depth,
                                    stream, launches);
        case 128:
            return launch_block<128>(d_states, count, d_out, d_per_state, d_board_of, d_level, d_lane_stats, count_unit, stack_depth,
                                     stream, launches);
        case 256:
            return launch_block<256>(d_states, count, d_out, d_per_state, d_board_of, d_level, d_lane_stats, count_unit, stack_depth,
                                     stream, launches);
        default:
            return NQB_E_INVALID;
    }
}

}  // namespace nqb
