// One search step of the DoubleSweep-light depth-first search, shared by the plain and
// batched kernels.  Device-only.
//
// A lane's search state is four 32-bit words kept in registers:
//   avail  candidate columns of the current row still to be searched below
//   nc     columns without a queen
//   l      columns of the NEXT row attacked along the left diagonals from above this row
//   r      columns of this row attacked along the right diagonals
// plus `sp`, the shared-memory byte address of the top entry of the lane's stack of
// pending rows.  Entries of a lane sit BLOCK x 16 bytes apart ([level][BLOCK] layout), so
// the 32 lanes of a warp touch 32 consecutive 16-byte slots and an LDS.128 / STS.128 needs
// no bank replays.
//
// Per step: if the row has no candidate left, pop the deepest pending row; place the
// lowest candidate b (avail & (avail - 1) is the row without it, and their XOR is b); push
// the row back only if candidates remain; step to the next
// row and "enter" it.  A row left without candidates is not pushed, so a row with one
// free column is filled without creating a branch point: the reference's unit-row
// propagation (GPU_NQueens.cu:392-408, n_queens.cuh:145-163).  The next row's masks are
// nc & ~b, l + 2b and r' = (r + b) >> 1 (b is a free column, so it is in neither diagonal
// mask and adding is setting).  Keeping l one row ahead makes its update one multiply-add.
//
// The entry at `base` is a sentinel with many candidates and a row whose columns are all
// attacked.  A lane whose search is over pops it, takes its lowest bit, pushes the rest back
// into the same slot and enters a row without candidates: nothing is counted, and no
// instruction guards the stack's bottom.  Each pop uses up one of the sentinel's bits, so the
// kernels call refresh_sentinel at least every kMaxParkedSteps steps.
//
// Entering a row counts every candidate of the row as a node at once: the search places
// each of them exactly once, so nodes = the sum of the candidate counts of the rows
// entered (the same placements the reference's kernel loop makes, unit and branch alike).
// A row entered with one free column is the last row: its candidate, if any, completes a
// board (a solution).
//
// Dead ends are then counted without being visited.  Placing candidate c leaves the next
// row with the candidates G & ~{c-1, c, c+1}, where G = nc & ~(l | (r >> 1)) are the
// columns free two rows down from the queens above (c's own column and diagonals aside).
// So c has a child exactly when G has a column g <= c - 2 or g >= c + 2, that is when c is
// above lowest(G) + 1 or below highest(G) - 1.  With H = 2G, which needs no right shift
// (2nc & ~(2l | r)), H ^ -H are the bits above lowest(G) + 1 and 0x1FFFFFFF >> clz(H) those
// below highest(G) - 1.  All other candidates are
// leaves, whose nodes were just counted, and are removed from `avail` before the row is
// searched.  At N=17..21 this removes 36% of the placements from the step loop.  The last
// row is always removed this way (G is at most its own column), so no step ever places a
// queen there, and a row entered by a step always has a candidate.
//
// What bounds a step: instruction issue and the shared-memory pipe (an LDS.128 and an
// STS.128, 4 wavefronts each whenever some lane of each 8 takes part) together.  At N=19,
// depth 7 a warp step issues 28.3 instructions (84% of the issue slots) and keeps the
// shared-memory pipe 93% busy; with five instructions taken out it runs 8% faster, at 98%
// of that pipe.  The step before it, with a filter for one-column G only, a compare that
// guarded the stack's bottom, and shifts where this one has multiply-adds, issued 32.2
// instructions and made 3.6% more steps: 1/16 of the N=20 depth-7 pool (1.18e11 nodes)
// took 80.2 ms against 71.7 ms.
//
// Stack bound: a row is pushed only while another candidate remains, and pushed rows are
// strictly deeper towards the top, so a search from a state with f free columns holds at
// most f - 1 entries.  Kernels check that bound once per item, so the step itself carries
// no bounds check.  Built with NQB_CHECKS (the checked library), every push is also
// compared with `top`, the lane's last slot: a push past it is dropped and sets bit 0 of the
// lane's `err`, which the kernels report as a device error.
//
// Lane counters are 32-bit: one step adds at most 31 nodes, so kernels fold them into
// 64-bit totals at least every 2^27 / 31 steps.
#pragma once

#include <cstdint>

namespace nqb {

// The sentinel.  Its row has two columns (29 and 30), both attacked there and in the rows
// after it, which the bits placed one after another (27 of them, all lower) do not change.
constexpr uint32_t kSentinelAvail = 0x07FFFFFFu, kSentinelNc = 0x60000000u, kSentinelL = 0xF0000000u;
constexpr int kMaxParkedSteps = 26;  // steps a parked lane may take between refreshes of its sentinel

struct Lane {
    uint32_t avail, nc, l, r;
    uint32_t sp;     // shared byte address of the top entry; == base when the stack is empty
    uint32_t sols;   // solutions since the last fold
    uint32_t nodes;  // placements since the last fold
    uint32_t placed; // instrumented kernels: steps that placed a queen since the last fold
    uint32_t err;    // NQB_CHECKS builds: bit 0 = a push would have passed the lane's last slot
};

// The candidates of the two rows a pair of steps entered (before dead ends are dropped).
struct StepInfo {
    uint32_t cand0, cand1;
};

// A stack entry's words lie in the order nc, avail, r, l (here and in the step): with
// avail, nc, l, r the step runs 1% slower, by the compiler's choice of registers alone.
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.y), "=r"(v.x), "=r"(v.w), "=r"(v.z)
                 : "r"(addr)
                 : "memory");
    return v;
}

__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.y), "r"(v.x), "r"(v.w), "r"(v.z)
                 : "memory");
}

__device__ __forceinline__ void write_sentinel(uint32_t addr) {
    sts128(addr, make_uint4(kSentinelAvail, kSentinelNc, kSentinelL, 0u));
}

// Gives the sentinel all its bits back.  Every lane may do so at any time: the slot at `base`
// never holds anything else.
__device__ __forceinline__ void refresh_sentinel(uint32_t base) {
    asm volatile("st.shared.u32 [%0+4], %1;" ::"r"(base), "r"(kSentinelAvail) : "memory");
}

// Candidates `a` of a row minus those whose placement leaves the next row empty (see the
// file comment); masks as in Lane.  Same arithmetic as the step's.
__device__ __forceinline__ uint32_t drop_leaves(uint32_t a, uint32_t nc, uint32_t l, uint32_t r) {
    const uint32_t h = (nc << 1) & ~((l << 1) | r);
    return h ? a & ((h ^ (0u - h)) | (0x1FFFFFFFu >> __clz(h))) : 0u;
}

// PTX of one step from the registers {a, n, l, r} into {A, N, L, R}: the previous and the next
// step's avail, nc, l, r.  `push` is the push of the quad {a, n, l, r}; c receives the
// candidates of the row entered.
#define NQB_STEP(a, n, l, r, A, N, L, R, c, push, count)                                                 \
    "setp.eq.u32 p, " a ", 0;\n\t" /* no candidate left: pop */                                          \
    count                                                                                                \
    "@p ld.shared.v4.u32 {" n ", " a ", " r ", " l "}, [%4];\n\t"                                        \
    "@p sub.u32 %4, %4, %10;\n\t"                                                                        \
    "sub.u32 x, " a ", 1;\n\t"                                                                           \
    "not.b32 w, x;\n\t"                                                                                  \
    "and.b32 b, " a ", w;\n\t"     /* the row's lowest candidate b */                                    \
    "and.b32 " a ", " a ", x;\n\t" /* the row without it */                                              \
    "setp.ne.u32 t, " a ", 0;\n\t" /* candidates remain: push the row */                                 \
    push                                                                                                 \
    "not.b32 x, b;\n\t"                                                                                  \
    "and.b32 " N ", " n ", x;\n\t"                                                                       \
    "mad.lo.u32 x, b, 2, " l ";\n\t"                                                                     \
    "shl.b32 " L ", x, 1;\n\t"                                                                           \
    "shl.b32 h, x, 2;\n\t"                                                                               \
    "add.u32 w, " r ", b;\n\t"                                                                           \
    "shr.u32 " R ", w, 1;\n\t"                                                                           \
    "or.b32 w, x, " R ";\n\t"                                                                            \
    "not.b32 w, w;\n\t"                                                                                  \
    "and.b32 " A ", " N ", w;\n\t" /* candidates of the entered row */                                   \
    "popc.b32 " c ", " A ";\n\t"                                                                         \
    "sub.u32 w, " N ", 1;\n\t"                                                                           \
    "and.b32 w, w, " N ";\n\t"                                                                           \
    "setp.eq.u32 u, w, 0;\n\t"        /* one free column: the last row */                                \
    "@u add.u32 %5, %5, " c ";\n\t"   /* its candidate is a solution */                                  \
    "shl.b32 x, " N ", 1;\n\t"                                                                           \
    "or.b32 w, h, " R ";\n\t"                                                                            \
    "not.b32 w, w;\n\t"                                                                                  \
    "and.b32 h, x, w;\n\t"            /* H */                                                            \
    "neg.s32 w, h;\n\t"                                                                                  \
    "xor.b32 w, w, h;\n\t"            /* above lowest(G) + 1 */                                          \
    "bfind.shiftamt.u32 x, h;\n\t"    /* clz(H), all ones for H = 0 */                                   \
    "shr.u32 x, k, x;\n\t"            /* below highest(G) - 1 */                                         \
    "or.b32 w, w, x;\n\t"                                                                                \
    "and.b32 " A ", " A ", w;\n\t"    /* drop the leaves */

#ifndef NQB_CHECKS
#define NQB_PUSH(a, n, l, r)       \
    "@t add.u32 %4, %4, %10;\n\t" \
    "@t st.shared.v4.u32 [%4], {" n ", " a ", " r ", " l "};\n\t"
#else
#define NQB_PUSH(a, n, l, r)                                          \
    "add.u32 x, %4, %10;\n\t" /* the push's slot must not pass top */ \
    "setp.gt.u32 ov, x, %12;\n\t"                                     \
    "and.pred ok, t, !ov;\n\t"                                        \
    "@ok mov.u32 %4, x;\n\t"                                          \
    "@ok st.shared.v4.u32 [%4], {" n ", " a ", " r ", " l "};\n\t"    \
    "and.pred ov, t, ov;\n\t"                                         \
    "@ov or.b32 %8, %8, 1;\n\t"
#endif

// Counts a step that places a queen: one that does not pop the sentinel.
#define NQB_COUNT_PLACED                 \
    "setp.ne.or.u32 q, %4, %11, !p;\n\t" \
    "@q add.u32 %9, %9, 1;\n\t"

#define NQB_TWO_STEPS(count)                                                                                    \
    asm volatile(                                                                                               \
        "{\n\t.reg .pred p, q, t, u, ov, ok;\n\t.reg .u32 b, x, h, w, k, a1, n1, l1, r1;\n\t"                   \
        "mov.u32 k, 0x1FFFFFFF;\n\t"                                                                            \
        NQB_STEP("%0", "%1", "%2", "%3", "a1", "n1", "l1", "r1", "%6", NQB_PUSH("%0", "%1", "%2", "%3"), count) \
        NQB_STEP("a1", "n1", "l1", "r1", "%0", "%1", "%2", "%3", "%7", NQB_PUSH("a1", "n1", "l1", "r1"), count) \
        "}"                                                                                                     \
        : "+r"(s.avail), "+r"(s.nc), "+r"(s.l), "+r"(s.r), "+r"(s.sp), "+r"(s.sols), "=&r"(o.cand0),            \
          "=&r"(o.cand1), "+r"(s.err), "+r"(s.placed)                                                           \
        : "n"(STRIDE), "r"(base), "r"(top)                                                                      \
        : "memory")

// Two steps (their candidate counts then join the node count in one addition); STRIDE is the byte distance between a lane's stack entries (BLOCK x 16); `top` is
// the byte address of the lane's last stack slot (checked builds only); LANES: s.placed counts
// the steps that place a queen.
template <int STRIDE, bool LANES>
__device__ __forceinline__ StepInfo search_two_steps(Lane& s, uint32_t base, uint32_t top) {
    StepInfo o;
    if (LANES) NQB_TWO_STEPS(NQB_COUNT_PLACED);
    else NQB_TWO_STEPS("");
    s.nodes += o.cand0 + o.cand1;  // each candidate is placed once: nodes
    return o;
}

// Loads a state {cols, ldiag, rdiag, meta} into a lane with an empty stack and enters its
// row: the lane's node and solution counters are set to that row's (a complete board handed
// in counts one solution).  Returns the stack depth the search needs (free columns - 1).
__device__ __forceinline__ uint32_t lane_load(Lane& s, const uint4 st, uint32_t base) {
    const uint32_t n = (st.w >> 8) & 0xFFu;
    const uint32_t mask = n >= 32 ? 0xFFFFFFFFu : ((1u << n) - 1u);
    s.nc = mask & ~st.x;
    s.l = st.y << 1;
    s.r = st.z;
    s.sp = base;
    const uint32_t a = s.nc & ~(st.y | st.z);
    const uint32_t pc = __popc(a);
    s.nodes = pc;
    s.sols = (s.nc & (s.nc - 1u)) == 0 ? pc + (s.nc == 0) : 0u;
    s.avail = drop_leaves(a, s.nc, s.l, s.r);
    const uint32_t f = __popc(s.nc);
    return f ? f - 1 : 0;
}

// Empties a lane: the next step pops the sentinel.
__device__ __forceinline__ void lane_park(Lane& s, uint32_t base) {
    s.avail = 0;
    s.nc = s.l = s.r = 0;
    s.sp = base;
}

// Re-splits work inside a warp: lanes with pending rows (`donors`) hand their shallowest one,
// the largest piece of what they have left, to the warp's idle lanes.  The receiver searches it
// as a new piece of the donor's item, from the bottom of its own stack (`base0`); the
// handed-over row's slot becomes the donor's sentinel, so its `base` moves up one slot.  All
// 32 lanes call it; `idle` and `donors` are their ballots.
template <int STRIDE>
__device__ __forceinline__ void share_rows(Lane& s, uint32_t& base, uint32_t base0, uint32_t& weight, uint32_t& item,
                                           uint32_t idle, uint32_t donors, uint32_t lane) {
    constexpr unsigned kAll = 0xFFFFFFFFu;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const uint32_t k = min(__popc(idle), __popc(donors));
    const uint32_t ri = __popc(idle & lt_mask);    // rank among idle lanes
    const uint32_t rd = __popc(donors & lt_mask);  // rank among donors
    const bool recv = ((idle >> lane) & 1u) && ri < k;
    const bool give = ((donors >> lane) & 1u) && rd < k;
    uint32_t src = lane;
    if (recv) {  // lane of the ri-th donor
        uint32_t m = donors;
        for (uint32_t j = 0; j < ri; ++j) m &= m - 1u;
        src = __ffs(m) - 1;
    }
    const uint32_t slot = __shfl_sync(kAll, base + STRIDE, src);  // donor's bottom row
    const uint32_t dw = __shfl_sync(kAll, weight, src);
    const uint32_t ditem = __shfl_sync(kAll, item, src);
    __syncwarp();
    if (recv) {
        const uint4 e = lds128(slot);
        base = base0;
        write_sentinel(base0);
        s.avail = e.x;
        s.nc = e.y;
        s.l = e.z;
        s.r = e.w;
        s.sp = base;
        weight = dw;
        item = ditem;
    }
    __syncwarp();
    if (give) {
        base += STRIDE;
        write_sentinel(base);
    }
}

__device__ __forceinline__ unsigned warp_or(unsigned v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v |= __shfl_down_sync(0xFFFFFFFFu, v, o);
    return v;
}

__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
    return v;
}

}  // namespace nqb
