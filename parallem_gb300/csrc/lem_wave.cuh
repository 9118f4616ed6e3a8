// lem_wave.cuh -- helpers shared by the two dependency waves (accumulation and
// sediment routing): float-float arithmetic, warp lists, donor tests.
#pragma once

#include <cooperative_groups.h>

#include "lem_ctx.cuh"

namespace lem {

// Unevaluated sum hi + lo of two floats (Knuth two-sum), ~44 significant bits.
__device__ __forceinline__ float2 ff_add(float2 a, float2 b) {
    const float s = __fadd_rn(a.x, b.x);
    const float bb = __fsub_rn(s, a.x);
    float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(b.x, bb));
    e = __fadd_rn(e, __fadd_rn(a.y, b.y));
    const float hi = __fadd_rn(s, e);
    return make_float2(hi, __fsub_rn(e, __fsub_rn(hi, s)));
}
__device__ __forceinline__ float2 ff_scale(float2 a, float p) {
    const float h = __fmul_rn(a.x, p);
    const float e = __fmaf_rn(a.x, p, -h);
    const float l = __fmaf_rn(a.y, p, e);
    const float hi = __fadd_rn(h, l);
    return make_float2(hi, __fsub_rn(l, __fsub_rn(hi, h)));
}
// order-preserving key of a canonical float-float value
__device__ __forceinline__ uint32_t fkey(float f) {
    uint32_t b = __float_as_uint(f);
    if (b == 0x80000000u) b = 0;
    return (b >> 31) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ unsigned long long ffkey(float2 v) {
    return ((unsigned long long)fkey(v.x) << 32) | fkey(v.y);
}

__device__ __forceinline__ int wsum(int v) { return __reduce_add_sync(0xffffffffu, v); }

__device__ __forceinline__ void wave_append(bool pred, int32_t value, int32_t* list, int32_t* count, int cap,
                                            uint32_t* err) {
    unsigned ballot = __ballot_sync(0xffffffffu, pred);
    if (!ballot) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(ballot) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(count, __popc(ballot));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pred) {
        const int pos = base + __popc(ballot & ((1u << lane) - 1));
        if (pos < cap)
            list[pos] = value;
        else
            raise_error(err, ErrFlags::kCapacity);
    }
}

// The neighbour in direction d of cell (x, y) donates to it when its code has
// the bit of the opposite direction.
__device__ __forceinline__ bool donates(uint8_t code_n, int d) { return (code_n & dir_bit((d + 4) & 7)) != 0; }

constexpr int32_t kBlocked = 0x40000000;  // pending flag of a cell with a donor that never completes

// Decrement with acquire-release semantics: the release publishes this
// thread's earlier stores (the finished cell) to whichever thread sees the
// count reach zero, and the acquire lets that thread read every donor.
__device__ __forceinline__ int32_t dec_acq_rel(int32_t* p) {
    int32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], -1;" : "=r"(old) : "l"(p) : "memory");
    return old;
}

// The general dependency wave (several receivers, contributing counts, steps the
// tiled waves cannot take), run by every thread of a cooperative launch.  Each
// cell's word counts its donors still to come in the low four bits (kBlocked:
// one never comes), and carries its donors that take part (bit k: direction
// scan_dir(k)) and its receivers that do (bits of its code), so that lowering a
// receiver's count brings all that is needed to go on with it.
//
// The ready cells stand in one list in which every cell appears once.  A warp
// without a cell holds a ticket, a place of the list, and watches it; a warp
// that finishes a cell lowers its receivers' counts, goes on with the first that
// became ready and appends the others, so a front spreads over all warps however
// few cells start ready.  inflight counts the cells ready and unfinished; the
// wave ends when it is 0.
//
// Bound by the chain of cells on the longest path: the last donor's release, the
// donors' values and the sum in order.  A warp takes one cell at a time, so no
// cell waits for another's turn (a lane per cell: 1.4 times as long), a lane
// reads each donor and lowers each receiver's count.  When each lane walked cells
// of its own and kept the ones it made ready, a smooth slope with few sources
// ran on as many lanes: 5 us a cell over all cells.
constexpr int32_t kWordReady = kBlocked | 15;  // the bits that are 0 in a ready cell's word
__device__ __forceinline__ int32_t wave_word(int count_and_block, uint32_t donors, uint32_t receivers) {
    return count_and_block | (int32_t)(donors << 8) | (int32_t)(receivers << 16);
}
constexpr int kWaveSpin = 1 << 26;  // polls of an idle warp before it gives up

// index step of direction d in a grid of width W
__device__ __forceinline__ int32_t grid_step(int d, int W) { return dir_dy(d) * W + dir_dx(d); }

// Op::donor(c, k, on) is called by every lane: lane k < 8 with its bit of the
// donors set (on) reads its donor's part; Op::cell(c, donors, part) combines the
// parts in scan order and stores cell c from lane 0.  The list starts with
// counters[0] cells.  Returns the cells this warp finished, in lane 0.
template <class Op>
__device__ int wave_walk(const Op& op, int32_t* word, int32_t* list, int W, int H, DevScalars* sc) {
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    const int32_t N = W * H;
    const size_t gtid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t gstride = (size_t)gridDim.x * blockDim.x;
    const int lane = threadIdx.x & 31;
    int32_t* const tail = &sc->counters[0];
    int32_t* const head = &sc->counters[1];
    int32_t* const inflight = &sc->counters[2];
    int32_t* const stop = &sc->counters[3];
    const int nin = *tail;
    if (nin == 0) return 0;  // the same in every thread
    for (size_t i = nin + gtid; i < (size_t)N; i += gstride) list[i] = -1;
    if (gtid == 0) {
        *head = *stop = 0;
        *inflight = nin;
    }
    grid.sync();
    const int b = lane & 7;  // a lane's receiver: bit b of the code
    const int32_t to = grid_step((b + 2) & 7, W);
    int done = 0;
    for (;;) {
        int32_t ticket = 0;
        if (lane == 0) ticket = atomicAdd(head, 1);
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        int32_t cur = -1;
        for (int spin = 0;; ++spin) {
            if (lane == 0 && ticket < N) cur = *((volatile int32_t*)(list + ticket));
            cur = __shfl_sync(0xffffffffu, cur, 0);
            if (cur >= 0) break;
            int end = 0;
            if (lane == 0 && (spin & 15) == 15) {  // seldom: every waiting warp reads this one word
                end = *((volatile int32_t*)inflight) == 0 || *((volatile int32_t*)stop);
                if (!end && spin > kWaveSpin) {
                    raise_error(&sc->err, ErrFlags::kNoConverge);
                    atomicExch(stop, 1);
                    end = 1;
                }
            }
            if (__shfl_sync(0xffffffffu, end, 0)) break;
            __nanosleep(32);
        }
        if (cur < 0) break;
        __threadfence();  // the donors' values, after the cell
        int32_t info = __ldcg(word + cur);
        while (cur >= 0) {
            const uint32_t donors = (uint32_t)(info >> 8) & 255u;
            op.cell(cur, donors, op.donor(cur, b, lane < 8 && ((donors >> b) & 1u)));
            ++done;
            __syncwarp();
            __threadfence();  // the finished cell, before its receivers' counts
            const bool on = lane < 8 && ((info >> (16 + b)) & 1);
            int32_t old = 0;
            if (on) old = atomicSub(word + cur + to, 1);
            const unsigned rdy = __ballot_sync(0xffffffffu, on && (old & kWordReady) == 1);
            __threadfence();  // the other donors' values, after the counts
            if (!rdy) break;
            const int first = __ffs(rdy) - 1, rest = __popc(rdy) - 1;
            if (rest) {
                int base = 0;
                if (lane == 0) {
                    atomicAdd(inflight, rest);
                    base = atomicAdd(tail, rest);
                    __threadfence();
                }
                base = __shfl_sync(0xffffffffu, base, 0);
                if (((rdy >> lane) & 1u) && lane != first)
                    *((volatile int32_t*)(list + base + __popc(rdy & ((1u << lane) - 1u)) - 1)) = cur + to;
            }
            cur += grid_step((first + 2) & 7, W);
            info = __shfl_sync(0xffffffffu, old, first);
        }
        if (lane == 0) atomicSub(inflight, 1);
    }
    return lane == 0 ? done : 0;
}

// ---------------------------------------------------------------------------
// 32x32 tiles of the two waves: cell classes of the halo, the kind of a cell's
// receiver, and the halo ring in a fixed order.
constexpr int kTH = kTile + 2;  // tile with its one-cell halo
constexpr uint8_t kKindIn = 0, kKindOutlet = 1, kKindEnd = 2;  // receiver: in the tile / in another tile / none
constexpr uint8_t kCellOff = 0;    // never a donor (outside the grid; for accumulation also nodata outside the catchment)
constexpr uint8_t kCellIn = 1;     // a cell the wave computes
constexpr uint8_t kCellBlock = 2;  // a donor that never completes

__device__ __forceinline__ bool in_tile(int lx, int ly) { return lx >= 0 && lx < kTile && ly >= 0 && ly < kTile; }
// index step of direction d inside a tile (row-major, kTile cells per row)
__device__ __forceinline__ int tile_step(int d) { return dir_dy(d) * kTile + dir_dx(d); }

// The outlets of a 32x32 tile (cells whose receiver lies in another tile) in
// cell order, with each outlet's slot: warp w ballots rows 4w..4w+3, and a
// prefix over the 8 warps' counts places them.  Called by all 256 threads;
// s_wcnt holds 8 ints; the caller synchronises before reading the lists.
__device__ __forceinline__ void list_outlets(const uint8_t* s_kind, int16_t* s_olist, int16_t* s_oslot, int* s_no,
                                             int* s_wcnt) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned m[4];
    int cnt = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        m[r] = __ballot_sync(0xffffffffu, s_kind[(4 * w + r) * kTile + lane] == kKindOutlet);
        cnt += __popc(m[r]);
    }
    if (lane == 0) s_wcnt[w] = cnt;
    __syncthreads();
    int base = 0;
    for (int i = 0; i < w; ++i) base += s_wcnt[i];
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int l = (4 * w + r) * kTile + lane;
        if ((m[r] >> lane) & 1u) {
            const int pos = base + __popc(m[r] & below);
            s_olist[pos] = (int16_t)l;
            s_oslot[l] = (int16_t)pos;
        }
        base += __popc(m[r]);
    }
    if (threadIdx.x == 255) *s_no = base;  // the last warp's end is the total
}

// Exclusive prefix sums over a tile's outlets (at most kTileEnt), by warp 0.
// Each count packs two numbers, one per 16-bit half, whose sums fit in theirs.
__device__ __forceinline__ void outlet_starts(const int32_t* s_count, int32_t* s_start, int no) {
    const int lane = threadIdx.x & 31;
    int carry = 0;
    for (int b = 0; b < no; b += 32) {
        const int v = b + lane < no ? s_count[b + lane] : 0;
        int incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += u;
        }
        if (b + lane < no) s_start[b + lane] = carry + incl - v;
        carry += __shfl_sync(0xffffffffu, incl, 31);
    }
}

// The halo ring in a fixed order: top row, bottom row, left column, right column.
constexpr int kRing = 4 * kTH - 4;
constexpr int kRingChunks = (kRing + 31) / 32;
__device__ __forceinline__ int ring_halo(int i) {
    if (i < kTH) return i;
    if (i < 2 * kTH) return (kTH - 1) * kTH + (i - kTH);
    if (i < 2 * kTH + kTile) return (i - 2 * kTH + 1) * kTH;
    return (i - 2 * kTH - kTile + 1) * kTH + kTH - 1;
}

// The in-tile dependency wave of one block, in rounds: a round takes every
// queued cell (all its donors in the tile finished), computes it with
// op(c, round), which returns the in-tile receiver it releases (or -1), and
// queues that receiver when c was its last donor.  Cells are queued once, in
// an order where every donor comes before its receiver.  Rounds with at least
// kWaveBlockMin cells (the first ones: the sources) run on every thread of the
// block; the narrow rounds after them run on warp 0 alone, with a warp barrier
// between rounds and the queue appended by ballot, while the block's other
// warps wait at one block barrier (the SM runs other blocks meanwhile).
constexpr int kWaveBlockMin = 96;
template <class Op>
__device__ __forceinline__ void tile_wave(const Op& op, int32_t* s_pend, int16_t* s_q, int* s_qn, int* s_end,
                                          const bool (&src)[4], int lx, int ly0) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (src[q]) s_q[atomicAdd(s_qn, 1)] = (int16_t)((ly0 + 8 * q) * kTile + lx);
    int start = 0, end = 0, round = 0;
    for (;; ++round) {
        __syncthreads();
        if (threadIdx.x == 0) *s_end = *s_qn;
        __syncthreads();
        end = *s_end;
        if (end - start < kWaveBlockMin) break;  // block-uniform
        for (int i = start + threadIdx.x; i < end; i += blockDim.x) {
            const int c = s_q[i];
            const int r = op(c, round);
            if (r >= 0 && atomicSub(&s_pend[r], 1) == 1) s_q[atomicAdd(s_qn, 1)] = (int16_t)r;
        }
        start = end;
    }
    if (threadIdx.x < 32) {
        const unsigned below = (1u << (threadIdx.x & 31)) - 1u;
        int qn = end;  // every append of the block rounds is in: the barrier above came after them
        for (; start < end && round <= kTile * kTile; ++round) {
            for (int i0 = start; i0 < end; i0 += 32) {
                const int i = i0 + (int)threadIdx.x;
                int r = -1;
                if (i < end) {
                    r = op(s_q[i], round);
                    if (r >= 0 && atomicSub(&s_pend[r], 1) != 1) r = -1;
                }
                const unsigned b = __ballot_sync(0xffffffffu, r >= 0);
                if (r >= 0) s_q[qn + __popc(b & below)] = (int16_t)r;
                qn += __popc(b);
            }
            __syncwarp();  // the round's cells and queue entries, for the next round
            start = end;
            end = qn;
        }
        if (threadIdx.x == 0) *s_qn = qn;
    }
    __syncthreads();
}

}  // namespace lem
