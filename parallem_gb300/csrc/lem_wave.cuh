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
// Polls of an idle warp, with no progress seen, before it gives up.  Progress is a
// change of the cells in flight, or of a count that a warp raises every kWaveBeat
// cells of a path: a path of one warp may hold every cell of the grid and takes about
// 1.7 us a cell (262144 cells: 0.46 s), so no fixed number of polls would do for it.
constexpr uint32_t kWaveSpin = 1 << 23;
constexpr int kWaveBeat = 256;

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
    int32_t* const beat = &sc->counters[4];
    const int nin = *tail;
    if (nin == 0) return 0;  // the same in every thread
    for (size_t i = nin + gtid; i < (size_t)N; i += gstride) list[i] = -1;
    if (gtid == 0) {
        *head = *stop = *beat = 0;
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
        int32_t seen = -1, heard = -1;  // inflight and beat when they last changed
        for (uint32_t spin = 0;; ++spin) {  // (lane 0's counts)
            if (lane == 0 && ticket < N) cur = *((volatile int32_t*)(list + ticket));
            cur = __shfl_sync(0xffffffffu, cur, 0);
            if (cur >= 0) break;
            int end = 0;
            if (lane == 0 && (spin & 15) == 15) {  // seldom: every waiting warp reads this one word
                const int32_t left = *((volatile int32_t*)inflight), at = *((volatile int32_t*)beat);
                end = left == 0 || *((volatile int32_t*)stop);
                if (left != seen || at != heard) {
                    seen = left;
                    heard = at;
                    spin = 0;
                } else if (!end && spin > kWaveSpin) {
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
            if ((++done & (kWaveBeat - 1)) == 0 && lane == 0) atomicAdd(beat, 1);
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

// The outlets of a 32x32 tile (cells whose receiver lies in another tile: kind
// kKindOutlet in `bits` of s_kind) in cell order, with each outlet's slot: warp w ballots rows 4w..4w+3, and a
// prefix over the 8 warps' counts places them.  Called by all 256 threads;
// s_wcnt holds 8 ints; the caller synchronises before reading the lists.
__device__ __forceinline__ void list_outlets(const uint8_t* s_kind, uint8_t bits, int16_t* s_olist, int16_t* s_oslot, int* s_no,
                                             int* s_wcnt) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned m[4];
    int cnt = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        m[r] = __ballot_sync(0xffffffffu, (s_kind[(4 * w + r) * kTile + lane] & bits) == kKindOutlet);
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

// Stages the direction codes and classes of a tile and its halo (256 threads; all
// loads of a thread in flight at once), class_of(grid cell, x, y) called for
// cells in the grid.  Every cell also announces itself to the cell of the tile it
// points at: s_dm (zero before, a barrier since) gets bit k of the receiver set
// when its neighbour in direction scan_dir(k) drains to it, in the low byte for
// cells of the tile and in the high byte for others; and s_bad the rows of the
// cells with a donor that never completes (a blocked cell, whose code may have
// several directions).  One push per cell in the place of eight tests.  Codes of
// more than one direction occur in blocked cells only.  The caller synchronises.
template <class ClassOf>
__device__ __forceinline__ void tile_stage(const uint8_t* __restrict__ fd, const ClassOf& class_of, int W, int H,
                                           int tx0, int ty0, uint8_t* s_code, uint8_t* s_cls, uint16_t* s_dm,
                                           uint32_t* s_bad) {
    constexpr int kTurns = (kTH * kTH + 255) / 256;
    uint8_t code[kTurns], cls[kTurns];
#pragma unroll
    for (int i = 0; i < kTurns; ++i) {
        const int j = threadIdx.x + 256 * i, hy = j / kTH, hx = j - hy * kTH;
        const int gx = tx0 - 1 + hx, gy = ty0 - 1 + hy;
        code[i] = 0;
        cls[i] = kCellOff;
        if (j < kTH * kTH && gx >= 0 && gx < W && gy >= 0 && gy < H) {
            const size_t g = (size_t)gy * W + gx;
            code[i] = fd[g];
            cls[i] = class_of(g, gx, gy);
        }
    }
#pragma unroll
    for (int i = 0; i < kTurns; ++i) {
        const int j = threadIdx.x + 256 * i, hy = j / kTH, hx = j - hy * kTH;
        if (j >= kTH * kTH) continue;
        s_code[j] = code[i];
        s_cls[j] = cls[i];
        if (cls[i] == kCellOff) continue;
        for (uint32_t m = code[i]; m; m &= m - 1) {
            const int b = __ffs(m) - 1, d = (b + 2) & 7;  // bit b of a code is direction (b + 2) % 8
            const int rx = hx - 1 + dir_dx(d), ry = hy - 1 + dir_dy(d);
            if (!in_tile(rx, ry)) continue;
            const int r = ry * kTile + rx;
            if (cls[i] == kCellBlock) {
                atomicOr(&s_bad[ry], 1u << rx);
            } else {
                const int k = scan_index((d + 4) & 7) + (in_tile(hx - 1, hy - 1) ? 0 : 8);
                atomicOr(reinterpret_cast<uint32_t*>(s_dm) + (r >> 1), 1u << (k + 16 * (r & 1)));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// The in-tile dependency order of one block (256 threads, thread (lx, ly0)
// holds the cells of column lx in rows ly0 + 8 q).
//
// s_pd of a cell: the cell its path reaches after 2^k steps, or where the path
// ends before that (low 10 bits), and the steps to it (above).  Doubling k
// takes every cell to its path's end, and on the way each cell hands the cell
// exactly 2^k steps down what lies above it: the length of the longest path
// that ends there (s_h, its level: every donor has a smaller one) and two flags
// (bit sets of 32 words, a row each).  A path that has not ended after 2^10
// steps runs into a cycle; its cells after as many steps, all of the cycle,
// join s_bad.  log2 of the longest path rounds, all threads at work, in the place
// of a queue of released cells whose order costs an atomic and a vote per cell.
constexpr int kPtr = kTile * kTile - 1;  // the pointer bits of s_pd
__device__ __forceinline__ void tile_paths(int32_t* s_pd, int32_t* s_h, uint32_t* s_wait, uint32_t* s_bad, int lx,
                                           int ly0) {
    for (int k = 0;; ++k) {
        int32_t next[4];
        int up[4];
        uint32_t flags = 0;
        bool any = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int l = (ly0 + 8 * q) * kTile + lx;
            const int32_t v = s_pd[l];
            up[q] = -1;
            next[q] = 0;
            if ((v >> 10) == 1 << k) {
                const int32_t v2 = s_pd[v & kPtr];
                next[q] = (v2 & kPtr) | (((v >> 10) + (v2 >> 10)) << 10);
                up[q] = (v & kPtr) | ((s_h[l] + (1 << k)) << 10);
                flags |= ((s_wait[l >> 5] >> lx) & 1u) << q | ((s_bad[l >> 5] >> lx) & 1u) << (q + 4);
                any = true;
            }
        }
        if (!__syncthreads_or(any)) break;
        if (k == 10) {  // into a cycle
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (up[q] >= 0) atomicOr(&s_bad[(up[q] & kPtr) >> 5], 1u << (up[q] & 31));
            break;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (up[q] < 0) continue;
            const int p = up[q] & kPtr;
            s_pd[(ly0 + 8 * q) * kTile + lx] = next[q];
            atomicMax(&s_h[p], up[q] >> 10);
            if ((flags >> q) & 1u) atomicOr(&s_wait[p >> 5], 1u << (p & 31));
            if ((flags >> (q + 4)) & 1u) atomicOr(&s_bad[p >> 5], 1u << (p & 31));
        }
        __syncthreads();
    }
    __syncthreads();
}

// Sorts the cells with key[q] >= 0 (below 2 * words) by key and counts them in
// *s_total (0 before): s_ent holds pack(q) of each.  s_bins (`words` words, 0
// before) then holds where each key's cells end, 16 bits a key, up to the last key
// used; the words 32 and more behind that one's stay 0.  Every thread calls it.
__device__ __forceinline__ int bin_end(const uint32_t* s_bins, int key) {
    return (s_bins[key >> 1] >> (16 * (key & 1))) & 0xffff;
}
template <class Pack>
__device__ __forceinline__ void tile_sort(const int (&key)[4], const Pack& pack, uint32_t* s_bins, int words,
                                          uint32_t* s_ent, int* s_total, int lx) {
    int mine = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (key[q] >= 0) atomicAdd(&s_bins[key[q] >> 1], 1u << (16 * (key[q] & 1)));
        mine += __popc(__ballot_sync(0xffffffffu, key[q] >= 0));
    }
    if (lx == 0 && mine) atomicAdd(s_total, mine);
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t total = (uint32_t)*s_total;
        uint32_t carry = 0;
        for (int b = lx; b < words && carry < total; b += 32) {
            const uint32_t v = s_bins[b], lo = v & 0xffff, n = lo + (v >> 16);
            uint32_t incl = n;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
                if (lx >= d) incl += u;
            }
            const uint32_t at = carry + incl - n;
            s_bins[b] = at | ((at + lo) << 16);
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q)
        if (key[q] >= 0) {
            const int sh = 16 * (key[q] & 1);
            const int at = (atomicAdd(&s_bins[key[q] >> 1], 1u << sh) >> sh) & 0xffff;
            s_ent[at] = pack(q);
        }
    __syncthreads();
}

// A cell of the sorted list with its first two in-tile donors: the cell in 11
// bits (kNoCell: a cell that the caller lays out behind the tile's, of no effect),
// the first donor as a step (7 bits), the second in 11 bits (kNoCell: none), and
// whether there are more.
constexpr int kNoCell = kTile * kTile;
constexpr uint32_t kNoEntry = kNoCell | (64u << 11) | ((uint32_t)kNoCell << 18);
constexpr uint32_t kMoreDonors = 1u << 29;
// index step of direction scan_dir(k): +1, +33, +32, +31, then their negatives
__device__ __forceinline__ int scan_step(int k) {
    const int v = (0x1F202101 >> (8 * (k & 3))) & 0xff;
    return k & 4 ? -v : v;
}
__device__ __forceinline__ uint32_t entry_of(int c, uint32_t donors) {  // donors: bit k for direction scan_dir(k)
    const uint32_t m = donors & (donors - 1);
    const int o0 = donors ? scan_step(__ffs(donors) - 1) : 0;
    const int d1 = m ? c + scan_step(__ffs(m) - 1) : kNoCell;
    return (uint32_t)c | (uint32_t)(o0 + 64) << 11 | (uint32_t)d1 << 18 | (m & (m - 1) ? kMoreDonors : 0u);
}
__device__ __forceinline__ int entry_cell(uint32_t e) { return e & 2047; }
__device__ __forceinline__ int entry_d0(uint32_t e) { return (int)(e & 2047) + (int)((e >> 11) & 127) - 64; }
__device__ __forceinline__ int entry_d1(uint32_t e) { return (e >> 18) & 2047; }

// Runs op(fetch(entry)) on the sorted entries of the keys from `first` on, key by
// key: a key's cells depend on smaller keys only.  A key has no more cells than
// the one before (each cell of a level has a donor of its own in the level
// above): the first keys, of more than 32 cells, run on every thread with a block
// barrier each, the others on warp 0 alone until one is empty.  There the chain of
// keys sets the time, and a warp issues in order, so nothing but op stands in it:
// entries are read two keys ahead and what fetch reads (nothing that op writes for
// another cell) one key ahead; finding the donors from direction bits in the chain
// took a third of it.
template <class Fetch, class Op>
__device__ __forceinline__ void tile_levels(const Fetch& fetch, const Op& op, int first, int keys,
                                            const uint32_t* s_bins, const uint32_t* s_ent) {
    int key = first, start = first ? bin_end(s_bins, first - 1) : 0;
    for (; key < keys; ++key) {
        const int end = bin_end(s_bins, key);
        if (end - start <= 32) break;  // block-uniform
        for (int i = start + threadIdx.x; i - (int)(threadIdx.x & 31) < end; i += blockDim.x)  // whole warps
            op(fetch(i < end ? s_ent[i] : kNoEntry));
        __syncthreads();
        start = end;
    }
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        auto end_of = [&](int k) { return k < keys ? bin_end(s_bins, k) : 0; };
        auto entry_at = [&](int from, int to) { return lane < to - from ? s_ent[from + lane] : kNoEntry; };
        int end = end_of(key), next = end_of(key + 1), after = end_of(key + 2);
        auto got = fetch(entry_at(start, end));
        uint32_t en = entry_at(end, next);
        while (end > start) {
            const uint32_t ea = entry_at(next, after);
            const auto gotn = fetch(en);
            start = end;
            end = next;
            next = after;
            after = end_of(++key + 2);
            op(got);
            __syncwarp();
            got = gotn;
            en = ea;
        }
    }
    __syncthreads();
}

// position of a halo cell of the ring in ring_halo's order
__device__ __forceinline__ int ring_index(int hx, int hy) {
    if (hy == 0) return hx;
    if (hy == kTH - 1) return kTH + hx;
    return 2 * kTH + (hx == 0 ? 0 : kTile) + hy - 1;
}

}  // namespace lem
