// lem_fa.cu -- flow-accumulation stage.
//
// computeRunOffWeights (MOD_kernels/runoffweight.cu:21-113), calcpropsSFD /
// calcprops (:115-354) and correctmfdflow (FA_kernels/mfd_simple.cu:33-384).
// The reference rescans the whole grid once per dependency level with a host
// round trip per launch; here every cell is computed once, after its donors.  Steps
// of one flow direction go by 32x32 tiles (k_fat_*), the others by the general wave
// (k_fa_walk), in which warps share one list of ready cells.  The sum of the donors
// is pulled in the reference's order E, SE, S, SW, W, NW, N, NE
// (mfd_simple.cu:95-165) as an fp32 pair (hi + lo) to keep ~44 bits.

#include <cooperative_groups.h>

#include <cstring>
#include <mutex>

#include "lem_wave.cuh"

namespace cg = cooperative_groups;

namespace lem {

namespace {

// k_fat_local's cell status: a donor in another tile, finished inside the tile,
// and waiting on an inflow from another tile somewhere upstream (its final value
// needs the coarse wave)
constexpr uint8_t kLaKind = 3, kLaEntry = 4, kLaDone = 8, kLaWaits = 16;  // (below them the cell's kind)
constexpr int32_t kRun = 1 << 30;  // k_fat_local: a waiting cell between nodes
constexpr int32_t kLaOutlet = -1;  // final-pass entry in the place of the node: an outlet (the coarse wave's; counted only)

// Sum over a block of 256 threads (every thread calls it; the result is valid in thread 0).
__device__ __forceinline__ int block_sum_i(int v) {
    __shared__ int part[8];
    v = wsum(v);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    int t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < 8; ++w) t += part[w];
    return t;
}

// calcrunoffweight (runoffweight.cu:21-58): runoff weights and soil moisture, and the
// accumulation's initial values.  A negative weight or a code with several directions
// sends the step off the tiled path.
__global__ void k_fa_prep(const uint8_t* __restrict__ mask, const uint8_t* __restrict__ fd,
                          const float* __restrict__ stone, const float* __restrict__ totB, float* __restrict__ soilM,
                          float* __restrict__ w, float2* __restrict__ fa, const int32_t* __restrict__ chunk_start,
                          ModelConsts k, DemCtx dc, DevScalars* sc) {
    const int W = k.W;
    const Chunk ch = chunk_of(chunk_start, dc);
    const DemIn& r = dc.in[ch.d];
    const float rain0 = (float)r.rain, rinc = (float)r.rain_inc;
    int nact = 0;
    bool untiled = false;
    // two cells per thread and iteration: both cells' inputs are loaded before
    // either is used, so each thread keeps two cells' loads in flight
    for (int64_t r0 = ch.first + threadIdx.x; r0 < ch.end; r0 += 2 * blockDim.x) {
        size_t i[2];
        int y[2];
        uint8_t mk[2] = {0, 0}, code[2] = {0, 0};
        float sto[2], tb[2], sm0[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int64_t ri = r0 + u * blockDim.x;
            int x;
            i[u] = ri < ch.end ? region_cell(r, ri, W, &x, &y[u]) : 0;
            if (ri < ch.end) {
                mk[u] = mask[i[u]];
                code[u] = fd[i[u]];
                sto[u] = stone[i[u]];
                tb[u] = totB[i[u]];
                sm0[u] = soilM[i[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (r0 + u * blockDim.x >= ch.end) continue;
            if (mk[u]) {
                ++nact;
                const float coeff =
                    (1.0f - 0.0085f * sto[u]) * expf(-0.0025f * tb[u] / 76.5f) * tanhf(0.6f + sm0[u] / 0.2f);
                const float myppt = (rain0 + (float)(y[u] - r.y0) * rinc) / 1000.0f;
                const float wi = myppt * coeff;
                float sm = sm0[u] + myppt * (1.0f - coeff);
                if (sm > 0.5f) sm = 0.5f;
                soilM[i[u]] = sm;
                w[i[u]] = wi;
                fa[i[u]] = make_float2(wi, 0.0f);
                untiled |= wi < 0.0f || (code[u] & (code[u] - 1));
            } else {
                w[i[u]] = -9999.0f;
                fa[i[u]] = make_float2(0.0f, 0.0f);
            }
        }
    }
    if (__syncthreads_or(untiled) && threadIdx.x == 0) sc->tiled_ok = 0;
    const int tot = __syncthreads_count(nact > 0) ? block_sum_i(nact) : 0;  // one atomic per block
    if (threadIdx.x == 0 && tot) atomicAdd(&dc.out[ch.d].n_active, tot);
}

// Words and sources of the general accumulation wave, for the steps that
// take it (MFD, or a step k_fa_prep sent off the tiled path).  A donor outside the
// catchment is complete from the start when its DEM is nodata (correctmfdflow's
// okgrid, mfd_simple.cu:279-285) and never otherwise.
__global__ void k_fa_pend(const double* __restrict__ z, const uint8_t* __restrict__ mask,
                          const uint8_t* __restrict__ fd, int32_t* __restrict__ word, int32_t* __restrict__ contrib,
                          int32_t* ready, const int32_t* __restrict__ chunk_start, ModelConsts k, DemCtx dc,
                          DevScalars* sc, int gate) {
    if (gate && sc->tiled_ok) return;  // the tiled path accumulates this step
    const int W = k.W, H = k.H;
    const size_t N = (size_t)W * H;
    const Chunk ch = chunk_of(chunk_start, dc);
    const DemIn& r = dc.in[ch.d];
    for (int64_t base = ch.first; base < ch.end; base += blockDim.x) {
        const int64_t ri = base + threadIdx.x;
        bool src = false;
        size_t i = 0;
        if (ri < ch.end) {
            int x, y;
            i = region_cell(r, ri, W, &x, &y);
            if (mask[i]) {
                if (contrib) contrib[i] = 1;
                int32_t pend = 0;
                uint32_t donors = 0, receivers = 0;
                const uint8_t code = fd[i];
#pragma unroll
                for (int d = 0; d < 8; ++d) {
                    const int nx = x + dir_dx(d), ny = y + dir_dy(d);
                    if (nx < 0 || nx >= W || ny < 0 || ny >= H) continue;
                    const size_t n = (size_t)ny * W + nx;
                    const bool in = mask[n];
                    if (in) receivers |= code & dir_bit(d);
                    if (!donates(fd[n], d)) continue;
                    if (in) {
                        ++pend;
                        donors |= 1u << scan_index(d);
                    } else if (z[n] != kNoData) {
                        pend |= kBlocked;
                    }
                }
                word[i] = wave_word(pend, donors, receivers);
                src = (pend == 0);
            } else {
                if (contrib) contrib[i] = 0;
                word[i] = kBlocked;
            }
        }
        wave_append(src, (int32_t)i, ready, &sc->counters[0], (int)N, &sc->err);
    }
}

// calcprops (runoffweight.cu:141-354): slope-proportional partition, forcing a
// single-direction code back to one direction (and rewriting its slopes).
__global__ void k_calcprops(const uint8_t* __restrict__ mask, const uint8_t* __restrict__ fd, float* slopes,
                            float* prop, size_t N) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        if (!mask[i]) continue;
        float s[8];
        float tot = 0.f;
        for (int j = 0; j < 8; ++j) {
            s[j] = slopes[8 * i + j];
            tot += s[j];
        }
        int cnt = 0;
        float p[8];
        for (int j = 0; j < 8; ++j) {
            p[j] = s[j] / tot;
            if (p[j] > 0) ++cnt;
        }
        const int d = bit_dir(fd[i]);
        if (d >= 0 && cnt > 1) {
            for (int j = 0; j < 8; ++j) {
                slopes[8 * i + j] = (j == d) ? 0.0001f : 0.0f;
                p[j] = (j == d) ? 1.0f : 0.0f;
            }
        }
        for (int j = 0; j < 8; ++j) prop[8 * i + j] = p[j];
    }
}

// One cell of correctmfdflow's CalcMFD (mfd_simple.cu:31-171): the weight plus
// the donors' accumulation in the order E, SE, S, SW, W, NW, N, NE, a negative
// donor sum clamped to zero.  A donor outside the catchment adds nothing, and
// the accumulation of a cell starts at its weight.
struct FaCell {
    const float* prop;
    float2* fa;
    int32_t* contrib;
    DemCtx dc;
    int W;
    struct Part {
        float2 v;  // the donor's accumulation, its share taken
        int32_t cnt;
    };
    __device__ __forceinline__ Part donor(int32_t cur, int kk, bool on) const {
        Part part{make_float2(0.f, 0.f), 0};
        const int d = scan_dir(kk);
        const int32_t n = cur + grid_step(d, W);
        if (on) {
            const float p = prop ? __ldg(prop + 8 * (size_t)n + ((d + 4) & 7)) : 1.0f;
            const float2 v = __ldcg(fa + n);
            part.v = p == 1.0f ? v : ff_scale(v, p);
            if (contrib) part.cnt = __ldcg(contrib + n);
        }
        return part;
    }
    __device__ __forceinline__ void cell(int32_t cur, uint32_t donors, Part part) const {
        const float2 w = __ldcg(fa + cur);
        float2 acc = make_float2(0.f, 0.f);
        for (uint32_t m = donors; m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            acc = ff_add(acc, make_float2(__shfl_sync(0xffffffffu, part.v.x, k), __shfl_sync(0xffffffffu, part.v.y, k)));
        }
        if (acc.x < 0.0f) acc = make_float2(0.f, 0.f);
        const int cnt = contrib ? wsum(part.cnt) : 0;
        if ((threadIdx.x & 31) == 0) {
            __stcg(fa + cur, ff_add(w, acc));
            if (contrib) __stcg(contrib + cur, 1 + cnt);
            if (dc.of) atomicAdd(&dc.out[dc.of[cur]].fa_done, 1);  // a batch: count per DEM
        }
    }
};

// The general accumulation wave.  With gate set it runs only when the tiled
// path is off.
__global__ void __launch_bounds__(256, 4)
    k_fa_walk(const float* __restrict__ prop, float2* fa, int32_t* word, int32_t* contrib, int32_t* list,
              ModelConsts k, DevScalars* sc, DemCtx dc, int gate) {
    if (gate && sc->tiled_ok) return;  // the tiled kernels did this step
    const FaCell op{prop, fa, contrib, dc, k.W};
    int done = wave_walk(op, word, list, k.W, k.H, sc);
    done = wsum(done);
    if (!dc.of && (threadIdx.x & 31) == 0 && done) atomicAdd(&dc.out[0].fa_done, done);
}

// ---------------------------------------------------------------------------
// Tiled accumulation for single-receiver codes (SFD).  A chain walk through
// global memory pays an L2 round trip per cell on the longest flow path; here
// the grid is cut into 32x32 tiles and most of the path runs in shared memory.
//   local : per tile, the accumulation from inside the tile (la), the outlet
//           each entry cell drains to, and per outlet its entries and the
//           number of inflows from other tiles it waits for;
//   coarse: a wave over the outlets only: F(o) = la(o) + the final values of
//           the outlets of neighbouring tiles that flow into o's entries;
//   final : per tile, every other cell by the reference formula, with the
//           donors in other tiles taken at their final values.
// All sums are pulled in a fixed order, so results do not depend on timing.
// The decomposition is exact while no donor sum can be negative (CalcMFD
// clamps those to zero); k_fa_prep disables the path for a step with a
// negative weight or a multi-direction code, and the walk then runs instead.


__global__ void __launch_bounds__(256, 6)
    k_fat_local(const double* __restrict__ z, const uint8_t* __restrict__ mask, const uint8_t* __restrict__ fd,
                const float* __restrict__ w, int4* __restrict__ t_rec, int32_t* __restrict__ t_dst,
                int32_t* __restrict__ t_pend, int32_t* __restrict__ t_ent, float2* __restrict__ fa,
                int32_t* __restrict__ n_meta, int32_t* __restrict__ n_ref, int2* __restrict__ f_idx,
                float2* __restrict__ f_la, int32_t* __restrict__ t_fcnt, int32_t* outs, ModelConsts k,
                DevScalars* sc, DemCtx dc, TileSet ts, int count) {
    if (!sc->tiled_ok) return;
    __shared__ uint8_t s_code[kTH * kTH];
    __shared__ uint8_t s_cls[kTH * kTH];
    __shared__ int32_t s_pd[kTile * kTile];  // the in-tile path (tile_paths): where it ends
    __shared__ int32_t s_h[kTile * kTile + 1];  // levels
    __shared__ float2 s_la[kTile * kTile + 1];
    __shared__ uint8_t s_info[kTile * kTile];  // kind, and kLa flags
    // donors, bit k for direction scan_dir(k): in the low byte those in the tile,
    // in the high byte those in other tiles, then with the waiting ones in the tile
    __shared__ __align__(4) uint16_t s_dm[kTile * kTile + 1];
    __shared__ uint32_t s_ent[kTile * kTile];  // the finished cells by level
    __shared__ uint32_t s_bins[kTile * kTile / 2];
    __shared__ uint32_t s_wait[kTile], s_bad[kTile];
    __shared__ int16_t s_olist[kTileEnt];
    __shared__ int32_t s_ocnt[kTileEnt];
    __shared__ int32_t s_ofill[kTileEnt];
    __shared__ int s_no, s_nn, s_fn, s_pool, s_qn;
    __shared__ int s_wcnt[9];  // per-warp counts of the outlet list and its append
    const int W = k.W, H = k.H, TW = (W + kTile - 1) / kTile;
    const int t = ts.tile(blockIdx.x);
    const int tx0 = (t % TW) * kTile, ty0 = (t / TW) * kTile;
    const int lx = threadIdx.x & 31, ly0 = threadIdx.x >> 5;
    float wq[4];  // the cells' weights, loaded alongside the halo
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int gx = tx0 + lx, gy = ty0 + ly0 + 8 * q;
        wq[q] = !w ? 1.0f : (gx < W && gy < H) ? w[(size_t)gy * W + gx] : 0.f;
    }
    if (threadIdx.x == 0) s_fn = s_pool = s_qn = 0;
    for (int i = threadIdx.x; i < kTile * kTile / 2; i += blockDim.x) {
        s_bins[i] = 0;
        reinterpret_cast<uint32_t*>(s_dm)[i] = 0;
    }
    if (threadIdx.x < kTile) s_bad[threadIdx.x] = 0;
    __syncthreads();
    tile_stage(
        fd,
        [&](size_t g, int, int) {
            return mask[g] ? kCellIn : (z[g] == kNoData ? kCellOff : kCellBlock);
        },
        W, H, tx0, ty0, s_code, s_cls, s_dm, s_bad);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx, hc = (ly + 1) * kTH + lx + 1;
        uint32_t dm = 0, kind = kKindEnd;
        int32_t pd = l;
        if (s_cls[hc] == kCellIn) {
            dm = s_dm[l];
            const int d = bit_dir(s_code[hc]);
            const int rlx = lx + dir_dx(d < 0 ? 0 : d), rly = ly + dir_dy(d < 0 ? 0 : d);
            if (d >= 0 && s_cls[(rly + 1) * kTH + rlx + 1] == kCellIn) {
                kind = in_tile(rlx, rly) ? kKindIn : kKindOutlet;
                if (kind == kKindIn) pd = (rly * kTile + rlx) | (1 << 10);
            }
        }
        const float2 wl = make_float2(s_cls[hc] == kCellIn ? wq[q] : 0.f, 0.f);
        const bool entry = dm >> 8;
        s_la[l] = dm & 255u ? wl : ff_add(wl, make_float2(0.f, 0.f));  // level 0: final
        s_pd[l] = pd;
        s_h[l] = 0;
        s_info[l] = (uint8_t)(kind | (entry ? kLaEntry : 0));
        s_dm[l] = (uint16_t)dm;
        const unsigned wb = __ballot_sync(0xffffffffu, entry);
        if (lx == 0) s_wait[ly] = wb;
    }
    __syncthreads();
    tile_paths(s_pd, s_h, s_wait, s_bad, lx, ly0);
    // a cell is finished here unless a donor upstream never completes; it waits
    // when an entry (a cell with a donor in another tile) lies upstream
    int level[4];
    bool stray = false;  // a waiting cell whose in-tile path ends inside the tile
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        uint32_t info = s_info[l];
        const bool done = s_cls[(ly + 1) * kTH + lx + 1] == kCellIn && !((s_bad[ly] >> lx) & 1u);
        const bool waits = done && ((s_wait[ly] >> lx) & 1u);
        level[q] = done ? s_h[l] : -1;
        info |= (done ? kLaDone : 0) | (waits ? kLaWaits : 0);
        s_info[l] = (uint8_t)info;
    }
    tile_sort(
        level,
        [&](int q) {
            const int l = (ly0 + 8 * q) * kTile + lx;
            return entry_of(l, s_dm[l] & 255u);
        },
        s_bins, kTile * kTile / 2, s_ent, &s_qn, lx);  // (its barriers also cover s_info)
    // What a waiting cell needs of the cells above it: s_nd holds 1 for a node
    // (an entry, a join of waiting branches, the outlet), else kRun and the cell
    // at the top of its run of single-input cells in the high half, found in
    // level order from its waiting donor.
    int32_t* const s_nd = s_h;  // the levels are spent
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        const uint32_t info = s_info[l];
        int32_t nd = 0;
        if (info & kLaWaits) {
            const uint32_t dm = s_dm[l];
            uint32_t wm = 0;
            for (uint32_t m = dm & 255u; m; m &= m - 1)
                if (s_info[l + scan_step(__ffs(m) - 1)] & kLaWaits) wm |= m & (0u - m);
            nd = (dm >> 8) || (wm & (wm - 1)) || (info & kLaKind) == kKindOutlet
                     ? 1
                     : kRun | ((l + scan_step(__ffs(wm) - 1)) << 16);
            s_dm[l] = (uint16_t)(dm | (wm << 8));
        }
        s_nd[l] = nd;
        const int e = s_pd[l] & kPtr;
        const bool out = (s_info[e] & kLaKind) == kKindOutlet;
        if (info & kLaEntry)
            t_dst[(size_t)(ty0 + ly) * W + tx0 + lx] =
                out ? (int32_t)((ty0 + e / kTile) * W + tx0 + (e & (kTile - 1))) : -1;
        stray |= (info & kLaWaits) && !out;
    }
    __syncthreads();
    if (threadIdx.x == 0) {  // kNoCell: a cell of nothing, its own donor
        s_la[kNoCell] = make_float2(0.f, 0.f);
        s_nd[kNoCell] = 0;
        s_dm[kNoCell] = 0;
    }
    __syncthreads();
    // accumulation from inside the tile, level by level; adding the zero of
    // kNoCell changes no pair
    struct Cell {
        float2 w;
        uint32_t e;
        int32_t nd;
    };
    tile_levels(
        [&](uint32_t e) { return Cell{s_la[entry_cell(e)], e, s_nd[entry_cell(e)]}; },
        [&](const Cell& f) {
            const int c = entry_cell(f.e);
            float2 acc = ff_add(s_la[entry_d0(f.e)], s_la[entry_d1(f.e)]);
            const int32_t top = s_nd[f.nd & kRun ? (f.nd >> 16) & kPtr : kNoCell];
            if (__any_sync(0xffffffffu, f.e & kMoreDonors) && (f.e & kMoreDonors)) {
                uint32_t m = s_dm[c] & 255u;
                m &= m - 1;
                for (m &= m - 1; m; m &= m - 1) acc = ff_add(acc, s_la[c + scan_step(__ffs(m) - 1)]);
            }
            const bool neg = acc.x < 0.0f;
            s_la[c] = ff_add(f.w, make_float2(neg ? 0.f : acc.x, neg ? 0.f : acc.y));
            s_nd[c] = top & kRun ? top : f.nd;
        },
        1, kTile * kTile, s_bins, s_ent);
    int16_t* const s_oslot = reinterpret_cast<int16_t*>(s_bins);  // the bins are spent
    const int qn = s_qn;                                          // finished cells
    // Such a tile keeps the second wave; every other tile writes its settled
    // cells here and leaves the final pass a program of nodes (see below).
    const bool second_wave = __syncthreads_or(stray);
    // outlets in cell order (they lie on the border: at most 124)
    list_outlets(s_info, kLaKind, s_olist, s_oslot, &s_no, s_wcnt);
    if (threadIdx.x < kTileEnt) s_ocnt[threadIdx.x] = 0;
    __syncthreads();
    // inflows: ring cells of the halo that flow into the tile, grouped by the
    // outlet their entry drains to, in ring order
    int key[kRingChunks];
    int32_t donor[kRingChunks];
#pragma unroll
    for (int c = 0; c < kRingChunks; ++c) {
        const int i = c * 32 + lx;
        key[c] = -1;
        donor[c] = 0;
        if (threadIdx.x < 32 && i < kRing) {
            const int h = ring_halo(i);
            const int d = s_cls[h] == kCellIn ? bit_dir(s_code[h]) : -1;
            if (d >= 0) {
                const int hx = h % kTH + dir_dx(d), hy = h / kTH + dir_dy(d);
                if (hx >= 1 && hx <= kTile && hy >= 1 && hy <= kTile && s_cls[hy * kTH + hx] == kCellIn) {
                    const int e = (hy - 1) * kTile + hx - 1;
                    const int o = s_pd[e] & kPtr;
                    if ((s_info[o] & kLaKind) == kKindOutlet) {
                        key[c] = s_oslot[o];
                        donor[c] = (ty0 - 1 + h / kTH) * W + tx0 - 1 + h % kTH;
                        atomicAdd(&s_ocnt[key[c]], 1);
                    }
                }
            }
        }
    }
    __syncthreads();
    const int no = s_no;
    if (threadIdx.x < 32) outlet_starts(s_ocnt, s_ofill, no);
    __syncthreads();
    const int j = threadIdx.x;
    const int ostart = j < no ? s_ofill[j] : 0;
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned below = (1u << lx) - 1u;
#pragma unroll
        for (int c = 0; c < kRingChunks; ++c) {
            const unsigned peers = __match_any_sync(0xffffffffu, key[c]);
            const int base = key[c] >= 0 ? s_ofill[key[c]] : 0;
            __syncwarp();
            if (key[c] >= 0) {
                t_ent[(size_t)t * kTileEnt + base + __popc(peers & below)] = donor[c];
                if ((peers & below) == 0) s_ofill[key[c]] = base + __popc(peers);
            }
            __syncwarp();
        }
    }
    int32_t og = 0;
    if (j < no) {
        const int o = s_olist[j];
        const int32_t opend = ((s_info[o] & kLaDone) ? 0 : kBlocked) + s_ocnt[j];
        og = (ty0 + o / kTile) * W + tx0 + (o & (kTile - 1));
        const float2 la = s_la[o];
        t_rec[og] = make_int4(__float_as_int(la.x), __float_as_int(la.y), (ostart << 16) | s_ocnt[j], -1);
        t_pend[og] = opend;
        if (opend == 0) {  // a source of the coarse wave: final already, and marked in the list
            fa[og] = la;
            og = ~og;
        }
    }
    block_append(j < no, og, outs, &sc->tile_src, W * H, &sc->err, s_wcnt);
    if (threadIdx.x == 0) t_fcnt[t] = -1;
    if (second_wave) return;  // block-uniform

    // The final pass's program.  A waiting cell's accumulation is its local
    // one plus the inflows of every entry upstream of it.  That sum is the same
    // along a run of single-input cells, so it is kept per node: the inflows the
    // node takes from other tiles plus the sums of the nodes at the top of its
    // waiting inputs.  s_nd: from here on a node's index + 1.
    int done = 0, dem = -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx, hc = (ly + 1) * kTH + lx + 1;
        const size_t g = (size_t)(ty0 + ly) * W + tx0 + lx;
        if (dem < 0 && s_cls[hc] == kCellIn) dem = dem_at(dc, g);
        if ((s_info[l] & (kLaDone | kLaWaits)) == kLaDone && (s_info[l] & kLaKind) != kKindOutlet) {
            fa[g] = s_la[l];  // (the coarse wave stores the outlets)
            ++done;
        }
    }
    done = wsum(done);
    dem = __reduce_max_sync(0xffffffffu, dem);  // one DEM per tile
    if (count && (threadIdx.x & 31) == 0 && done && dem >= 0) atomicAdd(&dc.out[dem].fa_done, done);
    // node indices in level order (inputs first): warp w numbers the nodes among entries 128 w .. 128 w + 127 of the sorted list
    {
        const int wq = threadIdx.x >> 5;
        const unsigned below = (1u << lx) - 1u;
        unsigned b[4];
        int cnt = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = wq * 128 + r * 32 + lx;
            bool isn = false;
            if (i < qn) {
                isn = (s_nd[entry_cell(s_ent[i])] & 0xffff) != 0;
            }
            b[r] = __ballot_sync(0xffffffffu, isn);
            cnt += __popc(b[r]);
        }
        if (lx == 0) s_wcnt[wq] = cnt;
        __syncthreads();
        int base = 0;
        for (int i = 0; i < wq; ++i) base += s_wcnt[i];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if ((b[r] >> lx) & 1u) s_nd[entry_cell(s_ent[wq * 128 + r * 32 + lx])] = base + __popc(b[r] & below) + 1;
            base += __popc(b[r]);
        }
        if (threadIdx.x == 255) s_nn = base;  // the last warp's end is the total
    }
    __syncthreads();
    const size_t tb = (size_t)t * kTile * kTile, pool = (size_t)t * kTilePool;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        const size_t g = (size_t)(ty0 + ly) * W + tx0 + lx;
        const int32_t v = s_nd[l];
        const bool waits = (s_info[l] & kLaWaits) != 0, outlet = (s_info[l] & kLaKind) == kKindOutlet;
        const int e = warp_slot(waits || outlet, &s_fn);
        if (outlet) {  // counted once the coarse wave stored it
            f_idx[tb + e] = make_int2((int)g, kLaOutlet);
        } else if (waits) {
            const int node = (v & 0xffff) ? (v & 0xffff) - 1 : (s_nd[(v >> 16) & kPtr] & 0xffff) - 1;
            f_idx[tb + e] = make_int2((int)g, node);
            f_la[tb + e] = s_la[l];
        }
        if (!waits || !(v & 0xffff)) continue;
        // the node's inputs, in the donors' scan order: cells of other tiles and
        // node indices (negated)
        const uint32_t dm = s_dm[l];
        const int nin = __popc(dm >> 8);
        const int start = atomicAdd(&s_pool, nin);
        if (start + nin > kTilePool) {
            raise_error(&sc->err, ErrFlags::kCapacity);
            continue;
        }
        int m = 0;
#pragma unroll 1
        for (uint32_t b = dm >> 8; b; b &= b - 1) {
            const int kk = __ffs(b) - 1;
            int32_t ref;
            if ((dm >> kk) & 1u) {
                const int32_t vu = s_nd[l + scan_step(kk)];
                ref = -((vu & 0xffff) ? (vu & 0xffff) : (s_nd[(vu >> 16) & kPtr] & 0xffff));
            } else {
                const int d = scan_dir(kk);
                ref = (ty0 + ly + dir_dy(d)) * W + tx0 + lx + dir_dx(d);
            }
            n_ref[pool + start + m] = ref;
            ++m;
        }
        n_meta[tb + (v & 0xffff) - 1] = start | (m << 11);
    }
    __syncthreads();
    if (threadIdx.x == 0) t_fcnt[t] = (s_nn << 16) | s_fn;
}

// The coarse wave: F(o) = la(o) + the final values of o's inflows, outlet by
// outlet downstream.  The sources (final since k_fat_local) release their
// receivers in one parallel pass, which also links every outlet to the outlet
// it drains to.  After it each warp takes a released outlet and walks
// downstream for as long as its outlet is the last inflow to arrive: an outlet
// has one receiver, so every outlet is reached once and no second list is
// needed.
//
// Bound by the longest chain of tile crossings (about 240 at 4096 x 4096
// cells, on average with 20 inflows each), so by the latency of one crossing:
// the last inflow's release, the other inflows' values, the sum in order.  A
// warp loads the inflows' values at once (a lane per outlet took them eight at
// a time, 1.07 ms), and the static data is read ahead: the inflow list of the
// next outlet and the record of the one after it.
__global__ void __launch_bounds__(256)
    k_fat_coarse(const uint8_t* __restrict__ fd, int4* __restrict__ t_rec, const int32_t* __restrict__ t_ent,
                 const int32_t* __restrict__ t_dst, float2* fa, int32_t* t_pend, const int32_t* __restrict__ outs,
                 int32_t* ready, ModelConsts k, DevScalars* sc) {
    if (!sc->tiled_ok) return;
    cg::grid_group grid = cg::this_grid();
    __shared__ int s_cnt[9];
    const int W = k.W, TW = (W + kTile - 1) / kTile;
    const size_t N = (size_t)W * k.H;
    const int n = sc->tile_src;
    int32_t* const n_ready = &sc->counters[0];
    int32_t* const head = &sc->counters[1];
    if (blockIdx.x == 0 && threadIdx.x == 0) *n_ready = *head = 0;
    grid.sync();
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < (size_t)n; base += (size_t)gridDim.x * blockDim.x) {
        const size_t i = base + threadIdx.x;
        int32_t nx = -1;
        bool rdy = false;
        if (i < (size_t)n) {
            const int32_t e = outs[i], o = e < 0 ? ~e : e;
            const int d = bit_dir(fd[o]);  // the receiver lies in another tile, in the catchment
            nx = t_dst[o + dir_dy(d) * W + dir_dx(d)];
            reinterpret_cast<int32_t*>(t_rec + o)[3] = nx;
            if (e < 0 && nx >= 0) rdy = atomicSub(t_pend + nx, 1) == 1;
        }
        block_append(rdy, nx, ready, n_ready, (int)N, &sc->err, s_cnt);
    }
    grid.sync();
    const int nin = *((volatile int32_t*)n_ready);
    const int lane = threadIdx.x & 31;
    auto inflows = [&](int32_t o, int rng) {
        return t_ent + (size_t)((o / W / kTile) * TW + (o % W) / kTile) * kTileEnt + (rng >> 16);
    };
    for (size_t guard = 0; guard <= N; ++guard) {
        int32_t o = -1;
        if (lane == 0) {
            const int it = atomicAdd(head, 1);
            if (it < nin) o = __ldcg(ready + it);
        }
        o = __shfl_sync(0xffffffffu, o, 0);
        if (o < 0) break;
        int4 r = __ldcg(t_rec + o), rn = make_int4(0, 0, 0, -1);  // the records of o and of the next outlet
        int32_t in = lane < (r.z & 0xffff) ? __ldg(inflows(o, r.z) + lane) : 0;  // a lane's inflow
        if (r.w >= 0) rn = __ldcg(t_rec + r.w);
        for (size_t chain = 0; o >= 0 && chain <= N; ++chain) {
            const int cnt = r.z & 0xffff;
            float2 v = make_float2(0.f, 0.f);
            if (lane < cnt) v = __ldcg(fa + in);
            int4 rnn = make_int4(0, 0, 0, -1);
            int32_t inn = 0;
            if (r.w >= 0) {
                if (lane < (rn.z & 0xffff)) inn = __ldg(inflows(r.w, rn.z) + lane);
                if (rn.w >= 0) rnn = __ldcg(t_rec + rn.w);
            }
            float2 acc = make_float2(__int_as_float(r.x), __int_as_float(r.y));
            for (int i0 = 0; i0 < cnt; i0 += 32) {
                if (i0 && i0 + lane < cnt) v = __ldcg(fa + __ldg(inflows(o, r.z) + i0 + lane));
                const int m = min(32, cnt - i0);
                for (int i = 0; i < m; ++i)
                    acc = ff_add(acc, make_float2(__shfl_sync(0xffffffffu, v.x, i), __shfl_sync(0xffffffffu, v.y, i)));
            }
            bool last = false;
            if (lane == 0) {
                __stcg(fa + o, acc);
                last = r.w >= 0 && dec_acq_rel(t_pend + r.w) == 1;
            }
            __syncwarp();
            o = __any_sync(0xffffffffu, last) ? r.w : -1;
            r = rn;
            rn = rnn;
            in = inn;
        }
    }
}

__global__ void __launch_bounds__(256)
    k_fat_final(const double* __restrict__ z, const uint8_t* __restrict__ mask, const uint8_t* __restrict__ fd,
                const float* __restrict__ w, const int32_t* __restrict__ t_pend, float2* fa,
                const int32_t* __restrict__ n_meta, const int32_t* __restrict__ n_ref, const int2* __restrict__ f_idx,
                const float2* __restrict__ f_la, const int32_t* __restrict__ t_fcnt, ModelConsts k, DevScalars* sc,
                DemCtx dc, TileSet ts, int count) {
    if (!sc->tiled_ok) return;
    __shared__ uint8_t s_code[kTH * kTH];
    __shared__ uint8_t s_cls[kTH * kTH];
    __shared__ float2 s_hval[kRing];  // the ring's accumulations
    __shared__ uint8_t s_hok[kRing];  //   and whether they are final
    __shared__ int32_t s_pd[kTile * kTile];
    __shared__ int32_t s_h[kTile * kTile];
    __shared__ float2 s_val[kTile * kTile + 1];
    __shared__ __align__(4) uint16_t s_dm[kTile * kTile];
    __shared__ uint32_t s_ent[kTile * kTile];
    __shared__ uint32_t s_bins[kTile * kTile / 2];
    __shared__ uint32_t s_wait[kTile], s_bad[kTile];
    __shared__ int s_done, s_dem, s_qn;
    const int W = k.W, H = k.H, TW = (W + kTile - 1) / kTile;
    const int t = ts.tile(blockIdx.x);
    const int fc = t_fcnt[t];
    if (fc >= 0) {
        // The tile's program: each node's sum of inflows, then every waiting
        // cell's local accumulation plus the sum of its node.  A node is valid
        // when every inflow upstream completed.
        const int ne = fc & 0xffff, nn = fc >> 16;
        const size_t tb = (size_t)t * kTile * kTile, pool = (size_t)t * kTilePool;
        float2* s_X = s_val;      // node sums
        int32_t* s_ok = s_pd;    // node valid
        // (the second wave's arrays are free here) per node: its largest input
        // node + 1 and its number of input nodes, and up to four input nodes
        int16_t* s_nin = reinterpret_cast<int16_t*>(s_h);         // (largest + 1) | count << 11
        int16_t* s_in4 = reinterpret_cast<int16_t*>(s_ent);       // [4 * node], a tile has fewer than 512 nodes
        for (int n = threadIdx.x; n < nn; n += blockDim.x) {
            const int meta = n_meta[tb + n];
            const int start = meta & 2047, nin = meta >> 11;
            float2 acc = make_float2(0.f, 0.f);
            int ok = 1, top = 0, cnt = 0;
            for (int j = 0; j < nin; ++j) {
                const int32_t ref = n_ref[pool + start + j];
                if (ref < 0) {  // an input node: added in the pass below
                    const int u = -ref - 1;
                    if (cnt < 4) s_in4[4 * n + cnt] = (int16_t)u;
                    ++cnt;
                    top = u + 1 > top ? u + 1 : top;
                    continue;
                }
                acc = ff_add(acc, __ldcg(fa + ref));
                ok &= t_pend[ref] == 0;
            }
            s_X[n] = acc;
            s_ok[n] = ok;
            s_nin[n] = (int16_t)(top | (cnt << 11));
        }
        __syncthreads();
        if (threadIdx.x < 32) {
            // in index order (a node's inputs have smaller indices), a run of
            // nodes with no input inside the run at a time
            const int lane = threadIdx.x;
            for (int i = 0; i < nn;) {
                const int n = i + lane;
                int info = 0;
                if (n < nn) info = s_nin[n];
                const bool dep = n < nn && (info & 2047) - 1 >= i;
                const unsigned b = __ballot_sync(0xffffffffu, dep);
                const int run = b ? __ffs(b) - 1 : 32;  // lane 0's inputs all lie before i
                if (lane < run && n < nn) {
                    float2 acc = s_X[n];
                    int ok = s_ok[n];
                    const int cnt = info >> 11;
                    if (cnt <= 4) {
                        for (int j = 0; j < cnt; ++j) {
                            const int u = s_in4[4 * n + j];
                            acc = ff_add(acc, s_X[u]);
                            ok &= s_ok[u];
                        }
                    } else {  // more input nodes than kept: from memory, in the same order
                        const int meta = n_meta[tb + n];
                        for (int j = 0; j < (meta >> 11); ++j) {
                            const int32_t ref = n_ref[pool + (meta & 2047) + j];
                            if (ref >= 0) continue;
                            acc = ff_add(acc, s_X[-ref - 1]);
                            ok &= s_ok[-ref - 1];
                        }
                    }
                    s_X[n] = acc;
                    s_ok[n] = ok;
                }
                __syncwarp();
                i += run;
            }
        }
        __syncthreads();
        int done = 0, dem = -1;
        for (int e = threadIdx.x; e < ne; e += blockDim.x) {
            const int2 id = f_idx[tb + e];
            dem = dem_at(dc, (size_t)id.x);
            if (id.y == kLaOutlet) {
                done += t_pend[id.x] == 0;
                continue;
            }
            if (!s_ok[id.y]) continue;
            fa[id.x] = ff_add(f_la[tb + e], s_X[id.y]);
            ++done;
        }
        done = wsum(done);
        dem = __reduce_max_sync(0xffffffffu, dem);
        if (count && (threadIdx.x & 31) == 0 && done && dem >= 0) atomicAdd(&dc.out[dem].fa_done, done);
        return;
    }
    // The second wave: every cell of the tile by the reference formula, in level
    // order, with the donors in other tiles (outlets of theirs) at their final
    // values.  A cell below a donor that never completes stays as it is, and an
    // outlet keeps the coarse wave's value.
    const int tx0 = (t % TW) * kTile, ty0 = (t / TW) * kTile;
    const int lx = threadIdx.x & 31, ly0 = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kTile * kTile / 2; i += blockDim.x) {
        s_bins[i] = 0;
        reinterpret_cast<uint32_t*>(s_dm)[i] = 0;
    }
    if (threadIdx.x < kTile) s_wait[threadIdx.x] = s_bad[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_done = s_qn = 0, s_dem = -1, s_val[kNoCell] = make_float2(0.f, 0.f);
    __syncthreads();
    tile_stage(
        fd, [&](size_t g, int, int) { return mask[g] ? kCellIn : (z[g] == kNoData ? kCellOff : kCellBlock); }, W, H, tx0,
        ty0, s_code, s_cls, s_dm, s_bad);
    if (threadIdx.x < kRing) {
        const int h = ring_halo(threadIdx.x);
        const int gx = tx0 - 1 + h % kTH, gy = ty0 - 1 + h / kTH;
        bool ok = false;
        float2 v = make_float2(0.f, 0.f);
        if (gx >= 0 && gx < W && gy >= 0 && gy < H && mask[(size_t)gy * W + gx]) {
            const size_t g = (size_t)gy * W + gx;
            ok = t_pend[g] == 0;
            v = fa[g];
        }
        s_hok[threadIdx.x] = ok;
        s_hval[threadIdx.x] = v;
    }
    __syncthreads();
    // the neighbour in direction scan_dir(k) of cell l when it lies in another tile
    auto ring_of = [&](int l, int k) {
        const int d = scan_dir(k);
        return ring_index((l & (kTile - 1)) + 1 + dir_dx(d), l / kTile + 1 + dir_dy(d));
    };
    auto sum = [&](int l) {  // CalcMFD's donor sum in scan order
        const uint32_t dm = s_dm[l];
        float2 acc = make_float2(0.f, 0.f);
        for (uint32_t m = (dm | (dm >> 8)) & 255u; m; m &= m - 1) {
            const int k = __ffs(m) - 1;
            acc = ff_add(acc, (dm >> k) & 1u ? s_val[l + scan_step(k)] : s_hval[ring_of(l, k)]);
        }
        return acc.x < 0.0f ? make_float2(0.f, 0.f) : acc;
    };
    int done = 0, dem = -1;  // one DEM per tile
    bool outlet[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx, hc = (ly + 1) * kTH + lx + 1;
        const size_t g = (size_t)(ty0 + ly) * W + tx0 + lx;
        int32_t pd = l;
        float wl = 0.f;
        outlet[q] = false;
        if (s_cls[hc] == kCellIn) {
            const int d = bit_dir(s_code[hc]);
            const int rlx = lx + dir_dx(d < 0 ? 0 : d), rly = ly + dir_dy(d < 0 ? 0 : d);
            if (d >= 0 && s_cls[(rly + 1) * kTH + rlx + 1] == kCellIn) {
                outlet[q] = !in_tile(rlx, rly);
                if (!outlet[q]) pd = (rly * kTile + rlx) | (1 << 10);
            }
            if (outlet[q] && t_pend[g] == 0) ++done;
            wl = w ? w[g] : 1.0f;
            if (dem < 0) dem = dem_at(dc, g);
            for (uint32_t m = s_dm[l] >> 8; m; m &= m - 1)
                if (!s_hok[ring_of(l, __ffs(m) - 1)]) atomicOr(&s_bad[ly], 1u << lx);
        }
        s_pd[l] = pd;
        s_h[l] = 0;
        s_val[l] = make_float2(wl, 0.f);
    }
    dem = __reduce_max_sync(0xffffffffu, dem);
    if (lx == 0 && dem >= 0) atomicMax(&s_dem, dem);
    __syncthreads();
    tile_paths(s_pd, s_h, s_wait, s_bad, lx, ly0);
    int level[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        const bool on = s_cls[(ly + 1) * kTH + lx + 1] == kCellIn && !((s_bad[ly] >> lx) & 1u) && !outlet[q];
        level[q] = on ? s_h[l] : -1;
        if (level[q] == 0) s_val[l] = ff_add(s_val[l], sum(l));  // donors in other tiles only
    }
    tile_sort(
        level,
        [&](int q) {
            const int l = (ly0 + 8 * q) * kTile + lx;
            return entry_of(l, s_dm[l] & 255u) | (s_dm[l] >> 8 ? kMoreDonors : 0u);
        },
        s_bins, kTile * kTile / 2, s_ent, &s_qn, lx);
    struct Cell {
        float2 w;
        uint32_t e;
    };
    tile_levels(
        [&](uint32_t e) { return Cell{s_val[entry_cell(e)], e}; },
        [&](const Cell& f) {
            const int c = entry_cell(f.e);
            float2 acc = ff_add(s_val[entry_d0(f.e)], s_val[entry_d1(f.e)]);
            if (acc.x < 0.0f) acc = make_float2(0.f, 0.f);
            if (f.e & kMoreDonors) acc = sum(c);
            s_val[c] = ff_add(f.w, acc);
        },
        1, kTile * kTile, s_bins, s_ent);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (level[q] < 0) continue;
        const int ly = ly0 + 8 * q;
        fa[(size_t)(ty0 + ly) * W + tx0 + lx] = s_val[ly * kTile + lx];
        ++done;
    }
    done = wsum(done);
    if ((threadIdx.x & 31) == 0 && done) atomicAdd(&s_done, done);
    __syncthreads();
    if (count && threadIdx.x == 0 && s_done && s_dem >= 0) atomicAdd(&dc.out[s_dem].fa_done, s_done);
}

// The contributing-cell counts of a tiled step are the accumulation of unit
// weights: the float pairs hold the whole numbers exactly (far beyond 2^31), so
// the same kernels give them, in the place of the int32 counts of the general
// wave (7.2 ms against 0.4 ms at 1501 x 1501 cells).  A cell the wave never
// finishes counts itself only.
__global__ void k_count_init(const uint8_t* __restrict__ mask, float2* __restrict__ cnt,
                             const int32_t* __restrict__ chunk_start, int W, DemCtx dc, DevScalars* sc) {
    if (!sc->tiled_ok) return;
    const Chunk ch = chunk_of(chunk_start, dc);
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->tile_src = 0;
    for (int64_t ri = ch.first + threadIdx.x; ri < ch.end; ri += blockDim.x) {
        int x, y;
        const size_t i = region_cell(dc.in[ch.d], ri, W, &x, &y);
        cnt[i] = make_float2(mask[i] ? 1.0f : 0.0f, 0.0f);
    }
}
__global__ void k_count_out(const float2* __restrict__ cnt, int32_t* __restrict__ contrib,
                            const int32_t* __restrict__ chunk_start, int W, DemCtx dc, DevScalars* sc) {
    if (!sc->tiled_ok) return;
    const Chunk ch = chunk_of(chunk_start, dc);
    for (int64_t ri = ch.first + threadIdx.x; ri < ch.end; ri += blockDim.x) {
        int x, y;
        const size_t i = region_cell(dc.in[ch.d], ri, W, &x, &y);
        const float2 v = cnt[i];
        contrib[i] = (int32_t)v.x + (int32_t)v.y;  // both are whole
    }
}

// The tiled accumulation of weights w (null: one each) into fa.  count: add the
// finished cells to the DEMs' counters.
struct FatArgs {
    const double* z;
    const uint8_t* mask;
    const uint8_t* fd;
    const float* w;
    float2* fa;
    int4* t_rec;
    int32_t* t_dst;
    int32_t* t_pend;
    int32_t* t_ent;
    int32_t* n_meta;
    int32_t* n_ref;
    int2* f_idx;
    float2* f_la;
    int32_t* t_fcnt;
    int32_t* outs;
    int32_t* ready;
    DevScalars* sc;
    DemCtx dc;
    int coarse_blocks;
};
lem_status launch_fat(const FatArgs& a, const ModelConsts& k, const TileSet& ts, int count, const Launch& L) {
    LEM_LAUNCH(L, k_fat_local, ts.n, 256, a.z, a.mask, a.fd, a.w, a.t_rec, a.t_dst, a.t_pend, a.t_ent, a.fa, a.n_meta,
               a.n_ref, a.f_idx, a.f_la, a.t_fcnt, a.outs, k, a.sc, a.dc, ts, count);
    const uint8_t* fd = a.fd;
    int4* trec = a.t_rec;
    const int32_t* tent = a.t_ent;
    const int32_t* tdst = a.t_dst;
    float2* fa = a.fa;
    int32_t* tpend = a.t_pend;
    const int32_t* outs = a.outs;  // the outlets, listed by k_fat_local
    int32_t* ready = a.ready;
    ModelConsts kk = k;
    DevScalars* sc = a.sc;
    void* args[] = {(void*)&fd,    (void*)&trec, (void*)&tent,  (void*)&tdst, (void*)&fa,
                    (void*)&tpend, (void*)&outs, (void*)&ready, (void*)&kk,   (void*)&sc};
    L.pre("k_fat_coarse");
    LEM_CUDA_TRY(coop_launch((const void*)k_fat_coarse, a.coarse_blocks, args, L.st));
    L.post();
    LEM_LAUNCH(L, k_fat_final, ts.n, 256, a.z, a.mask, a.fd, a.w, a.t_pend, a.fa, a.n_meta, a.n_ref, a.f_idx, a.f_la,
               a.t_fcnt, k, a.sc, a.dc, ts, count);
    return LEM_OK;
}

// correctmfdflow's first-iteration branch (mfd_simple.cu:336-349): the outlet
// becomes the first cell holding the largest accumulation.  Bound by memory once
// a warp makes one atomic: one for every cell queued up at the DEM's one word (484
// -> 18 us for twelve DEMs of 128 to 1024 cells a side).
__global__ void k_fa_argmax(const float2* __restrict__ fa, const int32_t* __restrict__ chunk_start, int W,
                            DemCtx dc, int phase) {
    const Chunk ch = chunk_of(chunk_start, dc);
    const DemIn& r = dc.in[ch.d];
    DemOut& o = dc.out[ch.d];
    if (!r.outlet_from_fa) return;
    unsigned long long best = 0;
    const unsigned long long top = phase == 0 ? 0ull : o.fa_max_key;
    int32_t first = 0x7fffffff;
    for (int64_t ri = ch.first + threadIdx.x; ri < ch.end; ri += blockDim.x) {
        int x, y;
        const size_t i = region_cell(r, ri, W, &x, &y);
        const float2 v = fa[i];
        if (v.x != v.x) continue;  // NaN never wins the host scan (mfd_simple.cu:341)
        const unsigned long long kk = ffkey(v);
        best = kk > best ? kk : best;
        if (phase != 0 && kk == top) first = min(first, (int32_t)i);
    }
    if (phase == 0) {
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, w);
            best = other > best ? other : best;
        }
        if ((threadIdx.x & 31) == 0 && best > __ldcg(&o.fa_max_key)) atomicMax(&o.fa_max_key, best);
    } else {
        first = __reduce_min_sync(0xffffffffu, first);
        if ((threadIdx.x & 31) == 0 && first < __ldcg(&o.argmax)) atomicMin(&o.argmax, first);
    }
}

// The DEM's outlet becomes the first cell of the largest accumulation; with
// none above zero the reference's scan leaves index 0, the region's first cell.
__global__ void k_fa_argmax_set(int W, DemCtx dc) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= dc.n || !dc.in[d].active || !dc.in[d].outlet_from_fa) return;
    const unsigned long long zero = ffkey(make_float2(0.f, 0.f));
    DemOut& o = dc.out[d];
    o.outlet = (o.fa_max_key > zero) ? o.argmax : dc.in[d].y0 * W + dc.in[d].x0;
}

__global__ void k_fa_reset(DevScalars* sc, DemCtx dc, int tiled) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d == 0) {
        sc->counters[0] = 0;
        sc->tiled_ok = tiled;
        sc->tile_src = 0;
    }
    if (d < dc.n) {
        DemOut& o = dc.out[d];
        o.fa_done = 0;
        o.n_active = 0;
        o.fa_max_key = 0ull;
        o.argmax = 0x7fffffff;
    }
}

}  // namespace

lem_status launch_flow_accumulation(const DevState& s, const ModelConsts& k, uint32_t flags, const Launch& L) {
    const size_t N = (size_t)k.W * k.H;
    const int T = 256;
    size_t nb = (N + T - 1) / T;
    const int blocks = (int)(nb > 152 * 32 ? 152 * 32 : nb);
    const int dem_blocks = (s.dems.n + 127) / 128;
    int32_t* contrib = (flags & LEM_STEP_CONTRIB) ? s.contrib : nullptr;
    const int tiled = k.flow_type == 0 ? 1 : 0;
    LEM_LAUNCH(L, k_fa_reset, dem_blocks, 128, s.sc, s.dems, tiled);
    const float* prop = nullptr;
    if (k.flow_type != 0 && k.mfd_props) {
        LEM_LAUNCH(L, k_calcprops, blocks, T, s.mask, s.fd, s.slopes, s.prop, N);
        prop = s.prop;
    }
    LEM_LAUNCH(L, k_fa_prep, s.n_chunks, T, s.mask, s.fd, s.stone, s.totB, s.soilM, s.w, s.fa, s.chunk_start, k,
               s.dems, s.sc);
    LEM_LAUNCH(L, k_fa_pend, s.n_chunks, T, s.z, s.mask, s.fd, s.pending, contrib, s.list_a, s.chunk_start, k, s.dems,
               s.sc, tiled);
    if (tiled) {
        const TileSet ts = tiles_of(s, k.W);
        FatArgs a{s.z, s.mask, s.fd, s.w, s.fa, s.t_rec, s.t_dst, s.t_pend, s.t_ent, s.n_meta, s.p_ref,
                  reinterpret_cast<int2*>(s.f_idx), s.f_ds, s.t_fcnt, s.list_b, s.list_a, s.sc, s.dems,
                  coop_for(s, k, kCkFatCoarse)};
        lem_status r = launch_fat(a, k, ts, 1, L);
        if (r != LEM_OK) return r;
        if (contrib) {
            a.w = nullptr;
            a.fa = reinterpret_cast<float2*>(s.p_map);  // free until the sediment programs: one pair per cell
            LEM_LAUNCH(L, k_count_init, s.n_chunks, T, s.mask, a.fa, s.chunk_start, k.W, s.dems, s.sc);
            if ((r = launch_fat(a, k, ts, 0, L)) != LEM_OK) return r;
            LEM_LAUNCH(L, k_count_out, s.n_chunks, T, a.fa, contrib, s.chunk_start, k.W, s.dems, s.sc);
        }
    }
    {
        float2* fa = s.fa;
        int32_t* word = s.pending;
        int32_t* list = s.list_a;
        ModelConsts kk = k;
        DevScalars* sc = s.sc;
        DemCtx dc = s.dems;
        int gate = tiled;
        void* args[] = {(void*)&prop, (void*)&fa, (void*)&word, (void*)&contrib, (void*)&list,
                        (void*)&kk,   (void*)&sc, (void*)&dc,   (void*)&gate};
        L.pre("k_fa_walk");
        LEM_CUDA_TRY(coop_launch((const void*)k_fa_walk, coop_for(s, k, kCkFaWalk), args, L.st));
        L.post();
    }
    if (flags & LEM_STEP_SET_OUTLET_FROM_FA) {  // some DEM moves its outlet this step
        LEM_LAUNCH(L, k_fa_argmax, s.n_chunks, T, s.fa, s.chunk_start, k.W, s.dems, 0);
        LEM_LAUNCH(L, k_fa_argmax, s.n_chunks, T, s.fa, s.chunk_start, k.W, s.dems, 1);
        LEM_LAUNCH(L, k_fa_argmax_set, dem_blocks, 128, k.W, s.dems);
    }
    LEM_CUDA_TRY(cudaGetLastError());
    return LEM_OK;
}

// ---------------------------------------------------------------------------
// lem_accumulate_flow_noalloc: the accumulation wave on caller-owned buffers,
// with its intermediate data in one file-scope device array.
namespace {

constexpr size_t kNaCells = LEM_NOALLOC_MAX_CELLS;
// The tiled accumulation's tables hold this many tiles, an eighth more than the
// cells fill: grids a few columns or rows over a multiple of 32 fit, narrow
// strips take the general wave.
constexpr size_t kNaTiles = kNaCells / (kTile * kTile) * 9 / 8;
constexpr size_t kNaSlots = kNaTiles * kTile * kTile;
constexpr size_t kNaHead = 1024;  // DevScalars and one DemOut, rounded up
constexpr size_t kNaOffDem = 512;
static_assert(sizeof(DevScalars) <= kNaOffDem && kNaOffDem + sizeof(DemOut) <= kNaHead, "scalar block");
constexpr size_t kNaOffFa = kNaHead;                          // float2 per cell
constexpr size_t kNaOffRec = kNaOffFa + 8 * kNaCells;         // int4
constexpr size_t kNaOffDst = kNaOffRec + 16 * kNaCells;       // int32
constexpr size_t kNaOffPend = kNaOffDst + 4 * kNaCells;       // int32 (the general wave's words)
constexpr size_t kNaOffOuts = kNaOffPend + 4 * kNaCells;      // int32 (and its list)
constexpr size_t kNaOffReady = kNaOffOuts + 4 * kNaCells;     // int32
constexpr size_t kNaOffW = kNaOffReady + 4 * kNaCells;        // float
constexpr size_t kNaOffFd = kNaOffW + 4 * kNaCells;           // u8
constexpr size_t kNaOffMask = kNaOffFd + kNaCells;            // u8
constexpr size_t kNaOffIdx = kNaOffMask + kNaCells;           // int2 per slot
constexpr size_t kNaOffLa = kNaOffIdx + 8 * kNaSlots;         // float2
constexpr size_t kNaOffMeta = kNaOffLa + 8 * kNaSlots;        // int32
constexpr size_t kNaOffRef = kNaOffMeta + 4 * kNaSlots;       // int32, kTilePool per tile
constexpr size_t kNaOffEnt = kNaOffRef + 4 * kTilePool * kNaTiles;  // int32, kTileEnt per tile
constexpr size_t kNaOffCnt = kNaOffEnt + 4 * kTileEnt * kNaTiles;   // int32 per tile
constexpr size_t kNaBytes = kNaOffCnt + 4 * kNaTiles;

// Scratch of the no-allocation entry point (every call shares it).
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

struct NaDevice {
    unsigned char* base = nullptr;  // device address of g_noalloc_scratch
    int walk_blocks = 0;            // co-resident blocks of k_fa_walk
    int coarse_blocks = 0;          //   and of k_fat_coarse
};
std::mutex g_na_mutex;
NaDevice g_na[64];

__global__ void k_na_reset(DevScalars* sc, DemOut* dem, int tiled) {
    dem->fa_done = 0;
    dem->n_active = 0;
    sc->counters[0] = 0;
    sc->tile_src = 0;
    sc->tiled_ok = tiled;
    sc->err = 0;
    sc->err_first = 0;
}

// Codes, mask, weights and the initial accumulation (the weight) from the
// caller's int32 codes and DEM (cells at -9999 are outside and complete with
// zero flow).  As in a step, a negative weight or a multi-direction code sends
// the call to the general wave.
__global__ void __launch_bounds__(256)
    k_na_prep(const int32_t* __restrict__ fd_in, const double* __restrict__ w_in, const double* __restrict__ dem,
              uint8_t* __restrict__ fd, uint8_t* __restrict__ mask, float* __restrict__ w, float2* __restrict__ fa,
              size_t N, DevScalars* sc, DemOut* dem_out) {
    int nact = 0;
    bool untiled = false;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        const bool in = dem[i] != kNoData;
        const uint32_t code = (uint32_t)fd_in[i] & 0xffu;
        const float wi = (float)w_in[i];
        fd[i] = (uint8_t)code;
        mask[i] = in ? 1 : 0;
        w[i] = wi;
        fa[i] = make_float2(in ? wi : 0.0f, 0.0f);
        nact += in;
        untiled |= in && (wi < 0.0f || (code & (code - 1)));
    }
    if (__syncthreads_or(untiled) && threadIdx.x == 0) sc->tiled_ok = 0;
    const int tot = block_sum_i(nact);
    if (threadIdx.x == 0 && tot) atomicAdd(&dem_out->n_active, tot);
}

// The general wave's words and sources.
__global__ void k_na_words(const uint8_t* __restrict__ fd, const uint8_t* __restrict__ mask,
                           int32_t* __restrict__ word, int32_t* ready, int W, int H, DevScalars* sc) {
    if (sc->tiled_ok) return;
    const size_t N = (size_t)W * H;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < N; base += (size_t)gridDim.x * blockDim.x) {
        const size_t i = base + threadIdx.x;
        bool src = false;
        if (i < N) {
            const int x = (int)(i % W), y = (int)(i / W);
            const bool in = mask[i];
            const uint32_t code = fd[i];
            int32_t pend = in ? 0 : kBlocked;
            uint32_t donors = 0, receivers = 0;
#pragma unroll
            for (int d = 0; d < 8; ++d) {
                const int nx = x + dir_dx(d), ny = y + dir_dy(d);
                if (!in || nx < 0 || nx >= W || ny < 0 || ny >= H) continue;
                const size_t n = (size_t)ny * W + nx;
                if (!mask[n]) continue;
                receivers |= code & dir_bit(d);
                if (donates(fd[n], d)) {
                    ++pend;
                    donors |= 1u << scan_index(d);
                }
            }
            word[i] = wave_word(pend, donors, receivers);
            src = in && pend == 0;
        }
        wave_append(src, (int32_t)i, ready, &sc->counters[0], (int)N, &sc->err);
    }
}

__global__ void k_na_out(const float2* __restrict__ fa, double* __restrict__ out, size_t N) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x)
        out[i] = (double)fa[i].x + (double)fa[i].y;
}

}  // namespace

extern "C" lem_status lem_accumulate_flow_noalloc(const int32_t* d_fd, const double* d_weight,
                                                  const double* d_dem, double* d_fa, int32_t width,
                                                  int32_t height, void* stream) {
    if (!d_fd || !d_weight || !d_dem || !d_fa || width < 1 || height < 1) return LEM_ERR_INVALID;
    const size_t N = (size_t)width * height;
    if (N > kNaCells) return LEM_ERR_CAPACITY;  // the static scratch holds LEM_NOALLOC_MAX_CELLS cells
    int dev = 0;
    LEM_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return LEM_ERR_INVALID;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    LEM_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
    NaDevice nd;
    {
        std::lock_guard<std::mutex> lock(g_na_mutex);
        if (cap == cudaStreamCaptureStatusNone || !g_na[dev].base) {
            // With that device current: the device address of the array.  It is
            // looked up again on every call outside a stream capture, so a
            // context torn down and created again (cudaDeviceReset) gets the
            // array's new address; inside a capture the address of the last
            // call on this device is used.
            void* ptr = nullptr;
            LEM_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));
            if (!g_na[dev].walk_blocks) {
                g_na[dev].walk_blocks = coop_blocks_for((const void*)k_fa_walk, 256, 0);
                g_na[dev].coarse_blocks = coop_blocks_for((const void*)k_fat_coarse, 256, 0);
            }
            g_na[dev].base = static_cast<unsigned char*>(ptr);
        }
        nd = g_na[dev];
    }
    DevScalars* sc = reinterpret_cast<DevScalars*>(nd.base);
    DemOut* dem = reinterpret_cast<DemOut*>(nd.base + kNaOffDem);
    auto at = [&](size_t off) { return static_cast<void*>(nd.base + off); };
    uint8_t* const fd = static_cast<uint8_t*>(at(kNaOffFd));
    uint8_t* const mask = static_cast<uint8_t*>(at(kNaOffMask));
    float* const w = static_cast<float*>(at(kNaOffW));
    float2* fa = static_cast<float2*>(at(kNaOffFa));
    int32_t* word = static_cast<int32_t*>(at(kNaOffPend));
    int32_t* list = static_cast<int32_t*>(at(kNaOffOuts));
    const int T = 256;
    const int blocks = (int)std::min<size_t>((N + T - 1) / T, 152 * 32);
    const int tw = (width + kTile - 1) / kTile, tiles = tw * ((height + kTile - 1) / kTile);
    const int tiled = (size_t)tiles <= kNaTiles;
    ModelConsts k{};
    k.W = width;
    k.H = height;
    const DemCtx dc{nullptr, nullptr, dem, 1, kChunkMax};
    uint64_t launches = 0;
    const Launch L{st, &launches, nullptr};
    k_na_reset<<<1, 1, 0, st>>>(sc, dem, tiled);  // the array keeps the previous call's contents
    k_na_prep<<<blocks, T, 0, st>>>(d_fd, d_weight, d_dem, fd, mask, w, fa, N, sc, dem);
    if (tiled) {
        const FatArgs a{d_dem, mask, fd, w, fa, static_cast<int4*>(at(kNaOffRec)), static_cast<int32_t*>(at(kNaOffDst)),
                        word, static_cast<int32_t*>(at(kNaOffEnt)), static_cast<int32_t*>(at(kNaOffMeta)),
                        static_cast<int32_t*>(at(kNaOffRef)), static_cast<int2*>(at(kNaOffIdx)),
                        static_cast<float2*>(at(kNaOffLa)), static_cast<int32_t*>(at(kNaOffCnt)), list,
                        static_cast<int32_t*>(at(kNaOffReady)), sc, dc, std::min(nd.coarse_blocks, 2 * tiles)};
        const lem_status r = launch_fat(a, k, TileSet{nullptr, tiles, tw}, 1, L);
        if (r != LEM_OK) return r;
    }
    k_na_words<<<blocks, T, 0, st>>>(fd, mask, word, list, width, height, sc);
    LEM_CUDA_TRY(cudaGetLastError());
    {
        const float* prop = nullptr;
        int32_t* contrib = nullptr;
        int gate = tiled;
        DemCtx d = dc;
        void* args[] = {(void*)&prop, (void*)&fa, (void*)&word, (void*)&contrib, (void*)&list,
                        (void*)&k,    (void*)&sc, (void*)&d,    (void*)&gate};
        LEM_CUDA_TRY(coop_launch((const void*)k_fa_walk, walk_blocks(nd.walk_blocks, N), args, st));
    }
    k_na_out<<<blocks, T, 0, st>>>(fa, d_fa, N);
    LEM_CUDA_TRY(cudaGetLastError());
    unsigned char head[kNaHead];  // the scalars and the counts in one copy
    LEM_CUDA_TRY(cudaMemcpyAsync(head, nd.base, sizeof head, cudaMemcpyDeviceToHost, st));
    LEM_CUDA_TRY(cudaStreamSynchronize(st));
    uint32_t err[2];  // err and err_first
    DemOut counts;
    std::memcpy(err, head + offsetof(DevScalars, err), sizeof err);
    std::memcpy(&counts, head + kNaOffDem, sizeof counts);
    if (err[1] == ErrFlags::kCapacity || (err[0] & ErrFlags::kCapacity && err[1] != ErrFlags::kNoConverge))
        return LEM_ERR_CAPACITY;
    if (err[0]) return LEM_ERR_NOCONVERGE;
    // in-catchment cells the wave never reached (a cycle in the codes, or a
    // donor chain through one): they hold their own weight, as correctmfdflow
    // leaves them (mfd_simple.cu:72), and the call says so
    if (counts.fa_done < counts.n_active) return LEM_ERR_NOCONVERGE;
    return LEM_OK;
}

const void* fa_coop_kernels[] = {(const void*)k_fa_walk, (const void*)k_fat_coarse};
extern const int fa_coop_kernel_count = 2;

}  // namespace lem
