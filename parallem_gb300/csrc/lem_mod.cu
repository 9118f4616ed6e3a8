// lem_mod.cu -- process stage: erosion, sediment routing, surface update.
//
// erosionGPU (MOD_kernels/erosion.cu:69-186) runs ten kernels and ~20 host
// copies per step.  Here it is three passes over the grid:
//   k_erosion  aveslope + diff_erosion + conc_erosion + gelifluction
//              (eroincidep.cu:8-198), budget sums and FA_max in the epilogue;
//   k_sed_*    sedmfdaccum / MFDsedbud (mfd_accum.cu:32-483) as a dependency
//              wave like the accumulation (lem_fa.cu);
//   k_final    surface_change + weathering + Update_Surface +
//              update_nutrient_content + grow_vegetation (eroincidep.cu:200-327,
//              updates.cu:23-139) fused, with their budget sums.
// The climate grids of SetClimateMatrices (Data.cpp:211-303) are generated on
// the fly from the row index and the DEM.

#include <cooperative_groups.h>

#include "lem_wave.cuh"

namespace cg = cooperative_groups;

namespace lem {

namespace {

constexpr double kMinHeight = 467.228;  // Data.cpp:252

// Temperature of cell i (tempmat): T - (z - 467.228) * 0.0065 with z the DEM the
// grids were built from (the initial DEM during run-in, the DEM at the start of
// the step otherwise; the outlet uses its value before the stage-1 adjustment).
__device__ __forceinline__ float clim_temp(const DemIn& c, const double* z, const double* z_init, size_t i,
                                           int outlet_clim, double outlet_z) {
    double zc = c.from_current_dem ? (((int)i == outlet_clim) ? outlet_z : z[i]) : z_init[i];
    float hi, lo;
    dsplit(zc, hi, lo);
    return (float)c.temp - ((hi - (float)kMinHeight) + lo) * 0.0065f;
}

// K sums of fp32 terms over a block of 256 threads: fp32 over a warp's 128 cells
// (four turns of the loop), fp64 from there on, so the totals depend on the size
// of the blocks only in the last bits of fp64.  turn() is called by every thread
// after every cell, finish() by every thread at the end; add_to's thread k < K
// then holds sum k.
template <int K>
struct BlockSums {
    double (*red)[K];  // [8] in shared memory
    float v[K];
    int turns = 0;
    __device__ __forceinline__ explicit BlockSums(double (*r)[K]) : red(r) {
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[k] = 0.f;
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = 0.0;
        }
    }
    __device__ __forceinline__ void flush() {
#pragma unroll
        for (int k = 0; k < K; ++k) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] += (double)v[k];
            v[k] = 0.f;
        }
    }
    __device__ __forceinline__ void turn() {
        if ((++turns & 3) == 0) flush();
    }
    __device__ __forceinline__ double finish() {
        if (turns & 3) flush();
        __syncthreads();
        double t = 0.0;
        if (threadIdx.x < K)
            for (int w = 0; w < 8; ++w) t += red[w][threadIdx.x];
        return t;
    }
};

__device__ __forceinline__ unsigned long long block_max_u64(unsigned long long v, unsigned long long* red) {
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long u = __shfl_xor_sync(0xffffffffu, v, o);
        v = u > v ? u : v;
    }
    const int wid = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[wid] = v;
    __syncthreads();
    unsigned long long m = 0;
    if (threadIdx.x == 0)
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) m = red[i] > m ? red[i] : m;
    return m;
}

// Six blocks per SM: a few spilled registers, measured faster than four or five (4096
// x 4096 cells: 350 us, 386 and 366; 334 with sums that left fp32 once per block, which
// depend on the size of the blocks).
__global__ void __launch_bounds__(256, 6)
    k_erosion(const double* __restrict__ z, const double* __restrict__ z_init, const uint8_t* __restrict__ mask,
              const float* __restrict__ slopes, const float2* __restrict__ fa, const float* __restrict__ fines,
              const float* __restrict__ nut, const float* __restrict__ soilT, const float* __restrict__ stone,
              const float* __restrict__ totB, float* __restrict__ slopeptr, float* __restrict__ ero,
              float* __restrict__ inci, float* __restrict__ geli, float* __restrict__ depo,
              const uint8_t* __restrict__ fd, const int32_t* __restrict__ chunk_start, ModelConsts k, DemCtx dc,
              DevScalars* sc) {
    __shared__ double red[8][3];
    __shared__ unsigned long long redk[8];
    const Chunk ch = chunk_of(chunk_start, dc);
    const DemIn& c = dc.in[ch.d];
    DemOut& o = dc.out[ch.d];
    const int W = k.W;
    const int outlet = o.outlet;
    const int outlet_clim = o.outlet_clim;  // the cell whose climate elevation is outlet_z_clim
    const double outlet_z = o.outlet_z_clim;
    if (ch.first == 0 && threadIdx.x == 0) o.base_level = z[outlet] - 0.00012;  // updates.cu:151
    BlockSums<3> sums(red);
    unsigned long long famax = 0;
    bool multi = false;
    auto cell = [&](int64_t ri) {
        int x, y;
        const size_t i = region_cell(c, ri, W, &x, &y);
        // every input of the cell in one batch of loads, ahead of the mask test
        // and the arithmetic (the region's cells outside the catchment are few)
        const float2 f2 = fa[i];
        const uint8_t mk = mask[i], code = fd[i];
        const float4 a = reinterpret_cast<const float4*>(slopes)[2 * i];
        const float4 b = reinterpret_cast<const float4*>(slopes)[2 * i + 1];
        const float st = soilT[i], tb = totB[i], fi = fines[i], nu = nut[i], sto = stone[i];
        float T = clim_temp(c, z, z_init, i, outlet_clim, outlet_z);
        const unsigned long long fk = ffkey(f2);
        if (f2.x == f2.x) famax = fk > famax ? fk : famax;  // the reduction skips NaN (thrust::maximum order)
        if (!mk) {
            ero[i] = inci[i] = geli[i] = 0.0f;
            slopeptr[i] = 0.0f;
            return;
        }
        // sedmfdaccum set-up (mfd_accum.cu:389-396): depo = 1e-5 in the catchment.
        // A multi-direction code among the routed cells (not row 0 / column 0,
        // mfd_accum.cu:42) sends the step's sediment routing to the walk.
        depo[i] = 0.00001f;
        if (x != 0 && y != 0) multi |= (code & (code - 1)) != 0;
        // aveslope (eroincidep.cu:8-37): mean of the positive entries
        const float sv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        float total = 0.f;
        int nonzero = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            total += sv[j];
            nonzero += sv[j] > 0.f;
        }
        const float sp = (total > 0.f && nonzero > 0) ? total / (float)nonzero : 0.f;
        slopeptr[i] = sp;
        const float fav = f2.x + f2.y;
        const float veg = expf(-0.07f * tb / 76.5f);
        // diff_erosion (eroincidep.cu:39-87)
        float erod = (2.77e-6f * powf(fi, 1.14f) * (12.0f - nu)) + k.erod_const;
        if (erod < 0.f) erod = 0.f;
        float OF = (fav * 1000.0f) / 25.0f;
        if (OF > k.q_threshold) OF = k.q_threshold;
        float slope = sp;
        if (slope == 0.f) slope = 0.0001f;
        if (slope > 5.0f) slope = 5.0f;
        float e = ((erod * OF * OF * powf(slope, 1.67f) * (powf(110.0f - sto, 0.877f) / 61.7023f))) * veg;
        if (e > st) e = st;
        // conc_erosion (eroincidep.cu:89-152)
        float cslope = sp;
        if (cslope > 0.5f) cslope = 0.5f;
        // fa * cs^2/1e4 - Qthreshold cancels near the threshold: evaluate it on the
        // (hi, lo) accumulation and the split constants
        float f_temp = fmaf(f2.x, k.rescale_conc, -k.q_threshold) +
                       (fmaf(f2.x, k.rescale_conc_lo, f2.y * k.rescale_conc) - k.q_threshold_lo);
        float in;
        if (f_temp < 0.0f) {
            f_temp = 0.0f;
            in = 0.0f;
        } else {
            in = k.flow_a * powf(f_temp, k.flow_b) * (cslope == 0.0f ? 0.01f : cslope) * veg;
        }
        if (in > k.max_incision) in = k.max_incision;
        if (in > st) {
            const float bed = (1.0f - (st / in)) * 0.0001f * powf(f_temp, k.flow_b) * cslope * veg;
            in = st + bed;
            if (in > k.max_incision) in = k.max_incision;
        }
        // gelifluction (eroincidep.cu:154-198).  The quartic kappa(T) cancels near
        // its roots (T ~ -16.8 and 8.6 C) and the range test has edges at -20 and 8.87 C:
        // there the temperature and kappa take the reference's fp64 arithmetic.
        float kappa = k.kappa;
        if (T >= -20.f && T <= 8.87f)
            kappa = 0.15711f - 0.011835f * T - 0.001195f * T * T + 0.000038f * T * T * T + 0.000002f * T * T * T * T;
        if (fabsf(T - 8.87f) < 1e-3f || fabsf(T + 20.0f) < 1e-3f || fabsf(kappa) < 4e-3f) {
            const double zc = c.from_current_dem ? (((int)i == outlet_clim) ? outlet_z : z[i]) : z_init[i];
            const double Td = c.temp - ((zc - kMinHeight) * 0.0065);
            double kd = (double)k.kappa;
            if (Td >= -20. && Td <= 8.87)
                kd = 0.15711 - 0.011835 * Td - 0.001195 * Td * Td + 0.000038 * Td * Td * Td +
                     0.000002 * Td * Td * Td * Td;
            kappa = (float)kd;
            T = (float)Td;
        }
        // 1 - fa/Gflowlim cancels where fa approaches Gflowlim
        const float gap = ((k.g_flowlim - f2.x) + k.g_flowlim_lo) - f2.y;
        float scaler = gap / (k.g_flowlim + k.g_flowlim_lo);
        if (gap < 0.0f) scaler = 0.0f;
        float sthr = sp;
        if (sthr > k.g_slope) sthr = k.g_slope;
        float g = kappa * sthr * scaler;
        if ((e + g) > st) g = st - e;
        if (g < 0.f) g = 0.f;
        ero[i] = e;
        inci[i] = in;
        geli[i] = g;
        sums.v[0] += e;
        sums.v[1] += in;
        sums.v[2] += g;
    };
    for (int64_t r0 = ch.first; r0 < ch.end; r0 += blockDim.x) {
        if (r0 + threadIdx.x < ch.end) cell(r0 + threadIdx.x);
        sums.turn();
    }
    const double total = sums.finish();
    if (threadIdx.x < 3) atomicAdd(threadIdx.x == 0 ? &o.tot_e : threadIdx.x == 1 ? &o.tot_i : &o.tot_g, total);
    const unsigned long long fm = block_max_u64(famax, redk);
    const bool any_multi = __syncthreads_or(multi) != 0;
    if (threadIdx.x == 0) {
        atomicMax(&o.fa_max_key, fm);
        if (any_multi) sc->sed_tiled_ok = 0;
    }
}

// The per-cell arithmetic of MFDsedbud (mfd_accum.cu:222-249), rounded the same
// way wherever it is evaluated (no contraction): deposition, the stone mix
// coefficients (stone = A + B * from, clamped, when the sediment column is not
// empty; stone kept otherwise) and the new soil thickness.
struct SedLocal {
    float dep, A, B, stn;
    bool nz;
};
__device__ __forceinline__ SedLocal sed_local(float ad, float ac, float ag, float e, float ic, float g, float st0,
                                              float stone0, float ddk, float dck, float dgk) {
    SedLocal r;
    r.dep = __fadd_rn(__fadd_rn(__fmul_rn(__fadd_rn(ad, e), ddk), __fmul_rn(__fadd_rn(ac, ic), dck)),
                      __fmul_rn(__fadd_rn(ag, g), dgk));
    const float sedthick = __fadd_rn(st0, r.dep);
    r.nz = sedthick != 0.0f;
    const float old = r.nz ? __fdiv_rn(st0, sedthick) : 0.0f;
    r.B = __fsub_rn(1.0f, old);
    r.A = r.nz ? __fmul_rn(old, stone0) : stone0;
    const float toterosion = __fadd_rn(__fadd_rn(e, ic), g);
    float stn = st0;
    if (toterosion >= sedthick) stn = 0.0f;
    if (sedthick > toterosion) stn = __fsub_rn(sedthick, toterosion);
    r.stn = stn;
    return r;
}
__device__ __forceinline__ float sed_mix(float A, float B, float from) {
    float sn = __fadd_rn(A, __fmul_rn(B, from));
    if (sn < 0.01f)
        sn = 0.01f;
    else if (sn > 99.9f)
        sn = 99.9f;
    return sn;
}
__device__ __forceinline__ void sed_store(size_t g, const SedLocal& L, float sn, float* depo, float* stone,
                                          float* fines, float* soilT) {
    depo[g] = L.dep;
    if (L.nz) {
        __stcg(stone + g, sn);
        fines[g] = __fsub_rn(100.0f, sn);
    }
    soilT[g] = L.stn;
}

// Words and sources of the general sediment wave, for the steps that take it
// (MFD, or a multi-direction code found by k_erosion): cells in row 0 or column
// 0 are never processed (mfd_accum.cu:42) and masked cells never complete, so a
// donor of either kind blocks its receiver for good.  Only the stone mix waits
// on the donors: every other part of a cell (MFDsedbud, mfd_accum.cu:32-254:
// deposition from the donors' erosion, new soil thickness, mix coefficients) is
// computed here.
__global__ void k_sed_prep(const uint8_t* __restrict__ mask, const uint8_t* __restrict__ fd,
                           const float* __restrict__ prop, const float* __restrict__ ero,
                           const float* __restrict__ inci, const float* __restrict__ geli,
                           const float* __restrict__ stone, const float* __restrict__ soilT, float4* __restrict__ coef,
                           uint8_t* __restrict__ nonzero, int32_t* __restrict__ word, int32_t* ready, ModelConsts k,
                           DevScalars* sc, TileSet ts) {
    if (sc->sed_tiled_ok) return;  // the tiled path routes this step
    const int W = k.W, H = k.H;
    const size_t N = (size_t)W * H;
    const float omd = 1.0f - k.ddk, omc = 1.0f - k.dck, omg = 1.0f - k.dgk;
    for (size_t base = (size_t)blockIdx.x * blockDim.x; base < ts.span(); base += (size_t)gridDim.x * blockDim.x) {
        int x, y;
        const bool in = ts.cell(base + threadIdx.x, W, H, x, y);
        const size_t i = (size_t)y * W + x;
        bool src = false;
        if (in) {
            int32_t pend = kBlocked;
            uint32_t donors = 0, receivers = 0;
            if (mask[i] && x != 0 && y != 0) {
                pend = 0;
                const uint8_t code = fd[i];
                float ad = 0.f, ac = 0.f, ag = 0.f;
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    const int d = scan_dir(kk);
                    const int nx = x + dir_dx(d), ny = y + dir_dy(d);
                    if (nx < 0 || nx >= W || ny < 0 || ny >= H) continue;
                    const size_t n = (size_t)ny * W + nx;
                    const bool live = mask[n] && nx != 0 && ny != 0;
                    if (live) receivers |= code & dir_bit(d);
                    if (!donates(fd[n], d)) continue;
                    if (live) {
                        ++pend;
                        donors |= 1u << kk;
                    } else {
                        pend |= kBlocked;
                    }
                    const float p = prop ? __ldg(prop + 8 * n + ((d + 4) & 7)) : 1.0f;
                    ad = __fadd_rn(ad, __fmul_rn(p, __fmul_rn(__ldg(ero + n), omd)));
                    ac = __fadd_rn(ac, __fmul_rn(p, __fmul_rn(__ldg(inci + n), omc)));
                    ag = __fadd_rn(ag, __fmul_rn(p, __fmul_rn(__ldg(geli + n), omg)));
                }
                const SedLocal L = sed_local(ad, ac, ag, __ldg(ero + i), __ldg(inci + i), __ldg(geli + i), soilT[i],
                                             stone[i], k.ddk, k.dck, k.dgk);
                coef[i] = make_float4(L.A, L.B, L.dep, L.stn);
                nonzero[i] = L.nz;
                src = (pend == 0);
            }
            word[i] = wave_word(pend, donors, receivers);
        }
        wave_append(src, (int32_t)i, ready, &sc->counters[0], (int)N, &sc->err);
    }
}

// A cell of the general sediment wave: its stone mixed with the donors' updated
// stone, by the coefficients of k_sed_prep.
struct SedCell {
    const float* prop;
    const float4* coef;
    const uint8_t* nonzero;
    float* depo;
    float* stone;
    float* fines;
    float* soilT;
    DemCtx dc;
    int W;
    __device__ __forceinline__ float donor(int32_t cur, int kk, bool on) const {
        const int d = scan_dir(kk);
        const int32_t n = cur + grid_step(d, W);
        if (!on) return 0.f;
        const float p = prop ? __ldg(prop + 8 * (size_t)n + ((d + 4) & 7)) : 1.0f;
        return __fmul_rn(p, __ldcg(stone + n));
    }
    __device__ __forceinline__ void cell(int32_t cur, uint32_t donors, float part) const {
        const float4 c = __ldg(coef + cur);
        SedLocal L;
        L.A = c.x;
        L.B = c.y;
        L.dep = c.z;
        L.stn = c.w;
        L.nz = __ldg(nonzero + cur) != 0;
        float from = 0.f;
        for (uint32_t m = donors; m; m &= m - 1)
            from = __fadd_rn(from, __shfl_sync(0xffffffffu, part, __ffs(m) - 1));
        if ((threadIdx.x & 31) == 0) {
            sed_store(cur, L, L.nz ? sed_mix(L.A, L.B, from) : 0.0f, depo, stone, fines, soilT);
            if (dc.of) atomicAdd(&dc.out[dc.of[cur]].sed_done, 1);  // a batch: count per DEM
        }
    }
};

// The general sediment wave.  With gate set it runs only when the tiled path is
// off.
__global__ void __launch_bounds__(256, 4)
    k_sed_walk(const float* __restrict__ prop, const float4* __restrict__ coef, const uint8_t* __restrict__ nonzero,
               float* depo, float* stone, float* fines, float* soilT, int32_t* word, int32_t* list, ModelConsts k,
               DevScalars* sc, DemCtx dc, int gate) {
    if (gate && sc->sed_tiled_ok) return;
    const SedCell op{prop, coef, nonzero, depo, stone, fines, soilT, dc, k.W};
    int done = wave_walk(op, word, list, k.W, k.H, sc);
    done = wsum(done);
    if (!dc.of && (threadIdx.x & 31) == 0 && done) atomicAdd(&dc.out[0].sed_done, done);
}

// ---------------------------------------------------------------------------
// Tiled sediment routing for single-receiver codes, on the tiles of the tiled
// accumulation.  Deposition and soil thickness are local; only the stone mix
// carries the donors' new values downstream, through a clamp, so the coarse
// level cannot add partial sums.  Instead:
//   local : per tile, cells with no donor outside the tile upstream are
//           settled and stored; the others ("waiting" cells) are written as a
//           program per outlet, in dependency order: A, B, the sum C of the
//           settled donors and references to the waiting donors (earlier
//           slots of the same program, or cells of other tiles);
//   coarse: a wave over the outlets: an outlet whose inflows are all final
//           runs its program and stores its own new values;
//   final : per tile, the remaining waiting cells by the per-cell formula.
// Cell classes follow MFDsedbud: in-catchment cells off row 0 and column 0 are
// computed; every other in-grid donor blocks its receiver.

constexpr int kFinNz = 1;      // final-pass slot: the cell's sediment column is not empty
constexpr int kFinOutlet = 2;  // final-pass slot: an outlet (the coarse wave stored it; counted only)
constexpr int kPool = kTilePool;

// Maps of a value through a run of single-input cells: v -> clamp(a*v + b, lo, hi)
// as float4(a, b, lo, hi); lo > hi encodes the constant b (a cell whose
// sediment column is empty keeps its stone whatever its donors carry).
__device__ __forceinline__ float4 map_identity() { return make_float4(1.0f, 0.0f, -INFINITY, INFINITY); }
__device__ __forceinline__ float4 map_const(float c) { return make_float4(0.0f, c, INFINITY, -INFINITY); }
__device__ __forceinline__ float map_apply(const float4 m, float v) {
    if (m.z > m.w) return m.y;
    const float y = __fadd_rn(__fmul_rn(m.x, v), m.y);
    return y < m.z ? m.z : (y > m.w ? m.w : y);
}
// a single-input cell: from = C + v, stone = clamp(A + B * from) (or its old stone S)
__device__ __forceinline__ float4 map_cell(float A, float B, float C, bool nz, float S) {
    if (!nz) return map_const(S);
    return make_float4(B, __fadd_rn(A, __fmul_rn(B, C)), 0.01f, 99.9f);
}
// outer after inner
__device__ __forceinline__ float4 map_compose(const float4 outer, const float4 inner) {
    if (outer.z > outer.w) return outer;
    if (inner.z > inner.w) return map_const(map_apply(outer, inner.y));
    const float a1 = outer.x, b1 = outer.y;
    if (a1 == 0.0f) return map_const(map_apply(outer, 0.0f));
    const float L = __fadd_rn(__fmul_rn(a1, a1 > 0.0f ? inner.z : inner.w), b1);
    const float U = __fadd_rn(__fmul_rn(a1, a1 > 0.0f ? inner.w : inner.z), b1);
    const float lo = fmaxf(L, outer.z), hi = fminf(U, outer.w);
    if (lo > hi) return map_const(U < outer.z ? outer.z : outer.w);
    return make_float4(__fmul_rn(a1, inner.x), __fadd_rn(__fmul_rn(a1, inner.y), b1), lo, hi);
}

// Static part of a cell: deposition from all donors (in scan order), the mix
// coefficients and the new soil thickness.
__device__ __forceinline__ SedLocal sed_init(const uint8_t* s_code, const uint8_t* s_cls, int lx, int ly, int tx0,
                                            int ty0, int W, const float* __restrict__ ero,
                                            const float* __restrict__ inci, const float* __restrict__ geli,
                                            const float* __restrict__ soilT, const float* stone, const ModelConsts& k) {
    const float omd = 1.0f - k.ddk, omc = 1.0f - k.dck, omg = 1.0f - k.dgk;
    const int hc = (ly + 1) * kTH + lx + 1;
    float ad = 0.f, ac = 0.f, ag = 0.f;
#pragma unroll
    for (int kk = 0; kk < 8; ++kk) {
        const int d = scan_dir(kk);
        const int nh = hc + dir_dy(d) * kTH + dir_dx(d);
        if (!donates(s_code[nh], d)) continue;
        if (s_cls[nh] != kCellIn) continue;
        const size_t n = (size_t)(ty0 + ly + dir_dy(d)) * W + tx0 + lx + dir_dx(d);
        ad = __fadd_rn(ad, __fmul_rn(1.0f, __fmul_rn(__ldg(ero + n), omd)));
        ac = __fadd_rn(ac, __fmul_rn(1.0f, __fmul_rn(__ldg(inci + n), omc)));
        ag = __fadd_rn(ag, __fmul_rn(1.0f, __fmul_rn(__ldg(geli + n), omg)));
    }
    const size_t g = (size_t)(ty0 + ly) * W + tx0 + lx;
    return sed_local(ad, ac, ag, __ldg(ero + g), __ldg(inci + g), __ldg(geli + g), soilT[g], __ldcg(stone + g), k.ddk,
                     k.dck, k.dgk);
}

// Sediment status of a cell in s_info, above its kind: a donor in another tile, a
// sediment column that is not empty, reached (every donor upstream completes),
// and downstream of an entry.
constexpr uint8_t kSedKind = 3, kSedEntry = 4, kSedNz = 8, kSedDone = 16, kSedTaint = 32;
constexpr int kMaxNodes = 512;  // nodes of a tile: entries (124 border cells), joins of their branches, outlets

// Bound by the chains of its one-warp phases (levels, runs) on few resident tiles
// rather than by memory.  The cells settle in level order (see tile_levels) in the
// place of a queue, donors and node inputs come from masks set while the codes are
// staged, runs follow stored links, and shared arrays are reused so that five tiles
// share an SM: 1.55 -> 1.16 ms at 4096 x 4096 cells, 53 -> 43 us for a few tiles.
__global__ void __launch_bounds__(256, 5)
    k_sedt_local(const uint8_t* __restrict__ mask, const uint8_t* __restrict__ fd, const float* __restrict__ ero,
                 const float* __restrict__ inci, const float* __restrict__ geli, float* depo, float* stone,
                 float* fines, float* soilT, int32_t* __restrict__ t_dst, int32_t* __restrict__ t_pend,
                 int4* __restrict__ t_rec, float4* __restrict__ p_abc, int32_t* __restrict__ p_ref,
                 float4* __restrict__ p_map, uint8_t* __restrict__ t_stat, int4* __restrict__ f_idx,
                 float4* __restrict__ f_map, float2* __restrict__ f_ds, int32_t* __restrict__ t_fcnt, int32_t* outs,
                 ModelConsts k, DevScalars* sc, DemCtx dc, TileSet ts) {
    if (!sc->sed_tiled_ok) return;
    constexpr int C = kTile * kTile;
    __shared__ uint8_t s_code[kTH * kTH];
    __shared__ uint8_t s_cls[kTH * kTH];
    __shared__ float s_new[C + 1];  // settled stone (the old stone until then)
    // A, B, deposition and soil thickness per cell, then (between nodes) the cell's
    // map; before them, the halo's erosion terms (3 kTH x kTH floats) for the set-up
    __shared__ float4 s_cf[C];
    float* const s_ero = reinterpret_cast<float*>(s_cf);
    float* const s_inc = s_ero + kTH * kTH;
    float* const s_gel = s_inc + kTH * kTH;
    // the in-tile paths (tile_paths), then where each ends, and the outlets' slots
    __shared__ int32_t s_pd[C];
    int16_t* const s_end = reinterpret_cast<int16_t*>(s_pd);
    int16_t* const s_oslot = s_end + C;
    // levels, then a node's number of inputs (0: not a node)
    __shared__ int32_t s_h[C];
    int32_t* const s_node = s_h;
    // donors, bit k for direction scan_dir(k): in the low byte those in the tile,
    // in the high byte those in other tiles, then with the waiting ones in the tile
    __shared__ __align__(4) uint16_t s_dm[C];
    __shared__ uint8_t s_info[C];
    // the settled cells by level, then the nodes by level and each node's slot
    __shared__ uint32_t s_ent[C];
    int16_t* const s_pos = reinterpret_cast<int16_t*>(s_ent + kMaxNodes);
    // sorting bins, then the cell below in a run (-1: none), then the node at the top
    // of a cell's run
    __shared__ uint32_t s_bins[C / 2];
    int16_t* const s_up = reinterpret_cast<int16_t*>(s_bins);
    __shared__ uint32_t s_wait[kTile], s_bad[kTile];
    __shared__ int16_t s_olist[kTileEnt];
    __shared__ int32_t s_ocnt[kTileEnt];
    // per outlet, its program's nodes in the low half and their inputs in the
    // high half: the counts, and where each starts
    __shared__ int32_t s_pcnt[kTileEnt];
    __shared__ int32_t s_pstart[kTileEnt];
    __shared__ int16_t s_pfill[kTileEnt];
    __shared__ int s_no, s_nt, s_done, s_dem, s_fn;
    __shared__ int s_wcnt[9];  // per-warp counts of the outlet list and its append
    const int W = k.W, H = k.H, TW = (W + kTile - 1) / kTile;
    const int t = ts.tile(blockIdx.x);
    const int tx0 = (t % TW) * kTile, ty0 = (t / TW) * kTile;
    const int lx = threadIdx.x & 31, ly0 = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < C / 2; i += blockDim.x) {
        s_bins[i] = 0;
        reinterpret_cast<uint32_t*>(s_dm)[i] = 0;
    }
    if (threadIdx.x < kTile) s_bad[threadIdx.x] = 0;
    if (threadIdx.x < kTileEnt) {
        s_ocnt[threadIdx.x] = 0;
        s_pcnt[threadIdx.x] = 0;
    }
    if (threadIdx.x == 0) s_done = s_fn = s_nt = 0, s_dem = -1, s_new[kNoCell] = 0.f;
    __syncthreads();
    tile_stage(
        fd, [&](size_t g, int x, int y) { return mask[g] && x != 0 && y != 0 ? kCellIn : kCellBlock; }, W, H, tx0, ty0,
        s_code, s_cls, s_dm, s_bad);
    for (int j = threadIdx.x; j < kTH * kTH; j += blockDim.x) {
        const int gx = tx0 - 1 + j % kTH, gy = ty0 - 1 + j / kTH;
        float e = 0.f, i = 0.f, g = 0.f;
        if (gx >= 0 && gx < W && gy >= 0 && gy < H) {
            const size_t c = (size_t)gy * W + gx;
            e = __ldg(ero + c);
            i = __ldg(inci + c);
            g = __ldg(geli + c);
        }
        s_ero[j] = e;
        s_inc[j] = i;
        s_gel[j] = g;
    }
    __syncthreads();
    float4 cf[4];                      // the cells' coefficients until the staged terms are spent
    int dem = -1;                      // one DEM per tile
    const float omd = 1.0f - k.ddk, omc = 1.0f - k.dck, omg = 1.0f - k.dgk;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx, hc = (ly + 1) * kTH + lx + 1;
        uint32_t info = kKindEnd, dm = 0;
        int32_t pd = l;
        float snew = 0.f;
        cf[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s_cls[hc] == kCellIn) {
            const size_t g = (size_t)(ty0 + ly) * W + tx0 + lx;
            snew = __ldcg(stone + g);
            const float st0 = soilT[g];
            dm = s_dm[l];
            float ad = 0.f, ac = 0.f, ag = 0.f;
            for (uint32_t m = (dm | (dm >> 8)) & 255u; m; m &= m - 1) {
                const int d = scan_dir(__ffs(m) - 1), nh = hc + dir_dy(d) * kTH + dir_dx(d);
                ad = __fadd_rn(ad, __fmul_rn(1.0f, __fmul_rn(s_ero[nh], omd)));
                ac = __fadd_rn(ac, __fmul_rn(1.0f, __fmul_rn(s_inc[nh], omc)));
                ag = __fadd_rn(ag, __fmul_rn(1.0f, __fmul_rn(s_gel[nh], omg)));
            }
            const SedLocal in =
                sed_local(ad, ac, ag, s_ero[hc], s_inc[hc], s_gel[hc], st0, snew, k.ddk, k.dck, k.dgk);
            cf[q] = make_float4(in.A, in.B, in.dep, in.stn);
            if (dem < 0) dem = dem_at(dc, g);
            const int d = bit_dir(s_code[hc]);
            const int rlx = lx + dir_dx(d < 0 ? 0 : d), rly = ly + dir_dy(d < 0 ? 0 : d);
            if (d >= 0 && s_cls[(rly + 1) * kTH + rlx + 1] == kCellIn) {
                info = in_tile(rlx, rly) ? kKindIn : kKindOutlet;
                if (info == kKindIn) pd = (rly * kTile + rlx) | (1 << 10);
            }
            info |= (in.nz ? kSedNz : 0) | (dm >> 8 ? kSedEntry : 0);
        }
        s_pd[l] = pd;
        s_h[l] = 0;
        s_info[l] = (uint8_t)info;
        s_new[l] = snew;
        const unsigned wb = __ballot_sync(0xffffffffu, (info & kSedEntry) != 0);
        if (lx == 0) s_wait[ly] = wb;
    }
    dem = __reduce_max_sync(0xffffffffu, dem);
    if (lx == 0 && dem >= 0) atomicMax(&s_dem, dem);
    __syncthreads();  // the staged erosion terms are spent
#pragma unroll
    for (int q = 0; q < 4; ++q) s_cf[(ly0 + 8 * q) * kTile + lx] = cf[q];
    tile_paths(s_pd, s_h, s_wait, s_bad, lx, ly0);
    int key[4];
    int16_t end[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        const uint32_t info = s_info[l];
        const bool done = s_cls[(ly + 1) * kTH + lx + 1] == kCellIn && !((s_bad[ly] >> lx) & 1u);
        const bool taint = (s_wait[ly] >> lx) & 1u;
        key[q] = done && !taint ? s_h[l] : -1;
        end[q] = (int16_t)(s_pd[l] & kPtr);
        s_info[l] = (uint8_t)(info | (done ? kSedDone : 0) | (taint ? kSedTaint : 0));
        // a settled cell without donors mixes with nothing
        if (key[q] == 0 && (info & kSedNz)) s_new[l] = sed_mix(s_cf[l].x, s_cf[l].y, 0.0f);
    }
    constexpr uint8_t kWaits = kSedDone | kSedTaint;
    tile_sort(
        key,
        [&](int q) {
            const int l = (ly0 + 8 * q) * kTile + lx;
            return entry_of(l, s_dm[l] & 255u);
        },
        s_bins, C / 2, s_ent, &s_nt, lx);  // (its barriers also cover s_info and the last reads of s_pd)
#pragma unroll
    for (int q = 0; q < 4; ++q) s_end[(ly0 + 8 * q) * kTile + lx] = end[q];
    // settle what depends on this tile only: every donor is inside the tile and
    // settled; the sum in scan order (adding the 0 of kNoCell changes nothing)
    struct Cell {
        float A, B;
        uint32_t e;
        bool nz;
    };
    tile_levels(
        [&](uint32_t e) {
            const int c = entry_cell(e) & kPtr;  // (kNoCell's coefficients are not used)
            return Cell{s_cf[c].x, s_cf[c].y, e, entry_cell(e) != kNoCell && (s_info[c] & kSedNz)};
        },
        [&](const Cell& f) {
            float from = __fadd_rn(__fadd_rn(0.f, s_new[entry_d0(f.e)]), s_new[entry_d1(f.e)]);
            if (__any_sync(0xffffffffu, f.e & kMoreDonors) && (f.e & kMoreDonors)) {
                const int c = entry_cell(f.e);
                uint32_t m = s_dm[c] & 255u;
                m &= m - 1;
                for (m &= m - 1; m; m &= m - 1) from = __fadd_rn(from, s_new[c + scan_step(__ffs(m) - 1)]);
            }
            const float sn = sed_mix(f.A, f.B, from);
            if (f.nz) s_new[entry_cell(f.e)] = sn;
        },
        1, C, s_bins, s_ent);
    // the settled cells' outputs (sed_store), one coalesced pass
    bool stray = false;  // a waiting cell whose in-tile path ends inside the tile (at the DEM's outlet, say)
    int done = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        const size_t g = (size_t)(ty0 + ly) * W + tx0 + lx;
        const uint32_t info = s_info[l];
        const int e = end[q];
        const bool out = (s_info[e] & kSedKind) == kKindOutlet;
        if ((info & kWaits) == kSedDone) {
            ++done;
            depo[g] = s_cf[l].z;
            if (info & kSedNz) {
                const float sn = s_new[l];
                __stcg(stone + g, sn);
                fines[g] = __fsub_rn(100.0f, sn);
            }
            soilT[g] = s_cf[l].w;
        }
        if (info & kSedEntry) t_dst[g] = out ? (int32_t)((ty0 + e / kTile) * W + tx0 + (e & (kTile - 1))) : -1;
        stray |= (info & kWaits) == kWaits && !out;
        if (tx0 + lx < W && ty0 + ly < H) t_stat[g] = (info & kSedDone) ? ((info & kSedTaint) ? 2 : 1) : 0;
    }
    // Such a tile keeps the second wave for its waiting cells; in every other
    // tile each waiting cell's stone is a map of one program node's value,
    // stored by the final pass.
    const bool second_wave = __syncthreads_or(stray);
    list_outlets(s_info, kSedKind, s_olist, s_oslot, &s_no, s_wcnt);
    for (int i = threadIdx.x; i < C / 2; i += blockDim.x) s_bins[i] = 0;  // for the nodes
    if (threadIdx.x == 0) s_nt = 0;
    __syncthreads();
    // inflows per outlet (ring cells flowing into the tile)
    if (threadIdx.x < kRing) {
        const int h = ring_halo(threadIdx.x);
        const int d = s_cls[h] == kCellIn ? bit_dir(s_code[h]) : -1;
        if (d >= 0) {
            const int hx = h % kTH + dir_dx(d), hy = h / kTH + dir_dy(d);
            if (hx >= 1 && hx <= kTile && hy >= 1 && hy <= kTile && s_cls[hy * kTH + hx] == kCellIn) {
                const int o = s_end[(hy - 1) * kTile + hx - 1];
                if ((s_info[o] & kSedKind) == kKindOutlet) atomicAdd(&s_ocnt[s_oslot[o]], 1);
            }
        }
    }
    // program nodes: waiting cells draining to an outlet that take an inflow
    // from another tile, join two waiting branches, or are the outlet.  The
    // waiting cells between nodes pass one value on; they become the maps of
    // the nodes' inputs.
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int l = (ly0 + 8 * q) * kTile + lx;
        int node = 0;
        key[q] = -1;
        if ((s_info[l] & kWaits) == kWaits && (s_info[end[q]] & kSedKind) == kKindOutlet) {
            const uint32_t dm = s_dm[l];
            uint32_t wm = 0;
            for (uint32_t m = dm & 255u; m; m &= m - 1)
                if (s_info[l + scan_step(__ffs(m) - 1)] & kSedTaint) wm |= m & (0u - m);
            // every input of a node is waiting or comes from another tile
            if ((dm >> 8) || (wm & (wm - 1)) || (s_info[l] & kSedKind) == kKindOutlet) {
                node = __popc(dm >> 8) + __popc(wm);
                key[q] = s_h[l];
            }
            s_dm[l] = (uint16_t)(dm | (wm << 8));
        }
        s_node[l] = node;  // (a cell's level is its own thread's to replace)
        if (node) atomicAdd(&s_pcnt[s_oslot[end[q]]], 1 | (node << 16));
    }
    tile_sort(
        key, [&](int q) { return (uint32_t)((ly0 + 8 * q) * kTile + lx); }, s_bins, C / 2, s_ent, &s_nt, lx);
    // Every waiting cell between nodes: its map v -> stone from its one waiting
    // in-tile donor (in place of its own coefficients, which only nodes need
    // from here on).  Every waiting cell of a tile without a second wave also
    // takes a final-pass slot, with its deposition and soil thickness.
    const size_t fbase = (size_t)t * C;
    int fslot[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int l = (ly0 + 8 * q) * kTile + lx;
        const bool waits = (s_info[l] & kWaits) == kWaits && (s_info[end[q]] & kSedKind) == kKindOutlet;
        fslot[q] = warp_slot(waits && !second_wave, &s_fn);
        if (!waits) continue;
        if (fslot[q] >= 0) f_ds[fbase + fslot[q]] = make_float2(s_cf[l].z, s_cf[l].w);
        if (s_node[l]) continue;
        float Cc = 0.f;
        const uint32_t dm = s_dm[l];
        for (uint32_t m = dm & ~(dm >> 8) & 255u; m; m &= m - 1)
            Cc = __fadd_rn(Cc, __fmul_rn(1.0f, s_new[l + scan_step(__ffs(m) - 1)]));
        s_cf[l] = map_cell(s_cf[l].x, s_cf[l].y, Cc, (s_info[l] & kSedNz) != 0, s_new[l]);
    }
    // the cell below in the same run: waiting and no node
    int16_t* const s_down = s_up;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        int c = -1;
        if ((s_info[l] & (kWaits | kSedKind)) == (kWaits | kKindIn)) {
            const int d = bit_dir(s_code[(ly + 1) * kTH + lx + 1]);
            c = l + dir_dy(d) * kTile + dir_dx(d);
            if ((s_info[c] & kWaits) != kWaits || s_node[c]) c = -1;
        }
        s_down[l] = (int16_t)c;
    }
    const int no = s_no, nt = s_nt;
    if (threadIdx.x < 32) outlet_starts(s_pcnt, s_pstart, no);
    __syncthreads();
    // The maps of the cells between nodes, composed down each run from the node
    // at its top: afterwards s_up of such a cell is that node and its map takes
    // the node's value to its own stone.  One walk per node; no two walks
    // share a cell (a cell between nodes has one waiting donor).
    for (int i = threadIdx.x; i < nt; i += blockDim.x) {
        const int l = (int)s_ent[i];
        float4 F = map_identity();
        for (int c = s_down[l], guard = 0; c >= 0 && guard < C; ++guard) {
            const int below = s_down[c];
            F = map_compose(s_cf[c], F);
            s_cf[c] = F;
            s_up[c] = (int16_t)l;
            c = below;
        }
    }
    const int j = threadIdx.x;
    const int pcnt = j < no ? s_pcnt[j] : 0, pstart = j < no ? s_pstart[j] : 0;
    int32_t* const s_ifill = s_pcnt;  // where the program's next node's inputs go (the counts are kept above)
    if (j < no) {
        s_ifill[j] = pstart >> 16;
        s_pfill[j] = (int16_t)(pstart & 0xffff);
    }
    __syncthreads();
    // node slots: grouped by outlet, in level order
    if (threadIdx.x < 32) {
        const unsigned below = (1u << lx) - 1u;
        for (int base = 0; base < nt; base += 32) {
            const int i = base + lx;
            int slot = -1, c = 0;
            if (i < nt) {
                c = (int)s_ent[i];
                slot = s_oslot[s_end[c]];
            }
            const unsigned peers = __match_any_sync(0xffffffffu, slot);
            const int fill = slot >= 0 ? s_pfill[slot] : 0;
            __syncwarp();
            if (slot >= 0) {
                s_pos[c] = (int16_t)(fill + __popc(peers & below));
                if ((peers & below) == 0) s_pfill[slot] = (int16_t)(fill + __popc(peers));
            }
            __syncwarp();
        }
    }
    __syncthreads();
    const size_t nbase = (size_t)t * C;
    const size_t pool = (size_t)t * kPool;
    for (int i = threadIdx.x; i < nt; i += blockDim.x) {
        const int l = (int)s_ent[i], ly = l / kTile, x = l & (kTile - 1);
        const int pos = s_pos[l], slot = s_oslot[s_end[l]];
        const int first = s_pstart[slot] & 0xffff;
        const int start = atomicAdd(&s_ifill[slot], s_node[l]);
        if (start + s_node[l] > kPool) {
            raise_error(&sc->err, ErrFlags::kCapacity);
            continue;
        }
        const uint32_t dm = s_dm[l];
        float Cc = 0.f;
        int m = 0;
#pragma unroll 1
        for (uint32_t b = (dm | (dm >> 8)) & 255u; b; b &= b - 1) {
            const int kk = __ffs(b) - 1;
            int cur = l + scan_step(kk);
            if (!((dm >> (8 + kk)) & 1u)) {  // settled in the tile
                Cc = __fadd_rn(Cc, __fmul_rn(1.0f, s_new[cur]));
                continue;
            }
            int32_t ref;
            float4 H = map_identity();
            if (!((dm >> kk) & 1u)) {
                const int d = scan_dir(kk);
                ref = (ty0 + ly + dir_dy(d)) * W + tx0 + x + dir_dx(d);
            } else {
                // the node that feeds this input, through the single-input cells in between
                if (!s_node[cur]) {
                    H = s_cf[cur];
                    cur = s_up[cur];
                }
                ref = -(s_pos[cur] - first + 1);
            }
            p_ref[pool + start + m] = ref;
            p_map[pool + start + m] = H;
            ++m;
        }
        p_abc[nbase + pos] = make_float4(s_cf[l].x, s_cf[l].y, Cc,
                                         __int_as_float(start | (m << 11) | (s_info[l] & kSedNz ? 1 << 15 : 0)));
    }
    // the final pass's slots: a node reads its own value, a cell between nodes
    // maps the value of the node at the top of its chain
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (fslot[q] < 0) continue;
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        const bool node = s_node[l] != 0;
        const int src_node = node ? l : s_up[l];
        const int e = end[q];
        const uint32_t info = s_info[l];
        f_idx[fbase + fslot[q]] = make_int4((ty0 + ly) * W + tx0 + lx, (int)(fbase + s_pos[src_node]),
                                            (ty0 + e / kTile) * W + tx0 + (e & (kTile - 1)),
                                            (info & kSedNz ? kFinNz : 0) |
                                                ((info & kSedKind) == kKindOutlet ? kFinOutlet : 0));
        f_map[fbase + fslot[q]] = node ? map_identity() : s_cf[l];
    }
    if (threadIdx.x == 0) t_fcnt[t] = second_wave ? -1 : s_fn;
    int32_t og = 0;
    if (j < no) {
        const int o = s_olist[j];
        const int32_t opend = ((s_info[o] & kSedDone) ? 0 : kBlocked) + s_ocnt[j];
        og = (ty0 + o / kTile) * W + tx0 + (o & (kTile - 1));
        // (the coefficients of a waiting outlet, a node, are still in place)
        t_rec[og] = make_int4((pstart << 16) | (pcnt & 0xffff), (pstart & ~0xffff) | (pcnt >> 16),
                              __float_as_int(s_cf[o].z), __float_as_int(s_cf[o].w));
        t_pend[og] = opend;
        if (opend == 0) og = ~og;  // settled here: a source of the coarse wave
    }
    block_append(j < no, og, outs, &sc->tile_src, W * H, &sc->err, s_wcnt);
    done = wsum(done);
    if (lx == 0 && done) atomicAdd(&s_done, done);
    __syncthreads();
    if (threadIdx.x == 0 && s_done && s_dem >= 0) atomicAdd(&dc.out[s_dem].sed_done, s_done);
}

// The coarse sediment wave over the tile outlets.  The sources (settled in
// their tiles) release their receivers in one parallel pass, which also links
// every outlet to the one it drains to; then each warp takes a released outlet,
// runs its program and walks downstream for as long as its outlet is the last
// inflow to arrive (an outlet has one receiver, so each is reached once).
//
// Bound by the longest chain of tile crossings (about 240 at 4096 x 4096
// cells, with 9 dependent nodes of a program each), so by the latency of one
// crossing.  A program is static but for the values from other tiles: it is
// copied to shared memory (cp.async) while the outlet above it is computed, and
// the records further down are read one outlet earlier still.  Each lane then
// holds one node with its first inputs in registers; a step computes every node
// whose input nodes are done, and the values pass between lanes by shuffles.
// Reading coefficients, references and maps level by level took 2150 cycles a
// level, 2.3 ms in all; a quarter of the outlets on the longest chains have more
// than 64 nodes, and such programs run from memory took 70000 cycles each.  The
// outlet's other outputs are stored behind the release.
constexpr int kGatherNodes = 64;   // larger programs are gathered 32 nodes at a time, when their turn comes
constexpr int kGatherInputs = 88;  //   (two buffers for each of the block's warps fit 48 KB)
constexpr int kGatherTurns = (kGatherInputs + 31) / 32;
constexpr int kHeldInputs = 3;     // inputs of a node held in registers (the others stay in shared memory)

struct SedProg {
    float4 abc[kGatherNodes];    // the nodes' coefficients
    float4 map[kGatherInputs];   // their inputs' maps; once the outlet is ready, the mapped value (.x) of an
    int32_t ref[kGatherInputs];  //   input from another tile, its ref 0; below 0 the feeding node
};

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__global__ void __launch_bounds__(256, 4)
    k_sedt_coarse(const uint8_t* __restrict__ fd, const int4* __restrict__ t_rec, int32_t* t_nxt,
                  const int32_t* __restrict__ t_dst, const float4* __restrict__ p_abc,
                  const int32_t* __restrict__ p_ref, const float4* __restrict__ p_map, float* p_val, float* depo,
                  float* stone, float* fines, float* soilT, int32_t* t_pend, const int32_t* __restrict__ outs,
                  int32_t* ready, ModelConsts k, DevScalars* sc) {
    if (!sc->sed_tiled_ok) return;
    cg::grid_group grid = cg::this_grid();
    __shared__ SedProg s_prog[8][2];
    __shared__ float s_vals[8][kGatherNodes];
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
            const int d = bit_dir(fd[o]);  // the receiver is a routed cell of another tile
            nx = t_dst[o + dir_dy(d) * W + dir_dx(d)];
            t_nxt[o] = nx;
            if (e < 0 && nx >= 0) rdy = atomicSub(t_pend + nx, 1) == 1;
        }
        block_append(rdy, nx, ready, n_ready, (int)N, &sc->err, s_cnt);
    }
    grid.sync();
    const int nin = *((volatile int32_t*)n_ready);
    const int lane = threadIdx.x & 31, wq = threadIdx.x >> 5;
    float* const vals = s_vals[wq];
    auto tile_of = [&](int32_t o) {
        const int y = o / W, x = o - y * W;
        return (y / kTile) * TW + x / kTile;
    };
    auto held = [](int4 r) { return (r.x & 0xffff) <= kGatherNodes && (r.y & 0xffff) <= kGatherInputs; };
    // starts copying the program of an outlet of tile t
    auto fetch = [&](SedProg& b, int t, int4 r) {
        const int cnt = r.x & 0xffff, ni = r.y & 0xffff;
        const float4* abc = p_abc + (size_t)t * kTile * kTile + (r.x >> 16);
        const size_t in0 = (size_t)t * kPool + (r.y >> 16);
        if (!held(r)) {  // a line of 128 bytes per lane
#pragma unroll 1
            for (int j = 8 * lane; j < cnt; j += 256) prefetch_l2(abc + j);
#pragma unroll 1
            for (int j = 8 * lane; j < ni; j += 256) {
                prefetch_l2(p_map + in0 + j);
                prefetch_l2(p_ref + in0 + j);
            }
            return;
        }
#pragma unroll 1
        for (int j = lane; j < cnt; j += 32) cp_async16(&b.abc[j], abc + j);
#pragma unroll 1
        for (int j = lane; j < ni; j += 32) {
            cp_async16(&b.map[j], p_map + in0 + j);
            cp_async4(&b.ref[j], p_ref + in0 + j);
        }
    };
    for (size_t guard = 0; guard <= N; ++guard) {
        int32_t o = -1;
        if (lane == 0) {
            const int it = atomicAdd(head, 1);
            if (it < nin) o = __ldcg(ready + it);
        }
        o = __shfl_sync(0xffffffffu, o, 0);
        if (o < 0) break;
        int4 r = __ldg(t_rec + o);
        int32_t d = __ldcg(t_nxt + o);
        int buf = 0, t = tile_of(o);
        fetch(s_prog[wq][0], t, r);
        int4 rd = make_int4(0, 0, 0, 0);  // the record of d and the outlet d drains to
        int32_t e = -1;
        if (d >= 0) {
            rd = __ldg(t_rec + d);
            e = __ldcg(t_nxt + d);
        }
        for (size_t chain = 0; o >= 0 && chain <= N; ++chain) {
            SedProg& pr = s_prog[wq][buf];
            const int cnt = r.x & 0xffff, ni = r.y & 0xffff;
            const size_t nbase = (size_t)t * kTile * kTile + (r.x >> 16);
            const size_t pool = (size_t)t * kPool;
            const int in0 = r.y >> 16;
            const bool gathered = held(r);
            cp_async_wait();
            __syncwarp();
            // the values from other tiles, final now that the outlet is ready
            if (gathered)
#pragma unroll 1
                for (int j = lane; j < ni; j += 32) {
                    const int32_t ref = pr.ref[j];
                    if (ref < 0) continue;
                    pr.map[j].x = map_apply(pr.map[j], __ldcg(stone + ref));
                    pr.ref[j] = 0;
                }
            // ahead of their use: the next outlet's program, the record after it
            int4 re = make_int4(0, 0, 0, 0);
            int32_t f = -1;
            if (d >= 0) {
                t = tile_of(d);
                fetch(s_prog[wq][buf ^ 1], t, rd);
                if (e >= 0) {
                    re = __ldg(t_rec + e);
                    f = __ldcg(t_nxt + e);
                }
            }
            __syncwarp();
            float sn = 0.f;  // the outlet's new stone: the last node of its program
            bool snz = false;
#pragma unroll 1
            for (int i = 0, m; i < cnt; i += m) {
                // The nodes i .. i + m - 1, one per lane.  An input from a node
                // among these is its lane's value through the map (bits of
                // need); one whose value is known becomes a constant map of
                // the lane's own value, still 0.
                const int j = i + lane;
                m = min(32, cnt - i);
                float4 c = make_float4(0.f, 0.f, 0.f, 0.f);
                if (lane < m) c = gathered ? pr.abc[j] : __ldg(p_abc + nbase + j);
                const int meta = __float_as_int(c.w);
                int nj = lane < m ? (meta >> 11) & 15 : 0;
                const bool nz = (meta >> 15) & 1;
                int b0 = (meta & 2047) - in0;
                if (!gathered) {
                    int incl = nj;
#pragma unroll
                    for (int d2 = 1; d2 < 32; d2 <<= 1) {
                        const int w = __shfl_up_sync(0xffffffffu, incl, d2);
                        if (lane >= d2) incl += w;
                    }
                    // as many nodes as have room for their inputs (at most 8 each)
                    m = min(m, __popc(__ballot_sync(0xffffffffu, incl <= kGatherInputs)));
                    b0 = incl - nj;
                    if (lane >= m) nj = 0;
                    // their places in the pool, then every input by its own lane
#pragma unroll 1
                    for (int q = 0; q < nj; ++q) pr.ref[b0 + q] = (meta & 2047) + q;
                    const int total = __shfl_sync(0xffffffffu, incl, m - 1);
                    __syncwarp();
                    int32_t ref[kGatherTurns];
                    float4 g[kGatherTurns];
#pragma unroll
                    for (int q = 0; q < kGatherTurns; ++q) {
                        const int at = lane + 32 * q;
                        if (at >= total) continue;
                        const size_t from = pool + pr.ref[at];
                        ref[q] = __ldg(p_ref + from);
                        g[q] = __ldg(p_map + from);
                    }
#pragma unroll
                    for (int q = 0; q < kGatherTurns; ++q) {
                        const int at = lane + 32 * q;
                        if (at >= total) continue;
                        if (ref[q] >= 0) g[q].x = map_apply(g[q], __ldcg(stone + ref[q]));
                        pr.map[at] = g[q];
                        pr.ref[at] = ref[q] >= 0 ? 0 : ref[q];
                    }
                    __syncwarp();
                }
                uint32_t need = 0;
                auto input = [&](int q, float4& f, int& src) {
                    const bool mine = q < nj;
                    const float4 g = pr.map[mine ? b0 + q : 0];
                    const int32_t ref = mine ? pr.ref[b0 + q] : 0;
                    bool known = ref == 0 || g.z > g.w;  // another tile's value, mapped; a constant map
                    float val = !mine ? 0.f : (ref == 0 ? g.x : g.y);
                    if (!known && -ref - 1 < i) {  // a node of an earlier turn
                        val = map_apply(g, gathered ? vals[-ref - 1] : __ldcg(p_val + nbase - ref - 1));
                        known = true;
                    }
                    f = make_float4(known ? 0.f : g.x, known ? val : g.y, known ? -INFINITY : g.z,
                                    known ? INFINITY : g.w);
                    src = known ? lane : -ref - 1 - i;
                    need |= known ? 0u : 1u << src;
                };
                auto through = [](const float4 f, float x) {  // map_apply of a map that is no constant
                    const float y = __fadd_rn(__fmul_rn(f.x, x), f.y);
                    return y < f.z ? f.z : (y > f.w ? f.w : y);
                };
                float4 f[kHeldInputs];
                int src[kHeldInputs];
#pragma unroll
                for (int q = 0; q < kHeldInputs; ++q) input(q, f[q], src[q]);
                const int most = __reduce_max_sync(0xffffffffu, nj);
#pragma unroll 1
                for (int q = kHeldInputs; q < most; ++q) {  // read again in each step
                    float4 f2;
                    int s2;
                    input(q, f2, s2);
                }
                uint32_t todo = m == 32 ? 0xffffffffu : (1u << m) - 1u;
                float v = 0.f;
#pragma unroll 1
                for (int step = 0; todo && step < 32; ++step) {
                    const bool act = ((todo >> lane) & 1u) && !(need & todo);
                    float from = c.z;
#pragma unroll
                    for (int q = 0; q < kHeldInputs; ++q)
                        from = __fadd_rn(from, through(f[q], __shfl_sync(0xffffffffu, v, src[q])));
#pragma unroll 1
                    for (int q = kHeldInputs; q < most; ++q) {
                        float4 f2;
                        int s2;
                        input(q, f2, s2);
                        from = __fadd_rn(from, through(f2, __shfl_sync(0xffffffffu, v, s2)));
                    }
                    const float sn2 = sed_mix(c.x, c.y, from);
                    v = act ? (nz ? sn2 : c.x) : v;
                    todo &= ~__ballot_sync(0xffffffffu, act);
                }
                if (lane < m) {
                    if (gathered)
                        vals[j] = v;
                    else
                        __stcg(p_val + nbase + j, v);
                }
                sn = __shfl_sync(0xffffffffu, v, m - 1);
                snz = __shfl_sync(0xffffffffu, (int)nz, m - 1) != 0;
                __syncwarp();
            }
            int32_t next = -1;
            if (lane == 0) {
                if (snz) __stcg(stone + o, sn);
                if (d >= 0 && dec_acq_rel(t_pend + d) == 1) next = d;
                depo[o] = __int_as_float(r.z);
                if (snz) fines[o] = __fsub_rn(100.0f, sn);
                soilT[o] = __int_as_float(r.w);
            }
            // the final pass maps every node's value onto its chain
            if (gathered)
#pragma unroll 1
                for (int j = lane; j < cnt; j += 32) p_val[nbase + j] = vals[j];
            o = __shfl_sync(0xffffffffu, next, 0);
            r = rd;
            d = e;
            rd = re;
            e = f;
            buf ^= 1;
        }
        cp_async_wait();  // the buffers are refilled for the next outlet
        __syncwarp();
    }
}

__global__ void __launch_bounds__(256, 6)
    k_sedt_final(const uint8_t* __restrict__ mask, const uint8_t* __restrict__ fd, const float* __restrict__ ero,
                 const float* __restrict__ inci, const float* __restrict__ geli, float* depo, float* stone,
                 float* fines, float* soilT, const int32_t* __restrict__ t_pend, const uint8_t* __restrict__ t_stat,
                 const int4* __restrict__ f_idx, const float4* __restrict__ f_map, const float2* __restrict__ f_ds,
                 const int32_t* __restrict__ t_fcnt, const float* __restrict__ p_val, ModelConsts k, DevScalars* sc,
                 DemCtx dc, TileSet ts) {
    if (!sc->sed_tiled_ok) return;
    const int t = ts.tile(blockIdx.x);
    const int nf = t_fcnt[t];
    const size_t fbase = (size_t)t * kTile * kTile;
    bool stalled = false;  // an outlet whose program never ran (a donor upstream never completes)
    // a thread's slots (a tile has at most kTile * kTile), kept for both passes
    int4 ev[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = (int)threadIdx.x + 256 * q;
        ev[q] = make_int4(0, 0, 0, kFinOutlet);
        if (nf >= 0 && i < nf) {
            ev[q] = f_idx[fbase + i];
            stalled |= t_pend[ev[q].z] != 0;
        }
    }
    if (nf >= 0 && !__syncthreads_or(stalled)) {
        // every waiting cell is a program node or lies on a chain below one:
        // its stone is the map of that node's value
        int done = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = (int)threadIdx.x + 256 * q;
            if (i >= nf) continue;
            const int4 e = ev[q];
            ++done;
            if (e.w & kFinOutlet) continue;
            const float2 ds = f_ds[fbase + i];
            const bool nz = (e.w & kFinNz) != 0;
            const float4 mp = nz ? f_map[fbase + i] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float pv = nz ? __ldcg(p_val + e.y) : 0.f;
            depo[e.x] = ds.x;
            soilT[e.x] = ds.y;
            if (nz) {
                const float sn = map_apply(mp, pv);
                __stcg(stone + e.x, sn);
                fines[e.x] = __fsub_rn(100.0f, sn);
            }
        }
        if (nf > 0) {
            done = wsum(done);
            const int dem = dem_at(dc, (size_t)f_idx[fbase].x);
            if ((threadIdx.x & 31) == 0 && done && dem >= 0) atomicAdd(&dc.out[dem].sed_done, done);
        }
        return;
    }
    // The second wave: the waiting cells by the per-cell formula, in level order,
    // with the donors in other tiles at their final values.  The levels count
    // waiting cells only; a cell below an inflow that never completes stays as it is,
    // and an outlet keeps the coarse wave's value.
    __shared__ uint8_t s_code[kTH * kTH];
    __shared__ uint8_t s_cls[kTH * kTH];
    __shared__ float s_hval[kRing];   // the ring's stone
    __shared__ uint8_t s_hok[kRing];  //   and whether it is final
    __shared__ int32_t s_pd[kTile * kTile];
    __shared__ int32_t s_h[kTile * kTile];
    __shared__ float s_new[kTile * kTile + 1];
    __shared__ float2 s_ab[kTile * kTile];  // a waiting cell's stone-mix coefficients
    __shared__ __align__(4) uint16_t s_dm[kTile * kTile];
    __shared__ uint32_t s_ent[kTile * kTile];
    __shared__ uint32_t s_bins[kTile * kTile / 2];
    __shared__ uint32_t s_wait[kTile], s_bad[kTile], s_nz[kTile];  // rows of cells
    __shared__ int s_done, s_dem, s_qn;
    const int W = k.W, H = k.H, TW = (W + kTile - 1) / kTile;
    const int tx0 = (t % TW) * kTile, ty0 = (t / TW) * kTile;
    const int lx = threadIdx.x & 31, ly0 = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kTile * kTile / 2; i += blockDim.x) {
        s_bins[i] = 0;
        reinterpret_cast<uint32_t*>(s_dm)[i] = 0;
    }
    if (threadIdx.x < kTile) s_wait[threadIdx.x] = s_bad[threadIdx.x] = 0;
    if (threadIdx.x == 0) s_done = s_qn = 0, s_dem = -1, s_new[kNoCell] = 0.f;
    __syncthreads();
    tile_stage(
        fd, [&](size_t g, int x, int y) { return mask[g] && x != 0 && y != 0 ? kCellIn : kCellBlock; }, W, H, tx0, ty0,
        s_code, s_cls, s_dm, s_bad);
    if (threadIdx.x < kRing) {
        const int h = ring_halo(threadIdx.x);
        const int gx = tx0 - 1 + h % kTH, gy = ty0 - 1 + h / kTH;
        bool ok = false;
        float v = 0.f;
        if (gx >= 0 && gx < W && gy >= 0 && gy < H) {
            const size_t g = (size_t)gy * W + gx;
            ok = t_pend[g] == 0;
            v = __ldcg(stone + g);
        }
        s_hok[threadIdx.x] = ok;
        s_hval[threadIdx.x] = v;
    }
    __syncthreads();
    // the neighbour in direction scan_dir(k) of cell l when it lies in another tile
    auto ring_of = [&](int l, int kk) {
        const int d = scan_dir(kk);
        return ring_index((l & (kTile - 1)) + 1 + dir_dx(d), l / kTile + 1 + dir_dy(d));
    };
    auto sum = [&](int l) {  // the donors' stone in scan order
        const uint32_t dm = s_dm[l];
        float from = 0.f;
        for (uint32_t m = (dm | (dm >> 8)) & 255u; m; m &= m - 1) {
            const int kk = __ffs(m) - 1;
            from = __fadd_rn(from, __fmul_rn(1.0f, (dm >> kk) & 1u ? s_new[l + scan_step(kk)] : s_hval[ring_of(l, kk)]));
        }
        return from;
    };
    int done = 0, dem = -1;  // one DEM per tile
    bool waits[4];
    float dep[4], stn[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx, hc = (ly + 1) * kTH + lx + 1;
        int32_t pd = l;
        float v = 0.f;
        bool nz = false;
        waits[q] = false;
        dep[q] = stn[q] = 0.f;
        if (s_cls[hc] == kCellIn) {
            const size_t g = (size_t)(ty0 + ly) * W + tx0 + lx;
            const int d = bit_dir(s_code[hc]);
            const int rlx = lx + dir_dx(d < 0 ? 0 : d), rly = ly + dir_dy(d < 0 ? 0 : d);
            const bool rin = d >= 0 && s_cls[(rly + 1) * kTH + rlx + 1] == kCellIn;
            const bool outlet = rin && !in_tile(rlx, rly);
            const bool st2 = t_stat[g] == 2;
            if (outlet && st2 && t_pend[g] == 0) ++done;
            v = __ldcg(stone + g);
            if (dem < 0) dem = dem_at(dc, g);
            if (st2 && !outlet) {
                waits[q] = true;
                if (rin) pd = (rly * kTile + rlx) | (1 << 10);
                const SedLocal in = sed_init(s_code, s_cls, lx, ly, tx0, ty0, W, ero, inci, geli, soilT, stone, k);
                s_ab[l] = make_float2(in.A, in.B);
                dep[q] = in.dep;
                stn[q] = in.stn;
                nz = in.nz;
                for (uint32_t m = s_dm[l] >> 8; m; m &= m - 1)
                    if (!s_hok[ring_of(l, __ffs(m) - 1)]) atomicOr(&s_bad[ly], 1u << lx);
            }
        }
        const unsigned nb = __ballot_sync(0xffffffffu, nz);
        if (lx == 0) s_nz[ly] = nb;
        s_pd[l] = pd;
        s_h[l] = 0;
        s_new[l] = v;
    }
    dem = __reduce_max_sync(0xffffffffu, dem);
    if (lx == 0 && dem >= 0) atomicMax(&s_dem, dem);
    __syncthreads();
    tile_paths(s_pd, s_h, s_wait, s_bad, lx, ly0);
    int level[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        level[q] = waits[q] && !((s_bad[ly] >> lx) & 1u) ? s_h[l] : -1;
        // no waiting donor in the tile (the others' stone is not written here)
        if (level[q] == 0 && ((s_nz[ly] >> lx) & 1u)) s_new[l] = sed_mix(s_ab[l].x, s_ab[l].y, sum(l));
    }
    tile_sort(
        level,
        [&](int q) {
            const int l = (ly0 + 8 * q) * kTile + lx;
            return entry_of(l, s_dm[l] & 255u) | (s_dm[l] >> 8 ? kMoreDonors : 0u);
        },
        s_bins, kTile * kTile / 2, s_ent, &s_qn, lx);
    struct Cell {
        float2 ab;
        uint32_t e;
        bool nz;
    };
    tile_levels(
        [&](uint32_t e) {
            const int c = entry_cell(e) & kPtr;
            return Cell{s_ab[c], e, entry_cell(e) != kNoCell && ((s_nz[c / kTile] >> (c & (kTile - 1))) & 1u)};
        },
        [&](const Cell& f) {
            float from = __fadd_rn(__fadd_rn(0.f, s_new[entry_d0(f.e)]), s_new[entry_d1(f.e)]);
            if (f.e & kMoreDonors) from = sum(entry_cell(f.e));
            const float sn = sed_mix(f.ab.x, f.ab.y, from);
            if (f.nz) s_new[entry_cell(f.e)] = sn;
        },
        1, kTile * kTile, s_bins, s_ent);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (level[q] < 0) continue;
        const int ly = ly0 + 8 * q, l = ly * kTile + lx;
        SedLocal L;
        L.dep = dep[q];
        L.stn = stn[q];
        L.nz = (s_nz[ly] >> lx) & 1u;
        sed_store((size_t)(ty0 + ly) * W + tx0 + lx, L, s_new[l], depo, stone, fines, soilT);
        ++done;
    }
    done = wsum(done);
    if ((threadIdx.x & 31) == 0 && done) atomicAdd(&s_done, done);
    __syncthreads();
    if (threadIdx.x == 0 && s_done && s_dem >= 0) atomicAdd(&dc.out[s_dem].sed_done, s_done);
}

__device__ __forceinline__ float dreybrodt(const float* tab, float T) {
    float u = (T - kTabT0) / kTabStep;
    u = fminf(fmaxf(u, 0.0f), (float)(kTabN - 2));
    const int j = (int)u;
    const float f = u - (float)j;
    return tab[j] + f * (tab[j + 1] - tab[j]);
}

// Bound by the instructions issued and by the FP64 pipe: three fp64 sums a cell,
// which takes two lanes a clock (the conversions and the test against the base
// level kept it busy as well: 441 -> 418 us at 4096 x 4096 cells without them).
// Six blocks per SM: a few spilled registers, measured faster than four.
__global__ void __launch_bounds__(256, 6)
    k_final(double* __restrict__ z, const double* __restrict__ z_init, const uint8_t* __restrict__ mask,
            const float2* __restrict__ fa, const float* __restrict__ ero, const float* __restrict__ inci,
            const float* __restrict__ geli, const float* __restrict__ depo, float* __restrict__ soilT,
            float* __restrict__ stone, float* __restrict__ fines, float* __restrict__ soilM,
            float* __restrict__ soilB, float* __restrict__ nut, float* __restrict__ totB, float* __restrict__ dz_out,
            float* __restrict__ wc_out, float* __restrict__ wp_out, const float* __restrict__ tab,
            const int32_t* __restrict__ chunk_start, ModelConsts k, DemCtx dc) {
    __shared__ double red[8][4];
    const int W = k.W;
    const Chunk ch = chunk_of(chunk_start, dc);
    const DemIn& c = dc.in[ch.d];
    DemOut& o = dc.out[ch.d];
    const int outlet = o.outlet;
    const int outlet_clim = o.outlet_clim;  // the cell whose climate elevation is outlet_z_clim
    const double outlet_z = o.outlet_z_clim;
    const double base = o.base_level;
    const uint64_t base_key = dkey(base);
    const float rain0 = (float)c.rain, rinc = (float)c.rain_inc;
    const float dtemp_scalar = (float)(c.temp - c.temp0);
    BlockSums<4> sums(red);
    auto cell = [&](int64_t ri) {
        int x, y;
        const size_t i = region_cell(c, ri, W, &x, &y);
        // every input of the cell in one batch of loads, ahead of the mask test
        // and the arithmetic (the region's cells outside the catchment are few)
        const uint8_t mk = mask[i];
        const float dp = depo[i];
        const float e = ero[i], ic = inci[i], gl = geli[i];
        const double zold = z[i], z0 = z_init[i];
        const float2 f2 = fa[i];
        const float st0 = soilT[i], sn0 = stone[i], sm0 = soilM[i], tb = totB[i], sb0 = soilB[i];
        sums.v[3] += dp;
        if (!mk) {
            totB[i] = 0.0f;  // grow_vegetation (updates.cu:102-105)
            if (dz_out) {
                dz_out[i] = 0.f;
                wc_out[i] = 0.f;
                wp_out[i] = 0.f;
            }
            return;
        }
        const float dz = dp - e - ic - gl;  // surface_change (eroincidep.cu:404)
        const double zc = c.from_current_dem ? (((int)i == outlet_clim) ? outlet_z : zold) : z0;
        float zch, zcl;
        dsplit(zc, zch, zcl);
        const float T = (float)c.temp - ((zch - (float)kMinHeight) + zcl) * 0.0065f;
        const float rain = rain0 + (float)(y - c.y0) * rinc;
        const float fav = f2.x + f2.y;
        // weathering type 1 (eroincidep.cu:220-327)
        const float PE = 1.44f * (T + 6.0f) * (T + 6.0f);
        const float surface_flow = fav * 1000.0f;
        const float evap_trans = (rain + surface_flow <= PE) ? rain + surface_flow : rain + surface_flow - PE;
        float st = st0;
        const float lpco2 = (st > 0.1f ? -2.5f : -3.5f) + ((T - 15.0f) / 10.0f);
        const float Ca2eq = exp10f((lpco2 + dreybrodt(tab, T)) * (1.0f / 3.0f));
        float wC = 0.0148148148f * Ca2eq * (surface_flow / k.rescale_weather);
        if (wC <= 0.0f) wC = 0.0f;
        if (wC > 0.001f) wC = 0.001f;
        const float wP = 7.7e-5f * expf(-2.3f * st);
        st = st + wC * 0.02f + wP;
        float sn = sn0, sm = sm0;
        if (st <= 0.0f) {
            st = 0.0f;
            sn = 0.0f;
            fines[i] = 0.0f;
            sm = 0.02f;
        } else {
            if (wP > 0.f)
                sn += sn * (tanhf(e / st) * -tanhf(wC / wP));
            else
                sn += sn * tanhf(e / st);
            if (sn < 0.01f)
                sn = 0.01f;
            else if (sn > 99.9f)
                sn = 99.9f;
            fines[i] = 100.0f - sn;
            sm -= (1.e-3f * evap_trans / st);
            if (sm < 0.02f)
                sm = 0.02f;
            else if (sm > 0.5f)
                sm = 0.5f;
        }
        soilT[i] = st;
        stone[i] = sn;
        soilM[i] = sm;
        // Update_Surface (updates.cu:23-46); the outlet takes base - 1.2e-4 (:165,174)
        double zn = zold;
        if ((int)i == outlet) {
            zn = base - 0.00012;
        } else {
            // the sums are fp64, the conversions and the test take the integer pipe
            zn = ((zn + dwiden(dz)) - dwiden(wC)) - dwiden(wP);
            const uint64_t kn = dkey(zn);
            if (kn != 0 && kn <= base_key) zn = base + 0.01;  // (NaN: no order)
        }
        z[i] = zn;
        // update_nutrient_content (updates.cu:48-76)
        float nu;
        const float leaf_fall = tb / (72.8f * logf(tb + 1.4f));
        const float decomposition = sb0 * expf(0.12f * T - 5.75f);
        const float sb = sb0 + leaf_fall - decomposition;
        soilB[i] = sb;
        if (st == 0.0f && sb > 0.0f)
            nu = 100.0f;
        else if (st == 0.0f)
            nu = 0.0f;
        else
            nu = (sb / (1300.0f * st)) * 100.0f;
        if (nu > 100.f) nu = 100.f;
        nut[i] = nu;
        // grow_vegetation (updates.cu:78-139): delta_temp against the initial
        // climate grids (copytolastclimate is disabled, lem.cpp:102).  During the
        // run-in both grids come from the same DEM and scalars, so it is 0.
        float dT = 0.0f;
        if (c.from_current_dem) {
            float h1, l1, h0, l0;
            dsplit(zc, h1, l1);
            dsplit(z0, h0, l0);
            dT = dtemp_scalar - ((h1 - h0) + (l1 - l0)) * 0.0065f;
            if (fabsf(dT) < 1.0e-3f) {  // decide the branch with the reference's fp64 arithmetic
                const double t1 = c.temp - ((zc - kMinHeight) * 0.0065);
                const double t0 = c.temp0 - ((z0 - kMinHeight) * 0.0065);
                const double dd = t1 - t0;
                dT = dd > 0.0 ? fmaxf((float)dd, 1.17549435e-38f) : (dd < 0.0 ? -fmaxf((float)(-dd), 1.17549435e-38f) : 0.0f);
            }
        }
        const float tempeffect = 100.0f + (100.0f / (T + 15.0f));
        const float total_cc = (3000.0f + (5.0f * (rain - tempeffect))) / k.rescale_veg;
        float nb = tb;
        if (dT > 0.f) {
            const float r_plus = dT * (1.0f + tanhf((T - k.temp_inflex) / k.temp_sens));
            nb += ((r_plus * nb) * (1.0f - (nb / total_cc)));
        }
        if (dT < 0.f) {
            const float r_minus = dT * (1.0f - tanhf((T - k.temp_inflex) / k.temp_sens));
            nb += ((r_minus * nb) * (nb / total_cc));
        }
        if (dT == 0.f) nb = total_cc;
        if (nb < 1.f) nb = 1.0f;
        totB[i] = nb;
        if (dz_out) {
            dz_out[i] = dz;
            wc_out[i] = wC;
            wp_out[i] = wP;
        }
        sums.v[0] += wC;
        sums.v[1] += wP;
        sums.v[2] += nb;
    };
    for (int64_t r0 = ch.first; r0 < ch.end; r0 += blockDim.x) {
        if (r0 + threadIdx.x < ch.end) cell(r0 + threadIdx.x);
        sums.turn();
    }
    const double total = sums.finish();
    if (threadIdx.x < 4)
        atomicAdd(threadIdx.x == 0   ? &o.tot_wc
                  : threadIdx.x == 1 ? &o.tot_wp
                  : threadIdx.x == 2 ? &o.tot_bio
                                     : &o.tot_d,
                  total);
}

__global__ void k_mod_reset(DevScalars* sc, DemCtx dc, int tiled) {
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d == 0) {
        sc->counters[0] = 0;
        sc->sed_tiled_ok = tiled;
        sc->tile_src = 0;
    }
    if (d < dc.n) {
        DemOut& o = dc.out[d];
        o.sed_done = 0;
        o.tot_e = o.tot_i = o.tot_g = o.tot_d = o.tot_wc = o.tot_wp = o.tot_bio = 0.0;
        o.fa_max_key = 0ull;
    }
}

}  // namespace

lem_status launch_erosion(const DevState& s, const ModelConsts& k, uint32_t flags, const Launch& L) {
    const int T = 256;
    const float* prop = (k.flow_type != 0 && k.mfd_props) ? s.prop : nullptr;
    const int tiled = (k.flow_type == 0 && !prop) ? 1 : 0;
    LEM_LAUNCH(L, k_mod_reset, (s.dems.n + 127) / 128, 128, s.sc, s.dems, tiled);
    LEM_LAUNCH(L, k_erosion, s.n_chunks, T, s.z, s.z_init, s.mask, s.slopes, s.fa, s.fines, s.nut, s.soilT, s.stone,
               s.totB, s.slopeptr, s.ero, s.inci, s.geli, s.depo, s.fd, s.chunk_start, k, s.dems, s.sc);
    const TileSet ts = tiles_of(s, k.W);
    {
        const size_t vb = (ts.span() + T - 1) / T;
        LEM_LAUNCH(L, k_sed_prep, (int)(vb > 152 * 32 ? 152 * 32 : vb), T, s.mask, s.fd, prop, s.ero, s.inci, s.geli,
                   s.stone, s.soilT, s.p_abc, s.t_stat, s.pending, s.list_a, k, s.sc, ts);
    }
    if (tiled) {
        const int tiles = ts.n;
        LEM_LAUNCH(L, k_sedt_local, tiles, 256, s.mask, s.fd, s.ero, s.inci, s.geli, s.depo, s.stone, s.fines,
                   s.soilT, s.t_dst, s.t_pend, s.t_rec, s.p_abc, s.p_ref, s.p_map, s.t_stat, s.f_idx, s.f_map,
                   s.f_ds, s.t_fcnt, s.list_b, k, s.sc, s.dems, ts);
        const uint8_t* fd = s.fd;
        const int4* trec = s.t_rec;
        int32_t* tnxt = s.t_nxt;
        const int32_t* tdst = s.t_dst;
        const float4* pabc = s.p_abc;
        const int32_t* pref = s.p_ref;
        const float4* pmap = s.p_map;
        float* pval = s.p_val;
        float* depo = s.depo;
        float* stone = s.stone;
        float* fines = s.fines;
        float* soilT = s.soilT;
        int32_t* tpend = s.t_pend;
        const int32_t* outs = s.list_b;  // the outlets, listed by k_sedt_local
        int32_t* ready = s.list_a;
        ModelConsts kk = k;
        DevScalars* sc = s.sc;
        void* args[] = {(void*)&fd,    (void*)&trec, (void*)&tnxt, (void*)&tdst,  (void*)&pabc, (void*)&pref,
                        (void*)&pmap,  (void*)&pval, (void*)&depo, (void*)&stone, (void*)&fines, (void*)&soilT,
                        (void*)&tpend, (void*)&outs, (void*)&ready, (void*)&kk,   (void*)&sc};
        L.pre("k_sedt_coarse");
        LEM_CUDA_TRY(coop_launch((const void*)k_sedt_coarse, coop_for(s, k, kCkSedCoarse), args, L.st));
        L.post();
        LEM_LAUNCH(L, k_sedt_final, tiles, 256, s.mask, s.fd, s.ero, s.inci, s.geli, s.depo, s.stone, s.fines,
                   s.soilT, s.t_pend, s.t_stat, s.f_idx, s.f_map, s.f_ds, s.t_fcnt, s.p_val, k, s.sc, s.dems,
                   ts);
    }
    {
        const float4* coef = s.p_abc;  // per cell (a tile has kTile * kTile of them)
        const uint8_t* nonzero = s.t_stat;
        float* depo = s.depo;
        float* stone = s.stone;
        float* fines = s.fines;
        float* soilT = s.soilT;
        int32_t* word = s.pending;
        int32_t* list = s.list_a;
        ModelConsts kk = k;
        DevScalars* sc = s.sc;
        DemCtx dc = s.dems;
        int gate = tiled;
        void* args[] = {(void*)&prop, (void*)&coef, (void*)&nonzero, (void*)&depo, (void*)&stone, (void*)&fines, (void*)&soilT,
                        (void*)&word, (void*)&list, (void*)&kk,      (void*)&sc,   (void*)&dc,    (void*)&gate};
        L.pre("k_sed_walk");
        LEM_CUDA_TRY(coop_launch((const void*)k_sed_walk, coop_for(s, k, kCkSedWalk), args, L.st));
        L.post();
    }
    const bool diag = (flags & LEM_STEP_KEEP_DIAGNOSTICS) != 0;
    LEM_LAUNCH(L, k_final, s.n_chunks, T, s.z, s.z_init, s.mask, s.fa, s.ero, s.inci, s.geli, s.depo, s.soilT,
               s.stone, s.fines, s.soilM, s.soilB, s.nut, s.totB, diag ? s.dz : nullptr, diag ? s.wc : nullptr,
               diag ? s.wp : nullptr, s.temp_tab, s.chunk_start, k, s.dems);
    LEM_CUDA_TRY(cudaGetLastError());
    return LEM_OK;
}

const void* mod_coop_kernels[] = {(const void*)k_sed_walk, (const void*)k_sedt_coarse};
extern const int mod_coop_kernel_count = 2;

}  // namespace lem
