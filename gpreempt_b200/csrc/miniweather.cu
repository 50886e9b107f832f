// miniWeather on the executor's kernel list: twelve preemptible semi-discrete steps per time step.
// Follows src/workloads/miniweather.cu of the reference (initial state :395-507, time step
// :182-200, kernels :222-372, reductions :650-677); arithmetic keeps the reference's types - the
// horizontal flux evaluates density, winds, temperature and pressure in double, everything else
// is float - so that results agree with it to rounding.
#include "stencil.h"

#include "model.h"
#include "quotients.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <thread>
#include <vector>

namespace gpx {

namespace {

// Physical constants of the reference (miniweather.cu:35-52), `real` = float.
constexpr float kPi = 3.14159265358979323846264338327;
constexpr float kGrav = 9.8;
constexpr float kCp = 1004.;
constexpr float kCv = 717.;
constexpr float kRd = 287.;
constexpr float kP0 = 1.e5;
constexpr float kC0 = 27.5629410929725921310572974482;
constexpr float kGamm = 1.40027894002789400278940027894;
constexpr float kXlen = 2.e4;
constexpr float kZlen = 1.e4;
constexpr float kHvBeta = 0.05;
constexpr float kCfl = 1.50;
constexpr float kMaxSpeed = 450;
constexpr int ID_DENS = 0, ID_UMOM = 1, ID_WMOM = 2, ID_RHOT = 3;

struct Grid {
    int nx, nz, W;   // W: row stride (nx + 4)
    unsigned plane;  // (nz + 4) * W; four planes stay below 2^31 elements (checked when the model is built)
};

__device__ __forceinline__ Grid grid_of(const StencilParams &p) {
    Grid g;
    g.nx = p.nx;
    g.nz = p.nz;
    g.W = p.nx + 2 * kMwHalo;
    g.plane = (unsigned)(p.nz + 2 * kMwHalo) * (unsigned)g.W;
    return g;
}


// Arithmetic with every rounding written out.  The reference is compiled with nvcc's default
// -fmad=true, which leaves the choice between a fused multiply-add and a rounded product plus a
// sum to the assembler; its choice depends on the surrounding code, so relying on it here would
// tie the results to register pressure.  These are the operations the reference's kernels
// execute (checked on a GPU against that code: all cells of all variables identical).
//
// The kernels are bound by instruction issue, and half of what they issued was divisions: eleven
// (eight along x, where three more are in double) with a divisor that is a constant, a parameter, or
// shared by three of them.  They are taken by reciprocals (quotients.cuh): the quotients of the divisions
// bit for bit, except that a numerator below 2^-100 (the fringe ahead of a disturbance, where values
// fall to nothing within cells) may miss by one or two in the last place.  A horizontal tile that reads an
// infinity, a NaN, a value of 1e15 or a density beyond half the hydrostatic one divides; along z
// div_by_any keeps infinities, and a density of zero, of which either way makes NaN, needs no care.
// 3200 x 1600, a time step: 1 727 us with divisions and pow, 958 like this; 777 with four cells a lane along x (451 ->
// 310 instructions a cell, loads a tile ahead: 84 -> 64 us a kernel) and steps unrolled along z with all of an
// SM's memory as cache (73 -> 64).
template <bool DIVIDE>
__device__ __forceinline__ float quotient(float a, float b, float y) { return DIVIDE ? __fdiv_rn(a, b) : div_by(a, b, y); }
template <bool DIVIDE>
__device__ __forceinline__ double quotient(double a, double b, double y) { return DIVIDE ? __ddiv_rn(a, b) : div_by(a, b, y); }

__device__ __forceinline__ float interp4_by_12(float s0, float s1, float s2, float s3) {
    // -s0 + 7*(s1 + s2) - s3
    return __fsub_rn(__fmaf_rn(7.f, __fadd_rn(s1, s2), -s0), s3);
}
__device__ __forceinline__ float third_derivative(float s0, float s1, float s2, float s3, float hv_coef) {
    // (-s0 + 3*(s1 - s2) + s3) * hv_coef
    return __fmul_rn(__fadd_rn(__fmaf_rn(3.f, __fsub_rn(s1, s2), -s0), s3), hv_coef);
}
__device__ __forceinline__ float advance(float init, float dt, float tend) { return __fmaf_rn(dt, tend, init); }

constexpr float kWild = 1.0e15f;  // (products of two, over a third of the density, stay finite)

struct Flux4 {
    float v[kMwVars];
};

// Flux through an interface along x from the interpolated values and third derivatives (compute_tendencies_x, :222-258).
template <bool DIVIDE>
__device__ __forceinline__ Flux4 flux_x(const float (&vals)[kMwVars], const float (&d3)[kMwVars], float hd, float hdt) {
    const double r = (double)__fadd_rn(vals[ID_DENS], hd);
    const double inv_r = DIVIDE ? 0.0 : reciprocal(r);
    const double u = quotient<DIVIDE>((double)vals[ID_UMOM], r, inv_r);
    const double w = quotient<DIVIDE>((double)vals[ID_WMOM], r, inv_r);
    const double t = quotient<DIVIDE>((double)__fadd_rn(vals[ID_RHOT], hdt), r, inv_r);
    const double pr = __dmul_rn((double)kC0, power(__dmul_rn(r, t), (double)kGamm));
    const double ru = __dmul_rn(r, u);
    // r*u feeds four fluxes; the mass flux subtracts from the rounded product, the others fuse
    Flux4 f;
    f.v[ID_DENS] = (float)__dsub_rn(ru, (double)d3[ID_DENS]);
    f.v[ID_UMOM] = (float)__dsub_rn(__fma_rn(ru, u, pr), (double)d3[ID_UMOM]);
    f.v[ID_WMOM] = (float)__fma_rn(ru, w, -(double)d3[ID_WMOM]);
    f.v[ID_RHOT] = (float)__fma_rn(ru, t, -(double)d3[ID_RHOT]);
    return f;
}

// The fluxes through a lane's four interfaces, two at a time; interface q reads staged cells q .. q + 3 of the lane's own
// four (at `own`) and the next lane's (at `next`).
template <bool DIVIDE>
__device__ __forceinline__ void lane_fluxes(const float *own, const float *next, float hv_coef, float hd, float hdt, Flux4 (&f)[kMwCells + 1]) {
#pragma unroll
    for (int h = 0; h < kMwCells; h += 2) {
        float vals[2][kMwVars], d3[2][kMwVars];
#pragma unroll
        for (int ll = 0; ll < kMwVars; ++ll) {
            const float4 a = *reinterpret_cast<const float4 *>(own + ll * kMwRowFloats);
            const float4 b = *reinterpret_cast<const float4 *>(next + ll * kMwRowFloats);
            const float s[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int o = h + q;
                vals[q][ll] = quotient<DIVIDE>(interp4_by_12(s[o], s[o + 1], s[o + 2], s[o + 3]), 12.f, 1.f / 12.f);
                d3[q][ll] = third_derivative(s[o], s[o + 1], s[o + 2], s[o + 3], hv_coef);
            }
        }
        f[h] = flux_x<DIVIDE>(vals[0], d3[0], hd, hdt);
        f[h + 1] = flux_x<DIVIDE>(vals[1], d3[1], hd, hdt);
    }
}

template <int BYTES>
__device__ __forceinline__ void copy_async(uint32_t dst, const float *src) {
    if (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}

// Horizontal tiles: four segments of at most 124 cells of a row, one to a warp.  compute_tendencies_x (:222-258) then
// compute_tendencies_x_r (:260-272).  The segment from two cells before its first to two behind its last is
// copied to shared memory, four cells a lane: a lane has four interfaces, and with its neighbour's first flux the
// four cells between them (the last lane has only that flux to give).  The cells beyond the ends of the row wrap around
// as set_halo_values_x (:331-341) would have written them, whichever segment reads them, and the segments at the ends of
// the row store those halo cells.  While a warp works on a segment its next one and the starting values of its cells are on
// their way, and the claim after that runs beside them.  (A claim for every warp is 41 600 of them in 70 us on
// one word and one cursor of a 3 200 x 1 600 grid, which is what bounded the kernel then.)  When the word goes up a CTA has up
// to three tiles to run, 14.6 us in the middle and 16.3 at most at that size (4.5 and 5.3 with a claim behind every tile); a kernel
// along z, whose tiles all run at once, lasts 65.
struct RowTile {
    int k, i0, n;       // row, first cell, cells
    unsigned at;        // array index of the first staged cell: column i0, which is cell i0 - 2
    float hd, hdt;      // the row's background
};
__device__ __forceinline__ RowTile row_tile(const StencilParams &p, const Grid &g, int tile, int warp) {
    RowTile r;
    const int seg = tile * (kMwThreads / 32) + warp;
    r.k = seg / p.segs_per_row;
    r.i0 = (seg - r.k * p.segs_per_row) * p.tile_x;
    r.n = r.k < g.nz ? min(p.tile_x, g.nx - r.i0) : 0;
    if (r.n == 0) r.k = 0, r.i0 = 0;  // (the last tile may have fewer than four)
    r.at = (unsigned)(r.k + kMwHalo) * (unsigned)g.W + (unsigned)r.i0;
    r.hd = p.hy_dens_cell[r.k + kMwHalo], r.hdt = p.hy_dens_theta_cell[r.k + kMwHalo];
    return r;
}

// VEC: floats a copy moves (rows of a multiple of VEC array columns are aligned to it).
template <int VEC>
__device__ __forceinline__ void fetch_row(const StencilParams &p, const Grid &g, const RowTile &r, float *stage, int lane) {
    const int left = g.W - r.i0 - kMwCells * lane;  // array columns from this lane's first on
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage) + (uint32_t)lane * kMwCells * 4;
    if (r.n && kMwCells * lane < r.n + 2 * kMwHalo)
#pragma unroll
        for (int ll = 0; ll < kMwVars; ++ll) {
            const float *f = p.forcing + ll * g.plane + r.at + kMwCells * lane, *i = p.init + ll * g.plane + r.at + kMwCells * lane;
#pragma unroll
            for (int c = 0; c < kMwCells; c += VEC)
                if (c < left) {
                    copy_async<4 * VEC>(dst + (ll * kMwRowFloats + c) * 4, f + c);
                    copy_async<4 * VEC>(dst + ((kMwVars + ll) * kMwRowFloats + c) * 4, i + c);
                }
        }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <int VEC>
__device__ __forceinline__ void work_row(const StencilParams &p, const Grid &g, const RowTile &r, float *stage, int lane, float hv_coef,
                                         float inv_dx) {
    if (r.n == 0) return;
    if (r.i0 == 0 || r.i0 + r.n > g.nx - kMwHalo) {
        // an end of the row (or both) is staged: the cells beyond it.  (The segment before a last one of a single cell
        // reads one of them as well, and stores what the last one stores there: without a branch for that, or the last staged
        // column in a register, 64 us a kernel at 3 200 x 1 600 instead of 69.)
        if (lane < 4 * kMwVars) {
            const int ll = lane >> 2, side = lane & 3;
            const int ca = side < 2 ? side : g.nx + side;  // array column
            if (side < 2 ? r.i0 == 0 : side < r.i0 + r.n + 2 * kMwHalo - g.nx) {
                const unsigned row = ll * g.plane + r.at - (unsigned)r.i0;
                const float v = p.forcing[row + (side < 2 ? ca + g.nx : ca - g.nx)];
                stage[ll * kMwRowFloats + ca - r.i0] = v;
                p.forcing[row + ca] = v;
            }
        }
        __syncwarp();
    }
    const float hd = r.hd, hdt = r.hdt;
    const float *own = stage + kMwCells * lane;
    // (the last lane has one interface, of its own cells; what it makes of the others is not used)
    const float *next = stage + kMwCells * min(lane + 1, 31);
    bool wild = !(fabsf(hdt) < kWild && hd > 1.0e-6f && hd < kWild);
    {
        float4 x[kMwVars];
#pragma unroll
        for (int ll = 0; ll < kMwVars; ++ll) {
            x[ll] = *reinterpret_cast<const float4 *>(own + ll * kMwRowFloats);
            const int staged = r.n + 2 * kMwHalo - kMwCells * lane;  // of this lane's four
            if (staged < 4) x[ll].w = 0.f;
            if (staged < 3) x[ll].z = 0.f;
            if (staged < 2) x[ll].y = 0.f;
            if (staged < 1) x[ll].x = 0.f;
        }
        const float dens = largest(largest(x[ID_DENS].x, x[ID_DENS].y, x[ID_DENS].z), x[ID_DENS].w, 0.f);
        float rest = 0.f;
#pragma unroll
        for (int ll = 1; ll < kMwVars; ++ll) rest = largest(largest(rest, x[ll].x, x[ll].y), x[ll].z, x[ll].w);
        // (four thirds of the largest density around is the most the interpolation makes of it)
        wild |= !(2.f * dens < hd && rest < kWild);
    }
    const bool divide = __any_sync(0xffffffffu, wild);
    Flux4 f[kMwCells + 1];
    if (divide)
        lane_fluxes<true>(own, next, hv_coef, hd, hdt, f);
    else
        lane_fluxes<false>(own, next, hv_coef, hd, hdt, f);
#pragma unroll
    for (int ll = 0; ll < kMwVars; ++ll) f[kMwCells].v[ll] = __shfl_down_sync(0xffffffffu, f[0].v[ll], 1);
    const int cells = r.n - kMwCells * lane;
    if (cells <= 0) return;
#pragma unroll
    for (int ll = 0; ll < kMwVars; ++ll) {
        const float *ini = stage + (kMwVars + ll) * kMwRowFloats + kMwCells * lane + kMwHalo;
        const float2 a = *reinterpret_cast<const float2 *>(ini), b = *reinterpret_cast<const float2 *>(ini + 2);
        const float init_v[kMwCells] = {a.x, a.y, b.x, b.y};
        float o[kMwCells];
#pragma unroll
        for (int c = 0; c < kMwCells; ++c) {
            const float d = __fsub_rn(f[c + 1].v[ll], f[c].v[ll]);
            const float tend = -(divide ? __fdiv_rn(d, p.dx) : div_by(d, p.dx, inv_dx));
            o[c] = advance(init_v[c], p.dt, tend);
        }
        float *out = p.out + ll * g.plane + r.at + kMwHalo + kMwCells * lane;
        if (VEC > 1 && cells >= kMwCells) {
            *reinterpret_cast<float2 *>(out) = make_float2(o[0], o[1]);
            *reinterpret_cast<float2 *>(out + 2) = make_float2(o[2], o[3]);
        } else {
#pragma unroll
            for (int c = 0; c < kMwCells; ++c)
                if (c < cells) out[c] = o[c];
        }
    }
}

// Value of variable ll in array row ka (a row outside the interior) of column ca as the
// reference's flux kernel reads it after set_halo_values_z (:346-372): the boundary row's value
// (scaled by the density ratio for the horizontal momentum, zero for the vertical momentum) where
// the reference's launch covers the cell, else what the array holds.  A derived value is stored.
__device__ __forceinline__ float halo_row_value(const StencilParams &p, const Grid &g, int ll, int ka, int ca) {
    const unsigned at = ll * g.plane + (unsigned)ka * (unsigned)g.W + (unsigned)ca;
    if (ll * g.W + ca >= p.halo_z_ids) return p.forcing[at];
    float v = 0.f;
    if (ll != ID_WMOM) {
        const bool low = ka < kMwHalo;
        v = p.forcing[ll * g.plane + (unsigned)(low ? kMwHalo : g.nz + kMwHalo - 1) * (unsigned)g.W + (unsigned)ca];
        if (ll == ID_UMOM) v = v * p.halo_ratio[low ? ka : ka - g.nz];
    }
    p.forcing[at] = v;
    return v;
}

// Vertical tile: kMwThreadsZ columns x up to kMwTileZRows rows; one thread walks down one column
// with the four stencil rows of every variable in registers.  compute_tendencies_z (:278-318)
// then compute_tendencies_z_r (:320-336).  Four steps are unrolled, so that the rows change their roles by name and
// no register is moved.
__device__ __forceinline__ void tile_z(const StencilParams &p, const Grid &g, int tile) {
    const int tr = tile / p.tiles_cols;
    const int i = (tile - tr * p.tiles_cols) * kMwThreadsZ + (int)threadIdx.x;  // cell column
    if (i >= g.nx) return;
    const int k0 = tr * p.tile_rows;
    const int nr = min(p.tile_rows, g.nz - k0);
    const int ca = i + kMwHalo;
    const float hv_coef = __fdiv_rn(__fmul_rn(-kHvBeta, p.dz), __fmul_rn(16.f, p.dt));
    const float inv_dz = __frcp_rn(p.dz);
    const float *__restrict__ forcing = p.forcing;
    auto row_value = [&](int ll, int ka) {  // of array row ka
        return ka >= kMwHalo && ka < g.nz + kMwHalo ? forcing[ll * g.plane + (unsigned)ka * (unsigned)g.W + (unsigned)ca]
                                                    : halo_row_value(p, g, ll, ka, ca);
    };
    float win[4][kMwVars];  // array row r of a step's stencil is win[(j + r) & 3]
#pragma unroll
    for (int ll = 0; ll < kMwVars; ++ll)
#pragma unroll
        for (int r = 0; r < 4; ++r) win[r][ll] = row_value(ll, k0 + r);
    float next_init[kMwVars] = {0.f, 0.f, 0.f, 0.f};
    float below[kMwVars] = {0.f, 0.f, 0.f, 0.f};  // flux through the interface under the cell about to be updated
    for (int j0 = 0; j0 <= nr; j0 += 4) {
#pragma unroll
        for (int ph = 0; ph < 4; ++ph) {
            const int j = j0 + ph;
            if (j > nr) break;
            const int k = k0 + j;  // interface below cell row k
            const unsigned cell = (unsigned)(k - 1 + kMwHalo) * (unsigned)g.W + (unsigned)ca;  // cell above interface k-1
            // Values of the next step are loaded one step ahead, before this step's stores (out may be
            // the array init points to, so a load could not move above a store by itself).
            float next_row[kMwVars], init_v[kMwVars];
#pragma unroll
            for (int ll = 0; ll < kMwVars; ++ll) {
                init_v[ll] = next_init[ll];
                if (j < nr) {
                    next_row[ll] = row_value(ll, k + 4);  // last row of the next interface's stencil
                    next_init[ll] = p.init[ll * g.plane + cell + (unsigned)g.W];  // cell row k, updated next step
                }
            }
            const float hd = p.hy_dens_int[k], hdt = p.hy_dens_theta_int[k];
            float vals[kMwVars], d3_vals[kMwVars];
#pragma unroll
            for (int ll = 0; ll < kMwVars; ++ll) {
                const float s0 = win[ph][ll], s1 = win[(ph + 1) & 3][ll], s2 = win[(ph + 2) & 3][ll], s3 = win[(ph + 3) & 3][ll];
                vals[ll] = div_by_any(interp4_by_12(s0, s1, s2, s3), 12.f, 1.f / 12.f);
                d3_vals[ll] = third_derivative(s0, s1, s2, s3, hv_coef);
            }
            const float r = __fadd_rn(vals[ID_DENS], hd);
            const float inv_r = reciprocal(r);
            const float u = div_by_any(vals[ID_UMOM], r, inv_r);
            float w = div_by_any(vals[ID_WMOM], r, inv_r);
            const float t = div_by_any(__fadd_rn(vals[ID_RHOT], hdt), r, inv_r);
            const float pr = __fmaf_rn(kC0, powf(__fmul_rn(r, t), kGamm), -p.hy_pressure_int[k]);
            if (k == 0 || k == g.nz) {
                w = 0;
                d3_vals[ID_DENS] = 0;
            }
            const float rw = __fmul_rn(r, w);
            float flux[kMwVars];
            flux[ID_DENS] = __fsub_rn(rw, d3_vals[ID_DENS]);  // from the rounded product, as along x
            flux[ID_UMOM] = __fmaf_rn(rw, u, -d3_vals[ID_UMOM]);
            flux[ID_WMOM] = __fsub_rn(__fmaf_rn(rw, w, pr), d3_vals[ID_WMOM]);
            flux[ID_RHOT] = __fmaf_rn(rw, t, -d3_vals[ID_RHOT]);
            if (j > 0) {
                // Cell row k-1, whose forcing values are array row k+1, the stencil's second.  When the reference
                // runs this stage with forcing and out in one array (the second Runge-Kutta stage) its
                // gravity term reads the density the same launch has already updated: its threads are
                // numbered variable-major (:322-324) and the density blocks run far ahead of the
                // momentum blocks.  `gravity_from_out` selects that value here, where out is a
                // separate array.
                float dens_new = 0.f;
#pragma unroll
                for (int ll = 0; ll < kMwVars; ++ll) {
                    float tend = -div_by_any(__fsub_rn(flux[ll], below[ll]), p.dz, inv_dz);
                    if (ll == ID_WMOM) tend = __fmaf_rn(-(p.gravity_from_out ? dens_new : win[(ph + 1) & 3][ID_DENS]), kGrav, tend);
                    const float v = advance(init_v[ll], p.dt, tend);
                    if (ll == ID_DENS) dens_new = v;
                    p.out[ll * g.plane + cell] = v;
                }
            }
#pragma unroll
            for (int ll = 0; ll < kMwVars; ++ll) {
                below[ll] = flux[ll];
                if (j < nr) win[ph][ll] = next_row[ll];
            }
        }
    }
}

}  // namespace

// One kernel per direction, so each gets its own register budget (the x direction holds doubles
// and a lane's fluxes, the z direction a 4 x 4 stencil window and two prefetched rows).
template <int VEC>
__global__ void __launch_bounds__(kMwThreads, 6)
miniweather_x_kernel(const __grid_constant__ StencilParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ __align__(16) float s_stage[kMwThreads / 32][2][2 * kMwVars * kMwRowFloats];
    if (threadIdx.x == 0) trace_begin(blp);
    const bool dynamic = blp.preempted != nullptr;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const Grid g = grid_of(p);
    const float hv_coef = __fdiv_rn(__fmul_rn(-kHvBeta, p.dx), __fmul_rn(16.f, p.dt));
    const float inv_dx = __frcp_rn(p.dx);
    __shared__ int s_tile[kClaimSlots];
    int tile, next = -1, iter = 0;
    // With a CTA for every tile each has one: a second claim would be two round trips to L2 for nothing.
    const bool more = blp.total_tiles > (int)gridDim.x;
    if (dynamic) {
        if (threadIdx.x == 0) s_tile[claim_slot(0)] = blp_claim(blp, 0);
        __syncthreads();
        tile = s_tile[claim_slot(0)];
    } else {
        tile = blp_claim(blp, 0);
    }
    RowTile now{}, ahead{};
    if (tile >= 0) {
        now = row_tile(p, g, tile, warp);
        fetch_row<VEC>(p, g, now, s_stage[warp][0], lane);
        if (more) {
            if (dynamic) {
                if (threadIdx.x == 0) s_tile[claim_slot(1)] = blp_claim(blp, 1);
                __syncthreads();
                next = s_tile[claim_slot(1)];
            } else {
                next = blp_claim(blp, 1);
            }
        }
    }
    while (tile >= 0) {
        int word = 0, after = -1;
        if (next >= 0) {
            if (dynamic && threadIdx.x == 0) word = load_word(blp.preempted);
            ahead = row_tile(p, g, next, warp);
            fetch_row<VEC>(p, g, ahead, s_stage[warp][(iter + 1) & 1], lane);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        // (the cursor's answer is looked at when the tile is through)
        const bool asks = next >= 0 && (!dynamic || threadIdx.x == 0), up = word != 0;
        if (asks) after = dynamic && !up ? atomicAdd(blp.executed, 1) : blp_claim(blp, iter + 2, word);
        work_row<VEC>(p, g, now, s_stage[warp][iter & 1], lane, hv_coef, inv_dx);
        ++iter;
        if (dynamic && next >= 0) {  // (next is the same for the whole CTA)
            if (threadIdx.x == 0) s_tile[claim_slot(iter + 1)] = after < blp.total_tiles ? after : -1;
            __syncthreads();
            after = s_tile[claim_slot(iter + 1)];
        } else {
            __syncwarp();  // the stage is the tile's after next
        }
        tile = next, now = ahead, next = after;
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

__global__ void __launch_bounds__(kMwThreadsZ, 8)
miniweather_z_kernel(const __grid_constant__ StencilParams p, BlpArgs blp) {
    pdl_enter();
    __shared__ int s_tile;
    const bool dynamic = blp.preempted != nullptr;
    if (threadIdx.x == 0) trace_begin(blp);
    const Grid g = grid_of(p);
    int iter = 0;
    for (;;) {
        int tile;
        if (dynamic) {
            __syncthreads();  // every thread has read the previous s_tile
            if (threadIdx.x == 0) s_tile = blp_claim(blp, iter);
            __syncthreads();
            tile = s_tile;
        } else {
            tile = blp_claim(blp, iter);
        }
        if (tile < 0) break;
        tile_z(p, g, tile);
        ++iter;
        if (blp.total_tiles <= (int)gridDim.x) break;  // a tile for every CTA: there is no second one to ask for
    }
    if (threadIdx.x == 0) trace_end(blp, iter);
}

namespace {

// ---- initial state (sci_init, miniweather.cu:376-507) --------------------------------------

// hydro_const_theta (:580-590): hydrostatic balance at constant potential temperature.
void hydro_const_theta(float z, float &r, float &t) {
    const float theta0 = 300.;
    const float exner0 = 1.;
    float p, exner, rt;
    t = theta0;
    exner = exner0 - kGrav * z / (kCp * theta0);
    p = kP0 * std::pow(exner, (kCp / kRd));
    rt = std::pow((p / kC0), (1. / kGamm));
    r = rt / t;
}

// sample_ellipse_cosine (:612-622).
float sample_ellipse_cosine(float x, float z, float amp, float x0, float z0, float xrad, float zrad) {
    float dist = std::sqrt(((x - x0) / xrad) * ((x - x0) / xrad) + ((z - z0) / zrad) * ((z - z0) / zrad)) * kPi / 2.;
    if (dist <= kPi / 2.) return amp * std::pow(std::cos(dist), 2.);
    return 0.;
}

// collision (:566-575): two thermals of opposite sign on one vertical line.
void collision(float x, float z, float &r, float &u, float &w, float &t, float &hr, float &ht) {
    hydro_const_theta(z, hr, ht);
    r = 0.;
    t = 0.;
    u = 0.;
    w = 0.;
    t = t + sample_ellipse_cosine(x, z, 20., kXlen / 2, 2000., 2000., 2000.);
    t = t + sample_ellipse_cosine(x, z, -20., kXlen / 2, 8000., 2000., 2000.);
}

constexpr int kQ = 3;
constexpr float kQPoints[kQ] = {0.112701665379258311482073460022E0, 0.500000000000000000000000000000E0,
                                0.887298334620741688517926539980E0};
constexpr float kQWeights[kQ] = {0.277777777777777777777777777779E0, 0.444444444444444444444444444444E0,
                                 0.277777777777777777777777777779E0};

struct HostFields {
    std::vector<float> state, hy_dens_cell, hy_dens_theta_cell, hy_dens_int, hy_dens_theta_int, hy_pressure_int;
};

void init_rows(HostFields &h, int nx, int nz, float dx, float dz, int k_from, int k_to) {
    const int W = nx + 2 * kMwHalo;
    const size_t plane = (size_t)(nz + 2 * kMwHalo) * W;
    for (int k = k_from; k < k_to; ++k)
        for (int i = 0; i < W; ++i) {
            float acc[kMwVars] = {0.f, 0.f, 0.f, 0.f};
            for (int kk = 0; kk < kQ; ++kk)
                for (int ii = 0; ii < kQ; ++ii) {
                    float x = (0 + i - kMwHalo + 0.5) * dx + (kQPoints[ii] - 0.5) * dx;
                    float z = (0 + k - kMwHalo + 0.5) * dz + (kQPoints[kk] - 0.5) * dz;
                    float r, u, w, t, hr, ht;
                    collision(x, z, r, u, w, t, hr, ht);
                    acc[ID_DENS] = acc[ID_DENS] + r * kQWeights[ii] * kQWeights[kk];
                    acc[ID_UMOM] = acc[ID_UMOM] + (r + hr) * u * kQWeights[ii] * kQWeights[kk];
                    acc[ID_WMOM] = acc[ID_WMOM] + (r + hr) * w * kQWeights[ii] * kQWeights[kk];
                    acc[ID_RHOT] = acc[ID_RHOT] + ((r + hr) * (t + ht) - hr * ht) * kQWeights[ii] * kQWeights[kk];
                }
            for (int ll = 0; ll < kMwVars; ++ll) h.state[ll * plane + (size_t)k * W + i] = acc[ll];
        }
}

void init_fields(HostFields &h, int nx, int nz, float dx, float dz) {
    const int W = nx + 2 * kMwHalo, R = nz + 2 * kMwHalo;
    h.state.assign((size_t)kMwVars * R * W, 0.f);
    unsigned nt = std::max(1u, std::min(16u, std::thread::hardware_concurrency()));
    std::vector<std::thread> pool;
    for (unsigned t = 0; t < nt; ++t) {
        int a = (int)((long long)R * t / nt), b = (int)((long long)R * (t + 1) / nt);
        pool.emplace_back([&h, nx, nz, dx, dz, a, b] { init_rows(h, nx, nz, dx, dz, a, b); });
    }
    for (auto &t : pool) t.join();
    // Hydrostatic background over cells: every quadrature point samples the cell centre
    // (miniweather.cu:461-475 omits the quadrature offset of z).
    h.hy_dens_cell.assign(R, 0.f);
    h.hy_dens_theta_cell.assign(R, 0.f);
    for (int k = 0; k < R; ++k)
        for (int kk = 0; kk < kQ; ++kk) {
            float z = (0 + k - kMwHalo + 0.5) * dz;
            float r, u, w, t, hr, ht;
            collision(0., z, r, u, w, t, hr, ht);
            h.hy_dens_cell[k] = h.hy_dens_cell[k] + hr * kQWeights[kk];
            h.hy_dens_theta_cell[k] = h.hy_dens_theta_cell[k] + hr * ht * kQWeights[kk];
        }
    // ... and at the interfaces (:477-488).
    h.hy_dens_int.assign(nz + 1, 0.f);
    h.hy_dens_theta_int.assign(nz + 1, 0.f);
    h.hy_pressure_int.assign(nz + 1, 0.f);
    for (int k = 0; k < nz + 1; ++k) {
        float z = (0 + k) * dz;
        float r, u, w, t, hr, ht;
        collision(0., z, r, u, w, t, hr, ht);
        h.hy_dens_int[k] = hr;
        h.hy_dens_theta_int[k] = hr * ht;
        h.hy_pressure_int[k] = kC0 * std::pow((hr * ht), kGamm);
    }
}

int add_field(gpx_model &m, const char *name, Storage::Kind kind, int rank, int64_t d0, int64_t d1, int64_t d2,
              const float *host, bool hidden) {
    Storage s;
    s.name = name;
    s.kind = kind;
    s.rank = rank;
    s.dims[0] = d0;
    s.dims[1] = d1;
    s.dims[2] = d2;
    s.dims[3] = 1;
    size_t n = (size_t)d0 * (rank > 1 ? d1 : 1) * (rank > 2 ? d2 : 1);
    s.bytes = n * sizeof(float);
    s.hidden = hidden;
    GPX_CUDA(cudaMalloc((void **)&s.dptr, s.bytes));
    GPX_CUDA(cudaMemcpy(s.dptr, host, s.bytes, cudaMemcpyHostToDevice));
    m.add_storage(s);
    return GPX_SUCC;
}

}  // namespace

typedef void (*StencilKernel)(const StencilParams, BlpArgs);
static StencilKernel stencil_kernel(int dir, int nx) {
    if (dir != 1) return miniweather_z_kernel;
    return nx % 4 == 0 ? miniweather_x_kernel<4> : (nx % 2 == 0 ? miniweather_x_kernel<2> : miniweather_x_kernel<1>);
}
// The kernels want the split of an SM's memory either way: stages of twenty-four warps, or all of it as cache (left as
// the horizontal kernel needs it, the vertical one takes 82 us instead of 72).
static cudaError_t stencil_prepare(int nx) {
    cudaError_t e = cudaFuncSetAttribute(stencil_kernel(1, nx), cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(stencil_kernel(2, nx), cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxL1);
}
static int stencil_threads(int dir) { return dir == 1 ? kMwThreads : kMwThreadsZ; }

int stencil_grid(int dir, int nx, int total_tiles, int sm_count) {
    int blocks = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, stencil_kernel(dir, nx), stencil_threads(dir), 0);
    if (blocks < 1) blocks = 1;
    return (int)std::max<long long>(1, std::min<long long>((long long)blocks * sm_count, total_tiles));
}

cudaError_t stencil_launch(const StencilParams &p, int grid, const BlpArgs &blp, cudaStream_t s) {
    return launch_layer(stencil_kernel(p.dir, p.nx), grid, stencil_threads(p.dir), 0, s, p, blp);
}

// "miniweather" is the reference's grid (3200 x 1600, miniweather.cu:21-22); "miniweather_tiny"
// (320 x 160) and "miniweather_<nx>x<nz>" exist for tests.
static bool parse_grid(const std::string &name, int &nx, int &nz) {
    if (name == "miniweather") {
        nx = 3200;
        nz = 1600;
        return true;
    }
    if (name == "miniweather_tiny") {
        nx = 320;
        nz = 160;
        return true;
    }
    int a = 0, b = 0;
    char tail = 0;
    if (sscanf(name.c_str(), "miniweather_%dx%d%c", &a, &b, &tail) == 2) {
        nx = a;
        nz = b;
        return true;
    }
    return false;
}

bool is_miniweather(const std::string &name) {
    int nx, nz;
    return parse_grid(name, nx, nz);
}

int build_miniweather(gpx_model &m, const std::string &name, const gpx_model_opts &) {
    int nx = 0, nz = 0;
    GPX_REQUIRE(parse_grid(name, nx, nz), GPX_NOT_FOUND, "unknown model '%s'", name.c_str());
    GPX_REQUIRE(nx >= 8 && nz >= 8 && nx <= 32768 && nz <= 32768 && (long long)nx * nz <= (1ll << 27), GPX_OUT_OF_RANGE,
                "%s: grid %d x %d is outside 8..32768 per side and 2^27 cells", name.c_str(), nx, nz);
    const DeviceInfo &d = device_info();
    GPX_REQUIRE(d.device >= 0, GPX_FAIL, "gpx_init was not called");
    m.device = d.device;
    m.sm_count = d.sm_count;
    m.sci = true;
    m.sci_nx = nx;
    m.sci_nz = nz;
    const float dx = kXlen / nx, dz = kZlen / nz;
    const float dt = std::min(dx, dz) / kMaxSpeed * kCfl;
    m.sci_dt = dt;
    m.sci_dx = dx;
    m.sci_dz = dz;

    HostFields h;
    init_fields(h, nx, nz, dx, dz);
    const int W = nx + 2 * kMwHalo, R = nz + 2 * kMwHalo;
    // state, state_tmp as the reference names them (:142-143); state_tmp2 receives the second
    // Runge-Kutta stage.  All three start from the initial state, halo cells included.
    GPX_TRY(add_field(m, "state", Storage::Table, 3, kMwVars, R, W, h.state.data(), false));
    GPX_TRY(add_field(m, "state_tmp", Storage::Table, 3, kMwVars, R, W, h.state.data(), false));
    GPX_TRY(add_field(m, "state_tmp2", Storage::Table, 3, kMwVars, R, W, h.state.data(), true));
    GPX_TRY(add_field(m, "hy_dens_cell", Storage::Vec, 1, R, 1, 1, h.hy_dens_cell.data(), false));
    GPX_TRY(add_field(m, "hy_dens_theta_cell", Storage::Vec, 1, R, 1, 1, h.hy_dens_theta_cell.data(), false));
    GPX_TRY(add_field(m, "hy_dens_int", Storage::Vec, 1, nz + 1, 1, 1, h.hy_dens_int.data(), false));
    GPX_TRY(add_field(m, "hy_dens_theta_int", Storage::Vec, 1, nz + 1, 1, 1, h.hy_dens_theta_int.data(), false));
    GPX_TRY(add_field(m, "hy_pressure_int", Storage::Vec, 1, nz + 1, 1, 1, h.hy_pressure_int.data(), false));
    m.sci_hy_dens_cell = h.hy_dens_cell;
    m.sci_hy_dens_theta_cell = h.hy_dens_theta_cell;
    m.sci_initial = std::move(h.state);

    StencilParams base{};
    base.hy_dens_cell = m.storages[m.find("hy_dens_cell")].dptr;
    base.hy_dens_theta_cell = m.storages[m.find("hy_dens_theta_cell")].dptr;
    base.hy_dens_int = m.storages[m.find("hy_dens_int")].dptr;
    base.hy_dens_theta_int = m.storages[m.find("hy_dens_theta_int")].dptr;
    base.hy_pressure_int = m.storages[m.find("hy_pressure_int")].dptr;
    // hy_dens_cell_const (:501-506)
    base.halo_ratio[0] = h.hy_dens_cell[0] / h.hy_dens_cell[kMwHalo];
    base.halo_ratio[1] = h.hy_dens_cell[1] / h.hy_dens_cell[kMwHalo];
    base.halo_ratio[2] = h.hy_dens_cell[nz + kMwHalo] / h.hy_dens_cell[nz + kMwHalo - 1];
    base.halo_ratio[3] = h.hy_dens_cell[nz + kMwHalo + 1] / h.hy_dens_cell[nz + kMwHalo - 1];
    base.dx = dx;
    base.dz = dz;
    base.nx = nx;
    base.nz = nz;
    GPX_CUDA(stencil_prepare(nx));
    // Segments of a row of equal width, in whole lanes.
    base.segs_per_row = (nx + kMwTileX - 1) / kMwTileX;
    base.tile_x = ((nx + base.segs_per_row - 1) / base.segs_per_row + kMwCells - 1) / kMwCells * kMwCells;
    base.segs_per_row = (nx + base.tile_x - 1) / base.tile_x;
    base.tiles_cols = (nx + kMwThreadsZ - 1) / kMwThreadsZ;
    // Rows per vertical tile: every tile recomputes one flux row and re-reads three stencil rows, so taller is
    // cheaper, but a step down a column takes 0.66 us however few CTAs an SM has, and 0.25 us for each of them where
    // that is more: the height with the least of rows x steps (3 200 x 1 600: 40 rows; 1 026 x 300: 7, where a
    // kernel takes 11 us instead of 30 with 40).
    {
        const int resident = stencil_grid(2, nx, 1 << 30, m.sm_count) / m.sm_count;
        double best = 0.0;
        for (int rows = 4; rows <= kMwTileZRowsMax; ++rows) {
            const long long tiles = (long long)base.tiles_cols * ((nz + rows - 1) / rows);
            long long left = (tiles + m.sm_count - 1) / m.sm_count;  // of the fullest SM
            double us = 0.0;
            for (; left > 0; left -= resident) us += (rows + 1.5) * std::max(0.66, 0.25 * (double)std::min<long long>(left, resident));
            if (best == 0.0 || us < best) {
                best = us;
                base.tile_rows = rows;
            }
        }
    }
    const char *cover = getenv("GPX_MINIWEATHER_FULL_HALO");
    base.halo_z_ids = (cover && cover[0] == '1') ? W * kMwVars
                                                 : (nx + 2 * kMwHalo * kMwVars + 255) / 256 * 256;

    float *state = m.storages[m.find("state")].dptr;
    float *tmp = m.storages[m.find("state_tmp")].dptr;
    float *tmp2 = m.storages[m.find("state_tmp2")].dptr;
    // perform_timestep (:182-200): x, z, z, x, each a three-stage Runge-Kutta sweep.
    const int dirs[4] = {1, 2, 2, 1};
    for (int sweep = 0; sweep < 4; ++sweep)
        for (int stage = 0; stage < 3; ++stage) {
            Kernel k;
            k.type = KernelType::Stencil;
            k.name = std::string("miniweather_step_kernel.") + (dirs[sweep] == 1 ? "x" : "z") + std::to_string(sweep) +
                     ".rk" + std::to_string(stage + 1);
            StencilParams p = base;
            p.dir = dirs[sweep];
            p.init = state;
            p.forcing = stage == 0 ? state : (stage == 1 ? tmp : tmp2);
            p.out = stage == 0 ? tmp : (stage == 1 ? tmp2 : state);
            p.dt = stage == 0 ? dt / 3 : (stage == 1 ? dt / 2 : dt / 1);
            p.gravity_from_out = stage == 1 ? 1 : 0;
            k.stencil = p;
            k.threads = stencil_threads(p.dir);
            k.total_tiles = p.dir == 1 ? (nz * p.segs_per_row + kMwThreads / 32 - 1) / (kMwThreads / 32)
                                       : p.tiles_cols * ((nz + p.tile_rows - 1) / p.tile_rows);
            k.grid = stencil_grid(p.dir, nx, k.total_tiles, m.sm_count);
            const double cells = (double)nx * nz;
            k.bytes = cells * kMwVars * 4.0 * 3.0;  // forcing and init read, out written
            k.flops = cells * (p.dir == 1 ? 120.0 : 100.0);
            m.kernels.push_back(k);
        }
    return GPX_SUCC;
}

}  // namespace gpx

extern "C" {

// reductions (miniweather.cu:650-677): domain mass and total energy in double from the float state.
int gpx_model_reductions(gpx_model *m, double *mass, double *te) {
    using namespace gpx;
    GPX_REQUIRE(m && mass && te, GPX_FAIL, "NULL argument");
    GPX_REQUIRE(m->sci && m->graph_algo < 0, GPX_NOT_FOUND, "model '%s' has no reductions (miniweather only)", m->name.c_str());
    const int nx = m->sci_nx, nz = m->sci_nz, W = nx + 2 * kMwHalo;
    const size_t plane = (size_t)(nz + 2 * kMwHalo) * W;
    std::vector<float> st(plane * kMwVars);
    GPX_CUDA(cudaMemcpy(st.data(), m->storages[m->find("state")].dptr, st.size() * sizeof(float),
                        cudaMemcpyDeviceToHost));
    double ms = 0, en = 0;
    const float dx = m->sci_dx, dz = m->sci_dz;
    for (int k = 0; k < nz; ++k)
        for (int i = 0; i < nx; ++i) {
            size_t at = (size_t)(k + kMwHalo) * W + i + kMwHalo;
            double r = st[ID_DENS * plane + at] + m->sci_hy_dens_cell[kMwHalo + k];
            double u = st[ID_UMOM * plane + at] / r;
            double w = st[ID_WMOM * plane + at] / r;
            double th = (st[ID_RHOT * plane + at] + m->sci_hy_dens_theta_cell[kMwHalo + k]) / r;
            double p = kC0 * pow(r * th, kGamm);
            double t = th / pow(kP0 / p, kRd / kCp);
            double ke = r * (u * u + w * w);
            double ie = r * kCv * t;
            ms += r * dx * dz;
            en += (ke + ie) * dx * dz;
        }
    *mass = ms;
    *te = en;
    return GPX_SUCC;
}

}  // extern "C"
