// cr_cube.cu -- the batched spectral cube: every channel weighted, planned
// and gridded (or degridded) by one sequence of launches whose number does
// not depend on the number of channels.
//
// Channel c's visibility batch is the unflagged samples of rows r = 0..R-1
// with u_lambda = u_m[r] * s_c, v_lambda = v_m[r] * s_c, s_c = f_c / c (the
// cube batch assembly of casars-imager/src/lib.rs:49571-49576, which leaves
// flagged samples out of the channel batch).  Per channel the path restates
//   * PerPlane density weighting (apply_weighting_with_density_source,
//     weighting.rs:1055-1180 with density_build_cell_convention /
//     density_cell_convention = CubeBriggsWeightor{Density,Lookup},
//     weighting.rs:1455-1483): the density is image-sized, a sample adds its
//     weight at the rounded cell of (u, v) and of (-u, -v)
//     (weight_density_cell_anchor, gridder.rs:1888-1934), f2 uses FP64 sums
//     of d and d^2 (weighting.rs:1108-1121) and the reweight is w / d or
//     w / (d f2 + 1) (casa_briggs_denominator, weighting.rs:2440-2443);
//   * the standard PSWF plan (sample_tap_span, gridder.rs:1976-1995) and
//     gridding (grid_sample_taps_real_complex_pair_planned_f64,
//     gridder.rs:1021-1071) with sumwt = sum of f64 weights (lib.rs:68433-68500);
//   * degridding (degrid_sample_taps_planned_normalized, gridder.rs:1278-1312).
//
// Layout: rows' u, v (f64 metres) are shared by all channels; vis, weight
// and flags are channel-major [C][R].  Planning makes one pass that builds
// the weight density and histograms the samples by (channel, 32 x 32 home
// tile, start cell), a scan, and a second pass that forms each imaging weight
// and scatters 16-byte records {cell | tap rows, sample, w vis} plus the
// weight into bin order.  The index selection runs on the integer fixed-point path of
// cr_fixed.cuh with the FP64 operations as the fallback.  Gridding gives
// every (channel, output tile) to one block, which takes the records of
// the four home tiles whose 7 x 7 footprints reach it (contiguous ranges, by
// the order of the cells), accumulates the tile in shared memory and writes
// it once with coalesced stores -- no memset and no global atomics on the
// output grids.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "cr_fixed.cuh"
#include "cr_internal.cuh"
#include "cr_runs.cuh"
#include "cr_tma.cuh"

namespace cr {

namespace {

constexpr int kCubeThreads = 256;
constexpr int kRowsPerBlock = 4096;   // rows of one channel per planning block
// Shared-memory tile rows are 39 floats apart (39 = 7 mod 32), so that the
// seven rows of a footprint fall in different banks.
constexpr int kRow = 39;
constexpr int kMaxTapRows = 255;      // oversampling up to 254, as the gridder's
// the tap table in floats, rows padded to 8
constexpr int kTapFloats = kMaxTapRows * 8;

struct CubeChan {
    double lscale;       // f / c
    FixScale kx, ky;     // lscale / du, lscale / dv
    FixScale kdx, kdy;   // lscale * nx cell_x, lscale * ny cell_y
    DfScale fx, fy, fdx, fdy;   // the same four as float32 pairs
};

struct CubeArgs {
    int64_t R;
    int32_t C;
    const double* u;
    const double* v;
    const float4* uvdf;        // per position (u_hi, u_lo, v_hi, v_lo); NaN u_hi: exact path only
    const uint32_t* rows;      // the row at each position, or null (in order)
    const CubeChan* ch;
    const float2* vis;
    const float* weight;
    const uint8_t* flags;
    // gridder
    double du, dv;
    int64_t gnx, gny;
    int32_t os, tap_rows;
    int64_t ntx, nty;
    long long cx_fix, cy_fix;
    // density
    int32_t nx, ny;
    double dus, dvs, dcx, dcy;
    long long dcx_fix, dcy_fix;
    int32_t mode;
    float* density;            // [C][nx][ny]
    const float* f2;           // [C]
    // planning
    uint32_t* hist;            // [C * ntiles]
    uint32_t* cursor;          // [C * ntiles]
    double* sumwt;             // [C]
    unsigned long long* counts;// [C][2]: gridded, skipped
    uint4* rec;                // {meta, c R + r, w vis.re, w vis.im}
    float* rec_w;
    // per-sample results kept between the passes ([C][R] by position)
    uint32_t* dcell;           // density cell x ny + y of (u, v), ~0 when none
    uint32_t* ev_tile;         // home tile, or kFlaggedSample / kUngriddedSample
    uint32_t* ev_meta;         // cell in tile | tap rows
};

// Rows' u, v as float32 pairs for the fast path, in the order of the
// positions (`order`, or the rows' own).  Rows whose coordinates are not
// finite, exceed 2^60 or are below 2^-60 (but not zero) get a NaN u_hi and
// always take the integer path.
__global__ void cube_rows_df_kernel(const double* u, const double* v, int64_t R,
                                    const uint32_t* order, uint32_t* rows, float4* out) {
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < R;
         p += (int64_t)gridDim.x * blockDim.x) {
        int64_t r = p;
        if (order) {
            // in range also after a sort that gave up
            r = min((int64_t)order[p], R - 1);
            rows[p] = (uint32_t)r;
        }
        const double um = u[r], vm = v[r];
        const bool ok = isfinite(um) && isfinite(vm) && fabs(um) < 0x1p60 &&
                        fabs(vm) < 0x1p60 && (um == 0.0 || fabs(um) > 0x1p-60) &&
                        (vm == 0.0 || fabs(vm) > 0x1p-60);
        const float uh = __double2float_rn(um), vh = __double2float_rn(vm);
        const float ul = __double2float_rn(__dsub_rn(um, (double)uh));
        const float vl = __double2float_rn(__dsub_rn(vm, (double)vh));
        out[p] = ok ? make_float4(uh, ul, vh, vl)
                    : make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
    }
}

// The key that puts rows near each other in the uv plane together: the home
// tile and cell of the row's point on the grid of the channel with the
// finest cells (su, sv: cells per metre there).  Any order is correct.
constexpr int kMaxKeyPasses = 5;
__global__ void __launch_bounds__(256) cube_row_keys_kernel(const double* u, const double* v,
                                                            int64_t R, double su, double sv,
                                                            int32_t gnx, int32_t gny,
                                                            uint32_t nty, KeyOut out) {
    __shared__ uint32_t s_counts[kMaxKeyPasses * kRadixBins];
    KeyCounts counts{s_counts};
    counts.begin(out);
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < R;
         r += (int64_t)gridDim.x * blockDim.x) {
        // (max and min drop a NaN)
        const float fx = fmaxf((float)(u[r] * su) + 0.5f * (float)gnx, 0.0f);
        const float fy = fmaxf((float)(-v[r] * sv) + 0.5f * (float)gny, 0.0f);
        const uint32_t x = (uint32_t)fminf(fx, (float)gnx - 1.0f);
        const uint32_t y = (uint32_t)fminf(fy, (float)gny - 1.0f);
        counts.put(out, r, (uint64_t)((x >> 5) * nty + (y >> 5)) << 10 | (x & 31u) << 5 |
                               (y & 31u));
    }
    counts.end(out);
}

// Lanes of a warp in runs of equal neighbouring keys.
struct LaneRuns {
    unsigned heads;   // lanes at which a run starts
    int start;        // the lane's own run's
    __device__ __forceinline__ LaneRuns(uint32_t key, int lane) {
        const uint32_t prev = __shfl_up_sync(0xffffffffu, key, 1);
        heads = __ballot_sync(0xffffffffu, lane == 0 || key != prev);
        start = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    }
    __device__ __forceinline__ int end(int lane) const {   // one past the run's last lane
        const unsigned after = lane == 31 ? 0u : heads >> (lane + 1);
        return after ? lane + __ffs(after) : 32;
    }
    // the sum of v over the run, complete in its last lane
    __device__ __forceinline__ float sum(float v, int lane) const {
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const float t = __shfl_up_sync(0xffffffffu, v, d);
            if (lane - d >= start) v += t;
        }
        return v;
    }
};

// The density cell (x, y) of x = s_x p_x + e_x + nx/2 (valid when 1 <= x <
// nx, likewise y) on the float32-pair path; false when undecided.  The cell
// of (-u, -v) is then (nx - x, ny - y), and valid with it.
__device__ __forceinline__ bool df_density_cell(float px, float ex, float py, float ey,
                                                int32_t nx, int32_t ny, int* x, int* y,
                                                bool* ok) {
    int ax, ay;
    float dh;
    if (!df_nearest(px, ex, (nx & 1) ? 0.5f : 0.0f, &ax, &dh) ||
        !df_nearest(py, ey, (ny & 1) ? 0.5f : 0.0f, &ay, &dh))
        return false;
    const int cx = (nx >> 1) + ax, cy = (ny >> 1) + ay;
    *ok = !(cx <= 0 || cy <= 0 || cx >= nx || cy >= ny);
    *x = cx;
    *y = cy;
    return true;
}

// weight_density_cell_anchor with the cube (rounded) conventions.
__device__ __forceinline__ bool density_cell(const CubeArgs& a, const CubeChan& ch, double um,
                                             double vm, bool mirror, int* ox, int* oy) {
    long long tx, ty;
    if (fix_mul(um, ch.kdx, &tx) && fix_mul(vm, ch.kdy, &ty)) {
        const long long X = (mirror ? -tx : tx) + a.dcx_fix;
        const long long Y = (mirror ? ty : -ty) + a.dcy_fix;
        long long ax, ay;
        if (fix_round(X, kFixMargin, &ax) && fix_round(Y, kFixMargin, &ay)) {
            if (ax <= 0 || ay <= 0 || ax >= a.nx || ay >= a.ny) return false;
            *ox = (int)ax;
            *oy = (int)ay;
            return true;
        }
    }
    double u = __dmul_rn(um, ch.lscale), v = __dmul_rn(vm, ch.lscale);
    if (mirror) {
        u = -u;
        v = -v;
    }
    const double x = __dadd_rn(__dmul_rn(u, a.dus), a.dcx);
    const double y = __dadd_rn(__dmul_rn(-v, a.dvs), a.dcy);
    if (!isfinite(x) || !isfinite(y)) return false;
    const double rx = round(x), ry = round(y);
    if (!(rx >= 1.0 && ry >= 1.0 && rx < (double)a.nx && ry < (double)a.ny)) return false;
    *ox = (int)rx;
    *oy = (int)ry;
    return true;
}

// Both density cells of row r at channel c, of (u, v) and of the mirror
// (-u, -v), from one pair of fixed-point products (FP64 fallback per cell):
// what the float32-pair path leaves undecided.  Out of line, so that the
// common path stays short in the instruction cache.
struct DensityCells {
    int x, y, xm, ym;
    bool ok, okm;
};
__device__ __noinline__ DensityCells density_cells(const CubeArgs& a, int c, int64_t r) {
    const CubeChan& ch = a.ch[c];
    const double um = a.u[r], vm = a.v[r];
    DensityCells d{0, 0, 0, 0, false, false};
    long long tx, ty;
    if (fix_mul(um, ch.kdx, &tx) && fix_mul(vm, ch.kdy, &ty)) {
        long long ax, ay;
        // (u, v): x = u s + c, y = -v s + c; mirror: x = -u s + c, y = v s + c
        if (fix_round(tx + a.dcx_fix, kFixMargin, &ax) &&
            fix_round(a.dcy_fix - ty, kFixMargin, &ay)) {
            d.ok = !(ax <= 0 || ay <= 0 || ax >= a.nx || ay >= a.ny);
            d.x = (int)ax;
            d.y = (int)ay;
        } else {
            d.ok = density_cell(a, ch, um, vm, false, &d.x, &d.y);
        }
        if (fix_round(a.dcx_fix - tx, kFixMargin, &ax) &&
            fix_round(a.dcy_fix + ty, kFixMargin, &ay)) {
            d.okm = !(ax <= 0 || ay <= 0 || ax >= a.nx || ay >= a.ny);
            d.xm = (int)ax;
            d.ym = (int)ay;
        } else {
            d.okm = density_cell(a, ch, um, vm, true, &d.xm, &d.ym);
        }
        return d;
    }
    d.ok = density_cell(a, ch, um, vm, false, &d.x, &d.y);
    d.okm = density_cell(a, ch, um, vm, true, &d.xm, &d.ym);
    return d;
}

__device__ __forceinline__ bool finite_f(float x) { return isfinite(x); }

struct Eval {
    bool ok;
    uint32_t tile;
    uint32_t meta;
    float w;
};

// sample_tap_span of a row of a channel: the home tile and meta = start cell
// in the tile | tap rows.
__device__ __forceinline__ void pack_sample(const CubeArgs& a, int32_t x0, int32_t y0, int32_t rx,
                                            int32_t ry, uint32_t* tile, uint32_t* meta) {
    *tile = (uint32_t)(x0 >> 5) * (uint32_t)a.nty + (uint32_t)(y0 >> 5);
    *meta = (uint32_t)(x0 & 31) << 27 | (uint32_t)(y0 & 31) << 22 | (uint32_t)rx << 11 |
            (uint32_t)ry;
}

// What the float32 pairs leave undecided: the integer path, then the
// reference's FP64 operations.
struct PlannedSample {
    bool ok;
    uint32_t tile, meta;
};
__device__ __noinline__ PlannedSample plan_sample_exact(const CubeArgs& a, int c, int64_t r) {
    const CubeChan& ch = a.ch[c];
    const double um = a.u[r], vm = a.v[r];
    PlannedSample out{false, 0u, 0u};
    int64_t x0 = 0, y0 = 0;
    int32_t rx = 0, ry = 0;
    int sx = -1, sy = -1;
    long long tx, ty;
    // x = u K_x + G/2, y = -v K_y + G/2
    if (fix_mul(um, ch.kx, &tx) && fix_mul(vm, ch.ky, &ty)) {
        sx = fix_tap_span(tx + a.cx_fix, a.gnx, a.os, a.tap_rows, &x0, &rx);
        if (sx != 0) sy = fix_tap_span(a.cy_fix - ty, a.gny, a.os, a.tap_rows, &y0, &ry);
        if (sx == 0 || sy == 0) return out;
    }
    if (sx < 0 || sy < 0) {
        const double u = __dmul_rn(um, ch.lscale), v = __dmul_rn(vm, ch.lscale);
        const double x = __dadd_rn(__ddiv_rn(u, a.du), (double)a.gnx / 2.0);
        const double y = __dadd_rn(__ddiv_rn(-v, a.dv), (double)a.gny / 2.0);
        if (!f64_tap_span(x, a.gnx, a.os, a.tap_rows, &x0, &rx) ||
            !f64_tap_span(y, a.gny, a.os, a.tap_rows, &y0, &ry))
            return out;
    }
    out.ok = true;
    pack_sample(a, (int32_t)x0, (int32_t)y0, rx, ry, &out.tile, &out.meta);
    return out;
}

// The scales of a channel's float32-pair path.
struct DfChan {
    DfScale fx, fy, fdx, fdy;
};
__device__ __forceinline__ DfChan df_chan(const CubeArgs& a, int c) {
    const CubeChan& ch = a.ch[c];
    return DfChan{ch.fx, ch.fy, ch.fdx, ch.fdy};
}

// False when the sample does not grid.
__device__ __forceinline__ bool plan_sample(const CubeArgs& a, const DfChan& ch, float4 uv, int c,
                                            int64_t r, uint32_t* tile, uint32_t* meta) {
    int32_t x0 = 0, y0 = 0, rx = 0, ry = 0;
    float px, ex, py, ey;
    df_product(uv.x, uv.y, ch.fx, &px, &ex);
    df_product(-uv.z, -uv.w, ch.fy, &py, &ey);
    const int sx = df_tap_span(px, ex, (int32_t)a.gnx, a.os, a.tap_rows, &x0, &rx);
    const int sy = df_tap_span(py, ey, (int32_t)a.gny, a.os, a.tap_rows, &y0, &ry);
    if (sx == 0 || sy == 0) return false;
    if (sx < 0 || sy < 0) {
        const PlannedSample p = plan_sample_exact(a, c, r);
        *tile = p.tile;
        *meta = p.meta;
        return p.ok;
    }
    pack_sample(a, x0, y0, rx, ry, tile, meta);
    return true;
}

// ev_tile values of samples without a home tile
constexpr uint32_t kFlaggedSample = ~0u;        // flagged: left out of the channel batch
constexpr uint32_t kUngriddedSample = ~0u - 1;  // unflagged, but no grid plan or weight

// Samples are evaluated kVec at a time per thread (rows row0 + 32 j): their
// loads are issued together, so each thread keeps kVec gathers in flight.
constexpr int kVec = 4;
constexpr int kWarpRows = 32 * kVec;

// kVec samples of channel c: flags, reweighting, validity and taps.
__device__ __forceinline__ void eval_samples(const CubeArgs& a, const DfChan& ch, float f2,
                                             int c, int64_t row0, int64_t r1,
                                             Eval (&e)[kVec]) {
    float w[kVec];
    float4 uv[kVec];
    bool live[kVec];
#pragma unroll
    for (int j = 0; j < kVec; ++j) {
        const int64_t r = row0 + 32 * j;
        e[j] = Eval{false, 0u, 0u, 0.0f};
        live[j] = r < r1;
        const int64_t i = (int64_t)c * a.R + (live[j] ? r : 0);
        if (live[j] && a.flags) live[j] = a.flags[i] == 0;
        w[j] = a.weight ? a.weight[i] : 1.0f;
        uv[j] = a.uvdf[live[j] ? r : 0];
    }
    if (a.mode != CR_WEIGHT_NATURAL) {
        float d[kVec];
        const float* dens = a.density + (int64_t)c * a.nx * a.ny;
        if (a.dcell) {
            uint32_t cell[kVec];
#pragma unroll
            for (int j = 0; j < kVec; ++j)
                cell[j] = live[j] ? a.dcell[(int64_t)c * a.R + row0 + 32 * j] : ~0u;
#pragma unroll
            for (int j = 0; j < kVec; ++j) d[j] = cell[j] != ~0u ? dens[cell[j]] : 0.0f;
        } else {
#pragma unroll
            for (int j = 0; j < kVec; ++j) {
                int x, y;
                d[j] = 0.0f;
                const int64_t r = row0 + 32 * j;
                if (live[j] && density_cell(a, a.ch[c], a.u[r], a.v[r], false, &x, &y))
                    d[j] = dens[(int64_t)x * a.ny + y];
            }
        }
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
            float nw = 0.0f;
            if (finite_f(w[j]) && w[j] > 0.0f && finite_f(d[j]) && d[j] > 0.0f)
                nw = a.mode == CR_WEIGHT_UNIFORM
                         ? __fdiv_rn(w[j], d[j])
                         : __fdiv_rn(w[j], __fadd_rn(__fmul_rn(d[j], f2), 1.0f));
            w[j] = nw;
        }
    }
#pragma unroll
    for (int j = 0; j < kVec; ++j) {
        if (!live[j] || !(finite_f(w[j]) && w[j] > 0.0f)) continue;
        if (!plan_sample(a, ch, uv[j], c, row0 + 32 * j, &e[j].tile, &e[j].meta)) continue;
        e[j].ok = true;
        e[j].w = w[j];
    }
}

// Records are binned by (channel, home tile, start cell in the tile), so that
// within a home tile they follow the cell order and records with one start
// cell are adjacent.  The order puts the cells in four groups: those whose
// footprint stays in the tile; those that reach the next tile in y only
// (y >= 26), in both directions, in x only.  The records that reach any one
// neighbour are then contiguous.
constexpr uint32_t kReachY = 26 * 26;                // first cell that reaches tile y + 1
constexpr uint32_t kReachXY = kReachY + 26 * 6;      // ... both x + 1 and y + 1
constexpr uint32_t kReachYEnd = kReachXY + 6 * 6;    // end of those reaching y + 1
__device__ __forceinline__ uint32_t cell_order(uint32_t x, uint32_t y) {
    return y >= 26 ? 6 * x + y + (kReachY - 26)
                   : 26 * x + y + (x >= 26 ? kReachYEnd - kReachY : 0u);
}

// the bin of a channel (all bins of a cube fit 32 bits)
__device__ __forceinline__ uint32_t cell_bin(uint32_t tile, uint32_t meta) {
    return tile << 10 | cell_order(meta >> 27, (meta >> 22) & 31u);
}
constexpr uint32_t kNoCell = ~0u;   // no bin's and no density cell's index

// Pass 1 over every sample: with DENSITY the weight density of both cells
// (u, v) and (-u, -v) and the sample's own density cell; then its grid plan
// and the histogram of (channel, home tile, cell) over the samples that can
// grid -- unflagged, a positive natural weight, an own density cell
// (DENSITY) and a plan.  This counts a superset of the gridded samples: the
// imaging weight w / d or w / (d f2 + 1), known only once every density is
// complete, must also come out positive; the scatter gives a sample for
// which it does not a null record, so the counts stay exact.
// With SORTED, positions are rows in uv order (a.rows): the lanes of a warp
// then share cells, and each run of equal cells adds once.  In row order a
// warp's samples lie in different cells, and the kernel is bound by the
// requests of its three adds a sample: 16 channels of 1.26 M rows 491 us
// against 347 us in uv order.
constexpr int kDensVec = 2;   // 4: 384 us
template <bool DENSITY, bool SORTED>
__global__ void __launch_bounds__(kCubeThreads, 5)
cube_density_kernel(const __grid_constant__ CubeArgs a) {
    const int c = blockIdx.y;
    const DfChan ch = df_chan(a, c);
    const int64_t ntiles = a.ntx * a.nty;
    const int64_t r0 = (int64_t)blockIdx.x * kRowsPerBlock;
    const int64_t r1 = min(a.R, r0 + kRowsPerBlock);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* dens = DENSITY ? a.density + (int64_t)c * a.nx * a.ny : nullptr;
    for (int64_t base = r0 + warp * 32 * kDensVec; base < r1; base += kCubeThreads * kDensVec) {
        float w[kDensVec];
        float4 uv[kDensVec];
        uint32_t row[kDensVec];
        bool live[kDensVec];
#pragma unroll
        for (int j = 0; j < kDensVec; ++j) {
            const int64_t p = base + lane + 32 * j;
            live[j] = p < r1;
            row[j] = SORTED ? a.rows[live[j] ? p : r0] : (uint32_t)(live[j] ? p : r0);
            uv[j] = a.uvdf[live[j] ? p : r0];
        }
#pragma unroll
        for (int j = 0; j < kDensVec; ++j) {
            const int64_t i = (int64_t)c * a.R + row[j];
            if (a.flags) live[j] = live[j] && a.flags[i] == 0;
            w[j] = a.weight ? a.weight[i] : 1.0f;
        }
#pragma unroll
        for (int j = 0; j < kDensVec; ++j) {
            const int64_t p = base + lane + 32 * j;
            const int64_t i = (int64_t)c * a.R + p;
            const bool pos = finite_f(w[j]) && w[j] > 0.0f;
            bool own = true;
            if (DENSITY) {
                uint32_t cell = kNoCell, mirror = kNoCell;
                bool add = false;
                if (live[j]) {
                    int x = 0, y = 0;
                    bool ok = false;
                    // float32 pairs first: (u, v) -> x = u s_x + nx/2,
                    // y = -v s_y + ny/2
                    float px, ex, py, ey;
                    df_product(uv[j].x, uv[j].y, ch.fdx, &px, &ex);
                    df_product(-uv[j].z, -uv[j].w, ch.fdy, &py, &ey);
                    if (df_density_cell(px, ex, py, ey, a.nx, a.ny, &x, &y, &ok)) {
                        if (ok) {
                            cell = (uint32_t)x * (uint32_t)a.ny + (uint32_t)y;
                            mirror = (uint32_t)(a.nx - x) * (uint32_t)a.ny + (uint32_t)(a.ny - y);
                            add = pos;
                        }
                    } else {
                        const DensityCells d = density_cells(a, c, row[j]);
                        if (d.ok) {
                            cell = (uint32_t)d.x * (uint32_t)a.ny + (uint32_t)d.y;
                            if (pos) atomicAdd(&dens[cell], w[j]);
                        }
                        if (d.okm && pos) atomicAdd(&dens[(int64_t)d.xm * a.ny + d.ym], w[j]);
                    }
                }
                if (SORTED) {
                    const LaneRuns runs(add ? cell : kNoCell, lane);
                    const float sum = runs.sum(add ? w[j] : 0.0f, lane);
                    if (add && runs.end(lane) == lane + 1) {
                        atomicAdd(&dens[cell], sum);
                        atomicAdd(&dens[mirror], sum);
                    }
                } else if (add) {
                    atomicAdd(&dens[cell], w[j]);
                    atomicAdd(&dens[mirror], w[j]);
                }
                if (p < r1) a.dcell[i] = cell;
                own = cell != kNoCell;
            }
            uint32_t tile = kUngriddedSample, meta = 0u;
            if (!live[j])
                tile = kFlaggedSample;
            else if (!(pos && own && plan_sample(a, ch, uv[j], c, row[j], &tile, &meta)))
                tile = kUngriddedSample;
            const bool bin = tile < kUngriddedSample;
            if (SORTED) {
                const uint32_t b = bin ? cell_bin(tile, meta) : kNoCell;
                const LaneRuns runs(b, lane);
                if (bin && runs.start == lane)
                    atomicAdd(&a.hist[((int64_t)c * ntiles << 10) + b],
                              (uint32_t)(runs.end(lane) - lane));
            } else if (bin) {
                atomicAdd(&a.hist[((int64_t)c * ntiles << 10) + cell_bin(tile, meta)], 1u);
            }
            if (p < r1) {
                a.ev_tile[i] = tile;
                a.ev_meta[i] = meta;
            }
        }
    }
}

// hi + lo += x without rounding error (Knuth's two-sum; lo collects errors)
__device__ __forceinline__ void two_sum(float& hi, float& lo, float x) {
    const float s = __fadd_rn(hi, x);
    const float bp = __fsub_rn(s, hi);
    const float err = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, bp)), __fsub_rn(x, bp));
    hi = s;
    lo = __fadd_rn(lo, err);
}

// Per channel: sum d and sum d^2 (d > 0) in FP64, then f2 (weighting.rs:1108-1121).
__global__ void __launch_bounds__(kCubeThreads) cube_density_sums(const float* density,
                                                                  int64_t cells, double* sums) {
    const int c = blockIdx.y;
    const float* d = density + (int64_t)c * cells;
    // per thread in float32 pairs (error-free sums and products: exact for
    // sums below 2^48 of integer-valued densities), FP64 only to combine
    float s_hi = 0.f, s_lo = 0.f, q_hi = 0.f, q_lo = 0.f;
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < cells;
         k += (int64_t)gridDim.x * blockDim.x) {
        const float v = d[k];
        two_sum(s_hi, s_lo, v);
        if (v > 0.0f) {
            const float p = __fmul_rn(v, v);
            two_sum(q_hi, q_lo, p);
            q_lo = __fadd_rn(q_lo, fmaf(v, v, -p));
        }
    }
    double s = (double)s_hi + (double)s_lo, s2 = (double)q_hi + (double)q_lo;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    __shared__ double sh[2][kCubeThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][warp] = s;
        sh[1][warp] = s2;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0, t2 = 0.0;
        for (int k = 0; k < kCubeThreads / 32; ++k) {
            t += sh[0][k];
            t2 += sh[1][k];
        }
        atomicAdd(&sums[2 * c], t);
        atomicAdd(&sums[2 * c + 1], t2);
    }
}

__global__ void cube_f2_kernel(const double* sums, int32_t C, double a2, float* f2) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const double s = sums[2 * c], s2 = sums[2 * c + 1];
    f2[c] = (s2 > 0.0 && s > 0.0) ? (float)__ddiv_rn(a2, __ddiv_rn(s2, s)) : 0.0f;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ unsigned long long warp_sum(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Tile-level starts from the cell-level exclusive scan.
__global__ void tile_starts_from_cells(const uint32_t* cell_start, int64_t nbins,
                                       uint32_t* bin_start) {
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b <= nbins;
         b += (int64_t)gridDim.x * blockDim.x)
        bin_start[b] = cell_start[b << 10];
}

// Pass 2: records scattered into (channel, home tile, cell) bins from pass
// 1's plans, kScatterVec samples per thread and iteration so that more
// cursor atomics are in flight.  The imaging weight is formed here, from the
// complete density: w itself, w / d (uniform) or w / (d f2 + 1) (Briggs,
// casa_briggs_denominator, weighting.rs:2440-2443).  A counted sample whose
// weight does not come out positive and finite gets a null record (zero
// weight and value, no sample index), which grids and degrids nothing.  The
// channel's sum of weights and its gridded and unflagged-but-not-gridded
// counts are summed here.
//
// With SORTED the lanes of a warp share cells: a run of equal cells takes its
// slots with one atomic and writes them side by side (16 channels of 1.26 M
// rows: 310 us against 452 us in row order).
constexpr int kScatterVec = 3;   // 6 at 4 blocks per SM: 324 us
constexpr uint32_t kNullSample = ~0u;   // sample index of a null record
template <bool SORTED>
__global__ void __launch_bounds__(kCubeThreads, 6) cube_scatter_kernel(CubeArgs a) {
    __shared__ double s_sum[kCubeThreads / 32];
    __shared__ unsigned long long s_ok[kCubeThreads / 32], s_skip[kCubeThreads / 32];
    const int c = blockIdx.y;
    const int64_t ntiles = a.ntx * a.nty;
    const int lane = threadIdx.x & 31;
    const int64_t r0 = (int64_t)blockIdx.x * kRowsPerBlock;
    const int64_t r1 = min(a.R, r0 + kRowsPerBlock);
    const int wp = threadIdx.x >> 5;
    const float f2 = a.mode == CR_WEIGHT_BRIGGS ? a.f2[c] : 0.0f;
    const float* dens = a.mode != CR_WEIGHT_NATURAL ? a.density + (int64_t)c * a.nx * a.ny
                                                    : nullptr;
    uint32_t* cursor = a.cursor + ((int64_t)c * ntiles << 10);
    // the channel's sum of weights as a float pair (no FP64 instruction per
    // sample), in FP64 from the warp sums on
    PairSum swp;
    unsigned long long n_ok = 0, n_skip = 0;
    for (int64_t base = r0 + wp * 32 * kScatterVec; base < r1;
         base += kCubeThreads * kScatterVec) {
        // loads first, then every cursor atomic, then the stores: the kScatterVec
        // atomics of a thread are in flight together
        uint32_t tile[kScatterVec], meta[kScatterVec], pos[kScatterVec], row[kScatterVec];
        float w[kScatterVec];
        float2 vv[kScatterVec];
#pragma unroll
        for (int j = 0; j < kScatterVec; ++j) {
            const int64_t p = base + lane + 32 * j;
            const int64_t q = p < r1 ? p : r0;
            tile[j] = p < r1 ? a.ev_tile[(int64_t)c * a.R + q] : kFlaggedSample;
            meta[j] = a.ev_meta[(int64_t)c * a.R + q];
            row[j] = SORTED ? a.rows[q] : (uint32_t)q;
        }
#pragma unroll
        for (int j = 0; j < kScatterVec; ++j) {
            const int64_t i = (int64_t)c * a.R + row[j];
            w[j] = a.weight ? a.weight[i] : 1.0f;
            vv[j] = a.vis[i];
        }
        if (dens) {
            float d[kScatterVec];
#pragma unroll
            for (int j = 0; j < kScatterVec; ++j) {
                const int64_t i = (int64_t)c * a.R + base + lane + 32 * j;
                d[j] = tile[j] < kUngriddedSample ? dens[a.dcell[i]] : 0.0f;
            }
#pragma unroll
            for (int j = 0; j < kScatterVec; ++j) {
                float nw = 0.0f;
                if (finite_f(w[j]) && w[j] > 0.0f && finite_f(d[j]) && d[j] > 0.0f)
                    nw = a.mode == CR_WEIGHT_UNIFORM
                             ? __fdiv_rn(w[j], d[j])
                             : __fdiv_rn(w[j], __fadd_rn(__fmul_rn(d[j], f2), 1.0f));
                w[j] = nw;
            }
        }
        int start[kScatterVec];
#pragma unroll
        for (int j = 0; j < kScatterVec; ++j) {
            const bool bin = tile[j] < kUngriddedSample;
            const uint32_t b = bin ? cell_bin(tile[j], meta[j]) : kNoCell;
            pos[j] = 0u;
            if (SORTED) {
                const LaneRuns runs(b, lane);
                start[j] = runs.start;
                if (bin && runs.start == lane)
                    pos[j] = atomicAdd(&cursor[b], (uint32_t)(runs.end(lane) - lane));
            } else if (bin) {
                pos[j] = atomicAdd(&cursor[b], 1u);
            }
        }
        if (SORTED) {
#pragma unroll
            for (int j = 0; j < kScatterVec; ++j)
                pos[j] = __shfl_sync(0xffffffffu, pos[j], start[j]) + (uint32_t)(lane - start[j]);
        }
#pragma unroll
        for (int j = 0; j < kScatterVec; ++j) {
            if (tile[j] == kFlaggedSample) continue;
            const bool ok = tile[j] != kUngriddedSample && finite_f(w[j]) && w[j] > 0.0f;
            if (!ok) ++n_skip;
            if (tile[j] == kUngriddedSample) continue;
            const int64_t i = (int64_t)c * a.R + row[j];
            float vr = 0.0f, vi = 0.0f, wr = 0.0f;
            uint32_t sample = kNullSample;
            if (ok) {
                if (finite_f(vv[j].x) && finite_f(vv[j].y)) {
                    vr = __fmul_rn(vv[j].x, w[j]);
                    vi = __fmul_rn(vv[j].y, w[j]);
                }
                wr = w[j];
                sample = (uint32_t)i;
                ++n_ok;
                swp.add(wr, 0.0f);
            }
            a.rec[pos[j]] = make_uint4(meta[j], sample, __float_as_uint(vr),
                                       __float_as_uint(vi));
            a.rec_w[pos[j]] = wr;
        }
    }
    double sw = (double)swp.h + (double)swp.l;
    sw = warp_sum(sw);
    n_ok = warp_sum(n_ok);
    n_skip = warp_sum(n_skip);
    const int warp = threadIdx.x >> 5;
    if (lane == 0) {
        s_sum[warp] = sw;
        s_ok[warp] = n_ok;
        s_skip[warp] = n_skip;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        unsigned long long o = 0, k = 0;
        for (int q = 0; q < kCubeThreads / 32; ++q) {
            t += s_sum[q];
            o += s_ok[q];
            k += s_skip[q];
        }
        if (t != 0.0) atomicAdd(&a.sumwt[c], t);
        if (o) atomicAdd(&a.counts[2 * c], o);
        if (k) atomicAdd(&a.counts[2 * c + 1], k);
    }
}

// Source records per gridding work item: chosen per cube shape by a
// first-use tuning pass over these candidates (the default before tuning).
constexpr uint32_t kGridChunkCandidates[3] = {1024, 2048, 4096};
constexpr uint32_t kGridChunkDefault = 2048;
constexpr uint32_t kGridChunkMin = 1024;
constexpr uint32_t kDegridChunk = 4096; // records per degridding work item

// Work lists.  Gridding: an output tile (channel, tx, ty) gathers the bins
// (tx, ty), (tx-1, ty), (tx, ty-1), (tx-1, ty-1); their records, taken in
// that order, are cut into chunks (of the tuned size).  A tile with one chunk is
// written with plain stores; the chunks of a heavier tile add into the grid
// with atomics after cube_zero_heavy zeroed it.  Degridding: each bin's
// records in chunks of kDegridChunk.
__device__ __forceinline__ uint32_t bin_count(const uint32_t* bin_start, int64_t bin) {
    return bin_start[bin + 1] - bin_start[bin];
}

// Start of cell bin cb: cell_end holds each cell bin's end (= the next
// bin's start) once the scatter has advanced the cursors.
__device__ __forceinline__ uint32_t cell_start(const uint32_t* cell_end, int64_t cb) {
    return cb == 0 ? 0u : cell_end[cb - 1];
}

// The records of one source of output tile (tx, ty) of channel c that reach
// it: source s is home tile (tx - (s & 1), ty - (s >> 1)); all of the tile's
// own, of the others the group of cells that reaches across.
__device__ __forceinline__ uint2 source_range(const uint32_t* bin_start,
                                              const uint32_t* cell_end, uint32_t c,
                                              uint32_t ntiles, uint32_t nty, uint32_t tx,
                                              uint32_t ty, int s) {
    const uint32_t dx = s & 1, dy = s >> 1;
    if (tx < dx || ty < dy) return make_uint2(0u, 0u);
    const int64_t sb = (int64_t)c * ntiles + (tx - dx) * nty + (ty - dy);
    const int64_t cb = sb << 10;
    return make_uint2(s == 0   ? bin_start[sb]
                      : s == 2 ? cell_start(cell_end, cb + kReachY)
                               : cell_start(cell_end, cb + kReachXY),
                      s < 2 ? bin_start[sb + 1] : cell_start(cell_end, cb + kReachYEnd));
}

// Channels whose plane_mask entry is 0 get no work items.
__global__ void cube_work_count(const uint32_t* bin_start, const uint32_t* cell_end,
                                int64_t nbins, int64_t ntiles, int64_t nty, uint32_t grid_chunk,
                                const uint8_t* plane_mask, uint32_t* grid_chunks,
                                uint32_t* degrid_chunks) {
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nbins;
         b += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t c = (uint32_t)b / (uint32_t)ntiles, T = (uint32_t)b % (uint32_t)ntiles;
        if (plane_mask && !plane_mask[c]) {
            grid_chunks[b] = degrid_chunks[b] = 0u;
            continue;
        }
        const uint32_t tx = T / (uint32_t)nty, ty = T % (uint32_t)nty;
        uint32_t n = 0;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const uint2 r = source_range(bin_start, cell_end, c, ntiles, nty, tx, ty, s);
            n += r.y - r.x;
        }
        grid_chunks[b] = n == 0 ? 1u : (n + grid_chunk - 1) / grid_chunk;
        degrid_chunks[b] = (bin_count(bin_start, b) + kDegridChunk - 1) / kDegridChunk;
    }
}

__global__ void cube_work_fill(const uint32_t* grid_chunks, const uint32_t* grid_first,
                               const uint32_t* degrid_chunks, const uint32_t* degrid_first,
                               int64_t nbins, uint2* grid_items, uint2* degrid_items) {
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nbins;
         b += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t n = grid_chunks[b], f = grid_first[b];
        for (uint32_t k = 0; k < n; ++k) grid_items[f + k] = make_uint2((uint32_t)b, k);
        const uint32_t nd = degrid_chunks[b], fd = degrid_first[b];
        for (uint32_t k = 0; k < nd; ++k) degrid_items[fd + k] = make_uint2((uint32_t)b, k);
    }
}

// The output tiles of several chunks zeroed, a warp per tile and row by row.
__global__ void cube_zero_heavy(const uint32_t* grid_chunks, int64_t nbins, int64_t ntiles,
                                int64_t nty, int64_t gnx, int64_t gny, float* psf,
                                float2* dirty) {
    const int lane = threadIdx.x & 31;
    for (int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < nbins;
         b += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        if (grid_chunks[b] <= 1) continue;
        const int64_t c = b / ntiles, T = b % ntiles;
        const int64_t x0 = (T / nty) * kTile, y = (T % nty) * kTile + lane;
        if (y >= gny) continue;
        for (int64_t x = x0; x < min(x0 + kTile, gnx); ++x) {
            const int64_t cell = (c * gnx + x) * gny + y;
            if (psf) psf[cell] = 0.0f;
            dirty[cell] = make_float2(0.0f, 0.0f);
        }
    }
}

struct CubeGridArgs {
    const uint4* rec;
    const float* rec_w;
    const uint32_t* bin_start;   // [C * ntiles + 1]
    const uint32_t* cell_end;    // [C * ntiles * 1024] end of each cell bin
    const float* taps;           // [tap_rows][8], rows padded with a zero
    int32_t tap_rows;
    uint32_t taps_bytes;
    int* status;                 // set to CR_TIMEOUT when a bounded wait gives up
    int64_t ntx, nty, gnx, gny;
    const uint2* items;          // (output tile bin, chunk)
    uint32_t grid_chunk;         // records per chunk
    const uint32_t* grid_chunks; // chunks of each output tile
    const unsigned long long* n_items;
    unsigned int* item_counter;
    float* psf;                  // [C][gnx][gny] real part of the PSF grid
    float2* dirty;               // [C][gnx][gny] (the residual grid with RESIDUAL)
    const float2* res;           // RESIDUAL: w (vis - pred) per record
    long long wait_polls;        // bound of the tap-table wait (the drain keeps the default)
};

// A block per work item: the chunk's records (from the four source bins)
// accumulate into a shared-memory copy of the output tile, which is then
// stored (single-chunk tile) or added (heavier tile) to the grid.
//
// The kernel is bound by instruction issue (some 18 M records of 49 taps on a
// 16-channel batch of 1.26 M rows), so records are summed by runs of one start
// cell, four at a time (cr_runs.cuh).  A vote over the records' cells ends a
// run, whose sums are added to the tile.  Records are decoded by a lane each,
// 32 ahead of their use; warp 0 fetches the next item's ranges before the tile
// is written; the tile is zeroed as it is read out.
//
// Four warps per block: an item has some 600 records, and every warp more
// cuts its runs once more (256 threads: 6 % slower; 96 and 64 lose occupancy
// to the tile's shared memory, 13 and 44 %).  16 channels of 1.26 M rows:
// 0.57 ms against 0.78 with a lane per tap (411 M instructions against 742 M).
constexpr int kGridThreads = 128, kGridBlocks = 8;

// With RESIDUAL the records carry w (vis - pred) from `res` and no PSF is
// formed.
// A work item as the block reads it.  The tile's sources one after the other
// give its records positions: source s holds [off[s], off[s + 1]) and
// position p is record p + rec[s].
struct GridItem {
    int32_t count;       // records of the chunk, from position `first`; -1: no more items
    uint32_t first;
    uint32_t off[5];
    uint32_t rec[4];
    int32_t x0, y0, rows, cols;   // the tile and its extent inside the grid
    int64_t plane;
    bool shared;         // the tile has several chunks
};

// The next work item into `out`, by one warp.
__device__ __forceinline__ void next_item(const CubeGridArgs& a, int lane, GridItem& out) {
    uint32_t item = 0;
    if (lane == 0) item = atomicAdd(a.item_counter, 1u);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= *a.n_items) {
        if (lane == 0) out.count = -1;
        return;
    }
    const uint2 it = a.items[item];
    const uint32_t nty = (uint32_t)a.nty, ntiles = (uint32_t)a.ntx * nty;
    const uint32_t c = it.x / ntiles, T = it.x % ntiles, tx = T / nty, ty = T % nty;
    const uint2 r = lane < 4 ? source_range(a.bin_start, a.cell_end, c, ntiles, nty, tx, ty, lane)
                             : make_uint2(0u, 0u);
    uint32_t end = r.y - r.x;   // inclusive sum over lanes 0-3
#pragma unroll
    for (int o = 1; o < 4; o *= 2) {
        const uint32_t up = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += up;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, end, 3);
    if (lane < 4) {
        out.off[lane + 1] = end;
        out.rec[lane] = r.y - end;
    }
    if (lane == 0) {
        const uint32_t lo = it.y * a.grid_chunk;
        out.off[0] = 0;
        out.first = lo;
        out.count = (int32_t)(min(total, lo + a.grid_chunk) - min(total, lo));
        out.x0 = (int32_t)(tx * kTile);
        out.y0 = (int32_t)(ty * kTile);
        out.rows = (int32_t)min((int64_t)kTile, a.gnx - tx * kTile);
        out.cols = (int32_t)min((int64_t)kTile, a.gny - ty * kTile);
        out.plane = c;
        out.shared = a.grid_chunks[it.x] > 1;
    }
}

template <bool RESIDUAL>
__global__ void __launch_bounds__(kGridThreads, kGridBlocks) cube_grid_kernel(CubeGridArgs a) {
    constexpr int kPlane = kTile * kRow, kComps = RESIDUAL ? 2 : 3;
    constexpr int kWarps = kGridThreads / 32;
    constexpr uint32_t kDone = ~0u;
    __shared__ __align__(16) float s_taps[kTapFloats];
    __shared__ float s_psf[RESIDUAL ? 1 : kPlane];
    __shared__ __align__(8) float2 s_ri[kPlane];
    __shared__ __align__(16) int4 s_ra[kGridThreads];
    __shared__ __align__(8) float2 s_rb[kGridThreads];
    __shared__ __align__(8) uint64_t s_bar;
    __shared__ GridItem s_items[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the tap table by one bulk copy
    if (tid == 0) {
        mbar_init(&s_bar, 1);
        mbar_fence_init();
        mbar_expect_tx(&s_bar, a.taps_bytes);
        bulk_load(s_taps, a.taps, a.taps_bytes, &s_bar);
    }
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(&s_bar, 0, a.wait_polls))) {
        if (tid == 0) {
            atomicExch(a.status, CR_TIMEOUT);
            mbar_wait(&s_bar, 0);   // let the copy land before the block exits
        }
        return;
    }
    if (warp == 0) next_item(a, lane, s_items[0]);
    // the tile is zero between items
    for (int k = tid; k < kPlane; k += kGridThreads) {
        if (!RESIDUAL) s_psf[k] = 0.0f;
        s_ri[k] = make_float2(0.0f, 0.0f);
    }
    int4* w_ra = s_ra + warp * 32;
    float2* w_rb = s_rb + warp * 32;
    const int g = lane >> 3, ix = lane & 7;
    const float* tap_x = s_taps + ix;
    RunSums<kComps> sums;
    for (int buf = 0;; buf ^= 1) {
        __syncthreads();
        const GridItem& it = s_items[buf];
        if (it.count < 0) break;
        // the sums of the run at cell (x, y) of the tile into the tile
        auto flush = [&](int x, int y) {
            float n[kComps][2];
            sums.exchange(lane, n);
            const bool row = ix < 7 && (unsigned)(x + ix) < kTile;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int iy = 2 * g + t;
                if (row && iy < 7 && (unsigned)(y + iy) < kTile) {
                    const int cell = (x + ix) * kRow + y + iy;
                    if (!RESIDUAL) atomicAdd(&s_psf[cell], n[0][t]);
                    shared_add2(&s_ri[cell], n[kComps - 2][t], n[kComps - 1][t]);
                }
            }
        };
        // each warp takes a contiguous share of the item's records
        const uint32_t n = (uint32_t)it.count;
        const uint32_t share = max(32u, (n + 4 * kWarps - 1) / (4 * kWarps) * 4u);
        const uint32_t w0 = it.first + min(n, warp * share);
        const uint32_t w1 = it.first + min(n, (warp + 1) * share);
        int open_x = 0, open_y = 0;
        bool any = false;
        sums.clear();
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
            const uint32_t lo = max(w0, it.off[s]), hi = min(w1, it.off[s + 1]);
            if (lo >= hi) continue;
            const uint32_t end = hi + it.rec[s];
            const int sx = (s & 1) * kTile, sy = (s >> 1) * kTile;
            uint32_t open = kDone - 1;   // the run's cell; none yet
            uint32_t meta = 0;
            float w = 0.0f;
            float2 v = make_float2(0.0f, 0.0f);
            auto load = [&](uint32_t i) {
                if (i < end) {
                    if (RESIDUAL) {
                        meta = a.rec[i].x;
                        v = a.res[i];
                    } else {
                        const uint4 q = a.rec[i];
                        meta = q.x;
                        w = a.rec_w[i];
                        v = make_float2(__uint_as_float(q.z), __uint_as_float(q.w));
                    }
                }
            };
            uint32_t base = lo + it.rec[s];
            load(base + lane);
#pragma unroll 1
            for (; base < end; base += 32) {
                // 32 records decoded by a lane each; the next 32 on their way
                __syncwarp();
                w_ra[lane] = make_int4(base + lane < end ? (int)(meta >> 22) : (int)kDone,
                                       (int)((meta >> 11) & 2047u) * 8, (int)(meta & 2047u) * 8,
                                       __float_as_int(w));
                w_rb[lane] = v;
                __syncwarp();
                load(base + 32 + lane);
                const int n_batch = (int)min(32u, end - base);
#pragma unroll 1
                for (int k = g; k - g < n_batch; k += 4) {
                    const int4 A = w_ra[k];
                    const float2 B = w_rb[k];
                    uint32_t cell = (uint32_t)A.x;
                    const float wq = __int_as_float(A.w);
                    const float wx = tap_x[A.y];
                    float2 y[4];
                    tap_pairs(s_taps + A.z, y);
                    for (;;) {
                        const bool mine = cell == open;
                        const unsigned match = __ballot_sync(0xffffffffu, mine);
                        if (match) {
                            sums.add(mine, wx, y, wq, B);
                            if (match == 0xffffffffu) break;
                            if (mine) cell = kDone;
                        }
                        const unsigned rest = __ballot_sync(0xffffffffu, cell != kDone);
                        if (!rest) break;
                        if (any) {
                            flush(open_x, open_y);
                            sums.clear();
                        }
                        any = true;
                        open = __shfl_sync(0xffffffffu, cell, __ffs(rest) - 1);
                        open_x = (int)(open >> 5) - sx;
                        open_y = (int)(open & 31u) - sy;
                    }
                }
            }
        }
        if (any) flush(open_x, open_y);
        if (warp == 0) next_item(a, lane, s_items[buf ^ 1]);
        __syncthreads();
        // the tile to the grid, a warp per row
        const int64_t x0 = it.x0, y0 = it.y0;
        const int rows = it.rows;
        const bool col = lane < it.cols, shared_tile = it.shared;
        const int64_t at0 = (it.plane * a.gnx + x0 + warp) * a.gny + y0 + lane;
        float* psf = RESIDUAL ? nullptr : a.psf + at0;
        float2* dirty = a.dirty + at0;
#pragma unroll 4
        for (int j = warp; j < kTile; j += kWarps) {
            const int cell = j * kRow + lane;
            const float vp = RESIDUAL ? 0.0f : s_psf[cell];
            const float2 v = s_ri[cell];
            if (!RESIDUAL) s_psf[cell] = 0.0f;
            s_ri[cell] = make_float2(0.0f, 0.0f);
            if (col && j < rows) {
                if (!shared_tile) {
                    if (!RESIDUAL) *psf = vp;
                    *dirty = v;
                } else {
                    if (!RESIDUAL && vp != 0.0f) atomicAdd(psf, vp);
                    if (v.x != 0.0f || v.y != 0.0f) atomicAdd(dirty, v);
                }
            }
            if (!RESIDUAL) psf += kWarps * a.gny;
            dirty += kWarps * a.gny;
        }
    }
}

struct CubeDegridArgs {
    const uint4* rec;
    const uint32_t* bin_start;   // [C * ntiles + 1]
    int32_t tap_rows;
    int64_t ntiles, nty, gnx, gny, R;
    const uint2* items;          // (bin, chunk)
    const unsigned long long* n_items;
    unsigned int* item_counter;
    const float* taps8;          // [tap_rows][8], rows padded to 32 bytes
    uint32_t taps8_bytes;
    const float2* grid;          // [C][gnx][gny]
    float2* pred;                // [C][R]
    const float* rec_w;          // RESIDUAL: imaging weight per record
    float2* res;                 // RESIDUAL: w vis - w pred per record
    int* status;                 // set to CR_TIMEOUT when a bounded wait gives up
    long long wait_polls;        // bound of the first waits (the drains keep the default)
};

// Bins in turn.  The block stages the 38 x 38 model footprint of its home
// tile in shared memory.  Records follow the cell order, so the 7 x 7 cells
// of a record are mostly those of the one before: a group of four lanes takes
// a record, lane ix holding rows 2 ix and 2 ix + 1 of the cells in registers
// until the cell changes, and a record costs it the tap rows and
// sum_ix wx[ix] sum_iy wy[iy] g[x0 + ix][y0 + iy] in paired FMAs.  The lanes'
// sums of four records are exchanged at once, and each lane writes its own.
// (Seven shared-memory loads of cells a lane and record had the load/store
// unit 91 % busy: 16 channels of 1.26 M rows 432 us, 223 us this way; eight
// lanes a record, one row each, 235 us; four blocks per SM spill, 299 us.)
// With RESIDUAL each record's w vis - w pred goes to res (record order)
// instead of pred (sample order).
// With TMA the footprints come as tensor-map boxes (float32 view
// [C][gnx][2 gny], box 76 x 38, zero-filled past the grid edge) into two
// buffers: while the block works on one item, the next item's footprint is
// already in flight.  Without TMA (a grid whose rows are not a multiple of
// 16 bytes, or an unaligned base) the block loads each footprint itself.
// The tap table arrives by one bulk copy in either case, its rows padded to
// 8 floats so that a record's 7 y taps come in two 16-byte loads.
constexpr int kDegridBlocks = 3;
template <bool RESIDUAL, bool TMA>
__global__ void __launch_bounds__(kCubeThreads, kDegridBlocks) cube_degrid_kernel(
    const __grid_constant__ CUtensorMap gmap, CubeDegridArgs a) {
    constexpr int kFoot = kTile + 6;
    constexpr int kPitch = TMA ? kFoot : kRow;   // float2 per footprint row
    constexpr int kBufs = TMA ? 2 : 1;
    constexpr uint32_t kBoxBytes = kFoot * kFoot * 8;
    // each buffer starts on a 128-byte boundary (tensor copy destinations)
    constexpr int kBufElems = (kFoot * kPitch * 8 + 127) / 128 * 16;
    __shared__ __align__(128) float2 s_g[kBufs][kBufElems];
    __shared__ __align__(8) uint64_t s_bar[3];   // footprint buffers 0, 1; taps
    __shared__ int s_item[2];
    // a warp's batch: cell in the footprint, x and y tap rows
    __shared__ __align__(16) int4 s_rec[kCubeThreads];
    extern __shared__ __align__(16) float s_taps[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sub = lane >> 2, ix = lane & 3;   // group of lanes, its pair of footprint rows
    int4* w_rec = s_rec + warp * 32;
    const unsigned long long n_items = *a.n_items;
    // thread 0: the footprint of `item` into buffer `buf`
    auto issue = [&](int item, int buf) {
        const int64_t bin = a.items[item].x;
        const int64_t c = bin / a.ntiles, T = bin % a.ntiles;
        const int gx0 = (int)((T / a.nty) * kTile), gy0 = (int)((T % a.nty) * kTile);
        mbar_expect_tx(&s_bar[buf], kBoxBytes);
        tensor_load_3d(&s_g[buf][0], &gmap, 2 * gy0, gx0, (int)c, &s_bar[buf]);
    };
    if (tid == 0) {
        for (int k = 0; k < 3; ++k) mbar_init(&s_bar[k], 1);
        mbar_fence_init();
        mbar_expect_tx(&s_bar[2], a.taps8_bytes);
        bulk_load(s_taps, a.taps8, a.taps8_bytes, &s_bar[2]);
        const int first = (int)atomicAdd(a.item_counter, 1u);
        s_item[0] = first;
        if (TMA) {
            tensormap_prefetch(&gmap);
            if ((unsigned long long)first < n_items) issue(first, 0);
        }
    }
    __syncthreads();
    if (!__syncthreads_and(mbar_wait(&s_bar[2], 0, a.wait_polls))) {
        if (tid == 0) {
            atomicExch(a.status, CR_TIMEOUT);
            // let this block's copies in flight land before it exits
            mbar_wait(&s_bar[2], 0);
            if (TMA && (unsigned long long)s_item[0] < n_items) mbar_wait(&s_bar[0], 0);
        }
        return;
    }
    uint32_t phase = 0u;   // bit k: parity of buffer k's next phase
    int b = 0;
    for (;;) {
        const int64_t item = s_item[b];
        if ((unsigned long long)item >= n_items) break;
        if (TMA) {
            if (tid == 0) {
                const int next = (int)atomicAdd(a.item_counter, 1u);
                s_item[b ^ 1] = next;
                if ((unsigned long long)next < n_items) issue(next, b ^ 1);
            }
        } else if (tid == 0) {
            s_item[b ^ 1] = (int)atomicAdd(a.item_counter, 1u);
        }
        const uint2 it = a.items[item];
        const int64_t bin = it.x;
        const uint32_t lo = a.bin_start[bin] + it.y * kDegridChunk;
        const uint32_t hi = min(a.bin_start[bin + 1], lo + kDegridChunk);
        const float2* sg = &s_g[TMA ? b : 0][0];
        if (TMA) {
            if (!__syncthreads_and(mbar_wait(&s_bar[b], (phase >> b) & 1u, a.wait_polls))) {
                if (tid == 0) {
                    atomicExch(a.status, CR_TIMEOUT);
                    // let this block's copies in flight land before it exits
                    mbar_wait(&s_bar[b], (phase >> b) & 1u);
                    if ((unsigned long long)s_item[b ^ 1] < n_items)
                        mbar_wait(&s_bar[b ^ 1], (phase >> (b ^ 1)) & 1u);
                }
                return;
            }
            phase ^= 1u << b;
        } else {
            const int64_t c = bin / a.ntiles, T = bin % a.ntiles;
            const int64_t gx0 = (T / a.nty) * kTile, gy0 = (T % a.nty) * kTile;
            const float2* g = a.grid + c * a.gnx * a.gny;
            for (int k = tid; k < kFoot * kFoot; k += kCubeThreads) {
                const int fx = k / kFoot, fy = k % kFoot;
                const int64_t x = gx0 + fx, y = gy0 + fy;
                float2 v = make_float2(0.0f, 0.0f);
                if (x < a.gnx && y < a.gny) v = __ldg(&g[x * a.gny + y]);
                s_g[0][fx * kPitch + fy] = v;
            }
            __syncthreads();
        }
        // each warp takes a contiguous share of the item's records
        const uint32_t n = hi - lo, share = (n + kCubeThreads - 1) / kCubeThreads * 32u;
        const uint32_t w0 = lo + min(n, warp * share), w1 = lo + min(n, (warp + 1) * share);
        // this lane's two rows of the 7 x 7 cells at `held`, two columns to a pair
        float2 row_re[2][4], row_im[2][4];
        int held = -1;
#pragma unroll
        for (int t = 0; t < 8; ++t)
            row_re[t >> 2][t & 3] = row_im[t >> 2][t & 3] = make_float2(0.0f, 0.0f);
        // records are loaded a batch ahead of their use, one per lane
        uint4 qn = make_uint4(0u, 0u, 0u, 0u);
        float wn = 0.0f;
        if (w0 + lane < w1) {
            qn = a.rec[w0 + lane];
            if (RESIDUAL) wn = a.rec_w[w0 + lane];
        }
#pragma unroll 1
        for (uint32_t base = w0; base < w1; base += 32) {
            const uint32_t k = base + lane;
            const uint4 q = qn;
            const float w = wn;
            __syncwarp();
            w_rec[lane] = make_int4((int)(q.x >> 27) * kPitch + (int)((q.x >> 22) & 31u),
                                    (int)((q.x >> 11) & 2047u) * 8, (int)(q.x & 2047u) * 8, 0);
            __syncwarp();
            if (k + 32 < w1) {
                qn = a.rec[k + 32];
                if (RESIDUAL) wn = a.rec_w[k + 32];
            }
            float re[4], im[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int4 A = w_rec[j * 8 + sub];
                if (A.x != held) {
                    held = A.x;
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (2 * ix + h < 7) {
                            const float2* cell = sg + held + (2 * ix + h) * kPitch;
#pragma unroll
                            for (int t = 0; t < 4; ++t) {
                                const float2 g0 = cell[2 * t];
                                const float2 g1 =
                                    t < 3 ? cell[2 * t + 1] : make_float2(0.0f, 0.0f);
                                row_re[h][t] = make_float2(g0.x, g1.x);
                                row_im[h][t] = make_float2(g0.y, g1.y);
                            }
                        }
                    }
                }
                const float2 wx = *reinterpret_cast<const float2*>(s_taps + A.y + 2 * ix);
                const float4* wy = reinterpret_cast<const float4*>(s_taps + A.z);
                const float4 y0 = wy[0], y1 = wy[1];
                const float2 y[4] = {make_float2(y0.x, y0.y), make_float2(y0.z, y0.w),
                                     make_float2(y1.x, y1.y), make_float2(y1.z, y1.w)};
                float2 r[2], i[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    r[h] = __fmul2_rn(row_re[h][0], y[0]);
                    i[h] = __fmul2_rn(row_im[h][0], y[0]);
#pragma unroll
                    for (int t = 1; t < 4; ++t) {
                        r[h] = __ffma2_rn(row_re[h][t], y[t], r[h]);
                        i[h] = __ffma2_rn(row_im[h][t], y[t], i[h]);
                    }
                }
                re[j] = __fmaf_rn(__fadd_rn(r[1].x, r[1].y), wx.y,
                                  __fmul_rn(__fadd_rn(r[0].x, r[0].y), wx.x));
                im[j] = __fmaf_rn(__fadd_rn(i[1].x, i[1].y), wx.y,
                                  __fmul_rn(__fadd_rn(i[0].x, i[0].y), wx.x));
            }
            // the rows' sums: lane ix of group `sub` ends with record 8 ix + sub,
            // which then goes to its own lane
#pragma unroll
            for (int o = 2; o > 0; o >>= 1) {
                const bool up = ix & o;
#pragma unroll
                for (int t = 0; t < o; ++t) {
                    re[t] = (up ? re[t + o] : re[t]) +
                            __shfl_xor_sync(0xffffffffu, up ? re[t] : re[t + o], o);
                    im[t] = (up ? im[t + o] : im[t]) +
                            __shfl_xor_sync(0xffffffffu, up ? im[t] : im[t + o], o);
                }
            }
            const int from = 4 * (lane & 7) + (lane >> 3);
            re[0] = __shfl_sync(0xffffffffu, re[0], from);
            im[0] = __shfl_sync(0xffffffffu, im[0], from);
            if (k < w1) {
                if (RESIDUAL) {
                    a.res[k] = make_float2(__fsub_rn(__uint_as_float(q.z), __fmul_rn(w, re[0])),
                                           __fsub_rn(__uint_as_float(q.w), __fmul_rn(w, im[0])));
                } else if (q.y != kNullSample) {
                    a.pred[q.y] = make_float2(re[0], im[0]);
                }
            }
        }
        __syncthreads();
        b ^= 1;
    }
}

// Per-sample plan of every channel (start cells, tap rows, imaging weight).
__global__ void __launch_bounds__(kCubeThreads) cube_taps_kernel(const __grid_constant__ CubeArgs a,
                                                                 CubeTaps t) {
    const int c = blockIdx.y;
    const DfChan ch = df_chan(a, c);
    const float f2 = a.mode == CR_WEIGHT_BRIGGS ? a.f2[c] : 0.0f;
    const int64_t r0 = (int64_t)blockIdx.x * kRowsPerBlock;
    const int64_t r1 = min(a.R, r0 + kRowsPerBlock);
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    for (int64_t base = r0 + wp * kWarpRows; base < r1; base += kCubeThreads * kVec) {
        Eval ev[kVec];
        eval_samples(a, ch, f2, c, base + lane, r1, ev);
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
            const int64_t r = base + lane + 32 * j;
            if (r >= r1) continue;
            const int64_t i = (int64_t)c * a.R + r;
            const Eval e = ev[j];
            if (e.ok) {
                const int64_t tx = e.tile / a.nty, ty = e.tile % a.nty;
                t.start_x[i] = (int32_t)(tx * kTile + (e.meta >> 27));
                t.start_y[i] = (int32_t)(ty * kTile + ((e.meta >> 22) & 31));
                t.row_x[i] = (int32_t)((e.meta >> 11) & 2047u);
                t.row_y[i] = (int32_t)(e.meta & 2047u);
                t.weight[i] = e.w;
            } else {
                t.start_x[i] = t.start_y[i] = t.row_x[i] = t.row_y[i] = -1;
                t.weight[i] = 0.0f;
            }
        }
    }
}

}  // namespace

void cube_upload_channels(cr_ctx* ctx, cr_gridder* g, const CubeInput& in) {
    const cr_grid_info& gi = g->info;
    const double dus = (double)g->geom.nx * g->geom.cell_x_rad;
    const double dvs = (double)g->geom.ny * g->geom.cell_y_rad;
    std::vector<CubeChan> chh((size_t)in.C);
    for (int c = 0; c < in.C; ++c) {
        const double s = in.lambda_scale[c];
        if (!(std::isfinite(s) && s > 0.0)) fail(CR_INVALID, "lambda_scale must be finite and > 0");
        chh[c].lscale = s;
        chh[c].kx = fix_scale_of(s, gi.du, false);
        chh[c].ky = fix_scale_of(s, gi.dv, false);
        chh[c].kdx = fix_scale_of(s, dus, true);
        chh[c].kdy = fix_scale_of(s, dvs, true);
        chh[c].fx = df_scale_of(s, gi.du, false);
        chh[c].fy = df_scale_of(s, gi.dv, false);
        chh[c].fdx = df_scale_of(s, dus, true);
        chh[c].fdy = df_scale_of(s, dvs, true);
    }
    CubeChan* chd = (CubeChan*)workspace(ctx, "cube_chan", chh.size() * sizeof(CubeChan));
    CR_CUDA_CHECK(cudaMemcpyAsync(chd, chh.data(), chh.size() * sizeof(CubeChan),
                                  cudaMemcpyHostToDevice, ctx->stream));
    // the pageable source must outlive the copy
    CR_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
}

// Rows are put in uv order when that pays: the sort costs some 35 us and
// 60 ps a row once, and saves up to 25 ps a sample in every channel where
// many rows share a cell.  Whole calls, in row order / in uv order: 1.26 M
// rows of 256 channels 32.3 / 26.9 ms, of 16 2.27 / 2.11 ms, of 1 414 /
// 505 us; 270,001 rows of 101 channels 3.65 / 3.53 ms; 262,144 rows of 48
// 1.43 / 1.47 ms; 8 M rows of 4 3.78 / 3.75 ms; 50,000 rows of 64 626 / 668 us.
static bool cube_rows_sorted(int64_t R, int32_t C) {
    return C >= 8 && R >= (1 << 18) && R * C >= (1 << 24);
}

CubeRecords cube_plan(cr_ctx* ctx, cr_gridder* g, const CubeInput& in, int32_t mode,
                      float robust, const CubeTaps* taps, Pool* keep) {
    // buffers the records and work lists live in: the plan's own pool when
    // given (a persistent plan), else the context's workspaces
    auto kept = [&](const char* name, size_t bytes) {
        return keep ? pool_alloc(ctx, *keep, name, bytes) : workspace(ctx, name, bytes);
    };
    if (mode != CR_WEIGHT_NATURAL && mode != CR_WEIGHT_UNIFORM && mode != CR_WEIGHT_BRIGGS)
        fail(CR_INVALID, "unknown weighting mode");
    if (in.C <= 0 || in.C > 65535) fail(CR_INVALID, "channels must lie in [1, 65535]");
    if (in.R < 0) fail(CR_INVALID, "negative row count");
    if ((uint64_t)in.C * (uint64_t)in.R >= (1ull << 32))
        fail(CR_INVALID, "cube larger than 2^32 samples");
    const cr_grid_info& gi = g->info;
    if (gi.oversampling > kMaxTapRows - 1) fail(CR_INVALID, "cube oversampling above 254");
    CubeRecords cr{};
    cr.R = in.R;
    cr.C = in.C;
    cr.ntx = (gi.grid_nx + kTile - 1) / kTile;
    cr.nty = (gi.grid_ny + kTile - 1) / kTile;
    cr.ntiles = cr.ntx * cr.nty;
    const int64_t nbins = (int64_t)in.C * cr.ntiles;
    const size_t ns = (size_t)std::max<int64_t>((int64_t)in.C * in.R, 1);
    // per-channel constants (uploaded before a capture by the caller)
    const double dus = (double)g->geom.nx * g->geom.cell_x_rad;
    const double dvs = (double)g->geom.ny * g->geom.cell_y_rad;
    if (!ctx->capturing) cube_upload_channels(ctx, g, in);
    CubeChan* chd = (CubeChan*)workspace(ctx, "cube_chan", (size_t)in.C * sizeof(CubeChan));
    cr.rec = (uint4*)kept("cube_rec", ns * 16);
    cr.rec_w = (float*)kept("cube_rec_w", ns * 4);
    cr.bin_start = (uint32_t*)kept("cube_bin_start", (size_t)(nbins + 1) * 4);
    const int64_t ncells = (nbins << 10) + 1;   // (channel, tile, cell) bins + total
    if (ncells >= (1ll << 32)) fail(CR_INVALID, "cube has too many (channel, tile, cell) bins");
    uint32_t* hist = (uint32_t*)kept("cube_hist", (size_t)ncells * 4);
    cr.sumwt = (double*)kept("cube_sumwt", (size_t)in.C * 8);
    cr.counts = (unsigned long long*)kept("cube_counts", (size_t)in.C * 16 + 8);
    cr.n_rec = cr.counts + 2 * in.C;
    CR_CUDA_CHECK(cudaMemsetAsync(hist, 0, (size_t)ncells * 4, ctx->stream));
    CR_CUDA_CHECK(cudaMemsetAsync(cr.sumwt, 0, (size_t)in.C * 8, ctx->stream));
    CR_CUDA_CHECK(cudaMemsetAsync(cr.counts, 0, (size_t)in.C * 16 + 8, ctx->stream));

    CubeArgs a{};
    a.R = in.R;
    a.C = in.C;
    a.u = in.u;
    a.v = in.v;
    a.ch = chd;
    a.vis = in.vis;
    a.weight = in.weight;
    a.flags = in.flags;
    a.du = gi.du;
    a.dv = gi.dv;
    a.gnx = gi.grid_nx;
    a.gny = gi.grid_ny;
    a.os = gi.oversampling;
    a.tap_rows = g->tap_rows;
    a.ntx = cr.ntx;
    a.nty = cr.nty;
    a.cx_fix = (long long)gi.grid_nx << (kFixF - 1);
    a.cy_fix = (long long)gi.grid_ny << (kFixF - 1);
    a.nx = g->geom.nx;
    a.ny = g->geom.ny;
    a.dus = dus;
    a.dvs = dvs;
    a.dcx = (double)g->geom.nx / 2.0;
    a.dcy = (double)g->geom.ny / 2.0;
    a.dcx_fix = (long long)g->geom.nx << (kFixF - 1);
    a.dcy_fix = (long long)g->geom.ny << (kFixF - 1);
    a.mode = mode;
    a.hist = hist;
    a.cursor = hist;
    a.sumwt = cr.sumwt;
    a.counts = cr.counts;
    a.rec = cr.rec;
    a.rec_w = cr.rec_w;
    const dim3 grid((unsigned)std::max<int64_t>((in.R + kRowsPerBlock - 1) / kRowsPerBlock, 1),
                    (unsigned)in.C);
    float4* uvdf = (float4*)workspace(ctx, "cube_uvdf", (size_t)std::max<int64_t>(in.R, 1) * 16);
    a.ev_tile = (uint32_t*)workspace(ctx, "cube_ev_tile", ns * 4);
    a.ev_meta = (uint32_t*)workspace(ctx, "cube_ev_meta", ns * 4);
    // (a context with an allocation limit keeps the smaller scratch)
    bool sorted = !taps && ctx->alloc_limit == 0 && cube_rows_sorted(in.R, in.C);
    int bits = 10;
    while (((uint64_t)cr.ntiles << 10) >> bits) ++bits;
    // the sort works in the per-sample results' memory, which is not yet in use
    sorted = sorted && radix_sort_bytes(in.R, bits) <= ns * 4;
    const uint32_t* order = nullptr;
    uint32_t* rows = nullptr;
    if (sorted) {
        rows = (uint32_t*)workspace(ctx, "cube_rows", (size_t)in.R * 4);
        double s_max = 0.0;
        for (int c = 0; c < in.C; ++c) s_max = std::max(s_max, in.lambda_scale[c]);
        RadixSort sort = radix_sort_begin(ctx, in.R, bits, a.ev_tile);
        const KeyOut out{sort.keys, sort.hist, sort.passes, nullptr};
        cube_row_keys_kernel<<<grid_blocks(in.R, 256 * 8), 256, 0, ctx->stream>>>(
            in.u, in.v, in.R, s_max / gi.du, s_max / gi.dv, (int32_t)gi.grid_nx,
            (int32_t)gi.grid_ny, (uint32_t)cr.nty, out);
        note_launch(ctx, "cube_row_keys_kernel");
        radix_sort_run(ctx, sort);
        order = sort.order;
    }
    if (in.R > 0) {
        cube_rows_df_kernel<<<grid_blocks(in.R, 256), 256, 0, ctx->stream>>>(
            in.u, in.v, in.R, order, rows, uvdf);
        note_launch(ctx, "cube_rows_df_kernel");
    }
    a.uvdf = uvdf;
    a.rows = rows;
    if (mode == CR_WEIGHT_NATURAL && in.R > 0) {
        if (sorted)
            cube_density_kernel<false, true><<<grid, kCubeThreads, 0, ctx->stream>>>(a);
        else
            cube_density_kernel<false, false><<<grid, kCubeThreads, 0, ctx->stream>>>(a);
        note_launch(ctx, "cube_plan_kernel");
    }
    if (mode != CR_WEIGHT_NATURAL) {
        const int64_t cells = (int64_t)g->geom.nx * g->geom.ny;
        a.density = (float*)workspace(ctx, "cube_density", (size_t)(in.C * cells) * 4);
        a.dcell = (uint32_t*)workspace(ctx, "cube_dcell", ns * 4);
        CR_CUDA_CHECK(cudaMemsetAsync(a.density, 0, (size_t)(in.C * cells) * 4, ctx->stream));
        if (in.R > 0) {
            if (sorted)
                cube_density_kernel<true, true><<<grid, kCubeThreads, 0, ctx->stream>>>(a);
            else
                cube_density_kernel<true, false><<<grid, kCubeThreads, 0, ctx->stream>>>(a);
            note_launch(ctx, "cube_density_kernel");
        }
        float* f2 = (float*)workspace(ctx, "cube_f2", (size_t)in.C * 4);
        if (mode == CR_WEIGHT_BRIGGS) {
            double* sums = (double*)workspace(ctx, "cube_dsums", (size_t)in.C * 16);
            CR_CUDA_CHECK(cudaMemsetAsync(sums, 0, (size_t)in.C * 16, ctx->stream));
            const dim3 sg((unsigned)std::min<int64_t>((cells + 255) / 256, 64), (unsigned)in.C);
            cube_density_sums<<<sg, 256, 0, ctx->stream>>>(a.density, cells, sums);
            note_launch(ctx, "cube_density_sums");
            const double am = 5.0 * std::pow(10.0, -(double)robust);
            cube_f2_kernel<<<(in.C + 127) / 128, 128, 0, ctx->stream>>>(sums, in.C, am * am, f2);
            note_launch(ctx, "cube_f2_kernel");
        }
        a.f2 = f2;
    }
    if (taps) {
        if (in.R > 0) {
            cube_taps_kernel<<<grid, kCubeThreads, 0, ctx->stream>>>(a, *taps);
            note_launch(ctx, "cube_taps_kernel");
        }
        return cr;
    }
    // in place: hist becomes each cell bin's first slot, the scatter's cursor
    exclusive_scan_u32(ctx, hist, hist, ncells, nullptr);
    tile_starts_from_cells<<<grid_blocks(nbins + 1, 256), 256, 0, ctx->stream>>>(hist, nbins,
                                                                                 cr.bin_start);
    note_launch(ctx, "tile_starts_from_cells");
    if (in.R > 0) {
        if (sorted)
            cube_scatter_kernel<true><<<grid, kCubeThreads, 0, ctx->stream>>>(a);
        else
            cube_scatter_kernel<false><<<grid, kCubeThreads, 0, ctx->stream>>>(a);
        note_launch(ctx, "cube_scatter_kernel");
    }
    // work-list buffers (the lists are made by cube_grid / cube_degrid)
    cr.grid_chunks = (uint32_t*)kept("cube_gchunks", (size_t)nbins * 4);
    cr.degrid_chunks = (uint32_t*)kept("cube_dchunks", (size_t)nbins * 4);
    cr.cell_end = hist;
    cr.grid_first = (uint32_t*)kept("cube_gfirst", (size_t)nbins * 4);
    cr.degrid_first = (uint32_t*)kept("cube_dfirst", (size_t)nbins * 4);
    cr.n_items = (unsigned long long*)kept("cube_nitems", 16);
    // sum over tiles of ceil(n / K) <= tiles + (sum n) / K, and each record is a
    // source of at most four output tiles
    const size_t max_grid_items = (size_t)nbins + 4 * ns / kGridChunkMin + 1;
    const size_t max_degrid_items = (size_t)nbins + ns / kDegridChunk + 1;
    cr.grid_items = (uint2*)kept("cube_gitems", max_grid_items * 8);
    cr.degrid_items = (uint2*)kept("cube_ditems", max_degrid_items * 8);
    return cr;
}

// Work lists for one gridding chunk size; with psf/dirty, heavy output tiles
// are zeroed for their atomic chunks.
static void make_work_lists(cr_ctx* ctx, cr_gridder* g, CubeRecords& cr, uint32_t chunk,
                            float* psf, float2* dirty, const uint8_t* plane_mask = nullptr) {
    const cr_grid_info& gi = g->info;
    const int64_t nbins = (int64_t)cr.C * cr.ntiles;
    cube_work_count<<<grid_blocks(nbins, 256), 256, 0, ctx->stream>>>(
        cr.bin_start, cr.cell_end, nbins, cr.ntiles, cr.nty, chunk, plane_mask, cr.grid_chunks,
        cr.degrid_chunks);
    note_launch(ctx, "cube_work_count");
    exclusive_scan_u32(ctx, cr.grid_chunks, cr.grid_first, nbins, cr.n_items);
    exclusive_scan_u32(ctx, cr.degrid_chunks, cr.degrid_first, nbins, cr.n_items + 1);
    cube_work_fill<<<grid_blocks(nbins, 256), 256, 0, ctx->stream>>>(
        cr.grid_chunks, cr.grid_first, cr.degrid_chunks, cr.degrid_first, nbins, cr.grid_items,
        cr.degrid_items);
    note_launch(ctx, "cube_work_fill");
    if (dirty) {
        cube_zero_heavy<<<grid_blocks(nbins * 32, 256), 256, 0, ctx->stream>>>(
            cr.grid_chunks, nbins, cr.ntiles, cr.nty, gi.grid_nx, gi.grid_ny, psf, dirty);
        note_launch(ctx, "cube_zero_heavy");
    }
    cr.grid_chunk = chunk;
    cr.fill_done = true;
    cr.lists_masked = plane_mask != nullptr;
}

template <bool RESIDUAL>
static void launch_cube_grid(cr_ctx* ctx, cr_gridder* g, const CubeRecords& cr, float* psf,
                             float2* dirty, const float2* res = nullptr) {
    const cr_grid_info& gi = g->info;
    unsigned int* counter = (unsigned int*)workspace(ctx, "cube_counter", 8);
    CR_CUDA_CHECK(cudaMemsetAsync(counter, 0, 8, ctx->stream));
    CubeGridArgs a{cr.rec, cr.rec_w, cr.bin_start, cr.cell_end, g->taps8_d, g->tap_rows,
                   (uint32_t)g->tap_rows * 32u, ctx->status_d, cr.ntx, cr.nty, gi.grid_nx,
                   gi.grid_ny, cr.grid_items, cr.grid_chunk, cr.grid_chunks, cr.n_items,
                   counter, psf, dirty, res, ctx->mbar_polls};
    int sms = 0;
    CR_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    int per_sm = 0;
    CR_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &per_sm, cube_grid_kernel<RESIDUAL>, kGridThreads, 0));
    cube_grid_kernel<RESIDUAL><<<sms * std::max(per_sm, 1), kGridThreads, 0, ctx->stream>>>(a);
    note_launch(ctx, RESIDUAL ? "cube_grid_kernel_residual" : "cube_grid_kernel");
}

static std::string cube_shape_key(const cr_gridder* g, const CubeRecords& cr) {
    return std::to_string(cr.C) + "x" + std::to_string(cr.ntx) + "x" + std::to_string(cr.nty) +
           "/" + std::to_string(g->info.oversampling);
}

bool cube_grid_chunk_valid(uint32_t chunk) {
    for (uint32_t c : kGridChunkCandidates)
        if (c == chunk) return true;
    return false;
}

void cube_grid(cr_ctx* ctx, cr_gridder* g, CubeRecords& cr, float* psf, float2* dirty) {
    const std::string key = cube_shape_key(g, cr);
    auto tuned = ctx->cube_chunk.find(key);
    if (tuned == ctx->cube_chunk.end() && !ctx->capturing && !ctx->cube_chunk_forced) {
        // first use of this cube shape: time the gridding pass (work lists
        // and kernel) for every candidate chunk size and keep the fastest
        cudaEvent_t e0 = ctx->kev[0], e1 = ctx->kev[1];
        float best_ms = 0.0f;
        uint32_t best = kGridChunkDefault;
        for (uint32_t chunk : kGridChunkCandidates) {
            CR_CUDA_CHECK(cudaEventRecord(e0, ctx->stream));
            make_work_lists(ctx, g, cr, chunk, psf, dirty);
            launch_cube_grid<false>(ctx, g, cr, psf, dirty);
            CR_CUDA_CHECK(cudaEventRecord(e1, ctx->stream));
            CR_CUDA_CHECK(cudaEventSynchronize(e1));
            float ms = 0.0f;
            CR_CUDA_CHECK(cudaEventElapsedTime(&ms, e0, e1));
            if (chunk == kGridChunkCandidates[0] || ms < best_ms) {
                best_ms = ms;
                best = chunk;
            }
        }
        ctx->cube_chunk[key] = best;
        tuned = ctx->cube_chunk.find(key);
    }
    uint32_t chunk = tuned != ctx->cube_chunk.end() ? tuned->second : kGridChunkDefault;
    if (ctx->cube_chunk_forced) chunk = ctx->cube_chunk_forced;
    make_work_lists(ctx, g, cr, chunk, psf, dirty);
    kernel_mark(ctx, 0, false);
    launch_cube_grid<false>(ctx, g, cr, psf, dirty);
    kernel_mark(ctx, 0, true);
}

template <bool RESIDUAL>
static void launch_cube_degrid(cr_ctx* ctx, cr_gridder* g, const CubeRecords& cr,
                               const float2* grid, float2* pred, float2* res) {
    const cr_grid_info& gi = g->info;
    unsigned int* counter = (unsigned int*)workspace(ctx, "cube_counter", 8);
    CR_CUDA_CHECK(cudaMemsetAsync(counter, 0, 8, ctx->stream));
    const uint32_t taps8_bytes = (uint32_t)g->tap_rows * 32u;
    CubeDegridArgs a{cr.rec, cr.bin_start, g->tap_rows, cr.ntiles, cr.nty, gi.grid_nx,
                     gi.grid_ny, cr.R, cr.degrid_items, cr.n_items + 1, counter, g->taps8_d,
                     taps8_bytes, grid, pred, cr.rec_w, res, ctx->status_d, ctx->mbar_polls};
    int sms = 0;
    CR_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    // the grids as float32 [C][gnx][2 gny] for footprint boxes of 76 x 38
    CUtensorMap map;
    std::memset(&map, 0, sizeof(map));
    const uint64_t row = (uint64_t)gi.grid_ny * 8;
    const bool tma = encode_tensor_map_3d(&map, grid, 2 * (uint64_t)gi.grid_ny,
                                          (uint64_t)gi.grid_nx, (uint64_t)cr.C, row,
                                          row * (uint64_t)gi.grid_nx, 2 * (kTile + 6), kTile + 6);
    if (tma)
        cube_degrid_kernel<RESIDUAL, true>
            <<<sms * kDegridBlocks, kCubeThreads, taps8_bytes, ctx->stream>>>(map, a);
    else
        cube_degrid_kernel<RESIDUAL, false>
            <<<sms * kDegridBlocks, kCubeThreads, taps8_bytes, ctx->stream>>>(map, a);
    note_launch(ctx, RESIDUAL ? "cube_degrid_kernel_residual" : "cube_degrid_kernel");
}

void cube_grid_residual(cr_ctx* ctx, cr_gridder* g, CubeRecords& cr, const float2* model,
                        float2* residual, const uint8_t* plane_mask) {
    auto tuned = ctx->cube_chunk.find(cube_shape_key(g, cr));
    uint32_t chunk = tuned != ctx->cube_chunk.end() ? tuned->second : kGridChunkDefault;
    if (ctx->cube_chunk_forced) chunk = ctx->cube_chunk_forced;
    // the lists skip masked planes and zero the heavy tiles of the others
    make_work_lists(ctx, g, cr, chunk, nullptr, residual, plane_mask);
    const size_t nrec = cr.n_records >= 0 ? (size_t)std::max<int64_t>(cr.n_records, 1)
                                          : (size_t)std::max<int64_t>((int64_t)cr.C * cr.R, 1);
    float2* res = (float2*)workspace(ctx, "cube_res", nrec * 8);
    kernel_mark(ctx, 1, false);
    launch_cube_degrid<true>(ctx, g, cr, model, nullptr, res);
    kernel_mark(ctx, 1, true);
    kernel_mark(ctx, 0, false);
    launch_cube_grid<true>(ctx, g, cr, nullptr, residual, res);
    kernel_mark(ctx, 0, true);
}

void cube_degrid(cr_ctx* ctx, cr_gridder* g, CubeRecords& cr, const float2* grid,
                 float2* pred) {
    CR_CUDA_CHECK(cudaMemsetAsync(pred, 0, (size_t)cr.C * cr.R * 8, ctx->stream));
    // the degridding work list without a gridding pass before it
    if (!cr.fill_done || cr.lists_masked)
        make_work_lists(ctx, g, cr, cr.fill_done ? cr.grid_chunk : kGridChunkDefault, nullptr,
                        nullptr);
    kernel_mark(ctx, 1, false);
    launch_cube_degrid<false>(ctx, g, cr, grid, pred, nullptr);
    kernel_mark(ctx, 1, true);
}

void cube_read_sums(cr_ctx* ctx, const CubeRecords& cr, cr_sums* out) {
    if (!out) return;
    std::vector<double> sw((size_t)cr.C);
    std::vector<unsigned long long> cnt((size_t)cr.C * 2);
    CR_CUDA_CHECK(cudaMemcpyAsync(sw.data(), cr.sumwt, sw.size() * 8, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    CR_CUDA_CHECK(cudaMemcpyAsync(cnt.data(), cr.counts, cnt.size() * 8, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    CR_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    for (int c = 0; c < cr.C; ++c) {
        out[c].normalization_sumwt = sw[c];
        out[c].reported_sumwt = sw[c];
        out[c].gridded = (int64_t)cnt[2 * c];
        out[c].skipped = (int64_t)cnt[2 * c + 1];
        out[c].unique_records = (int64_t)cnt[2 * c];
        out[c].taps = 49 * (int64_t)cnt[2 * c];
    }
}

}  // namespace cr
