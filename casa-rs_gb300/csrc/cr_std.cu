// cr_std.cu -- standard (prolate-spheroidal, 7 x 7 taps) gridding and
// degridding over deduplicated records.
//
// Gridding restates grid_sample_taps_real_complex_pair_planned_f64
// (gridder.rs:1021-1071): PSF += gw * wx*wy and dirty += vis*gw * wx*wy, the
// value times wx rounded in float32 before wy.  A warp sums the taps of
// consecutive records with one start cell in registers and adds them once per
// run to the home tile's 38 x 38 footprint in shared memory, which is flushed to
// the grid with FP32 atomics.
// Degridding restates degrid_sample_taps_planned_normalized
// (gridder.rs:1278-1312) with a warp per record.
#include "cr_fixed.cuh"
#include "cr_internal.cuh"
#include "cr_runs.cuh"

namespace cr {

namespace {

constexpr int kStdThreads = 256;
constexpr int kFoot = kTile + 6;   // 38
// footprint rows 39 cells apart (= 7 mod 32), so that the seven rows of a
// footprint fall in different banks
constexpr int kFootRow = 39;
constexpr int kStdMaxTaps = 255 * 8;   // oversampling up to 254
constexpr int kStdBlocksPerSm = 4;
// Work is measured in records, a home tile's flush counting as kStdTileCost
// of them: tile T's records lie at positions tile_start[T] + kStdTileCost T
// onwards.  An item is a range of positions, found by a search over the
// tiles, so no work list is built.  Items hold at least kStdMinItem positions
// (more blocks per tile would also mean more roundings at the size of the
// grid's sums) and at most kStdMaxItem, so that they spread over the blocks.
constexpr int kStdTileCost = 256;
constexpr int kStdMinItem = 512;
constexpr int kStdMaxItem = 4096;

struct StdGridArgs {
    const int2* xy;
    const uint32_t* meta;
    const float4* vsum;
    const float2* wsum;
    const float2* pred;
    const uint32_t* tile_start;
    const unsigned long long* counts;
    int64_t ntiles, nty;
    const float* taps;
    int32_t tap_floats;
    float* psf;
    int psf_step;
    float2* dirty;
    int64_t gnx, gny;
};

// Bound by the issue of the per-record work and, for small batches, by its
// latency.  Records are summed by runs of one start cell, four at a time
// (cr_runs.cuh).  4,001 samples of a 256^2 image, 126,360 (512^2) and 5.0 M
// (3000^2): 18, 17 and 140 us; with a lane per tap, and a shared-memory add
// per tap and run, 16, 18 and 261; with one add per tap and record, chunks of
// 2048 records of one tile and a work list, 68, 137 and 511.
template <bool RESIDUAL>
__global__ void __launch_bounds__(kStdThreads, kStdBlocksPerSm) std_grid_kernel(StdGridArgs a) {
    __shared__ float s_psf[RESIDUAL ? 1 : kFoot * kFootRow];
    __shared__ __align__(8) float2 s_ri[kFoot * kFootRow];
    __shared__ __align__(16) float s_taps[kStdMaxTaps];
    // per warp, 32 decoded records: {cell of the tile, tap row offsets,
    // weight} and the value
    __shared__ __align__(16) int4 s_ra[kStdThreads];
    __shared__ float2 s_rb[kStdThreads];
    constexpr int kComps = RESIDUAL ? 2 : 3;
    constexpr uint32_t kDone = ~0u;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t nrec = (int64_t)a.counts[2];
    const int64_t span = nrec + kStdTileCost * a.ntiles;
    const int64_t item = min((int64_t)kStdMaxItem,
                             max((int64_t)kStdMinItem,
                                 (span + 4 * gridDim.x - 1) / (4 * (int64_t)gridDim.x)));
    if (nrec == 0 || blockIdx.x * item >= span) return;
    for (int k = tid; k < a.tap_floats; k += kStdThreads) s_taps[k] = a.taps[k];
    for (int c = tid; c < kFoot * kFootRow; c += kStdThreads) {
        if (!RESIDUAL) s_psf[c] = 0.0f;
        s_ri[c] = make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    const int grp = lane >> 3, ix = lane & 7;
    const float* tap_x = s_taps + ix;
    RunSums<kComps> sums;
    int4* w_ra = s_ra + warp * 32;
    float2* w_rb = s_rb + warp * 32;
    for (int64_t v0 = blockIdx.x * item; v0 < span; v0 += gridDim.x * item) {
        const int64_t v1 = v0 + item;
        // the last tile whose position is <= v0, 256 probes at a time
        int64_t lo = 0, len = a.ntiles;
        while (len > 1) {
            const int64_t step = (len + kStdThreads - 1) / kStdThreads, T = lo + tid * step;
            const int below = __syncthreads_count(
                tid * step < len && (int64_t)a.tile_start[T] + kStdTileCost * T <= v0);
            lo += (below - 1) * step;
            len = min(step, len - (below - 1) * step);
        }
        int64_t s = a.tile_start[lo];
        s = min(s + (v0 - s - kStdTileCost * lo), (int64_t)a.tile_start[lo + 1]);
        while (s < nrec) {
            const int2 p = a.xy[s];
            const int x0 = p.x & ~31, y0 = p.y & ~31;
            const int64_t T = (p.x >> 5) * a.nty + (p.y >> 5);
            const int64_t e = min((int64_t)a.tile_start[T + 1], v1 - kStdTileCost * T);
            if (e <= s) break;   // the tile begins past the item's end
            const bool more = e == a.tile_start[T + 1];
            // each warp takes a contiguous share of the tile's records
            const uint32_t n = (uint32_t)(e - s), kWarps = kStdThreads / 32;
            const uint32_t share = max(32u, (n + 4 * kWarps - 1) / (4 * kWarps) * 4u);
            const uint32_t w0 = (uint32_t)s + min(n, warp * share);
            const uint32_t w1 = (uint32_t)s + min(n, (warp + 1) * share);
            uint32_t open = kDone - 1;   // the run's cell; none yet
            auto flush = [&]() {
                float v[kComps][2];
                sums.exchange(lane, v);
                const int c = ((open >> 5) + ix) * kFootRow + (open & 31u) + 2 * grp;
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    if (ix < 7 && 2 * grp + t < 7) {
                        if (!RESIDUAL) atomicAdd(&s_psf[c + t], v[0][t]);
                        shared_add2(&s_ri[c + t], v[kComps - 2][t], v[kComps - 1][t]);
                    }
                }
            };
            sums.clear();
#pragma unroll 1
            for (uint32_t g = w0; g < w1; g += 32) {
                const uint32_t r = g + lane;
                int4 ra = make_int4((int)kDone, 0, 0, 0);
                float2 val = make_float2(0.0f, 0.0f);
                if (r < w1) {
                    const int2 q = a.xy[r];
                    const uint32_t m = a.meta[r];
                    const float4 v = a.vsum[r];
                    const float2 w = a.wsum[r];
                    val = make_float2(v.x, v.z);
                    if (RESIDUAL) val = residual_value(v, w, a.pred[r]);
                    ra = make_int4((q.x & 31) << 5 | (q.y & 31), (int)(m & 0xffffu) * 8,
                                   (int)(m >> 16) * 8, __float_as_int(w.x));
                }
                __syncwarp();   // the slots' last readers are done
                w_ra[lane] = ra;
                w_rb[lane] = val;
                __syncwarp();
                const int nb = (int)min(32u, w1 - g);
#pragma unroll 1
                for (int k = grp; k - grp < nb; k += 4) {
                    const int4 A = w_ra[k];
                    const float2 B = w_rb[k];
                    uint32_t cell = (uint32_t)A.x;
                    const float wx = tap_x[A.y];
                    float2 y[4];
                    tap_pairs(s_taps + A.z, y);
                    // the groups' records belong to the run, or end it
                    for (;;) {
                        const bool mine = cell == open;
                        const unsigned match = __ballot_sync(0xffffffffu, mine);
                        if (match) {
                            sums.add(mine, wx, y, __int_as_float(A.w), B);
                            if (match == 0xffffffffu) break;
                            if (mine) cell = kDone;
                        }
                        const unsigned rest = __ballot_sync(0xffffffffu, cell != kDone);
                        if (!rest) break;
                        if (open != kDone - 1) {
                            flush();
                            sums.clear();
                        }
                        open = __shfl_sync(0xffffffffu, cell, __ffs(rest) - 1);
                    }
                }
            }
            if (open != kDone - 1) flush();
            __syncthreads();
            for (int k = tid; k < kFoot * kFoot; k += kStdThreads) {
                const int fx = k / kFoot, fy = k - fx * kFoot, c = fx * kFootRow + fy;
                const int64_t cell = (int64_t)(x0 + fx) * a.gny + (y0 + fy);
                const float2 d = s_ri[c];
                // cells past the grid's edge hold zeros
                if (!RESIDUAL && s_psf[c] != 0.0f) {
                    atomicAdd(&a.psf[cell * a.psf_step], s_psf[c]);
                    s_psf[c] = 0.0f;
                }
                if (d.x != 0.0f || d.y != 0.0f) {
                    atomicAdd(&a.dirty[cell], d);
                    s_ri[c] = make_float2(0.0f, 0.0f);
                }
            }
            __syncthreads();
            if (!more) break;
            s = e;
        }
    }
}

struct StdDegridArgs {
    const int2* xy;
    const uint32_t* meta;
    const unsigned long long* counts;
    const float* taps;
    const float2* grid;
    int64_t gny;
    float2* pred;
};

__global__ void __launch_bounds__(256) std_degrid_kernel(StdDegridArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t nrec = (int64_t)a.counts[2];
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < nrec;
         r += nwarps) {
        const int2 p = a.xy[r];
        const uint32_t m = a.meta[r];
        const float* wx = a.taps + (m & 0xffffu) * 7;
        const float* wy = a.taps + (m >> 16) * 7;
        const float2* g = a.grid + (int64_t)p.x * a.gny + p.y;
        float re = 0.f, im = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int t = lane + 32 * h;
            if (t < 49) {
                int tx = t / 7, ty = t - 7 * (t / 7);
                float wgt = __fmul_rn(__ldg(&wx[tx]), __ldg(&wy[ty]));
                float2 gv = g[(int64_t)tx * a.gny + ty];
                re = fmaf(gv.x, wgt, re);
                im = fmaf(gv.y, wgt, im);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            re += __shfl_xor_sync(0xffffffffu, re, o);
            im += __shfl_xor_sync(0xffffffffu, im, o);
        }
        if (lane == 0) a.pred[r] = make_float2(re, im);
    }
}

}  // namespace

void std_grid(cr_ctx* ctx, cr_gridder* g, const Records& r, float* psf, int psf_step,
              float2* dirty, int mode) {
    StdGridArgs a{r.rec_xy, r.rec_meta, r.rec_vsum, r.rec_wsum, r.rec_pred, r.tile_start,
                  r.counts, r.ntx * r.nty, r.nty, g->taps8_d, g->tap_rows * 8, psf, psf_step, dirty,
                  g->info.grid_nx, g->info.grid_ny};
    const unsigned blocks = (unsigned)(ctx->sms * kStdBlocksPerSm);
    kernel_mark(ctx, 0, false);
    if (mode == 0) {
        std_grid_kernel<false><<<blocks, kStdThreads, 0, ctx->stream>>>(a);
        note_launch(ctx, "std_grid_kernel");
    } else {
        std_grid_kernel<true><<<blocks, kStdThreads, 0, ctx->stream>>>(a);
        note_launch(ctx, "std_grid_kernel_residual");
    }
    kernel_mark(ctx, 0, true);
}

void std_degrid(cr_ctx* ctx, cr_gridder* g, const Records& r, const float2* grid) {
    StdDegridArgs a{r.rec_xy, r.rec_meta, r.counts, g->taps_d, grid,
                    g->info.grid_ny, r.rec_pred};
    kernel_mark(ctx, 1, false);
    std_degrid_kernel<<<ctx->sms * 8, 256, 0, ctx->stream>>>(a);
    note_launch(ctx, "std_degrid_kernel");
    kernel_mark(ctx, 1, true);
}

}  // namespace cr
