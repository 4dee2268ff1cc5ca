// cr_std.cu -- standard (prolate-spheroidal, 7 x 7 taps) gridding and
// degridding over deduplicated records.
//
// Gridding restates grid_sample_taps_real_complex_pair_planned_f64
// (gridder.rs:1021-1071): PSF += gw * wx*wy and dirty += vis*gw * wx*wy, the
// tap product wx*wy rounded in float32.  A warp sums the taps of consecutive
// records with one start cell in registers and adds them once per run to the
// home tile's 38 x 38 footprint in shared memory, which is flushed to the grid
// with FP32 atomics.
// Degridding restates degrid_sample_taps_planned_normalized
// (gridder.rs:1278-1312) with a warp per record.
#include "cr_fixed.cuh"
#include "cr_internal.cuh"

namespace cr {

namespace {

constexpr int kStdThreads = 256;
constexpr int kFoot = kTile + 6;   // 38
// footprint rows 39 floats apart (= 7 mod 32): the 49 taps of a record hit
// distinct banks within each warp-wide atomic
constexpr int kFootRow = 39;
constexpr int kStdMaxTaps = 255 * 7;   // oversampling up to 254
constexpr int kStdBlocksPerSm = 6;
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

// Bound by the issue of the per-record work (two tap slots per lane) and by
// shared-memory atomics per run.  With one atomic per tap and record, chunks of
// 2048 records of one tile and a work list: 68 us for 4,001 samples of a 256^2
// image, 137 for 126,360 (512^2), 511 for 5.0 M (3000^2); now 16, 18 and 265.
template <bool RESIDUAL>
__global__ void __launch_bounds__(kStdThreads) std_grid_kernel(StdGridArgs a) {
    __shared__ float s_psf[RESIDUAL ? 1 : kFoot * kFootRow];
    __shared__ float s_dr[kFoot * kFootRow];
    __shared__ float s_di[kFoot * kFootRow];
    __shared__ float s_taps[kStdMaxTaps];
    // per warp, 32 decoded records: {start cell, tap row offsets, weight}
    // and the value
    __shared__ int4 s_ra[kStdThreads];
    __shared__ float2 s_rb[kStdThreads];
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
        s_dr[c] = 0.0f;
        s_di[c] = 0.0f;
    }
    __syncthreads();
    // lane t holds taps t (slot 0) and t + 32 (slot 1, lanes 0-16; the other
    // lanes form a dummy product that is never added)
    const int ix0 = lane / 7, iy0 = lane % 7;
    const bool has1 = lane + 32 < 49;
    const int ix1 = has1 ? (lane + 32) / 7 : 0, iy1 = has1 ? (lane + 32) % 7 : 0;
    const int off0 = ix0 * kFootRow + iy0, off1 = ix1 * kFootRow + iy1;
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
            bool open = false;   // a run is being summed
            int cx = 0, cy = 0;
            // (psf slot 0, slot 1), (re, im) slot 0, (re, im) slot 1
            float2 pp = make_float2(0.f, 0.f), ri0 = pp, ri1 = pp;
            auto flush = [&]() {
                const int b = (cx - x0) * kFootRow + (cy - y0);
                if (!RESIDUAL) atomicAdd(&s_psf[b + off0], pp.x);
                atomicAdd(&s_dr[b + off0], ri0.x);
                atomicAdd(&s_di[b + off0], ri0.y);
                if (has1) {
                    if (!RESIDUAL) atomicAdd(&s_psf[b + off1], pp.y);
                    atomicAdd(&s_dr[b + off1], ri1.x);
                    atomicAdd(&s_di[b + off1], ri1.y);
                }
            };
            for (int64_t g = s + warp * 32; g < e; g += kStdThreads) {
                const int64_t r = g + lane;
                if (r < e) {
                    const int2 q = a.xy[r];
                    const uint32_t m = a.meta[r];
                    const float4 v = a.vsum[r];
                    const float2 w = a.wsum[r];
                    float2 val = make_float2(v.x, v.z);
                    if (RESIDUAL) val = residual_value(v, w, a.pred[r]);
                    w_ra[lane] = make_int4(q.x, q.y, (int)((m & 0xffffu) * 7u | ((m >> 16) * 7u) << 16),
                                           __float_as_int(w.x));
                    w_rb[lane] = val;
                }
                __syncwarp();
                const int n = (int)min((int64_t)32, e - g);
                for (int k = 0; k < n; ++k) {
                    const int4 A = w_ra[k];
                    const float2 B = w_rb[k];
                    if (!open || A.x != cx || A.y != cy) {
                        if (open) flush();
                        open = true;
                        cx = A.x;
                        cy = A.y;
                        pp = ri0 = ri1 = make_float2(0.f, 0.f);
                    }
                    const float* wx = s_taps + (A.z & 0xffff);
                    const float* wy = s_taps + ((unsigned)A.z >> 16);
                    const float pw = __int_as_float(A.w);
                    const float2 w = __fmul2_rn(make_float2(wx[ix0], wx[ix1]),
                                                make_float2(wy[iy0], wy[iy1]));
                    if (!RESIDUAL) pp = __ffma2_rn(make_float2(pw, pw), w, pp);
                    ri0 = __ffma2_rn(B, make_float2(w.x, w.x), ri0);
                    ri1 = __ffma2_rn(B, make_float2(w.y, w.y), ri1);
                }
                __syncwarp();   // the slots are refilled by the next batch
            }
            if (open) flush();
            __syncthreads();
            for (int k = tid; k < kFoot * kFoot; k += kStdThreads) {
                const int fx = k / kFoot, fy = k - fx * kFoot, c = fx * kFootRow + fy;
                const int64_t cell = (int64_t)(x0 + fx) * a.gny + (y0 + fy);
                const float2 d = make_float2(s_dr[c], s_di[c]);
                // cells past the grid's edge hold zeros
                if (!RESIDUAL && s_psf[c] != 0.0f) {
                    atomicAdd(&a.psf[cell * a.psf_step], s_psf[c]);
                    s_psf[c] = 0.0f;
                }
                if (d.x != 0.0f || d.y != 0.0f) {
                    atomicAdd(&a.dirty[cell], d);
                    s_dr[c] = 0.0f;
                    s_di[c] = 0.0f;
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
                  r.counts, r.ntx * r.nty, r.nty, g->taps_d, g->tap_rows * 7, psf, psf_step, dirty, g->info.grid_nx,
                  g->info.grid_ny};
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
