// cr_rows.cu -- row-runs to visibility samples on the device.
//
// Restates how casa-imaging turns MeasurementSet-shaped rows into weighted
// scalar samples (routed_weighted_grid_sample_from_run, lib.rs:880-1062, with
// the pair collapse of collapse_standard_mfs_pair_visibility,
// execution.rs:2323-2340, and ParallelHandBatch::collapse_with_transform,
// types.rs:2090-2160): per (row, channel) either one explicit correlation or
// a collapsed pair of parallel hands.  A sample is dropped when a used
// correlation is flagged, its visibility is not finite, a hand's weight is
// not finite and positive, the natural weight (the explicit weight, or the
// float32 mean 0.5 (w1 + w2) of a pair) is not finite and positive, or the
// plane's sumwt factor is not.  Weights come from WEIGHT_SPECTRUM when given,
// else from the row's WEIGHT.  u, v, w in wavelengths are the FP64 products
// uvw_m * lambda_scale; the density coordinates are the VisImagingWeight
// ones of casa_vis_imaging_weight_uv_lambda (weighting.rs:748-756): the
// float32 scale f/c, the FP64 product, rounded to float32.
//
// One launch: a tile of samples is loaded and judged, its kept samples are
// counted, the kept samples before it come by look-back over the earlier tiles'
// counts, and the tile writes its part of the compacted batch in (row, channel)
// order.  Each input is read once; the only FP64 instructions are the five
// products (conversions between float and double go by the bits).  1,263,600
// rows x 64 channels x 4 correlations: 2.9 -> 1.9 ms (a marking pass, a
// scan and a writing pass that read everything again, bound by the FP64
// pipe's conversions as much as by memory).
#include <algorithm>

#include "cr_fixed.cuh"
#include "cr_lookback.cuh"

namespace cr {

namespace {

struct RowArgs {
    int64_t R;
    int32_t C, ncorr;
    const double* uvw;
    const double* ls;          // [C] f / c, then [C] float32(f / c), device copy
    const float2* data;        // [R][C][ncorr]
    const uint8_t* flag;       // [R][C][ncorr]
    const float* weight;       // [R][ncorr]
    const float* spectrum;     // [R][C][ncorr] or null
    const uint8_t* gridable;   // [R] or null
    int32_t mode, corr0, corr1, transform;
    float sumwt_factor;
};

// StandardMfsPairCollapseTransform::collapse in num-complex's operations
// (Complex32 * f32 scales both parts; a complex product is
// (a c - b d, a d + b c) without fused operations).
__device__ __forceinline__ float2 collapse(float2 a, float2 b, int transform) {
    if (transform == 0)
        return make_float2(__fmul_rn(__fadd_rn(a.x, b.x), 0.5f), __fmul_rn(__fadd_rn(a.y, b.y), 0.5f));
    const float dr = __fsub_rn(a.x, b.x), di = __fsub_rn(a.y, b.y);
    if (transform == 1) return make_float2(__fmul_rn(dr, 0.5f), __fmul_rn(di, 0.5f));
    const float s = transform == 2 ? 0.5f : -0.5f;   // multiply by (0, s)
    return make_float2(__fsub_rn(__fmul_rn(dr, 0.0f), __fmul_rn(di, s)),
                       __fadd_rn(__fmul_rn(dr, s), __fmul_rn(di, 0.0f)));
}

__device__ __forceinline__ bool pos_finite(float w) { return isfinite(w) && w > 0.0f; }

struct RowOut {
    double *u, *v, *w, *du, *dv;
    float* weight;
    float* sumwt_factor;
    uint8_t* gridable;
    float2* vis;
};

constexpr int kRowThreads = 256;
constexpr int kRowItems = 8;
constexpr int kRowTile = kRowThreads * kRowItems;

__global__ void __launch_bounds__(kRowThreads, 4) rows_kernel(RowArgs a, RowOut o,
                                                              uint32_t* ticket,
                                                              unsigned long long* state,
                                                              unsigned long long* total,
                                                              int* status) {
    constexpr int kWarps = kRowThreads / 32;
    __shared__ uint32_t s_count[kRowItems * kWarps];
    __shared__ uint32_t s_base, s_tile;
    __shared__ int s_good;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const uint32_t n = (uint32_t)(a.R * a.C);   // below 2^31
    const uint32_t tile = s_tile, first = tile * (uint32_t)kRowTile + (uint32_t)tid;
    // item j of a thread is sample first + j * kRowThreads; every load of the
    // tile is issued before any is judged
    float2 va[kRowItems], vb[kRowItems];
    float wa[kRowItems], wb[kRowItems];
    uint32_t flagged = 0;
    const bool pair = a.mode != 0;
#pragma unroll
    for (int j = 0; j < kRowItems; ++j) {
        const uint32_t i = first + j * kRowThreads;
        va[j] = vb[j] = make_float2(0.0f, 0.0f);
        wa[j] = wb[j] = 0.0f;
        if (i < n) {
            const int64_t base = (int64_t)i * a.ncorr;
            va[j] = a.data[base + a.corr0];
            if (pair) vb[j] = a.data[base + a.corr1];
            if (a.flag) {
                if (a.flag[base + a.corr0]) flagged |= 1u << j;
                if (pair && a.flag[base + a.corr1]) flagged |= 1u << j;
            }
            const float* w = a.spectrum ? a.spectrum + base
                                        : a.weight + (int64_t)(i / (uint32_t)a.C) * a.ncorr;
            wa[j] = w[a.corr0];
            if (pair) wb[j] = w[a.corr1];
        }
    }
    uint32_t keep[kRowItems];   // the warp's kept lanes of item j
#pragma unroll
    for (int j = 0; j < kRowItems; ++j) {
        bool ok = pos_finite(a.sumwt_factor) && !((flagged >> j) & 1u) && pos_finite(wa[j]);
        if (pair) {
            ok = ok && pos_finite(wb[j]);
            va[j] = collapse(va[j], vb[j], a.transform);
            wa[j] = __fmul_rn(0.5f, __fadd_rn(wa[j], wb[j]));
            ok = ok && pos_finite(wa[j]);
        }
        // a sample past the end has weight zero
        keep[j] = __ballot_sync(0xffffffffu, ok && isfinite(va[j].x) && isfinite(va[j].y));
        if (lane == 0) s_count[j * kWarps + warp] = __popc(keep[j]);
    }
    __syncthreads();
    if (warp == 0) {
        // 64 counts in sample order: two per lane
        const uint32_t c0 = s_count[2 * lane], c1 = s_count[2 * lane + 1];
        uint32_t x = c0 + c1;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, k);
            if (lane >= k) x += y;
        }
        s_count[2 * lane] = x - c0 - c1;
        s_count[2 * lane + 1] = x - c1;
        const uint32_t sum = __shfl_sync(0xffffffffu, x, 31);
        bool good;
        const uint32_t before = tile_lookback(state, tile, sum, &good);
        if (lane == 0) {
            s_base = before;
            s_good = good;
            if (!good) atomicExch(status, CR_TIMEOUT);
            if ((tile + 1) * (uint64_t)kRowTile >= n) *total = (uint64_t)before + sum;
        }
    }
    __syncthreads();
    if (!s_good) return;
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < kRowItems; ++j) {
        if (!((keep[j] >> lane) & 1u)) continue;
        const uint32_t i = first + j * kRowThreads;
        const uint32_t r = i / (uint32_t)a.C, c = i - r * (uint32_t)a.C;
        const uint32_t k = s_base + s_count[j * kWarps + warp] + __popc(keep[j] & lt);
        const double ls = a.ls[c], ls32 = a.ls[a.C + c];
        const double um = a.uvw[3 * (int64_t)r], vm = a.uvw[3 * (int64_t)r + 1],
                     wm = a.uvw[3 * (int64_t)r + 2];
        o.u[k] = __dmul_rn(um, ls);
        o.v[k] = __dmul_rn(vm, ls);
        o.w[k] = __dmul_rn(wm, ls);
        o.du[k] = f2d(d2f(__dmul_rn(um, ls32)));
        o.dv[k] = f2d(d2f(__dmul_rn(vm, ls32)));
        o.weight[k] = wa[j];
        o.sumwt_factor[k] = a.sumwt_factor;
        o.gridable[k] = a.gridable ? (a.gridable[r] ? 1 : 0) : 1;
        o.vis[k] = va[j];
    }
}

}  // namespace

int64_t prepare_rows(cr_ctx* ctx, const cr_row_runs* rr, const cr_polarization* pol,
                     const RowsOut& out) {
    if (!rr || !pol) fail(CR_INVALID, "null argument");
    if (rr->rows < 0 || rr->channels <= 0 || rr->correlations <= 0)
        fail(CR_INVALID, "row runs need rows >= 0, channels > 0 and correlations > 0");
    if ((uint64_t)rr->rows * (uint64_t)rr->channels >= (1ull << 31))
        fail(CR_INVALID, "row runs larger than 2^31 samples");
    if (pol->mode != 0 && pol->mode != 1) fail(CR_INVALID, "polarization mode must be 0 or 1");
    if (pol->corr0 < 0 || pol->corr0 >= rr->correlations ||
        (pol->mode == 1 && (pol->corr1 < 0 || pol->corr1 >= rr->correlations)))
        fail(CR_INVALID, "polarization correlations exceed the correlation count");
    if (pol->mode == 1 && (pol->transform < 0 || pol->transform > 3))
        fail(CR_INVALID, "pair transform must be 0..3");
    if (!rr->lambda_scale) fail(CR_INVALID, "lambda_scale is null");
    const int64_t R = rr->rows, C = rr->channels, K = rr->correlations, n = R * C;
    if (R > 0 && (!rr->uvw_m || !rr->data || (!rr->weight && !rr->weight_spectrum)))
        fail(CR_INVALID, "row runs lack uvw, data or weights");
    RowArgs a{};
    a.R = R;
    a.C = (int32_t)C;
    a.ncorr = (int32_t)K;
    a.uvw = (const double*)device_input(ctx, rr->uvw_m, (size_t)R * 24, rr->location, "rr_uvw");
    a.data = (const float2*)device_input(ctx, rr->data, (size_t)n * K * 8, rr->location, "rr_data");
    a.flag = (const uint8_t*)device_input(ctx, rr->flag, (size_t)n * K, rr->location, "rr_flag");
    a.weight = (const float*)device_input(ctx, rr->weight, (size_t)R * K * 4, rr->location,
                                          "rr_weight");
    a.spectrum = (const float*)device_input(ctx, rr->weight_spectrum, (size_t)n * K * 4,
                                            rr->location, "rr_spectrum");
    a.gridable = (const uint8_t*)device_input(ctx, rr->gridable, (size_t)R, rr->location,
                                              "rr_gridable");
    // f / c and its float32 value, widened (casa_vis_imaging_weight_uv_lambda)
    std::vector<double> scales((size_t)C * 2);
    for (int64_t c = 0; c < C; ++c) {
        scales[(size_t)c] = rr->lambda_scale[c];
        scales[(size_t)(C + c)] = (double)(float)rr->lambda_scale[c];
    }
    double* ls = (double*)workspace(ctx, "rr_ls", (size_t)C * 16);
    CR_CUDA_CHECK(cudaMemcpyAsync(ls, scales.data(), (size_t)C * 16, cudaMemcpyHostToDevice,
                                  ctx->stream));
    a.ls = ls;
    a.mode = pol->mode;
    a.corr0 = pol->corr0;
    a.corr1 = pol->corr1;
    a.transform = pol->transform;
    a.sumwt_factor = pol->sumwt_factor;
    const size_t tiles = (size_t)((n + kRowTile - 1) / kRowTile);
    // the total, the ticket, and a look-back word per tile
    unsigned long long* work =
        (unsigned long long*)workspace(ctx, "rr_work", 16 + tiles * 8);
    unsigned long long* total = work;
    CR_CUDA_CHECK(cudaMemsetAsync(work, 0, 16 + tiles * 8, ctx->stream));
    if (n > 0) {
        RowOut o{out.u, out.v, out.w, out.du, out.dv, out.weight, out.sumwt_factor, out.gridable,
                 out.vis};
        rows_kernel<<<(unsigned)tiles, kRowThreads, 0, ctx->stream>>>(
            a, o, (uint32_t*)(work + 1), work + 2, total, ctx->status_d);
        note_launch(ctx, "rows_kernel");
    }
    unsigned long long h = 0;
    CR_CUDA_CHECK(cudaMemcpyAsync(&h, total, 8, cudaMemcpyDeviceToHost, ctx->stream));
    CR_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
    check_device_status(ctx);
    return (int64_t)h;
}

}  // namespace cr
