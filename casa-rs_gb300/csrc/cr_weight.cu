// cr_weight.cu -- natural, uniform and Briggs weighting.
//
// Restates apply_weighting_with_density_source (weighting.rs:1055-1180) in the
// Combined density mode, or with the cube PerPlane cells (rounded FP64
// u*scale + centre, weighting.rs:1455-1483): the density grid is image-sized, every sample
// with a finite positive weight adds its weight at its VisImagingWeight cell
// and at the cell of its Hermitian mirror (accumulate_density_sample_serial,
// weighting.rs:1831-1854; weight_density_cell_anchor, gridder.rs:1888-1934,
// whose float32 multiply-then-add order is kept with __fmul_rn/__fadd_rn);
// Briggs f2 = (5 * 10^-robust)^2 / (sum d^2 / sum d) with FP64 sums; the
// reweight divides by d (uniform) or by the CASA denominator d*f2 + 1 computed
// as a separate float multiply and add (casa_briggs_denominator,
// weighting.rs:2440-2443).
#include <cmath>

#include "cr_fixed.cuh"
#include "cr_internal.cuh"

namespace cr {

namespace {

struct DensityCellParams {
    int32_t nx, ny;
    float u_scale, v_scale, cx, cy;
    int32_t convention;          // 0 VisImagingWeight, 1 cube PerPlane (rounded, FP64)
    double du_scale, dv_scale, dcx, dcy;
};

// the VisImagingWeight cell of (u, v) with tx = u u_scale, ty = v v_scale
__device__ __forceinline__ bool float_cell(const DensityCellParams& p, float tx, float ty, int* ox,
                                           int* oy) {
    const float x = __fadd_rn(-tx, p.cx), y = __fadd_rn(ty, p.cy);
    if (!(isfinite(x) && isfinite(y))) return false;
    // trunc(x) in (0, nx) <=> 1 <= x < nx
    if (!(x >= 1.0f && x < (float)p.nx && y >= 1.0f && y < (float)p.ny)) return false;
    *ox = (int)x;
    *oy = (int)y;
    return true;
}

__device__ __forceinline__ bool density_cell(const DensityCellParams& p, double u, double v,
                                             int* ox, int* oy) {
    if (p.convention == 1) {
        // CubeBriggsWeightor{Density,Lookup}: u*scale + centre in FP64, rounded
        const double x = __dadd_rn(__dmul_rn(u, p.du_scale), p.dcx);
        const double y = __dadd_rn(__dmul_rn(-v, p.dv_scale), p.dcy);
        if (!isfinite(x) || !isfinite(y)) return false;
        const double rx = round(x), ry = round(y);
        if (!(rx >= 1.0 && ry >= 1.0 && rx < (double)p.nx && ry < (double)p.ny)) return false;
        *ox = (int)rx;
        *oy = (int)ry;
        return true;
    }
    return float_cell(p, __fmul_rn(d2f(u), p.u_scale), __fmul_rn(d2f(v), p.v_scale), ox, oy);
}

// the cells of (u, v) and of (-u, -v)
__device__ __forceinline__ void density_cells(const DensityCellParams& p, double u, double v,
                                              int* x, int* y, bool* ok, int* xm, int* ym,
                                              bool* okm) {
    if (p.convention == 1) {
        *ok = density_cell(p, u, v, x, y);
        *okm = density_cell(p, -u, -v, xm, ym);
        return;
    }
    const float tx = __fmul_rn(d2f(u), p.u_scale), ty = __fmul_rn(d2f(v), p.v_scale);
    *ok = float_cell(p, tx, ty, x, y);
    *okm = float_cell(p, -tx, -ty, xm, ym);
}

// A block takes contiguous samples, four to a thread at a time (their loads
// are in flight together; the float32 coordinates come from the bits, since
// the FP64 pipe converted four doubles a sample).
//
// With TABLE the block first collects its samples by cell in a hashed table
// in shared memory.  Samples are mostly in time order, and successive times
// of one baseline share a cell: added one by one, the few cells of the
// shortest baselines take tens of thousands of adds each, which memory works
// off one after the other.  A cell's mirror is as a rule the cell reflected,
// so one entry stands for both; a sample for which rounding or the edge makes
// it another, or whose slot another cell holds, is added directly.
// With / without the table: 10.1 M samples on 2048^2 62 / 316 us, 1.05 M on
// 512^2 14.0 / 26.7 us, 250,001 on 2048^2 9.8 / 15.8 us, 60,001 on 256^2
// 8.6 / 6.8 us.
constexpr int kDensityVec = 4, kDensityThreads = 512, kDensityBlocks = 2;
constexpr int kSlotBits = 13, kSlots = 1 << kSlotBits;
constexpr uint32_t kEmptySlot = ~0u;
constexpr int64_t kTableSamples = 1 << 17;

template <bool TABLE>
__global__ void __launch_bounds__(kDensityThreads, kDensityBlocks)
density_kernel(const double* u, const double* v, const float* weight, int64_t n,
               DensityCellParams p, float* density) {
    extern __shared__ uint32_t s_cell[];   // [kSlots], then their sums
    float* s_sum = reinterpret_cast<float*>(s_cell + kSlots);
    if (TABLE) {
        for (int k = threadIdx.x; k < kSlots; k += kDensityThreads) {
            s_cell[k] = kEmptySlot;
            s_sum[k] = 0.0f;
        }
        __syncthreads();
    }
    const int mx = p.convention == 1 ? p.nx : p.nx - 1, my = p.convention == 1 ? p.ny : p.ny - 1;
    const int64_t share = (n + gridDim.x - 1) / gridDim.x;
    const int64_t end = min(n, (blockIdx.x + 1) * share);
    for (int64_t base = blockIdx.x * share + threadIdx.x; base < end;
         base += kDensityThreads * kDensityVec) {
        float w[kDensityVec];
        double us[kDensityVec], vs[kDensityVec];
#pragma unroll
        for (int j = 0; j < kDensityVec; ++j) {
            const int64_t i = base + kDensityThreads * j;
            w[j] = i < end ? weight[i] : 0.0f;
            us[j] = i < end ? u[i] : 0.0;
            vs[j] = i < end ? v[i] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < kDensityVec; ++j) {
            if (!(isfinite(w[j]) && w[j] > 0.0f)) continue;
            int x = 0, y = 0, xm = 0, ym = 0;
            bool ok, okm;
            density_cells(p, us[j], vs[j], &x, &y, &ok, &xm, &ym, &okm);
            const uint32_t cell = (uint32_t)x * (uint32_t)p.ny + (uint32_t)y;
            if (TABLE && ok && okm && xm == mx - x && ym == my - y) {
                const uint32_t slot = (cell * 2654435761u) >> (32 - kSlotBits);
                uint32_t held = *(volatile uint32_t*)&s_cell[slot];
                if (held == kEmptySlot) {
                    held = atomicCAS(&s_cell[slot], kEmptySlot, cell);
                    if (held == kEmptySlot) held = cell;
                }
                if (held == cell) {
                    atomicAdd(&s_sum[slot], w[j]);
                    continue;
                }
            }
            if (ok) atomicAdd(&density[(int64_t)x * p.ny + y], w[j]);
            if (okm) atomicAdd(&density[(int64_t)xm * p.ny + ym], w[j]);
        }
    }
    if (TABLE) {
        __syncthreads();
        for (int k = threadIdx.x; k < kSlots; k += kDensityThreads) {
            const uint32_t cell = s_cell[k];
            if (cell == kEmptySlot) continue;
            const uint32_t x = cell / (uint32_t)p.ny, y = cell % (uint32_t)p.ny;
            atomicAdd(&density[cell], s_sum[k]);
            atomicAdd(&density[((uint32_t)mx - x) * (uint32_t)p.ny + ((uint32_t)my - y)], s_sum[k]);
        }
    }
}

// sum d and sum d^2 (d > 0) in FP64: one pair of adds a block (a pair a warp,
// 78,000 adds to two words, took most of 123 us for 2048^2), the conversions
// from the bits
__global__ void __launch_bounds__(256) density_sums_kernel(const float* d, int64_t n,
                                                           double* sums) {
    double s = 0.0, s2 = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        const float f = d[i];
        if (f == 0.0f) continue;
        const double v = f2d(f);
        s += v;
        if (v > 0.0) s2 += v * v;
    }
    __shared__ double sh[2][8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s += __shfl_xor_sync(0xffffffffu, s, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
        sh[0][warp] = s;
        sh[1][warp] = s2;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0.0;
        for (int k = 0; k < 8; ++k) t += sh[threadIdx.x][k];
        atomicAdd(&sums[threadIdx.x], t);
    }
}

__global__ void reweight_kernel(const double* u, const double* v, const float* weight, int64_t n,
                                DensityCellParams p, const float* density, int mode, float f2,
                                float* out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        float w = weight[i];
        if (mode == CR_WEIGHT_NATURAL) {
            out[i] = w;
            continue;
        }
        int x, y;
        float r = 0.0f;
        if (density_cell(p, u[i], v[i], &x, &y)) {
            float d = density[(int64_t)x * p.ny + y];
            if (isfinite(w) && w > 0.0f && isfinite(d) && d > 0.0f) {
                if (mode == CR_WEIGHT_UNIFORM)
                    r = __fdiv_rn(w, d);
                else
                    r = __fdiv_rn(w, __fadd_rn(__fmul_rn(d, f2), 1.0f));
            }
        }
        out[i] = r;
    }
}

}  // namespace

void apply_weighting(cr_ctx* ctx, cr_gridder* g, const DeviceBatch& b, int32_t mode,
                     float robust, float* out_weight, float* f2_out, int32_t convention,
                     const double* build_u, const double* build_v) {
    if (mode != CR_WEIGHT_NATURAL && mode != CR_WEIGHT_UNIFORM && mode != CR_WEIGHT_BRIGGS)
        fail(CR_INVALID, "unknown weighting mode");
    const int32_t nx = g->geom.nx, ny = g->geom.ny;
    DensityCellParams p;
    p.nx = nx;
    p.ny = ny;
    p.u_scale = (float)((double)nx * g->geom.cell_x_rad);
    p.v_scale = (float)((double)ny * g->geom.cell_y_rad);
    p.cx = (float)((double)nx / 2.0);
    p.cy = (float)((double)ny / 2.0);
    p.convention = convention;
    p.du_scale = (double)nx * g->geom.cell_x_rad;
    p.dv_scale = (double)ny * g->geom.cell_y_rad;
    p.dcx = (double)nx / 2.0;
    p.dcy = (double)ny / 2.0;
    float f2 = 0.0f;
    float* density = nullptr;
    if (mode != CR_WEIGHT_NATURAL) {
        density = (float*)workspace(ctx, "wt_density", (size_t)nx * ny * 4);
        CR_CUDA_CHECK(cudaMemsetAsync(density, 0, (size_t)nx * ny * 4, ctx->stream));
        if (b.n > 0) {
            // the density is built at build_u, build_v when given (the row
            // path's VisImagingWeight coordinates), looked up at u, v
            // (the table's keys are 32-bit cells)
            const bool table = b.n >= kTableSamples && (int64_t)nx * ny < kEmptySlot;
            auto kern = table ? density_kernel<true> : density_kernel<false>;
            const size_t smem = table ? (size_t)kSlots * 8 : 0;
            CR_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)smem));
            kern<<<grid_blocks(b.n, kDensityThreads * kDensityVec, 152 * kDensityBlocks),
                   kDensityThreads, smem, ctx->stream>>>(build_u ? build_u : b.u,
                                                         build_v ? build_v : b.v, b.weight, b.n,
                                                         p, density);
            note_launch(ctx, "density_kernel");
        }
        if (mode == CR_WEIGHT_BRIGGS) {
            double* sums = (double*)workspace(ctx, "wt_sums", 16);
            CR_CUDA_CHECK(cudaMemsetAsync(sums, 0, 16, ctx->stream));
            density_sums_kernel<<<grid_blocks((int64_t)nx * ny, 256, 152 * 8), 256, 0, ctx->stream>>>(
                density, (int64_t)nx * ny, sums);
            note_launch(ctx, "density_sums_kernel");
            double h[2];
            CR_CUDA_CHECK(cudaMemcpyAsync(h, sums, 16, cudaMemcpyDeviceToHost, ctx->stream));
            CR_CUDA_CHECK(cudaStreamSynchronize(ctx->stream));
            if (h[1] > 0.0 && h[0] > 0.0) {
                double a = 5.0 * std::pow(10.0, -(double)robust);
                f2 = (float)(a * a / (h[1] / h[0]));
            }
        }
    }
    if (b.n > 0) {
        reweight_kernel<<<grid_blocks(b.n, 256), 256, 0, ctx->stream>>>(b.u, b.v, b.weight, b.n, p,
                                                                        density, mode, f2, out_weight);
        note_launch(ctx, "reweight_kernel");
    }
    if (f2_out) *f2_out = f2;
}

}  // namespace cr
