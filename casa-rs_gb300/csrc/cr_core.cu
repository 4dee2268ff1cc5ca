// cr_core.cu -- context, workspaces, host tables, scan and radix sort.
#include <cmath>
#include <cstring>

#include <cudaTypedefs.h>

#include "cr_internal.cuh"
#include "cr_lookback.cuh"
#include "cr_tma.cuh"

namespace cr {

void fail(int code, const std::string& msg) { throw Error(code, msg); }

void check_cuda(cudaError_t e, const char* what) {
    if (e != cudaSuccess)
        fail(CR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

void check_cufft(cufftResult r, const char* what) {
    if (r != CUFFT_SUCCESS) fail(CR_CUDA, std::string(what) + ": cuFFT error " + std::to_string((int)r));
}

// Grow-only, stream-ordered buffers: a request larger than the current
// buffer frees it on the stream and allocates a larger one.
void* pool_alloc(cr_ctx* ctx, Pool& pool, const std::string& name, size_t bytes) {
    if (bytes == 0) bytes = 16;
    DevBuf& b = pool[name];
    if (b.bytes >= bytes) return b.ptr;
    if (ctx->capturing) fail(CR_CUDA, "workspace '" + name + "' grew during graph capture");
    if (ctx->alloc_limit > 0 && &pool == &ctx->ws) {
        size_t held = 0;
        for (const auto& kv : pool) held += kv.second.bytes;
        if (held - b.bytes + bytes > (size_t)ctx->alloc_limit)
            fail(CR_CUDA, "workspace '" + name + "' of " + std::to_string(bytes) +
                              " bytes exceeds the context's allocation limit (out of memory)");
    }
    ctx->ws_epoch++;
    if (b.ptr) CR_CUDA_CHECK(cudaFreeAsync(b.ptr, ctx->stream));
    size_t want = bytes + bytes / 8;
    want = (want + 255) & ~size_t(255);
    CR_CUDA_CHECK(cudaMallocAsync(&b.ptr, want, ctx->stream));
    b.bytes = want;
    return b.ptr;
}

void pool_free(cr_ctx* ctx, Pool& pool) {
    for (auto& kv : pool)
        if (kv.second.ptr) cudaFreeAsync(kv.second.ptr, ctx->stream);
    pool.clear();
}

void* workspace(cr_ctx* ctx, const std::string& name, size_t bytes) {
    return pool_alloc(ctx, ctx->ws, name, bytes);
}

void note_launch(cr_ctx* ctx, const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) fail(CR_CUDA, std::string("launch of ") + what + ": " + cudaGetErrorString(e));
    ctx->launches++;
}

void check_device_status(cr_ctx* ctx) {
    volatile int* st = ctx->status_h;
    if (!st) return;
    const int s = *st;
    if (s == 0) return;
    *st = 0;
    fail(s, "a kernel's bounded wait gave up");
}

void kernel_mark(cr_ctx* ctx, int which, bool end) {
    // a captured graph is timed as a whole; with timings off nothing is recorded
    if (ctx->capturing || !ctx->timings_enabled) return;
    CR_CUDA_CHECK(cudaEventRecord(ctx->kev[which * 2 + (end ? 1 : 0)], ctx->stream));
    if (end) ctx->kev_used |= 1 << which;
}

static cufftHandle cached_plan(cr_ctx* ctx,
                               std::map<std::pair<int64_t, int64_t>, cufftHandle>& plans,
                               int64_t nx, int64_t ny, cufftType type) {
    auto key = std::make_pair(nx, ny);
    auto it = plans.find(key);
    if (it != plans.end()) {
        check_cufft(cufftSetStream(it->second, ctx->stream), "cufftSetStream");
        return it->second;
    }
    cufftHandle h;
    check_cufft(cufftPlan2d(&h, (int)nx, (int)ny, type), "cufftPlan2d");
    check_cufft(cufftSetStream(h, ctx->stream), "cufftSetStream");
    plans[key] = h;
    return h;
}

cufftHandle fft_plan(cr_ctx* ctx, int64_t nx, int64_t ny) {
    return cached_plan(ctx, ctx->fft_plans, nx, ny, CUFFT_Z2Z);
}

cufftHandle fft_plan_c2c(cr_ctx* ctx, int64_t nx, int64_t ny) {
    return cached_plan(ctx, ctx->fft_plans_c2c, nx, ny, CUFFT_C2C);
}

cufftHandle fft_plan_type(cr_ctx* ctx, int64_t nx, int64_t ny, cufftType type) {
    return cached_plan(ctx, ctx->fft_plans_real[(int)type], nx, ny, type);
}

cufftHandle fft_plan_many(cr_ctx* ctx, int64_t nx, int64_t ny, cufftType type, int batch) {
    auto& plans = ctx->fft_plans_many[std::make_pair((int)type, batch)];
    auto key = std::make_pair(nx, ny);
    auto it = plans.find(key);
    if (it == plans.end()) {
        cufftHandle h;
        int n[2] = {(int)nx, (int)ny};
        check_cufft(cufftPlanMany(&h, 2, n, nullptr, 1, 0, nullptr, 1, 0, type, batch),
                    "cufftPlanMany");
        it = plans.emplace(key, h).first;
    }
    check_cufft(cufftSetStream(it->second, ctx->stream), "cufftSetStream");
    return it->second;
}

// ---- host tables --------------------------------------------------------------
// casa_composite_padded_len (gridder.rs:4152-4173).
int64_t casa_composite_padded_len(int64_t image_len, double padding) {
    int64_t padded = (int64_t)std::floor(padding * (double)image_len - 0.5);
    if (padded < image_len) padded = image_len;
    if (padded % 2) padded += 1;
    for (;;) {
        int64_t v = padded;
        for (int64_t f : {2, 3, 5})
            while (v > 1 && v % f == 0) v /= f;
        if (v == 1) return padded;
        padded += 2;
    }
}

int64_t image_blc(int64_t grid_len, int64_t image_len) {
    return (grid_len - image_len + (grid_len % 2 == 0 ? 1 : 0)) / 2;
}

// grdsf (gridder.rs:4230-4265), powers by repeated squaring.
double grdsf(double nu) {
    static const double P0[5] = {8.203343e-2, -3.644705e-1, 6.278660e-1, -5.335581e-1, 2.312756e-1};
    static const double P1[5] = {4.028559e-3, -3.697768e-2, 1.021332e-1, -1.201436e-1, 6.412774e-2};
    static const double Q0[3] = {1.0, 8.212018e-1, 2.078043e-1};
    static const double Q1[3] = {1.0, 9.599102e-1, 2.918724e-1};
    if (!(nu >= 0.0 && nu <= 1.0)) return 0.0;
    const bool lo = nu < 0.75;
    const double* p = lo ? P0 : P1;
    const double* q = lo ? Q0 : Q1;
    double e = lo ? 0.75 : 1.0;
    double d = nu * nu - e * e;
    double d2 = d * d;
    double pw[5] = {1.0, d, d2, d2 * d, d2 * d2};
    double num = 0.0, den = 0.0;
    for (int k = 0; k < 5; ++k) num = num + p[k] * pw[k];
    for (int k = 0; k < 3; ++k) den = den + q[k] * pw[k];
    return den == 0.0 ? 0.0 : num / den;
}

static float spheroidal_kernel(double distance, double support) {
    if (!(std::isfinite(distance) && distance <= support)) return 0.0f;
    double nu = distance / support;
    if (nu > 1.0) return 0.0f;
    return (float)((1.0 - nu * nu) * grdsf(nu));
}

// Kernel table (gridder.rs:407-416) and build_normalized_tap_weights
// (gridder.rs:2026-2051): rows for offsets -os/2..os/2, float32 sums.
std::vector<float> std_normalized_taps(int32_t os, int32_t support) {
    int64_t tlen = (int64_t)os * (support + 1);
    std::vector<float> table(tlen, 0.0f);
    for (int64_t i = 0; i < (int64_t)os * support; ++i) {
        double distance = (double)i / ((double)support * (double)os);
        table[i] = spheroidal_kernel(distance * (double)support, (double)support);
    }
    int32_t half = os / 2, taps = 2 * support + 1;
    std::vector<float> rows((size_t)(2 * half + 1) * taps);
    for (int32_t off = -half; off <= half; ++off) {
        float* row = &rows[(size_t)(off + half) * taps];
        float norm = 0.0f;
        for (int32_t t = 0; t < taps; ++t) {
            int64_t lookup = (int64_t)(t - support) * os + off;
            if (lookup < 0) lookup = -lookup;
            float w = lookup < tlen ? table[lookup] : 0.0f;
            row[t] = w;
            norm = norm + w;
        }
        if (norm > 0.0f)
            for (int32_t t = 0; t < taps; ++t) row[t] = row[t] / norm;
    }
    return rows;
}

// build_correction_axis (gridder.rs:4175-4188).
std::vector<float> correction_axis(int64_t size) {
    std::vector<float> out(size);
    double c = (double)size / 2.0;
    for (int64_t i = 0; i < size; ++i) {
        double nu = std::fabs((double)i - c) / c;
        nu = nu < 0.0 ? 0.0 : (nu > 1.0 ? 1.0 : nu);
        double v = grdsf(nu);
        out[i] = v > 1.0e-6 ? (float)(1.0 / v) : 0.0f;
    }
    return out;
}

// build_gridder_correction_axis (gridder.rs:4190-4198).
std::vector<float> gridder_correction_axis(int64_t size) {
    std::vector<float> out(size);
    double c = (double)size / 2.0;
    for (int64_t i = 0; i < size; ++i) {
        double nu = std::fabs((double)i - c) / c;
        nu = nu < 0.0 ? 0.0 : (nu > 1.0 ? 1.0 : nu);
        out[i] = (float)grdsf(nu);
    }
    return out;
}

// build_sinc_axis (gridder.rs:4211-4228).
std::vector<float> sinc_axis(int64_t size, int64_t conv_sampling) {
    std::vector<float> out(size);
    for (int64_t i = 0; i < size; ++i) {
        float offset = (float)(i - size / 2);
        float denom = (float)size * (float)conv_sampling;
        float arg = (float)(3.14159265358979323846 * (double)offset / (double)denom);
        out[i] = (i == size / 2) ? 1.0f : std::sin(arg) / arg;
    }
    return out;
}

// ---- exclusive scan (uint32) ------------------------------------------------------
// One launch: each tile is read once, the sum before it found by look-back, and
// written once.  419 M bins (a 256-channel cube): 1.56 -> 0.89 ms against block
// sums, their recursive scan and a second pass over the input.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 32;   // 16: 1.11 ms for 419 M bins
constexpr int kScanTile = kScanThreads * kScanItems;

__global__ void __launch_bounds__(kScanThreads) scan_kernel(const uint32_t* in, uint32_t* out,
                                                            int64_t n, uint32_t* ticket,
                                                            unsigned long long* state,
                                                            unsigned long long* total_dev,
                                                            int* status) {
    constexpr int kWarps = kScanThreads / 32;
    __shared__ uint32_t s_warp[kWarps];
    __shared__ uint32_t s_base, s_tile;
    __shared__ int s_good;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(ticket, 1u);
    __syncthreads();
    const int64_t tile = s_tile;
    // a warp's 1024 items in eight rows of 128; lane l holds items 4 l .. 4 l + 3
    // of each row
    const int64_t first = tile * kScanTile + warp * (32 * kScanItems) + 4 * lane;
    const bool whole = (tile + 1) * kScanTile <= n && !((uintptr_t)in & 15) &&
                       !((uintptr_t)out & 15);
    uint32_t v[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems / 4; ++k) {
        const int64_t i = first + 128 * k;
        if (whole) {
            const uint4 q = *reinterpret_cast<const uint4*>(in + i);
            v[4 * k] = q.x;
            v[4 * k + 1] = q.y;
            v[4 * k + 2] = q.z;
            v[4 * k + 3] = q.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[4 * k + j] = i + j < n ? in[i + j] : 0u;
        }
    }
    uint32_t run = 0;   // items of the warp before the row
    uint32_t before[kScanItems / 4];
#pragma unroll
    for (int k = 0; k < kScanItems / 4; ++k) {
        const uint32_t s = v[4 * k] + v[4 * k + 1] + v[4 * k + 2] + v[4 * k + 3];
        uint32_t x = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        before[k] = run + x - s;
        run += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) s_warp[warp] = run;
    __syncthreads();
    if (warp == 0) {
        const uint32_t sum =
            __reduce_add_sync(0xffffffffu, lane < kWarps ? s_warp[lane] : 0u);
        bool good;
        const uint32_t base = tile_lookback(state, tile, sum, &good);
        if (lane == 0) {
            s_base = base;
            s_good = good;
            if (!good) atomicExch(status, CR_TIMEOUT);
            if (total_dev && (tile + 1) * kScanTile >= n)
                *total_dev = good ? (unsigned long long)base + sum : 0ull;
        }
    }
    __syncthreads();
    // after a wait gave up the output is zeros: indices made from it stay in range
    uint32_t base = s_good ? s_base : 0u;
    for (int w = 0; w < warp; ++w) base += s_warp[w];
#pragma unroll
    for (int k = 0; k < kScanItems / 4; ++k) {
        const int64_t i = first + 128 * k;
        const uint32_t a = s_good ? base + before[k] : 0u, b = s_good ? a + v[4 * k] : 0u,
                       c = s_good ? b + v[4 * k + 1] : 0u, d = s_good ? c + v[4 * k + 2] : 0u;
        if (whole) {
            *reinterpret_cast<uint4*>(out + i) = make_uint4(a, b, c, d);
        } else {
            const uint32_t e[4] = {a, b, c, d};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + j < n) out[i + j] = e[j];
        }
    }
}

void exclusive_scan_u32(cr_ctx* ctx, const uint32_t* in, uint32_t* out, int64_t n,
                        unsigned long long* total_dev) {
    if (n <= 0) {
        if (total_dev) CR_CUDA_CHECK(cudaMemsetAsync(total_dev, 0, 8, ctx->stream));
        return;
    }
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    // a ticket, then a look-back word per tile
    unsigned long long* work =
        (unsigned long long*)workspace(ctx, "scan_state", (size_t)(tiles + 1) * 8);
    CR_CUDA_CHECK(cudaMemsetAsync(work, 0, (size_t)(tiles + 1) * 8, ctx->stream));
    scan_kernel<<<(unsigned)tiles, kScanThreads, 0, ctx->stream>>>(
        in, out, n, (uint32_t*)work, work + 1, total_dev, ctx->status_d);
    note_launch(ctx, "scan_kernel");
}

// ---- stable LSD radix sort, 8-bit digits ------------------------------------------
// One launch per digit: the digit counts of every pass come from the kernel
// that made the keys, and a tile learns how many items of each digit lie in
// the tiles before it by looking back over their published counts
// (Merrill and Garland's decoupled look-back; Adinets and Merrill's onesweep).
// Tiles take their numbers from a ticket counter, so every tile a block waits
// for has started.  The tile is reordered in shared memory and written in
// runs.  5.05 M keys, 5 passes: 425 -> 265 us against a histogram, a scan
// (1-3 launches) and an uncoalesced scatter per digit; 4,001 keys: 100 -> 33 us.
// Bound by instructions per key (a third of them the look-back's), not by the
// 24 bytes a key moves.
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
// Keys per thread: 16 fill the card from about half a million keys on; below
// kSortSmall keys 4 spread them over more blocks, each with a quarter of the
// serial ranking (4,001 keys: 8.9 -> 6.5 us per digit).
constexpr int kSortItems = 16, kSortItemsSmall = 4;
constexpr int64_t kSortSmall = 1 << 19;
static_assert(kSortThreads == kRadixBins, "a thread per digit");

struct RadixPass {
    const uint64_t* keys_in;
    const uint32_t* vals_in;    // null: the items' positions (first pass)
    uint64_t* keys_out;
    uint32_t* vals_out;
    int64_t n;
    uint32_t pass;              // the key's byte; tags this pass's state words
    const uint32_t* hist;       // digit counts of this pass
    uint32_t* ticket;
    unsigned long long* state;  // [tiles][256]
    unsigned int* fail;
    int* status;
};

__device__ __forceinline__ uint32_t key_byte(uint64_t key, uint32_t byte) {
    return __byte_perm((uint32_t)key, (uint32_t)(key >> 32), byte) & 255u;
}

// exclusive scan over the block's 256 threads of two sums at once
__device__ __forceinline__ unsigned long long scan256(unsigned long long v,
                                                      unsigned long long* s_warp) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    unsigned long long before = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w)
        if (w < warp) before += s_warp[w];
    return before + x - v;
}

template <int ITEMS>
__global__ void __launch_bounds__(kSortThreads, 2) radix_pass_kernel(RadixPass a) {
    constexpr int kTileItems = kSortThreads * ITEMS;
    extern __shared__ uint64_t s_keys[];   // [kTileItems], then the items' values
    uint32_t* s_vals = reinterpret_cast<uint32_t*>(s_keys + kTileItems);
    __shared__ uint32_t s_cnt[kSortWarps][kRadixBins];
    __shared__ uint32_t s_base[kRadixBins];
    __shared__ unsigned long long s_warp[kSortWarps];
    __shared__ uint32_t s_tile;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_tile = *(volatile unsigned int*)a.fail ? 0xffffffffu : atomicAdd(a.ticket, 1u);
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s_cnt[w][t] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;
    if (tile == 0xffffffffu) return;
    const int64_t base = (int64_t)tile * kTileItems;
    const int valid = (int)min((int64_t)kTileItems, a.n - base);
    // a warp holds 32 ITEMS consecutive items, item j of lane l at j * 32 + l
    const int first = warp * (32 * ITEMS) + lane;
    uint64_t key[ITEMS];
    uint32_t pos[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int i = first + 32 * j;
        key[j] = i < valid ? a.keys_in[base + i] : ~0ull;
    }
    const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const bool ok = first + 32 * j < valid;
        const uint32_t d = key_byte(key[j], a.pass);
        uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const uint32_t v = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= (d >> b) & 1u ? v : ~v;
        }
        const uint32_t before = s_cnt[warp][d];
        __syncwarp();
        if (ok && (peers & lt) == 0) s_cnt[warp][d] = before + __popc(peers);
        __syncwarp();
        pos[j] = before + __popc(peers & lt);
    }
    __syncthreads();
    // thread t: digit t
    uint32_t count = 0;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = s_cnt[w][t];
        s_cnt[w][t] = count;
        count += c;
    }
    // state words: count | kind << 32 (1 the tile's count, 2 the count up to
    // and including the tile) | (pass + 1) << 34, so words of earlier passes
    // read as not ready
    const unsigned long long tag = (unsigned long long)(a.pass + 1) << 34;
    volatile unsigned long long* st = a.state;
    if (tile > 0) st[(int64_t)tile * kRadixBins + t] = tag | 1ull << 32 | count;
    const unsigned long long sc =
        scan256((unsigned long long)a.hist[t] << 32 | count, s_warp);
    const uint32_t local = (uint32_t)sc;   // the tile's items of smaller digits
    uint32_t prefix = 0;
    bool good = true;
    for (int64_t p = (int64_t)tile - 1; p >= 0;) {
        // four predecessors at a time
        unsigned long long w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            w[q] = p - q >= 0 ? st[(p - q) * kRadixBins + t] : tag | 2ull << 32;
        bool done = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (done) break;
            for (long long polls = 0; (w[q] ^ tag) >> 34 || ((w[q] >> 32) & 3) == 0;) {
                if (++polls > kLookbackPolls) {
                    good = false;
                    break;
                }
                w[q] = st[(p - q) * kRadixBins + t];
            }
            prefix += (uint32_t)w[q];
            done = !good || ((w[q] >> 32) & 3) == 2;
        }
        if (done) break;
        p -= 4;
    }
    st[(int64_t)tile * kRadixBins + t] = tag | 2ull << 32 | (prefix + count);
    if (!__syncthreads_and(good)) {
        if (t == 0) {
            atomicExch(a.fail, 1u);
            atomicExch(a.status, CR_TIMEOUT);
        }
        return;
    }
    s_base[t] = (uint32_t)(sc >> 32) + prefix - local;
#pragma unroll
    for (int w = 0; w < kSortWarps; ++w) s_cnt[w][t] += local;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int i = first + 32 * j;
        if (i < valid) {
            const uint32_t at = pos[j] + s_cnt[warp][key_byte(key[j], a.pass)];
            s_keys[at] = key[j];
            s_vals[at] = a.vals_in ? a.vals_in[base + i] : (uint32_t)(base + i);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int i = t + kSortThreads * j;
        if (i < valid) {
            const uint64_t k = s_keys[i];
            const uint32_t at = s_base[key_byte(k, a.pass)] + i;
            a.keys_out[at] = k;
            a.vals_out[at] = s_vals[i];
        }
    }
}

// bytes of the keys, of the values and of the words that one memset clears:
// state, histograms, tickets, fail
struct RadixBytes {
    int passes;
    int64_t tiles;
    size_t keys, vals, state, rec, hist;
    size_t cleared() const { return state + rec + hist + 64; }
};

static RadixBytes radix_bytes(int64_t n, int bits) {
    RadixBytes b;
    b.passes = (bits + 7) / 8;
    const int64_t tile = kSortThreads * (n < kSortSmall ? kSortItemsSmall : kSortItems);
    b.tiles = (n + tile - 1) / tile;
    b.keys = (size_t)(n > 0 ? n : 1) * 8;
    b.vals = ((size_t)(n > 0 ? n : 1) * 4 + 7) & ~size_t(7);
    b.state = (size_t)b.tiles * kRadixBins * 8;
    b.rec = (size_t)((n + kRecTile - 1) / kRecTile) * 8;
    b.hist = (size_t)b.passes * kRadixBins * 4;
    return b;
}

size_t radix_sort_bytes(int64_t n, int bits) {
    const RadixBytes b = radix_bytes(n, bits);
    return 2 * b.keys + 2 * b.vals + b.cleared();
}

RadixSort radix_sort_begin(cr_ctx* ctx, int64_t n, int bits, void* mem) {
    const RadixBytes b = radix_bytes(n, bits);
    RadixSort s;
    s.n = n;
    s.passes = b.passes;
    s.tiles = b.tiles;
    char* m = (char*)mem;
    auto take = [&](const char* name, size_t bytes) {
        if (!mem) return (char*)workspace(ctx, name, bytes);
        char* p = m;
        m += bytes;
        return p;
    };
    s.keys = (uint64_t*)take("rec_keys", b.keys);
    s.keys_alt = (uint64_t*)take("sort_keys_alt", b.keys);
    s.vals[0] = (uint32_t*)take("rec_order", b.vals);
    s.vals[1] = (uint32_t*)take("sort_vals_alt", b.vals);
    char* w = take("sort_state", b.cleared());
    s.state = (unsigned long long*)w;
    s.rec_state = (unsigned long long*)(w + b.state);
    s.hist = (uint32_t*)(w + b.state + b.rec);
    s.tickets = (uint32_t*)(w + b.state + b.rec + b.hist);   // at most 8 passes
    s.rec_ticket = s.tickets + 8;
    s.fail = s.tickets + 9;
    CR_CUDA_CHECK(cudaMemsetAsync(w, 0, b.cleared(), ctx->stream));
    return s;
}

void radix_sort_run(cr_ctx* ctx, RadixSort& s) {
    uint64_t* kbuf[2] = {s.keys, s.keys_alt};
    uint32_t* vbuf[2] = {s.vals[0], s.vals[1]};
    const bool small = s.n < kSortSmall;
    auto kern = small ? radix_pass_kernel<kSortItemsSmall> : radix_pass_kernel<kSortItems>;
    const size_t smem = (size_t)kSortThreads * (small ? kSortItemsSmall : kSortItems) * 12;
    CR_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem));
    for (int p = 0; p < s.passes && s.n > 0; ++p) {
        RadixPass a{kbuf[p & 1], p ? vbuf[p & 1] : nullptr, kbuf[(p & 1) ^ 1], vbuf[(p & 1) ^ 1],
                    s.n, (uint32_t)p, s.hist + (size_t)p * kRadixBins, s.tickets + p,
                    s.state, s.fail, ctx->status_d};
        kern<<<(unsigned)s.tiles, kSortThreads, smem, ctx->stream>>>(a);
        note_launch(ctx, "radix_pass_kernel");
    }
    s.sorted_keys = kbuf[s.passes & 1];
    s.order = vbuf[s.passes & 1];
}

// ---- inputs and outputs ----------------------------------------------------------
const void* device_input(cr_ctx* ctx, const void* p, size_t bytes, int32_t location,
                         const char* name) {
    if (!p) return nullptr;
    if (location == CR_DEVICE) return p;
    if (location != CR_HOST) fail(CR_INVALID, "location must be CR_HOST or CR_DEVICE");
    void* d = workspace(ctx, std::string("in_") + name, bytes);
    CR_CUDA_CHECK(cudaMemcpyAsync(d, p, bytes, cudaMemcpyHostToDevice, ctx->stream));
    return d;
}

void copy_out(cr_ctx* ctx, void* dst, const void* src_dev, size_t bytes, int32_t location) {
    if (!dst || bytes == 0) return;
    if (location == CR_DEVICE) {
        if (dst != src_dev)
            CR_CUDA_CHECK(cudaMemcpyAsync(dst, src_dev, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
    } else if (location == CR_HOST) {
        CR_CUDA_CHECK(cudaMemcpyAsync(dst, src_dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    } else {
        fail(CR_INVALID, "location must be CR_HOST or CR_DEVICE");
    }
}

DeviceBatch device_batch(cr_ctx* ctx, const cr_vis_batch* b, bool need_w) {
    if (!b) fail(CR_INVALID, "batch is null");
    if (b->n < 0) fail(CR_INVALID, "batch size is negative");
    if (b->n >= (int64_t)1 << 31) fail(CR_INVALID, "batch larger than 2^31 samples");
    if (b->n > 0 && (!b->u || !b->v || !b->weight || !b->vis))
        fail(CR_INVALID, "batch lacks u, v, weight or vis");
    if (need_w && b->n > 0 && !b->w) fail(CR_INVALID, "W-projection needs w coordinates");
    DeviceBatch d;
    d.n = b->n;
    size_t n = (size_t)b->n;
    d.u = (const double*)device_input(ctx, b->u, n * 8, b->location, "u");
    d.v = (const double*)device_input(ctx, b->v, n * 8, b->location, "v");
    d.w = need_w ? (const double*)device_input(ctx, b->w, n * 8, b->location, "w") : nullptr;
    d.weight = (const float*)device_input(ctx, b->weight, n * 4, b->location, "weight");
    d.sumwt_factor = (const float*)device_input(ctx, b->sumwt_factor, n * 4, b->location, "sumwt");
    d.gridable = (const uint8_t*)device_input(ctx, b->gridable, n, b->location, "gridable");
    d.vis = (const float2*)device_input(ctx, b->vis, n * 8, b->location, "vis");
    return d;
}

// Host batches below this many samples are uploaded in one go.
constexpr int64_t kStageMinSamples = (int64_t)1 << 20;

StagedBatch::StagedBatch(cr_ctx* c, const cr_vis_batch* b, bool need_w) : ctx(c) {
    if (!b || b->location != CR_HOST || b->n < kStageMinSamples) {
        static_cast<DeviceBatch&>(*this) = device_batch(c, b, need_w);
        return;
    }
    // device_batch's checks
    if (b->n >= (int64_t)1 << 31) fail(CR_INVALID, "batch larger than 2^31 samples");
    if (!b->u || !b->v || !b->weight || !b->vis) fail(CR_INVALID, "batch lacks u, v, weight or vis");
    if (need_w && !b->w) fail(CR_INVALID, "W-projection needs w coordinates");
    const size_t n_s = (size_t)b->n;
    struct Col {
        const void* host;
        size_t elem;
        const char* name;
        void* dev;
    } cols[7] = {{b->u, 8, "u", nullptr},
                 {b->v, 8, "v", nullptr},
                 {need_w ? b->w : nullptr, 8, "w", nullptr},
                 {b->weight, 4, "weight", nullptr},
                 {b->sumwt_factor, 4, "sumwt", nullptr},
                 {b->gridable, 1, "gridable", nullptr},
                 {b->vis, 8, "vis", nullptr}};
    // the same workspaces as device_input's, allocated on the main stream
    // before the auxiliary stream is forked from it
    for (Col& col : cols)
        if (col.host) col.dev = workspace(c, std::string("in_") + col.name, n_s * col.elem);
    n = b->n;
    u = (const double*)cols[0].dev;
    v = (const double*)cols[1].dev;
    w = (const double*)cols[2].dev;
    weight = (const float*)cols[3].dev;
    sumwt_factor = (const float*)cols[4].dev;
    gridable = (const uint8_t*)cols[5].dev;
    vis = (const float2*)cols[6].dev;
    CR_CUDA_CHECK(cudaEventRecord(c->fork_ev, c->stream));
    CR_CUDA_CHECK(cudaStreamWaitEvent(c->aux_stream, c->fork_ev, 0));
    // from here on the destructor joins whatever was queued
    nchunks = kStageChunks;
    stage_ev = c->stage_ev;
    int64_t lo = 0;
    try {
        for (int k = 0; k < kStageChunks; ++k) {
            const int64_t hi = b->n * (k + 1) / kStageChunks;
            chunk_end[k] = hi;
            for (const Col& col : cols)
                if (col.host)
                    CR_CUDA_CHECK(cudaMemcpyAsync((char*)col.dev + lo * col.elem,
                                                  (const char*)col.host + lo * col.elem,
                                                  (size_t)(hi - lo) * col.elem,
                                                  cudaMemcpyHostToDevice, c->aux_stream));
            CR_CUDA_CHECK(cudaEventRecord(c->stage_ev[k], c->aux_stream));
            lo = hi;
        }
    } catch (...) {
        // no destructor runs for a half-built batch: join the copies here
        cudaEventRecord(c->join_ev, c->aux_stream);
        cudaStreamWaitEvent(c->stream, c->join_ev, 0);
        throw;
    }
}

StagedBatch::~StagedBatch() {
    if (nchunks > 0) cudaStreamWaitEvent(ctx->stream, ctx->stage_ev[nchunks - 1], 0);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link
// against the driver library).
bool encode_tensor_map_3d(CUtensorMap* map, const void* base, uint64_t d0, uint64_t d1,
                          uint64_t d2, uint64_t stride1, uint64_t stride2, uint32_t b0,
                          uint32_t b1) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000,
                                             cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            fn = nullptr;
        cudaGetLastError();
        return (PFN_cuTensorMapEncodeTiled_v12000)fn;
    }();
    if (!encode) return false;
    if (((uintptr_t)base & 15) || (stride1 & 15) || (stride2 & 15) || ((b0 * 4) & 15) ||
        b0 == 0 || b1 == 0 || b0 > 256 || b1 > 256 || d0 == 0 || d1 == 0 || d2 == 0)
        return false;
    const cuuint64_t dims[3] = {d0, d1, d2};
    const cuuint64_t strides[2] = {stride1, stride2};
    const cuuint32_t box[3] = {b0, b1, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<void*>(base), dims,
                  strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}


}  // namespace cr
