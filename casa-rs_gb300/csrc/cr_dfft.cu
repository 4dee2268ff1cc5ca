// cr_dfft.cu -- the image stage's centred transforms, in float-pair arithmetic or
// in float32.
//
// The dirty-product stage of the reference runs its centred FFTs in FP64
// (fft.rs:600-630 on Complex64 grids; DirtyProductFftPolicy's default,
// lib.rs:2435-2445): the grid correction 1/grdsf amplifies transform rounding
// near the image edge, so float32 transforms miss the 1e-5 image bar there.
// GB300 runs FP64 at a small fraction of its float32 rate, which made the
// two 5000^2 FP64 transforms of a W-projection dirty image a third of the
// end-to-end call.  These kernels compute the same transforms with every
// value held as an unevaluated sum of two floats (hi + lo, about 48
// significant bits): Knuth's two-sum and Dekker's product with a fused
// multiply-add give each addition and multiplication with an error of about
// 2^-44 of its operands, far below what the final float32 image keeps.
//
// One 2-D transform is two passes of 1-D transforms, one line per block: a
// mixed-radix decimation-in-time transform (radices 4, 2, 3, 5: the grids are
// even and 5-smooth, the composite padding of gridder.rs:4152-4173) whose first
// butterflies read global memory and whose last write it, with the line in
// shared memory between them, and twiddles exp(2 pi i k / N) split into float
// pairs on the host.
//   grid -> image: half of the grid's rows (only the image's columns kept,
//     stored transposed), then the image's columns, two to a line, whose output
//     goes straight through the crop and correction of crop_correct_body;
//   image -> grid: the image's columns first, two to a line (the apodised
//     image is zero outside them), then half of the grid's rows, written with
//     their mirror images as the float32 grid.
// So the grid, the largest array, is only read and written along its rows.
// The centring is the checkerboard modulation of cr_fft.cu.
//
// 3600^2 grid, 3000^2 image: grid to image 417 -> 231 us; 2560^2 and
// 2048^2: grid to image 219 -> 124 us, image to grid 219 -> 121 us
// (against scalar, renormalised pair arithmetic with every stage through
// shared memory, twiddles gathered from one table and the grid read and
// written by columns: the load/store unit was the bound, not the arithmetic).
#include <algorithm>
#include <cmath>
#include <memory>
#include <vector>

#include "cr_internal.cuh"

namespace cr {

struct DfPlan {
    int32_t n = 0, ns = 0;
    int32_t radix[16] = {}, tw_at[16] = {};
    int32_t* pos = nullptr;   // [n / radix[0]] where input p's butterfly goes
    // per stage (from the second), [radix - 1][m]: exp(+2 pi i q j / (m radix))
    // as (cos hi, sin hi, cos lo, sin lo), so that a warp reads rows; tw1 the
    // same as float32 (cos, sin)
    float4* tw = nullptr;
    float2* tw1 = nullptr;
    ~DfPlan() {
        cudaFree(pos);
        cudaFree(tw);
        cudaFree(tw1);
    }
};

namespace {

constexpr int kDfThreads = 512;
constexpr int kDfMaxStages = 16;
// lines up to this length fit one block's shared memory (16 bytes a point)
constexpr int64_t kDfMaxN = 13824;

struct DfStages {
    int32_t n, ns;
    int32_t sa, sb;                 // the line's swizzle (at())
    int32_t radix[kDfMaxStages];
    int32_t tw[kDfMaxStages];       // the stage's twiddles in the plan's table
    uint32_t magic[kDfMaxStages];   // ceil(2^32 / m), m the stage's span: exact below 2^16
};

struct DfConsts {
    float c1h, c1l, c2h, c2l;   // cos(2 pi / 5), cos(4 pi / 5)
    float s1h, s1l, s2h, s2l;   // sin(2 pi / 5), sin(4 pi / 5)
    float s3h, s3l;             // sin(2 pi / 3)
};

// A complex value as a float pair per part: h = (re, im) high parts, l the low
// ones.  Both parts go through paired float32 instructions (FADD2, FMUL2,
// FFMA2: two results per issue slot).  Sums are not renormalised: |l| stays
// below a few ulps of the largest |h| that went into a value, so the pair
// still holds about 2^-45 of it; the one rounding to float32 is at the end.
struct cdd {
    float2 h, l;
};
struct dd {
    float h, l;
};

__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a);
}
// s + e = a + b exactly (Knuth), the errors then summed with the low parts
__device__ __forceinline__ cdd cadd(cdd a, cdd b) {
    const float2 s = __fadd2_rn(a.h, b.h), v = sub2(s, a.h);
    const float2 e = __fadd2_rn(sub2(a.h, sub2(s, v)), sub2(b.h, v));
    return {s, __fadd2_rn(e, __fadd2_rn(a.l, b.l))};
}
__device__ __forceinline__ cdd csub(cdd a, cdd b) {
    const float2 s = sub2(a.h, b.h), v = sub2(s, a.h);
    const float2 e = sub2(sub2(a.h, sub2(s, v)), __fadd2_rn(b.h, v));
    return {s, __fadd2_rn(e, sub2(a.l, b.l))};
}
// times a real float pair: the high product's rounding error from one fused
// multiply-add (Dekker's product), the cross terms added to it
__device__ __forceinline__ cdd cscale(cdd a, dd c) {
    const float2 ch = dup(c.h), p = __fmul2_rn(a.h, ch);
    float2 e = __ffma2_rn(a.h, ch, make_float2(-p.x, -p.y));
    e = __ffma2_rn(a.h, dup(c.l), e);
    return {p, __ffma2_rn(a.l, ch, e)};
}
// a w with w = (wr, wi): (ar, ai) wr + (-ai, ar) wi, the two high products
// summed exactly, their errors and cross terms gathered in the low part
__device__ __forceinline__ cdd cmul(cdd a, float4 w) {
    const float2 rh = dup(w.x), rl = dup(w.z), ih = make_float2(-w.y, w.y),
                 il = make_float2(-w.w, w.w);
    const float2 sh = make_float2(a.h.y, a.h.x), sl = make_float2(a.l.y, a.l.x);
    const float2 p = __fmul2_rn(a.h, rh), q = __fmul2_rn(sh, ih);
    float2 t = __ffma2_rn(a.h, rh, make_float2(-p.x, -p.y));
    t = __ffma2_rn(a.h, rl, t);
    t = __ffma2_rn(a.l, rh, t);
    t = __fadd2_rn(t, __ffma2_rn(sh, ih, make_float2(-q.x, -q.y)));
    t = __ffma2_rn(sh, il, t);
    t = __ffma2_rn(sl, ih, t);
    const float2 s = __fadd2_rn(p, q), v = sub2(s, p);
    const float2 e = __fadd2_rn(sub2(p, sub2(s, v)), sub2(q, v));
    return {s, __fadd2_rn(e, t)};
}
// times +i for the inverse transform, -i for the forward one
template <bool INV>
__device__ __forceinline__ cdd mul_i(cdd a) {
    return INV ? cdd{make_float2(-a.h.y, a.h.x), make_float2(-a.l.y, a.l.x)}
               : cdd{make_float2(a.h.y, -a.h.x), make_float2(a.l.y, -a.l.x)};
}

// in memory: (re hi, im hi, re lo, im lo)
__device__ __forceinline__ cdd unpack(float4 v) {
    return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ float4 pack(cdd a) { return make_float4(a.h.x, a.h.y, a.l.x, a.l.y); }
__device__ __forceinline__ cdd exact(cdd*, float2 v) { return {v, make_float2(0.0f, 0.0f)}; }
__device__ __forceinline__ cdd halve(cdd a, float half) {
    return {__fmul2_rn(a.h, dup(half)), __fmul2_rn(a.l, dup(half))};
}
__device__ __forceinline__ cdd conj_of(cdd a) {
    return {make_float2(a.h.x, -a.h.y), make_float2(a.l.x, -a.l.y)};
}
__device__ __forceinline__ float2 rounded(cdd a) { return __fadd2_rn(a.h, a.l); }
__device__ __forceinline__ float2 low(cdd a) { return a.l; }
__device__ __forceinline__ float4 conj_mem(float4 w) { return make_float4(w.x, -w.y, w.z, -w.w); }

// A complex value in float32, for the float32 policy: the same operations.
struct cs1 {
    float2 h;
};
__device__ __forceinline__ cs1 cadd(cs1 a, cs1 b) { return {__fadd2_rn(a.h, b.h)}; }
__device__ __forceinline__ cs1 csub(cs1 a, cs1 b) { return {sub2(a.h, b.h)}; }
__device__ __forceinline__ cs1 cscale(cs1 a, dd c) { return {__fmul2_rn(a.h, dup(c.h))}; }
__device__ __forceinline__ cs1 cmul(cs1 a, float2 w) {
    return {__ffma2_rn(make_float2(a.h.y, a.h.x), make_float2(-w.y, w.y),
                       __fmul2_rn(a.h, dup(w.x)))};
}
template <bool INV>
__device__ __forceinline__ cs1 mul_i(cs1 a) {
    return INV ? cs1{make_float2(-a.h.y, a.h.x)} : cs1{make_float2(a.h.y, -a.h.x)};
}
__device__ __forceinline__ cs1 unpack(float2 v) { return {v}; }
__device__ __forceinline__ float2 pack(cs1 a) { return a.h; }
__device__ __forceinline__ cs1 exact(cs1*, float2 v) { return {v}; }
__device__ __forceinline__ cs1 halve(cs1 a, float half) { return {__fmul2_rn(a.h, dup(half))}; }
__device__ __forceinline__ cs1 conj_of(cs1 a) { return {make_float2(a.h.x, -a.h.y)}; }
__device__ __forceinline__ float2 rounded(cs1 a) { return a.h; }
__device__ __forceinline__ float2 low(cs1) { return make_float2(0.0f, 0.0f); }
__device__ __forceinline__ float2 conj_mem(float2 w) { return make_float2(w.x, -w.y); }

// V's form in memory and its share of a 128-byte row of banks
template <typename V>
struct Mem;
template <>
struct Mem<cdd> {
    using T = float4;
    static constexpr int kRowMask = 7;
};
template <>
struct Mem<cs1> {
    using T = float2;
    static constexpr int kRowMask = 15;
};
// two neighbouring values, the first at an even place of a 16-byte aligned row
__device__ __forceinline__ void store_two(float4* p, cdd a, cdd b) {
    p[0] = pack(a);
    p[1] = pack(b);
}
__device__ __forceinline__ void store_two(float2* p, cs1 a, cs1 b) {
    *reinterpret_cast<float4*>(p) = make_float4(a.h.x, a.h.y, b.h.x, b.h.y);
}

// A line in shared memory.  Position i lies at i with its place in a 128-byte
// row of banks exchanged by higher bits, so that the digit-reversed stores of
// the first stage and the strided reads of the second spread over the banks:
// counted over the stages, 1.9 (float pairs) and 3.1 (float32) wavefronts per
// ideal one without it, 1.1-1.3 with the shifts of stages().
template <typename V>
struct Line {
    using T = typename Mem<V>::T;
    T* sm;
    int sa, sb;
    __device__ __forceinline__ int at(int i) const {
        return i ^ (((i >> sa) ^ (i >> sb)) & Mem<V>::kRowMask);
    }
    __device__ __forceinline__ V ld(int i) const { return unpack(sm[at(i)]); }
    __device__ __forceinline__ void st(int i, V a) const { sm[at(i)] = pack(a); }
};

// DFTs of 2 to 5 values in place, with the transform's sign.
template <bool INV, typename V>
__device__ __forceinline__ void dft(V (&x)[2], const DfConsts&) {
    const V t = x[0];
    x[0] = cadd(t, x[1]);
    x[1] = csub(t, x[1]);
}

template <bool INV, typename V>
__device__ __forceinline__ void dft(V (&x)[3], const DfConsts& c) {
    const V t1 = cadd(x[1], x[2]), t2 = csub(x[1], x[2]);
    const V a = csub(x[0], halve(t1, 0.5f));
    const V b = mul_i<INV>(cscale(t2, dd{c.s3h, c.s3l}));
    x[0] = cadd(x[0], t1);
    x[1] = cadd(a, b);
    x[2] = csub(a, b);
}

template <bool INV, typename V>
__device__ __forceinline__ void dft(V (&x)[4], const DfConsts&) {
    const V t0 = cadd(x[0], x[2]), t1 = csub(x[0], x[2]), t2 = cadd(x[1], x[3]);
    const V t3 = mul_i<INV>(csub(x[1], x[3]));
    x[0] = cadd(t0, t2);
    x[1] = cadd(t1, t3);
    x[2] = csub(t0, t2);
    x[3] = csub(t1, t3);
}

template <bool INV, typename V>
__device__ __forceinline__ void dft(V (&x)[5], const DfConsts& c) {
    const dd c1{c.c1h, c.c1l}, c2{c.c2h, c.c2l}, s1{c.s1h, c.s1l}, s2{c.s2h, c.s2l};
    const V t1 = cadd(x[1], x[4]), t2 = cadd(x[2], x[3]), t3 = csub(x[1], x[4]),
              t4 = csub(x[2], x[3]);
    const V a1 = cadd(x[0], cadd(cscale(t1, c1), cscale(t2, c2)));
    const V a2 = cadd(x[0], cadd(cscale(t1, c2), cscale(t2, c1)));
    const V b1 = mul_i<INV>(cadd(cscale(t3, s1), cscale(t4, s2)));
    const V b2 = mul_i<INV>(csub(cscale(t3, s2), cscale(t4, s1)));
    x[0] = cadd(x[0], cadd(t1, t2));
    x[1] = cadd(a1, b1);
    x[2] = cadd(a2, b2);
    x[3] = csub(a2, b2);
    x[4] = csub(a1, b1);
}

// The first stage: input p + q n / R for q < R, out to shared memory.
template <bool INV, int R, typename V, typename Load>
__device__ __forceinline__ void first_stage(const Line<V>& line, const DfStages& s, const int32_t* pos,
                                            const DfConsts& c, Load load) {
    const int step = s.n / R;
    for (int p = threadIdx.x; p < step; p += blockDim.x) {
        V x[R];
#pragma unroll
        for (int q = 0; q < R; ++q) x[q] = load(p + q * step);
        dft<INV>(x, c);
        const int at = pos[p];
#pragma unroll
        for (int q = 0; q < R; ++q) line.st(at + q, x[q]);
    }
}

// A later stage of span m: values j + q m of group g, the q-th times its
// twiddle, a DFT of the radix, then out(position, value).
template <bool INV, int R, typename V, typename Out>
__device__ __forceinline__ void stage(const Line<V>& line, int n, int m, unsigned magic,
                                      const typename Mem<V>::T* tw, const DfConsts& c, Out out) {
    for (int b = threadIdx.x; b < n / R; b += blockDim.x) {
        const int g = (int)__umulhi((unsigned)b, magic), j = b - g * m, at = g * (m * R) + j;
        V x[R];
#pragma unroll
        for (int q = 0; q < R; ++q) x[q] = line.ld(at + q * m);
#pragma unroll
        for (int q = 1; q < R; ++q) {
            const auto w = __ldg(tw + (q - 1) * m + j);
            x[q] = cmul(x[q], INV ? w : conj_mem(w));
        }
        dft<INV>(x, c);
#pragma unroll
        for (int q = 0; q < R; ++q) out(at + q * m, x[q]);
    }
}

template <bool INV, typename V, typename Out>
__device__ __forceinline__ void any_stage(int r, const Line<V>& line, int n, int m, unsigned magic,
                                          const typename Mem<V>::T* tw, const DfConsts& c, Out out) {
    if (r == 4)
        stage<INV, 4>(line, n, m, magic, tw, c, out);
    else if (r == 5)
        stage<INV, 5>(line, n, m, magic, tw, c, out);
    else if (r == 3)
        stage<INV, 3>(line, n, m, magic, tw, c, out);
    else
        stage<INV, 2>(line, n, m, magic, tw, c, out);
}

// The transform of a line: load(index) gives its inputs, store(index, value)
// takes its outputs.  With KEEP the outputs stay in shared memory (after a
// barrier) and store is not called.
template <bool INV, bool KEEP, typename V, typename Load, typename Store>
__device__ __forceinline__ void line_transform(const Line<V>& line, const DfStages& s, const int32_t* pos,
                                               const typename Mem<V>::T* tw, const DfConsts& c, Load load,
                                               Store store) {
    if (s.radix[0] == 4)
        first_stage<INV, 4>(line, s, pos, c, load);
    else
        first_stage<INV, 2>(line, s, pos, c, load);
    __syncthreads();
    int m = s.radix[0];
    const int in_place = KEEP ? s.ns : s.ns - 1;
    for (int k = 1; k < in_place; ++k) {
        any_stage<INV>(s.radix[k], line, s.n, m, s.magic[k], tw + s.tw[k], c,
                       [&](int i, const V& v) { line.st(i, v); });
        __syncthreads();
        m *= s.radix[k];
    }
    if (KEEP) return;
    if (s.ns == 1) {
        for (int i = threadIdx.x; i < s.n; i += blockDim.x) store(i, line.ld(i));
        return;
    }
    any_stage<INV>(s.radix[s.ns - 1], line, s.n, m, s.magic[s.ns - 1], tw + s.tw[s.ns - 1], c,
                   store);
}

// Only real images leave and enter these transforms, so each works on half
// of the spectrum.  With gnx and gny even, negating both indices keeps the
// checkerboard's sign, and with g' the modulated grid:
//   grid -> image: the real part of the inverse transform of g' is the
//     inverse transform of its Hermitian part h(x, y) = (g'(x, y) +
//     conj(g'(-x, -y))) / 2.  After the pass along y, row -x of h is the
//     conjugate of row x, so only rows 0..gnx/2 are transformed, and each
//     image column is the real transform of a Hermitian line: two image
//     columns c1, c2 go through one complex line as c1 + i c2.
//   image -> grid: two real image columns go through one complex line as
//     m1 + i m2 and are separated by the same symmetry (rows 0..gnx/2
//     kept); then rows 0..gnx/2 are transformed along y and row -x
//     written as the conjugate of row x.
// The halves h, (Z + conj(Z')) / 2 are float-pair operations; h itself is
// exact (a two-sum halved).

// Up to kDfBatch grids of one geometry in a launch (blockIdx.y).
constexpr int kDfBatch = 16;
struct DfBatch {
    const float2* grid[kDfBatch];
    const float* real_grid[kDfBatch];   // real parts, where grid is null
    float* image[kDfBatch];
    unsigned int* peak[kDfBatch];       // max |image| (float bits), or null
    float sh[kDfBatch], sl[kDfBatch];   // the scale as a float pair
    float post[kDfBatch];               // a second float32 factor
};

// grid -> image, pass 1: row x (0 <= x <= gnx/2) of h transformed along y; the
// image's columns [by0, by0 + ny) kept in t[(y - by0) gnxh + x].
template <typename V>
__global__ void __launch_bounds__(kDfThreads, 2) dfft_inv_rows(
    const __grid_constant__ DfBatch im, int gnx, int gny, int gnxh, int by0, int ny,
    const int32_t* pos, const typename Mem<V>::T* tw, const __grid_constant__ DfStages s,
    DfConsts c, typename Mem<V>::T* t) {
    extern __shared__ float4 sm[];
    const Line<V> line{reinterpret_cast<typename Mem<V>::T*>(sm), s.sa, s.sb};
    const int x = blockIdx.x, xm = x ? gnx - x : 0, k = blockIdx.y;
    const float2* grid = im.grid[k];
    const float* real_grid = im.real_grid[k];
    const float2* ga = grid + (int64_t)x * gny;
    const float2* gb = grid + (int64_t)xm * gny;
    const float* ra = real_grid + (int64_t)x * gny;
    const float* rb = real_grid + (int64_t)xm * gny;
    const bool real = grid == nullptr;
    t += (int64_t)k * ny * gnxh + x;
    line_transform<true, false>(
        line, s, pos, tw, c,
        [&](int y) {
            const int ym = y ? gny - y : 0;
            const float2 a = real ? make_float2(ra[y], 0.0f) : ga[y];
            const float2 b = real ? make_float2(rb[ym], 0.0f) : gb[ym];
            const V z = cadd(exact((V*)nullptr, a), exact((V*)nullptr, make_float2(b.x, -b.y)));
            return halve(z, ((x + y) & 1) ? -0.5f : 0.5f);
        },
        [&](int y, const V& v) {
            const int yr = y - by0;
            if (yr >= 0 && yr < ny) t[(int64_t)yr * gnxh] = pack(v);
        });
}

// grid -> image, pass 2: image columns 2b and 2b + 1 as one
// Hermitian-extended line c1 + i c2 transformed along x (the real part is
// column 2b, the imaginary part column 2b + 1), then the crop and correction
// of crop_correct_body (the same operations on the FP64 value: the scaled
// value rounds to the float32 of the FP64 path but for ties at half an ulp),
// the second factor and the peak.
template <typename V>
__global__ void __launch_bounds__(kDfThreads, 2) dfft_inv_cols(
    const __grid_constant__ DfBatch im, const typename Mem<V>::T* t, int gnx, int gnxh, int nx,
    int ny, int bx0, int by0, int parity, const float* corr_x, const float* corr_y,
    const float* sx, const float* sy, int sinc_mode, const int32_t* pos,
    const typename Mem<V>::T* tw, const __grid_constant__ DfStages s, DfConsts c) {
    extern __shared__ float4 sm[];
    const Line<V> line{reinterpret_cast<typename Mem<V>::T*>(sm), s.sa, s.sb};
    const int y0 = 2 * blockIdx.x, k = blockIdx.y;
    const bool two = y0 + 1 < ny;
    const typename Mem<V>::T* col1 = t + ((int64_t)k * ny + y0) * gnxh;
    const typename Mem<V>::T* col2 = col1 + (two ? gnxh : 0);
    float* image = im.image[k] + y0;
    // both columns' pixels in one store (the columns start even)
    const bool vec = !(ny & 1) && !((uintptr_t)im.image[k] & 7);
    unsigned int* peak = im.peak[k];
    const float sh = im.sh[k], sl = im.sl[k], post = im.post[k];
    float cy[2], sfy[2] = {1.0f, 1.0f};
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int gy = by0 + y0 + (q && two);
        cy[q] = corr_y[gy];
        if (sinc_mode) sfy[q] = sy[gy];
    }
    float top = 0.0f;
    line_transform<true, false>(
        line, s, pos, tw, c,
        [&](int x) {
            const bool lower = x < gnxh;
            const int xx = lower ? x : gnx - x;
            V a = unpack(col1[xx]), b = unpack(col2[xx]);
            if (!two) b = exact((V*)nullptr, make_float2(0.0f, 0.0f));
            // c1 + i c2 with c(-x) = conj(c(x)) for the upper half
            if (!lower) {
                a = conj_of(a);
                b = conj_of(b);
            }
            return cadd(a, mul_i<true>(b));
        },
        [&](int gx, const V& w) {
            const int xr = gx - bx0;
            if (xr < 0 || xr >= nx) return;
            const float cx = corr_x[gx], sfx = sinc_mode ? sx[gx] : 1.0f;
            const float2 wl = low(w);
            float v[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const float flip = ((gx + by0 + y0 + q + parity) & 1) ? -1.0f : 1.0f;
                const float rh = flip * (q ? w.h.y : w.h.x), rl = flip * (q ? wl.y : wl.x);
                const float ph = __fmul_rn(rh, sh);
                float u = __fadd_rn(
                    ph, __fmaf_rn(rl, sh, __fmaf_rn(rh, sl, __fmaf_rn(rh, sh, -ph))));
                const float factor = __fmul_rn(cx, cy[q]);
                if (sinc_mode == 1) {
                    const float sf = __fmul_rn(sfx, sfy[q]);
                    u = fabsf(sf) > 1.0e-6f ? u * (factor / sf) : 0.0f;
                } else if (sinc_mode == 2) {
                    u = u * __fmul_rn(__fmul_rn(factor, sfx), sfy[q]);
                } else {
                    u = u * factor;
                }
                v[q] = __fmul_rn(u, post);
            }
            float* out = image + (int64_t)xr * ny;
            if (vec) {
                *reinterpret_cast<float2*>(out) = make_float2(v[0], v[1]);
            } else {
                out[0] = v[0];
                if (two) out[1] = v[1];
            }
            top = fmaxf(top, fabsf(v[0]));   // NaN never raises the peak
            if (two) top = fmaxf(top, fabsf(v[1]));
        });
    if (peak) {
        const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(top));
        if ((threadIdx.x & 31) == 0 && m) atomicMax(peak, m);
    }
}

// The models and model grids of a launch (blockIdx.y).
struct DfModels {
    const float* model[kDfBatch];
    float2* grid[kDfBatch];
};

// image -> grid, pass 1: columns 2b and 2b + 1 of the apodised, modulated
// model (zero outside the image's rows) as one line m1 + i m2 transformed
// along x, separated into each column's half spectrum t[x pitch + y], x <=
// gnx/2.
template <typename V>
__global__ void __launch_bounds__(kDfThreads, 2) dfft_fwd_cols(
    const __grid_constant__ DfModels im, int nx, int ny, int gnx, int gnxh, int bx0, int by0,
    int pitch, const float* corr_x, const float* corr_y, const float* sinc_x,
    const float* sinc_y, const int32_t* pos, const typename Mem<V>::T* tw,
    const __grid_constant__ DfStages s, DfConsts c, typename Mem<V>::T* t) {
    extern __shared__ float4 sm[];
    const Line<V> line{reinterpret_cast<typename Mem<V>::T*>(sm), s.sa, s.sb};
    const int y0 = 2 * blockIdx.x, gy0 = by0 + y0;
    const bool two = y0 + 1 < ny;
    const float* model = im.model[blockIdx.y] + y0;
    const bool vec = !(ny & 1) && !((uintptr_t)im.model[blockIdx.y] & 7);
    t += (int64_t)blockIdx.y * pitch * gnxh + y0;
    line_transform<false, true>(
        line, s, pos, tw, c,
        [&](int gx) {
            float v[2] = {0.0f, 0.0f};
            if (gx >= bx0 && gx < bx0 + nx) {
                const float* in = model + (int64_t)(gx - bx0) * ny;
                float2 px = make_float2(0.0f, 0.0f);
                if (vec) {
                    px = *reinterpret_cast<const float2*>(in);
                } else {
                    px.x = in[0];
                    if (two) px.y = in[1];
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q && !two) break;
                    const int gy = gy0 + q;
                    // apodize_body's operations
                    float f = __fmul_rn(corr_x[gx], corr_y[gy]);
                    if (sinc_x) f = __fmul_rn(__fmul_rn(f, sinc_x[gx]), sinc_y[gy]);
                    const float u = (q ? px.y : px.x) * f;
                    v[q] = ((gx + gy) & 1) ? -u : u;
                }
            }
            return exact((V*)nullptr, make_float2(v[0], v[1]));
        },
        [](int, const V&) {});
    for (int x = threadIdx.x; x < gnxh; x += blockDim.x) {
        const V a = line.ld(x), b = conj_of(line.ld(x ? gnx - x : 0));
        // column 1: (Z(x) + conj(Z(-x))) / 2; column 2: (Z(x) - conj(Z(-x))) / 2i
        // (the spare column of an odd last pair goes to the pitch's padding)
        store_two(t + (int64_t)x * pitch, halve(cadd(a, b), 0.5f),
                  halve(mul_i<false>(csub(a, b)), 0.5f));
    }
}

// image -> grid, pass 2: row x (0 <= x <= gnx/2) transformed along y
// (columns outside [by0, by0 + ny) are zero), the output checkerboard, float32
// grid; row -x written as the conjugate of row x at -y.
template <typename V>
__global__ void __launch_bounds__(kDfThreads, 2) dfft_fwd_rows(
    const __grid_constant__ DfModels im, const typename Mem<V>::T* t, int gnx, int gny, int gnxh,
    int ny, int by0, int pitch, int parity, const int32_t* pos, const typename Mem<V>::T* tw,
    const __grid_constant__ DfStages s, DfConsts c) {
    extern __shared__ float4 sm[];
    const Line<V> line{reinterpret_cast<typename Mem<V>::T*>(sm), s.sa, s.sb};
    const int x = blockIdx.x;
    const typename Mem<V>::T* row = t + ((int64_t)blockIdx.y * gnxh + x) * pitch;
    const bool mirror = x != 0 && x != gnxh - 1;
    float2* out = im.grid[blockIdx.y] + (int64_t)x * gny;
    float2* out_m = im.grid[blockIdx.y] + (int64_t)(gnx - x) * gny;
    line_transform<false, false>(
        line, s, pos, tw, c,
        [&](int y) {
            const int yr = y - by0;
            return yr >= 0 && yr < ny ? unpack(row[yr])
                                      : exact((V*)nullptr, make_float2(0.0f, 0.0f));
        },
        [&](int y, const V& w) {
            float2 v = rounded(w);
            if ((x + y + parity) & 1) v = make_float2(-v.x, -v.y);
            out[y] = v;
            if (mirror) out_m[y ? gny - y : 0] = make_float2(v.x, -v.y);
        });
}

void split(double v, float* h, float* l) {
    *h = (float)v;
    *l = (float)(v - (double)*h);
}

DfConsts consts() {
    const double pi = 3.14159265358979323846;
    DfConsts c;
    split(std::cos(2.0 * pi / 5.0), &c.c1h, &c.c1l);
    split(std::cos(4.0 * pi / 5.0), &c.c2h, &c.c2l);
    split(std::sin(2.0 * pi / 5.0), &c.s1h, &c.s1l);
    split(std::sin(4.0 * pi / 5.0), &c.s2h, &c.s2l);
    split(std::sqrt(3.0) / 2.0, &c.s3h, &c.s3l);
    return c;
}

// Radices for n (4s first, then 2, 3, 5); empty when n has another factor.
std::vector<int32_t> radices(int64_t n) {
    std::vector<int32_t> r;
    while (n % 4 == 0) {
        r.push_back(4);
        n /= 4;
    }
    for (int32_t f : {2, 3, 5})
        while (n % f == 0) {
            r.push_back(f);
            n /= f;
        }
    if (n != 1) r.clear();
    return r;
}

const DfPlan& plan_for(cr_ctx* ctx, int64_t n) {
    auto it = ctx->df_plans.find(n);
    if (it != ctx->df_plans.end()) return *it->second;
    const std::vector<int32_t> r = radices(n);
    if (r.empty() || (int)r.size() > kDfMaxStages) fail(CR_INVALID, "no float-pair plan");
    auto p = std::make_shared<DfPlan>();
    p->n = (int32_t)n;
    p->ns = (int32_t)r.size();
    for (size_t k = 0; k < r.size(); ++k) p->radix[k] = r[k];
    // position i = q0 + r0 (q1 + r1 (q2 + ...)) holds input sum_s q_s n / L_s
    // (L_s the product of the radices up to s); those with q0 = 0 are the
    // first stage's butterflies
    const int64_t r0 = r[0];
    std::vector<int32_t> pos((size_t)(n / r0));
    for (int64_t i = 0; i < n; i += r0) {
        int64_t rem = i, L = 1, v = 0;
        for (int32_t rs : r) {
            const int64_t q = rem % rs;
            rem /= rs;
            L *= rs;
            v += q * (n / L);
        }
        pos[(size_t)v] = (int32_t)i;
    }
    std::vector<float4> tw;
    const double pi = 3.14159265358979323846;
    int64_t m = r0;
    for (size_t k = 1; k < r.size(); ++k) {
        p->tw_at[k] = (int32_t)tw.size();
        const int64_t L = m * r[k];
        for (int64_t q = 1; q < r[k]; ++q)
            for (int64_t j = 0; j < m; ++j) {
                const double a = 2.0 * pi * (double)(q * j) / (double)L;
                float4 w;
                split(std::cos(a), &w.x, &w.z);
                split(std::sin(a), &w.y, &w.w);
                tw.push_back(w);
            }
        m = L;
    }
    if (tw.empty()) tw.push_back(make_float4(1.0f, 0.0f, 0.0f, 0.0f));
    CR_CUDA_CHECK(cudaMalloc((void**)&p->pos, pos.size() * 4));
    CR_CUDA_CHECK(cudaMalloc((void**)&p->tw, tw.size() * 16));
    CR_CUDA_CHECK(cudaMemcpy(p->pos, pos.data(), pos.size() * 4, cudaMemcpyHostToDevice));
    CR_CUDA_CHECK(cudaMemcpy(p->tw, tw.data(), tw.size() * 16, cudaMemcpyHostToDevice));
    std::vector<float2> tw1;
    for (const float4& w : tw) tw1.push_back(make_float2(w.x, w.y));
    CR_CUDA_CHECK(cudaMalloc((void**)&p->tw1, tw1.size() * 8));
    CR_CUDA_CHECK(cudaMemcpy(p->tw1, tw1.data(), tw1.size() * 8, cudaMemcpyHostToDevice));
    ctx->df_plans[n] = p;
    return *p;
}

DfStages stages(const DfPlan& p, bool single) {
    DfStages s{};
    s.n = p.n;
    s.ns = p.ns;
    // shifts with the fewest conflicts by the power of two in n (31: none)
    int e2 = 0;
    while (((p.n >> e2) & 1) == 0) ++e2;
    s.sa = e2 >= 3 ? 2 : e2 == 2 ? 8 : 31;
    s.sb = e2 >= 4 ? (p.n >= (single ? 2048 : 1024) ? 8 : 6) : e2 == 3 ? 3 : 31;
    int64_t m = 1;
    for (int k = 0; k < p.ns; ++k) {
        s.radix[k] = p.radix[k];
        s.tw[k] = p.tw_at[k];
        s.magic[k] = m > 1 ? (uint32_t)(((1ull << 32) + m - 1) / m) : 0u;
        m *= p.radix[k];
    }
    return s;
}

template <typename K>
void allow_smem(K kernel, size_t bytes) {
    CR_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)bytes));
}

}  // namespace

bool dfft_supported(int64_t gnx, int64_t gny) {
    for (int64_t n : {gnx, gny})
        if (n < 2 || n > kDfMaxN || (n & 1) || radices(n).empty()) return false;
    return true;
}

// Threads of a line's block: the radix-4 butterflies of one stage in equal
// rounds of at most kDfThreads.
static unsigned line_threads(int64_t n) {
    const int64_t nb = (n + 3) / 4, rounds = (nb + kDfThreads - 1) / kDfThreads;
    return (unsigned)(((nb + rounds - 1) / rounds + 31) / 32 * 32);
}

// whole rows of banks, which the swizzle permutes
template <typename V>
static size_t line_bytes(int64_t n) {
    return (size_t)((n + Mem<V>::kRowMask) & ~(int64_t)Mem<V>::kRowMask) *
           sizeof(typename Mem<V>::T);
}

static const float4* twiddles(const DfPlan& p, cdd*) { return p.tw; }
static const float2* twiddles(const DfPlan& p, cs1*) { return p.tw1; }

template <typename V>
static void grids_to_images(cr_ctx* ctx, cr_gridder* g, const std::vector<DfImage>& list,
                            const float* sx, const float* sy, int sinc_mode) {
    using T = typename Mem<V>::T;
    const int gnx = (int)g->info.grid_nx, gny = (int)g->info.grid_ny, gnxh = gnx / 2 + 1;
    const int nx = g->geom.nx, ny = g->geom.ny;
    const DfPlan& px = plan_for(ctx, gnx);
    const DfPlan& py = plan_for(ctx, gny);
    const DfConsts c = consts();
    const bool single = sizeof(T) == 8;
    const size_t most = std::min(list.size(), (size_t)kDfBatch);
    T* t = (T*)workspace(ctx, "dfft_t", most * ny * gnxh * sizeof(T));
    const size_t smx = line_bytes<V>(gnx), smy = line_bytes<V>(gny);
    allow_smem(dfft_inv_rows<V>, smy);
    allow_smem(dfft_inv_cols<V>, smx);
    const int parity = ((gnx / 2) + (gny / 2)) & 1;
    for (size_t k0 = 0; k0 < list.size(); k0 += kDfBatch) {
        const int nb = (int)std::min<size_t>(kDfBatch, list.size() - k0);
        DfBatch im{};
        for (int k = 0; k < nb; ++k) {
            const DfImage& e = list[k0 + k];
            im.grid[k] = e.grid;
            im.real_grid[k] = e.real_grid;
            im.image[k] = e.image;
            im.peak[k] = e.peak;
            split(e.scale, &im.sh[k], &im.sl[k]);
            im.post[k] = e.post;
        }
        dfft_inv_rows<V><<<dim3(gnxh, nb), line_threads(gny), smy, ctx->stream>>>(
            im, gnx, gny, gnxh, (int)g->info.blc_y, ny, py.pos, twiddles(py, (V*)nullptr),
            stages(py, single), c, t);
        note_launch(ctx, "dfft_inv_rows");
        dfft_inv_cols<V><<<dim3((ny + 1) / 2, nb), line_threads(gnx), smx, ctx->stream>>>(
            im, t, gnx, gnxh, nx, ny, (int)g->info.blc_x, (int)g->info.blc_y, parity,
            g->corr_x_d, g->corr_y_d, sx, sy, sinc_mode, px.pos, twiddles(px, (V*)nullptr),
            stages(px, single), c);
        note_launch(ctx, "dfft_inv_cols");
    }
}

void dfft_grids_to_images(cr_ctx* ctx, cr_gridder* g, const std::vector<DfImage>& list,
                          const float* sx, const float* sy, int sinc_mode, bool single) {
    if (single)
        grids_to_images<cs1>(ctx, g, list, sx, sy, sinc_mode);
    else
        grids_to_images<cdd>(ctx, g, list, sx, sy, sinc_mode);
}

template <typename V>
static void images_to_grids(cr_ctx* ctx, cr_gridder* g, const std::vector<DfModel>& list,
                            const float* sinc_x, const float* sinc_y) {
    using T = typename Mem<V>::T;
    const int gnx = (int)g->info.grid_nx, gny = (int)g->info.grid_ny, gnxh = gnx / 2 + 1;
    const int nx = g->geom.nx, ny = g->geom.ny;
    const int pitch = ny + (ny & 1);   // two columns in one sector
    const DfPlan& px = plan_for(ctx, gnx);
    const DfPlan& py = plan_for(ctx, gny);
    const DfConsts c = consts();
    const bool single = sizeof(T) == 8;
    const size_t most = std::min(list.size(), (size_t)kDfBatch);
    T* t = (T*)workspace(ctx, "dfft_t", most * pitch * gnxh * sizeof(T));
    const size_t smx = line_bytes<V>(gnx), smy = line_bytes<V>(gny);
    allow_smem(dfft_fwd_cols<V>, smx);
    allow_smem(dfft_fwd_rows<V>, smy);
    const int parity = ((gnx / 2) + (gny / 2)) & 1;
    for (size_t k0 = 0; k0 < list.size(); k0 += kDfBatch) {
        const int nb = (int)std::min<size_t>(kDfBatch, list.size() - k0);
        DfModels im{};
        for (int k = 0; k < nb; ++k) {
            im.model[k] = list[k0 + k].model;
            im.grid[k] = list[k0 + k].grid;
        }
        dfft_fwd_cols<V><<<dim3((ny + 1) / 2, nb), line_threads(gnx), smx, ctx->stream>>>(
            im, nx, ny, gnx, gnxh, (int)g->info.blc_x, (int)g->info.blc_y, pitch, g->corr_x_d,
            g->corr_y_d, sinc_x, sinc_y, px.pos, twiddles(px, (V*)nullptr), stages(px, single),
            c, t);
        note_launch(ctx, "dfft_fwd_cols");
        dfft_fwd_rows<V><<<dim3(gnxh, nb), line_threads(gny), smy, ctx->stream>>>(
            im, t, gnx, gny, gnxh, ny, (int)g->info.blc_y, pitch, parity, py.pos,
            twiddles(py, (V*)nullptr), stages(py, single), c);
        note_launch(ctx, "dfft_fwd_rows");
    }
}

void dfft_images_to_grids(cr_ctx* ctx, cr_gridder* g, const std::vector<DfModel>& list,
                          const float* sinc_x, const float* sinc_y, bool single) {
    if (single)
        images_to_grids<cs1>(ctx, g, list, sinc_x, sinc_y);
    else
        images_to_grids<cdd>(ctx, g, list, sinc_x, sinc_y);
}

}  // namespace cr
