// gemv.cu — y[r][n] = sum_k W[n][k] x[r][k] in F32 for a few activation rows: weights stream from HBM once.
//
// Serves every projection of the F32 layer stack (src/core/kernels.c:978-1090: GGML-layout W[out][in]) and those
// of the mixed stack's F32 models.
#include <math.h>

#include <algorithm>

#include "gemm_bf16.cuh"
#include "gemm_f32.cuh"
#include "gemv.cuh"
#include "warp_reduce.cuh"

namespace {

constexpr int kGemvThreads = 128;      // 4 warps per CTA
constexpr int kGemvWarps = kGemvThreads / 32;
constexpr int kChunk = 512;            // activation floats staged per row and pass

__device__ __forceinline__ float4 ldg_stream(const float *p)
{
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}

// ---- the GEMV pair ---------------------------------------------------------
//
// y[r][n] = sum_k W[n][k] * x[r][k], optionally with RMSNorm fused on x, and a
// residual add or SiLU(gate)*up on the way out.  Three kernels, one arithmetic:
// K is cut into four quarters; inside a quarter lane l takes the 16-byte
// vectors l, l+32, ... in ascending order with fused multiply-adds, starting
// from zero; lane l then adds its four quarter sums in order; the 32 lane sums
// are added by the xor butterfly (offsets 16, 8, 4, 2, 1).  The fused norm
// multiplies x by the norm weight first and the finished sum by
// 1/sqrt(mean(x^2)+eps) last, the sum of squares following the same quarter /
// lane / butterfly order.  Because all kernels compute every output by exactly
// this recipe, a row's bits do not depend on how many rows share the call (up to
// sixteen: more take gemm_f32.cu's arithmetic) or on which kernel served it.
//
//   gemv_splitk_kernel (<= 4 activation rows): a CTA owns C weight rows and
//     its four warps take one quarter each, so every lane has all its loads in
//     flight at once and nothing is staged; x comes straight from L2.  With few
//     rows the weights are all the traffic, and one warp per weight row would
//     leave most of the device idle on a narrow output (1024 rows = 7 warps/SM).
//   gemv_batch_kernel (5 to 16 activation rows): the same split, with the activations resident in shared memory.
//   gemv_rows_kernel (more rows, or rows too long to be resident; up to 16 rows per CTA): each warp owns NW weight rows
//     and walks the four quarters itself; the activation rows of the current
//     piece of a quarter sit in shared memory for all four warps, so x costs
//     RG/(4*NW) of the weight bytes instead of RG/C.

struct KQuarters {
    uint32_t vec, per;     // 16-byte vectors in K; vectors per quarter
    __device__ __forceinline__ explicit KQuarters(uint32_t k) : vec(k / 4), per((k / 4 + 3) / 4) {}
    __device__ __forceinline__ uint32_t lo(uint32_t q) const { return q * per < vec ? q * per : vec; }
    __device__ __forceinline__ uint32_t hi(uint32_t q) const { return (q + 1) * per < vec ? (q + 1) * per : vec; }
};

__device__ __forceinline__ float sumsq4(float ss, const float4 v)
{
    return fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, fmaf(v.x, v.x, ss))));
}
__device__ __forceinline__ float4 mul4(const float4 a, const float4 b)
{
    return make_float4(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z), __fmul_rn(a.w, b.w));
}
__device__ __forceinline__ float dot4(const float4 w, const float4 x, float acc)
{
    acc = fmaf(w.x, x.x, acc);
    acc = fmaf(w.y, x.y, acc);
    acc = fmaf(w.z, x.z, acc);
    return fmaf(w.w, x.w, acc);
}
__device__ __forceinline__ float inv_rms_of(float sumsq, uint32_t k, float eps)
{
    return 1.0f / sqrtf(__fadd_rn(__fdiv_rn(sumsq, (float)k), eps));
}
__device__ __forceinline__ float silu_mul(float g, float u)
{
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), u);
}

__device__ __forceinline__ float softplus(float x)
{
    return fmaxf(x, 0.0f) + log1pf(expf(-fabsf(x)));
}
// bias and activation of a finished sum, then the residual
__device__ __forceinline__ float finish(const GemvParams &p, uint32_t s, uint32_t n, uint32_t row, float y)
{
    if (p.bias && s == 0) y = __fadd_rn(y, p.bias[n]);
    if (p.act == WR_GEMV_ACT_SOFTPLUS) y = softplus(y);
    y = __fmul_rn(y, p.mul);
    if (p.add) y = __fadd_rn(p.add[(size_t)row * p.add_stride + n], y);
    return y;
}

// ... the residual at hand
__device__ __forceinline__ float finish(const GemvParams &p, uint32_t s, uint32_t n, float y, float resid)
{
    if (p.bias && s == 0) y = __fadd_rn(y, p.bias[n]);
    if (p.act == WR_GEMV_ACT_SOFTPLUS) y = softplus(y);
    y = __fmul_rn(y, p.mul);
    return p.add ? __fadd_rn(resid, y) : y;
}

// weight rows of a CTA / warp: plain, or swiglu (first half gate rows, second half the same rows of up)
template <int NR>
__device__ __forceinline__ void weight_rows(const GemvParams &p, const GemvSeg &seg, uint32_t n0,
                                            const float *(&wrow)[NR])
{
    constexpr int H = (NR >= 2) ? NR / 2 : 1;
#pragma unroll
    for (int c = 0; c < NR; ++c) {
        uint32_t n = p.swiglu ? n0 + (c % H) : n0 + c;
        const float *base = p.swiglu ? ((c < H) ? p.seg[0].w : p.seg[1].w) : seg.w;
        if (n >= seg.n) n = seg.n - 1;               // clamped rows are computed and dropped
        wrow[c] = base + (size_t)n * p.k;
    }
}

constexpr int kPrefetchRegs = 16;        // 16-byte weight vectors a lane holds before the dependency wait

template <int RG, int C>
__global__ void __launch_bounds__(kGemvThreads) gemv_splitk_kernel(const GemvParams p)
{
    __shared__ float part[kGemvWarps][C * RG + RG][32];      // per quarter (= warp): every lane's partial sums
    __shared__ float red[C * RG + RG];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t r0 = blockIdx.y * RG;
    uint32_t cta = blockIdx.x, s = 0;
    if (!p.swiglu) {
        while (s + 1 < p.n_seg && cta >= p.cta_end[s]) ++s;
        if (s > 0) cta -= p.cta_end[s - 1];
    }
    const GemvSeg seg = p.seg[s];
    constexpr int H = (C >= 2) ? C / 2 : 1;
    const uint32_t n0 = cta * (p.swiglu ? H : C);
    const float *wrow[C];
    weight_rows<C>(p, seg, n0, wrow);
    const float *xrow[RG];
#pragma unroll
    for (int r = 0; r < RG; ++r) {
        const uint32_t row = (r0 + r < p.rows) ? r0 + r : p.rows - 1;    // clamped rows are dropped at the end
        xrow[r] = p.x + (size_t)row * p.x_stride;
    }
    const KQuarters kq(p.k);
    const uint32_t v_lo = kq.lo(warp), v_hi = kq.hi(warp);

    float acc[C][RG], ss[RG];
#pragma unroll
    for (int r = 0; r < RG; ++r) {
        ss[r] = 0.f;
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c][r] = 0.f;
    }
    // Weights do not depend on the kernel before this one: the first PV vectors of the lane's walk
    // (all of it for K up to 512 * PV) are requested before the dependency wait, so their trip from
    // HBM overlaps that kernel's tail; the activations are read after it.
    constexpr int PV = kPrefetchRegs / C;
    float4 wbuf[PV][C];
#pragma unroll
    for (int i = 0; i < PV; ++i) {
        const uint32_t v = v_lo + lane + 32u * i;
        if (v < v_hi) {
#pragma unroll
            for (int c = 0; c < C; ++c) wbuf[i][c] = ldg_stream(wrow[c] + 4 * v);
        }
    }
    pdl_wait();
    // the residual that a finishing thread adds: on its way while the sums are worked out
    constexpr int kOut = C * RG;
    float resid = 0.f;
    if (!p.swiglu && p.add && tid < kOut) {
        const uint32_t n = n0 + tid / RG, row = r0 + tid % RG;
        if (n < seg.n && row < p.rows) resid = p.add[(size_t)row * p.add_stride + n];
    }
    auto step = [&](uint32_t v, const float4 (&w)[C]) {
        float4 nw = make_float4(1.f, 1.f, 1.f, 1.f);
        if (p.norm_w) nw = *reinterpret_cast<const float4 *>(p.norm_w + 4 * v);
#pragma unroll
        for (int r = 0; r < RG; ++r) {
            float4 xv = *reinterpret_cast<const float4 *>(xrow[r] + 4 * v);
            if (p.norm_w) {
                ss[r] = sumsq4(ss[r], xv);
                xv = mul4(xv, nw);
            }
#pragma unroll
            for (int c = 0; c < C; ++c) acc[c][r] = dot4(w[c], xv, acc[c][r]);
        }
    };
#pragma unroll
    for (int i = 0; i < PV; ++i) {
        const uint32_t v = v_lo + lane + 32u * i;
        if (v < v_hi) step(v, wbuf[i]);
    }
#pragma unroll 2
    for (uint32_t v = v_lo + lane + 32u * PV; v < v_hi; v += 32) {
        float4 w[C];
#pragma unroll
        for (int c = 0; c < C; ++c) w[c] = ldg_stream(wrow[c] + 4 * v);
        step(v, w);
    }
    constexpr int M = C * RG;
#pragma unroll
    for (int i = 0; i < M; ++i) part[warp][i][lane] = acc[i / RG][i % RG];
    if (p.norm_w) {
#pragma unroll
        for (int r = 0; r < RG; ++r) part[warp][M + r][lane] = ss[r];
    }
    __syncthreads();
    // every lane adds its four quarter sums in order, then the butterfly over the lanes
    for (int idx = warp; idx < M + (p.norm_w ? RG : 0); idx += kGemvWarps) {
        float t = part[0][idx][lane];
#pragma unroll
        for (int q = 1; q < kGemvWarps; ++q) t = __fadd_rn(t, part[q][idx][lane]);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
        if (lane == 0) red[idx] = t;
    }
    __syncthreads();
    const int n_out = p.swiglu ? H * RG : C * RG;
    if (tid < n_out) {
        const int c = tid / RG, r = tid % RG;
        const uint32_t n = n0 + c, row = r0 + r;
        if (n < seg.n && row < p.rows) {
            const float inv = p.norm_w ? inv_rms_of(red[M + r], p.k, p.eps) : 1.0f;
            float y = __fmul_rn(red[c * RG + r], inv);
            if (p.swiglu) {
                const float u = __fmul_rn(red[(c + H) * RG + r], inv);
                seg.out[(size_t)row * seg.out_stride + n] = silu_mul(y, u);
            } else {
                seg.out[(size_t)row * seg.out_stride + n] = finish(p, s, n, y, resid);
            }
        }
    }
}

// The same recipe for five to sixteen rows, with the activations resident.  16 rows of the Qwen3-0.6B shape, us per launch: o and
// down projections 32 -> 10.4, gate / up 47 -> 23, q / k / v 27 -> 16, head 446 -> 215; a step 7.75 -> 5.07 ms.
//  What bounded gemv_rows_kernel was latency:
// every 512 values of x were staged between two block-wide barriers, with two weight vectors in flight per lane (16 rows,
// 1024 x 3072: 32 us where HBM takes 1.9).  Here a CTA keeps RG rows of x in shared memory for good and walks tiles of
// 4 groups x 4 weight rows; a group's four warps take one quarter of K each, as in gemv_splitk_kernel, so that narrow
// outputs fill the device too, and no barrier stands between a warp's loads.  Row groups beyond RG rows are other CTAs
// that walk the same tiles at the same time: their weights come from L2.
// x lies as pairs of rows (two K-values of rows 2j and 2j + 1 to 16 bytes), so that one packed fused multiply-add serves
// two rows; shared memory is read RG * 4 bytes per four weights of each of four rows: at most 7 us per 16 million weights
// of 16 rows, under the 9.6 that HBM takes.
constexpr int kBatchThreads = 512, kBatchGroups = 4, kBatchC = 4;

__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t a, uint64_t b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

template <int RG> constexpr size_t batch_smem(uint32_t k) { return (size_t)RG * k * 4 + (size_t)kBatchGroups * 4 * kBatchC * RG * 128; }

template <int RG>
__global__ void __launch_bounds__(kBatchThreads, 1) gemv_batch_kernel(const GemvParams p, uint32_t tiles, uint32_t row_groups)
{
    constexpr int C = kBatchC, J = RG / 2, kVecs = 2;        // weight rows of a warp, row pairs, vectors in flight
    extern __shared__ float4 xs[];                            // [J][2][vec], then the quarters' sums
    __shared__ float inv_rms[RG];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, group = warp >> 2, quarter = warp & 3;
    const KQuarters kq(p.k);
    float *parts = reinterpret_cast<float *>(xs + (size_t)RG * kq.vec);
    const uint32_t r0 = (blockIdx.x % row_groups) * RG;       // (the grid is a multiple of row_groups)
    const uint32_t units = tiles * row_groups, v_lo = kq.lo(quarter) + lane, v_hi = kq.hi(quarter);

    const float *wrow[C];
    uint32_t s = 0, n0 = 0;
    auto find = [&](uint32_t unit) {
        uint32_t cta = unit / row_groups;
        s = 0;
        if (!p.swiglu) {
            while (s + 1 < p.n_seg && cta >= p.cta_end[s]) ++s;
            if (s > 0) cta -= p.cta_end[s - 1];
        }
        n0 = (cta * kBatchGroups + group) * (p.swiglu ? C / 2 : C);
        weight_rows<C>(p, p.seg[s], n0, wrow);
    };
    float4 w[kVecs][C];
    auto load = [&](uint32_t v) {
#pragma unroll
        for (int u = 0; u < kVecs; ++u)
            if (v + 32 * u < v_hi) {
#pragma unroll
                for (int c = 0; c < C; ++c) w[u][c] = ldg_stream(wrow[c] + 4 * (v + 32 * u));
            }
    };
    find(blockIdx.x);
    load(v_lo);                                               // weights need no kernel before this one
    pdl_wait();

    // x (times the norm weight) into shared memory: a warp per row pair and quarter, which also has the quarter's lane
    // sums of squares in the recipe's order
    if (warp < 4 * J) {
        const int j = warp >> 2;
        const float *xa = p.x + (size_t)(r0 + 2 * j) * p.x_stride, *xb = xa + p.x_stride;
        const bool a_in = r0 + 2 * j < p.rows, b_in = r0 + 2 * j + 1 < p.rows;
        float sa = 0.f, sb = 0.f;
#pragma unroll 4
        for (uint32_t v = v_lo; v < v_hi; v += 32) {
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
            if (a_in) a = *reinterpret_cast<const float4 *>(xa + 4 * v);
            if (b_in) b = *reinterpret_cast<const float4 *>(xb + 4 * v);
            if (p.norm_w) {
                const float4 nw = *reinterpret_cast<const float4 *>(p.norm_w + 4 * v);
                sa = sumsq4(sa, a);
                sb = sumsq4(sb, b);
                a = mul4(a, nw);
                b = mul4(b, nw);
            }
            xs[(size_t)(2 * j) * kq.vec + v] = make_float4(a.x, b.x, a.y, b.y);
            xs[(size_t)(2 * j + 1) * kq.vec + v] = make_float4(a.z, b.z, a.w, b.w);
        }
        parts[((2 * j) * 4 + quarter) * 32 + lane] = sa;
        parts[((2 * j + 1) * 4 + quarter) * 32 + lane] = sb;
    }
    __syncthreads();
    if (p.norm_w && warp < RG) {
        float t = parts[(warp * 4) * 32 + lane];
#pragma unroll
        for (int q = 1; q < 4; ++q) t = __fadd_rn(t, parts[(warp * 4 + q) * 32 + lane]);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
        if (lane == 0) inv_rms[warp] = inv_rms_of(t, p.k, p.eps);
    }
    __syncthreads();

    uint64_t *mine = reinterpret_cast<uint64_t *>(parts) + (size_t)group * 4 * C * J * 32;    // this group's [quarter][c][row pair][lane]
    for (uint32_t unit = blockIdx.x; unit < units; unit += gridDim.x) {
        uint64_t acc[C][J];
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int j = 0; j < J; ++j) acc[c][j] = 0;
        const uint32_t seg_at = s, n_at = n0;
        for (uint32_t v = v_lo; v < v_hi; v += 32 * kVecs) {
#pragma unroll
            for (int u = 0; u < kVecs; ++u) {
                const uint32_t at = v + 32 * u;
                if (at >= v_hi) break;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint64_t w0[C], w1[C];
#pragma unroll
                    for (int c = 0; c < C; ++c) {
                        w0[c] = h ? pack2(w[u][c].z, w[u][c].z) : pack2(w[u][c].x, w[u][c].x);
                        w1[c] = h ? pack2(w[u][c].w, w[u][c].w) : pack2(w[u][c].y, w[u][c].y);
                    }
#pragma unroll
                    for (int j = 0; j < J; ++j) {
                        const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(&xs[(size_t)(2 * j + h) * kq.vec + at]);
#pragma unroll
                        for (int c = 0; c < C; ++c) fma2(acc[c][j], w0[c], x.x);
#pragma unroll
                        for (int c = 0; c < C; ++c) fma2(acc[c][j], w1[c], x.y);
                    }
                }
            }
            if (v + 32 * kVecs < v_hi) load(v + 32 * kVecs);
        }
        if (unit + gridDim.x < units) {                       // the next tile's first vectors, ahead of this one's reduction
            find(unit + gridDim.x);
            load(v_lo);
        }
#pragma unroll
        for (int c = 0; c < C; ++c)
#pragma unroll
            for (int j = 0; j < J; ++j) mine[((quarter * C + c) * J + j) * 32 + lane] = acc[c][j];
        asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");
        // RG of the C * RG sums per warp, two rows to a pair: one weight row, or (swiglu) half the rows of a gate row and
        // its up row
        float v[RG];
#pragma unroll
        for (int i = 0; i < J; ++i) {
            const int c = !p.swiglu ? quarter : (quarter >> 1) + (i < J / 2 ? 0 : C / 2);
            const int j = !p.swiglu ? i : (quarter & 1) * (J / 2) + i % (J / 2);
            const uint64_t *from = mine + (c * J + j) * 32 + lane;
            uint64_t t = from[0];
#pragma unroll
            for (int q = 1; q < 4; ++q) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(t) : "l"(from[q * C * J * 32]));
            v[2 * i] = __uint_as_float((uint32_t)t);
            v[2 * i + 1] = __uint_as_float((uint32_t)(t >> 32));
        }
        const uint32_t at = warp_reduce_many<RG>(v, lane);
        const GemvSeg seg = p.seg[seg_at];
        if (!p.swiglu) {
            const uint32_t n = n_at + quarter, row = r0 + at;
            if (reduce_writer<RG>(lane) && n < seg.n && row < p.rows)
                seg.out[(size_t)row * seg.out_stride + n] =
                    finish(p, seg_at, n, row, __fmul_rn(v[0], p.norm_w ? inv_rms[at] : 1.0f));
        } else {
            const float up = __shfl_xor_sync(0xffffffffu, v[0], 16);      // (the index's highest bit is lane bit 4)
            const uint32_t n = n_at + (quarter >> 1), r = (quarter & 1) * (RG / 2) + at, row = r0 + r;
            if (reduce_writer<RG>(lane) && at < (uint32_t)RG / 2 && n < seg.n && row < p.rows) {
                const float inv = p.norm_w ? inv_rms[r] : 1.0f;
                seg.out[(size_t)row * seg.out_stride + n] = silu_mul(__fmul_rn(v[0], inv), __fmul_rn(up, inv));
            }
        }
        asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");   // the sums have been read
    }
}

// RG: activation rows per CTA (row group); NW: weight rows per warp.
template <int RG, int NW>
__global__ void __launch_bounds__(kGemvThreads) gemv_rows_kernel(const GemvParams p)
{
    constexpr int kPieceVec = kChunk / 4;            // 16-byte vectors of x staged per row and pass
    __shared__ __align__(16) float xs[RG][kChunk];
    __shared__ float inv_rms[RG];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t r0 = blockIdx.y * RG;
    uint32_t cta = blockIdx.x, s = 0;
    if (!p.swiglu) {
        while (s + 1 < p.n_seg && cta >= p.cta_end[s]) ++s;
        if (s > 0) cta -= p.cta_end[s - 1];
    }
    const GemvSeg seg = p.seg[s];
    constexpr int H = (NW >= 2) ? NW / 2 : 1;
    const uint32_t n0 = (cta * kGemvWarps + warp) * (p.swiglu ? H : NW);
    const float *wrow[NW];
    weight_rows<NW>(p, seg, n0, wrow);
    const KQuarters kq(p.k);
    pdl_wait();

    if (p.norm_w) {                                  // sum of squares in the shared order
        for (int r = warp; r < RG; r += kGemvWarps) {
            float t = 0.f;
            if (r0 + r < p.rows) {
                const float *xr = p.x + (size_t)(r0 + r) * p.x_stride;
#pragma unroll 1
                for (uint32_t q = 0; q < 4; ++q) {
                    float ss = 0.f;
                    for (uint32_t v = kq.lo(q) + lane; v < kq.hi(q); v += 32)
                        ss = sumsq4(ss, *reinterpret_cast<const float4 *>(xr + 4 * v));
                    t = (q == 0) ? ss : __fadd_rn(t, ss);
                }
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) t = __fadd_rn(t, __shfl_xor_sync(0xffffffffu, t, o));
            if (lane == 0) inv_rms[r] = inv_rms_of(t, p.k, p.eps);
        }
    }

    constexpr int M = NW * RG;
    constexpr int G = (M > 32) ? 32 : M;
    constexpr int NG = M / G;
    float lane_tot[NW][RG];                          // this lane's quarter sums, added in quarter order

#pragma unroll 1
    for (uint32_t q = 0; q < 4; ++q) {
        const uint32_t v_lo = kq.lo(q), v_hi = kq.hi(q);
        float acc[NW][RG];
#pragma unroll
        for (int c = 0; c < NW; ++c)
#pragma unroll
            for (int r = 0; r < RG; ++r) acc[c][r] = 0.f;
        for (uint32_t c0 = v_lo; c0 < v_hi; c0 += kPieceVec) {
            const uint32_t nvec = (v_hi - c0 < (uint32_t)kPieceVec) ? v_hi - c0 : (uint32_t)kPieceVec;
            __syncthreads();                         // the previous piece has been consumed
            for (uint32_t i = tid; i < RG * nvec; i += kGemvThreads) {
                const uint32_t r = i / nvec, vv = i % nvec;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (r0 + r < p.rows) {
                    v = *reinterpret_cast<const float4 *>(p.x + (size_t)(r0 + r) * p.x_stride + 4 * (c0 + vv));
                    if (p.norm_w) v = mul4(v, *reinterpret_cast<const float4 *>(p.norm_w + 4 * (c0 + vv)));
                }
                *reinterpret_cast<float4 *>(&xs[r][4 * vv]) = v;
            }
            __syncthreads();
#pragma unroll 2
            for (uint32_t vv = lane; vv < nvec; vv += 32) {
                float4 w[NW];
#pragma unroll
                for (int c = 0; c < NW; ++c) w[c] = ldg_stream(wrow[c] + 4 * (c0 + vv));
#pragma unroll
                for (int r = 0; r < RG; ++r) {
                    const float4 xv = *reinterpret_cast<const float4 *>(&xs[r][4 * vv]);
#pragma unroll
                    for (int c = 0; c < NW; ++c) acc[c][r] = dot4(w[c], xv, acc[c][r]);
                }
            }
        }
#pragma unroll
        for (int c = 0; c < NW; ++c)
#pragma unroll
            for (int r = 0; r < RG; ++r) lane_tot[c][r] = (q == 0) ? acc[c][r] : __fadd_rn(lane_tot[c][r], acc[c][r]);
    }
    // the butterfly over the lanes, once, for all NW * RG sums
    float tot[NG];
    int tot_idx[NG];
#pragma unroll
    for (int g = 0; g < NG; ++g) {
        float v[G];
#pragma unroll
        for (int i = 0; i < G; ++i) v[i] = lane_tot[(g * G + i) / RG][(g * G + i) % RG];
        tot_idx[g] = warp_reduce_many<G>(v, lane) + g * G;
        tot[g] = v[0];
    }
    __syncthreads();                                 // inv_rms is complete (and visible) for every warp

    if (!p.swiglu) {
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const uint32_t c = tot_idx[g] / RG, r = tot_idx[g] % RG, n = n0 + c, row = r0 + r;
            if (reduce_writer<G>(lane) && n < seg.n && row < p.rows) {
                float y = __fmul_rn(tot[g], p.norm_w ? inv_rms[r] : 1.0f);
                seg.out[(size_t)row * seg.out_stride + n] = finish(p, s, n, row, y);
            }
        }
    } else if constexpr (NW >= 2) {
        // flat index = c * RG + r over all NW rows: gate rows are c < H, up rows c >= H.  A lane that
        // holds gate (c, r) needs up (c + H, r): with M <= 32 it sits in the same group at index
        // + H*RG, whose owner differs in one lane bit; with two groups it is this lane's other total.
        if constexpr (NG == 2) {
            const uint32_t c = tot_idx[0] / RG, r = tot_idx[0] % RG, n = n0 + c, row = r0 + r;
            // group 0 holds rows [0, 32/RG) = gate, group 1 the same positions of up
            if (n < seg.n && row < p.rows) {
                const float inv = p.norm_w ? inv_rms[r] : 1.0f;
                seg.out[(size_t)row * seg.out_stride + n] =
                    silu_mul(__fmul_rn(tot[0], inv), __fmul_rn(tot[1], inv));
            }
        } else {
            // index bits are the top log2(M) lane bits; + H*RG = + M/2 flips the highest one (lane bit 4)
            const float other = __shfl_xor_sync(0xffffffffu, tot[0], 16);
            const uint32_t c = tot_idx[0] / RG, r = tot_idx[0] % RG, n = n0 + c, row = r0 + r;
            if (reduce_writer<G>(lane) && c < (uint32_t)H && n < seg.n && row < p.rows) {
                const float inv = p.norm_w ? inv_rms[r] : 1.0f;
                seg.out[(size_t)row * seg.out_stride + n] =
                    silu_mul(__fmul_rn(tot[0], inv), __fmul_rn(other, inv));
            }
        }
    }
}

template <int RG, int NW>
void launch_gemv_t(const GemvParams &p, uint32_t ctas, cudaStream_t st)
{
    dim3 grid(ctas, (p.rows + RG - 1) / RG);
    (void)wr_launch_pdl(gemv_rows_kernel<RG, NW>, grid, dim3(kGemvThreads), 0, st, p);
}

template <int RG, int C>
void launch_splitk_t(const GemvParams &p, uint32_t ctas, cudaStream_t st)
{
    dim3 grid(ctas, (p.rows + RG - 1) / RG);
    (void)wr_launch_pdl(gemv_splitk_kernel<RG, C>, grid, dim3(kGemvThreads), 0, st, p);
}

template <int C>
void launch_splitk(const GemvParams &p, uint32_t ctas, cudaStream_t st)
{
    if (p.rows == 1) launch_splitk_t<1, C>(p, ctas, st);
    else if (p.rows == 2) launch_splitk_t<2, C>(p, ctas, st);
    else launch_splitk_t<4, C>(p, ctas, st);
}

template <int NW>
void launch_gemv_rg(const GemvParams &p, uint32_t ctas, cudaStream_t st)
{
    if (p.rows <= 8) launch_gemv_t<8, NW>(p, ctas, st);
    else launch_gemv_t<16, NW>(p, ctas, st);
}

// Weight rows per warp from the total output width: narrow outputs take one row
// per warp so that the grid still covers the device.
int weight_rows_per_warp(uint32_t n_total)
{
    if (n_total >= 32768) return 4;
    if (n_total >= 2048) return 2;
    return 1;
}


constexpr uint32_t kSplitKRowsMax = 4;
constexpr size_t kSmemMax = 232448 - 1024;               // dynamic shared memory beside the kernel's own

// CTAs and running ends of the segments for tiles of `cols` output columns
uint32_t count_tiles(GemvParams &p, uint32_t cols)
{
    if (p.swiglu) return (p.seg[0].n + cols - 1) / cols;
    uint32_t ctas = 0;
    for (uint32_t s = 0; s < p.n_seg; ++s) {
        ctas += (p.seg[s].n + cols - 1) / cols;
        p.cta_end[s] = ctas;
    }
    return ctas;
}

template <int RG>
int launch_batch(wr_cuda_ctx *ctx, GemvParams &p)
{
    constexpr uint32_t flag = RG == 8 ? 1u << 19 : 1u << 20;
    if (!(ctx->attr_flags & flag)) {
        WR_CUDA_TRY(cudaFuncSetAttribute(gemv_batch_kernel<RG>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax));
        ctx->attr_flags |= flag;
    }
    const uint32_t tiles = count_tiles(p, kBatchGroups * (p.swiglu ? kBatchC / 2 : kBatchC));
    const uint32_t row_groups = (p.rows + RG - 1) / RG, most = std::max(1u, (uint32_t)ctx->sm_count / row_groups);
    WR_CUDA_TRY(wr_launch_pdl(gemv_batch_kernel<RG>, dim3(std::min(tiles, most) * row_groups), dim3(kBatchThreads),
                              batch_smem<RG>(p.k), ctx->stream, p, tiles, row_groups));
    WR_CUDA_TRY(cudaGetLastError());
    return WR_CUDA_OK;
}

// out = act(sum of the parts + bias) mul + add for columns n0 on of one product of many rows
__global__ void __launch_bounds__(256) finish_rows_kernel(const GemvParams p, const float *parts, uint32_t n_parts, uint32_t ld,
                                                          uint32_t n0)
{
    pdl_trigger();
    pdl_wait();
    const uint32_t row = blockIdx.y, c = blockIdx.x * blockDim.x + threadIdx.x, n = n0 + c;
    if (c >= ld || n >= p.seg[0].n) return;
    float y = parts[(size_t)row * ld + c];
    for (uint32_t j = 1; j < n_parts; ++j) y = __fadd_rn(y, parts[((size_t)j * p.rows + row) * ld + c]);
    p.seg[0].out[(size_t)row * p.seg[0].out_stride + n] = finish(p, 0, n, row, y);
}

// More rows than a decode batch: the tensor-core product of gemm_f32.cu, weights and rows split into the context's
// workspace on the way.  17 rows are two passes of the GEMV over the weights; this is three (in, out and in again, the
// last two in L2 where they fit) whatever the rows, and the products at the tensor cores' rate.  Two layers of the mixed stack in
// F32, the whole call: 17 rows of width 4096 2459 -> 1464 us, 40 of 2048 1268 -> 661, 700 of 1024 4568 -> 1172.
// Split weights take kWideBytes at most: larger ones go in slices of output columns, one after the other through the same memory
// (a 151936 x 4096 head would keep 2.5 GB; with half of it 17 rows through two layers of width 4096, whose 4096 x 12288 products
// then have too few tiles for the device, take 1799 us instead of 1440).  Columns are products of their own, so slices change no bits.  The split rows take what
// F32 rows would.  WR_CUDA_ERR_NOMEM: no workspace.
constexpr size_t kWideBytes = (size_t)256 << 20;

int launch_wide(wr_cuda_ctx *ctx, GemvParams &p)
{
    auto up256 = [](size_t n) { return (n + 255u) & ~(size_t)255u; };
    bool direct = !p.bias && p.act == WR_GEMV_ACT_NONE && p.mul == 1.f && !p.add;
    const uint32_t n_out = p.swiglu ? 1u : p.n_seg;
    for (uint32_t s = 0; s < n_out; ++s)
        direct = direct && !(p.seg[s].n & 3u) && !(p.seg[s].out_stride & 3u) && !((uintptr_t)p.seg[s].out & 15u);
    if (!direct && (p.swiglu || p.n_seg > 1)) return WR_CUDA_ERR_UNSUPPORTED;
    // columns: of all segments one after the other, or of gate and up
    uint32_t n = 0;
    for (uint32_t s = 0; s < n_out; ++s) n += p.seg[s].n;
    const uint32_t parts = direct ? 1u : wr_f32_gemm_k_parts((n + 3u) & ~3u, p.k), ld = wr_split_ld(p.k);
    if (!wr_f32_gemm_covers(p.k, parts)) return WR_CUDA_ERR_UNSUPPORTED;
    auto weight_rows_of = [&](uint32_t cols) { return p.swiglu ? (cols + 7u) / 8u * 16u : (cols + 3u) & ~3u; };
    const size_t col_bytes = std::max((size_t)(p.swiglu ? 2 : 1) * ld * 4, direct ? 0 : (size_t)parts * p.rows * 4);
    const uint32_t slice = (uint32_t)std::min<size_t>(n, std::max<size_t>(kWideBytes / col_bytes / kWBlock, 1) * kWBlock);
    const uint32_t most = weight_rows_of(slice);
    const size_t b_blocks = up256(wr_split_weight_bytes(most, p.k)), b_exponent = up256((size_t)most * 4);
    const size_t b_rows = up256((size_t)2 * p.rows * ld * 2), b_scale = up256(p.rows * sizeof(wr_split_scale));
    const size_t b_parts = direct ? 0 : (size_t)parts * p.rows * most * 4;
    int rc = wr_ctx_try_ws(ctx, b_blocks + b_exponent + b_rows + b_scale + b_parts);
    if (rc != WR_CUDA_OK) return rc;
    char *at = reinterpret_cast<char *>(ctx->ws);
    wr_f32_gemm_args a{};
    wr_split_weight &w = a.source.to;
    w.k = p.k;
    w.blocks = at;
    w.exponent = reinterpret_cast<int *>(at += b_blocks);
    wr_split_rows_args r{};
    r.x = const_cast<float *>(p.x); r.x_stride = p.x_stride; r.k = p.k; r.rows = p.rows;      // (no parts: x is only read)
    r.norm_w = p.norm_w; r.eps = p.eps;
    r.out = reinterpret_cast<__half *>(at += b_exponent); r.ld = ld; r.pad = p.rows;
    r.row_scale = reinterpret_cast<wr_split_scale *>(at += b_rows);
    float *sums = reinterpret_cast<float *>(at += b_scale);
    CUtensorMap map;
    if ((rc = wr_gemm_map_rows(&map, r.out, 2 * p.rows, ld, ld)) != WR_CUDA_OK) return rc;
    a.source.pair = p.swiglu; a.x = p.x; a.x_stride = p.x_stride; a.norm_w = p.norm_w;
    a.m = a.pad = p.rows; a.row_scale = r.row_scale; a.k_parts = parts;
    for (uint32_t c0 = 0; c0 < n; c0 += slice) {
        const uint32_t c1 = std::min(n, c0 + slice);
        w.n = weight_rows_of(c1 - c0);
        a.n_seg = 0;
        uint32_t at_col = 0, k = 0;
        for (uint32_t s = 0; s < n_out; ++s, at_col += p.seg[s - 1].n) {      // what of each segment lies in the slice
            const uint32_t lo = std::max(c0, at_col), hi = std::min(c1, at_col + p.seg[s].n);
            if (lo >= hi) continue;
            a.source.src[k] = p.seg[s].w + (size_t)(lo - at_col) * p.k;
            a.source.n[k++] = hi - lo;
            a.seg[a.n_seg++] = {p.seg[s].out + (lo - at_col), hi - lo, p.seg[s].out_stride};
            if (p.swiglu) {
                a.source.src[k] = p.seg[1].w + (size_t)lo * p.k;
                a.source.n[k++] = hi - lo;
            }
        }
        for (; k < 3; ++k) {
            a.source.src[k] = nullptr;
            a.source.n[k] = 0;
        }
        if (!direct) a.seg[0] = {sums, w.n, w.n};
        if ((rc = wr_split_weights_launch(ctx, &a.source, 1)) != WR_CUDA_OK) return rc;
        if (c0 == 0 && (rc = wr_split_rows_launch(ctx, r)) != WR_CUDA_OK) return rc;
        if ((rc = wr_f32_gemm_launch(ctx, map, a)) != WR_CUDA_OK) return rc;
        if (direct) continue;
        WR_CUDA_TRY(wr_launch_pdl(finish_rows_kernel, dim3((c1 - c0 + 255) / 256, p.rows), dim3(256), 0, ctx->stream, p,
                                  (const float *)sums, parts, w.n, c0));
        ctx->launches++;
        WR_CUDA_TRY(cudaGetLastError());
    }
    return WR_CUDA_OK;
}

}  // namespace

int wr_gemv_launch(wr_cuda_ctx *ctx, GemvParams &p, uint32_t n_total_for_width)
{
    if (p.rows > WR_CUDA_BATCH_MAX && p.rows <= 65535 && !(p.x_stride & 3u) && !((uintptr_t)p.x & 15u)) {
        const int rc = launch_wide(ctx, p);
        if (rc != WR_CUDA_ERR_NOMEM && rc != WR_CUDA_ERR_UNSUPPORTED) return rc;
    }
    if (p.rows <= kSplitKRowsMax) {
        // weight rows per CTA: 2 for narrow outputs (more CTAs), 4 otherwise
        const int c = (p.swiglu || n_total_for_width >= 4096) ? 4 : 2;
        const uint32_t ctas = count_tiles(p, p.swiglu ? (uint32_t)c / 2 : (uint32_t)c);
        if (c == 4) launch_splitk<4>(p, ctas, ctx->stream);
        else launch_splitk<2>(p, ctas, ctx->stream);
        WR_CUDA_TRY(cudaGetLastError());
        return WR_CUDA_OK;
    }
    // up to a decode batch: activations resident, eight rows to a CTA, or four where eight are too long
    if (p.rows <= WR_CUDA_BATCH_MAX) {
        if (batch_smem<8>(p.k) <= kSmemMax) return launch_batch<8>(ctx, p);
        if (batch_smem<4>(p.k) <= kSmemMax) return launch_batch<4>(ctx, p);
    }
    const int nw = p.swiglu ? 2 : weight_rows_per_warp(n_total_for_width);
    const uint32_t ctas = count_tiles(p, (p.swiglu ? 1u : (uint32_t)nw) * kGemvWarps);
    cudaStream_t st = ctx->stream;
    if (nw == 4) launch_gemv_rg<4>(p, ctas, st);
    else if (nw == 2) launch_gemv_rg<2>(p, ctas, st);
    else launch_gemv_rg<1>(p, ctas, st);
    WR_CUDA_TRY(cudaGetLastError());
    return WR_CUDA_OK;
}
