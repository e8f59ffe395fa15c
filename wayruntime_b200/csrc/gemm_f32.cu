// gemm_f32.cu — y[m][n] = sum_k x[m][k] W[n][k] for many F32 rows on the 5th-generation tensor cores.
//
// What bounds it: F32 FMAs.  The GEMV kernels (gemv.cu) stream the weights once per 16 rows; a prompt of 1000 rows of the
// Qwen3-0.6B shape took 121 ms = 8 TFLOP/s with them, and the FMA pipes as a whole end near 70.  The tensor cores have no
// F32 multiplier, but F32 values are two F16 values each (gemm_f32.cuh), and
//     x w = hi hi + (hi lo + lo hi) + lo lo,      the last term 2^-24 of the first and left out:
// three F16 products for one F32 product, a third of the tensor rate.
//
// Sums: tcgen05 adds into an F32 accumulator and rounds every sum towards zero; a K of thousands would lose hundreds of
// such roundings, all in one direction.  So an accumulator holds 64 K-values only (cross terms first, while it is small, then
// four additions of the large ones); eight warps fetch it and add it to F32 registers that keep what rounding loses
// (Kahan).  What the four roundings take on average is known, kTowardsZero, and put back at the end.  Error of one layer of
// products against float64 (2-norm), widths 1024 / 2048 / 4096: the GEMV 2.2 / 2.5 / 3.0e-7, accumulators of 64 K-values with plain
// sums 3.6 / 4.1 / 4.7e-7, this 2.4 / 2.5 / 2.5e-7.
// Accumulators: four of 128 columns, so that the fetch may lag behind.  A kept remainder in F32 would not fit the registers: with
// spills the fetch, not the products, set the pace (1000 x 4096 x 1024: 49.7 us, 37.3 without them; nothing fetched: 31.0).
// 1000 rows, us: 4096 x 1024 37, 6144 x 1024 58, 1024 x 3072 26 (= 660 to 740 TFLOP/s of F16 products, 220 to 245 of F32 ones).
// Stages: 64 K-values of hi and lo of both operands.  Persistent CTAs, tiles of 128 x BN, m fastest: the tiles in flight
// share weight rows in L2.
#include <math.h>

#include <algorithm>

#include "gemm_bf16.cuh"
#include "gemm_f32.cuh"
#include "tcgen05_dev.cuh"

namespace {

constexpr uint32_t kBM = 128, kBK = 64;
constexpr uint32_t kEpiWarps = 8, kThreads = 64 + 32 * kEpiWarps;
constexpr uint32_t kABytes = kBM * kBK * 2;          // one of hi / lo
constexpr uint32_t kAccs = 4;
// Rounding a sum towards zero takes half a unit of its last place on average: 2^-24 times the mean of 1 / mantissa, which
// is 1 / (2 ln 2) for mantissas spread evenly over their logarithm.  Of four additions of like size the j-th has j / 4 of
// the final value: 2.5 times that.
constexpr float kTowardsZero = 2.5f * 0.7213f * 5.9604645e-8f;

template <uint32_t BN> struct Tile {
    static constexpr uint32_t kBBytes = BN * kBK * 2;
    static constexpr uint32_t kStageBytes = 2 * (kABytes + kBBytes);
    static constexpr uint32_t kStages = 196608 / kStageBytes;        // 3 or 4
    static constexpr uint32_t kSmem = kStages * kStageBytes + 1024;
    static constexpr uint32_t kTmemCols = kAccs * BN;
    static constexpr uint32_t kCols = BN / 2;                        // columns a warp finishes
};

struct GemmParams {
    wr_f32_gemm_args a;
    wr_split_weight w;
    uint32_t m_tiles, n_tiles, k_blocks, part_blocks;
    long long wait_limit;
    int *err;
};

__device__ __forceinline__ float silu_mul(float g, float u)
{
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), u);
}

__device__ __forceinline__ uint64_t pair2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

template <uint32_t BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap x_map, const GemmParams p)
{
    using T = Tile<BN>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[T::kStages], empty[T::kStages], acc_full[kAccs], acc_empty[kAccs];
    __shared__ uint32_t tmem_slot;
    uint8_t *stages = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023u) & ~(uintptr_t)1023u);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_trigger();
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < T::kStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (uint32_t i = 0; i < kAccs; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kEpiWarps);
        }
        fence_barrier_init();
    }
    if (warp == 1) tc5::alloc(&tmem_slot, T::kTmemCols);
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    const uint32_t tmem = tmem_slot;
    pdl_wait();
    // a unit of work: a tile, and a part of K
    const uint32_t tiles = p.m_tiles * p.n_tiles, units = tiles * p.a.k_parts;

    if (warp == 0) {
        if (lane == 0) {
            const size_t lo_off = (size_t)wr_weight_blocks(p.w.n) * p.k_blocks * kWBlockBytes;
            uint32_t it = 0;
            bool ok = true;
            for (uint32_t unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
                const uint32_t tile = unit % tiles, k_lo = unit / tiles * p.part_blocks;
                const uint32_t k_hi = min(k_lo + p.part_blocks, p.k_blocks);
                const uint32_t m0 = (tile % p.m_tiles) * kBM, nb0 = (tile / p.m_tiles) * (BN / kWBlock);
                const uint32_t nb = min(BN / kWBlock, wr_weight_blocks(p.w.n) - nb0);
                for (uint32_t kb = k_lo; kb < k_hi; ++kb, ++it) {
                    const uint32_t st = it % T::kStages;
                    if (it >= T::kStages && !mbar_wait(&empty[st], (it / T::kStages - 1) & 1, p.wait_limit)) {
                        ok = false;
                        break;
                    }
                    uint8_t *a = stages + st * T::kStageBytes, *b = a + 2 * kABytes;
                    mbar_expect_tx(&full[st], 2 * (kABytes + nb * kWBlockBytes));
                    tc5::tma_load_2d(a, &x_map, (int)(kb * kBK), (int)m0, &full[st]);
                    tc5::tma_load_2d(a + kABytes, &x_map, (int)(kb * kBK), (int)(p.a.pad + m0), &full[st]);
                    const char *w = p.w.blocks + ((size_t)nb0 * p.k_blocks + kb) * kWBlockBytes;
                    for (uint32_t i = 0; i < nb; ++i, w += (size_t)p.k_blocks * kWBlockBytes) {
                        bulk_g2s(b + i * kWBlockBytes, w, kWBlockBytes, &full[st]);
                        bulk_g2s(b + T::kBBytes + i * kWBlockBytes, w + lo_off, kWBlockBytes, &full[st]);
                    }
                }
            }
            if (!ok) atomicCAS(p.err, 0, 61);
            // nothing of this CTA's may be in flight when it leaves (gemm_bf16.cu)
            const uint32_t last = it < T::kStages ? it : T::kStages;
            for (uint32_t i = it - last; i < it; ++i)
                (void)mbar_wait(ok ? &empty[i % T::kStages] : &full[i % T::kStages], (i / T::kStages) & 1, p.wait_limit);
        }
    } else if (warp == 1) {
        const bool lead = tc5::elect_one();
        const uint32_t idesc = tc5::idesc_f16(kBM, BN);
        uint32_t it = 0;
        bool ok = true;
        for (uint32_t unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
            const uint32_t k_lo = unit / tiles * p.part_blocks, k_hi = min(k_lo + p.part_blocks, p.k_blocks);
            for (uint32_t kb = k_lo; kb < k_hi; ++kb, ++it) {
                const uint32_t st = it % T::kStages, acc = it % kAccs;
                if ((it >= kAccs && !mbar_wait(&acc_empty[acc], (it / kAccs - 1) & 1, p.wait_limit)) ||
                    !mbar_wait(&full[st], (it / T::kStages) & 1, p.wait_limit)) {
                    ok = false;
                    break;
                }
                tc5::fence_after();
                const uint32_t a_addr = smem_u32(stages + st * T::kStageBytes), b_addr = a_addr + 2 * kABytes;
                const uint64_t ah = tc5::desc_kmajor(a_addr), al = tc5::desc_kmajor(a_addr + kABytes);
                const uint64_t bh = tc5::desc_kmajor(b_addr), bl = tc5::desc_kmajor(b_addr + T::kBBytes);
                const uint32_t d = tmem + acc * BN;
#pragma unroll
                for (uint32_t kk = 0; kk < kBK / 16; ++kk) {
                    if (lead) tc5::mma_ss(d, al + 2 * kk, bh + 2 * kk, idesc, kk != 0);
                    if (lead) tc5::mma_ss(d, ah + 2 * kk, bl + 2 * kk, idesc, 1);
                }
#pragma unroll
                for (uint32_t kk = 0; kk < kBK / 16; ++kk)
                    if (lead) tc5::mma_ss(d, ah + 2 * kk, bh + 2 * kk, idesc, 1);
                if (lead) tc5::commit(&empty[st]);
                if (lead) tc5::commit(&acc_full[acc]);
            }
        }
        if (!ok && lane == 0) atomicCAS(p.err, 0, 62);
    } else {
        const uint32_t quarter = warp & 3, c_lo = (warp - 2) / 4 * T::kCols;     // TMEM lanes and columns of this warp
        uint32_t it = 0;
        bool ok = true;
        for (uint32_t unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
            const uint32_t tile = unit % tiles, part = unit / tiles, k_lo = part * p.part_blocks;
            const uint32_t k_hi = min(k_lo + p.part_blocks, p.k_blocks);
            const uint32_t row = (tile % p.m_tiles) * kBM + quarter * 32 + lane, n0 = (tile / p.m_tiles) * BN + c_lo;
            // pairs; `lost` is what the sums' rounding took, itself rounded to two BF16 (2^-33 of the sum: as F32 it
            // would not fit the registers)
            uint64_t sum[T::kCols / 2];
            uint32_t lost[T::kCols / 2];
#pragma unroll
            for (uint32_t c = 0; c < T::kCols / 2; ++c) sum[c] = lost[c] = 0;
            for (uint32_t kb = k_lo; kb < k_hi; ++kb, ++it) {
                const uint32_t acc = it % kAccs;
                if (!mbar_wait(&acc_full[acc], (it / kAccs) & 1, p.wait_limit)) {
                    ok = false;
                    break;
                }
                tc5::fence_after();
#pragma unroll
                for (uint32_t c0 = 0; c0 < T::kCols; c0 += 16) {
                    float v[16];
                    tc5::ld16(tmem + ((quarter * 32) << 16) + acc * BN + c_lo + c0, v);
                    tc5::wait_ld();
#pragma unroll
                    for (uint32_t c = 0; c < 16; c += 2) {
                        uint64_t &s = sum[(c0 + c) / 2];
                        uint32_t &l = lost[(c0 + c) / 2];
                        const uint64_t old = pair2(__uint_as_float(l << 16), __uint_as_float(l & 0xffff0000u));
                        const uint64_t y = sub2(pair2(v[c], v[c + 1]), old), t = add2(s, y), e = sub2(sub2(t, s), y);
                        asm("cvt.rn.bf16x2.f32 %0, %1, %2;"
                            : "=r"(l) : "f"(__uint_as_float((uint32_t)(e >> 32))), "f"(__uint_as_float((uint32_t)e)));
                        s = t;
                    }
                }
                tc5::fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[acc]);
            }
            if (ok && row < p.a.m) {
                const float rs = p.a.row_scale[row];
                auto value = [&](uint32_t c) {
                    const float y = __uint_as_float((uint32_t)(sum[c / 2] >> (32 * (c & 1u))));
                    return __fmul_rn(__fmul_rn(fmaf(y, kTowardsZero, y), __ldg(p.w.unscale + n0 + c)), rs);
                };
                if (p.a.pair) {
#pragma unroll
                    for (uint32_t c = 0; c < T::kCols; c += 16) {
                        if (n0 + c >= p.w.n) continue;
                        float *o = p.a.seg[0].out + (size_t)row * p.a.seg[0].ld + (n0 + c) / 2;
                        float y[8];
#pragma unroll
                        for (uint32_t e = 0; e < 8; ++e) y[e] = silu_mul(value(c + e), value(c + 8 + e));
                        const uint32_t left = p.a.seg[0].n - (n0 + c) / 2;           // (a multiple of 4)
                        *reinterpret_cast<float4 *>(o) = make_float4(y[0], y[1], y[2], y[3]);
                        if (left > 4) *reinterpret_cast<float4 *>(o + 4) = make_float4(y[4], y[5], y[6], y[7]);
                    }
                } else {
#pragma unroll
                    for (uint32_t c = 0; c < T::kCols; c += 4) {
                        uint32_t n = n0 + c, s = 0;
                        if (n >= p.w.n) continue;
                        while (s + 1 < p.a.n_seg && n >= p.a.seg[s].n) n -= p.a.seg[s++].n;
                        float *o = p.a.seg[s].out + ((size_t)part * p.a.m + row) * p.a.seg[s].ld + n;
                        *reinterpret_cast<float4 *>(o) = make_float4(value(c), value(c + 1), value(c + 2), value(c + 3));
                    }
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicCAS(p.err, 0, 63);
    }
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    if (warp == 1) tc5::dealloc(tmem, T::kTmemCols);
}

// ---- splitting

// Power of two that puts a row whose largest |x| has these bits into [2^14, 2^15).  Rows of zeros, and rows that hold
// infinities or NaNs (products of which are not finite either way), stay as they are.
__device__ __forceinline__ int scale_exponent(uint32_t max_bits)
{
    if (max_bits == 0 || max_bits >= 0x7f800000u) return 0;
    const int e = (int)(max_bits >> 23) - 127;            // (denormal rows: -127)
    return min(14 - e, 126);
}
__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }

__device__ __forceinline__ void split4(const float4 v, float scale, uint2 &hi, uint2 &lo)
{
    split_half2(v.x * scale, v.y * scale, hi.x, lo.x);
    split_half2(v.z * scale, v.w * scale, hi.y, lo.y);
}
__device__ __forceinline__ uint32_t abs_bits(const float4 v)
{
    return max(max(__float_as_uint(v.x) & 0x7fffffffu, __float_as_uint(v.y) & 0x7fffffffu),
               max(__float_as_uint(v.z) & 0x7fffffffu, __float_as_uint(v.w) & 0x7fffffffu));
}

struct SplitWeights {
    wr_split_source s[kSplitSources];
    uint32_t end[kSplitSources];       // running count of 8-row groups
    uint32_t count;
};

constexpr uint32_t kSplitWarps = 8;

// A warp per weight row: the largest magnitude, then hi and lo pieces of eight values, 128 bytes of a block row per eight
// lanes.  HBM: 4 bytes in per weight; the 4 bytes out stay in L2 (a layer at a time) until the product has read them.
__global__ void __launch_bounds__(32 * kSplitWarps) split_weights_kernel(const SplitWeights p)
{
    pdl_trigger();
    uint32_t i = 0, g = blockIdx.x;
    while (i + 1 < p.count && g >= p.end[i]) ++i;
    if (i) g -= p.end[i - 1];
    const wr_split_source &s = p.s[i];
    const uint32_t lane = threadIdx.x & 31, row = g * kSplitWarps + (threadIdx.x >> 5), k = s.to.k;
    const float *src = nullptr;
    if (s.pair) {
        const uint32_t at = row / 16 * 8 + row % 8;
        if (at < s.n[0]) src = s.src[row / 8 & 1] + (size_t)at * k;
    } else {
        uint32_t at = row, j = 0;
        while (j < 2 && at >= s.n[j]) at -= s.n[j++];
        if (at < s.n[j]) src = s.src[j] + (size_t)at * k;
    }
    // weights are read before the wait: nothing ever writes them
    const uint32_t k_pad = (k + kWBlock - 1) / kWBlock * kWBlock;
    constexpr uint32_t kKeep = 4;                        // pieces of eight values that a lane holds
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 kept[kKeep][2];
    auto load = [&](uint32_t at, float4 (&v)[2]) {
        v[0] = src && at < k ? __ldg(reinterpret_cast<const float4 *>(src + at)) : zero;
        v[1] = src && at + 4 < k ? __ldg(reinterpret_cast<const float4 *>(src + at + 4)) : zero;
    };
    uint32_t top = 0;
#pragma unroll
    for (uint32_t u = 0; u < kKeep; ++u) {
        load(u * 256 + lane * 8, kept[u]);
        top = max(top, max(abs_bits(kept[u][0]), abs_bits(kept[u][1])));
    }
    for (uint32_t at = kKeep * 256 + lane * 8; at < k; at += 256) {
        float4 v[2];
        load(at, v);
        top = max(top, max(abs_bits(v[0]), abs_bits(v[1])));
    }
    top = __reduce_max_sync(0xffffffffu, top);
    const int e = scale_exponent(top);
    const float scale = pow2(e);
    pdl_wait();                                          // the blocks are read by the product before
    if (row >= wr_weight_blocks(s.to.n) * kWBlock) return;
    const size_t lo_off = (size_t)wr_weight_blocks(s.to.n) * (k_pad / kWBlock) * kWBlockBytes;
    auto store = [&](uint32_t at, const float4 (&v)[2]) {
        uint2 h0, l0, h1, l1;
        split4(v[0], scale, h0, l0);
        split4(v[1], scale, h1, l1);
        char *to = s.to.blocks + wr_weight_off(k, row, at);
        *reinterpret_cast<uint4 *>(to) = make_uint4(h0.x, h0.y, h1.x, h1.y);
        *reinterpret_cast<uint4 *>(to + lo_off) = make_uint4(l0.x, l0.y, l1.x, l1.y);
    };
#pragma unroll
    for (uint32_t u = 0; u < kKeep; ++u)
        if (u * 256 + lane * 8 < k_pad) store(u * 256 + lane * 8, kept[u]);
    for (uint32_t at = kKeep * 256 + lane * 8; at < k_pad; at += 256) {
        float4 v[2];
        load(at, v);
        store(at, v);
    }
    if (lane == 0 && row < s.to.n) s.to.unscale[row] = pow2(-e);
}

constexpr uint32_t kRowThreads = 256, kMaxParts = 4;

// One block per activation row: partial sums into the residual, sum of squares and largest magnitude, then the split.  What
// bounds it is one chain of round trips per row: everything a thread reads is requested at once, the norm's weights before the
// wait, and KEEP (vectors that a thread holds) is no larger than the row asks for, so that rows fit the device in one go.
template <uint32_t KEEP>
__global__ void __launch_bounds__(kRowThreads, KEEP == 1 ? 5 : 4) split_rows_kernel(const wr_split_rows_args p)
{
    __shared__ float part_ss[kRowThreads / 32];
    __shared__ uint32_t part_top[kRowThreads / 32];
    pdl_trigger();
    const uint32_t row = blockIdx.x, tid = threadIdx.x, vecs = p.k / 4;
    float4 *x = reinterpret_cast<float4 *>(p.x + (size_t)row * p.x_stride);
    const float4 *parts = reinterpret_cast<const float4 *>(p.parts + (p.parts ? (size_t)row * p.k : 0));
    const float4 *weight = reinterpret_cast<const float4 *>(p.norm_w);
    float4 w[KEEP], kept[KEEP];
#pragma unroll
    for (uint32_t u = 0; u < KEEP; ++u)
        if (weight && u * kRowThreads + tid < vecs) w[u] = __ldg(weight + u * kRowThreads + tid);
    pdl_wait();
    float ss = 0.f;
    uint32_t top = 0;
    auto take = [&](uint32_t i) {
        float4 v = x[i];
        if (p.parts) {
            float4 z[kMaxParts];
#pragma unroll
            for (uint32_t j = 0; j < kMaxParts; ++j)
                if (j < p.n_parts) z[j] = parts[(size_t)j * p.rows * vecs + i];
#pragma unroll
            for (uint32_t j = 1; j < kMaxParts; ++j)
                if (j < p.n_parts) z[0] = make_float4(z[0].x + z[j].x, z[0].y + z[j].y, z[0].z + z[j].z, z[0].w + z[j].w);
            v = make_float4(v.x + z[0].x, v.y + z[0].y, v.z + z[0].z, v.w + z[0].w);
            x[i] = v;
        }
        return v;
    };
    auto weigh = [&](float4 v, const float4 &w) {
        if (!weight) return v;
        return make_float4(__fmul_rn(v.x, w.x), __fmul_rn(v.y, w.y), __fmul_rn(v.z, w.z), __fmul_rn(v.w, w.w));
    };
    auto look = [&](float4 v, const float4 &w) {
        ss = fmaf(v.w, v.w, fmaf(v.z, v.z, fmaf(v.y, v.y, fmaf(v.x, v.x, ss))));
        v = weigh(v, w);
        top = max(top, abs_bits(v));
        return v;
    };
    auto weight_at = [&](uint32_t i) { return weight ? __ldg(weight + i) : make_float4(1.f, 1.f, 1.f, 1.f); };
#pragma unroll
    for (uint32_t u = 0; u < KEEP; ++u)
        if (u * kRowThreads + tid < vecs) kept[u] = take(u * kRowThreads + tid);
#pragma unroll
    for (uint32_t u = 0; u < KEEP; ++u)
        if (u * kRowThreads + tid < vecs) kept[u] = look(kept[u], w[u]);
    for (uint32_t i = KEEP * kRowThreads + tid; i < vecs; i += kRowThreads) (void)look(take(i), weight_at(i));
    if (!p.out) return;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((tid & 31) == 0) {
        part_ss[tid >> 5] = ss;
        part_top[tid >> 5] = top;
    }
    __syncthreads();
    ss = part_ss[0];
    top = part_top[0];
#pragma unroll
    for (uint32_t i = 1; i < kRowThreads / 32; ++i) {
        ss += part_ss[i];
        top = max(top, part_top[i]);
    }
    const int e = scale_exponent(top);
    const float scale = pow2(e);
    __half *hi = p.out + (size_t)row * p.ld, *lo = p.out + (size_t)(p.pad + row) * p.ld;
    auto store = [&](uint32_t i, float4 v) {
        uint2 h, l;
        split4(v, scale, h, l);
        *reinterpret_cast<uint2 *>(hi + 4 * i) = h;
        *reinterpret_cast<uint2 *>(lo + 4 * i) = l;
    };
#pragma unroll
    for (uint32_t u = 0; u < KEEP; ++u)
        if (u * kRowThreads + tid < vecs) store(u * kRowThreads + tid, kept[u]);
    for (uint32_t i = KEEP * kRowThreads + tid; i < vecs; i += kRowThreads) store(i, weigh(x[i], weight_at(i)));
    if (tid == 0) {
        const float inv = weight ? 1.0f / sqrtf(__fadd_rn(__fdiv_rn(ss, (float)p.k), p.eps)) : 1.0f;
        p.row_scale[row] = inv * pow2(-e);
    }
}

template <uint32_t BN>
int launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_split_weight &w, const wr_f32_gemm_args &a)
{
    constexpr uint32_t flag = BN == 128 ? 1u << 17 : 1u << 18;
    if (!(ctx->attr_flags & flag)) {
        WR_CUDA_TRY(cudaFuncSetAttribute(gemm_f32_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)Tile<BN>::kSmem));
        ctx->attr_flags |= flag;
    }
    GemmParams p;
    p.a = a;
    p.w = w;
    p.m_tiles = (a.m + kBM - 1) / kBM;
    p.n_tiles = (w.n + BN - 1) / BN;
    p.k_blocks = wr_weight_blocks(w.k);
    p.part_blocks = (p.k_blocks + a.k_parts - 1) / a.k_parts;
    p.wait_limit = ctx->wait_limit;
    p.err = ctx->dev_err;
    const uint32_t grid = std::min<uint32_t>(p.m_tiles * p.n_tiles * a.k_parts, (uint32_t)ctx->sm_count);
    WR_CUDA_TRY(wr_launch_pdl(gemm_f32_kernel<BN>, dim3(grid), dim3(kThreads), Tile<BN>::kSmem, ctx->stream, x, p));
    ctx->launches++;
    WR_CUDA_TRY(cudaGetLastError());
    return WR_CUDA_OK;
}

}  // namespace

size_t wr_split_weight_bytes(uint32_t n, uint32_t k) { return 2 * wr_weight_bytes(n, k); }

int wr_split_weights_launch(wr_cuda_ctx *ctx, const wr_split_source *list, uint32_t count)
{
    if (count == 0 || count > kSplitSources) return WR_CUDA_ERR_INVAL;
    SplitWeights p;
    p.count = count;
    uint32_t groups = 0;
    for (uint32_t i = 0; i < kSplitSources; ++i) {
        if (i < count) {
            p.s[i] = list[i];
            groups += wr_weight_blocks(list[i].to.n) * kWBlock / kSplitWarps;
        }
        p.end[i] = groups;
    }
    WR_CUDA_TRY(wr_launch_pdl(split_weights_kernel, dim3(groups), dim3(32 * kSplitWarps), 0, ctx->stream, p));
    ctx->launches++;
    WR_CUDA_TRY(cudaGetLastError());
    return WR_CUDA_OK;
}

int wr_split_rows_launch(wr_cuda_ctx *ctx, const wr_split_rows_args &a)
{
    if (a.rows == 0 || a.k == 0 || (a.k & 3u) || (a.x_stride & 3u) || (a.ld & 7u)) return WR_CUDA_ERR_INVAL;
    if (a.parts && (a.n_parts == 0 || a.n_parts > kMaxParts)) return WR_CUDA_ERR_INVAL;
    const dim3 grid(a.rows), block(kRowThreads);
    if (a.k <= 4 * kRowThreads) WR_CUDA_TRY(wr_launch_pdl(split_rows_kernel<1>, grid, block, 0, ctx->stream, a));
    else if (a.k <= 8 * kRowThreads) WR_CUDA_TRY(wr_launch_pdl(split_rows_kernel<2>, grid, block, 0, ctx->stream, a));
    else WR_CUDA_TRY(wr_launch_pdl(split_rows_kernel<4>, grid, block, 0, ctx->stream, a));
    ctx->launches++;
    WR_CUDA_TRY(cudaGetLastError());
    return WR_CUDA_OK;
}

uint32_t wr_f32_gemm_k_parts(uint32_t n, uint32_t k)
{
    // Narrow outputs have few tiles: 8 x 8 of 128 x 128 for 1000 rows of 1024 values.  Parts keep at least 512 K-values.
    uint32_t parts = n <= 512 ? 4u : n <= 1024 ? 2u : 1u;
    while (parts > 1 && k / parts < 512) parts /= 2;
    return parts;
}

int wr_f32_gemm_launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_split_weight &w, const wr_f32_gemm_args &a)
{
    if (a.m == 0 || w.n == 0 || w.k == 0 || a.n_seg == 0 || a.n_seg > 3 || a.k_parts == 0 || (a.k_parts > 1 && a.pair))
        return WR_CUDA_ERR_INVAL;
    for (uint32_t s = 0; s < a.n_seg; ++s)
        if ((a.seg[s].n & 3u) || (a.seg[s].ld & 3u)) return WR_CUDA_ERR_INVAL;
    // The tile width that finishes first: rounds over the device times a unit's time, which goes by shared memory: 64
    // K-values are 12 products that read 4 KB of x and 32 BN bytes of W each, and 32 KB + 256 BN that arrive.
    uint32_t best = 0;
    uint64_t best_cost = ~0ull;
    for (uint32_t bn : {128u, 64u}) {
        const uint64_t units = (uint64_t)((a.m + kBM - 1) / kBM) * ((w.n + bn - 1) / bn) * a.k_parts;
        const uint64_t cost = ((units + ctx->sm_count - 1) / ctx->sm_count) * (bn + 128u);
        if (cost < best_cost) {
            best_cost = cost;
            best = bn;
        }
    }
    if (best == 128) return launch<128>(ctx, x, w, a);
    return launch<64>(ctx, x, w, a);
}
