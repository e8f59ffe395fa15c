// gemm_f32.cu — y[m][n] = sum_k x[m][k] W[n][k] for many F32 rows on the 5th-generation tensor cores.
//
// What bounds it: F32 FMAs.  The GEMV kernels (gemv.cu) stream the weights once per 16 rows; a prompt of 1000 rows of the
// Qwen3-0.6B shape took 121 ms = 8 TFLOP/s with them, and the FMA pipes as a whole end near 70.  The tensor cores have no
// F32 multiplier, and in their F32 accumulators every sum is rounded towards zero; but they add integers exactly.  So a row is
// held as 32-bit integers under one power of two (gemm_f32.cuh), an integer as four signed digits of base 256,
//     x w = sum over i, j of x_i w_j 256^(6 - i - j),
// and the ten digit products with i + j <= 3 are summed over K into four S32 accumulators, one for each i + j.  Nothing is
// rounded until they are put together, once per result, in 64 bits.  The six products left out are below 2^-28 of the product of
// the two rows' largest values, and 2^-31 of it in the mean square.
// Error of one product against float64 (2-norm; rounding the exact result to F32 is 2.5e-8), K of 1024 / 2048 / 4096 and Gaussian
// rows: the GEMV 9.5e-8 / 1.1e-7 / 1.3e-7, this 4.5e-8 / 3.6e-8 / 3.6e-8 (with the rounding of the residual that it is added to).
// 1000 rows, us: 4096 x 1024 35.0, gate / up of 2 x 3072 x 1024 50.2, 1024 x 3072 25.7: 2400 to 2500 TOP/s of digit products, 240 to
// 250 TFLOP/s of F32 ones (37.4, 54.8, 26.1 with each sixteen sums finished and written before the next were fetched, and
// weights in 64-row blocks).  Sixteen warps fetch: with eight the gate / up product takes 63.2.  Back to back these products
// draw what the device may (980 of 1000 W): tiles of 256 x 64 on pairs of CTAs (gemm_bf16.cu), whose output overlaps the next
// tile's products, took 33.9 and 47.2 us alone and not a microsecond off a whole prompt, as they move more per product.
// Stages: 64 K-values, all digits of both operands.  Persistent CTAs, tiles of 128 x BN, m fastest: the tiles in flight
// share weight rows in L2.
#include <math.h>

#include <algorithm>

#include "gemm_bf16.cuh"
#include "gemm_f32.cuh"
#include "tcgen05_dev.cuh"

namespace {

constexpr uint32_t kBM = 128, kBK = 64;
constexpr uint32_t kEpiWarps = 16, kThreads = 64 + 32 * kEpiWarps;
constexpr uint32_t kABytes = kBM * kBK * 2;          // two digits of a stage's values
constexpr uint32_t kDiags = 4;
constexpr uint32_t kPartMost = 32704;                // |one accumulator| <= 4 * 2^14 * K < 2^31

template <uint32_t BN> struct Tile {
    static constexpr uint32_t kBBytes = BN * kBK * 2;
    static constexpr uint32_t kStageBytes = 2 * (kABytes + kBBytes);
    static constexpr uint32_t kStages = 196608 / kStageBytes;        // 3 or 4
    static constexpr uint32_t kSmem = kStages * kStageBytes + 1024;
    static constexpr uint32_t kAccs = 128 / BN;                      // sets of accumulators
    static constexpr uint32_t kTmemCols = 512;
    static constexpr uint32_t kCols = BN / 4;                        // columns a warp finishes
};

struct GemmParams {
    wr_f32_gemm_args a;
    uint32_t m_tiles, n_tiles, k_blocks, part_blocks;
    long long wait_limit;
    int *err;
};

__device__ __forceinline__ float silu_mul(float g, float u)
{
    return __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), u);
}

__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }

// Sixteen results of a thread as they go out: values y of row `row`, columns n on.
__device__ __forceinline__ void put16(const GemmParams &p, const float (&y)[16], uint32_t part, uint32_t row, uint32_t n_at)
{
    if (p.a.source.pair) {
        float *o = p.a.seg[0].out + (size_t)row * p.a.seg[0].ld + n_at / 2;
        float z[8];
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) z[i] = silu_mul(y[i], y[8 + i]);
        *reinterpret_cast<float4 *>(o) = make_float4(z[0], z[1], z[2], z[3]);
        if (p.a.seg[0].n - n_at / 2 > 4)                         // (a multiple of 4)
            *reinterpret_cast<float4 *>(o + 4) = make_float4(z[4], z[5], z[6], z[7]);
        return;
    }
#pragma unroll
    for (uint32_t i = 0; i < 16; i += 4) {
        uint32_t n = n_at + i, s = 0;
        if (n >= p.a.source.to.n) continue;
        while (s + 1 < p.a.n_seg && n >= p.a.seg[s].n) n -= p.a.seg[s++].n;
        float *o = p.a.seg[s].out + ((size_t)part * p.a.m + row) * p.a.seg[s].ld + n;
        *reinterpret_cast<float4 *>(o) = make_float4(y[i], y[i + 1], y[i + 2], y[i + 3]);
    }
}

// The same where a power of two is not a normal F32 number, or an infinity or a NaN is among the factors.  The latter is what
// plain F32 arithmetic makes of it.
__device__ __noinline__ void put16_rare(const GemmParams &p, const float *raw, const wr_split_scale rs, uint32_t part, uint32_t row,
                                        uint32_t n_at, uint32_t k_lo, uint32_t k_hi)
{
    const wr_f32_gemm_args &a = p.a;
    float y[16];
#pragma unroll 1
    for (uint32_t i = 0; i < 16; ++i) {
        y[i] = 0.f;
        if (n_at + i >= a.source.to.n) continue;
        const int e = rs.exponent + a.source.to.exponent[n_at + i];
        if (e < kNotFinite / 2) {
            const int first = min(max(e, -126), 127);
            y[i] = raw[i] * pow2(first) * pow2(min(max(e - first, -126), 127));
        } else if (e >= kNotNumbers / 2 + kNotFinite) {
            y[i] = __int_as_float(0x7fffffff);
        } else if (const float *w = wr_split_row(a.source, n_at + i)) {
            const float *x = a.x + (size_t)row * a.x_stride;
#pragma unroll 4
            for (uint32_t k = k_lo; k < min(k_hi, a.source.to.k); k += 4) {           // (K is a multiple of 4)
                float4 v = *reinterpret_cast<const float4 *>(x + k);
                const float4 u = *reinterpret_cast<const float4 *>(w + k);
                if (a.norm_w) {
                    const float4 nw = *reinterpret_cast<const float4 *>(a.norm_w + k);
                    v = make_float4(__fmul_rn(v.x, nw.x), __fmul_rn(v.y, nw.y), __fmul_rn(v.z, nw.z), __fmul_rn(v.w, nw.w));
                }
                y[i] = fmaf(v.w, u.w, fmaf(v.z, u.z, fmaf(v.y, u.y, fmaf(v.x, u.x, y[i]))));
            }
        }
        y[i] = __fmul_rn(y[i], rs.factor);
    }
    put16(p, y, part, row, n_at);
}

template <uint32_t BN>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ GemmParams p)
{
    using T = Tile<BN>;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full[T::kStages], empty[T::kStages], acc_full[T::kAccs], acc_empty[T::kAccs];
    __shared__ uint32_t tmem_slot;
    uint8_t *stages = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023u) & ~(uintptr_t)1023u);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_trigger();
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < T::kStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (uint32_t i = 0; i < T::kAccs; ++i) {
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
    const wr_split_weight &w = p.a.source.to;
    pdl_wait();
    // a unit of work: a tile, and a part of K
    const uint32_t tiles = p.m_tiles * p.n_tiles, units = tiles * p.a.k_parts;

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t w_rows = wr_weight_blocks(w.n) * kWBlock;
            uint32_t it = 0;
            bool ok = true;
            for (uint32_t unit = blockIdx.x; unit < units && ok; unit += gridDim.x) {
                const uint32_t tile = unit % tiles, k_lo = unit / tiles * p.part_blocks;
                const uint32_t k_hi = min(k_lo + p.part_blocks, p.k_blocks);
                const uint32_t m0 = (tile % p.m_tiles) * kBM, n0 = (tile / p.m_tiles) * BN;
                const uint32_t rows = min(BN, w_rows - n0);
                for (uint32_t kb = k_lo; kb < k_hi; ++kb, ++it) {
                    const uint32_t st = it % T::kStages;
                    if (it >= T::kStages && !mbar_wait(&empty[st], (it / T::kStages - 1) & 1, p.wait_limit)) {
                        ok = false;
                        break;
                    }
                    uint8_t *a = stages + st * T::kStageBytes, *b = a + 2 * kABytes;
                    mbar_expect_tx(&full[st], 2 * (kABytes + rows * 128));
                    tc5::tma_load_2d(a, &x_map, (int)(kb * kBK), (int)m0, &full[st]);
                    tc5::tma_load_2d(a + kABytes, &x_map, (int)(kb * kBK), (int)(p.a.pad + m0), &full[st]);
                    bulk_g2s(b, w.blocks + wr_weight_row(w.n, n0, kb), rows * 128, &full[st]);
                    bulk_g2s(b + T::kBBytes, w.blocks + wr_weight_row(w.n, n0, p.k_blocks + kb), rows * 128, &full[st]);
                }
            }
            if (!ok) atomicCAS(p.err, 0, 71);
            // nothing of this CTA's may be in flight when it leaves (gemm_bf16.cu)
            const uint32_t last = it < T::kStages ? it : T::kStages;
            for (uint32_t i = it - last; i < it; ++i)
                (void)mbar_wait(ok ? &empty[i % T::kStages] : &full[i % T::kStages], (i / T::kStages) & 1, p.wait_limit);
        }
    } else if (warp == 1) {
        const bool lead = tc5::elect_one();
        constexpr uint32_t one = tc5::idesc_i8(kBM, BN), two = tc5::idesc_i8(kBM, 2 * BN);
        uint32_t it = 0, turn = 0;
        bool ok = true;
        for (uint32_t unit = blockIdx.x; unit < units && ok; unit += gridDim.x, ++turn) {
            const uint32_t k_lo = unit / tiles * p.part_blocks, k_hi = min(k_lo + p.part_blocks, p.k_blocks);
            const uint32_t acc = turn % T::kAccs, d = tmem + acc * kDiags * BN;
            if (turn >= T::kAccs && !mbar_wait_warp(&acc_empty[acc], (turn / T::kAccs - 1) & 1, p.wait_limit)) {
                ok = false;
                break;
            }
            for (uint32_t kb = k_lo; kb < k_hi; ++kb, ++it) {
                const uint32_t st = it % T::kStages;
                if (!mbar_wait_warp(&full[st], (it / T::kStages) & 1, p.wait_limit)) {
                    ok = false;
                    break;
                }
                tc5::fence_after();
                const uint32_t a_addr = smem_u32(stages + st * T::kStageBytes), b_addr = a_addr + 2 * kABytes;
                // digit i of 32 K-values of x: 64 bytes in a row for an odd one, the second half from 2 on; digits i and i + 1 of the
                // weights (i even: digits of one kind lie BN rows behind the other), or of half the rows digit i alone
                auto a_of = [&](uint32_t i, uint32_t kk) { return tc5::desc_kmajor(a_addr + (i >> 1) * kABytes) + 4 * (i & 1) + 2 * kk; };
                auto b_of = [&](uint32_t i, uint32_t kk) { return tc5::desc_kmajor(b_addr) + 2 * i + 2 * kk; };
                if (lead) {
#pragma unroll
                    for (uint32_t kk = 0; kk < kBK / 32; ++kk) {
                        const uint32_t more = kb != k_lo || kk != 0;
                        tc5::mma_i8_ss(d, a_of(0, kk), b_of(0, kk), two, more);                  // 0 0, 0 1
                        tc5::mma_i8_ss(d + 2 * BN, a_of(0, kk), b_of(2, kk), two, more);         // 0 2, 0 3
                        tc5::mma_i8_ss(d + BN, a_of(1, kk), b_of(0, kk), two, 1);                // 1 0, 1 1
                        tc5::mma_i8_ss(d + 3 * BN, a_of(1, kk), b_of(2, kk), one, 1);            // 1 2
                        tc5::mma_i8_ss(d + 2 * BN, a_of(2, kk), b_of(0, kk), two, 1);            // 2 0, 2 1
                        tc5::mma_i8_ss(d + 3 * BN, a_of(3, kk), b_of(0, kk), one, 1);            // 3 0
                    }
                    tc5::commit(&empty[st]);
                    if (kb + 1 == k_hi) tc5::commit(&acc_full[acc]);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) atomicCAS(p.err, 0, 72);
    } else {
        const uint32_t quarter = warp & 3, c_lo = (warp - 2) / 4 * T::kCols;     // TMEM lanes and columns of this warp
        uint32_t turn = 0;
        bool ok = true;
        for (uint32_t unit = blockIdx.x; unit < units && ok; unit += gridDim.x, ++turn) {
            const uint32_t tile = unit % tiles, part = unit / tiles, acc = turn % T::kAccs;
            const uint32_t k_lo = part * p.part_blocks * kBK, k_hi = k_lo + p.part_blocks * kBK;
            const uint32_t row = (tile % p.m_tiles) * kBM + quarter * 32 + lane, n0 = (tile / p.m_tiles) * BN + c_lo;
            const bool in = row < p.a.m;
            const wr_split_scale rs = in ? p.a.row_scale[row] : wr_split_scale{0.f, 0};
            if (!mbar_wait_warp(&acc_full[acc], (turn / T::kAccs) & 1, p.wait_limit)) {
                ok = false;
                break;
            }
            tc5::fence_after();
            // all of the warp's sums first: with 128 columns the next tile's products wait for the accumulators
            float raw[T::kCols];
#pragma unroll
            for (uint32_t c = 0; c < T::kCols; c += 8) {
                int v[kDiags][8];
#pragma unroll
                for (uint32_t d = 0; d < kDiags; ++d)
                    tc5::ld8(tmem + ((quarter * 32) << 16) + (acc * kDiags + d) * BN + c_lo + c, reinterpret_cast<float *>(v[d]));
                tc5::wait_ld();
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j)
                    raw[c + j] = __ll2float_rn((long long)v[0][j] * (1 << 24) + (long long)v[1][j] * (1 << 16) + (long long)v[2][j] * 256 + v[3][j]);
            }
            tc5::fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
#pragma unroll
            for (uint32_t c = 0; c < T::kCols; c += 16) {
                if (!in || n0 + c >= w.n) continue;
                float y[16];
                bool odd = false;
#pragma unroll
                for (uint32_t i = 0; i < 16; i += 4) {
                    const int4 we = *reinterpret_cast<const int4 *>(w.exponent + n0 + c + i);      // (written while this kernel may be waiting)
                    const int es[4] = {we.x, we.y, we.z, we.w};
#pragma unroll
                    for (uint32_t j = i; j < i + 4; ++j) {
                        const int e = rs.exponent + es[j - i];
                        odd = odd || (uint32_t)(e + 126) > 253u;
                        y[j] = __fmul_rn(raw[c + j] * pow2(e), rs.factor);
                    }
                }
                if (!odd) {
                    put16(p, y, part, row, n0 + c);
                } else {
                    float z[16];
#pragma unroll
                    for (uint32_t i = 0; i < 16; ++i) z[i] = raw[c + i];
                    put16_rare(p, z, rs, part, row, n0 + c, k_lo, k_hi);
                }
            }
            __syncwarp();
        }
        if (!ok && lane == 0) atomicCAS(p.err, 0, 73);
    }
    tc5::fence_before();
    __syncthreads();
    tc5::fence_after();
    if (warp == 1) tc5::dealloc(tmem, T::kTmemCols);
}

// ---- splitting

// What a row whose largest |x| has these bits is multiplied by, as an exponent: the largest power of two that leaves all of it within
// four signed digits, |x| <= 0x7f7f7f7f.
__device__ __forceinline__ int scale_exponent(uint32_t max_bits)
{
    const int e = max(max_bits >> 23, 1u) - 127;          // (denormal rows: -126)
    return ((max_bits & 0x7fffffu) <= 0x7efefeu ? 30 : 29) - e;
}
// The exponent that undoes it; infinities and NaNs are marked.
__device__ __forceinline__ int undo_exponent(uint32_t max_bits)
{
    return max_bits > 0x7f800000u ? kNotNumbers : max_bits == 0x7f800000u ? kNotFinite : max_bits == 0 ? 0 : -scale_exponent(max_bits);
}
struct Scale {
    float a, b;                                           // two factors: together up to 2^156
    __device__ __forceinline__ explicit Scale(uint32_t max_bits)
    {
        const int s = max_bits >= 0x7f800000u || max_bits == 0 ? 0 : scale_exponent(max_bits);
        a = pow2(min(s, 126));
        b = pow2(max(s - 126, 0));
    }
};

// Digits of four values: w[i] holds digit i (0 the highest) of each.  x + 0x80808080 has digit + 128 in every byte.
__device__ __forceinline__ void digits4(const float4 v, const Scale &s, uint32_t (&w)[4])
{
    auto bytes = [&](float x) { return ((uint32_t)__float2int_rn(x * s.a * s.b) + 0x80808080u) ^ 0x80808080u; };
    const uint32_t x = bytes(v.x), y = bytes(v.y), z = bytes(v.z), u = bytes(v.w);
    const uint32_t xy_lo = __byte_perm(x, y, 0x5140), zu_lo = __byte_perm(z, u, 0x5140);
    const uint32_t xy_hi = __byte_perm(x, y, 0x7362), zu_hi = __byte_perm(z, u, 0x7362);
    w[3] = __byte_perm(xy_lo, zu_lo, 0x5410);
    w[2] = __byte_perm(xy_lo, zu_lo, 0x7632);
    w[1] = __byte_perm(xy_hi, zu_hi, 0x5410);
    w[0] = __byte_perm(xy_hi, zu_hi, 0x7632);
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

// A warp per weight row: the largest magnitude, then the digits, eight values to a lane: 64 bytes of each digit per eight lanes.
// HBM bounds it: 4 bytes in per weight and 4 out (which stay in L2 where a few MB are split for the product that follows).
__global__ void __launch_bounds__(32 * kSplitWarps) split_weights_kernel(const SplitWeights p)
{
    pdl_trigger();
    uint32_t i = 0, g = blockIdx.x;
    while (i + 1 < p.count && g >= p.end[i]) ++i;
    if (i) g -= p.end[i - 1];
    const wr_split_source &s = p.s[i];
    const uint32_t lane = threadIdx.x & 31, row = g * kSplitWarps + (threadIdx.x >> 5), k = s.to.k;
    const float *src = wr_split_row(s, row);
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
    const Scale scale(top);
    pdl_wait();                                          // the blocks are read by the product before
    if (row >= wr_weight_blocks(s.to.n) * kWBlock) return;
    auto store = [&](uint32_t at, const float4 (&v)[2]) {
        uint32_t a[4], b[4];
        digits4(v[0], scale, a);
        digits4(v[1], scale, b);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)
            *reinterpret_cast<uint2 *>(s.to.blocks + wr_split_off(s.to.n, k, row, i, at)) = make_uint2(a[i], b[i]);
    };
#pragma unroll
    for (uint32_t u = 0; u < kKeep; ++u)
        if (u * 256 + lane * 8 < k_pad) store(u * 256 + lane * 8, kept[u]);
    for (uint32_t at = kKeep * 256 + lane * 8; at < k_pad; at += 256) {
        float4 v[2];
        load(at, v);
        store(at, v);
    }
    if (lane == 0 && row < s.to.n) s.to.exponent[row] = undo_exponent(top) + 24;     // (digit products are in units of 2^24)
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
    const uint32_t row = blockIdx.x, tid = threadIdx.x, vecs = p.k / 4, padded = (p.k + kWBlock - 1) / kWBlock * kWBlock / 4;
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
    const Scale scale(top);
    char *out = reinterpret_cast<char *>(p.out) + (size_t)row * p.ld * 2;
    const size_t lo_off = (size_t)p.pad * p.ld * 2;
    auto store = [&](uint32_t i, float4 v) {
        uint32_t w[4];
        digits4(v, scale, w);
        char *to = out + i / 16 * 128 + i % 16 * 4;              // (64 K-values: 64 bytes of each digit)
#pragma unroll
        for (uint32_t d = 0; d < 4; ++d) *reinterpret_cast<uint32_t *>(to + (d >> 1) * lo_off + (d & 1) * 64) = w[d];
    };
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (uint32_t u = 0; u < KEEP; ++u)
        if (u * kRowThreads + tid < padded) store(u * kRowThreads + tid, u * kRowThreads + tid < vecs ? kept[u] : zero);
    for (uint32_t i = KEEP * kRowThreads + tid; i < padded; i += kRowThreads) store(i, i < vecs ? weigh(x[i], weight_at(i)) : zero);
    if (tid == 0) {
        const float inv = weight ? 1.0f / sqrtf(__fadd_rn(__fdiv_rn(ss, (float)p.k), p.eps)) : 1.0f;
        p.row_scale[row] = {inv, undo_exponent(top)};
    }
}

template <uint32_t BN>
int launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_f32_gemm_args &a)
{
    constexpr uint32_t flag = BN == 128 ? 1u << 17 : 1u << 18;
    if (!(ctx->attr_flags & flag)) {
        WR_CUDA_TRY(cudaFuncSetAttribute(gemm_f32_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)Tile<BN>::kSmem));
        ctx->attr_flags |= flag;
    }
    GemmParams p;
    p.a = a;
    p.m_tiles = (a.m + kBM - 1) / kBM;
    p.n_tiles = (a.source.to.n + BN - 1) / BN;
    p.k_blocks = wr_weight_blocks(a.source.to.k);
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
    if (a.rows == 0 || a.k == 0 || (a.k & 3u) || (a.x_stride & 3u) || a.ld < wr_split_ld(a.k) || (a.ld & 63u)) return WR_CUDA_ERR_INVAL;
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

bool wr_f32_gemm_covers(uint32_t k, uint32_t k_parts)
{
    return (wr_weight_blocks(k) + k_parts - 1) / k_parts * kBK <= kPartMost;
}

int wr_f32_gemm_launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_f32_gemm_args &a)
{
    const wr_split_weight &w = a.source.to;
    if (a.m == 0 || w.n == 0 || w.k == 0 || a.n_seg == 0 || a.n_seg > 3 || a.k_parts == 0 || (a.k_parts > 1 && a.source.pair))
        return WR_CUDA_ERR_INVAL;
    if (!wr_f32_gemm_covers(w.k, a.k_parts)) return WR_CUDA_ERR_UNSUPPORTED;
    for (uint32_t s = 0; s < a.n_seg; ++s)
        if ((a.seg[s].n & 3u) || (a.seg[s].ld & 3u)) return WR_CUDA_ERR_INVAL;
    // The tile width that finishes first: rounds over the device times a unit's time, in hundredths of a microsecond as measured
    // (16 to 64 blocks of K).  128 columns fill the accumulators, so nothing overlaps their filling and fetch; 64 columns have
    // two sets of them, but read x twice as often.  700 rows, us with 64 and 128 columns: 4096 x 1024 30.7, 34.8; 24576 x 4096 593, 504.
    const uint32_t blocks = (wr_weight_blocks(w.k) + a.k_parts - 1) / a.k_parts;
    auto rounds = [&](uint32_t bn) {
        const uint64_t units = (uint64_t)((a.m + kBM - 1) / kBM) * ((w.n + bn - 1) / bn) * a.k_parts;
        return (units + ctx->sm_count - 1) / ctx->sm_count;
    };
    if (rounds(128) * (blocks * 76u + 390u) <= rounds(64) * (blocks * 55u + 10u) + 300u) return launch<128>(ctx, x, a);
    return launch<64>(ctx, x, a);
}
