// gemm_bf16.cu — out[m][n] = act(x . w^T + bias) + add on the 5th-generation tensor cores.
//
// Persistent workers walk output tiles, m fastest so that the tiles in flight share weight rows in L2.  A worker is a
// pair of CTAs (cta_group::2, tiles of 256 rows: each rank holds its 128 rows of activations and half of the tile's
// weight rows) or one CTA (tiles of 128 rows: few rows, or row tiles with weights of their own).  Warp 0 and the last warp
// feed a ring of shared-memory stages with TMA, 64 K-values of both operands per stage: warp 0 the activations through a
// tensor map (what lies beyond K arrives as zeros), the last warp the weights, copies out of blocks stored in the operand's
// layout.  Warp 1 issues tcgen05.mma into one of two TMEM accumulators (in a pair the even rank's does; the odd rank's
// copies count on the even rank's barriers), warps 2-9 read the other one back and write the finished rows (bias, softplus,
// residual; F32, BF16 or saturated F16), so that a tile's output overlaps the next tile's products.  Columns may be gate /
// up pairs, of which the activation leaves (wr_pair_args), row tiles may have weights of their own (wr_group_args), and
// activations may come from a cache's pages.  Every wait is bounded by the context's wait limit; a warp that gives up
// records an error word and all of them leave.
//
// What bounds it: the way of the operands from L2 into the SMs while tiles are narrow, the tensor cores' power on long runs.
// Measured (us, one CTA per tile of 128 rows / pairs; rows x columns x K): 2048 x 8192 x 2048 68.8 / 49.1, 2048 x 2048 x 6144
// with a residual 62.8 / 39.2 (cuBLAS without one: 52 and 37).  What the pair is made of:
// - It reads two thirds of the operands.
// - A linear copy costs its thread about 50 ns to issue, so weights lie K-block by K-block and a stage's rows are one copy
//   (with one per 64 rows 61).
// - The odd rank's copies count on the even rank's barrier (a warp that relayed them: 70 against 61).
// - Eight warps bring a tile's last results out through shared memory in 7 us, four without it took 18.
// - Experts' weights that are read by a tile or two go out of L2 first (wr_group_args::once); else they push out what every prompt
//   reads, dense weights and activations.  Nurosun prompts without / with, us, tiles of 128 rows: 4 layers of width 1024, 17 rows
//   419 / 396, 300 rows 488 / 470; width 2048, 40 rows 680 / 663, 682 rows 895 / 872; 2 layers of width 4096, 100 rows 837 / 809, 500 rows
//   974 / 931.  Tiles of 256: width 2048, 1280 rows 1181 / 1135, 1792 rows 1385 / 1341; width 4096 1675 / 1593, 1978 / 1913.  Where an expert
//   has more rows its other tiles miss them: width 4096, tiles of 256, 2560 rows 2916 / 3045, 6000 rows 6463 / 6786.
// - Weights have a warp of their own, which does not wait for the kernel ahead: a prompt of 2048 rows, 8 layers of width
//   2048, 2614 -> 2597 us, one of 1501 rows, 4 layers with experts, 1300 -> 1286.
#include <cuda_bf16.h>

#include <algorithm>

#include "gemm_bf16.cuh"
#include "tcgen05_dev.cuh"

namespace {

using wr_plan::kBM;
using wr_plan::kMapRows;
using wr_plan::kMaxN;
using wr_plan::Plan;
constexpr uint32_t kBK = 64;                             // K-values of a stage
constexpr uint32_t kOutWarps = 8, kWeightWarp = 2 + kOutWarps, kThreads = 32 * (kWeightWarp + 1);
constexpr uint32_t kABytes = kBM * kBK * 2, kRowBytes = kBK * 2;
constexpr uint32_t kMaxStages = 8, kStageBudget = 196608;
constexpr uint32_t kOutBytes = 4096;                     // a warp's 32 x 32 results on their way out
constexpr uint32_t kSmem = kStageBudget + kOutWarps * kOutBytes + 1024;

struct GemmParams {
    wr_gemm_args a;
    wr_weight w;
    uint32_t m_tiles, n_tiles, k_blocks;
    uint32_t wide, bn0, bn1;                             // the first `wide` column tiles have bn0 columns, the others bn1
    uint32_t stages, stage_bytes;
    long long wait_limit;
    int *err;
};

__device__ __forceinline__ float softplus(float x) { return fmaxf(x, 0.0f) + log1pf(expf(-fabsf(x))); }

__device__ __forceinline__ uint32_t pack_bf16(float a, float b)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ uint32_t pack_f16(float a, float b)
{
    const __half2 h = __floats2half2_rn(fminf(fmaxf(a, -65504.f), 65504.f), fminf(fmaxf(b, -65504.f), 65504.f));
    return *reinterpret_cast<const uint32_t *>(&h);
}

struct TileAt {
    uint32_t strip, n0, bn;
    bool wide;
};
__device__ __forceinline__ TileAt tile_at(const GemmParams &p, uint32_t m_tiles, uint32_t tile)
{
    const uint32_t j = tile / m_tiles;
    const bool wide = j < p.wide;
    return {tile - j * m_tiles, wide ? j * p.bn0 : p.wide * p.bn0 + (j - p.wide) * p.bn1, wide ? p.bn0 : p.bn1, wide};
}

// Residual i of a 32 x 32 piece as finish() adds it: lane l has columns 4 (l % 8) .. + 3 of rows l / 8, l / 8 + 4, ...
__device__ __forceinline__ void fetch_add(const GemmParams &p, uint32_t row0, uint32_t col0, uint32_t lane, uint32_t i, float4 &r)
{
    const uint32_t col = col0 + 4 * (lane & 7u), row = row0 + (lane >> 3) + 4 * i;
    if (p.a.add && col < ((p.w.n + 7u) & ~7u) && (col & ~15u) < p.a.pair.from && row < p.a.m)
        r = *reinterpret_cast<const float4 *>(p.a.add + (size_t)row * p.a.add_ld + col);
}

// four gate values of a row and the up values that belong to them
__device__ __forceinline__ void put_pair(const GemmParams &p, uint32_t row, uint32_t at, const float4 &g, const float4 &u)
{
    const float y0 = wr_pair_act(p.a.pair.act, p.a.pair.alpha, p.a.pair.limit, g.x, u.x);
    const float y1 = wr_pair_act(p.a.pair.act, p.a.pair.alpha, p.a.pair.limit, g.y, u.y);
    const float y2 = wr_pair_act(p.a.pair.act, p.a.pair.alpha, p.a.pair.limit, g.z, u.z);
    const float y3 = wr_pair_act(p.a.pair.act, p.a.pair.alpha, p.a.pair.limit, g.w, u.w);
    *reinterpret_cast<uint2 *>((__nv_bfloat16 *)p.a.pair.out + (size_t)row * p.a.pair.ld + at) =
        make_uint2(pack_bf16(y0, y1), pack_bf16(y2, y3));
}

// A 32 x 32 piece of finished sums, a row to a lane as the tensor core leaves them, on through shared memory: eight lanes
// write (and read the residual of) 128 bytes of one row instead of each lane sixteen bytes of a row of its own.
__device__ __forceinline__ void lay_out(uint8_t *buf, const float (&v)[32], uint32_t lane)
{
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
        *reinterpret_cast<float4 *>(buf + lane * 128u + ((c ^ (lane & 7u)) << 4)) =
            make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
    __syncwarp();
}
// where lane l finds its four columns of row l / 8 + 4 i
__device__ __forceinline__ uint8_t *piece(uint8_t *buf, uint32_t lane, uint32_t i)
{
    const uint32_t rr = (lane >> 3) + 4 * i;
    return buf + rr * 128u + (((lane & 7u) ^ (rr & 7u)) << 4);
}

// The piece's plain columns.  A worker's last tile runs this alone, with two warps to a scheduler: reads, sums and writes
// of all rows go together, without a branch between them.
template <uint32_t TYPE>
__device__ __forceinline__ void finish(const GemmParams &p, uint8_t *buf, uint32_t row0, uint32_t col0, uint32_t lane,
                                       const float4 &bias, float4 (&r)[8], bool more, uint32_t next_col)
{
    const uint32_t col = col0 + 4 * (lane & 7u), row1 = row0 + (lane >> 3);
    const bool mine = col < ((p.w.n + 7u) & ~7u) && (col & ~15u) < p.a.pair.from;
    const uint32_t rows = mine && row1 < p.a.m ? (p.a.m - row1 + 3) / 4 : 0u;           // rows i < rows are there
    float4 u[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) u[i] = *reinterpret_cast<const float4 *>(piece(buf, lane, i));
    const bool add = p.a.add != nullptr;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        u[i].x = (u[i].x + bias.x) * p.a.mul; u[i].y = (u[i].y + bias.y) * p.a.mul;
        u[i].z = (u[i].z + bias.z) * p.a.mul; u[i].w = (u[i].w + bias.w) * p.a.mul;
        u[i].x = add ? u[i].x + r[i].x : u[i].x; u[i].y = add ? u[i].y + r[i].y : u[i].y;
        u[i].z = add ? u[i].z + r[i].z : u[i].z; u[i].w = add ? u[i].w + r[i].w : u[i].w;
    }
    const size_t at = (size_t)row1 * p.a.out_ld + col, step = (size_t)4 * p.a.out_ld;
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        if (TYPE == WR_GEMM_OUT_F32) {
            if (i < rows) *reinterpret_cast<float4 *>((float *)p.a.out + at + i * step) = u[i];
        } else {
            const uint2 h = TYPE == WR_GEMM_OUT_BF16 ? make_uint2(pack_bf16(u[i].x, u[i].y), pack_bf16(u[i].z, u[i].w))
                                                     : make_uint2(pack_f16(u[i].x, u[i].y), pack_f16(u[i].z, u[i].w));
            if (i < rows) *reinterpret_cast<uint2 *>((uint16_t *)p.a.out + at + i * step) = h;
        }
    }
    if (add && more) {                                   // the residual of this warp's next piece
#pragma unroll
        for (uint32_t i = 0; i < 8; ++i) fetch_add(p, row0, next_col, lane, i, r[i]);
    }
}

// What a piece may need besides, a row at a time: gate / up pairs, softplus (in place), the BF16 copy.
__device__ __forceinline__ void finish_pairs(const GemmParams &p, uint8_t *buf, uint32_t row0, uint32_t col0, uint32_t lane)
{
    const uint32_t c = lane & 7u, col = col0 + 4 * c, group = col & ~15u;
    const bool gate = group >= p.a.pair.from && col < ((p.w.n + 7u) & ~7u) && !(c & 2u);
#pragma unroll 2
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t row = row0 + (lane >> 3) + 4 * i;
        const float4 g = *reinterpret_cast<const float4 *>(piece(buf, lane, i));
        const float4 up = *reinterpret_cast<const float4 *>(piece(buf, lane ^ 2u, i));   // two lanes on
        if (gate && row < p.a.m) put_pair(p, row, (group - p.a.pair.from) / 2 + 4 * (c & 1u), g, up);
    }
}
__device__ __forceinline__ void finish_softplus(uint8_t *buf, uint32_t lane, float4 &bias)
{
#pragma unroll 1
    for (uint32_t i = 0; i < 8; ++i) {
        float4 *u = reinterpret_cast<float4 *>(piece(buf, lane, i));
        *u = make_float4(softplus(u->x + bias.x), softplus(u->y + bias.y), softplus(u->z + bias.z), softplus(u->w + bias.w));
    }
    bias = make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void finish_copy(const GemmParams &p, uint8_t *buf, uint32_t row0, uint32_t col0, uint32_t lane, const float4 &bias)
{
    const uint32_t col = col0 + 4 * (lane & 7u);
    const bool mine = col < ((p.w.n + 7u) & ~7u) && (col & ~15u) < p.a.pair.from;
#pragma unroll 2
    for (uint32_t i = 0; i < 8; ++i) {
        const uint32_t row = row0 + (lane >> 3) + 4 * i;
        const float4 u = *reinterpret_cast<const float4 *>(piece(buf, lane, i));
        if (mine && row < p.a.m)
            *reinterpret_cast<uint2 *>((__nv_bfloat16 *)p.a.out_bf16 + (size_t)row * p.a.out_bf16_ld + col) =
                make_uint2(pack_bf16(u.x + bias.x, u.y + bias.y), pack_bf16(u.z + bias.z, u.w + bias.w));
    }
}

template <bool PAIR>
__global__ void __launch_bounds__(kThreads, 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w0_map,
                 const __grid_constant__ CUtensorMap w1_map, const GemmParams p)
{
    constexpr uint32_t kRanks = PAIR ? 2 : 1;
    extern __shared__ uint8_t smem_raw[];
    // (a pair's full and acc_empty: those of the even rank)
    __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_slot;
    uint8_t *stages = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023u) & ~(uintptr_t)1023u);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? tc5::cluster_rank() : 0u;
    const uint32_t worker = blockIdx.x / kRanks, workers = gridDim.x / kRanks;
    pdl_trigger();
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < p.stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], kRanks * kOutWarps);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        if (PAIR) tc5::alloc2(&tmem_slot, 2 * kMaxN);
        else tc5::alloc(&tmem_slot, 2 * kMaxN);
    }
    tc5::fence_before();
    if (PAIR) tc5::cluster_sync();                       // (the other rank's barriers too)
    else __syncthreads();
    tc5::fence_after();
    const uint32_t tmem = tmem_slot;
    if (warp != kWeightWarp || p.a.group.list) pdl_wait();       // (weights depend on nothing)
    const uint32_t m_tiles = p.a.group.list ? *p.a.group.count : p.m_tiles, tiles = m_tiles * p.n_tiles;

    if (warp == 0 || warp == kWeightWarp) {
        if (lane == 0) {
            const bool weights = warp != 0;
            const uint32_t w_rows = wr_weight_blocks(p.w.n) * kWBlock;
            const uint64_t first_out = l2_policy_evict_first();      // (experts' weights: see above)
            uint32_t it = 0, st = 0, phase = 0;          // stage it % stages, round it / stages
            bool ok = true;
            for (uint32_t tile = worker; tile < tiles && ok; tile += workers) {
                const TileAt t = tile_at(p, m_tiles, tile);
                const uint32_t m0 = (t.strip * kRanks + rank) * kBM;
                const uint32_t share = t.bn / kRanks, r0 = t.n0 + rank * share;     // this rank's weight rows
                const uint32_t rows = r0 < w_rows ? min(share, w_rows - r0) : 0u;
                const char *blocks = static_cast<const char *>(p.w.blocks);
                uint32_t y0 = r0;                        // (in the weights' maps)
                if (p.a.group.list) {
                    const uint32_t e = p.a.group.list[t.strip];
                    blocks += e * p.a.group.stride;
                    y0 += e * (uint32_t)(p.a.group.stride / kRowBytes);
                }
                const uint32_t np = !p.a.pages || m0 >= p.a.m ? 0u : m0 + kPageTokens < p.a.m ? 2u : 1u;
                // (a pair's boxes count whole; what they bring from beyond the weight's rows belongs to no column)
                const uint32_t bytes = PAIR ? 2 * kABytes + t.bn * kRowBytes : (p.a.pages ? np * (kABytes / 2) : kABytes) + rows * kRowBytes;
                const CUtensorMap *w_map = t.wide ? &w0_map : &w1_map;
                for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                    if (it >= p.stages && !mbar_wait(&empty[st], phase ^ 1u, p.wait_limit)) {
                        ok = false;
                        break;
                    }
                    uint8_t *a = stages + st * p.stage_bytes, *b = a + kABytes;
                    // (a stage's bytes may come before they are expected: its barrier still waits for warp 0)
                    if (weights) {
                        if (PAIR && p.a.group.once) tc5::tma_load_2d_pair_hint(b, w_map, 0, (int)(kb * w_rows + y0), &full[st], first_out);
                        else if (PAIR) tc5::tma_load_2d_pair(b, w_map, 0, (int)(kb * w_rows + y0), &full[st]);
                        else if (rows && p.a.group.once) bulk_g2s_hint(b, blocks + wr_weight_row(p.w.n, r0, kb), rows * kRowBytes, &full[st], first_out);
                        else if (rows) bulk_g2s(b, blocks + wr_weight_row(p.w.n, r0, kb), rows * kRowBytes, &full[st]);
                    } else {
                        if (rank == 0) mbar_expect_tx(&full[st], bytes);
                        if (PAIR) {
                            tc5::tma_load_2d_pair(a, &x_map, (int)(kb * kBK), (int)m0, &full[st]);
                        } else if (p.a.pages) {
                            for (uint32_t i = 0; i < np; ++i)
                                bulk_g2s(a + i * kABytes / 2,
                                         reinterpret_cast<const char *>(p.a.pages[m0 / kPageTokens + i]) + kb * kABytes / 2, kABytes / 2,
                                         &full[st]);
                        } else {
                            tc5::tma_load_2d(a, &x_map, (int)(kb * kBK), (int)m0, &full[st]);
                        }
                    }
                    ++it;
                    if (++st == p.stages) {
                        st = 0;
                        phase ^= 1;
                    }
                }
            }
            if (!ok) atomicCAS(p.err, 0, 41);
            // nothing of this CTA's may be in flight when it leaves: the last loads have landed and (unless
            // a wait ran out) the products that read them have completed (a pair's odd rank waits the limit out then)
            const uint32_t last = it < p.stages ? it : p.stages;
            for (uint32_t i = it - last; i < it; ++i)
                (void)mbar_wait(ok ? &empty[i % p.stages] : &full[i % p.stages], (i / p.stages) & 1, p.wait_limit);
        }
    } else if (warp == 1 && rank == 0) {
        const bool lead = tc5::elect_one();
        uint32_t st = 0, phase = 0, n_tile = 0;
        bool ok = true;
        for (uint32_t tile = worker; tile < tiles && ok; tile += workers, ++n_tile) {
            const uint32_t bn = tile_at(p, m_tiles, tile).bn;
            const uint32_t idesc = p.a.pages ? tc5::idesc_f16(kRanks * kBM, bn) : tc5::idesc_bf16(kRanks * kBM, bn);
            const uint32_t acc = n_tile & 1;
            if (n_tile >= 2 && !mbar_wait_warp(&acc_empty[acc], (n_tile / 2 - 1) & 1, p.wait_limit)) {
                ok = false;
                break;
            }
            tc5::fence_after();
            for (uint32_t kb = 0; kb < p.k_blocks; ++kb) {
                if (!mbar_wait_warp(&full[st], phase, p.wait_limit)) {
                    ok = false;
                    break;
                }
                tc5::fence_after();
                const uint32_t a_addr = smem_u32(stages + st * p.stage_bytes);
                const uint64_t a = tc5::desc_kmajor(a_addr), b = tc5::desc_kmajor(a_addr + kABytes);
#pragma unroll
                for (uint32_t kk = 0; kk < kBK / 16; ++kk)
                    if (lead) {
                        if (PAIR) tc5::mma2_ss(tmem + acc * kMaxN, a + 2 * kk, b + 2 * kk, idesc, (kb | kk) != 0);
                        else tc5::mma_ss(tmem + acc * kMaxN, a + 2 * kk, b + 2 * kk, idesc, (kb | kk) != 0);
                    }
                if (lead) {
                    if (PAIR) tc5::commit2(&empty[st]);
                    else tc5::commit(&empty[st]);
                }
                if (++st == p.stages) {
                    st = 0;
                    phase ^= 1;
                }
            }
            if (ok && lead) {
                if (PAIR) tc5::commit2(&acc_full[acc]);
                else tc5::commit(&acc_full[acc]);
            }
        }
        if (!ok && lane == 0) atomicCAS(p.err, 0, 42);
    } else if (warp >= 2) {                              // (not the weights' warp, see above)
        const uint32_t quarter = warp & 3, half = (warp - 2) >> 2;       // TMEM lanes this warp may read; its pieces of 32 columns
        uint8_t *buf = stages + kStageBudget + (warp - 2) * kOutBytes;
        uint32_t n_tile = 0;
        bool ok = true;
        for (uint32_t tile = worker; tile < tiles && ok; tile += workers, ++n_tile) {
            const TileAt t = tile_at(p, m_tiles, tile);
            const uint32_t row0 = (t.strip * kRanks + rank) * kBM + quarter * 32, acc = n_tile & 1;
            const uint32_t end = min(t.bn, p.w.n > t.n0 ? p.w.n - t.n0 : 0u);
            float4 r[8];
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) fetch_add(p, row0, t.n0 + half * 32, lane, i, r[i]);
            if (!mbar_wait_warp(&acc_full[acc], (n_tile / 2) & 1, p.wait_limit)) {
                ok = false;
                break;
            }
            tc5::fence_after();
#pragma unroll 1
            for (uint32_t c0 = half * 32; c0 < end; c0 += 64) {
                float v[32];
                tc5::ld32(tmem + ((quarter * 32) << 16) + acc * kMaxN + c0, v);
                tc5::wait_ld();
                lay_out(buf, v, lane);
                const uint32_t col0 = t.n0 + c0, col = col0 + 4 * (lane & 7u);
                const bool more = c0 + 64 < end;
                if (col0 + 16 >= p.a.pair.from) finish_pairs(p, buf, row0, col0, lane);
                if (col0 < p.a.pair.from) {
                    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (p.a.bias && col < ((p.w.n + 7u) & ~7u)) bias = *reinterpret_cast<const float4 *>(p.a.bias + col);
                    if (p.a.act == WR_GEMM_ACT_SOFTPLUS) finish_softplus(buf, lane, bias);
                    if (p.a.out_bf16) finish_copy(p, buf, row0, col0, lane, bias);
                    if (p.a.out_type == WR_GEMM_OUT_F32) finish<WR_GEMM_OUT_F32>(p, buf, row0, col0, lane, bias, r, more, col0 + 64);
                    else if (p.a.out_type == WR_GEMM_OUT_BF16) finish<WR_GEMM_OUT_BF16>(p, buf, row0, col0, lane, bias, r, more, col0 + 64);
                    else finish<WR_GEMM_OUT_F16>(p, buf, row0, col0, lane, bias, r, more, col0 + 64);
                }
                __syncwarp();                            // the next piece takes the buffer
            }
            tc5::fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) tc5::arrive_rank(&acc_empty[acc], 0);
                else mbar_arrive(&acc_empty[acc]);
            }
        }
        if (!ok && lane == 0) atomicCAS(p.err, 0, 43);
    }
    __syncwarp();
    tc5::fence_before();
    if (PAIR) tc5::cluster_sync();                       // nobody leaves while its barriers or operands are still used
    else __syncthreads();
    tc5::fence_after();
    if (warp == 1) {
        if (PAIR) tc5::dealloc2(tmem, 2 * kMaxN);
        else tc5::dealloc(tmem, 2 * kMaxN);
    }
}

typedef CUresult (*encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                    const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                    CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                    CUtensorMapFloatOOBfill);

int map_2d(CUtensorMap *map, const void *base, uint32_t rows, uint32_t k, uint32_t ld, uint32_t box_rows,
           CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B)
{
    static encode_tiled_fn fn = nullptr;
    if (!fn) {
        void *sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess) {
            (void)cudaGetLastError();
            return WR_CUDA_ERR_INTERNAL;
        }
        fn = (encode_tiled_fn)sym;
    }
    const cuuint64_t dims[2] = {k, rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {kBK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? WR_CUDA_OK
               : WR_CUDA_ERR_INTERNAL;
}

template <bool PAIR>
int launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_weight &w, const wr_gemm_args &a, uint32_t m_tiles,
           uint32_t workers, const Plan &pl)
{
    constexpr uint32_t ranks = PAIR ? 2 : 1, flag = PAIR ? 16u : 32u;
    if (!(ctx->attr_flags & flag)) {
        WR_CUDA_TRY(cudaFuncSetAttribute(gemm_bf16_kernel<PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
        ctx->attr_flags |= flag;
    }
    GemmParams p;
    p.a = a;
    p.w = w;
    p.m_tiles = m_tiles;
    p.wide = pl.wide;
    p.bn0 = pl.bn0;
    p.bn1 = pl.bn1;
    p.n_tiles = pl.wide + (w.n > pl.wide * pl.bn0 ? (w.n - pl.wide * pl.bn0 + pl.bn1 - 1) / pl.bn1 : 0u);
    p.k_blocks = wr_weight_blocks(w.k);
    p.stage_bytes = kABytes + (pl.wide ? pl.bn0 : pl.bn1) / ranks * kRowBytes;
    p.stages = std::min(kMaxStages, kStageBudget / p.stage_bytes);
    p.wait_limit = ctx->wait_limit;
    p.err = ctx->dev_err;
    const uint32_t grid = ranks * (uint32_t)std::min<uint64_t>((uint64_t)m_tiles * p.n_tiles, workers);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = ranks;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = PAIR ? 2 : 1;
    WR_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_bf16_kernel<PAIR>, x, PAIR ? w.maps->box[pl.bn0 / 2 / kMapRows - 1] : x,
                                   PAIR ? w.maps->box[pl.bn1 / 2 / kMapRows - 1] : x, p));
    ctx->launches++;
    WR_CUDA_TRY(cudaGetLastError());
    return WR_CUDA_OK;
}

}  // namespace

int wr_gemm_map_rows(CUtensorMap *map, const void *x, uint32_t rows, uint32_t k, uint32_t ld)
{
    return map_2d(map, x, rows, k, ld, kBM);
}

int wr_gemm_map_weight(wr_weight_maps *maps, const void *blocks, uint32_t n, uint32_t k, uint32_t count, size_t stride)
{
    const uint32_t rows = wr_weight_blocks(n) * wr_weight_blocks(k) * kWBlock + (uint32_t)((count - 1) * (stride / kRowBytes));
    for (uint32_t i = 0; i < 4; ++i) {                   // (no box has more rows than there are: plan() takes no such tiles)
        const int rc = map_2d(&maps->box[i], blocks, rows, kBK, kBK, std::min((i + 1) * kMapRows, rows), CU_TENSOR_MAP_SWIZZLE_NONE);
        if (rc != WR_CUDA_OK) return rc;
    }
    return WR_CUDA_OK;
}

int wr_skinny_map_rows(CUtensorMap *map, const void *split_rows, uint32_t k, uint32_t ld, uint32_t groups)
{
    return map_2d(map, split_rows, groups * 2 * WR_CUDA_BATCH_MAX, k, ld, 2 * WR_CUDA_BATCH_MAX);
}

int wr_gemm_launch(wr_cuda_ctx *ctx, const CUtensorMap &x, const wr_weight &w, const wr_gemm_args &a)
{
    auto plan = [&](uint32_t ranks, const auto &m_tiles, uint32_t workers) {
        return wr_plan::plan(ranks, m_tiles, w.n, wr_weight_blocks(w.n) * kWBlock, workers);
    };
    if (a.m == 0 || w.n == 0 || w.k == 0 || (a.out_ld & 7u) || (a.out_bf16_ld & 7u) || (a.add_ld & 7u) ||
        (a.pair.from != ~0u && ((a.pair.from & 15u) || (a.pair.ld & 7u))))
        return WR_CUDA_ERR_INVAL;
    const uint32_t sms = (uint32_t)ctx->sm_count;
    if (a.group.list) {
        wr_plan::Tiles likely = a.group.likely;
        for (uint32_t *t : {&likely.few, &likely.usual, &likely.many}) *t = *t ? std::min(*t, a.group.max) : a.group.max;
        if (a.group.tile == kBM) return launch<false>(ctx, x, w, a, a.group.max, sms, plan(1, likely, sms));
        if (a.group.tile != 2 * kBM || !w.maps || a.group.stride % kRowBytes || sms < 2) return WR_CUDA_ERR_INVAL;
        return launch<true>(ctx, x, w, a, a.group.max, sms / 2, plan(2, likely, sms / 2));
    }
    const uint32_t m_one = (a.m + kBM - 1) / kBM, m_two = (m_one + 1) / 2;
    const Plan one = plan(1, m_one, sms);
    if (w.maps && !a.pages && a.m > kBM && sms >= 2) {
        const Plan two = plan(2, m_two, sms / 2);
        if (two.cost <= one.cost) return launch<true>(ctx, x, w, a, m_two, sms / 2, two);
    }
    return launch<false>(ctx, x, w, a, m_one, sms, one);
}
