// attn_step_small.cu — one layer-step of attention for short contexts, in ONE
// kernel: per-head QK-norm, RoPE on Q and K, the truncating F16 append of K / V
// and the attention of the new token over its session's keys.
//
// This is the reference's per-layer body between the projections and the
// output projection (src/core/session.c:458-496: wri_op_rmsnorm on the [heads,
// hd] views, wri_op_rope x2, kv_append_row x2, wri_op_gqa_attention) for the
// case the big kernels serve badly: one new token per session and at most
// kSmallMaxKeys keys, where three launches (norm, append, the split-KV decode
// kernel with its queue, arrival counters and merge warps) cost 20 us to move
// a few hundred KB.  One CTA per (session, kv head) does all of it out of shared
// memory.  Used by the device-resident layer stack (model_glue.cu) for every
// session whose own length allows it — the choice depends on that session
// alone, so a session's bits do not depend on its batch mates.
//
// Bit-level contracts kept: the cache bytes (norm as head_rmsnorm_kernel does
// it, RoPE with the reference's polynomials and separately rounded products,
// truncating F16 convert) are the ones the three-kernel path stores.  The
// softmax is the materialised form (all scores, one maximum, one sum) in F32
// with exp from the hardware; the reference's online form differs from it by
// float associativity only (kernels.c:1466-1470).
#include <algorithm>

#include "mathx_dev.cuh"
#include "wr_internal.cuh"

namespace {

// What bounds the kernel is round trips to L2: one per 256 keys for the scores and one per 128 for the values with 256 threads.
// A CTA has SETS times as many; sixteen groups of keys share the values as before, and each thread takes 8 / SETS dimensions, so
// every sum runs over the same terms in the same order whatever SETS is (the longest session of the launch decides).
// 48 CTAs, sessions of 200 to 1000 keys, 2 q heads per kv head: 34.4 -> 29.4 us.
constexpr uint32_t kSetThreads = 256;
__host__ __device__ constexpr uint32_t max_sets(uint32_t group) { return group > 4 ? 2u : 4u; }     // (registers)
inline uint32_t sets_for(uint32_t n_keys, uint32_t group)
{
    const uint32_t sets = n_keys <= 256 ? 1u : n_keys <= 512 ? 2u : 4u;
    return sets < max_sets(group) ? sets : max_sets(group);
}
constexpr uint32_t kSmallMaxKeys = WR_STEP_SMALL_MAX_KEYS;
constexpr uint32_t kSmallMaxGroup = 8;     // q heads per kv head
constexpr uint32_t kHd = 128;

struct step_small_params {
    wr_batch_desc b;                 // b.seq_len[s] = position of the new token of session s
    float *q;                        // [n_sess][n_q][128]: raw projections in, (normed, rotated) rows out
    const float *k, *v;              // [n_sess][n_kv][128] raw projections
    float *out;                      // [n_sess][n_q][128]
    const float *q_norm, *k_norm;    // [128] each, or both null
    uint32_t n_kv, n_q, n_rot;
    float eps, theta, scale;
};

__device__ __forceinline__ const char *row_chunk(const char *block, uint32_t tok, uint32_t c)
{
    // 16-byte chunk c (dims 8c .. 8c+7) of token `tok` inside a tiled (head, K|V) block
    return block + (c >> 3) * (kPageTokens * 128u) + tok * 128u + (((c & 7u) ^ (tok & 7u)) << 4);
}

// GM: upper bound of q heads per kv head this instantiation is unrolled for (the kernel runs its code
// once, on a handful of warps, so code size is time: a cold instruction line costs as much as a load).
template <int GM, int SETS>
__global__ void __launch_bounds__(kSetThreads * SETS) attn_step_small_kernel(const step_small_params p)
{
    constexpr uint32_t kSmallThreads = kSetThreads * SETS, kSmallWarps = kSmallThreads / 32;
    constexpr uint32_t kRaw = SETS == 4 ? 8 : 16;                // 16-byte pieces of a key row in flight per thread

    __shared__ __align__(16) float sq[GM][kHd];                  // this kv head's q rows
    __shared__ __align__(16) float sk[kHd], sv[kHd];
    __shared__ __align__(16) __half nk[kHd], nv[kHd];            // the new row as the cache holds it
    __shared__ float cs_tab[kHd / 2], sn_tab[kHd / 2];
    __shared__ float sc[GM][kSmallMaxKeys];                      // scores, then probabilities
    __shared__ float s_inv_l[GM];
    __shared__ float s_qnw[kHd], s_knw[kHd];                     // QK-norm weights
    __shared__ const char *s_page[kSmallMaxKeys / kPageTokens];  // this session's pages of this layer

    const uint32_t s = blockIdx.x / p.n_kv, kvh = blockIdx.x % p.n_kv;
    const uint32_t G = p.n_q / p.n_kv;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t pos = p.b.seq_len[s], n_keys = pos + 1;
    constexpr uint32_t half = kHd / 2;

    // ---- what does not depend on the kernel before this one (the projections): norm weights, the
    //      session's page pointers, the pair angles of this position (kernels.c:1400-1405).  The kernel
    //      behind this one may be scheduled meanwhile, and this part overlaps the one before.
    pdl_trigger();
    const uint64_t *pages = p.b.pages[s];
    if (p.q_norm) {
        if (tid < kHd) s_qnw[tid] = p.q_norm[tid];
        else if (tid < 2 * kHd) s_knw[tid - kHd] = p.k_norm[tid - kHd];
    }
    if (tid < (n_keys + kPageTokens - 1) / kPageTokens) s_page[tid] = (const char *)pages[tid];
    if (tid < p.n_rot) {
        float sn, cs;
        wrmath::rope_angle(pos, tid, kHd, wrmath::log_ref(p.theta), sn, cs);
        cs_tab[tid] = cs;
        sn_tab[tid] = sn;
    }
    // Short sessions: the K and V lines on their way into L2 (between two steps the weights have pushed them out): a hint, whatever
    // is still being written.  (28 layers, 64 to 192 keys: 1030 -> 1023 us a step.  With more keys they cost more than they bring: 16
    // sessions of 200 to 2000 keys 2973 -> 3001.  On the stream beside long sessions' kernels they make no difference: without / with
    // them, 15 sessions of 60 to 228 keys and one of 2000 2380 / 2384, 8 and 8 of 1200 to 1900 2471 / 2461, one and one 1455 / 1459.)
    if constexpr (SETS == 1) {
        __syncthreads();
        for (uint32_t i = tid; i < pos * 4; i += kSmallThreads) {
            const uint32_t key = i >> 2, which = (i >> 1) & 1u, line = i & 1u;
            const char *at = s_page[key / kPageTokens] + wr_block_off(kvh, which, kHd) + line * (kPageTokens * 128u) +
                             key % kPageTokens * 128u;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
        }
    }
    pdl_wait();
    // ---- rows in
    const size_t q_at = ((size_t)s * p.n_q + (size_t)kvh * G) * kHd;
    for (uint32_t i = tid; i < G * kHd; i += kSmallThreads) sq[i / kHd][i % kHd] = p.q[q_at + i];
    if (tid < kHd) sk[tid] = p.k[((size_t)s * p.n_kv + kvh) * kHd + tid];
    else if (tid < 2 * kHd) sv[tid - kHd] = p.v[((size_t)s * p.n_kv + kvh) * kHd + tid - kHd];
    __syncthreads();

    // ---- per-head RMSNorm of K and of the G q heads (one warp per vector), as head_rmsnorm_kernel
    if (p.q_norm) {
        for (uint32_t vct = warp; vct < G + 1; vct += kSmallWarps) {
            float *x = (vct == 0) ? sk : sq[vct - 1];
            const float *w = (vct == 0) ? s_knw : s_qnw;
            float ss = 0.f;
            for (uint32_t i = lane; i < kHd; i += 32) ss += x[i] * x[i];
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
            const float inv = 1.0f / sqrtf(ss / (float)kHd + p.eps);
            for (uint32_t i = lane; i < kHd; i += 32) x[i] = x[i] * inv * w[i];
        }
        __syncthreads();
    }

    // ---- RoPE (pairs j, j + 64; products rounded separately, kernels.c:1406-1407)
    for (uint32_t i = tid; i < (G + 1) * half; i += kSmallThreads) {
        const uint32_t vct = i / half, j = i % half;
        if (j < p.n_rot) {
            float *x = (vct == 0) ? sk : sq[vct - 1];
            const float cs = cs_tab[j], sn = sn_tab[j];
            const float x0 = x[j], x1 = x[j + half];
            x[j] = wrmath::sub(wrmath::mul(x0, cs), wrmath::mul(x1, sn));
            x[j + half] = wrmath::add(wrmath::mul(x0, sn), wrmath::mul(x1, cs));
        }
    }
    __syncthreads();

    // ---- append: the new K / V row into its page (truncating convert), and kept for this CTA's own use;
    //      the rotated q rows go back to the caller's buffer
    if (tid < kHd) {
        char *page = const_cast<char *>(s_page[pos / kPageTokens]);
        const uint32_t tk = pos % kPageTokens, off = wr_elem_off(tk, tid, kHd);
        const uint16_t kb = wr_f32_to_f16_trunc(sk[tid]), vb = wr_f32_to_f16_trunc(sv[tid]);
        *(uint16_t *)(page + wr_block_off(kvh, 0, kHd) + off) = kb;
        *(uint16_t *)(page + wr_block_off(kvh, 1, kHd) + off) = vb;
        nk[tid] = __ushort_as_half(kb);
        nv[tid] = __ushort_as_half(vb);
    }
    for (uint32_t i = tid; i < G * kHd; i += kSmallThreads) p.q[q_at + i] = sq[i / kHd][i % kHd];
    __syncthreads();

    // ---- scores: one thread per key, all G heads at once.  The sixteen 16-byte loads of a key row are
    //      issued together (the kernel is latency bound: what matters is the number of round trips).
    for (uint32_t key = tid; key < n_keys; key += kSmallThreads) {
        float dot[(uint32_t)GM];
#pragma unroll
        for (uint32_t g = 0; g < (uint32_t)GM; ++g) dot[g] = 0.f;
        const char *kb = s_page[key / kPageTokens] + wr_block_off(kvh, 0, kHd);
        const uint32_t tok = key % kPageTokens;
#pragma unroll
        for (uint32_t c0 = 0; c0 < kHd / 8; c0 += kRaw) {
            uint4 raw[kRaw];
#pragma unroll
            for (uint32_t i = 0; i < kRaw; ++i) {
                if (key == pos) raw[i] = *reinterpret_cast<const uint4 *>(&nk[8 * (c0 + i)]);
                else raw[i] = __ldg(reinterpret_cast<const uint4 *>(row_chunk(kb, tok, c0 + i)));
            }
#pragma unroll
            for (uint32_t c = c0; c < c0 + kRaw; ++c) {
                const __half2 *h2 = reinterpret_cast<const __half2 *>(&raw[c - c0]);
                float kf[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 f = __half22float2(h2[i]);
                    kf[2 * i] = f.x;
                    kf[2 * i + 1] = f.y;
                }
#pragma unroll
                for (uint32_t g = 0; g < (uint32_t)GM; ++g) {
                    if (g < G) {
                        const float4 qa = *reinterpret_cast<const float4 *>(&sq[g][8 * c]);
                        const float4 qb = *reinterpret_cast<const float4 *>(&sq[g][8 * c + 4]);
                        float d = dot[g];
                        d = fmaf(qa.x, kf[0], d); d = fmaf(qa.y, kf[1], d); d = fmaf(qa.z, kf[2], d); d = fmaf(qa.w, kf[3], d);
                        d = fmaf(qb.x, kf[4], d); d = fmaf(qb.y, kf[5], d); d = fmaf(qb.z, kf[6], d); d = fmaf(qb.w, kf[7], d);
                        dot[g] = d;
                    }
                }
            }
        }
#pragma unroll
        for (uint32_t g = 0; g < (uint32_t)GM; ++g)
            if (g < G) sc[g][key] = dot[g] * p.scale;
    }
    __syncthreads();

    // ---- softmax: warp g owns head g
    for (uint32_t g = warp; g < G; g += kSmallWarps) {
        float m = WR_NEG_SENTINEL;
        for (uint32_t key = lane; key < n_keys; key += 32) m = fmaxf(m, sc[g][key]);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float l = 0.f;
        for (uint32_t key = lane; key < n_keys; key += 32) {
            const float pw = __expf(sc[g][key] - m);
            sc[g][key] = pw;
            l += pw;
        }
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if (lane == 0) s_inv_l[g] = (l > 0.f) ? 1.0f / l : 0.f;
    }
    __syncthreads();

    // ---- P.V: thread = (W dimensions of the row, key group kg of 16); all G heads at once
    {
        constexpr uint32_t W = 8 / SETS;
        const uint32_t kg = lane & 15u, d0 = (warp * 2u + (lane >> 4)) * W;
        float acc[(uint32_t)GM][W];
#pragma unroll
        for (uint32_t g = 0; g < (uint32_t)GM; ++g)
#pragma unroll
            for (uint32_t i = 0; i < W; ++i) acc[g][i] = 0.f;
        constexpr uint32_t kBatch = SETS == 4 ? 16 : 8;  // V rows whose loads are in flight together
        for (uint32_t key0 = kg; key0 < n_keys; key0 += 16 * kBatch) {
            __align__(16) uint32_t raw[kBatch][W / 2];
#pragma unroll
            for (uint32_t u = 0; u < kBatch; ++u) {
                const uint32_t key = key0 + 16 * u;
#pragma unroll
                for (uint32_t i = 0; i < W / 2; ++i) raw[u][i] = 0u;
                if (key < n_keys) {
                    const char *from = reinterpret_cast<const char *>(&nv[d0]);
                    if (key != pos)
                        from = row_chunk(s_page[key / kPageTokens] + wr_block_off(kvh, 1, kHd), key % kPageTokens, d0 / 8) +
                               d0 % 8 * 2;
                    if constexpr (W == 8) *reinterpret_cast<uint4 *>(raw[u]) = *reinterpret_cast<const uint4 *>(from);
                    else if constexpr (W == 4) *reinterpret_cast<uint2 *>(raw[u]) = *reinterpret_cast<const uint2 *>(from);
                    else raw[u][0] = *reinterpret_cast<const uint32_t *>(from);
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < kBatch; ++u) {
                const uint32_t key = key0 + 16 * u;
                if (key >= n_keys) break;
                float vf[W];
#pragma unroll
                for (uint32_t i = 0; i < W / 2; ++i) {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&raw[u][i]));
                    vf[2 * i] = f.x;
                    vf[2 * i + 1] = f.y;
                }
#pragma unroll
                for (uint32_t g = 0; g < (uint32_t)GM; ++g) {
                    if (g < G) {
                        const float pw = sc[g][key];
#pragma unroll
                        for (uint32_t i = 0; i < W; ++i) acc[g][i] = fmaf(pw, vf[i], acc[g][i]);
                    }
                }
            }
        }
        // add the 16 key groups (lane bits 0-3)
#pragma unroll
        for (uint32_t g = 0; g < (uint32_t)GM; ++g) {
            if (g < G) {
#pragma unroll
                for (uint32_t i = 0; i < W; ++i) {
                    float a = acc[g][i];
                    a += __shfl_xor_sync(0xffffffffu, a, 8);
                    a += __shfl_xor_sync(0xffffffffu, a, 4);
                    a += __shfl_xor_sync(0xffffffffu, a, 2);
                    a += __shfl_xor_sync(0xffffffffu, a, 1);
                    acc[g][i] = a;
                }
                if (kg == 0) {
                    const float inv = s_inv_l[g];
                    float *o = p.out + q_at + (size_t)g * kHd + d0;
#pragma unroll
                    for (uint32_t i = 0; i < W; i += 2)
                        *reinterpret_cast<float2 *>(o + i) = make_float2(acc[g][i] * inv, acc[g][i + 1] * inv);
                }
            }
        }
    }
}

template <int GM, int SETS>
cudaError_t launch_sets(uint32_t grid, cudaStream_t st, bool side, const step_small_params &p)
{
    if (!side) return wr_launch_pdl(attn_step_small_kernel<GM, SETS>, dim3(grid), dim3(kSetThreads * SETS), 0, st, p);
    attn_step_small_kernel<GM, SETS><<<grid, kSetThreads * SETS, 0, st>>>(p);
    return cudaGetLastError();
}
template <int GM>
cudaError_t launch_small(uint32_t sets, uint32_t grid, cudaStream_t st, bool side, const step_small_params &p)
{
    if (sets == 1) return launch_sets<GM, 1>(grid, st, side, p);
    if (sets == 2) return launch_sets<GM, 2>(grid, st, side, p);
    if constexpr (max_sets(GM) == 4) return launch_sets<GM, 4>(grid, st, side, p);
    return cudaErrorInvalidValue;
}

}  // namespace

bool wr_step_small_covers(const wr_cuda_kv *kv, uint32_t layer, uint32_t n_q_heads, uint32_t position)
{
    const uint32_t n_kv = kv->hd_at(layer) == kHd ? kv->n_kv_at(layer) : 0u;
    return n_kv > 0 && n_q_heads % n_kv == 0 && n_q_heads / n_kv <= kSmallMaxGroup && position + 1 <= kSmallMaxKeys;
}

// Enqueue on device-resident rows.  Caller holds ctx->lock; every session must pass wr_step_small_covers and
// wr_kv_batch_check, and positions[s] < max_ctx.
int wr_step_small_launch(wr_cuda_ctx *ctx, uint32_t n_sess, wr_cuda_kv *const *kv, uint32_t layer,
                         const uint32_t *positions, const wr_step_small_args &a)
{
    if (n_sess == 0 || n_sess > WR_CUDA_BATCH_MAX) return WR_CUDA_ERR_LIMIT;
    step_small_params p;
    for (uint32_t s = 0; s < n_sess; ++s) {
        if (!wr_step_small_covers(kv[s], layer, a.n_q_heads, positions[s])) return WR_CUDA_ERR_UNSUPPORTED;
        if (positions[s] >= kv[s]->max_ctx) return WR_CUDA_ERR_CTX_FULL;
        p.b.pages[s] = kv[s]->d_pages + (size_t)layer * kv[s]->n_pages;
        p.b.seq_len[s] = positions[s];
    }
    constexpr uint32_t half = kHd / 2u;
    p.q = a.q;
    p.k = a.k;
    p.v = a.v;
    p.out = a.out;
    p.q_norm = a.q_norm;
    p.k_norm = a.k_norm;
    p.n_kv = kv[0]->n_kv_at(layer);
    p.n_q = a.n_q_heads;
    p.n_rot = (a.n_rot_pairs >= 1 && a.n_rot_pairs < half) ? a.n_rot_pairs : half;     // kernels.c:1381-1383
    p.eps = a.eps;
    p.theta = (a.theta_base < 1.0f) ? 10000.0f : a.theta_base;                       // kernels.c:1374
    p.scale = (a.scale_override > 0.0f) ? a.scale_override : 1.0f / sqrtf((float)kHd);
    const uint32_t group = a.n_q_heads / p.n_kv, grid = n_sess * p.n_kv;
    uint32_t sets = 1;                                           // the most that a session of this launch has
    for (uint32_t i = 0; i < n_sess; ++i) sets = std::max(sets, sets_for(positions[i] + 1, group));
    const cudaStream_t st = a.side ? a.side : ctx->stream;
    if (group == 1) WR_CUDA_TRY(launch_small<1>(sets, grid, st, a.side != nullptr, p));
    else if (group == 2) WR_CUDA_TRY(launch_small<2>(sets, grid, st, a.side != nullptr, p));
    else if (group <= 4) WR_CUDA_TRY(launch_small<4>(sets, grid, st, a.side != nullptr, p));
    else WR_CUDA_TRY(launch_small<8>(sets, grid, st, a.side != nullptr, p));
    ctx->launches++;
    WR_CUDA_TRY(cudaGetLastError());
    return WR_CUDA_OK;
}
