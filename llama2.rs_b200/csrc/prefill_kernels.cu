// Kernels of the batched forward pass transformer<B>, B >= 2 (src/models.rs:178-298), around the
// tcgen05 GEMM of gemm_tc.cu: embedding rows, row quantiser (adds the slices of the GEMM in front of it, residual add or SwiGLU,
// rmsnorm folded in), RoPE + cache append, causal attention over the cache.
#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cmath>

#include "kernels.cuh"

namespace l2 {

namespace {

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t peer_smem(const void* p, uint32_t rank) {  // the same shared-memory location of another CTA of the cluster
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace

// ---- x[m] = token_embedding_table[tokens[m]] (src/models.rs:189-191) ---------------------------
__global__ void embed_batch_kernel(const float* __restrict__ table, const int* __restrict__ tokens, float* __restrict__ x, int dim) {
    const int m = blockIdx.x;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const float4* src = reinterpret_cast<const float4*>(table + (size_t)tokens[m] * dim);
    float4* dst = reinterpret_cast<float4*>(x + (size_t)m * dim);
    for (int i = threadIdx.x; i < dim / 4; i += blockDim.x) dst[i] = src[i];
}

// ---- row quantiser ---------------------------------------------------------------------------------
// One token's row per cluster of CTAs.  The row is made first: a plain buffer, or the residual stream plus the output of the
// GEMM in front (its slices added in order, x updated in place), or silu(h1) * h3 of two GEMM outputs.  Every CTA makes its
// share, multiplies by the rmsnorm weight (linearity: the 1/sqrt(mean(x^2)+eps) factor goes into osc) and puts it into the shared
// memory of all CTAs of the cluster, with its part of the statistics; then every CTA cuts its share of each consumer's K order into
// digits, gathering from shared memory.  So the row is read once and the statistics (the same for every K order) are taken
// once, for up to three consumers.  A row that is in K order already (SwiGLU for w2, the longest of a layer) needs no gathering: a CTA's
// share is what it cuts, it keeps that alone and nothing but the statistics crosses.
//
// Digits: X = round(x * nw * 2^(22 - E)) with E the exponent of the row's largest |x * nw|, so |X| <= 2^23 (the 24 bits of an f32
// mantissa for the largest element), X = 4096 hi + lo with hi and lo in -2048..2048 (halves round to even), both exact in f16.  A NaN or an
// infinity becomes a digit that is not finite, which makes every output of its token NaN.  The digits go into the
// K-major, 128-byte-swizzled blocks the GEMM copies into shared memory: per K step two halves of 64 inputs, row digit * tq + token,
// inside a block of 8 inputs the order (0,4,1,5,2,6,3,7) in which a weight word separates into f16 pairs.
constexpr int RQ_THREADS = 256;
constexpr int RQ_MAX_CLUSTER = 8;

__global__ void __launch_bounds__(RQ_THREADS, 4) row_quant_kernel(const __grid_constant__ RowParams P) {
    extern __shared__ __align__(16) float xs[];  // the row (times the norm weight), natural order; or this CTA's share of it
    __shared__ float red[2][RQ_THREADS / 32];
    __shared__ float stat[RQ_MAX_CLUSTER][2];    // (largest |x nw|, sum of x^2) of every CTA's share
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int C = (int)gridDim.x, r = (int)cluster_rank(), m = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int tb = m / P.tq, t = m - tb * P.tq;
    // this CTA's share of the digits: blocks of 8 inputs, whole K steps; an item is a block of one consumer
    const int b0 = (int)((long long)P.KS * r / C) * 16, nb = min(P.in / 8, (int)((long long)P.KS * (r + 1) / C) * 16) - b0, items = P.nmat * nb;
    // and of the row: the same inputs if the row is in K order (a launch's rows are all permuted or none is)
    const bool own = !P.perm[0];
    const int n4 = P.in / 4, i0 = own ? 2 * b0 : (int)((long long)n4 * r / C), i1 = own ? 2 * (b0 + nb) : (int)((long long)n4 * (r + 1) / C);
    float4* xs4 = reinterpret_cast<float4*>(xs) - (own ? i0 : 0);  // element i of the row
    auto perm_of = [&](int item) {
        const int j = item / nb;
        const uint16_t* p = j == 0 ? P.perm[0] : j == 1 ? P.perm[1] : P.perm[2];
        return item < items && p ? __ldg(reinterpret_cast<const uint4*>(p) + b0 + (item - j * nb)) : make_uint4(0, 0, 0, 0);
    };
    // what does not depend on the kernel in front is requested before waiting for it
    const uint4 perm0 = perm_of(tid);
    float4 w0 = make_float4(1.f, 1.f, 1.f, 1.f);
    if (P.nw && i0 + tid < i1) w0 = __ldg(reinterpret_cast<const float4*>(P.nw) + i0 + tid);
    if (C > 1) cluster_barrier();  // every CTA of the cluster has started: its shared memory may be written
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float mx = 0.f, sq = 0.f;
    for (int i = i0 + tid; i < i1; i += RQ_THREADS) {
        float4 v;
        if (P.mode == ROW_SWIGLU) {  // src/models.rs:92-98
            const float4 a = tc_load4(P.a, m, tb, i * 4), b = tc_load4(P.b, m, tb, i * 4);
            v.x = (a.x * (1.0f / (1.0f + expf(-a.x)))) * b.x; v.y = (a.y * (1.0f / (1.0f + expf(-a.y)))) * b.y;
            v.z = (a.z * (1.0f / (1.0f + expf(-a.z)))) * b.z; v.w = (a.w * (1.0f / (1.0f + expf(-a.w)))) * b.w;
        } else {
            float4* xp = reinterpret_cast<float4*>(P.x + (size_t)m * P.ldx) + i;
            v = *xp;
            if (P.mode == ROW_RESID) {  // src/models.rs:47-51
                const float4 a = tc_load4(P.a, m, tb, i * 4);
                v.x += a.x; v.y += a.y; v.z += a.z; v.w += a.w;
                *xp = v;
            }
        }
        sq += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        if (P.nw) {
            const float4 w = i == i0 + tid ? w0 : __ldg(reinterpret_cast<const float4*>(P.nw) + i);
            v.x *= w.x; v.y *= w.y; v.z *= w.z; v.w *= w.w;
        }
        mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        xs4[i] = v;
        for (int c = 0; c < C && !own; c++)
            if (c != r)
                asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(peer_smem(xs + 4 * i, c)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        sq += __shfl_xor_sync(0xffffffffu, sq, o);
    }
    if (lane == 0) { red[0][warp] = mx; red[1][warp] = sq; }
    __syncthreads();
    if (tid < C) {  // thread c delivers this CTA's statistics to CTA c
        float a = 0.f, b = 0.f;
        for (int w = 0; w < RQ_THREADS / 32; w++) { a = fmaxf(a, red[0][w]); b += red[1][w]; }
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1,%2};" ::"r"(peer_smem(&stat[r][0], tid)), "f"(a), "f"(b) : "memory");
    }
    if (C > 1) cluster_barrier(); else __syncthreads();
    float total = 0.f;
    mx = 0.f;
    for (int c = 0; c < C; c++) { mx = fmaxf(mx, stat[c][0]); total += stat[c][1]; }
    const float rs = P.nw ? 1.0f / sqrtf(total / (float)P.in + P.eps) : 1.0f;  // src/models.rs:58-60
    int e = 0;
    if (mx > 0.f && mx < INFINITY) e = 22 - (int)((__float_as_uint(mx) >> 23) & 255u) + 127;  // |x| * scale < 2^23
    e = min(100, e);  // (at least 22 - 127: every finite row is scaled down far enough)
    const float scale = __uint_as_float((uint32_t)(127 + e) << 23);
    if (tid == 0 && r == 0) P.osc[m] = rs / scale;

    const size_t blk_bytes = (size_t)512 * P.tq;
    {
#pragma unroll 1
        for (int item = tid; item < items; item += RQ_THREADS) {
            const int j = item / nb, blk = b0 + (item - j * nb);
            uint8_t* img = (j == 0 ? P.img[0] : j == 1 ? P.img[1] : P.img[2]) + (size_t)tb * P.KS * blk_bytes;
            float v[8];
            if (!own) {
                const uint4 ix = item == tid ? perm0 : perm_of(item);
                v[0] = xs[ix.x & 0xFFFFu]; v[1] = xs[ix.x >> 16]; v[2] = xs[ix.y & 0xFFFFu]; v[3] = xs[ix.y >> 16];
                v[4] = xs[ix.z & 0xFFFFu]; v[5] = xs[ix.z >> 16]; v[6] = xs[ix.w & 0xFFFFu]; v[7] = xs[ix.w >> 16];
            } else {
                const float4 a = xs4[2 * blk], b = xs4[2 * blk + 1];
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
            }
            uint32_t hi[4], lo[4];
            constexpr int order[8] = {0, 4, 1, 5, 2, 6, 3, 7};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float x0 = rintf(v[order[2 * i]] * scale), x1 = rintf(v[order[2 * i + 1]] * scale);
                const float h0 = rintf(x0 * (1.0f / 4096.0f)), h1 = rintf(x1 * (1.0f / 4096.0f));
                const __half2 h = __floats2half2_rn(h0, h1), l = __floats2half2_rn(fmaf(h0, -4096.0f, x0), fmaf(h1, -4096.0f, x1));  // exact
                hi[i] = *reinterpret_cast<const uint32_t*>(&h);
                lo[i] = *reinterpret_cast<const uint32_t*>(&l);
            }
            // block `blk` of the K step: half (blk & 15) / 8, 16-byte chunk blk & 7 of the rows of both digits
            uint8_t* dst = img + (size_t)(blk >> 4) * blk_bytes + (size_t)((blk >> 3) & 1) * P.tq * 256;
            const uint32_t r0 = (uint32_t)t, r1 = (uint32_t)(P.tq + t), c = (uint32_t)blk & 7u;
            *reinterpret_cast<uint4*>(dst + r0 * 128 + ((c ^ (r0 & 7u)) << 4)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(dst + r1 * 128 + ((c ^ (r1 & 7u)) << 4)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    }
}

// ---- RoPE + cache append for M tokens (src/models.rs:100-129, 236-249) ----------------------------
// grid (M, slices of the row); a thread rotates four neighbouring pairs (i, i + 64) of one head.  Rotate-half as the reference does
// it in place: the second half uses the already rotated first half.
__device__ __forceinline__ void rotate4(const float4& a, const float4& b, const float4& c, const float4& s, float4& na, float4& nb) {
    na.x = __fsub_rn(__fmul_rn(a.x, c.x), __fmul_rn(b.x, s.x)); nb.x = __fadd_rn(__fmul_rn(b.x, c.x), __fmul_rn(na.x, s.x));
    na.y = __fsub_rn(__fmul_rn(a.y, c.y), __fmul_rn(b.y, s.y)); nb.y = __fadd_rn(__fmul_rn(b.y, c.y), __fmul_rn(na.y, s.y));
    na.z = __fsub_rn(__fmul_rn(a.z, c.z), __fmul_rn(b.z, s.z)); nb.z = __fadd_rn(__fmul_rn(b.z, c.z), __fmul_rn(na.z, s.z));
    na.w = __fsub_rn(__fmul_rn(a.w, c.w), __fmul_rn(b.w, s.w)); nb.w = __fadd_rn(__fmul_rn(b.w, c.w), __fmul_rn(na.w, s.w));
}
__global__ void __launch_bounds__(256) rope_append_kernel(const __grid_constant__ RopeParams P) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int m = blockIdx.x, pos = P.pos[m], tb = m / P.q.tq;
    const int KV = P.kv_stride ? P.kv_stride : P.n_kv_heads * HS;
    const int nq = P.n_heads * (HS / 8), nk = P.n_kv_heads * (HS / 8);  // units of four pairs
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < nq + 2 * nk; i += gridDim.y * blockDim.x) {
        const int u = i < nq ? i : i < nq + nk ? i - nq : i - nq - nk, h = u / (HS / 8), e = (u % (HS / 8)) * 4, o = h * HS + e;
        if (i < nq + nk) {
            const float4 c = *reinterpret_cast<const float4*>(P.rope_cos + (size_t)pos * (HS / 2) + e), s = *reinterpret_cast<const float4*>(P.rope_sin + (size_t)pos * (HS / 2) + e);
            const TcOut& T = i < nq ? P.q : P.k;
            const float4 a = tc_load4(T, m, tb, o), b = tc_load4(T, m, tb, o + HS / 2);
            float4 na, nb;
            rotate4(a, b, c, s, na, nb);
            float* dst = i < nq ? P.qout + (size_t)m * P.ldq + o : P.kc + (size_t)pos * KV + o;
            *reinterpret_cast<float4*>(dst) = na;
            *reinterpret_cast<float4*>(dst + HS / 2) = nb;
        } else {
            const float4 a = tc_load4(P.v, m, tb, o), b = tc_load4(P.v, m, tb, o + HS / 2);
            float* dst = P.vc + (size_t)pos * KV + o;
            *reinterpret_cast<float4*>(dst) = a;
            *reinterpret_cast<float4*>(dst + HS / 2) = b;
        }
    }
}

// ---- attention of M tokens over the cache, causal through 0..=pos[m] (src/models.rs:131-176) ------
// grid (n_heads, M), 128 threads: each warp walks the time steps t = warp, warp + 4, ... with an
// online softmax; the four warps are merged in shared memory.
__global__ void __launch_bounds__(128) attn_batch_kernel(const __grid_constant__ AttnBatchParams P) {
    __shared__ __align__(16) float sm_acc[4][HS];
    __shared__ float sm_m[4], sm_l[4];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int h = blockIdx.x, m = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = h / P.ag, KV = P.kv_stride ? P.kv_stride : P.n_kv_heads * HS;
    const int T = P.pos[m] + 1;
    const float4 q = reinterpret_cast<const float4*>(P.q + (size_t)m * P.ldq + (size_t)h * HS)[lane];
    const float4* kc = reinterpret_cast<const float4*>(P.kc) + (size_t)kvh * (HS / 4) + lane;
    const float4* vc = reinterpret_cast<const float4*>(P.vc) + (size_t)kvh * (HS / 4) + lane;
    const size_t rs = (size_t)KV / 4;
    const float div = sqrtf((float)HS);
    float mx = -INFINITY, l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int t = warp; t < T; t += 4) {
        const float4 k = kc[(size_t)t * rs], v = vc[(size_t)t * rs];
        float d = warp_sum_f(q.x * k.x + q.y * k.y + q.z * k.z + q.w * k.w);
        const float sc = __fdiv_rn(d, div);  // src/models.rs:158
        const float mn = fmaxf(mx, sc);
        const float corr = expf(mx - mn), pr = expf(sc - mn);
        l = l * corr + pr;
        acc.x = acc.x * corr + pr * v.x; acc.y = acc.y * corr + pr * v.y;
        acc.z = acc.z * corr + pr * v.z; acc.w = acc.w * corr + pr * v.w;
        mx = mn;
    }
    reinterpret_cast<float4*>(sm_acc[warp])[lane] = acc;
    if (lane == 0) { sm_m[warp] = mx; sm_l[warp] = l; }
    __syncthreads();
    float M = -INFINITY;
    for (int w = 0; w < 4; w++) M = fmaxf(M, sm_m[w]);
    float L = 0.f, A = 0.f;
    for (int w = 0; w < 4; w++) {
        const float e = sm_m[w] == -INFINITY ? 0.f : expf(sm_m[w] - M);
        L += sm_l[w] * e;
        A += sm_acc[w][tid] * e;
    }
    P.out[(size_t)m * P.ldo + (size_t)h * HS + tid] = A / L;
}

void launch_embed_batch(const float* table, const int* tokens, float* x, int dim, int M, cudaStream_t st) {
    g_launches++;
    embed_batch_kernel<<<M, 256, 0, st>>>(table, tokens, x, dim);
}
// A launch that may start while the kernel in front of it still runs (it waits inside for that one's results).
template <class K, class... A>
static cudaError_t launch_pdl(K kernel, dim3 grid, dim3 block, size_t smem, int cluster, cudaStream_t st, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[2];
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr; cfg.numAttrs = cluster > 0 ? 2 : 1;
    g_launches++;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

cudaError_t row_quant_init(int max_smem) { return cudaFuncSetAttribute(row_quant_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem); }

// As many CTAs per token as it takes to cover the SMs about twice with the batch (a row is 16 to 112 KB: one CTA walks it in 2 to
// 10 us, and nothing else of a small batch would hide that), never more than the K steps of the row.  Where a CTA holds its share
// alone, as many as it takes for four CTAs on an SM (a whole row of 28672 fills one; 7B shapes, 16 layers, 30 tokens: 1690 -> 1632 us, 1536
// tokens of the 70B shapes 29.6 -> 29.3 ms).
cudaError_t launch_row_quant(const RowParams& p, int sms, cudaStream_t st) {
    const bool own = !p.perm[0];
    auto share = [&](int C) { return own ? (size_t)((p.KS + C - 1) / C) * 512 : (size_t)p.in * 4; };
    int C = 1;
    while (C < RQ_MAX_CLUSTER && 2 * C <= p.KS && ((long long)p.M * C < sms || (own && share(C) > 48 * 1024))) C *= 2;
    return launch_pdl(row_quant_kernel, dim3(C, p.M), dim3(RQ_THREADS), share(C), C, st, p);
}

cudaError_t launch_rope_append(const RopeParams& p, int M, int sms, cudaStream_t st) {
    const int units = (p.n_heads + 2 * p.n_kv_heads) * (HS / 8);
    return launch_pdl(rope_append_kernel, dim3(M, std::max(1, std::min((units + 255) / 256, 4 * sms / M))), dim3(256), 0, 0, st, p);
}

// ---- the same attention with the cache rows shared by the queries that need them ---------------------------------------
// One CTA takes a kv head and a block of tokens: all their queries (AG heads per token) walk the cache together, 32
// positions at a time.  A tile of K and V rows is brought into shared memory once and used by up to 64 queries, instead of
// once per (head, token) as above — at a context of 1500 that kernel moved 64 times the cache through the L2 per kv head
// and was a fifth of a long prompt's prefill.  Scores: lane = position, the query comes as broadcast loads from shared
// memory; softmax state per query (online, one rescale per tile); values: lane = four of the 128 dimensions, the
// probabilities come by shuffle.  Plain f32 FMAs: the arithmetic is the reference's, only the order of the sums differs.
constexpr int AT_WARPS = 8, AT_TILE = 32, AT_KPAD = HS + 4;  // K rows padded: a lane reads "its" row without bank conflicts
template <int AG, int NQW>  // query heads per kv head; queries per warp (NQW / AG tokens)
__global__ void __launch_bounds__(32 * AT_WARPS) attn_batch_tiled_kernel(const __grid_constant__ AttnBatchParams P, int M) {
    extern __shared__ __align__(16) float at_smem[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int TPW = NQW / AG;                       // tokens per warp
    constexpr int QB = AT_WARPS * TPW;                  // tokens per CTA
    float* Qs = at_smem;                                // [AT_WARPS * NQW][HS]
    float* Ks = Qs + AT_WARPS * NQW * HS;               // [AT_TILE][AT_KPAD]
    float* Vs = Ks + AT_TILE * AT_KPAD;                 // [AT_TILE][HS]
    const int kvh = blockIdx.x, m0 = blockIdx.y * QB, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int KV = P.kv_stride ? P.kv_stride : P.n_kv_heads * HS;
    const float div = sqrtf((float)HS);
    // queries of this CTA: query i = (token m0 + i / AG, head kvh * AG + i % AG)
    for (int i = tid; i < AT_WARPS * NQW * (HS / 4); i += 32 * AT_WARPS) {
        const int qi = i / (HS / 4), c = i % (HS / 4), m = m0 + qi / AG;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < M) v = reinterpret_cast<const float4*>(P.q + (size_t)m * P.ldq + (size_t)(kvh * AG + qi % AG) * HS)[c];
        reinterpret_cast<float4*>(Qs)[i] = v;
    }
    int last[TPW];   // last position each of this warp's tokens attends to (-1: no such token)
    int tmax = -1;   // over the CTA
#pragma unroll
    for (int j = 0; j < TPW; j++) {
        const int m = m0 + warp * TPW + j;
        last[j] = m < M ? P.pos[m] : -1;
    }
    for (int m = m0; m < min(M, m0 + QB); m++) tmax = max(tmax, P.pos[m]);
    float mx[NQW], l[NQW];
    float4 acc[NQW];
#pragma unroll
    for (int q = 0; q < NQW; q++) { mx[q] = -INFINITY; l[q] = 0.f; acc[q] = make_float4(0.f, 0.f, 0.f, 0.f); }
    const float4* kc = reinterpret_cast<const float4*>(P.kc) + (size_t)kvh * (HS / 4);
    const float4* vc = reinterpret_cast<const float4*>(P.vc) + (size_t)kvh * (HS / 4);
    const size_t rs = (size_t)KV / 4;
    for (int t0 = 0; t0 <= tmax; t0 += AT_TILE) {
        __syncthreads();  // the previous tile has been used (and Qs is complete)
        for (int i = tid; i < AT_TILE * (HS / 4); i += 32 * AT_WARPS) {
            const int r = i / (HS / 4), c = i % (HS / 4), t = t0 + r;
            float4 k = make_float4(0.f, 0.f, 0.f, 0.f), v = k;
            if (t <= tmax) { k = kc[(size_t)t * rs + c]; v = vc[(size_t)t * rs + c]; }
            reinterpret_cast<float4*>(Ks + r * AT_KPAD)[c] = k;
            reinterpret_cast<float4*>(Vs + r * HS)[c] = v;
        }
        __syncthreads();
        // scores of position t0 + lane for this warp's queries
        float s[NQW];
#pragma unroll
        for (int q = 0; q < NQW; q++) s[q] = 0.f;
        const float4* krow = reinterpret_cast<const float4*>(Ks + lane * AT_KPAD);
        const float4* qrow = reinterpret_cast<const float4*>(Qs + (size_t)warp * NQW * HS);
#pragma unroll 4
        for (int c = 0; c < HS / 4; c++) {
            const float4 k = krow[c];
#pragma unroll
            for (int q = 0; q < NQW; q++) {
                const float4 qq = qrow[q * (HS / 4) + c];
                s[q] = fmaf(qq.x, k.x, s[q]); s[q] = fmaf(qq.y, k.y, s[q]); s[q] = fmaf(qq.z, k.z, s[q]); s[q] = fmaf(qq.w, k.w, s[q]);
            }
        }
        // online softmax per query, then the values
        float p[NQW];
#pragma unroll
        for (int q = 0; q < NQW; q++) {
            const bool valid = t0 + lane <= last[q / AG];
            const float sc = valid ? __fdiv_rn(s[q], div) : -INFINITY;  // src/models.rs:158
            float tm = sc;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
            const float mn = fmaxf(mx[q], tm);
            const float corr = mn == -INFINITY ? 1.f : expf(mx[q] - mn);
            p[q] = valid ? expf(sc - mn) : 0.f;
            const float ps = warp_sum_f(p[q]);
            l[q] = l[q] * corr + ps;
            acc[q].x *= corr; acc[q].y *= corr; acc[q].z *= corr; acc[q].w *= corr;
            mx[q] = mn;
        }
        const float4* vcol = reinterpret_cast<const float4*>(Vs) + lane;
#pragma unroll 4
        for (int t = 0; t < AT_TILE; t++) {
            const float4 v = vcol[t * (HS / 4)];
#pragma unroll
            for (int q = 0; q < NQW; q++) {
                const float pq = __shfl_sync(0xffffffffu, p[q], t);
                acc[q].x = fmaf(pq, v.x, acc[q].x); acc[q].y = fmaf(pq, v.y, acc[q].y);
                acc[q].z = fmaf(pq, v.z, acc[q].z); acc[q].w = fmaf(pq, v.w, acc[q].w);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < NQW; q++) {
        const int qi = warp * NQW + q, m = m0 + qi / AG;
        if (m < M) {
            const float inv = 1.0f / l[q];
            reinterpret_cast<float4*>(P.out + (size_t)m * P.ldo + (size_t)(kvh * AG + qi % AG) * HS)[lane] =
                make_float4(acc[q].x * inv, acc[q].y * inv, acc[q].z * inv, acc[q].w * inv);
        }
    }
}

// ---- the same for many queries: 16 per warp ------------------------------------------------------------------------------
// What bounds the kernel above is the way from shared memory into registers: 128 bytes per clock, broadcasts included, so a 16-byte load of a warp
// costs 4 clocks and feeds as many FMA clocks as there are values to combine it with (9 loads per 32 FMAs for the scores, a load and 8
// shuffles per 32 for the values: 1880 clocks per 8 queries and tile).  Hence register tiles:
//   scores: lane (pi, qi) has positions pi + 8 j (j < 4) of queries qi + 4 u (u < 4): 8 loads per 64 FMAs;
//   values: lane (half, dl) has dimensions 4 dl .. + 3 and 64 + 4 dl .. + 3 of 8 queries: 4 loads per 64 FMAs (the probabilities come
//   from shared memory, where the lanes that computed them put them).
// Rows of K are padded: the lanes of a load read different banks.  The shared memory is small enough for three CTAs per SM, so that the
// copies of one tile overlap the arithmetic of others.
constexpr int AW_WARPS = 4, AW_QW = 16, AW_PP = AW_QW + 4;
constexpr int AW_FLOATS = AW_WARPS * AW_QW * HS + AT_TILE * (AT_KPAD + HS) + AW_WARPS * AT_TILE * AW_PP;
static_assert(3 * (AW_FLOATS * 4 + 1024) <= 228 * 1024, "three CTAs per SM");

__device__ __forceinline__ float2 at_fma2(const float2& a, const float2& b, const float2& c) {
    float2 d;
    asm("{\n.reg .b64 a, b, c, d;\nmov.b64 a, {%2, %3};\nmov.b64 b, {%4, %5};\nmov.b64 c, {%6, %7};\nfma.rn.f32x2 d, a, b, c;\nmov.b64 {%0, %1}, d;\n}"
        : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return d;
}
__device__ __forceinline__ void at_copy16(float* dst, const float4* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int AG>  // query heads per kv head
__global__ void __launch_bounds__(32 * AW_WARPS, 3) attn_batch_wide_kernel(const __grid_constant__ AttnBatchParams P, int M) {
    extern __shared__ __align__(16) float at_smem[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    constexpr int TPW = AW_QW / AG, QB = AW_WARPS * TPW;        // tokens per warp, per CTA
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* Qs = at_smem;                                     // [AW_WARPS * 16][HS]
    float* Ks = Qs + AW_WARPS * AW_QW * HS;                     // [AT_TILE][AT_KPAD]
    float* Vs = Ks + AT_TILE * AT_KPAD;                     // [AT_TILE][HS]
    float* Ps = Vs + AT_TILE * HS + warp * AT_TILE * AW_PP;  // [AT_TILE][AW_PP] this warp's probabilities by place; behind them in rows 0-3
    float* Cs = Ps + AW_QW;                                  // a factor, in rows 4-7 the last position of the query in place 4 row + column
    int* Ls = reinterpret_cast<int*>(Cs + 4 * AW_PP);
    const int kvh = blockIdx.x, m0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * QB;  // (the blocks with the longest way start first)
    const int KV = P.kv_stride ? P.kv_stride : P.n_kv_heads * HS;
    const float div = sqrtf((float)HS);
    // queries of this CTA: query i = (token m0 + i / AG, head kvh * AG + i % AG)
    for (int i = tid; i < AW_WARPS * AW_QW * (HS / 4); i += 32 * AW_WARPS) {
        const int qi = i / (HS / 4), c = i % (HS / 4), m = m0 + qi / AG;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (m < M) v = reinterpret_cast<const float4*>(P.q + (size_t)m * P.ldq + (size_t)(kvh * AG + qi % AG) * HS)[c];
        *reinterpret_cast<float4*>(Qs + qi * HS + 4 * c) = v;
    }
    const int pi = lane & 7, qi = lane >> 3;
    // last position that query qi + 4 u attends to (-1: no such token); the last and the first of the warp's; the last of the CTA's
    int last[4], wlast = -1, wfirst = INT_MAX, tmax = -1;
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int m = m0 + warp * TPW + (qi + 4 * u) / AG;
        last[u] = m < M ? P.pos[m] : -1;
    }
    if (pi == 0) *reinterpret_cast<int4*>(Ls + qi * AW_PP) = make_int4(last[0], last[1], last[2], last[3]);  // query qi + 4 u has place 4 qi + u
    for (int m = m0 + warp * TPW; m < min(M, m0 + (warp + 1) * TPW); m++) { wlast = max(wlast, P.pos[m]); wfirst = min(wfirst, P.pos[m]); }
    for (int m = m0; m < min(M, m0 + QB); m++) tmax = max(tmax, P.pos[m]);
    float mx[4], l[4];
    float2 acc[8][4];  // 8 queries x 8 dimensions
#pragma unroll
    for (int u = 0; u < 4; u++) { mx[u] = -INFINITY; l[u] = 0.f; }
#pragma unroll
    for (int q = 0; q < 8; q++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[q][i] = make_float2(0.f, 0.f);
    const int half = lane >> 4, dl = lane & 15;
    const float4* kc = reinterpret_cast<const float4*>(P.kc) + (size_t)kvh * (HS / 4);
    const float4* vc = reinterpret_cast<const float4*>(P.vc) + (size_t)kvh * (HS / 4);
    const size_t rs = (size_t)KV / 4;
    const float* krow = Ks + pi * AT_KPAD;
    const float* qrow = Qs + (warp * AW_QW + qi) * HS;
    for (int t0 = 0; t0 <= tmax; t0 += AT_TILE) {
        __syncthreads();  // the previous tile has been used
        for (int i = tid; i < AT_TILE * (HS / 4); i += 32 * AW_WARPS) {
            const int r = i / (HS / 4), c = i % (HS / 4), t = min(t0 + r, tmax);  // (rows beyond the last are not used)
            at_copy16(Ks + r * AT_KPAD + 4 * c, kc + (size_t)t * rs + c);
            at_copy16(Vs + r * HS + 4 * c, vc + (size_t)t * rs + c);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (t0 > wlast) continue;
        float2 s2[4][4];  // [position][query], even and odd dimensions
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int u = 0; u < 4; u++) s2[j][u] = make_float2(0.f, 0.f);
#pragma unroll 2
        for (int c = 0; c < HS; c += 4) {
            float4 q[4];
#pragma unroll
            for (int u = 0; u < 4; u++) q[u] = *reinterpret_cast<const float4*>(qrow + 4 * u * HS + c);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 k = *reinterpret_cast<const float4*>(krow + 8 * j * AT_KPAD + c);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    s2[j][u] = at_fma2(make_float2(q[u].x, q[u].y), make_float2(k.x, k.y), s2[j][u]);
                    s2[j][u] = at_fma2(make_float2(q[u].z, q[u].w), make_float2(k.z, k.w), s2[j][u]);
                }
            }
        }
        // online softmax: one rescale per tile; a query's 32 scores are in 8 lanes
        float p[4][4], corr[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            float tm = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                p[j][u] = t0 + pi + 8 * j <= last[u] ? __fdiv_rn(s2[j][u].x + s2[j][u].y, div) : -INFINITY;  // src/models.rs:158
                tm = fmaxf(tm, p[j][u]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, o));
            const float mn = fmaxf(mx[u], tm);
            corr[u] = mn == -INFINITY ? 1.f : expf(mx[u] - mn);
            float ps = 0.f;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                p[j][u] = t0 + pi + 8 * j <= last[u] ? expf(p[j][u] - mn) : 0.f;
                ps += p[j][u];
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) ps += __shfl_xor_sync(0xffffffffu, ps, o);
            l[u] = l[u] * corr[u] + ps;
            mx[u] = mn;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) *reinterpret_cast<float4*>(Ps + (pi + 8 * j) * AW_PP + 4 * qi) = make_float4(p[j][0], p[j][1], p[j][2], p[j][3]);
        if (pi == 0) *reinterpret_cast<float4*>(Cs + qi * AW_PP) = make_float4(corr[0], corr[1], corr[2], corr[3]);
        __syncwarp();
        {
            const float4 c0 = *reinterpret_cast<const float4*>(Cs + 2 * half * AW_PP), c1 = *reinterpret_cast<const float4*>(Cs + (2 * half + 1) * AW_PP);
            const float f[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
            for (int q = 0; q < 8; q++)
#pragma unroll
                for (int i = 0; i < 4; i++) { acc[q][i].x *= f[q]; acc[q][i].y *= f[q]; }
        }
        auto values = [&](int t, auto&& attends) {
            const float4 v0 = *reinterpret_cast<const float4*>(Vs + t * HS + 4 * dl), v1 = *reinterpret_cast<const float4*>(Vs + t * HS + HS / 2 + 4 * dl);
            const float4 p0 = *reinterpret_cast<const float4*>(Ps + t * AW_PP + 8 * half), p1 = *reinterpret_cast<const float4*>(Ps + t * AW_PP + 8 * half + 4);
            const float f[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (attends(q)) {
                    const float2 pp = make_float2(f[q], f[q]);
                    acc[q][0] = at_fma2(pp, make_float2(v0.x, v0.y), acc[q][0]);
                    acc[q][1] = at_fma2(pp, make_float2(v0.z, v0.w), acc[q][1]);
                    acc[q][2] = at_fma2(pp, make_float2(v1.x, v1.y), acc[q][2]);
                    acc[q][3] = at_fma2(pp, make_float2(v1.z, v1.w), acc[q][3]);
                }
        };
        if (t0 + AT_TILE - 1 <= wfirst) {
#pragma unroll 2
            for (int t = 0; t < AT_TILE; t++) values(t, [](int) { return true; });
        } else {  // a row that a query does not attend to is left out, not multiplied by zero: it may hold anything
            const int4 l0 = *reinterpret_cast<const int4*>(Ls + 2 * half * AW_PP), l1 = *reinterpret_cast<const int4*>(Ls + (2 * half + 1) * AW_PP);
            const int lq[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll 1
            for (int t = 0; t < AT_TILE && t0 + t <= wlast; t++) values(t, [&](int q) { return t0 + t <= lq[q]; });
        }
        __syncwarp();  // the probabilities have been read
    }
    __syncwarp();
    if (pi == 0) *reinterpret_cast<float4*>(Cs + qi * AW_PP) = make_float4(l[0], l[1], l[2], l[3]);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; q++) {
        const int place = 8 * half + q, query = (place >> 2) + 4 * (place & 3), m = m0 + warp * TPW + query / AG;
        if (m < M) {
            const float inv = 1.0f / Cs[(place >> 2) * AW_PP + (place & 3)];
            float* o = P.out + (size_t)m * P.ldo + (size_t)(kvh * AG + query % AG) * HS + 4 * dl;
            *reinterpret_cast<float4*>(o) = make_float4(acc[q][0].x * inv, acc[q][0].y * inv, acc[q][1].x * inv, acc[q][1].y * inv);
            *reinterpret_cast<float4*>(o + HS / 2) = make_float4(acc[q][2].x * inv, acc[q][2].y * inv, acc[q][3].x * inv, acc[q][3].y * inv);
        }
    }
}

template <int AG, int NQW>
static cudaError_t launch_attn_tiled(const AttnBatchParams& p, int M, cudaStream_t st) {
    constexpr int QB = AT_WARPS * (NQW / AG);
    const size_t smem = (size_t)(AT_WARPS * NQW * HS + AT_TILE * AT_KPAD + AT_TILE * HS) * sizeof(float);
    return launch_pdl(attn_batch_tiled_kernel<AG, NQW>, dim3(p.n_kv_heads, (M + QB - 1) / QB), dim3(32 * AT_WARPS), smem, 0, st, p, M);
}
template <int AG>
static cudaError_t launch_attn_wide(const AttnBatchParams& p, int M, cudaStream_t st) {
    constexpr int QB = AW_WARPS * (AW_QW / AG);
    return launch_pdl(attn_batch_wide_kernel<AG>, dim3(p.n_kv_heads, (M + QB - 1) / QB), dim3(32 * AW_WARPS), AW_FLOATS * sizeof(float), 0, st, p, M);
}

// the tiled kernels' shared memory (77 KB at most) is above the default limit: once per device, at start-up
cudaError_t attn_batch_init() {
    const int smem = (AT_WARPS * 8 * HS + AT_TILE * AT_KPAD + AT_TILE * HS) * (int)sizeof(float);
    cudaError_t e;
#define L2_AT_ATTR(kernel, bytes) if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)) != cudaSuccess) return e;
    L2_AT_ATTR((attn_batch_tiled_kernel<1, 4>), smem) L2_AT_ATTR((attn_batch_tiled_kernel<2, 8>), smem)
    L2_AT_ATTR((attn_batch_tiled_kernel<4, 8>), smem) L2_AT_ATTR((attn_batch_tiled_kernel<8, 8>), smem)
    const int wide = AW_FLOATS * (int)sizeof(float);
    L2_AT_ATTR(attn_batch_wide_kernel<1>, wide) L2_AT_ATTR(attn_batch_wide_kernel<2>, wide)
    L2_AT_ATTR(attn_batch_wide_kernel<4>, wide) L2_AT_ATTR(attn_batch_wide_kernel<8>, wide)
#undef L2_AT_ATTR
    return cudaSuccess;
}

// Short contexts: one CTA per (head, token), which has more CTAs and less set-up (the cache is small and sits in the L2 anyway).  From
// `tiled` on (about 200 positions), the kernels that share cache tiles among queries: 16 queries per warp where that still gives the SMs
// three CTAs for every two of them (a batch of 499 tokens of the 7B shapes, 256 CTAs: 2000-token prompt on 16 layers 69.7 -> 61.5 ms; 70B
// shapes, 512 CTAs: 1536-token prompt on 4 layers 31.3 -> 29.6 ms; 296 tokens of the 7B shapes, 160 CTAs: 15.2 -> 16.2 ms).
cudaError_t launch_attn_batch(const AttnBatchParams& p, int n_heads, int M, bool tiled, int sms, cudaStream_t st) {
    const bool wide = (long long)p.n_kv_heads * ((M * p.ag + AW_WARPS * AW_QW - 1) / (AW_WARPS * AW_QW)) * 2 >= 3 * sms;
    return launch_attn_kind(p, n_heads, M, !tiled ? ATTN_HEAD : wide ? ATTN_WIDE : ATTN_TILED, st);
}
cudaError_t launch_attn_kind(const AttnBatchParams& p, int n_heads, int M, int kind, cudaStream_t st) {
    const bool wide = kind == ATTN_WIDE;
    switch (kind == ATTN_HEAD ? 0 : p.ag) {
        case 1: return wide ? launch_attn_wide<1>(p, M, st) : launch_attn_tiled<1, 4>(p, M, st);
        case 2: return wide ? launch_attn_wide<2>(p, M, st) : launch_attn_tiled<2, 8>(p, M, st);
        case 4: return wide ? launch_attn_wide<4>(p, M, st) : launch_attn_tiled<4, 8>(p, M, st);
        case 8: return wide ? launch_attn_wide<8>(p, M, st) : launch_attn_tiled<8, 8>(p, M, st);
        default: return launch_pdl(attn_batch_kernel, dim3(n_heads, M), dim3(128), 0, 0, st, p);
    }
}
// ---- all-gather of a column slice over peer memory (batched forward under tensor parallelism) ----------------------------
// Every CTA copies rows of this rank's columns into the peers' buffers with plain stores.  The CTA that finishes last
// (completion counter behind a system-wide fence) then tells every peer "my part of exchange seq is in your memory" and waits,
// bounded, until every peer has said the same: after this kernel the whole buffer is valid on this rank.
constexpr uint32_t TPG_WAIT_LIMIT = 1u << 22;
__global__ void __launch_bounds__(256) tp_gather_kernel(const __grid_constant__ TpGatherParams P) {
    __shared__ unsigned last;
    __shared__ unsigned long long seq_s;
    const int n4 = P.ncols / 4;
    for (int m = blockIdx.x; m < P.M; m += gridDim.x) {
        const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(P.pool[P.rank] + P.buf_off) + (size_t)m * P.ld + P.col0);
        for (int i = threadIdx.x; i < n4; i += blockDim.x) {
            const float4 v = src[i];
            for (int r = 0; r < P.world; r++)
                if (r != P.rank) reinterpret_cast<float4*>(reinterpret_cast<float*>(P.pool[r] + P.buf_off) + (size_t)m * P.ld + P.col0)[i] = v;
        }
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(P.done, 1u) == gridDim.x - 1 ? 1u : 0u;
    __syncthreads();
    if (!last) return;
    if (threadIdx.x == 0) { *P.done = 0; seq_s = ++*P.seq; }  // ready for the next launch; this exchange's number
    __threadfence_system();
    __syncthreads();
    const unsigned long long seq = seq_s;
    const int r = threadIdx.x;
    if (r < P.world && r != P.rank) {
        unsigned long long* theirs = reinterpret_cast<unsigned long long*>(P.pool[r] + P.flag_off) + P.rank;
        asm volatile("st.release.sys.global.u64 [%0], %1;" ::"l"(theirs), "l"(seq) : "memory");
        const unsigned long long* mine = reinterpret_cast<const unsigned long long*>(P.pool[P.rank] + P.flag_off) + r;
        bool ok = false;
#pragma unroll 1
        for (uint32_t it = 0; it < TPG_WAIT_LIMIT; it++) {
            unsigned long long v;
            asm volatile("ld.acquire.sys.global.u64 %0, [%1];" : "=l"(v) : "l"(mine) : "memory");
            if (v >= seq) { ok = true; break; }
            __nanosleep(200);
        }
        if (!ok && P.status) atomicCAS(P.status, 0, 3001);
    }
}
void launch_tp_gather(const TpGatherParams& p, cudaStream_t st) {
    g_launches++;
    tp_gather_kernel<<<std::min(p.M, 64), 256, 0, st>>>(p);
}

// ---- the output of a GEMM as a plain buffer (callers that cannot add slices themselves) ----------------------------------------
// dst (+)= the slices, or dst = silu(a) * b.  A destination that is slice 0 itself is only touched where there are more slices.
__global__ void __launch_bounds__(256) finish_kernel(TcOut a, TcOut b, int pair, float* dst, int ld, int add) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int o = (int)(blockIdx.x * blockDim.x + threadIdx.x) * 4, m = blockIdx.y, tb = m / a.tq;
    if (o >= a.rows) return;
    if (dst == a.out && tc_slices(a, tb, o) == 1) return;
    float4 v = tc_load4(a, m, tb, o);
    if (pair) {  // src/models.rs:92-98
        const float4 w = tc_load4(b, m, tb, o);
        v.x = (v.x * (1.0f / (1.0f + expf(-v.x)))) * w.x; v.y = (v.y * (1.0f / (1.0f + expf(-v.y)))) * w.y;
        v.z = (v.z * (1.0f / (1.0f + expf(-v.z)))) * w.z; v.w = (v.w * (1.0f / (1.0f + expf(-v.w)))) * w.w;
    }
    float4* d = reinterpret_cast<float4*>(dst + (size_t)m * ld + o);
    if (add) { const float4 x = *d; v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w; }
    *d = v;
}

void launch_finish(const TcOut& a, const TcOut* b, float* dst, int ld, bool add, cudaStream_t st) {
    launch_pdl(finish_kernel, dim3((a.rows / 4 + 255) / 256, a.M), dim3(256), 0, 0, st, a, b ? *b : a, b ? 1 : 0, dst, ld, add ? 1 : 0);
}

}  // namespace l2
