// Batched QLinear::matvec<B> (src/gptq.rs:94-176) for B >= 2 as a dense contraction on the
// 5th-generation tensor cores: tcgen05.mma kind::f16 on exact integer digits, weights and accumulators in tensor memory.
//
//   out[m][o] = f[m] * sum_g scale[o][g] * sum_{k in g} (q[o][k] - z[o][g]) * X[m][k]
//
// X[m][k] is the activation of token m as a 24-bit signed integer, X = 4096 hi + lo with |hi|, |lo| <= 2048 (see row_quant_kernel in
// prefill_kernels.cu).  Both digits and q - z are small integers, exact in f16, and so are their products and the sums over a
// quantisation group (at most 2^22) in the f32 accumulators: kind::f16 MMAs do exact integer arithmetic here.  f[m] carries the block
// exponent and the rmsnorm factor.
// (The alternative, three 8-bit digits on kind::i8, needs 3/4 of the MMA time but a third more accumulator columns, and their way
// from s32 columns to f32 sums (one multiply-add, two conversions, the zero-point correction) bounded the kernel at 1110 / 1770 clocks
// per 128 rows x 64 tokens x group of 64 / 128.  Here the accumulators are f32 already and the zero point is in the operand: two FMAs
// remain.)
//
// Work.  One launch covers up to three matrices that share an input length (wq/wk/wv, w1/w3).  A tile is RT x 128 output
// rows by up to 64 tokens; a K step is 128 inputs (1, 2 or 4 quantisation groups).  The (tile, K step) pairs of the launch
// form one line that is cut into equal pieces, one per SM: no tail wave, and the pipeline of a CTA fills once per launch.
// A tile that a cut goes through leaves several partial results (slices); whoever reads the output adds them in slice
// order, which costs nothing where the reader is a kernel that walks the rows anyway (row_quant_kernel, rope_append_kernel).
// RT = 2: two weight tiles share every digit block (32 KB per K step at 64 tokens, from the L2).
//
// Per K step and weight tile:
//   A  128 rows x 128 weights as f16 q - z in TENSOR MEMORY (64 columns, lane = row): written by the loaders with tcgen05.st and read by
//      the MMAs from there.  In shared memory the unpacked weights would cost 64 KB of write + read traffic per tile of a bandwidth
//      of 128 bytes per clock.
//   B  2 digits x tq tokens rows x 128 f16, one bulk copy of the block the quantiser wrote (two 128-byte-swizzled halves of 64 inputs);
//   D  per group: 128 x 2 tq f32 in one of three tensor-memory accumulators (GS / 16 MMAs of K = 16).
//      An accumulator is away from its commit until the drain has read it: with two, that chain bounded the kernel, so the A slots are
//      one per weight tile and D has three.  Clocks of a step of 256 rows x 64 tokens x 128 inputs (group 64), by stamps in the issuing
//      warp: 1406 issue (16 MMAs, 1024 of tensor time), 512 waits for an accumulator, 236 for B, 162 for A, 570 between, 2888 in all.
//      What bounds a step is the hand-overs between the roles (waits, fences, commits, arrivals), not the work between them: with the tensor-memory
//      stores of A, the loads of D and all MMAs but the first of a group left out together, and every hand-over kept, 8192 x 28672 at 256
//      tokens takes as long (243 us, back to back), and so it does with each left out alone or with a second issuing warp.
//
// Roles (they meet only through mbarriers):
//   warps 0-7    loaders, four warps per weight tile: a thread turns the 128 weights of one row into f16 (per 8 weights: a shift, four
//                and-or, four half2 operations).  Thread to row: the 8 threads of a shared-memory phase
//                read 8 different records, whose starts lie an odd number of 16-byte units apart: no bank conflicts.
//   warps 8-15   drain, four warps per weight tile: a warp reads the 32 tensor-memory lanes of its quadrant, 16 tokens at a time with
//                the next 16 in flight; packed f32 FMAs.
//                (Few warps with much work per hand-over: every wait, fence and arrival is issued by each warp of a role, and with the
//                weights or the tokens of a tile cut over twice as many warps those outnumbered the useful instructions.)
//   warp 16      raw weights: one bulk copy per 16-row record run (contiguous in memory), a ring as deep as shared memory allows.
//   warp 17      digit blocks.     warp 18  one thread issues the MMAs.
// The kernel is launched programmatically behind the quantiser: everything that does not read the quantiser's output (set-up,
// tensor-memory allocation, weight requests) runs while that kernel still does.
// Every wait on an mbarrier is bounded; a wait that gives up raises a flag that ends every loop.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "kernels.cuh"

namespace l2 {

namespace {

constexpr int TC_LOAD_WARPS = 8, TC_DRAIN_WARPS = 8;
constexpr int TC_RAW_WARP = TC_LOAD_WARPS + TC_DRAIN_WARPS, TC_B_WARP = TC_RAW_WARP + 1, TC_MMA_WARP = TC_RAW_WARP + 2;
constexpr int TC_THREADS = 640;   // the last warp has no work: register counts are set per group of four warps
constexpr int TC_KSTEP = 128;     // inputs per K step
constexpr int TC_B_SLOTS = 3, TC_MAX_RAW = 12;
constexpr uint32_t TC_A_COLS = 64;
// Tensor memory (512 columns) and registers by tokens per block (NT steps of 16).  Up to 32 tokens: four accumulators of 64 columns and two
// A slots per weight tile, and few enough registers that the row kernels in front of and behind a GEMM fit beside it (its weight
// requests start while they run).  More: three accumulators of 128 columns and one A slot per weight tile.
template <int NT> struct TcShape {
    static constexpr bool SMALL = NT <= 2;
    static constexpr int D_SLOTS = SMALL ? 4 : 3, A_SLOTS = SMALL ? 2 : 1;
    static constexpr uint32_t D_COLS = SMALL ? 64 : 128, A_COL0 = D_COLS * D_SLOTS;
    // registers a thread: at launch (640 threads), then loaders (8 warps), drain (8 warps), the others (4 warps); the split never exceeds the launch
    static constexpr int LAUNCH = SMALL ? 72 : 96, LOAD = SMALL ? 64 : 80, DRAIN = SMALL ? 96 : 136, REST = 40;
    static_assert(8 * LOAD + 8 * DRAIN + 4 * REST <= 20 * LAUNCH && A_COL0 + 2 * A_SLOTS * TC_A_COLS == 512, "register split and tensor memory");
};
constexpr uint32_t TC_WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// One poll of a barrier phase; the hardware parks the thread for a short time of its own choice if the phase is not complete.  (An
// explicit time hint of 2 microseconds, or a sleep between polls, made every hand-over between roles several hundred clocks longer.)
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}
// bounded: gives up after TC_WAIT_LIMIT polls or soon after another thread has given up
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* failed) {
#pragma unroll 1
    for (uint32_t i = 0; i < TC_WAIT_LIMIT; i++) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 63) == 63 && *failed) return false;
    }
    return false;
}
// the same for a whole warp (every lane polls: its reads are ordered behind the arrivals)
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* failed) {
    const bool ok = mbar_wait(bar, parity, failed);
    return __all_sync(0xffffffffu, ok);
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void commit_to(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
// K-major operand descriptor: rows of 128 bytes, 128-byte swizzle, 8-row atoms of 1024 bytes.  Low word: start address (16-byte units)
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t saddr) { return ((saddr >> 4) & 0x3FFFu) | (1u << 16); }
constexpr uint32_t UMMA_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
// D (+)= A (tensor memory) * B (shared memory), 128 x N x 16
template <bool ACC>
__device__ __forceinline__ void mma_f16(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc) {
    asm volatile("{\n.reg .pred p;\n.reg .b64 db;\nsetp.ne.b32 p, %5, 0;\nmov.b64 db, {%2, %3};\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n}"
                 ::"r"(d), "r"(a), "r"(b_lo), "n"(UMMA_DESC_HI), "r"(idesc), "n"(ACC ? 1 : 0) : "memory");
}
__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b));
    return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long d) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(d));
    return v;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint32_t hadd2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t hfma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// 8 weights of a row -> four f16 pairs q - z, inputs (0,4) (1,5) (2,6) (3,7).  0x6400 | n is 1024 + n in f16, 0x6400 | n << 4 is 1024 + 16 n;
// c1 = -(1024 + z), c2 = -(64 + z): every step is exact.
__device__ __forceinline__ void unpack8(uint32_t v, uint32_t c1, uint32_t c2, uint32_t* out) {
    constexpr uint32_t LO = 0x000F000Fu, HI = 0x00F000F0u, ONE = 0x64006400u, SIXTEENTH = 0x2C002C00u;
    const uint32_t w = v >> 8;
    out[0] = hadd2(and_or(v, LO, ONE), c1);
    out[1] = hfma2(and_or(v, HI, ONE), SIXTEENTH, c2);
    out[2] = hadd2(and_or(w, LO, ONE), c1);
    out[3] = hfma2(and_or(w, HI, ONE), SIXTEENTH, c2);
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]),
                   "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t (&v)[16], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
                   "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
template <int N> __device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// Bytes between record runs in shared memory: the run's records, padded so that runs start an odd number of 16-byte units apart (modulo 8)
__host__ __device__ constexpr uint32_t tc_run_bytes(int W) { return (uint32_t)(4 / W) * (256u * W + 80u) + (W == 4 ? 0u : 16u); }

// A CTA's piece of the line of (tile, K step) pairs, one tile at a time.
struct Seg { int mat, pair, tb, k0, k1, slice; };
struct Walk {
    int w, w1;
    __device__ __forceinline__ explicit Walk(const TcParams& P) : w((int)blockIdx.x * P.q), w1(min(P.total, ((int)blockIdx.x + 1) * P.q)) {}
    __device__ __forceinline__ bool next(const TcParams& P, Seg& s) {
        if (w >= w1) return false;
        const int T = w / P.KS;
        s.k0 = w - T * P.KS;
        s.k1 = min(P.KS, s.k0 + (w1 - w));
        s.slice = (int)blockIdx.x - (T * P.KS) / P.q;
        int begin = 0;
        s.mat = 0;
        while (s.mat + 1 < P.nmat && T >= P.mat[s.mat].tile_end) begin = P.mat[s.mat++].tile_end;
        s.pair = (T - begin) / P.ntb;
        s.tb = (T - begin) - s.pair * P.ntb;
        w += s.k1 - s.k0;
        return true;
    }
};

struct Drain {
    uint64_t *mma_done, *acc_free;
    volatile int* failed;
    uint32_t tmem_base;
    int warp, lane;
};

__device__ __forceinline__ void tmem_fetch(uint32_t (&c)[2][16], uint32_t col, int tq) {  // both digit columns of 16 tokens
    tmem_ld16(c[0], col);
    tmem_ld16(c[1], col + (uint32_t)tq);
}
// 16 tokens: scale * (4096 hi + lo), the digit sums being exact integers
__device__ __forceinline__ void add16(const uint32_t (&c)[2][16], unsigned long long* sum, unsigned long long s2, unsigned long long k4096) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const unsigned long long hi = pack2(__uint_as_float(c[0][2 * j]), __uint_as_float(c[0][2 * j + 1]));
        const unsigned long long lo = pack2(__uint_as_float(c[1][2 * j]), __uint_as_float(c[1][2 * j + 1]));
        sum[j] = fma2(s2, fma2(hi, k4096, lo), sum[j]);
    }
}

// The drain role of one warp: NT steps of 16 tokens per group.  A warp may read the 32 tensor-memory lanes of the quadrant given by its
// index in the CTA modulo 4; the first four drain warps take the first weight tile's accumulator, the others the second's.
template <int W, int NT>
__device__ __forceinline__ bool drain_tiles(const TcParams& P, const Drain& D, Walk& walk) {
    constexpr int RT = TC_TILE_ROWS / 128, tq = 16 * NT, GPS = 4 / W;
    using S = TcShape<NT>;
    constexpr uint32_t UB = 256u * W + 80u;
    const int quad = D.warp & 3, rec16 = D.lane & 7, rr = 4 * quad + (D.lane >> 3), rt = (D.warp - TC_LOAD_WARPS) >> 2;
    const uint32_t tquad = D.tmem_base + ((uint32_t)(32 * quad) << 16);
    const unsigned long long k4096 = pack2(4096.0f, 4096.0f);
    unsigned long long acc[8 * NT];                        // pairs of tokens
    uint32_t ca[2][16], cb[2][16];                         // digit columns of a step and of the next
    uint32_t d = rt, dph = 0;                              // accumulator of the next unit (every other unit is this warp's) and its parity
    while (walk.w < walk.w1) {
        Walk w0 = walk;
        Seg sg;
        walk.next(P, sg);
        const TcMat& X = P.mat[sg.mat];
        const int g0 = sg.k0 * GPS;
        int n = min(sg.k1 * GPS, P.G) - g0;                // groups of this tile
        // The row's scales come straight from its records in global memory (the L2 has them: the raw copies pass through it), three
        // groups ahead.  Read from shared memory when a group was ready they cost 200 clocks of every group: the memory is busy.
        const char* sp = reinterpret_cast<const char*>(X.rec) + ((size_t)min((sg.pair * RT + rt) * 8 + rec16, X.tiles16 - 1) * P.G + g0) * UB + 256 * W + 4 * rr;
        auto scale = [&](int ahead) { return __ldg(reinterpret_cast<const float*>(sp + (size_t)min(ahead, n - 1) * UB)); };
        float s_a = scale(0), s_b = scale(1), s_c = scale(2);
        // The tokens' factors, one or two per lane, well before they are needed.  They are the output of the kernel in front, which may run beside this
        // one until the wait above: no read-only loads.
        const int t0 = sg.tb * tq + D.lane;
        const float f0 = D.lane < tq && t0 < P.M ? P.osc[t0] : 0.f, f1 = NT > 2 && D.lane + 32 < tq && t0 + 32 < P.M ? P.osc[t0 + 32] : 0.f;
#pragma unroll
        for (int i = 0; i < 8 * NT; i++) acc[i] = 0ull;
#pragma unroll 1
        for (; n > 0; n--) {
            const uint32_t tcol = tquad + d * S::D_COLS;   // column of digit p, token t: p * tq + t
            if (!mbar_wait_warp(D.mma_done + d, dph, D.failed)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_fetch(ca, tcol, tq);
            const unsigned long long s2 = pack2(s_a, s_a);
            s_a = s_b; s_b = s_c; s_c = scale(3);
            sp += UB;
#pragma unroll
            for (int st = 0; st < NT; st++) {
                tmem_wait_ld();
                if (st + 1 < NT) {
                    if (S::SMALL) { add16(ca, acc + 8 * st, s2, k4096); tmem_fetch(ca, tcol + 16 * (st + 1), tq); continue; }  // (one set of registers)
                    if (st & 1) tmem_fetch(ca, tcol + 16 * (st + 1), tq); else tmem_fetch(cb, tcol + 16 * (st + 1), tq);
                } else {  // everything has been read: the accumulator is free again
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (D.lane == 0) mbar_arrive(D.acc_free + d);
                }
                add16(st & 1 && !S::SMALL ? cb : ca, acc + 8 * st, s2, k4096);
            }
            d += RT;
            if (d >= S::D_SLOTS) { d -= S::D_SLOTS; dph ^= 1u; }
        }
        w0.next(P, sg);  // (worked out again: the coordinates would take registers from the loop above)
        // ---- this tile's share of the output: slice 0 goes to the output rows, later slices to the part buffers
        if (__any_sync(0xffffffffu, *D.failed)) return false;  // (the whole warp: the factors below are shuffled)
        const int orow = (sg.pair * RT + rt) * 128 + rec16 * 16 + rr, m0 = sg.tb * tq;
        const size_t ld = sg.slice == 0 ? (size_t)X.ldo : (size_t)X.rows;
        float* dst = (sg.slice == 0 ? X.out : X.part + (size_t)(sg.slice - 1) * P.M * X.rows) + (size_t)m0 * ld + orow;
#pragma unroll
        for (int i = 0; i < 16 * NT; i += 2) {
            const float2 y = unpack2(acc[i / 2]);
            const float fa = __shfl_sync(0xffffffffu, i < 32 ? f0 : f1, i & 31), fb = __shfl_sync(0xffffffffu, i < 32 ? f0 : f1, (i + 1) & 31);
            if (orow < X.rows && m0 + i < P.M) dst[(size_t)i * ld] = y.x * fa;
            if (orow < X.rows && m0 + i + 1 < P.M) dst[(size_t)(i + 1) * ld] = y.y * fb;
        }
    }
    return true;
}

}  // namespace

template <int W, int NT>
__global__ void __maxnreg__(TcShape<NT>::LAUNCH) gemm_q4_tc_kernel(const __grid_constant__ TcParams P) {
    using S = TcShape<NT>;
    constexpr int RT = TC_TILE_ROWS / 128, tq = 16 * NT;     // weight tiles of a tile; tokens of a block
    constexpr int GS = 32 * W, GPS = TC_KSTEP / GS;          // inputs per group, groups per K step
    constexpr uint32_t UB = 256u * W + 80u;                  // bytes of a unit record
    constexpr uint32_t RUN = tc_run_bytes(W);                // room of a record run (16 rows x one K step)
    constexpr uint32_t RAW_BYTES = 8 * RUN;                  // raw weights of one 128-row tile and K step
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t raw_full[TC_MAX_RAW], raw_empty[TC_MAX_RAW], a_full[RT * S::A_SLOTS], a_empty[RT * S::A_SLOTS], b_full[TC_B_SLOTS], b_empty[TC_B_SLOTS],
        mma_done[S::D_SLOTS], acc_free[S::D_SLOTS];
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int failed;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    constexpr uint32_t b_bytes = 512u * tq;                   // a digit block
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* stage_b = smem;                                  // [TC_B_SLOTS][2 halves][2 tq rows][128 bytes]
    uint8_t* raw = stage_b + TC_B_SLOTS * b_bytes;            // [nraw][8 runs]

    if (tid == 0) {
        for (int i = 0; i < TC_MAX_RAW; i++) { mbar_init(&raw_full[i], 1); mbar_init(&raw_empty[i], 4); }
        for (int i = 0; i < RT * S::A_SLOTS; i++) { mbar_init(&a_full[i], 4); mbar_init(&a_empty[i], 1); }
        for (int i = 0; i < TC_B_SLOTS; i++) { mbar_init(&b_full[i], 1); mbar_init(&b_empty[i], 1); }
        for (int i = 0; i < S::D_SLOTS; i++) { mbar_init(&mma_done[i], 1); mbar_init(&acc_free[i], 4); }
        failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TC_MMA_WARP) {  // all 512 columns of tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_base_s)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_s;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");  // the kernel behind this one may set itself up

    // tensor-memory lane 32 q + l of a tile is row 16 (l & 7) + 4 q + (l >> 3) of its 128 rows
    const int quad = warp & 3, rec16 = lane & 7, rr = 4 * quad + (lane >> 3);
    Walk walk(P);
    Seg sg;
    if (warp < TC_LOAD_WARPS) {
        regs_down<S::LOAD>();
        // ================= loaders ==================================================================================
        // warps 0-3 take the first weight tile of every K step, warps 4-7 the second; a thread has a whole row of it
        const int rt = warp >> 2;
        const uint8_t* rec = raw + rec16 * RUN + rr * (16 * W);      // a row's words of a group follow one another
        const uint32_t z_shift = 4 * (rr & 7);
        const uint8_t* zeros = raw + rec16 * RUN + 256 * W + 64 + 4 * (rr >> 3);
        const uint32_t tquad = tmem_base + ((uint32_t)(32 * quad) << 16) + S::A_COL0;
        uint32_t rs = rt, rph = 0, as = rt, aph = 1;  // slot and parity of the raw ring and of this weight tile's A slots (a fresh "empty" barrier passes parity 1)
        bool ok = true;
        while (ok && walk.next(P, sg)) {
#pragma unroll 1
            for (int n = sg.k1 - sg.k0; n > 0; n--) {
                if (!mbar_wait_warp(&raw_full[rs], rph, &failed)) { ok = false; break; }
                const uint32_t so = rs * RAW_BYTES;
                constexpr int PER = 4 / GPS;                     // 32-weight pieces of a group
                uint4 v[4];
                uint32_t z[GPS];
#pragma unroll
                for (int i = 0; i < 4; i++) v[i] = *reinterpret_cast<const uint4*>(rec + so + (i / PER) * UB + (i % PER) * 16);
#pragma unroll
                for (int gg = 0; gg < GPS; gg++) z[gg] = *reinterpret_cast<const uint32_t*>(zeros + so + gg * UB);
                __syncwarp();
                if (lane == 0) mbar_arrive(&raw_empty[rs]);
                const uint32_t tcol = tquad + as * TC_A_COLS;
                auto unpack32 = [&](int i, uint32_t* a) {
                    const uint32_t zz = ((z[i / PER] >> z_shift) & 15u) + 1u;                                  // src/gptq.rs:148
                    const uint32_t c1 = 0xE400E400u + zz * 0x00010001u, c2 = 0xD400D400u + zz * 0x00100010u;  // -(1024 + z), -(64 + z), twice each
                    unpack8(v[i].x, c1, c2, a); unpack8(v[i].y, c1, c2, a + 4); unpack8(v[i].z, c1, c2, a + 8); unpack8(v[i].w, c1, c2, a + 12);
                };
                // with one A slot per weight tile the first half is turned into f16 before the slot is free
                constexpr int AHEAD = S::A_SLOTS == 1 ? 2 : 0;
                uint32_t early[2][16];
#pragma unroll
                for (int i = 0; i < AHEAD; i++) unpack32(i, early[i]);
                if (!mbar_wait_warp(&a_empty[as], aph, &failed)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int i = 0; i < AHEAD; i++) tmem_st16(tcol + i * 16, early[i]);
#pragma unroll
                for (int i = AHEAD; i < 4; i++) {
                    uint32_t a[16];
                    unpack32(i, a);
                    tmem_st16(tcol + i * 16, a);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[as]);
                rs += RT; if (rs >= (uint32_t)P.nraw) { rs -= P.nraw; rph ^= 1u; }
                as += RT; if (as >= RT * S::A_SLOTS) { as = rt; aph ^= 1u; }
            }
        }
        if (!ok && lane == 0) { failed = 1; if (P.status) atomicExch(P.status, 2003); }
    } else if (warp < TC_RAW_WARP) {
        regs_up<S::DRAIN>();
        // ================= drain warps ==================================================================================
        asm volatile("griddepcontrol.wait;" ::: "memory");     // the tokens' factors (and the output buffers) belong to the kernels in front of this one
        const Drain D{mma_done, acc_free, &failed, tmem_base, warp, lane};
        const bool ok = drain_tiles<W, NT>(P, D, walk);
        if (!ok && lane == 0) { failed = 1; if (P.status) atomicExch(P.status, 2002); }
    } else {
        regs_down<S::REST>();  // one instruction for the four warps: it is a warpgroup operation
        if (warp == TC_RAW_WARP) {
        // ================= raw weights: lanes 0-7 copy one record run each ================================================
        uint32_t rs = 0, rph = 1;
        bool ok = true;
        while (ok && walk.next(P, sg)) {
            const TcMat& X = P.mat[sg.mat];
            const uint8_t* base[RT];
#pragma unroll
            for (int rt = 0; rt < RT; rt++) {  // rows beyond the matrix read the last records (results dropped)
                const int t16 = min((sg.pair * RT + rt) * 8 + (lane & 7), X.tiles16 - 1);
                base[rt] = reinterpret_cast<const uint8_t*>(X.rec) + ((size_t)t16 * P.G + (size_t)sg.k0 * GPS) * UB;
            }
#pragma unroll 1
            for (int k = sg.k0; k < sg.k1 && ok; k++) {
                const uint32_t bytes = (uint32_t)min(GPS, P.G - k * GPS) * UB;
#pragma unroll
                for (int rt = 0; rt < RT; rt++) {
                    if (!mbar_wait_warp(&raw_empty[rs], rph, &failed)) { ok = false; break; }
                    if (lane == 0) mbar_expect_tx(&raw_full[rs], 8 * bytes);
                    __syncwarp();
                    if (lane < 8) bulk_g2s(smem_addr(raw) + rs * RAW_BYTES + lane * RUN, base[rt], bytes, &raw_full[rs]);
                    base[rt] += GPS * UB;
                    if (++rs == (uint32_t)P.nraw) { rs = 0; rph ^= 1u; }
                }
            }
        }
        if (!ok && lane == 0) { failed = 1; if (P.status) atomicExch(P.status, 2005); }
        } else if (warp == TC_B_WARP) {
        // ================= digit blocks: one thread ========================================================================
        if (lane == 0) {
            asm volatile("griddepcontrol.wait;" ::: "memory");  // the digit image is the output of the kernel in front of this one
            uint32_t bs = 0, bph = 1;
            bool ok = true;
            while (ok && walk.next(P, sg)) {
                const uint8_t* src = P.mat[sg.mat].img + ((size_t)sg.tb * P.KS + sg.k0) * b_bytes;
#pragma unroll 1
                for (int k = sg.k0; k < sg.k1; k++) {
                    if (!mbar_wait(&b_empty[bs], bph, &failed)) { ok = false; break; }
                    mbar_expect_tx(&b_full[bs], b_bytes);
                    bulk_g2s(smem_addr(stage_b) + bs * b_bytes, src, b_bytes, &b_full[bs]);
                    src += b_bytes;
                    if (++bs == TC_B_SLOTS) { bs = 0; bph ^= 1u; }
                }
            }
            if (!ok) { failed = 1; if (P.status) atomicExch(P.status, 2004); }
        }
        } else if (warp == TC_MMA_WARP) {
            // ================= MMA issue ===============================================================================
            // The whole warp walks the loop and one elected lane issues: the operands of tcgen05.mma are uniform registers, and values
            // that the compiler knows to be the same in all lanes need no move into them (inside an `if (lane == 0)` every MMA took
            // about 90 clocks to issue, more than it takes to execute).  The tensor memory allocated is all there is: it starts at 0.
            // Operand addresses are kept as the low words of the descriptors and advanced by constants: this warp shares its scheduler
            // with four busy ones and every instruction between two MMAs costs it about ten clocks.
            const bool leader = elect_one();
            constexpr uint32_t N = 2u * tq;
            // instruction descriptor: D f32, A and B f16, both K-major, N, M = 128
            constexpr uint32_t idesc = (1u << 4) | ((N >> 3) << 17) | ((128u >> 4) << 24);
            const uint32_t b_lo0 = umma_desc_lo(smem_addr(stage_b)), slot_units = b_bytes >> 4, half_units = N * 128 / 16;  // (N rows of 128 bytes per half)
            uint32_t as = 0, aph = 0, bs = 0, bph = 0, d = 0, dph = 1;
            bool ok = true;
            while (ok && walk.next(P, sg)) {
#pragma unroll 1
                for (int k = sg.k0; k < sg.k1 && ok; k++) {
                    const int ng = min(GPS, P.G - k * GPS);
                    const uint32_t b_half[2] = {b_lo0 + bs * slot_units, b_lo0 + bs * slot_units + half_units};
                    if (!mbar_wait_warp(&b_full[bs], bph, &failed)) { ok = false; break; }
#pragma unroll
                    for (int gg = 0; gg < GPS; gg++) {
                        if (gg >= ng) break;
#pragma unroll
                        for (int rt = 0; rt < RT; rt++) {
                            if (gg == 0 && ok) ok = mbar_wait_warp(&a_full[as + rt], aph, &failed);
                            if (ok) ok = mbar_wait_warp(&acc_free[d], dph, &failed);
                            if (!ok) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const uint32_t td = d * S::D_COLS, ta = S::A_COL0 + (as + rt) * TC_A_COLS;
                            if (leader) {
#pragma unroll
                                for (int j = 0; j < GS / 16; j++) {  // 16 inputs: 8 columns of A, 32 bytes of B
                                    const int k0 = gg * GS + 16 * j;
                                    if (j == 0) mma_f16<false>(td, ta + k0 / 2, b_half[k0 / 64] + (k0 % 64) / 8, idesc);
                                    else mma_f16<true>(td, ta + k0 / 2, b_half[k0 / 64] + (k0 % 64) / 8, idesc);
                                }
                                commit_to(&mma_done[d]);
                                if (gg == ng - 1) {
                                    commit_to(&a_empty[as + rt]);
                                    if (rt == RT - 1) commit_to(&b_empty[bs]);
                                }
                            }
                            __syncwarp();
                            if (++d == S::D_SLOTS) { d = 0; dph ^= 1u; }
                        }
                        if (!ok) break;
                    }
                    as += RT; if (as == RT * S::A_SLOTS) { as = 0; aph ^= 1u; }
                    if (++bs == TC_B_SLOTS) { bs = 0; bph ^= 1u; }
                }
            }
            if (!ok && lane == 0) { failed = 1; if (P.status) atomicExch(P.status, 2001); }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (failed && tid < TC_MAX_RAW + TC_B_SLOTS) {  // copies may still be on their way into this CTA's shared memory: a bounded time to land
        uint64_t* bar = tid < TC_MAX_RAW ? &raw_full[tid] : &b_full[tid - TC_MAX_RAW];
        for (int i = 0; i < 64; i++) { mbar_try_wait(bar, 0); mbar_try_wait(bar, 1); }
    }
    if (warp == TC_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
}

namespace {
int tc_max_smem = 200 * 1024;
size_t tc_fixed_bytes(int tq) { return 1024 + (size_t)TC_B_SLOTS * 512 * tq; }
size_t tc_raw_bytes(int gs) { return 8 * (size_t)tc_run_bytes(gs / 32); }
int tc_raw_slots(int gs, int tq) { return (int)std::min<size_t>(TC_MAX_RAW, (tc_max_smem - tc_fixed_bytes(tq)) / tc_raw_bytes(gs)); }
}  // namespace

void gemm_tc_tokens(int M, int* tq, int* ntb) {  // blocks of at most 64 tokens, as even as multiples of 16 allow
    *ntb = (M + TC_MAX_TOKENS - 1) / TC_MAX_TOKENS;
    *tq = ((M + *ntb - 1) / *ntb + 15) & ~15;
}

size_t gemm_tc_image_bytes(int in, int tokens) {
    return (size_t)((in + TC_KSTEP - 1) / TC_KSTEP) * 512 * ((tokens + TC_MAX_TOKENS - 1) / TC_MAX_TOKENS * TC_MAX_TOKENS);
}

// slices the most divided tile of a launch can have
int gemm_tc_slices(const TcParams& p) { return p.total <= p.q ? 1 : p.q >= p.KS ? (p.q % p.KS ? 2 : 1) : (p.KS - 2) / p.q + 2; }

// Fills in the geometry of a launch: p.mat[0 .. nmat) hold the matrices, p.G / p.M the groups and tokens.
void gemm_tc_plan(TcParams& p, int gs, int sms) {
    gemm_tc_tokens(p.M, &p.tq, &p.ntb);
    p.gs = gs;
    p.KS = (p.G * gs + TC_KSTEP - 1) / TC_KSTEP;
    int tiles = 0;
    for (int i = 0; i < p.nmat; i++) {
        tiles += (p.mat[i].tiles16 + TC_TILE_ROWS / 16 - 1) / (TC_TILE_ROWS / 16) * p.ntb;
        p.mat[i].tile_end = tiles;
    }
    p.total = tiles * p.KS;
    // equal pieces for the SMs, but no tile in more than TC_MAX_SLICES pieces
    p.q = std::max((p.total + sms - 1) / sms, (p.KS + TC_MAX_SLICES - 2) / (TC_MAX_SLICES - 1));
    p.grid = (p.total + p.q - 1) / p.q;
    p.nraw = tc_raw_slots(gs, p.tq);
}

cudaError_t gemm_tc_init(int max_smem) {
    tc_max_smem = max_smem;
    cudaError_t e;
#define L2_TC_ATTR(W, NT) if ((e = cudaFuncSetAttribute(gemm_q4_tc_kernel<W, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, tc_max_smem)) != cudaSuccess) return e;
#define L2_TC_ATTR_W(W) L2_TC_ATTR(W, 1) L2_TC_ATTR(W, 2) L2_TC_ATTR(W, 3) L2_TC_ATTR(W, 4)
    L2_TC_ATTR_W(4) L2_TC_ATTR_W(2) L2_TC_ATTR_W(1)
#undef L2_TC_ATTR_W
#undef L2_TC_ATTR
    return cudaSuccess;
}

// Launched programmatically behind the quantiser; the roles that read the quantiser's output wait for it inside the kernel.
cudaError_t launch_gemm_tc(const TcParams& p, cudaStream_t st) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(p.grid);
    cfg.blockDim = dim3(TC_THREADS);
    // (always more than half of an SM: one CTA, one owner of the tensor memory, per SM)
    cfg.dynamicSmemBytes = std::max<size_t>(120 * 1024, tc_fixed_bytes(p.tq) + (size_t)p.nraw * tc_raw_bytes(p.gs));
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    g_launches++;
    auto by_tokens = [&](auto w) {  // one instantiation per group size and 16-token steps
        constexpr int W = decltype(w)::value;
        switch (p.tq / 16) {
            case 1: return cudaLaunchKernelEx(&cfg, gemm_q4_tc_kernel<W, 1>, p);
            case 2: return cudaLaunchKernelEx(&cfg, gemm_q4_tc_kernel<W, 2>, p);
            case 3: return cudaLaunchKernelEx(&cfg, gemm_q4_tc_kernel<W, 3>, p);
            default: return cudaLaunchKernelEx(&cfg, gemm_q4_tc_kernel<W, 4>, p);
        }
    };
    if (p.gs == 128) return by_tokens(std::integral_constant<int, 4>());
    if (p.gs == 64) return by_tokens(std::integral_constant<int, 2>());
    return by_tokens(std::integral_constant<int, 1>());
}

}  // namespace l2
