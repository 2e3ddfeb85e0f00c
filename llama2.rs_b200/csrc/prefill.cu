// Host side of the batched forward pass transformer<B>, B >= 2 (src/models.rs:178-298): the
// sequence of launches for a batch of tokens.  Every QLinear is a tcgen05 GEMM on exact
// integer digits of the activations (gemm_tc.cu); no logits are produced, as in the reference.
#include <cstring>

#include "model.h"

namespace l2 {

void tc_set_matrix(TcParams& t, int i, const DevQ& q, const uint8_t* img, float* out, int ldo, float* part) {
    TcMat& m = t.mat[i];
    m.rec = q.rec; m.img = img; m.out = out; m.part = part;
    m.tiles16 = q.tiles; m.rows = q.out; m.ldo = ldo;
    t.G = q.G;
}

TcOut tc_out(const TcParams& t, int i) {
    TcOut o{};
    o.out = t.mat[i].out; o.part = t.mat[i].part; o.ldo = t.mat[i].ldo; o.rows = t.mat[i].rows;
    o.tile0 = i ? t.mat[i - 1].tile_end : 0;
    o.ntb = t.ntb; o.tq = t.tq; o.KS = t.KS; o.q = t.q; o.rq = 1.0f / (float)t.q; o.M = t.M;
    return o;
}

static RowParams row_params(int mode, int in, const TcParams& t) {
    RowParams r{};
    r.mode = mode; r.in = in; r.M = t.M; r.tq = t.tq; r.KS = t.KS;
    return r;
}

// out[m][:] = QLinear(x[m][:]) for m < M, x in natural order.  part: room for (slices - 1) * M * rows floats (part_floats).
int gemm_batched(const DevQ& q, const float* x, int M, uint8_t* img, float* osc, float* out, float* part, int* status, int sms, cudaStream_t st) {
    TcParams t{};
    t.nmat = 1; t.M = M; t.osc = osc; t.status = status;
    tc_set_matrix(t, 0, q, img, out, q.out, part);
    gemm_tc_plan(t, q.gs, sms);
    RowParams r = row_params(ROW_PLAIN, q.in, t);
    r.x = const_cast<float*>(x); r.ldx = q.in; r.nmat = 1; r.perm[0] = q.perm16; r.img[0] = img; r.osc = osc;
    L2_CUDA(launch_row_quant(r, sms, st));
    L2_CUDA(launch_gemm_tc(t, st));
    if (gemm_tc_slices(t) > 1) launch_finish(tc_out(t, 0), nullptr, out, q.out, false, st);
    return L2_OK;
}

// Floats of part buffer that launches of up to `cap` tokens over matrices of rows[0 .. n) rows (inputs: in) need.
size_t part_floats(const int* rows, int n, int in, int gs, int cap, int sms) {
    size_t most = 0, total_rows = 0;
    for (int i = 0; i < n; i++) total_rows += rows[i];
    for (int M = 2; M <= cap; M++) {
        TcParams t{};
        t.nmat = n; t.M = M; t.G = in / gs;
        for (int i = 0; i < n; i++) t.mat[i].tiles16 = (rows[i] + 15) / 16;
        gemm_tc_plan(t, gs, sms);
        most = std::max(most, (size_t)(gemm_tc_slices(t) - 1) * M * total_rows);
    }
    return most;
}

void free_batch(l2_model* m) {
    BatchBuffers* b = m->batch;
    if (!b) return;
    for (void* p : b->allocs) cudaFree(p);
    if (b->h_stage) cudaFreeHost(b->h_stage);
    delete b;
    m->batch = nullptr;
}

// The buffers of batches of up to `cap` tokens; cudaErrorMemoryAllocation (and no buffers) where the device does not have the room.
static cudaError_t alloc_batch(l2_model* m, int cap) {
    const bool tp = m->tp_world > 1;
    const l2_config& c = m->shape.c;
    const int T = m->tp_world, D = c.dim, KV = m->shape.kv_dim(), H = c.hidden_dim, Dl = D / T, KVl = KV / T, Hl = H / T, gs = c.group_size;
    BatchBuffers* b = m->batch = new BatchBuffers;
    b->cap = cap; b->tp = tp;
    const int qkv[3] = {Dl, KVl, KVl}, w13[2] = {Hl, Hl}, one[1] = {Dl};
    const size_t parts = std::max(std::max(part_floats(qkv, 3, D, gs, cap, m->sms), part_floats(w13, 2, D, gs, cap, m->sms)),
                                  std::max(part_floats(one, 1, D, gs, cap, m->sms), part_floats(one, 1, H, gs, cap, m->sms)));
    const size_t B = cap, outs = std::max<size_t>((size_t)Dl + 2 * KVl, 2 * (size_t)Hl);
    // one allocation, cut into pieces of whole 256-byte lines
    size_t total = 0;
    auto room = [&](size_t bytes) { const size_t at = total; total += (bytes + 255) & ~(size_t)255; return at; };
    const size_t x = tp ? 0 : room(B * D * 4), att = tp ? 0 : room(B * D * 4), q = room(B * Dl * 4), y = room(B * outs * 4), part = room(parts * 4), osc = room(B * 4);
    const size_t img0 = room(gemm_tc_image_bytes(std::max(D, H), cap)), img1 = room(gemm_tc_image_bytes(D, cap)), img2 = room(gemm_tc_image_bytes(D, cap));
    const size_t tok = room(2 * B * sizeof(int)), done = room(256);
    char* base = nullptr;
    if (cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&base), total)) {
        cudaGetLastError();  // (an answer here, not an error of a later launch)
        free_batch(m);
        return e;
    }
    b->allocs.push_back(base);
    auto at = [&](size_t off) { return reinterpret_cast<float*>(base + off); };
    b->x = at(x); b->att = at(att); b->q = at(q); b->y = at(y); b->part = at(part); b->osc = at(osc);
    b->img[0] = reinterpret_cast<uint8_t*>(base + img0); b->img[1] = reinterpret_cast<uint8_t*>(base + img1); b->img[2] = reinterpret_cast<uint8_t*>(base + img2);
    b->tok = reinterpret_cast<int*>(base + tok);
    if (tp) {  // the vectors every rank needs in full live in the model's pool, where the peers store their columns
        b->x = reinterpret_cast<float*>(m->tp_pool + m->tp_batch_off[0]);
        b->att = reinterpret_cast<float*>(m->tp_pool + m->tp_batch_off[1]);
        b->hb = reinterpret_cast<float*>(m->tp_pool + m->tp_batch_off[2]);
        b->tp_done = reinterpret_cast<unsigned*>(base + done);
        if (cudaError_t e = cudaMemsetAsync(b->tp_done, 0, 256, m->stream)) { free_batch(m); return e; }
    }
    if (cudaError_t e = cudaMallocHost(reinterpret_cast<void**>(&b->h_stage), sizeof(int) * 2 * B * BATCH_RING)) { free_batch(m); return e; }
    return cudaSuccess;
}

// The batched forward's buffers belong to the model: its calls run one after another on one stream and every call that uses
// them ends synchronised, so all run states share them.  They grow once, from the size of a short batch to that of a long one, or to
// the largest half, quarter ... of it that the device has room for.  *limit: tokens of one batch.
int reserve_batch(l2_model* m, int M, int* limit) {
    const int most = m->tp_world > 1 ? TC_MAX_TOKENS : MAX_BATCH;  // (the ranks' pools hold one token block)
    if (!m->batch || m->batch->cap < std::min(M, most)) {
        if (m->batch) {
            L2_CUDA(cudaStreamSynchronize(m->stream));
            free_batch(m);
        }
        for (int cap = M <= TC_MAX_TOKENS ? TC_MAX_TOKENS : most;; cap /= 2) {
            const cudaError_t e = alloc_batch(m, cap);
            if (e == cudaSuccess) break;
            if (e != cudaErrorMemoryAllocation || cap <= TC_MAX_TOKENS)
                return fail(L2_ECUDA, "buffers of the batched forward (%d tokens): %s", cap, cudaGetErrorString(e));
        }
    }
    *limit = m->batch->cap;
    return L2_OK;
}

// The kernels of one batched forward of M tokens (their ids and positions already at b->tok), enqueued on `st`: per layer
//   row_quant -> wq/wk/wv -> rope_append -> attention -> row_quant -> wo -> row_quant (+ residual) -> w1/w3 -> row_quant (SwiGLU) -> w2
// each launched programmatically behind the one before it.  The GEMMs leave slices of their outputs and the kernels behind them
// add those up while they read them.
static int enqueue_batch(l2_state* s, int M, bool long_context, cudaStream_t st) {
    l2_model* m = s->m;
    const l2_config& c = m->shape.c;
    BatchBuffers* b = m->batch;
    const int D = c.dim, KV = m->shape.kv_dim(), H = c.hidden_dim, gs = c.group_size;
    // this rank's share (everything on one GPU): rows of wq / wo (= heads), of wk / wv (= kv heads), of w1 / w3 / w2's inputs
    const int T = b->tp ? m->tp_world : 1, R = b->tp ? m->tp_rank : 0;
    const int Dl = D / T, KVl = KV / T, heads_l = c.n_heads / T, kvh_l = c.n_kv_heads / T;
    int* status = &s->ctl->status;
    const int* tok = b->tok;
    const int* pos = b->tok + M;
    // After a stage whose result every rank needs in full, this rank's columns go to the peers (stores over NVLink into their
    // pools) and the peers' columns are waited for: the same data flow as the tagged exchanges of the token kernel.  The
    // exchanges are numbered by a counter on the device (every rank makes the same exchanges in the same order).
    auto gather = [&](int which, int ld, int col0, int ncols) {
        if (!b->tp) return;
        TpGatherParams g{};
        for (int r = 0; r < 8; r++) g.pool[r] = r < T ? m->tp_peers[r] : nullptr;
        g.buf_off = m->tp_batch_off[which]; g.flag_off = m->tp_flag_off; g.seq = reinterpret_cast<unsigned long long*>(m->tp_pool + m->tp_flag_off + 128);  // in the pool: it outlives run states, like the peers' counters
        g.done = b->tp_done; g.status = status; g.rank = R; g.world = T; g.M = M; g.ld = ld; g.col0 = col0; g.ncols = ncols;
        launch_tp_gather(g, st);
    };
    // the four launches of a layer differ from layer to layer in their matrices only
    auto launch = [&](std::initializer_list<const DevQ*> mats, TcParams& t) {
        t = TcParams{};
        t.nmat = (int)mats.size(); t.M = M; t.osc = b->osc; t.status = status;
        float *y = b->y, *part = b->part;
        int i = 0;
        for (const DevQ* q : mats) {
            tc_set_matrix(t, i, *q, b->img[i], y, q->out, part);
            y += (size_t)M * q->out;
            i++;
        }
        gemm_tc_plan(t, gs, m->sms);
        const size_t extra = (size_t)(gemm_tc_slices(t) - 1) * M;
        for (i = 0; i < t.nmat; i++) { t.mat[i].part = part; part += extra * t.mat[i].rows; }
    };
    auto quant = [&](RowParams r, std::initializer_list<const DevQ*> mats, bool permuted) {
        int i = 0;
        for (const DevQ* q : mats) { r.perm[i] = permuted ? q->perm16 : nullptr; r.img[i] = b->img[i]; i++; }
        r.nmat = i; r.osc = b->osc; r.eps = m->eps;
        return launch_row_quant(r, m->sms, st);
    };
    launch_embed_batch(m->tok_emb, tok, b->x, D, M, st);  // src/models.rs:189-191 (every rank holds the table: no exchange)
    const size_t ls = (size_t)c.seq_len * KV;
    TcParams t{};
    TcOut resid{};          // output of the GEMM whose result has not been added to x yet
    bool pending = false;
    for (int l = 0; l < c.n_layers; l++) {
        const DevLayer& y = m->layers[l];
        auto with_x = [&](const float* nw) {
            RowParams r = row_params(pending ? ROW_RESID : ROW_PLAIN, D, t);
            r.x = b->x; r.ldx = D; r.a = resid; r.nw = nw;
            pending = false;
            return r;
        };
        // a residual projection: on one GPU the next row_quant adds it to x; under tensor parallelism it updates this rank's columns of x
        auto add_to_x = [&](const DevQ& q) {
            resid = tc_out(t, 0);
            if (b->tp) { launch_finish(resid, nullptr, b->x + q.row0, D, true, st); gather(0, D, q.row0, q.out); }
            else pending = true;
        };
        // rmsnorm + wq/wk/wv (:217-226)
        launch({&y.wq, &y.wk, &y.wv}, t);
        L2_CUDA(quant(with_x(y.rms_att), {&y.wq, &y.wk, &y.wv}, true));
        L2_CUDA(launch_gemm_tc(t, st));
        // rope, all rows into the cache (this rank's kv heads of the full-width cache rows), then attention (:228-256)
        RopeParams r{};
        r.q = tc_out(t, 0); r.k = tc_out(t, 1); r.v = tc_out(t, 2);
        r.qout = b->q; r.ldq = Dl;
        r.kc = s->kc + (size_t)l * ls + (size_t)R * KVl; r.vc = s->vc + (size_t)l * ls + (size_t)R * KVl;
        r.rope_cos = m->rope_cos; r.rope_sin = m->rope_sin; r.pos = pos;
        r.n_heads = heads_l; r.n_kv_heads = kvh_l; r.kv_stride = KV;
        L2_CUDA(launch_rope_append(r, M, m->sms, st));
        AttnBatchParams a{};
        a.q = b->q; a.kc = r.kc; a.vc = r.vc; a.pos = pos; a.out = b->att + (size_t)R * Dl;
        a.n_kv_heads = kvh_l; a.ag = m->shape.attn_groups(); a.ldq = Dl; a.ldo = D; a.kv_stride = KV;
        L2_CUDA(launch_attn_batch(a, heads_l, M, long_context, m->sms, st));
        gather(1, D, R * Dl, Dl);
        // wo + residual (:260-264)
        launch({&y.wo}, t);
        RowParams ra = row_params(ROW_PLAIN, D, t);
        ra.x = b->att; ra.ldx = D;
        L2_CUDA(quant(ra, {&y.wo}, true));
        L2_CUDA(launch_gemm_tc(t, st));
        add_to_x(y.wo);
        // rmsnorm + w1/w3 + SwiGLU (:266-276); their rows are stored in w2's K order
        launch({&y.w1, &y.w3}, t);
        L2_CUDA(quant(with_x(y.rms_ffn), {&y.w1, &y.w3}, true));
        L2_CUDA(launch_gemm_tc(t, st));
        const TcOut h1 = tc_out(t, 0), h3 = tc_out(t, 1);
        // w2 + residual (:279-285)
        launch({&y.w2}, t);
        RowParams rh = row_params(b->tp ? ROW_PLAIN : ROW_SWIGLU, H, t);
        rh.a = h1; rh.b = h3; rh.x = b->hb; rh.ldx = H;
        if (b->tp) { launch_finish(h1, &h3, b->hb + y.w1.row0, H, false, st); gather(2, H, y.w1.row0, y.w1.out); }
        L2_CUDA(quant(rh, {&y.w2}, false));
        L2_CUDA(launch_gemm_tc(t, st));
        add_to_x(y.w2);
    }
    L2_CUDA(cudaGetLastError());
    return L2_OK;
}

// One batched forward.  The ids and positions travel through a pinned ring.
int forward_batch(l2_state* s, int M, const int32_t* tokens, const int32_t* pos) {
    l2_model* m = s->m;
    if (m->tp_world > 1) {
        if (!m->tp_direct || !m->tp_pool) return fail(L2_EINVAL, "batched forward under tensor parallelism needs the peers' pools attached");
        if (!m->tp_pool_owner) m->tp_pool_owner = s;
        if (m->tp_pool_owner != s) return fail(L2_EINVAL, "batched forward under tensor parallelism: another run state of this model works in the pool");
    }
    int limit;
    if (int rc = reserve_batch(m, M, &limit)) return rc;
    if (M < 1 || M > limit) return fail(L2_EINVAL, "forward_batch: %d tokens", M);
    BatchBuffers* b = m->batch;
    cudaStream_t st = m->stream;
    // token ids and positions: own pinned slot per call until the copy has run
    if (++b->stage_slot >= BATCH_RING) { L2_CUDA(cudaStreamSynchronize(st)); b->stage_slot = 0; }
    int* hs = b->h_stage + (size_t)b->stage_slot * 2 * b->cap;
    memcpy(hs, tokens, sizeof(int) * M);
    memcpy(hs + M, pos, sizeof(int) * M);
    L2_CUDA(cudaMemcpyAsync(b->tok, hs, sizeof(int) * 2 * M, cudaMemcpyHostToDevice, st));
    int last = 0;
    for (int i = 0; i < M; i++) last = std::max(last, (int)pos[i]);
    return enqueue_batch(s, M, last >= 192, st);
}

}  // namespace l2
