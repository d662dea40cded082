// Whole-token persistent kernel: every operation of one or more decode steps in a single
// cooperative launch, one CTA per SM — this library's counterpart of the reference's megakernel
// (`worker_kernel`, crates/luminal_cuda/src/block/interpreter.cu:136-326, assembled by
// crates/luminal_cuda/src/block/mod.rs:702-935).
//
// The reference interprets a task queue: thread 0 of every CTA claims (task, iteration) pairs with
// atomics, spins on per-dependency barrier counters (no bound on the wait), and dispatches through a
// switch.  Decode of a Llama-style layer has no dynamic structure to interpret, so here the schedule
// is the code: per layer five phases (q,k,v projections -> attention -> o projection -> gate/up +
// SwiGLU -> down projection), each followed by one grid-wide barrier (a monotonic arrival counter
// with a bounded wait), then the vocabulary projection and the greedy sample.
//
// What this buys over one kernel per operation: decode is bound by the weight stream from HBM, and
// the stream does not depend on the activations.  Each CTA has a producer warp that walks the
// CTA's share of *all* weight matrices of the step in order and keeps a ring of shared-memory
// stages full with bulk copies, regardless of where the consumer warps are.  While the consumers sit
// in a grid barrier, run attention, or quantise the next activation vector, the producer is already
// fetching the next operation's weights, so HBM never waits for a kernel boundary.  The multiply-adds
// run on the tensor core (lum_gemv_dev.cuh), so that the consumers empty a full ring in a fraction of the
// time HBM took to fill it: a stall is paid for only to the extent that it outlasts the ring.
#include <cstdlib>

#include "lum_attn_dev.cuh"
#include "lum_gemv_dev.cuh"
#include "lum_mega.cuh"

namespace lum {


// ---- grid-wide barrier ----------------------------------------------------------------------------
// Arrival counter in global memory, only ever incremented; barrier number b (0-based since the counter
// was last zeroed by the host) completes when the counter reaches (b + 1) * gridDim.x.  Called by all
// consumer threads; thread 0 arrives and waits, the rest wait on the named barrier.  The wait is bounded
// (LUM_WAIT_BUDGET_CYCLES); once it runs out the kernel-wide abort flag is raised and every later wait
// in every CTA returns at once.  Returns whether this CTA has given up, the same answer in all of its workers: they skip phases (and the
// barriers inside them) together, whatever the producer warp raises meanwhile.
// Threads for attention and grid barriers; the first kConsumers of them are the consumers of the weight stream.  With the producer warp 16 warps, which leaves
// 128 registers a thread; attention without tensor cores takes 512 threads.  Measured, ms a token of the Llama-3-8B shape behind 512 / 3000 rows: 4.25 / 4.70, with
// 512 workers (96 registers) 4.51 / 4.92.
template <int HD, int GM, bool BF16>
__host__ __device__ constexpr int mega_workers() { return BF16 && attn_tc_fits(HD, GM) ? 480 : kAttnThreads; }
template <int W>
__device__ __forceinline__ bool grid_barrier(const MegaArgs& a, unsigned long long& seq, volatile int* cta_abort, int tid) {
    named_sync(1, W);                        // all of this CTA's writes of the phase are issued
    if (tid == 0) {
        __threadfence();
        // gbar[0] counts arrivals; gbar[16] (its own 128-byte line, so polls do not queue behind the atomics) holds the
        // number of barriers completed.  The last CTA to arrive publishes the new generation; the others poll it.
        const unsigned long long old = atomicAdd(a.gbar, 1ull);
        const unsigned long long gen = seq + 1ull;
        volatile unsigned long long* gword = a.gbar + 16;
        if (old + 1ull == gen * gridDim.x) {
            *gword = gen;
        } else {
            const long long t0 = clock64();
            unsigned int spins = 0;
            while (*gword < gen) {
                __nanosleep(20);
                if ((++spins & 255u) == 0) {
                    if (*cta_abort) break;
                    if (*(volatile int*)a.abort_flag) { *cta_abort = 1; break; }
                    if (clock64() - t0 > LUM_WAIT_BUDGET_CYCLES) {
                        atomicOr(a.status, LUM_ST_WAIT_GRID);
                        *(volatile int*)a.abort_flag = 1;
                        *cta_abort = 1;
                        break;
                    }
                }
            }
        }
        __threadfence();
    }
    seq++;
    return named_or(1, W, *cta_abort != 0);
}

__device__ __forceinline__ AttnArgs attn_phase_args(const MegaArgs& a, const MegaLayer& L, bool bf16) {
    AttnArgs t{};
    t.q = a.qkv; t.k_new = a.qkv + (size_t)a.n_q * a.hd; t.v_new = t.k_new + (size_t)a.n_kv * a.hd;
    t.k_cache = L.kc; t.v_cache = L.vc; t.out = a.attn; t.part = a.attn_part; t.counters = a.attn_cnt;
    t.q_gain = L.q_norm; t.k_gain = L.k_norm; t.gain_kind = a.gain_kind; t.qk_eps = a.qk_eps;
    t.n_q = a.n_q; t.n_kv = a.n_kv; t.hd = a.hd; t.n_splits = a.n_splits; t.kv_bf16 = bf16; t.rope_style = a.rope_style;
    t.c_inv_d = a.c_inv_d; t.c_ln_theta = a.c_ln_theta; t.c_log2e = a.c_log2e; t.c_half_pi = a.c_half_pi; t.theta = a.theta;
    t.window = 0; t.max_seq = a.max_seq; t.status = a.status;
    return t;
}
// The phase before it: the cached rows of earlier tokens are asked for while the projections stream.
template <int HD, int GM, bool BF16>
__device__ __forceinline__ void attn_phase_prefetch(const MegaArgs& a, const MegaLayer& L, int pos, int tid) {
    if constexpr (BF16 && attn_tc_fits(HD, GM)) {
        if ((int)blockIdx.x >= a.n_kv * a.n_splits) return;
        constexpr int W = mega_workers<HD, GM, BF16>();
        const AttnArgs t = attn_phase_args(a, L, BF16);
        int r0, r1;
        attn_tc_range(t, (int)blockIdx.x % a.n_splits, pos, &r0, &r1);
        attn_tc_prefetch<HD>(t, (int)blockIdx.x / a.n_splits, r0, r1, tid, W);
    }
}
template <int HD, int GM, bool BF16>
__device__ __noinline__ void attn_phase(const MegaArgs& a, const MegaLayer& L, unsigned char* scratch_smem, int pos, int tid) {
    const int items = a.n_kv * a.n_splits;
    if ((int)blockIdx.x >= items) return;           // uniform per CTA: the whole CTA skips, barriers inside stay matched
    constexpr int W = mega_workers<HD, GM, BF16>();
    const AttnArgs t = attn_phase_args(a, L, BF16);
    const int kvh = (int)blockIdx.x / a.n_splits, split = (int)blockIdx.x % a.n_splits;
    if constexpr (BF16 && attn_tc_fits(HD, GM)) {
        // The heads are prepared and the states merged by all workers, the rows (asked for in the phase before) taken by four warps.  Of a warp per key, 128 workers
        // and this, this was the fastest.
        AttnTile<HD> f;
        AttnPre<HD, W> pre;
        attn_tc_pre<HD, W>(t, pre, kvh, split, tid >> 5, tid & 31);
        attn_tc_body<HD, GM / 4, false, W, false>(t, scratch_smem, f, pre, kvh, split, pos, tid, 1, false);
    } else {
        attn_decode_body<HD, GM, BF16>(t, scratch_smem, kvh, split, pos, tid, 1);
    }
}

// What one phase streams and where its vectors are.  Kept in shared memory and filled by one thread: as locals of 512 threads these structs (whose matrices are
// picked by number) were a stack of 2 KB a thread, far beyond the L1 that the rings leave (7.0 / 7.5 ms a token, now 4.25 / 4.70).
struct MegaPhase { GemvArgs ga; GemvPlan plan; XSource xs; bool streams; };

// Phase p of layer l (p = 0..4), or the head phase (p = 5).  The attention phase (p == 1) streams no weights.  Where the down projection runs as K ranges, their
// partial vectors join the residual stream in the next prologue, which moves it from one of x, x2 to the other.
__device__ __noinline__ void mega_fill(const MegaArgs& a, int l, int p, int token, MegaPhase* out) {
    const int H = a.hidden, qd = a.n_q * a.hd, kvd = a.n_kv * a.hd;
    const int ranges = gemv_k_ranges(a.ffn, a.kc_f);
    const MegaLayer& L = a.layers[l];
    auto stream = [&](int layer) { return ranges > 1 && (layer & 1) ? a.x2 : a.x; };
    GemvArgs g{};
    XSource xs{};
    g.wkind = WK_Q8; g.gain_kind = a.gain_kind; g.eps = a.eps; g.status = a.status; g.nseg = 1; g.epi = EPI_STORE;
    const int joined = p == 0 ? l - 1 : p == 5 ? l : -1;             // the layer whose partial vectors join in this phase's prologue
    if (joined >= 0 && ranges > 1) { xs.parts = a.part; xs.n_parts = ranges; xs.part_stride = a.part_ld; }
    switch (p) {
        case 0:   // q, k, v projections (RMSNorm in the prologue)
            g.K = H; g.KC = a.kc_h; g.nseg = 3;
            g.seg[0] = {L.wq, nullptr, qd, a.kc_h}; g.seg[1] = {L.wk, nullptr, kvd, a.kc_h}; g.seg[2] = {L.wv, nullptr, kvd, a.kc_h};
            g.gain = L.attn_norm; g.y = a.qkv;
            if (l == 0) { xs.table = a.embed; xs.table_kind = a.embed_kind; xs.token = token; xs.x_out = a.x; }      // the embedding row is x
            else { xs.x = stream(l - 1); if (ranges > 1) xs.x_out = stream(l); }
            break;
        case 2:   // o projection + residual
            g.K = qd; g.KC = a.kc_o; g.epi = EPI_RESID; g.seg[0] = {L.wo, nullptr, H, a.kc_o};
            g.y = stream(l); g.resid = g.y; xs.x = a.attn;
            break;
        case 3:   // gate, up projections + SwiGLU (RMSNorm in the prologue)
            g.K = H; g.KC = a.kc_h; g.epi = EPI_SWIGLU; g.nseg = 2;
            g.seg[0] = {L.wg, nullptr, a.ffn, a.kc_h}; g.seg[1] = {L.wu, nullptr, a.ffn, a.kc_h};
            g.gain = L.mlp_norm; g.y = a.h; xs.x = stream(l);
            break;
        case 4:   // down projection
            g.K = a.ffn; g.KC = a.kc_f; g.seg[0] = {L.wd, nullptr, H, a.kc_f}; xs.x = a.h;
            g.ksplit = ranges;
            if (ranges > 1) { g.y = a.part; g.y_range_stride = a.part_ld; }
            else { g.epi = EPI_RESID; g.y = a.x; g.resid = a.x; }
            break;
        case 5:   // final RMSNorm + vocabulary projection + greedy sample
            g.K = H; g.KC = a.kc_h; g.epi = EPI_ARGMAX; g.seg[0] = {a.lm_head, nullptr, a.vocab, a.kc_h};
            g.gain = a.final_norm; g.y = a.logits; xs.x = stream(l);
            break;
        default: break;
    }
    out->streams = p != 1;
    if (p != 1) { out->ga = g; out->xs = xs; out->plan = gemv_plan(g, (int)blockIdx.x, (int)gridDim.x, 750); }
}

template <bool ONE>
__device__ __noinline__ void mega_consume(const MegaPhase& m, const GemvSmem& g, ConsumerRing& cr, int tid, ArgBest* best) {
    GainRegs gr;
    gemv_gain_preload(m.ga, tid, gr);
    gemv_consume<false, ONE>(m.ga, m.xs, blockIdx.x == 0, m.plan, g, cr, tid, m.ga.status, best, gr);
}

template <int HD, int GM, bool BF16>
__global__ void __launch_bounds__(mega_workers<HD, GM, BF16>() + 32, 1) decode_mega(const __grid_constant__ MegaArgs a) {
    constexpr int W = mega_workers<HD, GM, BF16>();
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    __shared__ int s_tok;
    __shared__ MegaPhase s_phase[2], s_stream;        // the workers' phase and the next one; the producer's, which runs ahead
    __shared__ GemvSmem g;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cta = (int)blockIdx.x, ncta = (int)gridDim.x;
    if (tid == 0) gemv_carve(smem, a.k_max, GemvRings{(a.stages + 1) / 2, a.stages / 2, kFillTiles, kFillTiles}, &s_abort, &g, attn_smem_bytes(HD, GM));
    __syncthreads();
    gemv_cta_begin(g, tid, &s_abort);

    const bool is_worker = warp < W / 32, is_producer = !is_worker;
    ProducerRing pring{};
    ConsumerRing cring{0, 0u};
    unsigned long long seq = a.gbar_base;             // grid barriers passed so far
    unsigned long long pseq = a.gbar_base;            // running phase number: picks the job-claim counter of each phase
    bool producing = true, gone = false;              // gone: this CTA's workers have given up
    int pos = 0, buf = 0;
    if (is_worker) {
        pos = a.state->pos;
        const int tok = a.forced ? a.forced[0] : a.state->tok;
        if (pos < 0 || pos + a.n_tokens > a.max_seq || tok < 0 || tok >= a.vocab) {
            // Refuse the whole launch the same way in every CTA (all read the same state): nothing was written yet.
            if (cta == 0 && tid == 0) atomicOr(a.status, pos < 0 || pos + a.n_tokens > a.max_seq ? LUM_ST_BAD_POS : LUM_ST_BAD_TOKEN);
            if (tid == 0) s_abort = 1;
            gone = true;
        }
        if (tid == 0) { mega_fill(a, 0, 0, tok, &s_phase[0]); s_tok = tok; }
        named_sync(1, W);
    }

    const int per_token = 5 * a.n_layers;             // phases per token before the head
#pragma unroll 1
    for (int t = 0; t < a.n_tokens; t++) {
        const bool head = a.head_every_token || t == a.n_tokens - 1;
        const int n_phase = per_token + (head ? 1 : 0);
#pragma unroll 1
        for (int ph = 0; ph < n_phase; ph++) {
            const int l = ph < per_token ? ph / 5 : a.n_layers - 1;
            const int p = ph < per_token ? ph - l * 5 : 5;
            const unsigned int slot = (unsigned int)(pseq % kJobCtrRing);
            // Re-zero the claim counter that phase pseq + 32 will use: its last user was phase pseq - 32, and no CTA can
            // be that far behind or ahead (a producer leads its consumers by at most one ring of stages, each phase
            // taking at least one).  Every phase does this, whether or not it streams weights itself.
            if (cta == 0 && tid < kMaxKRanges) a.job_ctr[(slot + kJobCtrRing / 2) % kJobCtrRing * kMaxKRanges + tid] = 0u;
            pseq++;
            if (is_producer) {
                if (p != 1 && elect_one() && producing) {
                    mega_fill(a, l, p, 0, &s_stream);
                    producing = gemv_produce(s_stream.ga, s_stream.plan, g, pring, a.job_ctr + slot * kMaxKRanges + s_stream.plan.range, a.status);
                }
                continue;
            }
            const MegaPhase& m = s_phase[buf];
            ArgBest best{-INFINITY, -1};
            if (!gone) {
                if (p == 1) {
                    // RoPE + cache append + attention
                    attn_phase<HD, GM, BF16>(a, a.layers[l], (unsigned char*)g.xq, pos, tid);
                } else {
                    if (p == 0) attn_phase_prefetch<HD, GM, BF16>(a, a.layers[l], pos, tid);
                    if (tid < kConsumers) {
                        if (m.plan.nt > kFillTiles && m.plan.nt <= kJobTiles) mega_consume<true>(m, g, cring, tid, &best);
                        else mega_consume<false>(m, g, cring, tid, &best);
                    }
                }
            }
            if (p == 5 && tid == 0) { a.part_val[cta] = best.v; a.part_idx[cta] = best.i; }
            // the next phase's, by a thread that does not stream; handed over by the barrier
            if (tid == W - 1) {
                const int nx = ph + 1 < n_phase ? ph + 1 : 0, nl = nx < per_token ? nx / 5 : a.n_layers - 1;
                mega_fill(a, nl, nx < per_token ? nx - nl * 5 : 5, nx == 0 && a.forced && t + 1 < a.n_tokens ? a.forced[t + 1] : 0, &s_phase[buf ^ 1]);
            }
            buf ^= 1;
            gone = grid_barrier<W>(a, seq, &s_abort, tid);
            if (p == 5) {
                // every CTA folds the per-CTA maxima itself: all of them need the token for the next embedding row
                if (warp == 0) {
                    const int fi = argmax_final(a.part_val, a.part_idx, ncta, lane).i;
                    if (lane == 0) {
                        s_tok = gone ? 0 : max(0, fi);
                        if (!a.forced) s_phase[buf].xs.token = s_tok;
                    }
                }
                named_sync(1, W);
                if (cta == 0 && tid == 0 && !gone) {
                    DecodeState* st = a.state;
                    const int step = st->step;
                    st->last_tok = s_tok;
                    if (st->log && a.tokens_out && step < st->max_steps) { a.tokens_out[step] = s_tok; st->step = step + 1; }
                }
                // part_val / part_idx are rewritten only after the next token's grid barriers, so no CTA can still
                // be reading them
            }
        }
        pos++;
    }

    if (is_producer) {
        if (elect_one() && (s_abort || !producing)) gemv_producer_drain(g, pring, a.status);
        return;
    }
    if (cta == 0 && tid == 0 && !gone) {
        a.state->pos = pos;
        a.state->tok = s_tok;
    }
}

// ------------------------------------------------------------------------------------------- host side

// the attention phase borrows the activation / reduction area; it is sized for the larger of the two uses
constexpr int kMegaSmem = 224 * 1024;      // dynamic shared memory at most: the phases' arguments are static
static size_t mega_scratch(int hd, int groups) { return attn_smem_bytes(hd, groups <= 4 ? 4 : 8); }
size_t mega_smem_bytes(int k_max, int stages, int hd, int groups) { return gemv_fixed_smem(k_max, mega_scratch(hd, groups)) + (size_t)stages * kFillBytes; }

int mega_pick_stages(int k_max, int hd, int groups) {
    int stages = (int)((kMegaSmem - (long)gemv_fixed_smem(k_max, mega_scratch(hd, groups))) / kFillBytes);
    if (stages > kMaxStages) stages = kMaxStages;
    static const int env_stages = [] { const char* e = getenv("LUM_MEGA_STAGES"); return e ? atoi(e) : 0; }();
    if (env_stages > 0 && env_stages < stages) stages = env_stages;
    return stages;
}

bool mega_supported(const MegaArgs& a) {
    if (a.hd != 64 && a.hd != 128) return false;
    if (!a.kc_h || !a.kc_o || !a.kc_f) return false;
    if (a.k_max > 16384) return false;
    if (a.n_kv <= 0 || a.n_q % a.n_kv || a.n_q / a.n_kv > 8 || a.n_splits < 1) return false;
    return mega_pick_stages(a.k_max, a.hd, a.n_q / a.n_kv) >= 2;
}

cudaError_t launch_mega(const MegaArgs& a_in, int sm_count, cudaStream_t st) {
    MegaArgs a = a_in;
    const void* fn = nullptr;
    const bool g4 = a.n_q / a.n_kv <= 4, bf = a.kv_bf16 != 0;
    if (a.hd == 128) fn = g4 ? (bf ? (const void*)decode_mega<128, 4, true> : (const void*)decode_mega<128, 4, false>)
                             : (bf ? (const void*)decode_mega<128, 8, true> : (const void*)decode_mega<128, 8, false>);
    else if (a.hd == 64) fn = g4 ? (bf ? (const void*)decode_mega<64, 4, true> : (const void*)decode_mega<64, 4, false>)
                                 : (bf ? (const void*)decode_mega<64, 8, true> : (const void*)decode_mega<64, 8, false>);
    else return cudaErrorInvalidValue;
    const int threads = 32 + (a.hd == 128 ? (g4 ? (bf ? mega_workers<128, 4, true>() : mega_workers<128, 4, false>()) : (bf ? mega_workers<128, 8, true>() : mega_workers<128, 8, false>()))
                                          : (g4 ? (bf ? mega_workers<64, 4, true>() : mega_workers<64, 4, false>()) : (bf ? mega_workers<64, 8, true>() : mega_workers<64, 8, false>())));
    if (a.n_kv * a.n_splits > sm_count) return cudaErrorInvalidValue;
    const size_t smem = mega_smem_bytes(a.k_max, a.stages, a.hd, a.n_q / a.n_kv);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kMegaSmem);
    if (e != cudaSuccess) return e;
    if (smem > kMegaSmem) return cudaErrorInvalidValue;
    // every CTA must be resident at once: the grid barrier relies on it
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorLaunchOutOfResources;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    void* params[] = {&a};
    return cudaLaunchKernelExC(&cfg, fn, params);
}

}  // namespace lum
