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
constexpr int kMegaWorkers = 512;        // attention, grid barriers; the first kConsumers of them are the consumers of the weight stream
constexpr int kMegaThreads = kMegaWorkers + 32;
__device__ __forceinline__ bool grid_barrier(const MegaArgs& a, unsigned long long& seq, volatile int* cta_abort, int tid) {
    named_sync(1, kMegaWorkers);                        // all of this CTA's writes of the phase are issued
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
    return named_or(1, kMegaWorkers, *cta_abort != 0);
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
        const AttnArgs t = attn_phase_args(a, L, BF16);
        int r0, r1;
        attn_tc_range(t, (int)blockIdx.x % a.n_splits, pos, &r0, &r1);
        attn_tc_prefetch<HD>(t, (int)blockIdx.x / a.n_splits, r0, r1, tid, kMegaWorkers);
    }
}
template <int HD, int GM, bool BF16>
__device__ __noinline__ void attn_phase(const MegaArgs& a, const MegaLayer& L, unsigned char* scratch_smem, int pos, int tid) {
    const int items = a.n_kv * a.n_splits;
    if ((int)blockIdx.x >= items) return;           // uniform per CTA: the whole CTA skips, barriers inside stay matched
    const AttnArgs t = attn_phase_args(a, L, BF16);
    const int kvh = (int)blockIdx.x / a.n_splits, split = (int)blockIdx.x % a.n_splits;
    if constexpr (BF16 && attn_tc_fits(HD, GM)) {
        // The heads are prepared and the states merged by all 512 workers, the rows (asked for in the phase before) taken by four warps.  Measured, ms a
        // token (32 layers of 32 / 8 heads of 128) behind 512 / 3000 rows: 5.13 / 5.68 with 128 workers and nothing asked for ahead, 4.89 / 5.28 this
        // way, 4.95 / 5.28 with a warp per key
        AttnTile<HD> f;
        AttnPre<HD, kMegaWorkers> pre;
        attn_tc_pre<HD, kMegaWorkers>(t, pre, kvh, split, tid >> 5, tid & 31);
        attn_tc_body<HD, GM / 4, false, kMegaWorkers, false>(t, scratch_smem, f, pre, kvh, split, pos, tid, 1, false);
    } else {
        attn_decode_body<HD, GM, BF16>(t, scratch_smem, kvh, split, pos, tid, 1);
    }
}

// Phase p of layer l (p = 0..4), or the head phase (p = 5): fill in the projection's arguments.
// Returns false for the attention phase (p == 1), which streams no weights.
__device__ __forceinline__ bool phase_gemv(const MegaArgs& a, const MegaLayer& L, int p, GemvArgs* out) {
    const int H = a.hidden, qd = a.n_q * a.hd, kvd = a.n_kv * a.hd;
    GemvArgs g{};
    g.wkind = WK_Q8; g.gain_kind = a.gain_kind; g.eps = a.eps; g.status = a.status;
    switch (p) {
        case 0:   // q, k, v projections (RMSNorm in the prologue)
            g.K = H; g.KC = a.kc_h; g.epi = EPI_STORE; g.nseg = 3;
            g.seg[0] = {L.wq, nullptr, qd, a.kc_h}; g.seg[1] = {L.wk, nullptr, kvd, a.kc_h}; g.seg[2] = {L.wv, nullptr, kvd, a.kc_h};
            g.gain = L.attn_norm; g.y = a.qkv;
            break;
        case 1:
            return false;
        case 2:   // o projection + residual
            g.K = qd; g.KC = a.kc_o; g.epi = EPI_RESID; g.nseg = 1; g.seg[0] = {L.wo, nullptr, H, a.kc_o};
            g.y = a.x; g.resid = a.x;
            break;
        case 3:   // gate, up projections + SwiGLU (RMSNorm in the prologue)
            g.K = H; g.KC = a.kc_h; g.epi = EPI_SWIGLU; g.nseg = 2;
            g.seg[0] = {L.wg, nullptr, a.ffn, a.kc_h}; g.seg[1] = {L.wu, nullptr, a.ffn, a.kc_h};
            g.gain = L.mlp_norm; g.y = a.h;
            break;
        case 4:   // down projection: its K ranges' partial vectors join the residual stream in the next prologue; one range: + residual
            g.K = a.ffn; g.KC = a.kc_f; g.nseg = 1; g.seg[0] = {L.wd, nullptr, H, a.kc_f};
            g.ksplit = gemv_k_ranges(a.ffn, a.kc_f);
            if (g.ksplit > 1) { g.epi = EPI_STORE; g.y = a.part; g.y_range_stride = a.part_ld; }
            else { g.epi = EPI_RESID; g.y = a.x; g.resid = a.x; }
            break;
        default:  // final RMSNorm + vocabulary projection + greedy sample
            g.K = H; g.KC = a.kc_h; g.epi = EPI_ARGMAX; g.nseg = 1; g.seg[0] = {a.lm_head, nullptr, a.vocab, a.kc_h};
            g.gain = a.final_norm; g.y = a.logits;
            break;
    }
    *out = g;
    return true;
}

template <int HD, int GM, bool BF16>
__global__ void __launch_bounds__(kMegaThreads, 1) decode_mega(const MegaArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    __shared__ int s_tok;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cta = (int)blockIdx.x, ncta = (int)gridDim.x;
    GemvSmem g;
    gemv_carve(smem, a.k_max, GemvRings{(a.stages + 1) / 2, a.stages / 2, kFillTiles, kFillTiles}, &s_abort, &g, attn_smem_bytes(HD, GM));
    gemv_cta_begin(g, tid, &s_abort);

    const bool is_worker = warp < kMegaWorkers / 32, is_producer = !is_worker;
    ProducerRing pring{};
    ConsumerRing cring{0, 0u};
    unsigned long long seq = a.gbar_base;             // grid barriers passed so far
    unsigned long long pseq = a.gbar_base;            // running phase number: picks the job-claim counter of each phase
    bool producing = true, gone = false;              // gone: this CTA's workers have given up
    int pos = 0, tok = 0;
    bool second = false;                              // the residual stream is in a.x2
    int pending = 0;                                  // partial vectors that have not joined it yet
    if (is_worker) {
        pos = a.state->pos;
        tok = a.forced ? a.forced[0] : a.state->tok;
        if (pos < 0 || pos + a.n_tokens > a.max_seq || tok < 0 || tok >= a.vocab) {
            // Refuse the whole launch the same way in every CTA (all read the same state): nothing was written yet.
            if (cta == 0 && tid == 0) atomicOr(a.status, pos < 0 || pos + a.n_tokens > a.max_seq ? LUM_ST_BAD_POS : LUM_ST_BAD_TOKEN);
            if (tid == 0) s_abort = 1;
            gone = true;
        }
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
            const MegaLayer& L = a.layers[l];
            GemvArgs ga;
            const bool streams = phase_gemv(a, L, p, &ga);
            GemvPlan plan{};
            if (streams) plan = gemv_plan(ga, cta, ncta, 750);
            unsigned int* ctr = a.job_ctr + (pseq % kJobCtrRing) * kMaxKRanges + plan.range;
            // Re-zero the claim counter that phase pseq + 32 will use: its last user was phase pseq - 32, and no CTA can
            // be that far behind or ahead (a producer leads its consumers by at most one ring of stages, each phase
            // taking at least one).  Every phase does this, whether or not it streams weights itself.
            if (cta == 0 && tid < kMaxKRanges) a.job_ctr[(pseq + kJobCtrRing / 2) % kJobCtrRing * kMaxKRanges + tid] = 0u;
            pseq++;
            if (is_producer) {
                if (streams && elect_one() && producing) {
                    producing = gemv_produce(ga, plan, g, pring, ctr, a.status);
                }
            } else if (!streams) {
                // RoPE + cache append + attention
                if (!gone) attn_phase<HD, GM, BF16>(a, L, (unsigned char*)g.xq, pos, tid);
                gone = grid_barrier(a, seq, &s_abort, tid);
            } else {
                XSource xs{};
                // the residual stream lives in a.x or a.x2, and moves to the other when partial vectors join it
                if (ph == 0) { xs.table = a.embed; xs.table_kind = a.embed_kind; xs.token = tok; xs.x_out = a.x; second = false; pending = 0; }   // the embedding row is x
                else xs.x = p == 2 ? a.attn : p == 4 ? a.h : second ? a.x2 : a.x;
                if (pending && (p == 0 || p == 5)) {
                    xs.parts = a.part; xs.n_parts = pending; xs.part_stride = a.part_ld;
                    if (p == 0) { xs.x_out = second ? a.x : a.x2; second = !second; }
                    pending = 0;
                }
                if (ga.epi == EPI_RESID) ga.y = second ? a.x2 : a.x;
                ga.resid = ga.y;
                if (p == 4 && ga.ksplit > 1) pending = ga.ksplit;
                ArgBest best{-INFINITY, -1};
                if (!gone) {
                    if (p == 0) attn_phase_prefetch<HD, GM, BF16>(a, L, pos, tid);
                    if (tid < kConsumers) {
                        GainRegs gr;
                        gemv_gain_preload(ga, tid, gr);
                        if (plan.nt > kFillTiles && plan.nt <= kJobTiles) gemv_consume<false, true>(ga, xs, cta == 0, plan, g, cring, tid, a.status, &best, gr);
                        else gemv_consume<false, false>(ga, xs, cta == 0, plan, g, cring, tid, a.status, &best, gr);
                    }
                }
                if (p == 5 && tid == 0) { a.part_val[cta] = best.v; a.part_idx[cta] = best.i; }
                gone = grid_barrier(a, seq, &s_abort, tid);
                if (p == 5) {
                    // every CTA folds the per-CTA maxima itself: all of them need the token for the next embedding row
                    if (warp == 0) {
                        const int fi = argmax_final(a.part_val, a.part_idx, ncta, lane).i;
                        if (lane == 0) s_tok = fi;
                    }
                    named_sync(1, kMegaWorkers);
                    const int sampled = gone ? 0 : max(0, s_tok);
                    if (cta == 0 && tid == 0 && !gone) {
                        DecodeState* st = a.state;
                        const int step = st->step;
                        st->last_tok = sampled;
                        if (st->log && a.tokens_out && step < st->max_steps) { a.tokens_out[step] = sampled; st->step = step + 1; }
                    }
                    tok = sampled;
                    // part_val / part_idx are rewritten only after the next token's grid barriers, so no CTA can still
                    // be reading them
                }
            }
        }
        if (is_worker && a.forced && t + 1 < a.n_tokens) tok = a.forced[t + 1];
        pos++;
    }

    if (is_producer) {
        if (elect_one() && (s_abort || !producing)) gemv_producer_drain(g, pring, a.status);
        return;
    }
    if (cta == 0 && tid == 0 && !gone) {
        a.state->pos = pos;
        a.state->tok = tok;
    }
}

// ------------------------------------------------------------------------------------------- host side

// the attention phase borrows the activation / reduction area; it is sized for the larger of the two uses
static size_t mega_scratch(int hd, int groups) { return attn_smem_bytes(hd, groups <= 4 ? 4 : 8); }
size_t mega_smem_bytes(int k_max, int stages, int hd, int groups) { return gemv_fixed_smem(k_max, mega_scratch(hd, groups)) + (size_t)stages * kFillBytes; }

int mega_pick_stages(int k_max, int hd, int groups) {
    int stages = (int)((226 * 1024 - (long)gemv_fixed_smem(k_max, mega_scratch(hd, groups))) / kFillBytes);
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
    if (a.n_kv * a.n_splits > sm_count) return cudaErrorInvalidValue;
    const size_t smem = mega_smem_bytes(a.k_max, a.stages, a.hd, a.n_q / a.n_kv);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(226 * 1024));
    if (e != cudaSuccess) return e;
    if (smem > 226 * 1024) return cudaErrorInvalidValue;
    // every CTA must be resident at once: the grid barrier relies on it
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kMegaThreads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorLaunchOutOfResources;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count);
    cfg.blockDim = dim3(kMegaThreads);
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
