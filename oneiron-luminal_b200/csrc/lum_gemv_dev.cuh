// Device-side building blocks of the streaming Q8_0 matrix-vector product, shared by the one-op
// kernel (lum_gemv.cu) and the whole-token persistent kernel (lum_mega.cu).  A "phase" is one
// y = W x over one CTA's share of the weight stream.  Two kinds of warps cooperate through mbarriers:
//
//   producer warp    gemv_produce()   one lane arms ring stages and issues one bulk copy (up to 4 tiles, 17 KiB) per stage.
//   consumer warps   gemv_consume()   eight warps quantise x into three int8 levels, then take a tile each off the ring: the
//                                     int8 weights go from shared memory through mma.sync.m16n8k32 against the levels as they
//                                     are, exact int32 sums land in registers; the block scales are applied in f32, rows are
//                                     reduced in a fixed order and the epilogue (store / residual add / SwiGLU / greedy
//                                     sample) runs on the finished rows.
//
// What bounds it: HBM while weights stream, and between two phases the time from the previous one's last row to this one's
// first: hand-over, activations, first tiles.  A CTA therefore takes half an SM (288 threads, 96 registers, 103 or 114 KB), so that
// under programmatic dependent launch the next phase's CTA is set up and has its ring full of weights while this one still
// works.  The form before it, tcgen05 kind::i8 over 576 threads and 512 columns of tensor memory, had an SM to itself: the next
// phase could not ask for a byte before it was gone.  The legacy tensor path is the right one here: a tile is 8 rows, one
// vector fills 2 of an instruction's 8 columns, and accumulators in registers need no hand-over to a draining warp.
//
// Arithmetic.  Q8_0 has one scale per 32 weights.  Converting int8 -> f32 costs a quarter-rate instruction per weight, which caps an SM near
// 29 weights a clock, barely above the 23 it must sustain at full HBM speed.  So the activations move to the integer side without
// giving up their f32 precision: each 32-block of x is written as
//     x ~= s * (a1 + a2/254 + a3/254^2),   a1, a2, a3 int8 vectors, s = max|x| / 127
// (three successive int8 roundings of the residual; |error| <= max|x| * 2^-24 per element, the order of f32 rounding).  A block
// then contributes d * s * (q.a1 + (q.a2)/254 + (q.a3)/254^2), d = the block's binary16 scale, with the three dot products exact.
//
// The ring keeps running across phases, so in the persistent kernel the producer streams the next
// operation's weights while the other warps are still finishing (or waiting for the grid-wide
// dependency of) the current one.
//
// Work is handed out in jobs (one row group of 8 rows with all its tiles; for narrow matrices several
// row groups).  Each CTA owns a static run of jobs; the rest sit in a pool that producers claim from with an
// atomic counter, so SMs that happen to get more HBM bandwidth take more of the matrix (equal static
// shares finished up to 30 % apart on B200).  Every ring stage carries the id of the row group it
// holds, and the producer ends a phase with an END marker stage.
#pragma once
#include "lum_kernels.cuh"

namespace lum {


constexpr int kConsumers = 256;          // eight consumer warps: activation prologue, tiles, epilogue
constexpr int kGemvThreads = kConsumers + 32;   // and the producer warp
constexpr int kTileK = 512;              // columns of one tile = 16 blocks of 32
constexpr int kTileRows = 8;             // weight rows of one tile (a "row group")
constexpr int kTileQ = 4096;             // int8 bytes of one tile: block b, row r at b * 256 + (byte / 16) * 128 + r * 16 + byte % 16
constexpr int kTileBytes = kTileQ + 256; // + the 128 binary16 scales, entry b * 8 + r
constexpr int kFillTiles = 4;            // tiles per ring stage, at most: one for each of the four warps that share a ring
constexpr int kJobTiles = 2 * kFillTiles;   // tiles one turn of both rings holds
constexpr int kFillBytes = kFillTiles * kTileBytes;
constexpr int kBarBytes = 640;           // mbarriers, 64 words of reduction scratch at 384
constexpr int kMaxStages = 16;
constexpr int kChunkRG = 16;             // row groups whose sums are held before an epilogue pass (>= 2 x 8: one SwiGLU job of one-tile rows)
constexpr int kRedFloats = kChunkRG * 64;   // [slot][consumer warp][row]
constexpr int kMetaEnd = -1;
constexpr int kXqTileBytes = 1536;       // operand bytes of x per tile: 512 columns x 3 levels

// fields of meta[stage].y: tiles of the fill, its first tile, row groups of the job part, flags
constexpr uint32_t kM2JobEnd = 1u << 16, kM2Up = 1u << 17, kM2First = 1u << 18;
__device__ __forceinline__ uint32_t m2_pack(int ntiles, int c0, int n_rg, bool job_end, int part, bool first) {
    return (uint32_t)ntiles | ((uint32_t)c0 << 4) | ((uint32_t)n_rg << 12) | (job_end ? kM2JobEnd : 0u) | (part ? kM2Up : 0u) | (first ? kM2First : 0u);
}
// The two rings of a CTA: stages [0, n0) belong to consumer warps 0-3, [n0, n0 + n1) to warps 4-7; a stage of ring w holds t_w tiles.
struct GemvRings {
    int n0, n1, t0, t1;
    __host__ __device__ int stages() const { return n0 + n1; }
    __host__ __device__ size_t bytes() const { return (size_t)(n0 * t0 + n1 * t1) * kTileBytes; }
};

// Shared-memory carve-up used by a streaming phase.
struct GemvSmem {
    uint32_t full0, empty0;      // per-stage mbarriers (shared-space addresses): bytes landed / stage released
    float* scratch;              // 64 words
    unsigned char* xq;           // activations as the B operand: per tile [4][24 lanes][16 B], see gemv_load_xfrag
    float* xsc;                  // K / 32 block scales of x
    float* red;                  // kRedFloats
    int* unit_of;                // kChunkRG: global row-group id held in each local slot of the current chunk
    int* pair_of;                // kChunkRG: SwiGLU: slot of the matching up rows (gate slots) or -1 (up slots)
    int* span_of;                // kChunkRG: the consumer warps that hold sums of the slot: first | number << 8
    int2* meta;                  // kMaxStages: x = first row-group id of the fill in each ring stage, or kMetaEnd;
                                 //             y = tiles / first tile / row groups / flags of the fill (m2_pack)
    unsigned char* stage0;       // the rings, 128-byte aligned
    GemvRings rings;
    __device__ int first(int w) const { return w ? rings.n0 : 0; }
    __device__ int count(int w) const { return w ? rings.n1 : rings.n0; }
    __device__ unsigned char* at(int w, int st) const { return stage0 + (size_t)(w ? rings.n0 * rings.t0 + st * rings.t1 : st * rings.t0) * kTileBytes; }
    volatile int* abort;         // CTA-wide: a wait ran out of budget; stop waiting, finish fast
};

// bytes of dynamic shared memory before the ring, for activations of length K.  `scratch_bytes`: the area behind the
// barriers (activation operand, scales, reduction scratch) is at least this large, for a caller that borrows it between
// phases (the persistent kernel's attention).
__host__ __device__ inline size_t gemv_fixed_smem(int K, size_t scratch_bytes = 0) {
    const size_t area = (size_t)K * 3 + (size_t)(K / 32) * 4 + (size_t)kRedFloats * 4;
    return (size_t)kBarBytes + (area > scratch_bytes ? area : scratch_bytes) + (size_t)(3 * kChunkRG + 2 * kMaxStages) * 4 + 256;
}

__device__ __forceinline__ void gemv_carve(unsigned char* smem, int K, const GemvRings& rings, volatile int* abort, GemvSmem* g, size_t scratch_bytes = 0) {
    g->full0 = smem_u32(smem);
    g->empty0 = g->full0 + 8u * kMaxStages;
    g->scratch = (float*)(smem + 384);
    g->xq = smem + kBarBytes;
    g->xsc = (float*)(g->xq + 3 * (size_t)K);
    g->red = g->xsc + (K >> 5);
    g->unit_of = (int*)(g->red + kRedFloats);
    if ((size_t)((unsigned char*)g->unit_of - g->xq) < scratch_bytes) g->unit_of = (int*)(g->xq + ((scratch_bytes + 15) & ~(size_t)15));
    g->pair_of = g->unit_of + kChunkRG;
    g->span_of = g->pair_of + kChunkRG;
    g->meta = (int2*)(g->span_of + kChunkRG);
    g->stage0 = (unsigned char*)(((uintptr_t)(g->meta + kMaxStages) + 127) & ~(uintptr_t)127);
    g->rings = rings;
    g->abort = abort;
}

__device__ __forceinline__ float load_gain(const void* g, int kind, int i) {
    return kind == WK_BF16 ? bf16_bits_to_f32(((const uint16_t*)g)[i]) : ((const float*)g)[i];
}

// Sum over the block's `nthreads` threads (a multiple of 32, <= 512); result in all threads.  `reuse`: the scratch words may be
// written again right after the call (costs a second barrier); false when the caller passes another barrier first anyway.
__device__ __forceinline__ float block_sum(float v, float* scratch, int tid, int nthreads, int bar_id, bool reuse = true) {
    v = warp_sum(v);
    if ((tid & 31) == 0) scratch[tid >> 5] = v;
    named_sync(bar_id, nthreads);
    float t = 0.0f;
    const int nw = nthreads >> 5;
    for (int w = 0; w < nw; w++) t += scratch[w];
    if (reuse) named_sync(bar_id, nthreads);
    return t;
}

// SiLU gate as the graph spells it: g * 1/(exp2(-g * 1.442695) + 1), times u.
__device__ __forceinline__ float swiglu(float g, float u) {
    const float sig = 1.0f / (exp2f((g * -1.0f) * 1.442695f) + 1.0f);
    return (g * sig) * u;
}

// Greedy-sample bookkeeping: (value, index) with "last maximum wins".
struct ArgBest { float v; int i; };
__device__ __forceinline__ void argbest_take(ArgBest& b, float ov, int oi) {
    if (oi >= 0 && (b.i < 0 || ov > b.v || (ov == b.v && oi > b.i))) { b.v = ov; b.i = oi; }
}

// Epilogue over the finished row groups of a chunk: slot s holds row group unit_of[s] (rows unit_of[s] * 8 ..), its 8 row
// sums vals(s*8 ..).  Plain phases: row group ids count over the concatenated segments.  SwiGLU phases: gate slots carry
// the slot of the matching up rows, pair_of(s) (up slots carry -1) and only they produce output.
// For EPI_ARGMAX the rows are stored and thread 0 folds the chunk's best into *best.
// PEER = false compiles the tensor-parallel paths out: the kernel's code size is latency (it has to stay well inside the
// instruction cache: measured, 100 KB -> 135 KB of code cost 12 % tokens/s on one GPU).  `range`: the K range of the sums (GemvArgs::ksplit).
template <bool PEER = false, typename Vals, typename Pair>
__device__ __forceinline__ void gemv_epilogue_units(const GemvArgs& a, Vals vals, const int* unit_of, Pair pair_of, int n_slots,
                                                    int tid, int nthreads, float* scratch, int bar_id, ArgBest* best, size_t range) {
    const int n = n_slots * kTileRows;
    if (a.epi == EPI_SWIGLU) {
        for (int i = tid; i < n; i += nthreads) {
            const int sl = i >> 3, r = i & 7, pr = pair_of(sl);
            if (pr >= 0) a.y[unit_of[sl] * kTileRows + r] = swiglu(vals(i), vals(pr * kTileRows + r));
        }
    } else if (a.epi == EPI_STORE) {
        for (int i = tid; i < n; i += nthreads) {
            const int row = unit_of[i >> 3] * kTileRows + (i & 7);
            a.y[range * a.y_range_stride + row] = (a.bias && range == 0) ? vals(i) + load_gain(a.bias, a.gain_kind, row) : vals(i);
        }
    } else if (a.epi == EPI_RESID) {
        for (int i = tid; i < n; i += nthreads) {
            const int row = unit_of[i >> 3] * kTileRows + (i & 7);
            const float v = a.bias ? vals(i) + load_gain(a.bias, a.gain_kind, row) : vals(i);
            a.y[row] = a.resid[row] + v;
        }
    } else if (PEER && a.epi == EPI_PEER) {
        for (int i = tid; i < n; i += nthreads) {
            const int row = unit_of[i >> 3] * kTileRows + (i & 7);
            const float v = vals(i);
            if (a.peer_ll) {
                const uint32_t word = peer_word(__ldcg(a.seq), a.peer_tag);
#pragma unroll
                for (int r = 0; r < kMaxPeers; r++)
                    if (r < a.n_peers) st_ll((uint2*)a.peer_out[r] + row, __float_as_uint(v), word);
            } else {
#pragma unroll
                for (int r = 0; r < kMaxPeers; r++)
                    if (r < a.n_peers) a.peer_out[r][row] = v;
            }
        }
    } else {  // EPI_ARGMAX
        ArgBest b{-INFINITY, -1};
        for (int i = tid; i < n; i += nthreads) {
            const int row = unit_of[i >> 3] * kTileRows + (i & 7);
            const float v = vals(i);
            a.y[row] = v;
            argbest_take(b, v, row);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, b.v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, b.i, o);
            argbest_take(b, ov, oi);
        }
        int* iscratch = (int*)(scratch + 32);
        if ((tid & 31) == 0) { scratch[tid >> 5] = b.v; iscratch[tid >> 5] = b.i; }
        named_sync(bar_id, nthreads);
        if (tid == 0) {
            for (int w = 1; w < (nthreads >> 5); w++) argbest_take(b, scratch[w], iscratch[w]);
            argbest_take(*best, b.v, b.i);
        }
        named_sync(bar_id, nthreads);
    }
}

// Same for a contiguous run of rows (the plain-load kernel): vals[i] is logical row row0 + i (SwiGLU: gate sums in
// vals[0..n), up sums in vals[n..2n)).  resid0: element tid of the residual.
__device__ __forceinline__ void gemv_epilogue_rows(const GemvArgs& a, const float* vals, int row0, int n, int tid, int nthreads,
                                                   float* scratch, int bar_id, ArgBest* best, float resid0) {
    if (a.epi == EPI_STORE) {
        for (int i = tid; i < n; i += nthreads) a.y[row0 + i] = a.bias ? vals[i] + load_gain(a.bias, a.gain_kind, row0 + i) : vals[i];
    } else if (a.epi == EPI_RESID) {
        for (int i = tid; i < n; i += nthreads) {
            const float v = a.bias ? vals[i] + load_gain(a.bias, a.gain_kind, row0 + i) : vals[i];
            a.y[row0 + i] = (i == tid ? resid0 : a.resid[row0 + i]) + v;
        }
    } else if (a.epi == EPI_SWIGLU) {
        for (int i = tid; i < n; i += nthreads) a.y[row0 + i] = swiglu(vals[i], vals[n + i]);
    } else if (a.epi == EPI_PEER) {
        for (int i = tid; i < n; i += nthreads) {
            const float v = vals[i];
            if (a.peer_ll) {
                const uint32_t word = peer_word(__ldcg(a.seq), a.peer_tag);
#pragma unroll
                for (int r = 0; r < kMaxPeers; r++)
                    if (r < a.n_peers) st_ll((uint2*)a.peer_out[r] + row0 + i, __float_as_uint(v), word);
            } else {
#pragma unroll
                for (int r = 0; r < kMaxPeers; r++)
                    if (r < a.n_peers) a.peer_out[r][row0 + i] = v;
            }
        }
    } else {  // EPI_ARGMAX
        ArgBest b{-INFINITY, -1};
        for (int i = tid; i < n; i += nthreads) {
            const float v = vals[i];
            a.y[row0 + i] = v;
            argbest_take(b, v, row0 + i);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, b.v, o);
            const int oi = __shfl_xor_sync(0xffffffffu, b.i, o);
            argbest_take(b, ov, oi);
        }
        int* iscratch = (int*)(scratch + 32);
        if ((tid & 31) == 0) { scratch[tid >> 5] = b.v; iscratch[tid >> 5] = b.i; }
        named_sync(bar_id, nthreads);
        if (tid == 0) {
            for (int w = 1; w < (nthreads >> 5); w++) argbest_take(b, scratch[w], iscratch[w]);
            argbest_take(*best, b.v, b.i);
        }
        named_sync(bar_id, nthreads);
    }
}

// Reduce the per-CTA partial maxima published in part_val / part_idx (one per CTA) to the sample.
// Called by one warp; every lane returns the winner.  Reads go through L2 (written by other CTAs).
__device__ __forceinline__ ArgBest argmax_final(const float* part_val, const int* part_idx, int n_cta, int lane) {
    ArgBest f{-INFINITY, -1};
    for (int c = lane; c < n_cta; c += 32) argbest_take(f, __ldcg(part_val + c), __ldcg(part_idx + c));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, f.v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, f.i, o);
        argbest_take(f, ov, oi);
    }
    return f;
}

// The greedy sampler's last step, run by the last CTA to arrive (one-op kernels) : fold the per-CTA
// maxima, log the token and advance the decode state.
__device__ __forceinline__ void argmax_finish(const GemvArgs& a, ArgBest mine, int tid, int nthreads, int bar_id) {
    __shared__ int s_last;
    if (tid == 0) {
        a.part_val[blockIdx.x] = mine.v;
        a.part_idx[blockIdx.x] = mine.i;
        __threadfence();
        const unsigned int ticket = atomicAdd(a.counter, 1u);
        s_last = (ticket == gridDim.x - 1) ? 1 : 0;
    }
    named_sync(bar_id, nthreads);
    if (s_last && tid < 32) {
        __threadfence();
        const ArgBest fb = argmax_final(a.part_val, a.part_idx, (int)gridDim.x, tid);
        const int fi = fb.i;
        if (tid == 0) {
            DecodeState* st = a.pair_out ? nullptr : a.state;
            if (a.pair_out) {   // tensor parallel: publish this shard's best; the ranks' pairs are folded after an all-gather ...
                const int pv = __float_as_int(fb.v), pi = fi >= 0 ? fi + a.row_offset : -1;
                a.pair_out[0] = pv;
                a.pair_out[1] = pi;
                if (a.n_peers > 0) {   // ... or are written into every rank's memory right here, followed by "landed" words
#pragma unroll
                    for (int r = 0; r < kMaxPeers; r++)
                        if (r < a.n_peers) { int* dst = (int*)a.peer_out[r]; dst[0] = pv; dst[1] = pi; }
                    __threadfence_system();
                    const uint32_t word = peer_word(__ldcg(a.seq), a.peer_tag);
#pragma unroll
                    for (int r = 0; r < kMaxPeers; r++)
                        if (r < a.n_peers) st_release_sys(a.peer_flag[r], word);
                }
            }
            if (st) {
                const int step = st->step;
                st->last_tok = fi;
                if (st->log && a.tokens_out && step < st->max_steps) { a.tokens_out[step] = fi; st->step = step + 1; }
                if (a.advance) { st->tok = fi; st->pos = st->pos + 1; }
            }
            *a.counter = 0u;
        }
    }
}

// Tensor parallel, producing side: called by all `nthreads` threads of every CTA after the kernel's last row has been
// stored into the ranks' buffers.  The last CTA to arrive tells every rank that this rank's partial vector is complete.
__device__ __forceinline__ void peer_publish(const GemvArgs& a, int tid, int nthreads, int bar_id) {
    named_sync(bar_id, nthreads);           // every thread's stores to the other GPUs are issued ...
    if (tid == 0) {
        __threadfence_system();             // ... and, through the barrier, ordered before this thread's arrival below (one fence per CTA)
        const unsigned int t = atomicAdd(a.peer_ticket, 1u);
        if (t == gridDim.x - 1) {
            *a.peer_ticket = 0u;
            __threadfence_system();
            const uint32_t word = peer_word(__ldcg(a.seq), a.peer_tag);
#pragma unroll
            for (int r = 0; r < kMaxPeers; r++)
                if (r < a.n_peers) st_release_sys(a.peer_flag[r], word);
        }
    }
}
// Consuming side: wait (bounded) until every rank's partial vector for this projection has landed in local memory.
__device__ __forceinline__ void peer_wait_parts(const uint32_t* flags, int n_parts, const uint32_t* seq, uint32_t tag, uint32_t* status,
                                                int tid, int nthreads, int bar_id) {
    if (tid < n_parts) {
        if (!wait_word_sys(flags + (size_t)tid * 32, peer_word(__ldcg(seq), tag))) atomicOr(status, LUM_ST_WAIT_PEER);
    }
    named_sync(bar_id, nthreads);
}

// Where a phase's activations come from.
struct XSource {
    const float* x;        // f32 vector [K] (null when the row of an embedding table is used)
    const float* x_add;    // optional second f32 vector added element-wise
    float* x_out;          // optional: CTA `writer_cta` stores the f32 activations here (must not alias x)
    const void* table;     // embedding table [vocab, K] (f32 or bf16) when x == null
    int table_kind;
    int token;
    // tensor parallel: partial vectors written by the ranks, added in rank order (see GemvArgs)
    const float* parts;
    const uint32_t* part_flags;
    int n_parts, part_stride;
    uint32_t parts_tag;
    const uint32_t* seq;
    int parts_ll;          // parts are {value bits, completion word} pairs, each waited for on its own word
};

// Four consecutive elements of a partial vector stored as {bits, word} pairs: both 16-byte loads are issued at once; an element
// whose word has not arrived yet is then waited for on its own (bounded).
static __device__ __noinline__ float4 ll_load4(const uint2* p, uint32_t word, uint32_t* status, long long budget) {   // out of line: the kernel's code size is latency
    const uint4 a = ld_ll2(p), b = ld_ll2(p + 2);
    float4 v = make_float4(__uint_as_float(a.x), __uint_as_float(a.z), __uint_as_float(b.x), __uint_as_float(b.z));
    bool ok = true;
    if (a.y != word) ok &= ld_ll_wait(p, word, &v.x, budget, status);
    if (a.w != word) ok &= ld_ll_wait(p + 1, word, &v.y, budget, status);
    if (b.y != word) ok &= ld_ll_wait(p + 2, word, &v.z, budget, status);
    if (b.w != word) ok &= ld_ll_wait(p + 3, word, &v.w, budget, status);
    if (!ok) atomicOr(status, LUM_ST_WAIT_PEER);
    return v;
}

// The RMSNorm gains do not depend on the previous operation, so a kernel can fetch them while it still waits for its
// grid dependency: thread tid keeps the gains of the first elements it will quantise (gemv_f4 of turn 0).
constexpr int kXTrips = 4;                  // float4 of x a consumer thread holds at a time: 4096 elements per CTA, a tile per warp
// number of the it-th float4 that a thread takes in turn b
__device__ __forceinline__ int gemv_f4(int tid, int b, int it) { return b * (kXTrips * kConsumers) + (tid >> 5) * (kTileK / 4) + it * 32 + (tid & 31); }
struct GainRegs { uint2 b[kXTrips]; bool loaded; };
__device__ __forceinline__ void gemv_gain_preload(const GemvArgs& a, int tid, GainRegs& gr) {
    gr.loaded = a.gain != nullptr && a.gain_kind == WK_BF16;
    if (!gr.loaded) return;
    const int n4 = a.K >> 2;
#pragma unroll
    for (int it = 0; it < kXTrips; it++) {
        const int f4 = gemv_f4(tid, 0, it);
        gr.b[it] = f4 < n4 ? ((const uint2*)a.gain)[f4] : make_uint2(0u, 0u);
    }
}

// How a phase's matrices are cut into jobs.
//   A matrix [N, K] (K a multiple of 512, N of 8) is a stream of tiles: row group rg = rows [8 rg, 8 rg + 8), tile t of it =
//   columns [512 t, 512 t + 512); tiles of a row group are consecutive, row groups follow each other.  tpr = K / 512.
//   A CTA works on the tiles [t0, t0 + nt) of every row group it takes: all of them, or (ksplit) one of the K ranges, which the
//   CTAs share out in proportion to their tiles.  A job is what one CTA must do as a whole: one row group, where it is whole and has up to 4 tiles as many (gpf) as make up to
//   8 tiles; for SwiGLU the same of the gate matrix followed by the same of the up matrix.  A job part is cut into fills of up to 4
//   tiles, which go to the two rings in turn (a part of one fill sends the second ring an empty one: both see every job).
struct GemvPlan {
    int tpr, t0, nt, gpf, sub;
    int range;        // which K range this CTA works on, cta / n_cta: its number among that range's CTAs
    int cta, n_cta;
    int J;            // jobs in the phase (of this range)
    int js;           // jobs every CTA owns without claiming: c, c + n_cta, ..; the others, from js * n_cta on, are claimed
    int seg_job0[4];  // first job of each segment (plain phases)
    int seg_rg0[4];   // first global row-group id of each segment
    int nrg[3];       // row groups per segment
};
__device__ __forceinline__ GemvPlan gemv_plan(const GemvArgs& a, int cta, int n_cta, int own_permille) {
    GemvPlan p;
    p.tpr = a.K / kTileK;
    p.range = 0; p.cta = cta; p.n_cta = n_cta; p.t0 = 0; p.nt = p.tpr;
    if (a.ksplit > 1) {
        for (int r = 0; r < a.ksplit; r++) {
            const int b0 = gemv_range_tile(p.tpr, a.ksplit, r), b1 = gemv_range_tile(p.tpr, a.ksplit, r + 1);
            const int c0 = b0 * n_cta / p.tpr, c1 = b1 * n_cta / p.tpr;
            if (cta >= c0 && cta < c1) { p.range = r; p.cta = cta - c0; p.n_cta = c1 - c0; p.t0 = b0; p.nt = b1 - b0; }
        }
    }
    p.gpf = p.nt > kFillTiles || p.nt < p.tpr ? 1 : kJobTiles / p.nt;      // (only whole row groups follow each other in memory)
    p.sub = a.epi == EPI_SWIGLU ? 2 : 1;
    int jobs = 0, rgs = 0;
    for (int i = 0; i < 3; i++) {
        const int n = i < a.nseg ? a.seg[i].rows / kTileRows : 0;
        p.nrg[i] = n;
        p.seg_job0[i] = jobs;
        p.seg_rg0[i] = rgs;
        if (a.epi != EPI_SWIGLU || i == 0) { jobs += (n + p.gpf - 1) / p.gpf; rgs += n; }
    }
    p.seg_job0[3] = jobs;
    p.seg_rg0[3] = rgs;
    p.J = jobs;
    // (a launch of one operation says how many it owns: those its rings hold)
    p.js = own_permille >= 0 ? (int)((long long)p.J * own_permille / 1000 / p.n_cta) : min(a.own_jobs, p.J / p.n_cta);
    return p;
}

// Four elements of a block that eight consecutive threads share -> four bytes of each level; returns the block's scale.  A block with an infinite or undefined
// element has no levels: its scale is NaN, and with it every sum that the block is part of.
__device__ __forceinline__ float gemv_levels(const float (&e)[4], uint32_t (&p)[3]) {
    float amax = max_nan(max_nan(fabsf(e[0]), fabsf(e[1])), max_nan(fabsf(e[2]), fabsf(e[3])));
    amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 4));
    amax = max_nan(amax, 0x1p-104f);                     // the third level's factor, 2^23 / amax, has to stay a number (smaller elements keep an error below 2^-127)
    const float s1 = amax * (1.0f / 127.0f);
    const float i1 = 127.0f / amax;
    const float s2 = s1 * (1.0f / 254.0f), i2 = i1 * 254.0f;
    const float i3 = i1 * 64516.0f;
    // Round to nearest by adding 1.5 * 2^23: the sum's low mantissa bits are the integer in two's complement,
    // so its low byte is the int8 value — no float->int conversion or rint (both quarter-rate instructions).
    // |e * i1| <= 127 and every residual is at most half a step of the level before, so no clamping is needed.
    constexpr float kMagic = 12582912.0f;
    p[0] = p[1] = p[2] = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float t1 = fmaf(e[j], i1, kMagic);
        const float r1 = fmaf(-s1, t1 - kMagic, e[j]);
        const float t2 = fmaf(r1, i2, kMagic);
        const float r2 = fmaf(-s2, t2 - kMagic, r1);
        const float t3 = fmaf(r2, i3, kMagic);
        p[0] |= (__float_as_uint(t1) & 0xffu) << (8 * j);
        p[1] |= (__float_as_uint(t2) & 0xffu) << (8 * j);
        p[2] |= (__float_as_uint(t3) & 0xffu) << (8 * j);
    }
    return amax < INFINITY ? s1 : __int_as_float(0x7fffffff);
}
// Where the first level's word j (columns 4 j .. 4 j + 3) of block blk goes in the operand (gemv_load_xfrag); the other levels 16 words further on each.
// Columns of the operand are (half of the tile, level); a block is number blk % 8 of its half.
__device__ __forceinline__ int gemv_level_word(int blk, int j) {
    const int i = blk & 7;
    return ((blk >> 4) * kXqTileBytes + (i >> 1) * 384 + (((blk >> 3) & 1) * 12 + (j & 3)) * 16 + (i & 1) * 8 + (j >> 2) * 4) >> 2;
}

// Prologue: activations (optionally RMS-normalised, times the gains) -> three int8 levels + one f32 scale per 32-block, laid out as
// the B operand of the tensor-core instruction (gemv_load_xfrag).  Runs on the kConsumers threads; 8 consecutive threads own one
// block, a warp a tile of every turn.  A thread issues the loads of up to four float4 (of every term) at once: the vector sits in L2, most of a microsecond away, and up
// to 4096 elements take one trip and stay in registers for both passes.  Longer vectors go around again, twice when they are normalised.
// x_out (if asked for) is the raw sum of the terms.  ONE: see gemv_consume.
template <bool PEER, bool ONE>
__device__ __forceinline__ void gemv_quantize_x(const GemvArgs& a, const XSource& xs, bool is_writer, const GemvPlan& p, const GemvSmem& g, int tid, const GainRegs& gr) {
    const int f40 = p.t0 * (kTileK / 4), n4 = p.nt * (kTileK / 4);          // this CTA's columns
    const int nb = ONE ? 1 : (n4 + kXTrips * kConsumers - 1) / (kXTrips * kConsumers);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    if (PEER && xs.n_parts > 0 && xs.part_flags) peer_wait_parts(xs.part_flags, xs.n_parts, xs.seq, xs.parts_tag, a.status, tid, kConsumers, 2);
    float4 xv[kXTrips];
    float ss = 0.0f, inv = 1.0f;
    // with a norm: one turn over the vector for its squares, then one to quantise (the same registers when it fits them)
#pragma unroll 1
    for (int step = a.gain ? 0 : nb; step < 2 * nb; step++) {
        const bool quant = step >= nb;
        const int b = quant ? step - nb : step;
        if (!(quant && a.gain && nb == 1)) {
            constexpr int kPartBatch = 2;
#pragma unroll
            for (int it = 0; it < kXTrips; it++) {
                const int f4 = gemv_f4(tid, b, it);
                xv[it] = zero;
                if (f4 < n4) {
                    if (xs.x) {
                        xv[it] = ((const float4*)xs.x)[f40 + f4];
                    } else if (xs.table_kind == WK_BF16) {
                        const uint2 r = ((const uint2*)((const uint16_t*)xs.table + (size_t)xs.token * a.K))[f4];
                        xv[it] = make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
                    } else {
                        xv[it] = ((const float4*)((const float*)xs.table + (size_t)xs.token * a.K))[f4];
                    }
                }
            }
            // the sums are formed in this order: x, the parts (ranks or K ranges) in theirs, the addend
            if (PEER && xs.parts_ll) {
                // every element carries its own completion word: the loads of two ranks' vectors go out together, stragglers are waited for one by one
                const uint32_t word = peer_word(__ldcg(xs.seq), xs.parts_tag);
#ifndef LUM_LL_BATCH
#define LUM_LL_BATCH 2
#endif
                // ranks whose vectors are requested together.  Measured on 2 GPUs, same call: 1 -> 558.7, 2 -> 553.6, 4 -> 495.2 tokens/s
                // (four ranks' loads in flight cost registers: the kernel spills); 2 is what the 4- and 8-GPU numbers were measured with
                constexpr int kLLBatch = LUM_LL_BATCH;
#pragma unroll 1
                for (int r0 = 0; r0 < xs.n_parts; r0 += kLLBatch) {
                    uint4 raw[kLLBatch][kXTrips][2];
#pragma unroll
                    for (int j = 0; j < kLLBatch; j++) {
                        const uint2* pr = (const uint2*)xs.parts + (size_t)min(r0 + j, xs.n_parts - 1) * xs.part_stride;
#pragma unroll
                        for (int it = 0; it < kXTrips; it++) {
                            const int f4 = min(gemv_f4(tid, b, it), n4 - 1);
                            raw[j][it][0] = ld_ll2(pr + 4 * f4);
                            raw[j][it][1] = ld_ll2(pr + 4 * f4 + 2);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < kLLBatch; j++) {
                        if (r0 + j < xs.n_parts) {
                            const uint2* pr = (const uint2*)xs.parts + (size_t)(r0 + j) * xs.part_stride;
#pragma unroll
                            for (int it = 0; it < kXTrips; it++) {
                                const int f4 = gemv_f4(tid, b, it);
                                if (f4 < n4) {
                                    const uint4 a4 = raw[j][it][0], b4 = raw[j][it][1];
                                    float4 v = make_float4(__uint_as_float(a4.x), __uint_as_float(a4.z), __uint_as_float(b4.x), __uint_as_float(b4.z));
                                    if (a4.y != word || a4.w != word || b4.y != word || b4.w != word) v = ll_load4(pr + 4 * f4, word, a.status, a.wait_cycles);
                                    xv[it].x += v.x; xv[it].y += v.y; xv[it].z += v.z; xv[it].w += v.w;
                                }
                            }
                        }
                    }
                }
            } else {
#pragma unroll 1
                for (int r0 = 0; r0 < xs.n_parts; r0 += kPartBatch) {
                    float4 u[kPartBatch][kXTrips];
#pragma unroll
                    for (int j = 0; j < kPartBatch; j++) {
                        const float4* pr = (const float4*)(xs.parts + (size_t)(r0 + j) * xs.part_stride);
#pragma unroll
                        for (int it = 0; it < kXTrips; it++) {
                            const int f4 = gemv_f4(tid, b, it);
                            u[j][it] = (r0 + j < xs.n_parts && f4 < n4) ? __ldcg(pr + f4) : zero;     // written by other GPUs / CTAs: read around L1
                        }
                    }
#pragma unroll
                    for (int j = 0; j < kPartBatch; j++) {
                        if (r0 + j < xs.n_parts) {
#pragma unroll
                            for (int it = 0; it < kXTrips; it++) { xv[it].x += u[j][it].x; xv[it].y += u[j][it].y; xv[it].z += u[j][it].z; xv[it].w += u[j][it].w; }
                        }
                    }
                }
            }
            if (xs.x_add) {
#pragma unroll
                for (int it = 0; it < kXTrips; it++) {
                    const int f4 = gemv_f4(tid, b, it);
                    if (f4 < n4) { const float4 u = ((const float4*)xs.x_add)[f4]; xv[it].x += u.x; xv[it].y += u.y; xv[it].z += u.z; xv[it].w += u.w; }
                }
            }
            if (xs.x_out && is_writer && (!quant || !a.gain)) {
#pragma unroll
                for (int it = 0; it < kXTrips; it++) {
                    const int f4 = gemv_f4(tid, b, it);
                    if (f4 < n4) ((float4*)xs.x_out)[f4] = xv[it];
                }
            }
        }
        if (!quant) {
#pragma unroll
            for (int it = 0; it < kXTrips; it++) {      // absent elements hold zeros
                const float4 t = xv[it];
                ss = fmaf(t.x, t.x, ss); ss = fmaf(t.y, t.y, ss); ss = fmaf(t.z, t.z, ss); ss = fmaf(t.w, t.w, ss);
            }
            if (b == nb - 1) {
                ss = block_sum(ss, g.scratch, tid, kConsumers, 2, false);   // (the next to use the scratch is the sampler's epilogue, behind gemv_consume's named_or)
                const float mean = ss * (1.0f / (float)(a.k_norm > 0 ? a.k_norm : a.K));
                inv = 1.0f / sqrtf(mean + a.eps);
            }
            continue;
        }
#pragma unroll
        for (int it = 0; it < kXTrips; it++) {
            const int f4 = gemv_f4(tid, b, it);
            if (f4 >= n4) continue;                      // n4 is a multiple of 128: a warp is in or out as a whole
            float e[4] = {xv[it].x, xv[it].y, xv[it].z, xv[it].w};
            if (a.gain) {
                if (gr.loaded) {
                    const uint2 gb = b == 0 ? gr.b[it] : ((const uint2*)a.gain)[f40 + f4];
                    e[0] = (inv * e[0]) * __uint_as_float(gb.x << 16); e[1] = (inv * e[1]) * __uint_as_float(gb.x & 0xffff0000u);
                    e[2] = (inv * e[2]) * __uint_as_float(gb.y << 16); e[3] = (inv * e[3]) * __uint_as_float(gb.y & 0xffff0000u);
                } else {
                    const float4 gf = ((const float4*)a.gain)[f40 + f4];
                    e[0] = (inv * e[0]) * gf.x; e[1] = (inv * e[1]) * gf.y; e[2] = (inv * e[2]) * gf.z; e[3] = (inv * e[3]) * gf.w;
                }
            }
            uint32_t lv[3];
            const float s1 = gemv_levels(e, lv);
            const int blk = f4 >> 3;
            uint32_t* dst = (uint32_t*)g.xq + gemv_level_word(blk, f4 & 7);
            dst[0] = lv[0]; dst[16] = lv[1]; dst[32] = lv[2];
            if ((tid & 7) == 0) g.xsc[blk] = s1;
        }
    }
    if (ONE) __syncwarp();                               // a warp multiplies by what it wrote itself
    else named_sync(2, kConsumers);
}

// Ring positions, carried across phases.
struct ProducerRing { int stage[2]; uint32_t par[2]; long long armed[2]; };
struct ConsumerRing { int stage; uint32_t par; };

// Producer side of one phase: ONE lane of the producer warp walks this CTA's own jobs, then claims others
// with atomicAdd on *job_ctr (two claims are in flight while a job is being issued: one takes about as long as a job), and
// closes the phase with an END marker in each ring.  With job_ctr == null the jobs are split evenly by CTA index instead.
// Returns false if a wait ran out of budget (or the CTA is already aborting).
__device__ __forceinline__ bool gemv_produce(const GemvArgs& a, const GemvPlan& p, const GemvSmem& g, ProducerRing& r,
                                             unsigned int* job_ctr, uint32_t* status) {
    // tiles > 0: a copy of them; 0: nothing to copy (an empty fill, the END marker)
    auto emit = [&](int w, const unsigned char* src, int tiles, int unit, uint32_t m2) -> bool {
        const int slot = g.first(w) + r.stage[w];
        if (*g.abort) return false;
        if (!mbar_wait_abortable(g.empty0 + 8u * slot, r.par[w] ^ 1u, g.abort)) {        // until the ring position is free
            if (!*g.abort) { atomicOr(status, LUM_ST_WAIT_EMPTY); *g.abort = 1; }
            return false;
        }
        const uint32_t fb = g.full0 + 8u * slot;
        g.meta[slot] = make_int2(unit, (int)m2);
        if (tiles > 0) {
            mbar_arrive_expect_tx(fb, (uint32_t)tiles * kTileBytes);
            bulk_g2s(smem_u32(g.at(w, r.stage[w])), src, (uint32_t)tiles * kTileBytes, fb);
        } else {
            mbar_arrive(fb);
        }
        r.armed[w]++;
        if (++r.stage[w] == g.count(w)) { r.stage[w] = 0; r.par[w] ^= 1u; }
        return true;
    };
    auto issue_job = [&](int j) -> bool {
        int sg = 0;
        if (a.epi != EPI_SWIGLU) while (sg < a.nseg - 1 && j >= p.seg_job0[sg + 1]) sg++;
        const int rg = (j - p.seg_job0[sg]) * p.gpf;                      // first row group of the job, inside its segment
        const int n_rg = min(p.gpf, p.nrg[sg] - rg), T = n_rg * p.nt;
#pragma unroll 1
        for (int part = 0; part < p.sub; part++) {
            const unsigned char* base = (const unsigned char*)a.seg[sg + part].w + ((size_t)rg * p.tpr + p.t0) * kTileBytes;
            const bool last_part = part == p.sub - 1;
#pragma unroll 1
            for (int c = 0; c < T; c += kJobTiles) {
                const int c1 = c + kFillTiles;
                if (!emit(0, base + (size_t)c * kTileBytes, min(kFillTiles, T - c), p.seg_rg0[sg] + rg, m2_pack(min(kFillTiles, T - c), c, n_rg, last_part && c + kJobTiles >= T, part, c == 0))) return false;
                if (c > 0 && c1 >= T) break;
                const int n1 = max(0, min(kFillTiles, T - c1));
                if (!emit(1, base + (size_t)c1 * kTileBytes, n1, p.seg_rg0[sg] + rg, m2_pack(n1, c1, n_rg, last_part && c1 + kJobTiles >= T, part, c == 0))) return false;
            }
        }
        return true;
    };

    if (job_ctr) {
        // A CTA that starts early (its SM was free while the previous kernel still ran elsewhere) could fill its whole ring
        // with claims before the others have started, and then has to drain it alone after the grid dependency resolves:
        // measured on the o projection, the last CTA finished 3-5 us after the median.  So a CTA takes at most its even
        // share plus one; a claim is only made when it will be used.
        const unsigned int base = (unsigned int)(p.js * p.n_cta), none = (unsigned int)p.J;
        const int cap = (p.J + p.n_cta - 1) / p.n_cta + (a.max_units > 0 ? a.max_units - 1 : 1) - p.js;   // a.max_units: tuning override of the slack
        unsigned int c0 = none, c1 = none;
        if (base < none && cap > 0) c0 = base + atomicAdd(job_ctr, 1u);     // these travel while the own jobs are issued
        if (base < none && cap > 1) c1 = base + atomicAdd(job_ctr, 1u);
        for (int i = 0; i < p.js; i++)
            if (!issue_job(p.cta + i * p.n_cta)) return false;
#pragma unroll 1
        for (int taken = 2; c0 < none; taken++) {
            const unsigned int nxt = taken < cap && c1 < none ? base + atomicAdd(job_ctr, 1u) : none;
            if (!issue_job((int)c0)) return false;
            c0 = c1; c1 = nxt;
        }
    } else {
#pragma unroll 1
        for (int j = p.cta; j < p.J; j += p.n_cta)
            if (!issue_job(j)) return false;
    }
    return emit(0, nullptr, 0, kMetaEnd, 0u) && emit(1, nullptr, 0, kMetaEnd, 0u);
}

// After an aborted run: never leave the CTA while a copy into its shared memory may still be in flight.
// Wait (bounded) for every fill armed in the last ring revolution to land.
__device__ __forceinline__ void gemv_producer_drain(const GemvSmem& g, const ProducerRing& r, uint32_t* status) {
    for (int w = 0; w < 2; w++) {
        const int S = g.count(w);
        int st = r.stage[w];
        uint32_t par = r.par[w];
        const long long back = r.armed[w] < S ? r.armed[w] : S;
        for (long long i = 0; i < back; i++) {
            if (st == 0) { st = S; par ^= 1u; }
            st--;
            if (!mbar_wait(g.full0 + 8u * (g.first(w) + st), par)) { atomicOr(status, LUM_ST_WAIT_DRAIN); return; }
        }
    }
}

// The operands of one tile.  A warp multiplies by m16n8k32 with the weights as A: rows 0-7 are the tile's 8 rows in block i, rows 8-15 the same
// 8 rows in block 8 + i; ldmatrix brings a row's weights 4 t .. 4 t + 3 of each half of a block to lane (row, t) as the instruction wants them.
// Column n = (half of the tile, level) of B holds that level of that half's block i (a half's fourth column repeats the third); the products of one half's rows with the
// other half's columns, and of the fourth columns, are not read.  Lane (g, t) ends up with row g of block (t / 2) * 8 + i: levels 1 and 2 (t even) or level 3 (t odd).
__device__ __forceinline__ void gemv_load_xfrag(const GemvSmem& g, int tile, int lane, uint32_t (&b)[4][4], float4& sx) {
    const int n = lane >> 2;
    const unsigned char* p = g.xq + (size_t)tile * kXqTileBytes + (((n >> 2) * 3 + min(n & 3, 2)) * 4 + (lane & 3)) * 16;
#pragma unroll
    for (int s = 0; s < 4; s++) {
        const uint4 v = *(const uint4*)(p + s * 384);
        b[s][0] = v.x; b[s][1] = v.y; b[s][2] = v.z; b[s][3] = v.w;
    }
    sx = *(const float4*)(g.xsc + tile * 16 + ((lane & 2) << 2) + ((lane & 1) << 2));
}
__device__ __forceinline__ void gemv_ldmatrix(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void gemv_mma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}

// Consumer side of one phase, called by the kConsumers threads: quantise x, then take fills off this warp's ring until the END marker, a tile
// of each fill.  A lane's share of a tile is one row in half of its blocks (even lanes: levels 1 and 2, odd ones: level 3), four lanes are folded with two
// shuffles, the warps' sums wait in shared memory and are added in a fixed order at the end of a
// chunk, followed by the epilogue.  For EPI_ARGMAX, *best (thread 0) receives this CTA's best row.
// ONE: five to eight tiles per row group (K of 2049 to 4096, or a K range): a job part is one fill of each ring, a warp has the same tile of every
// row group, whose columns it has quantised itself.  Most of what the loop does besides the tile falls away (270 -> 150 instructions a tile), and so does a barrier.
template <bool PEER, bool ONE>
__device__ __forceinline__ void gemv_consume(const GemvArgs& a, const XSource& xs, bool is_writer, const GemvPlan& p, const GemvSmem& g,
                                             ConsumerRing& cr, int tid, uint32_t* status, ArgBest* best, const GainRegs& gr) {
    gemv_quantize_x<PEER, ONE>(a, xs, is_writer, p, g, tid, gr);
    const int lane = tid & 31, warp = tid >> 5, wg = warp >> 2, wj = warp & 3;
    const int S = g.count(wg), first = g.first(wg);
    const uint32_t ring = smem_u32(g.at(wg, 0)) + (uint32_t)wj * kTileBytes + lane * 16, stride = (uint32_t)(wg ? g.rings.t1 : g.rings.t0) * kTileBytes;
    const uint32_t sc0 = kTileQ - lane * 16 + ((lane & 2) << 6) + ((lane & 1) << 6) + ((lane >> 2) << 1);           // this lane's first block scale in a tile
    float* const red = g.red + warp * 8 + (lane >> 2);
    uint32_t b[4][4];
    float4 sx;
    const bool odd = lane & 1, low = lane & 2;
    const int m1 = odd ? 1 : 254, m2c = odd ? 0 : 1;
    int cur = -1;                                        // the tile position whose activations b holds
    if (ONE && warp < p.nt) gemv_load_xfrag(g, warp, lane, b, sx);
    auto fail = [&](uint32_t code) { if (!*g.abort) { atomicOr(status, code); *g.abort = 1; } };
    int slot = 0, slot_base = 0;
    bool ended = false, gave_up = false;
#pragma unroll 1
    while (!ended) {
        slot = 0;
#pragma unroll 1
        for (;;) {
            const int st = first + cr.stage;
            if (!mbar_wait_warp(g.full0 + 8u * st, cr.par, g.abort)) { fail(LUM_ST_WAIT_FULL); gave_up = true; break; }
            const int2 mm = g.meta[st];
            const uint32_t m2 = (uint32_t)mm.y;
            const bool mine = ONE ? warp < p.nt && mm.x != kMetaEnd : wj < (int)(m2 & 15u);
            const uint32_t wp = ring + (uint32_t)cr.stage * stride;
            uint32_t wx[4][4], wy[4][4];
            uint16_t dw[4];
            if (mine) {
#pragma unroll
                for (int s = 0; s < 4; s++) {            // in the order they are multiplied
                    gemv_ldmatrix(wp + ((s & 1) * 2 + (s >> 1)) * 512, wx[(s & 1) * 2 + (s >> 1)]);
                    gemv_ldmatrix(wp + 2048 + ((s & 1) * 2 + (s >> 1)) * 512, wy[(s & 1) * 2 + (s >> 1)]);
                }
#pragma unroll
                for (int i = 0; i < 4; i++) asm volatile("ld.shared.u16 %0, [%1];" : "=h"(dw[i]) : "r"(wp + sc0 + i * 16) : "memory");
            }
            // The stage goes back when every load from it has returned.  (Behind their issue alone, about one pass in six of 16 steps of six Llama-3-8B layers came out
            // with scales of the next tile in some rows; waiting costs 0.6 % of a step, handing back behind the tile's arithmetic 2 %.)
            uint32_t seen = 0;
            if (mine) {
#pragma unroll
                for (int s = 0; s < 4; s++) seen ^= wx[s][0] ^ wy[s][0] ^ dw[s];
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(behind(g.empty0 + 8u * st, seen));
            if (++cr.stage == S) { cr.stage = 0; cr.par ^= 1u; }
            if (mm.x == kMetaEnd) { ended = true; break; }
            if (ONE) {
                if (warp == 7 && lane == 0) g.unit_of[slot] = mm.x;
                slot_base = slot++;
            } else if (m2 & kM2First) {                  // first fill of a job part: its row groups take new slots
                const int n_rg = (int)((m2 >> 12) & 15u);
                slot_base = slot;
                slot += n_rg;
                if (warp == 7 && lane < n_rg) {          // (a warp with less to do wherever a row group has fewer than eight tiles)
                    g.unit_of[slot_base + lane] = mm.x + lane;
                    g.pair_of[slot_base + lane] = (m2 & kM2Up) ? -1 : slot_base + n_rg + lane;
                    g.span_of[slot_base + lane] = (p.gpf > 1 ? lane * p.nt : 0) | min(p.nt, kJobTiles) << 8;
                }
            }
            if (mine) {
                int sl = slot_base;
                if (!ONE) {
                    int t = (int)((m2 >> 4) & 255u) + wj;
                    if (p.gpf > 1) { sl += t / p.nt; t %= p.nt; }
                    if (t != cur) { gemv_load_xfrag(g, t, lane, b, sx); cur = t; }
                }
                float v = 0.0f;
                // Lanes t and t ^ 1 hold levels 1, 2 and level 3 of the same row and blocks: of blocks i and i + 4 the even lane completes the first, the odd
                // one the second.  Four instructions are issued before the first result is used.
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    int c[4][4];
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        const int s = h + (k & 1) * 2, o = k & 2;                     // blocks 2 h, 2 h + 4, 2 h + 1, 2 h + 5
                        gemv_mma(c[k], wx[s][o], wy[s][o], wx[s][o + 1], wy[s][o + 1], b[s][o], b[s][o + 1]);
                    }
#pragma unroll
                    for (int k = 0; k < 4; k += 2) {
                        // i1 * 254 + i2 fits an int32 (|i1| <= 32 * 128 * 127): one conversion for both
                        const int qa = (low ? c[k][2] : c[k][0]) * m1 + (low ? c[k][3] : c[k][1]) * m2c;
                        const int qb = (low ? c[k + 1][2] : c[k + 1][0]) * m1 + (low ? c[k + 1][3] : c[k + 1][1]) * m2c;
                        const int got = __shfl_xor_sync(0xffffffffu, odd ? qa : qb, 1);
                        const int i12 = odd ? got : qa, i3 = odd ? qb : got;
                        const int i = 2 * h + (k >> 1);
                        const float x = i == 0 ? sx.x : i == 1 ? sx.y : i == 2 ? sx.z : sx.w;
                        const float tt = fmaf((float)i3, 1.0f / 64516.0f, (float)i12 * (1.0f / 254.0f));
                        v = fmaf(tt, x * __half2float(__ushort_as_half(dw[i])), v);
                    }
                }
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if ((lane & 3) == 0) red[sl * 64] = ONE || (m2 & kM2First) ? v : red[sl * 64] + v;
            }
            if (ONE ? slot == kChunkRG : (m2 & kM2JobEnd) && slot + p.sub * p.gpf > kChunkRG) break;
        }
        // A warp that gave up takes the others along: the two rings' warps then stand at different jobs, and nothing of this chunk is stored.  Otherwise every warp is
        // here with the same jobs behind it, and every barrier below is attended by all.
        if (named_or(2, kConsumers, gave_up)) return;
        // the warps' sums of a row, added in a fixed order, straight into the epilogue
        auto sum = [&](int i) {
            const int span = ONE ? p.nt << 8 : g.span_of[i >> 3];
            const float* rp = g.red + (size_t)(i >> 3) * 64 + (span & 255) * 8 + (i & 7);
            float t = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; w++) if (w < (span >> 8)) t += rp[w * 8];
            return t;
        };
        auto pair = [&](int sl) { return ONE ? (sl & 1 ? -1 : sl + 1) : g.pair_of[sl]; };
        if (slot > 0) gemv_epilogue_units<PEER>(a, sum, g.unit_of, pair, slot, tid, kConsumers, g.scratch, 2, best, (size_t)p.range);
        if (!ended) named_sync(2, kConsumers);
    }
}

// Kernel start (all threads of the CTA): barriers.
__device__ __forceinline__ void gemv_cta_begin(const GemvSmem& g, int tid, volatile int* abort_word) {
    if (tid == 0) {
        *abort_word = 0;
        for (int s = 0; s < g.rings.stages(); s++) {
            mbar_init(g.full0 + 8u * s, 1);
            mbar_init(g.empty0 + 8u * s, kConsumers / 64);
        }
        mbar_fence_init();
    }
    __syncthreads();
}

}  // namespace lum
