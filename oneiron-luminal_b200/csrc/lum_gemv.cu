// Matrix-vector kernels for single-token decode: y = W x with W row-major [N, K], K contiguous —
// the job `TileMatmulFullSplit`'s M == 1 path does in the reference
// (crates/luminal_cuda/src/block/ops.rs:1588-1651), and for block-quantised weights what
// `TileMatmulNvFp4` / `TileMatmulMxfp4` do (ops.rs:2148-2347, 2546-2733), here for Q8_0.
//
// Decode is bound by HBM bandwidth: every weight byte is read exactly once per token and nothing
// else is large.  Two kernels:
//
//  * q8_gemv_stream — the hot path (lum_gemv_dev.cuh).  A producer warp walks the CTA's share of the weight matrix in
//    tiles of 8 rows x 512 columns (4096 int8 plus their 128 binary16 scales) and fetches up to 4 of them per ring stage with
//    one bulk asynchronous copy (cp.async.bulk, completion counted on an mbarrier); eight consumer warps take a tile each.
//    A CTA is half an SM, so that under programmatic dependent launch the next projection's CTAs are resident, set up and
//    have filled their rings (the weight stream does not depend on the activations) while this one still works.
//  * gemv_direct — any K, f32 / bf16 / Q8_0 weights, plain vector loads, one warp per row (bf16: per four rows).
//    Used for the small all-f32 model and for shapes the streaming kernel does not take.
//
// Both fuse the RMSNorm that precedes the projection (`RowRMSNorm`, ops.rs:519-566; math per
// crates/luminal_nn/src/norm.rs:31-43) into their prologue and the residual add (`RowAdd`,
// ops.rs:135-146), SwiGLU (`RowSwishMul`, ops.rs:303-325) or the greedy sampler
// (examples/llama/src/main.rs:137-148) into their epilogue.
//
// The streaming kernel works on integer levels of the activations (lum_gemv_dev.cuh); the direct kernel keeps the plain
// f32 form sum_i float(q_i) * x_i.  (The CPU restatement multiplies each weight by its scale first and sums
// sequentially; all three differ by f32 rounding only.)
#include <algorithm>
#include <cstdlib>

#include "lum_gemv_dev.cuh"

namespace lum {

// Prologue of the plain-load kernel: bring x into shared memory as f32 (optionally RMS-normalised and
// scaled by the gains).  gain0: element tid's, asked for before the grid dependency was waited for.
__device__ __forceinline__ void gemv_load_x(const GemvArgs& a, float* xs, int tid, int nthreads, float* scratch, int bar_id, float gain0) {
    const int K = a.K;
    if (a.n_parts > 0 && a.part_flags) peer_wait_parts(a.part_flags, a.n_parts, a.seq, a.parts_tag, a.status, tid, nthreads, bar_id);
    // the raw activations first (x, plus a reduced partial or the ranks' partials in rank order), then the norm over them
    float ss = 0.0f;
    for (int k = tid; k < K; k += nthreads) {
        float v = a.x[k];
        if (a.x_add) v += a.x_add[k];
        for (int r = 0; r < a.n_parts; r++) {
            if (a.parts_ll) {
                float u;
                if (!ld_ll_wait((const uint2*)a.parts + (size_t)r * a.part_stride + k, peer_word(__ldcg(a.seq), a.parts_tag), &u, a.wait_cycles, a.status)) atomicOr(a.status, LUM_ST_WAIT_PEER);
                v += u;
            } else {
                v += __ldcg(a.parts + (size_t)r * a.part_stride + k);
            }
        }
        if ((a.x_add || a.n_parts > 0) && a.x_out && blockIdx.x == 0) a.x_out[k] = v;
        xs[k] = v;
        ss = fmaf(v, v, ss);
    }
    if (a.gain) {
        ss = block_sum(ss, scratch, tid, nthreads, bar_id, false);      // (a barrier follows before the scratch is written again)
        const float mean = ss * (1.0f / (float)(a.k_norm > 0 ? a.k_norm : K));
        const float inv = 1.0f / sqrtf(mean + a.eps);
        for (int k = tid; k < K; k += nthreads) xs[k] = (inv * xs[k]) * (k == tid ? gain0 : load_gain(a.gain, a.gain_kind, k));
    }
    named_sync(bar_id, nthreads);
}

__device__ __forceinline__ float dot4_s8(uint32_t w, float4 x, float acc) {
    acc = fmaf((float)(int)(int8_t)(w & 0xffu), x.x, acc);
    acc = fmaf((float)(int)(int8_t)((w >> 8) & 0xffu), x.y, acc);
    acc = fmaf((float)(int)(int8_t)((w >> 16) & 0xffu), x.z, acc);
    acc = fmaf((float)((int)w >> 24), x.w, acc);
    return acc;
}

// ------------------------------------------------------------------------------ streaming kernel (one op)


template <bool PEER, bool ONE>
__global__ void __launch_bounds__(kGemvThreads, PEER ? 1 : 2) q8_gemv_stream(const GemvArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    const int tid = threadIdx.x;
    GemvSmem g;
    const GemvPlan plan = gemv_plan(a, (int)blockIdx.x, (int)gridDim.x, -1);
    gemv_carve(smem, a.k_smem, GemvRings{a.ring_n[0], a.ring_n[1], a.ring_t[0], a.ring_t[1]}, &s_abort, &g);
    gemv_cta_begin(g, tid, &s_abort);
    if (a.use_pdl) pdl_launch_dependents();

    if (tid >= kConsumers) {
        // producer: the weight stream does not depend on the previous kernel, so it starts at once
        if (elect_one()) {
            ProducerRing pr{};
            if (!gemv_produce(a, plan, g, pr, a.job_ctr ? a.job_ctr + plan.range : nullptr, a.status)) gemv_producer_drain(g, pr, a.status);
        }
        return;
    }
    GainRegs gr;
    gemv_gain_preload(a, tid, gr);             // independent of the previous kernel: fetched while waiting for it
    if (a.use_pdl) pdl_grid_wait();
    XSource xs{};
    xs.x = a.x; xs.x_add = a.x_add; xs.x_out = a.x_out;
    xs.parts = a.parts; xs.part_flags = a.part_flags; xs.n_parts = a.n_parts; xs.part_stride = a.part_stride; xs.parts_tag = a.parts_tag; xs.seq = a.seq; xs.parts_ll = a.parts_ll;
    ArgBest best{-INFINITY, -1};
    ConsumerRing cr{0, 0u};
    gemv_consume<PEER, ONE>(a, xs, blockIdx.x == 0, plan, g, cr, tid, a.status, &best, gr);
    if (PEER && a.epi == EPI_PEER && !a.peer_ll) peer_publish(a, tid, kConsumers, 2);
    if (a.epi == EPI_ARGMAX) argmax_finish(a, best, tid, kConsumers, 2);
}

// ------------------------------------------------------------------------------ direct kernel

// N bf16 rows of 8 n8 elements (per lane; the caller folds the lanes).  A vocabulary-sized bf16 matrix (a head tied to the embedding) is hundreds
// of megabytes per token and must stream: 2 N 16-byte loads in flight per lane, and the activations' reads from shared memory — twice the
// bytes of a row's weights, which for one row at a time is what binds the SM — shared by the N rows.
template <int N>
__device__ __forceinline__ void bf16_rows_dot(const uint4* const (&w)[N], int n8, const float* xs, int lane, float (&acc)[N]) {
    auto dot8 = [](uint4 a, float4 x0, float4 x1, float s) {
        s = fmaf(__uint_as_float(a.x << 16), x0.x, s); s = fmaf(__uint_as_float(a.x & 0xffff0000u), x0.y, s);
        s = fmaf(__uint_as_float(a.y << 16), x0.z, s); s = fmaf(__uint_as_float(a.y & 0xffff0000u), x0.w, s);
        s = fmaf(__uint_as_float(a.z << 16), x1.x, s); s = fmaf(__uint_as_float(a.z & 0xffff0000u), x1.y, s);
        s = fmaf(__uint_as_float(a.w << 16), x1.z, s); s = fmaf(__uint_as_float(a.w & 0xffff0000u), x1.w, s);
        return s;
    };
    int i = lane;
    for (; i + 32 < n8; i += 64) {
        uint4 a[N], b[N];
#pragma unroll
        for (int r = 0; r < N; r++) { a[r] = __ldcs(w[r] + i); b[r] = __ldcs(w[r] + i + 32); }
        float4 x0 = *(const float4*)(xs + (size_t)i * 8), x1 = *(const float4*)(xs + (size_t)i * 8 + 4);
#pragma unroll
        for (int r = 0; r < N; r++) acc[r] = dot8(a[r], x0, x1, acc[r]);
        x0 = *(const float4*)(xs + (size_t)(i + 32) * 8); x1 = *(const float4*)(xs + (size_t)(i + 32) * 8 + 4);
#pragma unroll
        for (int r = 0; r < N; r++) acc[r] = dot8(b[r], x0, x1, acc[r]);
    }
    if (i < n8) {
        const float4 x0 = *(const float4*)(xs + (size_t)i * 8), x1 = *(const float4*)(xs + (size_t)i * 8 + 4);
#pragma unroll
        for (int r = 0; r < N; r++) acc[r] = dot8(__ldcs(w[r] + i), x0, x1, acc[r]);
    }
}

// pre: f32 rows: the first kRowAhead float4 of this lane, when they are there already
constexpr int kRowAhead = 4;
template <int WK>
__device__ __forceinline__ float row_dot(const GemvSeg& sg, int row, int K, const float* xs, int lane, const float4* pre = nullptr) {
    float acc = 0.0f;
    if (WK == WK_Q8) {
        // planes: quants [N,K] + scales [N,K/32].  packed (kc > 0): the streaming kernel's tile stream — per row group of
        // 8 rows K/512 tiles of 4352 bytes; inside a tile block b (0..15) of row r sits at b*256 + (byte/16)*128 + r*16 +
        // byte%16 and its scale is entry b*8 + r of the 128 binary16 values after the 4096 quants.
        const int kc = sg.kc;
        const unsigned char* gbase = kc ? (const unsigned char*)sg.w + (size_t)(row >> 3) * (K / kTileK) * kTileBytes : nullptr;
        const int8_t* q = (const int8_t*)sg.w + (size_t)row * K;
        const __half* sc = sg.s + (size_t)row * (K >> 5);
        for (int b = lane; b < (K >> 5); b += 32) {        // one 32-block per lane per trip
            uint4 w0, w1;
            float d;
            if (kc) {
                const unsigned char* t = gbase + (size_t)(b >> 4) * kTileBytes;
                const unsigned char* cm = t + ((b & 15) << 8) + ((row & 7) << 4);
                w0 = *(const uint4*)cm;
                w1 = *(const uint4*)(cm + 128);
                d = __half2float(((const __half*)(t + kTileQ))[((b & 15) << 3) + (row & 7)]);
            } else {
                const uint4* p = (const uint4*)(q + (size_t)b * 32);
                w0 = p[0]; w1 = p[1];
                d = __half2float(sc[b]);
            }
            const float4* x4 = (const float4*)(xs + (size_t)b * 32);
            float p0 = dot4_s8(w0.x, x4[0], 0.0f), p1 = dot4_s8(w0.y, x4[1], 0.0f);
            p0 = dot4_s8(w0.z, x4[2], p0); p1 = dot4_s8(w0.w, x4[3], p1);
            p0 = dot4_s8(w1.x, x4[4], p0); p1 = dot4_s8(w1.y, x4[5], p1);
            p0 = dot4_s8(w1.z, x4[6], p0); p1 = dot4_s8(w1.w, x4[7], p1);
            acc = fmaf(p0 + p1, d, acc);
        }
    } else if (WK == WK_F32) {
        const float* w = (const float*)sg.w + (size_t)row * K;
        if ((K & 3) == 0) {
            const float4* w4 = (const float4*)w;
            const float4* x4 = (const float4*)xs;
            int i = lane;
            if (pre) {
#pragma unroll
                for (int t = 0; t < kRowAhead; t++, i += 32)
                    if (i < (K >> 2)) {
                        const float4 a = pre[t], b = x4[i];
                        acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc); acc = fmaf(a.w, b.w, acc);
                    }
            }
            for (; i < (K >> 2); i += 32) {
                const float4 a = w4[i], b = x4[i];
                acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc); acc = fmaf(a.z, b.z, acc); acc = fmaf(a.w, b.w, acc);
            }
        } else {
            for (int i = lane; i < K; i += 32) acc = fmaf(w[i], xs[i], acc);
        }
    } else {
        const uint16_t* w = (const uint16_t*)sg.w + (size_t)row * K;
        if ((K & 7) == 0) {
            const uint4* const w8[1] = {(const uint4*)w};
            float r[1] = {0.0f};
            bf16_rows_dot<1>(w8, K >> 3, xs, lane, r);
            acc = r[0];
        } else {
            for (int i = lane; i < K; i += 32) acc = fmaf(bf16_bits_to_f32(w[i]), xs[i], acc);
        }
    }
    return warp_sum(acc);
}

constexpr int kDirectBf16Ctas = 3;                     // resident CTAs per SM of the bf16 form (four rows' loads in registers)
template <int WK>
__global__ void __launch_bounds__(256, WK == WK_BF16 ? kDirectBf16Ctas : 0) gemv_direct(const GemvArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const bool paired = a.epi == EPI_SWIGLU;
    int rows_total = 0;
    if (paired) rows_total = a.seg[0].rows;
    else for (int s = 0; s < a.nseg; s++) rows_total += a.seg[s].rows;
    const int row0 = (int)((long long)blockIdx.x * rows_total / gridDim.x);
    const int row1 = (int)((long long)(blockIdx.x + 1) * rows_total / gridDim.x);
    const int n = row1 - row0;

    float* scratch = (float*)smem;             // 64 words of reduction scratch
    float* xs = scratch + 64;                  // K floats (K rounded up to 4)
    float* vals = xs + ((a.K + 3) & ~3);       // 2 * max rows per CTA

    const int sub = paired ? 2 : 1;
    auto row_of = [&](int i, int* sg) {
        const int h = i / n;
        int row = row0 + i - h * n;
        *sg = 0;
        if (paired) *sg = h;
        else while (*sg < a.nseg - 1 && row >= a.seg[*sg].rows) { row -= a.seg[*sg].rows; (*sg)++; }
        return row;
    };
    if (a.use_pdl) pdl_launch_dependents();
    // What does not depend on the previous kernel is on its way before that is waited for: the gain of element tid, the start of each warp's first f32 row.  A small
    // model's step is a chain of trips to L2 (tiny_f32 of the configurations, 31 steps of 12 kernels: 1490 -> 1337 us).
    const float gain0 = a.gain && tid < a.K ? load_gain(a.gain, a.gain_kind, tid) : 0.0f;
    float4 pre[WK == WK_F32 ? kRowAhead : 1];
    const bool ahead = WK == WK_F32 && (a.K & 3) == 0 && warp < n * sub;
    if (ahead) {
        int sg;
        const int row = row_of(warp, &sg);
        const float4* w = (const float4*)((const float*)a.seg[sg].w + (size_t)row * a.K);
#pragma unroll
        for (int t = 0; t < kRowAhead; t++) pre[WK == WK_F32 ? t : 0] = lane + 32 * t < (a.K >> 2) ? __ldg(w + lane + 32 * t) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (a.use_pdl) pdl_grid_wait();
    const float resid0 = a.epi == EPI_RESID && tid < n ? a.resid[row0 + tid] : 0.0f;
    gemv_load_x(a, xs, tid, 256, scratch, 1, gain0);

    if (WK == WK_BF16 && (a.K & 7) == 0) {
        // Four rows at a time: vocabulary projection of 151936 x 2560 (778 MB) 222 us with one, 125 us = 6.2 TB/s with four.  At every size: where a CTA
        // has eight rows two of its warps work, and that is still no slower than eight with a row each (back to back, us with one / four:
        // 1024 x 512 6.2 / 5.9, 2048 x 512 6.2 / 6.1, 4096 x 1024 10.2 / 7.9, 4096 x 4096 16.9 / 15.9, 28672 x 4096 73.5 / 46.8)
        for (int i0 = warp * 4; i0 < n * sub; i0 += 32) {
            const uint4* w[4];
            float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int r = 0; r < 4; r++) {
                int sg;
                const int row = row_of(min(i0 + r, n * sub - 1), &sg);         // (rows past the end: the last one again, not stored)
                w[r] = (const uint4*)((const uint16_t*)a.seg[sg].w + (size_t)row * a.K);
            }
            const uint4* const (&wc)[4] = w;
            bf16_rows_dot<4>(wc, a.K >> 3, xs, lane, v);
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float t = warp_sum(v[r]);
                if (lane == 0 && i0 + r < n * sub) vals[i0 + r] = t;
            }
        }
    } else {
        for (int i = warp; i < n * sub; i += 8) {
            int sg;
            const int row = row_of(i, &sg);
            const float v = row_dot<WK>(a.seg[sg], row, a.K, xs, lane, ahead && i == warp ? pre : nullptr);
            if (lane == 0) vals[i] = v;
        }
    }
    named_sync(1, 256);
    ArgBest best{-INFINITY, -1};
    gemv_epilogue_rows(a, vals, row0, n, tid, 256, scratch, 1, &best, resid0);
    if (a.epi == EPI_ARGMAX) argmax_finish(a, best, tid, 256, 1);
    if (a.epi == EPI_PEER && !a.peer_ll) peer_publish(a, tid, 256, 1);
}

// ------------------------------------------------------------------------------ host side

// Packed layout: available when the matrix cuts into whole tiles (8 rows x 512 columns).  The "K-chunk" reported for a
// packed matrix is the tile width; 0 means the matrix stays in planes and is read by the direct kernel.
int q8_pack_kc(int rows, int K) {
    if (K <= 0 || K % kTileK || K > 16384 || rows <= 0 || rows % kTileRows) return 0;
    return kTileK;
}
size_t q8_packed_bytes(int rows, int K) {
    return q8_pack_kc(rows, K) ? (size_t)rows / kTileRows * (size_t)(K / kTileK) * kTileBytes : 0;
}

bool gemv_stream_supported(const GemvArgs& a) {
    if (a.wkind != WK_Q8 || a.force_direct) return false;
    if (a.K % kTileK || a.K > 16384 || ((uintptr_t)a.x & 15) || (a.x_add && ((uintptr_t)a.x_add & 15))) return false;
    for (int s = 0; s < a.nseg; s++)
        if (a.seg[s].rows % kTileRows || a.seg[s].kc != kTileK) return false;       // every segment must be in the packed layout
    if (a.epi == EPI_SWIGLU && (a.nseg != 2 || a.seg[0].rows != a.seg[1].rows)) return false;
    return true;
}

static cudaError_t launch_with_attrs(const void* fn, dim3 grid, dim3 block, size_t smem, cudaStream_t st, GemvArgs& a) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = a.use_pdl && !a.ordered ? 1 : 0;
    void* params[] = {&a};
    return cudaLaunchKernelExC(&cfg, fn, params);
}

cudaError_t launch_gemv(const GemvArgs& a_in, int sm_count, cudaStream_t st) {
    GemvArgs a = a_in;
    int rows_total = 0;
    if (a.epi == EPI_SWIGLU) rows_total = a.seg[0].rows;
    else for (int s = 0; s < a.nseg; s++) rows_total += a.seg[s].rows;
    if (rows_total <= 0 || a.K <= 0) return cudaErrorInvalidValue;

    if (gemv_stream_supported(a)) {
        static const int env_slack = [] { const char* e = getenv("LUM_CLAIM_SLACK"); return e ? atoi(e) + 1 : 0; }();
        if (a.max_units == 0) a.max_units = env_slack;
        a.KC = kTileK;
        const bool ranges = a.ksplit > 1 && a.epi == EPI_STORE && a.nseg == 1 && a.ksplit <= gemv_k_ranges(a.K, a.seg[0].kc) && sm_count >= a.K / kTileK && !a.gain && !a.x_add && !a.n_parts && !a.x_out;
        if (a.ksplit > 1 && !ranges) return cudaErrorInvalidValue;      // the caller's consumer expects that many partial vectors
        const int tpr = a.K / kTileK;
        a.k_smem = a.K;
        int grid = sm_count;
        if (ranges) {
            int most = 0;
            for (int r = 0; r < a.ksplit; r++) most = std::max(most, gemv_range_tile(tpr, a.ksplit, r + 1) - gemv_range_tile(tpr, a.ksplit, r));
            a.k_smem = most * kTileK;
        } else {
            const int gpf = tpr > kFillTiles ? 1 : kJobTiles / tpr, jobs = (rows_total / kTileRows + gpf - 1) / gpf;
            if (jobs < grid) grid = jobs;
        }
        const size_t fixed = gemv_fixed_smem(a.k_smem);
        // Up to 4096 elements a CTA takes half an SM: rings of 75 to 91 KB.  So that the next projection's CTAs can only spread one to an SM, whatever
        // order this one's leave in, every other projection asks for a little more than half (`wide_smem`): two of these don't fit an SM, nor
        // do one and two of the others.  Longer vectors take an SM to themselves.
        constexpr size_t kHalf = 109 * 1024 - 256, kWide = 114 * 1024, kAll = 226 * 1024;
        const int tiles = a.k_smem / kTileK;
        GemvRings rings{1, 1, kFillTiles, kFillTiles};
        if (tiles > kFillTiles && tiles < kJobTiles) rings.t1 = tiles - kFillTiles;
        const size_t room = fixed + 4 * kFillBytes <= kHalf ? kHalf : kAll;
        for (int i = 0; i < 2 * 3 - 2; i++) {                // in turn, up to three stages each
            GemvRings more = rings;
            (more.n0 > more.n1 ? more.n1 : more.n0)++;
            if (fixed + more.bytes() > room) break;
            rings = more;
        }
        if (const size_t need = fixed + rings.bytes(); need > kAll) return cudaErrorInvalidValue;
        a.ring_n[0] = rings.n0; a.ring_n[1] = rings.n1; a.ring_t[0] = rings.t0; a.ring_t[1] = rings.t1;
        const int fills = (a.epi == EPI_SWIGLU ? 2 : 1) * ((tiles + kJobTiles - 1) / kJobTiles);          // of a job, in the first ring
        a.own_jobs = a.job_ctr ? rings.n1 / fills : 0;
        size_t smem = fixed + rings.bytes();
        if (a.wide_smem && smem < kWide) smem = kWide;
        // instantiations: with and without the tensor-parallel paths (partial vectors of other ranks in, peer stores out); a tile of the row group per warp, or any K
        const bool peer = a.n_peers > 0 || a.parts_ll || a.part_flags != nullptr || a.epi == EPI_PEER;
        const int fewest = ranges ? tpr / a.ksplit : tpr;
        const bool one = fewest > kFillTiles && tiles <= kJobTiles;
        const void* fn = peer ? (one ? (const void*)q8_gemv_stream<true, true> : (const void*)q8_gemv_stream<true, false>)
                              : (one ? (const void*)q8_gemv_stream<false, true> : (const void*)q8_gemv_stream<false, false>);
        static std::atomic<uint64_t> raised[4] = {};
        if (const cudaError_t e = allow_smem(raised[(peer ? 2 : 0) + one], fn, (int)kAll, true)) return e;
        return launch_with_attrs(fn, dim3(grid), dim3(kGemvThreads), smem, st, a);
    }

    if (a.ksplit > 1) return cudaErrorInvalidValue;      // the caller's consumer expects several partial vectors: only the streaming kernel makes them
    // direct kernel: a few CTAs per SM's worth of rows, at least 8 rows per CTA; a large bf16 / f32 matrix gets as many CTAs as
    // an SM can hold, so that enough loads are in flight to keep HBM busy
    int grid = sm_count * (a.wkind != WK_Q8 && (long long)rows_total * a.K >= (1ll << 24) ? (a.wkind == WK_BF16 ? kDirectBf16Ctas : 8) : 2);
    if (grid > (rows_total + 7) / 8) grid = (rows_total + 7) / 8;
    if (a.epi == EPI_ARGMAX && grid > kArgmaxSlots) grid = kArgmaxSlots;       // one best-logit slot per CTA
    if (grid < 1) grid = 1;
    const int max_rows = (rows_total + grid - 1) / grid + 1;
    const size_t smem = 256 + (size_t)((a.K + 3) & ~3) * 4 + (size_t)max_rows * 2 * 4;
    const void* fn = a.wkind == WK_Q8 ? (const void*)gemv_direct<WK_Q8> : a.wkind == WK_F32 ? (const void*)gemv_direct<WK_F32> : (const void*)gemv_direct<WK_BF16>;
    if (a.wkind == WK_Q8 && (a.K % 32)) return cudaErrorInvalidValue;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(200 * 1024));
        if (e != cudaSuccess) return e;
        if (smem > 200 * 1024) return cudaErrorInvalidValue;
    }
    return launch_with_attrs(fn, dim3(grid), dim3(256), smem, st, a);
}

}  // namespace lum

// ------------------------------------------------------------------------------ sampling without allocating
//
// lum_op_sample_q8_0_static: the vocabulary projection + greedy sample of lum_op_sample_q8_0, for hosts that must
// not allocate device memory at call time.  That is the situation of a runtime embedded in a server that has
// already given every byte of HBM to its own arenas (weights, KV cache), where a cudaMalloc would fail — and of
// any caller on a latency-critical path, because cudaMalloc and cudaFree synchronise the whole device.
//
// The kernel's scratch (one best-logit / best-row pair per CTA, the arrival ticket, a status word) lives in the
// fixed array below instead of an allocated buffer.  Consequences, all part of the contract:
//   * capacity: 256 CTAs.  The kernel runs one CTA per SM, so a device with more than 256 SMs is refused.
//   * every GPU that loads this library carries the 4 KiB array until the process exits;
//   * every call on a device shares it, and it keeps the previous call's contents: the entry zeroes the arrival ticket on
//     the caller's stream before each launch, the per-CTA slots are overwritten by the kernel before it is read, and the
//     status word keeps a pending error until lum_op_status reports and clears it;
//   * two calls whose kernels could overlap on one GPU (different streams, no dependency) race on it — order them;
//   * the array's name is only a host-side handle; its device address is looked up with cudaGetSymbolAddress the first
//     time the entry is called on a device (with that device current).  That first call does this one-time set-up
//     and should therefore be made before any stream capture begins.
static __device__ __align__(256) unsigned char g_sample_static[4096];
constexpr int kStaticMaxCtas = 256;     // 256 floats + 256 ints + ticket + status = 2056 bytes of the 4096

static unsigned char* g_static_dev_ptr[64] = {nullptr};      // device address of the array, per device ordinal (set on first use)
// where lum_op_status finds this entry's status word on the current device (null: the entry was never used there)
uint32_t* lum_static_sample_status() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64 || !g_static_dev_ptr[dev]) return nullptr;
    return (uint32_t*)(g_static_dev_ptr[dev] + 2052);
}

extern "C" int32_t lum_op_sample_q8_0_static(const void* packed, int32_t n, int32_t k, const float* x, float* logits,
                                            int32_t* best, void* stream) {
    using namespace lum;
    unsigned char** dev_ptr = g_static_dev_ptr;
    const int kc = q8_pack_kc(n, k);
    if (!packed || !x || !logits || !best || !kc) {
        set_op_error("sample_q8_0_static: bad arguments or shape cannot be packed (needs K % 512 == 0, K <= 16384, N % 8 == 0)");
        return -1;
    }
    if ((uintptr_t)x & 15) {       // the streaming kernel copies x with 16-byte loads; no other kernel reads the packed layout
        set_op_error("sample_q8_0_static: x must be 16-byte aligned");
        return -1;
    }
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) { set_op_error("sample_q8_0_static: cannot query the current device"); return -2; }
    if (sms > kStaticMaxCtas) {
        set_op_error("sample_q8_0_static: this device has more than 256 SMs; the static scratch holds one slot per CTA for at most 256");
        return -3;
    }
    if (!dev_ptr[dev]) {
        // one-time set-up for this device: the symbol's device address (a kernel given the host-side name would fault)
        void* p = nullptr;
        e = cudaGetSymbolAddress(&p, g_sample_static);
        if (e != cudaSuccess || !p) { set_op_error("sample_q8_0_static: cudaGetSymbolAddress failed"); return -2; }
        dev_ptr[dev] = (unsigned char*)p;
    }
    unsigned char* base = dev_ptr[dev];
    cudaStream_t st = (cudaStream_t)stream;
    e = cudaMemsetAsync(base + 2048, 0, 4, st);         // the arrival ticket starts at zero (a status left by an earlier call
                                                        // stays until lum_op_status reads it; the array is zero when the library loads)
    if (e != cudaSuccess) { set_op_error("sample_q8_0_static: clearing the ticket failed"); return -2; }
    GemvArgs a{};
    a.nseg = 1; a.seg[0] = {packed, nullptr, n, kc}; a.K = k; a.wkind = WK_Q8; a.epi = EPI_ARGMAX; a.x = x; a.y = logits;
    a.part_val = (float*)base; a.part_idx = (int*)(base + 1024); a.counter = (unsigned int*)(base + 2048);
    a.status = (uint32_t*)(base + 2052); a.pair_out = best; a.row_offset = 0;
    e = launch_gemv(a, sms, st);
    if (e != cudaSuccess) { set_op_error(cudaGetErrorString(e)); return -2; }
    return 0;
}

