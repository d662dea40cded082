// Routed mixture-of-experts FFN for Q8_0 expert weights: the `MoeExperts` host op of the reference
// (examples/gpt_oss/src/model.rs:772-1118) with its two kernels `moe_gate_up_swiglu` (:821-900) and
// `moe_down_weighted_sum` (:903-962), plus the router product and the RMSNorm the graph places in front of it
// (:263-267).  The reference handles one token and has every CTA redo the top-k; here the routing is done once per
// token by its own kernel, the expert kernels take T tokens (T > 1 when an expert-parallel rank serves the tokens of
// the other ranks), and a rank only computes the experts it holds.
//
//   moe_route      a cluster of CTAs per token: xf = RMSNorm(x) * gain; logits = W_r xf + b_r; top-k by repeated arg-max (the first
//                  of equal maxima wins), softmax over the selected logits -> sel[t][k], wt[t][k]
//   moe_gate_up    gate / up = rows 2i / 2i+1 of a selected expert's gate_up matrix . xf + bias; gate <= limit, |up| <= limit;
//                  s = (up + 1) * gate * sigmoid(1.702 gate)
//   moe_down       sum over the token's selected LOCAL experts of wt * (W_down row . s + bias); added to the residual stream (one
//                  GPU) or left as this rank's partial
//
// Expert weights are Q8_0 planes (int8 [rows, K] and one binary16 scale per 32): a row is one contiguous run.  Converting every int8
// weight to f32 (a quarter-rate instruction each) binds such a kernel at about 1 TB/s, so — as in the streaming GEMV — the ACTIVATIONS
// go to the integer side instead: a CTA writes the token's activation vector as three int8 levels per 32-block, x ~= s (a1 + a2/254 +
// a3/254^2) (error <= 1.03 max|x| 2^-24), into shared memory once, and a weight block then costs 24 integer dot-product instructions (dp4a)
// and a few conversions.
#include "lum_gemv_dev.cuh"
#include "lum_moe.cuh"

namespace lum {

// x[0..K) (global, f32) -> three int8 levels [3][K] and K / 32 scales in shared memory.  All `nthreads` threads (a multiple of 8)
// call it; 8 consecutive threads own one 32-block.  Same levels as the GEMV prologue's.
__device__ __forceinline__ void x_levels_to_smem(const float* x, int K, int8_t* xq, float* xs, int tid, int nthreads) {
    const int n4 = K >> 2;
    constexpr int kAhead = 4;                            // loads on their way before the first is used
    for (int f0 = tid; f0 < ((n4 + nthreads - 1) / nthreads) * nthreads; f0 += nthreads * kAhead) {
      float4 vv[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; u++) vv[u] = f0 + u * nthreads < n4 ? __ldcg((const float4*)x + f0 + u * nthreads) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int u = 0; u < kAhead; u++) {
        const int f4 = f0 + u * nthreads;
        const bool in = f4 < n4;
        const float4 v = vv[u];
        const float e[4] = {v.x, v.y, v.z, v.w};
        uint32_t p[3];
        const float s1 = gemv_levels(e, p);
        if (in) {
            ((uint32_t*)xq)[f4] = p[0];
            ((uint32_t*)(xq + K))[f4] = p[1];
            ((uint32_t*)(xq + 2 * (size_t)K))[f4] = p[2];
            if ((f4 & 7) == 0) xs[f4 >> 3] = s1;
        }
      }
    }
}

// ---- Rows of experts, streamed.  A warp works through a list of units, each two consecutive weight rows of one expert (contiguous int8 planes): it
// keeps a ring of `stages` chunks (up to kMoeBlocks blocks of both rows) in shared memory, filled by bulk copies that one of its lanes issues, and
// never waits for another warp.  What bounds the kernels is how many bytes are on their way: 16 warps x 2 stages x 5.8 KB = 184 KB per SM, against
// the 12 KB that plain loads had in flight (8 warps x 4 stages: 34.25 against 31.25 ms for 16 tokens of the gpt-oss-20B shape).  Two lanes share a block (16 bytes each: no bank conflicts), the activation levels of a block
// serve both rows.  Scales and biases come with plain loads one unit ahead; nothing in the loop waits for a load made in the same turn.
constexpr int kMoeWarps = 16, kMoeTrips = 6, kMoeBlocks = 16 * kMoeTrips, kMoeMaxStages = 2;
struct MoeRing { unsigned char* base; uint32_t bars; int stages, blocks; uint32_t issued, taken; };      // blocks: of one row, per stage
__host__ __device__ inline size_t moe_ring_bytes(int stages, int blocks) { return (size_t)kMoeWarps * stages * blocks * 64; }

// rows(u): number of unit u's first row in the planes q [.., K] and sc [.., K / 32]; bias [..] of kind gain_kind.
// levels(u, &xq, &xs): activations.  done(u, r0, r1): the two rows' sums, biases added, in every lane.
template <typename Rows, typename Levels, typename Ready, typename Done>
__device__ __forceinline__ bool moe_stream(MoeRing& ring, int units, int K, const int8_t* q, const __half* sc, const void* bias, int gain_kind, int lane, Rows rows,
                                           Levels levels, Ready ready, Done done) {
    const int nb = K >> 5, chunks = (nb + ring.blocks - 1) / ring.blocks, total = units * chunks;
    auto count = [&](int c) { return min(ring.blocks, nb - c * ring.blocks); };
    auto issue = [&](int i, uint32_t seen) {                     // seen: see behind()
        const int u = i / chunks, c = i - u * chunks, n = count(c);
        const int8_t* src = q + rows(u) * K;
        const uint32_t st = ring.issued % ring.stages, bar = ring.bars + 8u * st;
        const uint32_t dst = behind(smem_u32(ring.base) + st * (uint32_t)ring.blocks * 64u, seen);
        if (elect_one()) {
            mbar_arrive_expect_tx(bar, (uint32_t)n * 64u);
            if (chunks == 1) bulk_g2s(dst, src, (uint32_t)n * 64u, bar);                // both rows are one run
            else {
                bulk_g2s(dst, src + (size_t)c * ring.blocks * 32, (uint32_t)n * 32u, bar);
                bulk_g2s(dst + (uint32_t)n * 32u, src + K + (size_t)c * ring.blocks * 32, (uint32_t)n * 32u, bar);
            }
        }
        ring.issued++;
    };
    auto scales = [&](int i, uint16_t (&d)[2][kMoeTrips], float (&b)[2]) {
        const int u = i / chunks, c = i - u * chunks, n = count(c);
        const size_t row = rows(u);
        const uint16_t* p = (const uint16_t*)(sc + row * nb) + c * ring.blocks + (lane >> 1);
#pragma unroll
        for (int t = 0; t < kMoeTrips; t++)
#pragma unroll
            for (int r = 0; r < 2; r++) d[r][t] = 16 * t + (lane >> 1) < n ? __ldg(p + r * nb + 16 * t) : (uint16_t)0;
        b[0] = load_gain(bias, gain_kind, (int)row);
        b[1] = load_gain(bias, gain_kind, (int)row + 1);
    };
    for (int i = 0; i < ring.stages && i < total; i++) issue(i, 0u);
    uint16_t dn[2][kMoeTrips], d[2][kMoeTrips];
    float bn[2], b[2];
    if (total > 0) scales(0, dn, bn);
    ready();                                                     // the activations are there
    float acc[2] = {0.0f, 0.0f};
    bool ok = true;
#pragma unroll 1
    for (int i = 0; i < total; i++) {
        const int u = i / chunks, c = i - u * chunks, n = count(c);
#pragma unroll
        for (int t = 0; t < kMoeTrips; t++) { d[0][t] = dn[0][t]; d[1][t] = dn[1][t]; }
        b[0] = bn[0]; b[1] = bn[1];
        if (i + 1 < total) scales(i + 1, dn, bn);
        const uint32_t st = ring.taken % ring.stages;
        if (!mbar_wait(ring.bars + 8u * st, (ring.taken / ring.stages) & 1u)) { ok = false; break; }
        const unsigned char* w = ring.base + (size_t)st * ring.blocks * 64;
        const int8_t* xq; const float* xs;
        levels(u, &xq, &xs);
        const int k0 = c * ring.blocks * 32;
#pragma unroll
        for (int t = 0; t < kMoeTrips; t++) {
            const int bl = 16 * t + (lane >> 1);
            if (bl < n) {
                const int off = t * 512 + lane * 16;
                const uint4 w0 = *(const uint4*)(w + off), w1 = *(const uint4*)(w + (size_t)n * 32 + off);
                int s0[3], s1[3];
#pragma unroll
                for (int lv = 0; lv < 3; lv++) {
                    const uint4 x = *(const uint4*)(xq + (size_t)lv * K + k0 + off);
                    s0[lv] = __dp4a((int)w0.w, (int)x.w, __dp4a((int)w0.z, (int)x.z, __dp4a((int)w0.y, (int)x.y, __dp4a((int)w0.x, (int)x.x, 0))));
                    s1[lv] = __dp4a((int)w1.w, (int)x.w, __dp4a((int)w1.z, (int)x.z, __dp4a((int)w1.y, (int)x.y, __dp4a((int)w1.x, (int)x.x, 0))));
                }
                const float sx = xs[(k0 >> 5) + bl];
                const float t0 = fmaf((float)s0[2], 1.0f / 64516.0f, (float)(s0[0] * 254 + s0[1]) * (1.0f / 254.0f));
                const float t1 = fmaf((float)s1[2], 1.0f / 64516.0f, (float)(s1[0] * 254 + s1[1]) * (1.0f / 254.0f));
                acc[0] = fmaf(t0, sx * __half2float(__ushort_as_half(d[0][t])), acc[0]);
                acc[1] = fmaf(t1, sx * __half2float(__ushort_as_half(d[1][t])), acc[1]);
            }
        }
        ring.taken++;
        __syncwarp();
        if (i + ring.stages < total) issue(i + ring.stages, __float_as_uint(acc[0]) ^ __float_as_uint(acc[1]));      // (both rows of the chunk have been added up)
        if (c == chunks - 1) {
            done(u, warp_sum(acc[0]) + b[0], warp_sum(acc[1]) + b[1]);
            acc[0] = acc[1] = 0.0f;
        }
    }
    // never leave while a copy into this CTA's shared memory may be in flight: wait (bounded) for what was issued
    if (!ok)
        for (uint32_t k = ring.taken; k < ring.issued; k++) mbar_wait(ring.bars + 8u * (k % ring.stages), (k / ring.stages) & 1u);
    return ok;
}
__device__ __forceinline__ void moe_ring_begin(MoeRing& r, unsigned char* base, unsigned long long* bars, int stages, int blocks, int tid) {
    if (tid < kMoeWarps * kMoeMaxStages) { mbar_init(smem_u32(bars + tid), 1); mbar_fence_init(); }
    r.base = base + (size_t)(tid >> 5) * stages * blocks * 64;
    r.bars = smem_u32(bars + (tid >> 5) * kMoeMaxStages);
    r.stages = stages; r.blocks = blocks; r.issued = r.taken = 0u;
    __syncthreads();
}
// This rank's selected experts of a token, into shared memory: their place in the selection and their number on this rank
struct MoeSel { int el, le; };
__device__ __forceinline__ int moe_selected(const MoeArgs& a, const float* xf, MoeSel* mine, int tid) {
    __syncthreads();                                             // the previous token's are no longer read
    int nl = 0;
    for (int el = 0; el < a.top_k; el++) {
        const int le = __ldcg((const int*)(xf + a.hidden) + el) - a.expert0;
        if (le < 0 || le >= a.n_local) continue;                 // another rank holds this expert
        if (tid == 0) mine[nl] = MoeSel{el, le};
        nl++;
    }
    __syncthreads();
    return nl;
}

// A cluster of eight CTAs per token: each normalises the row for itself and takes every eighth expert, a warp per expert; the first CTA gathers the logits
// and selects.  Gains and router rows do not depend on the previous kernel: a warp has its own on the way before it waits for that.
// Measured (gpt-oss-20B shape, cold caches): 16.3 us with one CTA of 512 threads, 8.5 us this way.
constexpr int kRouteCtas = 8, kRouteWarps = 4, kRouteAhead = 12, kRouteTrips = 8;
__global__ void __launch_bounds__(kRouteWarps * 32) moe_route(const MoeArgs a) {
    extern __shared__ __align__(16) float mr_smem[];          // xf [H], logits [E]
    __shared__ float scratch[kRouteWarps];
    constexpr int T = kRouteWarps * 32;
    const int t = blockIdx.x / kRouteCtas, rank = blockIdx.x % kRouteCtas, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int H = a.hidden, E = a.n_experts, n8 = H >> 3, n4 = H >> 2;
    float* xf = mr_smem;
    float* logits = xf + H;
    const bool bf = a.gain_kind == WK_BF16, wide = bf && (H & 7) == 0;
    const int e_first = warp * kRouteCtas + rank;
    uint4 ahead[kRouteAhead];
#pragma unroll
    for (int u = 0; u < kRouteAhead; u++)
        ahead[u] = wide && e_first < E && lane + 32 * u < n8 ? __ldg((const uint4*)((const uint16_t*)a.router + (size_t)e_first * H) + lane + 32 * u) : make_uint4(0u, 0u, 0u, 0u);
    uint2 gain[kRouteTrips];                                  // the gains of this thread's first float4s
#pragma unroll
    for (int u = 0; u < kRouteTrips; u++) gain[u] = bf && tid + T * u < n4 ? __ldg((const uint2*)a.gain + tid + T * u) : make_uint2(0u, 0u);
    if (a.use_pdl) { pdl_launch_dependents(); pdl_grid_wait(); }
    const float4* x = (const float4*)(a.x + (size_t)t * a.x_ld);
    float4* out = (float4*)(a.xf + (size_t)t * a.slot);
    float4 xv[kRouteTrips];
    float ss = 0.0f;
#pragma unroll
    for (int u = 0; u < kRouteTrips; u++) xv[u] = tid + T * u < n4 ? __ldcg(x + tid + T * u) : make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](float4 v) { ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss); };
#pragma unroll
    for (int u = 0; u < kRouteTrips; u++) add(xv[u]);
    for (int i = tid + T * kRouteTrips; i < n4; i += T) { const float4 v = __ldcg(x + i); ((float4*)xf)[i] = v; add(v); }
    ss = block_sum(ss, scratch, tid, T, 1, false);
    const float inv = 1.0f / sqrtf(ss * (1.0f / (float)H) + a.eps);
    auto put = [&](int i, float4 v, float g0, float g1, float g2, float g3) {
        v.x = (inv * v.x) * g0; v.y = (inv * v.y) * g1; v.z = (inv * v.z) * g2; v.w = (inv * v.w) * g3;
        ((float4*)xf)[i] = v;
        if (rank == 0) out[i] = v;
    };
#pragma unroll
    for (int u = 0; u < kRouteTrips; u++) {
        const int i = tid + T * u;
        if (i < n4) {
            if (bf) put(i, xv[u], __uint_as_float(gain[u].x << 16), __uint_as_float(gain[u].x & 0xffff0000u), __uint_as_float(gain[u].y << 16), __uint_as_float(gain[u].y & 0xffff0000u));
            else put(i, xv[u], load_gain(a.gain, a.gain_kind, i * 4), load_gain(a.gain, a.gain_kind, i * 4 + 1), load_gain(a.gain, a.gain_kind, i * 4 + 2), load_gain(a.gain, a.gain_kind, i * 4 + 3));
        }
    }
    for (int i = tid + T * kRouteTrips; i < n4; i += T)        // each thread's own elements
        put(i, ((const float4*)xf)[i], load_gain(a.gain, a.gain_kind, i * 4), load_gain(a.gain, a.gain_kind, i * 4 + 1), load_gain(a.gain, a.gain_kind, i * 4 + 2), load_gain(a.gain, a.gain_kind, i * 4 + 3));
    __syncthreads();
    auto dot8 = [&](uint4 w, int i, float acc) {               // 8 weights per 16-byte load
        const float4 x0 = *(const float4*)(xf + (size_t)i * 8), x1 = *(const float4*)(xf + (size_t)i * 8 + 4);
        acc = fmaf(__uint_as_float(w.x << 16), x0.x, acc); acc = fmaf(__uint_as_float(w.x & 0xffff0000u), x0.y, acc);
        acc = fmaf(__uint_as_float(w.y << 16), x0.z, acc); acc = fmaf(__uint_as_float(w.y & 0xffff0000u), x0.w, acc);
        acc = fmaf(__uint_as_float(w.z << 16), x1.x, acc); acc = fmaf(__uint_as_float(w.z & 0xffff0000u), x1.y, acc);
        acc = fmaf(__uint_as_float(w.w << 16), x1.z, acc); acc = fmaf(__uint_as_float(w.w & 0xffff0000u), x1.w, acc);
        return acc;
    };
    for (int e = e_first; e < E; e += kRouteCtas * kRouteWarps) {
        float acc = 0.0f;
        if (wide) {
            const uint4* w8 = (const uint4*)((const uint16_t*)a.router + (size_t)e * H);
            if (e == e_first) {
#pragma unroll
                for (int u = 0; u < kRouteAhead; u++)
                    if (lane + 32 * u < n8) acc = dot8(ahead[u], lane + 32 * u, acc);
            }
#pragma unroll 4
            for (int i = lane + (e == e_first ? 32 * kRouteAhead : 0); i < n8; i += 32) acc = dot8(__ldg(w8 + i), i, acc);
        } else if (bf) {
            const uint16_t* w = (const uint16_t*)a.router + (size_t)e * H;
            for (int i = lane; i < H; i += 32) acc = fmaf(bf16_bits_to_f32(w[i]), xf[i], acc);
        } else {
            const float* w = (const float*)a.router + (size_t)e * H;
            for (int i = lane; i < H; i += 32) acc = fmaf(w[i], xf[i], acc);
        }
        acc = warp_sum(acc);
        if (lane == 0) logits[e] = acc + load_gain(a.router_bias, a.gain_kind, e);
    }
    cluster_arrive_release();
    cluster_wait_acquire();
    if (rank == 0 && warp == 0) {
        for (int e = lane; e < E; e += 32)
            if (e % kRouteCtas) logits[e] = cluster_ld_f32(cluster_map(smem_u32(logits + e), (uint32_t)(e % kRouteCtas)));
        __syncwarp();
        // the token's routing travels with its activations: [H floats][top_k expert ids][top_k weights]
        int* sel = (int*)(a.xf + (size_t)t * a.slot + H);
        float* wt = a.xf + (size_t)t * a.slot + H + a.top_k;
        float mx = 0.0f, se = 0.0f;
        for (int ki = 0; ki < a.top_k; ki++) {                 // the first of equal maxima wins
            float best = -1e30f; int bi = 0x7fffffff;
            for (int e = lane; e < E; e += 32) if (logits[e] > best) { best = logits[e]; bi = e; }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
            }
            if (bi == 0x7fffffff) bi = 0;
            if (ki == 0) mx = best;                            // (the largest comes first)
            if (lane == 0) { sel[ki] = bi; wt[ki] = best; logits[bi] = -1e30f; }
            __syncwarp();
        }
        if (lane == 0) {
            for (int ki = 0; ki < a.top_k; ki++) { wt[ki] = expf(wt[ki] - mx); se += wt[ki]; }
            const float iv = 1.0f / se;
            for (int ki = 0; ki < a.top_k; ki++) wt[ki] *= iv;
        }
    }
    cluster_arrive_release();                                  // nobody leaves while the first CTA may still read its logits
    cluster_wait_acquire();
}

// One CTA per SM: its warps take (selected expert, position) pairs in turn; gate and up are rows 2 i and 2 i + 1.
// Measured (gpt-oss-20B shape, 4 experts, 70.5 MB, cold caches): 31.5 us with plain loads, 29.5 us with 8 warps of four stages, 24.4 us with 16 of two.
__global__ void __launch_bounds__(kMoeWarps * 32, 1) moe_gate_up(const MoeArgs a, const int stages, const int blocks) {
    extern __shared__ __align__(128) unsigned char me_smem[];
    __shared__ __align__(8) unsigned long long bars[kMoeWarps * kMoeMaxStages];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int H = a.hidden, F = a.ffn, nb = H >> 5;
    MoeRing ring;
    moe_ring_begin(ring, me_smem, bars, stages, blocks, tid);
    int8_t* xq = (int8_t*)(me_smem + moe_ring_bytes(stages, blocks));        // [3][H]
    float* xs = (float*)(xq + 3 * (size_t)H);                                // [H / 32]
    MoeSel* mine = (MoeSel*)(xs + nb);                                       // [top_k]
    // The routing must be there before the weights can be asked for.  The kernel after this one asks for its own as soon as it starts, so
    // it may only start now that the routing is.
    if (a.use_pdl) { pdl_grid_wait(); pdl_launch_dependents(); }
    for (int t = 0; t < a.n_tokens; t++) {
        const float* xf = a.xf_in + (size_t)t * a.slot;
        const int nl = moe_selected(a, xf, mine, tid);
        const int total = nl * F, w0 = blockIdx.x * kMoeWarps + warp, step = gridDim.x * kMoeWarps;
        const int units = w0 < total ? (total - w0 + step - 1) / step : 0;
        const bool ok = moe_stream(ring, units, H, a.gu_q, a.gu_s, a.gu_bias, a.gain_kind, lane,
            [&](int u) { const int p = w0 + u * step, n = p / F; return (size_t)mine[n].le * 2 * F + 2 * (size_t)(p - n * F); },
            [&](int, const int8_t** q, const float** s) { *q = xq; *s = xs; },
            [&] { x_levels_to_smem(xf, H, xq, xs, tid, kMoeWarps * 32); __syncthreads(); },
            [&](int u, float gate, float up) {
                if (lane == 0) {
                    const int p = w0 + u * step, n = p / F;
                    gate = fminf(gate, a.limit);
                    up = fmaxf(fminf(up, a.limit), -a.limit);
                    const float glu = gate * (1.0f / (1.0f + expf(-gate * 1.702f)));
                    a.sw[((size_t)t * a.top_k + mine[n].el) * F + (p - n * F)] = (up + 1.0f) * glu;
                }
            });
        if (!ok && lane == 0) atomicOr(a.status, LUM_ST_WAIT_FULL);
    }
}

// One CTA per SM takes pairs of output columns; a warp's unit is a pair's rows of one selected expert, and the experts' shares of a column meet in
// shared memory, added in the order of the selection.  The routing was complete before this kernel could start (see moe_gate_up), so the
// weights are on their way before the previous kernel is waited for.
// Measured (gpt-oss-20B shape, 4 experts, 35.3 MB, cold caches): 37 us with plain loads and a warp per column, 22.2 us with 8 warps of four stages,
// 21.3 us with 16 of two.
__global__ void __launch_bounds__(kMoeWarps * 32, 1) moe_down(const MoeArgs a, const int stages, const int blocks) {
    extern __shared__ __align__(128) unsigned char me_smem[];
    __shared__ __align__(8) unsigned long long bars[kMoeWarps * kMoeMaxStages];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int H = a.hidden, F = a.ffn, nbf = F >> 5;
    // per selected expert: levels [3][F], then scales [F / 32]
    const size_t per = (3 * (size_t)F + (size_t)nbf * 4 + 15) & ~(size_t)15;     // every expert's levels start 16-byte aligned (they are read with 128-bit loads)
    MoeRing ring;
    moe_ring_begin(ring, me_smem, bars, stages, blocks, tid);
    unsigned char* acts = me_smem + moe_ring_bytes(stages, blocks);
    const int pairs = (H / 2 - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;        // this CTA's: blockIdx.x, + gridDim.x, ..
    MoeSel* mine = (MoeSel*)(acts + a.top_k * per);                              // [top_k]
    float* res = (float*)(mine + a.top_k);                                       // [pairs][selected][2]
    if (a.use_pdl) pdl_launch_dependents();
    for (int t = 0; t < a.n_tokens; t++) {
        const float* xf = a.xf_in + (size_t)t * a.slot;
        const float* wt = xf + H + a.top_k;
        const int nl = moe_selected(a, xf, mine, tid);
        const int total = pairs * nl, units = warp < total ? (total - warp + kMoeWarps - 1) / kMoeWarps : 0;
        const bool ok = moe_stream(ring, units, F, a.dn_q, a.dn_s, a.dn_bias, a.gain_kind, lane,
            [&](int u) {
                const int v = warp + u * kMoeWarps, j = v / nl;
                return (size_t)mine[v - j * nl].le * H + 2 * ((size_t)blockIdx.x + (size_t)j * gridDim.x);
            },
            [&](int u, const int8_t** q, const float** s) {
                const unsigned char* x = acts + mine[(warp + u * kMoeWarps) % nl].el * per;
                *q = (const int8_t*)x; *s = (const float*)(x + 3 * (size_t)F);
            },
            [&] {
                if (a.use_pdl) pdl_grid_wait();
                for (int n = 0; n < nl; n++) {
                    const int el = mine[n].el;
                    x_levels_to_smem(a.sw + ((size_t)t * a.top_k + el) * F, F, (int8_t*)(acts + el * per), (float*)(acts + el * per + 3 * (size_t)F), tid, kMoeWarps * 32);
                }
                __syncthreads();
            },
            [&](int u, float r0, float r1) { if (lane == 0) *(float2*)(res + 2 * (warp + u * kMoeWarps)) = make_float2(r0, r1); });
        if (!ok && lane == 0) atomicOr(a.status, LUM_ST_WAIT_FULL);
        __syncthreads();
        for (int i = tid; i < pairs * 2; i += kMoeWarps * 32) {
            const int col = 2 * ((int)blockIdx.x + (i >> 1) * (int)gridDim.x) + (i & 1);
            float ov = 0.0f;
            for (int n = 0; n < nl; n++) ov = fmaf(__ldcg(wt + mine[n].el), res[2 * ((i >> 1) * nl + n) + (i & 1)], ov);
            if (a.out_add) a.out_add[(size_t)t * a.out_ld + col] += ov;     // one GPU: straight into the residual stream
            else a.out[(size_t)t * a.out_ld + col] = ov;                    // expert parallel: this rank's share of the token's output
        }
    }
}

// Expert parallel, after the combine exchange: x[col] += sum over the ranks' shares of this rank's token.
__global__ void moe_combine(float* x, const float* parts, int n_parts, int part_ld, int H) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= H) return;
    float v = 0.0f;
    for (int r = 0; r < n_parts; r++) v += parts[(size_t)r * part_ld + i];
    x[i] += v;
}

static cudaError_t launch1(const void* fn, dim3 grid, dim3 block, size_t smem, void** params, int cluster, int use_pdl, cudaStream_t st) {
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)cluster; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
        n++;
    }
    if (use_pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelExC(&cfg, fn, params);
}

cudaError_t launch_moe_route(const MoeArgs& a_in, int n_tokens, cudaStream_t st) {
    MoeArgs a = a_in;
    if (a.hidden % 4 || a.x_ld % 4 || a.slot % 4 || ((uintptr_t)a.x & 15)) return cudaErrorInvalidValue;
    void* params[] = {&a};
    return launch1((const void*)moe_route, dim3(n_tokens * kRouteCtas), dim3(kRouteWarps * 32), ((size_t)a.hidden + a.n_experts) * 4, params, kRouteCtas, a.use_pdl, st);
}
// Shared memory of an expert kernel beside its ring: activation levels and block scales, the selection, and (down) a CTA's results
size_t moe_gate_up_bytes(int H, int top_k) { return 3 * (size_t)H + (size_t)(H / 32) * 4 + (size_t)top_k * sizeof(MoeSel); }
size_t moe_down_bytes(int H, int F, int top_k, int sm_count) {
    const size_t pairs = ((size_t)H / 2 + sm_count - 1) / sm_count;
    return (size_t)top_k * ((3 * (size_t)F + (size_t)(F / 32) * 4 + 15) & ~(size_t)15) + (size_t)top_k * sizeof(MoeSel) + pairs * top_k * 8;
}
// The ring beside `act` bytes: two stages of whole rows (up to 96 blocks) where they fit, then shorter ones, then one stage; 0 where not even
// a block per warp fits.  Whatever 200 KB of levels and scales hold is taken (hidden up to 65536, eight experts of ffn up to 8192).
int moe_ring_fit(size_t act, int K, int* stages, int* blocks) {
    constexpr size_t kMost = 226 * 1024;
    int s = kMoeMaxStages, b = K / 32 < kMoeBlocks ? K / 32 : kMoeBlocks;
    while (act + moe_ring_bytes(s, b) > kMost && (s > 1 || b > 1)) {
        if (b > 16) b = b / 2 < 16 ? 16 : b / 2;
        else if (s > 1) s--;
        else b = b / 2;
    }
    *stages = s; *blocks = b;
    return act + moe_ring_bytes(s, b) <= kMost;
}
cudaError_t launch_moe_experts(const MoeArgs& a_in, int sm_count, cudaStream_t st) {
    MoeArgs a = a_in;
    if ((a.hidden % 32) || (a.ffn % 32) || a.top_k < 1) return cudaErrorInvalidValue;
    auto launch = [&](const void* fn, size_t act, int K) -> cudaError_t {
        int stages, blocks;
        if (!moe_ring_fit(act, K, &stages, &blocks)) return cudaErrorInvalidValue;
        void* params[] = {&a, &stages, &blocks};
        return launch1(fn, dim3(sm_count), dim3(kMoeWarps * 32), act + moe_ring_bytes(stages, blocks), params, 1, a.use_pdl, st);
    };
    cudaError_t e = launch((const void*)moe_gate_up, moe_gate_up_bytes(a.hidden, a.top_k), a.hidden);
    if (e != cudaSuccess) return e;
    return launch((const void*)moe_down, moe_down_bytes(a.hidden, a.ffn, a.top_k, sm_count), a.ffn);
}
cudaError_t launch_moe_combine(float* x, const float* parts, int n_parts, int part_ld, int H, cudaStream_t st) {
    moe_combine<<<(H + 255) / 256, 256, 0, st>>>(x, parts, n_parts, part_ld, H);
    return cudaGetLastError();
}

}  // namespace lum
