// Device-side body of single-token attention, shared by the one-op kernel (lum_attn.cu) and the whole-token
// persistent kernel (lum_mega.cu).  See lum_attn.cu for what it computes and which reference code it follows.
#pragma once
#include "lum_kernels.cuh"

namespace lum {

__device__ __forceinline__ float gain_at(const void* g, int kind, int i) {
    return kind == WK_BF16 ? bf16_bits_to_f32(((const uint16_t*)g)[i]) : ((const float*)g)[i];
}

// cos/sin of the rotation for pair index i at position pos.
// RS: the rotation convention known at compile time (0 / 1), or -1 to decide at run time — each convention brings its own
// precise transcendental functions, several KB of code apiece.
template <int RS = -1>
__device__ __forceinline__ void rope_cs(const AttnArgs& a, int i, int pos, float* cs, float* sn) {
    if (RS == 0 || (RS < 0 && a.rope_style == 0)) {
        // the graph's chain, constant by constant: f = 2i * (1/d); inv = 1/exp2((f * ln theta) * log2 e);
        // emb = pos * inv; sin(emb); cos as sin(-emb + pi/2)
        const float f = (float)(2 * i) * a.c_inv_d;
        const float inv = 1.0f / exp2f((f * a.c_ln_theta) * a.c_log2e);
        const float emb = (float)pos * inv;
        *sn = sinf(emb);
        *cs = sinf(emb * -1.0f + a.c_half_pi);
    } else if (a.rope_style == 2) {
        // YaRN table (examples/gpt_oss/src/model.rs:557-567): angle = pos * inv_freq[i], cos and sin times the attention factor
        const float ang = (float)pos * a.inv_freq[i];
        *sn = sinf(ang) * a.attn_factor;
        *cs = cosf(ang) * a.attn_factor;
    } else {
        const float freq = powf(a.theta, -((float)(2 * i)) / (float)a.hd);
        const float ang = (float)pos * freq;
        *sn = sinf(ang);
        *cs = cosf(ang);
    }
}

// The last step of a head's softmax: an optional sink logit (no value row) joins the denominator
// (examples/gpt_oss/src/model.rs:727-757), then the division.
__device__ __forceinline__ float attn_finish(float O, float M, float L, const void* sinks, int kind, int head) {
    if (sinks) {
        const float s = gain_at(sinks, kind, head);
        const float mn = fmaxf(M, s);
        const float c = expf(M - mn);
        L = L * c + expf(s - mn);
        O = O * c;
    }
    return O * (1.0f / L);
}

// One (kv head, split) of cached rows per CTA; all G <= GM query heads that share the KV head together.
//
// Phase A (whole CTA): this step's q heads of the group — and, in the CTA that owns the last split, the
// step's own k and v — are staged in shared memory, RMS-normalised per head if the model asks for it,
// rotated, and (k, v) rounded to the cache type and appended to the cache.
// Phase B: one warp per cached row and trip; lane i holds dims [i*DPL, (i+1)*DPL) of every head's q and
// running output, so a thread needs only 2 * G * DPL registers for them and the kernel fits beside the
// streaming GEMV's register budget in the persistent kernel.
// Loops stay rolled where they can: the code runs once per CTA, so its size in instruction-cache lines is latency.
constexpr int kAttnThreads = 512;
constexpr int kAttnWarps = kAttnThreads / 32;

// bytes of shared memory the body needs for G query heads per KV head
constexpr int kMaxSplits = 32;
constexpr int kMaxClusterSplits = 16;      // largest cluster the hardware schedules (above 8 the kernel has to opt in)
__host__ __device__ inline size_t attn_smem_bytes(int HD, int G) {
    return (size_t)(9 * HD + HD + 2 * kAttnWarps * 8 + 4 + HD) * 4 + (size_t)kAttnWarps * G * HD * 4;
}
// where the rotation table (cos, sin per dimension pair) lives in the attention scratch (`states`: partial states merged in the CTA)
__device__ __forceinline__ float* attn_rope_table(unsigned char* smem, int HD, int states = kAttnWarps) { return (float*)smem + 9 * HD + HD + 2 * states * 8 + 4; }
// The table depends only on the position: a kernel can fill it while it still waits for the projections (threads 0 .. HD/2-1).
template <int HD, int RS = -1>
__device__ __forceinline__ void attn_fill_rope(const AttnArgs& a, float* tab, int p, int tid) {
    if (tid < HD / 2) {
        float cs, sn;
        rope_cs<RS>(a, tid, p, &cs, &sn);
        tab[2 * tid] = cs;
        tab[2 * tid + 1] = sn;
    }
}

// DPL consecutive cache elements as the bits they are stored in (bf16: 2 bytes each, else f32)
template <bool BF16, int DPL> struct RawRow;
template <> struct RawRow<true, 4> { using type = uint2; };
template <> struct RawRow<true, 2> { using type = uint32_t; };
template <> struct RawRow<false, 4> { using type = float4; };
template <> struct RawRow<false, 2> { using type = float2; };
template <bool BF16, int DPL>
__device__ __forceinline__ typename RawRow<BF16, DPL>::type raw_load(const void* base, size_t elem_off) {
    using T = typename RawRow<BF16, DPL>::type;
    return BF16 ? *(const T*)((const uint16_t*)base + elem_off) : *(const T*)((const float*)base + elem_off);
}
__device__ __forceinline__ void raw_to_float_impl(uint2 r, float* out) {
    out[0] = __uint_as_float(r.x << 16); out[1] = __uint_as_float(r.x & 0xffff0000u);
    out[2] = __uint_as_float(r.y << 16); out[3] = __uint_as_float(r.y & 0xffff0000u);
}
__device__ __forceinline__ void raw_to_float_impl(uint32_t r, float* out) { out[0] = __uint_as_float(r << 16); out[1] = __uint_as_float(r & 0xffff0000u); }
__device__ __forceinline__ void raw_to_float_impl(float4 r, float* out) { out[0] = r.x; out[1] = r.y; out[2] = r.z; out[3] = r.w; }
__device__ __forceinline__ void raw_to_float_impl(float2 r, float* out) { out[0] = r.x; out[1] = r.y; }
template <bool BF16, int DPL>
__device__ __forceinline__ void raw_to_float(typename RawRow<BF16, DPL>::type r, float* out) { raw_to_float_impl(r, out); }

// The cached rows a CTA will walk do not depend on the projections of the current step (rows [.., p) were written by earlier
// steps), so a kernel that still waits for those projections can already ask for them to be brought into L2: one request
// per 128-byte line of every K and V row of this (KV head, split).
template <int HD, bool BF16>
__device__ __forceinline__ void attn_prefetch_rows(const AttnArgs& a, int kvh, int split, int p, int tid) {
    const int lo = (a.window > 0 && p + 1 > a.window) ? p + 1 - a.window : 0;
    const int n_cached = p - lo;
    const int per = (n_cached + a.n_splits - 1) / a.n_splits;
    const int r0 = lo + split * per;
    const int nc = max(0, min(p, r0 + per) - r0);
    constexpr int kRowBytes = HD * (BF16 ? 2 : 4), kLines = kRowBytes / 128;        // lines per K (or V) row of one head
    const size_t row_bytes = (size_t)a.n_kv * kRowBytes;
    for (int i = tid; i < nc * 2 * kLines; i += kAttnThreads) {
        const int r = i / (2 * kLines), w = i - r * (2 * kLines);
        const char* base = (const char*)(w < kLines ? a.k_cache : a.v_cache) + kv_phys_row(a.pg, 0, 0, r0 + r) * row_bytes + (size_t)kvh * kRowBytes + (size_t)(w % kLines) * 128;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(base));
    }
}

// Merging the splits of a KV head from a.part, called by all T threads of every CTA that holds one: the last CTA to arrive does it.
template <int HD>
__device__ __forceinline__ void attn_merge_ticket(const AttnArgs& a, int* s_last, int kvh, int G, int tid, int T, int bar_id) {
    __threadfence();
    named_sync(bar_id, T);
    if (tid == 0) {
        const unsigned int t = atomicAdd(&a.counters[kvh], 1u);
        *s_last = (t == (unsigned int)a.n_splits - 1u) ? 1 : 0;
    }
    named_sync(bar_id, T);
    if (!*s_last) return;
    __threadfence();
    // The partials were written by other CTAs: read them through L2 (ld.cg).  All loads of a batch of 8 splits
    // are issued before any is used, so a batch costs one round trip; batches fold into a running (max, sum, out).
    constexpr int kBatch = 8;
#pragma unroll 1
    for (int idx = tid; idx < G * HD; idx += T) {
        const int g = idx / HD, e = idx - g * HD;
        const float* src = a.part + ((size_t)kvh * a.n_splits * G + g) * (HD + 2);
        const size_t sstride = (size_t)G * (HD + 2);
        float M = -INFINITY, L = 0.0f, O = 0.0f;
#pragma unroll 1
        for (int s0 = 0; s0 < a.n_splits; s0 += kBatch) {
            float mv[kBatch], lv[kBatch], ov[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; j++) {
                const bool in = s0 + j < a.n_splits;
                const float* q2 = src + (size_t)(in ? s0 + j : 0) * sstride;
                mv[j] = in ? __ldcg(q2 + HD) : -INFINITY;
                lv[j] = __ldcg(q2 + HD + 1);
                ov[j] = __ldcg(q2 + e);
            }
            float Mb = M;
#pragma unroll
            for (int j = 0; j < kBatch; j++) Mb = fmaxf(Mb, mv[j]);
            const float c0 = (M == -INFINITY) ? 0.0f : expf(M - Mb);
            L *= c0; O *= c0;
#pragma unroll
            for (int j = 0; j < kBatch; j++) {
                const float c = (mv[j] == -INFINITY) ? 0.0f : expf(mv[j] - Mb);
                L = fmaf(lv[j], c, L);
                O = fmaf(ov[j], c, O);
            }
            M = Mb;
        }
        a.out[((size_t)kvh * G + g) * HD + e] = attn_finish(O, M, L, a.sinks, a.gain_kind, kvh * G + g);
    }
    if (tid == 0) a.counters[kvh] = 0u;
}

// Runs on exactly kAttnThreads threads (tid 0..511) that synchronise on named barrier `bar_id`.
// p = position of the token being processed (rows [.., p) are cached, row p is this step's own).
// smem: attn_smem_bytes(HD, G) bytes, 16-byte aligned.
// CL: the CTAs of one KV head form a thread-block cluster (cluster rank = split, 2 <= n_splits <= kMaxClusterSplits); the
// splits are then merged through distributed shared memory — every CTA finishes its own slice of the outputs — instead of
// through global partials and an arrival ticket.
template <int HD, int GM, bool BF16, bool CL = false>
__device__ __forceinline__ void attn_decode_body(const AttnArgs& a, unsigned char* smem, int kvh, int split, int p, int tid, int bar_id,
                                                 bool rope_ready = false) {
    constexpr int DPL = HD / 32;            // dims per lane
    constexpr int NW = kAttnWarps;
    const int warp = tid >> 5, lane = tid & 31;
    const int G = a.n_q / a.n_kv;
    auto sync = [bar_id] { named_sync(bar_id, kAttnThreads); };
    float (*s_q)[HD] = (float (*)[HD])smem;                 // [9][HD]: rotated q heads; row G = this step's k
    float* s_v = (float*)smem + 9 * HD;                     // [HD]
    float (*s_m)[8] = (float (*)[8])(s_v + HD);             // [NW][8]
    float (*s_l)[8] = (float (*)[8])(s_v + HD + NW * 8);    // [NW][8]
    int& s_last = *(int*)(s_v + HD + 2 * NW * 8);
    float* s_rope = s_v + HD + 2 * NW * 8 + 4;              // [HD/2][2]: cos, sin
    float* s_o = s_rope + HD;                               // [NW][G][HD]
    const int d0 = lane * DPL;
    const size_t row_elems = (size_t)a.n_kv * HD;

    // rows [lo, p) come from the cache; row p is this step's own
    const int lo = (a.window > 0 && p + 1 > a.window) ? p + 1 - a.window : 0;
    const int n_cached = p - lo;
    const int per = (n_cached + a.n_splits - 1) / a.n_splits;
    const int r0 = lo + split * per;
    const int r1 = min(p, r0 + per);
    const int nc = max(0, r1 - r0);                    // cached rows of this CTA
    const bool owns_new = split == a.n_splits - 1;
    const int n_rows = nc + (owns_new ? 1 : 0);
    const float scale = 1.0f / sqrtf((float)HD);

    // ---- phase A
    const int nheads = G + (owns_new ? 1 : 0);
    for (int idx = tid; idx < nheads * HD; idx += kAttnThreads) {
        const int h = idx / HD, e = idx - h * HD;
        float v = h < G ? a.q[((size_t)kvh * G + h) * HD + e] : a.k_new[(size_t)kvh * HD + e];
        if (h < G) { if (a.q_bias) v = v + gain_at(a.q_bias, a.gain_kind, (kvh * G + h) * HD + e); }
        else if (a.k_bias) v = v + gain_at(a.k_bias, a.gain_kind, kvh * HD + e);
        s_q[h][e] = v;
    }
    if (owns_new)
        for (int e = tid; e < HD; e += kAttnThreads) {
            float v = a.v_new[(size_t)kvh * HD + e];
            if (a.v_bias) v = v + gain_at(a.v_bias, a.gain_kind, kvh * HD + e);
            s_v[e] = v;
        }
    if (!rope_ready) attn_fill_rope<HD>(a, s_rope, p, tid);
    sync();
    if (a.q_gain || a.k_gain) {
        // per-head RMSNorm: x * 1/sqrt(mean(x^2) + eps) * g   (one warp per head)
#pragma unroll 1
        for (int h = warp; h < nheads; h += NW) {
            const void* gain = h < G ? a.q_gain : a.k_gain;
            if (!gain) continue;
            float ss = 0.0f;
            for (int e = lane; e < HD; e += 32) ss = fmaf(s_q[h][e], s_q[h][e], ss);
            ss = warp_sum(ss);
            const float inv = 1.0f / sqrtf(ss * (1.0f / (float)HD) + a.qk_eps);
            for (int e = lane; e < HD; e += 32) s_q[h][e] = (inv * s_q[h][e]) * gain_at(gain, a.gain_kind, e);
        }
        sync();
    }
#pragma unroll 1
    for (int idx = tid; idx < nheads * (HD / 2); idx += kAttnThreads) {
        const int h = idx / (HD / 2), i = idx - h * (HD / 2);
        const float cs = s_rope[2 * i], sn = s_rope[2 * i + 1];
        const int e0 = a.rope_style == 0 ? 2 * i : i, e1 = a.rope_style == 0 ? 2 * i + 1 : i + HD / 2;
        const float x0 = s_q[h][e0], x1 = s_q[h][e1];
        // separately rounded products and sums, as the graph's Mul / Add nodes produce them
        if (a.rope_style == 0) {
            s_q[h][e0] = __fadd_rn(__fmul_rn(x0, cs), __fmul_rn(__fmul_rn(x1, sn), -1.0f));
            s_q[h][e1] = __fadd_rn(__fmul_rn(x0, sn), __fmul_rn(x1, cs));
        } else {
            s_q[h][e0] = __fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn));
            s_q[h][e1] = __fadd_rn(__fmul_rn(x1, cs), __fmul_rn(x0, sn));
        }
    }
    sync();
    if (owns_new) {
        // append this step's row to the cache; keep the rounded values for our own use
        const size_t off = kv_phys_row(a.pg, 0, 0, p) * row_elems + (size_t)kvh * HD;
        for (int e = tid; e < HD; e += kAttnThreads) {
            if (BF16) {
                const __nv_bfloat16 kb = __float2bfloat16_rn(s_q[G][e]), vb = __float2bfloat16_rn(s_v[e]);
                ((__nv_bfloat16*)a.k_cache)[off + e] = kb;
                ((__nv_bfloat16*)a.v_cache)[off + e] = vb;
                s_q[G][e] = __bfloat162float(kb);
                s_v[e] = __bfloat162float(vb);
            } else {
                ((float*)a.k_cache)[off + e] = s_q[G][e];
                ((float*)a.v_cache)[off + e] = s_v[e];
            }
        }
        sync();
    }

    // ---- phase B
    float q[GM][DPL], o[GM][DPL], m[GM], l[GM];
#pragma unroll
    for (int g = 0; g < GM; g++) {
        m[g] = -INFINITY; l[g] = 0.0f;
#pragma unroll
        for (int i = 0; i < DPL; i++) { q[g][i] = g < G ? s_q[g][d0 + i] : 0.0f; o[g][i] = 0.0f; }
    }
    // rows of this CTA: cached rows r0 .. r1-1, then (last split only) the step's own row from shared memory.  A warp takes rows
    // warp, warp + NW, ...; the next row's K and V are requested (raw bits, converted only when used) before the current row is
    // worked on, so a warp waits for memory once, not once per row.
    using Raw = typename RawRow<BF16, DPL>::type;
    Raw kn = Raw(), vn = Raw();
    if (warp < nc) {
        const size_t off = kv_phys_row(a.pg, 0, 0, r0 + warp) * row_elems + (size_t)kvh * HD + d0;
        kn = raw_load<BF16, DPL>(a.k_cache, off);
        vn = raw_load<BF16, DPL>(a.v_cache, off);
    }
#pragma unroll 1
    for (int j = warp; j < n_rows; j += NW) {
        float kr[DPL], vr[DPL];
        const Raw kc = kn, vc = vn;
        if (j + NW < nc) {
            const size_t off = kv_phys_row(a.pg, 0, 0, r0 + j + NW) * row_elems + (size_t)kvh * HD + d0;
            kn = raw_load<BF16, DPL>(a.k_cache, off);
            vn = raw_load<BF16, DPL>(a.v_cache, off);
        }
        if (j < nc) {
            raw_to_float<BF16, DPL>(kc, kr);
            raw_to_float<BF16, DPL>(vc, vr);
        } else {
#pragma unroll
            for (int i = 0; i < DPL; i++) { kr[i] = s_q[G][d0 + i]; vr[i] = s_v[d0 + i]; }
        }
#pragma unroll
        for (int g = 0; g < GM; g++) {
            if (g < G) {
                float d = 0.0f;
#pragma unroll
                for (int i = 0; i < DPL; i++) d = fmaf(q[g][i], kr[i], d);
                d = warp_sum(d);
                const float logit = d * scale;
                const float mn = fmaxf(m[g], logit);
                const float corr = (m[g] == -INFINITY) ? 0.0f : expf(m[g] - mn);
                const float w = expf(logit - mn);
                l[g] = l[g] * corr + w;
#pragma unroll
                for (int i = 0; i < DPL; i++) o[g][i] = fmaf(w, vr[i], o[g][i] * corr);
                m[g] = mn;
            }
        }
    }
    // every warp publishes its running state; then the CTA merges them
#pragma unroll
    for (int g = 0; g < GM; g++) {
        if (g < G) {
            if (lane == 0) { s_m[warp][g] = m[g]; s_l[warp][g] = l[g]; }
#pragma unroll
            for (int i = 0; i < DPL; i++) s_o[((size_t)warp * G + g) * HD + d0 + i] = o[g][i];
        }
    }
    sync();
#pragma unroll 1
    for (int idx = tid; idx < G * HD; idx += kAttnThreads) {
        const int g = idx / HD, e = idx - g * HD;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < NW; w++) M = fmaxf(M, s_m[w][g]);
        float L = 0.0f, O = 0.0f;
#pragma unroll 2
        for (int w = 0; w < NW; w++) {
            const float c = (s_m[w][g] == -INFINITY) ? 0.0f : expf(s_m[w][g] - M);
            L = fmaf(s_l[w][g], c, L);
            O = fmaf(s_o[((size_t)w * G + g) * HD + e], c, O);
        }
        if (CL) {
            // q lives in registers by now: the staging area becomes this CTA's [G][HD + 2] result, read by the whole cluster
            float* dst = (float*)smem + (size_t)g * (HD + 2);
            dst[e] = O;
            if (e == 0) { dst[HD] = M; dst[HD + 1] = L; }
        } else if (a.n_splits == 1) {
            a.out[((size_t)kvh * G + g) * HD + e] = attn_finish(O, M, L, a.sinks, a.gain_kind, kvh * G + g);      // no other split to merge with
        } else {
            float* dst = a.part + (((size_t)kvh * a.n_splits + split) * G + g) * (HD + 2);
            dst[e] = O;
            if (e == 0) { dst[HD] = M; dst[HD + 1] = L; }
        }
    }
    if (CL) {
        // The own k row (row G of the staging area) was last read inside the row loop, before the barrier above, so the
        // writes just made collide with nothing.  Cluster barrier: every split's result is in place.
        cluster_arrive_release();
        cluster_wait_acquire();
        const int S = a.n_splits, total = G * HD;
        const int chunk = (total + S - 1) / S;          // outputs this CTA finishes: [split * chunk, (split + 1) * chunk)
        float* t = s_o;                                 // [S][chunk][3] staged (max, sum, out); the per-warp states are spent
        const uint32_t base = smem_u32(smem);
#pragma unroll 1
        for (int idx = tid; idx < S * chunk; idx += kAttnThreads) {
            const int s = idx / chunk, oi = idx - s * chunk, oidx = split * chunk + oi;
            if (oidx < total) {
                const int g = oidx / HD, e = oidx - g * HD;
                const uint32_t r = cluster_map(base + (uint32_t)(g * (HD + 2)) * 4u, (uint32_t)s);
                t[idx * 3] = cluster_ld_f32(r + HD * 4u);
                t[idx * 3 + 1] = cluster_ld_f32(r + (HD + 1) * 4u);
                t[idx * 3 + 2] = cluster_ld_f32(r + (uint32_t)e * 4u);
            }
        }
        sync();
        cluster_arrive_release();                       // this CTA has read what it needs from the others
        if (tid < chunk && split * chunk + tid < total) {
            // the same folding as the ticket path below — batches of 8 splits into a running (max, sum, out) — so both paths
            // give the same bits
            float M = -INFINITY, L = 0.0f, O = 0.0f;
#pragma unroll 1
            for (int s0 = 0; s0 < S; s0 += 8) {
                const int nb = min(8, S - s0);
                float Mb = M;
                for (int j = 0; j < nb; j++) Mb = fmaxf(Mb, t[((s0 + j) * chunk + tid) * 3]);
                const float c0 = (M == -INFINITY) ? 0.0f : expf(M - Mb);
                L *= c0; O *= c0;
                for (int j = 0; j < nb; j++) {
                    const float* v = t + (size_t)((s0 + j) * chunk + tid) * 3;
                    const float c = (v[0] == -INFINITY) ? 0.0f : expf(v[0] - Mb);
                    L = fmaf(v[1], c, L);
                    O = fmaf(v[2], c, O);
                }
                M = Mb;
            }
            a.out[(size_t)kvh * G * HD + split * chunk + tid] = attn_finish(O, M, L, a.sinks, a.gain_kind, kvh * G + (split * chunk + tid) / HD);
        }
        __syncwarp();
        cluster_wait_acquire();                         // nobody leaves while a neighbour may still read its memory
        return;
    }
    if (a.n_splits == 1) return;

    attn_merge_ticket<HD>(a, &s_last, kvh, G, tid, kAttnThreads, bar_id);
}

// ---- Products of attention on m16n8k16 tensor-core instructions (bf16 operands) without giving up f32 operands: K and V are bf16
// already; an f32 query or softmax weight is the sum of THREE bf16 terms (24 bits: all of it), and the terms take the rows of the first
// operand that a group of four query heads leaves free: row h holds head h's first term, rows 4 + h and 12 + h its second and third, so that
// the two small ones meet in one thread and the sum of the three is rounded once.
//
// The tensor core cuts every sum it hands back to 24 bits, always towards zero: carried from instruction to instruction, the loss grows with the
// number of keys and does not cancel (30000 keys, one split: 2.1e-5 of the result, 2.5e-7 with f32 additions).  So a sum leaves the tensor
// core after one instruction (16 products), and the rest is added up in f32, rounded to nearest: scores pairwise, values tile by tile.
__device__ __forceinline__ void attn_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1, float c2, float c3) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f), "f"(0.0f), "f"(c2), "f"(c3));
}
// Scores of eight keys, two of them this thread's: the sums of the KS instructions of 16 dimensions each; the third terms' row, 2^-16 of the rest,
// is carried along inside
template <int KS> struct AttnScore { float d[KS][2], c2, c3; };
template <int KS>
__device__ __forceinline__ void attn_mma_score(AttnScore<KS>& s, int ks, const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float d[4];
    attn_mma(d, a, b0, b1, ks ? s.c2 : 0.0f, ks ? s.c3 : 0.0f);
    s.d[ks][0] = d[0]; s.d[ks][1] = d[1]; s.c2 = d[2]; s.c3 = d[3];
}
template <int KS>
__device__ __forceinline__ float attn_score(AttnScore<KS>& s, int e) {
#pragma unroll
    for (int w = 1; w < KS; w *= 2)
#pragma unroll
        for (int i = 0; i + w < KS; i += 2 * w) s.d[i][e] += s.d[i + w][e];
    const float x = s.d[0][e] + (e ? s.c3 : s.c2);                   // first term, or second and third
    return x + __shfl_xor_sync(0xffffffffu, x, 16);
}
// values: 16 more keys, behind what the old ones are worth under the new maximum
__device__ __forceinline__ void attn_mma_value(float (&o)[2], float corr, const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float d[4];
    attn_mma(d, a, b0, b1, 0.0f, 0.0f);
    o[0] = fmaf(o[0], corr, d[0] + d[2]);
    o[1] = fmaf(o[1], corr, d[1] + d[3]);
}
// Two neighbouring elements for this thread's two rows, g = lane / 4 and g + 8: the first terms of head g (g < 4) and nothing, or the second and
// the third terms of head g - 4
__device__ __forceinline__ void attn_terms(float x0, float x1, bool second, uint32_t* lo_row, uint32_t* hi_row) {
    const __nv_bfloat162 t1 = __floats2bfloat162_rn(x0, x1);
    const float r0 = x0 - __low2float(t1), r1 = x1 - __high2float(t1);
    const __nv_bfloat162 t2 = __floats2bfloat162_rn(r0, r1);
    const __nv_bfloat162 t3 = __floats2bfloat162_rn(r0 - __low2float(t2), r1 - __high2float(t2));
    *lo_row = second ? *(const uint32_t*)&t2 : *(const uint32_t*)&t1;
    *hi_row = second ? *(const uint32_t*)&t3 : 0u;
}

// An infinity breaks the sum of terms (infinity times a zero term, or a first term rounded up to infinity): where a warp's state does not come out
// finite, it takes its keys once more, element by element in f32.  Keys first + 64 i .. + 15 below `end`; q [G][HD].
template <int HD>
__device__ __noinline__ void attn_plain_keys(const __nv_bfloat16* k, const __nv_bfloat16* v, KvPages pg, int seq, int max_seq, size_t row_elems, int first, int end,
                                             const float* q, int G, int lane, float* s_m, float* s_l, float* s_o) {
    constexpr int N = HD / 32;
    const float scale = 1.0f / sqrtf((float)HD);
    __syncwarp();                                                    // (the state in place is overwritten)
#pragma unroll 1
    for (int h = 0; h < G; h++) {
        float x[N], o[N], mx = -INFINITY, l = 0.0f;
#pragma unroll
        for (int i = 0; i < N; i++) { x[i] = q[h * HD + lane + 32 * i]; o[i] = 0.0f; }
#pragma unroll 1
        for (int j0 = first; j0 < end; j0 += 64)
#pragma unroll 1
            for (int j = j0; j < min(end, j0 + 16); j++) {
                const size_t off = kv_phys_row(pg, seq, max_seq, j) * row_elems + lane;
                float d = 0.0f;
#pragma unroll
                for (int i = 0; i < N; i++) d = fmaf(x[i], __bfloat162float(k[off + 32 * i]), d);
                const float logit = warp_sum(d) * scale, mn = fmaxf(mx, logit);
                const float corr = mx == -INFINITY ? 0.0f : expf(mx - mn), w = logit == -INFINITY ? 0.0f : expf(logit - mn);
                l = l * corr + w;
#pragma unroll
                for (int i = 0; i < N; i++) o[i] = fmaf(w, __bfloat162float(v[off + 32 * i]), o[i] * corr);
                mx = mn;
            }
        if (lane == 0) { s_m[h] = mx; s_l[h] = l; }
#pragma unroll
        for (int i = 0; i < N; i++) s_o[h * HD + lane + 32 * i] = o[i];
    }
}

// ---- Single-token attention over a bf16 cache on the tensor core: the form every decode step takes whose heads fit it (up to four query heads
// of 128 dimensions or eight of 64 per KV head; others, and f32 caches, take the form above).
//
// Bound by latency, not by bytes (2 to 12 MB a layer): what counts is the chain of trips to memory, barriers and shuffles.
//   * 128 threads; a warp takes 16 keys at a time and holds their K and V in registers exactly as the tensor core reads them — no shared
//     memory, no barrier.  The contraction does not care about the order of the dimensions, so a thread's 16-byte load of a K row is
//     four pairs of two consecutive K = 16 steps; the outputs' order is free too, so a 16-byte load of a V row serves eight column tiles.
//   * The cached rows were written by earlier steps: the first 16 keys of every warp are requested before the grid dependency is waited for, the
//     rest is prefetched into L2, and inside the loop a tile's K is replaced while its softmax runs, its V right after use.
//   * The step's own row never passes through memory: one warp of the CTA that owns it adds it as one more partial state.
//   * In a cluster every CTA stores its results straight into the shared memory of the CTA that finishes them: one barrier, no trip back.
// Measured, whole decode steps (this form against the one above): 36 layers of 32 / 8 heads of 128 behind 3000 rows 2.48 -> 2.28 ms a token, 32 such
// layers behind 512 rows 2.265 -> 2.232 ms, 24 layers of 64 / 8 heads of 64 behind 700 rows (half of them with a window of 128) 2.14 -> 2.12 ms; with
// sums added up outside the tensor core and the test for infinities (2.28 -> 2.30, the others within 0.4 %).
// The plain form takes a warp per key, five shuffles and two exponentials per key and head in a chain.  Tried: the cluster's results fetched by their
// readers instead of pushed (two barriers and a trip: 3 % of a step behind 512 rows); 64 registers in the projections, so that a CTA of this
// kernel fits beside theirs (their prologue spills: 48 against 36 ms for 16 tokens).
constexpr int kAttnTcThreads = 128, kAttnTcWarps = kAttnTcThreads / 32, kAttnTcTile = 16;
__host__ __device__ constexpr bool attn_tc_fits(int HD, int G) { return HD * ((G + 3) / 4) <= 128; }
__host__ __device__ inline size_t attn_tc_smem_bytes(int HD, int G) {
    return (size_t)(9 * HD + HD + 2 * (kAttnTcWarps + 1) * 8 + 4 + HD + (G + 3) / 4 * (HD / 16) * 128) * 4 + (size_t)(kAttnTcWarps + 1) * G * HD * 4 +
           (size_t)(G * HD + kMaxClusterSplits) * 16;
}
// cached rows of a split: [r0, r1), whole tiles except at the end
__device__ __forceinline__ void attn_tc_range(const AttnArgs& a, int split, int p, int* r0, int* r1) {
    const int lo = (a.window > 0 && p + 1 > a.window) ? p + 1 - a.window : 0;
    const int per = ((p - lo + a.n_splits - 1) / a.n_splits + kAttnTcTile - 1) / kAttnTcTile * kAttnTcTile;
    *r0 = min(p, lo + split * per);
    *r1 = min(p, *r0 + per);
}
// asks for rows [r0, r1) of a KV head to be brought into L2, one request per 128-byte line
template <int HD>
__device__ __forceinline__ void attn_tc_prefetch(const AttnArgs& a, int kvh, int r0, int r1, int tid, int threads) {
    constexpr int kLines = HD * 2 / 128;
    for (int i = tid; i < (r1 - r0) * 2 * kLines; i += threads) {
        const int r = r0 + i / (2 * kLines), w = i % (2 * kLines);
        const char* base = (const char*)(w < kLines ? a.k_cache : a.v_cache) + (kv_phys_row(a.pg, 0, 0, r) * a.n_kv + kvh) * (HD * 2) + (w % kLines) * 128;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(base));
    }
}
template <int HD> struct AttnTile { uint4 k[2][HD / 32], v[4][HD / 64]; };
template <int HD>
__device__ __forceinline__ void attn_tc_load_k(const AttnArgs& a, AttnTile<HD>& f, int kvh, int j0, int r1, int lane) {
#pragma unroll
    for (int x = 0; x < 2; x++) {
        const int row = j0 + 8 * x + (lane >> 2);
        const bool in = row < r1;
        const uint4* p = (const uint4*)((const __nv_bfloat16*)a.k_cache + (kv_phys_row(a.pg, 0, 0, in ? row : 0) * a.n_kv + kvh) * HD) + (lane & 3);
#pragma unroll
        for (int j = 0; j < HD / 32; j++) f.k[x][j] = in ? __ldcg(p + 4 * j) : make_uint4(0u, 0u, 0u, 0u);
    }
}
template <int HD>
__device__ __forceinline__ void attn_tc_load_v(const AttnArgs& a, AttnTile<HD>& f, int kvh, int j0, int r1, int lane) {
#pragma unroll
    for (int x = 0; x < 4; x++) {
        const int row = j0 + 8 * (x >> 1) + 2 * (lane & 3) + (x & 1);
        const bool in = row < r1;
        const uint4* p = (const uint4*)((const __nv_bfloat16*)a.v_cache + (kv_phys_row(a.pg, 0, 0, in ? row : 0) * a.n_kv + kvh) * HD) + (lane >> 2);
#pragma unroll
        for (int j = 0; j < HD / 64; j++) f.v[x][j] = in ? __ldcg(p + 8 * j) : make_uint4(0u, 0u, 0u, 0u);
    }
}
// Gains and biases of the heads this warp prepares (every T / 32nd: the group's queries, then the step's own key and value): they do not depend
// on the previous kernel either.
__host__ __device__ constexpr int attn_tc_heads(int T) { return (10 + T / 32 - 1) / (T / 32); }                  // up to 8 queries + key + value
template <int HD, int T> struct AttnPre { float gain[attn_tc_heads(T)][HD / 32], bias[attn_tc_heads(T)][HD / 32]; };
template <int HD, int T>
__device__ __forceinline__ void attn_tc_pre(const AttnArgs& a, AttnPre<HD, T>& pre, int kvh, int split, int warp, int lane) {
    const int G = a.n_q / a.n_kv;
#pragma unroll
    for (int k = 0; k < attn_tc_heads(T); k++) {
        const int h = warp + T / 32 * k;
        const bool in = h < G || (h < G + 2 && split == a.n_splits - 1);
        const void* gain = h < G ? a.q_gain : h == G ? a.k_gain : nullptr;
        const void* bias = h < G ? a.q_bias : h == G ? a.k_bias : a.v_bias;
        const int off = (h < G ? kvh * G + h : kvh) * HD;
#pragma unroll
        for (int i = 0; i < HD / 32; i++) {
            pre.gain[k][i] = in && gain ? gain_at(gain, a.gain_kind, lane + 32 * i) : 0.0f;
            pre.bias[k][i] = in && bias ? gain_at(bias, a.gain_kind, off + lane + 32 * i) : 0.0f;
        }
    }
}
__device__ __forceinline__ uint32_t attn_word(const uint4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Runs on exactly T threads (tid 0 ..) that synchronise on named barrier `bar_id`; `pre` holds this warp's heads' gains and biases.  AHEAD: `f` holds
// its first tile (attn_tc_load_*); otherwise it is loaded when the heads are ready.  Keys are taken by the first kAttnTcWarps warps.
template <int HD, int MT, bool CL, int T, bool AHEAD>
__device__ __forceinline__ void attn_tc_body(const AttnArgs& a, unsigned char* smem, AttnTile<HD>& f, const AttnPre<HD, T>& pre, int kvh, int split, int p, int tid, int bar_id,
                                             bool rope_ready) {
    constexpr int NW = kAttnTcWarps, NP = NW + 1, TW = T / 32, NH = attn_tc_heads(T), KS = HD / 16, NT = HD / 8, N = HD / 32;
    const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const bool second = g >= 4;
    const int G = a.n_q / a.n_kv;
    auto sync = [bar_id] { named_sync(bar_id, T); };
    float (*s_q)[HD] = (float (*)[HD])smem;                 // [9][HD]: rotated q heads; row G = this step's k
    float* s_v = (float*)smem + 9 * HD;                     // [HD]
    float (*s_m)[8] = (float (*)[8])(s_v + HD);             // [NP][8]: one state per warp, and the own row's
    float (*s_l)[8] = (float (*)[8])(s_v + HD + NP * 8);
    int& s_last = *(int*)(s_v + HD + 2 * NP * 8);
    float* s_rope = s_v + HD + 2 * NP * 8 + 4;              // [HD/2][2]: cos, sin
    uint4* s_a = (uint4*)(s_rope + HD);                     // [MT][KS][32]: the queries as the tensor core's first operand
    float* s_o = (float*)(s_a + MT * KS * 32);              // [NP][G][HD]
    float4* s_t = (float4*)(s_o + NP * G * HD);             // [splits][chunk]: the cluster's (max, sum, out) of the outputs this CTA finishes
    const size_t row_elems = (size_t)a.n_kv * HD;
    if (CL) cluster_arrive_release();                       // (waited for before the first store into another CTA: it has started)
    int r0, r1;
    attn_tc_range(a, split, p, &r0, &r1);
    const bool owns_new = split == a.n_splits - 1;
    const float scale = 1.0f / sqrtf((float)HD);

    // ---- this step's q heads of the group and, in the owner of the last split, its k and v: a warp per head, in registers (lane l holds the
    // elements l, l + 32, ..: the rotation's partner is in the next lane or in the same one)
    const int nheads = G + (owns_new ? 2 : 0);
    if (!rope_ready) attn_fill_rope<HD>(a, s_rope, p, tid);
    float x[NH][N];
#pragma unroll
    for (int k = 0; k < NH; k++) {
        const int h = warp + TW * k;
        if (h < nheads) {
            const float* src = h < G ? a.q + ((size_t)kvh * G + h) * HD : h == G ? a.k_new + (size_t)kvh * HD : a.v_new + (size_t)kvh * HD;
#pragma unroll
            for (int i = 0; i < N; i++) x[k][i] = __ldcg(src + lane + 32 * i);
        }
    }
    sync();                                                  // (the rotation table is there)
#pragma unroll
    for (int k = 0; k < NH; k++) {
        const int h = warp + TW * k;
        if (h < nheads) {
            if (h < G ? a.q_bias != nullptr : h == G ? a.k_bias != nullptr : a.v_bias != nullptr) {
#pragma unroll
                for (int i = 0; i < N; i++) x[k][i] = x[k][i] + pre.bias[k][i];
            }
            if (h > G) {
#pragma unroll
                for (int i = 0; i < N; i++) s_v[lane + 32 * i] = x[k][i];
            } else {
                if (h < G ? a.q_gain != nullptr : a.k_gain != nullptr) {
                    float ss = 0.0f;
#pragma unroll
                    for (int i = 0; i < N; i++) ss = fmaf(x[k][i], x[k][i], ss);
                    ss = warp_sum(ss);
                    const float inv = 1.0f / sqrtf(ss * (1.0f / (float)HD) + a.qk_eps);
#pragma unroll
                    for (int i = 0; i < N; i++) x[k][i] = (inv * x[k][i]) * pre.gain[k][i];
                }
                // separately rounded products and sums, as the graph's Mul / Add nodes produce them
                if (a.rope_style == 0) {
#pragma unroll
                    for (int i = 0; i < N; i++) {
                        const float cs = s_rope[2 * ((lane + 32 * i) >> 1)], sn = s_rope[2 * ((lane + 32 * i) >> 1) + 1];
                        const float other = __shfl_xor_sync(0xffffffffu, x[k][i], 1);
                        x[k][i] = (lane & 1) ? __fadd_rn(__fmul_rn(other, sn), __fmul_rn(x[k][i], cs))
                                             : __fadd_rn(__fmul_rn(x[k][i], cs), __fmul_rn(__fmul_rn(other, sn), -1.0f));
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < N / 2; i++) {
                        const float cs = s_rope[2 * (lane + 32 * i)], sn = s_rope[2 * (lane + 32 * i) + 1];
                        const float x0 = x[k][i], x1 = x[k][i + N / 2];
                        x[k][i] = __fsub_rn(__fmul_rn(x0, cs), __fmul_rn(x1, sn));
                        x[k][i + N / 2] = __fadd_rn(__fmul_rn(x1, cs), __fmul_rn(x0, sn));
                    }
                }
#pragma unroll
                for (int i = 0; i < N; i++) s_q[h][lane + 32 * i] = x[k][i];
            }
        }
    }
    sync();
    // queries -> operand: step ks of thread column t covers dimensions 32 (ks / 2) + 8 t + 4 (ks % 2) .. + 3
#pragma unroll 1
    for (int idx = tid; idx < MT * KS * 32; idx += T) {
        const int ln = idx & 31, ks = (idx >> 5) % KS, h = (idx >> 5) / KS * 4 + ((ln >> 2) & 3);
        const float4 q = h < G ? *(const float4*)&s_q[h][(ks >> 1) * 32 + (ln & 3) * 8 + (ks & 1) * 4] : make_float4(0.f, 0.f, 0.f, 0.f);
        uint4 w;
        attn_terms(q.x, q.y, ln >= 16, &w.x, &w.y);
        attn_terms(q.z, q.w, ln >= 16, &w.z, &w.w);
        s_a[idx] = w;
    }
    if (owns_new && warp == TW - 1) {
        // append this step's row to the cache; the rounded values are one more state: score, weight 1, value
        const size_t off = kv_phys_row(a.pg, 0, 0, p) * row_elems + (size_t)kvh * HD;
        float k[N], v[N];
#pragma unroll
        for (int i = 0; i < N; i++) {
            const __nv_bfloat16 kb = __float2bfloat16_rn(s_q[G][lane + 32 * i]), vb = __float2bfloat16_rn(s_v[lane + 32 * i]);
            ((__nv_bfloat16*)a.k_cache)[off + lane + 32 * i] = kb;
            ((__nv_bfloat16*)a.v_cache)[off + lane + 32 * i] = vb;
            k[i] = __bfloat162float(kb); v[i] = __bfloat162float(vb);
        }
#pragma unroll 1
        for (int h = 0; h < G; h++) {
            float d = 0.0f;
#pragma unroll
            for (int i = 0; i < N; i++) d = fmaf(s_q[h][lane + 32 * i], k[i], d);
            d = warp_sum(d);
            if (lane == 0) { s_m[NW][h] = d * scale; s_l[NW][h] = 1.0f; }
#pragma unroll
            for (int i = 0; i < N; i++) s_o[((size_t)NW * G + h) * HD + lane + 32 * i] = v[i];
        }
    }
    sync();

    // ---- the cached rows
    if (T == kAttnTcThreads || warp < NW) {
    if (!AHEAD) {
        attn_tc_load_k<HD>(a, f, kvh, r0 + warp * kAttnTcTile, r1, lane);
        attn_tc_load_v<HD>(a, f, kvh, r0 + warp * kAttnTcTile, r1, lane);
    }
    float o[MT][NT][2], mx[MT], l[MT];
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        mx[mt] = -INFINITY; l[mt] = 0.0f;
#pragma unroll
        for (int n = 0; n < NT; n++) o[mt][n][0] = o[mt][n][1] = 0.0f;
    }
#pragma unroll 1
    for (int j0 = r0 + warp * kAttnTcTile; j0 < r1; j0 += NW * kAttnTcTile) {
        AttnScore<KS> s[MT][2];
#pragma unroll
        for (int ks = 0; ks < KS; ks++) {
#pragma unroll
            for (int mt = 0; mt < MT; mt++) {
                const uint4 w = s_a[(mt * KS + ks) * 32 + lane];
                const uint32_t qa[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                for (int y = 0; y < 2; y++) attn_mma_score(s[mt][y], ks, qa, attn_word(f.k[y][ks >> 1], 2 * (ks & 1)), attn_word(f.k[y][ks >> 1], 2 * (ks & 1) + 1));
            }
        }
        const int jn = j0 + NW * kAttnTcTile;
        if (jn < r1) attn_tc_load_k<HD>(a, f, kvh, jn, r1, lane);
        const int j = j0 + 2 * t;                                     // this thread's keys: j, j + 1, j + 8, j + 9
        uint32_t pa[MT][4];
        float corr[MT];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float y = attn_score(s[mt][e >> 1], e & 1);
                v[e] = j + (e >> 1) * 8 + (e & 1) < r1 ? y * scale : -INFINITY;
            }
            float tm = fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3]));
            tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 1));
            tm = fmaxf(tm, __shfl_xor_sync(0xffffffffu, tm, 2));
            const float mn = fmaxf(mx[mt], tm);                       // a tile always holds at least one live key
            corr[mt] = mx[mt] == -INFINITY ? 0.0f : expf(mx[mt] - mn);
            mx[mt] = mn;
            float ps = 0.0f;
#pragma unroll
            for (int e = 0; e < 4; e++) { v[e] = v[e] == -INFINITY ? 0.0f : expf(v[e] - mn); ps += v[e]; }
            l[mt] = l[mt] * corr[mt] + ps;                            // per-lane partial sums, folded at the end
            attn_terms(v[0], v[1], second, &pa[mt][0], &pa[mt][1]);
            attn_terms(v[2], v[3], second, &pa[mt][2], &pa[mt][3]);
        }
        // column g of tile 8 jj + i is dimension 64 jj + 8 g + i
#pragma unroll
        for (int jj = 0; jj < HD / 64; jj++)
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const uint32_t sel = (i & 1) ? 0x7632u : 0x5410u;
                const uint32_t b0 = __byte_perm(attn_word(f.v[0][jj], i >> 1), attn_word(f.v[1][jj], i >> 1), sel);
                const uint32_t b1 = __byte_perm(attn_word(f.v[2][jj], i >> 1), attn_word(f.v[3][jj], i >> 1), sel);
#pragma unroll
                for (int mt = 0; mt < MT; mt++) attn_mma_value(o[mt][jj * 8 + i], corr[mt], pa[mt], b0, b1);
            }
        if (jn < r1) attn_tc_load_v<HD>(a, f, kvh, jn, r1, lane);
    }
    // ---- add up the terms' rows and the lanes' sums, then the warps
    float odd[2] = {0.0f, 0.0f};                            // sums of x * 0: 0, or NaN where something is not finite
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        const int h = mt * 4 + (g & 3);
        float lt = l[mt];
        lt += __shfl_xor_sync(0xffffffffu, lt, 1);
        lt += __shfl_xor_sync(0xffffffffu, lt, 2);
        if (t == 0 && !second) { s_m[warp][h] = mx[mt]; s_l[warp][h] = lt; }
        odd[0] = fmaf(mx[mt], 0.0f, odd[0]); odd[1] = fmaf(lt, 0.0f, odd[1]);
#pragma unroll
        for (int n = 0; n < NT; n++) {
            float x0 = o[mt][n][0], x1 = o[mt][n][1];
            x0 += __shfl_xor_sync(0xffffffffu, x0, 16);
            x1 += __shfl_xor_sync(0xffffffffu, x1, 16);
            odd[0] = fmaf(x0, 0.0f, odd[0]); odd[1] = fmaf(x1, 0.0f, odd[1]);
            float* dst = s_o + ((size_t)warp * G + h) * HD + (n >> 3) * 64 + 16 * t + (n & 7);
            if (!second && h < G) { dst[0] = x0; dst[8] = x1; }
        }
    }
    const int j_first = r0 + warp * kAttnTcTile;
    if (j_first < r1 && __any_sync(0xffffffffu, odd[0] + odd[1] != 0.0f))
        attn_plain_keys<HD>((const __nv_bfloat16*)a.k_cache + (size_t)kvh * HD, (const __nv_bfloat16*)a.v_cache + (size_t)kvh * HD, a.pg, 0, 0, row_elems, j_first, r1,
                            &s_q[0][0], G, lane, s_m[warp], s_l[warp], s_o + (size_t)warp * G * HD);
    }
    sync();
    const int parts = owns_new ? NP : NW;
    const int S = a.n_splits, total = G * HD, chunk = (total + S - 1) / S;      // outputs CTA r of the cluster finishes: [r * chunk, (r + 1) * chunk)
    if (CL) cluster_wait_acquire();
#pragma unroll 1
    for (int idx = tid; idx < total; idx += T) {
        const int h = idx / HD, e = idx - h * HD;
        float M = -INFINITY, L = 0.0f, O = 0.0f;
#pragma unroll
        for (int w = 0; w < NP; w++) if (w < parts) M = fmaxf(M, s_m[w][h]);
#pragma unroll
        for (int w = 0; w < NP; w++)
            if (w < parts) {
                const float c = s_m[w][h] == -INFINITY ? 0.0f : expf(s_m[w][h] - M);
                L = fmaf(s_l[w][h], c, L);
                O = fmaf(s_o[(size_t)w * G * HD + idx], c, O);
            }
        if (CL) {
            const int r = idx / chunk;
            const uint32_t dst = cluster_map(smem_u32(s_t + split * chunk + (idx - r * chunk)), (uint32_t)r);
            asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "f"(M), "f"(L), "f"(O), "f"(0.0f) : "memory");
        } else if (S == 1) {
            a.out[(size_t)kvh * total + idx] = attn_finish(O, M, L, a.sinks, a.gain_kind, kvh * G + h);      // no other split to merge with
        } else {
            float* dst = a.part + (((size_t)kvh * S + split) * G + h) * (HD + 2);
            dst[e] = O;
            if (e == 0) { dst[HD] = M; dst[HD + 1] = L; }
        }
    }
    if (CL) {
        cluster_arrive_release();
        cluster_wait_acquire();
        for (int oi = tid; oi < chunk && split * chunk + oi < total; oi += T) {
            // the ticket path's folding: batches of 8 splits into a running (max, sum, out)
            float M = -INFINITY, L = 0.0f, O = 0.0f;
#pragma unroll 1
            for (int s0 = 0; s0 < S; s0 += 8) {
                float4 v[8];
                float Mb = M;
#pragma unroll
                for (int j = 0; j < 8; j++) v[j] = s0 + j < S ? s_t[(s0 + j) * chunk + oi] : make_float4(-INFINITY, 0.f, 0.f, 0.f);
#pragma unroll
                for (int j = 0; j < 8; j++) Mb = fmaxf(Mb, v[j].x);
                const float c0 = (M == -INFINITY) ? 0.0f : expf(M - Mb);
                L *= c0; O *= c0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float c = (v[j].x == -INFINITY) ? 0.0f : expf(v[j].x - Mb);
                    L = fmaf(v[j].y, c, L);
                    O = fmaf(v[j].z, c, O);
                }
                M = Mb;
            }
            a.out[(size_t)kvh * total + split * chunk + oi] = attn_finish(O, M, L, a.sinks, a.gain_kind, kvh * G + (split * chunk + oi) / HD);
        }
    } else if (S > 1) {
        attn_merge_ticket<HD>(a, &s_last, kvh, G, tid, T, bar_id);
    }
}

}  // namespace lum
