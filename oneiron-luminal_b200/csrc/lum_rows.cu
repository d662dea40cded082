// Kernels around the tensor-core GEMM for steps that carry MORE THAN ONE row: a prompt's tokens (rows of one sequence at
// consecutive positions) or one token of each of several sequences (batched decode).  Every row has a token, a sequence
// and a position; the K/V cache holds `max_batch` sequences side by side.
//
// What they replace in the reference, which runs these ops for all `s` rows of a step
// (examples/llama/src/model.rs:91-113; launch ranges `[s]` / `[kv_heads, groups, s]`, model.rs:240-246):
//   embed_rows         `RowEmbed`  (crates/luminal_cuda/src/block/ops.rs:1921-1944)
//   rope_append_rows   `RowRope` on q and k (ops.rs:917-957; the graph's own formula: examples/llama/src/model.rs:128-163),
//                      Qwen's per-head RMSNorm (examples/qwen/src/model.rs:434-450) and the cache append that group 0 of the
//                      attention op performs (examples/llama/src/model.rs:388-402)
//   attn_rows          `LlamaAttention` / `QwenAttention` (examples/llama/src/model.rs:415-488): causal attention of each row
//                      over the cache rows of its sequence up to its own position
//   argmax_rows        `sample` per row (examples/llama/src/main.rs:137-148: last maximum wins)
// The arithmetic (rotation, norm, rounding to the cache type) is the decode kernels' (lum_attn_dev.cuh), so a cache row
// written here equals the row the single-token path writes for the same inputs.
#include "lum_attn_dev.cuh"
#include "lum_gemv_dev.cuh"
#include <cstdlib>

#include "lum_rows.cuh"

namespace lum {

// ---------------------------------------------------------------------------------------------------- embedding rows
__global__ void __launch_bounds__(256) embed_rows(const void* table, int kind, int H, int vocab, const int* row_tok, float* x, int ldx, int M,
                                                  const int* row_pos, const double* pos_freq, uint32_t* status) {
    const int m = blockIdx.x;
    if (m >= M) return;
    const int tok = row_tok[m];
    if (tok < 0 || tok >= vocab) {
        if (threadIdx.x == 0) atomicOr(status, LUM_ST_BAD_TOKEN);
        return;
    }
    embed_row_into(table, kind, H, tok, pos_freq, pos_freq ? row_pos[m] : 0, x + (size_t)m * ldx, threadIdx.x, 256);
}

// ---------------------------------------------------------------------------------------------------- RoPE + cache append
// A warp per head, eight heads of a row per CTA (they share the table of cosines and sines).  A row's q | k | v is the sum of the
// projection's K-split partial planes; q and k heads are RMS-normalised (Qwen; same operation order as the decode kernel) and
// rotated, q goes to q_rot, k and v are rounded to the cache type and stored at (sequence, position).  Lane l holds the elements
// l, l + 32, ..: the rotation's partner is in the next lane (adjacent pairs) or in the same one (split halves).
// Measured (32 rows of 32 + 2 x 8 heads of 128): 11.7 us with one CTA of 256 threads per row, 5.0 us this way — the kernel
// is a chain of trips to L2, and a row's 48 warps take them side by side.
template <int HD>
__global__ void __launch_bounds__(256) rope_append_rows(const RopeRowsArgs a) {
    constexpr int N = HD / 32;
    __shared__ float2 tab[HD / 2];                       // cos, sin
    const int tid = threadIdx.x, lane = tid & 31;
    const int nq = a.n_q, nkv = a.n_kv, heads = nq + 2 * nkv, W = heads * HD;
    const int per_row = (heads + 7) / 8, m = blockIdx.x / per_row, h = (blockIdx.x - m * per_row) * 8 + (tid >> 5);
    if (a.use_pdl) { pdl_launch_dependents(); pdl_grid_wait(); }
    const int pos = a.row_pos[m];
    const int seq = a.row_seq ? a.row_seq[m] : a.seq0;
    if (pos < 0 || pos >= a.max_seq || seq < 0 || seq >= a.max_batch) {
        if (h == 0 && lane == 0) atomicOr(a.status, LUM_ST_BAD_POS);
        return;                                          // (the whole CTA: its warps share a row)
    }
    float x[N];
#pragma unroll
    for (int i = 0; i < N; i++) x[i] = 0.0f;
    const float* src = a.qkv + (size_t)m * W + (size_t)(h < heads ? h : 0) * HD + lane;
#pragma unroll 4
    for (int p = 0; p < a.n_parts; p++)
#pragma unroll
        for (int i = 0; i < N; i++) x[i] += __ldcg(src + p * a.part_stride + 32 * i);
    if (tid < HD / 2) {
        AttnArgs t{};
        t.rope_style = a.rope_style; t.c_inv_d = a.c_inv_d; t.c_ln_theta = a.c_ln_theta; t.c_log2e = a.c_log2e; t.c_half_pi = a.c_half_pi;
        t.theta = a.theta; t.hd = HD;
        float cs, sn;
        rope_cs<-1>(t, tid, pos, &cs, &sn);
        tab[tid] = make_float2(cs, sn);
    }
    __syncthreads();
    if (h >= heads) return;
    if (h < nq + nkv) {
        const void* gain = h < nq ? a.q_gain : a.k_gain;
        if (gain) {
            float ss = 0.0f;
#pragma unroll
            for (int i = 0; i < N; i++) ss = fmaf(x[i], x[i], ss);
            ss = warp_sum(ss);
            const float inv = 1.0f / sqrtf(ss * (1.0f / (float)HD) + a.qk_eps);
#pragma unroll
            for (int i = 0; i < N; i++) x[i] = (inv * x[i]) * gain_at(gain, a.gain_kind, lane + 32 * i);
        }
        if (a.rope_style == 0) {
#pragma unroll
            for (int i = 0; i < N; i++) {
                const float2 c = tab[(lane + 32 * i) >> 1];
                const float other = __shfl_xor_sync(0xffffffffu, x[i], 1);
                x[i] = (lane & 1) ? __fadd_rn(__fmul_rn(other, c.y), __fmul_rn(x[i], c.x))
                                  : __fadd_rn(__fmul_rn(x[i], c.x), __fmul_rn(__fmul_rn(other, c.y), -1.0f));
            }
        } else {
#pragma unroll
            for (int i = 0; i < N / 2; i++) {
                const float2 c = tab[lane + 32 * i];
                const float x0 = x[i], x1 = x[i + N / 2];
                x[i] = __fsub_rn(__fmul_rn(x0, c.x), __fmul_rn(x1, c.y));
                x[i + N / 2] = __fadd_rn(__fmul_rn(x1, c.x), __fmul_rn(x0, c.y));
            }
        }
    }
    if (h < nq) {
        float* dst = a.q_rot + ((size_t)m * nq + h) * HD + lane;
#pragma unroll
        for (int i = 0; i < N; i++) dst[32 * i] = x[i];
        return;
    }
    const bool is_k = h < nq + nkv;
    void* cache = is_k ? a.k_cache : a.v_cache;
    const size_t off = kv_phys_row(a.pg, seq, a.max_seq, pos) * ((size_t)nkv * HD) + (size_t)(h - nq - (is_k ? 0 : nkv)) * HD + lane;
#pragma unroll
    for (int i = 0; i < N; i++) {
        if (a.kv_bf16) ((__nv_bfloat16*)cache)[off + 32 * i] = __float2bfloat16_rn(x[i]);
        else ((float*)cache)[off + 32 * i] = x[i];
    }
}

// ---------------------------------------------------------------------------------------------------- attention over the cache
// One CTA per (KV head, row): 8 warps take the cached positions lo .. pos of the row's sequence in turn (the row's own
// position was appended before this kernel runs); all G query heads of the group share each K/V read; lanes split the
// head dimension.  Online softmax per warp, merged in shared memory.
template <int HD, int GM, bool BF16>
__global__ void __launch_bounds__(256) attn_rows(const AttnRowsArgs a) {
    constexpr int DPL = HD / 32, NW = 8;
    __shared__ float s_m[NW][GM], s_l[NW][GM];
    __shared__ float s_o[NW][GM][HD];
    const int kvh = blockIdx.x, m = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int G = a.n_q / a.n_kv;
    const int pos = a.row_pos[m];
    const int seq = a.row_seq ? a.row_seq[m] : a.seq0;
    if (pos < 0 || pos >= a.max_seq || seq < 0 || seq >= a.max_batch) return;       // flagged by the append kernel
    const int lo = (a.window > 0 && pos + 1 > a.window) ? pos + 1 - a.window : 0;
    const size_t row_elems = (size_t)a.n_kv * HD;
    const size_t base = (size_t)kvh * HD + lane * DPL;
    auto row_off = [&](int r) { return base + kv_phys_row(a.pg, seq, a.max_seq, r) * row_elems; };
    const float scale = 1.0f / sqrtf((float)HD);
    float q[GM][DPL], o[GM][DPL], mx[GM], l[GM];
#pragma unroll
    for (int g = 0; g < GM; g++) {
        mx[g] = -INFINITY; l[g] = 0.0f;
#pragma unroll
        for (int i = 0; i < DPL; i++) {
            q[g][i] = g < G ? a.q_rot[(size_t)m * a.n_q * HD + ((size_t)kvh * G + g) * HD + lane * DPL + i] : 0.0f;
            o[g][i] = 0.0f;
        }
    }
    using Raw = typename RawRow<BF16, DPL>::type;
    Raw kn = Raw(), vn = Raw();
    int j = lo + warp;
    if (j <= pos) {
        kn = raw_load<BF16, DPL>(a.k_cache, row_off(j));
        vn = raw_load<BF16, DPL>(a.v_cache, row_off(j));
    }
#pragma unroll 1
    for (; j <= pos; j += NW) {
        float kr[DPL], vr[DPL];
        const Raw kc = kn, vc = vn;
        if (j + NW <= pos) {
            kn = raw_load<BF16, DPL>(a.k_cache, row_off(j + NW));
            vn = raw_load<BF16, DPL>(a.v_cache, row_off(j + NW));
        }
        raw_to_float<BF16, DPL>(kc, kr);
        raw_to_float<BF16, DPL>(vc, vr);
#pragma unroll
        for (int g = 0; g < GM; g++) {
            if (g < G) {
                float d = 0.0f;
#pragma unroll
                for (int i = 0; i < DPL; i++) d = fmaf(q[g][i], kr[i], d);
                d = warp_sum(d);
                const float logit = d * scale;
                const float mn = fmaxf(mx[g], logit);
                const float corr = (mx[g] == -INFINITY) ? 0.0f : expf(mx[g] - mn);
                const float w = expf(logit - mn);
                l[g] = l[g] * corr + w;
#pragma unroll
                for (int i = 0; i < DPL; i++) o[g][i] = fmaf(w, vr[i], o[g][i] * corr);
                mx[g] = mn;
            }
        }
    }
#pragma unroll
    for (int g = 0; g < GM; g++) {
        if (g < G) {
            if (lane == 0) { s_m[warp][g] = mx[g]; s_l[warp][g] = l[g]; }
#pragma unroll
            for (int i = 0; i < DPL; i++) s_o[warp][g][lane * DPL + i] = o[g][i];
        }
    }
    __syncthreads();
    for (int idx = tid; idx < G * HD; idx += 256) {
        const int g = idx / HD, e = idx - g * HD;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < NW; w++) M = fmaxf(M, s_m[w][g]);
        float L = 0.0f, O = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const float c = (s_m[w][g] == -INFINITY) ? 0.0f : expf(s_m[w][g] - M);
            L = fmaf(s_l[w][g], c, L);
            O = fmaf(s_o[w][g][e], c, O);
        }
        a.out[(size_t)m * a.n_q * HD + ((size_t)kvh * G + g) * HD + e] = O * (1.0f / L);
    }
}

// The same attention for rows of a bfloat16 cache: batched decode (every row its own sequence with a long context), and the rows of a
// prompt that do not take the tcgen05 kernel.  Bound by the cache's bytes.  What counts is how many of them are on their way and how
// few instructions a key costs:
//   * a cluster of CTAs per (KV head, row), one CTA per split of the cached positions, four warps per CTA.  Warps do not wait for
//     each other: each takes 16 keys at a time and fetches their K and V (cp.async, coalesced 16-byte pieces, rows swizzled so that
//     ldmatrix reads them without bank conflicts) into its own ring in shared memory, ar_stages - 1 tiles ahead.
//   * both products are tensor-core instructions over three bf16 terms of the f32 operand (attn_terms), whose 24 bits they keep; what goes
//     beyond one instruction is added up in f32 (attn_mma).
//   * warps merge in shared memory, splits through the cluster's distributed shared memory: no partial results in global memory and no
//     second kernel.
// Measured (32 sequences x 2049 keys, 8 KV heads x 4 query heads, head dimension 128; 268 MB of cache): 53.4 us with sums left in the
// tensor core, 55.4 us this way.  The form before it, with
// a lane per key and the products on CUDA cores (1700 instructions per warp and 32 keys, 16-byte loads 2 KiB apart), took 147 us and
// 6 us more to merge.
__device__ __forceinline__ void ar_ldsm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ar_ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ar_cp16(uint32_t dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
constexpr int kArTile = 16;                                        // keys per warp and step
__host__ __device__ constexpr int ar_stages(int hd) { return hd == 128 ? 2 : 3; }
__host__ __device__ constexpr int ar_smem(int hd) { return 4 * ar_stages(hd) * 2 * kArTile * hd * 2; }

// MT: groups of four query heads (G <= 4 MT)
template <int HD, int MT>
__global__ void __launch_bounds__(128, 3) attn_rows_split(const AttnRowsArgs a, int n_splits) {
    constexpr int NW = 4, NT = HD / 8, KS = HD / 16, CH = HD / 8, GM = 4 * MT, NS = ar_stages(HD);
    constexpr int kSide = kArTile * HD * 2, kStage = 2 * kSide;     // bytes of one tile's K (or V); of both
    extern __shared__ __align__(128) unsigned char ar_sm[];
    static_assert((NW * GM * HD + GM * HD + 2 * NW * GM + 2 * GM) * 4 <= ar_smem(HD), "the merge reuses the ring");
    const int kvh = blockIdx.x, m = blockIdx.y, sp = blockIdx.z, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = lane >> 2, t = lane & 3;                           // row and column group of the fragments
    const bool second = g >= 4;
    const int G = a.n_q / a.n_kv;
    if (a.use_pdl) { pdl_launch_dependents(); pdl_grid_wait(); }
    const int pos = a.row_pos[m];
    const int seq = a.row_seq ? a.row_seq[m] : a.seq0;
    if (pos < 0 || pos >= a.max_seq || seq < 0 || seq >= a.max_batch) return;       // flagged by the append kernel (the whole cluster returns)
    const int n_keys = pos + 1;
    const int per = ((n_keys + n_splits - 1) / n_splits + 63) & ~63;                // keys per split, whole steps of the four warps
    const int k0 = sp * per, k1 = min(n_keys, k0 + per);
    const size_t row_elems = (size_t)a.n_kv * HD;
    const __nv_bfloat16* kc = (const __nv_bfloat16*)a.k_cache + (size_t)kvh * HD;
    const __nv_bfloat16* vc = (const __nv_bfloat16*)a.v_cache + (size_t)kvh * HD;
    const float scale = 1.0f / sqrtf((float)HD);
    const uint32_t ring = smem_u32(ar_sm) + (uint32_t)warp * (NS * kStage);
    const int j_first = k0 + warp * kArTile;
    const int n_it = j_first < k1 ? (k1 - j_first + 63) / 64 : 0;

    auto load = [&](int i) {
        if (i < n_it) {
            const int j0 = j_first + 64 * i;
            // the tile's 16 keys start on a multiple of 16: one sequence slot or one page holds them all
            const size_t base = kv_phys_row(a.pg, seq, a.max_seq, j0);
            const uint32_t dst = ring + (uint32_t)(i % NS) * kStage;
#pragma unroll
            for (int x = 0; x < kArTile * CH / 32; x++) {
                const int r = (x * 32 + lane) / CH, c = (x * 32 + lane) % CH;
                const bool in = j0 + r < k1;                          // rows past the end read as zeros
                const size_t off = (base + (in ? r : 0)) * row_elems + c * 8;
                const uint32_t d = dst + (uint32_t)(r * HD * 2 + ((c ^ (r & 7)) << 4));
                ar_cp16(d, kc + off, in ? 16u : 0u);
                ar_cp16(d + kSide, vc + off, in ? 16u : 0u);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < NS - 1; i++) load(i);

    uint32_t qa[MT][KS][4];
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        const int h = mt * 4 + (g & 3);
        const float* q = a.q_rot + (size_t)m * a.n_q * HD + ((size_t)kvh * G + h) * HD + 2 * t;
#pragma unroll
        for (int ks = 0; ks < KS; ks++)
#pragma unroll
            for (int e = 0; e < 2; e++) {
                const float2 v = h < G ? *(const float2*)(q + ks * 16 + e * 8) : make_float2(0.0f, 0.0f);
                attn_terms(v.x, v.y, second, &qa[mt][ks][2 * e], &qa[mt][ks][2 * e + 1]);
            }
    }
    float o[MT][NT][2], mx[MT], l[MT];
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        mx[mt] = -INFINITY; l[mt] = 0.0f;
#pragma unroll
        for (int n = 0; n < NT; n++) o[mt][n][0] = o[mt][n][1] = 0.0f;
    }
    const int kkey = ((lane >> 4) << 3) + (lane & 7), kch = (lane >> 3) & 1;       // this lane's row and 16-byte group in a ldmatrix of K ...
    const int vkey = (((lane >> 3) & 1) << 3) + (lane & 7), vch = lane >> 4;        // ... and of V
#pragma unroll 1
    for (int i = 0; i < n_it; i++) {
        load(i + NS - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(NS - 1) : "memory");
        __syncwarp();
        const uint32_t kb = ring + (uint32_t)(i % NS) * kStage, vb = kb + kSide;
        AttnScore<KS> s[MT][2];
#pragma unroll
        for (int ks = 0; ks < KS; ks++) {
            uint32_t b[4];
            ar_ldsm4(kb + (uint32_t)(kkey * HD * 2 + (((ks * 2 + kch) ^ (kkey & 7)) << 4)), b);
#pragma unroll
            for (int mt = 0; mt < MT; mt++) { attn_mma_score(s[mt][0], ks, qa[mt][ks], b[0], b[1]); attn_mma_score(s[mt][1], ks, qa[mt][ks], b[2], b[3]); }
        }
        const int j = j_first + 64 * i + 2 * t;                       // this thread's keys: j, j + 1, j + 8, j + 9
        uint32_t pa[MT][4];
        float corr[MT];
#pragma unroll
        for (int mt = 0; mt < MT; mt++) {
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const float x = attn_score(s[mt][e >> 1], e & 1);
                v[e] = j + (e >> 1) * 8 + (e & 1) < k1 ? x * scale : -INFINITY;
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
#pragma unroll
        for (int np = 0; np < NT / 2; np++) {
            uint32_t b[4];
            ar_ldsm4_t(vb + (uint32_t)(vkey * HD * 2 + (((np * 2 + vch) ^ (vkey & 7)) << 4)), b);
#pragma unroll
            for (int mt = 0; mt < MT; mt++) { attn_mma_value(o[mt][2 * np], corr[mt], pa[mt], b[0], b[1]); attn_mma_value(o[mt][2 * np + 1], corr[mt], pa[mt], b[2], b[3]); }
        }
        __syncwarp();
    }
    // ---- add up the terms' rows and the lanes' sums, then the warps
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float* s_o = (float*)ar_sm;                    // [NW][GM][HD]
    float* s_f = s_o + NW * GM * HD;               // [GM][HD]: this CTA's split
    float* s_m = s_f + GM * HD;                    // [NW][GM]
    float* s_l = s_m + NW * GM;                    // [NW][GM]
    float* s_fm = s_l + NW * GM;                   // [GM]
    float* s_fl = s_fm + GM;                       // [GM]
    float odd[2] = {0.0f, 0.0f};                   // sums of x * 0: 0, or NaN where something is not finite
#pragma unroll
    for (int mt = 0; mt < MT; mt++) {
        const int h = mt * 4 + (g & 3);
        float lt = l[mt];
        lt += __shfl_xor_sync(0xffffffffu, lt, 1);
        lt += __shfl_xor_sync(0xffffffffu, lt, 2);
        if (t == 0 && !second) { s_m[warp * GM + h] = mx[mt]; s_l[warp * GM + h] = lt; }
        odd[0] = fmaf(mx[mt], 0.0f, odd[0]); odd[1] = fmaf(lt, 0.0f, odd[1]);
#pragma unroll
        for (int n = 0; n < NT; n++) {
            float x0 = o[mt][n][0], x1 = o[mt][n][1];
            x0 += __shfl_xor_sync(0xffffffffu, x0, 16);
            x1 += __shfl_xor_sync(0xffffffffu, x1, 16);
            odd[0] = fmaf(x0, 0.0f, odd[0]); odd[1] = fmaf(x1, 0.0f, odd[1]);
            if (!second) *(float2*)(s_o + (warp * GM + h) * HD + n * 8 + 2 * t) = make_float2(x0, x1);
        }
    }
    if (n_it > 0 && __any_sync(0xffffffffu, odd[0] + odd[1] != 0.0f))
        attn_plain_keys<HD>(kc, vc, a.pg, seq, a.max_seq, row_elems, j_first, k1, a.q_rot + ((size_t)m * a.n_q + (size_t)kvh * G) * HD, G, lane, s_m + warp * GM,
                            s_l + warp * GM, s_o + warp * GM * HD);
    __syncthreads();
    float* out = a.out + ((size_t)m * a.n_q + (size_t)kvh * G) * HD;
    for (int idx = tid; idx < G * HD; idx += 128) {
        const int h = idx / HD;
        float M = -INFINITY;
#pragma unroll
        for (int w = 0; w < NW; w++) M = fmaxf(M, s_m[w * GM + h]);
        float L = 0.0f, O = 0.0f;
#pragma unroll
        for (int w = 0; w < NW; w++) {
            const float c = s_m[w * GM + h] == -INFINITY ? 0.0f : expf(s_m[w * GM + h] - M);
            L = fmaf(s_l[w * GM + h], c, L);
            O = fmaf(s_o[w * GM * HD + idx], c, O);
        }
        if (n_splits == 1) out[idx] = O * (1.0f / L);
        else {
            s_f[idx] = O;
            if (idx % HD == 0) { s_fm[h] = M; s_fl[h] = L; }            // a split without keys leaves M = -inf, L = 0
        }
    }
    if (n_splits == 1) return;
    cluster_arrive_release();
    cluster_wait_acquire();
    for (int idx = sp * 128 + tid; idx < G * HD; idx += n_splits * 128) {
        const int h = idx / HD;
        float M = -INFINITY;
        for (int r = 0; r < n_splits; r++) M = fmaxf(M, cluster_ld_f32(cluster_map(smem_u32(s_fm + h), (uint32_t)r)));
        float L = 0.0f, O = 0.0f;
        for (int r = 0; r < n_splits; r++) {
            const float ms = cluster_ld_f32(cluster_map(smem_u32(s_fm + h), (uint32_t)r));
            const float c = ms == -INFINITY ? 0.0f : expf(ms - M);
            L = fmaf(cluster_ld_f32(cluster_map(smem_u32(s_fl + h), (uint32_t)r)), c, L);
            O = fmaf(cluster_ld_f32(cluster_map(smem_u32(s_f + idx), (uint32_t)r)), c, O);
        }
        out[idx] = O * (1.0f / L);
    }
    cluster_arrive_release();                       // nobody leaves while another CTA may still read its shared memory
    cluster_wait_acquire();
}

// ---------------------------------------------------------------------------------------------------- greedy sample per row
// One CTA per row: logits[m][:] = sum of the vocabulary projection's partial planes (written back to plane 0), the greedy
// sample (last maximum wins), and the bookkeeping of a batched decode step: the sample becomes the row's next token, its
// position advances, and the token is logged.
__global__ void __launch_bounds__(1024) argmax_rows(const ArgmaxRowsArgs a) {
    __shared__ float s_v[32];
    __shared__ int s_i[32];
    const int m = blockIdx.x, tid = threadIdx.x;
    if (a.use_pdl) { pdl_launch_dependents(); pdl_grid_wait(); }
    if (m >= a.M) return;
    float* plane0 = a.logits + (size_t)m * a.vocab;
    ArgBest b{-INFINITY, -1};
    // eight elements per thread and plane on their way at once: a row is read by one CTA, and the trips to L2 are what it waits for
    // (128256 elements: 27.6 us with one element per thread and 512 threads, 22.1 us)
    constexpr int T = 1024, U = 8;
    for (int i0 = tid; i0 < a.vocab; i0 += T * U) {
        float v[U];
#pragma unroll
        for (int u = 0; u < U; u++) v[u] = i0 + u * T < a.vocab ? __ldcg(plane0 + i0 + u * T) : 0.0f;
        for (int p = 1; p < a.n_parts; p++)
#pragma unroll
            for (int u = 0; u < U; u++)
                if (i0 + u * T < a.vocab) v[u] += __ldcg(plane0 + p * a.part_stride + i0 + u * T);
#pragma unroll
        for (int u = 0; u < U; u++)
            if (i0 + u * T < a.vocab) {
                if (a.n_parts > 1) plane0[i0 + u * T] = v[u];
                argbest_take(b, v[u], i0 + u * T);
            }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, b.v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, b.i, o);
        argbest_take(b, ov, oi);
    }
    if ((tid & 31) == 0) { s_v[tid >> 5] = b.v; s_i[tid >> 5] = b.i; }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < 32; w++) argbest_take(b, s_v[w], s_i[w]);
        const int tok = b.i < 0 ? 0 : b.i;
        if (a.best) a.best[m] = tok;
        if (a.row_tok) a.row_tok[m] = tok;
        if (a.row_pos) a.row_pos[m] += 1;
        if (a.log && a.step) {
            const int s = *a.step;                       // advanced by row 0's CTA of the NEXT step's first kernel
            if (s < a.max_steps) a.log[(size_t)s * a.M + m] = tok;
        }
    }
}
// advances the batched decode's step counter (a kernel of its own: every row's CTA of argmax_rows reads the old value)
__global__ void step_advance(int* step) { *step += 1; }

// ---------------------------------------------------------------------------------------------------- launchers

cudaError_t launch_embed_rows(const void* table, int kind, int H, int vocab, const int* row_tok, float* x, int M, uint32_t* status, cudaStream_t st) {
    embed_rows<<<M, 256, 0, st>>>(table, kind, H, vocab, row_tok, x, H, M, nullptr, nullptr, status);
    return cudaGetLastError();
}
cudaError_t launch_embed_rows_sinusoid(const void* table, int kind, int H, int vocab, const int* row_tok, const int* row_pos, const double* pos_freq, float* x, int ldx,
                                       int M, uint32_t* status, cudaStream_t st) {
    embed_rows<<<M, 256, 0, st>>>(table, kind, H, vocab, row_tok, x, ldx, M, row_pos, pos_freq, status);
    return cudaGetLastError();
}

static cudaError_t launch_rows_pdl(const void* fn, dim3 grid, dim3 block, void** params, int use_pdl, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = use_pdl ? 1 : 0;
    return cudaLaunchKernelExC(&cfg, fn, params);
}

cudaError_t launch_rope_append_rows(const RopeRowsArgs& a, cudaStream_t st) {
    const void* fn = a.hd == 128 ? (const void*)rope_append_rows<128> : a.hd == 64 ? (const void*)rope_append_rows<64> : nullptr;
    if (!fn) return cudaErrorInvalidValue;
    RopeRowsArgs b = a;
    void* params[] = {&b};
    return launch_rows_pdl(fn, dim3((unsigned)(a.M * ((a.n_q + 2 * a.n_kv + 7) / 8))), dim3(256), params, a.use_pdl, st);
}

cudaError_t launch_attn_rows(const AttnRowsArgs& a, int sm_count, cudaStream_t st) {
    const int G = a.n_kv > 0 ? a.n_q / a.n_kv : 0;
    static const int env_split = [] { const char* e = getenv("LUM_ATTN_ROWS_SPLIT"); return e ? atoi(e) : 1; }();
    if (env_split && a.kv_bf16 && a.window == 0 && (a.hd == 128 || a.hd == 64) && G >= 1 && G <= (a.hd == 128 ? 4 : 8) && (((uintptr_t)a.k_cache | (uintptr_t)a.v_cache) & 15) == 0 &&
        ((size_t)a.n_kv * a.hd * 2) % 16 == 0) {
        const void* fn = a.hd == 128 ? (const void*)attn_rows_split<128, 1> : (G <= 4 ? (const void*)attn_rows_split<64, 1> : (const void*)attn_rows_split<64, 2>);
        const size_t smem = (size_t)ar_smem(a.hd);
        if (smem > 48 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
        // Splits per (KV head, row): rounds of resident CTAs (three per SM: what the ring of a 128-dimension head and the registers allow; counted for
        // the others too) times the keys of one, plus what a CTA costs beside its keys — about the time of 100 of them.  The positions are on
        // the device, so a context of middling length (1024 keys) stands for all.
        const long long pairs = (long long)a.n_kv * a.M, slots = 3ll * sm_count;
        int splits = 1;
        for (int s = 2; s <= kAttnRowsMaxSplits; s++) {
            auto cost = [&](int n) { return (double)((pairs * n + slots - 1) / slots) * (1024.0 / n + 100.0); };
            if (cost(s) < cost(splits)) splits = s;
        }
        AttnRowsArgs b = a;
        void* params[] = {&b, &splits};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(a.n_kv, a.M, splits);
        cfg.blockDim = dim3(128);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute at[2];
        int n_at = 0;
        if (splits > 1) {
            at[n_at].id = cudaLaunchAttributeClusterDimension;
            at[n_at].val.clusterDim.x = 1; at[n_at].val.clusterDim.y = 1; at[n_at].val.clusterDim.z = (unsigned)splits;
            n_at++;
        }
        if (a.use_pdl) {
            at[n_at].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[n_at].val.programmaticStreamSerializationAllowed = 1;
            n_at++;
        }
        cfg.attrs = at;
        cfg.numAttrs = n_at;
        return cudaLaunchKernelExC(&cfg, fn, params);
    }
    const void* fn = nullptr;
    const bool bf = a.kv_bf16 != 0;
    if (a.hd == 128 && G >= 1 && G <= 4) fn = bf ? (const void*)attn_rows<128, 4, true> : (const void*)attn_rows<128, 4, false>;
    else if (a.hd == 64 && G >= 1 && G <= 4) fn = bf ? (const void*)attn_rows<64, 4, true> : (const void*)attn_rows<64, 4, false>;
    else if (a.hd == 64 && G <= 8) fn = bf ? (const void*)attn_rows<64, 8, true> : (const void*)attn_rows<64, 8, false>;
    if (!fn) return cudaErrorInvalidValue;
    AttnRowsArgs b = a;
    void* params[] = {&b};
    return cudaLaunchKernel(fn, dim3(a.n_kv, a.M), dim3(256), params, 0, st);
}

cudaError_t launch_argmax_rows(const ArgmaxRowsArgs& a, cudaStream_t st) {
    ArgmaxRowsArgs b = a;
    void* params[] = {&b};
    return launch_rows_pdl((const void*)argmax_rows, dim3(a.M), dim3(1024), params, a.use_pdl, st);
}
cudaError_t launch_step_advance(int* step, cudaStream_t st) {
    step_advance<<<1, 1, 0, st>>>(step);
    return cudaGetLastError();
}

}  // namespace lum
