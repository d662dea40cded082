// Q8_0 products of two to five rows: batched steps of a few sequences, the shortest prompts.  Between the matrix-vector kernel (lum_gemv.cu) and the
// products of up to 64 rows (lum_gemm.cu): there is still so little to do per weight that HBM should be the bound, but converting every weight to two binary16
// operands, as the larger products do, takes longer than HBM takes to deliver it.  So the rows are written as three int8 levels per 32-block, like the vector of
// the matrix-vector kernel, and the weights go to the tensor core as they are (mma.sync m16n8k32, exact int32 sums).
//
//  * rows_levels — forms the rows (sum of the previous product's planes, residual, norm or SwiGLU) and writes the levels in operand order.
//  * q8_few — one CTA per SM: a producer warp keeps two rings of weight tiles full (lum_gemv_dev.cuh), two groups of eight consumer warps take pairs of row
//    groups in turn, a warp the same tile of both.  An instruction multiplies one block of the pair's 16 rows by eight columns, a column
//    being one level of one row of x.  The levels of all rows' columns (a K range of at most 4096) lie in shared memory.
#include <algorithm>

#include "lum_gemv_dev.cuh"
#include "lum_rows.cuh"

namespace lum {

constexpr int kFewRows = kFewMax;                    // rows at most: three levels of five rows are 15 of 16 columns, and their levels leave room for eight stages
constexpr int kFewStages = 4;                        // per ring, two for each group of consumers: a group sees every phase of its own stages
constexpr int kFewThreads = 2 * kConsumers + 32;
constexpr int kFewBar = kBarBytes;

__host__ __device__ inline int few_tiles(int M) { return (3 * M + 7) / 8; }      // eight columns of the operand each

// ---------------------------------------------------------------------------------------------------------------- rows
// Operand: per pair of blocks and eight columns 512 bytes, lane (column % 8, t) having words t and t + 4 of the even block, then of the odd one (the B operand of
// m16n8k32).  Row m's levels are columns 3 m, 3 m + 1, 3 m + 2 of tiles = ceil(3 M / 8) groups of eight.  Scales: [K / 32][8 tiles], the levels' factors included.
// A cluster of C CTAs forms one row, like rows_quantize; a block's scale is its own, so only the norm's sum of squares goes round.
__global__ void __launch_bounds__(256) rows_levels(const RowsArgs a, const int C) {
    extern __shared__ __align__(16) float rowbuf[];          // this CTA's columns (behind a norm)
    __shared__ float scratch[8], s_x;
    const int part = blockIdx.x % C, m = blockIdx.x / C, tid = threadIdx.x;
    const int K = a.K, nb = K >> 5;
    const int s0 = (int)((long long)nb * part / C), s1 = (int)((long long)nb * (part + 1) / C);     // this CTA's blocks
    const int k0 = s0 << 5, n4 = (s1 - s0) << 3;
    if (a.use_pdl) { pdl_launch_dependents(); pdl_grid_wait(); }
    const int tiles = few_tiles(a.M);
    // eight consecutive threads own a block: four of its columns each
    auto store = [&](int f4, float4 v) {
        const float e[4] = {v.x, v.y, v.z, v.w};
        uint32_t p[3];
        const float s1 = gemv_levels(e, p);
        if (f4 < n4) {
            const int blk = s0 + (f4 >> 3), j = f4 & 7;
#pragma unroll
            for (int l = 0; l < 3; l++) {
                const int c = 3 * m + l;
                *(uint32_t*)(a.xq + ((size_t)(blk >> 1) * tiles + (c >> 3)) * 512 + ((c & 7) * 4 + (j & 3)) * 16 + (blk & 1) * 8 + (j >> 2) * 4) = p[l];
                if (j == 0) a.sx[((size_t)blk * tiles + (c >> 3)) * 8 + (c & 7)] = s1 * (l == 0 ? 1.0f : l == 1 ? 1.0f / 254.0f : 1.0f / 64516.0f);
            }
        }
    };
    float ss = 0.0f;
    for (int b = 0; b < n4; b += 256) {
        const int f4 = b + tid;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f), u = v;
        if (f4 < n4) {
            const size_t at = (size_t)m * a.ld + k0 + f4 * 4;
#pragma unroll 4
            for (int p = 0; p < a.n_parts; p++) {
                const float4 t = __ldcg((const float4*)(a.a + p * a.part_stride + at));
                v.x += t.x; v.y += t.y; v.z += t.z; v.w += t.w;
                if (a.b) {
                    const float4 s = __ldcg((const float4*)(a.b + p * a.part_stride + at));
                    u.x += s.x; u.y += s.y; u.z += s.z; u.w += s.w;
                }
            }
            if (a.b) { v.x = swiglu(v.x, u.x); v.y = swiglu(v.y, u.y); v.z = swiglu(v.z, u.z); v.w = swiglu(v.w, u.w); }
            if (a.resid) {
                const float4 r = __ldcg((const float4*)(a.resid + (size_t)m * a.resid_ld + k0) + f4);
                v.x = r.x + v.x; v.y = r.y + v.y; v.z = r.z + v.z; v.w = r.w + v.w;
            }
            if (a.out) ((float4*)(a.out + (size_t)m * a.out_ld + k0))[f4] = v;
        }
        if (!a.gain) { store(f4, v); continue; }
        if (f4 < n4) ((float4*)rowbuf)[f4] = v;
        ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss);
    }
    if (!a.gain) return;
    ss = block_sum(ss, scratch, tid, 256, 1, false);
    if (C > 1) {
        if (tid == 0) s_x = ss;
        cluster_arrive_release();
        cluster_wait_acquire();
        ss = 0.0f;
        for (int r = 0; r < C; r++) ss += cluster_ld_f32(cluster_map(smem_u32(&s_x), (uint32_t)r));
        cluster_arrive_release();                            // waited for at the end: nobody leaves while its s_x may still be read
    }
    const float inv = 1.0f / sqrtf(ss * (1.0f / (float)K) + a.eps);
    for (int b = 0; b < n4; b += 256) {                      // each thread revisits the elements it wrote
        const int f4 = b + tid;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (f4 < n4) {
            v = ((const float4*)rowbuf)[f4];
            float4 g;
            if (a.gain_kind == WK_BF16) {
                const uint2 r = __ldg((const uint2*)((const uint16_t*)a.gain + k0) + f4);
                g = make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
            } else {
                g = __ldg((const float4*)((const float*)a.gain + k0) + f4);
            }
            v.x = (inv * v.x) * g.x; v.y = (inv * v.y) * g.y; v.z = (inv * v.z) * g.z; v.w = (inv * v.w) * g.w;
        }
        store(f4, v);
    }
    if (C > 1) cluster_wait_acquire();
}

// ---------------------------------------------------------------------------------------------------------------- product
struct FewSmem { size_t x, sx, red, ring, total; };          // byte offsets
__host__ __device__ inline int few_red_ld(int tiles) { return 8 * tiles + 1; }      // floats per weight row of a warp's sums
__host__ __device__ inline FewSmem few_smem(int tiles, int k, size_t ring) {
    FewSmem s;
    s.x = kFewBar;
    s.sx = s.x + (size_t)(k / 64) * tiles * 512;
    s.red = s.sx + (size_t)(k / 32) * tiles * 32;
    s.ring = (s.red + (size_t)2 * 8 * 16 * few_red_ld(tiles) * 4 + 127) / 128 * 128;
    s.total = s.ring + ring;
    return s;
}

// T: groups of eight columns.  y[range][m][column] = sums of the range (planes part_stride apart, rows ldy).
// The accumulators start at 1.5 * 2^23 as a float's bits, so that an int32 sum comes out as that float plus the sum: an addition instead of a conversion.
// Measured, 5 rows of a Llama-3-8B layer (q8_gemm_tc_skinny / this): gate | up 45 -> 32 us, vocabulary projection 151 -> 111 us; a step of five sequences 4.08 -> 2.95 ms.
// With a warp per (tile, row) instead of columns of all rows: 3.70 ms (issue slots).
template <int T>
__global__ void __launch_bounds__(kFewThreads, 1) q8_few(const GemvArgs a, const int M, const int8_t* xq, const float* sx, const int ldy, const size_t part_stride) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    __shared__ int2 s_meta[kMaxStages];
    const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) & 7, grp = tid >> 8;
    const GemvPlan p = gemv_plan(a, (int)blockIdx.x, (int)gridDim.x, -1);
    GemvSmem g{};
    g.full0 = smem_u32(smem); g.empty0 = g.full0 + 8u * kMaxStages;
    const uint32_t xbar = g.empty0 + 8u * kMaxStages;
    g.rings = GemvRings{a.ring_n[0], a.ring_n[1], a.ring_t[0], a.ring_t[1]};
    const FewSmem fs = few_smem(T, a.k_smem, g.rings.bytes());
    g.meta = s_meta; g.stage0 = smem + fs.ring; g.abort = &s_abort;
    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < g.rings.stages(); s++) { mbar_init(g.full0 + 8u * s, 1); mbar_init(g.empty0 + 8u * s, 4); }
        mbar_init(xbar, 1);
        mbar_fence_init();
    }
    __syncthreads();
    if (a.use_pdl) pdl_launch_dependents();
    if (grp == 2) {
        if (elect_one()) {
            ProducerRing pr{};
            if (!gemv_produce(a, p, g, pr, nullptr, a.status)) gemv_producer_drain(g, pr, a.status);
        }
        return;
    }
    if (a.use_pdl) pdl_grid_wait();
    if (tid < 32 && elect_one()) {                           // this range's columns of every row
        const uint32_t nx = (uint32_t)p.nt * 8u * T * 512u, ns = (uint32_t)p.nt * 16u * T * 32u;
        mbar_arrive_expect_tx(xbar, nx + ns);
        bulk_g2s(smem_u32(smem + fs.x), xq + (size_t)p.t0 * 8 * T * 512, nx, xbar);
        bulk_g2s(smem_u32(smem + fs.sx), sx + (size_t)p.t0 * 16 * T * 8, ns, xbar);
    }
    __syncwarp();
    auto fail = [&](uint32_t code) { if (!s_abort) { atomicOr(a.status, code); *(volatile int*)&s_abort = 1; } };
    if (!mbar_wait_warp(xbar, 0u, g.abort)) fail(LUM_ST_WAIT_FULL);

    const int wg = warp >> 2, wj = warp & 3, first = g.first(wg);
    constexpr int S = kFewStages;
    const uint32_t ring = smem_u32(g.at(wg, 0)) + (uint32_t)wj * kTileBytes, stride = (uint32_t)(wg ? g.rings.t1 : g.rings.t0) * kTileBytes;
    const bool mine = warp < p.nt;
    const unsigned char* const xw = smem + fs.x + (size_t)min(warp, p.nt - 1) * 8 * T * 512 + lane * 16;
    const float* const sw = (const float*)(smem + fs.sx) + (size_t)min(warp, p.nt - 1) * 16 * T * 8 + (lane & 3) * 2;
    constexpr int LD = 8 * T + 1;
    float* const red = (float*)(smem + fs.red) + (size_t)grp * 8 * 16 * LD;
    // The jobs are dealt out (row groups blockIdx.x, + n_cta, ..): fill number f of either ring is row group f of this CTA's, pair q is fills 2 q and 2 q + 1.  With four
    // stages a ring the even pairs always lie in the first two and the odd ones in the others: no group waits for a phase of a stage whose phases before it has not seen.
    const int n_fill = p.cta < p.J ? (p.J - p.cta + p.n_cta - 1) / p.n_cta : 0;
#pragma unroll 1
    for (int q = grp; 2 * q < n_fill; q += 2) {
        const int f0 = 2 * q, f1 = min(f0 + 1, n_fill - 1);                   // (a last row group on its own is its own partner)
        const int st0 = f0 % S, st1 = f1 % S;
        bool ok = mbar_wait_warp(g.full0 + 8u * (first + st0), (uint32_t)(f0 / S) & 1u, g.abort);
        ok = ok && mbar_wait_warp(g.full0 + 8u * (first + st1), (uint32_t)(f1 / S) & 1u, g.abort);
        if (!ok) fail(LUM_ST_WAIT_FULL);
        float acc[T][4];
#pragma unroll
        for (int t = 0; t < T; t++)
#pragma unroll
            for (int i = 0; i < 4; i++) acc[t][i] = 0.0f;
        if (mine && ok) {
            const uint32_t w0 = ring + (uint32_t)st0 * stride, w1 = ring + (uint32_t)st1 * stride;
#pragma unroll 2
            for (int s = 0; s < 8; s++) {                    // two blocks at a time
                uint32_t x0[4], x1[4];
                gemv_ldmatrix(w0 + s * 512 + lane * 16, x0);
                gemv_ldmatrix(w1 + s * 512 + lane * 16, x1);
                uint4 b[T];
#pragma unroll
                for (int t = 0; t < T; t++) b[t] = *(const uint4*)(xw + (s * T + t) * 512);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint16_t u0, u1;
                    const uint32_t so = kTileQ + (2 * s + h) * 16 + (lane >> 2) * 2;
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u0) : "r"(w0 + so) : "memory");
                    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u1) : "r"(w1 + so) : "memory");
                    const float d0 = __half2float(__ushort_as_half(u0)), d1 = __half2float(__ushort_as_half(u1));
#pragma unroll
                    for (int t = 0; t < T; t++) {
                        constexpr int kMagicBits = 0x4b400000;                // 12582912.0f
                        int c[4];
                        asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                                     : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
                                     : "r"(x0[2 * h]), "r"(x1[2 * h]), "r"(x0[2 * h + 1]), "r"(x1[2 * h + 1]), "r"(h ? b[t].z : b[t].x), "r"(h ? b[t].w : b[t].y), "r"(kMagicBits));
                        const float2 x = *(const float2*)(sw + ((2 * s + h) * T + t) * 8);
                        acc[t][0] = fmaf(__int_as_float(c[0]) - 12582912.0f, d0 * x.x, acc[t][0]);
                        acc[t][1] = fmaf(__int_as_float(c[1]) - 12582912.0f, d0 * x.y, acc[t][1]);
                        acc[t][2] = fmaf(__int_as_float(c[2]) - 12582912.0f, d1 * x.x, acc[t][2]);
                        acc[t][3] = fmaf(__int_as_float(c[3]) - 12582912.0f, d1 * x.y, acc[t][3]);
                    }
                }
            }
            float* const r0 = red + (size_t)(warp * 16 + (lane >> 2)) * LD + (lane & 3) * 2;
#pragma unroll
            for (int t = 0; t < T; t++) {
                r0[8 * t] = acc[t][0]; r0[8 * t + 1] = acc[t][1];
                r0[8 * LD + 8 * t] = acc[t][2]; r0[8 * LD + 8 * t + 1] = acc[t][3];
            }
        }
        const int unit0 = p.cta + f0 * p.n_cta, unit1 = p.cta + f1 * p.n_cta;      // (one row group per job: not read from the stage's words, which a refill replaces)
        __syncwarp();
        if (lane == 0) {                                     // the tiles have been read: their sums are stored
            mbar_arrive(g.empty0 + 8u * (first + st0));
            if (f1 != f0) mbar_arrive(g.empty0 + 8u * (first + st1));
        }
        // the warps' sums of a row and its three levels, added in a fixed order (a warp that gave up takes its group along)
        if (named_or(2 + grp, kConsumers, !ok)) break;
        for (int i = tid & 255; i < 16 * M; i += kConsumers) {
            const int r = i & 15, m = i >> 4;
            if (r >= 8 && f1 == f0) continue;
            const float* rp = red + (size_t)r * LD + 3 * m;
            float v = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; w++)
                if (w < p.nt) v += (rp[(size_t)w * 16 * LD + 2] + rp[(size_t)w * 16 * LD + 1]) + rp[(size_t)w * 16 * LD];
            a.y[p.range * part_stride + (size_t)m * ldy + (r < 8 ? unit0 : unit1) * kTileRows + (r & 7)] = v;
        }
        named_sync(2 + grp, kConsumers);
    }
    // after a run that was given up: not before the copies of x have landed (the producer sees to the ring's)
    if (tid < 32 && elect_one() && *(volatile int*)&s_abort && !mbar_wait(xbar, 0u)) atomicOr(a.status, LUM_ST_WAIT_DRAIN);
}

// ---------------------------------------------------------------------------------------------------------------- host side
// Whether a product of K columns can run here, and in how many K ranges: every range five to eight tiles, so that a warp has the same tile of every row group.
int few_ranges(int K, int sm_count) {
    const int tpr = K / kTileK, r = gemv_k_ranges(K, kTileK);
    if (K % kTileK || tpr / r <= kFillTiles || (tpr + r - 1) / r > kJobTiles || sm_count < tpr) return 0;
    return r;
}
size_t few_xq_bytes(int M, int K) { return (size_t)(K / 64) * few_tiles(M) * 512; }
size_t few_sx_floats(int M, int K) { return (size_t)(K / 32) * few_tiles(M) * 8; }

cudaError_t launch_rows_levels(const RowsArgs& a_in, int sm_count, cudaStream_t st) {
    RowsArgs a = a_in;
    if (a.M < 1 || a.M > kFewRows || a.K <= 0 || (a.K % kTileK) || a.n_parts < 1) return cudaErrorInvalidValue;
    int C = 1;
    while (C < 8 && a.M * C * 2 <= 4 * sm_count && (a.K >> 5) / (C * 2) >= 8) C *= 2;
    const size_t smem = a.gain ? (size_t)(((a.K >> 5) + C - 1) / C) * 128 : 0;
    if (smem > 48 * 1024) return cudaErrorInvalidValue;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.M * C);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (C > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = (unsigned)C; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
        n++;
    }
    if (a.use_pdl) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    void* params[] = {&a, &C};
    return cudaLaunchKernelExC(&cfg, (const void*)rows_levels, params);
}

cudaError_t launch_few(const FewArgs& f, int sm_count, cudaStream_t st) {
    const int R = few_ranges(f.K, sm_count);
    if (!R || f.M < 1 || f.M > kFewRows || f.nseg < 1 || f.nseg > 3) return cudaErrorInvalidValue;
    GemvArgs a{};
    a.nseg = f.nseg; a.K = f.K; a.wkind = WK_Q8; a.epi = EPI_STORE; a.ksplit = R; a.y = f.y; a.status = f.status; a.use_pdl = f.use_pdl;
    int groups = 0;
    for (int s = 0; s < f.nseg; s++) {
        if (f.rows[s] <= 0 || f.rows[s] % kTileRows) return cudaErrorInvalidValue;
        a.seg[s] = {f.w[s], nullptr, f.rows[s], kTileK};
        groups += f.rows[s] / kTileRows;
    }
    const int tpr = f.K / kTileK;
    int most = 0;
    for (int r = 0; r < R; r++) most = std::max(most, gemv_range_tile(tpr, R, r + 1) - gemv_range_tile(tpr, R, r));
    a.k_smem = most * kTileK;
    int grid = sm_count;
    if (R == 1 && groups < grid) grid = groups;
    constexpr size_t kAll = 226 * 1024;
    const GemvRings rings{kFewStages, kFewStages, kFillTiles, most < kJobTiles ? most - kFillTiles : kFillTiles};
    const size_t smem = few_smem(few_tiles(f.M), a.k_smem, rings.bytes()).total;
    if (smem > kAll) return cudaErrorInvalidValue;
    a.ring_n[0] = rings.n0; a.ring_n[1] = rings.n1; a.ring_t[0] = rings.t0; a.ring_t[1] = rings.t1;
    const int t = few_tiles(f.M);
    const void* fn = t == 1 ? (const void*)q8_few<1> : (const void*)q8_few<2>;
    static std::atomic<uint64_t> raised[2] = {};
    if (const cudaError_t e = allow_smem(raised[t - 1], fn, (int)kAll)) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kFewThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = f.use_pdl ? 1 : 0;
    int M = f.M, ldy = f.ldy;
    const int8_t* xq = f.xq;
    const float* sx = f.sx;
    size_t stride = f.part_stride;
    void* params[] = {&a, &M, &xq, &sx, &ldy, &stride};
    return cudaLaunchKernelExC(&cfg, fn, params);
}

}  // namespace lum
