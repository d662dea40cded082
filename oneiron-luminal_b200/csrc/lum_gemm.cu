// Q8_0 matrix-matrix product for more than one activation row — batched decode and prompt processing:
// Y[M, N] = X[M, K] W[N, K]^T with W in the packed tile stream of the streaming GEMV.  This is the M > 1 path of
// `TileMatmulFullSplit` (crates/luminal_cuda/src/block/ops.rs:1653-1738: 64 x 64 tiles, one thread per output element with a
// serial k loop and atomicAdd) and of `TileMatmulNvFp4` / `TileMatmulMxfp4` (ops.rs:2148-2347, 2546-2733), here for Q8_0
// on the 5th-generation tensor cores.
//
// Arithmetic.  The CPU restatement multiplies f32 activations by exactly dequantised weights, and greedy decoding over a
// large vocabulary only stays token-exact at f32-level accuracy, so neither operand may simply be rounded to 16 bits.
// Both are written as short sums of binary16 terms instead, and the tensor core (tcgen05.mma kind::f16, f32 accumulators in
// tensor memory) adds up the products of the terms:
//   * a weight w = q * d (q int8, d binary16) has at most 18 significant bits.  1024 w = hi + lo EXACTLY, with
//     hi = f16(q * 1024 d) and lo = q * 1024 d - hi (one fused multiply-add); the factor 1024 keeps lo out of the binary16
//     subnormals whatever d is.  Two instructions per pair of weights, on the packed-half units.
//   * an activation row is scaled by a power of two that puts its largest magnitude in [2^13, 2^14) and split into two
//     terms x1 + x2 (binary16 roundings of the value and of the residual): 22 bits.
//   * three products are accumulated: hi x1, hi x2, lo x1.  What is left out (lo x2 and the activation's third term) is
//     below 2^-21 of |w| |x| per element — the size of the differences that the ORDER of an f32 summation over K >= 2048
//     terms makes anyway (the CPU restatement sums sequentially, the tensor core in its own order), so the result is
//     as close to the restatement as any f32 evaluation of the same dot product is.  (Five products, with a third activation
//     term, reproduce every bit of the operands; measured, they cost 1.6x the time and change no token and no test.)
// Q8_0's per-32 scales therefore never leave the operand: ONE accumulator per output tile runs over the whole K range and is
// read back once, instead of once per 32-block (which is what binds an integer formulation: the read-back, not the tensor core).
// The power-of-two factors (1024 and the row's) are undone exactly when the accumulator is stored.
//
// Two kernels:
//  * rows_quantize — one CTA per activation row.  Forms the row (sum of the previous product's K-split partials, residual
//    add, SwiGLU), optionally RMS-normalises it (`RowRMSNorm`, ops.rs:519-566; `RowSwishMul`, ops.rs:303-325; `RowAdd`,
//    ops.rs:135-146 are fused here), writes the two terms in tensor-core operand order and the row's output factor.
//  * q8_gemm_tc — 80 to 128 activation rows per chunk (prompts).  Persistent CTAs over work items (256 weight rows = two tensor-core tiles
//    that share every activation slice, one chunk, one K range).  One lane fills a ring of six 32 KiB activation stages with bulk
//    copies; 16 warps read their rows' weights straight from global memory (32 bytes per row and slice, two steps ahead, in
//    registers), turn them into the hi / lo operands and store those to tensor memory (the A operand is read from there: shared
//    memory and its bandwidth belong to the activation operand); one thread issues the tensor-core instructions (24 of N = chunk rows per
//    step of two 32-column slices) and commits the buffers free; the 16 warps store the two accumulators when the K range is done.
//    Bound by the tensor core, if everything else keeps up: 24 instructions of 65 clocks a step.  Measured, alone (issued TFLOP/s, 6 per
//    weight and row; 8 warps that converted after the wait for their buffer / 16 that convert before it): 28672 x 4096 at 512 rows
//    909 -> 1342, at 4096 rows 1177 -> 1649 (constant operands; a prompt's run into the power limit), 128 rows 771 -> 1188.
//  * q8_gemm_tc_skinny — up to 64 rows (batched decode): see its own header further down.
//    Outputs are plain f32 stores of K-split partial planes; whoever consumes them (the next rows_quantize) adds them up.
#include <cstdlib>

#include <cuda_fp16.h>

#include "lum_gemv_dev.cuh"
#include "lum_rows.cuh"

namespace lum {

constexpr int kGmHB = 2;                            // tensor-core tiles (128 weight rows) per work item; they share every activation slice
constexpr int kGmRows = 128 * kGmHB;                // weight rows per work item
constexpr int kGmMaxChunk = 128;                    // activation rows per chunk: 16, 32 or 64, or (q8_gemm_tc) 80 .. 128 (gemm_shape)
constexpr int kGmXTerms = 2;                        // binary16 terms per activation element
constexpr int kGmStep = 2;                          // 32-column slices per hand-over between the warps (every hand-over costs each single-threaded role
                                                    // several hundred cycles of its own, whatever the amount of work behind it)
constexpr int kGmAhead = 2;                         // steps whose weights a converter thread has on their way from global memory
constexpr int kGmXStageMax = kGmStep * kGmXTerms * kGmMaxChunk * 32 * 2;   // 32768: one activation stage (the terms of one step of a 128-row chunk)
constexpr int kGmCvtBufs = 2, kGmXStages = 6;
constexpr uint32_t kGmCvtCols = 32 * kGmHB * kGmStep;        // tensor-memory columns of one converted step: per slice and 128-row tile hi (16 columns: 32 binary16
                                                             // per row) | lo (16)
constexpr int kGmCvtWarps = 16;
constexpr int kGmThreads = (kGmCvtWarps + 2) * 32;   // + activation producer warp + tensor-core warp
constexpr int kGmBarBytes = 512;
constexpr size_t kGmSmem = kGmBarBytes + 128 + (size_t)kGmXStages * kGmXStageMax;
constexpr int kGmWExp = 10;                         // weights enter as 2^10 w
constexpr uint32_t kGmTmemCols = 512;               // one accumulator of 128 columns per 128-row tile, then the converted-weight buffers
constexpr uint32_t kGmCvtCol0 = 128 * kGmHB;

__device__ __forceinline__ float block_max(float v, float* scratch, int tid, int nthreads, int bar_id) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    named_sync(bar_id, nthreads);
    if ((tid & 31) == 0) scratch[tid >> 5] = v;
    named_sync(bar_id, nthreads);
    float t = 0.0f;
    for (int w = 0; w < (nthreads >> 5); w++) t = fmaxf(t, scratch[w]);
    return t;
}

// activation operand: [chunk][K / 32 slices][4 groups of 8 columns][kGmXTerms terms][chunk rows][16 bytes]: within a column group the
// rows of the first term are followed by the rows of the second, so ONE operand descriptor of 2 x chunk rows covers both terms
//
// A cluster of C CTAs forms one row, each K / C of its columns (whole 32-column slices); the sum of squares and the largest magnitude go
// round through distributed shared memory.  With few rows this kernel is bound by its chain of trips to L2 and by how many loads are
// on their way, so a row is spread over as many SMs as there are.  Measured (32 rows, the four of a Llama-3-8B layer, K 4096 and
// 14336): 70 us a layer with one CTA per row, 31 us with eight.
//
// With many rows (no cluster) a CTA forms TWO of them, 256 threads each, and stores both together: a row's 16-byte pieces of the operand lie between its
// neighbours', and two make a whole 32-byte sector.  What bounds it then is memory and issue slots about equally (packed conversions, gains by four).  Measured,
// gate | up of a Llama-3-8B layer, 705 MB for 4096 rows: 263 -> 180 us, a row of 4096 columns behind a norm 53 -> 47.
constexpr int kRqMaxCluster = 8;
constexpr int kRqPad = 16;                               // floats behind a row in shared memory: the two rows' pieces lie in different banks
template <int ROWS>
__global__ void __launch_bounds__(256 * ROWS) rows_quantize(const RowsArgs a, const int C) {
    extern __shared__ __align__(16) float rows[];            // this CTA's columns of its rows
    __shared__ float scratch_of[ROWS][8], s_x[2];
    __shared__ float s_up[ROWS];
    const int half = ROWS > 1 ? (int)threadIdx.x >> 8 : 0, tid = threadIdx.x & 255, bar = 1 + half;
    const int part = ROWS > 1 ? 0 : blockIdx.x % C, m = ROWS > 1 ? (int)blockIdx.x * ROWS + half : (int)blockIdx.x / C;
    float* const scratch = scratch_of[half];
    const int K = a.K, nb = K >> 5;
    float* const rowbuf = rows + (size_t)half * (K + kRqPad);
    const int s0 = (int)((long long)nb * part / C), s1 = (int)((long long)nb * (part + 1) / C);     // this CTA's slices
    const int k0 = s0 << 5, n4 = (s1 - s0) << 3;             // its first column, its float4
    if (a.use_pdl) { pdl_launch_dependents(); pdl_grid_wait(); }
    const int nc = a.nc;
    const size_t slice_bytes = (size_t)kGmXTerms * 4 * nc * 16;
    unsigned char* xq_chunk = (unsigned char*)a.xq + (size_t)(m / nc) * nb * slice_bytes;
    const int ml = m % nc;
    if (ROWS == 1 && m >= a.M) {
        // padding row of the last chunk: zeros (the whole cluster returns)
        for (int ch = s0 * kGmXTerms * 4 + tid; ch < s1 * kGmXTerms * 4; ch += 256) {
            const int s = ch / (kGmXTerms * 4), tc = ch - s * (kGmXTerms * 4);           // (column group, term) of slice s
            *(uint4*)(xq_chunk + (size_t)s * slice_bytes + (size_t)tc * nc * 16 + ml * 16) = make_uint4(0u, 0u, 0u, 0u);
        }
        if (tid == 0 && part == 0) a.sx[m] = 0.0f;
        return;
    }
    const bool live = m < a.M;                               // (a padding row is a row of zeros)
    float ss = 0.0f, amax = 0.0f;
    for (int f4 = tid; f4 < n4; f4 += 256) {
        const size_t at = (size_t)m * a.ld + k0 + f4 * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f), u = v;
        if (ROWS == 1 || live) {
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
        ((float4*)rowbuf)[f4] = v;
        if (a.gain) { ss = fmaf(v.x, v.x, ss); ss = fmaf(v.y, v.y, ss); ss = fmaf(v.z, v.z, ss); ss = fmaf(v.w, v.w, ss); }
        else amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    // one number per CTA -> the cluster's, combined in the order of its CTAs
    auto exchange = [&](float v, int slot, bool maximum) -> float {
        if (C == 1) return v;
        if (tid == 0) s_x[slot] = v;
        cluster_arrive_release();
        cluster_wait_acquire();
        float t = cluster_ld_f32(cluster_map(smem_u32(&s_x[slot]), 0u));
        for (int r = 1; r < C; r++) {
            const float x = cluster_ld_f32(cluster_map(smem_u32(&s_x[slot]), (uint32_t)r));
            t = maximum ? fmaxf(t, x) : t + x;
        }
        return t;
    };
    if (a.gain) {
        // the normalised row, and its largest magnitude
        ss = exchange(block_sum(ss, scratch, tid, 256, bar), 0, false);
        const float inv = 1.0f / sqrtf(ss * (1.0f / (float)K) + a.eps);
        for (int f4 = tid; f4 < n4; f4 += 256) {            // each thread revisits the elements it wrote
            float4 v = ((const float4*)rowbuf)[f4], g;
            if (a.gain_kind == WK_BF16) {
                const uint2 r = __ldg((const uint2*)((const uint16_t*)a.gain + k0) + f4);
                g = make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16), __uint_as_float(r.y & 0xffff0000u));
            } else {
                g = __ldg((const float4*)((const float*)a.gain + k0) + f4);
            }
            v.x = (inv * v.x) * g.x; v.y = (inv * v.y) * g.y; v.z = (inv * v.z) * g.z; v.w = (inv * v.w) * g.w;
            ((float4*)rowbuf)[f4] = v;
            amax = fmaxf(amax, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
        }
    }
    amax = exchange(block_max(amax, scratch, tid, 256, bar), 1, true);     // (its barriers also publish the row to the other threads)
    if (C > 1) cluster_arrive_release();                    // waited for at the end: nobody leaves while its s_x may still be read
    // power of two that puts the maximum in [2^13, 2^14); a zero (or non-finite) row keeps factor 1
    int ex = 0;
    if (amax > 0.0f && amax < INFINITY) frexpf(amax, &ex);
    else ex = 14;
    if (tid == 0 && part == 0) a.sx[m] = ROWS == 1 || live ? ldexpf(1.0f, ex - 14 - kGmWExp) : 0.0f;       // undoes this factor and the weights' 2^10
    float up = ldexpf(1.0f, 14 - ex);
    const float* src = rowbuf;
    int c0 = tid, cn = 256;                                  // this thread's pieces of 8 columns, of the row it stores
    unsigned char* dst0 = xq_chunk + ml * 16;
    if (ROWS > 1) {
        if (tid == 0) s_up[half] = up;
        __syncthreads();
        const int r = threadIdx.x % ROWS;
        up = s_up[r]; src = rows + (size_t)r * (K + kRqPad);
        c0 = threadIdx.x / ROWS;
        const int mr = (int)blockIdx.x * ROWS + r;
        dst0 = (unsigned char*)a.xq + (size_t)(mr / nc) * nb * slice_bytes + (mr % nc) * 16;
    }
    for (int c8 = c0; c8 < (n4 >> 1); c8 += cn) {
        const float4 v0 = ((const float4*)src)[2 * c8], v1 = ((const float4*)src)[2 * c8 + 1];
        const float e[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        uint32_t t1[4], t2[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float x0 = e[2 * j] * up, x1 = e[2 * j + 1] * up;          // exact: a power of two
            const __half2 h = __floats2half2_rn(x0, x1);
            const float2 f = __half22float2(h);
            const __half2 l = __floats2half2_rn(x0 - f.x, x1 - f.y);         // (the differences are exact in f32)
            t1[j] = *(const uint32_t*)&h;
            t2[j] = *(const uint32_t*)&l;
        }
        const int s = s0 + (c8 >> 2), cg = c8 & 3;
        unsigned char* dst = dst0 + (size_t)s * slice_bytes + (size_t)cg * kGmXTerms * nc * 16;
        *(uint4*)(dst) = make_uint4(t1[0], t1[1], t1[2], t1[3]);
        *(uint4*)(dst + (size_t)nc * 16) = make_uint4(t2[0], t2[1], t2[2], t2[3]);
    }
    if (C > 1) cluster_wait_acquire();
}

struct GemmItem { int seg, rg0, n_rg, mc, t0, t1, ks; };
__device__ __forceinline__ GemmItem gemm_item(const GemmArgs& a, int item, int tpr, int rows_per_item = kGmRows) {
    GemmItem it;
    it.mc = item % a.m_chunks;
    int rest = item / a.m_chunks;
    it.ks = rest % a.ksplit;
    int tile = rest / a.ksplit;
    it.seg = 0;
    for (int s = 0; s < a.nseg - 1; s++) {
        const int nt = (a.seg[s].rows + rows_per_item - 1) / rows_per_item;
        if (it.seg == s && tile >= nt) { tile -= nt; it.seg = s + 1; }
    }
    it.rg0 = tile * (rows_per_item / kTileRows);
    it.n_rg = min(rows_per_item / kTileRows, a.seg[it.seg].rows / kTileRows - it.rg0);
    it.t0 = (int)((long long)it.ks * tpr / a.ksplit);
    it.t1 = (int)((long long)(it.ks + 1) * tpr / a.ksplit);
    return it;
}

// packed binary16 arithmetic on plain 32-bit registers
__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b) { uint32_t d; asm("sub.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t h2_mul(uint32_t a, uint32_t b) { uint32_t d; asm("mul.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t h2_fma(uint32_t a, uint32_t b, uint32_t c) { uint32_t d; asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d; }

// kind::f16 with binary16 operands, f32 accumulators, both operands K-major, shape M x N (K = 16)
__host__ __device__ constexpr uint32_t umma_idesc_f16(int M, int N) { return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24); }
// The A operand lies in tensor memory: lane = row, 32-bit column j = elements 2j, 2j + 1 of the row.  The B descriptor is given as its two halves
// (the high half is the same for every operand of a kernel).
__device__ __forceinline__ void umma_f16_ts2(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tsetp.ne.b32 p, %5, 0;\n\tmov.b64 db, {%2, %3};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// whole warp: 16 consecutive 32-bit columns of this thread's lane
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]),
                 "r"(v[14]), "r"(v[15])
                 : "memory");
}
__device__ __forceinline__ uint32_t h2_neg(uint32_t a) { uint32_t d; asm("neg.f16x2 %0, %1;" : "=r"(d) : "r"(a)); return d; }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__global__ void __launch_bounds__(kGmThreads, 1) q8_gemm_tc(const GemmArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bars = smem_u32(smem);
    const uint32_t xfull = bars, xempty = bars + 64, cfull = bars + 128, cempty = bars + 160, afull = bars + 192, aempty = bars + 200,
                   fin = bars + 208, tmem_slot = bars + 216;
    static_assert(kGmXStages <= 8 && kGmCvtBufs <= 4 && kGmCvtCol0 + kGmCvtBufs * kGmCvtCols <= kGmTmemCols && kGmXTerms == 2 && kGmStep == 2 &&
                  kGmHB == 2 && 16 % (kGmAhead * kGmStep) == 0, "barrier area / tensor memory / the converter's unrolled loop");
    unsigned char* xst = (unsigned char*)(((uintptr_t)smem + kGmBarBytes + 127) & ~(uintptr_t)127);
    volatile int* abort = &s_abort;
    if (tid == 0) {
        s_abort = 0;
        mbar_init(afull, 1); mbar_init(aempty, kGmCvtWarps);
        for (int i = 0; i < kGmCvtBufs; i++) { mbar_init(cfull + 8u * i, kGmCvtWarps); mbar_init(cempty + 8u * i, 1); }
        for (int i = 0; i < kGmXStages; i++) { mbar_init(xfull + 8u * i, 1); mbar_init(xempty + 8u * i, 1); }
        mbar_init(fin, 1);
        mbar_fence_init();
    }
    if (warp == kGmCvtWarps + 1) tmem_alloc(tmem_slot, kGmTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
    // The weights do not depend on the previous kernel: they are on their way while it still runs.  Its results are waited for where they
    // are read (activation copies, row factors) or where what it may still read is overwritten (the sums).
    if (a.use_pdl) pdl_launch_dependents();

    const int tpr = a.K / kTileK, nb = a.K >> 5;
    const int nc = a.nc;                                   // activation rows per chunk
    const uint32_t x_cg = (uint32_t)kGmXTerms * (uint32_t)nc * 16u;      // bytes of one column group of a slice: both terms' rows
    const uint32_t x_slice = 4u * x_cg;
    constexpr uint32_t ncb = kGmCvtBufs, nxs = kGmXStages;
    constexpr int sps = kGmStep;                           // slices per activation stage: one step, one 32 KiB copy
    int tiles = 0;
    for (int s = 0; s < a.nseg; s++) tiles += (a.seg[s].rows + kGmRows - 1) / kGmRows;
    const int n_items = tiles * a.ksplit * a.m_chunks;
    auto fail = [&](uint32_t code) { if (!*abort) { atomicOr(a.status, code); *abort = 1; } };

    if (warp == kGmCvtWarps) {
        // ---------------------------------------------------------------- activation producer: one lane, one 32 KiB copy per stage
        if (elect_one()) {
            uint32_t xi = 0;
            bool ok = true;
            if (a.use_pdl) pdl_grid_wait();
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                const GemmItem it = gemm_item(a, item, tpr);
                for (int t = it.t0; t < it.t1 && ok; t++) {
                    for (int s = 0; s < 16; s += sps) {
                        const uint32_t xs = xi % nxs;
                        if (!mbar_wait_abortable(xempty + 8u * xs, ((xi / nxs) & 1u) ^ 1u, abort)) { fail(LUM_ST_WAIT_EMPTY); ok = false; break; }
                        mbar_arrive_expect_tx(xfull + 8u * xs, x_slice * (uint32_t)sps);
                        bulk_g2s(smem_u32(xst + (size_t)xs * kGmXStageMax), (const unsigned char*)a.xq + ((size_t)it.mc * nb + (size_t)t * 16 + s) * x_slice,
                                 x_slice * (uint32_t)sps, xfull + 8u * xs);
                        xi++;
                    }
                }
            }
            // never leave while a copy into this CTA's shared memory may be in flight: wait (bounded) for what was armed
            if (!ok)
                for (uint32_t k = 0; k < nxs && k < xi; k++) { const uint32_t i = xi - 1 - k; mbar_wait(xfull + 8u * (i % nxs), (i / nxs) & 1u); }
        }
        return;
    }
    if (warp == kGmCvtWarps + 1) {
        // ---------------------------------------------------------------- tensor-core warp: one lane issues
        if (elect_one()) {
            uint32_t xi = 0, ci = 0, ic = 0;
            bool ok = true;
            // hi x1, hi x2, lo x1 as three instructions of N = nc into one accumulator
            const uint32_t idesc = umma_idesc_f16(128, nc);
            // activation operand descriptors: start address in the low 14 bits; column groups x_cg bytes apart, 8-row groups 128
            const uint32_t x_lo = ((x_cg >> 4) & 0x3fffu) << 16, x_base = smem_u32(xst);
            constexpr uint32_t x_hi = umma_desc_hi(128u);
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ic++) {
                const GemmItem it = gemm_item(a, item, tpr);
                if (!mbar_wait_abortable(aempty, (ic & 1u) ^ 1u, abort)) { fail(LUM_ST_WAIT_TMEM); break; }      // the previous item's sums were stored
                tc_fence_after_sync();
                uint32_t started = 0;
                for (int t = it.t0; t < it.t1 && ok; t++) {
                    for (int s = 0; s < 16; s += kGmStep) {
                        const uint32_t cb = ci % ncb, xs = xi % nxs;
                        if (!mbar_wait_abortable(cfull + 8u * cb, (ci / ncb) & 1u, abort) || !mbar_wait_abortable(xfull + 8u * xs, (xi / nxs) & 1u, abort)) {
                            fail(LUM_ST_WAIT_FULL); ok = false; break;
                        }
                        tc_fence_after_sync();
                        const uint32_t wt = tmem + kGmCvtCol0 + cb * kGmCvtCols;
                        const uint32_t xb = x_base + xs * (uint32_t)kGmXStageMax;
#pragma unroll
                        for (int kk = 0; kk < 2 * kGmStep; kk++) {     // K = 16 per instruction: two per 32-column slice
                            // weights: tensor memory, 8 columns (16 binary16) per instruction; activations: shared memory,
                            // [column group of 8][term][row][16 bytes], an instruction reads two adjacent column groups
                            const uint32_t xo = xb + (uint32_t)(kk >> 1) * x_slice + (uint32_t)(kk & 1) * 2u * x_cg;
                            const uint32_t x1 = x_lo | ((xo >> 4) & 0x3fffu), x2 = x_lo | (((xo + (uint32_t)nc * 16u) >> 4) & 0x3fffu);
#pragma unroll
                            for (int hb = 0; hb < kGmHB; hb++) {      // the 128-row tiles of the item
                                const uint32_t acc = tmem + (uint32_t)hb * 128u;
                                const uint32_t hi = wt + (uint32_t)((kk >> 1) * kGmHB + hb) * 32u + (uint32_t)(kk & 1) * 8u;
                                umma_f16_ts2(acc, hi, x1, x_hi, idesc, kk > 0 ? 1u : started);
                                umma_f16_ts2(acc, hi, x2, x_hi, idesc, 1u);
                                umma_f16_ts2(acc, hi + 16u, x1, x_hi, idesc, 1u);
                            }
                        }
                        started = 1u;
                        umma_commit(cempty + 8u * cb);        // arrive when the instructions that read these operands have retired
                        umma_commit(xempty + 8u * xs);
                        ci++;
                        xi++;
                    }
                }
                if (ok) umma_commit(afull);
            }
            umma_commit(fin);
            if (!mbar_wait(fin, 0u)) atomicOr(a.status, LUM_ST_WAIT_TMEM);
        }
        __syncwarp();
        named_sync(4, kGmCvtWarps * 32 + 32);
        tc_fence_after_sync();
        tmem_dealloc(tmem, kGmTmemCols);
        return;
    }

    // -------------------------------------------------------------------- converting / storing warps
    {
        // A warp reaches the 32 tensor-memory lanes of its quarter: thread = weight row of a 128-row tile; of a step's four operands (two
        // slices of two tiles) it converts slice ss of tile hb (and stores half of that tile's sums).  The weights come straight from global
        // memory: a thread's 2 x 16 bytes of a slice are the columns of its row in the tile stream (8 rows x 16 bytes of a tile are
        // contiguous: full 32-byte sectors), kGmAhead steps ahead of their use, in registers — no shared-memory staging, no copy engine, and
        // the 139 KiB a staged K-tile of 256 rows would take go to the activation stages instead.  A step is converted before its
        // buffer is waited for: between "the tensor core has let go of it" and "it is full again" lie only the stores.
        const int q = warp & 3, z = warp >> 2, hb = z >> 1, ss = z & 1;
        const int n = (q << 5) + lane, r = n & 7;                    // row inside a 128-row tile
        const uint32_t lane_addr = (uint32_t)(q << 5) << 16;
        uint32_t ci = 0, ic = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ic++) {
            const GemmItem it = gemm_item(a, item, tpr);
            const int g = (n >> 3) + hb * 16;
            const bool live = g < it.n_rg;                           // row groups past the matrix's end contribute zeros (and are never read)
            const unsigned char* base = a.seg[it.seg].w + (size_t)(it.rg0 + (live ? g : 0)) * tpr * kTileBytes;
            uint4 rq[kGmAhead][2];
            uint32_t rs[kGmAhead];
            const int si0 = it.t0 * 16 + ss, si1 = it.t1 * 16;
            auto fetch = [&](int si, uint4 (&dq)[2], uint32_t& ds) {
                const unsigned char* tile = base + (size_t)(si >> 4) * kTileBytes;
                dq[0] = live ? __ldg((const uint4*)(tile + (si & 15) * 256 + r * 16)) : make_uint4(0u, 0u, 0u, 0u);
                dq[1] = live ? __ldg((const uint4*)(tile + (si & 15) * 256 + 128 + r * 16)) : make_uint4(0u, 0u, 0u, 0u);
                ds = live ? (uint32_t)__ldg((const unsigned short*)(tile + kTileQ + ((si & 15) * 8 + r) * 2)) : 0u;
            };
#pragma unroll
            for (int d = 0; d < kGmAhead; d++) fetch(si0 + d * kGmStep, rq[d], rs[d]);          // (an item holds whole K-tiles: at least 16 slices)
#pragma unroll 1
            for (int si = si0; si < si1 && ok; si += kGmAhead * kGmStep) {
#pragma unroll
                for (int d = 0; d < kGmAhead; d++) {
                    const uint32_t cb = ci % ncb;
                    const uint32_t dd = h2_mul(rs[d] | (rs[d] << 16), 0x64006400u);            // 1024 d, exact
                    const uint32_t w8[8] = {rq[d][0].x, rq[d][0].y, rq[d][0].z, rq[d][0].w, rq[d][1].x, rq[d][1].y, rq[d][1].z, rq[d][1].w};
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        // bytes (q + 128) into the mantissas of 1024 + (q + 128), two at a time; minus 1152 leaves q, exactly
                        const uint32_t w = w8[j] ^ 0x80808080u;
                        const uint32_t q0 = h2_sub(__byte_perm(w, 0x64646464u, 0x4140), 0x64806480u);
                        const uint32_t q1 = h2_sub(__byte_perm(w, 0x64646464u, 0x4342), 0x64806480u);
                        hi[2 * j] = h2_mul(q0, dd); hi[2 * j + 1] = h2_mul(q1, dd);
                        lo[2 * j] = h2_fma(q0, dd, h2_neg(hi[2 * j]));             // q d' - hi: the rounding error of hi, exactly
                        lo[2 * j + 1] = h2_fma(q1, dd, h2_neg(hi[2 * j + 1]));
                    }
                    if (si + (d + kGmAhead) * kGmStep < si1) fetch(si + (d + kGmAhead) * kGmStep, rq[d], rs[d]);     // this slot's next step
                    if (!mbar_wait_abortable(cempty + 8u * cb, ((ci / ncb) & 1u) ^ 1u, abort)) { fail(LUM_ST_WAIT_EMPTY); ok = false; break; }
                    tc_fence_after_sync();
                    const uint32_t wt = tmem + lane_addr + kGmCvtCol0 + cb * kGmCvtCols + (uint32_t)(ss * kGmHB + hb) * 32u;
                    tmem_st16(wt, hi);
                    tmem_st16(wt + 16u, lo);
                    tmem_st_wait();
                    tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(cfull + 8u * cb);
                    ci++;
                }
            }
            if (!ok) break;
            // ---- the item's K range is done: store the accumulators (lane = weight row, columns = activation rows)
            if (!mbar_wait_abortable(afull, ic & 1u, abort)) { fail(LUM_ST_WAIT_TMEM); ok = false; break; }
            if (a.use_pdl) pdl_grid_wait();              // (long over: the sums are there)
            tc_fence_after_sync();
            const GemmSeg& sg = a.seg[it.seg];
            {
                const int n_st = hb * 128 + n, m0 = it.mc * nc;          // this warp's half of the chunk's rows: every second block of 16
                const bool row_live = (n_st >> 3) < it.n_rg;
                float* yp = a.y + (size_t)it.ks * a.part_stride + sg.col0 + it.rg0 * kTileRows + n_st;
#pragma unroll 1
                for (int c0 = 16 * ss; c0 < nc; c0 += 32) {
                    uint32_t v[16];
                    const float sx_lane = __ldcg(a.sx + m0 + c0 + (lane & 15));
                    tmem_ld16(tmem + lane_addr + (uint32_t)hb * 128u + (uint32_t)c0, v);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const int m = m0 + c0 + i;
                        const float sum = __uint_as_float(v[i]) * __shfl_sync(0xffffffffu, sx_lane, i);
                        if (row_live && m < a.M) yp[(size_t)m * a.ldy] = sum;
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(aempty);
        }
        tc_fence_before_sync();
        named_arrive(4, kGmCvtWarps * 32 + 32);
    }
}


// ===== The kernel for up to 64 activation rows (batched decode, short prompts) =====
// Same arithmetic, but the regime is the other one: the weights are the stream that matters (HBM-bound), and everything else has to
// keep up with 23 bytes of them per SM and clock, which is 187 clocks per 32-column slice of 128 weight rows.
//   * Work items are runs of up to 32 row groups of 8 weight rows, over the concatenated matrices, times a range of K-tiles: the row groups
//     are dealt out evenly (gemm_plan), so that all SMs finish together whatever the K ranges (planes of partial sums).  An item of
//     more than 16 row groups is two tensor-core tiles that take turns on each K-tile and share its activation slices in shared memory.
//   * Weights are staged by bulk copies of whole 4352-byte tiles, half an item's row groups of one K-tile per stage, two stages.
//   * 16 warps convert: four per quarter of the tensor-memory lanes, each one slice of the four of a hand-over (two loads, 32 weights in
//     registers, two stores of 16 columns).  With 8 warps of half a slice the loads' and stores' latencies were exposed.
//   * Tensor core: per 16 columns of K two instructions, hi x [x1 | x2] of N = 2 nc (its two halves are added when the sums are stored) and
//     lo x x1 of N = nc: 33 + 17 clocks at nc = 32.  lo x x1 joins the half of hi x x2, whose values are as small: every addition to an
//     accumulator is cut to 24 bits, so the large half takes one per 16 columns and not two (whole-model error against 64 bits 3.8e-5
//     with both in the large half).
//   * Activations: a chunk is 16, 32 or 64 rows, whichever holds the step; a slice is 128 bytes per row, and with 32 rows a CTA reads as many
//     bytes of them from L2 as of weights from HBM if it has one tensor-core tile, half as many if it has two.
// Measured, alone, back to back over weights that L2 does not hold (us at 32 rows / 5 rows; before: q8_gemm_tc_layer_shapes of the profiles, a chunk
// of 32 rows for both): qkv 6144 x 4096 39.5 -> 16.5 / 14.8, gate|up 28672 x 4096 111.3 -> 52.1 / 45.2 (three K ranges, which gemm_least_split asks for;
// one range: 43.3 / 41.1), down 4096 x 14336 68.8 -> 26.7 / 22.7, vocabulary 128256 x 4096 323.1 -> 152.8 / 141.0 (3.7 and 4.0 TB/s of weights).
// 33 to 64 rows, with their rows' preparation: gate|up 135 -> 76 at 33 rows, 140 -> 85 at 64; down 79 -> 51, 80 -> 52; vocabulary 431 -> 221, 435 ->
// 219.  What is left is latency: set-up and first copies, about 5 us
// that a dependent launch hides, and hand-overs of about 800 clocks per four slices where the conversion's issue slots are 440.
constexpr int kGsRG = 16;                           // row groups per tensor-core tile
constexpr int kGsWRow = kTileBytes;                 // 4352: one tile, quants then scales, as streamed
constexpr int kGsWStage = kGsRG * kGsWRow;          // 69632
constexpr int kGsStep = 4;                          // 32-column slices per hand-over between the warps
constexpr int kGsXStage = 16384;                    // one activation stage: 16384 / (128 nc) slices
constexpr int kGsWStages = 2, kGsCvtBufs = 3, kGsXStages = 4;
constexpr uint32_t kGsSliceCols = 32;               // tensor-memory columns of one converted slice: hi (16: 32 binary16 per row) | lo (16)
constexpr uint32_t kGsCvtCols = kGsStep * kGsSliceCols;
constexpr int kGsCvtWarps = 16;
constexpr int kGsThreads = (kGsCvtWarps + 3) * 32;   // + activation producer warp + tensor-core warp + weight producer warp
constexpr int kGsBarBytes = 256;
constexpr double kGsCvtUs = 1.5;                    // measured: one K-tile (16 slices) of one tensor-core tile through the converting warps
constexpr size_t kGsSmem = kGsBarBytes + 128 + (size_t)kGsWStages * kGsWStage + (size_t)kGsXStages * kGsXStage;
constexpr uint32_t kGsTmemCols = 512;
constexpr uint32_t kGsAccCols = 64, kGsCvtCol0 = 128;   // accumulators: 2 nc <= 64 columns per tile, or (nc = 64, one tile) 128

// item -> row groups [g0, g0 + n) of the concatenated matrices, K-tiles [t0, t1), part of the sums
struct SkinnyItem { int g0, n, t0, t1, ks; };
__device__ __forceinline__ SkinnyItem skinny_item(const GemmArgs& a, int item, int tpr, int groups) {
    SkinnyItem it;
    it.ks = item % a.ksplit;
    const int c = item / a.ksplit;
    it.g0 = (int)((long long)c * groups / a.row_chunks);
    it.n = (int)((long long)(c + 1) * groups / a.row_chunks) - it.g0;
    it.t0 = (int)((long long)it.ks * tpr / a.ksplit);
    it.t1 = (int)((long long)(it.ks + 1) * tpr / a.ksplit);
    return it;
}
// matrix and row group inside it of row group g of the concatenation
__device__ __forceinline__ int skinny_seg(const GemmArgs& a, int& g) {
    int s = 0;
    while (s < a.nseg - 1 && g >= a.seg[s].rows / kTileRows) { g -= a.seg[s].rows / kTileRows; s++; }
    return s;
}
// NC: activation rows of the chunk (a compile-time number: with the index arithmetic done at run time the issuing thread took 86 clocks per
// instruction)
template <int NC>
__global__ void __launch_bounds__(kGsThreads, 1) q8_gemm_tc_skinny(const GemmArgs a) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t bars = smem_u32(smem);
    const uint32_t wfull = bars, wempty = bars + 16, xfull = bars + 32, xempty = bars + 64, cfull = bars + 96, cempty = bars + 128,
                   afull = bars + 160, aempty = bars + 168, fin = bars + 176, tmem_slot = bars + 184;
    static_assert(kGsXStages <= 4 && kGsCvtBufs <= 4 && kGsCvtCol0 + kGsCvtBufs * kGsCvtCols <= kGsTmemCols && kGmXTerms == 2, "barrier area / tensor memory");
    unsigned char* wst = (unsigned char*)(((uintptr_t)smem + kGsBarBytes + 127) & ~(uintptr_t)127);
    unsigned char* xst = wst + (size_t)kGsWStages * kGsWStage;
    volatile int* abort = &s_abort;
    if (tid == 0) {
        s_abort = 0;
        for (int i = 0; i < kGsWStages; i++) { mbar_init(wfull + 8u * i, 1); mbar_init(wempty + 8u * i, kGsCvtWarps); }
        mbar_init(afull, 1); mbar_init(aempty, kGsCvtWarps);
        for (int i = 0; i < kGsCvtBufs; i++) { mbar_init(cfull + 8u * i, kGsCvtWarps); mbar_init(cempty + 8u * i, 1); }
        for (int i = 0; i < kGsXStages; i++) { mbar_init(xfull + 8u * i, 1); mbar_init(xempty + 8u * i, 1); }
        mbar_init(fin, 1);
        mbar_fence_init();
    }
    if (warp == kGsCvtWarps + 1) tmem_alloc(tmem_slot, kGsTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot));
    // The weights do not depend on the previous kernel: they are on their way while it still runs.  Its results are waited for where they
    // are read (activation copies, row factors) or where what it may still read is overwritten (the sums).
    if (a.use_pdl) pdl_launch_dependents();

    const int tpr = a.K / kTileK;
    constexpr int nc = NC;
    constexpr uint32_t x_cg = (uint32_t)kGmXTerms * (uint32_t)nc * 16u;      // bytes of one column group of a slice: both terms' rows
    constexpr uint32_t x_slice = 4u * x_cg;
    constexpr int sps = kGsXStage / (int)x_slice;          // slices per activation stage: 8, 4 or 2
    int groups = 0;
    for (int s = 0; s < a.nseg; s++) groups += a.seg[s].rows / kTileRows;
    const int n_items = a.row_chunks * a.ksplit;
    auto fail = [&](uint32_t code) { if (!*abort) { atomicOr(a.status, code); *abort = 1; } };
    // row groups of tensor-core tile hb of an item of n: all of them, or halves
    auto tiles_of = [](int n) { return n > kGsRG ? 2 : 1; };
    auto first_of = [](int n, int hb) { return hb ? (n + 1) / 2 : 0; };
    auto count_of = [](int n, int hb) { return n <= kGsRG ? n : hb ? n / 2 : (n + 1) / 2; };

    if (warp == kGsCvtWarps + 2) {
        // ---------------------------------------------------------------- weight producer warp: lane = row group
        uint32_t wi = 0;
        int ok = 1;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            const SkinnyItem it = skinny_item(a, item, tpr, groups);
            const int hbs = tiles_of(it.n);
            const unsigned char* src[2];                   // this lane's row group of each tensor-core tile
#pragma unroll
            for (int hb = 0; hb < 2; hb++) {
                int g = it.g0 + first_of(it.n, hb) + (lane < count_of(it.n, hb) ? lane : 0);
                if (hb >= hbs) g = it.g0;
                const int sg = skinny_seg(a, g);
                src[hb] = a.seg[sg].w + (size_t)g * tpr * kTileBytes;
            }
            for (int t = it.t0; t < it.t1 && ok; t++) {
                for (int hb = 0; hb < hbs; hb++) {
                    const uint32_t ws = wi % kGsWStages;
                    const int cnt = count_of(it.n, hb);
                    if (lane == 0) {
                        if (!mbar_wait_abortable(wempty + 8u * ws, ((wi / kGsWStages) & 1u) ^ 1u, abort)) { fail(LUM_ST_WAIT_EMPTY); ok = 0; }
                        else mbar_arrive_expect_tx(wfull + 8u * ws, (uint32_t)cnt * kGsWRow);
                    }
                    ok = __shfl_sync(0xffffffffu, ok, 0);
                    if (!ok) break;
                    if (lane < cnt)
                        bulk_g2s(smem_u32(wst + (size_t)ws * kGsWStage + (size_t)lane * kGsWRow), (hb ? src[1] : src[0]) + (size_t)t * kTileBytes, kTileBytes, wfull + 8u * ws);
                    wi++;
                }
            }
        }
        // never leave while a copy into this CTA's shared memory may be in flight: wait (bounded) for what was armed
        if (!ok && lane == 0)
            for (uint32_t k = 0; k < kGsWStages && k < wi; k++) { const uint32_t i = wi - 1 - k; mbar_wait(wfull + 8u * (i % kGsWStages), (i / kGsWStages) & 1u); }
        return;
    }
    if (warp == kGsCvtWarps) {
        // ---------------------------------------------------------------- activation producer: one lane, one copy per stage
        if (elect_one()) {
            uint32_t xi = 0;
            bool ok = true;
            if (a.use_pdl) pdl_grid_wait();
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                const SkinnyItem it = skinny_item(a, item, tpr, groups);
                for (int s = it.t0 * 16; s < it.t1 * 16; s += sps) {
                    const uint32_t xs = xi % kGsXStages;
                    if (!mbar_wait_abortable(xempty + 8u * xs, ((xi / kGsXStages) & 1u) ^ 1u, abort)) { fail(LUM_ST_WAIT_EMPTY); ok = false; break; }
                    mbar_arrive_expect_tx(xfull + 8u * xs, kGsXStage);
                    bulk_g2s(smem_u32(xst + (size_t)xs * kGsXStage), (const unsigned char*)a.xq + (size_t)s * x_slice, kGsXStage, xfull + 8u * xs);
                    xi++;
                }
            }
            if (!ok)
                for (uint32_t k = 0; k < kGsXStages && k < xi; k++) { const uint32_t i = xi - 1 - k; mbar_wait(xfull + 8u * (i % kGsXStages), (i / kGsXStages) & 1u); }
        }
        return;
    }
    if (warp == kGsCvtWarps + 1) {
        // ---------------------------------------------------------------- tensor-core warp: one thread issues
        if (elect_one()) {
            uint32_t x0 = 0, ci = 0, ic = 0;               // x0: activation stages before the current K-tile
            bool ok = true;
            constexpr uint32_t idesc2 = umma_idesc_f16(128, 2 * nc), idesc1 = umma_idesc_f16(128, nc);
            // activation operand descriptors: start address in the low 14 bits; column groups x_cg bytes apart, 8-row groups 128
            constexpr uint32_t x_lo = ((x_cg >> 4) & 0x3fffu) << 16, x_hi = umma_desc_hi(128u);
            const uint32_t x_base = smem_u32(xst);
            constexpr int spt = 16 / sps;                  // activation stages per K-tile
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ic++) {
                const SkinnyItem it = skinny_item(a, item, tpr, groups);
                const int hbs = tiles_of(it.n);
                if (!mbar_wait_abortable(aempty, (ic & 1u) ^ 1u, abort)) { fail(LUM_ST_WAIT_TMEM); break; }      // the previous item's sums were stored
                tc_fence_after_sync();
                for (int t = it.t0; t < it.t1 && ok; t++, x0 += (uint32_t)spt) {
                    for (int hb = 0; hb < hbs && ok; hb++) {
                        const uint32_t acc = tmem + (uint32_t)hb * kGsAccCols;
#pragma unroll
                        for (int s = 0; s < 16; s += kGsStep, ci++) {
                            const uint32_t cb = ci % kGsCvtBufs;
                            if (!mbar_wait_abortable(cfull + 8u * cb, (ci / kGsCvtBufs) & 1u, abort)) { fail(LUM_ST_WAIT_FULL); ok = false; break; }
                            tc_fence_after_sync();
                            const uint32_t wt = tmem + kGsCvtCol0 + cb * kGsCvtCols;
#pragma unroll
                            for (int ss = 0; ss < kGsStep; ss++) {
                                const int sub = (s + ss) % sps;               // the slice inside its activation stage
                                const uint32_t xi = x0 + (uint32_t)((s + ss) / sps), xs = xi % kGsXStages;
                                if (sub == 0 && hb == 0 && !mbar_wait_abortable(xfull + 8u * xs, (xi / kGsXStages) & 1u, abort)) { fail(LUM_ST_WAIT_FULL); ok = false; break; }
                                const uint32_t xb = x_base + xs * (uint32_t)kGsXStage + (uint32_t)sub * x_slice;
#pragma unroll
                                for (int kk = 0; kk < 2; kk++) {      // K = 16 per instruction: two per 32-column slice
                                    // weights: tensor memory, 8 columns (16 binary16) per instruction; activations: shared memory,
                                    // [column group of 8][term][row][16 bytes], an instruction reads two adjacent column groups
                                    const uint32_t x12 = x_lo | (((xb + (uint32_t)kk * 2u * x_cg) >> 4) & 0x3fffu);
                                    const uint32_t hi = wt + (uint32_t)ss * kGsSliceCols + (uint32_t)kk * 8u;
                                    umma_f16_ts2(acc, hi, x12, x_hi, idesc2, (t > it.t0 || s + ss + kk > 0) ? 1u : 0u);
                                    umma_f16_ts2(acc + (uint32_t)nc, hi + 16u, x12, x_hi, idesc1, 1u);
                                }
                                if (sub == sps - 1 && hb == hbs - 1) umma_commit(xempty + 8u * xs);       // the tile that reads it last has done so
                            }
                            if (!ok) break;
                            umma_commit(cempty + 8u * cb);        // arrive when the instructions that read these operands have retired
                        }
                    }
                }
                if (ok) umma_commit(afull);
            }
            umma_commit(fin);
            if (!mbar_wait(fin, 0u)) atomicOr(a.status, LUM_ST_WAIT_TMEM);
        }
        __syncwarp();
        named_sync(4, kGsCvtWarps * 32 + 32);
        tc_fence_after_sync();
        tmem_dealloc(tmem, kGsTmemCols);
        return;
    }

    // -------------------------------------------------------------------- converting / storing warps
    {
        // a warp reaches the 32 tensor-memory lanes of its quarter: thread = weight row of the tile (lane of tensor memory); of a
        // hand-over's four slices it converts number z (and stores columns 16 z .. of the sums)
        const int q = warp & 3, z = warp >> 2;
        const int n = (q << 5) + lane, g = n >> 3, r = n & 7;        // row, row group inside the tile, row inside that
        const uint32_t lane_addr = (uint32_t)(q << 5) << 16;
        uint32_t wi = 0, ci = 0, ic = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x, ic++) {
            const SkinnyItem it = skinny_item(a, item, tpr, groups);
            const int hbs = tiles_of(it.n);
            for (int t = it.t0; t < it.t1 && ok; t++) {
                for (int hb = 0; hb < hbs && ok; hb++) {
                    const uint32_t ws = wi % kGsWStages;
                    if (!mbar_wait_abortable(wfull + 8u * ws, (wi / kGsWStages) & 1u, abort)) { fail(LUM_ST_WAIT_FULL); ok = false; break; }
                    // a quarter without rows converts nothing (its lanes' sums are never stored); lanes past the last row read stale bytes
                    // of the stage, for the same reason
                    const bool live = q * 4 < count_of(it.n, hb);
                    const unsigned char* tile = wst + (size_t)ws * kGsWStage + (size_t)g * kGsWRow;
#pragma unroll 2
                    for (int s0 = 0; s0 < 16; s0 += kGsStep, ci++) {
                        const uint32_t cb = ci % kGsCvtBufs;
                        const int s = s0 + z;
                        // converted before the buffer is waited for: the wait then costs no arithmetic
                        uint32_t hi[16], lo[16];
                        if (live) {
                            const uint4 raw0 = *(const uint4*)(tile + s * 256 + r * 16), raw1 = *(const uint4*)(tile + s * 256 + 128 + r * 16);
                            const uint32_t d16 = (uint32_t)*(const unsigned short*)(tile + kTileQ + (s * 8 + r) * 2);
                            const uint32_t dd = h2_mul(d16 | (d16 << 16), 0x64006400u);            // 1024 d, exact
                            const uint32_t w8[8] = {raw0.x, raw0.y, raw0.z, raw0.w, raw1.x, raw1.y, raw1.z, raw1.w};
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                // bytes (q + 128) into the mantissas of 1024 + (q + 128), two at a time; minus 1152 leaves q, exactly
                                const uint32_t w = w8[j] ^ 0x80808080u;
                                const uint32_t q0 = h2_sub(__byte_perm(w, 0x64646464u, 0x4140), 0x64806480u);
                                const uint32_t q1 = h2_sub(__byte_perm(w, 0x64646464u, 0x4342), 0x64806480u);
                                hi[2 * j] = h2_mul(q0, dd); hi[2 * j + 1] = h2_mul(q1, dd);
                                lo[2 * j] = h2_fma(q0, dd, h2_neg(hi[2 * j]));             // q d' - hi: the rounding error of hi, exactly
                                lo[2 * j + 1] = h2_fma(q1, dd, h2_neg(hi[2 * j + 1]));
                            }
                        }
                        if (!mbar_wait_abortable(cempty + 8u * cb, ((ci / kGsCvtBufs) & 1u) ^ 1u, abort)) { fail(LUM_ST_WAIT_EMPTY); ok = false; break; }
                        tc_fence_after_sync();
                        if (live) {
                            const uint32_t wt = tmem + lane_addr + kGsCvtCol0 + cb * kGsCvtCols + (uint32_t)z * kGsSliceCols;
                            tmem_st16(wt, hi);
                            tmem_st16(wt + 16u, lo);
                            tmem_st_wait();
                        }
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(cfull + 8u * cb);
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(wempty + 8u * ws);
                    wi++;
                }
            }
            if (!ok) break;
            // ---- the item's K range is done: store the accumulators (lane = weight row, columns = activation rows)
            if (!mbar_wait_abortable(afull, ic & 1u, abort)) { fail(LUM_ST_WAIT_TMEM); ok = false; break; }
            if (a.use_pdl) pdl_grid_wait();              // (long over: the sums are there)
            tc_fence_after_sync();
            if (16 * z < nc && 16 * z < a.M) {
                // one request per warp: every CTA wants the same few bytes at the same time (a load per row and warp cost 2 us at 32 rows)
                const float sx_lane = __ldcg(a.sx + 16 * z + (lane & 15));
#pragma unroll 1
                for (int hb = 0; hb < hbs; hb++) {
                    const bool row_live = g < count_of(it.n, hb);
                    int rg = it.g0 + first_of(it.n, hb) + (row_live ? g : 0);
                    const int sg = skinny_seg(a, rg);
                    float* yp = a.y + (size_t)it.ks * a.part_stride + a.seg[sg].col0 + rg * kTileRows + r;
                    uint32_t v[16], v2[16];
                    const uint32_t col = tmem + lane_addr + (uint32_t)hb * kGsAccCols + (uint32_t)(16 * z);
                    tmem_ld16(col, v);
                    tmem_ld16(col + (uint32_t)nc, v2);              // the x2 half of the accumulator
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        const int m = 16 * z + i;
                        const float sum = (__uint_as_float(v[i]) + __uint_as_float(v2[i])) * __shfl_sync(0xffffffffu, sx_lane, i);
                        if (row_live && m < a.M) yp[(size_t)m * a.ldy] = sum;
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(aempty);
        }
        tc_fence_before_sync();
        named_arrive(4, kGsCvtWarps * 32 + 32);
    }
}


// ---------------------------------------------------------------------------------------------------------- host side

// rows of the activation operand: M and what fills the last chunk, whatever the chunk
static int gemm_padded_rows(int M) { return M <= 64 ? 64 : M + kGmMaxChunk - 1; }
size_t gemm_xq_bytes(int M, int K) { return (size_t)gemm_padded_rows(M) * K * 2 * kGmXTerms; }
size_t gemm_sx_bytes(int M, int K) { (void)K; return (size_t)gemm_padded_rows(M) * 4; }

// Shapes hold for whole blocks of 16 rows: whoever sizes a buffer for every row count asks once per block (gemm_parts_rows).
constexpr int kGmBlock = 16;
static int block_first(int M) { return (M - 1) / kGmBlock * kGmBlock + 1; }
static int block_last(int M) { return (M + kGmBlock - 1) / kGmBlock * kGmBlock; }

// The fewest K ranges a product may be cut into.  An accumulator's additions are cut to 24 bits, always towards zero: longer ranges cost accuracy,
// and with operands of one sign the loss grows with the length.  So the split that a first, coarse estimate of the time gives (chunks of 32, 64
// or 128 rows, items of 128 or 256 weight rows) is never undercut, whatever the finer estimates below would gain.
// Measured, 28672 x 4096 at 2 to 64 rows, one range / three, error against 64 bits: normal operands 4.9e-6 / 1.7e-6, operands of one sign
// 2.6e-5 / 8.0e-6; 16384 x 16384, one / eight: 1.07e-4 / 1.3e-5.
static int gemm_least_split(int n_rows_total, int M, int K, int sm_count) {
    const int nc = M <= 32 ? 32 : M <= 64 ? 64 : 128, tile_rows = M > 64 ? kGmRows : 128;
    const int items = (n_rows_total + tile_rows - 1) / tile_rows * ((M + nc - 1) / nc), tpr = K / kTileK;
    const double tile_us = M > 64 ? 14.4 : 16.0 * (0.16 + 0.43 * nc / 128.0), plane_us = (double)block_first(M) * n_rows_total * 8.0 / 6.5e6;
    auto cost = [&](int k) { return (double)(((long long)items * k + sm_count - 1) / sm_count) * ((double)tpr / k + 0.33) * tile_us + (k - 1) * plane_us; };
    int best = 1;
    for (int ks = 2; ks <= kMaxKsplit && ks <= tpr; ks++)
        if (cost(ks) < cost(best) * 0.97) best = ks;                          // a larger split has to pay for itself
    return best;
}

// Up to 64 rows: K ranges (at least `least`) and runs of row groups of a product.  An SM's time for one K-tile of n row groups is the largest of: its
// share of HBM (4352 n bytes at 44 GB/s), the conversion (kGsCvtUs per tensor-core tile), and what comes
// in from L2 and HBM together (90 GB/s); an item costs about 2.5 us beside that, a plane of partial sums its write and read at the copy rate.
struct SkinnyPlan { int ks, chunks; };
static SkinnyPlan gemm_plan(int groups, int nc, int K, int sms, int least) {
    const int tpr = K / kTileK, most = nc == 64 ? kGsRG : 2 * kGsRG;       // two tiles share activation slices that are all resident
    SkinnyPlan best{least, (groups + most - 1) / most};
    double best_t = 1e30;
    for (int ks = least; ks <= kMaxKsplit && ks <= tpr; ks++) {
        const double plane_us = (double)nc * groups * kTileRows * 8.0 / 6.5e6;
        for (int p = 1; p <= 64; p++) {                                     // items per SM
            int chunks = (int)((long long)sms * p / ks);
            if (chunks < 1) continue;
            if (chunks > groups) chunks = groups;
            const int n = (groups + chunks - 1) / chunks;
            if (n > most) continue;
            const double hbm = 4352.0 * n / 44e3, cvt = kGsCvtUs * (n > kGsRG ? 2 : 1), in = (4352.0 * n + 16.0 * 128.0 * nc) / 90e3;
            const double tile_us = hbm > cvt ? (hbm > in ? hbm : in) : (cvt > in ? cvt : in);
            const int rounds = (int)(((long long)chunks * ks + sms - 1) / sms);
            const double t = rounds * ((double)((tpr + ks - 1) / ks) * tile_us + 2.5) + (ks - 1) * plane_us;
            if (t < best_t * 0.98) { best_t = t; best = {ks, chunks}; }
            if (chunks == groups) break;
        }
    }
    return best;
}

// More rows: rows per chunk and K ranges (at least `least`) per product.  Work items are equal, so a product takes ceil(items / SMs) rounds of one item
// each: with few items per SM the last, partly filled round is a large share of the time (448 items over 148 SMs: 4 rounds for 3.03 rounds of work), and so are the
// rows that fill up the last chunk (387 rows in chunks of 128: a quarter).  Smaller chunks and more K ranges make both finer, but every item pays
// its own pipeline fill and store, every extra range writes (and the consumer reads) another plane of partial sums, and the
// converting warps set a floor.  Constants: measured, us per K-tile of one item (28672 x 4096 in chunks of 80 / 112 / 128 rows: 6.6 / 8.1 / 8.75),
// an item's own cost a third of that, planes at the HBM copy rate.
// Measured, alone, us (chunks of 128 / as chosen): 28672 x 4096 at 65 rows 74 / 58, 129 rows 143 / 109, 387 rows 264 / 231, 1000 rows 487 / 449.
// Other products, with their rows' preparation, against the kernel of chunks of 128 before it: 4096 x 14336 at 65 / 387 / 1000 rows 85 / 232 / 439 -> 52 / 159 /
// 308, 19456 x 2560 82 / 235 / 347 -> 51 / 171 / 242, 2560 x 9728 63 / 124 / 234 -> 41 / 93 / 182.
static GemmShape gemm_shape_wide(int n_rows_total, int M, int K, int sm_count, int least) {
    const int tiles = (n_rows_total + kGmRows - 1) / kGmRows, tpr = K / kTileK;
    const double plane_us = (double)block_last(M) * n_rows_total * 8.0 / 6.5e6;   // write + read of one plane of partial sums
    auto cost = [&](int nc, int ks, double t_tile) {
        const int rounds = (tiles * ((M + nc - 1) / nc) * ks + sm_count - 1) / sm_count;
        return (double)rounds * ((double)((tpr + ks - 1) / ks) * t_tile + 0.33 * t_tile) + (ks - 1) * plane_us;
    };
    GemmShape best{kGmMaxChunk, least};
    auto tile = [](int nc) { return 2.9 + 5.85 * nc / kGmMaxChunk; };
    double best_t = cost(kGmMaxChunk, least, tile(kGmMaxChunk));
    for (int nc = kGmMaxChunk; nc >= 80; nc -= 16)
        for (int ks = least; ks <= kMaxKsplit && ks <= tpr; ks++) {
            const double t = cost(nc, ks, tile(nc));
            if (t < best_t * 0.98) { best_t = t; best = {nc, ks}; }
        }
    return best;
}
GemmShape gemm_shape(int n_rows_total, int M, int K, int sm_count) {
    const int least = gemm_least_split(n_rows_total, M, K, sm_count);
    if (M > 64) return gemm_shape_wide(n_rows_total, M, K, sm_count, least);
    const int nc = M <= 16 ? 16 : M <= 32 ? 32 : 64;
    return {nc, gemm_plan(n_rows_total / kTileRows, nc, K, sm_count, least).ks};
}
// The most rows of partial sums (K ranges times rows) a product of up to `cap` rows needs.  Larger row counts come first, and those that even the
// largest split could not bring above what was found are not looked at: a model's four products of up to 4096 rows take 0.25 ms (3.4 ms row by
// row), once, when its buffers are made.
size_t gemm_parts_rows(int n_rows_total, int K, int cap, int sm_count) {
    size_t worst = 0;
    for (int m = cap; m >= 1 && (size_t)kMaxKsplit * m > worst; m = block_first(m) - 1) {
        const size_t need = (size_t)gemm_shape(n_rows_total, m, K, sm_count).ks * m;
        if (need > worst) worst = need;
    }
    return worst;
}

cudaError_t launch_rows_quantize(const RowsArgs& a_in, int sm_count, cudaStream_t st) {
    RowsArgs a = a_in;
    if (a.M <= 0 || a.K <= 0 || (a.K % 32) || a.n_parts < 1 || a.nc < 16 || a.nc > kGmMaxChunk || a.nc % 16) return cudaErrorInvalidValue;
    const int nc = a.nc;
    const int rows = (a.M + nc - 1) / nc * nc;            // padding rows of the last chunk are zeroed by their own CTAs
    // CTAs per row: up to eight while the rows alone leave SMs idle, of at least eight slices each
    int C = 1;
    while (C < kRqMaxCluster && rows * C * 2 <= 4 * sm_count && (a.K >> 5) / (C * 2) >= 8) C *= 2;
    // Two rows per CTA where there is one CTA per row and both fit (`rows` is a multiple of 16): see the kernel
    const size_t two = (size_t)2 * (a.K + kRqPad) * 4;
    const bool pair = C == 1 && two <= 200 * 1024;
    const size_t smem = pair ? two : (size_t)(((a.K >> 5) + C - 1) / C) * 128;
    if (smem > 200 * 1024) return cudaErrorInvalidValue;
    const void* fn = pair ? (const void*)rows_quantize<2> : (const void*)rows_quantize<1>;
    if (smem > 48 * 1024) {
        static std::atomic<uint64_t> raised[2] = {};
        if (const cudaError_t e = allow_smem(raised[pair], fn, 200 * 1024)) return e;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pair ? rows / 2 : rows * C);
    cfg.blockDim = dim3(pair ? 512 : 256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    int n_at = 0;
    if (C > 1) {
        at[n_at].id = cudaLaunchAttributeClusterDimension;
        at[n_at].val.clusterDim.x = (unsigned)C; at[n_at].val.clusterDim.y = 1; at[n_at].val.clusterDim.z = 1;
        n_at++;
    }
    if (a.use_pdl) {
        at[n_at].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n_at].val.programmaticStreamSerializationAllowed = 1;
        n_at++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n_at;
    void* params[] = {&a, &C};
    return cudaLaunchKernelExC(&cfg, fn, params);
}

bool gemm_supported(const GemmArgs& a) {
    if (a.nseg < 1 || a.nseg > 3 || a.K <= 0 || a.K % kTileK || a.M <= 0) return false;
    for (int s = 0; s < a.nseg; s++)
        if (a.seg[s].rows <= 0 || a.seg[s].rows % kTileRows || ((uintptr_t)a.seg[s].w & 15)) return false;
    return a.ksplit >= 1 && a.ksplit <= a.K / kTileK;
}

cudaError_t launch_gemm(const GemmArgs& a_in, int sm_count, cudaStream_t st) {
    GemmArgs a = a_in;
    if (a.M <= 0 || (a.M <= 64 ? a.nc != 16 && a.nc != 32 && a.nc != 64 : a.nc < 80) || a.nc > kGmMaxChunk || a.nc % 16 || (a.M <= 64 && a.nc < a.M)) return cudaErrorInvalidValue;
    a.m_chunks = (a.M + a.nc - 1) / a.nc;
    if (!gemm_supported(a)) return cudaErrorInvalidValue;
    // more than 64 rows (prompts): the tensor core is the resource; fewer (batched decode): the weight stream is
    const bool wide = a.nc > 64;
    const void* fn = wide ? (const void*)q8_gemm_tc : a.nc == 16 ? (const void*)q8_gemm_tc_skinny<16> : a.nc == 32 ? (const void*)q8_gemm_tc_skinny<32> : (const void*)q8_gemm_tc_skinny<64>;
    const size_t smem = wide ? kGmSmem : kGsSmem;
    const int threads = wide ? kGmThreads : kGsThreads;
    static std::atomic<uint64_t> raised[4] = {};
    if (const cudaError_t e = allow_smem(raised[wide ? 3 : a.nc / 32], fn, (int)smem)) return e;
    long long items = 0;
    if (wide) {
        for (int s = 0; s < a.nseg; s++) items += (a.seg[s].rows + kGmRows - 1) / kGmRows;
        items *= (long long)a.ksplit * a.m_chunks;
    } else {
        // the row groups of one K range over the SMs it has, in as many rounds as the plan takes (the split itself was the caller's choice)
        int groups = 0;
        for (int s = 0; s < a.nseg; s++) groups += a.seg[s].rows / kTileRows;
        const SkinnyPlan p = gemm_plan(groups, a.nc, a.K, sm_count, gemm_least_split(groups * kTileRows, a.M, a.K, sm_count));
        const int most = a.nc == 64 ? kGsRG : 2 * kGsRG;
        a.row_chunks = p.ks == a.ksplit ? p.chunks : (groups + most - 1) / most;
        items = (long long)a.row_chunks * a.ksplit;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items < sm_count ? items : sm_count));
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = a.use_pdl ? 1 : 0;
    void* params[] = {&a};
    return cudaLaunchKernelExC(&cfg, fn, params);
}

// y[m][n] = sum over parts (stand-alone operator only: inside a model the next rows_quantize adds the parts up)
__global__ void gemm_sum_parts(const float* parts, int n_parts, size_t part_stride, float* y, size_t total) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    float v = 0.0f;
    for (int p = 0; p < n_parts; p++) v += parts[p * part_stride + i];
    y[i] = v;
}

}  // namespace lum

// ---------------------------------------------------------------------------------------------------------- C ABI

extern "C" size_t lum_op_gemm_q8_0_workspace(int32_t n, int32_t k, int32_t m) {
    using namespace lum;
    if (n <= 0 || k <= 0 || m <= 0 || k % kTileK || n % kTileRows) return 0;
    const int ks = gemm_shape(n, m, k, 148).ks;
    return gemm_xq_bytes(m, k) + gemm_sx_bytes(m, k) + (size_t)ks * m * n * 4 + 1024;
}

extern "C" int32_t lum_op_gemm_q8_0_packed(const void* packed, int32_t n, int32_t k, const float* x, int32_t m, float* y, void* workspace,
                                           size_t workspace_bytes, void* stream) {
    using namespace lum;
    const size_t need = lum_op_gemm_q8_0_workspace(n, k, m);
    if (!packed || !x || !y || !workspace || !need || workspace_bytes < need || !q8_pack_kc(n, k)) {
        set_op_error("gemm_q8_0_packed: bad arguments (needs K % 512 == 0, K <= 16384, N % 8 == 0 and a workspace of lum_op_gemm_q8_0_workspace bytes)");
        return -1;
    }
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
    unsigned char* ws = (unsigned char*)(((uintptr_t)workspace + 255) & ~(uintptr_t)255);
    int8_t* xq = (int8_t*)ws;
    float* sx = (float*)(ws + gemm_xq_bytes(m, k));
    float* parts = (float*)(ws + gemm_xq_bytes(m, k) + gemm_sx_bytes(m, k));
    static uint32_t* status[64] = {nullptr};
    if (dev < 0 || dev >= 64) { set_op_error("gemm_q8_0_packed: device ordinal"); return -2; }
    if (!status[dev]) {
        if (cudaMalloc((void**)&status[dev], 4) != cudaSuccess) { set_op_error("gemm_q8_0_packed: status word"); return -5; }
        cudaMemset(status[dev], 0, 4);
    }
    const GemmShape shape = gemm_shape(n, m, k, 148);
    RowsArgs r{};
    r.nc = shape.nc; r.a = x; r.n_parts = 1; r.part_stride = 0; r.ld = k; r.M = m; r.K = k; r.xq = xq; r.sx = sx;
    cudaError_t e = launch_rows_quantize(r, sms, st);
    GemmArgs g{};
    g.nseg = 1; g.seg[0] = {(const unsigned char*)packed, n, 0}; g.K = k; g.xq = xq; g.sx = sx; g.M = m;
    g.nc = shape.nc; g.ksplit = shape.ks;
    g.y = g.ksplit > 1 ? parts : y; g.ldy = n; g.part_stride = (size_t)m * n; g.status = status[dev];
    if (e == cudaSuccess) e = launch_gemm(g, sms, st);
    if (e == cudaSuccess && g.ksplit > 1) {
        const size_t total = (size_t)m * n;
        gemm_sum_parts<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(parts, g.ksplit, g.part_stride, y, total);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) { set_op_error(cudaGetErrorString(e)); return -2; }
    return 0;
}
