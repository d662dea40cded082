// Kernels called through the library's own launchers, without a model around them, against sums in 64 bits.  One check per command; prints a line
// per case: name, largest or relative error, bound.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "lum_dense.cuh"
#include "lum_gemv_dev.cuh"
#include "lum_moe.cuh"
#include "lum_rows.cuh"

using namespace lum;

#define CK(x) do { const cudaError_t e_ = (x); if (e_ != cudaSuccess) { std::printf("%s: %s\n", #x, cudaGetErrorString(e_)); std::exit(2); } } while (0)

static int failures = 0;
static void report(const std::string& what, double err, double bound) {
    const bool ok = err <= bound;                       // (false for a NaN)
    if (!ok) failures++;
    std::printf("%s %s: %.3e, bound %.3e\n", ok ? "ok" : "FAILED", what.c_str(), err, bound);
}

template <typename T> struct Dev {                      // a device array, filled from or read into a vector
    T* p = nullptr; size_t n;
    explicit Dev(size_t n_) : n(n_) { CK(cudaMalloc(&p, n * sizeof(T))); CK(cudaMemset(p, 0, n * sizeof(T))); }
    explicit Dev(const std::vector<T>& v) : Dev(v.size()) { put(v); }
    ~Dev() { cudaFree(p); }
    Dev(const Dev&) = delete;
    void put(const std::vector<T>& v) { CK(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice)); }
    std::vector<T> get() const { std::vector<T> v(n); CK(cudaDeviceSynchronize()); CK(cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost)); return v; }
};

static std::vector<float> normal(std::mt19937& rng, size_t n, float std, float mean = 0.0f) {
    std::normal_distribution<float> d(mean, std);
    std::vector<float> v(n);
    for (float& x : v) x = d(rng);
    return v;
}
static uint16_t bf16_bits(float x) { uint32_t u; std::memcpy(&u, &x, 4); return (uint16_t)((u + 0x7fffu + ((u >> 16) & 1u)) >> 16); }
static float bf16_value(uint16_t b) { const uint32_t u = (uint32_t)b << 16; float x; std::memcpy(&x, &u, 4); return x; }
static std::vector<uint16_t> to_bf16(const std::vector<float>& v) { std::vector<uint16_t> b(v.size()); for (size_t i = 0; i < v.size(); i++) b[i] = bf16_bits(v[i]); return b; }
static double rel(const std::vector<float>& got, const std::vector<double>& want) {
    double a = 0, b = 0;
    for (size_t i = 0; i < want.size(); i++) { a += (got[i] - want[i]) * (got[i] - want[i]); b += want[i] * want[i]; }
    return std::sqrt(a / b);
}

// ---- attention of one token behind n cached rows of bf16 keys and values; queries as given (the rotation's angles are zero)
struct Attention {
    int nq, nkv, hd, n, max_seq;
    std::vector<float> q;
    std::vector<uint16_t> k, v;                         // n + 1 rows: the last is the token's own
    Attention(int nq_, int nkv_, int hd_, int n_, float q_std, float v_mean) : nq(nq_), nkv(nkv_), hd(hd_), n(n_), max_seq((n_ + 64) / 64 * 64 + 64) {
        std::mt19937 rng(n + nq);
        q = normal(rng, (size_t)nq * hd, q_std);
        k = to_bf16(normal(rng, (size_t)max_seq * nkv * hd, 1.0f));
        v = to_bf16(normal(rng, (size_t)max_seq * nkv * hd, 1.0f, v_mean));
    }
    std::vector<double> exact() const {
        std::vector<double> out((size_t)nq * hd), w(n + 1);
        for (int h = 0; h < nq; h++) {
            const size_t col = (size_t)(h / (nq / nkv)) * hd, ld = (size_t)nkv * hd;
            double mx = -INFINITY, l = 0;
            for (int j = 0; j <= n; j++) {
                double d = 0;
                for (int e = 0; e < hd; e++) d += (double)q[(size_t)h * hd + e] * bf16_value(k[j * ld + col + e]);
                w[j] = d * (double)(1.0f / std::sqrt((float)hd));
                mx = std::fmax(mx, w[j]);
            }
            for (int j = 0; j <= n; j++) l += w[j] = std::exp(w[j] - mx);
            for (int j = 0; j <= n; j++)
                for (int e = 0; e < hd; e++) out[(size_t)h * hd + e] += w[j] / l * bf16_value(v[j * ld + col + e]);
        }
        return out;
    }
    std::vector<float> own(const std::vector<uint16_t>& c) const {
        std::vector<float> r((size_t)nkv * hd);
        for (size_t i = 0; i < r.size(); i++) r[i] = bf16_value(c[(size_t)n * nkv * hd + i]);
        return r;
    }
    // one decode step's kernel
    std::vector<float> step(int splits, bool cluster) const {
        DecodeState s{};
        s.pos = n; s.max_seq = max_seq;
        Dev<float> dq(q), dk(own(k)), dv(own(v)), out(q.size()), part((size_t)nq * splits * (hd + 2)), inv_freq((size_t)hd / 2);
        Dev<uint16_t> kc(k), vc(v);
        Dev<unsigned int> counters((size_t)nkv);
        Dev<uint32_t> status(1);
        Dev<DecodeState> state(std::vector<DecodeState>{s});
        AttnArgs a{};
        a.q = dq.p; a.k_new = dk.p; a.v_new = dv.p; a.k_cache = kc.p; a.v_cache = vc.p; a.out = out.p; a.part = part.p; a.counters = counters.p; a.state = state.p;
        a.n_q = nq; a.n_kv = nkv; a.hd = hd; a.n_splits = splits; a.kv_bf16 = 1; a.rope_style = 2; a.inv_freq = inv_freq.p; a.attn_factor = 1.0f; a.max_seq = max_seq;
        a.status = status.p; a.cluster = cluster;
        CK(launch_attn_decode(a, nullptr));
        return out.get();
    }
    // the same token as one of a step of several rows
    std::vector<float> row() const {
        Dev<float> dq(q), out(q.size());
        Dev<uint16_t> kc(k), vc(v);
        Dev<uint32_t> status(1);
        Dev<int> pos(std::vector<int>{n});
        AttnRowsArgs a{};
        a.q_rot = dq.p; a.k_cache = kc.p; a.v_cache = vc.p; a.row_pos = pos.p; a.out = out.p; a.M = 1; a.n_q = nq; a.n_kv = nkv; a.hd = hd; a.kv_bf16 = 1;
        a.max_seq = max_seq; a.max_batch = 1; a.status = status.p;
        CK(launch_attn_rows(a, 148, nullptr));
        return out.get();
    }
};

// Rows of a prompt behind `first` cached ones: tiles of 128 keys and of 128 / (heads per K/V head) rows, on and off their edges; a cache of pages.
static void attention_prompt() {
    struct Case { int nq, nkv, rows, first; bool pages; };
    const std::vector<Case> cases = {{8, 2, 16, 0, false},   {4, 4, 128, 0, false},  {4, 4, 129, 127, false}, {8, 2, 33, 95, false},  {16, 2, 17, 111, true},
                                     {8, 2, 96, 1000, true}, {8, 4, 65, 191, true},  {4, 1, 31, 383, false},  {8, 1, 200, 56, false}, {2, 2, 300, 1, true}};
    for (const Case& c : cases) {
        const int hd = 128, n = c.first + c.rows, max_seq = (n + 63) / 64 * 64, G = c.nq / c.nkv;
        std::mt19937 rng(n * 7 + c.nq);
        const size_t ld = (size_t)c.nkv * hd, qd = (size_t)c.nq * hd;
        const std::vector<float> q = normal(rng, (size_t)c.rows * qd, 1.0f);
        std::vector<uint16_t> k = to_bf16(normal(rng, max_seq * ld, 1.0f)), v = to_bf16(normal(rng, max_seq * ld, 1.0f, 0.5f));
        std::vector<int> pos(c.rows), table(max_seq / 64);
        for (int i = 0; i < c.rows; i++) pos[i] = c.first + i;
        std::vector<uint16_t> kp = k, vp = v;               // with pages: in another order, and what no row may see is not a number
        for (int i = 0; i < max_seq / 64; i++) table[i] = c.pages ? max_seq / 64 - 1 - i : i;
        for (int j = 0; j < max_seq; j++)
            for (size_t e = 0; e < ld; e++) {
                const size_t to = ((size_t)table[j / 64] * 64 + j % 64) * ld + e;
                kp[to] = j < n ? k[j * ld + e] : 0x7fc0; vp[to] = j < n ? v[j * ld + e] : 0x7fc0;
            }
        Dev<float> dq(q), out(q.size());
        Dev<uint16_t> kc(kp), vc(vp);
        Dev<int> dpos(pos), dtable(table);
        Dev<uint32_t> status(1);
        AttnRowsArgs a{};
        a.q_rot = dq.p; a.k_cache = kc.p; a.v_cache = vc.p; a.row_pos = dpos.p; a.out = out.p; a.M = c.rows; a.n_q = c.nq; a.n_kv = c.nkv; a.hd = hd; a.kv_bf16 = 1;
        a.max_seq = max_seq; a.max_batch = 1; a.status = status.p;
        if (c.pages) { a.pg.table = dtable.p; a.pg.lg = 6; a.pg.pages_per_seq = max_seq / 64; }
        CK(launch_attn_prompt_tc(a, nullptr));
        std::vector<double> want(q.size()), w(n);
        for (int m = 0; m < c.rows; m++)
            for (int h = 0; h < c.nq; h++) {
                const size_t col = (size_t)(h / G) * hd, row = (size_t)m * qd + (size_t)h * hd;
                double mx = -INFINITY, l = 0;
                for (int j = 0; j <= pos[m]; j++) {
                    double d = 0;
                    for (int e = 0; e < hd; e++) d += (double)q[row + e] * bf16_value(k[j * ld + col + e]);
                    w[j] = d / std::sqrt((double)hd);
                    mx = std::fmax(mx, w[j]);
                }
                for (int j = 0; j <= pos[m]; j++) l += w[j] = std::exp(w[j] - mx);
                for (int j = 0; j <= pos[m]; j++)
                    for (int e = 0; e < hd; e++) want[row + e] += w[j] / l * bf16_value(v[j * ld + col + e]);
            }
        // queries and weights keep 2^-17 of themselves in two bf16 terms; a score of 128 products then moves by less than 2^-17 on average, and a sum of
        // 16 instructions is cut to 24 bits that many times
        report(std::to_string(c.nq) + " / " + std::to_string(c.nkv) + " heads, rows " + std::to_string(c.first) + " + " + std::to_string(c.rows) + (c.pages ? ", pages" : ""), rel(out.get(), want), std::exp2(-16.0));
        report("status", status.get()[0], 0);
    }
}

// The same kernel for layers described one by one: windows, chunks, a bias by distance, one to eight query heads per K/V head.  What no row of a CTA sees, before its
// first row's window or chunk and behind its last row, is not a number; with pages (in another order), it is on pages of its own.
static void attention_band() {
    struct Case { int nq, nkv, rows, first, window, chunk; bool bias, pages; };
    const std::vector<Case> cases = {{4, 4, 130, 0, 0, 0, true, false},     {8, 4, 65, 300, 128, 0, true, false},     {8, 2, 97, 1000, 300, 0, true, false}, {8, 1, 50, 255, 1, 0, true, false},
                                     {8, 2, 129, 511, 512, 0, false, true}, {8, 1, 33, 127, 0, 100, true, false},     {4, 2, 200, 64, 0, 256, false, true},  {4, 1, 40, 900, 129, 0, true, false},
                                     {8, 2, 32, 1003, 300, 0, true, true},  {8, 1, 16, 447, 192, 0, false, false},    {8, 1, 16, 400, 0, 336, true, true},   {4, 4, 128, 765, 128, 0, true, true}};
    for (const Case& c : cases) {
        const int hd = 128, n = c.first + c.rows, max_seq = (n + 63) / 64 * 64, G = c.nq / c.nkv, chunks = c.nq * hd / 64;
        std::mt19937 rng(n * 5 + c.nq + c.window);
        const size_t ld = (size_t)c.nkv * hd, qd = (size_t)c.nq * hd;
        const std::vector<float> q = normal(rng, (size_t)c.rows * qd, 0.09f);
        const std::vector<uint16_t> k = to_bf16(normal(rng, max_seq * ld, 1.0f)), v = to_bf16(normal(rng, max_seq * ld, 1.0f, 0.5f));
        const int low = c.window ? std::max(0, c.first + 1 - c.window) : c.chunk ? c.first / c.chunk * c.chunk : 0;
        std::vector<uint16_t> kp = k, vp = v;
        std::vector<int> table(max_seq / 64);
        for (int i = 0; i < max_seq / 64; i++) table[i] = c.pages ? max_seq / 64 - 1 - i : i;
        for (int j = 0; j < max_seq; j++)
            for (size_t e = 0; e < ld; e++) {
                const size_t to = ((size_t)table[j / 64] * 64 + j % 64) * ld + e;
                kp[to] = j >= low && j < n ? k[j * ld + e] : 0x7fc0; vp[to] = j >= low && j < n ? v[j * ld + e] : 0x7fc0;
            }
        std::vector<float> r1(c.nq), r2(c.nq);
        for (int h = 0; h < c.nq; h++) { r1[h] = 0.1f + 0.2f * h; r2[h] = 0.05f + 0.07f * h; }
        std::vector<int> pos(c.rows);
        for (int i = 0; i < c.rows; i++) pos[i] = c.first + i;
        const int rows_up = (c.rows + 127) / 128 * 128;
        Dev<float> dq(q), d1(r1), d2(r2);
        Dev<uint16_t> kc(kp), vc(vp), out((size_t)rows_up * qd);
        Dev<int> dpos(pos), dtable(table);
        Dev<uint32_t> status(1);
        BandArgs a{};
        if (c.pages) { a.pg.table = dtable.p; a.pg.lg = 6; a.pg.pages_per_seq = max_seq / 64; }
        a.p.n_q = c.nq; a.p.n_kv = c.nkv; a.p.dk = a.p.dv = a.p.dkp = a.p.dvp = hd; a.p.maps = 1;
        a.q = dq.p; a.k_cache = kc.p; a.v_cache = vc.p; a.kv_bf16 = 1; a.row_pos = dpos.p; a.M = c.rows; a.window = c.window; a.chunk = c.chunk; a.max_seq = max_seq; a.max_batch = 1;
        if (c.bias) { a.r1 = d1.p; a.r2 = d2.p; }
        a.out_kind = WK_BF16; a.out.p = out.p; a.out.chunks = chunks; a.status = status.p;
        CK(launch_band_prompt_tc(a, nullptr));
        const std::vector<uint16_t> raw = out.get();
        std::vector<float> got(q.size());
        std::vector<double> want(q.size()), w(n);
        for (int m = 0; m < c.rows; m++)
            for (size_t e = 0; e < qd; e++)
                got[m * qd + e] = bf16_value(raw[((((size_t)(m >> 7) * chunks + (e >> 6)) * 16 + ((m & 127) >> 3)) * 1024 + ((e >> 3) & 7) * 128 + (m & 7) * 16 + (e & 7) * 2) / 2]);
        for (int m = 0; m < c.rows; m++)
            for (int h = 0; h < c.nq; h++) {
                const size_t col = (size_t)(h / G) * hd, row = (size_t)m * qd + (size_t)h * hd;
                int j0 = 0;
                if (c.window) j0 = std::max(0, pos[m] + 1 - c.window);
                if (c.chunk) j0 = pos[m] / c.chunk * c.chunk;
                double mx = -INFINITY, l = 0;
                for (int j = j0; j <= pos[m]; j++) {
                    double d = 0;
                    for (int e = 0; e < hd; e++) d += (double)q[row + e] * bf16_value(k[j * ld + col + e]);
                    w[j] = d - (c.bias ? r1[h] * std::log1p((double)r2[h] * (pos[m] - j)) : 0.0);
                    mx = std::fmax(mx, w[j]);
                }
                for (int j = j0; j <= pos[m]; j++) l += w[j] = std::exp(w[j] - mx);
                for (int j = j0; j <= pos[m]; j++)
                    for (int e = 0; e < hd; e++) want[row + e] += w[j] / l * bf16_value(v[j * ld + col + e]);
            }
        // outputs are rounded to bf16: at most 2^-9 of each
        report(std::to_string(c.nq) + " / " + std::to_string(c.nkv) + " heads, rows " + std::to_string(c.first) + " + " + std::to_string(c.rows) + ", window " + std::to_string(c.window) + ", chunk " +
               std::to_string(c.chunk) + (c.bias ? ", bias" : "") + (c.pages ? ", pages" : ""), rel(got, want), std::exp2(-9.0));
        report("status", status.get()[0], 0);
    }
}

// Long sums stay sums of 32 bits.  A split's values are added up tile by tile, 64 keys of a CTA at a time: m additions of relative error 2^-24 at most
// walk about sqrt(m) of them away, and scores, weights and each tile's own sum (cut, not rounded) are a few more.
static void attention_sums() {
    for (int hd : {64, 128})
        for (float v_mean : {0.0f, 1.0f}) {
            const Attention a(4, 1, hd, 30000, 1.0f, v_mean);
            const std::vector<double> want = a.exact();
            auto bound = [&](int splits) { return (4 + std::sqrt(a.n / 64.0 / splits)) * std::exp2(-24.0); };
            const std::string what = std::to_string(hd) + (v_mean ? " same sign" : " both signs");
            report("step, 1 split, " + what, rel(a.step(1, false), want), bound(1));
            report("step, 8 splits, " + what, rel(a.step(8, false), want), bound(8));
            report("step, cluster of 8, " + what, rel(a.step(8, true), want), bound(8));
            report("row, " + what, rel(a.row(), want), bound(8));
        }
}

// Infinite, undefined and huge elements go where the plain sums take them, and nowhere else.
static void attention_specials() {
    const float inf = INFINITY;
    for (int hd : {64, 128})
        for (int n : {40, 700})
            for (int what = 0; what < 6; what++) {
                Attention a(8, hd == 64 ? 1 : 2, hd, n, 1.0f, 0.0f);
                const int key = n / 2 + 1, e = 5;
                const size_t at = ((size_t)key * a.nkv) * hd + e;                    // element e of the first KV head's key
                for (int h = 0; h < a.nq; h++) a.q[(size_t)h * hd + e] = 0.75f + 0.001f * h;
                const char* name[] = {"a key of minus infinity", "a value of infinity", "an undefined value", "the lowest key", "the largest query", "two infinite values of one column"};
                if (what == 0) a.k[at] = bf16_bits(-inf);
                if (what == 1) a.v[at] = bf16_bits(inf);
                if (what == 2) a.v[at] = 0x7fc0;
                if (what == 3) a.k[at] = 0xff7f;
                if (what == 4) {
                    for (int h = 0; h < a.nq; h++) a.q[(size_t)h * hd + e] = 3.4e38f;
                    for (int j = 0; j <= n; j++) for (int g = 0; g < a.nkv; g++) a.k[((size_t)j * a.nkv + g) * hd + e] = bf16_bits(j % 3 ? 2e-38f : -2e-38f);
                }
                if (what == 5) { a.v[at] = bf16_bits(-inf); a.v[at + (size_t)a.nkv * hd * 3] = bf16_bits(-inf); }
                const std::vector<double> want = a.exact();
                auto worst = [&](const std::vector<float>& got) {
                    double m = 0;
                    for (size_t i = 0; i < want.size(); i++) {
                        if (std::isnan(want[i]) || std::isinf(want[i])) { if (!(std::isnan(want[i]) ? std::isnan(got[i]) : (double)got[i] == want[i])) return (double)INFINITY; }
                        else if (!(std::fabs(got[i] - want[i]) <= m)) m = std::isnan(got[i]) ? INFINITY : std::fabs(got[i] - want[i]);
                    }
                    return m;
                };
                // values of size one, scores of up to ten: a hundred roundings
                const std::string where = std::string(name[what]) + ", " + std::to_string(hd) + ", " + std::to_string(n);
                report("step, 1 split, " + where, worst(a.step(1, false)), 100 * std::exp2(-24.0));
                report("step, cluster of 4, " + where, worst(a.step(4, true)), 100 * std::exp2(-24.0));
                report("row, " + where, worst(a.row()), 100 * std::exp2(-24.0));
            }
}

// Routed experts of several tokens, as an expert-parallel rank has them: some, all or none of a token's experts are this rank's.
static void experts() {
    struct Size { int hidden, ffn, n_experts, top_k; };
    // (the last: activations that leave the ring four blocks)
    for (const Size z : {Size{256, 128, 8, 3}, Size{3200, 96, 6, 2}, Size{96, 3136, 5, 4}, Size{64, 8960, 8, 8}}) {
        const int H = z.hidden, F = z.ffn, E = z.n_experts, K = z.top_k, T = 5, slot = (H + 2 * K + 3) / 4 * 4;
        std::mt19937 rng(H + F);
        auto ints = [&](size_t n, int lo, int hi) { std::vector<int> v(n); for (int& x : v) x = std::uniform_int_distribution<int>(lo, hi)(rng); return v; };
        auto planes = [&](size_t rows, int k, std::vector<int8_t>& q, std::vector<__half>& d) {
            q.resize(rows * k); d.resize(rows * k / 32);
            const std::vector<int> i = ints(q.size(), -127, 127);
            for (size_t j = 0; j < q.size(); j++) q[j] = (int8_t)i[j];
            for (__half& x : d) x = __float2half(0.02f / std::sqrt((float)k) * (1 + std::uniform_real_distribution<float>(0, 1)(rng)));
        };
        std::vector<int8_t> gq, dq;
        std::vector<__half> gs, ds;
        planes((size_t)E * 2 * F, H, gq, gs);
        planes((size_t)E * H, F, dq, ds);
        const std::vector<float> gb = normal(rng, (size_t)E * 2 * F, 0.1f), db = normal(rng, (size_t)E * H, 0.1f);
        std::vector<float> xf((size_t)T * slot);         // per token: activations, chosen experts, their weights
        std::vector<int> chosen((size_t)T * K);
        for (int t = 0; t < T; t++) {
            const std::vector<float> x = normal(rng, H, 1.0f);
            std::memcpy(&xf[(size_t)t * slot], x.data(), H * 4);
            for (int k = 0; k < K; k++) {
                // token 0: the first experts, 1: the last, then a mixture
                const int e = t == 0 ? k : t == 1 ? E - 1 - k : (t * 3 + k * 2 + (2 * k >= E ? 1 : 0)) % E;
                chosen[(size_t)t * K + k] = e;
                std::memcpy(&xf[(size_t)t * slot + H + k], &e, 4);
                xf[(size_t)t * slot + H + K + k] = 0.1f + 0.2f * k;
            }
        }
        Dev<int8_t> dgq(gq), ddq(dq);
        Dev<__half> dgs(gs), dds(ds);
        Dev<float> dgb(gb), ddb(db), dxf(xf), sw((size_t)T * K * F);
        Dev<uint32_t> status(1);
        for (int first : {0, E / 2})
            for (int n_local : {E - first, 2})
                for (int tokens : {1, 2, T}) {
                    if (F > 4096 && tokens > 2) continue;
                    Dev<float> out((size_t)T * H);
                    MoeArgs a{};
                    a.hidden = H; a.ffn = F; a.n_experts = E; a.top_k = K; a.slot = slot; a.xf_in = dxf.p; a.n_tokens = tokens; a.expert0 = first; a.n_local = n_local;
                    a.gu_q = dgq.p + (size_t)first * 2 * F * H; a.gu_s = dgs.p + (size_t)first * 2 * F * H / 32; a.gu_bias = dgb.p + (size_t)first * 2 * F;
                    a.dn_q = ddq.p + (size_t)first * H * F; a.dn_s = dds.p + (size_t)first * H * F / 32; a.dn_bias = ddb.p + (size_t)first * H;
                    a.gain_kind = WK_F32; a.sw = sw.p; a.limit = 7.0f; a.status = status.p; a.out = out.p; a.out_ld = H;
                    CK(launch_moe_experts(a, 148, nullptr));
                    const std::vector<float> got = out.get();
                    double num = 0, den = 0;
                    for (int t = 0; t < tokens; t++) {
                        std::vector<double> want(H);
                        for (int k = 0; k < K; k++) {
                            const int e = chosen[(size_t)t * K + k];
                            if (e < first || e >= first + n_local) continue;
                            std::vector<double> s(F);
                            auto row = [&](const std::vector<int8_t>& q, const std::vector<__half>& d, size_t r, int n, auto x) {
                                double v = 0;
                                for (int i = 0; i < n; i++) v += (double)q[r * n + i] * (double)__half2float(d[(r * n + i) / 32]) * x(i);
                                return v;
                            };
                            auto x = [&](int i) { return (double)xf[(size_t)t * slot + i]; };
                            for (int i = 0; i < F; i++) {
                                const size_t r = (size_t)e * 2 * F + 2 * i;
                                const double g = std::fmin(row(gq, gs, r, H, x) + gb[r], 7.0), u = std::fmax(std::fmin(row(gq, gs, r + 1, H, x) + gb[r + 1], 7.0), -7.0);
                                s[i] = (u + 1) * g / (1 + std::exp(-1.702 * g));
                            }
                            for (int c = 0; c < H; c++)
                                want[c] += (double)xf[(size_t)t * slot + H + K + k] * (row(dq, ds, (size_t)e * H + c, F, [&](int i) { return s[i]; }) + db[(size_t)e * H + c]);
                        }
                        for (int c = 0; c < H; c++) { const double d = got[(size_t)t * H + c] - want[c]; num += d * d; den += want[c] * want[c]; }
                    }
                    for (size_t i = (size_t)tokens * H; i < got.size(); i++) num += (double)got[i] * got[i];          // nothing behind the last token
                    // three levels keep 2^-24 of the largest magnitude, the rest are roundings of two sums in a row
                    report(std::to_string(H) + " x " + std::to_string(F) + ", experts " + std::to_string(first) + " + " + std::to_string(n_local) + ", " + std::to_string(tokens) + " tokens",
                           den > 0 ? std::sqrt(num / den) : num, 32 * std::exp2(-24.0));
                }
        uint32_t st = status.get()[0];
        report("status", st, 0);
    }
}

// bf16 matrices in the plain matrix-vector kernel, four rows per warp: rows per block that are no multiple of four or of 32, matrices that end inside a
// group of four, columns that are no multiple of a warp's trip, the paired epilogue.
static void matvec_bf16() {
    struct Case { std::vector<int> rows; int k; bool pair; };
    const std::vector<Case> cases = {{{1}, 8, false},      {{3}, 264, false},         {{37}, 2568, false},     {{9, 2, 5}, 512, false}, {{130, 33, 34}, 264, false},
                                     {{5003}, 520, false}, {{6, 6}, 512, true},       {{45, 45}, 264, true},   {{2501, 2501}, 1032, true}, {{40003}, 512, false}, {{20000, 3, 1001}, 1024, false}};
    for (const Case& c : cases) {
        std::mt19937 rng(c.k + c.rows[0]);
        const std::vector<float> x = normal(rng, c.k, 1.0f);
        Dev<float> dx(x);
        GemvArgs a{};
        a.nseg = (int)c.rows.size(); a.K = c.k; a.wkind = WK_BF16; a.epi = c.pair ? EPI_SWIGLU : EPI_STORE; a.x = dx.p; a.gain_kind = WK_F32;
        std::vector<std::vector<uint16_t>> w;
        std::vector<Dev<uint16_t>*> dw;
        std::vector<std::vector<double>> sums;
        int total = 0;
        for (int n : c.rows) {
            w.push_back(to_bf16(normal(rng, (size_t)n * c.k, 1.0f / std::sqrt((float)c.k))));
            dw.push_back(new Dev<uint16_t>(w.back()));
            a.seg[sums.size()] = {dw.back()->p, nullptr, n, 0};
            sums.emplace_back(n);
            for (int r = 0; r < n; r++)
                for (int i = 0; i < c.k; i++) sums.back()[r] += (double)bf16_value(w.back()[(size_t)r * c.k + i]) * x[i];
            total += n;
        }
        std::vector<double> want;
        if (c.pair) { total = c.rows[0]; for (int r = 0; r < total; r++) want.push_back(sums[0][r] / (1 + std::exp(-sums[0][r])) * sums[1][r]); }
        else for (const auto& s : sums) want.insert(want.end(), s.begin(), s.end());
        Dev<float> y((size_t)total + 8);                  // (eight behind the end: stay zero)
        Dev<uint32_t> status(1);
        a.y = y.p; a.status = status.p;
        CK(launch_gemv(a, 148, nullptr));
        std::vector<float> got = y.get();
        for (int i = 0; i < 8; i++) if (got[total + i] != 0.0f) report("behind the end", 1, 0);
        got.resize(total);
        std::string what;
        for (int n : c.rows) what += std::to_string(n) + " ";
        // 32-bit sums of k products, folded over a warp
        report(what + "x " + std::to_string(c.k) + (c.pair ? " paired" : ""), rel(got, want), (4 + std::sqrt(c.k / 32.0)) * std::exp2(-23.0));
        for (auto* p : dw) delete p;
    }
}

// Q8_0 matrices in the streaming matrix-vector kernel: every number of tiles a row group can have (a tile per warp, several row groups per job, several turns
// of the rings), K ranges, jobs claimed or dealt out, all epilogues but the sampler's, vectors made of several terms.
static void matvec_q8() {
    struct Case { std::vector<int> rows; int k, ranges, parts; bool pair, resid, claims, norm; };
    const std::vector<Case> cases = {
        {{8}, 512, 1, 0, false, false, false, false},          {{264, 16, 8}, 512, 1, 0, false, false, true, false}, {{40, 40}, 512, 1, 0, true, false, true, true},
        {{72, 8}, 1024, 1, 2, false, false, true, true},       {{1208}, 1536, 1, 0, false, true, true, false},       {{24, 24}, 1536, 1, 0, true, false, false, true},
        {{136, 8, 8}, 2048, 1, 4, false, false, true, true},   {{2560}, 2560, 1, 3, false, true, true, true},        {{1240, 1240}, 2560, 1, 0, true, false, true, true},
        {{648}, 3072, 1, 0, false, true, false, false},        {{512, 40, 40}, 3584, 1, 0, false, false, true, true}, {{4096}, 4096, 1, 1, false, false, true, true},
        {{2008, 2008}, 4096, 1, 4, true, false, true, true},   {{96}, 4608, 1, 0, false, false, true, true},         {{64, 64}, 6144, 1, 2, true, false, true, true},
        {{264}, 4608, 2, 0, false, false, true, false},        {{1208}, 9728, 3, 0, false, false, true, false},      {{1200}, 14336, 4, 0, false, false, true, false},
        {{40}, 14336, 4, 0, false, false, false, false},       {{328}, 14336, 1, 0, false, true, true, false},       {{80}, 16384, 4, 0, false, false, true, false}};
    for (const Case& c : cases) {
        std::mt19937 rng(c.k + c.rows[0] + c.parts);
        const int K = c.k, nb = K / 32;
        std::vector<std::vector<float>> terms;
        for (int i = 0; i <= c.parts; i++) terms.push_back(normal(rng, K, 1.0f));
        std::vector<float> x = terms[0], parts;
        for (int i = 1; i <= c.parts; i++) { for (int j = 0; j < K; j++) x[j] += terms[i][j]; parts.insert(parts.end(), terms[i].begin(), terms[i].end()); }
        const std::vector<uint16_t> gain = to_bf16(normal(rng, K, 0.1f, 1.0f));
        std::vector<double> xe(x.begin(), x.end());
        if (c.norm) {
            double ss = 0;
            for (double v : xe) ss += v * v;
            for (int j = 0; j < K; j++) xe[j] *= bf16_value(gain[j]) / std::sqrt(ss / K + 1e-5);
        }
        Dev<float> dx(terms[0]), dparts(parts.empty() ? std::vector<float>(1) : parts), dxo(K);
        Dev<uint16_t> dgain(gain);
        Dev<unsigned int> ctr(kMaxKRanges);
        Dev<uint32_t> status(1);
        GemvArgs a{};
        a.nseg = (int)c.rows.size(); a.K = K; a.wkind = WK_Q8; a.epi = c.pair ? EPI_SWIGLU : c.resid ? EPI_RESID : EPI_STORE; a.x = dx.p; a.gain_kind = WK_BF16; a.status = status.p;
        if (c.norm) { a.gain = dgain.p; a.eps = 1e-5f; }
        if (c.parts) { a.parts = dparts.p; a.n_parts = c.parts; a.part_stride = K; a.x_out = dxo.p; }
        if (c.claims) a.job_ctr = ctr.p;
        std::vector<Dev<unsigned char>*> packed;
        std::vector<std::vector<double>> sums;
        int total = 0;
        for (int n : c.rows) {
            std::vector<int8_t> q((size_t)n * K);
            std::vector<__half> s((size_t)n * nb);
            for (auto& v : q) v = (int8_t)((int)(rng() % 256) - 128);
            for (auto& v : s) v = __float2half(0.0005f + 0.001f * (rng() % 1000) / 1000.0f);
            Dev<int8_t> dq(q);
            Dev<__half> ds(s);
            packed.push_back(new Dev<unsigned char>(q8_packed_bytes(n, K)));
            CK(launch_q8_pack_units(dq.p, ds.p, n, K, q8_pack_kc(n, K), packed.back()->p, nullptr));
            CK(cudaDeviceSynchronize());
            a.seg[sums.size()] = {packed.back()->p, nullptr, n, q8_pack_kc(n, K)};
            sums.emplace_back(n);
            for (int r = 0; r < n; r++)
                for (int b = 0; b < nb; b++) {
                    double t = 0;
                    for (int i = 0; i < 32; i++) t += (double)q[(size_t)r * K + b * 32 + i] * xe[b * 32 + i];
                    sums.back()[r] += t * (double)__half2float(s[(size_t)r * nb + b]);
                }
            total += n;
        }
        std::vector<float> res = normal(rng, total, 1.0f);
        std::vector<double> want;
        if (c.pair) { total = c.rows[0]; for (int r = 0; r < total; r++) want.push_back(sums[0][r] / (1 + std::exp(-sums[0][r])) * sums[1][r]); }
        else for (const auto& s : sums) want.insert(want.end(), s.begin(), s.end());
        if (c.resid) for (int r = 0; r < total; r++) want[r] += res[r];
        Dev<float> y((size_t)total * c.ranges + 8), dres(res);
        a.y = y.p; a.resid = dres.p;
        if (c.ranges > 1) { a.ksplit = c.ranges; a.y_range_stride = total; }
        CK(launch_gemv(a, 148, nullptr));
        std::vector<float> raw = y.get(), got(total);
        for (int i = 0; i < 8; i++) if (raw[(size_t)total * c.ranges + i] != 0.0f) report("behind the end", 1, 0);
        for (int r = 0; r < c.ranges; r++) for (int i = 0; i < total; i++) got[i] += raw[(size_t)r * total + i];
        std::string what;
        for (int n : c.rows) what += std::to_string(n) + " ";
        // three levels keep 2^-24 of a block's largest magnitude (about two to three standard deviations), every sum of the vector's terms and of the blocks rounds once more
        report(what + "x " + std::to_string(K) + " in " + std::to_string(c.ranges) + " ranges, epilogue " + std::to_string(a.epi) + ", " + std::to_string(c.parts) + " terms more" + (c.claims ? ", claimed" : ""),
               rel(got, want), 16 * std::exp2(-24.0));
        if (c.parts) { const std::vector<float> xo = dxo.get(); report("the vector itself", rel(xo, std::vector<double>(x.begin(), x.end())), std::exp2(-24.0)); }
        report("status", status.get()[0], 0);
        for (auto* p : packed) delete p;
    }
}

// The matrix-vector kernel's tensor-parallel paths, on one GPU: partial vectors as {value, completion word} pairs that are there already, rows stored as such pairs or
// as values with a word behind them; and the sampler's epilogue, where the last of equal best rows wins.
static void matvec_peer() {
    struct Case { int k, n, parts, epi; bool ll; };
    const std::vector<Case> cases = {{2560, 1208, 1, EPI_STORE, true}, {2560, 264, 2, EPI_PEER, true},   {4096, 4096, 3, EPI_STORE, true},  {4096, 1208, 5, EPI_PEER, false}, {4608, 96, 2, EPI_STORE, true},
                                     {4608, 640, 3, EPI_PEER, true},   {1024, 72, 2, EPI_PEER, false},   {2560, 5000, 0, EPI_ARGMAX, true}, {4096, 1208, 1, EPI_ARGMAX, true}, {512, 264, 0, EPI_ARGMAX, true},
                                     {4608, 640, 2, EPI_ARGMAX, true}, {2048, 3000, 0, EPI_PEER, false}};
    for (const Case& c : cases) {
        const int K = c.k, N = c.n, nb = K / 32;
        std::mt19937 rng(K + N + c.parts);
        Dev<uint32_t> seq(std::vector<uint32_t>{41}), status(1), flag(32);
        const uint32_t word[2] = {peer_word(41, 7), peer_word(41, 9)};
        const std::vector<float> x0 = normal(rng, K, 1.0f);
        std::vector<float> x = x0;
        std::vector<uint2> pairs((size_t)c.parts * K + 1);
        for (int r = 0; r < c.parts; r++) {
            const std::vector<float> v = normal(rng, K, 1.0f);
            for (int i = 0; i < K; i++) { uint32_t b; std::memcpy(&b, &v[i], 4); pairs[(size_t)r * K + i] = make_uint2(b, word[0]); x[i] += v[i]; }
        }
        std::vector<int8_t> q((size_t)N * K);
        std::vector<__half> s((size_t)N * nb, __float2half(0.001f));
        for (auto& v : q) v = (int8_t)((int)(rng() % 255) - 127);
        const int first = N / 3, last = N - 3;               // two equal rows that no other row comes near
        if (c.epi == EPI_ARGMAX) for (int i = 0; i < K; i++) q[(size_t)first * K + i] = q[(size_t)last * K + i] = x[i] > 0 ? 127 : -127;
        std::vector<double> want(N);
        for (int n = 0; n < N; n++)
            for (int i = 0; i < K; i++) want[n] += (double)q[(size_t)n * K + i] * x[i] * (double)__half2float(s[0]);
        Dev<int8_t> dq(q);
        Dev<__half> ds(s);
        Dev<unsigned char> w(q8_packed_bytes(N, K));
        CK(launch_q8_pack_units(dq.p, ds.p, N, K, q8_pack_kc(N, K), w.p, nullptr));
        Dev<float> dx(x0), dxo(K), y((size_t)N), part_val(256);
        Dev<uint2> dparts(pairs), out((size_t)N);
        Dev<int> part_idx(256), tokens(4);
        Dev<unsigned int> counter(1), ticket(1);
        DecodeState st{};
        st.max_steps = 4; st.log = 1; st.pos = 11; st.vocab = N;
        Dev<DecodeState> state(std::vector<DecodeState>{st});
        GemvArgs a{};
        a.nseg = 1; a.seg[0] = {w.p, nullptr, N, q8_pack_kc(N, K)}; a.K = K; a.wkind = WK_Q8; a.epi = c.epi; a.x = dx.p; a.y = y.p; a.status = status.p; a.seq = seq.p; a.wait_cycles = 10000000;
        if (c.parts) { a.parts = (const float*)dparts.p; a.parts_ll = 1; a.n_parts = c.parts; a.part_stride = K; a.parts_tag = 7; a.x_out = dxo.p; }
        if (c.epi == EPI_PEER) { a.n_peers = 1; a.peer_out[0] = (float*)out.p; a.peer_flag[0] = flag.p; a.peer_ticket = ticket.p; a.peer_tag = 9; a.peer_ll = c.ll; }
        if (c.epi == EPI_ARGMAX) { a.part_val = part_val.p; a.part_idx = part_idx.p; a.counter = counter.p; a.state = state.p; a.tokens_out = tokens.p; a.advance = 1; }
        const std::string what = std::to_string(N) + " x " + std::to_string(K) + ", " + std::to_string(c.parts) + " parts, epilogue " + std::to_string(c.epi) + (c.ll ? "" : ", values") + ": ";
        for (int turn = 0; turn < 2; turn++) {               // (tickets are left at zero)
            CK(launch_gemv(a, 148, nullptr));
            std::vector<float> got(N);
            if (c.epi == EPI_PEER) {
                const std::vector<uint2> o = out.get();
                double late = 0;
                for (int n = 0; n < N; n++) {
                    if (c.ll) { std::memcpy(&got[n], &o[n].x, 4); late += o[n].y != word[1]; }
                    else std::memcpy(&got[n], (const float*)o.data() + n, 4);
                }
                if (!c.ll) late = flag.get()[0] != word[1];
                report(what + "words", late, 0);
            } else {
                got = y.get();
            }
            report(what + "rows", rel(got, want), 16 * std::exp2(-24.0));
            if (c.epi == EPI_ARGMAX) {
                const DecodeState d = state.get()[0];
                report(what + "best row", std::fabs((double)d.last_tok - last) + std::fabs((double)tokens.get()[turn] - last) + std::fabs(d.pos - 12.0 - turn) + std::fabs(d.step - 1.0 - turn), 0);
            }
            report("status", status.get()[0], 0);
        }
        if (c.parts) report(what + "the vector itself", rel(dxo.get(), std::vector<double>(x.begin(), x.end())), std::exp2(-24.0));
    }
}

// A step's chain: an embedding row that zeroes the claim counters, projections behind it that claim from them under programmatic launch and change places between the
// two sizes of shared memory.  Every row of every step is there (a claim from an old count leaves rows out), and what is captured says why: the first projection
// waits for the counters in plain stream order, the others may come early.
static void claims() {
    const int V = 64, H = 2560, P = 4, steps = 60;
    const int N[P] = {2560, 1208, 4096, 264};
    std::mt19937 rng(11);
    Dev<float> table(normal(rng, (size_t)V * H, 1.0f)), x((size_t)H);
    Dev<uint32_t> status(1);
    DecodeState s{};
    s.tok = 5; s.vocab = V;
    Dev<DecodeState> state(std::vector<DecodeState>{s});
    Dev<unsigned int> ctr(std::vector<unsigned int>(P * kMaxKRanges, 7u));            // (left over from a step before)
    std::vector<Dev<unsigned char>*> packed;
    size_t total = 0;
    for (int n : N) {
        std::vector<int8_t> q((size_t)n * H);
        std::vector<__half> d((size_t)n * H / 32);
        for (auto& v : q) v = (int8_t)((int)(rng() % 255) - 127);
        for (auto& v : d) v = __float2half(0.001f);
        Dev<int8_t> dq(q);
        Dev<__half> ds(d);
        packed.push_back(new Dev<unsigned char>(q8_packed_bytes(n, H)));
        CK(launch_q8_pack_units(dq.p, ds.p, n, H, q8_pack_kc(n, H), packed.back()->p, nullptr));
        CK(cudaDeviceSynchronize());
        total += n;
    }
    Dev<float> y(total * (steps + 1));
    cudaStream_t st;
    CK(cudaStreamCreate(&st));
    auto step = [&](int i) {
        EmbedArgs e{};
        e.table = table.p; e.kind = WK_F32; e.H = H; e.x = x.p; e.state = state.p; e.status = status.p; e.zero_ctr = ctr.p; e.n_zero = P * kMaxKRanges;
        CK(launch_embed(e, st));
        float* to = y.p + (size_t)i * total;
        for (int p = 0; p < P; to += N[p], p++) {
            GemvArgs a{};
            a.nseg = 1; a.seg[0] = {packed[p]->p, nullptr, N[p], q8_pack_kc(N[p], H)}; a.K = H; a.wkind = WK_Q8; a.epi = EPI_STORE; a.x = x.p; a.y = to; a.status = status.p;
            a.use_pdl = 1; a.job_ctr = ctr.p + p * kMaxKRanges; a.ordered = p == 0; a.wide_smem = (p & 1) == 0;
            CK(launch_gemv(a, 148, st));
        }
    };
    for (int i = 0; i < steps; i++) step(i);
    CK(cudaStreamSynchronize(st));
    const std::vector<float> got = y.get();
    size_t differ = 0, zero = 0;
    for (size_t i = 0; i < (size_t)steps * total; i++) { differ += got[i] != got[i % total]; zero += got[i] == 0.0f; }
    report("rows of a step that differ from the first step's", (double)differ, 0);
    report("rows that nobody wrote", (double)zero, 0);
    report("status", status.get()[0], 0);

    cudaGraph_t graph;
    CK(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
    step(steps);
    CK(cudaStreamEndCapture(st, &graph));
    size_t n = 0;
    CK(cudaGraphGetEdges_v2(graph, nullptr, nullptr, nullptr, &n));
    std::vector<cudaGraphNode_t> from(n), to(n);
    std::vector<cudaGraphEdgeData> how(n);
    CK(cudaGraphGetEdges_v2(graph, from.data(), to.data(), how.data(), &n));
    report("edges", std::fabs((double)n - P), 0);
    int programmatic = 0;
    for (size_t i = 0; i < n; i++) {
        const bool first = std::find(to.begin(), to.end(), from[i]) == to.end();          // an edge from the embedding
        const bool pdl = how[i].type == cudaGraphDependencyTypeProgrammatic;
        programmatic += pdl;
        if (first) report("the first projection in plain order", pdl, 0);
    }
    report("the others programmatic", std::fabs(programmatic - (P - 1.0)), 0);
    CK(cudaGraphDestroy(graph));
    CK(cudaStreamDestroy(st));
    for (auto* p : packed) delete p;
}

// Two to five rows: rows formed and quantised (plain, behind a norm, SwiGLU of two sums; planes, residual), then multiplied; every number of tiles, K ranges.
static void few_rows() {
    struct Case { std::vector<int> rows; int k, m, planes; bool norm, pair; };
    const std::vector<Case> cases = {{{8}, 2560, 2, 1, false, false},        {{1200, 40, 8}, 4096, 5, 4, true, false}, {{9600}, 4096, 5, 1, false, false}, {{264}, 3072, 3, 2, true, false},
                                     {{640}, 14336, 5, 1, false, true},      {{72, 72}, 3584, 5, 3, true, false},      {{1192}, 9728, 4, 2, false, true},   {{96}, 8192, 3, 1, false, false},
                                     {{16, 7184}, 2560, 5, 1, true, false},  {{88}, 5120, 2, 1, false, true},          {{4096}, 3584, 1, 1, false, false}};
    for (const Case& c : cases) {
        const int K = c.k, M = c.m, nb = K / 32, ld = c.pair ? 2 * K : K, R = few_ranges(K, 148);
        std::mt19937 rng(K + M);
        const std::vector<float> in = normal(rng, (size_t)c.planes * M * ld, 1.0f), resid = normal(rng, (size_t)M * K, 1.0f);
        const std::vector<uint16_t> gain = to_bf16(normal(rng, K, 0.1f, 1.0f));
        std::vector<double> x((size_t)M * K);
        for (int m = 0; m < M; m++) {
            double ss = 0;
            for (int i = 0; i < K; i++) {
                double v = 0, u = 0;
                for (int p = 0; p < c.planes; p++) { v += in[((size_t)p * M + m) * ld + i]; if (c.pair) u += in[((size_t)p * M + m) * ld + K + i]; }
                if (c.pair) v = v / (1 + std::exp(-v)) * u;
                if (c.norm) v += resid[(size_t)m * K + i];
                x[(size_t)m * K + i] = v;
                ss += v * v;
            }
            if (c.norm) for (int i = 0; i < K; i++) x[(size_t)m * K + i] *= bf16_value(gain[i]) / std::sqrt(ss / K + 1e-5);
        }
        Dev<float> din(in), dres(resid), out((size_t)M * K), sx(few_sx_floats(M, K));
        Dev<uint16_t> dgain(gain);
        Dev<int8_t> xq(few_xq_bytes(M, K));
        Dev<uint32_t> status(1);
        RowsArgs r{};
        r.a = din.p; r.n_parts = c.planes; r.part_stride = (size_t)M * ld; r.ld = ld; r.M = M; r.K = K; r.xq = xq.p; r.sx = sx.p; r.gain_kind = WK_BF16;
        if (c.pair) r.b = din.p + K;
        if (c.norm) { r.gain = dgain.p; r.eps = 1e-5f; r.resid = dres.p; r.resid_ld = K; r.out = out.p; r.out_ld = K; }
        CK(launch_rows_levels(r, 148, nullptr));
        FewArgs f{};
        f.nseg = (int)c.rows.size(); f.K = K; f.M = M; f.xq = xq.p; f.sx = sx.p; f.status = status.p;
        std::vector<Dev<unsigned char>*> packed;
        int total = 0;
        for (int n : c.rows) total += n;
        std::vector<double> want((size_t)M * total);
        int col = 0;
        for (size_t sg = 0; sg < c.rows.size(); sg++) {
            const int n = c.rows[sg];
            std::vector<int8_t> q((size_t)n * K);
            std::vector<__half> s((size_t)n * nb);
            for (auto& v : q) v = (int8_t)((int)(rng() % 256) - 128);
            for (auto& v : s) v = __float2half(0.0005f + 0.001f * (rng() % 1000) / 1000.0f);
            Dev<int8_t> dq(q);
            Dev<__half> ds(s);
            packed.push_back(new Dev<unsigned char>(q8_packed_bytes(n, K)));
            CK(launch_q8_pack_units(dq.p, ds.p, n, K, q8_pack_kc(n, K), packed.back()->p, nullptr));
            CK(cudaDeviceSynchronize());
            f.w[sg] = packed.back()->p; f.rows[sg] = n;
            for (int m = 0; m < M; m++)
                for (int i = 0; i < n; i++)
                    for (int b = 0; b < nb; b++) {
                        double t = 0;
                        for (int e = 0; e < 32; e++) t += (double)q[(size_t)i * K + b * 32 + e] * x[(size_t)m * K + b * 32 + e];
                        want[(size_t)m * total + col + i] += t * (double)__half2float(s[(size_t)i * nb + b]);
                    }
            col += n;
        }
        Dev<float> y((size_t)R * M * total + 8);
        f.y = y.p; f.ldy = total; f.part_stride = (size_t)M * total;
        CK(launch_few(f, 148, nullptr));
        const std::vector<float> raw = y.get();
        std::vector<float> got((size_t)M * total);
        for (int i = 0; i < 8; i++) if (raw[(size_t)R * M * total + i] != 0.0f) report("behind the end", 1, 0);
        for (int k = 0; k < R; k++) for (size_t i = 0; i < got.size(); i++) got[i] += raw[(size_t)k * M * total + i];
        // as for one vector: three levels, a norm's factor and the sums of blocks and of planes round
        report(std::to_string(total) + " x " + std::to_string(K) + ", " + std::to_string(M) + " rows, " + std::to_string(R) + " ranges", rel(got, want), 16 * std::exp2(-24.0));
        report("status", status.get()[0], 0);
        for (auto* p : packed) delete p;
    }
}

// Products on integer levels, one vector and several rows: an infinite or undefined element makes its own row undefined, as a sum over it would be, and no other.
// A row of tiny elements (`special` 0) keeps its 24 bits, or errors below 2^-127 an element.
static void level_specials() {
    const float inf = INFINITY, nan = std::nanf("");
    const int N = 72;
    for (int K : {512, 2560, 4096})
        for (int M : {1, 2, 5}) {
            if (M > 1 && !few_ranges(K, 148)) continue;
            for (float special : {nan, inf, -inf, 0.0f}) {
                const int nb = K / 32, bad = M - 1, at = K / 2 + 37;
                std::mt19937 rng(K + M);
                std::vector<float> x = normal(rng, (size_t)M * K, 1.0f);
                if (special != 0.0f) x[(size_t)bad * K + at] = special;
                else for (int e = 0; e < K; e++) x[(size_t)bad * K + e] *= 3e-33f;
                std::vector<int8_t> q((size_t)N * K);
                std::vector<__half> s((size_t)N * nb);
                for (auto& v : q) v = (int8_t)((int)(rng() % 255) - 127);
                for (auto& v : s) v = __float2half(0.01f);
                std::vector<double> want((size_t)M * N);
                for (int m = 0; m < M; m++)
                    for (int i = 0; i < N; i++)
                        for (int e = 0; e < K; e++) want[(size_t)m * N + i] += (double)q[(size_t)i * K + e] * x[(size_t)m * K + e] * (double)__half2float(s[(size_t)i * nb + e / 32]);
                Dev<int8_t> dq(q);
                Dev<__half> ds(s);
                Dev<unsigned char> w(q8_packed_bytes(N, K));
                CK(launch_q8_pack_units(dq.p, ds.p, N, K, q8_pack_kc(N, K), w.p, nullptr));
                Dev<float> dx(x), y((size_t)M * N), sx(few_sx_floats(M, K));
                Dev<int8_t> xq(few_xq_bytes(M, K));
                Dev<uint32_t> status(1);
                if (M == 1) {
                    GemvArgs a{};
                    a.nseg = 1; a.seg[0] = {w.p, nullptr, N, q8_pack_kc(N, K)}; a.K = K; a.wkind = WK_Q8; a.epi = EPI_STORE; a.x = dx.p; a.y = y.p; a.status = status.p;
                    CK(launch_gemv(a, 148, nullptr));
                } else {
                    RowsArgs r{};
                    r.a = dx.p; r.n_parts = 1; r.part_stride = (size_t)M * K; r.ld = K; r.M = M; r.K = K; r.xq = xq.p; r.sx = sx.p;
                    CK(launch_rows_levels(r, 148, nullptr));
                    FewArgs f{};
                    f.nseg = 1; f.w[0] = w.p; f.rows[0] = N; f.K = K; f.M = M; f.xq = xq.p; f.sx = sx.p; f.y = y.p; f.ldy = N; f.part_stride = (size_t)M * N; f.status = status.p;
                    CK(launch_few(f, 148, nullptr));
                }
                const std::vector<float> got = y.get();
                int defined = 0;
                for (int i = 0; i < N; i++) defined += !std::isnan(got[(size_t)bad * N + i]);
                const std::string what = (special == 0.0f ? "tiny ones" : std::to_string(special)) + " among " + std::to_string(K) + ", " + std::to_string(M) + " rows";
                if (special == 0.0f)
                    report(what, rel(std::vector<float>(got.begin() + (size_t)bad * N, got.end()), std::vector<double>(want.begin() + (size_t)bad * N, want.end())), 16 * std::exp2(-24.0) + std::exp2(-127.0) / 3e-33);
                else
                    report(what + ": outputs of its row that look defined", defined, 0);
                if (M > 1) report(what + ": the other rows", rel(got, std::vector<double>(want.begin(), want.begin() + (size_t)bad * N)), 16 * std::exp2(-24.0));
                report("status", status.get()[0], 0);
            }
        }
}

// The consumers of a weight stream whose producer gives up: three row groups' first halves come, one row group's second half, then the abort flag and nothing more.
// The warps of the two rings stand at different jobs by then.  All of them return, nothing is stored, no row is the best one.
template <bool ONE>
__global__ void __launch_bounds__(kGemvThreads) consume_short(const GemvArgs a, const int fills0, const int fills1, int* back) {
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ int s_abort;
    const int tid = threadIdx.x;
    GemvSmem g;
    const GemvPlan plan = gemv_plan(a, 0, 1, -1);
    gemv_carve(smem, a.K, GemvRings{a.ring_n[0], a.ring_n[1], a.ring_t[0], a.ring_t[1]}, &s_abort, &g);
    gemv_cta_begin(g, tid, &s_abort);
    if (tid >= kConsumers) {
        if (elect_one()) {
            bool ok = true;
            for (int w = 0; w < 2; w++)
                for (int f = 0; f < (w ? fills1 : fills0); f++) {            // (no more than the ring has stages)
                    const int slot = g.first(w) + f;
                    g.meta[slot] = make_int2(f, (int)m2_pack(kFillTiles, w * kFillTiles, 1, true, 0, true));
                    mbar_arrive_expect_tx(g.full0 + 8u * slot, kFillBytes);
                    bulk_g2s(smem_u32(g.at(w, f)), (const unsigned char*)a.seg[0].w + ((size_t)f * plan.tpr + w * kFillTiles) * kTileBytes, kFillBytes, g.full0 + 8u * slot);
                }
            for (int w = 0; w < 2; w++)
                for (int f = 0; f < (w ? fills1 : fills0); f++) ok = mbar_wait(g.full0 + 8u * (g.first(w) + f), 0u) && mbar_wait(g.empty0 + 8u * (g.first(w) + f), 0u) && ok;
            if (!ok) atomicOr(a.status, 1u << 31);
            *(volatile int*)&s_abort = 1;
        }
        return;
    }
    XSource xs{};
    xs.x = a.x;
    ArgBest best{-INFINITY, -1};
    ConsumerRing cr{0, 0u};
    GainRegs gr;
    gemv_gain_preload(a, tid, gr);
    gemv_consume<false, ONE>(a, xs, false, plan, g, cr, tid, a.status, &best, gr);
    atomicAdd(back, 1);
    if (tid == 0) back[1] = best.i;
}
static void gave_up() {
    const int K = 4096, N = 64;
    std::mt19937 rng(3);
    Dev<float> x(normal(rng, K, 1.0f));
    Dev<unsigned char> w(q8_packed_bytes(N, K));          // (zeros)
    for (bool one : {true, false})
        for (int epi : {EPI_STORE, EPI_RESID, EPI_ARGMAX})
            for (int fills0 : {3, 1}) {
                Dev<float> y(std::vector<float>(N, 7.0f)), res((size_t)N);
                Dev<int> back(2);
                Dev<uint32_t> status(1);
                GemvArgs a{};
                a.nseg = 1; a.seg[0] = {w.p, nullptr, N, q8_pack_kc(N, K)}; a.K = K; a.wkind = WK_Q8; a.epi = epi; a.x = x.p; a.y = y.p; a.resid = res.p; a.status = status.p;
                a.ring_n[0] = a.ring_n[1] = 3; a.ring_t[0] = a.ring_t[1] = kFillTiles;
                const size_t smem = gemv_fixed_smem(K) + 6 * kFillBytes;
                const void* fn = one ? (const void*)consume_short<true> : (const void*)consume_short<false>;
                CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
                int f0 = fills0, f1 = 4 - fills0;
                int* bp = back.p;
                void* params[] = {&a, &f0, &f1, &bp};
                CK(cudaLaunchKernel(fn, dim3(1), dim3(kGemvThreads), params, smem, nullptr));
                const std::vector<int> b = back.get();
                const std::string what = std::string(one ? "a tile per warp" : "any K") + ", epilogue " + std::to_string(epi) + ", fills " + std::to_string(f0) + " / " + std::to_string(f1) + ": ";
                report(what + "threads that did not return", kConsumers - b[0], 0);
                report(what + "a best row", b[1] != -1, 0);
                double stored = 0;
                for (float v : y.get()) stored += v != 7.0f;
                report(what + "rows stored", stored, 0);
                report(what + "the producer's own waits", status.get()[0] >> 31, 0);
            }
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "attention-sums") attention_sums();
    else if (what == "attention-specials") attention_specials();
    else if (what == "attention-prompt") attention_prompt();
    else if (what == "attention-band") attention_band();
    else if (what == "experts") experts();
    else if (what == "matvec-bf16") matvec_bf16();
    else if (what == "matvec-q8") matvec_q8();
    else if (what == "matvec-peer") matvec_peer();
    else if (what == "claims") claims();
    else if (what == "few-rows") few_rows();
    else if (what == "level-specials") level_specials();
    else if (what == "gave-up") gave_up();
    else { std::printf("unknown check\n"); return 2; }
    return failures ? 1 : 0;
}
