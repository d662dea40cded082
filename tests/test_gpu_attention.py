"""Attention over a bf16 cache at the edges of its tiles: rows of several sequences (one batched step) against each sequence alone (one decode
step), and single steps against the same step over a cache in 32 bits, which takes the plain kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# tiles of 16 keys per warp, 64 per CTA, splits of whole 64s (rows) or 16s (single steps)
CONTEXTS = [1, 2, 14, 15, 16, 17, 62, 63, 64, 65, 127, 128, 129, 300, 511, 700]
# (query heads, KV heads, head size): four and fewer per KV head, five to eight, one
HEADS = [(8, 2, 128), (8, 2, 64), (12, 4, 128), (16, 2, 64), (40, 8, 64), (8, 8, 64), (16, 2, 128)]


def bf16(x):
    u = np.ascontiguousarray(x, dtype=np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


def rows_of(rng, n, width):
    """Keys and values of a conversation; values of rows at the tiles' edges and of a few others stand out, so that a lost key shows."""
    k, v = rng.normal(0, 0.3, (n, width)), rng.normal(0, 1, (n, width))
    for r in (0, 15, 16, 63, 64, n - 2, n - 1):
        if 0 <= r < n:
            v[r] *= 30
    return bf16(k), bf16(v)


def model(pkg, heads, **kw):
    nq, nkv, hd = heads
    return pkg.CONFIGS["small_q8"].copy(n_layers=1, n_q_heads=nq, n_kv_heads=nkv, head_dim=hd, max_seq=1024, **kw)


def err(a, b):
    return float(np.linalg.norm(a.astype(np.float64) - b) / np.linalg.norm(b.astype(np.float64)))


@pytest.mark.parametrize("heads", HEADS[:-1], ids=lambda h: "%dx%dx%d" % h)          # (batches take at most four heads of 128 per KV head)
@pytest.mark.parametrize("page", [0, 64])
def test_batched_step_equals_single_steps(pkg, heads, page):
    rng = np.random.default_rng(sum(heads) + page)
    d = model(pkg, heads, max_batch=len(CONTEXTS), kv_page_rows=page)
    rt = pkg.B200Runtime.initialize(device=0)
    try:
        rt.load_model(d)
        rt.synth(5)
        alone = []
        for s, n in enumerate(CONTEXTS):
            rt.seq_select(s)
            for which, rows in zip("kv", rows_of(rng, n, heads[1] * heads[2])):
                rt.kv_load(0, which, n, rows.view(np.uint8))
            rt.set_data([7 * s + 3])
            rt.execute({"s": 1, "p": n})
            alone.append(rt.get_f32())
        rt.batch_begin([7 * s + 3 for s in range(len(CONTEXTS))], CONTEXTS)
        rt.batch_decode(1)
        for s, n in enumerate(CONTEXTS):
            # the step's own key and value may round the other way (2^-9 of one row among n + 1), the rest is sums of 32 bits
            assert err(rt.batch_get_logits(s), alone[s]) < 3e-3, f"{n} cached rows"
    finally:
        rt.close()


@pytest.mark.parametrize("heads", HEADS, ids=lambda h: "%dx%dx%d" % h)
@pytest.mark.parametrize("splits", [0, 1, 3])
def test_single_step_equals_plain_kernels(pkg, heads, splits):
    rng = np.random.default_rng(sum(heads) * 3 + splits)
    out = []
    for kv in ("bf16", "f32"):
        rng = np.random.default_rng(sum(heads) * 3 + splits)
        rt = pkg.B200Runtime.initialize(device=0, attn_splits=splits)
        try:
            rt.load_model(model(pkg, heads, kv_dtype=pkg.DTYPE[kv]))
            rt.synth(5)
            got = []
            for s, n in enumerate(CONTEXTS):
                for which, rows in zip("kv", rows_of(rng, n, heads[1] * heads[2])):
                    data = rows if kv == "bf16" else (rows.astype(np.uint32) << 16).view(np.float32)
                    rt.kv_load(0, which, n, np.ascontiguousarray(data).view(np.uint8))
                rt.set_data([7 * s + 3])
                rt.execute({"s": 1, "p": n})
                got.append(rt.get_f32())
            out.append(got)
        finally:
            rt.close()
    for n, a, b in zip(CONTEXTS, *out):
        # rounded against unrounded: one key and value of n + 1, 2^-9 of theirs each
        assert err(a, b) < 4e-3, f"{n} cached rows"
