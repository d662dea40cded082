"""Routed experts at sizes where their kernels change shape: rows longer than one ring stage, more experts than one pass of the router, widths that
are no multiple of a warp's trip."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import OracleModel  # noqa: E402


@pytest.mark.parametrize("over", [
    dict(hidden=3584, ffn=3200, n_layers=1),              # 112 and 100 blocks per row: two chunks each
    dict(n_experts=40, top_k=3),                          # a second pass of the router's warps, an odd selection
    dict(hidden=544, ffn=96, top_k=1),                    # 17 and 3 blocks per row
    dict(ffn=2880, top_k=8),                              # every expert; a ring squeezed by the activations
], ids=["long", "experts40", "narrow", "all"])
def test_routed_experts_match_oracle(pkg, over):
    desc = pkg.CONFIGS["small_oss"].copy(**over)
    orc = OracleModel(desc)
    orc.synth(17)
    prompt = orc.synth_tokens(17, 6)
    want, lo, margins = orc.generate(prompt, 6, return_last_logits=True, return_margins=True)
    rt = pkg.B200Runtime.initialize(device=0)
    try:
        rt.load_model(desc)
        rt.synth(17)
        got, lg = rt.generate(prompt, 6), rt.get_f32()
    finally:
        rt.close()
    assert got == want, f"min oracle top-1/top-2 margin {min(margins):.3e}"
    # the other tests of these layers allow 1e-2 of the largest logit; f32 sums over a bf16 cache differ far less
    assert np.max(np.abs(lg.astype(np.float64) - lo)) <= 5e-3 * np.max(np.abs(lo))
