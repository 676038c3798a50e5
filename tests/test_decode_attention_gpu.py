"""Decode attention: which of its two kernels a model takes, and what each of them owes."""
import os

import numpy as np
import pytest

from util import rel_l2

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "kquant_steps.npz")


def kquant_steps():
    """Logits of a small Q4_K_M model: a prompt that goes token by token, then steps over two, three, ... pages."""
    from forge_llm_b200 import configs, runtime, synth
    c = configs.with_proj_quant(configs.tiny(12, hd=64, nq=8, nkv=2, layers=4, ffn=512, vocab=256), v=14, down=14, lm_head=14)
    gm = runtime.Model(c, synth.make_weights_bin(c))
    kv = gm.new_cache(max_seq=400)
    toks = synth.prompt_tokens(c, 200)
    got = [gm.forward_prefill(toks[:90], kv)] + [gm.forward(int(t), kv) for t in toks[90:]]
    kv.close()
    gm.close()
    return np.stack(got[::10])


def test_kquant_steps_keep_their_logits():
    """Models with K-quants round every row to 8 bits in front of a product, so that a last bit of the attention that comes out otherwise now and
    then moves a whole step of that rounding (6e-3 of a step's logits here).  The stored logits are those of attention by f32 multiply-adds in a
    fixed order; 1e-6 leaves room for f32 rounding and for no such step."""
    assert rel_l2(kquant_steps(), np.load(GOLDEN)["logits"]) < 1e-6
