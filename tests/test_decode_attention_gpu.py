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


def attend(q, k, v, seq, window=0, fn=None):
    """The operator's result for float32 queries [heads][hd] over fp16 rows [seq][kv heads][hd], everything on the GPU."""
    import torch
    from forge_llm_b200._lib import check, lib
    (nq, hd), nkv = q.shape, k.shape[1]
    out = torch.full((nq, hd), 7.0, device="cuda")
    p = [x.data_ptr() for x in (out, q, k, v)]
    if window:
        check(lib.forge_attention_sliding(*p, seq, window, nq, nkv, hd, None))
    else:
        check((fn or lib.forge_attention_flash)(*p, seq, nq, nkv, hd, None))
    torch.cuda.synchronize()
    return out


def attend64(q, k, v, seq, window=0):
    """The same in 64 bits."""
    import torch
    (nq, hd), nkv = q.shape, k.shape[1]
    lo = max(0, seq - window) if window else 0
    s = torch.einsum("ngd,tnd->ngt", q.double().view(nkv, nq // nkv, hd), k[lo:seq].double()) / hd ** 0.5
    p = torch.exp(s - s.amax(-1, keepdim=True))
    return (torch.einsum("ngt,tnd->ngd", p, v[lo:seq].double()) / p.sum(-1, keepdim=True)).reshape(nq, hd)


def inputs(hd, nq, nkv, seq, q_scale=1.0, k_scale=0.5):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(hd + 7 * nq + 31 * nkv + seq)
    q = q_scale * torch.randn(nq, hd, generator=g, device="cuda")
    k, v = torch.randn(2, seq, nkv, hd, generator=g, device="cuda")
    return q, (k_scale * k).half(), v.half()


def error(got, want):
    return ((got.double() - want).norm() / want.norm()).item()


@pytest.mark.parametrize("hd,nq,nkv", [(64, 9, 1), (64, 32, 2), (96, 12, 1), (128, 16, 1), (128, 24, 2)])
@pytest.mark.parametrize("seq,window", [(1100, 0), (2100, 0), (4096, 0), (8192, 0), (8191, 3000), (8300, 0), (8300, 5000)])
def test_two_passes_over_more_pages_than_the_ring_holds(hd, nq, nkv, seq, window):
    """Nine to sixteen query heads per KV head take two passes over a CTA's pages; here the pages of the first pass fill the ring, so that the copies
    of the second can only begin as pages are read, and the CTAs of a cluster meet behind both."""
    from forge_llm_b200._lib import lib
    q, k, v = inputs(hd, nq, nkv, seq)
    want = attend64(q, k, v, seq, window)
    assert error(attend(q, k, v, seq, window), want) < 3e-6
    if not window:
        assert error(attend(q, k, v, seq, fn=lib.forge_attention_flash_static), want) < 3e-6


@pytest.mark.parametrize("hd,nq,nkv", [(64, 16, 1), (128, 12, 1)])
def test_steps_of_models_with_many_heads_per_kv_head(hd, nq, nkv):
    """The same through a session: a step behind n tokens gives the logits of a prompt of n + 1 (the prompt's attention is another kernel)."""
    from forge_llm_b200 import configs, runtime, synth
    c = configs.tiny(8, hd=hd, nq=nq, nkv=nkv, layers=2)
    gm = runtime.Model(c, synth.make_weights_bin(c))
    toks = synth.prompt_tokens(c, 3001)
    kv = gm.new_cache(max_seq=3100)
    want = gm.forward_prefill(toks, kv)
    kv.reset()
    gm.forward_prefill(toks[:3000], kv, want_logits=False)
    got = gm.forward(int(toks[3000]), kv)
    assert rel_l2(got, want) < 1e-3    # the prompt's queries and weights enter its products as plain fp16
    kv.close()
    gm.close()


@pytest.mark.parametrize("hd,nq,nkv", [(64, 14, 2), (96, 6, 2), (128, 8, 1)])
@pytest.mark.parametrize("q_scale,k_scale", [(1e-30, 1.0), (1e-3, 1e3), (1e2, 1e-2), (4e6, 1e-6), (1e7, 1e-7)])
def test_queries_of_any_size(hd, nq, nkv, q_scale, k_scale):
    """A query is an f32 number: its size may not cost bits, and a large one may not overflow."""
    q, k, v = inputs(hd, nq, nkv, 700, q_scale, k_scale)
    assert error(attend(q, k, v, 700), attend64(q, k, v, 700)) < 3e-6


@pytest.mark.parametrize("hd,nq,nkv,seq", [(64, 32, 8, 8192), (64, 14, 2, 20000), (96, 128, 128, 4096), (128, 32, 32, 8192), (128, 16, 2, 8192)])
def test_long_sums_keep_f32(hd, nq, nkv, seq):
    """Thousands of weights of one size: what an f32 result owes.  A sum of independent roundings of 2^-24 stays below 2.5e-7; sums that a tensor core carries from
    page to page lose a bit toward zero at every step and come to 3.5e-7 and more."""
    q, k, v = inputs(hd, nq, nkv, seq, q_scale=0.1)
    assert error(attend(q, k, v, seq), attend64(q, k, v, seq)) < 2.8e-7


@pytest.mark.parametrize("hd,nq,nkv", [(64, 14, 2), (128, 32, 32)])
@pytest.mark.parametrize("above", [5, 10, 14])
def test_weights_beside_a_first_token_that_takes_almost_all(hd, nq, nkv, above):
    """A first token whose score lies far above the others' and whose value is zero: the result is made of weights of e^-above, and each of them
    still has the bits of an f32 number."""
    seq = 1000
    q, k, v = inputs(hd, nq, nkv, seq, q_scale=0.1)
    q[:, 0] = 4.0
    k[:, :, 0] = 0
    k[0, :, :] = 0
    k[0, :, 0] = above * hd ** 0.5 / 4
    v[0] = 0
    assert error(attend(q, k, v, seq), attend64(q, k, v, seq)) < 1e-6


@pytest.mark.parametrize("hd,nq,nkv,seq,window", [(64, 14, 2, 100, 0), (64, 12, 1, 3000, 0), (64, 8, 2, 9000, 700), (96, 6, 2, 700, 0), (128, 16, 16, 2000, 300), (128, 4, 2, 20000, 0)])
def test_infinite_keys_and_values(hd, nq, nkv, seq, window):
    """What f32 arithmetic gives: an infinite value reaches the result with its sign, a key whose score is minus infinity has no weight, one whose
    score is plus infinity takes the row with it.  Rows and KV heads without one are as they would be."""
    import torch
    q, k, v = inputs(hd, nq, nkv, seq)
    G = nq // nkv
    v[seq - 9, 0, 5], v[seq - 70, 0, 6] = float("inf"), float("-inf")
    v[seq - 1, 0, 7] = v[seq - 30, 0, 7] = float("inf")
    k[seq - 20, nkv - 1, 3] = float("-inf")
    if nkv > 1:   # the last KV head's first query: with a positive value there the key is ignored, with a negative one the row is lost
        q[(nkv - 1) * G, 3] = q[(nkv - 1) * G, 3].abs()
    got, want = attend(q, k, v, seq, window), attend64(q, k, v, seq, window)
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()].sign().double(), want[want.isinf()].sign())
    ok = want.isfinite()
    assert ok.any() and error(got[ok], want[ok]) < 3e-6


def test_steps_of_fewer_sequences_than_the_cache_holds():
    """A long cache of many sequences, stepped by one and by three of them: their launches take more context splits than one of all sequences
    would, and the logits are those of a cache of their own."""
    from forge_llm_b200 import configs, runtime, synth
    c = configs.tiny(8, hd=64, nq=4, nkv=1, layers=1)
    gm = runtime.Model(c, synth.make_weights_bin(c))
    prompts = [synth.prompt_tokens(c, n, seed=n) for n in (4000, 2500, 130)]
    own = []
    for p in prompts:
        kv = gm.new_cache(max_seq=4096)
        gm.forward_prefill(p, kv, want_logits=False)
        own.append(gm.forward(int(p[0]), kv))
        kv.close()
    kv = gm.new_cache(max_seq=4096, batch=64)
    for i, p in enumerate(prompts):
        gm.forward_prefill(p, kv, seq=i, want_logits=False)
    got = gm.forward_batch([int(p[0]) for p in prompts], kv)
    for a, b in zip(got, own):
        assert rel_l2(a, b) < 1e-4    # products of several rows round otherwise
    kv.reset()
    gm.forward_prefill(prompts[0], kv, want_logits=False)
    assert rel_l2(gm.forward(int(prompts[0][0]), kv), own[0]) < 1e-5
    kv.close()
    gm.close()


@pytest.mark.parametrize("hd,nq,nkv", [(64, 7, 1), (64, 28, 2), (96, 8, 1), (96, 6, 6), (96, 20, 2), (128, 14, 2), (128, 16, 1)])
@pytest.mark.parametrize("seq,window", [(40, 17), (129, 64), (130, 65), (1000, 500), (2500, 2400), (8300, 1), (8300, 4100), (20000, 19937)])
def test_windows_with_every_group(hd, nq, nkv, seq, window):
    """Windows that begin within a warp's keys, at a page and beyond whole splits, for one to sixteen query heads per KV head: what lies in front of them
    has no weight, whatever it holds."""
    q, k, v = inputs(hd, nq, nkv, seq)
    want = attend64(q, k, v, seq, window)
    k[:seq - window], v[:seq - window] = float("nan"), float("inf")
    assert error(attend(q, k, v, seq, window), want) < 3e-6
