"""Products of prompts and the decode attention at the sizes where their tiles, slices and splits begin and end.

Tolerances: the products carry both operands to 22 bits; their error is the tensor core's rounding toward zero, which grows with K and
stays below 3e-5 at K = 8192 (the bound of the batched products' own test, 6e-5, holds with room).  The decode attention is held to the
3e-6 of its own test (what its f32 sums owe, and its contexts beyond a cluster's splits, are in test_decode_attention_gpu.py)."""
import numpy as np
import pytest

from util import dev, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("quant", [8, 4])
@pytest.mark.parametrize("m,K,N", [(33, 64, 2), (64, 256, 256), (65, 320, 257), (128, 64, 130), (129, 192, 300), (191, 576, 254), (193, 128, 512), (256, 1024, 20), (257, 448, 131),
                                   (700, 2048, 18992)])
def test_prompt_product_edges(oracle, quant, m, K, N):
    """Token tiles, row tiles, K of one step, of part of a stage, of several stages, outputs with and without
    aligned rows (N a multiple of 4 or not, a buffer that does not begin on 16 bytes), several rounds of tiles."""
    import ctypes as C
    import torch
    from forge_llm_b200 import synth
    from forge_llm_b200._lib import check, lib
    rng = np.random.default_rng(quant + m + K + N)
    w = synth.quantize(quant, rng.standard_normal((N, K), dtype=np.float32) * 0.02)
    x = rng.standard_normal((m, K), dtype=np.float32)
    rows = np.unique(np.r_[0:4, m // 2, m - 4:m])     # the oracle's rows
    ref = oracle.matmul_mat(quant, x[rows], w, K, N)
    dx, dw = dev(x), dev(w)
    pk = C.c_void_p()
    check(lib.forge_packed_create(quant, dw.data_ptr(), K, N, None, C.byref(pk)))
    first = None
    for skew in (0, 1) + (0,) * 30:   # the same bits every time: a stage or a buffer given back too early shows here
        buf = torch.full((m * N + 2,), 7.0, dtype=torch.float32, device="cuda")
        out = buf[skew:skew + m * N]
        check(lib.forge_matmul_mat_packed(out.data_ptr(), m, dx.data_ptr(), pk, None))
        check(lib.forge_packed_check(pk, None))
        got = out.cpu().numpy().reshape(m, N)
        assert rel_l2(got[rows], ref) < 6e-5
        assert np.isfinite(got).all() and buf[skew + m * N:].eq(7.0).all() and buf[:skew].eq(7.0).all()   # nothing outside is written
        first = got if first is None else first
        assert np.array_equal(got, first)    # the way out does not change a bit
    lib.forge_packed_destroy(pk)


@pytest.mark.parametrize("quant,hidden,ffn,n", [(4, 2048, 4096, 33), (8, 2048, 5120, 200), (4, 3072, 2048, 65), (8, 1024, 8192, 449)])
def test_prompt_slices(oracle, quant, hidden, ffn, n):
    """K slices of products, added up by the pair that owns the tile or left as partial outputs, ragged last tiles, the SiLU epilogue.  The bound is eight products
    of 3e-5 each and twice what rounding K and V to fp16 makes of a difference of 6e-6 (sqrt(6e-6 * 2^-11))."""
    from forge_llm_b200 import configs, runtime, synth
    c = configs.tiny(quant, hd=64, nq=hidden // 64, nkv=hidden // 128, layers=2, hidden=hidden, ffn=ffn, vocab=1000)
    blob = synth.make_weights_bin(c)
    gm = runtime.Model(c, blob)
    om = oracle.OracleModel(c, blob, kv_mode=oracle.KV_F16)
    p = synth.prompt_tokens(c, n, seed=n)
    want = om.forward_prefill(p)
    kv = gm.new_cache(max_seq=n + 2, batch=1)
    first = None
    for _ in range(5):
        kv.reset()
        got = gm.forward_prefill(p, kv)
        assert rel_l2(got, want) < 3.5e-4
        first = got if first is None else first
        assert np.array_equal(got, first)
    kv.close()
    gm.close()


@pytest.mark.parametrize("hd,nq,nkv", [(64, 16, 1), (64, 18, 2), (96, 9, 1), (128, 7, 7), (128, 16, 2)])
@pytest.mark.parametrize("seq", [1, 15, 16, 17, 63, 65, 511, 513, 8300])
def test_decode_attention_edges(oracle, hd, nq, nkv, seq):
    """One to sixteen query heads per KV head (more than eight take two passes, here over pages that fit the ring), contexts around a warp's keys, a page and
    eight splits, and one whose splits are merged through global memory where KV heads are few."""
    import torch
    from forge_llm_b200._lib import check, lib
    rng = np.random.default_rng(hd + nq + seq)
    q = rng.standard_normal(nq * hd, dtype=np.float32)
    k = (rng.standard_normal((seq, nkv * hd), dtype=np.float32) * 0.5).astype(np.float16)
    v = rng.standard_normal((seq, nkv * hd), dtype=np.float32).astype(np.float16)
    ref = oracle.attention_flash(q, oracle.KV_F16, k.astype(np.float32), v.astype(np.float32), None, None, seq, nq, nkv, hd)
    dq, dk, dv = dev(q), dev(k.view(np.uint16)), dev(v.view(np.uint16))
    for fn in (lib.forge_attention_flash, lib.forge_attention_flash_static):
        out = torch.full((nq * hd,), float("nan"), dtype=torch.float32, device="cuda")
        check(fn(out.data_ptr(), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), seq, nq, nkv, hd, None))
        torch.cuda.synchronize()
        assert rel_l2(out.cpu().numpy(), ref) < 3e-6


def test_batched_steps_of_every_size_agree(oracle):
    """Steps of 1 .. 66 sequences take different products (one row, rows by rows, 8, 32 and 64 rows, K slices): the logits of the same sequences agree, and the
    first nine are the oracle's.  The oracle's bound is the products' 3e-5 through two layers, twice (attention and feed-forward) each."""
    from forge_llm_b200 import configs, runtime, synth
    c = configs.tiny(8, hd=64, nq=6, nkv=2, layers=2, hidden=1024, ffn=1536, vocab=1000)
    blob = synth.make_weights_bin(c)
    gm = runtime.Model(c, blob)
    om = oracle.OracleModel(c, blob, kv_mode=oracle.KV_F16)
    prompts = [synth.prompt_tokens(c, 3 + 7 * i % 150, seed=50 + i) for i in range(66)]
    want = []
    for p in prompts[:9]:
        om.reset()
        om.forward_prefill(p)
        want.append(om.forward(int(p[0])))
    ref = None
    for batch in (66, 64, 33, 32, 9, 8, 2, 1):
        kv = gm.new_cache(max_seq=200, batch=batch)
        for i in range(batch):
            gm.forward_prefill(prompts[i], kv, seq=i, want_logits=False)
        got = gm.forward_batch([int(p[0]) for p in prompts[:batch]], kv)
        if ref is None:
            ref = got
        assert np.abs(got - ref[:batch]).max() < 1e-3   # fp16 cache rows and the products' last bits
        for a, b in zip(got, want):
            assert rel_l2(a, b) < 1.2e-4
        kv.close()
    gm.close()


@pytest.mark.parametrize("quant,hidden", [(8, 160), (4, 160), (8, 256)])
def test_small_batched_steps_by_both_products(quant, hidden):
    """Steps of 2 .. 8 sequences: rows of whole 64-column steps take the tcgen05 products, others the mma.sync one; both agree with single steps to the products' and the
    fp16 cache's last bits (3e-5 a product, eight of them)."""
    from forge_llm_b200 import configs, runtime, synth
    c = configs.tiny(quant, hd=64, nq=4, nkv=2, layers=2, hidden=hidden, ffn=384, vocab=1000)
    gm = runtime.Model(c, synth.make_weights_bin(c))
    prompts = [synth.prompt_tokens(c, 5 + 9 * i, seed=70 + i) for i in range(8)]
    want = []
    for p in prompts:
        kv = gm.new_cache(max_seq=100)
        gm.forward_prefill(p, kv)
        want.append(gm.forward(int(p[0]), kv))
        kv.close()
    for batch in (2, 3, 5, 8):
        kv = gm.new_cache(max_seq=100, batch=batch)
        for i in range(batch):
            gm.forward_prefill(prompts[i], kv, seq=i)
        got = gm.forward_batch([int(p[0]) for p in prompts[:batch]], kv)
        assert max(rel_l2(a, b) for a, b in zip(got, want)) < 2.4e-4
        kv.close()
    gm.close()
