"""Token rows of the qwen3moe engine: the tensor-core K-quant product at the edges of its tiles (and at the largest integers its
accumulators can meet), and prompts that walk the layers together against the one-token step."""
import ctypes as C

import numpy as np
import pytest

from conftest import bits, to_dev
from cpubrrr_b200 import synth as S

pytestmark = pytest.mark.gpu


def P(t):
    return C.c_void_p(t.data_ptr())


def extreme(w, kind):
    """Every weight of the first rows at the end of its range, with scales and minima at theirs."""
    w = w.copy()
    nsb = w.shape[1] if w.ndim == 3 else w.reshape(w.shape[0], -1).shape[1] // (144 if kind == 12 else 210)
    b = w.reshape(w.shape[0], nsb, -1)
    if kind == 12:
        b[:3, :, 4:16] = 0xFF
        b[0, :, 16:] = 0xFF
        b[1, :, 16:] = 0xF0
    else:
        b[:2, :, 192:208] = 0x7F
        b[2, :, 192:208] = 0x80
        b[0, :, :192] = 0x00
        b[1, :, :192] = 0xFF
        b[2, :, :192] = 0x00
    return w


@pytest.mark.parametrize("kind", [12, 14])
@pytest.mark.parametrize("rows,cols,ntok", [(128, 256, 1), (768, 2048, 16), (128, 768, 17), (256, 512, 33), (2048, 768, 70), (640, 4096, 512)])
def test_kquant_rows_equal_one_token_products(brrr, dev, kind, rows, cols, ntok):
    import torch
    L = brrr.lib()
    w = S.synth_q4k(rows, rows, cols) if kind == 12 else S.synth_q6k(rows, rows, cols)
    w = extreme(np.asarray(w).reshape(rows, -1), kind)
    dw = to_dev(w.reshape(-1), dev)
    g = torch.Generator(device=dev); g.manual_seed(ntok)
    x = torch.randn((ntok, cols), device=dev, generator=g)
    x[0] = 3.0                                        # every quant 127: the largest sums
    if ntok > 2:
        x[1] = -3.0
        x[2] = 0.0
    y = torch.empty((ntok, rows), device=dev)
    assert L.brrr_kquant_rows(P(dw), kind, rows, cols, P(x), ntok, P(y), None) == 0
    q = torch.empty((ntok, cols), dtype=torch.int8, device=dev); s = torch.empty((ntok, cols // 256), device=dev)
    b = torch.empty((ntok, cols // 32), dtype=torch.int32, device=dev)
    assert L.brrr_quant_q8k(P(x), x.numel(), P(q), P(s), P(b), None) == 0
    want = torch.empty((ntok, rows), device=dev)
    for t in range(ntok):
        if kind == 12:
            assert L.brrr_q4k_matvec(P(dw), rows, cols, P(q[t]), P(s[t]), P(b[t]), P(want[t]), None, None) == 0
        else:
            assert L.brrr_q6k_matvec(P(dw), rows, cols, P(q[t]), P(s[t]), P(want[t]), None, None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(bits(y.cpu().numpy()), bits(want.cpu().numpy()))
    assert L.brrr_kquant_rows(P(dw), kind, rows, cols, P(x), 513, P(y), None) == 1


@pytest.mark.parametrize("shape,lengths", [
    (dict(n_embd=256, n_layer=2, n_head=2, n_head_kv=1, n_expert=8, n_expert_used=2, n_ff_exp=256, n_vocab=512), [2, 3, 31, 64, 600]),
    (dict(n_embd=512, n_layer=3, n_head=8, n_head_kv=2, n_expert=40, n_expert_used=8, n_ff_exp=768, n_vocab=2051), [5, 33, 130]),
    (dict(n_embd=768, n_layer=2, n_head=8, n_head_kv=1, n_expert=128, n_expert_used=8, n_ff_exp=512, n_vocab=1000), [17, 300]),
    (dict(n_embd=256, n_layer=1, n_head=8, n_head_kv=1, n_expert=8, n_expert_used=2, n_ff_exp=256, n_vocab=300), [1300, 2400]),
    (dict(n_embd=768, n_layer=2, n_head=6, n_head_kv=6, n_expert=128, n_expert_used=8, n_ff_exp=512, n_vocab=1000), [9]),      # token by token
])
def test_qwen_prefill_rows_equal_steps(brrr, shape, lengths):
    """Logits, hidden state and the cache (through later steps) of a prompt fed at once against the same tokens one by one."""
    cfg = brrr.make_qwen_cfg(**shape)
    eng = brrr.QwenEngine.synth(cfg, 23)
    for n in lengths:
        prompt = S.synth_prompt(23 + n, n, cfg.n_vocab)
        tok = 0
        for i, t in enumerate(prompt):
            tok = eng.run(int(t), i, i == n - 1)
        lg, hid, toks = bits(eng.logits()), bits(eng.hidden()), eng.decode(tok, n, 6)
        lg2 = bits(eng.logits())
        assert eng.prefill(prompt) == tok, n
        assert np.array_equal(bits(eng.logits()), lg) and np.array_equal(bits(eng.hidden()), hid), n
        assert np.array_equal(eng.decode(tok, n, 6), toks) and np.array_equal(bits(eng.logits()), lg2), n
        if n > 4:                                     # a prompt in two parts: rows over keys that are already there
            eng.prefill(prompt[:n // 3])
            assert eng.prefill(prompt[n // 3:], n // 3) == tok
            assert np.array_equal(bits(eng.logits()), lg), n
    with pytest.raises(Exception):
        eng.prefill([cfg.n_vocab])
    eng.close()
