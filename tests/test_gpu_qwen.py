"""Whole-model parity of the qwen3moe engine on the GPU: the decode step (one CUDA graph per token)
against the CPU oracle on seeded synthetic models.

Bar: identical greedy tokens for >= 128 steps; logits, hidden state and the per-layer trace
bit-identical to the oracle (0 ulp), which implies the 1e-2 relative-L2 logit bound."""
import json
import os

import numpy as np
import pytest

from conftest import bits
from cpubrrr_b200 import synth as S

pytestmark = pytest.mark.gpu
GOLD = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")


def ocfg_of(orc, c):
    return orc.make_qcfg(d=c.n_embd, nh=c.n_head, nkv=c.n_head_kv, hd=c.head_dim, nl=c.n_layer, ne=c.n_expert, topk=c.n_expert_used,
                         ff=c.n_ff_exp, nvocab=c.n_vocab, rope_base=c.rope_freq_base, rms_eps=c.rms_eps)


def greedy(run, prompt, n):
    tok = 0
    for i, t in enumerate(prompt):
        tok = run(int(t), i, i == len(prompt) - 1)
    out, pos = [], len(prompt)
    for _ in range(n):
        out.append(tok)
        tok = run(tok, pos, True)
        pos += 1
    return out


def test_qwen_golden_tokens_tiny(brrr):
    g = json.load(open(os.path.join(GOLD, "qwen_tiny_tokens.json")))
    c = g["cfg"]
    eng = brrr.QwenEngine.synth(brrr.make_qwen_cfg(c["d"], c["nl"], c["nh"], c["nkv"], c["ne"], c["topk"], c["ff"], c["nvocab"]), g["seed"])
    first = eng.prefill(g["prompt"])
    toks = eng.decode(first, len(g["prompt"]), len(g["tokens"]))
    assert [first] + [int(t) for t in toks[:-1]] == g["tokens"]
    assert [int(b) for b in bits(eng.logits())[:8]] != []      # logits are readable after a decode run
    eng.close()


@pytest.mark.parametrize("shape", [
    dict(n_embd=256, n_layer=2, n_head=2, n_head_kv=1, n_expert=8, n_expert_used=2, n_ff_exp=256, n_vocab=512),
    dict(n_embd=512, n_layer=3, n_head=8, n_head_kv=2, n_expert=40, n_expert_used=8, n_ff_exp=768, n_vocab=2051),
    dict(n_embd=768, n_layer=2, n_head=6, n_head_kv=6, n_expert=128, n_expert_used=8, n_ff_exp=512, n_vocab=1000),
])
def test_qwen_tokens_logits_hidden_bit_exact(brrr, orc, shape):
    cfg = brrr.make_qwen_cfg(**shape)
    seed = 41
    eng = brrr.QwenEngine.synth(cfg, seed)
    om = orc.QwenModel.synth(ocfg_of(orc, cfg), seed)
    prompt = S.synth_prompt(seed, 11, cfg.n_vocab)
    n = 136
    want = greedy(om.run, prompt, n)
    got = greedy(eng.run, prompt, n)
    assert got == want
    assert np.array_equal(bits(eng.logits()), bits(om.logits()))
    assert np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    first = eng.prefill(prompt)
    toks = eng.decode(first, len(prompt), n)
    assert [first] + [int(t) for t in toks[:-1]] == want
    assert eng.launches_per_step(True) == 2 + 7 * cfg.n_layer + 2      # embed, first norm; seven per layer; head, finish
    assert eng.bytes_per_step(10) > 0
    eng.close()


@pytest.mark.parametrize("shape", [
    dict(n_embd=2304, n_layer=2, n_head=4, n_head_kv=2, n_expert=33, n_expert_used=4, n_ff_exp=512, n_vocab=1003),      # nine superblocks: a second pass of one
    dict(n_embd=4096, n_layer=3, n_head=8, n_head_kv=2, n_expert=40, n_expert_used=8, n_ff_exp=1024, n_vocab=700),      # down behind the router's end
])
def test_qwen_rows_wider_than_eight_superblocks(brrr, orc, shape):
    """n_embd above 2048: the two-pass rows of q|k|v, gate/up and the head; no step is run again."""
    cfg = brrr.make_qwen_cfg(**shape)
    eng = brrr.QwenEngine.synth(cfg, 29)
    om = orc.QwenModel.synth(ocfg_of(orc, cfg), 29)
    prompt = S.synth_prompt(29, 5, cfg.n_vocab)
    want = greedy(om.run, prompt, 12)
    assert greedy(eng.run, prompt, 12) == want
    assert np.array_equal(bits(eng.logits()), bits(om.logits())) and np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    first = eng.prefill(prompt)
    assert [first] + [int(t) for t in eng.decode(first, len(prompt), 12)[:-1]] == want
    assert np.array_equal(bits(eng.logits()), bits(om.logits())) and np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    assert (eng.spec_redos(), eng.wait_fallbacks()) == (0, 0)
    eng.close(); om.close()


@pytest.mark.parametrize("ne,topk", [(1, 1), (8, 8), (33, 5), (128, 8), (129, 8), (256, 8)])
def test_qwen_picks_of_the_estimate(brrr, orc, ne, topk):
    """Expert counts at the edges of the selection (four experts a lane up to 128, eight above): the estimate's picks are the router's, so
    no step is run again, and the tokens are the oracle's.  With ff = 256 and eight slots a CTA's rows meet several slots."""
    cfg = brrr.make_qwen_cfg(256, 2, 2, 1, ne, topk, 256, 512)
    eng = brrr.QwenEngine.synth(cfg, 43)
    om = orc.QwenModel.synth(ocfg_of(orc, cfg), 43)
    prompt = S.synth_prompt(43, 5, cfg.n_vocab)
    want = greedy(om.run, prompt, 24)
    assert greedy(eng.run, prompt, 24) == want
    assert eng.spec_redos() == 0
    eng.close()


def test_qwen_layer_trace_bit_exact(brrr, orc):
    cfg = brrr.make_qwen_cfg(512, 4, 4, 2, 16, 4, 256, 772)
    eng = brrr.QwenEngine.synth(cfg, 5)
    om = orc.QwenModel.synth(ocfg_of(orc, cfg), 5)
    tr = om.enable_trace()
    prompt = S.synth_prompt(5, 40, cfg.n_vocab)
    for i, t in enumerate(prompt):
        om.run(int(t), i, True)
        got = eng.run_trace(int(t), i)
        assert np.array_equal(bits(got), bits(tr)), f"position {i}"
    eng.close()


def test_qwen_long_context_bit_exact(brrr, orc):
    """Attention over more than a thousand keys (several passes of the 32-key score loop, long
    serial sums): feed a long prompt without the head, compare the hidden state and the next tokens."""
    cfg = brrr.make_qwen_cfg(256, 2, 4, 1, 8, 2, 256, 640)
    eng = brrr.QwenEngine.synth(cfg, 9)
    om = orc.QwenModel.synth(ocfg_of(orc, cfg), 9)
    prompt = S.synth_prompt(9, 1100, cfg.n_vocab)
    a = b = 0
    for i, t in enumerate(prompt):
        last = i == len(prompt) - 1
        a = om.run(int(t), i, last)
        b = eng.run(int(t), i, last)
    assert a == b
    assert np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    assert np.array_equal(bits(eng.logits()), bits(om.logits()))
    toks = eng.decode(b, len(prompt), 8)
    want = []
    tok, pos = a, len(prompt)
    for _ in range(8):
        tok = om.run(tok, pos, True); pos += 1
        want.append(tok)
    assert [int(t) for t in toks] == want
    eng.close()


def test_qwen_data_dir_load(brrr, orc, tmp_path):
    """brrr_qwen_open on a GGUF blob + data directory == the synthetic builder (same bytes)."""
    import refdata
    cfg, d, blob = refdata.case_data_dir(str(tmp_path / "qw"), "qwen_d256", 12)
    eng = brrr.QwenEngine.open(d, blob)
    ref = brrr.QwenEngine.synth(cfg, 12)
    assert eng.cfg.n_ff_exp == 256 and eng.cfg.n_vocab == 600
    prompt = S.synth_prompt(12, 7, cfg.n_vocab)
    assert greedy(eng.run, prompt, 40) == greedy(ref.run, prompt, 40)
    assert np.array_equal(bits(eng.logits()), bits(ref.logits()))
    eng.close(); ref.close()


def test_qwen_mixed_kquant_types_per_tensor(brrr, orc, tmp_path):
    """A file that mixes K-quant types per tensor the way real files do (attn_v of layer 0 stored as
    Q6_K, the down experts of layer 1 as Q4_K; the reference dispatches on the manifest's type,
    src/bin/engine_qwen2.rs:202-212): the engine and the oracle load the same directory and agree
    bit for bit, and the result differs from the all-default-types model of the same seed."""
    import refdata
    cfg, d, blob = refdata.case_data_dir(str(tmp_path / "qm"), "qwen_mixed", 12)
    man = open(os.path.join(d, "manifest.txt")).read()
    assert "blk.0.attn_v.weight 14 " in man and "blk.1.ffn_down_exps.weight 12 " in man
    eng = brrr.QwenEngine.open(d, blob)
    om = orc.QwenModel.open(d, blob)
    prompt = S.synth_prompt(12, 7, cfg.n_vocab)
    got, want = greedy(eng.run, prompt, 40), greedy(om.run, prompt, 40)
    assert got == want
    assert np.array_equal(bits(eng.logits()), bits(om.logits()))
    assert np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    plain = brrr.QwenEngine.synth(cfg, 12)
    greedy(plain.run, prompt, 40)
    assert not np.array_equal(bits(plain.hidden()), bits(eng.hidden()))
    eng.close(); plain.close(); om.close()


@pytest.mark.parametrize("ktypes", [
    {"blk.0.ffn_gate_exps.weight": 14, "blk.1.ffn_up_exps.weight": 14},                                     # gate 6 / up 4 bits, then 4 / 6
    {"blk.0.ffn_gate_exps.weight": 14, "blk.0.ffn_up_exps.weight": 14, "blk.1.attn_output.weight": 14,      # both 6
     "blk.1.attn_q.weight": 14, "blk.1.attn_k.weight": 14, "output.weight": 12},
])
def test_qwen_kquant_types_of_gate_up_and_head(brrr, orc, tmp_path, ktypes):
    """Every pair of types the gate/up kernel takes, Q6_K projections, a Q4_K head: steps, device-chained steps and token rows."""
    import refdata
    cfg, d, blob = refdata.case_data_dir(str(tmp_path / "qt"), "qwen_mixed", 12)
    refdata.retype_qwen(d, blob, cfg, 12, ktypes)
    eng = brrr.QwenEngine.open(d, blob)
    om = orc.QwenModel.open(d, blob)
    prompt = S.synth_prompt(12, 40, cfg.n_vocab)
    want = greedy(om.run, prompt, 20)
    for prefill in (False, True):
        if prefill:
            first = eng.prefill(prompt)
            got = [first] + [int(t) for t in eng.decode(first, len(prompt), 20)[:-1]]
        else:
            got = greedy(eng.run, prompt, 20)
        assert got == want
        assert np.array_equal(bits(eng.logits()), bits(om.logits())) and np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    assert (eng.spec_redos(), eng.wait_fallbacks()) == (0, 0)
    eng.close(); om.close()


@pytest.mark.parametrize("mode", ["qwen_sabotage", "qwen_mute", "qwen_memory"])
def test_qwen_failures_are_recovered(brrr, mode):
    """A step whose estimate missed an expert, and one whose exact router stays silent, run again without the estimate; a model without
    memory for the rows' scratch feeds prompts token by token: results are the oracle's and the counters name the steps (test-hook
    build of the library, tests/hooks_worker.py)."""
    import subprocess
    import sys
    from cpubrrr_b200 import build
    env = dict(os.environ, BRRR_LIBRARY=build.build_hooks())
    worker = os.path.join(os.path.dirname(GOLD), "hooks_worker.py")
    r = subprocess.run([sys.executable, worker, mode], env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "hooks_worker ok" in r.stdout, r.stdout[-2000:] + r.stderr[-4000:]


def test_qwen_open_errors(brrr, tmp_path):
    import ctypes as C
    L = brrr.lib()
    h = C.c_void_p()
    assert L.brrr_qwen_open(str(tmp_path).encode(), b"/nonexistent", 0, C.byref(h)) == 2
    bad = brrr.make_qwen_cfg(256, 1, 2, 1, 4, 2, 256, 100, head_dim=64)
    assert L.brrr_qwen_open_synth(C.byref(bad), 1, 0, C.byref(h)) == 1
    eng = brrr.QwenEngine.synth(brrr.make_qwen_cfg(256, 1, 2, 1, 4, 2, 256, 100), 1)
    out = C.c_uint32()
    assert L.brrr_qwen_forward(eng._h, 100, 0, 1, C.byref(out)) == 5
    assert L.brrr_qwen_forward(eng._h, 0, 4096, 1, C.byref(out)) == 5
    eng.close()


def test_full_size_qwen3_30b_a3b_parity_and_properties(brrr, orc):
    """Qwen3-30B-A3B architecture at full size (48 layers, 128 experts top-8, vocab 151936): a short
    prompt and greedy steps against the oracle, then size-independent properties (replay determinism,
    prefill idempotence) over a longer device-chained run."""
    cfg = brrr.qwen3_30b_a3b_cfg()
    eng = brrr.QwenEngine.synth(cfg, 3)
    om = orc.QwenModel.synth(ocfg_of(orc, cfg), 3)
    prompt = S.synth_prompt(3, 6, cfg.n_vocab)
    want = greedy(om.run, prompt, 10)
    got = greedy(eng.run, prompt, 10)
    assert got == want
    assert np.array_equal(bits(eng.logits()), bits(om.logits()))
    assert np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    om.close()
    first = eng.prefill(prompt)
    a = eng.decode(first, len(prompt), 140)
    assert [first] + [int(t) for t in a[:9]] == want
    assert eng.prefill(prompt) == first
    assert np.array_equal(a, eng.decode(first, len(prompt), 140))
    assert eng.bytes_per_step(100) > 1.5e9
    eng.close()


def test_full_size_qwen3_30b_a3b_64_token_prompt_128_steps(brrr, orc):
    """The qwen3moe configuration as stated: Qwen3-30B-A3B architecture at full size, a 64-token prompt,
    then 128 greedy decode steps: every token identical to the oracle's (device-chained decode loop),
    last logits and hidden state identical on their bit patterns."""
    cfg = brrr.qwen3_30b_a3b_cfg()
    eng = brrr.QwenEngine.synth(cfg, 3)
    om = orc.QwenModel.synth(ocfg_of(orc, cfg), 3)
    prompt = S.synth_prompt(3, 64, cfg.n_vocab)
    tok = 0
    for i, t in enumerate(prompt):
        tok = om.run(int(t), i, i == len(prompt) - 1)
    want, pos, gap = [tok], len(prompt), float("inf")
    for _ in range(128):
        tok = om.run(tok, pos, True); pos += 1
        want.append(tok)
        a = np.partition(om.logits(), -2)[-2:]
        gap = min(gap, float(a[1] - a[0]))
    first = eng.prefill(prompt)
    toks = eng.decode(first, len(prompt), 128)
    assert [first] + [int(t) for t in toks] == want
    assert np.array_equal(bits(eng.logits()), bits(om.logits()))
    assert np.array_equal(bits(eng.hidden()), bits(om.hidden()))
    print(f"Qwen3-30B-A3B 64+128: min top-1/top-2 gap {gap:.3e}, distinct tokens {len(set(want))}")
    eng.close(); om.close()
