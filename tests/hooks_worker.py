"""Child process of the GPU tests that need the test-hook build of the library (libbrrr_hooks.so,
-DBRRR_TEST_HOOKS): the parent sets BRRR_LIBRARY to it, so this process loads it instead of the
default build, which contains no hook.  No GPU fault is provoked: a missed speculation is a
flagged step, a silent router is a bounded wait that runs out and is reported.

    python tests/hooks_worker.py sabotage | mute | memory | exponents | qwen_sabotage | qwen_mute | qwen_memory
"""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))


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


def qwen(mode):
    """The same two failures in the qwen3moe engine: a missed expert and a silent router, through host-driven steps
    (brrr_qwen_forward) and through the device-chained run (brrr_qwen_decode_wait)."""
    import cpubrrr_b200 as B
    from cpubrrr_b200 import synth as S
    from oracle import oracle as O
    bits = lambda a: np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
    shape = dict(n_embd=512, n_layer=3, n_head=8, n_head_kv=2, n_expert=40, n_expert_used=8, n_ff_exp=768, n_vocab=515)
    cfg = B.make_qwen_cfg(**shape)
    om = O.QwenModel.synth(O.make_qcfg(d=512, nh=8, nkv=2, hd=128, nl=3, ne=40, topk=8, ff=768, nvocab=515), 17)
    prompt = S.synth_prompt(17, 9, cfg.n_vocab)
    want = greedy(om.run, prompt, 40)          # positions 0 .. 48

    def check(eng):
        assert np.array_equal(bits(eng.logits()), bits(om.logits())) and np.array_equal(bits(eng.hidden()), bits(om.hidden()))

    def hooked(var, value="1"):
        os.environ[var] = value
        eng = B.QwenEngine.synth(cfg, 17)
        del os.environ[var]
        return eng

    def chained(eng):
        first = eng.prefill(prompt)            # token rows: no speculation in it
        toks = eng.decode(first, len(prompt), 40)
        assert [first] + [int(t) for t in toks[:-1]] == want
        check(eng)

    if mode == "qwen_memory":
        # the rows' scratch does not fit: prompts go token by token
        import ctypes as C
        taken = B.lib().brrr_debug_qwen_taken
        taken.restype, taken.argtypes = C.c_uint64, [C.c_void_p]
        eng = B.QwenEngine.synth(cfg, 17)
        assert eng.uses_rows
        chained(eng)
        most = taken(eng._h)
        eng.close()
        eng = hooked("BRRR_TEST_MEM_BYTES", str(most - 1))
        assert not eng.uses_rows
        chained(eng)
    elif mode == "qwen_sabotage":
        # the estimate is spoiled where the position is a multiple of three: exactly those steps run twice
        eng = hooked("BRRR_SPEC_SABOTAGE")
        assert greedy(eng.run, prompt, 40) == want
        check(eng)
        assert (eng.spec_redos(), eng.wait_fallbacks()) == (17, 0)         # 0, 3 .. 48
        chained(eng)
        assert (eng.spec_redos(), eng.wait_fallbacks()) == (17 + 14, 0)    # 9, 12 .. 48
        clean = B.QwenEngine.synth(cfg, 17)
        assert greedy(clean.run, prompt, 40) == want
        check(clean)
        chained(clean)
        assert (clean.spec_redos(), clean.wait_fallbacks()) == (0, 0)
        clean.close()
    else:
        # the router never publishes: the first combine's wait (about a second) runs out, the step runs again with the routing
        # in the chain, and the model does without speculation from there on
        eng = hooked("BRRR_ROUTER_MUTE")
        assert greedy(eng.run, prompt, 40) == want
        check(eng)
        chained(eng)
        assert (eng.spec_redos(), eng.wait_fallbacks()) == (1, 1)
        eng.close()
        eng = hooked("BRRR_ROUTER_MUTE")       # the same, met inside a device-chained run first
        chained(eng)
        assert (eng.spec_redos(), eng.wait_fallbacks()) == (1, 1)
        assert greedy(eng.run, prompt, 40) == want
        assert (eng.spec_redos(), eng.wait_fallbacks()) == (1, 1)
    eng.close()
    om.close()


def memory(cfg, prompt):
    """Copies and workspaces that do not fit: what goes without them, and that nothing changes but the path."""
    import ctypes as C
    import cpubrrr_b200 as B
    from cpubrrr_b200 import synth as S
    bits = lambda a: np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
    taken = B.lib().brrr_debug_taken
    taken.restype, taken.argtypes = C.c_uint64, [C.c_void_p]
    limit = lambda n: os.environ.__setitem__("BRRR_TEST_MEM_BYTES", str(n))
    free = lambda: os.environ.pop("BRRR_TEST_MEM_BYTES", None)
    PROJ, HEAD, KEYS = 1, 2, 4
    long = S.synth_prompt(5, 70, 500)

    def use(eng, nseq):
        """A prompt, a batch whose sequences have prompts of their own, a step of as many rows."""
        out = [eng.prefill(long), bits(eng.logits())]
        for s in range(nseq):
            eng.batch_prefill(s, long[:20 + s])
        toks, lg = eng.batch_step(list(long[:nseq]), [20 + s for s in range(nseq)], list(range(nseq)), logits=True)
        return out + [toks, bits(lg)]

    def same(a, b):
        return all(np.array_equal(x, y) for x, y in zip(a, b))

    n = 16                                                  # rows enough for the tensor-core projections and head
    eng = B.Engine.synth(cfg, 17)
    eng.batch_open(n)
    want = use(eng, n)
    assert eng.row_paths == PROJ | HEAD | KEYS and eng.uses_tensor_experts
    eng.close()
    # neither copy fits beside the rest (2 GB are kept free): integer units throughout
    limit(1 << 30)
    eng = B.Engine.synth(cfg, 17)
    eng.batch_open(n)
    assert eng.row_paths == KEYS and not eng.uses_tensor_experts
    assert same(use(eng, n), want) and eng.row_paths == KEYS
    eng.close()
    # the workspace of the prompt rows does not fit: the other attention kernel
    free()
    eng = B.Engine.synth(cfg, 17)
    eng.batch_open(n)
    limit(taken(eng._h) + 4096)
    assert same(use(eng, n), want) and eng.row_paths == PROJ | HEAD
    eng.close()
    # the caches fit only where the projections' copies were, after a prompt has run on those
    free()
    eng = B.Engine.synth(cfg, 17)
    eng.prefill(long)
    at = taken(eng._h)
    limit(at + (64 << 20))
    assert B.lib().brrr_batch_open(eng._h, 256) == 4        # 256 caches fit neither way: BRRR_ERR_NOMEM, and the model as it was
    assert taken(eng._h) == at and eng.row_paths == PROJ | KEYS
    assert eng.prefill(long) == want[0] and np.array_equal(bits(eng.logits()), want[1])
    need = 2 * cfg.n_layer * cfg.n_head_kv * 4096 * 64 * 4 * n + 512 * (cfg.n_vocab + 1) * 4
    limit(at + need - 4096)
    eng.batch_open(n)
    assert eng.row_paths == KEYS and taken(eng._h) < at + need
    assert same(use(eng, n), want)
    eng.close()
    free()


def exponents():
    """The form each layer's expert matrices run in (brrr_debug_wide: bit 0 = gate | up, bit 1 = down)."""
    import ctypes as C
    import tempfile
    import cpubrrr_b200 as B
    import refdata
    from test_gpu_mxt import EXPONENTS
    wide_of = B.lib().brrr_debug_wide
    wide_of.restype, wide_of.argtypes = C.c_int, [C.c_void_p, C.c_int]
    for exps, wide in EXPONENTS:
        for kind, bit in (("gate", 1), ("up", 1), ("down", 2)):
            with tempfile.TemporaryDirectory() as tmp:
                _, d, blob = refdata.case_data_dir(tmp, "gptoss_d128", 12)
                refdata.set_exponents(d, blob, f"blk.1.ffn_{kind}_exps.weight", exps)
                eng = B.Engine.open(d, blob)
                assert (wide_of(eng._h, 0), wide_of(eng._h, 1)) == (0, bit if wide else 0), (exps, kind)
                eng.close()


def main(mode):
    assert os.environ.get("BRRR_LIBRARY", "").endswith("libbrrr_hooks.so")
    if mode.startswith("qwen"):
        qwen(mode)
        print("hooks_worker ok:", mode)
        return
    if mode == "exponents":
        exponents()
        print("hooks_worker ok:", mode)
        return
    import cpubrrr_b200 as B
    from cpubrrr_b200 import synth as S
    from oracle import oracle as O
    bits = lambda a: np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)
    cfg = B.make_cfg(128, 2, 4, 2, 8, 4, 512, sliding_window=8)
    om = O.Model.synth(O.make_cfg(d=128, nh=4, nkv=2, hd=64, nl=2, ne=8, topk=4, nvocab=512, swa=8), 17)
    prompt = S.synth_prompt(17, 9, 500)
    want = greedy(om.run, prompt, 40)
    if mode == "sabotage":
        # the estimate is spoiled on every third position: those steps are flagged and run again
        os.environ["BRRR_SPEC_SABOTAGE"] = "1"
        eng = B.Engine.synth(cfg, 17)
        del os.environ["BRRR_SPEC_SABOTAGE"]
        assert greedy(eng.run, prompt, 40) == want                  # host-driven steps
        assert np.array_equal(bits(eng.logits()), bits(om.logits()))
        first = eng.prefill(prompt)
        toks = eng.decode(first, len(prompt), 40)                   # device-chained run with redos inside
        assert [first] + [int(t) for t in toks[:-1]] == want
        assert eng.spec_redos() > 10 and eng.wait_fallbacks() == 0
        clean = B.Engine.synth(cfg, 17)                             # without the hook the estimate practically never misses
        assert greedy(clean.run, prompt, 40) == want and clean.spec_redos() == 0
        eng.close(); clean.close()
    elif mode == "mute":
        # the exact router never publishes: the fold's bounded wait (about a second) runs out in the
        # first speculative step; the host re-runs that step with the plain graph, stops speculating
        # on this model, and every result is still the oracle's
        os.environ["BRRR_ROUTER_MUTE"] = "1"
        eng = B.Engine.synth(cfg, 17)
        del os.environ["BRRR_ROUTER_MUTE"]
        assert greedy(eng.run, prompt, 40) == want
        assert np.array_equal(bits(eng.logits()), bits(om.logits()))
        assert eng.wait_fallbacks() == 1
        first = eng.prefill(prompt)
        toks = eng.decode(first, len(prompt), 40)
        assert [first] + [int(t) for t in toks[:-1]] == want and eng.wait_fallbacks() == 1
        eng.close()
        # the same through the device-chained loop first (the recovery inside brrr_decode_wait)
        os.environ["BRRR_ROUTER_MUTE"] = "1"
        eng = B.Engine.synth(cfg, 17)
        del os.environ["BRRR_ROUTER_MUTE"]
        tok = 0
        for i, t in enumerate(prompt):
            tok = om.run(int(t), i, True)       # (oracle state only)
        first = eng.prefill(prompt)
        assert first == want[0]
        toks = eng.decode(first, len(prompt), 12)
        assert [first] + [int(t) for t in toks[:-1]] == want[:12]
        assert eng.wait_fallbacks() == 1
        eng.close()
    elif mode == "memory":
        memory(cfg, prompt)
    else:
        raise SystemExit("mode?")
    print("hooks_worker ok:", mode)


if __name__ == "__main__":
    main(sys.argv[1])
