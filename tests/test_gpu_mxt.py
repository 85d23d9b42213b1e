"""Expert matvecs on the tensor cores in native fp4 (tcgen05.mma kind::mxf4.block_scale, kernels_mxt.cu):
the MoE FFN step through them equals the oracle bit for bit, at the gpt-oss-20b layer shape and at
ragged small shapes (partial last tile of down, partial last ring stage, one block pair), and the
decode step that uses them emits the same tokens and logits as the integer-unit kernels."""
import ctypes as C

import numpy as np
import pytest

from conftest import bits, to_dev
from cpubrrr_b200 import synth as S
from test_gpu_model import _run_with_hooks, greedy, ocfg_of

pytestmark = pytest.mark.gpu


def _ffn_oracle(orc, om, ocfg, xn, il=0):
    Lo = orc.lib()
    vp = lambda a: a.ctypes.data_as(C.c_void_p)
    d, k = ocfg.d, ocfg.topk
    y = np.zeros(d, np.float32)
    top = np.zeros(k, np.int32); wts = np.zeros(k, np.float32)
    Lo.orc_moe_ffn_step(C.byref(ocfg), vp(xn), Lo.orc_layer_f32(om.h, il, S.T["ROUTER_W"]), Lo.orc_layer_f32(om.h, il, S.T["ROUTER_B"]),
                        Lo.orc_layer_mx(om.h, il, 0), Lo.orc_layer_mx(om.h, il, 1), Lo.orc_layer_mx(om.h, il, 2),
                        Lo.orc_layer_f32(om.h, il, S.T["GATE_B"]), Lo.orc_layer_f32(om.h, il, S.T["UP_B"]), Lo.orc_layer_f32(om.h, il, S.T["DOWN_B"]),
                        vp(y), vp(top), vp(wts))
    return y, top, wts


@pytest.mark.parametrize("shape", [
    dict(n_embd=2880, n_layer=1, n_head=64, n_head_kv=8, n_expert=32, n_expert_used=4, n_vocab=256),     # gpt-oss-20b layer
    dict(n_embd=64, n_layer=1, n_head=2, n_head_kv=1, n_expert=4, n_expert_used=2, n_vocab=256),         # one block pair, half a down tile
    dict(n_embd=320, n_layer=1, n_head=10, n_head_kv=2, n_expert=8, n_expert_used=8, n_vocab=256),       # 5 pairs: ragged stage, ragged down tile
    dict(n_embd=1024, n_layer=1, n_head=16, n_head_kv=4, n_expert=6, n_expert_used=1, n_vocab=256),      # top-1, 16 pairs: ring wraps
])
def test_moe_ffn_step_tensor_cores_bit_exact(brrr, orc, dev, shape):
    import torch
    cfg = brrr.make_cfg(**shape)
    d, k = cfg.n_embd, cfg.n_expert_used
    eng = brrr.Engine.synth(cfg, 5)
    assert eng.uses_tensor_experts
    ocfg = ocfg_of(orc, cfg)
    om = orc.Model.synth(ocfg, 5)
    for trial in range(3):
        x = S.synth_input(10 + trial, d)
        xn = orc.rmsnorm(x, np.ones(d, np.float32), 1e-5) * np.float32(1.0 + 3.0 * trial)
        want_y, want_top, want_w = _ffn_oracle(orc, om, ocfg, xn)
        dy = torch.zeros(d, dtype=torch.float32, device=dev)
        dt = torch.zeros(k, dtype=torch.int32, device=dev); dw = torch.zeros(k, dtype=torch.float32, device=dev)
        dxn = to_dev(xn, dev)
        torch.cuda.synchronize()
        P = lambda t: C.c_void_p(t.data_ptr())
        eng.moe_ffn_step_tc(0, P(dxn), P(dy), P(dt), P(dw))
        assert np.array_equal(dt.cpu().numpy(), want_top)
        assert np.array_equal(bits(dw.cpu().numpy()), bits(want_w))
        assert np.array_equal(bits(dy.cpu().numpy()), bits(want_y))
        # and the integer-unit kernels give the same bits
        dy2 = torch.zeros(d, dtype=torch.float32, device=dev)
        eng.moe_ffn_step(0, P(dxn), P(dy2), P(dt), P(dw))
        assert np.array_equal(bits(dy2.cpu().numpy()), bits(want_y))
    # the fold adds onto what the residual already holds, and the arrival counters are back at zero
    dy = to_dev(x, dev)
    eng.moe_ffn_step_tc(0, P(dxn), P(dy), None, None)
    eng.moe_ffn_step_tc(0, P(dxn), P(dy), None, None)
    ref = to_dev(x, dev)
    eng.moe_ffn_step(0, P(dxn), P(ref), None, None)
    eng.moe_ffn_step(0, P(dxn), P(ref), None, None)
    assert np.array_equal(bits(dy.cpu().numpy()), bits(ref.cpu().numpy()))
    eng.close()


def test_worst_case_magnitudes_stay_exact(brrr, orc, dev):
    """Activation bytes at +-127 in every position (the largest lane sums; digits 2, 0, -1 and -2, 0, 1), and at -36 and 92 in all but one of a
    block's (digits 0, -4, -4 and 2, -4, -4: the largest sums of a digit plane), against all weight codes."""
    import torch
    cfg = brrr.make_cfg(n_embd=256, n_layer=1, n_head=4, n_head_kv=2, n_expert=4, n_expert_used=4, n_vocab=256)
    eng = brrr.Engine.synth(cfg, 9)
    ocfg = ocfg_of(orc, cfg)
    om = orc.Model.synth(ocfg, 9)
    rng = np.random.default_rng(3)
    P = lambda t: C.c_void_p(t.data_ptr())
    for trial in range(6):
        sign = rng.integers(0, 2, 256) * 2 - 1
        xn = (sign * (1.0 + 0.001 * (trial == 3) * rng.random(256))).astype(np.float32)     # every |x| equal: every byte +-127
        if trial >= 4:
            xn = np.full(256, (-36, 92)[trial - 4], np.float32)
            xn[rng.integers(0, 32, 8) + 32 * np.arange(8)] = 127.0
        want_y, want_top, _ = _ffn_oracle(orc, om, ocfg, xn)
        dy = torch.zeros(256, dtype=torch.float32, device=dev)
        eng.moe_ffn_step_tc(0, P(to_dev(xn, dev)), P(dy), None, None)
        assert np.array_equal(bits(dy.cpu().numpy()), bits(want_y))
    eng.close()


def test_decode_same_with_and_without_tensor_experts(brrr, orc, monkeypatch):
    cfg = brrr.make_cfg(n_embd=256, n_layer=3, n_head=8, n_head_kv=4, n_expert=16, n_expert_used=4, n_vocab=1024)
    prompt = S.synth_prompt(4, 9, cfg.n_vocab)
    eng = brrr.Engine.synth(cfg, 4)
    assert eng.uses_tensor_experts
    got = greedy(eng.run, prompt, 64)
    lg = eng.logits()
    eng.close()
    monkeypatch.setenv("BRRR_NOMXT", "1")
    old = brrr.Engine.synth(cfg, 4)
    assert not old.uses_tensor_experts
    assert greedy(old.run, prompt, 64) == got
    assert np.array_equal(bits(old.logits()), bits(lg))
    old.close()
    om = orc.Model.synth(ocfg_of(orc, cfg), 4)
    assert greedy(om.run, prompt, 64) == got
    assert np.array_equal(bits(om.logits()), bits(lg))


EXPONENTS = [
    ([49, 134, 120, 60], False),         # the ends of the range whose scaled products are exact
    ([(0, 0), (48, 0), 49], False),      # zero blocks below it
    ([48], True),                        # values other than zero below it, any block above it: scales in the epilogue
    ([135], True),
    ([0, 1, 2, 190], True),
    ([(255, 0)], True),
]


@pytest.mark.parametrize("kind", ["gate", "up", "down"])
@pytest.mark.parametrize("exponents,wide", EXPONENTS)
def test_block_exponents_of_any_size(brrr, orc, dev, tmp_path, exponents, wide, kind):
    """Blocks with the given exponents (pairs: exponent of a block of zeros) among the synthetic ones of one layer's matrix: the experts stay on the
    tensor cores and the oracle's tokens and logits come out, and the stage call answers, with activations from the smallest scale to huge ones."""
    import torch
    import refdata
    cfg, d, blob = refdata.case_data_dir(str(tmp_path), "gptoss_d128", 12)
    refdata.set_exponents(d, blob, f"blk.1.ffn_{kind}_exps.weight", exponents)
    eng, om = brrr.Engine.open(d, blob), orc.Model.open(d, blob)
    assert eng.uses_tensor_experts
    prompt = S.synth_prompt(12, 7, 500)
    assert greedy(eng.run, prompt, 24) == greedy(om.run, prompt, 24)
    assert np.array_equal(bits(eng.logits()), bits(om.logits()))
    # the same prompt as token rows
    assert eng.run_tile([int(t) for t in prompt], 0, True) == greedy(om.run, prompt, 1)[0]
    P = lambda t: C.c_void_p(t.data_ptr())
    for scale in (1e-30, 1.0, 2.0 ** 66):
        xn = S.synth_input(7, cfg.n_embd) * np.float32(scale)
        dxn, y = to_dev(xn, dev), [torch.zeros(cfg.n_embd, dtype=torch.float32, device=dev) for _ in range(2)]
        eng.moe_ffn_step_tc(1, P(dxn), P(y[0]), None, None)
        eng.moe_ffn_step(1, P(dxn), P(y[1]), None, None)
        tc, iu = (bits(t.cpu().numpy()) for t in y)
        assert np.array_equal(tc, iu)
        largest = max(e[0] if isinstance(e, tuple) else e for e in exponents)
        if scale > 1 and largest >= 190:         # the block's scale, 2^62 x 2^66 and more, overflows: sums that are no numbers (inf - inf, 0 x inf)
            continue
        assert np.array_equal(tc, bits(_ffn_oracle(orc, om, ocfg_of(orc, cfg), xn, 1)[0]))
    eng.close()


def test_block_exponents_choose_the_form(brrr):
    """Which form the matrices of a layer run in: by the layer's own blocks, gate | up and down each by themselves."""
    _run_with_hooks(brrr, "exponents")


# gate and up exponent, down exponent, whether the matrices run in the wide form, activation scale (gate of the order of one, or h below
# the quantiser's smallest block maximum of 1e-12)
WHOLE = [
    (49, 49, False, 2.0 ** 70),
    (134, 134, False, 2.0 ** -14),
    (123, 49, False, 2.0 ** -43),        # activation and h both at the smallest block scale, 1e-12 / 127
    (49, 134, False, 2.0 ** 70),
    (48, 48, True, 2.0 ** 71),
    (135, 135, True, 2.0 ** -15),
    (1, 0, True, 2.0 ** 118),            # block scales that are subnormal numbers
    (190, 190, True, 2.0 ** -43),
]


@pytest.mark.parametrize("gate_up,down,wide,scale", WHOLE)
def test_matrices_of_one_block_exponent(brrr, orc, dev, tmp_path, gate_up, down, wide, scale):
    """Every block of a matrix at one end of a form's range, no bias, a residual of zero: nothing absorbs or clamps a product that is not exact.  Five
    block pairs (a whole group of scales and half of one), a ragged tile of down."""
    import torch
    import refdata
    cfg = brrr.make_cfg(320, 1, 4, 2, 8, 4, 256)

    def edit(name, raw):
        if name.endswith("_exps.bias"):
            return bytes(len(raw))
        if not name.endswith("_exps.weight"):
            return raw
        blocks = np.frombuffer(raw, np.uint8).reshape(-1, 17).copy()
        blocks[:, 0] = down if "down" in name else gate_up
        return blocks.tobytes()

    d, blob = refdata.plain_data_dir(str(tmp_path), cfg, 21, edit)
    eng, om = brrr.Engine.open(d, blob), orc.Model.open(d, blob)
    assert eng.uses_tensor_experts
    P = lambda t: C.c_void_p(t.data_ptr())
    for seed in range(3):
        xn = S.synth_input(40 + seed, cfg.n_embd) * np.float32(scale)
        want = _ffn_oracle(orc, om, ocfg_of(orc, cfg), xn)[0]
        assert np.isfinite(want).all() and np.count_nonzero(want) > 300 and len(np.unique(np.abs(want))) > 300      # (subnormal sums coincide at times)
        dxn, y = to_dev(xn, dev), [torch.zeros(cfg.n_embd, dtype=torch.float32, device=dev) for _ in range(2)]
        eng.moe_ffn_step_tc(0, P(dxn), P(y[0]), None, None)
        eng.moe_ffn_step(0, P(dxn), P(y[1]), None, None)
        for got in y:
            assert np.array_equal(bits(got.cpu().numpy()), bits(want))
    eng.close()
