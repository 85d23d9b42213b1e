"""Attention of prompt rows (attn_rows_kernel: 32 (head, row) pairs per CTA share tiles of 64 keys) against the oracle, which runs token by token: hidden
state and logits of a prompt's last token after four layers, so that every row's output of a layer reaches it through the caches of the
next.  Lengths and offsets around the tiles, all head groupings, scores spread over the exponential's whole range, sinks at its ends."""
import numpy as np
import pytest

from conftest import bits
from cpubrrr_b200 import synth as S
from test_gpu_model import ocfg_of
import refdata

pytestmark = pytest.mark.gpu
LENGTHS = [2, 3, 31, 32, 33, 63, 64, 65, 66, 70, 71, 127, 128, 129, 135, 191, 193, 260]


def _scale_bf16(raw, k):
    """bf16 values x 2^k"""
    w = (np.frombuffer(raw, np.uint16).astype(np.uint32) << 16).view(np.float32) * np.float32(2.0 ** k)
    return (w.view(np.uint32) >> 16).astype(np.uint16).tobytes()


def _edit(k, sinks):
    def edit(name, raw):
        if name.endswith("attn_q.weight"):
            return _scale_bf16(raw, k)
        if name.endswith("attn_q.bias"):
            return (np.frombuffer(raw, np.float32) * np.float32(2.0 ** k)).tobytes()
        if name.endswith("attn_sinks") and sinks is not None:
            return np.resize(np.float32(sinks), len(raw) // 4).tobytes()
        return raw
    return edit


@pytest.mark.parametrize("nh,nkv,k,sinks", [
    (4, 2, 0, None), (4, 4, 0, None), (8, 1, 0, None), (32, 1, 0, None),
    # q x 256 and x 1024: of the first layer's exponents 6 and 91 % lie below -104, 10 and 2 % have a subnormal result
    (4, 2, 8, None), (4, 2, 10, None), (8, 1, 10, None),
    (4, 2, 8, [-np.inf, -300.0, 300.0, 60.0]),
])
def test_prompt_rows_equal_the_oracle(brrr, orc, tmp_path, nh, nkv, k, sinks):
    cfg = brrr.make_cfg(128, 4, nh, nkv, 8, 4, 512, sliding_window=70)
    d, blob = refdata.plain_data_dir(str(tmp_path), cfg, 21, _edit(k, sinks))
    om = orc.Model.open(d, blob)
    toks = [int(t) for t in S.synth_prompt(21, max(LENGTHS), 500)]
    want = {}
    for i, t in enumerate(toks):
        tok = om.run(t, i, i + 1 in LENGTHS)
        if i + 1 in LENGTHS:
            want[i + 1] = tok, bits(om.hidden()), bits(om.logits())
    eng = brrr.Engine.open(d, blob)

    def check(n, first):
        assert first == want[n][0] and np.array_equal(bits(eng.hidden()), want[n][1]) and np.array_equal(bits(eng.logits()), want[n][2]), n

    for n in LENGTHS:
        check(n, eng.prefill(toks[:n]))
    assert eng.row_paths & 4                      # BRRR_ROWS_SHARED_KEYS
    # a prompt in parts: rows whose windows and caches start inside a tile
    for cuts in ([33, 66, 193], [5, 71, 135, 260], [128, 191], [64, 128, 260]):
        at = 0
        for n in cuts:
            first = eng.run_tile(toks[at:n], at, n in want)
            if n in want:
                check(n, first)
            at = n
    eng.close()


@pytest.mark.parametrize("tensor,value", [("attn_sinks", np.inf), ("attn_sinks", np.nan), ("attn_q.bias", np.nan), ("attn_k.bias", np.inf), ("attn_v.bias", -np.inf)])
def test_prompt_rows_without_numbers_equal_tokens(brrr, tmp_path, tensor, value):
    """One head's sink, or one element of a head's bias, infinite or NaN: prompt rows give the bits of token after token."""
    def edit(name, raw):
        if name != f"blk.1.{tensor}":
            return raw
        v = np.frombuffer(raw, np.float32).copy()
        v[1] = value
        return v.tobytes()
    cfg = brrr.make_cfg(128, 3, 4, 2, 8, 4, 512, sliding_window=70)
    d, blob = refdata.plain_data_dir(str(tmp_path), cfg, 22, edit)
    eng = brrr.Engine.open(d, blob)
    toks = [int(t) for t in S.synth_prompt(22, 131, 500)]
    for n in (64, 65, 131):
        out = []
        for tiles in (False, True):
            eng.set_tile_prefill(tiles)
            out.append((eng.prefill(toks[:n]), bits(eng.hidden()), bits(eng.logits())))
        assert out[0][0] == out[1][0] and np.array_equal(out[0][1], out[1][1]) and np.array_equal(out[0][2], out[1][2])
    eng.close()
