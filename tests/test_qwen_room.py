"""The rule by which the qwen3moe step lets its down projection poll for the router's words (qw_router_room, kernels_qwen.cu): it may
only where the kernels that wait can never keep the router off every SM.  Host arithmetic of the test-hook build; no GPU."""
import ctypes as C
import itertools

import pytest

SMS, SM_SMEM, CTA_RESERVE = 148, 228 * 1024, 1024


@pytest.fixture(scope="module")
def room(brrr):
    from cpubrrr_b200 import build
    f = C.CDLL(build.build_hooks()).brrr_debug_qwen_room
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p]

    def rule(cfg, type_qkv, type_down):
        out = (C.c_uint64 * 6)()
        assert f(C.byref(cfg), type_qkv, type_down, out) == 0
        return [int(v) for v in out]
    return rule


def test_down_polls_at_the_qwen3_30b_a3b_shape(brrr, room):
    down, nxt, down_smem, next_smem, router_smem, ok = room(brrr.qwen3_30b_a3b_cfg(), 12, 14)
    assert ok and down == 137 and nxt == 139                       # 2048 rows of 15 per CTA, 5120 of 37


def test_down_waits_where_its_grid_fills_the_chip(brrr, room):
    """293 CTAs of the down projection, two per SM, would all poll while no SM takes a router CTA of 133 KB."""
    cfg = brrr.make_qwen_cfg(4096, 1, 32, 4, 128, 8, 1024, 1000)
    down, nxt, down_smem, next_smem, router_smem, ok = room(cfg, 12, 14)
    assert down == 293 and 2 * (down_smem + CTA_RESERVE) < SM_SMEM and not ok


def test_no_shape_polls_without_room(brrr, room):
    polls = waits = 0
    for d, ff, ne, topk, heads, types in itertools.product((256, 768, 1536, 2048, 2304, 2816, 4096), (256, 768, 1024), (8, 32, 33, 128, 256), (1, 4, 8),
                                                           ((2, 1), (32, 4), (32, 32)), ((12, 12), (12, 14), (14, 14))):
        if topk > ne:
            continue
        down, nxt, down_smem, next_smem, router_smem, ok = room(brrr.make_qwen_cfg(d, 1, heads[0], heads[1], ne, topk, ff, 1000), *types)
        # CTAs of the waiting kernels an SM must hold before it refuses a router CTA: by registers two (launch bounds give each half an SM)
        largest = max(down_smem, next_smem) + CTA_RESERVE
        refuses = 1 if largest + router_smem + CTA_RESERVE > SM_SMEM else 2
        if ok:
            polls += 1
            assert down + nxt < refuses * SMS, (d, ff, ne, topk, heads, types)
        else:
            waits += 1
    assert polls > 100 and waits > 100
