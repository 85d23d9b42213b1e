"""The tensor-core row kernels at the sizes where their dispatch changes or a launch runs more CTAs than fit at once:
tokens per CTA 8 / 16 / 32, ragged last chunks, several chunks per matrix, 2 .. 64 block pairs."""
import ctypes as C

import numpy as np
import pytest

from conftest import bits, to_dev
from cpubrrr_b200 import synth as S

pytestmark = pytest.mark.gpu


def P(t):
    return C.c_void_p(t.data_ptr())


@pytest.mark.parametrize("rows,cols,ntok", [(5120, 2880, 30), (5120, 2880, 49), (2880, 4096, 30), (2880, 4096, 70), (20000, 2880, 17), (130, 192, 8), (5120, 448, 512)])
def test_q8_rows_tensor_cores_equal_integer_units(brrr, dev, rows, cols, ntok):
    """Both engines run the same chains (the integer one is compared with the oracle elsewhere): equal bits."""
    import torch
    L = brrr.lib()
    w = torch.empty(rows * cols, dtype=torch.int16, device=dev)
    assert L.brrr_synth_tensor(rows + ntok, 1, S.T["WQ"], 30, rows * cols, P(w), None) == 0
    h = C.c_void_p()
    assert L.brrr_q8mat_from_bf16(P(w), rows, cols, C.byref(h), None) == 0
    g = torch.Generator(device=dev); g.manual_seed(ntok)
    x = torch.randn((ntok, cols), device=dev, generator=g)
    q = torch.empty((ntok, cols), dtype=torch.int8, device=dev); s = torch.empty((ntok, cols // 32), device=dev)
    assert L.brrr_quant_q8(P(x), x.numel(), P(q), P(s), None) == 0
    ys = []
    for tensor_cores in (0, 1, 1):
        y = torch.full((ntok, rows + 1), 5.0, device=dev)
        assert L.brrr_q8_matmul_rows(h, P(q), P(s), ntok, P(y), rows + 1, tensor_cores, None) == 0
        ys.append(y)
    torch.cuda.synchronize()
    assert np.array_equal(bits(ys[0].cpu().numpy()), bits(ys[1].cpu().numpy())) and torch.equal(ys[1], ys[2])
    L.brrr_q8mat_free(h)


def test_q8_operand_units_are_made_when_wanted(brrr, dev):
    """A matrix that is only multiplied by vectors takes its Q8 bytes; the tensor-core product adds its copy once, and none of its
    own where the stream is being captured."""
    import torch
    L = brrr.lib()
    rows, cols, ntok = 24576, 4096, 9
    q8 = rows * cols * 9 // 8
    w = torch.empty(rows * cols, dtype=torch.int16, device=dev)
    assert L.brrr_synth_tensor(7, 1, S.T["WQ"], 30, rows * cols, P(w), None) == 0
    x = torch.randn((ntok, cols), device=dev)
    q = torch.empty((ntok, cols), dtype=torch.int8, device=dev); s = torch.empty((ntok, cols // 32), device=dev)
    assert L.brrr_quant_q8(P(x), x.numel(), P(q), P(s), None) == 0
    ys = [torch.zeros((ntok, rows), device=dev) for _ in range(4)]

    def taken():
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0]

    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    h = C.c_void_p()
    assert L.brrr_q8mat_from_bf16(P(w), rows, cols, C.byref(h), None) == 0
    assert L.brrr_q8_matmul_rows(h, P(q), P(s), ntok, P(ys[0]), rows, 0, None) == 0
    assert taken() < q8 + (8 << 20)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        assert L.brrr_q8_matmul_rows(h, P(q), P(s), ntok, P(ys[1]), rows, 1, C.c_void_p(side.cuda_stream)) == 0
    graph.replay()
    for y in ys[2:]:
        assert L.brrr_q8_matmul_rows(h, P(q), P(s), ntok, P(y), rows, 1, None) == 0
    torch.cuda.synchronize()
    for y in ys[1:]:
        assert torch.equal(y, ys[0])
    del graph
    L.brrr_q8mat_free(h)


@pytest.mark.parametrize("rows,blocks,ntok", [(2880, 90, 9), (2880, 90, 30), (2880, 90, 333), (272, 128, 33), (4096, 4, 8)])
def test_mx_tile_equals_one_token_kernel(brrr, dev, rows, blocks, ntok):
    import torch
    L = brrr.lib()
    raw = to_dev(S.synth_mxfp4(rows + ntok, 2, S.T["UP"], rows * blocks), dev)
    h = C.c_void_p()
    assert L.brrr_mxmat_from_gguf(P(raw), rows, blocks, C.byref(h), None) == 0
    g = torch.Generator(device=dev); g.manual_seed(ntok)
    x = torch.randn((ntok, blocks * 32), device=dev, generator=g)
    x[0] *= 1e4                                       # one row of large scales beside ordinary ones
    q = torch.empty((ntok, blocks * 32), dtype=torch.int8, device=dev); s = torch.empty((ntok, blocks), device=dev)
    assert L.brrr_quant_q8(P(x), x.numel(), P(q), P(s), None) == 0
    y = torch.empty((ntok, rows), device=dev); want = torch.empty((ntok, rows), device=dev)
    assert L.brrr_mx_matmul_tile(h, 0, rows, P(q), P(s), ntok, P(y), rows, None) == 0
    for t in range(ntok):
        assert L.brrr_mx_matvec(h, 0, rows, P(q[t]), P(s[t]), P(want[t]), None, None) == 0
    torch.cuda.synchronize()
    assert np.array_equal(bits(y.cpu().numpy()), bits(want.cpu().numpy()))
    L.brrr_mxmat_free(h)
