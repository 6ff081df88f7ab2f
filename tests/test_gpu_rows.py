"""Feature rows off the 32-byte grid: an encoding with L levels writes, bit for bit, the first columns
of one with more levels whose rows are aligned (a level does not depend on the others).  Level counts
around the steps of 8 values, more levels than are staged at once, a single level; the batch is large
enough for the kernels that work in whole steps, and its last block is ragged."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
N = 80001


@pytest.mark.parametrize("ordered", [False, True])
@pytest.mark.parametrize("levels", [1, 2, 3, 5, 6, 7, 9, 34, 37])
@pytest.mark.parametrize("d,feat", [(2, 2), (3, 2), (5, 2), (7, 2), (3, 4)])
def test_shifted_rows_equal_aligned_rows(d, feat, levels, ordered):
    from permutohedral_encoding_b200 import _native as nat
    wide, cap = (levels + 3) // 4 * 4 + 4, 2 ** 10
    gen = torch.Generator(device=DEV).manual_seed(levels)
    sig = np.geomspace(1.0, 1e-2, wide)
    table = torch.randn((wide, cap, feat), device=DEV, generator=gen)
    shift = torch.randn((wide, d), device=DEV, generator=gen) * 10
    pos = torch.rand((N, d), device=DEV, generator=gen)
    dpg = torch.randn((N, d), device=DEV, generator=gen)
    window = torch.rand(wide, device=DEV, generator=gen)

    def run(count):
        fx = nat.EncodingFixedParams(d, cap, count, feat, sig[:count], shift[:count].contiguous(), False, 1.0)
        enc = nat.EncodingWrapper.create(d, feat, fx)
        inp = nat.EncodingInput(table[:count].contiguous(), pos, window[:count].contiguous(), True, True)
        inp.m_order = enc.order(inp) if ordered else None
        grad = torch.ones((N, feat * count), device=DEV)
        return enc.forward(inp), enc.double_backward_from_positions(inp, dpg, grad, need_lattice_grad=False)[1]

    for got, want in zip(run(levels), run(wide)):
        assert torch.equal(got, want[:, :feat * levels])
