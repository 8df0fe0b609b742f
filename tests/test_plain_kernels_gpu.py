"""The plain kernels at the edges of their tiles: every variant a size picks, against 64-bit, and rows that do not
depend on the batch they come in."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_inference_lab_b200.kernels import ops as module
    return module


# Rows on both sides of every choice (few rows by 2, 4, 8, 16, 32; tiles of 16 and of 32), columns that end inside a
# tile, k's that end inside a load, a part and a stage, rows that are whole 16-byte units or not.
@pytest.mark.parametrize("gated", [False, True])
@pytest.mark.parametrize("N,K", [(5, 3), (33, 20), (70, 65), (130, 132), (900, 72), (257, 300)])
def test_product_rows_do_not_depend_on_their_batch(N, K, gated):
    g = torch.Generator(device=DEV).manual_seed(N + K)
    x = torch.randn(530, K, device=DEV, generator=g)
    w = torch.randn(2 * N if gated else N, K, device=DEV, generator=g)
    full = ops().gemm_plain(x, w, gated=gated)
    want = x.double() @ w.double().T
    if gated:
        want = torch.nn.functional.silu(want[:, :N]) * want[:, N:]
    # every rounding is at most 2^-24 of a partial sum, of which there are K / 8 in a chain, below |x| |w|; the gate's
    # slope is at most 1.1 and its factors |x| |w|
    size = x.abs().double() @ w.abs().double().T
    size = 2.2 * size[:, :N] * size[:, N:] if gated else size
    assert bool(((full.double() - want).abs() <= (K / 8 + 8) * 2.0 ** -24 * size + 1e-30).all())
    for rows in (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 47, 64, 100, 200):
        assert torch.equal(ops().gemm_plain(x[:rows], w, gated=gated), full[:rows]), rows
    bias = torch.randn(w.shape[0], device=DEV, generator=g)
    if not gated:
        assert torch.equal(ops().gemm_plain(x[3:40], w, bias), ops().gemm_plain(x, w, bias)[3:40])
