"""The decode attention that sums, rotates and stores its own step's projections: the same bits as the two kernels apart, in the
output and in the cache."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_inference_lab_b200.kernels import ops as module
    return module


@pytest.mark.parametrize("n_q,n_kv,d,lens,window,parts,page", [
    (14, 2, 64, [520] * 8, 0, 7, 16), (14, 2, 64, [1, 2, 32, 33, 64, 65, 129, 1000], 0, 0, 16), (28, 4, 128, [4097] * 5, 0, 5, 16),
    (16, 1, 64, [300, 31, 1], 0, 13, 8), (3, 3, 80, [50, 700, 16], 0, 4, 16), (8, 2, 16, [17, 90], 0, 1, 4),
    (14, 2, 64, [700, 64, 40], 48, 3, 16), (14, 2, 64, [40000], 0, 2, 64), (12, 2, 128, [600] * 70, 0, 0, 16)])
def test_same_as_rotation_and_attention_apart(n_q, n_kv, d, lens, window, parts, page):
    R, width = len(lens), (n_q + 2 * n_kv) * d
    g = torch.Generator(device=DEV).manual_seed(sum(lens) + d)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    bf = torch.bfloat16
    # a request without a row beside the others, and of the last one a row without a slot (padding) if there are several
    rows = [1] * R + [0]
    t = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)  # noqa: E731
    pages = -(-max(lens) // page)
    bt = torch.randperm((R + 1) * pages, device=DEV, generator=g).to(torch.int32).view(R + 1, pages)
    kv = np.array(lens + [0])
    slots = np.array([int(bt[r, (n - 1) // page]) * page + (n - 1) % page for r, n in enumerate(lens)])
    if R > 2:
        slots[-1] = -1
    ck, cv = rand((R + 1) * pages, n_kv, page, d).to(bf), rand((R + 1) * pages, n_kv, page, d).to(bf)
    qkv = rand(parts, R, width) if parts else rand(R, width).to(bf)
    bias = rand(width).to(bf) if parts > 1 else None
    positions, inv_freq = t(kv[:R] - 1), 10000.0 ** (-torch.arange(0, d, 2, device=DEV, dtype=torch.float32) / d)
    ctx = SimpleNamespace(q_start=t(np.concatenate([[0], np.cumsum(rows)])), kv_len=t(kv), pos0=t(np.maximum(kv - 1, 0)), n_requests=R + 1,
                          q_lens=rows, max_q_len=1, max_kv_len=max(lens))
    group = SimpleNamespace(block_table=bt)
    assert ops().attention_rotates(ctx, n_q, n_kv, d, d, ck)
    k1, v1, k2, v2 = ck.clone(), cv.clone(), ck.clone(), cv.clone()
    got = ops().attention_rotated(qkv.clone(), bias, positions, inv_freq, t(slots), k1, v1, ctx, group, n_q, n_kv, d, window, d ** -0.5)
    q = ops().rope_kv_write(qkv.clone(), positions, inv_freq, d, t(slots), k2, v2, n_q, n_kv, d, bias=bias)
    want = ops().attention(q, k2, v2, ctx, group, n_q, n_kv, d, window, d ** -0.5)
    ops().take_device_errors()
    assert torch.equal(k1, k2) and torch.equal(v1, v2) and not torch.equal(k1, ck)
    assert torch.equal(got, want) and torch.isfinite(got.float()).all()


def test_a_slot_beyond_the_pages_is_an_error():
    ck = torch.zeros(4, 2, 16, 64, device=DEV, dtype=torch.bfloat16)
    t = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = SimpleNamespace(q_start=t([0, 1]), kv_len=t([5]), n_requests=1, q_lens=[1], max_q_len=1, max_kv_len=5)
    ops().attention_rotated(torch.zeros(1, 18 * 64, device=DEV, dtype=torch.bfloat16), None, t([4]), torch.ones(32, device=DEV), t([64]), ck,
                            ck.clone(), ctx, SimpleNamespace(block_table=t([[0]])), 14, 2, 64, 0, 0.125)
    with pytest.raises(ops().KernelError):
        ops().take_device_errors()
    assert not ck.any()


def test_rows_or_a_bias_off_16_bytes_are_refused():
    ck = torch.zeros(4, 2, 16, 64, device=DEV, dtype=torch.bfloat16)
    t = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    ctx = SimpleNamespace(q_start=t([0, 1]), kv_len=t([5]), n_requests=1, q_lens=[1], max_q_len=1, max_kv_len=5)
    width, bf = 18 * 64, torch.bfloat16
    run = lambda rows, bias: ops().attention_rotated(rows, bias, t([4]), torch.ones(32, device=DEV), t([4]), ck, ck.clone(), ctx,  # noqa: E731
                                                     SimpleNamespace(block_table=t([[0]])), 14, 2, 64, 0, 0.125)
    run(torch.zeros(2, 1, width, device=DEV), torch.zeros(width, device=DEV, dtype=bf))
    for rows, bias in ((torch.zeros(width + 1, device=DEV, dtype=bf)[1:].view(1, width), None),
                       (torch.zeros(2, 1, width, device=DEV), torch.zeros(width + 1, device=DEV, dtype=bf)[1:])):
        with pytest.raises(ops().KernelError):
            run(rows, bias)
    ops().take_device_errors()
