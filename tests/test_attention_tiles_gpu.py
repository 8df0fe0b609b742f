"""Attention on the ordinary units: tiles of 32, 16 and 8 rows give a row the same bits, and those of the softmax in 64-bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_inference_lab_b200.kernels import ops as module
    return module


@pytest.mark.parametrize("bad", [None, float("inf"), float("nan")])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n_q,n_kv,lens,past", [(14, 2, [1300], [0]), (14, 2, [1, 700, 33, 640], [90, 5, 0, 64]), (40, 1, [610], [3])])
def test_a_row_is_the_same_in_every_tile(n_q, n_kv, lens, past, dtype, bad):
    d, page, T = 64, 16, sum(lens)
    g = torch.Generator(device=DEV).manual_seed(T)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g).to(dtype)  # noqa: E731
    pages = -(-max(n + p for n, p in zip(lens, past)) // page)
    q, ck, cv = rand(T, n_q * d), rand(len(lens) * pages, n_kv, page, d), rand(len(lens) * pages, n_kv, page, d)
    t = lambda a: torch.tensor(np.asarray(a), dtype=torch.int32, device=DEV)  # noqa: E731
    bt = torch.randperm(len(lens) * pages, device=DEV, generator=g).to(torch.int32).view(len(lens), pages)
    req, pos = t(np.repeat(np.arange(len(lens)), lens)), t(np.concatenate([np.arange(n) + p for n, p in zip(lens, past)]))
    q_start = t(np.concatenate([[0], np.cumsum(lens)]))
    where = lens[-1] // 2      # a position of the last request
    if bad is not None:
        cv[bt[-1, where // page].long(), 0, where % page, 5] = bad

    def run(a, b, **k):
        return ops().attention_plain(q[a:b], ck, cv, req[a:b].contiguous(), pos[a:b].contiguous(), bt, n_q, n_kv, d, 0, d ** -0.5, **k)

    together = run(0, T, q_start=q_start, requests=len(lens))
    assert -(-T // max(1, 32 // (n_q // n_kv))) * -(-(n_q // n_kv) // 32) * n_kv >= 4 * ops().sm_count()
    ops().take_device_errors()
    same = lambda a, b: torch.equal(torch.nan_to_num(a, 1e3, 2e3, 3e3), torch.nan_to_num(b, 1e3, 2e3, 3e3))  # noqa: E731
    for a, n in ((0, 40), (T - 40, 40), (T - lens[-1] + where - 3, 7), (1, 1), (T // 2, 160)):
        assert same(run(a, a + n), together[a: a + n])
    if bad is not None:      # the rows that see the position, at the heads of its kv head
        seen = torch.zeros(T, dtype=torch.bool, device=DEV)
        seen[T - lens[-1] + max(0, where - past[-1]):] = True
        hit = ~torch.isfinite(together.view(T, n_q, d)).all(2)
        assert not hit[~seen].any() and not hit[:, n_q // n_kv:].any() and hit[seen][:, : n_q // n_kv].all()
        return
    for row in (0, 1, T // 3, T - 1):
        r, n = int(req[row]), int(pos[row]) + 1
        k, v = (c[bt[r].long()].permute(1, 0, 2, 3).reshape(n_kv, -1, d)[:, :n].double().repeat_interleave(n_q // n_kv, 0) for c in (ck, cv))
        w = torch.softmax((k @ q[row].view(n_q, d, 1).double()).squeeze(2) * d ** -0.5, dim=1)
        want = (w.unsqueeze(2) * v).sum(1).view(-1)
        # 32-bit roundings of scores of a few units and sums of up to 1,300 terms; one rounding to 16 bits
        assert (together[row].double() - want).abs().max() < (2e-6 if dtype == torch.float32 else 2.0 ** -8) * want.abs().max().clamp(min=1.0)
