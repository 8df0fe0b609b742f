"""The generalized delta rule by blocks of four tokens against the recurrence in 64-bit: portions that end inside a block and
inside a chunk, requests whose first rows lie anywhere in the batch, single tokens beside them, rows of padding."""
import numpy as np
import pytest
import torch

from test_segments_gpu import DEV, context, ops

pytestmark = pytest.mark.gpu


def plain(r, k, v, a, decay, S):
    """S [keys, values] is advanced; the outputs o = S^T r, row by row, each over its root mean square"""
    out = []
    for t in range(len(r)):
        unit = k[t] / np.sqrt((k[t] ** 2).sum() + 1e-6)
        S = decay[t][:, None] * S - np.outer(a[t] * unit, unit @ S) + np.outer(k[t], v[t])
        o = S.T @ r[t]
        out.append(o / np.sqrt((o ** 2).mean() + 1e-6))
    return np.array(out), S


@pytest.mark.parametrize("D,heads", [(32, 3), (64, 9), (128, 2), (256, 1)])
@pytest.mark.parametrize("lens", [[32], [33, 1, 2, 67], [1, 130, 35, 4, 3], [34, 36]])
def test_blocks_of_four_tokens(D, heads, lens, monkeypatch):
    assert ops().delta_rule_blocks(max(lens))
    monkeypatch.setattr(ops(), "delta_blocks_pay", lambda *a: True)
    g = torch.Generator(device=DEV).manual_seed(D + sum(lens))
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    T, hd, rate = sum(lens), heads * D, 0.6
    slots = [(3 * i + 1) % 7 for i in range(len(lens))]
    if len(lens) > 2:
        slots[-1] = -1
    proj, decay_pre = rand(T, 5 * hd + 3)[:, : 5 * hd], rand(T, hd)
    decay_bias, rate_bias, weight = ((rand(hd) + m).bfloat16() for m in (-1.0, 0.0, 1.0))
    state = rand(7, heads, D, D)
    start, n = state.clone(), lambda t: t.double().cpu().numpy()
    run = lambda write: ops().delta_rule(proj, decay_pre, decay_bias, rate_bias, weight, state, context(lens, slots), heads, D,  # noqa: E731
                                         1e-6, rate, write=write)
    out = run(False)
    assert torch.equal(state, start)
    assert torch.equal(run(True), out)
    ops().take_device_errors()
    sigmoid = lambda z: 1.0 / (1.0 + np.exp(-z))  # noqa: E731
    r, k, v, gate, a = (n(proj[:, i * hd: (i + 1) * hd]).reshape(T, heads, D) for i in range(5))
    decay = np.exp(-rate * sigmoid(n(decay_pre) + n(decay_bias))).reshape(T, heads, D)
    a = sigmoid(a + n(rate_bias).reshape(heads, D))
    at = 0
    for length, slot in zip(lens, slots):
        rows = slice(at, at + length)
        at += length
        if slot < 0:
            continue
        for h in range(heads):
            want, S = plain(r[rows, h], k[rows, h], v[rows, h], a[rows, h], decay[rows, h], n(start[slot, h]))
            want = want * n(weight)[h * D: (h + 1) * D] * sigmoid(gate[rows, h])
            got = n(out[rows])[:, h * D: (h + 1) * D]
            # bfloat16 results: half a unit of 2^-8 of themselves; the state: 32-bit roundings over its memory of a few tokens
            assert np.abs(got - want).max() <= 2 ** -8 * np.abs(want).max()
            assert np.abs(n(state[slot, h]) - S).max() <= 1e-5 * np.abs(S).max()
    used = [s for s in slots if s >= 0]
    rest = [s for s in range(7) if s not in used]
    assert torch.equal(state[rest], start[rest])


@pytest.mark.parametrize("D,heads", [(32, 1), (64, 2)])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("row", [0, 1, 2, 3, 8, 17, 22, 31])
def test_rows_before_a_non_finite_one_are_as_they_were(D, heads, bad, row, monkeypatch):
    """Every place of a block, of a portion's first block and of later ones; one entry of r, k, v, the gate, the rate or the decay."""
    T, hd = 35, heads * D
    assert ops().delta_rule_blocks(T)
    monkeypatch.setattr(ops(), "delta_blocks_pay", lambda *a: True)
    g = torch.Generator(device=DEV).manual_seed(row)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    proj, decay_pre, start = rand(T, 5 * hd), rand(T, hd), rand(1, heads, D, D)
    bias, weight = rand(hd).bfloat16(), rand(hd).bfloat16()

    def run(proj, decay_pre):
        return ops().delta_rule(proj, decay_pre, bias, bias, weight, start.clone(), context([T], [0]), heads, D, 1e-6, 0.6)

    clean = run(proj, decay_pre)
    assert clean.isfinite().all()
    for i in range(5):
        spoilt = proj.clone()
        spoilt[row, i * hd + 5] = bad
        out = run(spoilt, decay_pre)
        assert torch.equal(out[:row], clean[:row]), i
        if i < 3:
            assert not out[row, :D].isfinite().all(), i
        assert torch.equal(out[:, D:], clean[:, D:])      # the other heads
    spoilt = decay_pre.clone()
    spoilt[row, 5] = bad
    assert torch.equal(run(proj, spoilt)[:row], clean[:row])
    ops().take_device_errors()


@pytest.mark.parametrize("D,heads", [(32, 3), (64, 9), (128, 2), (256, 1)])
def test_blocks_and_single_rows_agree(D, heads, monkeypatch):
    """The two walks of the same step, single rows beside a portion: 32-bit roundings of the states, one of the outputs."""
    lens = [1, 50, 1, 3, 33, 1]
    g = torch.Generator(device=DEV).manual_seed(D)
    T, hd = sum(lens), heads * D
    proj, decay_pre = torch.randn(T, 5 * hd, device=DEV, generator=g), torch.randn(T, hd, device=DEV, generator=g)
    bias, weight = (torch.randn(hd, device=DEV, generator=g).bfloat16() for _ in range(2))
    start, got = torch.randn(6, heads, D, D, device=DEV, generator=g), {}
    for blocks in (True, False):
        monkeypatch.setattr(ops(), "delta_blocks_pay", lambda *a: blocks)
        state = start.clone()
        out = ops().delta_rule(proj, decay_pre, bias, bias, weight, state, context(lens, [4, 0, 5, 2, 1, 3]), heads, D, 1e-6, 0.6)
        got[blocks] = out.float(), state
    ops().take_device_errors()
    (a, S), (b, R) = got[True], got[False]
    assert not torch.equal(S, R) and float((S - R).abs().max()) <= 1e-5 * float(R.abs().max())
    # (an entry near zero takes the error of the whole row's)
    assert bool(((a - b).abs() <= 2.0 ** -7 * b.abs() + 1e-5 * b.abs().amax(1, keepdim=True)).all())
