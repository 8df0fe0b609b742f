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
def test_blocks_of_four_tokens(D, heads, lens):
    assert ops().delta_rule_blocks(max(lens))
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
