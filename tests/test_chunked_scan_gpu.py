"""The decayed recurrence over chunks of 64 rows side by side: against the recurrence in 64-bit, at the edges of chunks, of tiles
and of the slices of columns."""
from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def ops():
    from llm_inference_lab_b200.kernels import ops as module
    return module


def context(q_lens, slots):
    t = lambda a: torch.tensor(a, dtype=torch.int32, device=DEV)  # noqa: E731
    return SimpleNamespace(q_start=t([0] + list(np.cumsum(q_lens))), state_slot=t(slots), n_requests=len(q_lens), max_q_len=max(q_lens))


# less than a chunk, a whole one, one row more, several and a rest; padding (slot -1) in between and last
Q_LENS = [1, 63, 7, 64, 65, 129, 300, 3]
SLOTS = [4, 0, -1, 2, 5, 1, 6, -1]
LIVE = np.repeat(np.array(SLOTS) >= 0, Q_LENS)


@pytest.mark.parametrize("heads,groups,keys,vdim,per_token,silu", [
    (4, 2, 64, 68, True, False), (2, 1, 50, 33, True, True), (3, 3, 16, 20, False, True), (1, 1, 3, 1, True, False),
    (2, 2, 128, 132, True, False), (1, 1, 65, 144, False, False), (2, 1, 12, 72, True, False)])
def test_chunks(heads, groups, keys, vdim, per_token, silu, monkeypatch):
    monkeypatch.setattr(ops(), "decay_scan_chunks", lambda *a: True)
    g = torch.Generator(device=DEV).manual_seed(keys + vdim)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    T = sum(Q_LENS)
    qk, v = rand(T, 2 * groups * keys), rand(T, heads * vdim)
    gates = torch.stack([torch.exp(-torch.rand(T, heads, device=DEV, generator=g) * 0.2), rand(T, heads)], dim=1)
    gates[70, 0] = 0.0      # a decay that forgets everything
    fixed = 1.0 - torch.rand(heads, device=DEV, generator=g) * 0.1
    state = rand(7, heads, keys, vdim)
    start, ctx = state.clone(), context(Q_LENS, SLOTS)
    how = dict(a_tok=gates[:, 0], s_tok=gates[:, 1]) if per_token else dict(a_head=fixed)
    for write in (False, True):
        out = ops().decay_scan(qk[:, : groups * keys], qk[:, groups * keys:], v, state, ctx, heads, groups, keys, vdim, silu=silu,
                               write=write, **how)
        assert write or torch.equal(state, start)
    ops().take_device_errors()
    n = lambda t: t.double().cpu().numpy()  # noqa: E731
    act = (lambda z: z / (1 + np.exp(-z))) if silu else (lambda z: z)
    Q, K = (act(n(t)).reshape(T, groups, keys).repeat(heads // groups, axis=1) for t in (qk[:, : groups * keys], qk[:, groups * keys:]))
    V, W = act(n(v)).reshape(T, heads, vdim), n(start)
    a, s = (n(gates[:, 0]), n(gates[:, 1])) if per_token else (np.tile(n(fixed), (T, 1)), np.ones((T, heads)))
    want, at = np.zeros((T, heads, vdim)), 0
    for length, slot in zip(Q_LENS, SLOTS):
        for t in range(at, at + length) if slot >= 0 else ():
            W[slot] = a[t][:, None, None] * W[slot] + (s[t][:, None] * K[t])[:, :, None] * V[t][:, None, :]
            want[t] = (W[slot] * Q[t][:, :, None]).sum(1)
        at += length
    # as for the walk: 32-bit roundings over a memory of ten tokens or so and sums of up to 128; SiLU's exponential is off by 2^-21
    off = lambda got, want: np.abs(n(got) - want).max() / np.abs(want).max()  # noqa: E731
    assert off(out[torch.from_numpy(LIVE).to(DEV)], want.reshape(T, -1)[LIVE]) < 2e-5 and off(state, W) < 2e-5


@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("row", [0, 5, 63, 64, 100])
def test_rows_before_a_non_finite_one_are_as_they_were(bad, row, monkeypatch):
    monkeypatch.setattr(ops(), "decay_scan_chunks", lambda *a: True)
    T, H, N, V = 130, 2, 64, 68
    g = torch.Generator(device=DEV).manual_seed(row)
    q, k, v = (torch.randn(T, H * w, device=DEV, generator=g) for w in (N, N, V))
    qk, decay = torch.cat([q, k], dim=1), torch.full((H,), 0.9, device=DEV)
    run = lambda qk, v: ops().decay_scan(qk[:, : H * N], qk[:, H * N:], v, torch.zeros(1, H, N, V, device=DEV),  # noqa: E731
                                         context([T], [0]), H, H, N, V, a_head=decay)
    clean = run(qk, v)
    v_bad, k_bad = v.clone(), qk.clone()
    v_bad[row, 3], k_bad[row, H * N + 3] = bad, bad
    for out in (run(qk, v_bad), run(k_bad, v)):
        assert torch.equal(out[:row], clean[:row]) and not torch.isfinite(out[row]).all()
