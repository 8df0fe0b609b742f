"""Recurrences whose rows are cut into segments walked side by side: against the recurrence in 64-bit, for every number of
segments, at the edges of chunks and segments."""
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
    return SimpleNamespace(q_start=t([0] + list(np.cumsum(q_lens))), state_slot=t(slots), n_requests=len(q_lens), max_q_len=max(q_lens),
                           n_tokens=sum(q_lens), row_req=t(np.repeat(np.arange(len(q_lens)), q_lens)))


def off(got, want):
    got, want = got.double().cpu().numpy(), np.asarray(want)
    return np.abs(got - want).max() / max(1e-30, np.abs(want).max())


# one token, a chunk and one more, several chunks; a row of padding (slot -1) last
Q_LENS = [1, 33, 64, 150, 97, 2]
SLOTS = [4, 0, 2, 5, 1, -1]


@pytest.mark.parametrize("segments", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("channels,N", [(40, 16), (33, 3), (36, 20), (8, 64), (20, 100), (5, 256)])
def test_selective_scan_segments(channels, N, segments, monkeypatch):
    monkeypatch.setattr(ops(), "scan_segments", lambda ctas, longest: segments)
    g = torch.Generator(device=DEV).manual_seed(channels + N)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    T = sum(Q_LENS)
    x, dt_pre, z, bc = rand(T, channels), rand(T, channels) - 3, rand(T, channels), rand(T, 2 * N)
    a_log, skip, bias = rand(channels, N), rand(channels), rand(channels)
    state = rand(6, channels, N)
    start, ctx = state.clone(), context(Q_LENS, SLOTS)
    for write in (False, True):
        out = ops().selective_scan(x, dt_pre, bc, 0, N, z, a_log, skip, bias, state, ctx, write=write)
        assert write or torch.equal(state, start)
    ops().take_device_errors()
    n = lambda t: t.double().cpu().numpy()  # noqa: E731
    X, Z, B, A, W = n(x), n(z), n(bc), -np.exp(n(a_log)), n(start)
    dt = np.log1p(np.exp(n(dt_pre) + n(bias)))
    want, at = np.zeros((T, channels)), 0
    for length, slot in zip(Q_LENS, SLOTS):
        for t in range(at, at + length) if slot >= 0 else ():
            W[slot] = np.exp(dt[t][:, None] * A) * W[slot] + (dt[t] * X[t])[:, None] * B[t, None, :N]
            want[t] = (W[slot] @ B[t, N:] + n(skip) * X[t]) * Z[t] / (1 + np.exp(-Z[t]))
        at += length
    # 32-bit roundings, a few units of 2^-24 a token where the state's memory is long (150 tokens) and sums of up to 256
    assert off(out, want) < 2e-5 and off(state, W) < 2e-5
