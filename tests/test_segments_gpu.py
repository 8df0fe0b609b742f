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
    monkeypatch.setattr(ops(), "scan_segments_pay", lambda *a: True)
    g = torch.Generator(device=DEV).manual_seed(channels + N)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    T = sum(Q_LENS)
    x, dt_pre, z, bc = rand(T, channels), rand(T, channels) - 3, rand(T, channels), rand(T, 2 * N)
    a_log, skip, bias = rand(channels, N), rand(channels), rand(channels)
    state = rand(6, channels, N)
    start, ctx = state.clone(), context(Q_LENS, SLOTS)
    for write in (False, True):
        before = ops().COUNTER.launches
        out = ops().selective_scan(x, dt_pre, bc, 0, N, z, a_log, skip, bias, state, ctx, write=write)
        assert ops().COUNTER.launches - before == min(segments, 2)
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


@pytest.mark.parametrize("segments", [1, 2, 3, 5, 9])
@pytest.mark.parametrize("heads,groups,keys,vdim,per_token,silu", [(4, 2, 64, 68, True, False), (3, 3, 16, 20, False, True),
                                                                   (2, 1, 50, 33, True, False), (2, 2, 128, 128, True, False),
                                                                   (1, 1, 200, 8, False, False), (2, 1, 130, 33, True, False),
                                                                   (3, 3, 256, 96, True, True), (4, 2, 144, 68, True, False),
                                                                   (1, 1, 129, 1, False, True)])
def test_decay_scan_segments(heads, groups, keys, vdim, per_token, silu, segments, monkeypatch):
    monkeypatch.setattr(ops(), "decay_scan_segments", lambda *a: segments)
    g = torch.Generator(device=DEV).manual_seed(keys + vdim)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    T = sum(Q_LENS)
    qk, v = rand(T, 2 * groups * keys), rand(T, heads * vdim)
    gates = torch.stack([torch.exp(-torch.rand(T, heads, device=DEV, generator=g) * 0.2), rand(T, heads)], dim=1)
    fixed = 1.0 - torch.rand(heads, device=DEV, generator=g) * 0.1
    state = rand(6, heads, keys, vdim)
    start, ctx = state.clone(), context(Q_LENS, SLOTS)
    how = dict(a_tok=gates[:, 0], s_tok=gates[:, 1]) if per_token else dict(a_head=fixed)
    for write in (False, True):
        before = ops().COUNTER.launches
        out = ops().decay_scan(qk[:, : groups * keys], qk[:, groups * keys:], v, state, ctx, heads, groups, keys, vdim, silu=silu,
                               write=write, **how)
        # (up to 128 key channels never go in segments)
        assert ops().COUNTER.launches - before == (min(segments, 2) if keys > 128 else 1)
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
    live = T - Q_LENS[-1]      # (a row of padding leaves nothing)
    # 32-bit roundings over a memory of ten tokens or so and sums of up to 200; SiLU's exponential is off by 2^-21
    assert off(out[:live], want.reshape(T, -1)[:live]) < 2e-5 and off(state, W) < 2e-5


@pytest.mark.parametrize("heads", [1, 5, 14])
def test_running_maximum_of_any_length(heads):
    g = torch.Generator(device=DEV).manual_seed(heads)
    lens, slots = [1, 7, 8, 255, 256, 257, 700, 2], [3, 0, 7, 5, 1, 6, 2, -1]
    T, ctx = sum(lens), context(lens, slots)
    gates = torch.randn(T, 2, heads, device=DEV, generator=g) * 3
    gates[:, 1] = -torch.nn.functional.softplus(gates[:, 1])
    m_state = torch.randn(8, heads, device=DEV, generator=g)
    log_i, log_f, M = (t.double().cpu().numpy() for t in (gates[:, 0], gates[:, 1], m_state))
    m = ops().memory_stabilize(gates, m_state, ctx)
    got, at = [t.double().cpu().numpy() for t in (m, gates[:, 0], gates[:, 1])], 0
    for length, slot in zip(lens, slots):
        for t in range(at, at + length) if slot >= 0 else ():
            top = np.maximum(log_f[t] + M[slot], log_i[t])
            # up to 700 roundings of sums of a few tens
            assert np.abs(got[0][t] - top).max() < 1e-3
            assert np.abs(got[1][t] - np.exp(log_f[t] + M[slot] - top)).max() < 1e-3
            assert np.abs(got[2][t] - np.exp(log_i[t] - top)).max() < 1e-3
            M[slot] = top
        at += length
    assert np.abs(m_state.double().cpu().numpy() - M).max() < 1e-3


@pytest.mark.parametrize("segments", [1, 2, 3, 5, 9])
# (200 key channels: in one piece whatever the rule says)
@pytest.mark.parametrize("heads,groups,keys,vdim", [(4, 2, 64, 64), (3, 1, 20, 36), (2, 2, 128, 100), (1, 1, 200, 24), (2, 1, 16, 130)])
def test_delta_walk_segments(heads, groups, keys, vdim, segments, monkeypatch):
    monkeypatch.setattr(ops(), "delta_walk_segments", lambda *a: segments)
    g = torch.Generator(device=DEV).manual_seed(keys + vdim)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    T, taps, H, G = sum(Q_LENS), 4, heads, groups
    gd, hv = G * keys, H * vdim
    proj = rand(T, 2 * gd + hv + 2 * H)
    conv, a_log, bias = rand(2 * gd + hv, taps) * 0.5, rand(H), rand(H) - 2
    state, kept = rand(6, H, keys, vdim), rand(6, taps - 1, 2 * gd + hv)
    start, kept_start, ctx = state.clone(), kept.clone(), context(Q_LENS, SLOTS)
    for write in (False, True):
        operands = ops().delta_prepare(proj, 2 * gd + hv, 2 * gd + hv + H, taps, H, G, keys, vdim, conv, a_log, bias, kept, ctx,
                                       keys ** -0.5, 1e-6)
        out = ops().delta_walk(*operands, state, ctx, H, G, keys, vdim, write=write, proj=proj, kept=kept)
        assert write or torch.equal(state, start) and torch.equal(kept, kept_start)
    ops().take_device_errors()
    n = lambda t: t.double().cpu().numpy()  # noqa: E731
    P, W, want, at = n(proj), n(start), np.zeros((T, H, vdim)), 0
    silu = lambda z: z / (1 + np.exp(-z))  # noqa: E731
    for length, slot in zip(Q_LENS, SLOTS):
        if slot < 0:
            continue
        full = np.concatenate([n(kept_start)[slot], P[at: at + length, : 2 * gd + hv]])
        assert np.array_equal(n(kept)[slot], full[-(taps - 1):])
        u = silu(sum(full[j: j + length] * n(conv)[:, j] for j in range(taps)))
        q, k = (u[:, i * gd: (i + 1) * gd].reshape(length, G, keys) for i in (0, 1))
        q, k = (m / np.sqrt((m * m).sum(-1, keepdims=True) + 1e-6) for m in (q, k))
        q, k, v = q.repeat(H // G, 1) * keys ** -0.5, k.repeat(H // G, 1), u[:, 2 * gd:].reshape(length, H, vdim)
        rate = 1 / (1 + np.exp(-P[at: at + length, 2 * gd + hv: 2 * gd + hv + H]))
        decay = np.exp(-np.exp(n(a_log)) * np.log1p(np.exp(P[at: at + length, 2 * gd + hv + H:] + n(bias))))
        for t in range(length):
            S = decay[t][:, None, None] * W[slot]
            new = rate[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1))
            W[slot] = S + k[t][:, :, None] * new[:, None, :]
            want[at + t] = (W[slot] * q[t][:, :, None]).sum(1)
        at += length
    live = T - Q_LENS[-1]
    # 32-bit roundings over the state's memory (decays near 0.9) and sums of up to 200
    assert off(out[:live], want.reshape(T, -1)[:live]) < 2e-5 and off(state, W) < 2e-5


def test_decays_go_by_the_running_maximum_that_is_kept():
    g = torch.Generator(device=DEV).manual_seed(11)
    lens, slots, heads = [9, 700, 1, 256], [1, 0, 3, 2], 3
    T, ctx = sum(lens), context(lens, slots)
    log_i = torch.randn(T, heads, device=DEV, generator=g) * 3 + torch.tensor([0.0, 4900.0, 5100.0], device=DEV)
    log_f = -torch.rand(T, heads, device=DEV, generator=g)
    gates, m_state = torch.stack([log_i, log_f], dim=1), torch.full((4, heads), 5000.0, device=DEV)
    m = ops().memory_stabilize(gates, m_state, ctx).cpu().numpy()
    decay, scale = (gates[:, i].cpu().numpy() for i in (0, 1))
    log_i, log_f, at = log_i.cpu().numpy(), log_f.cpu().numpy(), 0
    for length, slot in zip(lens, slots):
        before = np.concatenate([np.full((1, heads), 5000.0, dtype=np.float32), m[at: at + length - 1]])
        now = m[at: at + length]
        carried = log_f[at: at + length] + before      # 32-bit, as the kernel forms it
        # the exponentials' arguments are differences of 32-bit numbers: what is left is the exponentials' own rounding
        assert np.abs(decay[at: at + length] - np.exp((carried - now).astype(np.float64))).max() < 1e-6
        assert np.abs(scale[at: at + length] - np.exp((log_i[at: at + length] - now).astype(np.float64))).max() < 1e-6
        assert np.array_equal(m_state[slot].cpu().numpy(), now[-1])
        at += length


@pytest.mark.parametrize("heads,keys,vdim", [(12, 128, 128), (9, 100, 68), (7, 256, 96), (14, 64, 64)])
def test_decay_scan_of_many_requests_has_the_bits_of_one(heads, keys, vdim):
    """Steps of many CTAs of more than 64 key channels run a build with fewer registers."""
    g = torch.Generator(device=DEV).manual_seed(keys)
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    lens = [1] * 12 + [17, 40, 3, 16, 1, 33]
    T, slots = sum(lens), list(np.random.default_rng(keys).permutation(len(lens)))
    qk, v, state = rand(T, 2 * heads * keys), rand(T, heads * vdim), rand(len(lens), heads, keys, vdim)
    decay, scale = torch.exp(-torch.rand(T, heads, device=DEV, generator=g) * 0.2), rand(T, heads)
    gates = torch.stack([decay, scale], dim=1)

    def walk(a, b, lens, slots, state):
        return ops().decay_scan(qk[a:b, : heads * keys], qk[a:b, heads * keys:], v[a:b], state, context(lens, slots), heads, heads, keys,
                                vdim, a_tok=gates[a:b, 0], s_tok=gates[a:b, 1], in_order=True)

    together, at = state.clone(), 0
    out = walk(0, T, lens, slots, together)
    ops().take_device_errors()
    assert len(lens) * heads * -(-vdim // 32) > 2 * ops().sm_count() or keys <= 64
    for n, slot in zip(lens, slots):
        alone = state.clone()
        assert torch.equal(walk(at, at + n, [n], [slot], alone), out[at: at + n]) and torch.equal(alone[slot], together[slot])
        at += n
