"""The decays of the selective scan: the exponential by itself, what is no number or infinite, and slow decays over
thousands of tokens, in one piece and in segments."""
import numpy as np
import pytest
import torch

from test_segments_gpu import DEV, context, ops

pytestmark = pytest.mark.gpu


def scan(x, dt_pre, bc, a_log, state, lens, slots, segments, monkeypatch):
    monkeypatch.setattr(ops(), "scan_segments", lambda *a: segments)
    N, zeros = a_log.shape[1], torch.zeros_like(a_log[:, 0])
    out = ops().selective_scan(x, dt_pre, bc, 0, N, torch.ones_like(x), a_log, zeros, zeros, state, context(lens, slots))
    ops().take_device_errors()
    return out


def test_decay_is_the_exponential(monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(1)
    requests, channels = 64, 2048
    dt = torch.exp(torch.rand(requests, channels, device=DEV, generator=g) * np.log(87.0 / 1e-6) + np.log(1e-6))
    dt[0, :3] = torch.tensor([86.0, 86.5, 85.5], device=DEV)
    dt_pre = torch.where(dt > 20, dt, torch.log(torch.expm1(dt)))
    a_log = torch.zeros(channels, 4, device=DEV)      # A = -1
    a_log[:, 1:] = -20.0
    ones = torch.ones(requests, 8, device=DEV)
    run = lambda x, state: scan(x, dt_pre, ones, a_log, state, [1] * requests, range(requests), 1, monkeypatch)  # noqa: E731
    step, decay = torch.zeros(requests, channels, 4, device=DEV), torch.ones(requests, channels, 4, device=DEV)
    run(torch.ones_like(dt), step)         # 0 * decay + dt * 1 * 1: the step size as the kernel has it
    run(torch.zeros_like(dt), decay)       # 1 * decay + 0: the decay
    want = np.exp(-step[:, :, 0].double().cpu().numpy())
    ulp = np.spacing(want.astype(np.float32)).astype(np.float64)
    # CUDA states at most two units in the last place for expf, whatever the argument
    assert (np.abs(decay[:, :, 0].double().cpu().numpy() - want) <= 2 * ulp).all()


@pytest.mark.parametrize("N", [16, 6])
@pytest.mark.parametrize("segments", [1, 3])
def test_no_numbers_and_infinities_pass_through(segments, N, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(2)
    T, channels, nan, inf = 150, 40, float("nan"), float("inf")
    rand = lambda *s: torch.randn(s, device=DEV, generator=g)  # noqa: E731
    x, dt_pre, bc, a_log, state = rand(T, channels), rand(T, channels) - 3, rand(T, 2 * N), rand(channels, N), rand(1, channels, N)
    clean_state = state.clone()
    clean = scan(x, dt_pre, bc, a_log, clean_state, [T], [0], segments, monkeypatch)
    a_log[1, 2] = nan                                 # a decay that is no number
    a_log[5, 0], dt_pre[:, 5] = inf, -200.0           # exp(0 * -inf)
    a_log[9, 1] = inf                                 # exp(-inf): nothing is kept
    dt_pre[30, 13] = nan
    a_log[17] = 3.0
    dt_pre[40, 17], x[40, 17] = 300.0, 0.0            # decays below the least number: the state is left empty
    x[60, 21] = inf
    out = scan(x, dt_pre, bc, a_log, state, [T], [0], segments, monkeypatch)
    bad = [1, 5, 9, 13, 17, 21]
    fine = [c for c in range(channels) if c not in bad]
    assert torch.equal(out[:, fine], clean[:, fine]) and torch.equal(state[0, fine], clean_state[0, fine])
    assert bool(out[:, [1, 5]].isnan().all()) and bool(state[0, 1, 2].isnan()) and bool(state[0, 5, 0].isnan())
    assert bool(out[:, 9].isfinite().all())
    last = x[-1, 9] * torch.nn.functional.softplus(dt_pre[-1, 9]) * bc[-1, 1]
    assert abs(float(state[0, 9, 1] - last)) <= 1e-6 * abs(float(last))
    assert bool(out[30:, 13].isnan().all()) and torch.equal(out[:30, 13], clean[:30, 13])
    assert float(out[40, 17]) == 0.0 and bool(out[:, 17].isfinite().all())
    assert torch.equal(out[:60, 21], clean[:60, 21]) and not bool(out[60:, 21].isfinite().any())
    # an infinite x times B is an infinity of B's sign in every entry: only a sum of both signs is no number
    assert not bool(state[0, 21].isnan().any())


def test_slow_decays_lose_no_more_than_the_library_exponential(monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(3)
    T, channels, N = 4096, 64, 4
    x = torch.rand(T, channels, device=DEV, generator=g)
    dt_pre = torch.full((T, channels), float(np.log(np.expm1(1e-3))), device=DEV)
    dt_pre += torch.randn(1, channels, device=DEV, generator=g)
    bc, a_log = torch.ones(T, 2 * N, device=DEV), torch.rand(channels, N, device=DEV, generator=g) * 3 - 2
    # the step sizes as the kernel has them
    probe = torch.zeros(1, channels, N, device=DEV)
    scan(torch.ones_like(x[:1]), dt_pre[:1], bc[:1], a_log, probe, [1], [0], 1, monkeypatch)
    dt = probe[0, :, :1]
    decay = torch.exp(dt * -torch.exp(a_log))
    plain, exact = torch.zeros(channels, N, device=DEV), torch.zeros(channels, N, device=DEV, dtype=torch.float64)
    exact_decay = torch.exp(dt.double() * -torch.exp(a_log.double()))
    for t in range(T):
        dx = dt * x[t, :, None]
        plain = torch.addcmul(dx, decay, plain)
        exact = dt.double() * x[t, :, None].double() + exact_decay * exact
    off = lambda s: float(((s.double() - exact) / exact).norm()) / exact.numel() ** 0.5  # noqa: E731
    for segments in (1, 4, 16):
        state = torch.zeros(1, channels, N, device=DEV)
        scan(x, dt_pre, bc, a_log, state, [T], [0], segments, monkeypatch)
        # (segments: the opening state takes one exponential over a segment's sum of step sizes)
        assert off(state[0]) <= 1.25 * off(plain), (segments, off(state[0]), off(plain))
