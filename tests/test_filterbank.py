"""Batched ragged FIR -> cascaded-biquad filter bank (forward + adjoint).

CPU: the FP64 restatement's adjoint against central finite differences (pins
the reference the GPU path is compared with), and the plan entry points'
export.  GPU: the C-ABI forward/backward against the FP64 restatement, bitwise
repeatability, autograd, and CUDA-graph replay."""
import numpy as np
import pytest

from filterbank_ref import bank_adjoint, bank_forward, channel_adjoint, channel_forward, stable_sections


def _loss(x, h, c, w):
    y, _ = channel_forward(x, h, c)
    return float(w @ y)


@pytest.mark.parametrize("L,T,S", [(40, 5, 2), (17, 1, 3), (9, 9, 1), (30, 4, 0)])
def test_fp64_adjoint_matches_finite_differences(L, T, S):
    rng = np.random.default_rng(L * 100 + T * 10 + S)
    x = rng.standard_normal(L)
    h = rng.standard_normal(T)
    c = stable_sections(rng, S).reshape(-1)
    w = rng.standard_normal(L - T + 1)
    gx, gh, gc = channel_adjoint(x, h, c, w)
    eps = 1e-6
    for vec, grad in ((x, gx), (h, gh), (c, gc.reshape(-1))):
        fd = np.zeros_like(vec)
        for i in range(len(vec)):
            vp = vec.copy()
            vm = vec.copy()
            vp[i] += eps
            vm[i] -= eps
            args_p = [vp if vec is a else a for a in (x, h, c)]
            args_m = [vm if vec is a else a for a in (x, h, c)]
            fd[i] = (_loss(*args_p, w) - _loss(*args_m, w)) / (2 * eps)
        np.testing.assert_allclose(grad, fd, rtol=1e-6, atol=1e-7)


def test_reference_composed_step_matches_fp64():
    """The CPU baseline step built from the reference's natural-C kernels computes the same gradients."""
    import oracle
    from oracle.filterbank import channel_step

    if not oracle.ref_available():
        pytest.skip("oracle/_ref not built")
    rng = np.random.default_rng(11)
    L, T, S = 3000, 37, 3
    x = rng.standard_normal(L).astype(np.float32)
    h = (rng.standard_normal(T) / np.sqrt(T)).astype(np.float32)
    c = stable_sections(rng, S).astype(np.float32)
    target = rng.standard_normal(L - T + 1).astype(np.float32)
    n = L - T + 1
    loss, gx, gh, gc = channel_step(x, h, c, target, n)
    y64, _ = channel_forward(x, h, c)
    gy64 = 2.0 * (y64 - target) / n
    gx64, gh64, gc64 = channel_adjoint(x, h, c, gy64)
    assert loss == pytest.approx(float((y64 - target) @ (y64 - target)) / n, rel=1e-5)
    for got, want in ((gx, gx64), (gh, gh64), (gc, gc64)):
        assert np.abs(got - want).max() <= 1e-4 * np.abs(want).max()


def test_plan_symbols_exported():
    from c7x_dsplib_b200 import lib

    L = lib()
    for n in ("DSPLIB_gpu_raggedPlanCreate", "DSPLIB_gpu_raggedPlanSize", "DSPLIB_gpu_raggedPlanDestroy",
              "DSPLIB_gpu_firBiquadBatched_fwd", "DSPLIB_gpu_firBiquadBatched_bwd"):
        assert hasattr(L, n)


# ---------------------------------------------------------------------------------- GPU


def _bank_case(seed, C, Lrange=(64, 20000), Tmax=64, Smax=6, force=()):
    rng = np.random.default_rng(seed)
    lengths, taps, stages = [], [], []
    for _ in range(C):
        T = int(rng.integers(1, Tmax + 1))
        L = int(rng.integers(max(T, Lrange[0]), Lrange[1] + 1))
        lengths.append(L)
        taps.append(T)
        stages.append(int(rng.integers(0, Smax + 1)))
    for L, T, S in force:
        lengths.append(L)
        taps.append(T)
        stages.append(S)
    x = rng.standard_normal(sum(lengths))
    h = np.concatenate([rng.standard_normal(T) / np.sqrt(T) for T in taps])
    c = np.concatenate([stable_sections(rng, S).reshape(-1) for S in stages] + [np.zeros(0)])
    return lengths, taps, stages, x, h, c


def _per_channel_err(lengths, offsets_len, got, want):
    """max |got - want| / max(|want|) per channel segment."""
    worst = 0.0
    o = 0
    for n in offsets_len:
        if n:
            peak = max(np.abs(want[o:o + n]).max(), 1e-30)
            worst = max(worst, np.abs(got[o:o + n] - want[o:o + n]).max() / peak)
        o += n
    return worst


# Tolerance (FP32 kernels against the FP64 restatement, max error relative to
# each channel's peak magnitude, for y, gx, gtaps and gcoefs): 1e-4.
Y_TOL = 1e-4
G_TOL = 1e-4


def _run_bank(lengths, taps, stages, x, h, c, gy):
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    bank = RaggedFilterBank(lengths, taps, stages)
    dev = "cuda"
    xt = torch.tensor(x, dtype=torch.float32, device=dev)
    ht = torch.tensor(h, dtype=torch.float32, device=dev)
    ct = torch.tensor(c, dtype=torch.float32, device=dev)
    gyt = torch.tensor(gy, dtype=torch.float32, device=dev)
    y = torch.empty(bank.sizes[0], device=dev)
    work = torch.empty(bank.sizes[3], device=dev)
    bank.forward_raw(xt, ht, ct, y, work)
    gx, gh, gc = torch.empty_like(xt), torch.empty_like(ht), torch.empty_like(ct)
    scratch = torch.empty(bank.sizes[4], device=dev)
    bank.backward_raw(xt, ht, ct, work, gyt, gx, gh, gc, scratch)
    torch.cuda.synchronize()
    return bank, [t.cpu().numpy().astype(np.float64) for t in (y, gx, gh, gc)]


def _check_bank(lengths, taps, stages, x, h, c, seed=0):
    rng = np.random.default_rng(seed + 99)
    # inputs as the GPU sees them (FP32-rounded), reference in FP64
    x = x.astype(np.float32).astype(np.float64)
    h = h.astype(np.float32).astype(np.float64)
    c = c.astype(np.float32).astype(np.float64)
    gy = rng.standard_normal(len(x)).astype(np.float32).astype(np.float64)
    out_len = [L - T + 1 for L, T in zip(lengths, taps)]
    gy_masked = gy.copy()
    o = 0
    for L, n in zip(lengths, out_len):
        gy_masked[o + n:o + L] = 0.0
        o += L
    bank, (y, gx, gh, gc) = _run_bank(lengths, taps, stages, x, h, c, gy)
    y64 = bank_forward(lengths, taps, stages, x, h, c)
    gx64, gh64, gc64 = bank_adjoint(lengths, taps, stages, x, h, c, gy_masked)
    # tail samples of y are zero
    o = 0
    for L, n in zip(lengths, out_len):
        assert np.all(y[o + n:o + L] == 0.0)
        o += L
    ey = _per_channel_err(lengths, lengths, y, y64)
    egx = _per_channel_err(lengths, lengths, gx, gx64)
    egh = _per_channel_err(lengths, taps, gh, gh64)
    egc = _per_channel_err(lengths, [5 * s for s in stages], gc, gc64)
    assert ey <= Y_TOL, ey
    assert egx <= G_TOL, egx
    assert egh <= G_TOL, egh
    assert egc <= G_TOL, egc
    return bank


@pytest.mark.gpu
def test_bank_small_mixed():
    _check_bank(*_bank_case(1, 12, Lrange=(16, 3000), Tmax=32, Smax=4,
                            force=[(1, 1, 2), (5, 5, 0), (7, 1, 0), (33, 32, 3), (200, 7, 1)]))


@pytest.mark.gpu
def test_bank_multi_window_long_channels():
    # channels longer than one 8192-sample scan window, deep cascades
    _check_bank(*_bank_case(2, 6, Lrange=(8000, 70000), Tmax=128, Smax=10,
                            force=[(8192 + 63, 64, 8), (16384, 1, 12), (8193, 2, 1)]))


@pytest.mark.gpu
def test_bank_long_taps():
    _check_bank(*_bank_case(3, 5, Lrange=(600, 5000), Tmax=512, Smax=3, force=[(512, 512, 2), (2600, 300, 1)]))


@pytest.mark.gpu
@pytest.mark.parametrize("T", [2, 65, 66, 193, 444, 512])
def test_bank_gradient_tile_edges(T):
    """Channels whose outputs end around a 64-sample row, a 1024-sample step, a 4096-sample
    gradient tile, an 8192-output FIR tile and a 16-tile run of the taps gradient; taps around
    the 128-position accumulator tiles, next to channels of few taps (accumulators of
    neighbouring runs); with two taps the gradient plane keeps the input's packing."""
    outs = [1, 63, 65, 1023, 1025, 4095, 4097, 8191, 8193, 12289, 16 * 8192 + 3]
    taps = [T if k % 3 else min(T, 3) for k in range(len(outs))]
    rng = np.random.default_rng(T)
    lengths = [n + t - 1 for n, t in zip(outs, taps)]
    stages = [k % 3 for k in range(len(outs))]
    x = rng.standard_normal(sum(lengths))
    h = np.concatenate([rng.standard_normal(t) / np.sqrt(t) for t in taps])
    c = np.concatenate([stable_sections(rng, S).reshape(-1) for S in stages])
    _check_bank(lengths, taps, stages, x, h, c, seed=T)


@pytest.mark.gpu
@pytest.mark.parametrize("S", [1, 4, 5, 9, 16, 17, 33, 64])
def test_bank_cascade_unit_edges(S):
    """Channels that end around a 16-sample chunk, a lane's 32 samples, a 1024-sample unit and a
    group of 32 units; stage counts around the adjoint's groups of four, the two chain
    kernels and a warp's entry states, next to channels without stages.  All-pass sections
    (poles of radius up to 0.6) keep every stage's signal at unit level; a stage's FP32
    rounding is a few 2^-24 / (1 - r) of it, 64 stages stay below the bar of 1e-4."""
    outs = [1, 16, 17, 32, 33, 1023, 1024, 1025, 2047, 2049, 32 * 1024, 32 * 1024 + 1, 5000]
    rng = np.random.default_rng(500 + S)
    taps = [1 + k % 4 for k in range(len(outs))]
    stages = [S if k != 3 else 0 for k in range(len(outs))]
    lengths = [n + t - 1 for n, t in zip(outs, taps)]
    x = rng.standard_normal(sum(lengths))
    h = np.concatenate([rng.standard_normal(t) / np.sqrt(t) + (np.arange(t) == 0) for t in taps])
    r, th = rng.uniform(0.2, 0.6, sum(stages)), rng.uniform(0.3, 2.8, sum(stages))
    a1, a2 = -2 * r * np.cos(th), r * r
    c = np.stack([a2, a1, np.ones_like(a1), a1, a2], 1).reshape(-1)
    _check_bank(lengths, taps, stages, x, h, c, seed=S)


@pytest.mark.gpu
def test_bank_many_channels():
    _check_bank(*_bank_case(4, 300, Lrange=(256, 4000), Tmax=64, Smax=6))


@pytest.mark.gpu
def test_backward_bitwise_repeatable():
    import torch

    lengths, taps, stages, x, h, c = _bank_case(5, 20, Lrange=(100, 9000), Tmax=48, Smax=5)
    gy = np.random.default_rng(7).standard_normal(len(x))
    _, a = _run_bank(lengths, taps, stages, x, h, c, gy)
    _, b = _run_bank(lengths, taps, stages, x, h, c, gy)
    for u, v in zip(a, b):
        assert np.array_equal(u, v)
    del torch


@pytest.mark.gpu
def test_autograd_and_graph_replay():
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    lengths, taps, stages, x, h, c = _bank_case(6, 16, Lrange=(100, 12000), Tmax=40, Smax=4)
    bank = RaggedFilterBank(lengths, taps, stages)
    dev = "cuda"
    xt = torch.tensor(x, dtype=torch.float32, device=dev, requires_grad=True)
    ht = torch.tensor(h, dtype=torch.float32, device=dev, requires_grad=True)
    ct = torch.tensor(c, dtype=torch.float32, device=dev, requires_grad=True)
    target = torch.randn(bank.sizes[0], device=dev)
    mask = bank.output_mask(dev)
    n = mask.sum()
    y = bank.apply(xt, ht, ct)
    loss = (((y - target) * mask) ** 2).sum() / n
    loss.backward()
    # same step captured in a CUDA graph
    xs, hs, cs = xt.detach().clone(), ht.detach().clone(), ct.detach().clone()
    replay, out = bank.graph_step(xs, hs, cs, target)
    replay()
    torch.cuda.synchronize()
    assert torch.allclose(out["loss"], loss.detach(), rtol=1e-5, atol=0)
    assert torch.allclose(out["gx"], xt.grad, rtol=1e-5, atol=1e-9)
    assert torch.allclose(out["gtaps"], ht.grad, rtol=1e-5, atol=1e-9)
    assert torch.allclose(out["gcoefs"], ct.grad, rtol=1e-5, atol=1e-9)
    # replay after refilling the inputs in place follows the new values
    xs.mul_(0.5)
    replay()
    torch.cuda.synchronize()
    y2 = bank.apply(xs, hs, cs).detach()
    assert torch.allclose(out["y"], y2, rtol=0, atol=0)


@pytest.mark.gpu
def test_mse_grad():
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    lengths, taps, stages = [5000, 64, 3000, 9000], [16, 64, 1, 200], [1, 0, 2, 3]
    bank = RaggedFilterBank(lengths, taps, stages)
    rng = np.random.default_rng(12)
    y = rng.standard_normal(bank.sizes[0]).astype(np.float32)
    t = rng.standard_normal(bank.sizes[0]).astype(np.float32)
    yd, td = torch.from_numpy(y).cuda(), torch.from_numpy(t).cuda()
    gy = torch.full_like(yd, 7.0)
    loss = torch.empty(1, device="cuda")
    scratch = torch.empty(bank.sizes[4], device="cuda")
    bank.mse_grad_raw(yd, td, gy, loss, scratch)
    torch.cuda.synchronize()
    mask = bank.output_mask("cpu").numpy() > 0
    n = int(mask.sum())
    assert n == bank.sizes[5]
    d = (y - t).astype(np.float32)
    want_gy = np.where(mask, np.float32(2.0 / n) * d, np.float32(0.0))
    assert np.array_equal(gy.cpu().numpy(), want_gy)
    want = float(np.sum(d[mask].astype(np.float64) ** 2) / n)
    assert float(loss.item()) == pytest.approx(want, rel=1e-6)


# ------------------------------------------------------------------ poles near the unit circle


def _fp32_channel_step(x, h, c, gy):
    """The same step in sequential FP32 (numpy / scipy single-precision recursions): the
    error an FP32 implementation of this filter makes anyway, the yardstick for the
    bound below."""
    from scipy.signal import lfilter

    f = np.float32
    u = np.convolve(x.astype(f), h.astype(f), "valid").astype(f)
    coefs = np.asarray(c, f).reshape(-1, 5)
    acts = [u]
    for b0, b1, b2, a1, a2 in coefs:
        acts.append(lfilter(np.array([b0, b1, b2], f), np.array([1, a1, a2], f), acts[-1]).astype(f))
    g = gy.astype(f)
    gc = np.zeros_like(coefs)
    for s in range(len(coefs) - 1, -1, -1):
        b0, b1, b2, a1, a2 = coefs[s]
        uu, yy = acts[s], acts[s + 1]
        v = lfilter(np.array([1], f), np.array([1, a1, a2], f), g[::-1]).astype(f)[::-1]
        vp = np.concatenate([v, np.zeros(2, f)])
        g = (b0 * vp[:-2] + b1 * vp[1:-1] + b2 * vp[2:]).astype(f)
        gc[s] = [v @ uu, v[1:] @ uu[:-1], v[2:] @ uu[:-2], -(v[1:] @ yy[:-1]), -(v[2:] @ yy[:-2])]
    gx = np.convolve(g, h.astype(f)[::-1], "full").astype(f)
    gh = np.correlate(x.astype(f), g, "valid")[::-1].astype(f)
    return acts[-1], gx, gh, gc.reshape(-1)


def _rel(got, want):
    return float(np.abs(np.asarray(got, np.float64) - want).max() / max(np.abs(want).max(), 1e-30))


@pytest.mark.gpu
@pytest.mark.parametrize("radius", [0.99, 0.995, 0.999])
def test_bank_poles_near_unit_circle(radius):
    """Every pole at radius 0.99 / 0.995 / 0.999 (the regime the FP64-formed transition
    powers exist for), channels of many scan segments, against FP64.  Bound per channel
    and quantity: max(1e-4, 4 x the error of the sequential FP32 step), the FP32
    recursion's own error growing like 1 / (1 - r)."""
    rng = np.random.default_rng(int(radius * 1000))
    lengths, taps, stages = [70000, 23000, 9000, 4200], [64, 17, 200, 1], [2, 3, 4, 1]
    x = rng.standard_normal(sum(lengths)).astype(np.float32).astype(np.float64)
    h = np.concatenate([rng.standard_normal(T) / np.sqrt(T) for T in taps]).astype(np.float32).astype(np.float64)
    c = np.concatenate([stable_sections(rng, S, radius=(radius, radius)).reshape(-1) for S in stages])
    c = c.astype(np.float32).astype(np.float64)
    gy = rng.standard_normal(len(x)).astype(np.float32).astype(np.float64)
    o = 0
    for L, T in zip(lengths, taps):
        gy[o + L - T + 1:o + L] = 0.0
        o += L
    bank, (y, gx, gh, gc) = _run_bank(lengths, taps, stages, x, h, c, gy)
    xo = ho = co = 0
    for L, T, S in zip(lengths, taps, stages):
        xs, hs, cs = x[xo:xo + L], h[ho:ho + T], c[co:co + 5 * S]
        gys = gy[xo:xo + L - T + 1]
        y64, _ = channel_forward(xs, hs, cs)
        gx64, gh64, gc64 = channel_adjoint(xs, hs, cs, gys)
        y32, gx32, gh32, gc32 = _fp32_channel_step(xs, hs, cs, gys)
        for name, got, want, seq in (("y", y[xo:xo + L - T + 1], y64, y32), ("gx", gx[xo:xo + L], gx64, gx32),
                                     ("gtaps", gh[ho:ho + T], gh64, gh32),
                                     ("gcoefs", gc[co:co + 5 * S], gc64.reshape(-1), gc32)):
            bound = max(1e-4, 4 * _rel(seq, want))
            assert _rel(got, want) <= bound, (radius, L, name, _rel(got, want), _rel(seq, want))
        xo, ho, co = xo + L, ho + T, co + 5 * S


@pytest.mark.gpu
@pytest.mark.parametrize("C,L,T,S", [(1, 5, 5, 1), (7, 1100, 64, 8), (5, 2049, 1, 64), (3, 5000, 17, 16), (2, 300000, 256, 4)])
def test_plan_sizes(C, L, T, S):
    """Work and scratch stay within the sizes that the header states."""
    from c7x_dsplib_b200.filterbank import SCRATCH, WORK, RaggedFilterBank

    sizes = RaggedFilterBank([L] * C, [T] * C, [S] * C).sizes
    out = L - T + 1
    units, groups = -(-out // 1024), -(-out // 32768)
    work = 4 * -(-out // 16) * 16 + 16 * units * S + 128 * S + 64 * S * (S + 1) + 8 * S * groups
    assert 4 * sizes[WORK] <= C * work + 6 * 16
    runs = -(-out // 8192)
    scratch = 4 * L + 36 * units * S + 8 * S * groups + 4 * 512 * runs
    assert 4 * sizes[SCRATCH] <= C * (scratch + 8 * units) + 8 * 16


def _bank_tensors(lengths, taps, stages, seed):
    """A bank and two sets of tensors for its calls: (bank, x, h, c, gy, sets), a set being
    y, work, gx, gtaps, gcoefs, scratch."""
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    bank = RaggedFilterBank(lengths, taps, stages)
    gen = torch.Generator("cuda").manual_seed(seed)
    n, nh, nk, nw, ns = (bank.sizes[k] for k in range(5))
    x, gy = (torch.randn(n, device="cuda", generator=gen) for _ in range(2))
    h = torch.randn(nh, device="cuda", generator=gen) / 4
    c = torch.tensor([0.5, 0.2, 0.1, -0.9, 0.4], device="cuda").repeat(nk // 5)
    sets = [[torch.empty(k, device="cuda") for k in (n, nw, n, nh, nk, ns)] for _ in range(2)]
    return bank, x, h, c, gy, sets


def _beside_a_capture(lengths, taps, stages):
    """Forward and adjoint of a plan, eager on another stream, while a capture that holds a forward of
    the same plan goes on: both give what they give alone."""
    import torch

    bank, x, h, c, gy, (a, b) = _bank_tensors(lengths, taps, stages, len(lengths))

    def call(t):
        bank.forward_raw(x, h, c, t[0], t[1])
        bank.backward_raw(x, h, c, t[1], gy, *t[2:])

    call(a)
    want = [t.clone() for t in (a[0], *a[2:5])]
    side = torch.cuda.Stream()
    for t in (*a, *b):
        t.fill_(7.0)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        bank.forward_raw(x, h, c, a[0], a[1])
        with torch.cuda.stream(side):
            call(b)
        bank.backward_raw(x, h, c, a[1], gy, *a[2:])
    g.replay()
    torch.cuda.synchronize()
    for t in (a, b):
        for u, v in zip((t[0], *t[2:5]), want):
            assert torch.equal(u, v)
    del g


@pytest.mark.gpu
def test_uniform_plan_eager_beside_a_capture():
    """One stage count, few samples: the eager calls stay on their stream altogether."""
    _beside_a_capture([3000] * 5, [17] * 5, [3] * 5)


@pytest.mark.gpu
@pytest.mark.parametrize("lengths", [[3000, 700, 5000, 1100], [600_000] * 4], ids=["small", "large"])
def test_plan_eager_beside_a_capture(lengths):
    """Several stage counts, and more samples than calls outside a capture leave on one stream."""
    _beside_a_capture(lengths, [17, 16, 3, 1], [3, 1, 2, 0])


@pytest.mark.gpu
@pytest.mark.parametrize("S", [5, 8, 17, 64])
def test_adjoint_stage_groups(S):
    """A channel's results do not depend on how many units the plan has, and so not on how many stages
    a unit of the adjoint keeps at once (all of them down to four)."""
    import torch

    want = None
    for more in (0, 300, 1000, 5000):  # units beside the channel's three
        bank, x, h, c, gy, (a, b) = _bank_tensors([3000, 1] + [1024] * more, [17, 1] + [1] * more, [S, 0] + [1] * more, S)
        rng = torch.Generator("cuda").manual_seed(S)
        x[:3000], gy[:3000] = (torch.randn(3000, device="cuda", generator=rng) for _ in range(2))
        h[:17] = torch.randn(17, device="cuda", generator=rng)
        bank.forward_raw(x, h, c, a[0], a[1])
        bank.backward_raw(x, h, c, a[1], gy, *a[2:])
        torch.cuda.synchronize()
        got = [t.clone() for t in (a[0][:3000], a[2][:3000], a[3][:17], a[4][:5 * S])]
        want = want or got
        for u, v in zip(got, want):
            assert torch.isfinite(u).all() and torch.equal(u, v), more


@pytest.mark.gpu
@pytest.mark.parametrize("v", [np.inf, np.nan])
def test_bank_not_finite_samples(v):
    """One sample of x and one of gy that are not finite, in channels without stages at any offset: of y
    and gx they spoil the rows of 64 whose window holds them (whole groups of 16 samples) and no more."""
    import torch

    taps = [1, 2, 17, 34, 64, 255, 512, 3, 130]
    lengths = [9001 + T + k for k, T in enumerate(taps)]
    bank, x, h, c, gy, (a, _) = _bank_tensors(lengths, taps, [0] * len(taps), 11)
    place = [0, 63, 64, 64 * 40 - 1, 64 * 128 - 2, 64 * 33 - 3, 700, 8191, 8999]
    results = []
    for bad in (False, True):
        if bad:
            for o, q in zip(bank.x_off, place):
                x[o + q] = gy[o + q] = v
        bank.forward_raw(x, h, c, a[0], a[1])
        bank.backward_raw(x, h, c, a[1], gy, *a[2:])
        results.append([t.cpu().numpy().copy() for t in (a[0], a[2])])
    for k, (T, L, q) in enumerate(zip(taps, lengths, place)):
        K = (63 + T + 15) // 16 * 16
        for got, want, n, start in zip(results[1], results[0], (L - T + 1, L), (0, -(T - 1))):
            got, want = (r[bank.x_off[k]:bank.x_off[k] + n] for r in (got, want))
            row = np.arange(n) // 64 * 64 + start
            clean = (q < row) | (q >= row + K)
            assert clean.any() and np.isfinite(got[clean]).all(), (k, start)
            assert np.abs(got[clean] - want[clean]).max() <= 1e-5 * np.abs(want).max(), (k, start)


@pytest.mark.gpu
@pytest.mark.parametrize("C,S", [(8, 3), (74, 8), (75, 8), (49, 9), (50, 9)])
def test_captured_step_beside_and_in_turn(C, S):
    """Captured steps of plans whose tables are made beside the FIR and of plans just too large for that
    (one run a channel on 148 SMs) equal the eager calls."""
    import torch

    bank, x, h, c, target, (a, b) = _bank_tensors([1500] * C, [20] * C, [S] * C, C)
    y, work, gx, gh, gc, scratch = a
    gy, loss = torch.empty_like(x), torch.empty(1, device="cuda")
    bank.step_mse_raw(x, h, c, target, y, gy, loss, gx, gh, gc, work, scratch)
    replay, out = bank.graph_step(x, h, c, target)
    for t in out.values():
        t.fill_(7.0)
    replay()
    torch.cuda.synchronize()
    for k, t in (("y", y), ("gx", gx), ("gtaps", gh), ("gcoefs", gc), ("loss", loss)):
        assert torch.equal(out[k], t), k


@pytest.mark.gpu
def test_plan_in_two_captures_at_once():
    import torch

    bank, x, h, c, gy, sets = _bank_tensors([3000, 700, 5000], [17, 16, 3], [3, 1, 2], 4)

    def call(t):
        bank.forward_raw(x, h, c, t[0], t[1])
        bank.backward_raw(x, h, c, t[1], gy, *t[2:])

    call(sets[0])
    want = [t.clone() for t in (sets[0][0], *sets[0][2:5])]
    streams, graphs = [torch.cuda.Stream() for _ in sets], [torch.cuda.CUDAGraph() for _ in sets]
    for t in (*sets[0], *sets[1]):
        t.fill_(7.0)
    torch.cuda.synchronize()
    for s, g in zip(streams, graphs):
        with torch.cuda.stream(s):
            g.capture_begin(capture_error_mode="relaxed")
    for _ in range(2):  # in turn
        for s, t in zip(streams, sets):
            with torch.cuda.stream(s):
                call(t)
    for s, g in zip(streams, graphs):
        with torch.cuda.stream(s):
            g.capture_end()
    for g in graphs:
        g.replay()
    torch.cuda.synchronize()
    for t in sets:
        for u, v in zip((t[0], *t[2:5]), want):
            assert torch.equal(u, v)
    del graphs


@pytest.mark.gpu
@pytest.mark.parametrize("L,radius,start", [(3000, 1.1, 2600), (2100, 1.12, 1700), (100_000, 1.003, 85_000)])
def test_bank_unstable_cascades_before_the_signal_begins(L, radius, start):
    """Poles outside the unit circle and a signal (for the adjoint: a gradient) of zeros but for its last
    (first) samples: finite and as exact as ever, although the response over a unit, or over 32 of them,
    is beyond FP32."""
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    rng = np.random.default_rng(L)
    S, th = 2, 0.7
    bank = RaggedFilterBank([L], [1], [S])
    c = np.array([[1.0, 0.3, 0.2, -2 * radius * np.cos(th), radius * radius], [0.8, -0.1, 0.1, -0.9, 0.4]], np.float32)
    x, gy = np.zeros(L, np.float32), np.zeros(L, np.float32)
    x[start:] = rng.standard_normal(L - start)
    gy[:L - start] = rng.standard_normal(L - start)
    d = [torch.tensor(a, device="cuda") for a in (x, np.ones(1, np.float32), c.reshape(-1), gy)]
    y, work = torch.empty(L, device="cuda"), torch.empty(bank.sizes[3], device="cuda")
    gx, gh, gc = (torch.empty_like(t) for t in d[:3])
    bank.forward_raw(*d[:3], y, work)
    bank.backward_raw(*d[:3], work, d[3], gx, gh, gc, torch.empty(bank.sizes[4], device="cuda"))
    h64 = np.ones(1)
    y64 = bank_forward([L], [1], [S], x.astype(np.float64), h64, c.astype(np.float64).reshape(-1))
    gx64 = bank_adjoint([L], [1], [S], x.astype(np.float64), h64, c.astype(np.float64).reshape(-1), gy.astype(np.float64))[0]
    for got, want in ((y, y64), (gx, gx64)):
        got = got.cpu().numpy().astype(np.float64)
        assert np.isfinite(want).all() and np.isfinite(got).all()
        assert np.abs(got - want).max() <= Y_TOL * np.abs(want).max()


@pytest.mark.gpu
def test_bank_deep_cascades_beyond_shared_memory():
    """24 and 22 stages beside shallow ones: the unit transitions of deep cascades
    (48 x 48 state) and the adjoint's per-stage sequences in shared memory."""
    lengths, taps, stages, x, h, c = _bank_case(8, 5, Lrange=(2000, 12000), Tmax=32, Smax=4,
                                                force=[(9000, 16, 24), (3000, 3, 22)])
    _check_bank(lengths, taps, stages, x, h, c)


@pytest.mark.gpu
def test_fused_step_equals_separate_calls():
    """DSPLIB_gpu_firBiquadBatched_stepMse against forward + MSE + adjoint as three calls:
    y, gy and every gradient bitwise equal, the loss to FP64 summation order."""
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    lengths, taps, stages, x, h, c = _bank_case(13, 20, Lrange=(100, 30000), Tmax=96, Smax=6,
                                                force=[(70000, 33, 4), (600, 1, 0)])
    bank = RaggedFilterBank(lengths, taps, stages)
    dev = "cuda"
    xt, ht, ct = (torch.tensor(a, dtype=torch.float32, device=dev) for a in (x, h, c))
    target = torch.randn(bank.sizes[0], device=dev, generator=torch.Generator(dev).manual_seed(3))
    n = bank.sizes[0]
    sep = {k: torch.empty(n, device=dev) for k in ("y", "gy", "gx")}
    sep["gtaps"], sep["gcoefs"] = torch.empty_like(ht), torch.empty_like(ct)
    sep["loss"] = torch.empty(1, device=dev)
    work = torch.empty(bank.sizes[3], device=dev)
    scratch = torch.empty(bank.sizes[4], device=dev)
    bank.forward_raw(xt, ht, ct, sep["y"], work)
    bank.mse_grad_raw(sep["y"], target, sep["gy"], sep["loss"], scratch)
    bank.backward_raw(xt, ht, ct, work, sep["gy"], sep["gx"], sep["gtaps"], sep["gcoefs"], scratch)
    fus = {k: torch.full_like(v, 7.0) for k, v in sep.items()}
    work2 = torch.empty_like(work)
    scratch2 = torch.empty_like(scratch)
    bank.step_mse_raw(xt, ht, ct, target, fus["y"], fus["gy"], fus["loss"], fus["gx"], fus["gtaps"],
                      fus["gcoefs"], work2, scratch2)
    torch.cuda.synchronize()
    for k in ("y", "gy", "gx", "gtaps", "gcoefs"):
        assert torch.equal(fus[k], sep[k]), k
    assert float(fus["loss"]) == pytest.approx(float(sep["loss"]), rel=1e-6)


@pytest.mark.gpu
@pytest.mark.parametrize("pinned", [True, False])
def test_host_step_equals_device_step(pinned):
    """DSPLIB_gpu_firBiquadBatched_stepMseHost on host tensors (several pipelined channel
    segments: 7.3 M samples at 2 M samples per segment) against the device call:
    y, gy and every gradient bitwise equal, the loss to FP64 summation order; twice in a
    row, then with gy omitted and the taps / coefficients left on the device."""
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    lengths, taps, stages, x, h, c = _bank_case(21, 60, Lrange=(1000, 240000), Tmax=300, Smax=8,
                                                force=[(262144, 512, 8), (300, 300, 0)])
    bank = RaggedFilterBank(lengths, taps, stages)
    assert bank.sizes[0] > 6_000_000
    dev = "cuda"
    xt, ht, ct = (torch.tensor(a, dtype=torch.float32, device=dev) for a in (x, h, c))
    target = torch.randn(bank.sizes[0], device=dev, generator=torch.Generator(dev).manual_seed(5))
    n = bank.sizes[0]
    ref = {k: torch.empty(n, device=dev) for k in ("y", "gy", "gx")}
    ref["gtaps"], ref["gcoefs"], ref["loss"] = torch.empty_like(ht), torch.empty_like(ct), torch.empty(1, device=dev)
    bank.step_mse_raw(xt, ht, ct, target, ref["y"], ref["gy"], ref["loss"], ref["gx"], ref["gtaps"], ref["gcoefs"],
                      torch.empty(bank.sizes[3], device=dev), torch.empty(bank.sizes[4], device=dev))
    torch.cuda.synchronize()
    ref = {k: v.cpu() for k, v in ref.items()}

    def host(t):
        t = t.cpu()
        return t.pin_memory() if pinned else t.clone()

    hx, hh, hc, ht_ = host(xt), host(ht), host(ct), host(target)
    for rep in range(3):
        out = {k: host(torch.full_like(v, 7.0)) for k, v in ref.items()}
        taps_in, coefs_in, gy_out = (hh, hc, out["gy"]) if rep < 2 else (ht, ct, None)
        if rep == 2:
            out["gtaps"], out["gcoefs"] = torch.full_like(ht, 7.0), torch.full_like(ct, 7.0)
        bank.step_mse_host(hx, taps_in, coefs_in, ht_, out["y"], gy_out, out["loss"], out["gx"], out["gtaps"],
                           out["gcoefs"])
        for k in ("y", "gy", "gx", "gtaps", "gcoefs"):
            if k == "gy" and gy_out is None:
                continue
            assert torch.equal(out[k].cpu(), ref[k]), (rep, k)
        assert float(out["loss"]) == pytest.approx(float(ref["loss"]), rel=1e-6)


@pytest.mark.gpu
def test_host_step_async_two_plans_in_flight():
    """Two plans of the same bank, each DSPLIB_gpu_raggedPlanSetAsync(plan, 1), calls queued
    on two streams before either finishes (one call's copies out overlap the next's copies
    in), three rounds: every result bitwise equal to the device step's."""
    import torch

    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    lengths, taps, stages, x, h, c = _bank_case(22, 40, Lrange=(1000, 240000), Tmax=300, Smax=6)
    dev = "cuda"
    xt, ht, ct = (torch.tensor(a, dtype=torch.float32, device=dev) for a in (x, h, c))
    ref_bank = RaggedFilterBank(lengths, taps, stages)
    target = torch.randn(ref_bank.sizes[0], device=dev, generator=torch.Generator(dev).manual_seed(9))
    n = ref_bank.sizes[0]
    ref = {k: torch.empty(n, device=dev) for k in ("y", "gy", "gx")}
    ref["gtaps"], ref["gcoefs"], ref["loss"] = torch.empty_like(ht), torch.empty_like(ct), torch.empty(1, device=dev)
    ref_bank.step_mse_raw(xt, ht, ct, target, ref["y"], ref["gy"], ref["loss"], ref["gx"], ref["gtaps"],
                          ref["gcoefs"], torch.empty(ref_bank.sizes[3], device=dev),
                          torch.empty(ref_bank.sizes[4], device=dev))
    torch.cuda.synchronize()
    ref = {k: v.cpu() for k, v in ref.items()}
    hx, hh, hc, htg = (t.cpu().pin_memory() for t in (xt, ht, ct, target))
    banks = [RaggedFilterBank(lengths, taps, stages) for _ in range(2)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    outs = []
    for b in banks:
        assert b.set_async(True) == 0
        outs.append({k: torch.full(v.shape, 7.0).pin_memory() for k, v in ref.items() if k != "gy"})
    for rnd in range(3):
        for b, st, o in zip(banks, streams, outs):
            st.synchronize()  # this slot's previous call finished: its buffers may be reused
            with torch.cuda.stream(st):
                b.step_mse_host(hx, hh, hc, htg, o["y"], None, o["loss"], o["gx"], o["gtaps"], o["gcoefs"])
        for b, st, o in zip(banks, streams, outs):
            st.synchronize()
            assert b.status() == 0
            for k in ("y", "gx", "gtaps", "gcoefs"):
                assert torch.equal(o[k], ref[k]), (rnd, k)
            assert float(o["loss"]) == pytest.approx(float(ref["loss"]), rel=1e-6)
