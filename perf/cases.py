"""Performance cases of the filtering path, through its public entry points.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges;
``prepare`` makes what a program holds before the call (device inputs from a seed, handles,
plans, graphs), ``run`` is one pass, ``work`` the bytes and operations a pass cannot do
without and ``exact`` its results in 64 bits, without this package.

Kinds of case:

* ``stream``     ``FirStream.exec``: one block of a running overlap-save filter (integer
                 blocks as an audio or radio front end feeds them).
* ``fir``        ``FirHandle.exec``: a whole batch of channels, int8 / int16 (Q mode or the
                 natural-C wrap) or FP32 (plain or split-BF16), shared or per-channel taps.
* ``fir_train``  ``torch.ops.dsplib_gpu.fir`` forward and backward: an FIR layer whose taps
                 and input both take gradients.
* ``biquad``     ``BiquadHandle.exec``: one block of a running biquad cascade (the state
                 carries over from pass to pass), any form, shared or per-channel coefficients.
* ``bank_grad``  ``RaggedFilterBank.apply`` and ``torch.autograd.grad``: the uneven
                 FIR -> biquad bank inside a larger differentiable program.
* ``bank_step``  ``RaggedFilterBank.graph_step``: its training step (forward, loss, adjoint)
                 replayed from a CUDA graph.
* ``frontend``   interleaved Q.15 frames to float channel rows and back: deinterleave,
                 q15tofl, fltoq15, interleave.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import c7x_dsplib_b200 as D

FORMS = {"tif": D.TIF, "df1": D.DF1, "df2": D.DF2, "tdf2": D.TDF2}
INTS = {"int8": (D.INT8, torch.int8, 8), "int16": (D.INT16, torch.int16, 16)}
TIF_GROUP = 7  # stages per gain group of the transposed-form coefficients


# ----------------------------------------------------------------- the cases


def listed():
    return [
        # the smallest calls: one block of a 16-channel Q15 stream, 64 shared taps
        dict(name="stream_i16_small", kind="stream", dtype="int16", channels=16, block=4096, taps=64, nch=False,
             qmode=True),
        # int8 batch at the benchmark's size, Q7 output
        dict(name="fir_i8_large", kind="fir", dtype="int8", channels=4096, samples=16384, taps=128, nch=False,
             qmode=True, split=False),
        # int16, natural-C wrap, every channel its own taps; odd row length (unaligned rows)
        dict(name="fir_i16_odd_rows", kind="fir", dtype="int16", channels=1000, samples=10007, taps=201, nch=True,
             qmode=False, split=False),
        # FP32 at the default precision, a middling batch with per-channel taps
        dict(name="fir_f32_plain", kind="fir", dtype="float32", channels=256, samples=32768, taps=255, nch=True,
             qmode=False, split=False),
        # FP32 on the tensor cores (split-BF16), the benchmark's size
        dict(name="fir_f32_split", kind="fir", dtype="float32", channels=1024, samples=65536, taps=256, nch=True,
             qmode=False, split=True),
        # an FIR layer in training: forward and both gradients
        dict(name="fir_layer_train", kind="fir_train", channels=64, samples=16384, taps=128, nch=True),
        # one block of 32 channels: a latency-bound call
        dict(name="biquad_small", kind="biquad", form="df2", channels=32, samples=8192, stages=4, nch=False),
        # a full batch of channels
        dict(name="biquad_large", kind="biquad", form="df2", channels=4096, samples=8192, stages=4, nch=False),
        # ragged in every size, per-channel coefficients in the reference's own transposed form
        dict(name="biquad_odd_tif", kind="biquad", form="tif", channels=203, samples=20011, stages=7, nch=True),
        # a middling bank differentiated by autograd (forward call, backward call)
        dict(name="bank_grad_256", kind="bank_grad", channels=256, shortest=256, longest=262144),
        # the benchmark's bank: one training step over 2048 uneven channels
        dict(name="bank_step_2048", kind="bank_step", channels=2048, shortest=256, longest=262144),
        # stereo Q.15 frames to float rows and back
        dict(name="frontend_stereo", kind="frontend", channels=2, frames=8 << 20),
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], uniform in its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["stream", "fir", "fir", "fir", "fir_train", "biquad", "biquad", "bank_grad", "bank_step",
                       "frontend"])
    if kind == "stream":
        return dict(kind=kind, dtype=rng.choice(["int8", "int16"]), channels=_log(rng, 1, 64),
                    block=_log(rng, 64, 8192), taps=rng.randint(8, 256), nch=rng.random() < 0.5,
                    qmode=rng.random() < 0.5)
    if kind == "fir":
        dtype = rng.choice(["int8", "int16", "float32", "float32"])
        samples = _log(rng, 1024, 65536)
        channels = _log(rng, 16, max(16, min(4096, (1 << 26 if dtype != "float32" else 1 << 24) // samples)))
        return dict(kind=kind, dtype=dtype, channels=channels, samples=samples, taps=rng.randint(16, 256),
                    nch=rng.random() < 0.5, qmode=dtype != "float32" and rng.random() < 0.5,
                    split=dtype == "float32" and rng.random() < 0.5)
    if kind == "fir_train":
        return dict(kind=kind, channels=_log(rng, 4, 256), samples=_log(rng, 1024, 16384), taps=rng.randint(16, 256),
                    nch=rng.random() < 0.5)
    if kind == "biquad":
        samples = _log(rng, 256, 32768)
        return dict(kind=kind, form=rng.choice(sorted(FORMS)), channels=_log(rng, 1, min(4096, (1 << 25) // samples)),
                    samples=samples, stages=rng.randint(1, 8), nch=rng.random() < 0.5)
    if kind in ("bank_grad", "bank_step"):
        longest = _log(rng, 4096, 262144)
        return dict(kind=kind, channels=_log(rng, 8, 512), shortest=rng.randint(256, 1024), longest=longest)
    return dict(kind="frontend", channels=rng.choice([2, 3, 4, 8]), frames=_log(rng, 4096, 1 << 21))


# ----------------------------------------------------------------- inputs


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gen(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=_device())


def _int(g, dtype, *shape):
    """Full-range samples of an integer type."""
    _, td, bits = INTS[dtype]
    return torch.randint(-(1 << (bits - 1)), 1 << (bits - 1), shape, generator=g, device=_device(), dtype=td)


def _lowpass(rng, rows, T):
    """Windowed-sinc low-pass taps, cutoff U[0.05, 0.45] of Nyquist, unit gain at DC; stored order."""
    n = np.arange(T) - (T - 1) / 2.0
    fc = rng.uniform(0.05, 0.45, (rows, 1))
    h = fc * np.sinc(fc * n) * np.hamming(T)
    return (h / h.sum(axis=1, keepdims=True))[:, ::-1].astype(np.float32)


def _sections(rng, n, rmax):
    """n stable sections [b0 b1 b2 a1 a2]: conjugate poles of radius U[0.5, rmax], zeros in the
    unit disc, gain about 1 at DC."""
    r, th = rng.uniform(0.5, rmax, n), rng.uniform(0.05, math.pi - 0.05, n)
    rz, tz = rng.uniform(0, 1, n), rng.uniform(0, math.pi, n)
    a1, a2 = -2 * r * np.cos(th), r * r
    b = np.stack([np.ones(n), -2 * rz * np.cos(tz), rz * rz], 1)
    b *= ((1 + a1 + a2) / np.maximum(np.abs(b.sum(1)), 0.2))[:, None]
    return np.concatenate([b, a1[:, None], a2[:, None]], 1).astype(np.float32)


def _fir_inputs(case, seed):
    """(x, stored taps, Q-mode shift) of a stream, fir or fir_train case."""
    C, T, dtype = case["channels"], case["taps"], case.get("dtype", "float32")
    N = case["block"] if case["kind"] == "stream" else case["samples"]
    rows = C if case["nch"] else 1
    g = _gen(seed)
    if dtype == "float32":
        h = torch.from_numpy(_lowpass(np.random.default_rng(seed), rows, T)).to(_device())
        return _randn(g, C, N), h, 0
    return _int(g, dtype, C, N), _int(g, dtype, rows, T), INTS[dtype][2] - 1


def _biquad_inputs(case, seed):
    """(x [N, C], natural coefficients [1 or C, 5 S])."""
    C, N, S = case["channels"], case["samples"], case["stages"]
    rows = C if case["nch"] else 1
    nat = _sections(np.random.default_rng(seed), rows * S, 0.95).reshape(rows, 5 * S)
    return _randn(_gen(seed), N, C), nat


def _bank_shape(case):
    """Channel lengths (log-uniform), taps and stages of a bank: part of the case, not of the inputs."""
    C = case["channels"]
    rng = np.random.default_rng(5)
    lengths = np.exp(rng.uniform(math.log(case["shortest"]), math.log(case["longest"]), C)).astype(np.int64)
    taps = np.minimum(rng.integers(32, 512, size=C, endpoint=True), lengths)
    return lengths, taps, rng.integers(2, 8, size=C, endpoint=True)


def _bank_inputs(case, seed):
    """(x, taps, coefficients, target or output gradient), packed."""
    lengths, taps, stages = _bank_shape(case)
    rng, g = np.random.default_rng(seed), _gen(seed)
    n = int(lengths.sum())
    scale = np.repeat(1 / np.sqrt(taps), taps)
    h = torch.from_numpy((rng.standard_normal(int(taps.sum())) * scale).astype(np.float32)).to(_device())
    c = torch.from_numpy(_sections(rng, int(stages.sum()), 0.98).reshape(-1)).to(_device())
    return _randn(g, n), h, c, _randn(g, n)


# ----------------------------------------------------------------- one pass


def prepare(case, seed):
    return {"kind": case["kind"], **globals()["_prepare_" + case["kind"]](case, seed)}


def run(state):
    return globals()["_run_" + state["kind"]](state)


def _prepare_stream(case, seed):
    x, h, shift = _fir_inputs(case, seed)
    s = D.FirStream(INTS[case["dtype"]][0], case["channels"], case["block"], case["taps"], nch=case["nch"],
                    shift=shift, qmode=case["qmode"])
    D.lib().DSPLIB_gpu_setAsync(s.h, 1)
    return dict(stream=s, x=x, h=h, y=torch.empty_like(x))


def _run_stream(s):
    return s["stream"].exec(s["x"], s["h"], s["y"])


def _prepare_fir(case, seed):
    x, h, shift = _fir_inputs(case, seed)
    code = {torch.int8: D.INT8, torch.int16: D.INT16, torch.float32: D.FLOAT32}[x.dtype]
    C, N, T = case["channels"], case["samples"], case["taps"]
    handle = D.FirHandle()
    handle._check("init", handle.init(*D.fir_setup(code, C, N, T, nch=case["nch"], shift=shift)))
    handle.set_precision(D.FIR_BF16X3 if case["split"] else D.FIR_SIMT)
    handle.set_qmode(case["qmode"])
    handle.set_async(True)
    return dict(handle=handle, x=x, h=h, y=torch.empty((C, N - T + 1), dtype=x.dtype, device=x.device))


def _run_fir(s):
    s["handle"]._check("exec", s["handle"].exec(s["x"], s["h"], s["y"]))
    return s["y"]


def _prepare_fir_train(case, seed):
    import c7x_dsplib_b200.torch_ops  # noqa: F401  (registers the operators)

    x, h, _ = _fir_inputs(case, seed)
    gy = _randn(_gen(seed + 7), case["channels"], case["samples"] - case["taps"] + 1)
    return dict(x=x.requires_grad_(), h=h.requires_grad_(), gy=gy, nch=case["nch"])


def _run_fir_train(s):
    y = torch.ops.dsplib_gpu.fir(s["x"], s["h"], s["nch"], D.FIR_SIMT, False, 0)
    gx, gh = torch.autograd.grad(y, (s["x"], s["h"]), s["gy"])
    return y.detach(), gx, gh


def _prepare_biquad(case, seed):
    x, nat = _biquad_inputs(case, seed)
    form, C, N, S = FORMS[case["form"]], case["channels"], case["samples"], case["stages"]
    opt, popt = D.opt_coefficients(nat, form, int(case["nch"]), C)
    args, pin, pout, pvar, _, _ = D.biquad_descs(C, N, S, form, int(case["nch"]))
    handle = D.BiquadHandle()
    handle._check("init", handle.init(args, pin, popt, pvar, pout))
    handle.set_async(True)
    state = torch.zeros((S * (4 if form == D.DF1 else 2), C), device=x.device)
    return dict(handle=handle, x=x, coef=torch.from_numpy(opt).to(x.device), state=state, y=torch.empty_like(x))


def _run_biquad(s):
    s["handle"]._check("exec", s["handle"].exec(s["x"], s["coef"], s["state"], s["y"]))
    return s["y"], s["state"]


def _prepare_bank_grad(case, seed):
    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    x, h, c, gy = _bank_inputs(case, seed)
    return dict(bank=RaggedFilterBank(*_bank_shape(case)), x=x.requires_grad_(), h=h.requires_grad_(),
                c=c.requires_grad_(), gy=gy)


def _run_bank_grad(s):
    y = s["bank"].apply(s["x"], s["h"], s["c"])
    return (y.detach(), *torch.autograd.grad(y, (s["x"], s["h"], s["c"]), s["gy"]))


def _prepare_bank_step(case, seed):
    from c7x_dsplib_b200.filterbank import RaggedFilterBank

    x, h, c, target = _bank_inputs(case, seed)
    bank = RaggedFilterBank(*_bank_shape(case))
    replay, out = bank.graph_step(x, h, c, target)
    return dict(bank=bank, replay=replay, out=out, inputs=(x, h, c, target))


def _run_bank_step(s):
    s["replay"]()
    return s["out"]


def _prepare_frontend(case, seed):
    C, n = case["channels"], case["frames"]
    x = _int(_gen(seed), "int16", n, C)
    rows_q = torch.empty((C, n), dtype=torch.int16, device=x.device)
    rows = torch.empty((C, n), device=x.device)
    back_q, back = torch.empty_like(rows_q), torch.empty_like(x)
    style, conv = D.StyleInitArgs(funcStyle=D.OPTIMIZED), D.ConvertInitArgs(funcStyle=D.OPTIMIZED, dataSize=C * n)
    frames_d, rows_d = D.bp(D.INT16, C, n, 2 * C), D.bp(D.INT16, n, C, 2 * n)
    q_d, f_d = D.BufParams1D(D.INT16, C * n), D.BufParams1D(D.FLOAT32, C * n)
    calls = []
    for handle, args, pin, pout, src, dst in (
            (D.LayoutHandle("DSPLIB_deinterleave"), style, frames_d, rows_d, x, rows_q),
            (D.Q15toflHandle(), conv, q_d, f_d, rows_q, rows),
            (D.Fltoq15Handle(), conv, f_d, q_d, rows, back_q),
            (D.LayoutHandle("DSPLIB_interleave"), style, rows_d, frames_d, back_q, back)):
        handle._check("init", handle.init(args, pin, pout))
        handle.set_async(True)
        calls.append((handle, src, dst))
    return dict(calls=calls, rows=rows, back=back)


def _run_frontend(s):
    for handle, src, dst in s["calls"]:
        handle._check("exec", handle.exec(src, dst))
    return s["rows"], s["back"]


# ----------------------------------------------------------------- necessary work


def work(case):
    kind = case["kind"]
    if kind in ("stream", "fir", "fir_train"):
        C, T = case["channels"], case["taps"]
        e = {"int8": 1, "int16": 2, "float32": 4}[case.get("dtype", "float32")]
        N = case["block"] + T - 1 if kind == "stream" else case["samples"]
        out, rows = N - T + 1, C if case["nch"] else 1
        if kind == "fir_train":  # y = fir(x, h); gx from gy and h; gh from gy and x
            return {"bytes": 4.0 * (3 * C * N + 3 * C * out + 3 * rows * T), "flops": 6.0 * C * out * T}
        hist = 2 * C * (T - 1) if kind == "stream" else 0  # the history is read and written
        return {"bytes": float(e * (C * (N - hist // (2 * C)) + C * out + rows * T + hist)),
                "flops": 2.0 * C * out * T}
    if kind == "biquad":
        C, N, S = case["channels"], case["samples"], case["stages"]
        states = S * C * (4 if case["form"] == "df1" else 2)
        return {"bytes": 4.0 * (2 * C * N + 5 * S * (C if case["nch"] else 1) + 2 * states), "flops": 9.0 * C * N * S}
    if kind in ("bank_grad", "bank_step"):
        lengths, taps, stages = (v.astype(np.float64) for v in _bank_shape(case))
        out = lengths - taps + 1
        # x, y forward; target and gradient (loss); x, gradient and gx (adjoint)
        return {"bytes": float((20 if kind == "bank_step" else 16) * lengths.sum()),
                "flops": float((6 * taps * out + 27 * stages * out).sum())}
    n = case["channels"] * case["frames"]
    return {"bytes": 20.0 * n, "flops": 4.0 * n}  # 2 + 2, 2 + 4, 4 + 2 and 2 + 2 bytes a sample


# ----------------------------------------------------------------- 64-bit results


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _correlate(x, h, out):
    """sum_c x[:, j + c] h[:, T - 1 - c] in 64 bits (exact for the integer types)."""
    acc = torch.zeros((x.shape[0], out), dtype=torch.float64, device=x.device)
    x, h, T = x.double(), h.double(), h.shape[1]
    for c in range(T):
        acc += x[:, c:c + out] * h[:, T - 1 - c, None]
    return acc


def _to_int(acc, case, shift):
    _, td, bits = INTS[case["dtype"]]
    v = acc.to(torch.int64)
    if case["qmode"]:
        v = (v + (1 << (shift - 1))) >> shift
        return v.clamp(-(1 << (bits - 1)), (1 << (bits - 1)) - 1).to(td)
    return (((v + (1 << (bits - 1))) & ((1 << bits) - 1)) - (1 << (bits - 1))).to(td)


def _exact_fir(case, seed):
    x, h, shift = _fir_inputs(case, seed)
    acc = _correlate(x, h, case["samples"] - case["taps"] + 1)
    return acc if case["dtype"] == "float32" else _to_int(acc, case, shift)


def _exact_stream(case, seed):
    x, h, shift = _fir_inputs(case, seed)
    x = torch.nn.functional.pad(x.double(), (case["taps"] - 1, 0))  # the stream starts from zeros
    return _to_int(_correlate(x, h, case["block"]), case, shift)


def _exact_fir_train(case, seed):
    x, h, _ = _fir_inputs(case, seed)
    T, out = case["taps"], case["samples"] - case["taps"] + 1
    gy = _randn(_gen(seed + 7), case["channels"], out).double()
    gx = _correlate(torch.nn.functional.pad(gy, (T - 1, T - 1)), torch.flip(h, [1]), case["samples"])
    x64 = x.double()
    gh = torch.stack([(gy * x64[:, c:c + out]).sum(1) for c in range(T - 1, -1, -1)], 1)
    return _correlate(x, h, out), gx, gh if case["nch"] else gh.sum(0, keepdim=True)


DECAY = 4096  # samples after which a section's response (poles of radius at most 0.98) is nothing


def _grid(n):
    """An FFT length for n samples and the sections' decay."""
    return 1 << (n + DECAY - 1).bit_length()


def _z(M, dev):
    return torch.exp(-2j * math.pi * torch.arange(M // 2 + 1, dtype=torch.float64, device=dev) / M)


def _poly(c, z):
    return c[0] + z * (c[1] + z * c[2])


def _exact_biquad(case, seed):
    x, nat = _biquad_inputs(case, seed)
    C, N, S, form = case["channels"], case["samples"], case["stages"], case["form"]
    M = _grid(N)
    z = _z(M, x.device)[:, None]
    k = torch.from_numpy(nat).to(x.device).double().reshape(-1, S, 5).permute(1, 2, 0)  # [S, 5, 1 or C]
    one, zero = torch.ones_like(k[0, 0]), torch.zeros_like(k[0, 0])

    def filt(v, b, a):
        spec = torch.fft.rfft(v, M, dim=0)
        return torch.fft.irfft(spec * (_poly(b, z) / _poly((one, *a), z)), M, dim=0)[:N]

    v, states = x.double(), []
    for s in range(S):
        b, a = (k[s, 0], k[s, 1], k[s, 2]), (k[s, 3], k[s, 4])
        last = torch.nn.functional.pad(v, (0, 0, 2, 0))[-2:]
        if form == "df2":
            w = torch.nn.functional.pad(filt(v, (one, zero, zero), a), (0, 0, 2, 0))
            states += [w[-1], w[-2]]
            v = filt(v, b, a)
        elif form == "df1":
            v = filt(v, b, a)
            o = torch.nn.functional.pad(v, (0, 0, 2, 0))
            states += [last[1], last[0], o[-1], o[-2]]
        else:  # tdf2; tif is the same on sections of b0 = 1, the gain applied at the group's end
            if form == "tif":
                gain = b[0] if s % TIF_GROUP == 0 else gain * b[0]
                b = (one, b[1] / b[0], b[2] / b[0])
            v = filt(v, b, a)
            o = torch.nn.functional.pad(v, (0, 0, 2, 0))
            states += [b[1] * last[1] + b[2] * last[0] - a[0] * o[-1] - a[1] * o[-2], b[2] * last[1] - a[1] * o[-1]]
            if form == "tif" and (s % TIF_GROUP == TIF_GROUP - 1 or s == S - 1):
                v = v * gain
    return v, torch.stack([t.expand(C) for t in states])


def _bank_channel(x, h, c, grad_of):
    """One channel in 64 bits: y, its output gradient's adjoint (gx, gh, gc)."""
    L, T, Lu = len(x), len(h), len(x) - len(h) + 1
    M = _grid(L + T)
    z = _z(M, x.device)
    fx, fh = torch.fft.rfft(x, M), torch.fft.rfft(h, M)
    acts = [torch.fft.irfft(fx * fh, M)[T - 1:L]]
    spec = torch.fft.rfft(acts[0], M)
    for k in c:
        spec = spec * (_poly(k[:3], z) / (1 + z * (k[3] + z * k[4])))
        acts.append(torch.fft.irfft(spec, M)[:Lu])
    y, gc = acts[-1], []
    spec = torch.fft.rfft(torch.flip(grad_of(y), [0]), M)  # the adjoint runs back in time
    for s in range(len(c) - 1, -1, -1):
        k = c[s]
        spec = spec / (1 + z * (k[3] + z * k[4]))
        v = torch.flip(torch.fft.irfft(spec, M)[:Lu], [0])
        u, o = acts[s], acts[s + 1]
        gc.insert(0, torch.stack([v @ u, v[1:] @ u[:-1], v[2:] @ u[:-2], -(v[1:] @ o[:-1]), -(v[2:] @ o[:-2])]))
        spec = spec * _poly(k[:3], z)
    g = torch.flip(torch.fft.irfft(spec, M)[:Lu], [0])
    fg = torch.fft.rfft(g, M)
    gx = torch.fft.irfft(fg * torch.fft.rfft(torch.flip(h, [0]), M), M)[:L]
    gh = torch.flip(torch.fft.irfft(fx * fg.conj(), M)[:T], [0])
    return y, gx, gh, torch.cat(gc)


def _exact_bank(case, seed, grad_of):
    lengths, taps, stages = (v.tolist() for v in _bank_shape(case))
    x, h, c, t = (v.double() for v in _bank_inputs(case, seed))
    y, gx, gh, gc = torch.zeros_like(x), torch.empty_like(x), torch.empty_like(h), torch.empty_like(c)
    xo = ho = co = 0
    for L, T, S in zip(lengths, taps, stages):
        Lu = L - T + 1
        got = _bank_channel(x[xo:xo + L], h[ho:ho + T], c[co:co + 5 * S].reshape(S, 5),
                            lambda v: grad_of(v, t[xo:xo + Lu]))
        y[xo:xo + Lu], gx[xo:xo + L], gh[ho:ho + T], gc[co:co + 5 * S] = got
        xo, ho, co = xo + L, ho + T, co + 5 * S
    return y, gx, gh, gc


def _exact_bank_grad(case, seed):
    return _exact_bank(case, seed, lambda y, gy: gy)


def _exact_bank_step(case, seed):
    lengths, taps, _ = _bank_shape(case)
    n, sq = float((lengths - taps + 1).sum()), []

    def grad(y, target):
        sq.append((y - target).square().sum())
        return (2 / n) * (y - target)

    y, gx, gh, gc = _exact_bank(case, seed, grad)
    return {"loss": (sum(sq) / n).reshape(1), "y": y, "gx": gx, "gtaps": gh, "gcoefs": gc}


def _exact_frontend(case, seed):
    x = _int(_gen(seed), "int16", case["frames"], case["channels"])
    return x.t().double() / 32768, x
