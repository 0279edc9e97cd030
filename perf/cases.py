"""The work a user has this framework do, as cases that can be timed.

Each case is a dict of plain values; :func:`prepare` makes what the user's program holds before the call (inputs from a
seed, planned and uploaded batches, handles), :func:`run` is one pass through the public entry points, :func:`work` what
such a pass cannot do without.  Source parameters are the benchmark's draws (``emri_kludge_suite_b200.workloads``), the
likelihood's templates the benchmark's fiducial source and its neighbourhood.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from emri_kludge_suite_b200 import aak, workloads
from emri_kludge_suite_b200.gpuAAK import GPUAAK
from emri_kludge_suite_b200.LISAnoise import LISA_Noise, generate_noise_frequencies, generate_noise_single_channel
from emri_kludge_suite_b200.parmap_mlp import ParMapMLP, init_params, input_features

DT = workloads.DT
# gpu_gen_AAK order: iota, s, p, e, M, mu, gamma, psi, alph, theta_S, phi_S, theta_K, phi_K, D
FIDUCIAL = (0.785, 0.5, 8.0, 0.2, 1e6, 10.0, 0.0, 0.0, 0.0, 0.5, 1.0, 0.8, 2.0, 1.0)


def listed():
    return [
        # AAKwrapper.wave of one short source: host parameters in, host arrays out; the call of a user's first script
        dict(name="wave_one", kind="wave", length=20011, lisa=True, backint=False),
        # a handful of short sources on the device (snapshots, a sampler's few walkers): launches and latency count;
        # detector-frame response, integrated backwards from the plunge end
        dict(name="waves_few", kind="batch", nsrc=4, lo=4001, hi=20011, e_max=0.5, precision=0, graph=False, lisa=False,
             backint=True, modes="reference"),
        # the ordinary batch: sources of 0.1 to 1 yr in FP64, the default precision, with the LISA response
        dict(name="waves_fp64", kind="batch", nsrc=32, lo=315581, hi=3155814, e_max=0.5, precision=0, graph=False,
             lisa=True, backint=False, modes="thirty"),
        # the largest batch, split precision, replayed as one CUDA graph: the benchmark's headline call
        dict(name="waves_split", kind="batch", nsrc=64, lo=315581, hi=3155814, e_max=0.5, precision=1, graph=True,
             lisa=True, backint=False, modes="thirty"),
        # eccentric sources (e0 up to 0.7, 11 to 61 harmonics) in FP64
        dict(name="waves_eccentric", kind="batch", nsrc=12, lo=200003, hi=2000003, e_max=0.7, precision=0, graph=False,
             lisa=True, backint=False, modes="eccentric"),
        # the phase product of a batch (eight FP64 rows a sample)
        dict(name="phases", kind="phase", nsrc=16, lo=315581, hi=3155814),
        # a sampler's likelihood call at the full length (3.2e6 samples, 1 yr), FP64, in chunks of 64
        dict(name="likelihood_fp64", kind="likelihood", length=3200000, n=128, max_batch=64, precision=0),
        # the same with FP32 transform and products, shorter data, two default chunks
        dict(name="likelihood_fp32", kind="likelihood", length=800000, n=512, max_batch=256, precision=2),
        # Fisher matrices of several points (14 parameters, 28 templates each)
        dict(name="fisher", kind="fisher", length=1600000, npts=4),
        # frequency-domain TDI, host parameters in, host rows out
        dict(name="tdi", kind="tdi", nsrc=2, lo=200003, hi=400009),
        # the warm-start network's prediction for many coarse points
        dict(name="mlp_predict", kind="predict", n=1000003),
        # its backward direction: one minibatch's gradient in training
        dict(name="mlp_gradient", kind="gradient", n=8192, rows=131072),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["wave", "batch", "batch", "batch", "phase", "likelihood", "likelihood", "fisher", "tdi", "predict",
                       "gradient"])
    if kind == "wave":
        return dict(kind=kind, length=_log_int(rng, 1000, 400000), lisa=rng.random() < 0.75, backint=rng.random() < 0.25)
    if kind == "batch":
        precision = int(rng.random() < 0.3)
        modes = rng.choice(["reference", "thirty", "eccentric"])
        hi = _log_int(rng, 8000, 3155814 if modes != "eccentric" else 2000003)
        return dict(kind=kind, nsrc=_log_int(rng, 1, 64 if precision else 32 if modes != "eccentric" else 12),
                    lo=_log_int(rng, max(1000, hi // 10), hi), hi=hi, e_max=0.7 if modes == "eccentric" else 0.5,
                    precision=precision, graph=rng.random() < 0.5, lisa=rng.random() < 0.75, backint=rng.random() < 0.25,
                    modes=modes)
    if kind == "phase":
        hi = _log_int(rng, 8000, 3155814)
        return dict(kind=kind, nsrc=_log_int(rng, 1, 16), lo=_log_int(rng, max(1000, hi // 10), hi), hi=hi)
    if kind == "likelihood":
        # transform lengths as a user picks them: 2^a 5^b near the span wanted
        length = rng.choice([2 ** a * 5 ** b for a in range(4, 15) for b in range(0, 6) if 50000 <= 2 ** a * 5 ** b <= 3200000])
        n = _log_int(rng, 8, min(512, 128 * 3200000 // length))
        return dict(kind=kind, length=length, n=n, max_batch=rng.choice([32, 64]), precision=rng.choice([0, 0, 1, 2]))
    if kind == "fisher":
        return dict(kind=kind, length=rng.choice([100000, 320000, 500000, 800000, 1600000]), npts=rng.randint(1, 4))
    if kind == "tdi":
        hi = _log_int(rng, 20000, 400009)
        return dict(kind=kind, nsrc=rng.randint(1, 2), lo=_log_int(rng, hi // 5, hi), hi=hi)
    if kind == "predict":
        return dict(kind=kind, n=_log_int(rng, 64, 1000003))
    return dict(kind=kind, n=_log_int(rng, 100, 8192), rows=_log_int(rng, 8192, 131072))


# --------------------------------------------------------------------------- sources
def _lengths(case):
    """nsrc lengths evenly spread from lo to hi (the mean one for a single source)."""
    n = case["nsrc"]
    if n == 1:
        return [(case["lo"] + case["hi"]) // 2]
    return [case["lo"] + (case["hi"] - case["lo"]) * i // (n - 1) for i in range(n)]


def _source(rng, length, e_max, lisa=True, backint=False):
    """A benchmark draw of the given length (the start radius keeps the plunge after the span)."""
    p = workloads.draw_source(rng, e_max=e_max)
    rr = (p["M"] * workloads.MSUN_SEC) ** 2 / (p["mu"] * workloads.MSUN_SEC)
    end = 10.0 + 3.0 * p["e"]
    p.update(length=length, T=length * DT / workloads.YEAR, LISA=lisa, backint=backint,
             p=min(max((end**4 + 2.0 * (256.0 / 5.0) * length * DT / rr) ** 0.25, 9.0), 80.0))
    return p


def _sources(case, seed):
    rng = np.random.default_rng(seed)
    return [_source(rng, n, case.get("e_max", 0.5), case.get("lisa", True), case.get("backint", False))
            for n in _lengths(case)]


def _one_source(case, seed):
    """A source that plans without an error (a single call raises where a batch reports a status)."""
    rng = np.random.default_rng(seed)
    check = aak.WaveBatch(-1)
    while True:
        p = _source(rng, case["length"], 0.5, case["lisa"], case["backint"])
        if check.plan([p]).status[0] == 0:
            return p


def _modes(case, sources):
    if case["modes"] == "thirty":
        return [workloads.NMODES] * len(sources)
    if case["modes"] == "eccentric":
        return [min(100, math.ceil(10.0 / (1.0 - p["e"]) ** 1.5)) for p in sources]
    return None  # the reference's rule


def _templates(n, seed):
    rng = np.random.default_rng(seed)
    X = np.tile(np.array(FIDUCIAL), (n, 1))
    for j in (2, 4, 5):
        X[:, j] *= 1.0 + 1e-5 * rng.standard_normal(n)
    for j in (0, 6, 7, 8, 9, 10, 11, 12):
        X[:, j] += 1e-3 * rng.standard_normal(n)
    return X


def _likelihood(length, seed):
    """The likelihood object with its weights and data (the fiducial signal in seeded LISA-coloured noise)."""
    g = GPUAAK(1.0, 100, length, 100.0, DT, True, False)
    freqs = generate_noise_frequencies(length * DT, 1 / DT)
    freqs[0] = freqs[1] / 10.0
    w = np.sqrt(DT / length) / np.sqrt(LISA_Noise(freqs, dur=1))
    ones, zero, nb = np.ones_like(w), np.zeros(len(w), dtype=np.complex128), len(w)
    g.input_data(zero, zero, ones, ones)
    g.gpu_gen_AAK(*FIDUCIAL)
    g.Likelihood()
    _, sI, sII = g.GetWaveform(is_Fourier=True)
    rng = np.random.default_rng(seed)
    data = []
    for s in (sI, sII):
        noise = generate_noise_single_channel(LISA_Noise, [], {"dur": 1}, 1.0 / (length * DT), freqs, rng)
        data.append(w * (s[0:2 * nb:2] + 1j * s[1:2 * nb:2] + noise))
    g.input_data(data[0], data[1], w, w)
    return g


def _points(n, seed):
    """Points of the warm start's distribution (p above a simple separatrix bound) and smooth targets."""
    rng = np.random.default_rng(seed)
    e, iota, a = rng.uniform(1e-3, 0.7, n), rng.uniform(0.0, math.pi, n), rng.uniform(0.0, 0.95, n)
    p = rng.uniform(0.0, 1.0, n) * (13.9 - 2.0 * e) + 6.1 + 2.0 * e
    x = np.stack([p, e, iota, a], axis=1).astype(np.float32)
    y = np.stack([1.0 + 0.3 / p + 0.02 * e * e, 1.0 - 0.8 / p + 0.1 * a * np.cos(iota), 0.1 * a * e + 0.2 / p], axis=1)
    return x, y.astype(np.float32)


def _norm(x, y):
    f = input_features(x.astype(np.float64))
    return [v.astype(np.float32) for v in (f.mean(0), 1.0 / f.std(0), y.mean(0, dtype=np.float64), y.std(0, dtype=np.float64))]


def _mlp_inputs(case, seed):
    rows = case.get("rows", case["n"])
    x, y = _points(rows, seed)
    perm = np.random.default_rng(seed + 1).permutation(rows)[: case["n"]].astype(np.int32)
    return x, y, perm, _norm(*_points(4096, 1)), init_params(seed)


# --------------------------------------------------------------------------- the cases
def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "wave":
        s["pars"] = _one_source(case, seed)
    elif kind in ("batch", "phase"):
        src = _sources(case, seed)
        wb = s["wb"] = aak.WaveBatch(0)
        wb.plan(src, nmodes=_modes(case, src) if kind == "batch" else None)
        wb.upload()
        n = wb.total_samples
        if kind == "phase":
            s["rows"] = torch.empty((8, n), dtype=torch.float64, device="cuda")
        else:
            s["hI"], s["hII"] = (torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(2))
    elif kind == "likelihood":
        g = s["g"] = _likelihood(case["length"], seed)
        g.set_precision(case["precision"])
        s["X"] = _templates(case["n"], seed)
    elif kind == "fisher":
        s["g"] = _likelihood(case["length"], seed)
        step = 1e-6 * np.maximum(np.abs(np.array(FIDUCIAL)), 1.0)
        X = np.repeat(_templates(case["npts"], seed)[:, None, :], 28, axis=1)
        for i in range(14):
            X[:, 2 * i, i] += step[i]
            X[:, 2 * i + 1, i] -= step[i]
        s["X"], s["scale"] = X, 0.5e6
    elif kind == "tdi":
        s["src"], s["wb"] = _sources(case, seed), aak.WaveBatch(0)
    else:
        x, y, perm, norm, params = _mlp_inputs(case, seed)
        s["model"] = ParMapMLP(0, params=params)
        s["model"].set_norm(*norm)
        s["x"], s["y"], s["perm"] = (torch.as_tensor(v, device="cuda") for v in (x, y, perm))
        if kind == "predict":
            s["out"] = torch.empty((case["n"], 3), dtype=torch.float32, device="cuda")
        else:
            s["out"] = torch.empty(params.size, dtype=torch.float32, device="cuda")
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "wave":
        t, hI, hII, _ = aak.wave(s["pars"])
        return t, hI, hII
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "batch":
        if case["graph"]:
            s["wb"].run_graph(s["hI"].data_ptr(), s["hII"].data_ptr(), precision=case["precision"], stream=stream)
        else:
            s["wb"].run(s["hI"].data_ptr(), s["hII"].data_ptr(), precision=case["precision"], stream=stream)
        return s["hI"], s["hII"]
    if kind == "phase":
        s["wb"].run_phase(s["rows"].data_ptr(), s["rows"].shape[1], stream=stream)
        return s["rows"]
    if kind == "likelihood":
        return s["g"].likelihood_batch(s["X"], max_batch=case["max_batch"])
    if kind == "fisher":
        return s["g"].fisher_gram_batch(s["X"], s["scale"])
    if kind == "tdi":
        rows, _, status = s["wb"].tdi_host(s["src"])
        return list(rows), status
    if kind == "predict":
        s["model"].forward_device(s["x"].data_ptr(), s["out"].data_ptr(), case["n"], stream=stream)
        return s["out"]
    loss = s["model"].gradients_device(s["x"].data_ptr(), s["y"].data_ptr(), case["n"], s["out"].data_ptr(),
                                       perm_ptr=s["perm"].data_ptr(), stream=stream)
    return s["out"], np.float32(loss)


# --------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Waveforms: 60 flops a sample and 54 a sample and harmonic (an FMA is two), outputs written once.  Likelihoods and
    Fisher matrices: that, and a real transform (2.5 n log2 n) with its half spectrum."""
    kind = case["kind"]
    if kind == "wave":
        return {"bytes": 24.0 * case["length"], "flops": (60.0 + 54.0 * 10) * case["length"]}
    if kind == "batch":
        modes = {"reference": 10, "thirty": 30, "eccentric": 22}[case["modes"]]
        n = float(sum(_lengths(case)))
        return {"bytes": 16.0 * n, "flops": (60.0 + 54.0 * modes) * n}
    if kind == "phase":
        n = float(sum(_lengths(case)))
        return {"bytes": 64.0 * n, "flops": 100.0 * n}
    if kind in ("likelihood", "fisher"):
        n = float(case["n"] if kind == "likelihood" else 28 * case["npts"])
        size = 4.0 if case.get("precision") == 2 else 8.0
        N = float(case["length"])
        return {"bytes": n * 2 * N * size * 2, "flops": n * N * (60.0 + 54.0 * 6 + 2 * 2.5 * math.log2(N))}
    if kind == "tdi":
        n = float(sum(_lengths(case)))
        return {"bytes": 24.0 * n, "flops": 1000.0 * n}
    layers = 2.0 * (4 * 128 + 2 * 128 * 128 + 3 * 128)
    if kind == "predict":
        return {"bytes": 28.0 * case["n"], "flops": layers * case["n"]}
    return {"bytes": 32.0 * case["n"] + 4.0 * 34051, "flops": 3 * layers * case["n"]}


# --------------------------------------------------------------------------- the network in 64 bits
def _unpack(params):
    out, o = [], 0
    for shape in ((128, 4), (128,), (128, 128), (128,), (128, 128), (128,), (3, 128), (3,)):
        k = math.prod(shape)
        p = params[o:o + k].reshape(shape)
        # the model's weights are BF16, its biases FP32
        out.append(p.to(torch.bfloat16).double() if len(shape) == 2 else p.double())
        o += k
    return out


def exact(case, seed):
    """The network's values in 64 bits on its BF16 weights.  The waveform products have no short statement outside the
    library (a Kerr inspiral, a nonlinear map and two recurrences of millions of steps): None."""
    if case["kind"] not in ("predict", "gradient"):
        return None
    x, y, perm, norm, params = _mlp_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x, y = (torch.as_tensor(v, device=dev).double() for v in (x, y))
    shift, scale, oshift, oscale = (torch.as_tensor(v, device=dev).double() for v in norm)
    if case["kind"] == "gradient":
        idx = torch.as_tensor(perm.astype(np.int64), device=dev)
        x, y = x[idx], y[idx]
    weights = [w.requires_grad_(True) for w in _unpack(torch.as_tensor(params, device=dev))]
    W1, b1, W2, b2, W3, b3, W4, b4 = weights
    a = (torch.stack([x[:, 0].rsqrt(), x[:, 1], x[:, 2].cos(), x[:, 3]], dim=1) - shift) * scale
    for W, b in ((W1, b1), (W2, b2), (W3, b3)):
        a = torch.nn.functional.silu(a @ W.T + b)
    z = a @ W4.T + b4
    if case["kind"] == "predict":
        return (z * oscale + oshift).detach()
    loss = ((z - (y - oshift) / oscale) ** 2).mean()
    grads = torch.autograd.grad(loss, weights)
    return torch.cat([g.reshape(-1) for g in grads]), float(loss)
