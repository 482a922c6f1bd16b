"""The work that programs give this framework, as cases that can be timed and checked.

A case is a dict of plain values; `kind` names the public entry points it goes
through:

* ``fastconv``  ``Fastconv(weights, rows)(x, y)``: pulse compression, one
  spectrum for all rows (``weights="vector"``) or one per row ("matrix").
* ``phased``    ``Fftm`` forward, ``vmmul``, ``Fftm`` inverse scaled by 1/n: the
  same computation as three calls, as programs written against the separate
  operations make it.
* ``fftm``      one ``Fftm`` over rows (``axis="row"``) or columns ("col").
* ``real``      ``FftmReal`` forward and inverse on independent data.
* ``fft2d``     one ``Fft2d``.
* ``batch``     ``Batch.run()``: uneven fast-convolution jobs in one launch.
* ``host``      ``Fastconv`` on numpy arrays: the whole call, copies included.

Data are complex Gaussian samples (radar noise and clutter look like that);
replicas are linear-FM chirps.  Plans, weights and output arrays are made once,
as programs keep them across pulses.
"""
import math

import numpy as np
import torch

import openvsip_b200 as ov
from openvsip_b200 import synth
from openvsip_b200.batch import Batch


def listed():
    return [
        # one coherent processing interval of a small radar: a call of a few
        # microseconds, where the launch and the host's share count
        {"name": "fastconv_64x2048", "kind": "fastconv", "rows": 64, "n": 2048, "weights": "vector"},
        # the benchmark's pulse compression: many long pulses, one replica
        {"name": "fastconv_1024x16384", "kind": "fastconv", "rows": 1024, "n": 16384, "weights": "vector"},
        # the longest rows that one plan takes, at the length sweep's 256 rows
        {"name": "fastconv_256x65536", "kind": "fastconv", "rows": 256, "n": 65536, "weights": "vector"},
        # a matrix of coefficients: every row with a spectrum of its own
        {"name": "coefs_512x4096", "kind": "fastconv", "rows": 512, "n": 4096, "weights": "matrix"},
        # the three separate operations of the phased benchmark form
        {"name": "phased_1024x8192", "kind": "phased", "rows": 1024, "n": 8192},
        # an ordinary Doppler-sized transform of the row sweep, inverse
        {"name": "fftm_256x1024_inv", "kind": "fftm", "rows": 256, "n": 1024, "axis": "row", "inverse": True},
        # image formation: the range transform of a SAR kernel (1072 rows of 1144)
        {"name": "fftm_1072x1144", "kind": "fftm", "rows": 1072, "n": 1144, "axis": "row", "inverse": False},
        # and its cross-range transform: 1144 columns of 756, inverse
        {"name": "fftm_cols_756x1144_inv", "kind": "fftm", "rows": 1144, "n": 756, "axis": "col", "inverse": True},
        # real samples from a receiver to half spectra, and back
        {"name": "real_2048x4096", "kind": "real", "rows": 2048, "n": 4096},
        # one large image
        {"name": "fft2d_4096x4096", "kind": "fft2d", "rows": 4096, "n": 4096, "inverse": False},
        # a queue of uneven jobs (16 to 512 pulses of 1024 to 32768 samples), each with its own replica
        {"name": "batch_64_jobs", "kind": "batch", "jobs": 64, "mix": 3},
        # a program whose data live in ordinary host arrays
        {"name": "host_256x4096", "kind": "host", "rows": 256, "n": 4096},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _length(rng, lo, hi):
    """A row length: most are powers of two, many others products of small
    primes (sizes are chosen for their FFTs), some whatever the data had."""
    u = rng.random()
    t = _log_uniform(rng, lo, hi)
    if u < 0.55:
        return 1 << min(int(math.log2(hi)), max(int(math.ceil(math.log2(lo))), round(math.log2(t))))
    t = min(t, 16384)
    if u < 0.85:
        n = t
        while True:
            m = n
            for p in (2, 3, 5, 7):
                while m % p == 0:
                    m //= p
            if m == 1:
                return n
            n += 1
    return t


def _rows(rng, n, samples):
    """Rows for at most `samples` samples in all (at least 4096, as long as there is one row)."""
    return max(1, _log_uniform(rng, max(1, 4096 // n), max(2, samples // n)))


def draw(rng):
    kind = rng.choice(["fastconv", "fastconv", "fastconv", "phased", "fftm", "fftm", "fftm", "real", "fft2d",
                       "batch", "host"])
    if kind == "fastconv":
        weights = rng.choice(["vector", "vector", "matrix"])
        n = _length(rng, 64, 65536)
        pow2 = n & (n - 1) == 0
        return {"kind": kind, "rows": _rows(rng, n, 1 << (24 if pow2 else 22)), "n": n, "weights": weights}
    if kind == "phased":
        n = _length(rng, 256, 32768)
        return {"kind": kind, "rows": _rows(rng, n, 1 << 22), "n": n}
    if kind == "fftm":
        n = _length(rng, 64, 65536)
        pow2 = n & (n - 1) == 0
        axis = rng.choice(["row", "row", "col"])
        return {"kind": kind, "rows": _rows(rng, n, 1 << (24 if pow2 and axis == "row" else 22)), "n": n,
                "axis": axis, "inverse": rng.random() < 0.5}
    if kind == "real":
        n = _length(rng, 128, 65536)
        return {"kind": kind, "rows": _rows(rng, n, 1 << 23), "n": n}
    if kind == "fft2d":
        n = _length(rng, 64, 4096)
        m = _length(rng, 64, min(4096, (1 << 22) // n) + 1)
        return {"kind": kind, "rows": m, "n": n, "inverse": rng.random() < 0.5}
    if kind == "batch":
        return {"kind": kind, "jobs": _log_uniform(rng, 4, 40), "mix": rng.randrange(1 << 20)}
    n = _length(rng, 256, 16384)
    return {"kind": kind, "rows": _rows(rng, n, 1 << 20), "n": n}


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _gauss(g, rows, n):
    return torch.view_as_complex(torch.randn(rows, n, 2, generator=g, device="cuda"))


def _spectra(case, seed):
    """Replica spectra: matched filters of linear-FM chirps, their bandwidth drawn from the seed."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    rows = case["rows"] if case.get("weights") == "matrix" else 1
    tbp = rng.uniform(0.05, 0.6, size=(rows, 1)) * n
    t = torch.arange(n, dtype=torch.float64, device="cuda") / n - 0.5
    phase = torch.from_numpy(np.pi * tbp).cuda() * t ** 2
    w = torch.fft.fft(torch.polar(torch.ones_like(phase), phase)).conj().to(torch.complex64)
    return w.contiguous() if rows > 1 else w.reshape(n).contiguous()


def _real_inputs(case, seed):
    g = _generator(seed)
    rows, n = case["rows"], case["n"]
    x = torch.randn(rows, n, generator=g, device="cuda")
    s = _gauss(g, rows, n // 2 + 1)  # the half spectrum of a real signal: real at the ends
    s[:, 0] = s[:, 0].real
    if n % 2 == 0:
        s[:, -1] = s[:, -1].real
    return x, s


def _data(case, seed):
    kind = case["kind"]
    if kind == "fftm" and case["axis"] == "col":
        return _gauss(_generator(seed), case["n"], case["rows"])
    return _gauss(_generator(seed), case["rows"], case["n"])


def _host_data(case, seed):
    rng = np.random.default_rng(seed)
    return synth.cgauss(rng, (case["rows"], case["n"]))


def _batch_jobs(case, seed):
    """(data, replica) of every job: the shapes are the case's, the data the seed's."""
    g = _generator(seed)
    return [(_gauss(g, j["pulses"], j["n"]), synth.job_replica(j).astype(np.complex64))
            for j in synth.uneven_jobs(seed=case["mix"], njobs=case["jobs"])]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "batch":
        jobs = _batch_jobs(case, seed)
        b = Batch()
        ids = [b.add_replica(r, kind="matched") for _, r in jobs]
        s["out"] = [torch.empty_like(x) for x, _ in jobs]
        s["keep"] = jobs
        b.set_stream(torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        b.set_jobs([(x, y, i) for (x, _), y, i in zip(jobs, s["out"], ids)])
        s["batch"] = b
        return s
    rows, n = case["rows"], case["n"]
    if kind == "host":
        s["x"] = _host_data(case, seed)
        s["y"] = np.empty_like(s["x"])
        s["plan"] = ov.Fastconv(_spectra(case, seed).cpu().numpy(), rows)
        return s
    if kind == "real":
        s["x"], s["s"] = _real_inputs(case, seed)
        s["fwd"] = ov.FftmReal(rows, n, ov.fft_fwd)
        s["inv"] = ov.FftmReal(rows, n, ov.fft_inv, 1.0 / n)
        s["X"] = torch.empty_like(s["s"])
        s["y"] = torch.empty_like(s["x"])
        return s
    s["x"] = _data(case, seed)
    s["y"] = torch.empty_like(s["x"])
    if kind == "fastconv":
        w = _spectra(case, seed)
        torch.cuda.synchronize()  # a plan reads its weights on a stream of its own
        s["plan"] = ov.Fastconv(w, rows)
    elif kind == "phased":
        s["w"] = _spectra(case, seed)
        s["fwd"] = ov.Fftm(rows, n, ov.fft_fwd)
        s["inv"] = ov.Fftm(rows, n, ov.fft_inv, 1.0 / n)
        s["X"] = torch.empty_like(s["x"])
    elif kind == "fft2d":
        d = ov.fft_inv if case["inverse"] else ov.fft_fwd
        s["plan"] = ov.Fft2d(rows, n, d, 1.0 / (rows * n) if case["inverse"] else 1.0)
    else:
        d = ov.fft_inv if case["inverse"] else ov.fft_fwd
        scale = 1.0 / n if case["inverse"] else 1.0
        if case["axis"] == "col":
            s["plan"] = ov.Fftm(n, rows, d, scale, axis=ov.col)
        else:
            s["plan"] = ov.Fftm(rows, n, d, scale)
    return s


def run(s):
    kind = s["case"]["kind"]
    if kind == "batch":
        s["batch"].run()
        return s["out"]
    if kind == "phased":
        s["fwd"](s["x"], s["X"])
        ov.vmmul(s["w"], s["X"], s["X"])
        return s["inv"](s["X"], s["y"])
    if kind == "real":
        return s["fwd"](s["x"], s["X"]), s["inv"](s["s"], s["y"])
    return s["plan"](s["x"], s["y"])


def work(case):
    def fft(rows, n):
        return 5.0 * rows * n * math.log2(n)

    kind = case["kind"]
    if kind == "batch":
        jobs = synth.uneven_jobs(seed=case["mix"], njobs=case["jobs"])
        return {"bytes": sum(16.0 * j["pulses"] * j["n"] + 8.0 * j["n"] for j in jobs),
                "flops": sum(2 * fft(j["pulses"], j["n"]) + 6.0 * j["pulses"] * j["n"] for j in jobs)}
    rows, n = case["rows"], case["n"]
    samples = float(rows) * n
    if kind == "real":
        return {"bytes": 2 * rows * (4.0 * n + 8.0 * (n // 2 + 1)), "flops": fft(rows, n)}
    if kind == "fft2d":
        return {"bytes": 16.0 * samples, "flops": 5.0 * samples * math.log2(samples)}
    if kind == "fftm":
        return {"bytes": 16.0 * samples, "flops": fft(rows, n)}
    weights = samples if case.get("weights") == "matrix" else n
    return {"bytes": 16.0 * samples + 8.0 * weights, "flops": 2 * fft(rows, n) + 6.0 * samples}


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        out = []
        for x, r in _batch_jobs(case, seed):
            w = torch.fft.fft(torch.from_numpy(r).cuda().to(torch.complex128)).conj()
            out.append(torch.fft.ifft(torch.fft.fft(x.to(torch.complex128)) * w))
        return out
    if kind == "real":
        x, s = _real_inputs(case, seed)
        return torch.fft.rfft(x.double()), torch.fft.irfft(s.to(torch.complex128), case["n"])
    if kind == "host":
        x = torch.from_numpy(_host_data(case, seed)).cuda().to(torch.complex128)
        w = _spectra(case, seed).to(torch.complex128)
        return torch.fft.ifft(torch.fft.fft(x) * w).cpu().numpy()
    x = _data(case, seed).to(torch.complex128)
    if kind == "fft2d":
        return torch.fft.ifft2(x) if case["inverse"] else torch.fft.fft2(x)
    if kind == "fftm":
        d = 0 if case["axis"] == "col" else 1
        return torch.fft.ifft(x, dim=d) if case["inverse"] else torch.fft.fft(x, dim=d)
    return torch.fft.ifft(torch.fft.fft(x) * _spectra(case, seed).to(torch.complex128))
