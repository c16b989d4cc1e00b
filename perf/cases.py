"""Measured workloads of the filter + whiten path, through the public API.

Each case is one call that a program of this package makes on device data it
already holds: `prepare` makes the recording (seeded, the package's own
synthetic model), `run` makes the call, `exact` gives the same result from
plain torch in 64 bits.  The listed sizes are those of the repository's
configurations, benchmark and tests (32 channels x 60 s, 384-channel probes, 4
shanks x 384 channels as int16, an uneven batch of {16, 32, 64, 128, 384}
channels), with tetrodes, odd channel counts and ragged lengths beside them.
The reference's window geometry depends on the thread count; it is 16
throughout, as in the benchmark.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mountainsort_b200 import api as ms
from mountainsort_b200 import synth

FS, FMIN, FMAX, FWID = 30000.0, 300.0, 6000.0, 1000.0
THREADS = 16
OVERLAP = 60000  # timepoints of overlap on each side of a filter window


def listed():
    return [
        # clips cut around a sorting run's events, whitened with a known matrix: the smallest call
        {"name": "clips_32ch", "kind": "clips", "M": 32, "T": 50, "L": 300},
        # a few seconds of a 16-channel probe: two windows, mostly latency
        {"name": "filter_16ch_snippet", "kind": "filter", "M": 16, "N": 130001},
        # a tetrode: few channels give the reference's long windows (699050 points)
        {"name": "filter_tetrode", "kind": "filter", "M": 4, "N": 3000001},
        # an odd channel count recorded and stored as int16
        {"name": "filter_63ch_int16_out", "kind": "filter", "M": 63, "N": 777777, "i16": True, "q": 0.25},
        # four shanks of 384 channels, int16 input, filtered as one recording
        {"name": "filter_1536ch_int16", "kind": "filter", "M": 1536, "N": 600000, "i16": True},
        # a 200-channel probe, the mixed-precision form
        {"name": "whiten_200ch_mixed", "kind": "whiten", "M": 200, "N": 1500000, "precision": "mixed"},
        # four shanks of 384 channels, each whitened on its own
        {"name": "whiten_4_shanks", "kind": "blocks", "M": 1536, "N": 300000, "blocks": 4},
        # one minute of a 32-channel probe, filter + whiten
        {"name": "fused_32ch_minute", "kind": "fused", "M": 32, "N": 1800000},
        # several minutes of a 384-channel probe, filter + whiten: the largest call
        {"name": "fused_384ch_minutes", "kind": "fused", "M": 384, "N": 6000000},
        # uneven recordings in one call
        {"name": "batch_uneven", "kind": "batch", "Ms": "16,32,64,128,384,32", "Ns": "900001,1500000,640000,420000,300000,60001"},
        # artifact masking of a filtered recording
        {"name": "mask_64ch", "kind": "mask", "M": 64, "N": 3000000, "interval": 2000},
        # event detection on a whitened recording
        {"name": "detect_64ch", "kind": "detect", "M": 64, "N": 1800000, "sign": 0},
    ]


def _between(rng, a, b):
    """Log-uniform integer in [a, b]."""
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["clips", "filter", "filter", "whiten", "whiten", "fused", "fused", "blocks", "batch", "mask", "detect"])
    if kind == "clips":
        return {"kind": kind, "M": _between(rng, 1, 384), "T": rng.choice([30, 50, 51, 100]), "L": _between(rng, 100, 20000)}
    if kind == "batch":
        k = rng.randint(2, 8)
        Ms = [rng.choice([16, 32, 64, 128, 384]) for _ in range(k)]
        return {"kind": kind, "Ms": ",".join(map(str, Ms)), "Ns": ",".join(str(_between(rng, 30000, 1000000)) for _ in range(k))}
    if kind == "blocks":
        b = rng.choice([2, 3, 4])
        per = _between(rng, 4, 384)
        return {"kind": kind, "M": b * per, "N": _between(rng, 30000, max(30000, min(3000000, 1000000000 // (b * per)))), "blocks": b}
    M = _between(rng, 1, 1536) if kind == "filter" else _between(rng, 1, 384)
    if rng.random() < 0.5:
        M = min(1536, (M + 3) // 4 * 4)  # probes come in multiples of four more often than not
    N = _between(rng, 20000, min(10000000, 2000000000 // M))
    c = {"kind": kind, "M": M, "N": N}
    if kind == "filter":
        c["i16"] = rng.random() < 0.4
        c["q"] = 0.25 if rng.random() < 0.2 else 0.0
        c["sub"] = rng.choice([1, 1, 1, 2, 3])
    if kind in ("whiten", "fused"):
        c["precision"] = rng.choice(["plain", "plain", "mixed"])
        c["q"] = 0.01 if rng.random() < 0.2 else 0.0
    if kind == "mask":
        c["interval"] = rng.choice([500, 2000, 3001])
    if kind == "detect":
        c["sign"] = rng.choice([-1, 0, 1])
    return c


# ---------------------------------------------------------------- inputs


def _raw(M, N, seed):
    """An extracellular recording, (N, M) float32 on the GPU."""
    return synth.generate_torch(M, N, FS, K=max(1, min(64, M)), seed=seed)


def _band(X):
    """X band-limited to the spike band (what a filtered recording looks like), in place."""
    N, M = X.shape
    f = torch.fft.rfftfreq(N, 1.0 / FS, device=X.device)
    gain = (1 + torch.erf(3.0 * (f - FMIN) / FMIN)) * (1 - torch.erf((f - FMAX) / FWID)) / 4
    gain[0] = 0
    gain = gain.clamp_(min=0).sqrt_()
    for m in range(0, M, 16):
        X[:, m:m + 16] = torch.fft.irfft(torch.fft.rfft(X[:, m:m + 16].T.contiguous()) * gain, n=N).T
    return X


def _int16(X):
    return torch.clamp(torch.round(X / 0.195), -32768, 32767).to(torch.int16)


def _matrix(M, seed):
    """A symmetric whitening matrix of a correlated M-channel covariance, float64."""
    g = torch.Generator(device="cuda").manual_seed(seed + 17)
    A = torch.eye(M, device="cuda", dtype=torch.float64)
    A += 0.3 * torch.randn((M, M), generator=g, device="cuda", dtype=torch.float64) / math.sqrt(M)
    w, v = torch.linalg.eigh(100.0 * A @ A.T)
    return (v / w.sqrt()) @ v.T


def _ints(text):
    return [int(t) for t in text.split(",")]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "clips":
        M, T, L = case["M"], case["T"], case["L"]
        X = _band(_raw(M, max(4096, T * L), seed))[:T * L]
        s["X"], s["W"] = X.reshape(L, T, M).contiguous(), _matrix(M, seed)
    elif kind == "batch":
        s["jobs"] = [{"X": _raw(M, N, seed + 1000 * k), "samplerate": FS, "freq_min": FMIN, "freq_max": FMAX,
                      "freq_wid": FWID, "num_threads": THREADS}
                     for k, (M, N) in enumerate(zip(_ints(case["Ms"]), _ints(case["Ns"])))]
    elif kind == "detect":
        M, N = case["M"], case["N"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        X = torch.randn((N, M), generator=g, device="cuda")
        k = max(1, N // 600)  # spikes of a few samples, about 50 a second on each of their channels
        t = torch.randint(0, max(1, N - 8), (k * M,), generator=g, device="cuda")
        m = torch.arange(M, device="cuda").repeat(k)
        size = 4 + 4 * torch.rand(k * M, generator=g, device="cuda")
        for j, w in enumerate((0.4, -1.0, -0.6, 0.3, 0.2)):
            X.view(-1).index_put_((((t + j).clamp(max=N - 1)) * M + m,), w * size, accumulate=True)
        s["X"] = torch.floor(X.double() / 1e-4 + 0.5).mul_(1e-4).float()
    elif kind == "filter":
        X = _raw(case["M"], case["N"], seed)
        s["X"] = _int16(X) if case.get("i16") else X
    elif kind == "fused":
        s["X"] = _raw(case["M"], case["N"], seed)
    else:  # whiten, blocks, mask: a filtered recording
        s["X"] = _band(_raw(case["M"], case["N"], seed))
        if kind == "mask":
            g = torch.Generator(device="cuda").manual_seed(seed + 3)
            I, n = case["interval"], case["N"] // case["interval"]
            for i in torch.randint(0, max(1, n), (max(1, n // 100),), generator=g, device="cuda").tolist():
                s["X"][i * I:(i + 1) * I] *= 8.0
        if kind == "blocks":
            per = case["M"] // case["blocks"]
            s["blocks"] = [list(range(1 + b * per, 1 + (b + 1) * per)) for b in range(case["blocks"])]
    return s


# ---------------------------------------------------------------- the calls


def run(state):
    c = state["case"]
    kind = c["kind"]
    q, precision = c.get("q", 0.0), c.get("precision", "plain")
    if kind == "clips":
        return ms.whiten_clips(state["X"], state["W"])
    if kind == "batch":
        return ms.bandpass_whiten_batch(state["jobs"])
    X = state["X"]
    if kind == "filter":
        return ms.bandpass_filter(X, FS, FMIN, FMAX, FWID, quantization_unit=q, subsample_factor=c.get("sub", 1), num_threads=THREADS)
    if kind == "whiten":
        return ms.whiten(X, quantization_unit=q, precision=precision)
    if kind == "blocks":
        return ms.whiten_blocks(X, state["blocks"])
    if kind == "fused":
        return ms.bandpass_whiten(X, FS, FMIN, FMAX, FWID, num_threads=THREADS, quantization_unit=q, precision=precision)
    if kind == "mask":
        out, kept = ms.mask_out_artifacts(X, 6.0, c["interval"], return_kept=True)
        return {"out": out, "kept": kept}
    times = ms.detect_events(X, 3.5, 10.0, c["sign"])
    # the event times channel after channel, in an array of one length for all recordings of a size
    flat = np.full(X.numel() // 128 + 4096, -1, np.int64)
    np.concatenate(times, out=flat[:sum(map(len, times))])
    return {"times": flat, "counts": np.array([len(t) for t in times])}


# ---------------------------------------------------------------- 64 bits


def _chunk(M):
    return max(2 * OVERLAP, int(1.0 * 2 ** 30 / (6 * 4 * M * THREADS) - 2 * OVERLAP))


def _exact_filter(X, sub=1):
    """The windowed FFT filter in complex128, float64 (N // sub, M)."""
    N, M = X.shape
    chunk = _chunk(M)
    L = chunk + 2 * OVERLAP
    i = torch.arange(L, device=X.device, dtype=torch.float64)
    df = 1.0 / (L / FS)
    f = torch.where(i <= (L + 1) // 2, df * i, df * (i - L)).abs()
    K = (1 + torch.erf(3.0 * (f - FMIN) / FMIN)) / 2
    K[0] = 0
    K = (K * (1 - torch.erf((f - FMAX) / FWID)) / 2).sqrt()
    out = torch.zeros((N // sub, M), device=X.device, dtype=torch.float64)
    step = max(1, min(M, 2 ** 27 // L))
    for t in range(0, N, chunk):
        lo, hi = max(0, t - OVERLAP), min(N, t - OVERLAP + L)
        for m in range(0, M, step):
            w = torch.zeros((min(step, M - m), L), device=X.device, dtype=torch.float64)
            w[:, lo - t + OVERLAP:hi - t + OVERLAP] = X[lo:hi, m:m + step].T
            y = torch.fft.ifft(torch.fft.fft(w) * K).real[:, OVERLAP:OVERLAP + chunk]
            y = y[:, 0:(chunk // sub) * sub:sub]
            o = t // sub
            n = min(y.shape[1], N // sub - o)
            if n > 0:
                out[o:o + n, m:m + step] = y[:, :n].T
    return out


def _exact_matrix(X):
    """The whitening matrix of the reference's ten-step power iteration, float64."""
    N, M = X.shape
    C = torch.zeros((M, M), device=X.device, dtype=torch.float64)
    for t in range(0, N, 1 << 20):
        x = X[t:t + (1 << 20)].double()
        C += x.T @ x
    if N > 1:
        C /= N - 1
    v0 = torch.sin(torch.arange(1, M + 1, device=X.device, dtype=torch.float64))
    v0 = v0 / v0.norm()
    W = torch.zeros_like(C)
    for _ in range(M):
        v = v0
        for _ in range(10):
            v = C @ v
            size = v.norm()
            v = v / size
        u = C @ v
        C = C - torch.outer(v, u) - torch.outer(u, v) + (v @ u) * torch.outer(v, v)
        W += torch.outer(v, v) / size.sqrt()
    return W


def _exact_apply(X, W, rounded=True):
    out = torch.empty(X.shape, device=X.device, dtype=torch.float64)
    for t in range(0, X.shape[0], 1 << 20):
        y = X[t:t + (1 << 20)].double() @ W
        out[t:t + (1 << 20)] = torch.floor(y / 1e-4 + 0.5) * 1e-4 if rounded else y
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "detect" or case.get("q"):
        return None  # whole numbers
    s = prepare(case, seed)
    if kind == "clips":
        L, T, M = s["X"].shape
        return _exact_apply(s["X"].reshape(L * T, M), s["W"], rounded=False).reshape(L, T, M)
    if kind == "batch":
        out = []
        for j in s["jobs"]:
            filt = _exact_filter(j["X"])
            out.append(_exact_apply(filt, _exact_matrix(filt)))
        return out
    X = s.pop("X")
    if kind == "filter":
        return _exact_filter(X, case.get("sub", 1))
    if kind == "fused":
        filt = _exact_filter(X)
        del X
        return _exact_apply(filt, _exact_matrix(filt))
    if kind == "whiten":
        return _exact_apply(X, _exact_matrix(X))
    if kind == "blocks":
        out = torch.empty(X.shape, device=X.device, dtype=torch.float64)
        for b in s["blocks"]:
            x = X[:, b[0] - 1:b[-1]].contiguous()
            out[:, b[0] - 1:b[-1]] = _exact_apply(x, _exact_matrix(x))
        return out
    # mask: intervals whose norm is far out on any channel go to zero with their neighbours
    N, M = X.shape
    I = case["interval"]
    n = N // I
    norms = X[:n * I].reshape(n, I, M).double().square().sum(1).sqrt()
    limit = norms.mean(0) + 6.0 * (norms.std(0) if n >= 2 else torch.zeros(M, device=X.device, dtype=torch.float64))
    bad = (norms > limit).any(1)
    keep = ~bad
    keep[1:] &= ~bad[:-1]
    keep[:-1] &= ~bad[1:]
    out = torch.zeros((N, M), device=X.device, dtype=torch.float64)
    out[:n * I] = torch.where(keep.repeat_interleave(I)[:, None], X[:n * I].double(), 0.0)
    return {"out": out, "kept": None}


# ---------------------------------------------------------------- work


def _filter_flops(M, N):
    chunk = _chunk(M)
    L = chunk + 2 * OVERLAP
    return 5.0 * L * math.log2(L) * M * math.ceil(N / chunk)  # one complex transform each way for two channels


def _whiten_flops(M, N):
    return 1.0 * M * M * N + 22.0 * M ** 3 + 2.0 * M * M * N  # covariance (half of it), ten steps and deflation, apply


def work(case):
    kind = case["kind"]
    if kind == "clips":
        n = case["M"] * case["T"] * case["L"]
        return {"bytes": 8.0 * n + 8.0 * case["M"] ** 2, "flops": 2.0 * case["M"] * n}
    if kind == "batch":
        w = [work({"kind": "fused", "M": M, "N": N}) for M, N in zip(_ints(case["Ms"]), _ints(case["Ns"]))]
        return {"bytes": sum(x["bytes"] for x in w), "flops": sum(x["flops"] for x in w)}
    M, N = case["M"], case["N"]
    out = 2.0 if case.get("q") else 4.0
    if kind == "filter":
        return {"bytes": M * N * (2.0 if case.get("i16") else 4.0) + M * (N // case.get("sub", 1)) * out, "flops": _filter_flops(M, N)}
    if kind in ("fused", "whiten"):  # read for the covariance, read again for the output
        return {"bytes": M * N * (8.0 + out), "flops": _whiten_flops(M, N) + (_filter_flops(M, N) if kind == "fused" else 0.0)}
    if kind == "blocks":
        b = case["blocks"]
        return {"bytes": 12.0 * M * N, "flops": b * _whiten_flops(M // b, N)}
    if kind == "mask":
        return {"bytes": 12.0 * M * N, "flops": 2.0 * M * N}
    return {"bytes": 8.0 * M * N, "flops": 6.0 * M * N}  # detect: statistics, then candidates
