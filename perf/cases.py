"""Performance cases of spectrum_gb300: the calls its users make, over the sizes they make them at.

listed() gives the fixed cases, draw(rng) one more of the same ranges, prepare(case, seed) what a
program holds before the call (inputs on the GPU or in page-locked host memory, a batch plan, a
network), run(state) one pass through the public entry points, work(case) the bytes and operations
of a pass and exact(case, seed) the same outputs in 64 bits by plain torch.

Samples are sums of complex tones in circular Gaussian noise, as in spectrum_gb300/synth.py.
"""
import math

import numpy as np
import torch

import spectrum_gb300 as spx
from spectrum_gb300.batch import Batch
from spectrum_gb300.learned import LAYOUT, N_PARAMS, MLPRefiner

WINDOWS = {"none": spx.WINDOW_NONE, "hann": spx.WINDOW_HANN, "hamming": spx.WINDOW_HAMMING,
           "blackman": spx.WINDOW_BLACKMAN, "blackman_harris": spx.WINDOW_BLACKMAN_HARRIS}
FS = 12.0e6        # sample rate of the peak searches, Hz
MAX_MAXIMA = 1000  # output capacity per beam of an all-maxima search


def listed():
    return [
        # one snapshot of a small array, the strongest tones wanted at once: the shortest call
        {"name": "topk_small", "kind": "topk", "beams": 8, "n": 4096, "nfft": 4096, "k": 5},
        # ordinary two-sided peak search (left and right of zero) of antenna beams, odd length
        {"name": "two_peaks", "kind": "two", "beams": 256, "n": 3001, "nfft": 8192, "two": True},
        # wide-band survey: every maximum above six sigma of long zero-padded beams
        {"name": "maxima_large", "kind": "all", "beams": 256, "n": 65536, "nfft": 131072},
        # the same search from host memory to host memory, a receiver's buffer as it arrives
        {"name": "maxima_host", "kind": "host", "beams": 64, "n": 16384, "nfft": 32768},
        # beams of uneven length in one batch, the eight strongest tones of each
        {"name": "batch_uneven", "kind": "batch", "beams": 1024, "lo": 1000, "hi": 100000, "k": 8},
        # power spectra of short frames (a spectrogram's block)
        {"name": "fft_frames", "kind": "fft", "beams": 8192, "n": 4096, "nfft": 4096, "window": "hann", "out": "mag2"},
        # high dynamic range spectra of very long beams: the largest transform in ordinary use
        {"name": "fft_long", "kind": "fft", "beams": 64, "n": 1048576, "nfft": 1048576, "window": "blackman_harris",
         "out": "complex"},
        # magnitude and phase of a 2^a 3^b length, ragged samples
        {"name": "fft_smooth", "kind": "fft", "beams": 300, "n": 48001, "nfft": 49152, "window": "hamming",
         "out": "magphase"},
        # a length with other prime factors (CpuFFT takes any)
        {"name": "fft_odd", "kind": "fft", "beams": 1024, "n": 5000, "nfft": 5000, "window": "none", "out": "complex"},
        # back to samples
        {"name": "inverse", "kind": "ifft", "beams": 2048, "nfft": 16384},
        # one tone per beam with learned sub-bin refinement
        {"name": "learned_peaks", "kind": "learned", "beams": 4096, "n": 8192, "nfft": 8192, "k": 1},
        # one training minibatch of the refinement network: loss and gradients
        {"name": "learned_grad", "kind": "grad", "rows": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["topk", "two", "all", "host", "batch", "fft", "fft", "fft_long", "fft_any", "ifft", "learned",
                       "grad"])
    pow2 = spx.next_pow2
    if kind == "topk":
        n = _log(rng, 1000, 16384)
        return {"kind": "topk", "beams": _log(rng, 1, 64), "n": n, "nfft": pow2(n), "k": rng.randint(1, 8)}
    if kind == "two":
        n = _log(rng, 500, 16000)
        return {"kind": "two", "beams": _log(rng, 16, 1024), "n": n, "nfft": pow2(n) * rng.choice([1, 2]),
                "two": rng.random() < 0.5}
    if kind == "all":
        n = _log(rng, 10000, 65536)
        return {"kind": "all", "beams": _log(rng, 8, 256), "n": n, "nfft": 2 * pow2(n)}
    if kind == "host":
        n = _log(rng, 4096, 65536)
        return {"kind": "host", "beams": _log(rng, 8, 64), "n": n, "nfft": 2 * pow2(n)}
    if kind == "batch":
        return {"kind": "batch", "beams": _log(rng, 64, 1024), "lo": 1000, "hi": rng.randint(20000, 100000),
                "k": rng.randint(1, 8)}
    if kind == "learned":
        n = rng.choice([4096, 8192, 16384])
        return {"kind": "learned", "beams": _log(rng, 64, 4096), "n": n, "nfft": n, "k": 1}
    if kind == "grad":
        return {"kind": "grad", "rows": _log(rng, 256, 16384)}
    if kind == "ifft":
        nfft = spx.next_smooth23(_log(rng, 1024, 131072))
        return {"kind": "ifft", "beams": max(1, _log(rng, 1 << 18, 1 << 25) // nfft), "nfft": nfft}
    window = rng.choice(sorted(WINDOWS))
    out = rng.choice(["complex", "mag", "mag2", "magphase"])
    if kind == "fft_long":
        n = _log(rng, 1 << 18, 1 << 20)
        nfft = pow2(n)
        total = _log(rng, 1 << 22, 1 << 26)
    elif kind == "fft_any":  # lengths as they come: 2^a 3^b or not
        n = _log(rng, 500, 100000)
        nfft = n if rng.random() < 0.5 else spx.next_smooth23(n)
        total = _log(rng, 1 << 18, 1 << 23)
    else:
        n = _log(rng, 1000, 100000)
        nfft = pow2(n)
        total = _log(rng, 1 << 18, 1 << 25)
    return {"kind": "fft", "beams": max(1, total // nfft), "n": n, "nfft": nfft, "window": window, "out": out}


# ---- inputs ---------------------------------------------------------------------------------
def _tones(gen, lengths, count, snr_db):
    """Samples of the beams back to back (complex64): up to `count` tones of U[0, 0.5) cycles a sample
    and amplitudes log-uniform in [0.1, 1] per beam (the first always on), noise at an SNR of
    U[snr_db] dB below the strongest."""
    dev = gen.device
    b = len(lengths)

    def uniform(*shape):
        return torch.rand(*shape, generator=gen, device=dev, dtype=torch.float64)

    f, p = 0.5 * uniform(count, b), uniform(count, b)
    a = torch.exp(math.log(0.1) * uniform(count, b))
    on = uniform(count, b) < 0.5
    on[0] = True
    a = a * on
    sigma = a.max(0).values * 10.0 ** (-(snr_db[0] + (snr_db[1] - snr_db[0]) * uniform(b)) / 20.0)
    same = len(set(lengths)) == 1
    if same:
        t = torch.arange(lengths[0], device=dev, dtype=torch.float64)[None, :]
        spread = lambda v: v[:, None]  # noqa: E731
        shape = (b, lengths[0])
    else:
        n = torch.tensor(lengths, device=dev)
        beam = torch.repeat_interleave(torch.arange(b, device=dev), n)
        first = torch.cumsum(n, 0) - n
        t = (torch.arange(beam.numel(), device=dev) - first[beam]).double()
        spread = lambda v: v[beam]  # noqa: E731
        shape = (beam.numel(),)
    x = torch.zeros(shape + (2,), device=dev, dtype=torch.float32)
    for i in range(count):
        cyc = torch.remainder(spread(f[i]) * t + spread(p[i]), 1.0)
        ph = (2 * math.pi) * cyc
        amp = spread(a[i])
        x[..., 0] += (amp * torch.cos(ph)).float()
        x[..., 1] += (amp * torch.sin(ph)).float()
    s = (spread(sigma) / math.sqrt(2.0)).float()
    x += s[..., None] * torch.randn(x.shape, generator=gen, device=dev, dtype=torch.float32)
    return torch.view_as_complex(x)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _lengths(case, seed):
    if case["kind"] == "batch":
        return [int(v) for v in np.random.default_rng(seed).integers(case["lo"], case["hi"] + 1, case["beams"])]
    return [case["n"]] * case["beams"]


def _samples(case, seed):
    kind = case["kind"]
    if kind == "ifft":
        x = torch.randn((case["beams"], case["nfft"], 2), generator=_gen(seed), device="cuda")
        return torch.view_as_complex(x)
    tones, snr = {"topk": (3, (30.0, 40.0)), "two": (2, (10.0, 40.0)), "learned": (1, (20.0, 20.0)),
                  "batch": (8, (0.0, 40.0)), "all": (8, (0.0, 40.0)), "host": (8, (0.0, 40.0))}.get(
                      kind, (2, (20.0, 140.0)))
    return _tones(_gen(seed), _lengths(case, seed), tones, snr)


def _network(seed):
    """Parameters of the refinement network at the scale of its initialisation, small outputs."""
    rng = np.random.default_rng(seed)
    parts = []
    for name, shape, _ in LAYOUT:
        scale = {"W1": 0.5, "W2": 0.2, "W3": 0.03}.get(name, 0.05)
        parts.append((rng.standard_normal(int(np.prod(shape))) * scale).astype(np.float32))
    p = np.concatenate(parts)
    assert p.size == N_PARAMS
    return p


def _rows(case, seed):
    """Feature rows, targets and mask of a minibatch: magnitude ratios and phases around main lobes."""
    g = _gen(seed)
    r = case["rows"]
    ratio = torch.rand((r, 5), generator=g, device="cuda")
    ratio[:, 2] = 1.0
    phase = 0.2 * torch.randn((r, 5), generator=g, device="cuda")
    phase[:, 2] = 0.0
    t = torch.rand((r, 2), generator=g, device="cuda") - 0.5
    mask = (torch.rand(r, generator=g, device="cuda") < 0.95).to(torch.int32)
    return torch.cat([ratio, phase], 1).contiguous(), t, mask


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind == "grad":
        s["net"] = MLPRefiner(seed=0)
        s["net"].set_params(_network(seed))
        s["x"], s["t"], s["mask"] = _rows(case, seed)
        return s
    x = _samples(case, seed)
    if kind == "learned":
        s["net"] = MLPRefiner(seed=0)
        s["net"].set_params(_network(seed))
    elif kind == "batch":
        s["batch"] = Batch(_lengths(case, seed), window=spx.WINDOW_HANN, k=case["k"], sample_rate=FS)
    elif kind == "host":
        host = torch.empty(x.shape, dtype=x.dtype, pin_memory=True)
        host.copy_(x)
        x = host
        s["peaks"] = torch.zeros((case["beams"], MAX_MAXIMA, 8), dtype=torch.int32, pin_memory=True)
        s["counts"] = torch.zeros(case["beams"], dtype=torch.int32, pin_memory=True)
    s["x"] = x
    return s


# ---- one pass -------------------------------------------------------------------------------
def _peaks(out, counts):
    """MaxValue words: the whole ones (index, pad) and the FP32 fields, as the user reads them."""
    return {"words": out[..., ::7], "values": out.view(torch.float32)[..., 1:7], "counts": counts}


def run(s):
    kind = s["kind"]
    if kind == "fft":
        return spx.fft(s["x"], s["nfft"], WINDOWS[s["window"]], s["out"])
    if kind == "ifft":
        return spx.ifft(s["x"])
    if kind == "grad":
        grad, loss = s["net"].gradients(s["x"], s["t"], s["mask"])
        return {"grad": grad, "loss": loss}
    if kind == "topk":
        return _peaks(*spx.fft_peaks(s["x"], s["nfft"], spx.WINDOW_HANN, spx.PEAK_TOPK, sample_rate=FS,
                                     max_per_beam=s["k"], refine=spx.REFINE_PARABOLIC))
    if kind == "two":
        out, _ = spx.fft_peaks(s["x"], s["nfft"], spx.WINDOW_HANN, spx.PEAK_TWO if s["two"] else spx.PEAK_ONE,
                               sample_rate=FS)
        return _peaks(out, None)
    if kind == "all":
        return _peaks(*spx.fft_peaks(s["x"], s["nfft"], spx.WINDOW_HANN, spx.PEAK_ALL, sample_rate=FS,
                                     max_per_beam=MAX_MAXIMA, refine=spx.REFINE_PARABOLIC, thresh_sigma=6.0))
    if kind == "host":
        return _peaks(*spx.fft_peaks_host(s["x"], s["nfft"], spx.WINDOW_HANN, spx.PEAK_ALL, sample_rate=FS,
                                          max_per_beam=MAX_MAXIMA, refine=spx.REFINE_PARABOLIC, thresh_sigma=6.0,
                                          out=s["peaks"], counts=s["counts"]))
    if kind == "batch":
        return _peaks(*s["batch"].run(s["x"]))
    out, counts, amp, used = s["net"].fft_peaks(s["x"], s["nfft"], spx.WINDOW_HANN, s["k"], FS)
    return {**_peaks(out, counts), "amplitude": amp, "used": used}


def _fft_flops(n):
    return 5.0 * n * math.log2(n)


def work(case):
    kind = case["kind"]
    if kind == "grad":
        # forward and backward of 10 -> 64 -> 64 -> 2: every weight three products a row (two in layer 1)
        return {"bytes": case["rows"] * 52.0 + 4 * N_PARAMS * 2, "flops": case["rows"] * 2.0 * (2 * 640 + 3 * 4096 + 3 * 128)}
    beams = case["beams"]
    if kind == "ifft":
        return {"bytes": 16.0 * beams * case["nfft"], "flops": beams * _fft_flops(case["nfft"])}
    if kind == "fft":
        out = {"complex": 8, "magphase": 8, "mag": 4, "mag2": 4}[case["out"]]
        return {"bytes": beams * (8.0 * case["n"] + out * case["nfft"]), "flops": beams * _fft_flops(case["nfft"])}
    if kind == "batch":  # lengths are U[lo, hi]; the transform sizes lie a few per cent above
        n = 0.5 * (case["lo"] + case["hi"])
        return {"bytes": beams * (8.0 * n + 32 * case["k"] + 4), "flops": beams * _fft_flops(1.04 * n)}
    rows = {"topk": case.get("k", 0), "learned": case.get("k", 0), "two": 8 if case.get("two") else 4,
            "all": 40, "host": 40}[kind]
    return {"bytes": beams * (8.0 * case["n"] + 32 * rows + 4), "flops": beams * _fft_flops(case["nfft"])}


# ---- the same in 64 bits ----------------------------------------------------------------------
def _window64(name, n):
    if name == "none" or n < 2:
        return torch.ones(n, dtype=torch.float64, device="cuda")
    t = torch.arange(n, dtype=torch.float64, device="cuda") / (n - 1)
    c = [torch.cos(2 * math.pi * k * t) for k in range(4)]
    if name == "hann":
        return torch.sin(math.pi * t) ** 2
    if name == "hamming":
        return 0.54 - 0.46 * c[1]
    if name == "blackman":
        return 0.42 - 0.5 * c[1] + 0.08 * c[2]
    return 0.35875 - 0.48829 * c[1] + 0.14128 * c[2] - 0.01168 * c[3]


def _spectrum64(x, nfft, window):
    return torch.fft.fft(x.to(torch.complex128) * _window64(window, x.shape[-1]), n=nfft)


def _parabola(yl, yc, yr):
    den = yl - 2 * yc + yr
    return torch.where(den.abs() > 1e-10, (0.5 * (yl - yr) / den).clamp(-0.5, 0.5), torch.zeros_like(den))


def _records(spec, mag, k, nfft):
    """[real, imag, |X|, phase, offset, frequency] of the maxima at bins k [beams, R]."""
    z, yc = spec.gather(1, k), mag.gather(1, k)
    d = _parabola(mag.gather(1, k - 1), yc, mag.gather(1, k + 1))
    return torch.stack([z.real, z.imag, yc, torch.rad2deg(z.angle()), d, (k + d) * (FS / nfft)], -1)


def _maxima(mag):
    """Strict local maxima of bins [1, nfft / 2)."""
    end = mag.shape[1] // 2
    c = mag[:, 1:end]
    return (c > mag[:, :end - 1]) & (c > mag[:, 2:end + 1])


def _top64(spec, k):
    nfft = spec.shape[1]
    mag = spec.abs()
    ok = _maxima(mag)
    key = torch.where(ok, mag[:, 1:nfft // 2], torch.full_like(mag[:, 1:nfft // 2], -1.0))
    top = key.topk(k, dim=1)
    rec = _records(spec, mag, top.indices + 1, nfft)
    return rec * (top.values >= 0)[..., None], top.indices + 1


def _all64(spec):
    nfft = spec.shape[1]
    mag = spec.abs()
    end = nfft // 2
    thr = torch.empty(spec.shape[0], dtype=torch.float64, device="cuda")
    factor = (math.sqrt(math.pi / 2) + 6.0 * math.sqrt(2 - math.pi / 2)) / math.sqrt(2 * math.log(2))
    n = end - 1
    r = (n - 1) // 2
    edges = (torch.arange(4097, device="cuda").to(torch.int32) << 19).view(torch.float32).double()
    for b in range(spec.shape[0]):  # the noise median, interpolated in its histogram bucket
        h = torch.bincount((mag[b, 1:end].float().view(torch.int32) >> 19).long(), minlength=4096)
        c = torch.cumsum(h, 0)
        i = torch.searchsorted(c, torch.tensor(r, device="cuda"), right=True)
        frac = (r - (c[i] - h[i]) + 0.5) / h[i]
        thr[b] = (edges[i] + (edges[i + 1] - edges[i]) * frac) * factor
    ok = _maxima(mag) & (mag[:, 1:end] > thr[:, None])
    beam, bin_ = ok.nonzero(as_tuple=True)
    rank = torch.cumsum(ok, 1)[beam, bin_] - 1
    cap = min((end - 1) // 2, MAX_MAXIMA)
    rows = torch.zeros((spec.shape[0], cap, 6), dtype=torch.float64, device="cuda")
    keep = rank < cap
    beam, bin_, rank = beam[keep], bin_[keep] + 1, rank[keep]
    z, yc = spec[beam, bin_], mag[beam, bin_]
    d = _parabola(mag[beam, bin_ - 1], yc, mag[beam, bin_ + 1])
    rows[beam, rank] = torch.stack([z.real, z.imag, yc, torch.rad2deg(z.angle()), d, (bin_ + d) * (FS / nfft)], -1)
    return rows


def _sided64(spec, two):
    nfft = spec.shape[1]
    mag = spec.abs()
    half = nfft // 4 // 2
    left = mag[:, :half].max(1)
    right = mag[:, nfft - half:].max(1)
    il, ir = left.indices, right.indices + nfft - half

    def four(i, mirror):  # interpolated, left, centre, right
        hl, hr = i > 0, i < nfft - 1
        at = [i, (i - 1).clamp(min=0), i, (i + 1).clamp(max=nfft - 1)]
        on = [torch.ones_like(hl), hl, torch.ones_like(hl), hr]
        z = [spec.gather(1, k[:, None])[:, 0] * o for k, o in zip(at, on)]
        d = torch.where(hl & hr, _parabola(z[1].abs(), z[0].abs(), z[3].abs()), torch.zeros(1, device="cuda").double())
        rows = []
        for j, (k, o, v) in enumerate(zip(at, on, z)):
            off = d if j == 0 else torch.zeros_like(d)
            fr = (k + off) * (FS / nfft)
            fr = torch.where(mirror & o, FS - fr, fr) * o
            rows.append(torch.stack([v.real, v.imag, v.abs(), torch.rad2deg(v.angle()) * o, off, fr], -1))
        return torch.stack(rows, 1)

    if two:
        return torch.cat([four(il, torch.zeros_like(il, dtype=torch.bool)),
                          four(ir, torch.ones_like(ir, dtype=torch.bool))], 1)
    r = right.values > left.values
    return four(torch.where(r, ir, il), r)


def _net64(p):
    """The network's tensors: products read the weights rounded to BF16, biases are FP32."""
    t, pos = {}, 0
    for name, shape, dt in LAYOUT:
        n = int(np.prod(shape))
        v = torch.from_numpy(p[pos:pos + n]).cuda().reshape(shape)
        t[name] = (v.bfloat16() if dt == "bf16" else v).double()
        pos += n
    return t


def _forward64(t, x):
    gelu = torch.nn.functional.gelu
    h = gelu(x @ t["W1"].T + t["b1"])
    return gelu(h @ t["W2"].T + t["b2"]) @ t["W3"].T + t["b3"]


def _learned64(case, spec, net):
    nfft = case["nfft"]
    rec, k = _top64(spec, case["k"])
    d = torch.arange(-2, 3, device="cuda")
    at = (k[..., None] + d).clamp(0, nfft - 1)
    z = spec.gather(1, at.reshape(at.shape[0], -1)).reshape(at.shape)
    c = z[..., 2:3]
    ph = (z * c.conj()).angle() + math.pi * (case["n"] - 1) / nfft * d
    ph = ph - 2 * math.pi * torch.round(ph / (2 * math.pi))
    ph = torch.where(d == 0, torch.zeros_like(ph), ph)
    y = _forward64(_net64(net), torch.cat([z.abs() / c.abs(), ph], -1))
    use = (k >= 2) & (k + 2 < nfft) & (y[..., 0].abs() <= 0.5)
    rec[..., 4] = torch.where(use, y[..., 0], rec[..., 4])
    rec[..., 5] = torch.where(use, (k + y[..., 0]) * (FS / nfft), rec[..., 5])
    return rec, torch.where(use, rec[..., 2] * torch.exp(y[..., 1]), rec[..., 2])


def exact(case, seed):
    kind = case["kind"]
    if kind == "grad":
        x, t, mask = _rows(case, seed)
        net = {n: v.requires_grad_() for n, v in _net64(_network(seed)).items()}
        err = (_forward64(net, x.double()) - t.double()) * mask[:, None]
        loss = (err ** 2).sum() / (2 * case["rows"])
        loss.backward()
        return {"grad": torch.cat([net[n].grad.reshape(-1) for n, _, _ in LAYOUT]), "loss": loss.detach().reshape(1)}
    x = _samples(case, seed)
    if kind == "ifft":
        return torch.fft.ifft(x.to(torch.complex128))
    if kind == "fft":
        out = torch.empty((case["beams"], case["nfft"]), dtype=torch.complex128, device="cuda")
        step = max(1, (1 << 24) // case["nfft"])
        for b in range(0, case["beams"], step):
            out[b:b + step] = _spectrum64(x[b:b + step], case["nfft"], case["window"])
        if case["out"] == "complex":
            return out
        if case["out"] == "magphase":
            return torch.stack([out.abs(), out.angle()], -1)
        return out.abs() if case["out"] == "mag" else out.real ** 2 + out.imag ** 2
    if kind == "batch":
        rows, pos = [], 0
        for n in _lengths(case, seed):
            rows.append(_top64(_spectrum64(x[None, pos:pos + n], spx.next_smooth23(n), "hann"), case["k"])[0])
            pos += n
        return {"words": None, "values": torch.cat(rows), "counts": None}
    spec = _spectrum64(x, case["nfft"], "hann")
    if kind == "two":
        return {"words": None, "values": _sided64(spec, case["two"]), "counts": None}
    if kind == "learned":
        rec, amp = _learned64(case, spec, _network(seed))
        return {"words": None, "values": rec, "counts": None, "amplitude": amp, "used": None}
    values = _top64(spec, case["k"])[0] if kind == "topk" else _all64(spec)
    return {"words": None, "values": values, "counts": None}
