"""Workloads of the phasing path that are timed from one state of the code to the next.

Each case is one call (or one short sequence of calls) that a user's program
makes through the package's public entry points, on inputs with the
statistics the path meets in use: Poisson-noise diffraction moduli of
ellipse objects, square and multi-part supports, noisy reconstructions.
Sizes are those of the package's workloads, benchmark and tests, and odd
ones between them.

A case is a dict with a ``kind``:

``iterate``   the drop-in call on one reconstruction: ``phasing.iterate`` from
              a given start, a few tens of iterations as between two
              refinements of the support.  Launch-bound at small N.
``trials``    ``phasing.iterate_trials``: random-phase starts advanced
              together; coherent, with an ipsf, with an energy spectrum, both.
``uneven``    one ``Engine.solve`` over trials of different sizes and
              algorithms, as the serving loop issues them.
``refine``    ``refine_support`` (shrinkwrap) on the crop of a support.
``align``     ``align_frames_subpixel`` of a batch's crops to the first.
``prtf``      ``prtf`` of a batch's crops with its azimuthal average.
``rftf``      ``gpu_rftf`` of a batch's crops against the goal modulus.
"""
import math

import numpy as np
import torch

from als_speckle_b200 import phasing as P
from als_speckle_b200.engine import Engine, TrialSpec

# pixel-iterations of the largest listed case (128 trials of 512^2, 10
# iterations); drawn cases stay below it
MOST_PX = 128 * 512 * 512 * 10

ORDERS = {
    "hio": (("hio", 1000),),
    "er": (("er", 1000),),
    "raar": (("raar", 1000),),
    "dm": (("dm", 1000),),
    "hio_er": (("hio", 9), ("er", 1)),
    "raar_dm": (("raar", 12), ("dm", 8)),
}


def listed():
    return [
        # one reconstruction at a time, the reference's own way of working: the smallest
        # work, where launches and latency count
        {"name": "iterate_256", "kind": "iterate", "N": 256, "its": 20, "order": "hio_er", "beta": 0.9},
        # one large reconstruction between two shrinkwraps, two projections per DM iteration
        {"name": "iterate_1024_raar_dm", "kind": "iterate", "N": 1024, "its": 20, "order": "raar_dm", "beta": 0.87},
        # the benchmark's batch: 128 random starts of one 512^2 pattern
        {"name": "trials_512x128", "kind": "trials", "N": 512, "trials": 128, "its": 10, "order": "hio_er",
         "beta": 0.9, "ipsf": False, "spectrum": 0},
        # a middling batch of small patterns that does not fill the GPU evenly
        {"name": "trials_256x45", "kind": "trials", "N": 256, "trials": 45, "its": 12, "order": "raar",
         "beta": 0.87, "ipsf": False, "spectrum": 0},
        # a few very large patterns (full detector frames)
        {"name": "trials_2048x4", "kind": "trials", "N": 2048, "trials": 4, "its": 8, "order": "hio",
         "beta": 0.9, "ipsf": False, "spectrum": 0},
        # transverse partial coherence on a batch
        {"name": "trials_512x32_ipsf", "kind": "trials", "N": 512, "trials": 32, "its": 6, "order": "hio",
         "beta": 0.9, "ipsf": True, "spectrum": 0},
        # both coherence corrections, seven spectral samples
        {"name": "trials_512x16_both", "kind": "trials", "N": 512, "trials": 16, "its": 6, "order": "hio",
         "beta": 0.9, "ipsf": True, "spectrum": 7},
        # a round of the serving loop: sizes and algorithms mixed in one call
        {"name": "uneven_round", "kind": "uneven", "n256": 16, "n512": 8, "n1024": 3, "n2048": 1, "its": 10},
        # shrinkwrap on the crop of a 320^2 support, every 20 iterations of a run
        {"name": "refine_340", "kind": "refine", "rows": 340, "cols": 340, "blur": 2.0},
        # end of a batched job: 128 crops aligned to the first ...
        {"name": "align_128x180", "kind": "align", "frames": 128, "rows": 180, "cols": 180, "upsample": 64},
        # ... their phase-retrieval transfer function and its radial curve ...
        {"name": "prtf_128x180", "kind": "prtf", "N": 512, "frames": 128, "rows": 180, "cols": 180},
        # ... and the Fourier-error counterpart against the measured modulus
        {"name": "rftf_37x173", "kind": "rftf", "N": 512, "frames": 37, "rows": 173, "cols": 181},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate"] * 4 + ["trials"] * 7 + ["uneven"] * 2 + ["refine"] * 2
                      + ["align"] * 2 + ["prtf"] * 2 + ["rftf"])
    if kind == "iterate":
        order = rng.choice(["hio_er", "raar_dm", "raar", "dm", "er"])
        return {"kind": kind, "N": 2 ** rng.randint(6, 11), "its": rng.randint(5, 20), "order": order,
                "beta": rng.choice([0.9, 0.87, 0.8])}
    if kind == "trials":
        N = 2 ** rng.randint(6, 11)
        ipsf, spectrum = rng.choice([(False, 0)] * 4 + [(True, 0), (False, 5), (True, 7)])
        its = rng.randint(4, 8) if ipsf or spectrum else rng.randint(6, 12)
        most = MOST_PX // (N * N * its) // (4 if ipsf or spectrum else 1)
        return {"kind": kind, "N": N, "trials": _log_int(rng, 2, max(2, min(most, 150))), "its": its,
                "order": rng.choice(["hio_er", "hio", "raar", "er"]), "beta": rng.choice([0.9, 0.87]),
                "ipsf": ipsf, "spectrum": spectrum}
    if kind == "uneven":
        return {"kind": kind, "n256": rng.randint(1, 40), "n512": rng.randint(1, 20), "n1024": rng.randint(0, 5),
                "n2048": rng.randint(0, 2), "its": rng.randint(5, 12)}
    rows, cols = _log_int(rng, 60, 400), 0
    cols = max(60, min(400, rows + rng.randint(-20, 20)))
    if kind == "refine":
        return {"kind": kind, "rows": rows, "cols": cols, "blur": round(rng.uniform(0.7, 3.0), 2)}
    frames = _log_int(rng, 4, 128)
    if kind == "align":
        if max(rows, cols) > 256:
            frames = min(frames, 40)
        return {"kind": kind, "frames": frames, "rows": rows, "cols": cols, "upsample": rng.choice([16, 50, 64, 100])}
    N = 512 if max(rows, cols) > 250 else rng.choice([256, 512, 1024])
    if N == 1024:
        frames = min(frames, 32)
    return {"kind": kind, "N": N, "frames": frames, "rows": rows, "cols": cols}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _u(g, shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _object(rows, cols, seed, count, margin=0):
    """(rows, cols) complex128 object: anti-aliased ellipses, one phase each,
    inside a frame of `margin` pixels."""
    g = _gen(seed)
    r = torch.arange(rows, device="cuda", dtype=torch.float64)[:, None]
    c = torch.arange(cols, device="cuda", dtype=torch.float64)[None, :]
    ax = min(15.0, (min(rows, cols) - 2 * margin) / 6.0)
    p = _u(g, (count, 6)).cpu().tolist()
    amp = torch.zeros((rows, cols), device="cuda", dtype=torch.float64)
    ph = torch.zeros_like(amp)
    for u in p:
        a0, a1 = ax * (0.2 + 0.8 * u[0]), ax * (0.2 + 0.8 * u[1])
        lo = margin + ax + 1
        cy, cx = lo + u[2] * max(0.0, rows - 2 * lo), lo + u[3] * max(0.0, cols - 2 * lo)
        th = math.pi * u[4]
        y = (r - cy) * math.cos(th) + (c - cx) * math.sin(th)
        x = (c - cx) * math.cos(th) - (r - cy) * math.sin(th)
        d = torch.sqrt((y / a0) ** 2 + (x / a1) ** 2) * min(a0, a1)
        e = 1 - torch.clamp(d - min(a0, a1), 0, 1)
        take = e > amp
        amp = torch.where(take, e, amp)
        ph = torch.where(take, torch.full_like(ph, (u[5] - 0.5) * math.pi / 2), ph)
    return torch.polar(amp, ph)


def _pattern(N, seed, photons=1e6):
    """(modulus, support) float32 on the GPU: the Poisson-noise modulus of an
    object in the middle N/4 box, and the square 5/16 N support."""
    box = N // 4
    o = torch.zeros((N, N), dtype=torch.complex128, device="cuda")
    a = (N - box) // 2
    o[a:a + box, a:a + box] = _object(box, box, seed, 30)
    i = torch.fft.fft2(o).abs() ** 2
    i *= photons / i.max()
    m = torch.sqrt(torch.poisson(i, generator=_gen(seed + 0x5EED))).float()
    s = torch.zeros((N, N), dtype=torch.float32, device="cuda")
    e = 5 * N // 16
    b = (N - e) // 2
    s[b:b + e, b:b + e] = 1
    return m, s


def _ipsf(N):
    """Transform of a normalised Gaussian point spread of sigma 2 pixels."""
    q = np.fft.fftfreq(N) * N
    g = np.exp(-0.5 * q ** 2 / 4.0)
    f = np.fft.fft(g / g.sum())
    return (f[:, None] * f[None, :]).astype(np.complex64)


def _spectrum(n):
    """(energies, weights): n samples over +-5%, a Gaussian line."""
    return np.stack([np.linspace(0.95, 1.05, n), np.exp(-0.5 * np.linspace(-2, 2, n) ** 2)])


def _frames(case, seed, shifted):
    """Noisy reconstructions of one object: each with its own global phase and,
    if `shifted`, its own subpixel shift."""
    F, rows, cols = case["frames"], case["rows"], case["cols"]
    o = _object(rows, cols, seed, 24, margin=10)
    g = _gen(seed + 77)
    ph = _u(g, (F, 1, 1), -math.pi, math.pi)
    sh = _u(g, (F, 2), -5.0, 5.0)
    f = torch.polar(torch.ones_like(ph), ph) * o
    if shifted:
        ky = torch.fft.fftfreq(rows, device="cuda", dtype=torch.float64)
        kx = torch.fft.fftfreq(cols, device="cuda", dtype=torch.float64)
        t = -2 * math.pi * (sh[:, :1, None] * ky[None, :, None] + sh[:, 1:, None] * kx[None, None, :])
        f = torch.fft.ifft2(torch.fft.fft2(f) * torch.polar(torch.ones_like(t), t))
    n = torch.randn((F, rows, cols, 2), generator=g, device="cuda", dtype=torch.float32)
    return (f.to(torch.complex64) + 0.05 * torch.view_as_complex(n)).contiguous()


def _goal(case, seed):
    """Measured modulus (N, N) of the reconstructed object, at least a photon everywhere."""
    N = case["N"]
    o = torch.zeros((N, N), dtype=torch.complex128, device="cuda")
    o[:case["rows"], :case["cols"]] = _object(case["rows"], case["cols"], seed, 24, margin=10)
    i = torch.fft.fft2(o).abs() ** 2
    return torch.sqrt(torch.poisson(i, generator=_gen(seed + 5)) + 1).float()


def _start(N, s, seed):
    """A start in the support: uniform real and imaginary parts."""
    v = torch.rand((N, N, 2), generator=_gen(seed + 9), device="cuda", dtype=torch.float32)
    return torch.view_as_complex(v) * s


def _uneven_plan(case):
    """(N, algorithm, beta, index) of every trial of a mixed round."""
    algs = [("hio", 0.9), ("raar", 0.87), ("dm", 0.9), ("er", 0.9)]
    plan, k = [], 0
    for N in (256, 512, 1024, 2048):
        for _ in range(case["n%d" % N]):
            plan.append((N,) + algs[k % 4] + (k,))
            k += 1
    return plan


def prepare(case, seed):
    kind = case["kind"]
    if kind == "iterate":
        N = case["N"]
        m, s = _pattern(N, seed)
        r = P.phasing()
        r.load(modulus=m.cpu().numpy(), support=s.cpu().numpy(), numtrials=1)
        return {"case": case, "r": r, "start": _start(N, s, seed)}
    if kind == "trials":
        N = case["N"]
        m, s = _pattern(N, seed, 1e4 if case["ipsf"] or case["spectrum"] else 1e6)
        r = P.phasing()
        r.load(modulus=m.cpu().numpy(), support=s.cpu().numpy(), numtrials=case["trials"],
               ipsf=_ipsf(N) if case["ipsf"] else None,
               spectrum=_spectrum(case["spectrum"]) if case["spectrum"] else None)
        return {"case": case, "r": r, "seed": seed}
    if kind == "uneven":
        pats = {N: _pattern(N, seed + N) for N in (256, 512, 1024, 2048) if case["n%d" % N]}
        specs = []
        for N, alg, beta, k in _uneven_plan(case):
            psi = torch.zeros((N, N), dtype=torch.complex64, device="cuda")
            specs.append(TrialSpec(psi=psi, modulus=pats[N][0], support=pats[N][1], iterations=case["its"],
                                   order=ORDERS[alg], beta=beta, random_phase=True, seed=seed, trial=k))
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        return {"case": case, "engine": Engine(use_graph=True), "stream": stream, "specs": specs}
    if kind == "refine":
        rows, cols = case["rows"], case["cols"]
        o = _object(rows, cols, seed, 24, margin=10)
        n = torch.randn((rows, cols, 2), generator=_gen(seed + 3), device="cuda", dtype=torch.float64)
        avg = (o + 0.03 * torch.view_as_complex(n)).to(torch.complex64)
        # a support of several parts: the object grown by a few pixels
        grown = torch.nn.functional.max_pool2d((o.abs() > 0.1).float()[None, None], 9, 1, 4)[0, 0]
        return {"case": case, "avg": avg, "support": grown.cpu().numpy()}
    if kind == "align":
        return {"case": case, "frames": _frames(case, seed, True)}
    if kind == "prtf":
        return {"case": case, "frames": _frames(case, seed, False)}
    return {"case": case, "frames": _frames(case, seed, False), "goal": _goal(case, seed)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "iterate":
        r = state["r"]
        r.psi_in.copy_(state["start"])
        r.numtrial = 0
        r.iterate(case["its"], order=ORDERS[case["order"]], beta=case["beta"])
        return r.psi_in, r.savebuffer[0], r.errors
    if kind == "trials":
        r = state["r"]
        r.numtrial = 0
        psis = r.iterate_trials(case["its"], case["trials"], order=ORDERS[case["order"]], beta=case["beta"],
                                seed=state["seed"])
        return psis, r.savebuffer[:case["trials"]]
    if kind == "uneven":
        state["engine"].solve(state["specs"], stream=state["stream"])
        return [s.psi for s in state["specs"]]
    if kind == "refine":
        return P.refine_support(state["support"], state["avg"], blur=case["blur"], local_threshold=0.15,
                                global_threshold=0.02)
    if kind == "align":
        return P.align_frames_subpixel(state["frames"], upsample=case["upsample"])
    if kind == "prtf":
        return P.prtf(state["frames"], N=case["N"], prtfq=True)
    return P.gpu_rftf(None, state["frames"], state["goal"])


# ------------------------------------------------------------------ cost
def _fft2(N):
    """Operations of one N x N complex transform."""
    return 5 * N * N * math.log2(N * N)


def work(case):
    """An iteration reads psi, the modulus and the support and writes psi (24
    bytes a pixel; an ipsf adds 8 and two transforms, a spectrum four taps a
    sample); everything else reads its inputs and writes its outputs once."""
    kind = case["kind"]
    if kind in ("iterate", "trials"):
        N, n = case["N"], case.get("trials", 1) * case["its"]
        dm = 0.4 * (case["order"] == "raar_dm") + (case["order"] == "dm")
        ipsf, sp = bool(case.get("ipsf")), case.get("spectrum", 0)
        px = N * N * n
        return {"bytes": px * (24 + 8 * ipsf),
                "flops": n * _fft2(N) * 2 * (1 + dm) * (2 if ipsf else 1) + px * (20 + 12 * sp)}
    if kind == "uneven":
        b = f = 0
        for N, alg, _, _ in _uneven_plan(case):
            b += 24 * N * N * case["its"]
            f += case["its"] * (_fft2(N) * 2 * (2 if alg == "dm" else 1) + 20 * N * N)
        return {"bytes": b, "flops": f}
    rows, cols = case["rows"], case["cols"]
    if kind == "refine":
        # the support comes from and the two maps go back to host arrays
        return {"bytes": rows * cols * (8 + 4 + 4 + 8), "flops": rows * cols * 4 * 8 * case["blur"]}
    F = case["frames"]
    if kind == "align":
        N = 8
        while N < max(rows, cols):
            N *= 2
        M = math.ceil(1.5 * case["upsample"])
        return {"bytes": 16 * F * rows * cols,
                "flops": F * (3 * _fft2(N) + 8 * N * N * M + 8 * N * M * M + 20 * N * N)}
    N = case["N"]
    return {"bytes": F * rows * cols * 8 + 4 * N * N * (1 if kind == "prtf" else 2),
            "flops": F * (_fft2(N) + 8 * N * N)}


# ------------------------------------------------------------------ 64 bits
def _random_start(m, s, seed, trial):
    """S IFFT2(M exp(2 pi i u)), u from the start's counter-based hash."""
    N = m.shape[-1]
    mask = 0xFFFFFFFF
    idx = torch.arange(N * N, device="cuda", dtype=torch.int64)

    def mul(x, c):  # low 32 bits of x * c without overflowing 64
        return ((x & 0xFFFF) * c + ((((x >> 16) * c) & 0xFFFF) << 16)) & mask

    h = (((seed & mask) * 0x9E3779B1) & mask) ^ (((trial & mask) * 0x85EBCA77) & mask)
    h = mul(idx, 0xC2B2AE3D) ^ h
    h ^= h >> 16
    h = mul(h, 0x7FEB352D)
    h ^= h >> 15
    h = mul(h, 0x846CA68B)
    h ^= h >> 16
    u = (h >> 8).double().reshape(N, N) * (2 * math.pi / 16777216.0)
    return s * torch.fft.ifft2(torch.polar(m, u))


def _rescale(d2, spectrum):
    """The radial rescale of the squared divisor: each sample's bilinear gather
    at coordinates divided by its energy ratio, times its weight."""
    N = d2.shape[-1]
    e, w = spectrum
    r = (e / e[w.argmax()]).astype(np.float32)
    w = w.astype(np.float32)
    x = torch.arange(N, device="cuda")
    x = torch.where(x > N // 2 - 1, x - N, x).to(torch.float32)
    out = torch.zeros_like(d2)
    for k in range(len(r)):
        # tap positions in single precision, as the operator defines them
        rc = x / torch.tensor(r[k], device="cuda")
        taps = []
        for c in (torch.floor(rc), torch.floor(rc) + 1):
            ok = (c > -(N // 2)) & (c < N // 2)
            i = torch.where(c < 0, c + N, c).long()
            taps.append((torch.where(ok, i, torch.zeros_like(i)),
                         torch.where(ok, 1 - (c - rc).abs(), torch.zeros_like(c)).double()))
        for iy, wy in taps:
            for ix, wx in taps:
                out += float(w[k]) * wy[:, None] * wx[None, :] * d2[iy][:, ix]
    return out


def _iterate64(psi, m, s, its, order, beta, ipsf=None, spectrum=None):
    """(psi, error sums) after `its` iterations in double precision."""
    beta = float(np.float32(beta))
    flat = [a for a, n in order for _ in range(min(n, its))]
    period = [a for a, n in order for _ in range(n)] if sum(n for _, n in order) <= 100 else flat
    errs = []

    def project(x):
        f = torch.fft.fft2(x)
        div = f.abs()
        e = div - m
        if ipsf is not None or spectrum is not None:
            d2 = div ** 2
            if ipsf is not None:
                d2 = torch.fft.ifft2(torch.fft.fft2(d2) * ipsf).abs()
            if spectrum is not None:
                d2 = _rescale(d2, spectrum)
            div = torch.sqrt(d2)
        p = torch.where(div > 0, f * (m / torch.where(div > 0, div, torch.ones_like(div))), m.to(f.dtype))
        return torch.fft.ifft2(p), e

    for i in range(its):
        alg = period[i % len(period)]
        po, e = project(psi)
        errs.append(torch.stack([(e * e).sum(), e.abs().sum()]))
        if alg == "hio":
            psi = (1 - s) * (psi - beta * po) + s * po
        elif alg == "er":
            psi = s * po
        elif alg == "raar":
            psi = (1 - s) * (beta * psi + (1 - 2 * beta) * po) + s * po
        else:
            g = 1 / beta
            t, _ = project(psi * (-g + (1 + g) * s))
            psi = psi + po * (-beta + (1 + 2 * beta) * s) - s * beta * t
    return psi, torch.stack(errs)


def _box(s):
    """The crop of the support: its bounding box and 10 pixels around it."""
    nz = (s > 1e-10).nonzero()
    n = s.shape[0]
    lo, hi = (nz.min(0).values - 10).clamp(min=0).tolist(), (nz.max(0).values + 11).clamp(max=n).tolist()
    return lo[0], hi[0], lo[1], hi[1]


def exact(case, seed):
    kind = case["kind"]
    if kind == "iterate":
        m, s = _pattern(case["N"], seed)
        psi, errs = _iterate64(_start(case["N"], s, seed).to(torch.complex128), m.double(), s.double(),
                               case["its"], ORDERS[case["order"]], case["beta"])
        a, b, c, d = _box(s)
        return psi, psi[a:b, c:d], errs
    if kind == "trials":
        N = case["N"]
        m, s = _pattern(N, seed, 1e4 if case["ipsf"] or case["spectrum"] else 1e6)
        ipsf = torch.from_numpy(_ipsf(N)).cuda().to(torch.complex128) if case["ipsf"] else None
        sp = _spectrum(case["spectrum"]) if case["spectrum"] else None
        a, b, c, d = _box(s)
        m, s = m.double(), s.double()
        psis = torch.stack([_iterate64(_random_start(m, s, seed, k), m, s, case["its"], ORDERS[case["order"]],
                                       case["beta"], ipsf, sp)[0].to(torch.complex128)
                            for k in range(case["trials"])])
        return psis, psis[:, a:b, c:d].contiguous()
    if kind == "uneven":
        pats = {N: _pattern(N, seed + N) for N in (256, 512, 1024, 2048) if case["n%d" % N]}
        out = []
        for N, alg, beta, k in _uneven_plan(case):
            m, s = pats[N][0].double(), pats[N][1].double()
            out.append(_iterate64(_random_start(m, s, seed, k), m, s, case["its"], ORDERS[alg], beta)[0])
        return out
    if kind == "refine":
        avg = prepare(case, seed)["avg"].to(torch.complex128).abs()
        k = []
        for n in avg.shape:
            x = torch.arange(n, device="cuda", dtype=torch.float64)
            g = torch.exp(-(x - n // 2) ** 2 / (2 * float(case["blur"]) ** 2))
            k.append(torch.fft.fft(torch.fft.fftshift(g) / g.sum()))
        return None, torch.fft.ifft2(torch.fft.fft2(avg) * k[0][:, None] * k[1][None, :]).real
    if kind == "align":
        return _align64(prepare(case, seed)["frames"].to(torch.complex128), case["upsample"])
    N, rows, cols = case["N"], case["rows"], case["cols"]
    state = prepare(case, seed)
    f = torch.zeros((N, N), dtype=torch.complex128, device="cuda")
    acc = torch.zeros((N, N), dtype=torch.complex128, device="cuda")
    for x in state["frames"]:
        f.zero_()
        f[:rows, :cols] = x
        t = torch.fft.fft2(f)
        if kind == "prtf":
            acc += t / t.abs()
        else:
            g = state["goal"].double()
            acc += 1 / torch.sqrt(1 + (g - t.abs()) ** 2 / (g * g))
    return (torch.fft.fftshift(acc.abs() / case["frames"]), None) if kind == "prtf" else \
        torch.fft.fftshift(acc.real / case["frames"])


def _align64(t, U):
    F, rows, cols = t.shape
    N = 8
    while N < max(rows, cols):
        N *= 2
    f = torch.zeros((F, N, N), dtype=torch.complex128, device="cuda")
    f[:, :rows, :cols] = t
    f = torch.fft.fft2(f)
    x = f * f[0].conj()
    peak = torch.fft.fftshift(torch.fft.ifft2(x).abs(), dim=(1, 2)).reshape(F, -1).argmax(1)
    d0 = torch.stack([peak // N - N // 2, peak % N - N // 2], 1).double()
    k = torch.arange(N, device="cuda", dtype=torch.float64)
    k = torch.where(k >= N // 2, k - N, k)
    M = (3 * U + 1) // 2
    q = torch.arange(M, device="cuda", dtype=torch.float64) - M // 2

    def turn(v):
        return torch.polar(torch.ones_like(v), 2 * math.pi * v)

    w = turn(k[:, None] * q[None, :] / (U * N))
    x = x * turn((d0[:, :1] * k) / N)[:, :, None] * turn((d0[:, 1:] * k) / N)[:, None, :]
    up = w.T @ (x @ w)
    best = up.abs().reshape(F, -1).argmax(1)
    theta = up.reshape(F, -1).gather(1, best[:, None]).angle()
    d = d0 + torch.stack([q[best // M], q[best % M]], 1) / U
    f = f * turn(d[:, :1] * k / N)[:, :, None] * turn(d[:, 1:] * k / N)[:, None, :]
    f = f * torch.polar(torch.ones_like(theta), -theta)[:, :, None]
    return torch.fft.ifft2(f)[:, :rows, :cols].contiguous()
