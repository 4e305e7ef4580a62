"""Timed cases of the wavelet transforms.

A case is one pass through the public entry points on one GPU: the device
API (`s2dw_b200.device.Plan`) for programs that keep maps in GPU memory, and
the drop-in host functions (`s2dw_b200.core`) for programs that hold numpy
arrays.  `listed()` names the fixed cases, `draw()` gives more of the same
ranges, `prepare()` makes what a program has before the call, `run()` is the
pass, `work()` its unavoidable bytes and operations, and `exact()` the same
outputs from plain numpy and torch in 64 bits (direct sums with the Wigner d
functions at the sample angles, and torch.fft), without the library.

The kernel tables are the S2DW harmonic tiling and steerable directionality,
evaluated here so that the library and `exact()` start from the same numbers.
"""
import functools
import math

import numpy as np
import torch

from s2dw_b200 import core
from s2dw_b200.device import Plan

KINDS = ("analysis", "synthesis", "pair", "moments", "batch", "host")


def listed():
    return [
        # the smallest transform: a low-resolution map in an interactive
        # loop, where launches and latency are all there is
        {"name": "analysis_b32_n3", "kind": "analysis", "B": 32, "N": 3, "alpha": 2.0, "maps": 1},
        # a small map back to harmonic space, five orientations
        {"name": "synthesis_b64_n5", "kind": "synthesis", "B": 64, "N": 5, "alpha": 2.0, "maps": 1},
        # a band limit that is not a power of two (every scale ragged)
        {"name": "analysis_b100_n4", "kind": "analysis", "B": 100, "N": 4, "alpha": 2.0, "maps": 1},
        # axisymmetric wavelets (N = 1): filtering a map and putting it back
        {"name": "pair_b128_n1", "kind": "pair", "B": 128, "N": 1, "alpha": 2.0, "maps": 1},
        # the ordinary directional round trip of a degraded map
        {"name": "pair_b256_n5", "kind": "pair", "B": 256, "N": 5, "alpha": 2.0, "maps": 1},
        # few, wide scales (alpha = 3) at an odd band limit: a survey's lmax + 1
        {"name": "synthesis_b301_n2_a3", "kind": "synthesis", "B": 301, "N": 2, "alpha": 3.0, "maps": 1},
        # full resolution, each direction: the headline configuration
        {"name": "analysis_b1024_n4", "kind": "analysis", "B": 1024, "N": 4, "alpha": 2.0, "maps": 1},
        {"name": "synthesis_b1024_n4", "kind": "synthesis", "B": 1024, "N": 4, "alpha": 2.0, "maps": 1},
        # the statistics of simulations: analysis of a few maps, moments of
        # the masked coefficients per scale, coefficients left on the GPU
        {"name": "moments_b512_n4_x4", "kind": "moments", "B": 512, "N": 4, "alpha": 2.0, "maps": 4},
        # a Monte-Carlo batch through the split-precision form, both ways
        {"name": "batch_b512_n4_x32", "kind": "batch", "B": 512, "N": 4, "alpha": 2.0, "maps": 32},
        # a reference program's call: numpy arrays in, numpy arrays out
        {"name": "host_b256_n4", "kind": "host", "B": 256, "N": 4, "alpha": 2.0, "maps": 1},
        # the largest band limit with eight orientations
        {"name": "pair_b2048_n8", "kind": "pair", "B": 2048, "N": 8, "alpha": 2.0, "maps": 1},
    ]


def draw(rng):
    """One more case: every kind, band limits over their logarithm (half of
    them powers of two, as the reference's programs use, half any number)."""
    kind = rng.choice(("analysis", "synthesis", "pair", "analysis", "synthesis", "pair", "moments", "batch", "host"))
    lo, hi = {"moments": (32, 512), "batch": (32, 320), "host": (32, 512)}.get(kind, (32, 1100))
    B = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5:
        B = 1 << int(round(math.log2(B)))
    B = min(B, hi)
    return {
        "kind": kind,
        "B": B,
        "N": rng.randint(1, 5 if kind == "batch" else 8),
        "alpha": rng.choice((2.0, 2.0, 2.0, 3.0, 1.7)),
        "maps": rng.randint(2, 6) if kind == "moments" else rng.randint(16, 32) if kind == "batch" else 1,
    }


# ---------------------------------------------------------------------------
# Parameters and kernel tables
# ---------------------------------------------------------------------------
def _near_int(x, otherwise):
    r = round(x)
    return int(r) if abs(x - r) < 1e-5 else int(otherwise(x))


def _jmax(B, alpha):
    return _near_int(math.log(B) / math.log(alpha), math.ceil)


def _bands(B, alpha, J):
    """(bl_hi, bl_lo) of every scale: scale j holds bl_lo < l < bl_hi."""
    return [(min(B, _near_int(B / alpha ** (j - 1), math.ceil)), max(0, _near_int(B / alpha ** (j + 1), math.floor)))
            for j in range(J + 1)]


def _phi2(bw, lo, B):
    """Scaling function squared, l < B: the tail integral of
    exp(-2/(1-t^2))/k over (lo, bw), 1 below lo and 0 above bw."""
    t, w = np.polynomial.legendre.leggauss(48)
    k = np.arange(lo, bw)[:, None] + 0.5 * (t + 1.0)
    u = 2.0 * (k - lo) / (bw - lo) - 1.0
    part = (np.exp(-2.0 / (1.0 - u * u)) / k * (0.5 * w)).sum(1)
    tail = np.cumsum(part[::-1])[::-1]
    out = np.zeros(max(B, bw) + 1)
    out[:lo + 1] = 1.0
    out[lo:bw] = tail / tail[0]
    return out[:B]


@functools.lru_cache(maxsize=64)
def _tables(B, N, alpha):
    """J, K_gamma (J+1, B), Phi2 (B,), bl_scoeff and Slm (B, N)."""
    J = _jmax(B, alpha)
    bw = [_near_int(B / alpha ** (j - 1), math.ceil) for j in range(J + 2)]
    phi2 = np.stack([_phi2(b, _near_int(b / alpha, math.floor), B) for b in bw])
    K = np.sqrt(np.maximum(phi2[:-1] - phi2[1:], 0.0))
    S = np.zeros((B, N), dtype=np.complex128)
    for l in range(1, B):
        g = min(N - 1, l - (0 if (N + l) % 2 else 1))
        for m in range(min(l, N - 1) + 1):
            if (N + m) % 2:
                S[l, m] = math.sqrt(math.comb(g, (g - m) // 2) / 2.0 ** g) if m <= g else 0.0
    if N % 2 == 0:
        S = S * 1j
    return J, np.asfortranarray(K), phi2[-1].copy(), bw[-1], np.asfortranarray(S)


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _flm(B, rng):
    """Harmonic coefficients of a real Gaussian map, C_l = 1/(l(l+1)), l >= 2,
    as flm[l, m], m <= l."""
    l = np.arange(B, dtype=np.float64)
    c = np.zeros(B)
    c[2:] = 1.0 / (l[2:] * (l[2:] + 1.0))
    f = rng.standard_normal((B, B)) + 1j * rng.standard_normal((B, B))
    f *= np.sqrt(0.5 * c)[:, None]
    f[:, 0] = rng.standard_normal(B) * np.sqrt(c)
    return np.asfortranarray(np.tril(f))


def _flms(case, seed):
    rng = np.random.default_rng([seed, 1])
    return [_flm(case["B"], rng) for _ in range(case["maps"])]


def _wav_shapes(case, J):
    return [(case["N"], 2 * hi, 2 * hi - 1) for hi, _ in _bands(case["B"], case["alpha"], J)]


def _wavs(case, seed, J, bs):
    """Noise coefficients per scale (packed, each (N, 2bl, 2bl-1) in C order)
    whose level grows with the scale as a map's do, and a scaling part."""
    rng = np.random.default_rng([seed, 2])
    wav = [rng.standard_normal(s) * (0.02 * 1.5 ** j) for j, s in enumerate(_wav_shapes(case, J))]
    sc = np.tril(rng.standard_normal((bs, bs)) + 1j * rng.standard_normal((bs, bs)))
    sc[:, 0] = sc[:, 0].real
    return wav, np.asfortranarray(sc)


def _mask(case, seed, J):
    """A mask of one map's coefficients: 1 kept, 0 removed (a band around the
    equator and scattered holes)."""
    rng = np.random.default_rng([seed, 3])
    out = []
    for n, nb, na in _wav_shapes(case, J):
        m = (rng.random((n, nb, na)) > 0.05).astype(np.float64)
        m[:, int(0.46 * nb):int(0.54 * nb)] = 0.0
        out.append(m)
    return out


def _pack(parts):
    return np.concatenate([p.reshape(-1) for p in parts])


def prepare(case, seed):
    B, N, alpha, maps, kind = case["B"], case["N"], case["alpha"], case["maps"], case["kind"]
    J, K, P, bs, S = _tables(B, N, alpha)
    if kind == "host":
        return {"kind": kind, "flm": _flms(case, seed)[0], "args": (K, S, J, B, N, bs, alpha),
                "back": (K, P, S, J, B, N, bs, alpha)}
    plan = Plan(B, N, alpha, J, form=Plan.SPLIT if kind == "batch" else Plan.FP64)
    plan.set_tables(K, P, S, bs)
    if kind == "batch":
        plan.reserve(maps)
    st = {"kind": kind, "plan": plan}
    lead = () if kind in ("analysis", "synthesis", "pair") else (maps,)
    if kind == "synthesis":
        wav, sc = _wavs(case, seed, J, bs)
        st["wav"] = torch.from_numpy(_pack(wav)).cuda()
        st["scoeff"] = torch.from_numpy(np.ascontiguousarray(sc.T)).cuda()
    else:
        f = np.stack([np.ascontiguousarray(x.T) for x in _flms(case, seed)])
        st["flm"] = torch.from_numpy(f.reshape(lead + (B, B))).cuda()
        st["wav"] = torch.empty(lead + (plan.wav_size,), dtype=torch.float64, device="cuda")
        st["scoeff"] = torch.empty(lead + (bs, bs), dtype=torch.complex128, device="cuda")
    if kind in ("synthesis", "pair", "batch"):
        st["out"] = torch.empty(lead + (B, B), dtype=torch.complex128, device="cuda")
    if kind == "moments":
        st["mask"] = torch.from_numpy(_pack(_mask(case, seed, J))).cuda()
        st["moments"] = torch.empty((maps, J + 1, 6), dtype=torch.float64, device="cuda")
    return st


def run(st):
    kind = st["kind"]
    if kind == "host":
        wav, sc = core.s2dw_core_analysis_flm2wav_dynamic(st["flm"], *st["args"])
        kept = list(wav)  # the synthesis empties its list, as the reference does
        flm = core.s2dw_core_synthesis_wav2flm_dynamic(wav, sc, *st["back"])
        return {"wav": kept, "scoeff": sc, "flm": flm}
    plan = st["plan"]
    if kind == "analysis":
        plan.analysis(st["flm"], st["wav"], st["scoeff"])
        return {"wav": st["wav"], "scoeff": st["scoeff"]}
    if kind == "synthesis":
        plan.synthesis(st["wav"], st["scoeff"], st["out"])
        return {"flm": st["out"]}
    if kind == "pair":
        plan.analysis(st["flm"], st["wav"], st["scoeff"])
        plan.synthesis(st["wav"], st["scoeff"], st["out"])
        return {"wav": st["wav"], "scoeff": st["scoeff"], "flm": st["out"]}
    if kind == "moments":
        plan.analysis_batch(st["flm"], st["wav"], st["scoeff"])
        plan.stat_moments(st["wav"], st["moments"], st["mask"])
        return {"wav": st["wav"], "scoeff": st["scoeff"], "moments": st["moments"]}
    plan.analysis_batch(st["flm"], st["wav"], st["scoeff"])
    plan.synthesis_batch(st["wav"], st["scoeff"], st["out"])
    return {"wav": st["wav"], "scoeff": st["scoeff"], "flm": st["out"]}


def work(case):
    """Bytes: flm (l >= m), wavelets, scaling part (and mask, moments), each
    once per direction.  Operations per scale and direction: the
    multiply-adds of the l / m' contractions (one real d factor times a complex value per
    (l, m, m', n); the analysis needs both signs of n, the synthesis n >= 0)
    and 5 L log2 L per complex beta (L = 2bl) and packed alpha (L = 2bl-1)
    transform."""
    B, N, maps, kind = case["B"], case["N"], case["maps"], case["kind"]
    J = _jmax(B, case["alpha"])
    bands = _bands(B, case["alpha"], J)
    npos = len([n for n in range(N) if (N + n) % 2])
    nall = N
    wav = sum((2 * hi - 1) * 2 * hi * N for hi, _ in bands)
    bs = _near_int(B / case["alpha"] ** J, math.ceil)
    ana = syn = 0.0
    for hi, lo in bands:
        mac = sum((l + 1.0) ** 2 for l in range(lo + 1, hi))
        beta, alpha = (5.0 * L * math.log2(max(2, L)) for L in (2 * hi, 2 * hi - 1))
        ana += 4.0 * mac * nall + N * hi * (beta + alpha)
        syn += 4.0 * mac * npos + npos * hi * beta + N * hi * alpha
    one = 16.0 * B * (B + 1) / 2 + 8.0 * wav + 16.0 * bs * bs
    both = kind in ("pair", "batch", "host")
    flops = syn if kind == "synthesis" else ana + syn if both else ana
    nbytes = 2 * one if both else one
    if kind == "moments":
        nbytes += 8.0 * wav / maps + 48.0 * (J + 1)
        flops += 12.0 * wav
    return {"bytes": nbytes * maps, "flops": flops * maps}


# ---------------------------------------------------------------------------
# The same outputs from direct sums in 64 bits
# ---------------------------------------------------------------------------
def _wigner(bl, n, beta):
    """Yields (l, d) for l = |n|..bl-1 with d[m, b] = d^l_{mn}(beta_b),
    m = 0..l (for l >= |n|), by the three-term recurrence in l started from
    the closed forms at l = max(m, |n|)."""
    dev, an = beta.device, abs(n)
    c, s, x = torch.cos(beta / 2), torch.sin(beta / 2), torch.cos(beta)
    cur = torch.zeros((bl, beta.numel()), dtype=torch.float64, device=dev)
    prev = torch.zeros_like(cur)
    for m in range(min(an, bl - 1) + 1):
        co = math.sqrt(math.comb(2 * an, an + m))
        if n >= 0:
            cur[m] = co * c ** (an + m) * s ** (an - m)
        else:
            cur[m] = (-1) ** (m + an) * co * c ** (an - m) * s ** (an + m)
    edge = cur[min(an, bl - 1)].clone()  # d^m_{mn} at m = |n|
    ms = torch.arange(bl, dtype=torch.float64, device=dev)
    for l in range(an, bl):
        yield l, cur[:l + 1]
        if l + 1 == bl:
            return
        r = ms[:l + 1]
        if l == 0:
            nxt = cur[:1] * x
        else:
            den = l * torch.sqrt((l + 1 - r) * (l + 1 + r) * float((l + 1) ** 2 - n * n))
            a = ((2 * l + 1) * l * (l + 1.0) / den)[:, None]
            b = ((2 * l + 1) * r * n / den)[:, None]
            q = ((l + 1) * torch.sqrt((l - r) * (l + r) * float(l * l - n * n)) / den)[:, None]
            nxt = torch.addcmul((a * x - b) * cur[:l + 1], q, prev[:l + 1], value=-1.0)
        edge = -math.sqrt((2 * l + 1) * (2 * l + 2) / float((l + 1 + n) * (l + 1 - n))) * edge * c * s
        prev[:l + 1] = cur[:l + 1]
        cur[:l + 1] = nxt
        cur[l + 1] = edge


def _beta(bl, dev):
    return math.pi * (2.0 * torch.arange(2 * bl, dtype=torch.float64, device=dev) + 1.0) / (4.0 * bl)


def _nset(N, signed):
    return [n for n in range(-(N - 1) if signed else 0, N) if (N + n) % 2]


def _phase(n, N, dev):
    g = torch.arange(N, dtype=torch.float64, device=dev) * (math.pi * n / N)
    return torch.complex(torch.cos(g), torch.sin(g))


def _analysis(f, hi, lo, K, S, N):
    """One scale's coefficients (maps, N, 2bl, 2bl-1) of f (maps, l, m)."""
    dev, maps = f.device, f.shape[0]
    X = torch.zeros((maps, N, hi, 2 * hi), dtype=torch.complex128, device=dev)
    for n in _nset(N, True):
        acc = torch.zeros((maps, 2, hi, 2 * hi), dtype=torch.float64, device=dev)
        for l, d in _wigner(hi, n, _beta(hi, dev)):
            if l > lo:
                kap = (-1) ** n * K[l] * S[l, -n] if n < 0 else np.conj(K[l] * S[l, n])
                v = f[:, l, :l + 1] * complex(kap)
                acc[:, :, :l + 1].addcmul_(torch.stack((v.real, v.imag), 1)[..., None], d)
        X += _phase(n, N, dev)[:, None, None] * torch.complex(acc[:, 0], acc[:, 1])[:, None]
    if hi == 1:
        return X.real.transpose(2, 3).contiguous()
    return torch.fft.irfft(X, n=2 * hi - 1, dim=2, norm="forward").transpose(2, 3).contiguous()


def _synthesis(wav, sc, bands, K, P, S, B, N):
    """flm (maps, l, m) from per-scale wav (maps, N, 2bl, 2bl-1) and sc (maps, l, m)."""
    dev, maps = sc.device, sc.shape[0]
    out = torch.zeros((maps, B, B), dtype=torch.complex128, device=dev)
    for j, (hi, lo) in enumerate(bands):
        if lo + 1 >= hi:
            continue
        be = _beta(hi, dev)
        k = 2.0 * torch.arange(hi, dtype=torch.float64, device=dev) + 1.0
        q = (2.0 / hi) * torch.sin(be) * (torch.sin(be[:, None] * k) / k).sum(1)
        Y = torch.fft.rfft(wav[j], dim=3).transpose(2, 3) * (4.0 * math.pi ** 2 / N / (2 * hi - 1))
        for n in _nset(N, False):
            Z = (Y * _phase(-n, N, dev)[:, None, None]).sum(1) * q  # (maps, m, b)
            Z = torch.stack((Z.real, Z.imag), 1)
            for l, d in _wigner(hi, n, be):
                if l > lo:
                    fac = (1 if n == 0 else 2) * (2 * l + 1) / (8.0 * math.pi ** 2) * K[j, l] * S[l, n]
                    v = (Z[:, :, :l + 1] * d).sum(-1)
                    out[:, l, :l + 1] += complex(fac) * torch.complex(v[:, 0], v[:, 1])
    bs = sc.shape[1]
    out[:, :bs, :bs] += torch.from_numpy(P[:bs, None]).to(dev) * sc
    return out


def _moments(w, mask):
    """mean, variance, skewness, excess kurtosis, fifth and excess sixth
    standardised moments of the kept values of each map's scale."""
    keep = mask.reshape(-1) > 0.5
    x = w.reshape(w.shape[0], -1)[:, keep]
    nj = float(x.shape[1])
    mu = x.mean(1, keepdim=True)
    s = x - mu
    v = ((s * s).sum(1) - s.sum(1) ** 2 / nj) / (nj - 1.0)
    ok = v >= 1e-12
    sd = torch.sqrt(torch.where(ok, v, torch.ones_like(v)))
    hig = [(s ** p).sum(1) / (nj * sd ** p) - e for p, e in ((3, 0.0), (4, 3.0), (5, 0.0), (6, 15.0))]
    hig = [torch.where(ok, h, torch.zeros_like(h)) for h in hig]
    return torch.stack([mu[:, 0], v] + hig, 1)


def exact(case, seed):
    B, N, alpha, maps, kind = case["B"], case["N"], case["alpha"], case["maps"], case["kind"]
    if B > 1200:  # the start values of the recurrence leave the double range
        return None
    J, K, P, bs, S = _tables(B, N, alpha)
    bands = _bands(B, alpha, J)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "synthesis":
        wav, sc = _wavs(case, seed, J, bs)
        w = [torch.from_numpy(x)[None].to(dev) for x in wav]
        flm = _synthesis(w, torch.from_numpy(np.ascontiguousarray(sc)).to(dev)[None], bands, K, P, S, B, N)
        return {"flm": flm[0].T.contiguous()}
    f = torch.from_numpy(np.stack([np.ascontiguousarray(x) for x in _flms(case, seed)])).to(dev)
    w = [_analysis(f, hi, lo, K[j], S, N) for j, (hi, lo) in enumerate(bands)]
    sc = f[:, :bs, :bs]
    if kind == "host":
        flm = _synthesis(w, sc, bands, K, P, S, B, N)[0]
        return {"wav": [x[0].permute(2, 1, 0).cpu().numpy() for x in w], "scoeff": sc[0].cpu().numpy(),
                "flm": flm.cpu().numpy()}
    out = {"wav": torch.cat([x.reshape(maps, -1) for x in w], 1), "scoeff": sc.transpose(1, 2).contiguous()}
    if kind == "moments":
        mask = [torch.from_numpy(m).to(dev) for m in _mask(case, seed, J)]
        out["moments"] = torch.stack([_moments(x, m) for x, m in zip(w, mask)], 1)
        return out
    if kind in ("pair", "batch"):
        out["flm"] = _synthesis(w, sc, bands, K, P, S, B, N).transpose(1, 2).contiguous()
    if kind in ("analysis", "pair"):
        out = {k: v[0] for k, v in out.items()}
    return out
