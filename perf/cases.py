"""Workloads of the acquisition engine, for timing it and comparing its results.

Every case is one call (or one short sequence of calls) of the public Python
binding, tart-gnss_b200/tga.py, on host data as the TART observation files
hold it: packed one-bit rows, one row per antenna.  The recordings are
synthetic: satellites of every constellation searched with random code
phase, Doppler within +-4 kHz, per-epoch sign flips and per-antenna carrier
phase, in unit noise, quantised to one bit, made on the GPU from the seed.

A program keeps one engine context per arithmetic for its whole life and
sends one recording after another through it, so the contexts are kept here
as well, one per precision; a state holds one recording.

Results that the engine computes in 32 bits (peaks, second peaks, C/N0 and
block powers, widened to f64 by the reference's result structs) are returned
in 32 bits; lags, bins and hypotheses as whole numbers.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "tart-gnss_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import tga  # noqa: E402

FS = 16.368e6  # the TART receiver's rate, 16 samples per C/A chip
IF = 4.092e6
BAND = 6000.0
CONST = {"gps": tga.GPS, "galileo": tga.GALILEO, "beidou": tga.BEIDOU, "sbas": tga.SBAS, "l1c": tga.L1C,
         "qzss": tga.QZSS}
PRECISION = {"fp32": tga.PRECISION_FP32, "tc": tga.PRECISION_FP16_TC}
# rates with a whole number of samples per chip; S of 1, 2, 4 and 8 are left
# out because there the 4.092 MHz carrier is a multiple of half the rate and
# the bins +f and -f of a real recording tie exactly
SAMPLES_PER_CHIP = (6, 10, 12, 14, 16, 18, 20)


def _single(name, const, prn, fs=FS, precision="fp32"):
    return {"name": name, "kind": "single", "const": const, "prn": prn, "fs": fs, "precision": precision}


def _cells(name, consts, n_ant, ms=100, fs=FS, n_prn=0, ant_step=1, cn0=False, precision="fp32"):
    return {"name": name, "kind": "cells", "consts": consts, "n_ant": n_ant, "ms": ms, "fs": fs, "n_prn": n_prn,
            "ant_step": ant_step, "cn0": cn0, "precision": precision}


def _nc(name, consts, n_ant, periods, blocks, step, bins, n_prn=0, ms=100, cn0_lo=38.0, cn0_hi=50.0,
        precision="fp32"):
    # periods, blocks, step and bins of a C/A search; the longer codes take
    # the same span of time per block and bins as fine (see _nc_searches)
    return {"name": name, "kind": "nc", "consts": consts, "n_ant": n_ant, "periods": periods, "blocks": blocks,
            "step": step, "bins": bins, "n_prn": n_prn, "ms": ms, "cn0_lo": cn0_lo, "cn0_hi": cn0_hi,
            "precision": precision}


ALL = "gps galileo beidou sbas l1c qzss"


def listed():
    return [
        # one PRN on one antenna, the smallest call a program makes (the
        # tool's --benchmark and every acquire_full of the library): latency
        _single("single_gps", "gps", 11),
        # the same call on the longest code, 10 ms of BOC chips
        _single("single_l1c", "l1c", 5),
        # a rate with no whole number of samples per chip: the generic path
        _single("single_gps_16mhz", "gps", 7, fs=16.0e6),
        # one constellation, some antennas and PRNs, another sampling rate
        # (18 samples per chip): a receiver that looks for few satellites
        _cells("cells_odd", "gps beidou", 5, ms=40, fs=18 * 1.023e6, n_prn=13, ant_step=2, cn0=True),
        # a whole-sky search on one antenna, tensor cores
        _cells("all_1ant_tc", ALL, 1, cn0=True, precision="tc"),
        # the tool's --all on a 24-antenna TART recording, in the default
        # arithmetic and on the tensor cores with --cn0
        _cells("all_24ant_fp32", ALL, 24),
        _cells("all_24ant_tc", ALL, 24, cn0=True, precision="tc"),
        # plain non-coherent GPS search: 1 ms x 10, 21 bins of 500 Hz
        _nc("nc_plain_gps", "gps", 1, 1, 10, 500.0, 21, n_prn=32, ms=10),
        # weak signals: 10 ms x 10 over 201 bins of 50 Hz, 24 antennas
        _nc("nc_weak_gps_tc", "gps", 24, 10, 10, 50.0, 201, n_prn=32, cn0_lo=28.0, cn0_hi=36.0, precision="tc"),
        # non-coherent whole-sky search over 100 ms, one antenna
        _nc("nc_all_1ant_tc", ALL, 1, 1, 100, 500.0, 21, precision="tc"),
        # refinement of 12 found satellites over 24 antennas and 10 ms
        {"name": "fine_24ant", "kind": "fine", "n_ant": 24, "n_sat": 12, "ms": 10, "precision": "fp32"},
        # interference scan of a 24-antenna recording of 100 ms
        {"name": "rfi_24ant", "kind": "rfi", "n_ant": 24, "ms": 100, "precision": "fp32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "cells", "cells", "cells", "nc", "nc", "fine", "rfi"])
    precision = rng.choice(["fp32", "tc"])
    if kind == "single":
        const = rng.choice(sorted(CONST))
        lo, hi = tga.PRN_RANGE[CONST[const]]
        generic = const in ("gps", "galileo") and rng.random() < 0.25
        fs = 16.0e6 if generic else 1.023e6 * rng.choice(SAMPLES_PER_CHIP)
        c = _single("", const, rng.randint(lo, min(hi, lo + 31)), fs, "fp32" if generic else precision)
    elif kind == "cells":
        consts = " ".join(sorted(rng.sample(sorted(CONST), rng.choice([1, 1, 2, 3, 6]))))
        same_prns = all(k in ("gps", "galileo", "beidou", "l1c") for k in consts.split())
        n_ant = _log(rng, 1, 12 if precision == "fp32" else 24)
        c = _cells("", consts, n_ant, ms=rng.choice([20, 33, 50, 100]), fs=1.023e6 * rng.choice(SAMPLES_PER_CHIP[:5]),
                   n_prn=rng.randint(1, 37) if same_prns else 0, ant_step=rng.choice([1, 1, 2]),
                   cn0=rng.random() < 0.5, precision=precision)
    elif kind == "nc":
        consts = " ".join(sorted(rng.sample(sorted(CONST), rng.choice([1, 1, 2]))))
        same_prns = all(k in ("gps", "galileo", "beidou", "l1c") for k in consts.split())
        periods = rng.choice([1, 2, 5, 10])
        n_ant = _log(rng, 1, 4)
        blocks = rng.randint(1, max(1, 60 // periods))
        c = _nc("", consts, n_ant, periods, blocks, 500.0 / periods, rng.choice([11, 21, 31, 41]),
                n_prn=rng.randint(1, 37) if same_prns else 0, ms=max(20, 10 * -(-periods * blocks // 10)),
                precision=precision)
    elif kind == "fine":
        c = {"kind": "fine", "n_ant": _log(rng, 2, 24), "n_sat": rng.randint(1, 16), "ms": rng.choice([4, 8, 10]),
             "precision": "fp32"}
    else:
        c = {"kind": "rfi", "n_ant": _log(rng, 1, 24), "ms": rng.choice([20, 33, 50, 100]), "precision": "fp32"}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------------------
# recordings
# ---------------------------------------------------------------------------
def _period(c, fs):
    return int(fs / 1000.0) if c in (tga.GPS, tga.SBAS, tga.QZSS) else int(fs * (0.004 if c == tga.GALILEO else 0.010))


def _prns(c, n):
    lo, hi = tga.PRN_RANGE[c]
    return list(range(lo, hi + 1)) if not n else list(range(lo, min(hi, lo + n - 1) + 1))


def _recording(seed, consts, n_ant, n, fs, n_prn=0, per_const=8, cn0=(38.0, 50.0), interferer=False):
    """Packed rows [n_ant, n / 8] and the satellites in them."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    t = torch.arange(n, device="cuda", dtype=torch.int64)
    v = torch.randn((n_ant, n), generator=gen, device="cuda")
    sats = []
    for c in consts:
        prns = _prns(c, n_prn)
        P = _period(c, fs)
        for prn in rng.choice(prns, size=min(per_const, len(prns)), replace=False):
            s = dict(c=c, prn=int(prn), P=P, delay=int(rng.integers(0, P)), dop=float(rng.uniform(-4000, 4000)),
                     cn0=float(rng.uniform(*cn0)))
            code = torch.from_numpy(tga.code_resampled(c, int(prn), float(P), P)).cuda()
            flips = torch.from_numpy(rng.choice([-1.0, 1.0], size=n // P + 2).astype(np.float32)).cuda()
            amp = 2.0 * math.sqrt(10.0 ** (s["cn0"] / 10.0) / fs)
            i = t + s["delay"]
            chip = amp * code[i % P] * flips[i // P]
            ph = 2 * math.pi * torch.frac(((IF + s["dop"]) / fs) * t.double()).float()
            re, im = chip * torch.cos(ph), chip * torch.sin(ph)
            for a, th in enumerate(rng.uniform(0, 2 * math.pi, size=n_ant)):
                v[a] += math.cos(th) * re - math.sin(th) * im
            sats.append(s)
    if interferer:
        ph = 2 * math.pi * torch.frac((float(rng.uniform(1.0e6, 7.0e6)) / fs) * t.double()).float()
        v += 0.4 * torch.sign(torch.cos(ph))
    w = torch.tensor([128, 64, 32, 16, 8, 4, 2, 1], device="cuda", dtype=torch.uint8)
    bits = ((v >= 0).to(torch.uint8).view(n_ant, n // 8, 8) * w).sum(2, dtype=torch.uint8)
    return bits.cpu().numpy(), sats


_contexts = {}


def _context(precision):
    if precision not in _contexts:
        ctx = tga.Context(0)
        ctx.set_precision(PRECISION[precision])
        _contexts[precision] = ctx
    return _contexts[precision]


def _consts(case):
    return sorted(CONST[k] for k in case["consts"].split())


def _nc_searches(case):
    out = []
    for c in _consts(case):
        ratio = {tga.GALILEO: 4, tga.BEIDOU: 10, tga.L1C: 10}.get(c, 1)  # code periods of 1, 4 and 10 ms
        total = case["periods"] * case["blocks"]
        periods = max(1, case["periods"] // ratio)
        blocks = max(1, total // (periods * ratio))
        d = dict(constellation=c, prns=_prns(c, case["n_prn"]), coherent_periods=periods, blocks=blocks, start=0)
        if ratio == 1 or case["periods"] >= ratio:
            d.update(bin_step_hz=case["step"], n_bins=case["bins"])
        else:  # a block of one longer period: bins of 1 / (2 T) over the same span
            n = int(case["step"] * (case["bins"] - 1) / (500.0 / ratio)) + 1
            d.update(bin_step_hz=500.0 / ratio, n_bins=n)
        out.append(d)
    return out


def prepare(case, seed):
    s = {"case": case, "ctx": _context(case["precision"])}
    kind = case["kind"]
    if kind == "single":
        c, fs = CONST[case["const"]], case["fs"]
        P = _period(c, fs)
        rng = np.random.default_rng(seed)
        code = tga.code_resampled(c, case["prn"], float(P), P).astype(np.float64)
        t = np.arange(2 * P)
        x = 2.0 * math.sqrt(10.0 ** 4.5 / fs) * code[(t + int(rng.integers(0, P))) % P] * np.cos(
            2 * np.pi * np.mod((IF + float(rng.uniform(-4000, 4000))) / fs * t, 1.0) + rng.uniform(0, 2 * np.pi))
        b = np.where(x + rng.standard_normal(2 * P) >= 0, 1.0, -1.0)
        s.update(c=c, P=P, sig=(b - b.mean()).astype(np.float32), pp=(2 * math.pi / fs) * np.arange(2 * P, dtype=np.float64))
    elif kind == "cells":
        n = int(case["fs"] * case["ms"] / 1000.0) // 8 * 8
        s["bits"], _ = _recording(seed, _consts(case), case["n_ant"], n, case["fs"], case["n_prn"])
        s["ants"] = list(range(0, case["n_ant"], case["ant_step"]))
    elif kind == "nc":
        n = int(FS * case["ms"] / 1000.0) // 8 * 8
        s["bits"], _ = _recording(seed, _consts(case), case["n_ant"], n, FS, case["n_prn"],
                                  cn0=(case["cn0_lo"], case["cn0_hi"]))
        s["searches"] = _nc_searches(case)
    elif kind == "fine":
        n = int(FS * case["ms"] / 1000.0) // 8 * 8
        consts = [tga.GPS, tga.GALILEO]
        s["bits"], sats = _recording(seed, consts, case["n_ant"], n, FS, per_const=-(-case["n_sat"] // 2),
                                     cn0=(45.0, 47.0))
        # grid estimates as the search gives them: a whole sample, 300 Hz bins
        s["tasks"] = [(q["c"], q["prn"], float(-q["delay"] % q["P"]), IF + 300.0 * round(q["dop"] / 300.0), 0, n)
                      for q in sats[:case["n_sat"]]]
    else:
        n = int(FS * case["ms"] / 1000.0) // 8 * 8
        s["bits"], _ = _recording(seed, [tga.GPS], case["n_ant"], n, FS, interferer=True)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "single":
        r = ctx.acquire_single(s["c"], s["sig"], s["pp"], case["fs"], IF, BAND, case["prn"], s["P"])
        return {"strength": np.float32(r.signal_strength), "second": np.float32(r.second_peak),
                "frac": r.codephase_frac, "frequency": r.frequency, "lag": r.best_codephase, "bin": r.best_freq_idx,
                "hypothesis": r.hypothesis}
    if kind == "cells":
        mask = sum(1 << c for c in _consts(case))
        prns = _prns(_consts(case)[0], case["n_prn"]) if case["n_prn"] else None
        x = ctx.acquire_cells(s["bits"], case["fs"], mask=mask, ant_filter=s["ants"], prn_filter=prns,
                              cn0=case["cn0"])
        out = {}
        for c in _consts(case):
            r = x[x["constellation"] == c]
            out[tga.NAMES[c]] = {
                "strength": r["signal_strength"].astype(np.float32), "second": r["second_peak"].astype(np.float32),
                "cn0": r["cn0_acr"].astype(np.float32), "frac": r["codephase_frac"], "frequency": r["frequency"],
                "which": np.stack([r["prn"], r["antenna"], r["best_freq_idx"], r["best_codephase"], r["hypothesis"],
                                   r["cn0_valid"]])}
        return out
    if kind == "nc":
        if len(s["searches"]) == 1:
            found = [ctx.search_noncoherent(s["bits"], FS, **s["searches"][0])]
        else:
            found = ctx.search_noncoherent_multi(s["bits"], FS, s["searches"])
        return {tga.NAMES[d["constellation"]]: {
            "power": r["power"].astype(np.float32), "second": r["second_power"].astype(np.float32),
            "frequency": r["frequency"],
            "which": np.stack([r["prn"], r["antenna"], r["best_freq_idx"], r["best_codephase"]])}
            for d, r in zip(s["searches"], found)}
    if kind == "fine":
        res, phases = ctx.fine_acquire(s["bits"], FS, s["tasks"])
        keys = ("code_phase", "frequency", "power", "power_start")
        return {"tasks": np.array([[r[k] for k in keys] for r in res], dtype=np.float32),
                "phases": np.stack([np.cos(phases), np.sin(phases)]).astype(np.float32)}
    res = ctx.rfi_scan(s["bits"], FS)
    lines = np.full((len(res), 3, 2), -1.0)
    for i, r in enumerate(res):
        for k, q in enumerate(r["lines"]):
            lines[i, k] = q["frequency"], q["excess_db"]
    return {"acf": np.array([[r["acf_lag1"], r["acf_lag3"], r["acf_lag16"]] for r in res]), "lines": lines,
            "found": np.array([len(r["lines"]) for r in res])}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _row_flops(P):
    """One product, one inverse transform and |y|^2 over P lags."""
    return 5.0 * P * math.log2(P) + 9.0 * P


def work(case):
    kind = case["kind"]
    if kind == "single":
        P = _period(CONST[case["const"]], case["fs"])
        return {"bytes": 2.0 * P * 12, "flops": 41 * (2 * _row_flops(P) + 10.0 * P * math.log2(P) + 20.0 * P)}
    n = int(case.get("fs", FS) * case["ms"] / 1000.0)
    data = case["n_ant"] * n / 8.0
    if kind == "cells":
        n_ant, b, f = len(range(0, case["n_ant"], case["ant_step"])), data, 0.0
        for c in _consts(case):
            P, k = _period(c, case["fs"]), len(_prns(c, case["n_prn"]))
            f += n_ant * 41 * (2 * k * _row_flops(P) + 10.0 * P * math.log2(P) + 20.0 * P)
            b += n_ant * k * 80.0
        return {"bytes": b, "flops": f}
    if kind == "nc":
        b, f = data, 0.0
        for d in _nc_searches(case):
            P, k = _period(d["constellation"], FS), len(d["prns"])
            rows = case["n_ant"] * d["n_bins"] * d["blocks"]
            f += rows * (k * _row_flops(P) + 5.0 * P * math.log2(P) + 10.0 * P * d["coherent_periods"])
            b += case["n_ant"] * k * 48.0
        return {"bytes": b, "flops": f}
    if kind == "fine":
        # a frequency scan and about six Newton evaluations, 24 flops a sample
        return {"bytes": data + case["n_ant"] * case["n_sat"] * 8.0,
                "flops": case["n_ant"] * case["n_sat"] * n * 24.0 * 10}
    return {"bytes": data + case["n_ant"] * 80.0, "flops": case["n_ant"] * (2.5 * n * math.log2(n) + 4.0 * n)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
# G2 delays of GPS PRN 1-37 (IS-GPS-200), and the 0 that the searched table has for PRN 38
G2_DELAY = (5, 6, 7, 8, 17, 18, 139, 140, 141, 251, 252, 254, 255, 256, 257, 258, 469, 470, 471, 472, 473, 474, 509,
            512, 513, 514, 515, 516, 859, 860, 861, 862, 863, 950, 947, 948, 950, 0)


def _ca_code(prn, P):
    """One period of P samples of a GPS C/A code."""
    g1, g2, a, b = [1] * 10, [1] * 10, [], []
    for _ in range(1023):
        a.append(g1[9])
        b.append(g2[9])
        g1 = [g1[2] ^ g1[9]] + g1[:9]
        g2 = [g2[1] ^ g2[2] ^ g2[5] ^ g2[7] ^ g2[8] ^ g2[9]] + g2[:9]
    a, b = np.array(a), np.array(b)
    chips = 1.0 - 2.0 * (a ^ np.roll(b, G2_DELAY[prn - 1]))
    return chips[np.floor(np.arange(P) / (P / 1023.0)).astype(np.int64) % 1023]


def _peaks(power, cw):
    """Largest value of each row and the largest more than cw lags from it."""
    n = power.shape[-1]
    p, at = power.max(-1)
    d = (torch.arange(n, device=power.device)[None] - at[:, None]).abs()
    d = torch.minimum(d, n - d)
    return p, torch.where(d > cw, power, torch.zeros_like(power)).max(-1).values


def _coherent_exact(sig, pp, codes, P, cw):
    """(signal strength, second peak) per code: wipe-off by the f32 carrier
    phase, the [c, c] and [c, -c] correlations over two periods, the
    strongest of all bins and hypotheses."""
    n = int(round(2 * BAND / 300.0)) + 1
    fc = [(IF - BAND) + i * (2 * BAND) / (n - 1.0) for i in range(n)]
    x = torch.from_numpy(sig.astype(np.float64)).cuda()
    ph = [torch.from_numpy((pp * f).astype(np.float32).astype(np.float64)).cuda() for f in fc]
    X = torch.fft.fft(torch.stack([torch.polar(torch.ones_like(p), p) * x for p in ph]))
    out = []
    for c in codes:
        c = torch.from_numpy(c).cuda()
        best = (-1.0, 0.0)
        for sign in (1.0, -1.0):
            C = torch.fft.fft(torch.cat([c, sign * c])).conj()
            y = torch.fft.ifft(X * C).abs() * math.sqrt(2.0 * P)
            y = y[:, :P]
            p, s = _peaks(y, cw)
            k = int(p.argmax())
            if float(p[k]) > best[0]:
                best = (float(p[k]), float(s[k]))
        out.append(best)
    return np.array(out)


def _demeaned(row, n):
    b = 2.0 * np.unpackbits(row).astype(np.float64) - 1.0
    return (b - b.mean())[:n].astype(np.float32)


def exact(case, seed):
    kind = case["kind"]
    cw = math.ceil(case.get("fs", FS) / 1.023e6)
    if kind == "single":
        if case["const"] != "gps":
            return None
        s = prepare(case, seed)
        p = _coherent_exact(s["sig"], s["pp"], [_ca_code(case["prn"], s["P"])], s["P"], cw)[0]
        return {"strength": np.array(p[0]), "second": np.array(p[1])}
    if kind == "cells":
        if "gps" not in case["consts"].split():
            return None
        s = prepare(case, seed)
        P = _period(tga.GPS, case["fs"])
        codes = [_ca_code(k, P) for k in _prns(tga.GPS, case["n_prn"])]
        pp = (2 * math.pi / case["fs"]) * np.arange(2 * P, dtype=np.float64)
        r = np.stack([_coherent_exact(_demeaned(s["bits"][a], 2 * P), pp, codes, P, cw) for a in s["ants"]], 1)
        return {"gps": {"strength": r[..., 0].reshape(-1), "second": r[..., 1].reshape(-1)}}
    if kind == "nc":
        gps = [d for d in _nc_searches(case) if d["constellation"] == tga.GPS]
        if not gps:
            return None
        d, s = gps[0], prepare(case, seed)
        P = _period(tga.GPS, FS)
        K, B, nb = d["coherent_periods"], d["blocks"], d["n_bins"]
        if case["n_ant"] * nb * B * len(d["prns"]) > 3_000_000:
            return None
        N = K * P
        codes = torch.from_numpy(np.stack([_ca_code(k, P) for k in d["prns"]])).cuda()
        C = torch.fft.fft(codes.to(torch.complex128)).conj()
        got = np.zeros((len(d["prns"]), case["n_ant"], 2))
        for a in range(case["n_ant"]):
            x = torch.from_numpy(_demeaned(s["bits"][a], N * B).astype(np.float64)).cuda().view(B, N)
            best = torch.full((len(d["prns"]), 2), -1.0, dtype=torch.float64, device="cuda")
            for i in range(nb):
                f = IF + (i - (nb - 1) // 2) * d["bin_step_hz"]
                ph = 2 * math.pi * torch.frac((f / FS) * torch.arange(N, dtype=torch.float64, device="cuda"))
                X = torch.fft.fft((torch.polar(torch.ones_like(ph), ph) * x).view(B, K, P).sum(1))
                y = torch.zeros((len(d["prns"]), P), dtype=torch.float64, device="cuda")
                for b in range(B):
                    y += torch.view_as_real(torch.fft.ifft(X[b] * C)).square().sum(-1)
                p, q = _peaks(N * y, cw)
                better = p >= best[:, 0]
                best = torch.where(better[:, None], torch.stack([p, q], 1), best)
            got[:, a] = best.cpu().numpy()
        return {"gps": {"power": got[..., 0].reshape(-1), "second": got[..., 1].reshape(-1)}}
    if kind == "rfi":
        s = prepare(case, seed)
        acf = []
        for row in s["bits"]:
            b = 2.0 * np.unpackbits(row).astype(np.float64) - 1.0
            z = b - b.mean()
            acf.append([float(np.dot(z[:-k], z[k:])) / (len(z) - k) for k in (1, 3, 16)])
        return {"acf": np.array(acf)}
    return None
