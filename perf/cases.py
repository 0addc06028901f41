"""The work a user of this framework has it do, as cases to be timed.

A case is one full multivariate empirical mode decomposition (all IMFs, all
sifts) through the Python binding's Plan: one record or a batch of records, in
the FP64, FP32 or mixed form, with a fixed number of sifts or the stop
criterion, natural or not-a-knot splines, the reference's record ends or
mirrored ones.

listed()            the cases
draw(rng)           one more case of the same ranges
prepare(case, seed) records, directions, output buffer and plan
run(state)          one decomposition
work(case)          bytes and operations it cannot do without
exact(case, seed)   the same decomposition in plain torch, FP64
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "memd-gpu_gb300", "py"))

FORMS = {"f64": 0, "f32": 1, "mixed": 2}
# exact() is left out above this many direction-channel-samples x sifts
EXACT_MOST = 6e10


def case_(name, form, channels, length, directions, num_imfs, max_iter=10, signal="eeg", epochs=0, stop=False,
          spline="natural", boundary="reference", window=True):
    """epochs > 0: a batch of that many records of length / 8 .. length samples."""
    d = {"form": form, "signal": signal, "channels": channels, "length": length, "directions": directions,
         "num_imfs": num_imfs, "max_iter": max_iter, "epochs": epochs, "stop": stop, "spline": spline,
         "boundary": boundary, "window": window}
    return {"name": name, **d} if name else d


def listed():
    return [
        # a short record of a few channels, as the golden tests have it: latency and launches
        case_("f64_4x1000", "f64", 4, 1000, 8, 6, signal="tones"),
        # the smoke test's and the benchmark's tone record, sifted until the stop criterion
        case_("f64_stop_8x2000", "f64", 8, 2000, 64, 5, 200, signal="tones", stop=True),
        case_("mixed_stop_8x2000", "mixed", 8, 2000, 64, 10, 200, signal="tones", stop=True),
        # an odd channel count and record length, MATLAB's spline ends, extrema over the whole record
        case_("f64_nak_19x7501", "f64", 19, 7501, 50, 7, spline="nak", window=False),
        # mirrored ends, mixed form
        case_("mixed_mirror_16x12003", "mixed", 16, 12003, 64, 7, boundary="mirror"),
        # the reference main()'s record (32 channels, 30,504 samples, 64 directions,
        # 9 slots x 10 sifts) in the drop-in precision and in the reference's own
        case_("f64_32x30504", "f64", 32, 30504, 64, 9),
        case_("f32_32x30504", "f32", 32, 30504, 64, 9),
        # the benchmark's headline: the same record, 128 directions, mixed form
        case_("mixed_32x30504", "mixed", 32, 30504, 128, 9),
        # epochs of uneven lengths decomposed in one call
        case_("mixed_batch_64x32", "mixed", 32, 8192, 64, 9, epochs=64),
        case_("f64_batch_12x32", "f64", 32, 8192, 64, 9, epochs=12),
        # many channels
        case_("mixed_128x10000", "mixed", 128, 10000, 256, 9),
        # a long recording
        case_("mixed_64x262144", "mixed", 64, 262144, 128, 6),
    ]


def lengths_of(case):
    """The samples of each record."""
    if not case["epochs"]:
        return [case["length"]]
    rng = random.Random(1000003 * case["epochs"] + case["length"])
    return [rng.randint(max(4, case["length"] // 8), case["length"]) for _ in range(case["epochs"])]


def sifts_of(case):
    """Sifts of a fixed run; for the stop criterion, which decides by the data, a usual number."""
    return (case["num_imfs"] - 1) * (min(case["max_iter"], 12) if case["stop"] else case["max_iter"])


def cost_of(case):
    """Relative cost of a case, for draw()'s limit: direction-channel-samples x sifts, by form."""
    weight = {"f64": 8.0, "f32": 1.2, "mixed": 1.0}[case["form"]]
    if case["form"] == "mixed" and (case["stop"] or case["boundary"] == "mirror"):
        weight = 3.0
    return weight * case["directions"] * case["channels"] * sum(lengths_of(case)) * sifts_of(case)


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    most = 0.6 * max(cost_of(c) for c in listed())
    while True:
        form = rng.choice(["f64", "mixed", "mixed", "f32"])
        epochs = spread(2, 64) if rng.random() < 0.25 else 0
        stop = not epochs and rng.random() < 0.25
        length = spread(1024, 8192) if epochs else spread(500, 5000 if stop else 262144)
        channels, directions = spread(1, 128), spread(4, 256)
        shortest = length // 8 if epochs else length
        slots = max(2, min(10, int(math.log2(shortest)) - 4))
        num_imfs = rng.randint(2, slots)
        spline = "nak" if rng.random() < 0.15 else "natural"
        boundary = "mirror" if not epochs and rng.random() < 0.1 else "reference"
        case = case_(None, form, channels, length, directions, num_imfs, 50 if stop else rng.choice([5, 8, 10, 10]),
                     signal=rng.choice(["eeg", "eeg", "tones"]), epochs=epochs, stop=stop, spline=spline,
                     boundary=boundary, window=rng.random() < 0.7)
        if cost_of(case) <= most:
            return case


# ---- inputs ----------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _record(signal, channels, length, gen):
    """channels x length, FP64, values a float32 can hold (so that every form decomposes the same numbers)."""
    dev = gen.device
    n = torch.arange(length, device=dev, dtype=torch.float64)

    def uniform(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=gen, device=dev, dtype=torch.float64)

    def normal(*shape):
        return torch.randn(*shape, generator=gen, device=dev, dtype=torch.float64)

    if signal == "tones":  # 5, 20 and 60 Hz at 1 kHz, and noise
        y = 0.1 * normal(channels, length)
        for f in (5.0, 20.0, 60.0):
            y += uniform(0.5, 1.5, channels, 1) * torch.sin(2 * math.pi * f * n / 1000.0 + uniform(0, 2 * math.pi, channels, 1))
        return y.float().double()
    # EEG-shaped at 256 Hz: 1/f sources (flat below 1/64 Hz, steeper above 64 Hz) mixed over the channels, a 10 Hz
    # rhythm in bursts, a slow drift, tens of microvolts
    fs = 256.0
    spec = torch.fft.rfft(normal(channels, length))
    f = torch.fft.rfftfreq(length, 1.0 / fs, device=dev, dtype=torch.float64)
    src = torch.fft.irfft(spec / torch.sqrt(f.clamp_min(1.0 / 64.0) * (1 + (f / 64.0) ** 2)), n=length)
    src /= src.square().mean(dim=1, keepdim=True).sqrt()
    y = (normal(channels, channels) / math.sqrt(channels)) @ src
    burst = (torch.sin(2 * math.pi * 0.05 * n / fs + uniform(0, 2 * math.pi, 1)) - 0.4).clamp_min(0.0)
    y += 1.5 * normal(channels, 1) * burst * torch.sin(2 * math.pi * 10.0 * n / fs)
    y += uniform(0.5, 1.5, channels, 1) * torch.sin(2 * math.pi * 0.5 * n / fs + uniform(0, 2 * math.pi, channels, 1))
    return (30.0 * y).float().double()


def _inputs(case, seed):
    """(records, directions) of a case, FP64: directions spread evenly over the sphere."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    ys = [_record(case["signal"], case["channels"], n, gen) for n in lengths_of(case)]
    d = torch.randn(case["directions"], case["channels"], generator=gen, device=dev, dtype=torch.float64)
    d /= d.norm(dim=1, keepdim=True)
    return ys, d.float().double()


def prepare(case, seed):
    import memd_gb300 as mg

    ys, d = _inputs(case, seed)
    dt = torch.float64 if case["form"] == "f64" else torch.float32
    lens = lengths_of(case)
    plan = mg.Plan(case["channels"], case["length"], case["directions"], case["num_imfs"], case["max_iter"],
                   FORMS[case["form"]], max_epochs=case["epochs"],
                   stop_mode=mg.STOP_CRITERION if case["stop"] else mg.STOP_FIXED,
                   spline_end=mg.SPLINE_NOT_A_KNOT if case["spline"] == "nak" else mg.SPLINE_NATURAL,
                   boundary=mg.BOUNDARY_MIRROR if case["boundary"] == "mirror" else mg.BOUNDARY_REFERENCE,
                   ref_window=1 if case["window"] else 0)
    state = {"plan": plan, "d": d.to(dt).contiguous(), "lens": lens, "batched": case["epochs"] > 0}
    if case["epochs"]:
        state["y"] = torch.cat([y.reshape(-1) for y in ys]).to(dt)
        state["off"] = [case["channels"] * sum(lens[:i]) for i in range(len(lens))]
        state["imfs"] = torch.zeros(case["num_imfs"] * case["channels"] * sum(lens), dtype=dt, device=d.device)
    else:
        state["y"] = ys[0].to(dt).contiguous()
        state["imfs"] = torch.zeros(case["num_imfs"], case["channels"], case["length"], dtype=dt, device=d.device)
    return state


def run(state):
    if state["batched"]:
        state["plan"].run_batched(state["y"], state["lens"], state["off"], state["d"], state["imfs"], stats=False)
    else:
        state["plan"].run(state["y"], state["d"], state["imfs"], stats=False)
    return {"imfs": state["imfs"]}


def work(case):
    """The record and the directions read once, the IMFs written once.  Operations of every sift: the projection (2 per
    direction, channel and sample), the splines at their knots (about 30 per knot and channel, setup, solution and mean;
    a knot every 3.6 samples in the first IMF of a record with noise, every 7 in the second, and so on) and the update
    of the signal (4 per channel and sample)."""
    size = 8 if case["form"] == "f64" else 4
    c, k, n = case["channels"], case["directions"], sum(lengths_of(case))
    per_imf = sifts_of(case) / max(1, case["num_imfs"] - 1)
    knots = sum(2.0 * k * n / (3.6 * 2 ** i) for i in range(case["num_imfs"] - 1)) * per_imf
    return {"bytes": size * (c * n * (1 + case["num_imfs"]) + k * c),
            "flops": sifts_of(case) * (2.0 * k * c * n + 4.0 * c * n) + 30.0 * c * knots}


# ---- the same decomposition in plain torch, FP64 -----------------------------
def _pack(flags, extra=0):
    """Positions of each row's set flags, padded to a common length, and their counts."""
    count = flags.sum(dim=1)
    rows, at = flags.nonzero(as_tuple=True)
    start = count.cumsum(0) - count
    x = torch.zeros(flags.shape[0], max(2, int(count.max())) + extra, dtype=torch.int64, device=flags.device)
    x[rows, torch.arange(rows.numel(), device=flags.device) - start[rows]] = at
    return x, count


def _mirror_ends(P, imax, imin):
    """The knots mirrored past the ends of one direction (Rilling et al. 2003, two extrema an end): the symmetry samples
    and the source samples of the left and right knots, for maxima and minima."""
    last = len(P) - 1
    if imax[0] < imin[0]:
        if P[0] > P[imin[0]]:
            lx, ln, ls = imax[1:3][::-1], imin[:2][::-1], imax[0]
        else:
            lx, ln, ls = imax[:2][::-1], imin[:1] + [0], 0
    elif P[0] < P[imax[0]]:
        lx, ln, ls = imax[:2][::-1], imin[1:3][::-1], imin[0]
    else:
        lx, ln, ls = imax[:1] + [0], imin[:2][::-1], 0
    if 2 * ls - lx[0] > 0 or 2 * ls - ln[0] > 0:
        if ls == imax[0]:
            lx = imax[:2][::-1]
        else:
            ln = imin[:2][::-1]
        ls = 0
    if imax[-1] < imin[-1]:
        if P[last] < P[imax[-1]]:
            rx, rn, rs = imax[-2:][::-1], imin[-3:-1][::-1], imin[-1]
        else:
            rx, rn, rs = [last, imax[-1]], imin[-2:][::-1], last
    elif P[last] > P[imin[-1]]:
        rx, rn, rs = imax[-3:-1][::-1], imin[-2:][::-1], imax[-1]
    else:
        rx, rn, rs = imax[-2:][::-1], [last, imin[-1]], last
    if 2 * rs - rx[-1] < last or 2 * rs - rn[-1] < last:
        if rs == imax[-1]:
            rx = imax[-2:][::-1]
        else:
            rn = imin[-2:][::-1]
        rs = last
    return (ls, rs), (lx, ln), (rx, rn)


def _knots(X, d, case):
    """Knot positions (2K x E, maxima then minima), the samples their values come from, their counts, the interior
    extrema, and the envelopes whose ends are clamped."""
    L, K = X.shape[0], d.shape[0]
    P = d @ X.T
    n = torch.arange(L, device=X.device)
    cov = 240 * ((L + 241) // 242) if case["window"] else L
    inner = (n >= 1) & (n <= min(cov, L - 2))
    up, dn = torch.zeros_like(P, dtype=torch.bool), torch.zeros_like(P, dtype=torch.bool)
    a, b, c = P[:, :-2], P[:, 1:-1], P[:, 2:]
    up[:, 1:-1] = (b > a) & (b > c) & inner[1:-1]
    dn[:, 1:-1] = (b < a) & (b < c) & inner[1:-1]
    flags = torch.cat([up, dn])
    interior = flags.sum(dim=1)
    if case["boundary"] != "mirror":
        flags[:, 0] = flags[:, L - 1] = True
        x, count = _pack(flags)
        return x, x, count, interior
    x0, count0 = _pack(flags, 4)
    rows, ends = x0.tolist(), P.tolist()
    src, pos, count = [], [], []
    for r in range(2 * K):
        k, e = r % K, r // K
        im = [rows[k][:int(count0[k])], rows[k + K][:int(count0[k + K])]]
        mine = im[e]
        left, right, sym = [], [], (0, 0)
        if len(im[0]) >= 2 and len(im[1]) >= 2:
            sym, lefts, rights = _mirror_ends(ends[k], im[0], im[1])
            left, right = lefts[e], rights[e]
        src.append(left + mine + right)
        pos.append([2 * sym[0] - s for s in left] + mine + [2 * sym[1] - s for s in right])
        count.append(len(src[-1]))
    width = max(2, max(count))
    pad = [torch.tensor([v + [0] * (width - len(v)) for v in m], device=X.device) for m in (pos, src)]
    return pad[0], pad[1], torch.tensor(count, device=X.device), interior


def _second(x, count, y, nak):
    """Half the second derivative at the knots of each row's spline (R x E x C), by parallel cyclic reduction."""
    R, E = x.shape
    i = torch.arange(E, device=x.device).expand(R, E)
    valid = i < count[:, None]
    h = torch.ones(R, E, dtype=torch.float64, device=x.device)
    h[:, :-1] = torch.where(i[:, 1:] < count[:, None], (x[:, 1:] - x[:, :-1]).double(), h[:, :-1])
    slope = torch.zeros_like(y)
    slope[:, :-1] = (y[:, 1:] - y[:, :-1]) / h[:, :-1, None]
    hl = torch.cat([h[:, :1], h[:, :-1]], dim=1)
    row = valid & (i > 0) & (i < count[:, None] - 1)
    a, b, c = torch.where(row, hl, 0.0), torch.where(row, 2 * (hl + h), 1.0), torch.where(row, h, 0.0)
    r = torch.zeros_like(y)
    r[:, 1:] = 3 * (slope[:, 1:] - slope[:, :-1])
    r *= row[:, :, None]
    if nak:  # the end rows eliminated by equal third derivatives across the second and second-to-last knots
        four = count[:, None] >= 4
        first, last = four & (i == 1), four & (i == count[:, None] - 2)
        a, b, c = torch.where(first, 0.0, a), torch.where(first, hl + 2 * h, b), torch.where(first, h - hl, c)
        r = torch.where(first[:, :, None], r * (h / (hl + h))[:, :, None], r)
        a, b, c = torch.where(last, hl - h, a), torch.where(last, 2 * hl + h, b), torch.where(last, 0.0, c)
        r = torch.where(last[:, :, None], r * (hl / (hl + h))[:, :, None], r)
    step = 1
    while step < min(E, 128):  # couplings fall by a factor of two or more a knot: nothing is left of them past 64

        def back(v, fill):
            out = torch.full_like(v, fill)
            out[:, step:] = v[:, :-step]
            return out

        def ahead(v, fill):
            out = torch.full_like(v, fill)
            out[:, :-step] = v[:, step:]
            return out

        al, be = -a / back(b, 1.0), -c / ahead(b, 1.0)
        r = r + al[:, :, None] * back(r, 0.0) + be[:, :, None] * ahead(r, 0.0)
        b, a, c = b + al * back(c, 0.0) + be * ahead(a, 0.0), al * back(a, 0.0), be * ahead(c, 0.0)
        step *= 2
    s = r / b[:, :, None]
    if nak:
        q = torch.arange(R, device=x.device)[count >= 4]
        e = count[q]
        s[q, 0] = s[q, 1] + (h[q, 0] / h[q, 1])[:, None] * (s[q, 1] - s[q, 2])
        s[q, e - 1] = s[q, e - 2] + (h[q, e - 2] / h[q, e - 3])[:, None] * (s[q, e - 2] - s[q, e - 3])
    return s


def _envelopes(X, x, src, count, env, clamp, nak):
    """The envelopes (R x L x C) through the knots of each row; env: 0 for rows of maxima, 1 for minima."""
    R, E = x.shape
    L = X.shape[0]
    y = X[src]
    rows = torch.arange(R, device=X.device)
    if clamp:  # an end value is raised (lowered) to the line through its two neighbours
        sign = torch.where(env == 0, 1.0, -1.0).double()[:, None]
        for end in (0, 1):
            q = rows[count > 5]
            e = count[q] - 1
            j = [torch.zeros_like(e), torch.ones_like(e), torch.full_like(e, 2)] if end == 0 else [e, e - 1, e - 2]
            v = [y[q, t] for t in j]
            p = [x[q, t].double()[:, None] for t in j]
            line = v[1] + (v[2] - v[1]) / (p[2] - p[1]) * (p[0] - p[1])
            y[q, j[0]] = torch.where((line - v[0]) * sign[q] > 0, line, v[0])
    s = _second(x, count, y, nak)
    n = torch.arange(L, device=X.device)
    padded = torch.where(torch.arange(E, device=X.device)[None] < count[:, None], x, 1 << 40)
    iv = torch.searchsorted(padded, n.expand(R, L).contiguous()) - 1
    iv = torch.minimum(iv.clamp_min(0), (count - 2).clamp_min(0)[:, None])
    g = rows[:, None]
    h = (x[g, iv + 1] - x[g, iv]).double()[:, :, None]
    t = (n[None] - x[g, iv]).double()[:, :, None]
    y0, s0, s1 = y[g, iv], s[g, iv], s[g, iv + 1]
    b = (y[g, iv + 1] - y0) / h - h / 3 * (2 * s0 + s1)
    return y0 + t * (b + t * (s0 + t * ((s1 - s0) / (3 * h))))


def _mean(X, d, case, want_spread):
    """(mean envelope L x C, qualified directions, mean of the directions' half spreads, whether all have few extrema)."""
    K, (L, C) = d.shape[0], X.shape
    x, src, count, interior = _knots(X, d, case)
    few = bool(((interior[:K] + interior[K:]) < 3).all())
    good = torch.arange(K, device=X.device)[(interior[:K] >= 2) & (interior[K:] >= 2)]
    total, spread = torch.zeros_like(X), torch.zeros(L, dtype=torch.float64, device=X.device)
    block = max(1, int(1.5e8 // (2 * L * C)))
    for at in range(0, len(good), block):
        k = good[at:at + block]
        rows = torch.cat([k, k + K])
        width = int(count[rows].max())
        env = (rows >= K).long()
        v = _envelopes(X, x[rows, :width], src[rows, :width], count[rows], env, case["boundary"] != "mirror",
                       case["spline"] == "nak")
        total += v.sum(dim=0)
        if want_spread:
            spread += (v[:len(k)] - v[len(k):]).square().sum(dim=2).sqrt().sum(dim=0) / 2
    q = len(good)
    nan = float("nan")
    return total / (2 * q) if q else total * nan, q, spread / q if q else spread, few


def _decompose(y, d, case):
    """num_imfs x C x L of one record (C x L)."""
    run_, out = y.T.contiguous(), []
    slots = case["num_imfs"] - 1
    while len(out) < slots:
        X, few = run_.clone(), False
        for i in range(case["max_iter"]):
            m, q, spread, few_now = _mean(X, d, case, case["stop"])
            if case["stop"]:
                few = i == 0 and few_now
                if few or q == 0:
                    break
                sigma = m.square().sum(dim=1).sqrt() / spread
                if float((sigma > 0.075).double().mean()) <= 0.075 and not bool((sigma > 0.75).any()):
                    break
            X = X - m
        if few:
            break
        out.append(X.T.clone())
        run_ = run_ - X
    out += [torch.zeros_like(y)] * (slots - len(out))
    return torch.stack(out + [run_.T])


def exact(case, seed):
    if case["directions"] * case["channels"] * sum(lengths_of(case)) * sifts_of(case) > EXACT_MOST:
        return None
    ys, d = _inputs(case, seed)
    got = [_decompose(y, d, case) for y in ys]
    return {"imfs": got[0] if not case["epochs"] else torch.cat([v.reshape(-1) for v in got])}
