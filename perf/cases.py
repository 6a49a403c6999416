"""The work that programs built on this framework have it do, as measurable cases.

Each case is one call (or the few calls that belong together) a program makes
per snapshot, box or optimiser step, through the public entry points of
genpk_gb300.api, with the inputs already where such a program has them.

kinds
  spectrum       clear a grid, deposit the particles, P(k) of the grid
                 (Context.zero, deposit, power): what gen-pk does per particle
                 type.  `chunks` > 0: host arrays handed over in that many
                 pieces, as a snapshot reader does.
  step           the per-species loop: dark matter, gas and stars deposited and
                 every auto and cross spectrum (Context.power_step).
  boxes          the auto spectra of many boxes in one call (Batch.power).
  grad           a P(k) likelihood and its gradient with respect to the
                 particles (deposit, power, adjoint): one optimiser step of a
                 field reconstruction.
  fieldize       the reference's own deposit call on host arrays (api.fieldize).
  powerspectrum  the reference's own binning call on a host half-complex
                 spectrum (api.powerspectrum).

orders (the order the particles lie in)
  lattice        initial-condition lattice order, x slowest (Zel'dovich sets)
  curve          along a Morton curve, as codes write their snapshots
  random         no spatial order (catalogues, resampled or shuffled sets)
  clustered      no spatial order, lognormal density, a mass per particle

Results whose rounding depends on a timed choice are pinned by programs that
want to reproduce them: the boxes run in the grouped mode, and the drawn cases
of particles in no order leave out the counts where the two deposit engines
(and with them the transform) are about as fast as each other.
"""
import math

import numpy as np
import torch

from genpk_gb300 import api, synth

BOX = 25000.0
NRBINS = 64


def listed():
    return [
        # a small box or one patch of a larger one: bound by launches and latency
        {"name": "random_64", "kind": "spectrum", "n": 64, "order": "random", "count": 40_000},
        # the smallest configuration: 128^3 unordered particles, one per cell
        {"name": "random_128", "kind": "spectrum", "n": 128, "order": "random", "count": 128 ** 3},
        # a galaxy or halo sample with a mass per object on a grid that is not a power of two
        {"name": "clustered_200", "kind": "spectrum", "n": 200, "order": "clustered",
         "count": 3_300_001},
        # an evolved snapshot in the order its code wrote it, on the grid of gen-pk's rule
        {"name": "curve_512", "kind": "spectrum", "n": 512, "order": "curve", "side": 384},
        # the headline workload: 512^3 particles in lattice order on 512^3
        {"name": "lattice_512", "kind": "spectrum", "n": 512, "order": "lattice", "side": 512},
        # the largest configuration: 1024^3 on 1024^3
        {"name": "lattice_1024", "kind": "spectrum", "n": 1024, "order": "lattice", "side": 1024},
        # dark matter, gas and massive stars of one snapshot: three autos, three crosses
        {"name": "species_512", "kind": "step", "n": 512, "side": 256, "stars": 12_000_000},
        # a suite of boxes of uneven sizes
        {"name": "boxes_16", "kind": "boxes", "boxes": 16, "small": 128, "large": 256,
         "least": 100_000, "most": 30_000_000},
        # one step of a field reconstruction at the headline size
        {"name": "grad_512", "kind": "grad", "n": 512, "order": "lattice", "side": 512},
        # the same for unordered particles whose masses are parameters too
        {"name": "grad_clustered_160", "kind": "grad", "n": 160, "order": "clustered",
         "count": 2_000_003},
        # a program linked against the reference's functions: its host grid...
        {"name": "fieldize_128", "kind": "fieldize", "n": 128, "count": 1_000_000},
        # ... and the spectrum its own FFT made of it
        {"name": "powerspectrum_128", "kind": "powerspectrum", "n": 128},
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pow2_at_least(v):
    return 1 << max(0, math.ceil(math.log2(v)))


def _draw_random(rng):
    """Particles in no order: a count and a grid (see the module's note)."""
    n = rng.choice([32, 48, 64, 75, 96, 128, 130, 200, 256, 320, 384, 512])
    # 64..512, powers of two: below the lower or above the upper count one
    # engine is clearly the faster; other grids have one transform for both
    low, high = (900_000, 4_200_000) if n == 512 else (380_000, 2_097_152)
    most = 30_000_000
    while True:
        count = _between(rng, 3_000, most)
        if n not in (64, 128, 256, 512) or not low < count < high:
            return {"n": n, "order": "random", "count": count}


def _draw_lattice(rng, most):
    side = _between(rng, 110, most)
    n = rng.choice([_pow2_at_least(side), _pow2_at_least(side), side])
    return {"n": n, "order": rng.choice(["lattice", "lattice", "curve"]), "side": side}


def _draw_clustered(rng):
    return {"n": rng.choice([40, 90, 100, 150, 160, 200, 250, 300, 384]), "order": "clustered",
            "count": _between(rng, 3_000, 20_000_000)}


def draw(rng):
    kind = rng.choice(["spectrum"] * 10 + ["grad"] * 4 +
                      ["step", "boxes", "fieldize", "powerspectrum"])
    if kind == "spectrum":
        pick = rng.choice(["random", "lattice", "lattice", "clustered", "host"])
        if pick == "host":
            return {"kind": kind, "n": rng.choice([96, 150, 200, 250]), "order": "random",
                    "count": _between(rng, 20_000, 4_000_000), "chunks": rng.choice([1, 2, 3])}
        case = {"random": lambda: _draw_random(rng), "lattice": lambda: _draw_lattice(rng, 640),
                "clustered": lambda: _draw_clustered(rng)}[pick]()
        return {"kind": kind, **case}
    if kind == "grad":
        case = rng.choice([lambda: _draw_lattice(rng, 480), lambda: _draw_clustered(rng)])()
        return {"kind": kind, **case}
    if kind == "step":
        return {"kind": kind, "n": rng.choice([200, 256, 384, 512]), "side": _between(rng, 110, 288),
                "stars": _between(rng, 1_200_000, 12_000_000)}
    if kind == "boxes":
        small, large = rng.choice([(64, 128), (128, 256), (96, 200)])
        return {"kind": kind, "boxes": rng.randint(2, 16), "small": small, "large": large,
                "least": _between(rng, 20_000, 100_000),
                "most": _between(rng, 1_000_000, 30_000_000)}
    if kind == "fieldize":
        return {"kind": kind, "n": _between(rng, 30, 160), "count": _between(rng, 1_000, 4_000_000)}
    return {"kind": kind, "n": _between(rng, 30, 160)}


# ---- inputs -----------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _morton_sites(side):
    """Lattice sites (x slowest) in the order of a Morton curve."""
    i = torch.arange(side, device="cuda")
    spread = torch.zeros_like(i)
    for b in range(10):
        spread |= ((i >> b) & 1) << (3 * b)
    code = (spread[:, None, None] << 2) | (spread[None, :, None] << 1) | spread[None, None, :]
    return torch.argsort(code.reshape(-1))


def _lognormal(count, seed, box, mesh=64, ordered=False):
    """count particles of a lognormal density (sigma 1.5) on a mesh, placed at
    random in their mesh cells, with lognormal masses; ordered: cell by cell."""
    g = _gen(seed)
    white = torch.randn((mesh,) * 3, generator=g, device="cuda", dtype=torch.float64)
    k = torch.fft.fftfreq(mesh, device="cuda", dtype=torch.float64) * mesh
    kz = torch.arange(mesh // 2 + 1, device="cuda", dtype=torch.float64)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    smooth = torch.exp(-0.5 * k2 / (0.25 * mesh) ** 2)
    f = torch.fft.irfftn(torch.fft.rfftn(white) * smooth, s=(mesh,) * 3)
    rho = torch.exp(1.5 * f / f.std())
    edges = torch.cumsum(rho.reshape(-1), 0)
    u = torch.rand(count, generator=g, device="cuda", dtype=torch.float64) * edges[-1]
    cell = torch.searchsorted(edges, u).clamp_(max=mesh ** 3 - 1)
    if ordered:
        cell = torch.sort(cell).values
    site = torch.stack([cell // (mesh * mesh), (cell // mesh) % mesh, cell % mesh], dim=1).float()
    pos = (site + torch.rand((count, 3), generator=g, device="cuda")) * (box / mesh)
    pos = torch.where(pos >= box, torch.zeros_like(pos), pos)
    mass = torch.exp(-5.0 + 0.8 * torch.randn(count, generator=g, device="cuda"))
    return pos.contiguous(), mass


def _particles(case, seed):
    """(positions, masses or None) on the GPU."""
    order = case["order"]
    if order in ("lattice", "curve"):
        pos = synth.zeldovich(case["side"], BOX, seed=seed, device="cuda")
        return (pos[_morton_sites(case["side"])].contiguous() if order == "curve" else pos), None
    if order == "clustered":
        return _lognormal(case["count"], seed, BOX)
    return synth.uniform(case["count"], BOX, seed=seed, device="cuda"), None


def _norm(pos, masses):
    """The normalising mass as gen-pk forms it: the sum of the masses plus one."""
    return (float(masses.double().sum()) if masses is not None else float(pos.shape[0])) + 1.0


def _species(case, seed):
    stars, mass = _lognormal(case["stars"], seed + 2000, BOX, mesh=128, ordered=True)
    pos = [synth.zeldovich(case["side"], BOX, seed=seed, device="cuda"),
           synth.zeldovich(case["side"], BOX, seed=seed + 1000, device="cuda"), stars]
    pairs = [(0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2)]
    norm = [_norm(pos[0], None), _norm(pos[1], None), _norm(stars, mass)]
    return pos, [None, None, mass], pairs, [(norm[a], norm[b]) for a, b in pairs]


def _box_counts(case):
    """Counts spread over their logarithm, in a fixed shuffled order."""
    k = case["boxes"]
    at = [((i * 7) % k + 0.5) / k if math.gcd(7, k) == 1 else (i + 0.5) / k for i in range(k)]
    return [int(case["least"] * (case["most"] / case["least"]) ** t) | 1 for t in at]


def _box_dims(case, counts):
    return [case["large"] if c >= 4_000_000 else case["small"] for c in counts]


def _target(case):
    """The spectrum the likelihood compares with: shot noise and a power law."""
    shot = 1.0 / (case["side"] ** 3 if "side" in case else case["count"])
    return shot * (1.0 + 100.0 / (1.0 + np.arange(NRBINS)))


def _host_field(case, seed):
    pos = synth.uniform(case["count"], BOX, seed=seed, device="cuda").cpu().numpy()
    ln = torch.randn(case["count"], generator=_gen(seed + 1), device="cuda")
    return pos, torch.exp(0.5 * ln).cpu().numpy()


def _host_spectrum(case, seed):
    n = case["n"]
    g = _gen(seed)
    k = torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * n
    kz = torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    f = torch.randn((n, n, n // 2 + 1, 2), generator=g, device="cuda", dtype=torch.float64)
    return (torch.view_as_complex(f) * (1.0 + k2) ** -0.5).cpu().numpy()


def prepare(case, seed):
    seed = int(seed)
    kind = case["kind"]
    if kind in ("spectrum", "grad"):
        pos, masses = _particles(case, seed)
        norm = _norm(pos, masses)
        state = {"case": case, "pos": pos, "masses": masses, "norm": norm,
                 "ctx": api.Context(case["n"], NRBINS)}
        if kind == "grad":
            state["target"] = _target(case)
        if case.get("chunks"):
            host = pos.cpu().numpy()
            state["pos"] = [np.ascontiguousarray(c) for c in np.array_split(host, case["chunks"])]
        return state
    if kind == "step":
        pos, masses, pairs, norms = _species(case, seed)
        return {"case": case, "pos": pos, "masses": masses, "pairs": pairs, "norms": norms,
                "ctx": api.Context(case["n"], NRBINS, nfields=3)}
    if kind == "boxes":
        counts = _box_counts(case)
        batch = api.Batch(_box_dims(case, counts), NRBINS)
        batch.set_mode("grouped")
        return {"case": case, "batch": batch, "norm": [c + 1.0 for c in counts],
                "pos": [synth.uniform(c, BOX, seed=seed + 100 * i, device="cuda")
                        for i, c in enumerate(counts)]}
    if kind == "fieldize":
        n = case["n"]
        pos, mass = _host_field(case, seed)
        return {"case": case, "pos": pos, "mass": mass, "grid": np.zeros((n, n, 2 * (n // 2 + 1)))}
    if kind == "powerspectrum":
        return {"case": case, "spectrum": _host_spectrum(case, seed)}
    raise ValueError(kind)


# ---- the calls --------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "spectrum":
        ctx = state["ctx"]
        ctx.zero(0)
        for pos in state["pos"] if case.get("chunks") else [state["pos"]]:
            ctx.deposit(0, BOX, pos, state["masses"], 1.0)
        return ctx.power(0, 0, state["norm"], state["norm"])
    if kind == "step":
        return state["ctx"].power_step(BOX, state["pos"], state["pairs"], state["norms"],
                                       masses_list=state["masses"], mass=1.0)
    if kind == "boxes":
        return state["batch"].power(BOX, state["pos"], state["norm"], mass=1.0)
    if kind == "grad":
        # chi^2 = sum_b count_b (P_b - T_b)^2 / (2 T_b^2), the variance of a Gaussian field
        ctx, pos, masses = state["ctx"], state["pos"], state["masses"]
        norm, target = state["norm"], state["target"]
        ctx.zero(0)
        ctx.deposit(0, BOX, pos, masses, 1.0)
        power, count, _ = ctx.power(0, 0, norm, norm)
        slope = count * (power - target) / target ** 2
        gpos, gmass, gnorm = ctx.adjoint(0, BOX, pos, slope, norm, masses=masses, mass=1.0)
        return (power, gpos, gnorm) if gmass is None else (power, gpos, gnorm, gmass)
    if kind == "fieldize":
        state["grid"][...] = 0.0  # gen-pk clears its field before each type
        api.fieldize(BOX, case["n"], state["grid"], state["pos"], state["mass"])
        return state["grid"]
    norm = float(case["n"]) ** 3
    return api.powerspectrum(case["n"], state["spectrum"], None, NRBINS, norm, norm)


# ---- bytes and operations ---------------------------------------------------


def _fft_flops(n):
    return 2.5 * n ** 3 * math.log2(n ** 3) + 5.0 * n ** 3


def work(case):
    kind = case["kind"]
    if kind in ("spectrum", "grad"):
        count = case["side"] ** 3 if "side" in case else case["count"]
        masses = case["order"] == "clustered"
        each = 16 if masses else 12  # read, and for the gradient written, per particle
        bytes_, flops = count * each + 20 * NRBINS, 40.0 * count + _fft_flops(case["n"])
        if kind == "grad":
            bytes_, flops = bytes_ + count * each, 2.0 * flops
    elif kind == "step":
        lattice = 2 * case["side"] ** 3
        bytes_ = 12 * lattice + 16 * case["stars"] + 60 * NRBINS
        flops = 40.0 * (lattice + case["stars"]) + 3 * _fft_flops(case["n"])
    elif kind == "boxes":
        counts = _box_counts(case)
        bytes_ = 12 * sum(counts) + 20 * NRBINS * case["boxes"]
        flops = 40.0 * sum(counts) + sum(_fft_flops(n) for n in _box_dims(case, counts))
    elif kind == "fieldize":
        n = case["n"]
        bytes_, flops = 16 * case["count"] + 8 * n * n * 2 * (n // 2 + 1), 40.0 * case["count"]
    else:
        n = case["n"]
        bytes_, flops = 16 * n * n * (n // 2 + 1) + 20 * NRBINS, 10.0 * n * n * (n // 2 + 1)
    return {"bytes": float(bytes_), "flops": float(flops)}


# ---- the same in 64 bits ----------------------------------------------------


def _cells(pos, n, box):
    x = pos.double() * (n / box)
    f = torch.floor(x)
    return torch.remainder(f.long(), n), x - f


def _corners(cell, d, n, row):
    """Index and weight of a chunk's eight corners, and the corner's offsets."""
    up = (cell + 1) % n
    for k in range(8):
        side = [(k >> a) & 1 for a in range(3)]
        at = [up[:, a] if s else cell[:, a] for a, s in enumerate(side)]
        w = [d[:, a] if s else 1.0 - d[:, a] for a, s in enumerate(side)]
        yield (at[0] * n + at[1]) * row + at[2], w, side


def _density(pos, masses, n, row=None):
    row = n if row is None else row
    grid = torch.zeros(n * n * row, device="cuda", dtype=torch.float64)
    for first in range(0, pos.shape[0], 1 << 23):
        p = pos[first:first + (1 << 23)]
        m = None if masses is None else masses[first:first + (1 << 23)]
        cell, d = _cells(p, n, BOX)
        for at, w, _ in _corners(cell, d, n, row):
            v = w[0] * w[1] * w[2]
            grid.index_add_(0, at, v if m is None else v * m.double())
    return grid.view(n, n, row)


def _modes(n):
    """Wave numbers, the bins of integer |k|^2, and the window and weight factors."""
    half = n // 2
    i = torch.arange(n, device="cuda")
    k = torch.where(i <= half, i, i - n)
    kk2 = torch.arange(1, 3 * half * half + 1, dtype=torch.float64)
    per = (NRBINS - 1) / math.log(math.sqrt(3) * n / 2.0)
    bins = torch.floor(per * 0.5 * torch.log(kk2)).long()
    bins = torch.cat([torch.zeros(1, dtype=torch.long), bins]).cuda()
    kd = k.double()
    window = torch.where(k != 0, math.pi * kd / (n * torch.sin(math.pi * kd / n)),
                         torch.ones_like(kd))
    window = window.float().double()  # single precision per axis is the reference's definition
    weight = torch.full((half + 1,), 2.0, device="cuda", dtype=torch.float64)
    weight[0] = weight[half] = 1.0
    return k, bins, window, weight


def _slabs(n):
    step = max(1, (1 << 25) // (n * (n // 2 + 1)))
    return [(a, min(n, a + step)) for a in range(0, n, step)]


def _slab_modes(tables, n, a, b):
    k, bins, window, weight = tables
    kz = torch.arange(n // 2 + 1, device="cuda")
    kk2 = k[a:b, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    v = (window[a:b, None, None] * window[None, :, None] * window[None, None, :n // 2 + 1]) ** 4
    c = weight[None, None, :].expand(kk2.shape).clone()
    if a == 0:
        c[0, 0, 0] = 0.0
    return bins[kk2], v, c, kk2


def _power(fa, fb, n, norm_a, norm_b):
    tables = _modes(n)
    power, count, keff = (torch.zeros(NRBINS, device="cuda", dtype=torch.float64) for _ in range(3))
    for a, b in _slabs(n):
        bins, v, c, kk2 = _slab_modes(tables, n, a, b)
        x, y = fa[a:b], fb[a:b]
        value = c * v * (x.real * y.real + x.imag * y.imag)
        for total, w in ((power, value), (count, c), (keff, c * torch.sqrt(kk2.double()))):
            total += torch.bincount(bins.reshape(-1), weights=w.reshape(-1), minlength=NRBINS)
    full = count.clamp(min=1.0)
    return ((power / (norm_a * norm_b * full)).cpu().numpy(),
            count.cpu().numpy().astype(np.int32), (keff / full).cpu().numpy())


def _gradient(pos, masses, n, spectrum, slope, count, norm, power):
    tables = _modes(n)
    coef = np.where(count > 0, 2.0 * slope / (norm * norm * np.maximum(count, 1)), 0.0)
    coef = torch.from_numpy(coef).cuda()
    mult = torch.full((n // 2 + 1,), 2.0, device="cuda", dtype=torch.float64)
    mult[0] = 1.0
    if n % 2 == 0:
        mult[n // 2] = 1.0
    for a, b in _slabs(n):
        bins, v, c, _ = _slab_modes(tables, n, a, b)
        spectrum[a:b] *= coef[bins] * v * c / mult
    field = torch.fft.irfftn(spectrum, s=(n, n, n), norm="forward").reshape(-1)
    gnorm = float(np.sum(slope * (-2.0 * power / norm)))
    gpos = torch.zeros(pos.shape, device="cuda", dtype=torch.float64)
    gmass = torch.zeros(pos.shape[0], device="cuda", dtype=torch.float64)
    for first in range(0, pos.shape[0], 1 << 23):
        p = pos[first:first + (1 << 23)]
        m = 1.0 if masses is None else masses[first:first + (1 << 23)].double()
        cell, d = _cells(p, n, BOX)
        for at, w, side in _corners(cell, d, n, n):
            g = field[at]
            gmass[first:first + p.shape[0]] += g * w[0] * w[1] * w[2]
            for ax in range(3):
                rest = w[(ax + 1) % 3] * w[(ax + 2) % 3]
                gpos[first:first + p.shape[0], ax] += (1.0 if side[ax] else -1.0) * g * rest * m * (n / BOX)
    return gpos, gnorm, gmass + gnorm


def exact(case, seed):
    seed = int(seed)
    kind, n = case["kind"], case.get("n")
    if kind in ("spectrum", "grad"):
        pos, masses = _particles(case, seed)
        norm = _norm(pos, masses)
        f = torch.fft.rfftn(_density(pos, masses, n))
        power, count, keff = _power(f, f, n, norm, norm)
        if kind == "spectrum":
            return power, count, keff
        target = _target(case)
        slope = count * (power - target) / target ** 2
        gpos, gnorm, gmass = _gradient(pos, masses, n, f, slope, count, norm, power)
        return (power, gpos, gnorm) if masses is None else (power, gpos, gnorm, gmass)
    if kind == "step":
        pos, masses, pairs, norms = _species(case, seed)
        f = [torch.fft.rfftn(_density(p, m, n)) for p, m in zip(pos, masses)]
        got = [_power(f[a], f[b], n, *norm) for (a, b), norm in zip(pairs, norms)]
        return np.stack([g[0] for g in got]), got[0][1], got[0][2]
    if kind == "boxes":
        counts, got = _box_counts(case), []
        for i, (c, n) in enumerate(zip(counts, _box_dims(case, counts))):
            pos = synth.uniform(c, BOX, seed=seed + 100 * i, device="cuda")
            f = torch.fft.rfftn(_density(pos, None, n))
            got.append(_power(f, f, n, c + 1.0, c + 1.0))
        return tuple(np.stack([g[j] for g in got]) for j in range(3))
    if kind == "fieldize":
        pos, mass = _host_field(case, seed)
        pos, mass = torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda()
        return _density(pos, mass, n, 2 * (n // 2 + 1)).cpu().numpy()
    f = torch.from_numpy(_host_spectrum(case, seed)).cuda()
    return _power(f, f, n, float(n) ** 3, float(n) ** 3)
