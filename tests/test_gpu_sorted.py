"""The sorted engine's two sorts (chunks binned in shared memory, up to 8192
tiles; a counting sort over the pass beyond) at the edges of their ranges.

Every engine adds the same integers and rounds each cell once, so the grids
are compared with the stream engine's bit for bit; the oracle bounds both:
2e-6 of the largest cell (FP32 rounding of a cell and of its mean) and 1e-5
per bin of P(k), whose last bin is the corner mode the sort sums itself.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gp(native_lib):
    import torch
    assert torch.cuda.is_available(), "GPU tests need a CUDA device"
    import genpk_gb300
    return genpk_gb300


def particles(n, box, seed, kind):
    rng = np.random.default_rng(seed)
    pos = (rng.random((n, 3)) * box).astype(np.float32)
    if kind == "clustered":  # most of them in one tile, in runs of one tile
        pos[: n // 2] = (pos[: n // 2] * 0.05).astype(np.float32)
    if kind == "outside":    # periodic images, cell edges, the origin's neighbourhood
        pos[::3] += np.float32(box)
        pos[1::5] -= np.float32(2 * box)
        pos[2::7] = 0.0
        pos[3::11] = np.float32(-1e-6 * box)
    return pos


@pytest.mark.parametrize("dims,tile,n,kind,mass", [
    (8, (8, 8, 8), 1, "uniform", "one"),              # one tile, one particle
    (17, (16, 16, 16), 1023, "outside", "each"),      # partial tiles, odd grid, below one chunk row
    (64, (8, 8, 8), 1025, "uniform", "one"),
    (64, (16, 16, 8), 152 * 1024 + 1, "uniform", "each"),  # one chunk more than the CTAs
    (100, (16, 16, 16), 300_001, "clustered", "signed"),
    (128, (8, 8, 8), 200_000, "outside", "negative"),  # 4096 tiles of 8^3
    (160, (8, 8, 8), 400_000, "uniform", "each"),      # 8000 tiles: the largest binned
    (168, (8, 8, 8), 400_000, "clustered", "one"),     # 9261 tiles: the counting sort
    (130, (16, 16, 16), 152 * 12288 + 5, "uniform", "one"),  # a second round of full chunks
    (330, (16, 16, 16), 500_000, "outside", "each"),   # 9261 tiles of 16^3
    (280, (8, 8, 8), 100_000, "uniform", "signed"),    # 42875 tiles: counted in global memory
])
def test_sorts_at_their_edges(gp, dims, tile, n, kind, mass):
    box = 1000.0
    pos = particles(n, box, dims + n, kind)
    rng = np.random.default_rng(n)
    masses, uniform = None, {"one": 1.5, "negative": -0.75}.get(mass, 0.0)
    if mass in ("each", "signed"):
        masses = rng.lognormal(0.0, 1.0, n).astype(np.float32)
        if mass == "signed":
            masses[::4] *= -1
            masses[1::9] = 0.0
    norm = 1.0 + float(np.abs(masses).sum(dtype=np.float64)) if masses is not None else n * abs(uniform) + 1.0
    grids, powers = [], []
    with gp.Context(dims, 16) as ctx:
        for eng in (gp.api.ENGINE_SORTED, gp.api.ENGINE_STREAM):
            ctx.set_engine(eng)
            ctx.set_tile(*tile)
            ctx.zero(0)
            ctx.deposit(0, box, pos, masses, uniform)
            grids.append(ctx.read_field(0))
            assert ctx.last_engine == eng
            powers.append(ctx.power(0, 0, norm, norm))
    assert np.array_equal(grids[0], grids[1])
    ref = O.deposit(pos, box, dims, masses, uniform)
    assert np.abs(grids[0] - ref).max() <= 2e-6 * np.abs(ref).max()
    f = O.rfft_padded(ref)
    pr, cr, _ = O.port().powerspectrum(dims, f, f, 16, norm, norm)
    for p, c, _ in powers:
        assert np.array_equal(c, cr)
        ok = cr > 0
        assert np.abs(p[ok] - pr[ok]).max() <= 1e-5 * np.abs(pr[ok]).max()
        if n >= 100_000 and dims % 2 == 0:
            assert abs(p[-1] - pr[-1]) <= 1e-5 * abs(pr[-1])


@pytest.mark.parametrize("dims,n", [(64, 5000), (100, 300_000), (330, 70_000)])
def test_skipped_particles_leave_the_others_mean(gp, dims, n):
    """Non-finite and far positions are skipped and reported; the grid is that
    of the others, their mean included, and the next pass starts clean."""
    box = 1000.0
    pos = particles(n, box, 3, "uniform")
    bad = pos.copy()
    bad[5, 0] = np.nan
    bad[n // 2, 1] = np.inf
    bad[n - 1, 2] = 1e30
    keep = np.ones(n, bool)
    keep[[5, n // 2, n - 1]] = False
    with gp.Context(dims, 16) as ctx:
        ctx.set_engine(gp.api.ENGINE_SORTED)
        ctx.set_tile(16, 16, 16)
        ctx.deposit(0, box, pos[keep], None, 1.0)
        want = ctx.read_field(0)
        for _ in range(2):
            ctx.zero(0)
            ctx.deposit(0, box, bad, None, 1.0)
            with pytest.raises(gp.GenPKError) as e:
                ctx.read_field(0)
            assert "3 particle(s)" in str(e.value)
            assert np.array_equal(ctx.read_field(0), want)
        ctx.zero(0)
        ctx.deposit(0, box, pos[keep], None, 1.0)
        assert np.array_equal(ctx.read_field(0), want)


@pytest.mark.parametrize("dims,n", [(64, 70_000), (128, 200_000), (256, 500_000)])
def test_transform_of_unordered_passes_does_not_depend_on_the_engine(gp, dims, n):
    """Particles in no order: whichever engine the timed trials keep, the
    spectrum has the same bits (the z pass reads the FP32 grid or the
    accumulator)."""
    import torch
    pos = torch.from_numpy(particles(n, 1000.0, n, "uniform")).cuda()
    got = []
    for _ in range(4):
        with gp.Context(dims, 32) as ctx:
            for _ in range(2):
                ctx.zero(0)
                ctx.deposit(0, 1000.0, pos, None, 1.0)
                got.append(ctx.power(0, 0, n + 1.0, n + 1.0)[0])
    assert all(np.array_equal(got[0], g) for g in got)
