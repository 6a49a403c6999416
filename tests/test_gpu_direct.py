"""Direct passes (particles in no order, too few for a sort to pay) at the edges
of their range: the automatic engine's grid against the sorted engine's bit for
bit, and P(k) against the oracle, 1e-5 per bin (the last bin is the corner mode).
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


@pytest.mark.parametrize("dims,n,mass", [
    (3, 1, 1.0),            # odd grid, one lane of one pair
    (5, 31, -2.0),          # a warp short of one lane
    (64, 257, 1.0),         # one particle past a block
    (75, 4001, 0.25),       # odd grid: half-padded rows
    (264, 65535, 3.0),      # the largest grid and count of an untuned direct pass
    (265, 5000, 1.0),       # one past that grid: the sort
    (128, 0, 1.0),
])
def test_small_unordered_passes(gp, dims, n, mass):
    box = 1000.0
    rng = np.random.default_rng(dims)
    pos = (rng.random((n, 3)) * box).astype(np.float32)
    if n > 100:
        pos[::7] += np.float32(box)       # periodic images
        pos[1::9, 2] = np.float32(box * (1 - 0.3 / dims))  # the wrapped upper z cell
        pos[2::11] = 0.0
    norm = abs(mass) * n + 1.0
    with gp.Context(dims, 8) as ctx:
        got = []
        for _ in range(3):  # the accumulator is clear again after each
            ctx.zero(0)
            ctx.deposit(0, box, pos, None, mass)
            got.append((ctx.read_field(0), ctx.power(0, 0, norm, norm)[0]))
        assert all(np.array_equal(g[0], got[0][0]) and np.array_equal(g[1], got[0][1]) for g in got)
        # two passes onto one grid: each adds its own, each minus its own mean
        ctx.zero(0)
        ctx.deposit(0, box, pos, None, mass)
        ctx.sync()
        ctx.deposit(0, box, pos, None, mass)
        twice = ctx.read_field(0)
        ctx.set_engine(gp.api.ENGINE_SORTED)
        ctx.zero(0)
        ctx.deposit(0, box, pos, None, mass)
        assert np.array_equal(ctx.read_field(0), got[0][0])
        ctx.sync()
        ctx.deposit(0, box, pos, None, mass)
        assert np.array_equal(ctx.read_field(0), twice)
    if n >= 1000:
        pr, cr, _ = O.pk(pos, box, dims, 8, None, mass, m_norm=norm)
        ok = cr > 0
        assert (np.abs(got[0][1][ok] - pr[ok]) / pr[ok]).max() <= 1e-5


def test_skipped_particles_in_a_direct_pass(gp):
    box, n, dims = 1000.0, 3000, 64
    pos = (np.random.default_rng(1).random((n, 3)) * box).astype(np.float32)
    bad = pos.copy()
    bad[[0, 33, n - 1], [0, 1, 2]] = [np.nan, np.inf, -1e30]
    keep = np.ones(n, bool)
    keep[[0, 33, n - 1]] = False
    with gp.Context(dims, 8) as ctx:
        ctx.deposit(0, box, pos[keep], None, 1.0)
        want = ctx.read_field(0)
        for _ in range(2):
            ctx.zero(0)
            ctx.deposit(0, box, bad, None, 1.0)
            with pytest.raises(gp.GenPKError) as e:
                ctx.read_field(0)
            assert "3 particle(s)" in str(e.value)
            assert np.array_equal(ctx.read_field(0), want)


@pytest.mark.parametrize("mass", ["one", "signed"])
@pytest.mark.parametrize("dims", [75, 128])
def test_tuned_unordered_passes(gp, dims, mass):
    """Counts that the tuner times: whichever of the direct pass and the sort it
    keeps, the grid is the sorted engine's."""
    box, n = 1000.0, 70_001
    rng = np.random.default_rng(dims)
    pos = (rng.random((n, 3)) * box).astype(np.float32)
    m = None
    if mass == "signed":
        m = (rng.lognormal(0.0, 1.0, n) * np.where(rng.random(n) < 0.3, -1, 1)).astype(np.float32)
        m[::50] = 0.0
    with gp.Context(dims, 8) as ctx:
        ctx.deposit(0, box, pos, m, 1.0)
        auto = ctx.read_field(0)
        assert ((0, 0, 0), 0) in [(t, c) for t, c, _ in ctx.deposit_trials()]
        ctx.set_engine(gp.api.ENGINE_SORTED)
        ctx.zero(0)
        ctx.deposit(0, box, pos, m, 1.0)
        assert np.array_equal(ctx.read_field(0), auto)


@pytest.mark.parametrize("masses,count,own", [(True, 2_200_001, True), (False, 2_200_001, False),
                                              (False, 2_000_003, True)])
def test_transform_of_unordered_particles_follows_their_count(gp, masses, count, own):
    """On 512^3 the own z, y and x passes take fewer than 2^21 particles without
    order, or 3 * 2^21 with masses; the spectrum is the other transform's to FP32
    rounding (the FP32 transforms' 1e-5 against FP64)."""
    import torch
    from genpk_gb300 import api, synth

    pos = synth.uniform(count, 1.0, seed=5, device="cuda")
    m = torch.rand(count, device="cuda") + 0.5 if masses else None
    total = float(m.double().sum()) if masses else float(count)
    with api.Context(512, 32, timing=True) as ctx:
        ctx.deposit(0, 1.0, pos, m, 1.0)
        p, c, _ = ctx.power(0, 0, total, total)
        assert ("zfft" in ctx.stage_times()) == own
    with api.Context(512, 32) as ctx:
        ctx.set_fft_mode(1)  # cuFFT's 3-D transform
        ctx.deposit(0, 1.0, pos, m, 1.0)
        q, d, _ = ctx.power(0, 0, total, total)
    np.testing.assert_array_equal(c, d)
    np.testing.assert_allclose(p[c > 0], q[c > 0], rtol=1e-5)


@pytest.mark.parametrize("masses", [False, True])
def test_unordered_particles_on_1024_take_the_kz_major_transform(gp, masses):
    """The direct pass stays in the accumulator, which the kz-major z pass reads;
    the spectrum is the library transform's to FP32 rounding (1e-5)."""
    import torch
    from genpk_gb300 import api, synth

    n = 300_001
    pos = synth.uniform(n, 1.0, seed=9, device="cuda")
    m = torch.rand(n, device="cuda") + 0.5 if masses else None
    total = float(m.double().sum()) if masses else float(n)
    with api.Context(1024, 32, timing=True) as ctx:
        got = []
        for _ in range(2):  # the binning leaves the accumulator clear
            ctx.zero(0)
            ctx.timing_reset()
            ctx.deposit(0, 1.0, pos, m, 1.0)
            got.append(ctx.power(0, 0, total, total))
            stages = ctx.stage_times()
            assert "direct_deposit" in stages and "zfft_kz" in stages
            assert "direct_convert" not in stages or "tune" in stages
    with api.Context(1024, 32) as ctx:
        ctx.set_fft_mode(1)  # cuFFT's 3-D transform
        ctx.deposit(0, 1.0, pos, m, 1.0)
        q, d, _ = ctx.power(0, 0, total, total)
    for p, c, _ in got:
        np.testing.assert_array_equal(c, d)
        np.testing.assert_allclose(p[c > 0], q[c > 0], rtol=1e-5)


@pytest.mark.parametrize("dims,n,mass,masses,direct", [
    (269, 65535, 1.0, False, True),   # the largest accumulator and count of an untuned direct pass
    (270, 65535, 1.0, False, False),  # one past that accumulator: the sort
    (269, 5000, 1.0, True, False),    # masses: the sort
])
def test_where_untuned_direct_passes_end(gp, dims, n, mass, masses, direct):
    rng = np.random.default_rng(dims)
    pos = rng.random((n, 3)).astype(np.float32)
    m = rng.random(n).astype(np.float32) if masses else None
    with gp.Context(dims, 8, timing=True) as ctx:
        ctx.deposit(0, 1.0, pos, m, mass)
        got = ctx.read_field(0)
        stages = ctx.stage_times()
        assert ("direct_deposit" in stages) == direct and ("dep_tile" in stages) != direct
        ctx.set_engine(gp.api.ENGINE_SORTED)
        ctx.zero(0)
        ctx.deposit(0, 1.0, pos, m, mass)
        assert np.array_equal(ctx.read_field(0), got)
