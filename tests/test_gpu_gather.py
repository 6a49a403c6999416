"""The gradient's gather: four particles per thread with 32-bit offsets against
the one-particle kernel, which splits every coordinate and indexes in general."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

BOX = 1.0


def _positions(dims, order):
    """Particles in every place that the fast split treats apart: cell corners
    and the last cell of each axis, outside the box, and non-finite ones."""
    rng = np.random.default_rng(7)
    if order == "lattice":
        g = (np.arange(32) + 0.5) / 32
        pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
        pos = pos + rng.normal(0, 0.2 / dims, pos.shape)
    else:
        pos = rng.random((20003, 3))
    pos = pos.astype(np.float32)
    cell = np.float32(1.0 / dims)
    k = rng.integers(0, dims + 1, (3000, 3)).astype(np.float32)
    pos[1000:4000] = k * cell  # corners, with 0 and the box's end
    pos[4000:4600, 2] = np.nextafter(np.float32(1), np.float32(0))
    pos[4600:4700, 1] = np.nextafter(np.float32(1), np.float32(0))
    pos[4700:4800, 0] = np.nextafter(np.float32(1), np.float32(0))
    pos[4800:5000] -= np.float32(1.25)
    pos[5000:5100] += np.float32(3.0)
    bad = np.array([np.nan, np.inf, -np.inf, 3e38], np.float32)
    for i, v in enumerate(np.tile(bad, 12)):
        pos[5100 + 5 * i, i % 3] = v
    return pos


@pytest.mark.parametrize("masses", [False, True])
@pytest.mark.parametrize("order", ["random", "lattice"])
@pytest.mark.parametrize("dims", [16, 33, 64, 100, 1024])
def test_gather_kernels_agree(dims, order, masses):
    from genpk_gb300 import api

    pos = _positions(dims, order)
    n = len(pos) - len(pos) % 4 + 3
    pos = np.concatenate([pos, pos])[:n]
    finite = np.isfinite(pos * np.float32(dims)).all(axis=1)
    m = np.random.default_rng(3).random(n).astype(np.float32) + 0.5
    rng = np.random.default_rng(5)
    dep = torch.tensor(rng.random((40000, 3)).astype(np.float32), device="cuda")
    slope = rng.normal(size=16)

    def gradients(shift):
        # the same values at a 16-byte boundary and 4 bytes past one
        p = torch.empty(3 * n + 1, device="cuda")[shift:shift + 3 * n].view(n, 3)
        p.copy_(torch.tensor(pos))
        w = None
        if masses:
            w = torch.empty(n + 1, device="cuda")[shift:shift + n]
            w.copy_(torch.tensor(m))
        with api.Context(dims, 16) as ctx:
            if order == "lattice":
                ctx.set_engine(3)  # the gather follows the latest pass's engine
            ctx.zero(0)
            ctx.deposit(0, BOX, dep, None, 1.0)
            ctx.power(0, 0, 4e4, 4e4)
            gp, gm, _ = ctx.adjoint(0, BOX, p, slope, 4e4, masses=w, mass=1.0, recompute=False)
            return gp.cpu().numpy(), None if gm is None else gm.cpu().numpy()

    (ga, ma), (gb, mb) = gradients(0), gradients(1)
    assert (ga[finite] != 0).any()
    np.testing.assert_array_equal(ga.view(np.uint32), gb.view(np.uint32))
    assert (ga[~np.isfinite(pos).all(axis=1)] == 0).all()
    if masses:
        np.testing.assert_array_equal(ma.view(np.uint32), mb.view(np.uint32))


@pytest.mark.parametrize("nrbins", [1, 512, 513])
def test_coefficients_by_value_and_by_copy(nrbins):
    """Up to 512 per-bin coefficients go up as a kernel parameter, more by a
    copy; both give the oracle's gradient within the adjoint tests' 1e-4."""
    from genpk_gb300 import api, synth
    from oracle import oracle as O

    dims, box = 36, 1000.0
    pos = synth.zeldovich(dims, box, seed=21)
    m = O.total_mass(len(pos), None, 1.0)
    with api.Context(dims, nrbins) as ctx:
        ctx.deposit(0, box, pos, None, 1.0)
        p, c, _ = ctx.power(0, 0, m, m)
        g = np.where(c > 0, 1.0 + np.cos(np.arange(nrbins)), 0.0)
        gpos, _, _ = ctx.adjoint(0, box, pos, g, m, mass=1.0)
    ref, _, _ = O.reference_gradient(pos, box, dims, nrbins, g, None, 1.0, m_norm=m)
    assert np.abs(gpos - ref).max() <= 1e-4 * np.abs(ref).max()


def _gather_form(ctx, call):
    """The last template argument of the gather kernel that `call` launches
    (2: single cells, 3: z pairs); None where kernels cannot be traced."""
    import re
    from torch.profiler import ProfilerActivity, profile

    kinds = [ProfilerActivity.CPU, ProfilerActivity.CUDA]
    with profile(activities=kinds):  # (the first trace of a process may come back empty)
        torch.ones(1, device="cuda")
        torch.cuda.synchronize()
    with profile(activities=kinds) as prof:
        call()
        torch.cuda.synchronize()
    names = [e.key for e in prof.key_averages() if "k_gather" in e.key]
    if not names:
        return None
    return int(re.search(r"k_gather4<\w+, (\d)>", names[0].replace("(int)", "")).group(1))


def test_gather_form_follows_the_fields_order():
    """The tuner's direct pass has particles in no order: z pairs.  With the
    forward pass kept, the field's own latest pass counts, not the context's."""
    from genpk_gb300 import api, synth

    dims, n = 128, 400_000
    random = synth.uniform(n, BOX, seed=3, device="cuda")
    lattice = synth.zeldovich(128, BOX, seed=3, device="cuda")
    slope = np.ones(16)
    with api.Context(dims, 16, nfields=2) as ctx:
        def grad(field, pos):
            ctx.power(field, field, float(n), float(n))
            return ctx.adjoint(field, BOX, pos, slope, float(n), mass=1.0, recompute=False)

        def deposit(field, pos):
            ctx.zero(field)
            ctx.deposit(field, BOX, pos, None, 1.0)
            ctx.sync()

        deposit(0, random)
        assert ((0, 0, 0), 0) in [(t, c) for t, c, _ in ctx.deposit_trials()]
        form = _gather_form(ctx, lambda: grad(0, random))
        if form is None:
            pytest.skip("no kernel trace on this machine")
        assert form == 3
        deposit(0, lattice)  # found to be in order: the stream engine
        assert ctx.last_engine == api.ENGINE_STREAM
        deposit(1, random)
        assert _gather_form(ctx, lambda: grad(0, lattice)) == 2
        deposit(0, lattice)
        deposit(1, random)
        assert _gather_form(ctx, lambda: grad(1, random)) == 3
