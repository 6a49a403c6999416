"""Host grids and spectra through the reference-named calls, at the sizes where
they cross the pinned ring's slots (2^20 floats), the device buffer of a host
spectrum (2^23 doubles) and the single-threaded loops (2^18 values).

A cell that comes back is one FP32 value plus the pass mean: 2e-6 of the
largest cell covers both roundings.
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


@pytest.mark.parametrize("dims,extra", [(2, 1), (5, 1), (62, 0), (64, 1), (101, 1), (160, 0), (160, 1)])
def test_fieldize_adds_rows_of_any_ring_slot(gp, dims, extra):
    box, n = 1000.0, 20_000
    rng = np.random.default_rng(dims)
    pos = (rng.random((n, 3)) * box).astype(np.float32)
    m = rng.lognormal(0.0, 0.5, n).astype(np.float32)
    row = 2 * (dims // 2 + extra)
    before = rng.random((dims, dims, row))
    out = before.copy()
    assert gp.fieldize(box, dims, out, pos, m, 0.0, extra) == 0
    ref = O.deposit(pos, box, dims, m)[:, :, :dims]
    assert np.abs(out[:, :, :dims] - before[:, :, :dims] - ref).max() <= 2e-6 * ref.max()
    assert np.array_equal(out[:, :, dims:], before[:, :, dims:])  # padding untouched
    with gp.Context(dims, 4) as ctx:  # the same cells as read_field's
        ctx.deposit(0, box, pos, m)
        assert np.array_equal(before[:, :, :dims] + ctx.read_field(0)[:, :, :dims], out[:, :, :dims])
    bad = pos.copy()
    bad[7, 1] = np.nan
    held = out.copy()
    with pytest.raises(gp.GenPKError):
        gp.fieldize(box, dims, out, bad, m, 0.0, extra)
    assert np.array_equal(out, held)


@pytest.mark.parametrize("dims", [2, 31, 208])
def test_host_spectrum_in_pieces(gp, dims):
    rng = np.random.default_rng(dims)
    shape = (dims, dims, dims // 2 + 1)
    f = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    p, c, _ = gp.powerspectrum(dims, f, None, 8, 2.0, 2.0)
    pr, cr, _ = O.port().powerspectrum(dims, f, f, 8, 2.0, 2.0)
    assert np.array_equal(c, cr)
    ok = cr > 0
    assert (np.abs(p[ok] - pr[ok]) / pr[ok]).max() <= 1e-5


@pytest.mark.parametrize("engine", [0, 1, 2, 3])
def test_loaded_spectrum_replaces_a_deposit(gp, engine):
    """A deposit still in the accumulator when a spectrum is loaded in its place
    does not come back over it."""
    import torch
    dims = 128
    rng = np.random.default_rng(3)
    shape = (dims, dims, dims // 2 + 1)
    f = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    pos = torch.tensor(rng.random((300_000, 3)).astype(np.float32), device="cuda")
    with gp.Context(dims, 8) as ctx:
        ctx.load_spectrum(0, f)
        want = ctx.power(0, 0, 2.0, 2.0)[0]
    with gp.Context(dims, 8, nfields=2) as ctx:
        ctx.set_engine(engine)
        ctx.deposit(0, 1.0, pos, None, 1.0)
        ctx.sync()
        ctx.load_spectrum(0, f)
        assert np.array_equal(ctx.power(0, 0, 2.0, 2.0)[0], want)
        ctx.deposit(1, 1.0, pos, None, 1.0)  # a later pass starts from a clear accumulator
        ctx.power(1, 1, 3e5, 3e5)
        assert np.array_equal(ctx.power(0, 0, 2.0, 2.0)[0], want)
