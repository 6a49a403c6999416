"""Uniform masses around the end of the fixed-point shift's range (2^-73): the
window, stream and direct kernels give the sorted engine's grid bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,n", [(75, 5000), (128, 5000), (128, 70_001)])
@pytest.mark.parametrize("mass", [2.0 ** -72, 2.0 ** -73, 2.0 ** -74 * 1.75, 1.7e-24, -3e-26,
                                  2.0 ** -104, 2.0 ** -105, 1.2e-38, 1e-39, 3e38])
def test_uniform_mass_at_the_shift_limit(mass, dims, n):
    from genpk_gb300 import api, synth

    pos = synth.uniform(n, 1.0, seed=n, device="cuda")

    def grid(engine):
        with api.Context(dims, 8) as ctx:
            ctx.set_engine(engine)
            ctx.deposit(0, 1.0, pos, None, mass)
            return ctx.read_field(0)

    want = grid(api.ENGINE_SORTED)
    if 2.0 ** -80 < abs(mass) < 1e30:  # (a weight's unit is 2^-100 at the limit)
        assert abs(want.sum() / (n * mass) - 1) < 1e-5
    for engine in (api.ENGINE_AUTO, api.ENGINE_STREAM, api.ENGINE_WINDOW):
        np.testing.assert_array_equal(grid(engine), want, err_msg=f"engine {engine}")
