"""The window engine's flush: windows with short z rows (all cells in order) and
long ones (a row to a warp) give the sorted engine's grid bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("masses", [False, True])
@pytest.mark.parametrize("dims", [71, 160])
@pytest.mark.parametrize("depth", [0, 1, 8, 61, 62, 63, 64, 200])
def test_flush_matches_sorted(depth, dims, masses):
    from genpk_gb300 import api

    # Blocks of 5000 particles (more than a window chunk), each in a box of
    # 3 x 7 cells by `depth`, the boxes running over the grid's ends.
    rng = np.random.default_rng(11 * depth + dims)
    blocks = []
    for k in range(9):
        org = rng.integers(0, dims, 3)
        org[k % 3] = dims - 2
        ext = np.array([3, 7, min(depth, dims)], float)
        if k % 2:
            ext[:2] = ext[1::-1]
        blocks.append((org + rng.random((5000, 3)) * ext) % dims)
    pos = (np.concatenate(blocks) / dims).astype(np.float32)
    pos = torch.tensor(np.where(pos >= 1, np.float32(0), pos), device="cuda")
    m = None
    if masses:
        m = torch.tensor(rng.random(len(pos)).astype(np.float32) + 0.25, device="cuda")

    def grid(engine):
        with api.Context(dims, 16) as ctx:
            ctx.set_engine(engine)
            ctx.zero(0)
            ctx.deposit(0, 1.0, pos, m, 1.0)
            return ctx.read_field(0)

    a, b = grid(api.ENGINE_SORTED), grid(api.ENGINE_WINDOW)
    np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32))
