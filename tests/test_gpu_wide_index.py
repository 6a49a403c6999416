"""Kernels that index with 64 bits: forced on small grids (the GENPK_WIDE_INDEX=1
hook, read once, so in a child process), and the one grid size on which a 32-bit
pair count would wrap.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

_DIRECT = """
import sys, numpy as np, torch
sys.path.insert(0, {root!r})
from genpk_gb300 import api
rng = np.random.default_rng(2)
for dims, n in ((64, 5000), (75, 4001), (75, 70001), (100, 70001)):
    pos = torch.tensor(rng.random((n, 3)).astype(np.float32), device="cuda")
    pos[::9, 2] = 1.0 - 0.3 / dims  # the wrapped upper z cell
    m = None if n < 65536 else torch.tensor(rng.normal(size=n).astype(np.float32), device="cuda")
    with api.Context(dims, 8, timing=True) as ctx:
        for w in (None, m):
            got = []
            for _ in range(2):  # the accumulator is zero again after each
                ctx.zero(0)
                ctx.timing_reset()
                ctx.deposit(0, 1.0, pos, w, 1.0)
                ctx.sync()
                direct = "direct_convert" in ctx.stage_times()
                ctx.deposit(0, 1.0, pos, w, 1.0)
                got.append(ctx.read_field(0))
            assert n > 65536 or direct
            ctx.set_engine(api.ENGINE_SORTED)
            ctx.zero(0)
            ctx.deposit(0, 1.0, pos, w, 1.0)
            ctx.sync()
            ctx.deposit(0, 1.0, pos, w, 1.0)
            want = ctx.read_field(0)
            ctx.set_engine(api.ENGINE_AUTO)
            assert np.array_equal(got[0], want) and np.array_equal(got[1], want)
print("wide ok")
"""


def test_direct_passes_64bit_indices():
    r = subprocess.run([sys.executable, "-c", _DIRECT.format(root=ROOT)],
                       env={**os.environ, "GENPK_WIDE_INDEX": "1"}, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "wide ok" in r.stdout, r.stdout + r.stderr


# The four-particle gather with 64-bit indices against the one-particle kernel
# (arrays off a 16-byte boundary), bit for bit.
_GATHER = """
import sys, numpy as np, torch
sys.path.insert(0, {root!r})
from genpk_gb300 import api
rng = np.random.default_rng(2)
n = 20003
values = rng.random((n, 3)).astype(np.float32)
values[::50] += 2.0
values[7] = np.nan
weights = rng.random(n).astype(np.float32) + 0.5
for dims in (33, 64):
    for masses in (False, True):
        out = []
        for shift in (0, 1):
            p = torch.empty(3 * n + 1, device="cuda")[shift:shift + 3 * n].view(n, 3)
            p.copy_(torch.tensor(values))
            w = None
            if masses:
                w = torch.empty(n + 1, device="cuda")[shift:shift + n]
                w.copy_(torch.tensor(weights))
            with api.Context(dims, 16) as ctx:
                ctx.deposit(0, 1.0, p[:7].contiguous(), None, 1.0)
                ctx.power(0, 0, 7.0, 7.0)
                gp, gm, _ = ctx.adjoint(0, 1.0, p, np.cos(np.arange(16.0)), 7.0, masses=w,
                                        mass=1.0, recompute=False)
                out.append((gp.cpu().numpy(), None if gm is None else gm.cpu().numpy()))
        assert (out[0][0][:5] != 0).all() and (out[0][0][7] == 0).all()
        for a, b in zip(*out):
            assert a is b or np.array_equal(a.view(np.uint32), b.view(np.uint32))
print("wide ok")
"""


def test_gather_64bit_indices():
    r = subprocess.run([sys.executable, "-c", _GATHER.format(root=ROOT)],
                       env={**os.environ, "GENPK_WIDE_INDEX": "1"}, capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0 and "wide ok" in r.stdout, r.stdout + r.stderr


def test_unordered_particles_on_2048():
    """2048^3 cells are 2^32 + 4194304 pairs of padded elements: every cell of the
    automatic engine's grid (the direct pass: few particles on many cells) is
    converted and the accumulator is left clear.  The same cells give the same
    transform; the exact corner mode is summed in another order (1e-6)."""
    from genpk_gb300 import api, synth

    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 220e9:
        pytest.skip("needs 220 GB of free device memory")
    n = 100_003
    pos = synth.uniform(n, 1.0, seed=4, device="cuda")
    with api.Context(2048, 32) as ctx:
        got = []
        for _ in range(2):
            ctx.zero(0)
            ctx.deposit(0, 1.0, pos, None, 1.0)
            got.append(ctx.power(0, 0, float(n), float(n))[0])
        assert ((0, 0, 0), 0) in [(t, c) for t, c, _ in ctx.deposit_trials()]
        assert ctx.last_engine == api.ENGINE_STREAM
    with api.Context(2048, 32) as ctx:
        ctx.set_engine(api.ENGINE_SORTED)
        ctx.set_tile(16, 16, 16)
        ctx.deposit(0, 1.0, pos, None, 1.0)
        want, count, _ = ctx.power(0, 0, float(n), float(n))
    ok = count > 0
    for p in got:
        np.testing.assert_allclose(p[ok], want[ok], rtol=1e-6)
