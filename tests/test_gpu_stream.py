"""The stream mode's chunks, handed out in order to whichever CTA is free: the
spectrum (its last bin is the corner mode, summed across chunks) has the same
bits every time, and the oracle's value: 1e-5 per bin, the last one included.
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
    (64, 4095, "one"),                 # one partial chunk
    (64, 2 * 152 * 4096 + 1, "one"),   # the fixed first two chunks of every CTA and one more
    (128, 700_001, "signed"),          # masses scaled to the pass's largest
    (64, 4 * 152 * 8192 + 8191, "negative"),  # 8192-particle chunks
])
def test_stream_spectrum_does_not_depend_on_the_chunks_order(gp, dims, n, mass):
    import torch
    box = 1000.0
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 3)) * box).astype(np.float32)
    masses, uniform = None, {"one": 1.0, "negative": -2.5}.get(mass, 0.0)
    if mass == "signed":
        masses = (rng.lognormal(0.0, 1.0, n) * np.where(rng.random(n) < 0.2, -1, 1)).astype(np.float32)
    norm = float(n)
    dpos = torch.from_numpy(pos).cuda()
    dm = None if masses is None else torch.from_numpy(masses).cuda()
    got = []
    with gp.Context(dims, 24) as ctx:
        ctx.set_engine(gp.api.ENGINE_STREAM)
        for _ in range(4):
            ctx.zero(0)
            ctx.deposit(0, box, dpos, dm, uniform)
            got.append(ctx.power(0, 0, norm, norm)[0])
    assert all(np.array_equal(got[0], g) for g in got)
    pr, cr, _ = O.pk(pos, box, dims, 24, masses, uniform, m_norm=norm)
    ok = cr > 0
    assert (np.abs(got[0][ok] - pr[ok]) / pr[ok]).max() <= 1e-5
