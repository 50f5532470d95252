"""Limited flux at the edges of its launch: cell groups cut by the grid,
row walks of 2, of a few and of 32 rows, and values where a limiter's branch and
the sign of a zero decide. Bit for bit against the oracle's loop body."""
import numpy as np
import pytest

from oracle.flux import limited_flux

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(5, 6, 1), (6, 7, 2), (7, 8, 33), (8, 9, 5), (300, 12, 3), (66, 1100, 16),
                                   (517, 129, 31), (700, 1025, 24)])
def test_bitwise(shape):
    import torch

    from titus_b200.flux import limited_flux_device

    rng = np.random.default_rng(sum(shape))
    phi = rng.standard_normal(shape)
    # plateaus, signed zeros, denormals and values near the overflow of a doubled difference
    pick = rng.random(shape)
    phi[pick < 0.25] = 0.0
    phi[(pick > 0.25) & (pick < 0.4)] = -0.0
    phi[(pick > 0.4) & (pick < 0.5)] = 1.0
    phi[(pick > 0.5) & (pick < 0.55)] *= 1e-310
    phi[(pick > 0.55) & (pick < 0.6)] *= 1e150
    ox, oz = rng.uniform(-1, 1, shape[2]), rng.uniform(-1, 1, shape[2])
    ox[0] = 0.0
    f0 = rng.standard_normal(shape)
    dev = torch.device("cuda", 0)
    d_flux = torch.from_numpy(f0).to(dev)
    limited_flux_device(torch.from_numpy(phi).to(dev), d_flux, torch.from_numpy(ox).to(dev),
                        torch.from_numpy(oz).to(dev), 0.013, 0.021)
    ref = limited_flux(phi, ox, oz, 0.013, 0.021, f0)
    assert np.array_equal(d_flux.cpu().numpy().view(np.int64), ref.view(np.int64))
