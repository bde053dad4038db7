"""States in units far from one: the fast build's fluxes follow the strict build's
(the reference's operations) wherever its intermediate results fit in a double."""
import numpy as np
import pytest

from alpaca_b200 import api
from alpaca_b200 import native as N

pytestmark = pytest.mark.gpu


def fluxes(variant, rho, c, strict):
    """Face fluxes of a block of random gas states with densities of order rho and
    sound speeds of order c."""
    import torch
    rng = np.random.default_rng(5)
    shp = (1, 24, 24, 24)
    r, p = 1.0 + 0.5 * rng.random(shp), 1.0 + 0.5 * rng.random(shp)
    v = [rng.random(shp) - 0.5 for _ in range(3)]
    u = np.stack([r, p / 0.4 + 0.5 * r * sum(x * x for x in v)] + [r * x for x in v], axis=1)
    u[:, 0] *= rho
    u[:, 1] *= rho * c * c
    u[:, 2:] *= rho * c
    f = api.convective_fluxes(torch.from_numpy(u).cuda(), 3, variant, N.Material.make(1.4), 0.1,
                              strict=strict)
    return [x.cpu().numpy() for x in f]


# The tolerance is that of unit states (about 1e3 roundings of 1.1e-16, WENO5-Z and
# TENO5 a factor of ten more through their indicators).
@pytest.mark.parametrize("variant,rho,c", [
    ("fvchar", 1e-12, 1e3), ("fvchar", 1e12, 1e7), ("fvchar", 1e14, 1e7), ("fvchar", 1e0, 1e14),
    ("fvchar_hll", 1e14, 1e7), ("fvchar_weno5z", 1e14, 1e7), ("fvchar_teno5", 1e14, 1e7),
    ("fvprim_hll", 1e9, 1e7), ("fvprim_teno5", 1e9, 1e7),
    ("fsroe", 1e-20, 1e0), ("fsroe", 1e-40, 1e0), ("fsroe", 1e-100, 1e-3), ("fsroe", 1e9, 1e7),
    ("fsroe", 1e15, 1e2), ("fs_llf", 1e-20, 1e0), ("fs_llf", 1e-100, 1e-3), ("fs_llf", 1e14, 1e7),
    ("fs_llf", 1e0, 1e14), ("fs_teno5", 1e-40, 1e0), ("fs_teno5", 1e14, 1e7),
    ("fs_weno3", 1e-40, 1e0), ("fs_glf_weno5z", 1e-40, 1e0)])
def test_units_far_from_one(cuda, monkeypatch, variant, rho, c):
    monkeypatch.setitem(N.EXT_SCHEMES, "fvprim_hll", ("fvprim", {"riemann_solver": N.RIEMANN_HLL}))
    fast, want = fluxes(variant, rho, c, False), fluxes(variant, rho, c, True)
    for a, b in zip(fast, want):
        assert np.isfinite(a).all() and np.abs(b).max() > 0.0
        for f in range(5):
            assert np.abs(a[:, f] - b[:, f]).max() <= 1e-12 * np.abs(b[:, f]).max(), f
