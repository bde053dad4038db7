"""Exchanging the axes of a state exchanges the axes of its fluxes, to the bit, in
the forms that promise it: primitive reconstruction (FP64 and FP32 flux), prime
states and the time-step size."""
import itertools

import numpy as np
import pytest

from alpaca_b200 import api
from alpaca_b200 import native as N

pytestmark = pytest.mark.gpu


def state(dim, gamma, B, seed):
    rng = np.random.default_rng(seed)
    shp = (2,) + tuple(24 if d < dim else 1 for d in range(3))
    rho, p = 1.0 + 0.5 * rng.random(shp), 1.0 + 0.5 * rng.random(shp)
    v = [rng.random(shp) - 0.5 for _ in range(dim)]
    e = (p + gamma * B) / (gamma - 1.0) + 0.5 * rho * sum(x * x for x in v)
    return np.stack([rho, e] + [rho * x for x in v], axis=1)


def exchanged(a, perm, first=2):
    """New axis d is old axis perm[d], of the grid and of the vector that starts at
    field `first`."""
    dim = len(perm)
    fields = list(range(a.shape[1]))
    for d, q in enumerate(perm):
        fields[first + d] = first + q
    axes = [0, 1] + [2 + q for q in perm] + list(range(2 + dim, 5))
    return np.ascontiguousarray(a[:, fields].transpose(axes))


def exchanges(dim):
    return [p for p in itertools.permutations(range(dim)) if p != tuple(range(dim))]


@pytest.mark.parametrize("variant,precision", [("fvprim", N.FP64), ("fvprim", N.FP32_FLUX),
                                               ("fvprim_teno5", N.FP64), ("fvprim_hll", N.FP64)])
@pytest.mark.parametrize("gamma,B,safe", [(1.4, 0.0, False), (1.4, 0.0, True),
                                          (6.12, 3430.0, False)])
@pytest.mark.parametrize("dim", [2, 3])
def test_primitive_fluxes(cuda, monkeypatch, dim, gamma, B, safe, variant, precision):
    import torch
    if variant == "fvprim_hll":
        if dim == 2:
            pytest.skip("HLL's energies in 2D add two products in axis order")
        monkeypatch.setitem(N.EXT_SCHEMES, variant, ("fvprim", {"riemann_solver": N.RIEMANN_HLL}))
    u = state(dim, gamma, B, 3)
    mat = N.Material.make(gamma, B, safe)

    def fluxes(a):
        f = api.convective_fluxes(torch.from_numpy(a).cuda(), dim, variant, mat, 0.1, precision)
        return [x.cpu().numpy() for x in f[:dim]]

    f = fluxes(u)
    for p in exchanges(dim):
        g = fluxes(exchanged(u, p))
        for d in range(dim):
            assert np.array_equal(exchanged(f[p[d]], p), g[d]), (p, d)


@pytest.mark.parametrize("gamma,B", [(1.4, 0.0), (6.12, 3430.0)])
def test_prime_states_and_time_step(cuda, gamma, B):
    import torch
    mat = N.Material.make(gamma, B)
    for seed in range(8):
        u = state(3, gamma, B, seed)
        prim = api.prime_states(torch.from_numpy(u).cuda(), 3, mat).cpu().numpy()
        dt = api.timestep_size(torch.from_numpy(u).cuda(), 3, mat, 0.1, 0.6)
        for p in exchanges(3):
            v = torch.from_numpy(exchanged(u, p)).cuda()
            assert np.array_equal(exchanged(prim, p), api.prime_states(v, 3, mat).cpu().numpy())
            assert api.timestep_size(v, 3, mat, 0.1, 0.6) == dt
