"""The forms in which the face-flux path runs a step (kernels chosen by size) give
the bits of the plain form, face fluxes of every direction and a stage update per
batch of blocks (stepping candidate 3): the last direction fused with the update
(many blocks) and whole steps in one cluster launch (few 1D / 2D blocks)."""
import numpy as np
import pytest

from alpaca_b200 import api, cases
from alpaca_b200 import native as N

pytestmark = pytest.mark.gpu

PLAIN = 3


def box(dim, n, edge, seed, B=0.0):
    """Seeded modes with a Mach-2 front on an n[0] x n[1] x n[2] block grid."""
    g = cases.BlockGrid(dim, n, (edge,) * dim, 1.0 / (16 * max(n)))
    x = g.cell_centres()
    shp = g.cells_shape()
    rng = np.random.default_rng(seed)
    rho = 1.0 + 0.1 * cases.fourier_modes(rng, shp, x, dim)
    p = 1.0 + 0.1 * cases.fourier_modes(rng, shp, x, dim)
    vel = [0.2 * cases.fourier_modes(rng, shp, x, dim) for _ in range(dim)]
    r2, u2, p2 = cases.rankine_hugoniot(rho, vel[0], p + B, 1.4, 2.0)
    behind = x[0] < 0.25
    rho, p = np.where(behind, r2, rho), np.where(behind, p2 - B, p)
    vel[0] = np.where(behind, u2, vel[0])
    return cases.Case("box", g, g.scatter(cases.primes_to_conservatives(dim, rho, p, vel, 1.4, B)),
                      1.4, B, 0.6, 1e300, 0)


def run(dim, cs, scheme, precision, path, steps, strict=False):
    e = api.Engine(dim, N.Scheme.make(scheme, precision), strict=strict, max_cases=len(cs) + 1,
                   capacity_blocks=sum(c.grid.nb for c in cs))
    ids = [e.add_case(c, max_steps=s) for c, s in zip(cs, steps)]
    e.set_path(path)
    e.step(1)
    e.step(max(steps) - 1)
    out = [e.get(i) for i in ids]
    n = e.launches(4)
    e.close()
    return out, n


def same(a, b):
    for (u, t, s), (v, tv, sv) in zip(a, b):
        assert s == sv and t == tv and np.array_equal(u, v)


# 3D from 128 blocks, 2D from 1200 blocks: 8 lines to a warp at these counts
@pytest.mark.parametrize("scheme,precision", [("fvchar", N.FP64), ("fvprim", N.FP64),
                                              ("fsroe", N.FP64), ("fvchar", N.FP32_FLUX),
                                              ("fsroe", N.FP32_FLUX), ("fvchar_weno3_hll", N.FP64),
                                              ("fs_glf_weno5z", N.FP64), ("rk2_fvchar_weno7", N.FP64)])
@pytest.mark.parametrize("dim,n,edge", [(3, (5, 5, 5), True), (3, (7, 5, 4), cases.SYMMETRY),
                                        (2, (35, 36, 1), False)])
def test_sweep_matches_plain_form(cuda, scheme, precision, dim, n, edge):
    cs = [box(dim, n, edge, 5)]
    if dim == 3:
        cs.append(box(dim, (2, 1, 2), False, 6))
    steps = [3, 2][:len(cs)]
    a, _ = run(dim, cs, scheme, precision, 0, steps)
    b, _ = run(dim, cs, scheme, precision, PLAIN, steps)
    same(a, b)


@pytest.fixture(scope="module")
def large():
    """Boxes of the larger sweeps, built once."""
    built = {}

    def get(dim, n, edge):
        if (dim, n) not in built:
            built[dim, n] = box(dim, n, edge, 8)
        return built[dim, n]
    return get


# 16 lines to a warp from 444 3D blocks and from 7104 2D blocks, 32 from 888 3D
# blocks, where every lane computes a line's last face; an odd number of 2D blocks
# leaves the last warp of the launch without lines
@pytest.mark.parametrize("scheme,precision", [("fvchar", N.FP64), ("fvprim", N.FP64),
                                              ("fsroe", N.FP64), ("fvchar", N.FP32_FLUX),
                                              ("fvchar_weno3_hll", N.FP64)])
@pytest.mark.parametrize("dim,n,edge", [(3, (10, 9, 5), True), (3, (10, 9, 10), False),
                                        (2, (35, 203, 1), True)])
def test_longer_sweeps_match_plain_form(cuda, large, scheme, precision, dim, n, edge):
    cs = [large(dim, n, edge)]
    a, _ = run(dim, cs, scheme, precision, 0, [2])
    b, _ = run(dim, cs, scheme, precision, PLAIN, [2])
    same(a, b)


@pytest.mark.parametrize("strict", [False, True])
@pytest.mark.parametrize("scheme,precision", [("fvchar", N.FP64), ("fvprim", N.FP64),
                                              ("fsroe", N.FP64), ("fvprim", N.FP32_FLUX)])
@pytest.mark.parametrize("dim,shapes,edge", [(1, ((1,),), False), (1, ((8,), (3,), (64,)), True), (1, ((240,),), False),
                                             (2, ((1, 1),), True), (2, ((3, 1), (2, 2)), False),
                                             (2, ((2, 3),), cases.SYMMETRY)])
def test_small_steps_match_plain_form(cuda, scheme, precision, dim, shapes, edge, strict):
    """One to three cases with different step budgets; the short ones stop inside
    the launch."""
    cs = [box(dim, s + (1,) * (3 - len(s)), edge, 7 + k) for k, s in enumerate(shapes)]
    steps = [9, 4, 6][:len(cs)]
    a, n = run(dim, cs, scheme, precision, 0, steps, strict)
    b, _ = run(dim, cs, scheme, precision, PLAIN, steps, strict)
    assert n == 1
    same(a, b)


def test_small_steps_rk2_and_long_calls(cuda):
    """RK2's two stages, and a call of more steps than one launch runs."""
    c = box(1, (4, 1, 1), False, 9)
    s = N.Scheme.make("fvchar")
    s.time_integrator = N.RK2
    out = []
    for path in (0, PLAIN):
        e = api.Engine(1, s, capacity_blocks=4, max_cases=1)
        i = e.add_case(c)
        e.set_path(path)
        e.step(300)
        out.append(e.get(i))
        e.close()
    same(out[:1], out[1:])


@pytest.mark.parametrize("mode", [N.HALO_ALL, N.HALO_FACES])
@pytest.mark.parametrize("dim,n,nfields", [(1, (3,), 3), (2, (3, 2), 4), (3, (2, 3, 2), 5),
                                           (3, (2, 2, 1), 1), (3, (1, 2, 3), 7)])
def test_halo_regions(cuda, dim, n, nfields, mode):
    """Periodic halos of random blocks against the periodic global field."""
    import torch
    g = cases.BlockGrid(dim, n, (True,) * dim, 1.0)
    rng = np.random.default_rng(3)
    glob = rng.standard_normal((nfields,) + g.cells_shape())
    u = g.scatter(glob)
    want = u.copy()
    for b, c in enumerate(g.coords):
        ax = [(np.arange(-4, 20) + 16 * c[d]) % (16 * g.nblocks[d]) if d < dim else np.zeros(1, int)
              for d in range(3)]
        full = glob[(slice(None),) + np.ix_(*ax)]
        if mode == N.HALO_FACES:
            out = 0
            for d in range(dim):
                shape = [1, 1, 1]
                shape[d] = 24
                out = out + np.isin(np.arange(24), np.r_[0:4, 20:24]).astype(int).reshape(shape)
            full = np.where(out == 1, full, want[b])
        want[b] = np.where(want[b] != 0.0, want[b], full)
    d_u = torch.from_numpy(u).cuda()
    api.halo_update(d_u, dim, torch.from_numpy(np.ascontiguousarray(g.nbr26)).cuda(), mode)
    assert np.array_equal(d_u.cpu().numpy(), want)


@pytest.mark.parametrize("variant", ["fvchar", "fvprim", "fsroe"])
@pytest.mark.parametrize("precision,tol", [(N.FP64, 1e-12), (N.FP32_FLUX, 1e-6)])
@pytest.mark.parametrize("rho,c", [(1e-8, 1.0), (1e-4, 1e-3), (1e3, 1e2), (1.0, 1e4)])
def test_scaled_states(cuda, variant, precision, tol, rho, c):
    """The reconstruction's eps is absolute, so states far from unit size take
    other weights: at densities of order rho and sound speeds of order c the fast
    build still follows the strict one. FP64 tolerance as for unit states; FP32:
    16 float roundings of 6e-8, for pressure differences below 2e9 (the square
    of a float smoothness indicator, (10/3 g^2)^2, must stay below 3.4e38)."""
    import torch
    case = box(3, (2, 1, 1), True, 11)
    u = case.u.copy()
    u[:, 0] *= rho
    u[:, 1] *= rho * c * c
    u[:, 2:] *= rho * c
    d_u = torch.from_numpy(u).cuda()
    api.halo_update(d_u, 3, torch.from_numpy(np.ascontiguousarray(case.grid.nbr26)).cuda())
    mat = N.Material.make(1.4, 0.0)
    a = api.space_rhs(d_u, 3, variant, mat, case.grid.cell_size, precision).cpu().numpy()
    b = api.space_rhs(d_u, 3, variant, mat, case.grid.cell_size, N.FP64, strict=True).cpu().numpy()
    assert np.isfinite(a).all()
    for f in range(5):
        assert np.abs(a[:, f] - b[:, f]).max() <= tol * np.abs(b[:, f]).max(), f
