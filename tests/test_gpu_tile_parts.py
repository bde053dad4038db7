"""The fused tile path with quarter, half and whole blocks as items (148 SMs: up to
37, up to 147, from 148 blocks) against the face-flux path: equal bits."""
import numpy as np
import pytest

from alpaca_b200 import api, cases
from alpaca_b200 import native as N
from test_gpu_step_forms import box, same

pytestmark = pytest.mark.gpu

FACE, TILE16, TILE12 = 0, 4, 5


def run(cs, scheme, precision, path, steps, strict=False):
    e = api.Engine(3, N.Scheme.make(scheme, precision), strict=strict, max_cases=len(cs),
                   capacity_blocks=sum(c.grid.nb for c in cs))
    ids = [e.add_case(c, max_steps=s) for c, s in zip(cs, steps)]
    e.set_path(path)
    e.step(2)
    e.step(max(steps) - 2)
    out = [e.get(i) for i in ids]
    e.close()
    return out


@pytest.mark.parametrize("scheme,precision", [("fvchar", N.FP64), ("fsroe", N.FP64),
                                              ("fvprim", N.FP32_FLUX)])
@pytest.mark.parametrize("n,edge", [((1, 1, 1), True), ((1, 1, 1), False),
                                    ((2, 1, 3), cases.SYMMETRY), ((37, 1, 1), True),
                                    ((19, 2, 1), cases.SYMMETRY), ((7, 7, 3), False),
                                    ((37, 2, 2), True)])
def test_items_match_face_path(cuda, scheme, precision, n, edge):
    cs = [box(3, n, edge, 21)]
    want = run(cs, scheme, precision, FACE, [4])
    for path in (TILE16, TILE12):
        same(run(cs, scheme, precision, path, [4]), want)


@pytest.mark.parametrize("strict", [False, True])
def test_cases_of_different_length(cuda, strict):
    """Three cases in part-block items, two of which end inside a call, and RK2."""
    cs = [box(3, (2, 2, 1), True, 22), box(3, (1, 2, 1), False, 23), box(3, (3, 1, 1), True, 24)]
    for scheme in ("fvchar", "fsroe"):
        s = N.Scheme.make(scheme)
        for integrator in (N.RK3, N.RK2):
            s.time_integrator = integrator
            out = []
            for path in (TILE16, FACE):
                e = api.Engine(3, s, strict=strict, max_cases=3, capacity_blocks=9)
                ids = [e.add_case(c, max_steps=k) for c, k in zip(cs, (7, 3, 5))]
                e.set_path(path)
                e.step(4)
                e.step(4)
                out.append([e.get(i) for i in ids])
                e.close()
            same(out[0], out[1])
            assert [g[2] for g in out[0]] == [7, 3, 5]
