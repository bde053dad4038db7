"""The fast build's refined reciprocals against correctly rounded values."""
import ctypes as C

import numpy as np
import pytest

from alpaca_b200 import build as B

pytestmark = pytest.mark.gpu


def arguments():
    """Every exponent whose reciprocal is normal with random mantissas, mantissas just
    beside the powers of two, and many arguments of order one."""
    rng = np.random.default_rng(1)
    x = [np.ldexp(1.0 + rng.random(64), e) for e in range(-1022, 1022)]
    eps = np.finfo(float).eps
    edge = np.array([1.0, 1.0 + eps, 1.0 + 2 * eps, 2.0 - eps, 2.0 - 2 * eps, 1.5])
    x += [np.ldexp(edge, e) for e in range(-1022, 1022)]
    x += [np.ldexp(np.linspace(1.0, 4.0, 1 << 18), 0)]
    x = np.concatenate(x)
    return np.concatenate([x, -x])


# In units in the last place of the result. rcp: 1/2 from the last rounding and 2^-7
# from the cube of the seed's 2^-20. rsqrt: as much, and 1/2 from the rounding of x y
# (2^-53 in e, half of which reaches y). Measured: 0.504 and 0.981.
@pytest.mark.parametrize("which,bound", [("rcp", 0.52), ("rsqrt", 1.02)])
def test_within_rounding(cuda, which, bound):
    import torch
    lib = C.CDLL(B.PROBE_LIB)
    x = arguments()
    d = torch.from_numpy(x).cuda()
    r, q = torch.empty_like(d), torch.empty_like(d)
    p = [C.c_void_p(t.data_ptr()) for t in (d, r, q)]
    assert lib.alp_probe_reciprocals(*p, C.c_int(x.size)) == 0
    a = np.abs(x) if which == "rsqrt" else x
    want = 1 / np.sqrt(a.astype(np.longdouble)) if which == "rsqrt" else 1 / a.astype(np.longdouble)
    got = (q if which == "rsqrt" else r).cpu().numpy()
    ulps = np.abs(got.astype(np.longdouble) - want) / np.spacing(np.abs(want).astype(float))
    print(which, "largest error", float(ulps.max()), "units in the last place")
    assert np.isfinite(got).all()
    assert ulps.max() <= bound
