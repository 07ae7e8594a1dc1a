"""The projection of the conformal metric to unit determinant, near it and far
from it (a host may upload any metric)."""
import numpy as np
import pytest

from parity_util import C1, params

pytestmark = pytest.mark.gpu


# around the line between the series in det - 1 and the reciprocal cube root
# (2^-9), and determinants of 10^-24 and 10^24
@pytest.mark.parametrize("scale", [1e-8, 0.7, 1.0 - 2.0 ** -10, 1.0, 1.0 + 2.0 ** -11, 1.0 + 2.0 ** -10, 3.0, 1e8])
def test_projection_is_accurate_for_any_determinant(scale):
    from ollin.gpu import Evolution
    cfg = dict(C1, nrtotal=24, nztotal=20, nl0=0)
    e = Evolution(params(cfg))
    e.initial_data()
    e.initialize()
    e.step()
    rng = np.random.default_rng(3)
    shape = e.download(0, "A").shape
    near = abs(scale - 1.0) < 0.01
    f = {nm: scale * (1.0 + (1e-4 if near else 0.3) * rng.uniform(-1.0, 1.0, shape)) for nm in ("A", "B", "H")}
    r = (np.arange(shape[0]) - 2.5) * cfg["dr0"]
    f["C"] = (1e-4 if near else 0.1) * scale * rng.uniform(-1.0, 1.0, shape) / np.abs(r).max()
    for nm, v in f.items():
        e.upload(0, nm, v)
    e.aux(0)
    w = {nm: v.astype(np.longdouble) for nm, v in f.items()}
    det = (w["A"] * w["B"] - (r.astype(np.longdouble)[:, None] * w["C"]) ** 2) * w["H"]
    factor = np.cbrt(1.0 / det)
    for nm in f:
        want = w[nm] * factor
        # the determinant to four roundings, a third of that in its root, which
        # has an ulp of its own, and the product's rounding
        assert np.max(np.abs(e.download(0, nm) - want) / np.abs(want)) <= 2.0 ** -51, nm
