"""The RCS far-field sum (calc_RCS, modRCS.f90:60-153) against the oracle where
its launch changes: one angle (edges split over many CTAs), more angles than
the split covers, fewer edges than a CTA's threads, and a body so small in
wavelengths' terms beside its observation radius that the square-root form runs.

Tolerance: the oracle forms k R in double, R up to 10^4 lambda, so a phase is
off by up to 2 pi 1e4 2^-53 ~ 1e-11; random currents cancel to a few per cent
of the sum of moduli, hence 1e-9 of the largest value."""
import numpy as np
import pytest

from oracle import core
from oracle.rwg import RWG as ORWG

pytestmark = pytest.mark.gpu


def _plate(size):
    p = np.array([[0, 0, 0], [1, 0, 0], [1, 1, 0.2], [0, 1, 0.1]], dtype=float) * size
    return np.array([[p[0], p[1], p[2]], [p[0], p[2], p[3]]])


@pytest.mark.parametrize("body,nang", [("ico1", 1), ("ico1", 3), ("ico3", 1), ("ico3", 257), ("ico3", 4001),
                                       ("plate", 1), ("plate", 40)])
def test_rcs_sum(body, nang, gpu_lib):
    from lywell_gb300 import RWG, MoM, meshes
    tris = _plate(5.0) if body == "plate" else meshes.icosphere(int(body[3]), 1.0)
    rng = np.random.default_rng(nang)
    with MoM(RWG(tris), lam=1.0) as m:
        cur = (rng.standard_normal(m.N) + 1j * rng.standard_normal(m.N)) * 1e-3
        pol = rng.standard_normal(3) + 1j * rng.standard_normal(3)
        th, ph = rng.uniform(0, np.pi, nang), rng.uniform(0, 2 * np.pi, nang)
        for _ in range(2):   # the second call finds the edge data and the workspace laid out
            s = m.rcs(cur, pol, th, ph, ctte=0.5 + 1j)
            ref = core.sigma_rcs(ORWG(tris), 1.0, cur, pol, th, ph, ctte=0.5 + 1j)
            assert np.abs(s - ref).max() < 1e-9 * np.abs(ref).max()
