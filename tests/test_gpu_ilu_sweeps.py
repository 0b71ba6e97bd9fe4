"""ILU sweeps on the GPU (lusol0C) against a host solve with the exported
factors in 64 bits: the one-CTA sweeps (narrow dependency levels) at sizes
around a warp's and a CTA's share of rows, several columns, and the sweeps by
levels (vectors too long for one CTA's shared memory)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lusol(alu, jlu, ju, y):
    """lusol0C (modIterativo.f90:504-560) on 1-based MSR factors."""
    a = alu.astype(np.complex128)
    x = y.astype(np.complex128).copy()
    n = len(ju)
    for i in range(n):
        k = slice(jlu[i] - 1, ju[i] - 1)
        x[i] -= a[k] @ x[jlu[k] - 1]
    for i in range(n - 1, -1, -1):
        k = slice(ju[i] - 1, jlu[i + 1] - 1)
        x[i] = a[i] * (x[i] - a[k] @ x[jlu[k] - 1])
    return x


@pytest.mark.parametrize("level,radius,kind", [(2, 0.6, "ilu0"), (2, 0.6, "ilut"), (3, 1.0, "ilu0"), (4, 1.5, "ilu0"),
                                               (5, 3.0, "ilu0")])
def test_sweeps_match_the_factors(level, radius, kind, gpu_lib):
    from lywell_gb300 import MLFMA, RWG, meshes
    with MLFMA(RWG(meshes.icosphere(level, radius)), lam=1.0, ladomax=0.25) as m:
        assert (m.ilutC() if kind == "ilut" else m.ilu0C()) == 0
        alu, jlu, ju = m.ilu0_factors()
        rng = np.random.default_rng(level)
        y = rng.standard_normal((m.N, 3)) + 1j * rng.standard_normal((m.N, 3))
        x = m.lusol0C(y)
        for c in range(3):
            # rounding: 2^-53 times the length of the sums (up to ~300) times the factors' growth
            # on these bodies (below 1e3) stays under 1e-10
            ref = _lusol(alu, jlu, ju, y[:, c])
            assert np.linalg.norm(x[:, c] - ref) < 1e-10 * np.linalg.norm(ref)
        assert np.array_equal(m.lusol0C(y[:, 1]), x[:, 1])   # a column does not depend on its neighbours


def test_sweeps_carry_nan(gpu_lib):
    """A NaN in the right-hand side reaches the rows that depend on it and no wait runs out."""
    from lywell_gb300 import MLFMA, RWG, meshes
    with MLFMA(RWG(meshes.icosphere(3, 1.0)), lam=1.0, ladomax=0.25) as m:
        assert m.ilu0C() == 0
        y = np.ones(m.N, dtype=np.complex128)
        y[m.N // 2] = np.nan
        x = m.lusol0C(y)
        assert np.isnan(x).any()
        y[m.N // 2] = 1.0
        assert np.isfinite(m.lusol0C(y)).all()


@pytest.mark.parametrize("level,radius,fill,droptol", [(2, 0.6, 1.0, 1e-2), (2, 0.6, 60.0, 1e-6), (3, 1.0, 5.0, 1e-3),
                                                       (3, 1.0, 20.0, 1e-5)])
def test_narrow_levels(level, radius, fill, droptol, gpu_lib):
    """ILUT factors of few rows a level: rows of less than half a batch of 32
    entries up to rows of several loads of four batches; NaN is carried."""
    from lywell_gb300 import MLFMA, RWG, meshes
    with MLFMA(RWG(meshes.icosphere(level, radius)), lam=1.0, ladomax=0.25) as m:
        assert m.ilut(fill, droptol) == 0
        alu, jlu, ju = m.ilu0_factors()
        rng = np.random.default_rng(level)
        y = rng.standard_normal((m.N, 2)) + 1j * rng.standard_normal((m.N, 2))
        x = m.lusol0C(y)
        for c in range(2):
            ref = _lusol(alu, jlu, ju, y[:, c])   # same bound as above
            assert np.linalg.norm(x[:, c] - ref) < 1e-10 * np.linalg.norm(ref)
        y[m.N // 2, 0] = np.nan
        z = m.lusol0C(y)
        assert np.isnan(z[:, 0]).any() and np.array_equal(z[:, 1], x[:, 1])
