"""FP64 operator on blocks of columns where the near field, the aggregation and
the receive run on digit splits (full leaf boxes): against the single-column
operator, at column counts around the tile of 12, ragged boxes, and inputs with
a wide range, zeros, NaN and Inf.

Tolerance: both sides round; the single-column sums have up to 3000 terms, so
they are off by about 3000^0.5 2^-53 to 3000 2^-53 (6e-15 to 3e-13) of the
largest partial sums: 1e-12."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def spheroid(gpu_lib):
    from lywell_gb300 import MLFMA, RWG, meshes
    m = MLFMA(RWG(meshes.spheroid(4, (0.75, 0.1875, 0.1875), noise=0.0025, seed=1234)), lam=1.0, ladomax=0.25)
    assert m.N >= 112 * m.levels[m.nlev]["nb"] / 2   # blocks of two columns and more take the split path
    yield m
    m.close()


def _columns(m, nrhs, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((m.N, nrhs)) + 1j * rng.standard_normal((m.N, nrhs))


def _off(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("nrhs", [2, 3, 11, 12, 13, 25])
def test_blocks_match_single_columns(spheroid, nrhs):
    m = spheroid
    X = _columns(m, nrhs, nrhs)
    Y = m.matvec(X)
    for c in range(nrhs):
        assert _off(Y[:, c], m.matvec(X[:, c])) < 1e-12
    assert np.array_equal(m.matvec(X), Y)   # the same sums every time


def test_fmm_blocks(gpu_lib):
    """One level: the receive reads the translated fields themselves."""
    from lywell_gb300 import FMM, RWG, meshes
    with FMM(RWG(meshes.spheroid(4, (1.5, 0.375, 0.375))), lam=1.0, side=0.5) as m:
        X = _columns(m, 5, 1)
        Y = m.matvec(X)
        for c in range(5):
            assert _off(Y[:, c], m.matvec(X[:, c])) < 1e-12


def test_range_of_inputs(spheroid):
    """Entries over six decades, columns 1e250 and 1e-250 in one block, a zero column."""
    m = spheroid
    X = _columns(m, 5, 7)
    X[:, 0] *= 10.0 ** np.random.default_rng(8).uniform(-6, 0, m.N)
    X[:, 1] *= 1e250
    X[:, 2] *= 1e-250
    X[:, 3] = 0
    Y = m.matvec(X)
    assert not Y[:, 3].any()
    for c, s in ((0, 1.0), (1, 1e-250), (2, 1e250), (4, 1.0)):
        assert _off(Y[:, c] * s, m.matvec(X[:, c] * s)) < 1e-12


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_not_finite_stays_in_its_column(spheroid, bad):
    m = spheroid
    X = _columns(m, 4, 9)
    Y = m.matvec(X)
    X[m.N // 3, 2] = bad
    Z = m.matvec(X)
    assert not np.isfinite(Z[:, 2]).all()
    for c in (0, 1, 3):
        assert _off(Z[:, c], Y[:, c]) < 1e-14


@pytest.mark.parametrize("level,nrhs", [(0, 2), (1, 3), (2, 13), (2, 2), (3, 2), (3, 25)])
def test_dense_blocks(level, nrhs, gpu_lib):
    """The dense operator: fewer rows than a tile, ragged last blocks of 32 unknowns."""
    from lywell_gb300 import RWG, MoM, meshes
    with MoM(RWG(meshes.icosphere(level, 0.6))) as m:
        X = _columns(m, nrhs, level)
        if nrhs == 13:
            X[:, 3] *= 1e100
            X[:, 4] = 0
        Y = m.matvec(X)
        for c in range(nrhs):
            ref = m.matvec(X[:, c])
            assert np.linalg.norm(Y[:, c] - ref) <= 1e-12 * np.linalg.norm(ref)
