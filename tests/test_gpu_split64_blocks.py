"""FP64 products of blocks of columns on digit splits (full leaf boxes, and the
dense operator): blocks of different sizes one after the other on one context.

A product of a block is a fixed sequence of sums, so a context that has seen
other blocks gives the bits of a new one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _columns(n, nrhs, seed):
    rng = np.random.default_rng(seed)
    return rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))


def _body(kind):
    from lywell_gb300 import MLFMA, MoM, RWG, meshes
    if kind == "dense":
        return MoM(RWG(meshes.icosphere(3, 0.6)))
    tris = {"spheroid4": lambda: meshes.spheroid(4, (0.75, 0.1875, 0.1875)),
            "spheroid5": lambda: meshes.spheroid(5, (1.5, 0.375, 0.375)),
            "superellipsoid": lambda: meshes.superellipsoid(4, (1.0, 0.5, 0.5))}[kind]()
    return MLFMA(RWG(tris), lam=1.0, ladomax=0.25)


@pytest.mark.parametrize("kind", ["spheroid4", "spheroid5", "superellipsoid", "dense"])
def test_smaller_block_first(kind, gpu_lib):
    sizes = (12, 18, 24, 64)
    with _body(kind) as m:
        X = _columns(m.N, 64, 5)
        after = [m.matvec(X[:, :n]) for n in sizes]
    for n, y in zip(sizes, after):
        with _body(kind) as m:
            assert np.array_equal(m.matvec(X[:, :n]), y)


@pytest.mark.parametrize("kind", ["spheroid4", "dense"])
@pytest.mark.parametrize("size", [1e-12, 1e15])
def test_finite_columns_beside_a_nan(kind, size, gpu_lib):
    """Columns of another magnitude than one beside a column with a NaN.  Against the
    columns alone: both sides round, sums of up to 3000 terms, 1e-13 of the norm."""
    with _body(kind) as m:
        X = size * _columns(m.N, 14, 11)
        X[m.N // 3, 2] = np.nan
        Y = m.matvec(X)
        assert np.isnan(Y[:, 2]).any()
        for c in (0, 3, 13):
            ref = m.matvec(X[:, c])
            assert np.linalg.norm(Y[:, c] - ref) < 1e-13 * np.linalg.norm(ref)
