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


def _neighbours(m, kind):
    """Columns whose ranges differ: flat, over twelve decades along the body (up and
    down), unit vectors, spikes."""
    X = _columns(m.N, 14, 12)
    along = np.linspace(0.0, 12.0, m.N)
    X[:, 1] *= 10.0 ** along
    X[:, 2] *= 10.0 ** -along
    X[:, 3] = 0
    X[m.N // 2, 3] = 1.0
    X[:, 4] = 0
    X[m.N // 2 + 1, 4] = 1e-9j
    X[::97, 5] *= 1e12
    X[::89, 6] *= 1e-12
    X[:, 7] = X[:, 7].real
    X[:, 8] *= 1e-120
    return X


@pytest.mark.parametrize("kind", ["spheroid4", "superellipsoid", "dense"])
def test_columns_of_different_ranges(kind, gpu_lib):
    """A column's accuracy does not depend on its neighbours: each against itself
    alone, over the norm and, for the dense operator, row by row (relative to the
    row's terms).  A warp's sums of n <= 3000 terms have n / 32 + 5 = 100 roundings in
    a row: under 100 2^-53 = 1.1e-14 of the terms' sum, which is up to n^0.5 times the
    result, and of either sign, so 100^0.5 2^-53 n^0.5 = 6e-14 of the norm."""
    with _body(kind) as m:
        X = _neighbours(m, kind)
        Y = m.matvec(X)
        for c in range(X.shape[1]):
            ref = m.matvec(X[:, c])
            assert np.linalg.norm(Y[:, c] - ref) < 1e-13 * np.linalg.norm(ref), c
        if kind == "dense":
            Z = m.matvec(np.eye(m.N, 64))   # |Z| of 64 sources at a time
            A = np.concatenate([np.abs(m.matvec(np.roll(np.eye(m.N, 64), k, 0))) for k in range(0, m.N, 64)], 1)
            assert np.array_equal(np.abs(Z), A[:, :64])
            for c in range(X.shape[1]):
                terms = A @ np.abs(X[:, c])
                assert (np.abs(Y[:, c] - m.matvec(X[:, c])) <= 1e-14 * terms).all(), c


@pytest.mark.parametrize("nrhs", [1, 3, 60])
def test_first_dense_block_under_capture(nrhs, gpu_lib):
    """A dense operator's products allocate nothing and wait for nothing: the first
    one of a context, of any number of columns, can be captured in a CUDA graph."""
    import torch
    with _body("dense") as m:
        x = torch.from_numpy(np.ascontiguousarray(_columns(m.N, nrhs, 3).T)).cuda()
        y = torch.zeros_like(x)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            m.matvec_device(x.data_ptr(), y.data_ptr(), nrhs, s.cuda_stream)
        graph.replay()
        torch.cuda.synchronize()
        ref = m.matvec(x.cpu().numpy().T)
        assert np.array_equal(y.cpu().numpy().T, ref.reshape(m.N, nrhs))


@pytest.mark.parametrize("nrhs", [65536, 66000, 70001])
def test_more_dense_columns_than_a_grid_has_rows(nrhs, gpu_lib):
    """A tetrahedron's six unknowns.  Against the matrix itself; sums of six terms,
    1e-14 of the norm."""
    from lywell_gb300 import RWG, MoM
    v = 0.3 * np.array([[1.0, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]])
    tris = v[np.array([[0, 1, 2], [0, 3, 1], [0, 2, 3], [1, 3, 2]])]
    with MoM(RWG(tris)) as m:
        assert m.N == 6
        Z = m.matvec(np.eye(6) + 0j)
        X = _columns(6, nrhs, 1)
        assert np.linalg.norm(m.matvec(X) - Z @ X) < 1e-14 * np.linalg.norm(Z @ X)
