"""The tcgen05 engine, its tiles cut into parts by equal shares of the chunks, in
rings of either depth, against the FP64 operator.

Bodies: about 46 tiles of 145 rows (four or five parts each; rings of four stages,
the receive's three), 184 tiles of 42 rows (one or two parts; at most 96 rows: five
stages, the receive's four) and 736 tiles of 42 rows (most in one part, as before).
The aggregation's tiles are rows of directions, with a depth of their own.
Columns: the fewest, one over half a column tile, one over a whole one, and back
to few in the workspaces of the larger block.

Tolerance: the FP32 operator's own accuracy against FP64 with 0.25 lambda
leaves, 2e-5; parts change only the order of FP32 sums.  (The mma.sync engine is
no oracle here: it is 2.6e-5 from FP64 on the first body.)
"""
import numpy as np
import pytest

from lywell_gb300 import MLFMA, RWG, meshes

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float(np.linalg.norm(np.ravel(a - b)) / np.linalg.norm(np.ravel(b)))


@pytest.mark.parametrize("level,axis", [(4, 0.75), (4, 1.5), (5, 3.0)])
def test_parts_and_rings(gpu_lib, level, axis):
    tris = meshes.spheroid(level, (axis, axis / 4, axis / 4), noise=0.005, seed=1234)
    m = MLFMA(RWG(tris), lam=1.0, ladomax=0.25)
    rng = np.random.default_rng(level)
    for nrhs in (2, 33, 65, 3):
        X = rng.standard_normal((m.N, nrhs)) + 1j * rng.standard_normal((m.N, nrhs))
        X[:, -1] *= 1e3
        m.set_block_engine(4)
        Y4 = m.matvec32(X)
        assert np.array_equal(Y4, m.matvec32(X))
        for k in range(nrhs):
            assert _rel(Y4[:, k], m.matvec(X[:, k])) < 2e-5

    # the near-pattern preconditioner on the same items
    assert m.nearinv(own_only=True) == 0
    B = rng.standard_normal((m.N, 3)) + 1j * rng.standard_normal((m.N, 3))
    out = m.solve(B, errmax=1e-3, maxit=2000, precond="nearinv", mixed=True)
    for k in range(3):
        assert out["status"][k] == "converged"
        assert np.linalg.norm(m.matvec(out["x"][:, k]) - B[:, k]) / np.linalg.norm(B[:, k]) < 1e-3
    m.close()


@pytest.mark.parametrize("cut,nrhs", [(1, 2), (7, 31), (30, 33), (5, 17)])
def test_ragged_blocks(gpu_lib, cut, nrhs):
    """An open body whose unknowns fill no tile of 32 rows: the block's copy to box
    order and the sums back, all engines.  A misplaced row is an error of order one;
    the FP32 operator is 2e-5 from FP64, the bound five times that."""
    tris = meshes.icosphere(3, 1.0)[:-cut]
    m = MLFMA(RWG(tris), lam=1.0, ladomax=0.25)
    assert m.N % 32
    rng = np.random.default_rng(cut)
    X = rng.standard_normal((m.N, nrhs)) + 1j * rng.standard_normal((m.N, nrhs))
    X[3, 0] = 0.0
    Y = np.stack([m.matvec(X[:, k].copy()) for k in range(nrhs)], 1)
    for engine in (0, 1, 3, 4, -1):
        m.set_block_engine(engine)
        Y32 = m.matvec32(X)
        assert max(_rel(Y32[:, k], Y[:, k]) for k in range(nrhs)) < 1e-4
    m.close()
