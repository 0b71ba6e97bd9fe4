"""ILU sweeps on both sides of the rule that sends factors to the kernel for the
narrowest levels, and on more columns than the GPU has SMs: each column against
a host solve with the exported factors, and against itself alone.

ILUT by fill and drop tolerance: under four rows a level with under 600 entries
in them go to the narrow kernel, more to the one-CTA sweeps."""
import numpy as np
import pytest

from test_gpu_ilu_sweeps import _lusol

pytestmark = pytest.mark.gpu


def _levels(jlu, ju):
    n = len(ju)
    up, down = np.zeros(n, int), np.zeros(n, int)
    for i in range(n):
        up[i] = 1 + max(up[jlu[jlu[i] - 1:ju[i] - 1] - 1], default=-1)
    for i in range(n - 1, -1, -1):
        down[i] = 1 + max(down[jlu[ju[i] - 1:jlu[i + 1] - 1] - 1], default=-1)
    return up.max() + down.max() + 2


@pytest.mark.parametrize("body,fill,drop,narrow", [("sphere", 5.0, 1e-3, True), ("spheroid", 5.0, 1e-2, True),
                                                   ("spheroid", 0.3, 5e-2, True), ("spheroid", 50.0, 1e-7, False)])
def test_sweeps_on_both_sides_of_the_rule(body, fill, drop, narrow, gpu_lib):
    from lywell_gb300 import MLFMA, RWG, meshes
    tris = meshes.icosphere(2, 0.6) if body == "sphere" else meshes.spheroid(3, (0.6, 0.3, 0.3))
    with MLFMA(RWG(tris), lam=1.0, ladomax=0.25 if body == "sphere" else 0.1) as m:
        assert m.ilut(fill, drop) == 0
        alu, jlu, ju = m.ilu0_factors()
        levels = _levels(jlu, ju)
        assert (2 * m.N < 4 * levels and 2 * len(alu) < 600 * levels) == narrow, (2 * m.N / levels, len(alu) / m.N)
        rng = np.random.default_rng(7)
        y = rng.standard_normal((m.N, 160)) + 1j * rng.standard_normal((m.N, 160))
        x = m.lusol0C(y)
        for c in (0, 151, 159):
            # rounding: 2^-53 times the length of the sums (up to ~500) times the factors'
            # growth on these bodies (below 1e3) stays under 1e-10
            ref = _lusol(alu, jlu, ju, y[:, c])
            assert np.linalg.norm(x[:, c] - ref) < 1e-10 * np.linalg.norm(ref)
        assert all(np.array_equal(m.lusol0C(y[:, c]), x[:, c]) for c in range(0, 160, 13))
