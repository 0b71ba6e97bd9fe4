"""Blocks of columns with a leading dimension above N: the bits of the block with
ld = N, and nothing written between the columns.  FP64 operator on digit splits
and on FMAs, dense operator, FP32 operator on every engine."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nrhs,engine", [("digits", 14, None), ("fma", 3, None), ("dense", 5, None),
                                              ("dense", 50, None), ("dense_small", 2, None), ("fp32", 5, 0),
                                              ("fp32", 34, 1), ("fp32", 5, 2), ("fp32", 5, 3), ("fp32", 66, 4),
                                              ("fp32", 1, -1)])
def test_padded_columns(kind, nrhs, engine, gpu_lib):
    import torch

    from lywell_gb300 import MLFMA, MoM, RWG, _capi, meshes
    if kind.startswith("dense"):
        m = MoM(RWG(meshes.icosphere(2 if kind == "dense_small" else 3, 0.6)))
    elif kind == "fma":
        m = MLFMA(RWG(meshes.icosphere(3, 1.0)), lam=1.0, ladomax=0.25)
    else:
        m = MLFMA(RWG(meshes.spheroid(3, (0.75, 0.1875, 0.1875))), lam=1.0, ladomax=0.25)
    with m:
        if engine is not None:
            m.set_block_engine(engine)
        product = gpu_lib.mlf_matvec_device if engine is None else gpu_lib.mlf_matvec32_device
        g = torch.Generator(device="cuda").manual_seed(1)
        x = torch.randn(nrhs, m.N, dtype=torch.complex128, device="cuda", generator=g)
        y = torch.full_like(x, float("nan"))
        ld = m.N + 37
        xp = torch.full((nrhs, ld), float("nan"), dtype=torch.complex128, device="cuda")   # read: a NaN shows
        xp[:, :m.N] = x
        yp = torch.full((nrhs, ld), -5.0, dtype=torch.complex128, device="cuda")
        torch.cuda.synchronize()
        for a, b, n in ((x, y, m.N), (xp, yp, ld)):
            st = product(m.handle, ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(b.data_ptr()), nrhs, n, None)
            assert st == 0, _capi.load().mlf_last_error(m.handle)
            torch.cuda.synchronize()
        assert torch.isfinite(torch.view_as_real(y)).all()
        assert torch.equal(yp[:, :m.N], y)
        assert (yp[:, m.N:] == -5.0).all()
