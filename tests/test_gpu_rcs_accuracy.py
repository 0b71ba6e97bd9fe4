"""The RCS far-field sum against the same sum in extended precision (numpy's long
double).

Tolerance: a term's phase k (R - R0) is up to 40 on this body and rounds by 40 2^-53 =
4e-15, its other factors by a few 1e-16; random currents cancel to 3 per cent of the
sum of moduli and the square doubles: 2 * 4e-15 / 0.03 = 3e-13 of the largest value if
all erred alike; 5e-13.  (A sum over distances of 10^4 lambda in double is off by
1e-11.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MU, EPS = 1.2566370614e-6, 8.8541878176e-12


@pytest.mark.parametrize("nang", [1, 37])
def test_against_extended_precision(nang, gpu_lib):
    from lywell_gb300 import RWG, MoM, meshes
    ld = np.longdouble
    if np.finfo(ld).eps > 1e-18:
        pytest.skip("long double is double here")
    rwg = RWG(meshes.icosphere(3, 3.0))
    rng = np.random.default_rng(nang)
    cur = (rng.standard_normal(len(rwg.e_long)) + 1j * rng.standard_normal(len(rwg.e_long))) * 1e-3
    pol = np.array([1.0, 0.5j, 0.25])
    th, ph = rng.uniform(0, np.pi, nang), rng.uniform(0, 2 * np.pi, nang)
    with MoM(rwg, lam=1.0) as m:
        s = m.rcs(cur, pol, th, ph)
    # the constants as the library has them, in double
    vp = 1.0 / np.sqrt(MU * EPS)
    w = 2 * np.pi * (vp / 1.0)
    k, lam = w * np.sqrt(MU * EPS), 2 * np.pi / (w * np.sqrt(MU * EPS))
    lo, hi = rwg.e_centro.min(0), rwg.e_centro.max(0)
    D = np.sqrt(((hi - lo) ** 2).sum())
    R0 = ld(10 * max(2 * D * D / lam, 50 * D, 20 * lam))
    cp, cm = (rwg.t_baric[rwg.e_t[:, i]].astype(ld) for i in (0, 1))
    mid, dip = (cp + cm) / 2 - (0.5 * (hi + lo)).astype(ld), (cm - cp) * rwg.e_long.astype(ld)[:, None]
    re, im = cur.real.astype(ld)[:, None], cur.imag.astype(ld)[:, None]
    ref = []
    for t, p in zip(th, ph):
        t, p = ld(t), ld(p)
        r = R0 * np.array([np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)]) - mid
        d = np.sqrt((r * r).sum(1, keepdims=True))
        u = r / d
        v = (u * (dip * u).sum(1, keepdims=True) - dip) / d
        c, sn = np.cos(ld(k) * (d - R0)), np.sin(ld(k) * (d - R0))
        er, ei = (v * (c * re + sn * im)).sum(0), (v * (c * im - sn * re)).sum(0)
        ref.append((er * er + ei * ei).sum())
    ref = np.array(ref) * ld(w * MU / (4 * np.pi)) ** 2 * ld(4 * np.pi) * R0 * R0 / ld((np.abs(pol) ** 2).sum())
    assert np.abs(s - ref).max() < 5e-13 * ref.max()
