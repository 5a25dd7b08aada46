"""The throughput build's square root (qsqrt in physics.cuh) against the correctly rounded one,
and what an infinite sound speed does to the time step.

qsqrt corrects a Newton step by its residual; its comment claims one unit in the last place, on
the whole range: subnormals, both sides of the scaling limit 2^-900, the largest finite values;
0 and Inf are their own roots and NaN stays NaN.
"""
import ctypes

import numpy as np
import pytest

from nuc3d_b200 import _LIB_PATH


def _qsqrt(x):
    lib = ctypes.CDLL(str(_LIB_PATH.with_name("libnuc3d_probe.so")))
    P = ctypes.POINTER(ctypes.c_double)
    lib.nuc3d_probe_qsqrt.restype = ctypes.c_int
    lib.nuc3d_probe_qsqrt.argtypes = [ctypes.c_int, P, P, ctypes.c_longlong]
    x = np.ascontiguousarray(x, dtype=np.float64)
    r = np.empty_like(x)
    assert lib.nuc3d_probe_qsqrt(0, x.ctypes.data_as(P), r.ctypes.data_as(P), x.size) == 0
    return r


@pytest.mark.gpu
def test_qsqrt_within_one_ulp():
    rng = np.random.default_rng(9)
    n = 1 << 22
    edge = 2.0 ** np.array([-1074.0, -1060, -1023, -1022, -901, -900, -899, -1, 0, 1, 1022, 1023])
    x = np.concatenate([
        rng.uniform(1.0, 4.0, n),                                            # every significand
        rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-1022, 1024, n),      # every binade
        rng.integers(1, 1 << 52, 1 << 16).view(np.float64),                  # subnormals
        edge, np.nextafter(edge, 0.0), np.nextafter(edge, np.inf), [np.finfo(np.float64).max],
        (1.0 + np.arange(1 << 12) * 2.0 ** -52) ** 2, np.arange(1.0, 4097.0) ** 2])
    x = x[(x > 0.0) & np.isfinite(x)]
    got, want = _qsqrt(x), np.sqrt(x)
    ulp = np.abs(got.view(np.int64) - want.view(np.int64))
    assert int(ulp.max()) <= 1, (int(ulp.max()), x[int(ulp.argmax())])
    assert np.array_equal(_qsqrt([0.0, np.inf]), [0.0, np.inf])
    assert np.isnan(_qsqrt([np.nan])[0])


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(16, 12, 14), (72, 64, 64)])  # tiles, and the marching sweeps
@pytest.mark.parametrize("scheme", ["weno5z", "weno7js", "upwind1st"])
def test_infinite_energy_stops_the_step(shape, scheme):
    """One cell of infinite energy: its sound speed is Inf, so is the largest eigenvalue, and
    dt is 0 in both builds."""
    import nuc3d_b200 as nb
    from nuc3d_b200 import cases as C
    q, m = C.taylor_green(shape, mach=0.8)
    q[4, shape[2] // 2, shape[1] // 2, shape[0] // 2] = np.inf
    for exact in (True, False):
        s = nb.Solver(nb.Config(scheme_ivs=(scheme,) * 3, riemann="AUSM", mach=0.8, exact=exact))
        b = s.add_block(*shape, *C.periodic_faces())
        s.set_metrics(b, *[m[k] for k in ("jac", "xi_xyz", "eta_xyz", "zeta_xyz", "dxyz")])
        s.finalize()
        s.set_q(b, q)
        assert s.rhs() == 0.0, exact
        s.close()
