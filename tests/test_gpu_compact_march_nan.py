"""Values that are not finite on a line of the marching crweno5 sweeps: a NaN or Inf inside makes
the line's system NaN, but the faces next to the line's ends are explicit and lie outside it, so
the same cells stay finite as in the three-kernel path (rows, Thomas, faces), whose elimination
is the reference's (src/crweno5.cpp:207-218)."""
import numpy as np
import pytest

from nuc3d_b200 import cases as C

IDS = {"outlet": 1, "wall": 2}


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("place", [0.5, 0.0, 0.99])   # inside, at the first and at the last cell
@pytest.mark.parametrize("faces", [(None,) * 6, (None, None, "wall", "outlet", "outlet", "wall")])
def test_same_cells_stay_finite(value, place, faces):
    import nuc3d_b200 as nb
    shape = (96, 64, 65)
    q, m = C.gaussian_pulse(shape)
    t, i = C.periodic_faces()
    for f, kind in enumerate(faces):
        if kind:
            t[f], i[f] = -1, IDS[kind]
    at = tuple(int(place * n) for n in shape[::-1])
    q[(4,) + at] = value
    out = []
    for fused in (True, False):
        s = nb.Solver(nb.Config(scheme_ivs=("weno5z", "crweno5", "crweno5"), riemann="AUSM", mach=1.0, exact=False))
        b = s.add_block(*shape, t, i)
        s.set_metrics(b, *[m[k] for k in ("jac", "xi_xyz", "eta_xyz", "zeta_xyz", "dxyz")])
        s.finalize()
        s.set_compact_solver(fused)
        s.set_q(b, q)
        s.rhs()
        out.append(s.get_rhs(b))
        s.close()
    a, b = (np.isfinite(x) for x in out)
    assert np.array_equal(a, b), (int(a.sum()), int(b.sum()))
    assert not a.all() and a.any()
    assert np.max(np.abs(out[0][a] - out[1][a])) <= 1e-11 * np.max(np.abs(out[1][a]))
