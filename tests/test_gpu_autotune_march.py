"""nuc3d_autotune times only kernels that differ: a marching direction (throughput build, WENO5 eta
and zeta of 2^18 cells or more) has no tiles, so it keeps its shape and is timed once."""
import pytest

from nuc3d_b200 import cases as C


def _solver(shape, scheme, exact):
    import nuc3d_b200 as nb
    q, m = C.taylor_green(shape, mach=0.8)
    s = nb.Solver(nb.Config(scheme_ivs=(scheme,) * 3, riemann="AUSM", mach=0.8, exact=exact))
    b = s.add_block(*shape, *C.periodic_faces())
    s.set_metrics(b, *[m[k] for k in ("jac", "xi_xyz", "eta_xyz", "zeta_xyz", "dxyz")])
    s.finalize()
    s.set_q(b, q)
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("tiles", [(0, 0, 0), (2, 1, 2)])
def test_marching_directions_keep_their_shape(tiles):
    s = _solver((64 + 2 * tiles[0], 66, 64), "weno5z", False)  # (a grid of its own: choices are cached)
    s.set_tiles(tiles)
    r = s.autotune(reps=2)
    assert r["shape"][1:] == tiles[1:]
    assert all(x is not None for x in r["ms"][0])
    for d in (1, 2):
        assert [x is not None for x in r["ms"][d]] == [k == tiles[d] for k in range(3)]
