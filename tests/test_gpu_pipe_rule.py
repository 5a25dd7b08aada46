"""Which launches run pipelined (pipe_pays in kernels.cuh), and that those with many tiles per CTA
give what the one-tile-per-CTA sweeps give: bit for bit in the reference-order build, to 1e-11 of
the largest value in the throughput build.  The low-order schemes, whose sweeps wait for their
tiles, are faster pipelined."""
import numpy as np
import pytest

from nuc3d_b200 import cases as C


def _solver(shape, scheme, model, exact, blocks=1):
    import nuc3d_b200 as nb
    nx, ny, nz = shape
    q, m = C.taylor_green((nx, ny * blocks, nz), mach=0.8)
    q = q * (1.0 + 0.02 * np.random.default_rng(3).uniform(-1.0, 1.0, q.shape))
    s = nb.Solver(nb.Config(scheme_ivs=(scheme,) * 3, scheme_vis=("cd2",) * 3, riemann="AUSM", model=model,
                            mach=0.8, reynolds=200.0, cfl=0.2, exact=exact))
    for b in range(blocks):
        t, i = C.periodic_faces(b)
        if blocks > 1:
            t[2], t[3] = (b - 1) % blocks, (b + 1) % blocks
        s.add_block(nx, ny, nz, t, i)
        at = np.s_[..., b * ny:(b + 1) * ny, :]
        s.set_metrics(b, *[np.ascontiguousarray(m[k][at]) for k in ("jac", "xi_xyz", "eta_xyz", "zeta_xyz", "dxyz")])
    s.finalize()
    for b in range(blocks):
        s.set_q(b, np.ascontiguousarray(q[:, :, b * ny:(b + 1) * ny]))
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("shape,scheme,exact,dirs", [
    ((64, 64, 64), "upwind1st", True, 7),
    ((64, 64, 64), "upwind1st", False, 7),
    ((64, 64, 64), "weno3js", False, 7),
    ((32, 32, 32), "weno5z", True, 7),
    ((32, 32, 32), "weno5z", False, 6),   # no pipelined kernel along xi
    ((64, 64, 64), "weno5z", False, 0),   # eta and zeta march
    ((63, 64, 64), "upwind1st", True, 0),  # odd rows
])
def test_directions_that_may_run_pipelined(shape, scheme, exact, dirs):
    s = _solver(shape, scheme, "Euler3d", exact)
    assert s.pipeline() == dirs
    s.set_pipeline(False)
    assert s.pipeline() == 0
    s.set_pipeline(True)
    assert s.pipeline() == dirs


@pytest.mark.gpu
@pytest.mark.parametrize("scheme", ["upwind1st", "weno3js"])
@pytest.mark.parametrize("model", ["Euler3d", "NavierStokes3d"])
@pytest.mark.parametrize("shape,blocks", [((130, 50, 66), 1), ((66, 38, 70), 2)])
def test_many_tiles_per_cta(scheme, model, shape, blocks):
    for exact in (True, False):
        out = []
        for on in (True, False):
            s = _solver(shape, scheme, model, exact, blocks)
            s.set_pipeline(on)
            dt = s.rhs()
            r = [s.get_rhs(b) for b in range(blocks)]
            s.step(2)
            out.append((dt, r + [s.get_q(b) for b in range(blocks)], s.residual()))
            s.close()
        a, b = out
        if exact:
            assert a[0] == b[0] and a[2] == b[2]
            assert all(np.array_equal(x, y) for x, y in zip(a[1], b[1]))
        else:
            assert abs(a[0] - b[0]) <= 1e-12 * b[0]
            for x, y in zip(a[1], b[1]):
                assert np.max(np.abs(x - y)) <= 1e-11 * np.max(np.abs(y))


@pytest.mark.gpu
@pytest.mark.parametrize("exact", [True, False])
def test_low_order_is_faster_pipelined(exact):
    """128^3 Euler upwind1st: 0.6 to 0.8 of the plain sweeps' time where it was measured."""
    s = _solver((128, 128, 128), "upwind1st", "Euler3d", exact)
    for d in range(3):
        t = {}
        for on in (True, False, True, False):
            s.set_pipeline(on)
            t[on] = min(t.get(on, 1e9), s.profile_sweep(d, 10))
        assert t[True] < 0.95 * t[False], (d, t)
