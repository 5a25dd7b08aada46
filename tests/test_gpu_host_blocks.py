"""nuc3d_solve_host on many small blocks whose eta and zeta sweeps march (throughput build, 2^18
cells or more in all): stage 2 runs by groups of blocks, with the bits of the device-resident
steps, and is not slower than the whole step between whole copies."""
import time

import numpy as np
import pytest

from nuc3d_b200 import cases as C


def _make(sizes, model):
    """Blocks of the given extents in a row along eta, periodic as a whole."""
    import nuc3d_b200 as nb
    nx, nz = 16, 16
    q, m = C.taylor_green((nx, sum(sizes), nz), mach=0.8)
    s = nb.Solver(nb.Config(scheme_ivs=("weno5z",) * 3, riemann="AUSM", model=model, mach=0.8, reynolds=200.0,
                            cfl=0.2, exact=False))
    out, lo = [], 0
    for b, ny in enumerate(sizes):
        t, i = C.periodic_faces(b)
        t[2], t[3] = (b - 1) % len(sizes), (b + 1) % len(sizes)
        s.add_block(nx, ny, nz, t, i)
        at = np.s_[..., lo:lo + ny, :]
        s.set_metrics(b, *[np.ascontiguousarray(m[k][at]) for k in ("jac", "xi_xyz", "eta_xyz", "zeta_xyz", "dxyz")])
        out.append(np.ascontiguousarray(q[at]))
        lo += ny
    s.finalize()
    for b, qb in enumerate(out):
        s.set_q(b, qb)
    return s, out


@pytest.mark.gpu
@pytest.mark.parametrize("model", ["Euler3d", "NavierStokes3d"])
@pytest.mark.parametrize("sizes", [[16] * 80,                            # groups of 16 blocks
                                   [1100, 16, 16, 900, 140, 1024, 20]])  # of 1, 3 and the last ones
def test_groups_equal_device_steps(sizes, model):
    s1, q = _make(sizes, model)
    s1.step(2)
    s2, _ = _make(sizes, model)
    host = [x.copy() for x in q]
    s2.solve_host([h.ctypes.data for h in host], 2)
    for b in range(len(sizes)):
        assert np.array_equal(host[b], s1.get_q(b)), b
    assert s1.time_dt() == s2.time_dt() and s1.residual() == s2.residual()


@pytest.mark.gpu
def test_small_blocks_are_not_slower_than_whole_steps():
    """80 blocks of 16^3: 1.3 times the time of whole steps between whole copies at most (block by
    block the marching sweeps took more than twice)."""
    import torch
    t = {}
    for on in (True, False):
        s, q = _make([16] * 80, "Euler3d")
        s.set_host_pipeline(on)
        host = [torch.from_numpy(x.copy()).pin_memory() for x in q]
        ptrs = [h.data_ptr() for h in host]
        s.solve_host(ptrs, 2)
        best = []
        for _ in range(5):
            t0 = time.perf_counter()
            s.solve_host(ptrs, 2)
            best.append(time.perf_counter() - t0)
        t[on] = min(best)
        s.close()
    assert t[True] <= 1.3 * t[False], t
