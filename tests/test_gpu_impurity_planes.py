"""The impurity spectrum that a handle keeps between evaluations (spec[4],
csrc/fft.cu fft_r2c_box).  Its planes outside the particle box hold exact zeros
however long the box stays put, on grids whose pairs of rows straddle two planes
too (odd ny): the split evaluation, which reads every plane, gives a long-used
handle the bits of a fresh one, and the oracle's fields to the tolerances of
test_gpu_impurity_box.py and test_gpu_mixed_fft.py."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / max(np.max(np.abs(b)), 1e-300))


# z with and without two-step kernels (40, 36 | 30: every evaluation is split);
# the two clouds one plane apart put the box's faces on planes of both parities
@pytest.mark.parametrize("shape", [(48, 45, 40), (36, 45, 30), (64, 75, 36)])
@pytest.mark.parametrize("plane", [0, 1])
def test_still_box(pkg, ora, shape, plane):
    w = pkg.workloads
    nx, ny, nz = shape
    h, npar = 0.6, 300
    p = w.make_params(nx, h, npar, ny=ny, nz=nz)
    o = ora.Oracle(p)
    vq = np.ascontiguousarray(o.get_kernel("vq"))
    q = pkg.abi.He4Params.from_buffer_copy(p)
    q.pot_kind = pkg.abi.HE4_POT_TABLE
    q.vq_table = vq.ctypes.data_as(C.POINTER(C.c_double))
    psi = w.droplet_psi(p, 60)
    r, v = w.particles(npar, 3, 0.0, center=(0.3, 0.2, 0.5 + h * plane), width=0.2)
    dt = w.deltat_fs(0.01)  # the particles stay in their cells
    o.set_state(psi, r, v)
    with pkg.He4Step(q) as g:
        g.set_state(psi, r, v)
        g.run(40, dt)
        uimp = g.get_field("uimp")
        assert np.isfinite(uimp).all()
        s = g.get_state()
        with pkg.He4Step(q) as fresh:
            fresh.set_state(*s[:3])
            fresh.field()
            assert np.array_equal(g.get_field("denx"), fresh.get_field("denx"))
            assert np.array_equal(uimp, fresh.get_field("uimp"))
        if nz == 30:
            o.run(40, dt)
            assert rel(g.get_field("pot4"), o.get_field("pot4")) < 1e-10
            assert rel(s[0], o.get_state()[0]) < 1e-10
            o.set_state(psi, r, v)
        g.set_state(psi, r, v)
        Eg = g.energy()
        g.field()
        o.field()
        for name in ("uimp", "pot4"):
            assert rel(g.get_field(name), o.get_field(name)) < 1e-11, name
        Eo = o.energy()
        for k in Eo:
            assert abs(Eg[k] - Eo[k]) <= 1e-10 * max(abs(Eo[k]), 1e-30), (k, Eg[k], Eo[k])
        first = [g.get_field(n) for n in ("uimp", "pot4")]
        for _ in range(60):
            g.field()
        for a, n in zip(first, ("uimp", "pot4")):
            assert np.array_equal(a, g.get_field(n)), n
    o.close()
