"""Energies of the FP32-convolution form after time steps.  Its real grids are
FP64 for the energies whichever evaluation came last: the merged one of a time
step, which keeps float grids, gives the terms of a split evaluation of the same
state (he4_field).  The two form the same FP32 spectra from sources that differ
in FP64 rounding only, 1e-16, so a source rounds to another float at about one
point in 1e8 and a term moves by less than 1e-12; 1e-10 is asked.  (With
gradients and alpha_s products rounded to float ealphas moves by 1e-9 to 1e-8.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# register stencils (64), streamed stencils (128 along x), 13 points, the core without alpha_s
@pytest.mark.parametrize("shape,npd,core", [((64, 64, 64), 7, "OTC"), ((128, 32, 64), 7, "OTC"),
                                            ((64, 32, 64), 13, "OTC"), ((64, 32, 32), 7, "OT")])
def test_energies_after_steps(pkg, shape, npd, core):
    w, abi = pkg.workloads, pkg.abi
    nx, ny, nz = shape
    p = w.make_params(nx, 0.5, 400, ny=ny, nz=nz, npd=npd,
                      core4=abi.HE4_CORE_OTC if core == "OTC" else abi.HE4_CORE_OT)
    p.precision = abi.HE4_PREC_FP32CONV
    psi = w.droplet_psi(p, 60) * np.exp(0.2j)
    r, v = w.particles(400, 6, 150.0, center=(0.0, 0.0, 1.0))
    with pkg.He4Step(p) as g:
        g.set_state(psi, r, v)
        g.run(7, w.deltat_fs(1.0))
        merged = g.energy()
        pot4 = g.get_field("pot4")
        g.field()
        split = g.energy()
        for k in merged:
            assert abs(merged[k] - split[k]) <= 1e-10 * abs(split[k]), (k, merged[k], split[k])
        # the energies leave the evaluation they follow as it was
        g.set_state(psi, r, v)
        g.run(7, w.deltat_fs(1.0))
        assert np.array_equal(pot4, g.get_field("pot4"))
        a = g.get_state()
        g.set_state(psi, r, v)
        g.run(4, w.deltat_fs(1.0))
        g.energy()
        g.run(3, w.deltat_fs(1.0))
        for x, y in zip(a, g.get_state()):
            assert np.array_equal(x, y)
