"""he4_run beyond the 4096 steps whose results it buffers on the device: the
errors, means and state of one call are those of two shorter ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_run_longer_than_its_buffer(pkg):
    w = pkg.workloads
    p = w.make_params(16, 0.8, 32)
    psi = w.droplet_psi(p, 10)
    r, v = w.particles(32, 2, 50.0, center=(0.0, 0.0, 1.0))
    dt = w.deltat_fs(0.05)
    with pkg.He4Step(p) as a, pkg.He4Step(p) as b:
        a.set_state(psi, r, v)
        b.set_state(psi, r, v)
        ea, ma = a.run(4200, dt)
        parts = [b.run(n, dt) for n in (2000, 2200)]
        assert np.array_equal(ea, np.concatenate([x[0] for x in parts]))
        assert np.array_equal(ma, np.concatenate([x[1] for x in parts]))
        assert np.all(ea[4096:, 0] > 0) and len(np.unique(ma[4090:4110, 2])) == 20
        for x, y in zip(a.get_state(), b.get_state()):
            assert np.array_equal(x, y)
