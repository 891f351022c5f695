"""he4_energy's convolution energies, summed over k (csrc/fft_mix.cuh
k_mix_zenergy), against the sums over the grid of the fields they stand for:
every z length with a two-step transform, whose CTAs have 48 to 216 threads at work,
few of them a multiple of 32, on x and y axes that leave tiles with a remainder.
Both are sums of a few thousand products in FP64: they agree to 1e-12 of the sum of
the magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [16, 32, 36, 40, 45, 48, 50, 54, 60, 64, 72, 75, 80, 81, 90, 96, 100, 108, 120, 125, 128, 135, 144, 150, 160,
           162, 180, 192, 200, 216, 225, 240, 243, 250, 256]


@pytest.mark.parametrize("nz", LENGTHS)
def test_convolution_energies(pkg, nz):
    w = pkg.workloads
    p = w.make_params(20, 0.6, 200, ny=15, nz=nz)
    psi = w.droplet_psi(p, 40)
    r, v = w.particles(200, 4, 100.0, center=(0.0, 0.0, 1.0))
    with pkg.He4Step(p) as g:
        g.set_state(psi, r, v)
        g.field()
        E = g.energy()
        den, dxyz = g.get_field("den"), 0.6 ** 3
        for name, field, c in (("elj4", "delj4", 0.5), ("eHeX", "uimp", 1.0)):
            terms = c * g.get_field(field) * den * dxyz
            assert abs(E[name] - terms.sum()) <= 1e-12 * np.abs(terms).sum(), (name, E[name], terms.sum())
