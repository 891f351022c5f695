"""Device memory of a handle, and the fields whose room a time step borrows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(128, "HE4_PREC_FP64"), (128, "HE4_PREC_FP32CONV")])
def test_memory_per_handle(pkg, n, precision):
    """The arrays that the state, its histories, the named fields and one
    branch of transforms need, and no more than 3 % beside them."""
    import torch
    w = pkg.workloads
    p = w.make_params(n, 0.5, 1000)
    p.precision = getattr(pkg.abi, precision)
    fp32 = precision == "HE4_PREC_FP32CONV"
    pkg.He4Step(p).close()  # modules, contexts
    torch.cuda.synchronize()
    free0 = torch.cuda.mem_get_info()[0]
    hs = [pkg.He4Step(p) for _ in range(4)]
    used = (free0 - torch.cuda.mem_get_info()[0]) / len(hs)
    N, H = n ** 3, (n // 2 + 1) * n * n
    # psi and histories 9, real fields 26 (3 with the room of a spectrum), counts,
    # spectra 6, kernels 5; the FP32 form's kernels 4 and float grids 9; each array in
    # the allocator's units of 2 MiB
    arrays = 9 * [16 * N] + 23 * [8 * N] + 3 * [16 * H] + [4 * N] + 6 * [16 * H] + 5 * [8 * H]
    if fp32:
        arrays += 4 * [4 * H] + 9 * [4 * N]
    need = sum(-(-a // (1 << 21)) << 21 for a in arrays)
    for h in hs:
        h.close()
    assert used <= 1.03 * need, (used / 1e6, need / 1e6)


@pytest.mark.parametrize("core,icon,n", [("OTC", 8, 48), ("OT", 8, 40), ("OTC", 13, 45)])
def test_named_fields_after_steps(pkg, core, icon, n):
    """Every named field after time steps is that of he4_field on the same state, in
    whatever order they are asked for: the same bits, but for pot4, which the
    merged evaluation of a step sums in another order."""
    w, abi = pkg.workloads, pkg.abi
    p = w.make_params(n, 0.6, 300, core4=abi.HE4_CORE_OTC if core == "OTC" else abi.HE4_CORE_OT)
    p.icon = icon
    psi = w.droplet_psi(p, 80) * np.exp(0.2j)
    r, v = w.particles(300, 8, 120.0)
    names = ["fx", "delj4", "corr", "penalty", "ualphas", "falfs", "uimp", "fz", "pot4"]
    with pkg.He4Step(p) as g:
        for order in (names, names[::-1]):
            g.set_state(psi, r, v)
            g.run(6, w.deltat_fs(1.0))
            got = {k: g.get_field(k) for k in order}
            g.field()
            for k in order:
                want = g.get_field(k)
                if k == "pot4":
                    assert np.max(np.abs(got[k] - want)) <= 1e-11 * np.max(np.abs(want))
                else:
                    assert np.array_equal(got[k], want), k
