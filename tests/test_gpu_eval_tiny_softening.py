"""The evaluation where the softening is so small that its square lies below the
packed loops' bound: down to the smallest normal square they take the mass last,
and below it (or without softening) the general kernel skips a particle's own
entry, groups of at most 16 as several copies. Compared with the CPU restatement
at the fast form's tolerance (|da| <= 2e-5 |a| + 1e-6 of the median); counts must
be equal. Heavy particles: m / eps^3 of a particle's own entry overflows."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.0, 1e-20, 1.05e-19, 1.2e-19, 1e-15, 1e-13, 5e-13, 9.0e-13, 9.2e-13])
@pytest.mark.parametrize("group_size", [1, 5, 8, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("form,quad", [(0, True), (1, True), (0, False), (1, False)])
def test_tiny_softening(native, oracle, eps, group_size, form, quad):
    from astro_gb300 import ic
    from test_gpu_parity import acc_close, run_gpu

    L = native.layouts
    flags = L.FLAG_OPEN_DELTA | (L.FLAG_QUADRUPOLE if quad else 0)
    p = native.default_params(L.PRESET_PHYSICAL, lbits=7, form=form, group_size=group_size, softening=eps,
                              far_ratio=0.2 if group_size in (5, 32, 64) else 0.0, flags=flags, force_clamp=3e38)
    pm, vr = ic.plummer(1500, seed=group_size)
    if 0.0 < eps < 9.1e-13:
        pm["mass"] *= 1e6  # 667 each; above the bound a mass below 2^128 eps^3 is asked for
    out = run_gpu(native, p, pm, vr, dt=1e-9, steps=1)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-9, steps=1)
    ok, rel = acc_close(out["acc4"], ref["acc4"])
    assert ok.all(), f"{(~ok).sum()} particles outside tolerance, worst {rel.max():.3e}"
    assert out["interactions"] == ref["interactions"] and out["far_interactions"] == ref["far_interactions"]
