"""A particle at the origin of the coordinates under a tiny softening: what the
staged lists are padded with must not meet it at distance zero, where a
quadrupole's 1 / r^5 is infinite. Compared with the CPU restatement at the fast
form's tolerance (|da| <= 2e-5 |a| + 1e-6 of the median)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [1e-12, 1e-11, 1e-10, 1e-9, 1e-8, 3e-8, 1e-7])
@pytest.mark.parametrize("group_size", [8, 16, 32, 64])
@pytest.mark.parametrize("form", [0, 1])
def test_particle_at_the_origin(native, oracle, eps, group_size, form):
    from astro_gb300 import ic
    from test_gpu_parity import acc_close, run_gpu

    L = native.layouts
    flags = L.FLAG_QUADRUPOLE | L.FLAG_OPEN_DELTA
    p = native.default_params(L.PRESET_PHYSICAL, lbits=7, form=form, group_size=group_size, softening=eps,
                              far_ratio=0.2 if group_size == 16 else 0.0, flags=flags)
    pm, vr = ic.plummer(2500, seed=21)
    pm["position"][0] = 0.0
    out = run_gpu(native, p, pm, vr, dt=1e-3, steps=1)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=1)
    assert np.abs(ref["acc4"]).max() < p.force_clamp
    ok, rel = acc_close(out["acc4"], ref["acc4"])
    assert ok.all(), f"{(~ok).sum()} particles outside tolerance, worst {rel.max():.3e}"
    assert out["interactions"] == ref["interactions"]
