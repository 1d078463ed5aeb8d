"""Groups of one to five particles, whose lists all the warp's lanes split: list
lengths below, at and above the number of parts, both forms. Compared with the
CPU restatement at the fast form's tolerance (|da| <= 2e-5 |a| + 1e-6 of the
median); counts must be equal."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group_size", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n,lbits,bucket", [(1, 2, 0), (2, 21, 0), (5, 1, 8), (31, 3, 1), (34, 3, 40), (65, 2, 0),
                                            (3001, 8, 8)])
@pytest.mark.parametrize("form", [0, 1])
def test_small_groups(native, oracle, group_size, n, lbits, bucket, form):
    from astro_gb300 import ic
    from test_gpu_parity import acc_close, run_gpu

    L = native.layouts
    p = native.default_params(L.PRESET_PHYSICAL, lbits=lbits, form=form, group_size=group_size, softening=0.01,
                              bucket=bucket, far_ratio=0.2 if group_size % 2 else 0.0)
    pm, vr = ic.plummer(n, seed=40 + n)
    out = run_gpu(native, p, pm, vr, dt=1e-3, steps=1)
    ref = oracle.phys_run(p, pm.copy(), vr.copy(), dt=1e-3, steps=1)
    ok, rel = acc_close(out["acc4"], ref["acc4"])
    assert ok.all(), f"{(~ok).sum()} particles outside tolerance, worst {rel.max():.3e}"
    assert out["interactions"] == ref["interactions"] and out["far_interactions"] == ref["far_interactions"]
