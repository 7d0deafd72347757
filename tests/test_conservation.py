"""Mass and angular momentum of mixed disks just above 2^20 zones, where the gravity turns to
FP32 transforms: 300 steps of the standard disk's seed, in every hydro form, with the bounds of
the 4096^2 disk's test (mass to 1e-11, angular momentum to 1e-8)."""
import pytest

import diskgpu as D


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["packed", "tile", "warp"])
@pytest.mark.parametrize("Nu,Nphi", [(1152, 1152), (1280, 1024), (1536, 768), (1024, 1920)])
def test_mass_drift_above_2_20_zones(Nu, Nphi, form, monkeypatch):
    monkeypatch.setenv("DISKGPU_HYDRO32", form)
    with D.Disk(Nu, Nphi, eps=0.005, amp=1e-3, precision="mixed") as d:
        d.init_standard()
        m0, L0 = d.conserved()
        d.run_steps(300, 0.3)
        m1, L1 = d.conserved()
    assert abs(m1 - m0) <= 1e-11 * m0, (m1 - m0) / m0
    assert abs(L1 - L0) <= 1e-8 * abs(L0), (L1 - L0) / L0
