"""The tuner's choices are kept per form of the gravity: a disk that is told to run the products
where disks run FFTs by default does not take over what was found and said for those."""
import pytest

import diskgpu as D


@pytest.mark.gpu
def test_products_do_not_take_the_fft_disks_tuning(monkeypatch):
    monkeypatch.delenv("DISKGPU_HYDRO32", raising=False)
    monkeypatch.delenv("DISKGPU_STAGES", raising=False)
    with D.Disk(1152, 1024, eps=0.01, precision="mixed") as d:
        d.init_standard()
        assert "FFT" in d.tuning()
    monkeypatch.setenv("DISKGPU_STAGES", "0,0,0,0,0,0")
    with D.Disk(1152, 1024, eps=0.01, precision="mixed") as d:
        d.init_standard()
        info = d.tuning()
    assert "gravity stages fixed 0 0 0 0 0 0" in info and "FFT" not in info and "cached" not in info
