"""The plain path's FFT passes over transform lengths: single-stage and odd lengths, every
radix, the edges of the shared-memory table form (512 / 540), odd row counts, and the longest
transform of each direction.  Round-off of two FFTs of up to 2^13 points is a few 1e-15 of the
field; the bound is the 1e-12 of the other potential tests."""
import numpy as np
import pytest

import diskgpu as D
import oracle as O
from helpers import rel_err


@pytest.mark.gpu
@pytest.mark.parametrize("Nu,Nphi", [(2, 2), (3, 5), (8, 4), (27, 45), (25, 16), (15, 128), (120, 96), (512, 9),
                                     (540, 512), (9, 540), (1000, 30), (4096, 6), (6, 8192)])
def test_potential_over_lengths(Nu, Nphi):
    r = np.random.RandomState(Nu * 8209 + Nphi)
    Sig = r.uniform(0.1, 1.0, (Nu, Nphi))
    got = D.KalnajsSolver(Nu, Nphi, eps=0.01).potential(Sig)
    want = O.Kalnajs(Nu, Nphi, eps=0.01).potential(Sig)
    assert rel_err(got, want) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("Nu,Nphi", [(64, 64), (128, 256), (256, 128), (384, 512), (512, 384), (768, 64), (64, 768),
                                     (1024, 128), (128, 1024), (2048, 64), (64, 2048), (150, 256), (6, 128)])
def test_potential_over_compile_time_lengths(Nu, Nphi):
    r = np.random.RandomState(Nu * 8209 + Nphi)
    Sig = r.uniform(0.1, 1.0, (Nu, Nphi))
    got = D.KalnajsSolver(Nu, Nphi, eps=0.01).potential(Sig)
    want = O.Kalnajs(Nu, Nphi, eps=0.01).potential(Sig)
    assert rel_err(got, want) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("Nu,Nphi", [(384, 4096), (4096, 384), (512, 2560), (2560, 512), (640, 2048), (2048, 640),
                                     (768, 1536), (1536, 768), (1280, 1024), (1024, 1280), (3072, 384), (384, 3072),
                                     (256, 8192), (1152, 1152), (1920, 640)])
def test_mixed_potential_over_lengths(Nu, Nphi):
    """FP32 transforms (grids above 2^20 zones) against the FP64 ones: two real transforms there
    and back, some 25 levels of butterflies of 6e-8 each adding up in quadrature, stay below
    1e-6 of the field."""
    r = np.random.RandomState(Nu * 8209 + Nphi)
    Sig = r.uniform(0.1, 1.0, (Nu, Nphi))
    want = D.KalnajsSolver(Nu, Nphi, eps=0.01).potential(Sig)
    with D.Disk(Nu, Nphi, eps=0.01, precision="mixed") as d:
        got = d.potential(Sig)
    assert rel_err(got, want) < 1e-6
