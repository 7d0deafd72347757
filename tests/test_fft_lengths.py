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
