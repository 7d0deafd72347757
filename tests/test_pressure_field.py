"""Gamma != 2 in FP64: the pressure that steps hand on, the one that the CFL pass computes from an
uploaded density and the one that a step takes straight after an upload computes by itself are
the same bits, so a run interrupted by an upload of its own state goes on as if it had not been."""
import numpy as np
import pytest

import diskgpu as D

DT = 2e-3


@pytest.mark.gpu
@pytest.mark.parametrize("Nu,Nphi", [(6, 5), (72, 60), (40, 108)])
@pytest.mark.parametrize("path", ["step", "forces", "no_forces", "timestep", "advance", "graph"])
def test_uploaded_state_goes_on_with_the_same_bits(Nu, Nphi, path):
    r = np.random.RandomState(Nu)
    gR, gp = (r.uniform(-0.2, 0.2, (Nu, Nphi)) for _ in "ab")

    def go(d):
        if path == "forces":
            d.step_forces(DT, gR, gp)
        elif path == "no_forces":
            d.step_forces(DT)
        elif path == "timestep":
            d.step(0.5 * d.timestep(0.3))
        elif path == "advance":
            d.advance(0.02)
        elif path == "graph":
            d.run_steps(70)
        else:
            d.step(DT)
        return d.get_state()

    with D.Disk(Nu, Nphi, eps=0.01, amp=0.05, gamma_gas=1.7) as a, D.Disk(Nu, Nphi, eps=0.01, amp=0.05,
                                                                          gamma_gas=1.7) as b:
        a.init_standard()
        if path == "advance":
            state = a.get_state()  # (advance goes by the disk's own time: both start at t = 0)
        else:
            a.step(DT)
            a.step(DT)
            state = a.get_state()
        if path == "graph":
            b.set_state(*state)
            b.capture_graph()
        for again in range(2):  # the second time the pressure is a step's
            b.set_state(*state)
            got = go(b)
            if path == "advance":
                a.set_state(*state)
                a.timestep(0.3)
            want = go(a)
            for x, y in zip(got, want):
                assert np.array_equal(x, y), (path, again)
            state = want
