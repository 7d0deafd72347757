"""The FP64 hydro step on grids at the edges of its strips (26 columns) and bands: fewer
columns than a strip's halo, one column more or less than whole strips, one to many strips
per CTA, few rows, general Gamma, with caller forces and without.  One step from a rough state
against the oracle: some hundred roundings, of quantities up to a few times the fields' size,
stay under 1e-13 of the field; three more steps under 1e-12."""
import numpy as np
import pytest

import diskgpu as D
import oracle as O
from helpers import rel_err


@pytest.mark.gpu
@pytest.mark.parametrize("Nu,Nphi", [(2, 2), (3, 5), (5, 25), (4, 27), (16, 30), (36, 54), (20, 80), (24, 108),
                                     (9, 135), (64, 160), (40, 810), (1000, 9)])
@pytest.mark.parametrize("gamma,forces", [(2.0, False), (2.0, True), (1.6, True)])
def test_steps_match_oracle(Nu, Nphi, gamma, forces):
    r = np.random.RandomState(Nu * 1009 + Nphi)
    h = D.DiskHydro(Nu, Nphi, gamma=gamma)
    ref = O.Hydro(Nu, Nphi, gamma=gamma)
    h.Sig = r.uniform(0.2, 1.0, (Nu, Nphi))
    h.vR = r.uniform(-0.5, 0.5, (Nu, Nphi))
    h.vp = r.uniform(-0.5, 1.5, (Nu, Nphi))
    ref.set_state(h.Sig, h.vR, h.vp)
    gR, gp = (r.uniform(-1.0, 1.0, (Nu, Nphi)) for _ in "ab") if forces else (None, None)
    for k in range(4):
        dt = ref.timestep(0.1)
        ref.step(dt, gR, gp)
        h.step(dt, gR, gp)
        for got, want in zip((h.Sig, h.vR, h.vp), ref.state()):
            assert rel_err(got, want) < (1e-13 if k == 0 else 1e-12)
    assert abs(h.timestep(0.3) - ref.timestep(0.3)) < 1e-12 * ref.timestep(0.3)


@pytest.mark.gpu
def test_restart_rebuilds_the_pressure_field(tmp_path):
    """Gamma != 2: the pressure a step stored and the one a restart computes from the saved
    density are the same bits, so the runs stay equal."""
    path = str(tmp_path / "s.snap")
    with D.Disk(72, 60, eps=0.01, amp=0.05, gamma_gas=1.7) as a, D.Disk(72, 60, eps=0.01, amp=0.05, gamma_gas=1.7) as b:
        a.init_standard()
        a.run_steps(17)
        a.save(path)
        b.load(path)
        a.run_steps(9)
        b.run_steps(9)
        for x, y in zip(a.get_state(), b.get_state()):
            assert np.array_equal(x, y)
