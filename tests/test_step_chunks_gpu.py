"""However a run is cut into calls (graphs of 16 and 8 steps, the rest kernel
by kernel), it is the same run: every count around the graphs' lengths against
single steps, bit for bit, with averages."""
import numpy as np
import pytest

from test_parity_gpu import AVG_FIELDS, BASIC, jet_cfg

pytestmark = pytest.mark.gpu


def test_every_way_to_cut_a_run(pflbm):
    c = jet_cfg(pflbm, 19, nx=24, ny=24, nz=30, diam=6, noise=1)
    c.flags = pflbm.FLAG_TIME_AVERAGE | pflbm.FLAG_REYNOLDS_MOMENTS
    counts = (1, 7, 8, 9, 15, 16, 17, 23, 24, 25, 31, 33, 40)
    with pflbm.Simulation(c) as a, pflbm.Simulation(c) as b:
        for n in counts:
            a.step(n)
            for _ in range(n):
                b.step(1)
            assert a.current_step == b.current_step
            for f in BASIC + AVG_FIELDS:
                assert np.array_equal(a.get_field(f), b.get_field(f)), (n, f)
