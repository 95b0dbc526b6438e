"""The column kernel's forces against 64 bits: no further off than the cell kernel's, whose relative error in this
fluid (DPD at 12.5 a cell, 50 neighbours a particle) is 1.49e-7."""
import numpy as np
import pytest

from mechanica_b200 import workloads as W
from oracle import restatement as R

from golden_util import rel_rms

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [1, 2])
def test_dpd_forces_are_as_exact_as_the_cell_kernels(variant):
    grid = [200, 5, 4]
    scn = W.dpd(n=50000, dims=[float(c) for c in grid], seed=1)
    scn["cells"] = grid
    scn["pots"] = [("dpd", (25.0, 4.5, 3.0, 1.0, 0), 0, 0)]
    u = W.build_gpu(scn)
    u.force_config(variant, 1 << 20)
    u.force()
    x, v, f, c, xr = u.state()
    tasks = u.tasks()
    u.close()
    tasks = tasks[(tasks[:, 0] == 1) | (tasks[:, 0] == 2)]
    f64 = R.nonbond(scn, xr, v, c, tasks, np.array(grid, dtype=np.int32), precision=64)[0]
    assert rel_rms(f, f64) <= 1.49e-7
