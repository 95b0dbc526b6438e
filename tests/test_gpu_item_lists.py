"""The item list of the pair counts and the virial, which is the force pass's own where no space goes by columns: it
takes no device memory of its own there."""
import numpy as np
import pytest
import torch

import mechanica_b200 as m
from mechanica_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _bytes(cubic):
    """Device bytes of an engine over 120 x 100 x 100 cells (some 15.6 million items' words in a list)."""
    cells = (120, 100, 100)
    rng = np.random.default_rng(0)
    dim = [float(c) for c in cells] if cubic else [float(c) * (1 + 0.01 * k) for k, c in enumerate(cells)]
    n = 1000
    x = rng.uniform(0, 1, size=(n, 3)) * dim
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    u = W.build_gpu(dict(dim=dim, cells=list(cells), cutoff=1.0, dt=0.01, bc=("periodic",) * 3, types=[(1.0, 0.1, m.Newtonian)],
                         pots=[("dpd", (25.0, 4.5, 3.0, 1.0, 0), 0, 0)], forces=[], x=x, v=np.zeros((n, 3), np.float32),
                         t=np.zeros(n, dtype=np.int32)))
    u.force()
    assert u.candidate_pairs() >= 0
    used = free - torch.cuda.mem_get_info()[0]
    u.close()
    return used


def test_one_list_where_one_is_enough():
    _bytes(True)  # loads the kernels
    columns, cells = _bytes(True), _bytes(False)
    # by columns: one list of cells' items (16 bytes each) and one of columns; by cells: one list of cells' items and its
    # order; a second list would be 1.2 million times 16 bytes more
    assert cells - columns <= 12 << 20
