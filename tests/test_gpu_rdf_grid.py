"""The radial distribution's histogram and gradient over the cell grid (mxg_rdf from 1,024
particles, boxes of at least three reaches) against a dense FP64 evaluation of every pair: the
smallest grid (three cells on an axis), a box longer than the most cells on an axis, particles
outside the box, a third type, one type against itself, and a box too small for the grid."""
import ctypes
import math

import numpy as np
import pytest
import torch

from mechanica_b200._native import check, lib

pytestmark = pytest.mark.gpu

NBINS, DR, SIGMA = 16, 0.1, 0.1  # reach 16 * 0.1 + 4 * 0.1 + 0.01


def _dense(x, t, box, ta, tb, coef):
    """(histogram, gradient of coef . histogram) in FP64, and the number of (pair, bin) terms."""
    L = torch.tensor(box, dtype=torch.float64, device="cuda")
    c = (torch.arange(NBINS, dtype=torch.float64, device="cuda") + 0.5) * DR
    y = x.double().requires_grad_(True)
    a, b = torch.nonzero(t == ta).ravel(), torch.nonzero(t == tb).ravel()
    d = y[a][:, None] - y[b][None]
    d = d - L * torch.round(d.detach() / L)
    r2 = (d * d).sum(2)
    keep = (a[:, None] != b[None]) & (r2.detach() < (NBINS * DR + 4 * SIGMA) ** 2)
    u = (r2[keep].sqrt()[:, None] - c) / SIGMA
    near = u.detach().abs() <= 4
    k = torch.where(near, torch.exp(-0.5 * u * u) - math.exp(-8.0), torch.zeros_like(u)) / (math.sqrt(2 * math.pi) * SIGMA)
    hist = k.sum(0)
    grad, = torch.autograd.grad((hist * coef).sum(), y)
    return hist.detach(), grad, int(near.sum())


@pytest.mark.parametrize("n,box,ta,tb", [(1024, (6.1, 9.3, 7.0), 0, 1), (1531, (6.04, 6.04, 70.0), 1, 0),
                                         (2049, (8.5, 7.7, 12.2), 1, 1), (1100, (5.9, 8.0, 8.0), 0, 1)])
def test_grid_matches_every_pair(n, box, ta, tb):
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.4, 1.4, size=(n, 3)) * np.asarray(box)  # some particles outside the box
    t = torch.tensor(rng.integers(0, 3, size=n).astype(np.int32))
    x4 = torch.tensor(np.c_[x, np.zeros(n)], dtype=torch.float32)
    x4[:, 3] = t.view(torch.float32)
    x4 = x4.cuda()
    coef = torch.tensor(rng.normal(size=NBINS), device="cuda")
    hist = torch.zeros(NBINS, dtype=torch.int64, device="cuda")
    grad = torch.full((n, 4), float("nan"), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    p = [ctypes.c_void_p(q.data_ptr()) for q in (x4, hist, grad)]
    check(lib().mxg_rdf(p[0], n, (ctypes.c_double * 3)(*box), ta, tb, NBINS, DR, SIGMA, p[1],
                        ctypes.cast(coef.data_ptr(), ctypes.POINTER(ctypes.c_double)), p[2], None), "rdf")
    torch.cuda.synchronize()
    h64, g64, terms = _dense(x4[:, :3], t.cuda(), box, ta, tb, coef)
    # each term is rounded to 2^-32 once; the FP64 arithmetic is far below that
    assert (hist.double() / 2.0 ** 32 - h64).abs().max().item() <= terms * 2.0 ** -32
    # FP32 storage of an FP64 sum
    assert (grad[:, :3].double() - g64).abs().max().item() <= 1e-6 * g64.abs().max().item()
    assert not grad[:, 3].any() and not grad[t.cuda() == 2, :3].any()
