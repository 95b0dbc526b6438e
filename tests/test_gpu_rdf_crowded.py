"""The radial distribution of particles crowded into one cell of the grid: the values against an FP64 evaluation of
every pair, and the time against the same particles spread over the box, where each meets far fewer partners:
the cell's particles have as many pairs as the all-pairs kernels test, and the grid must not add to that."""
import ctypes
import math

import numpy as np
import pytest
import torch

from mechanica_b200._native import check, lib

pytestmark = pytest.mark.gpu

NBINS, DR, SIGMA = 64, 2.5 / 64, 2.5 / 64


def _rdf(x4, box, hist, coef, grad, scratch):
    p = [ctypes.c_void_p(q.data_ptr()) for q in (x4, hist, coef, grad, scratch)]
    check(lib().mxg_rdf_in(p[0], len(x4), (ctypes.c_double * 3)(*box), 0, 1, NBINS, DR, SIGMA, p[1], p[2], p[3], p[4],
                           scratch.numel(), None), "rdf")


def _scratch(n, box):
    need = ctypes.c_size_t()
    check(lib().mxg_rdf_scratch(n, (ctypes.c_double * 3)(*box), NBINS, DR, SIGMA, ctypes.byref(need)), "rdf")
    return torch.empty(need.value, dtype=torch.uint8, device="cuda")


def test_a_crowded_cell():
    n, L = 8192, 320.0  # 32 cells of 10: all particles in one
    rng = np.random.default_rng(1)
    x4 = torch.zeros((n, 4), dtype=torch.float32)
    x4[:, :3] = torch.tensor(rng.uniform(101, 109, size=(n, 3)))
    x4[:, 3] = torch.tensor((np.arange(n) % 2).astype(np.int32)).view(torch.float32)
    x4 = x4.cuda()
    coef = torch.tensor(rng.normal(size=NBINS), device="cuda")
    hist = torch.zeros(NBINS, dtype=torch.int64, device="cuda")
    grad = torch.zeros((n, 4), device="cuda")
    torch.cuda.synchronize()
    _rdf(x4, [L] * 3, hist, coef, grad, _scratch(n, [L] * 3))
    torch.cuda.synchronize()
    y = x4[:, :3].double()
    c = (torch.arange(NBINS, dtype=torch.float64, device="cuda") + 0.5) * DR
    a, b = y[0::2], y[1::2]
    want = torch.zeros(NBINS, dtype=torch.float64, device="cuda")
    g = torch.zeros_like(a)
    terms = 0
    for k in range(0, len(a), 64):
        d = a[k:k + 64, None] - b[None]
        r = d.norm(dim=2)
        u = (r[..., None] - c) / SIGMA
        near = (u.abs() <= 4) & (r < NBINS * DR + 4 * SIGMA)[..., None]
        e = torch.where(near, torch.exp(-0.5 * u * u), torch.zeros_like(u))
        want += ((e - math.exp(-8.0) * near) / (math.sqrt(2 * math.pi) * SIGMA)).sum((0, 1))
        s = -(e * u * coef).sum(2) / (math.sqrt(2 * math.pi) * SIGMA * SIGMA)
        g[k:k + 64] = ((s / r)[..., None] * d).sum(1)
        terms += int(near.sum())
    assert (hist.double() / 2.0 ** 32 - want).abs().max().item() <= terms * 2.0 ** -32 + 1e-9 * want.abs().max().item()
    assert (grad[0::2, :3].double() - g).abs().max().item() <= 1e-6 * g.abs().max().item()


def test_the_grid_adds_little_time_to_a_crowded_cell():
    """16,384 particles in one cell against the all-pairs kernels on the same particles in a box too small for the
    grid (two reaches wide and a little more): no more than 1.5 times their time."""
    n = 16384
    rng = np.random.default_rng(2)
    x = rng.uniform(0, 8, size=(n, 3))
    ms = {}
    for name, L in (("grid", 320.0), ("all", 8.1)):
        x4 = torch.zeros((n, 4), dtype=torch.float32)
        x4[:, :3] = torch.tensor(x + (101 if name == "grid" else 0))
        x4[:, 3] = torch.tensor((np.arange(n) % 2).astype(np.int32)).view(torch.float32)
        x4 = x4.cuda()
        coef = torch.ones(NBINS, dtype=torch.float64, device="cuda")
        hist = torch.zeros(NBINS, dtype=torch.int64, device="cuda")
        grad = torch.zeros((n, 4), device="cuda")
        scratch, t = _scratch(n, [L] * 3), []
        for _ in range(7):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda.synchronize()
            ev[0].record(torch.cuda.default_stream())
            _rdf(x4, [L] * 3, hist, coef, grad, scratch)
            ev[1].record(torch.cuda.default_stream())
            torch.cuda.synchronize()
            t.append(ev[0].elapsed_time(ev[1]))
        ms[name] = sorted(t)[3]
    assert ms["grid"] <= 1.5 * ms["all"]
