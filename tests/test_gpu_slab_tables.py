"""Slabs of a fluid with a table potential at a density where a slab's engine, which has the whole grid and only its
own particles and ghosts, looks sparser than the undivided box: 13 particles a cell in all, 8 seen from one of
two slabs. Every slab takes the kernel that the undivided box takes, so states agree to the bit, as in
test_gpu_slab.py. Run as a program, the file is one rank of the test."""
import datetime
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [HERE, os.path.dirname(HERE)]

pytestmark = pytest.mark.gpu

K, N = 3, 13 * 16 * 8 * 8


def _build():
    from mechanica_b200 import workloads as W
    scn = W.dpd(n=N, dims=(16.0, 8.0, 8.0), seed=11)
    scn["pots"] = [("morse", (0.2, 5.0, 0.6, 1e-4, 2.0, 1e-3), 0, 0)]
    scn["types"] = [(1.0, 0.7, scn["types"][0][2])]
    scn["dt"] = 1e-4
    return W.build_gpu(scn)


def _rank(out):
    import torch
    import torch.distributed as dist
    rank, world = int(os.environ["RANK"]), int(os.environ["WORLD_SIZE"])
    dist.init_process_group("gloo", rank=rank, world_size=world, timeout=datetime.timedelta(seconds=120))
    try:
        torch.cuda.set_device(0)
        from mechanica_b200 import slab
        u = _build()
        s = slab.Slab(u, rank, world)
        s.steps(K)
        c, xr, v = s.gather()
        if rank == 0:
            np.savez(out, cell=c, xr=xr, v=v)
        u.close()
    finally:
        dist.destroy_process_group()


@pytest.mark.parametrize("world", [2, 3])
def test_slabs_of_a_table_fluid_match_the_undivided_box(tmp_path, world):
    from slab_launch import free_port
    u = _build()
    u.steps(K)
    x, v0, f, c0, xr0 = u.state()
    u.close()
    out, port = str(tmp_path / "slab.npz"), free_port()
    procs = [subprocess.Popen([sys.executable, os.path.abspath(__file__), out],
                              env=dict(os.environ, RANK=str(r), WORLD_SIZE=str(world), LOCAL_RANK=str(r),
                                       MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port)),
                              stdout=subprocess.PIPE, stderr=subprocess.STDOUT) for r in range(world)]
    try:
        for p in procs:
            log, _ = p.communicate(timeout=300)
            assert p.returncode == 0, log.decode(errors="replace")[-2000:]
    finally:
        for p in procs:
            if p.poll() is None:
                p.kill()
                p.wait()
    z = np.load(out)
    assert np.array_equal(z["cell"], c0)
    assert np.array_equal(z["xr"].view(np.uint32), xr0.view(np.uint32))
    assert np.array_equal(z["v"].view(np.uint32), v0.view(np.uint32))


if __name__ == "__main__":
    _rank(sys.argv[1])
