"""The Sz correlators on a device with little room left.

``measure_sz`` takes the environments of many sites through the chain together; where the
device has no room for them it takes fewer, down to one at a time.  A 26-site chain with
bonds up to 1800 takes about 130 MB that way and 420 MB together; with 200 MB left it has
to give what it gave with the device empty.  In a process of its own: a pool that an
earlier context has grown would serve it.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
import numpy as np, torch, tt_b200
ctx, fill = tt_b200.Context(0), []
psi = tt_b200.QMPS.load(sys.argv[1] + ".ttmps")
ctx.sync()
while (more := (torch.cuda.mem_get_info()[0] - (200 << 20)) >> 21) > 1:
    fill.append(torch.empty(min(more, 1 << 13) << 21, dtype=torch.uint8, device="cuda"))
np.savez(sys.argv[1] + ".npz", *psi.measure_sz())
del psi
ctx.close()
"""


def test_with_200_megabytes_left(tmp_path):
    import tt_b200
    L, fn = 26, str(tmp_path / "psi")
    h = np.random.default_rng(1).uniform(-1.0, 1.0, L)
    ctx = tt_b200.Context(0)
    try:
        psi = tt_b200.QMPS(L, [i % 2 for i in range(L)])
        H = tt_b200.QMPO(L, list(h))
        tt_b200.QDMRG(psi, H).run(4, [64, 256, 1024, 2048], [1e-30], [2])
        sz, szsz = psi.measure_sz()
        psi.save(fn)
        del psi, H
    finally:
        ctx.close()
    path = os.pathsep.join([os.path.join(ROOT, "tensor-tools_b200"), os.environ.get("PYTHONPATH", "")])
    out = subprocess.run([sys.executable, "-c", CHILD, fn], env={**os.environ, "PYTHONPATH": path}, timeout=300,
                         stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert out.returncode == 0, out.stdout[-2000:]
    with np.load(fn + ".npz") as got:
        assert np.abs(got["arr_0"] - sz).max() <= 1e-13 and np.abs(got["arr_1"] - szsz).max() <= 1e-13
