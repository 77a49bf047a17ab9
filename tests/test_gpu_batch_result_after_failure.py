"""mg_batch_cell_result after a relaxation that failed in its list build: the
build had moved the batch's arrays to larger ones (a wider skin makes more
ghosts) before the next cell could not be built, and the result still comes
from arrays that exist -- finite positions of every cell, the forces and the
state of the last relaxation that went through."""
import tempfile

import numpy as np
import pytest

from mapp_b200 import fixtures as fx

pytestmark = pytest.mark.gpu


def test_result_after_a_failed_build():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb

    builder = mb.system_from_workload(fx.write_workload(tempfile.mkdtemp(), "dmd", n=2, style="DMD_I"))
    cells = [fx.make_dmd_cell(4, 4, 4, sigma=0.03, seed=1), fx.make_dmd_cell(1, 1, 1, sigma=0.0, seed=2)]
    B = mb.Batch(builder)
    for c in cells:
        B.add_cell(c)
    B.set_params(5, 5, 1e-5, 1e-8, 60)
    B.relax()
    before = [B.cell_result(k) for k in range(2)]
    # 18 A of skin: the first cell's ghosts grow from some 1500 to 15000, the one
    # of four sites needs images 6 boxes away in every dimension, more swaps than
    # a ghost's image chain holds
    builder.set_skin(18.0)
    with pytest.raises(mb.MGError):
        B.relax()
    for (xb, fb, rb), c, k in zip(before, cells, range(2)):
        x, f, r = B.cell_result(k)
        edges = np.diag(c.H())
        assert np.all(np.isfinite(x)) and np.all(x[:, :3] >= -1.0) and np.all(x[:, :3] <= edges + 1.0)
        assert np.array_equal(f, fb) and r["energy"] == rb["energy"] and r["iterations"] == rb["iterations"]
    builder.set_skin(0.5)
    B.relax()
    for k in range(2):
        assert abs(B.cell_result(k)[2]["energy"] - before[k][2]["energy"]) <= 1e-9 * abs(before[k][2]["energy"])
    B.close()
