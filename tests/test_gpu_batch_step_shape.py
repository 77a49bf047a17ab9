"""The built-in shape of the minimiser's step on both sides of each line, for
both forms and methods: small cells 256 threads, medium ones 512, large ones
1024 with as many CTAs a cell as fit the GPU; and every cell ends where the
same cell relaxed by 256 threads and one CTA does."""
import tempfile

import numpy as np
import pytest

from mapp_b200 import fixtures as fx

pytestmark = pytest.mark.gpu

# cell shapes (4 sites a unit), expected threads and CTAs a cell
CASES = [([(1, 1, 1)], 256, 1), ([(4, 4, 4), (2, 2, 2)], 256, 1), ([(4, 4, 5)], 512, 1), ([(5, 5, 10), (2, 3, 3)], 512, 1),
         ([(5, 5, 11)], 1024, 4), ([(2, 2, 2)] * 36 + [(6, 6, 7)], 1024, 4), ([(2, 2, 2)] * 37 + [(6, 6, 7)], 1024, 2),
         ([(2, 2, 2)] * 74 + [(6, 6, 7)], 1024, 1)]


@pytest.mark.parametrize("form", ["fp64", "fp32"])
@pytest.mark.parametrize("cg", [False, True])
@pytest.mark.parametrize("shapes,threads,ctas", CASES)
def test_built_in_shape(shapes, threads, ctas, form, cg):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb

    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the counts are those of 148 SMs")
    builder = mb.system_from_workload(fx.write_workload(tempfile.mkdtemp(), "dmd", n=2, style="DMD_I"))

    def relax(launch):
        B = mb.Batch(builder)
        for k, sh in enumerate(shapes):
            B.add_cell(fx.make_dmd_cell(*sh, sigma=0.03, seed=k, mean_cA=0.5))
        B.set_params(5, 1, 1e-5, 1e-8, 60)
        B.set_form(mb.MG_FORM_FP32 if form == "fp32" else mb.MG_FORM_FP64)
        if cg:
            B.set_method(mb.MG_MIN_CG)
        if launch:
            B.set_launch(0, 0, *launch)
        st = B.relax()
        out = [B.cell_result(k) for k in range(len(shapes))]
        B.close()
        return st, out

    st, out = relax(None)
    assert (st["lbfgs_threads"], st["lbfgs_cluster"]) == (threads, ctas)
    for (x, f, r), (xr, fr, rr) in zip(out, relax((256, 1))[1]):
        # one iteration along the gradient: sums in another order (FP32: of pair
        # forces rounded to 24 bits; a step length differs by no more than the forces)
        tol = 1e-9 if form == "fp64" else 1e-3
        assert abs(r["energy"] - rr["energy"]) <= (1e-10 if form == "fp64" else 1e-6) * abs(rr["energy"])
        assert np.max(np.abs(x[:, :3] - xr[:, :3])) <= tol
        assert np.all(np.isfinite(f))
