"""mg_last_time("list"): the last list build that went through, also after one
that failed on the way (a skin that needs more ghost swaps than an image chain
holds), and again after the next good one."""
import pytest

from mapp_b200 import fixtures as fx

pytestmark = pytest.mark.gpu


def test_list_time_after_a_failed_build(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb

    w = fx.write_workload(str(tmp_path), "dmd", cfg=fx.make_dmd_cell(1, 1, 1, seed=2), style="DMD_I")
    s = mb.system_from_workload(w)
    good = s.last_time("list")
    assert 0.0 < good < 1000.0
    for _ in range(2):
        s.set_skin(18.0)
        for _ in range(2):
            with pytest.raises(mb.MGError):
                s.init()
            assert s.last_time("list") == good
        s.set_skin(0.5)
        s.init()
        good = s.last_time("list")
        assert 0.0 < good < 1000.0
