"""energy_calc right after an update_x whose skin test nobody has read: the same
energy as with the test read first, inside the skin and beyond it (the list is
rebuilt), and the system goes on as usual.  Against the oracle, 1e-10 relative."""
import numpy as np
import pytest

from mapp_b200 import fixtures as fx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,kw", [("eam", dict(n=4)), ("fs", dict(n=4, nt=2)), ("dmd", dict(n=4, sigma=0.02, style="DMD_I"))])
@pytest.mark.parametrize("move", [0.05, 0.9])
def test_energy_with_a_pending_skin_test(tmp_path, kind, kw, move):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb
    from oracle.restated import Oracle

    w = fx.write_workload(str(tmp_path), kind, **kw)
    s, o = mb.system_from_workload(w), Oracle(w)
    x = s.get_x()
    rng = np.random.default_rng(5)
    x[:, :3] += rng.uniform(-0.02, 0.02, size=(len(x), 3))
    x[7, 0] += move
    s.update_x(x, report=False)
    e = s.energy_calc()
    o.update_x(x)
    assert abs(e - o.energy()) <= 1e-10 * abs(o.energy())
    assert s.counts()["npairs"] == o.counts()["npairs"]
    f, en = s.force_calc(1)
    fo, eno = o.force(1)
    assert np.max(np.abs(f - fo)) <= 1e-10 * np.max(np.abs(fo))
    assert abs(en[0] - eno[0]) <= 1e-10 * abs(eno[0])
