"""EAM / FS pair passes at the sizes where a warp's stretch of pairs can go
wrong: few atoms, atom counts and pair counts that fill no warp or block, atoms
with very different neighbour counts (a crystal with atoms taken out), one and
two species.  Against the oracle, forces within 1e-10 of the largest one,
energies and virial within 1e-10 relative (FP64 sums in another order: 1e-13)."""
import numpy as np
import pytest

from mapp_b200 import fixtures as fx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,nt,fmt,n,keep", [
    ("eam", 1, "SetFL", 2, 1), ("eam", 1, "SetFL", 2, 3), ("eam", 1, "SetFL", 3, 33), ("eam", 2, "FS", 3, 64),
    ("eam", 2, "FS", 4, 255), ("eam", 1, "SetFL", 6, 769), ("fs", 1, None, 3, 107), ("fs", 2, None, 4, 251),
])
def test_pair_passes_on_ragged_systems(tmp_path, kind, nt, fmt, n, keep):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb
    from oracle.restated import Oracle

    kw = dict(fmt=fmt) if fmt else {}
    w = fx.write_workload(str(tmp_path), kind, n=n, nt=nt, sigma=0.05, seed=3 + keep, **kw)
    cfg = w["cfg"]
    pick = np.sort(np.random.default_rng(keep).permutation(cfg.natms)[:keep])
    cfg.s, cfg.type = cfg.s[pick], cfg.type[pick]
    fx.write_cfg(w["cfg_path"], cfg)
    s, o = mb.system_from_workload(w), Oracle(w)
    assert s.counts()["npairs"] == o.counts()["npairs"]
    f, en = s.force_calc(1)
    fo, eno = o.force(1)
    assert np.max(np.abs(f - fo)) <= 1e-10 * np.max(np.abs(fo))
    assert np.max(np.abs(en - eno)) <= 1e-10 * np.max(np.abs(eno))
    assert abs(s.energy_calc() - o.energy()) <= 1e-10 * abs(o.energy())
