"""The ghost build and half list where their launches change: one CTA and
several per cluster, boxes that need two swap passes in some dimensions and one
in others, and the sizes on both sides of the limit above which each pass is a
launch of its own.  Ghosts, their order and the list as a set are bit-exact
with the oracle's."""
import numpy as np
import pytest

from mapp_b200 import fixtures as fx
from tests.test_gpu_parity import check_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,keep", [((1, 1, 1), 3), ((2, 5, 3), None), ((6, 6, 1), 141), ((8, 8, 8), 2047),
                                        ((8, 8, 9), 2049), ((16, 16, 17), 17001), ((22, 22, 22), 39999),
                                        ((22, 22, 22), 40001)])
def test_ghosts_and_list(tmp_path, shape, keep):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb
    from oracle.restated import Oracle

    cfg = fx.make_dmd_cell(*shape, sigma=0.03, seed=17, nt=1)
    if keep:
        pick = np.sort(np.random.default_rng(keep).permutation(cfg.natms)[:keep])
        cfg.s, cfg.alpha, cfg.c = cfg.s[pick], cfg.alpha[pick], cfg.c[pick]
    w = fx.write_workload(str(tmp_path), "dmd", cfg=cfg, style="DMD_I")
    check_state(mb.system_from_workload(w), Oracle(w))
