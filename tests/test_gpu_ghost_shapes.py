"""The ghost build on thin boxes, where several CTAs of the cluster read, in one
swap pass, ghosts that others made in the pass before: slabs and rods of one
or two cells across, in every direction, with ghost arrays that have to grow,
and boxes on both sides of the line (by owned and ghost sites) above which each
pass is a launch of its own.  Ghosts, their order and the list as a set are
bit-exact with the oracle's."""
import numpy as np
import pytest

from mapp_b200 import fixtures as fx
from tests.test_gpu_parity import check_state

pytestmark = pytest.mark.gpu

CUT = 5.0 + 1.224744871391589 / np.sqrt(20.0) + 0.5  # table, furthest of three nodes at the lowest alpha, skin
LINE = 75000.0


def total(shape, natms, a=3.58):
    """Owned and ghost sites by the edges alone, as the dispatch counts them."""
    return natms * float(np.prod([1.0 + 2.0 * CUT / (a * k) for k in shape]))


# shape, sites kept (None: all), below the line
CASES = [((1, 26, 26), None, True), ((26, 2, 26), 2601, True), ((2, 40, 40), None, True), ((1, 1, 700), None, True),
         ((700, 1, 2), None, True), ((1, 9, 1), 33, True), ((1, 1, 1040), None, True), ((1, 1, 1070), None, False),
         ((1, 1060, 1), 4180, True), ((23, 23, 23), None, True), ((24, 24, 24), 51600, False)]


@pytest.mark.parametrize("shape,keep,below", CASES)
def test_the_line(shape, keep, below):
    assert (total(shape, keep or 4 * int(np.prod(shape))) <= LINE) == below


@pytest.mark.parametrize("shape,keep,below", CASES)
def test_thin_boxes(tmp_path, shape, keep, below):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb
    from oracle.restated import Oracle

    cfg = fx.make_dmd_cell(*shape, sigma=0.03, seed=23, nt=1)
    if keep:
        pick = np.sort(np.random.default_rng(keep).permutation(cfg.natms)[:keep])
        cfg.s, cfg.alpha, cfg.c = cfg.s[pick], cfg.alpha[pick], cfg.c[pick]
    w = fx.write_workload(str(tmp_path), "dmd", cfg=cfg, style="DMD_I")
    s = mb.system_from_workload(w)
    check_state(s, Oracle(w))
    if shape in ((1, 1, 700), (1, 1, 1070)):  # arrays start at four times the owned sites and 1024
        assert s.counts()["nph"] > 3 * cfg.natms + 1024
