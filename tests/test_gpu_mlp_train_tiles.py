"""The training step at one tile, an odd number of tiles and more tiles than
SMs: the gradient of every weight matrix and bias against the CPU FP64
reference (relative 1e-2 a block, the BF16 products' rounding; 0.9999 cosine),
and two training runs of the same seed give the same weights bit for bit."""
import numpy as np
import pytest

from mapp_b200 import fixtures as fx
from tests import mlp_reference as ref

pytestmark = pytest.mark.gpu

BOX = (1.8, 5.0, 0.05, 0.20)
BLOCKS = {"W1": (0, 4 * 64), "b1": (1024, 1088), "W2": (1088, 5184), "b2": (5184, 5248), "W3": (5248, 9344),
          "b3": (9344, 9408), "W4": (9408, 9920)}


def _system(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb

    return mb.system_from_workload(fx.write_workload(str(tmp_path / "w"), "dmd", n=3, sigma=0.03, style="DMD_I"))


@pytest.mark.parametrize("n,kind", [(64, 1), (64 * 3, 2), (64 * 201, 2)])
def test_gradient_blocks(tmp_path, n, kind):
    s = _system(tmp_path)
    s.mlp_set_activation(kind)
    s.mlp_init(*BOX, seed=4)
    rng = np.random.default_rng(n)
    x = np.stack([rng.uniform(1.8, 5.0, n), rng.uniform(0.05, 0.2, n), rng.uniform(0.05, 0.2, n),
                  rng.integers(0, 3, n)], axis=1).astype(np.float32)
    y = rng.normal(0, 1, (n, 6)).astype(np.float32)
    p, scaling = s.mlp_state()
    g, loss = s.mlp_grad(x, y)
    loss_ref, g_ref = ref.loss_and_grad(p, x, y, scaling, BOX, kind)
    assert abs(loss - loss_ref) <= 1e-3 * loss_ref
    for name, (lo, hi) in BLOCKS.items():
        a, b = g[lo:hi].astype(np.float64), g_ref[lo:hi]
        assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b), name
        assert a @ b >= 0.9999 * np.linalg.norm(a) * np.linalg.norm(b), name


@pytest.mark.parametrize("steps", [60, 200])
def test_training_is_reproducible(tmp_path, steps):
    """Also on the legacy default stream and with a larger sample set before."""
    s = _system(tmp_path)
    runs = []
    for k in range(3):
        if k == 2:
            s.mlp_train(nsamples=20000, steps=2, batch=64, seed=1)
            s.set_stream(0)
        s.mlp_init(*BOX, seed=9)
        s.mlp_train(nsamples=5000, steps=steps, batch=640, seed=3)
        runs.append((s.mlp_state()[0], s.mlp_loss_history(steps)))
    for p, h in runs[1:]:
        assert np.array_equal(runs[0][0].view(np.uint32), p.view(np.uint32))
        assert np.array_equal(runs[0][1], h)
