"""The training step's output bias (summed by a warp of its own) against the CPU
FP64 reference, and the padded parameters -- rows 4 to 15 of the first weights,
columns 6 and 7 of the last and their biases -- whose gradient must be zero
exactly, or Adam would move what no input or output uses; they stay zero
through a run.  Tolerance: the BF16 rounding of the layers before the output
(2^-9 relative a product), as for the other blocks 1e-2 of the norm."""
import numpy as np
import pytest

from mapp_b200 import fixtures as fx
from tests import mlp_reference as ref

pytestmark = pytest.mark.gpu

BOX = (1.8, 5.0, 0.05, 0.20)
W1, W4, B4 = slice(0, 1024), slice(9408, 9920), slice(9920, 9928)


def padding(p):
    return np.concatenate([p[W1].reshape(16, 64)[4:].ravel(), p[W4].reshape(64, 8)[:, 6:].ravel(), p[B4][6:]])


@pytest.mark.parametrize("n", [64, 64 * 5, 64 * 150])
def test_output_bias_and_padding(tmp_path, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb

    s = mb.system_from_workload(fx.write_workload(str(tmp_path / "w"), "dmd", n=3, sigma=0.03, style="DMD_I"))
    s.mlp_set_activation(2)
    s.mlp_init(*BOX, seed=4)
    rng = np.random.default_rng(n)
    x = np.stack([rng.uniform(1.8, 5.0, n), rng.uniform(0.05, 0.2, n), rng.uniform(0.05, 0.2, n),
                  rng.integers(0, 3, n)], axis=1).astype(np.float32)
    y = rng.normal(0.5, 1, (n, 6)).astype(np.float32)
    p, scaling = s.mlp_state()
    assert np.all(padding(p) == 0.0)
    g, _ = s.mlp_grad(x, y)
    g_ref = ref.loss_and_grad(p, x, y, scaling, BOX, 2)[1]
    a, b = g[B4][:6].astype(np.float64), g_ref[B4][:6]
    assert np.linalg.norm(a - b) <= 1e-2 * np.linalg.norm(b)
    assert np.all(padding(g) == 0.0)
    s.mlp_train(nsamples=5000, steps=20, batch=640, seed=3)
    assert np.all(padding(s.mlp_state()[0]) == 0.0)
