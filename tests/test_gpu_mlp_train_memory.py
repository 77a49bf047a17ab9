"""Training sets: a small one's buffers stay with the system, a large one's
memory is given back when the run ends (320 MB here; a set may have 2^31 - 1
samples of 40 bytes), and a run on a kept buffer gives the same weights as a
run on a fresh one."""
import numpy as np
import pytest

from mapp_b200 import fixtures as fx

pytestmark = pytest.mark.gpu


def test_a_large_training_set_is_given_back(tmp_path):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import mapp_b200 as mb

    s = mb.system_from_workload(fx.write_workload(str(tmp_path / "w"), "dmd", n=3, sigma=0.03, style="DMD_I"))

    def train(n):
        s.mlp_init(seed=9)
        s.mlp_train(nsamples=n, steps=4, batch=128, seed=3)
        return s.mlp_state()

    first = train(20000)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    train(8_000_000)
    torch.cuda.synchronize()
    after = torch.cuda.mem_get_info()[0]
    assert before - after <= 100 << 20
    again = train(20000)
    assert np.array_equal(first[0], again[0]) and np.array_equal(first[1], again[1])
