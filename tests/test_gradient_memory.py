"""csp_mlp_gradient keeps at most 64 MB of device memory from call to call, and none once a
handle has been destroyed."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_memory_goes_back(pkg, synth):
    import torch
    torch.cuda.init()
    rng = np.random.default_rng(1)
    p = pkg.mlp_init(1)

    def gradient(n):
        pkg.mlp_gradient(p, rng.random((n, 8), dtype=np.float32), rng.random((n, 5), dtype=np.float32))

    def free():
        return torch.cuda.mem_get_info()[0]

    pkg.Simulation(synth.tiny((12, 12, 16)), dict(h=6.0, tstop=1.0, seed=1)).close()
    gradient(1000)
    pkg.Simulation(synth.tiny((12, 12, 16)), dict(h=6.0, tstop=1.0, seed=1)).close()
    before = free()
    gradient(5_000_000)                                  # 260 MB
    assert before - free() <= 64 << 20
    gradient(200_000)                                    # 10 MB: kept for the next call
    assert before - free() <= 64 << 20
    pkg.Simulation(synth.tiny((12, 12, 16)), dict(h=6.0, tstop=1.0, seed=1)).close()
    assert before - free() <= 4 << 20
