"""Memory kept between calls is bounded over all objects (needs a GPU): 256 MiB of scratch over all
states, 256 MiB of training rows over all networks, however many are alive."""
import numpy as np
import pytest

import ruqu_b200 as rq
from ruqu_b200.warmstart import Mlp

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_scratch_of_many_live_states():
    states = [rq.QuantumState(20, k, "f64") for k in range(60)]
    states[0].probability_of_qubit(0)
    before = _free()
    for s in states:                                  # 8 MiB of scratch each
        assert s.probabilities()[0] == 1.0
    assert before - _free() <= 256 * MIB + 16 * MIB
    for s in states:
        assert s.state_vector()[0] == 1.0


def test_training_rows_of_many_networks():
    r = np.random.default_rng(0)
    n = 60000                                         # 115 MiB of rows each
    x = (r.random((n, 325)) < 0.1).astype(np.float32)
    t = r.standard_normal((n, 8)).astype(np.float32)
    nets = [Mlp() for _ in range(5)]
    alone = [net.train(x[:256], t[:256], batch=256, steps=2) for net in nets]
    before = _free()
    losses = [net.train(x, t, batch=256, steps=2) for net in nets]
    assert before - _free() <= 256 * MIB + 16 * MIB
    assert len(set(alone)) == 1 and len(set(losses)) == 1
