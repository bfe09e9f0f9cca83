"""The autotuner's choice can be written down: what Context.autotune_trace returns, set on another context,
launches the same kernel with the same refill threshold."""
import numpy as np
import pytest
import torch

from rbr_b200 import Context, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("refill", [1, 3, 8])
def test_choice_is_complete(any_hit, refill):
    w = scenes.random_world(400, 1500, False, seed=5)
    rays = scenes.random_test_rays(800_000, seed=3)[:300_001]
    dev = torch.from_numpy(np.frombuffer(rays.tobytes(), np.uint8).copy()).cuda()
    with Context(0) as a, Context(0) as b:
        a.upload(w)
        b.upload(w)
        defaults = {k: b.get_param(k) for k in NAMES}
        a.set_param("trace.refill_min", refill)
        chosen = a.autotune_trace(dev.data_ptr(), len(rays), any_hit)
        assert chosen.pop("us_per_launch") > 0
        for k, v in chosen.items():
            b.set_param(k, v)
        for k in NAMES:
            assert b.get_param(k) == a.get_param(k), k
            assert k in chosen or a.get_param(k) == defaults[k]


NAMES = ["trace.kernel", "trace.blocks_per_sm", "trace.refill_min", "trace.min_blocks", "trace.order", "trace.node_test",
         "trace.stream_io", "trace.l2_persist"]
