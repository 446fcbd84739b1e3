"""GPU tests of the RWKV-4 time scan where it is cut: several segments, several CTAs of a cluster and several steps of
the cluster, with start flags and lengths on and next to the cuts, against the CPU oracle."""
import numpy as np
import pytest
import torch

import oracle
from test_gpu_wkv4 import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T", [127, 129, 256, 513, 600])
def test_segments_ctas_and_cluster_steps(T, dtype):
    d = oracle.make_wkv4_inputs(4, T, 40, seed=70 + T, default_state=False)      # 40 channels: a ragged second group
    ns = np.zeros((4, T), dtype=bool)
    ns[0, [0, 16, 31, 128 % T, T - 1]] = True
    ns[1, [127 % T, (T // 2) & ~15]] = True
    ns[2] = np.random.default_rng(T).random(T) < 0.02
    d["new_starts"] = ns
    d["length"] = np.asarray([T, (T // 2) & ~15, max(T - 17, 1), 128 % T], dtype=np.uint32)
    check(d, dtype)
