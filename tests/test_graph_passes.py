"""The second evaluation of a later pass is replayed: weights overwritten between two passes, and a
generation bumped by another shape, must still give the eager run's samples."""
import pytest
import torch

import cases
from test_gpu_unet import build

pytestmark = pytest.mark.gpu


def test_overwritten_weights_between_passes(cuda):
    import modiff_b200 as m
    c = next(u for u in cases.UNET_CASES if u["name"] == "w4a4_split_b2_s10")
    betas = torch.from_numpy(m.get_beta_schedule()).float()
    seq = cases.unet_sequence(c)[-5:]
    x = cases.unet_noise(c).to(cuda)
    runs = {}
    for use_graph in (False, True):
        qnn = build(c, cuda)
        outs = []
        for k in range(3):
            if k == 2:
                with torch.no_grad():
                    layer = [q for q in qnn.modules() if isinstance(q, m.QuantModule)][7]
                    layer.weight.mul_(1.25)
            qnn.reset_cache()
            xs, _ = m.generalized_steps(x, seq, qnn, betas, eta=0.0, cuda_graph=use_graph)
            outs.append(xs[-1].clone())
        runs[use_graph] = outs
    assert m.device_status() == 0
    for a, b in zip(runs[False], runs[True]):
        assert torch.equal(a, b)
    assert not torch.equal(runs[True][1], runs[True][2])
