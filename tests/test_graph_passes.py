"""The second evaluation of a later pass is replayed: weights overwritten between two passes, and
passes at another batch size in between (dynamic and static scales, and PLMS, whose second evaluation
belongs to its first step), must still give the eager run's samples."""
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


def _model(kind, cuda):
    import modiff_b200 as m
    if kind == "plms":
        torch.manual_seed(0)
        net = m.UNetModel(**cases.LDM_CONFIG).eval()
        m.rerandomize_zero_tensors(net, seed=1234)
        wq, aq = cases.quant_params(cases.LDM_CASES[0])
    else:
        c = next(u for u in cases.UNET_CASES if u["name"] == ("w8a8_b2_s10" if kind == "static" else "w4a4_split_b2_s10"))
        torch.manual_seed(0)
        net = m.Model(m.make_config(split_shortcut=c["split"])).eval()
        wq, aq = cases.quant_params(c)
    aq = dict(aq, dynamic=kind != "static")
    qnn = m.QuantModel(net, wq, aq, sm_abit=8, modulate=True).to(cuda).eval()
    qnn.set_quant_state(True, True)
    return qnn


@pytest.mark.parametrize("kind", ["dynamic", "static", "plms"])
def test_another_batch_size_between_passes(cuda, kind):
    import modiff_b200 as m
    betas = torch.from_numpy(m.get_beta_schedule()).float()
    seq = cases.unet_sequence(cases.UNET_CASES[-1])[-5:]
    shape = (4, 32, 32) if kind == "plms" else (3, 32, 32)
    runs = {}
    for use_graph in (False, True):
        qnn = _model(kind, cuda)
        g = torch.Generator().manual_seed(6)
        outs = []
        for b in (2, 2, 3, 2, 2):
            x = torch.randn((b,) + shape, generator=g).to(cuda)
            qnn.reset_cache()
            if kind == "plms":
                out, _ = m.PLMSSampler(qnn, **cases.LDM_SCHEDULE).sample(50, b, shape, x_T=x, max_steps=4,
                                                                        cuda_graph=use_graph)
            else:
                xs, _ = m.generalized_steps(x, seq, qnn, betas, eta=0.0, cuda_graph=use_graph)
                out = xs[-1]
            outs.append(out.clone())
        runs[use_graph] = outs
    for k, (a, b) in enumerate(zip(runs[False], runs[True])):
        assert torch.equal(a, b), k
