"""Linear layers that share one input, used at several batch sizes in turn: below the group's limit
one launch writes every layer's output, above it each layer runs its own GEMM.  Every output is
written exactly once in every evaluation, whatever ran at another size before."""
import ctypes as C

import pytest
import torch

CIN, COUT = 768, 640        # to_k / to_v of a 640-channel cross-attention
ROWS = [154, 308, 154, 308]  # two prompts' tokens (grouped: 76 M multiply-adds a layer), four (151 M: not)


def _layers(device="cpu", cin=CIN, couts=(COUT, COUT)):
    import modiff_b200 as m
    torch.manual_seed(3)
    wq = {'n_bits': 8, 'channel_wise': True, 'scale_method': 'max'}
    aq = {'n_bits': 8, 'symmetric': True, 'channel_wise': False, 'scale_method': 'max',
          'leaf_param': True, 'dynamic': True}
    layers = [m.QuantModule(torch.nn.Linear(cin, c, bias=False), wq, aq, modulate=True).to(device)
              for c in couts]
    for q in layers:
        q.set_quant_state(True, True)
    return layers


def _evaluate(layers, x):
    owner = layers[0]
    return [owner(x)] + [q.forward_shared(owner, x) for q in layers[1:]]


def test_every_output_is_written_once_an_evaluation(monkeypatch):
    """On the CPU, with the launches recorded instead of made."""
    from modiff_b200 import _lib
    written = []

    def record(name, *args, **kw):
        if name == 'modiff_igemm_conv':
            written.append(args[6])
        elif name == 'modiff_linear_group':
            blocks = (C.c_int32 * (2 * args[6])).from_address(args[5])
            for i in sorted(set(blocks[0::2])):
                written.append(_lib.LinearItem.from_address(args[4] + i * C.sizeof(_lib.LinearItem)).o_hat)

    class Stream:
        def synchronize(self):
            pass

    monkeypatch.setattr(_lib, 'call', record)
    monkeypatch.setattr(_lib, 'require_cuda', lambda *a: None)
    monkeypatch.setattr(_lib, 'stream_ptr', lambda: 0)
    monkeypatch.setattr(torch.cuda, 'current_stream', lambda *a: Stream())
    layers = _layers()
    with torch.no_grad():
        for rows in ROWS:
            for q in layers:
                q.reset_cache()
            for step in range(4):
                written.clear()
                _evaluate(layers, torch.zeros(rows, CIN))
                if step:              # the first evaluation creates the caches
                    assert sorted(written) == sorted(q.o_hat.data_ptr() for q in layers), (rows, step)


@pytest.mark.gpu
@pytest.mark.parametrize("cin,couts,sizes", [(CIN, (COUT, COUT), ROWS),
                                             (1280, (1280, 1280, 1280), [64, 128, 96, 128]),
                                             (1280, (320, 1280) * 9, [150, 200, 150])])
def test_outputs_are_a_fresh_layers_at_every_size(cuda, cin, couts, sizes):
    import modiff_b200 as m
    used = _layers(cuda, cin, couts)
    g = torch.Generator().manual_seed(1)
    with torch.no_grad():
        for rows in sizes:
            x = torch.randn(rows, cin, generator=g)
            xs = [(x + 0.1 * s * torch.randn(rows, cin, generator=g)).to(cuda) for s in range(4)]
            fresh = _layers(cuda, cin, couts)
            for q in used:
                q.reset_cache()
            for step, xi in enumerate(xs):
                for a, b in zip(_evaluate(used, xi), _evaluate(fresh, xi)):
                    assert torch.equal(a, b), (rows, step)
    assert m.device_status() == 0


def _small_transformer(device):
    import modiff_b200 as m
    torch.manual_seed(0)
    net = m.UNetModel(image_size=8, in_channels=4, out_channels=4, model_channels=640,
                      attention_resolutions=[1], num_res_blocks=1, channel_mult=[1], num_heads=8,
                      use_spatial_transformer=True, transformer_depth=1, context_dim=CIN,
                      legacy=False).eval()
    m.rerandomize_zero_tensors(net, seed=1)
    wq = {"n_bits": 8, "channel_wise": True, "scale_method": "max"}
    aq = {"n_bits": 8, "symmetric": True, "channel_wise": False, "scale_method": "max",
          "leaf_param": True, "dynamic": True}
    qnn = m.QuantModel(net, wq, aq, sm_abit=8, modulate=True).to(device).eval()
    qnn.set_quant_state(True, True)
    return qnn


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
def test_guided_batches_in_turn(cuda, graph):
    """A small transformer UNet (cross-attention 768 -> 640, 77 tokens a prompt), guided, at batch 1,
    2, 4, 1, 4 with a pass repeated: the samples of a fresh model at each size."""
    import modiff_b200 as m
    g = torch.Generator().manual_seed(2)
    used = _small_transformer(cuda)

    def sample(qnn, b, x, cond, uncond, use_graph):
        qnn.reset_cache()
        out, _ = m.DDIMSampler(qnn, linear_start=0.00085, linear_end=0.0120).sample(
            5, b, tuple(x.shape[1:]), conditioning=cond, x_T=x, unconditional_guidance_scale=3.0,
            unconditional_conditioning=uncond, cuda_graph=use_graph)
        return out.clone()

    for b in (1, 2, 2, 4, 1, 4):
        x = torch.randn(b, 4, 8, 8, generator=g).to(cuda)
        cond, uncond = (torch.randn(b, 77, CIN, generator=g).to(cuda) for _ in range(2))
        got = sample(used, b, x, cond, uncond, graph)
        want = sample(_small_transformer(cuda), b, x, cond, uncond, False)
        assert torch.equal(got, want), b
