"""The attention kernel at the edges of its key blocks (128 keys, two score buffers) and of its two
operand layouts (heads of up to 64 channels keep q in shared memory), with maxima that keep growing
along the keys (every block rescales the accumulated output), against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grow", [0.0, 6.0])
@pytest.mark.parametrize("b,c,t,tk", [(2, 40, 128, 65), (3, 64, 64, 128), (2, 64, 256, 129), (1, 72, 128, 192),
                                      (2, 24, 1024, 300), (1, 200, 64, 640), (2, 256, 128, 321),
                                      (1, 64, 4096, 16)])
def test_attention_matches_float64(cuda, b, c, t, tk, grow):
    from modiff_b200 import ops
    import modiff_b200 as m
    torch.manual_seed(tk)
    q, k, v = torch.randn(b, c, t), torch.randn(b, c, tk), torch.randn(b, c, tk)
    q[:, 0] = 1.0
    k[:, 0] = torch.linspace(0.0, grow * c ** 0.5, tk)      # scores rise by `grow` along the keys
    scale = float(c) ** -0.5
    for s in (scale, -scale):
        w = torch.softmax(q.double().transpose(1, 2) @ k.double() * s, dim=2)
        exp = v.double() @ w.transpose(1, 2)
        got = ops.attention(q.to(cuda), k.to(cuda), v.to(cuda), s)
        torch.cuda.synchronize()
        assert m.device_status() == 0
        # operands keep 2^-17 of themselves: a score moves by at most 2^-16 sum |q k| scale, about
        # 2^-16 (c^0.5 + grow), its probability by as much relatively, the output by twice that
        bound = 2.0 ** -15 * (c ** 0.5 + grow) / 4 + 2e-6
        err = (got.cpu().double() - exp).abs().max() / exp.abs().max()
        assert err < bound, (err, bound)
