"""Kernels that share a row or a query between threads when there are few of them: the grouped small
linear layers (integer sums, exact) and the attention of at most 64 tokens."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 2, 3, 8, 37, 154, 300])
@pytest.mark.parametrize("cin,couts", [(16, [16]), (512, [256, 40, 16]), (1280, [320, 24])])
def test_grouped_linears_match_the_integer_sums(cuda, rows, cin, couts):
    from modiff_b200 import _lib
    g = torch.Generator().manual_seed(rows * 7 + cin)
    codes = torch.randint(-128, 128, (rows, cin), generator=g, dtype=torch.int8)
    kp = -(-cin // 128) * 128
    xs, dev_codes = torch.tensor([0.03125], device=cuda), codes.to(cuda)
    items, block_map, keep = (_lib.LinearItem * len(couts))(), [], []
    for i, co in enumerate(couts):
        w = torch.randint(-128, 128, (co, cin), generator=g, dtype=torch.int8)
        packed = torch.zeros(-(-co // 128) * 128, kp, dtype=torch.int8)
        packed[:co, :cin] = w
        corr = torch.randint(-9, 10, (co,), generator=g, dtype=torch.int32)
        t = [packed.to(cuda), torch.full((co,), 0.5, device=cuda), corr.to(cuda),
             torch.randn(rows, co, generator=g).to(cuda)]
        items[i] = _lib.LinearItem(t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), t[3].data_ptr(), co, 0)
        block_map += [(i, c0) for c0 in range(0, co, 16)]
        acc = codes.long() @ w.long().t() + codes.long().sum(1, keepdim=True) * corr.long()
        # scales are powers of two and |acc| < 2^24 + ..: the fused multiply-add rounds once
        keep.append((t, (t[3].cpu().double() + acc.double() * 0.015625).float()))
    table = torch.frombuffer(bytearray(bytes(items)), dtype=torch.uint8).to(cuda)
    blocks = torch.tensor(block_map, dtype=torch.int32, device=cuda)
    _lib.call('modiff_linear_group', dev_codes.data_ptr(), xs.data_ptr(), rows, cin, table.data_ptr(),
              blocks.data_ptr(), len(block_map), _lib.stream_ptr())
    for t, want in keep:
        # sums beyond 2^24 lose their last bits in the conversion to fp32 as well: one more rounding
        assert torch.allclose(t[3].cpu(), want, rtol=2.0 ** -22, atol=2.0 ** -20)


# images from four a SM on (592): one block each, except few pairs and wide heads
@pytest.mark.parametrize("b,c,t,tk", [(1, 256, 16, 16), (3, 24, 64, 64), (2, 130, 7, 33), (5, 768, 4, 4),
                                      (2, 64, 9, 1), (1, 64, 1, 64), (591, 24, 64, 64), (592, 24, 64, 64),
                                      (600, 130, 7, 33), (600, 64, 9, 1), (600, 96, 4, 4), (600, 260, 9, 16)])
def test_small_attention(cuda, b, c, t, tk):
    from modiff_b200 import _lib
    g = torch.Generator().manual_seed(t)
    q, k, v = (torch.randn(b, c, n, generator=g) for n in (t, tk, tk))
    out = torch.empty(b, c, t, device=cuda)
    scale = c ** -0.5
    d = [x.to(cuda) for x in (q, k, v)]
    _lib.call('modiff_attention_small', d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), out.data_ptr(),
              b, c, t, tk, scale, _lib.stream_ptr())
    w = torch.softmax(q.double().transpose(1, 2) @ k.double() * scale, dim=-1)
    ref = v.double() @ w.transpose(1, 2)
    # fp32 sums over c channels of unit values move a score by about sqrt(c) 2^-24 * scale * sqrt(c),
    # a probability by as much relatively: 2e-6 with the sums over the keys
    assert float((out.cpu().double() - ref).abs().max()) < 2e-6 * max(1.0, float(ref.abs().max()))
