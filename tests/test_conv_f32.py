"""The tensor-core fp32 convolution (three bf16 planes per operand) against the same convolution in
64 bits, at the edges of its tiles: ragged channel counts, one chunk and several, widths that are
not powers of two, images smaller than a tile, few output channels."""
import pytest
import torch
import torch.nn.functional as F


def _layer(conv):
    import modiff_b200 as m
    return m.QuantModule(conv, {'n_bits': 8, 'channel_wise': True, 'scale_method': 'max'},
                         {'n_bits': 8, 'symmetric': True, 'channel_wise': False,
                          'scale_method': 'max', 'leaf_param': True, 'dynamic': True})


def _bound(x, w, pad):
    """Largest error of any output.  Products leave out at most 2^-24 of themselves; a chunk of 64
    channels adds 24 terms in the tensor core, each rounded (or cut off) at 2^-23 of a partial sum
    that stays below sum |x||w|, and the chunks and the bias are added in fp32.  A worst case: a lost
    plane can stay below it; `test_error_is_no_larger_than_the_fp32_kernels` is the one that shows it."""
    chunks = w.shape[2] * w.shape[3] * -(-w.shape[1] // 64)
    return (24 + chunks + 2) * 2.0 ** -23 * F.conv2d(x.abs(), w.abs(), padding=pad) + 1e-30


@pytest.mark.gpu
@pytest.mark.parametrize("b,cin,cout,h,w,k,pad", [
    (1, 32, 16, 8, 8, 3, 1), (3, 40, 3, 5, 7, 3, 1), (1, 64, 128, 16, 16, 1, 0),
    (2, 130, 72, 24, 24, 3, 1), (1, 128, 3, 4, 512, 3, 1), (130, 64, 20, 1, 1, 1, 0),
    (5, 96, 200, 6, 40, 5, 2), (1, 512, 512, 32, 32, 3, 1), (1, 256, 130, 64, 128, 3, 0)])
def test_matches_64_bit_convolution(cuda, b, cin, cout, h, w, k, pad):
    import modiff_b200 as m
    torch.manual_seed(b + cin)
    conv = torch.nn.Conv2d(cin, cout, k, padding=pad).to(cuda)
    x = torch.randn(b, cin, h, w, device=cuda) * torch.rand(b, cin, 1, 1, device=cuda) * 3
    y = _layer(conv)(x)
    torch.cuda.synchronize()
    assert m.device_status() == 0
    wd, bd = conv.weight.detach().double().cpu(), conv.bias.detach().double().cpu()
    xd = x.double().cpu()
    ref = F.conv2d(xd, wd, bd, padding=pad)
    err = (y.double().cpu() - ref).abs()
    bound = _bound(xd, wd, pad) + 2.0 ** -23 * ref.abs()
    assert bool((err <= bound).all()), float((err / bound).max())


@pytest.mark.gpu
@pytest.mark.parametrize("b,cin,cout,h,w,up2", [(2, 64, 32, 8, 8, False), (1, 96, 40, 7, 5, False),
                                                (1, 128, 128, 64, 96, False), (2, 64, 48, 5, 6, True)])
def test_norm_silu_upsample_and_residual_around_the_convolution(cuda, b, cin, cout, h, w, up2):
    torch.manual_seed(7)
    conv = torch.nn.Conv2d(cin, cout, 3, padding=1).to(cuda)
    norm = torch.nn.GroupNorm(32, cin, eps=1e-6).to(cuda)
    with torch.no_grad():
        norm.weight.normal_(1.0, 0.3)
        norm.bias.normal_()
    x = torch.randn(b, cin, h, w, device=cuda) + 4.0
    s = 2 if up2 else 1
    res = torch.randn(b, cout, s * h, s * w, device=cuda)
    y = _layer(conv).conv_plain(x, norm=norm, silu=True, up2=up2, residual=res)
    n = F.silu(F.group_norm(x.double(), 32, norm.weight.double(), norm.bias.double(), 1e-6))
    if up2:
        n = F.interpolate(n, scale_factor=2.0, mode="nearest")
    ref = F.conv2d(n.cpu(), conv.weight.double().cpu(), conv.bias.double().cpu(), padding=1) + res.double().cpu()
    # fp32 GroupNorm of values around 4 (mean subtracted: 2^-22 of 4 over a deviation of 1) and a
    # SiLU of about 2 ulp, both multiplied through the sum of |w|: 1e-5 of the largest value
    assert float((y.double().cpu() - ref).abs().max() / ref.abs().max()) < 1e-5


@pytest.mark.gpu
def test_infinities_and_large_values_are_those_of_the_plain_sum(cuda):
    torch.manual_seed(9)
    conv = torch.nn.Conv2d(64, 16, 3, padding=1).to(cuda)
    x = torch.randn(1, 64, 8, 8, device=cuda)
    x[0, 3, 1, 1], x[0, 5, 6, 6], x[0, 9, 1, 6] = float("inf"), float("nan"), 3.4e38
    y = _layer(conv)(x).cpu()
    ref = F.conv2d(x.cpu(), conv.weight.detach().cpu(), conv.bias.detach().cpu(), padding=1)
    assert torch.equal(torch.isnan(y), torch.isnan(ref))
    assert torch.equal(torch.isinf(y), torch.isinf(ref))
    assert torch.equal(y[torch.isinf(y)], ref[torch.isinf(ref)])
    fin = torch.isfinite(ref)
    assert torch.allclose(y[fin], ref[fin], rtol=1e-5, atol=1e-4)


SHORT_AND_LONG = [(1, 32, 16, 8, 1), (8, 32, 64, 32, 1), (1, 32, 32, 8, 3), (4, 40, 16, 16, 3), (8, 64, 64, 32, 1),
                  (1, 128, 128, 4, 3), (1, 512, 256, 16, 1), (1, 512, 512, 16, 3)]


def _operands(b, cin, cout, hw, k, positive):
    torch.manual_seed(b * 131 + cin + k)
    conv = torch.nn.Conv2d(cin, cout, k, padding=k // 2)
    x = torch.randn(b, cin, hw, hw)
    if positive:
        with torch.no_grad():
            conv.weight.abs_()
        x = x.abs()
    return conv, x


def _rms(err):
    return float(err.double().pow(2).mean().sqrt())


@pytest.mark.gpu
@pytest.mark.parametrize("positive", [False, True])
@pytest.mark.parametrize("b,cin,cout,hw,k", SHORT_AND_LONG)
def test_error_is_no_larger_than_the_fp32_kernels(cuda, b, cin, cout, hw, k, positive):
    """rms error against 64 bits of the tensor-core kernel and of the plain fp32 kernel on the same
    inputs, from 32 products a sum to 4608, also where nothing cancels (observed 0.14 - 0.73 of it)."""
    conv, x = _operands(b, cin, cout, hw, k, positive)
    ref = F.conv2d(x.double(), conv.weight.detach().double(), conv.bias.detach().double(), padding=k // 2)
    layer, xd = _layer(conv.to(cuda)), x.to(cuda)
    got = layer(xd)
    plain = torch.empty_like(got)
    layer._conv_fp32(xd, layer._org_weights_kn(), layer.org_bias, layer._geom(xd, 0), plain)
    err, err_plain = _rms(got.cpu() - ref), _rms(plain.cpu() - ref)
    assert err <= err_plain, (err, err_plain)


@pytest.mark.gpu
def test_single_products_keep_their_low_planes(cuda):
    """One channel and tap other than zero: an output is one product.  2^-24 of it is left out and five
    additions of its parts round at 2^-23 of it each; a lost low plane would be 2^-17 of it."""
    g = torch.Generator().manual_seed(4)
    for c in (0, 37, 63):
        x, conv = torch.zeros(1, 64, 8, 8), torch.nn.Conv2d(64, 32, 1, bias=False)
        x[0, c] = 1.0 + torch.rand(8, 8, generator=g)
        with torch.no_grad():
            conv.weight.zero_()
            conv.weight[:, c, 0, 0] = -1.0 - torch.rand(32, generator=g)
        ref = conv.weight.detach().double()[None, :, c] * x.double()[:, c:c + 1]
        got = _layer(conv.to(cuda))(x.to(cuda)).cpu().double()
        assert float(((got - ref) / ref).abs().max()) <= 2.0 ** -24 + 5 * 2.0 ** -23


@pytest.mark.parametrize("b,cin,cout,hw,k,positive", [
    (1, 32, 16, 8, 1, False), (1, 32, 32, 8, 3, False), (1, 64, 64, 8, 1, False), (1, 128, 32, 4, 3, False),
    (1, 32, 16, 8, 1, True), (1, 64, 64, 8, 1, True)])
def test_a_lost_plane_or_product_would_be_seen(b, cin, cout, hw, k, positive):
    """The comparison with the fp32 kernel, on the CPU with every sum of plane products in 64 bits (so
    that only what is left out counts): the kernel's six products stay far below the fp32 chain's error, two
    planes and any five of the six products lie above it.  (Long sums of one sign are left out: there the
    chain's own rounding outgrows what is lost.)"""
    conv, x = _operands(b, cin, cout, hw, k, positive)
    w = conv.weight.detach()
    # the fp32 kernel's chain: one fused multiply-add a product, channels and taps in order
    cols = F.unfold(x[:1], k, padding=k // 2)[0].double()
    chain = torch.zeros(cout, cols.shape[1])
    for i, row in enumerate(cols):
        chain = (chain.double() + w.flatten(1)[:, i:i + 1].double() * row).float()
    exact = w.flatten(1).double() @ cols
    err_chain = _rms(chain.double() - exact)

    def planes(v):
        out = []
        for _ in range(3):
            out.append(v.bfloat16().float())
            v = v - out[-1]
        return out

    px = planes(F.unfold(x[:1], k, padding=k // 2)[0])
    pw = planes(w.flatten(1))
    parts = {(i, j): pw[j].double() @ px[i].double() for i in range(3) for j in range(3)}
    six = [(0, 0), (0, 1), (1, 0), (1, 1), (0, 2), (2, 0)]
    error = lambda pairs: _rms(sum(parts[p] for p in pairs) - exact)
    assert error(six) < 0.25 * err_chain
    assert error([(0, 0), (0, 1), (1, 0), (1, 1)]) > 1.5 * err_chain          # two planes
    for lost in six[1:]:
        assert error([p for p in six if p != lost]) > 1.5 * err_chain, lost


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["conv1d_k1_pow2", "conv1d_k1", "conv1d_k3", "implicit_pad", "channels_last", "sliced",
                                  "offset", "weights_channels_last", "no_bias"])
def test_every_form_of_the_layer_agrees_with_the_fp32_kernel(cuda, form):
    """Orders, strides, alignments and paddings that the unquantised layer takes, against modiff_conv_fp32
    on the same layer: both are fp32 sums of 32 - 288 products, 1e-5 of the largest output apart at most
    (their own errors are below 1e-6 of the root mean square)."""
    torch.manual_seed(11)
    if form.startswith("conv1d"):
        k = 3 if form.endswith("k3") else 1
        conv = torch.nn.Conv1d(32, 24, k, padding=k // 2)
        x = torch.randn(2, 32, 64 if form.endswith("pow2") else 21, device=cuda)
    else:
        conv = torch.nn.Conv2d(32, 24, 3, padding=0 if form == "implicit_pad" else 1, bias=form != "no_bias")
        x = torch.randn(2, 32, 10, 7, device=cuda)
    conv = conv.to(cuda)
    if form == "weights_channels_last":
        conv = conv.to(memory_format=torch.channels_last)
    layer = _layer(conv)
    if form == "implicit_pad":
        layer.implicit_pad = (0, 1, 0, 1)          # right and bottom, as the UNet's downsampling pads
    plain_in = x
    if form == "channels_last":
        x = x.contiguous(memory_format=torch.channels_last)
    elif form == "sliced":
        x = torch.cat([x, x], dim=1)[:, :32]
    elif form == "offset":                         # contiguous, four bytes off a 16-byte boundary
        x = torch.cat([x.new_zeros(1), x.flatten()])[1:].view(x.shape)
        assert x.data_ptr() % 16 == 4
    y = layer(x)
    g = layer._geom(plain_in, 0)
    ref = torch.empty_like(y)
    layer._conv_fp32(plain_in, layer._org_weights_kn(), layer.org_bias, g, ref)
    assert float((y - ref).abs().max()) <= 1e-5 * float(ref.abs().max())
