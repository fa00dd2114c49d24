"""The work that users of this package have it do, as cases to be timed.

A case is one call of a sampler (or of the first-stage decoder) as a user's program makes it, on
a model that the program holds: the modulated-quantisation sampling pass of the pixel UNet, the
latent UNet (LSUN-churches kl-8 shapes) and the Stable-Diffusion-v1 UNet, and the decoder that
turns the latent models' samples into pixels.  Random-init weights and N(0, 1) noise / context
stand in for checkpoints and prompts.

Ranges: batch 1 (one image for one user) to 256 (bulk generation) in any size, 10 to 100 sampling
steps, W8A8 / W4A4 codes, symmetric (`--a_sym`) and asymmetric activation quantisers, dynamic and
calibrated (static) activation scales, the split shortcut, floating-point and integer attention,
DDIM and PLMS, guided and unguided, latents of 32x32 and 64x64.
"""
import math

import torch
import torch.nn.functional as F

import modiff_b200 as m
from modiff_b200.ldm_unet import LSUN_CHURCHES_KL8, SD_V1

DEVICE = "cuda"


def _case(name, net, batch, steps, w_bits=8, a_bits=8, sym=True, static=False, split=False,
          int8_attention=False, sampler="ddim"):
    return dict(name=name, net=net, batch=batch, steps=steps, w_bits=w_bits, a_bits=a_bits, sym=sym,
                static=static, split=split, int8_attention=int8_attention, sampler=sampler)


def listed():
    return [
        # one image while somebody waits, few steps: launches and latency decide
        _case("pixel_w8a8_b1", "pixel", 1, 20),
        # the W8A8 configuration of the pixel UNet at its quoted batch and length
        _case("pixel_w8a8_b8", "pixel", 8, 100),
        # an odd remainder of a bulk job, 4-bit codes with the split shortcut
        _case("pixel_w4a4_b37", "pixel", 37, 100, 4, 4, split=True),
        # bulk generation, the headline configuration of the pixel UNet
        _case("pixel_w4a4_b256", "pixel", 256, 100, 4, 4, split=True),
        # a calibrated checkpoint: activation scales are read, not measured
        _case("pixel_w8a8_static_b100", "pixel", 100, 50, static=True),
        # the latent drivers' default quantisers (no --a_sym), a handful of images
        _case("ldm_w8a8_asym_b5", "ldm", 5, 50, sym=False),
        # latent UNet at its quoted batch, integer attention
        _case("ldm_w8a8_b32", "ldm", 32, 50, int8_attention=True),
        # text to image for one prompt: guided PLMS, floating-point attention
        _case("sd_w8a8_plms_b1", "sd", 1, 20, sampler="plms"),
        # text to image at the quoted batch: guided DDIM, integer attention
        _case("sd_w8a8_b8", "sd", 8, 20, int8_attention=True),
        # the samples of a latent batch to 256x256 pixels
        _case("decode_32_b8", "decoder32", 8, 1),
        # one image of a 64x64 latent to 512x512 pixels
        _case("decode_64_b1", "decoder64", 1, 1),
    ]


def _between(rng, lo, hi):
    """A whole number, uniform over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    net = rng.choice(["pixel"] * 5 + ["ldm"] * 3 + ["sd"] * 2 + ["decoder32", "decoder64"])
    if net.startswith("decoder"):
        return _drawn(net, _between(rng, 1, 12 if net == "decoder32" else 3), 1)
    if net == "pixel":
        w_bits, a_bits = rng.choice([(8, 8), (8, 8), (4, 4)])
        static = w_bits == 8 and rng.random() < 0.25
        batch = _between(rng, 1, 256)
        steps = rng.choice([20, 50, 100]) if w_bits == 8 else 100
        return _drawn(net, batch, steps, w_bits, a_bits, static=static,
                      split=w_bits == 4 or rng.random() < 0.3)
    sym = rng.random() < 0.7
    return _drawn(net, _between(rng, 1, 48 if net == "ldm" else 8), rng.choice([20, 25, 40, 50]) if
                  net == "ldm" else rng.choice([10, 20]), sym=sym,
                  int8_attention=sym and rng.random() < 0.6,
                  sampler="plms" if rng.random() < 0.3 else "ddim")


def _drawn(*args, **kw):
    c = _case("", *args, **kw)
    del c["name"]
    return c


def _redraw_zeros(net, generator):
    """Latent UNets zero-initialise the last layer of every block; a trained model has weights
    there.  Drawn small: a residual branch of random weights amplifies last-bit differences from
    step to step, which a trained one does not."""
    with torch.no_grad():
        for p in net.parameters():
            if not bool(p.any()):
                p.normal_(0.0, 0.005, generator=generator)


def prepare(case, seed):
    torch.manual_seed(seed)
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    kind, b = case["net"], case["batch"]
    if kind.startswith("decoder"):
        size = int(kind[len("decoder"):])
        with torch.device(DEVICE):
            dec = m.FirstStageDecoder().eval()
        return dict(case=case, decoder=dec, z=torch.randn(b, 4, size, size, generator=g,
                                                          device=DEVICE))
    wq = {"n_bits": case["w_bits"], "channel_wise": True, "scale_method": "max"}
    aq = {"n_bits": case["a_bits"], "symmetric": case["sym"], "channel_wise": False,
          "scale_method": "max", "leaf_param": True, "dynamic": not case["static"]}
    with torch.device(DEVICE):
        if kind == "pixel":
            net = m.Model(m.make_config(split_shortcut=case["split"])).eval()
        else:
            net = m.UNetModel(**(SD_V1 if kind == "sd" else LSUN_CHURCHES_KL8)).eval()
            _redraw_zeros(net, g)
        qnn = m.QuantModel(net, wq, aq, sm_abit=8, modulate=True,
                           int8_attention=case["int8_attention"]).to(DEVICE).eval()
    qnn.set_quant_state(True, True)
    state = dict(case=case, qnn=qnn)
    if kind == "pixel":
        state["betas"] = torch.from_numpy(m.get_beta_schedule()).float()
        state["seq"] = m.make_timestep_sequence(1000, case["steps"], "quad")
        state["x"] = torch.randn(b, 3, 32, 32, generator=g, device=DEVICE)
    else:
        sd = kind == "sd"
        cls = m.PLMSSampler if case["sampler"] == "plms" else m.DDIMSampler
        state["sampler"] = cls(qnn, linear_start=0.00085 if sd else 0.0015,
                               linear_end=0.0120 if sd else 0.0155)
        size = 64 if sd else 32
        state["x"] = torch.randn(b, 4, size, size, generator=g, device=DEVICE)
        if sd:
            state["cond"] = torch.randn(b, 77, 768, generator=g, device=DEVICE)
            state["uncond"] = torch.randn(b, 77, 768, generator=g, device=DEVICE)
    if case["static"]:
        # the calibrated scales of a checkpoint: what each layer measures at its first
        # quantised evaluation, kept from then on
        t = torch.full((b,), float(state["seq"][-1]), device=DEVICE)
        for k in range(2):
            qnn(state["x"] + 0.05 * k * torch.randn(state["x"].shape, generator=g, device=DEVICE), t)
    return state


def run(state):
    case = state["case"]
    if "decoder" in state:
        return state["decoder"].decode(state["z"])
    state["qnn"].reset_cache()
    if case["net"] == "pixel":
        xs, _ = m.generalized_steps(state["x"], state["seq"], state["qnn"], state["betas"], eta=0.0)
        return xs[-1]
    kw = {}
    if case["net"] == "sd":
        kw = dict(conditioning=state["cond"], unconditional_conditioning=state["uncond"],
                  unconditional_guidance_scale=7.5)
    x = state["x"]
    out, _ = state["sampler"].sample(case["steps"], case["batch"], tuple(x.shape[1:]), eta=0.0, x_T=x,
                                     **kw)
    return out


# Of one image and evaluation, summed over the quantised layers' shapes: elements of the distinct
# cached inputs, elements of the cached outputs, multiply-adds of the layers, multiply-adds of
# the attention products; and the weights of the model.
_SUMS = {"pixel": (5.70e6, 4.77e6, 6.054e9, 0.17e9, 35.69e6),
         "ldm": (11.53e6, 12.63e6, 18.64e9, 2.3e9, 294.7e6),
         "sd": (185.2e6, 236.7e6, 338.6e9, 63.0e9, 859.1e6)}


def _decoder_sums(size):
    """(multiply-adds of one image, weights) of the kl-f8 decoder."""
    macs = weights = 0

    def conv(cin, cout, k, res):
        nonlocal macs, weights
        macs += cin * cout * k * k * res * res
        weights += cin * cout * k * k

    def block(cin, cout, res):
        conv(cin, cout, 3, res)
        conv(cout, cout, 3, res)
        if cin != cout:
            conv(cin, cout, 1, res)

    res, ch = size, 512
    conv(4, 4, 1, res)
    conv(4, ch, 3, res)
    block(ch, ch, res)
    for _ in range(4):
        conv(ch, ch, 1, res)
    macs += 2 * (size * size) ** 2 * ch
    block(ch, ch, res)
    for level, out in reversed(list(enumerate((128, 256, 512, 512)))):
        for _ in range(3):
            block(ch, out, res)
            ch = out
        if level:
            res *= 2
            conv(ch, ch, 3, res)
    conv(ch, 3, 3, res)
    return macs, weights


def work(case):
    """Per evaluation every layer's cached input and cached output are read and written once (the
    state that modulation keeps from step to step, fp32) and the weight codes read once."""
    kind, b = case["net"], case["batch"]
    if kind.startswith("decoder"):
        size = int(kind[len("decoder"):])
        macs, weights = _decoder_sums(size)
        return {"bytes": 4.0 * (weights + b * (4 * size * size + 3 * 64 * size * size)),
                "flops": 2.0 * macs * b}
    inputs, outputs, macs, attention, weights = _SUMS[kind]
    rows = b * (2 if kind == "sd" else 1)
    evals = case["steps"]
    if kind != "pixel":
        evals = len(range(0, 1000, 1000 // case["steps"])) + (case["sampler"] == "plms")
    per_eval = 8.0 * rows * (inputs + outputs) + weights * case["w_bits"] / 8.0
    return {"bytes": evals * per_eval, "flops": evals * rows * 2.0 * (macs + attention)}


def tolerance(case):
    """Sampling quantises the differences between nearly equal tensors of successive steps, so a
    last-bit difference anywhere moves some codes by one and the samples by far more than one
    rounding.  Stated is about four times what the first evaluation's sums in another order, or
    1e-6 of noise on x_T, did to the samples (W4A4: 0.014, pixel W8A8: 0.0013 at 20 steps, static
    scales 0.0003, latent 0.0003, SD 0.0033 at 10 steps); the decoder's is four times its distance
    from the same network in 64 bits."""
    kind = case["net"]
    if kind.startswith("decoder"):
        return {"rel": 4e-5, "max": 3e-4}
    if kind == "pixel":
        if case["w_bits"] == 4:
            return {"rel": 0.03, "max": 0.3}
        return {"rel": 0.0012, "max": 0.006} if case["static"] else {"rel": 0.006, "max": 0.025}
    return {"rel": 0.002, "max": 0.008} if kind == "ldm" else {"rel": 0.013, "max": 0.05}


def _conv64(x, p, name):
    """Stride-1 'same' convolution in 64 bits, one image at a time as a matrix product."""
    w, b = p[name + ".weight"], p[name + ".bias"]
    k = w.shape[-1]
    images = [(w.flatten(1) @ F.unfold(im[None], k, padding=k // 2)[0]).view(-1, *x.shape[2:])
              for im in x]
    return torch.stack(images) + b.view(1, -1, 1, 1)


def _norm64(x, p, name, silu=True):
    y = F.group_norm(x, 32, p[name + ".weight"], p[name + ".bias"], eps=1e-6)
    return F.silu(y) if silu else y


def _block64(x, p, name):
    h = _conv64(_norm64(x, p, name + ".norm1"), p, name + ".conv1")
    h = _conv64(_norm64(h, p, name + ".norm2"), p, name + ".conv2")
    return h + (_conv64(x, p, name + ".nin_shortcut") if name + ".nin_shortcut.weight" in p else x)


def exact(case, seed):
    """The decoder in plain 64-bit torch.  A sampler has no such value: it rounds residuals of
    nearly equal tensors to codes, and where a code falls decides more than any sum's precision."""
    if not case["net"].startswith("decoder"):
        return None
    state = prepare(case, seed)
    p = {k.removeprefix("decoder."): v.double() for k, v in state["decoder"].state_dict().items()}
    h = _conv64(_conv64(state["z"].double(), p, "post_quant_conv"), p, "conv_in")
    h = _block64(h, p, "mid.block_1")
    n = _norm64(h, p, "mid.attn_1.norm", silu=False)
    q, k, v = (_conv64(n, p, "mid.attn_1." + s).flatten(2) for s in "qkv")
    a = torch.softmax(q.transpose(1, 2) @ k * q.shape[1] ** -0.5, dim=2) @ v.transpose(1, 2)
    h = h + _conv64(a.transpose(1, 2).reshape(h.shape), p, "mid.attn_1.proj_out")
    h = _block64(h, p, "mid.block_2")
    for level in (3, 2, 1, 0):
        for i in range(3):
            h = _block64(h, p, f"up.{level}.block.{i}")
        if level:
            h = _conv64(F.interpolate(h, scale_factor=2.0, mode="nearest"), p,
                        f"up.{level}.upsample.conv")
    return _conv64(_norm64(h, p, "norm_out"), p, "conv_out")
