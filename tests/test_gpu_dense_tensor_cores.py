"""Dense layers on the tensor cores: around the row tile (128) and the smallest batch that takes them (512), contractions of
one slice (32), of three and of those that two to four blocks share, one to three tiles of 64 outputs, both layouts of the
weight -- against float64; contractions taken in several runs; operands that are not finite; weight and bias gradients, which
only a layer has, against framework products, and the weights' against float64 up to 65 537 atoms."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _linear(x, w, b, r, relu, kn):
    from crystalframer_b200 import _lib
    p = _lib.ptr
    y = torch.full((x.shape[0], w.shape[1 if kn else 0]), float("nan"), device=x.device)
    _lib.invoke("cfb200_linear", 1, x.device, p(x), p(w), None if b is None else p(b), None if r is None else p(r),
                x.shape[0], y.shape[1], x.shape[1], relu, kn, p(y))
    assert _lib.read_status(x.device) == 0
    return y


def _draw(rows, outs, inner, kn):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    dev = torch.device("cuda:0")
    g = torch.Generator().manual_seed(rows + outs + inner)
    x, b, r = (torch.randn(s, generator=g).to(dev) for s in ((rows, inner), (outs,), (rows, outs)))
    return x, torch.randn((inner, outs) if kn else (outs, inner), generator=g).to(dev), b, r


@pytest.mark.parametrize("rows", [512, 513, 640, 1000])
@pytest.mark.parametrize("outs,inner,kn", [(64, 32, 0), (64, 32, 1), (192, 96, 0), (64, 96, 1), (128, 160, 0), (128, 256, 1),
                                           (64, 416, 0), (128, 544, 1), (512, 128, 0)])
def test_products(rows, outs, inner, kn):
    """Exact splits into three bf16 numbers and six products leave 2^-23 of a product; the accumulators cut off 2^-23 of
    themselves per 16 terms, and four of them are added: inner / 16 + 5 times 2^-23 of the sum of the terms' sizes."""
    x, w, b, r = _draw(rows, outs, inner, kn)
    W = w.double() if kn else w.double().t()
    size = x.double().abs() @ W.abs()
    want = x.double() @ W
    y = _linear(x, w, None, None, 0, kn)
    assert ((y.double() - want).abs() <= (inner / 16 + 5) * 2.0 ** -23 * size).all()
    # and no larger on the whole than that of a chain of FP32 additions, 0.2 sqrt(inner / 2) 2^-23 of the result and more
    assert float((y.double() - want).norm() / want.norm()) <= 1.5e-7
    y2 = _linear(x, w, b, r, 1, kn)
    want = (want + b.double() + r.double()).clamp_min(0)
    size += b.double().abs() + r.double().abs()
    assert ((y2.double() - want).abs() <= (inner / 16 + 7) * 2.0 ** -23 * size).all()
    assert torch.equal(y2, _linear(x, w, b, r, 1, kn))


@pytest.mark.parametrize("rows,outs,inner", [(10000, 192, 512), (10000, 192, 544), (10000, 192, 576), (10000, 192, 768), (10000, 192, 1024),
                                             (513, 64, 1056), (700, 128, 2080), (520, 64, 8192)])
@pytest.mark.parametrize("kn", [0, 1])
@pytest.mark.parametrize("signs", [1, 2])
def test_products_of_long_contractions(rows, outs, inner, kn, signs):
    """Contractions above 512 terms, which one block takes in runs of eight slices (last runs of one, of two and of eight), or
    which blocks share: distance from float64, of the result's norm, for operands of both signs and of one.  The accumulators
    cut off what does not fit, on average 2^-24 of their size: a run's eight times (16 where one takes 512 terms), while they
    grow, so half of 8 (16) times that, and the runs' FP32 sum adds below 2^-24 per eighth of their number's root."""
    x, w, _, _ = _draw(rows, outs, inner, kn)
    if signs == 1:
        x, w = x.abs(), w.abs()
    y = _linear(x, w, None, None, 0, kn)
    want = x.double() @ (w.double() if kn else w.double().t())
    error = float((y.double() - want).norm() / want.norm())
    assert error <= (4 if inner > 512 else 8) * 2.0 ** -24 * 1.25, error
    x[5, 7], x[rows - 1, inner - 1] = float("inf"), float("nan")
    z = _linear(x, w, None, None, 0, kn)
    assert z[rows - 1].isnan().all() and not z[5].isfinite().any() and torch.equal(z[128:rows // 128 * 128], y[128:rows // 128 * 128])


@pytest.mark.parametrize("atoms", [600, 2560, 2593, 3500, 4000, 4600, 16384, 65537])
@pytest.mark.parametrize("signs", [1, 2])
def test_weight_gradients_of_large_batches(atoms, signs):
    """Feed-forward weight gradients of a layer against float64 on the activations that the layer's own products give: splits
    of the atoms that one run takes (up to 160) and of two to 33 runs of four slices, last ones of one, two, three and four.
    The accumulators of the large products are cut off four times by 2^-24 of their size on average, while they grow: 2 2^-24
    at most for operands of one sign, less the first of each, which cuts nothing off; the FP32 sums of the runs and of the 16
    splits add roundings of either sign, below 2^-24 in all.  Of both signs the result is smaller than its parts: twice that."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from crystalframer_b200 import _lib, data, synth
    from crystalframer_b200.latticeformer import Latticeformer, ModelParams
    dev = torch.device("cuda:0")
    torch.manual_seed(1)
    model = Latticeformer(ModelParams(num_layers=1, frame_method="no", value_pe_angle_real=0, symm_break_noise=0.0)).to(dev).train()
    layer = model.encoder.layers[0]
    with torch.no_grad():
        model(data.host_batch(synth.make_batch(16, 3), np.zeros((16, 1), np.float32), pinned=False).to(dev, non_blocking=False))
        layer.self_attn.out_proj.weight.zero_()                 # the feed-forward block's input is the layer's
    g = torch.Generator().manual_seed(atoms)
    x, up = (torch.randn(atoms, 128, generator=g).to(dev) for _ in range(2))
    if signs == 1:
        x, up = x.abs(), up.abs()
    eye = torch.eye(3, device=dev).expand(atoms, 3, 3).contiguous()
    one = torch.arange(atoms, device=dev)
    model.zero_grad(set_to_none=True)
    layer(x, one, one.repeat(2, 1), torch.zeros(atoms, 3, device=dev), None, 6 * eye, None, eye, None).backward(up)
    w1, b1, w2 = (p.detach() for p in (layer.linear1.weight, layer.linear1.bias, layer.linear2.weight))
    h = _linear(x, w1, b1, None, 1, 0)
    gh = torch.where(h > 0, _linear(up, w2, None, None, 0, 1), 0.0)
    for got, want in ((layer.linear2.weight.grad, up.double().t() @ h.double()), (layer.linear1.weight.grad, gh.double().t() @ x.double())):
        error = float((got.double() - want).norm() / want.norm())
        assert error <= 2.5 * signs * 2.0 ** -24, error


@pytest.mark.parametrize("kn", [0, 1])
def test_operands_that_are_not_finite(kn):
    """An infinity has no split: its tiles give what FP32 gives, and the others are untouched."""
    x, w, _, _ = _draw(700, 128, 512, kn)
    clean = _linear(x, w, None, None, 0, kn)
    x[5, 7], x[200, 500], x[201, 3], x[640, 100] = float("inf"), float("nan"), -float("inf"), 3.4e38
    y = _linear(x, w, None, None, 0, kn)
    want = (x.double() @ (w.double() if kn else w.double().t())).float()
    assert torch.equal(y.isnan(), want.isnan())
    assert torch.equal(y.isinf(), want.isinf()) and torch.equal(y[y.isinf()], want[want.isinf()])
    fine = want.isfinite()
    assert ((y - want).abs()[fine] <= 1e-4 * (1 + want.abs()[fine])).all()
    assert torch.equal(y[256:512], clean[256:512])


@pytest.mark.parametrize("atoms", [512, 560, 1100])
def test_gradients_of_a_layer(atoms):
    """Every gradient of a one-call layer (slices of the batch's rows that end in the middle of one of 32) against the layer
    operator by operator: 1e-4 of the largest entry, the bound of the layer's own tests."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from crystalframer_b200 import data, encoder, synth
    from crystalframer_b200.latticeformer import Latticeformer, ModelParams
    dev = torch.device("cuda:0")
    torch.manual_seed(1)
    model = Latticeformer(ModelParams(num_layers=1, symm_break_noise=0.0)).to(dev).train()
    b = synth.make_batch(atoms // 4, 2, size_dist="uniform", size_lo=4, size_hi=4)
    tb = data.host_batch(b, np.zeros((len(b.sizes), 1), np.float32), pinned=False).to(dev, non_blocking=False)
    with torch.no_grad():
        model(data.host_batch(synth.make_batch(16, 3), np.zeros((16, 1), np.float32), pinned=False).to(dev, non_blocking=False))
    results = []
    try:
        for one_call in (False, True):
            encoder.FUSED_LAYER = one_call
            model.zero_grad(set_to_none=True)
            out = model(tb)
            out.square().sum().backward()
            results.append([out.detach()] + [p.grad.clone() for p in model.parameters() if p.grad is not None])
    finally:
        encoder.FUSED_LAYER = True
    for x, y in zip(*results):
        assert (x - y).abs().max() <= 1e-4 * x.abs().max() + 1e-9, (x.shape, float((x - y).abs().max()), float(x.abs().max()))
