"""The training forward of models with weighted-PCA frames keeps its order of summation: its predictions on a few batches
are, bit for bit, those that were recorded (``golden/weighted_pca_outputs.json``) before the attention kernels worked in
tiles of pairs and the dense layers split their contractions.  Signs and directions of eigenvectors, and the ReLUs behind
them, turn on a last bit, and where a batch's errors have balanced signs one turned ReLU is a quarter of the mean gradient.
Then the kernel that does it, against the tiles of the prediction, at the sizes where it can go wrong."""
import json
import os

import numpy as np
import pytest
import torch

from crystalframer_b200 import data, fused_layer, synth
from parity_util import cuda

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "weighted_pca_outputs.json")

# crystals, atoms from / to, cell vectors from / to, angle Gaussians, seed: chunked and whole tasks, one to three list
# ranges, narrow and wide angle bases, batches below and above 32 pairs per atom
BATCHES = [(16, 100, 200, 10.0, 25.0, 64, 1), (5, 100, 200, 10.0, 25.0, 64, 2), (1, 100, 200, 10.0, 25.0, 64, 3),
           (24, 20, 100, 6.0, 20.0, 64, 4), (2, 20, 100, 6.0, 20.0, 32, 5), (9, 20, 100, 6.0, 20.0, 16, 6),
           (40, 4, 40, 4.0, 12.0, 48, 7)]


def _model_and_batch(crystals, lo, hi, len_lo, len_hi, angles, seed, dev, layers=4):
    from crystalframer_b200.latticeformer import Latticeformer, ModelParams
    torch.manual_seed(seed)
    model = Latticeformer(ModelParams(num_layers=layers, frame_method="weighted_pca", value_pe_angle_real=angles)).to(dev).train()

    def batch(b):
        y = np.random.default_rng(seed).normal(size=(len(b.sizes), 1)).astype(np.float32)
        return data.host_batch(b, y, pinned=False).to(dev, non_blocking=False)
    with torch.no_grad():
        model(batch(synth.make_batch(32, 77)))              # the first forward measures the coefficient statistics
    return model, batch(synth.make_batch(crystals, seed, size_dist="uniform", size_lo=lo, size_hi=hi, len_lo=len_lo, len_hi=len_hi))


def _predict(model, tb, seed):
    np.random.seed(seed)
    torch.manual_seed(seed)
    return model(tb)


def outputs(spec, dev):
    """Predictions of a training forward, as the bits of their floats."""
    model, tb = _model_and_batch(*spec, dev)
    return _predict(model, tb, spec[-1]).detach().cpu().numpy().ravel().view(np.uint32).tolist()


@pytest.mark.parametrize("row", range(len(BATCHES)))
def test_training_forward_repeats_to_the_bit(row):
    with open(GOLDEN) as f:
        want = json.load(f)[row]
    assert outputs(BATCHES[row], cuda()) == want


# small cells and Gaussians three times as wide: ranges beyond the lists beside ranges within; recorded before the sums of
# tasks with lists were formed in tiles
WIDE = [(6, 4, 40, 4.0, 12.0, 32, 6), (8, 1, 64, 3.0, 15.0, 16, 11), (12, 4, 40, 4.0, 12.0, 64, 18)]
WIDE_GOLDEN = os.path.join(os.path.dirname(GOLDEN), "weighted_pca_wide_outputs.json")


def wide_outputs(spec, dev):
    model, tb = _model_and_batch(*spec, dev, layers=2)
    with torch.no_grad():
        for n, p in model.named_parameters():
            if "lattice_pos" in n:
                p.mul_(3.0)
    return _predict(model, tb, spec[-1]).detach().cpu().numpy().ravel().view(np.uint32).tolist()


@pytest.mark.parametrize("row", range(len(WIDE)))
def test_training_forward_of_wide_gaussians_repeats_to_the_bit(row):
    with open(WIDE_GOLDEN) as f:
        want = json.load(f)[row]
    assert wide_outputs(WIDE[row], cuda()) == want


@pytest.mark.parametrize("sizes", [(1, 2, 3, 5, 31, 32, 33, 65)])
@pytest.mark.parametrize("angles", [16, 64])
@pytest.mark.parametrize("chunked", [False, True])
@pytest.mark.parametrize("listed", [False, True])
def test_pair_after_pair_against_tiles(sizes, angles, chunked, listed, monkeypatch):
    """One layer, whose frames both routes share to the bit: what is left is the rounding of sums of a few hundred terms,
    each route 4 sqrt(terms) 2^-24 = 5e-6 at most, and the dense layers behind it at most double that."""
    dev = cuda()
    monkeypatch.setattr(fused_layer, "SPLIT_TASKS", chunked)
    if not listed:
        from crystalframer_b200.cuda_funcs import common
        monkeypatch.setattr(common, "pair_list_fits", lambda *a: False)
    model, _ = _model_and_batch(1, 4, 5, 4.0, 8.0, angles, 3, dev, layers=1)
    b = synth.concat([synth.make_batch(1, 40 + n, size_dist="uniform", size_lo=n, size_hi=n, len_lo=3.0, len_hi=10.0) for n in sizes])
    tb = data.host_batch(b, np.zeros((len(sizes), 1), np.float32), pinned=False).to(dev, non_blocking=False)
    seen = []
    taps = []
    monkeypatch.setattr(fused_layer, "FRAME_TAP", taps)
    orig = fused_layer.FusedEncoderLayerFunc.forward

    def spy(ctx, *a):
        out = orig(ctx, *a)
        seen.append(out.detach().clone())
        return out
    monkeypatch.setattr(fused_layer.FusedEncoderLayerFunc, "forward", staticmethod(spy))
    _predict(model, tb, 5)
    with torch.no_grad():
        _predict(model, tb, 5)
    assert len(seen) == 2 and torch.equal(taps[0], taps[1])
    err = (seen[0].double() - seen[1].double()).abs().max() / seen[1].double().square().mean().sqrt()
    assert err < 2e-5, float(err)
