"""Squeeze-and-excite module: the CUDA launch against the oracle on the reference's ten shapes
(cpp/efficientnet/test_efficientnet_se_module.py:13-23) and on shapes it does not dispatch."""
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from oracle import souffle_oracle as so  # noqa: E402

pytestmark = pytest.mark.gpu

REF_SHAPES = [(1, 112, 112, 32, 8), (1, 56, 56, 96, 4), (1, 56, 56, 144, 6), (1, 28, 28, 144, 6), (1, 28, 28, 240, 10),
              (1, 14, 14, 240, 10), (1, 14, 14, 480, 20), (1, 14, 14, 672, 28), (1, 7, 7, 672, 28), (1, 7, 7, 1152, 48)]


def _case(b, h, w, c, r, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(b, c, h, w, generator=g)
    wr = torch.randn(r, c, generator=g) * 0.2
    we = torch.randn(c, r, generator=g) * 0.5
    return x, wr, we


@pytest.mark.parametrize("shape", REF_SHAPES + [(2, 10, 13, 40, 5), (3, 1, 1, 8, 2), (1, 224, 224, 3, 1)])
def test_se_module_matches_oracle(shape):
    from souffle_models_b200 import efficientnet
    b, h, w, c, r = shape
    x, wr, we = _case(b, h, w, c, r, 7 + c)
    pooled, out = efficientnet.se_module(x.cuda(), wr.cuda(), we.cuda())
    want_pooled, want = so.se_module(x, wr, we)
    assert (pooled.cpu() - want_pooled).abs().max() < 1e-5
    assert (out.cpu() - want).abs().max() < 2e-5
    pooled2, out2 = efficientnet.se_module(x.cuda(), wr.cuda(), we.cuda())       # the workspace cleans itself up
    assert torch.equal(out, out2) and torch.equal(pooled, pooled2)


def test_drop_in_entry_returns_the_reference_shapes():
    sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "shims"))
    import efficientnet_se_module_binding as ref_name
    x, wr, we = _case(1, 14, 14, 240, 10, 3)
    pooled, out = ref_name.torch_dispatch_efficientnet_se_module_v2_short_cut_fused(x.cuda(), wr.cuda(), we.cuda(), 2)
    assert tuple(pooled.shape) == (1, 240) and tuple(out.shape) == (1, 14, 14, 240)
    _, want = so.se_module(x, wr, we)
    assert (out.cpu().reshape(1, 240, 14, 14) - want).abs().max() < 2e-5       # NCHW memory under the declared shape


def test_bad_arguments():
    from souffle_models_b200 import efficientnet
    x, wr, we = _case(1, 7, 7, 16, 4, 1)
    with pytest.raises(ValueError):
        efficientnet.se_module(x.cuda().half(), wr.cuda(), we.cuda())
    with pytest.raises(ValueError):
        efficientnet.se_module(x.cuda(), we.cuda(), wr.cuda())
    with pytest.raises(Exception):
        efficientnet.se_module(x.cuda(), torch.zeros(80, 16).cuda(), torch.zeros(16, 80).cuda())      # reduce > 64


@pytest.mark.parametrize("shape", [(5, 9, 7, 33, 64), (40, 56, 56, 144, 6), (3, 150, 149, 7, 3), (2, 8, 8, 4096, 64), (1, 1, 5, 2, 1)])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_slices_at_every_alignment(shape, shift):
    """Odd image sizes and inputs that start off a 16-byte boundary (edges of the 16-byte pieces), slices that fit shared
    memory and that do not, reduce weights too large to stage.  Bound: fp32 sums of n terms are within 1e-6 of the
    largest term for the orders compared here."""
    from souffle_models_b200 import efficientnet
    b, h, w, c, r = shape
    x, wr, we = _case(b, h, w, c, r, 11 + c)
    we = we / r ** 0.5
    flat = torch.zeros(x.numel() + 8)
    flat[shift:shift + x.numel()] = x.reshape(-1)
    xin = flat.cuda()[shift:shift + x.numel()].view(b, c, h, w)
    pooled, out = efficientnet.se_module(xin, wr.cuda(), we.cuda())
    want_pooled, want = so.se_module(x, wr, we)
    assert (pooled.cpu() - want_pooled).abs().max() < 1e-5
    assert (out.cpu() - want).abs().max() < 2e-5


@pytest.mark.parametrize("shape", [(1, 7, 7, 1152, 48), (2, 14, 14, 672, 28), (8, 14, 14, 240, 10), (2, 8, 8, 4096, 64), (3, 3, 3, 1801, 64),
                                   (5, 7, 7, 101, 64)])
@pytest.mark.parametrize("shift", [0, 1])
def test_reduce_weights_staged_and_not_at_every_alignment(shape, shift):
    """Reduce weights that fill shared memory to the last hundred bytes, that do not fit, that start off a 16-byte boundary,
    rows that are no multiple of four; runs of items that divide an image and runs that cannot.  Bound of the test above."""
    from souffle_models_b200 import efficientnet
    b, h, w, c, r = shape
    x, wr, we = _case(b, h, w, c, r, 23 + c)
    we = we / r ** 0.5
    flat = torch.zeros(wr.numel() + 4)
    flat[shift:shift + wr.numel()] = wr.reshape(-1)
    pooled, out = efficientnet.se_module(x.cuda(), flat.cuda()[shift:shift + wr.numel()].view(r, c), we.cuda())
    want_pooled, want = so.se_module(x, wr, we)
    assert (pooled.cpu() - want_pooled).abs().max() < 1e-5
    assert (out.cpu() - want).abs().max() < 2e-5


@pytest.mark.parametrize("shape", [(1, 3, 3, 2368, 64), (1, 3, 3, 2369, 64), (1, 32, 32, 2368, 7), (1, 25, 41, 2368, 7), (300, 5, 5, 2, 3),
                                   (3000, 5, 5, 2, 3), (12000, 1, 3, 1, 64), (20, 7, 73, 160, 9), (20, 16, 32, 160, 9), (33, 19, 27, 37, 5)])
@pytest.mark.parametrize("shift", [0, 1])
def test_one_slice_a_warp_and_many_images_a_block(shape, shift):
    """As many slices as a B200 has warps, one more, a slice of 1024 floats and the next longer one (kept in registers or in
    shared memory); blocks that meet two images, twenty, more than are worked on together; images just under and over the
    512 floats from where they are added one by one.  Bound of the tests above; the same call twice gives the same bits."""
    from souffle_models_b200 import efficientnet
    b, h, w, c, r = shape
    x, wr, we = _case(b, h, w, c, r, 31 + c)
    wr, we = wr * (32.0 / c) ** 0.5 if c > 32 else wr, we / r ** 0.5
    flat = torch.zeros(x.numel() + 4)
    flat[shift:shift + x.numel()] = x.reshape(-1)
    xin, wr_d, we_d = flat.cuda()[shift:shift + x.numel()].view(b, c, h, w), wr.cuda(), we.cuda()
    pooled, out = efficientnet.se_module(xin, wr_d, we_d)
    want_pooled, want = so.se_module(x, wr, we)
    assert (pooled.cpu() - want_pooled).abs().max() < 1e-5
    assert (out.cpu() - want).abs().max() < 2e-5
    pooled2, out2 = efficientnet.se_module(xin, wr_d, we_d)
    assert torch.equal(out, out2) and torch.equal(pooled, pooled2)
