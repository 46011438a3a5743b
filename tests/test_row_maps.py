"""The multiply-high quotients of the Swin row maps are exact over the sizes a plan takes (host arithmetic: the kernel
uses the same 32-bit formula), and a token grid past that range goes through the plain divisions."""
import pytest
import torch

from oracle import souffle_oracle as so


def _magic(d):
    return 0 if d <= 1 else (2 ** 32 + d - 1) // d


@pytest.mark.parametrize("res,win,rows", [(7, 7, 1 << 20), (14, 7, 1 << 20), (56, 7, 1 << 20), (64, 8, (1 << 20) - 4096), (120, 8, 291600),
                                          (252, 7, 63504)])
def test_quotients_are_exact(res, win, rows):
    import numpy as np
    nwr = res // win
    assert rows * res * res < 2 ** 32            # the rule by which the host hands out a multiplier at all
    for d, top in ((res * res, rows), (res, res * res), (win, res), (nwr * nwr, rows // 64 + 1), (nwr, nwr * nwr), (win, 64)):
        if d > 1:
            n = np.arange(top, dtype=np.uint64)
            assert ((n * np.uint64(_magic(d))) >> np.uint64(32) == n // np.uint64(d)).all(), (d, top)


@pytest.mark.gpu
@pytest.mark.parametrize("res,window,shift,dim", [(256, 8, 3, 128), (8, 8, 0, 128), (21, 7, 2, 128), (35, 7, 3, 256), (7, 7, 0, 1024)])
def test_block_on_grids_at_the_ends_of_the_range(res, window, shift, dim):
    """256 x 256 tokens: no exact 32-bit multiplier; one window; odd numbers of windows, with one (window, head) per
    attention item (9 x 4, 1 x 32 problems) and with two by two (25 x 8: the last item has a single window)."""
    from souffle_models_b200 import swin
    cfg = so.SwinConfig(res=res, dim=dim, heads=dim // 32, window=window)
    p = so.make_swin_params(cfg, 5, zero_bias=False)
    x = torch.randn(res * res, dim, generator=torch.Generator().manual_seed(res)).half()
    blk = swin.SwinBlock(1, res, dim, dim // 32, window, shift, {k: v.cuda() for k, v in p.items()})
    y = blk.forward(x.cuda())
    blk.status()
    want = so.swin_block(cfg, x, p, shift)
    # the bound of the block test (fp16 storage of values up to ~6)
    assert (y.float().cpu() - want).abs().max() < 1.5e-2 and (y.float().cpu() - want).pow(2).mean().sqrt() < 2e-3
