"""The multiply-high quotients of the Swin row maps are exact over the sizes a plan takes (the library's own multipliers,
with the kernel's multiply-high in 64 bits), and a token grid past that range goes through the plain divisions."""
import os
import shutil
import subprocess

import pytest
import torch

from oracle import souffle_oracle as so

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "souffle_models_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include <cstdlib>
#include "stage_program.h"
int main(int argc, char** argv) {       // pairs: divisor, number of numerators
  for (int i = 1; i + 1 < argc; i += 2) {
    const uint32_t d = (uint32_t)atol(argv[i]), top = (uint32_t)atol(argv[i + 1]), mg = souffle::fast_div_magic(d);
    for (uint32_t n = 0; n < top; ++n)
      if ((d <= 1 ? n : (uint32_t)(((uint64_t)n * mg) >> 32)) != n / d) { printf("%u / %u", n, d); return 1; }
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def quotients(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    tmp = tmp_path_factory.mktemp("quotients")
    (tmp / "q.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-O2", "-I", CSRC, "-o", str(tmp / "q"), str(tmp / "q.cpp")], check=True)
    return str(tmp / "q")


@pytest.mark.parametrize("res,win,rows", [(7, 7, 1 << 20), (14, 7, 1 << 20), (56, 7, 1 << 20), (64, 8, (1 << 20) - 4096), (120, 8, 291600),
                                          (252, 7, 63504)])
def test_quotients_are_exact(quotients, res, win, rows):
    nwr = res // win
    assert rows * res * res < 2 ** 32            # the rule by which the host hands out a multiplier at all
    pairs = ((res * res, rows), (res, res * res), (win, res), (nwr * nwr, rows // 64 + 1), (nwr, nwr * nwr), (win, 64))
    run = subprocess.run([quotients] + [str(v) for pair in pairs for v in pair], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout


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
