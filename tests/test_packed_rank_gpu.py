"""Forward at the edges of the packed rank 96 (ranks 64 to 97 at head_dim 32), with both scale kinds, masks and ragged tiles,
against the CPU checker."""
import math

import pytest
import torch

from flashbias_b200 import check_device_status
from flashbias_b200.flash_bias import flash_bias_forward
from oracle import flashbias_oracle as orc
from tests.helpers import check_close, kernels_taken

pytestmark = pytest.mark.gpu


# (rank, head_dim, scale (None: split), dtype, masked)
@pytest.mark.parametrize("R,D,scale,dtype,masked", [
    (64, 32, 1.0, torch.float16, False), (65, 32, 1.0, torch.float16, False), (81, 24, 0.25, torch.bfloat16, False),
    (96, 32, 1.0, torch.float16, False), (96, 32, None, torch.bfloat16, False), (96, 32, 1.0, torch.float16, True),
    (97, 32, 1.0, torch.float16, False), (96, 64, 0.125, torch.bfloat16, False)])
def test_forward(R, D, scale, dtype, masked):
    B, H, Sq, Sk = 3, 4, 257, 390
    g = torch.Generator().manual_seed(R + D)
    q = torch.randn(B, Sq, H, D, generator=g).to(dtype)
    k, v = (torch.randn(B, Sk, H, D, generator=g).to(dtype) for _ in range(2))
    qb, kb = (torch.tanh(torch.randn(1, S, H, R, generator=g)).mul(0.3).to(dtype) for S in (Sq, Sk))
    mask = torch.where(torch.rand(B, 1, Sq, Sk, generator=g) < 0.3, -100.0, 0.0) if masked else None
    scale = scale or 1.0 / math.sqrt(D)
    dev = [t.cuda() for t in (q, k, v, qb, kb)] + [mask.cuda() if masked else None]
    assert kernels_taken(*dev)[0] == "fwd_tiled"
    o, _, _ = flash_bias_forward(*dev, False, scale)
    torch.cuda.synchronize()
    check_device_status()
    o_ref, _ = orc.attention_forward(*(t.float() for t in (q, k, v, qb, kb)), mask, False, scale, dtype=torch.float64)
    check_close("packed_rank/R%dD%d%s" % (R, D, "m" if masked else ""), o, o_ref, dtype)
