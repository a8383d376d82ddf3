"""Item boundaries of the persistent backward: items of one query tile behind longer ones (causal), repeated until a race
between the product chains of neighbouring items would show as a different dk or dv."""
import pytest
import torch

from flashbias_b200 import _lib, check_device_status
from flashbias_b200.flash_bias import flash_bias_backward, flash_bias_forward

pytestmark = pytest.mark.gpu


# (B, H, Sq, Sk, R, causal): last items of one query tile; items of one tile only; packed rank 64
@pytest.mark.parametrize("B,H,Sq,Sk,R,causal", [(8, 40, 512, 512, 8, True), (64, 12, 100, 300, 4, False), (4, 40, 384, 384, 24, True)])
def test_repeated_persistent_backward_is_bit_identical(B, H, Sq, Sk, R, causal):
    g = torch.Generator().manual_seed(B + Sq)
    q, do = (torch.randn(B, Sq, H, 32, generator=g).bfloat16().cuda() for _ in range(2))
    k, v = (torch.randn(B, Sk, H, 32, generator=g).bfloat16().cuda() for _ in range(2))
    qb, kb = ((torch.randn(1, S, H, R, generator=g) * 0.5).bfloat16().cuda() for S in (Sq, Sk))
    o, lse, sc = flash_bias_forward(q, k, v, qb, kb, None, causal, None)
    args = (do, q, k, v, o, qb, kb, lse, None, causal, sc)
    want = flash_bias_backward(*args, flags=_lib.FB_FLAG_BWD_ONE_ITEM)
    for _ in range(100):
        got = flash_bias_backward(*args, flags=_lib.FB_FLAG_BWD_PERSISTENT)
        assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    torch.cuda.synchronize()
    check_device_status()
