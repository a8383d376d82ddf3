"""Item boundaries of the persistent backward: items of one query tile behind longer ones (causal), repeated until a race
between the product chains of neighbouring items would show as a different dk or dv."""
import pytest
import torch

from flashbias_b200 import _lib, check_device_status
from flashbias_b200.flash_bias import flash_bias_backward, flash_bias_forward
from tests.helpers import kernels_taken

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


# (head_dim 16: scale 1/4, a power of two; 32: a split scale)
@pytest.mark.parametrize("S,D,R,causal,kernel", [
    (2560, 32, 16, False, "bwd_persistent"), (2561, 32, 16, False, "bwd_two_stream"), (5120, 32, 16, True, "bwd_persistent"),
    (512, 32, 17, False, "bwd_persistent"), (513, 32, 17, False, "bwd_two_stream"), (1024, 32, 32, True, "bwd_persistent"),
    (896, 16, 17, False, "bwd_persistent"), (897, 16, 17, False, "bwd_two_stream"), (1793, 16, 32, True, "bwd_two_stream")])
def test_query_tiles_up_to_which_the_persistent_form_is_taken(S, D, R, causal, kernel):
    q, k, v = (torch.empty(16, S, 16, D, dtype=torch.bfloat16, device="cuda") for _ in range(3))
    qb, kb = (torch.empty(1, S, 16, R, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    assert kernels_taken(q, k, v, qb, kb, causal=causal)[1] == kernel
