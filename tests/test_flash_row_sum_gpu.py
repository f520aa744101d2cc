"""Order in which the attention forward adds up a row's probabilities."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sq,sk", [(1, 128), (300, 128)])
def test_row_sum_runs_over_key_pairs_in_order(sq, sk):
    """One key of weight 1 and 127 of weight p, 0.7 * 2^-24 < p < 0.78 * 2^-24.  In fp32 a pair of the small ones (1.4 .. 1.56 * 2^-24)
    added to 1 rounds up to one unit 2^-23, while one of them alone is rounded away.  Keys taken pair after pair give
    1 + 63 * 2^-23; sums of even and odd keys that meet at the end give about 1 + 35 * 2^-23.  The logarithm's absolute error near 1 is
    2^-21.4."""
    from mindspeed_b200.ops import gemm as G
    from mindspeed_b200.ops.flash_sm100_impl import flash_fwd
    q, k = torch.zeros(sq, 1, 1, 128, device="cuda"), torch.zeros(sk, 1, 1, 128, device="cuda")
    q[..., 0] = 1.0
    k[1:, ..., 0] = -24.375                                  # scores in units of log 2: exp(score * log 2) = 0.77 * 2^-24
    _, lse = flash_fwd(q.bfloat16(), k.bfloat16(), torch.ones_like(k).bfloat16(), False, math.log(2.0))
    torch.cuda.synchronize()
    G.check_status()
    assert (lse.double() - math.log1p(63 * 2.0 ** -23)).abs().max().item() < 5e-7
