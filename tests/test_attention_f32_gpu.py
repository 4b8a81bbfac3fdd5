"""The 32-bit attention kernel at the sizes its words and columns a thread change at, from aligned and from odd addresses."""

import pytest
import torch

from test_gizulorn_gpu import hide_the_passed
from test_pabavik_gpu import attention_problem, run_attention

from freetoken_b200.kernels import ops

pytestmark = pytest.mark.gpu
DEV = "cuda"


def odd(x):
    """The same values one element off a 16-byte boundary."""
    return torch.empty(x.numel() + 1, dtype=x.dtype, device=DEV)[1:].view(x.shape).copy_(x)


@pytest.mark.parametrize("D", [16, 48, 64, 80, 128, 144, 256])
@pytest.mark.parametrize("window,keep", [(None, 0), (37, 5)])
@pytest.mark.parametrize("tied", [True, False])
def test_heads_of_every_width(D, window, keep, tied):
    for segs, kw in (([(70, 70), (1, 33), (1, 32), (17, 200), (2, 2)], {}), ([(5, 700)], dict(force_split=True))):
        problem = attention_problem(torch.float32, 6, 2, D, 16, segs, seed=6)
        if window:
            problem = hide_the_passed(problem, window, keep, 16)
        q, ks, vs, bt, seg = problem
        vs = ks if tied else vs
        out, want, _ = run_attention(torch.float32, 6, 2, D, 16, segs, 16, window, None, problem=(q, ks, vs, bt, seg), keep_first=keep, **kw)
        # sums of at most D and of 700 terms in 32 bits: a few units of 2^-24 of values of size up to 4
        torch.testing.assert_close(out, want, rtol=2e-5, atol=2e-5)
        ko = odd(ks)
        off, _, _ = run_attention(torch.float32, 6, 2, D, 16, segs, 16, window, None, problem=(odd(q), ko, ko if tied else odd(vs), bt, seg),
                                  keep_first=keep, **kw)
        assert torch.equal(off, out)
    assert ops.read_status() == 0
