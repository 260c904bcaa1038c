"""Sizes that the kernel library refuses before it launches anything."""
import pytest

from monarch_b200.ops import kernels as K

BAD_ARGUMENTS = 1001


@pytest.mark.parametrize("call", [
    lambda l: l.mb200_rope_inplace(0, 0, 0, 4, 4, 0, 64, 64, 0, 0),      # no head to rotate
    lambda l: l.mb200_rope_inplace(0, 0, 0, 4, 4, 1, 0, 64, 0, 0),
    lambda l: l.mb200_rope_inplace(0, 0, 0, 4, 4, 1, 40, 64, 0, 0),
    lambda l: l.mb200_swiglu_fwd(0, 0, 4, 0, 0),
    lambda l: l.mb200_swiglu_bwd(0, 0, 0, 4, 0, 0),
    lambda l: l.mb200_swiglu_fwd(0, 0, 4, 12, 0),
    lambda l: l.mb200_embedding_bwd(0, 0, 0, 4, 0, 0),
    lambda l: l.mb200_embedding_bwd(0, 0, 0, 4, 3, 0),
    lambda l: l.mb200_rmsnorm_bwd(0, 0, 0, 0, 0, 0, 0, 0, 0, 4, 8200, 0, 0),
])
def test_refused(call):
    assert call(K.lib()) == BAD_ARGUMENTS
