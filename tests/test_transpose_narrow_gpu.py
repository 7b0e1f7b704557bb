"""Transposes of matrices with a narrow side."""
import itertools

import pytest

pytestmark = pytest.mark.gpu


# sides on both sides of the 16-wide tiles, in every order of the dims
@pytest.mark.parametrize("shape", [(3, 5, 16, 64), (2, 3, 64, 16), (7, 1, 17, 33), (2, 2, 16, 33), (1, 3, 33, 16), (4, 31, 8, 65), (2, 70, 3, 15)])
@pytest.mark.parametrize("dtype", ["uint8", "float16", "float32", "int64"])
def test_transpose_narrow(cuda, shape, dtype):
    import torch
    from rmlk_b200 import kernels as K
    x = torch.randint(0, 200, shape, device=cuda).to(getattr(torch, dtype))
    for perm in itertools.permutations(range(4)):
        assert torch.equal(K.transpose(x, list(perm)), x.permute(perm).contiguous()), perm
