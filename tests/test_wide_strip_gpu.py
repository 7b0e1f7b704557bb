"""Small-M MatMul whose K splits are added inside a thread-block cluster."""
import pytest

pytestmark = pytest.mark.gpu


# rows 1 .. 16 (every register block), columns with a partial strip, K from one row to many rounds: no split, a cluster, more splits than one takes
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("k,n", [(1, 128), (63, 260), (129, 132), (777, 1000), (2048, 2052), (4100, 516), (2049, 8196)])
def test_wide_strip(cuda, m, k, n):
    import torch
    from rmlk_b200 import kernels as K
    g = torch.Generator(device=cuda)
    g.manual_seed(m + k + n)
    a, b = torch.randn(m, k, device=cuda, generator=g), torch.randn(k, n, device=cuda, generator=g)
    want, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    ws = torch.empty(max(16, K.matmul_workspace_bytes(1, m, n, k)), dtype=torch.uint8, device=cuda)
    for workspace in (None, ws):
        got = K.matmul(a, b, out=torch.full((m, n), float("nan"), device=cuda), workspace=workspace)
        # fp32 FMA chains of at most K terms: K 2^-24 of the magnitudes at the very worst, some sqrt(K) of it in practice
        assert bool(((got.double() - want).abs() <= mag * 2.0 ** -24 * (k ** 0.5 * 2 + 8)).all())
        assert torch.equal(got, K.matmul(a, b, workspace=workspace))  # added in a fixed order
