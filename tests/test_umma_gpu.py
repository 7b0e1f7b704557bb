"""MatMul on the f16-kind tensor-core kernel (umma_gemm.cu) against float64."""
import pytest

pytestmark = pytest.mark.gpu


# edges of the row tiles (16 .. 256), of the 128- and 256-column tiles, of the 64-wide k-blocks and of the stage rings, with remainders
@pytest.mark.parametrize("m", [1, 15, 16, 17, 33, 64, 65, 127, 129, 192, 257, 600])
@pytest.mark.parametrize("n,k", [(128, 64), (136, 72), (8, 8), (384, 640), (2048, 1032), (2048, 2048)])
def test_f16(cuda, m, n, k):
    import torch
    from rmlk_b200 import kernels as K
    g = torch.Generator(device=cuda)
    g.manual_seed(m * 131 + n + k)
    a = torch.randn(m, k, device=cuda, generator=g).half()
    b = (torch.randn(k, n, device=cuda, generator=g) * 0.1).half()
    got = K.matmul(a, b).double()
    want, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    # one rounding to f16, and one truncated fp32 addition per 16 products
    bound = want.abs() * 2.0 ** -11 + mag * 2.0 ** -23 * (k / 16 + 1) + 2.0 ** -24
    assert bool(((got - want).abs() <= bound).all()), float(((got - want).abs() / bound).max())


def test_f16_large_tiles(cuda):
    import torch
    from rmlk_b200 import kernels as K
    for m, n, k in ((1024, 8192, 512), (2500, 4360, 200), (4096, 1024, 4096)):
        a = torch.randn(m, k, device=cuda).half()
        b = (torch.randn(k, n, device=cuda) * 0.1).half()
        got = K.matmul(a, b).double()
        want, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
        bound = want.abs() * 2.0 ** -11 + mag * 2.0 ** -23 * (k / 16 + 1) + 2.0 ** -24
        assert bool(((got - want).abs() <= bound).all()), (m, n, k)
