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


def _check_f32(a, b, got):
    import torch
    want, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    k = a.shape[1]
    # the operands hold 22 bits (2^-22 for either one and for the dropped product of the low parts), sums lose one truncated fp32
    # addition per 16 products
    bound = mag * (3 * 2.0 ** -22 + 2.0 ** -23 * (k / 16 + 2))
    assert bool(((got.double() - want).abs() <= bound).all()), float(((got.double() - want).abs() / bound).max())


# what the splitting pass pads (K to 64, N to 128), row tiles, K splits; sizes that no other tensor-core kernel takes
@pytest.mark.parametrize("m", [256, 300, 513])
@pytest.mark.parametrize("n,k", [(64, 64), (100, 65), (129, 200), (512, 2048), (1000, 777), (3072, 2048)])
def test_f32_split(cuda, m, n, k):
    import torch
    from rmlk_b200 import kernels as K
    g = torch.Generator(device=cuda)
    g.manual_seed(m + n + k)
    a = torch.randn(m, k, device=cuda, generator=g)
    b = torch.randn(k, n, device=cuda, generator=g) * 0.02
    ws = torch.empty(K.matmul_workspace_bytes(1, m, n, k), dtype=torch.uint8, device=cuda)
    _check_f32(a, b, K.matmul(a, b, workspace=ws))


def test_f32_split_scales(cuda):
    """Rows and columns of very different size, values far below their row's largest, zeros, the ends of the exponent range."""
    import torch
    from rmlk_b200 import kernels as K
    m, n, k = 320, 256, 512
    a = torch.randn(m, k, device=cuda) * torch.exp2(torch.randint(-60, 60, (m, 1), device=cuda).float())
    b = torch.randn(k, n, device=cuda) * torch.exp2(torch.randint(-60, 60, (1, n), device=cuda).float())
    a *= torch.exp2(-torch.rand(m, k, device=cuda) * 24)   # a range of 2^24 inside every row
    b *= torch.exp2(-torch.rand(k, n, device=cuda) * 24)
    a[5] = 0
    b[:, 7] = 0
    a[9] = 2.0 ** -120
    a[11] = 2.0 ** 100
    b[:, 13] = 2.0 ** -130   # denormal
    ws = torch.empty(K.matmul_workspace_bytes(1, m, n, k), dtype=torch.uint8, device=cuda)
    got = K.matmul(a, b, workspace=ws)
    want, mag = a.double() @ b.double(), a.double().abs() @ b.double().abs()
    bound = mag * (3 * 2.0 ** -22 + 2.0 ** -23 * (k / 16 + 2)) + 2.0 ** -125
    fine = want.abs() < 2.0 ** 127
    assert bool(((got.double() - want).abs() <= bound)[fine].all())


@pytest.mark.parametrize("n,k", [(200, 100), (256, 512)])
def test_f32_split_non_finite_and_extreme(cuda, n, k):
    """Infinities and NaNs come out where fp32 puts them; scales whose product is in range although one alone takes the sum out of it."""
    import torch
    from rmlk_b200 import kernels as K
    m = 300
    a, b = torch.randn(m, k, device=cuda), torch.randn(k, n, device=cuda)
    a[:, 3] = a[:, 3].abs() + 1.0
    b[3] = 1.0                    # exact in f16: its low part is zero
    a[4, 3] = float("inf")
    a[5, 3] = float("-inf")
    a[6, 9] = float("nan")
    a[7, 3], a[7, 8] = float("inf"), float("-inf")
    b[8] = 2.0
    b[11, 17] = float("-inf")
    a[:, 11] = 1.0
    a[20] *= 2.0 ** -120
    b[:, 30] *= 2.0 ** 118
    a[21] *= 2.0 ** 110
    b[:, 31] *= 2.0 ** -122
    ws = torch.empty(K.matmul_workspace_bytes(1, m, n, k), dtype=torch.uint8, device=cuda)
    got = K.matmul(a, b, workspace=ws).double()
    want = a.double() @ b.double()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    inf = torch.isinf(want)
    assert bool((got[inf] == want[inf]).all())
    fine = torch.isfinite(want) & (want.abs() < 2.0 ** 127)
    mag = torch.nan_to_num(a.double().abs(), posinf=0.0) @ torch.nan_to_num(b.double().abs(), posinf=0.0)
    bound = mag * (3 * 2.0 ** -22 + 2.0 ** -23 * (k / 16 + 2)) + 2.0 ** -125
    assert bool(((got - want).abs() <= bound)[fine].all())


@pytest.mark.parametrize("m,k,n", [(1000, 777, 1003), (300, 4100, 260), (2048, 2050, 516), (512, 1025, 100)])
def test_f32_split_ragged_accuracy(cuda, m, k, n):
    """Sizes that FMA chains would otherwise take are no less accurate than those: 2-norm error at most that of fp32 sums over K."""
    import torch
    from rmlk_b200 import kernels as K
    g = torch.Generator(device=cuda)
    g.manual_seed(k)
    a, b = torch.randn(m, k, device=cuda, generator=g), torch.randn(k, n, device=cuda, generator=g) * 0.02
    ws = torch.empty(K.matmul_workspace_bytes(1, m, n, k), dtype=torch.uint8, device=cuda)
    want = a.double() @ b.double()
    # the same call without workspace runs on the FMA kernel
    split, fma = K.matmul(a, b, workspace=ws).double(), K.matmul(a, b).double()
    assert float((split - want).norm()) <= float((fma - want).norm())
