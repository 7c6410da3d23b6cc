"""Plain updates of deep k at the sizes where the part count and the tile side change: two parts (from k = 2048, up to
eight 64 x 64 tiles per SM of 148), one part where the tiles run together, and batches, which add the same parts.

Tolerance: a sum of k products of |a|, |b| <= 1 added to c has error at most (k + 1) u per unit of
|A||B| + |c| in any order; the result and the FP64 reference each have that much.
"""
import pytest

torch = pytest.importorskip("torch")

from fmm_gen_b200 import build, runtime as rt  # noqa: E402

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return rt.load_library()


@pytest.mark.parametrize("m,n", [
    (490, 511),    # 256 tiles of 32: two parts of their own
    (577, 575),    # 361: one part but for the depth
    (1088, 1088),  # 289 of 64: two per SM at the same time
    (1344, 1344),  # 441: three
    (1409, 1407),  # 529
    (2176, 2240),  # 1190: past eight per SM
])
@pytest.mark.parametrize("k", [2047, 2048, 2063])
@pytest.mark.parametrize("pad", [0, 1])
def test_deep_updates(lib, m, n, k, pad):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)

    def matrix(rows, cols):
        flat = torch.full(((rows + pad) * cols,), float("nan"), dtype=torch.float64, device="cuda")
        v = torch.as_strided(flat, (rows, cols), (1, rows + pad), 0)
        v.copy_(torch.rand(rows, cols, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1)
        return v

    A, B, C = matrix(m, k), matrix(k, n), matrix(m, n)
    C0, batch_C = C.clone(), rt.colmajor(m, n, device="cuda").copy_(C)
    rt.plain_gemm(A, B, C)
    rt.batch_submit([None], [A], [B], [batch_C])
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    over = (C - (C0 + A @ B)).abs() - 2 * (k + 2) * U * (A.abs() @ B.abs() + C0.abs())
    assert torch.isfinite(C).all() and over.max().item() <= 0
    assert torch.equal(C, batch_C)
