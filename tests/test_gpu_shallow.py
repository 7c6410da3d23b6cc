"""Updates of little k, which C's traffic bounds: the plain kernel that brings C to L2 ahead and streams its stores,
and FMM calls of the abc type whose units are tiles with all their products.

Plain tolerance: a sum of k products of |a|, |b| <= 1 added to c has error at most (k + 1) u per unit of
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


def matrix(rows, cols, ld, off, gen):
    """(view, flat): column-major rows x cols in a buffer of NaN, its base `off` doubles past 16 bytes."""
    flat = torch.full((off + ld * cols + 2,), float("nan"), dtype=torch.float64, device="cuda")
    v = torch.as_strided(flat, (rows, cols), (1, ld), off)
    v.copy_(torch.rand(rows, cols, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1)
    return v, flat


# one round of CTAs and less, several rounds (tiles of another round are prefetched), partial tiles
@pytest.mark.parametrize("m,n", [(1, 1), (63, 130), (2049, 1031), (3000, 2900)])
@pytest.mark.parametrize("k", [1, 8, 17, 48, 49, 128, 129])
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (2, 1), (3, 0)])
def test_plain_updates_of_little_k(lib, m, n, k, pad, off):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    (A, _), (B, _), (C, flat) = (matrix(r, c, r + pad, off, gen) for r, c in ((m, k), (k, n), (m, n)))
    C0 = C.clone()
    rt.plain_gemm(A, B, C)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    over = (C - (C0 + A @ B)).abs() - 2 * (k + 2) * U * (A.abs() @ B.abs() + C0.abs())
    assert torch.isfinite(C).all() and over.max().item() <= 0
    assert int(torch.isnan(flat).sum()) == flat.numel() - m * n  # nothing outside C was written


@pytest.mark.parametrize("algs,shape", [
    (["222"], (7700, 7712, 512)),     # blocks of 61 x 61 tiles, eight rounds of three CTAs on 148 SMs; ks = 256
    (["222"], (7700, 7713, 511)),     # odd columns: every fringe
    (["232"], (7720, 7700, 250)),
    (["333"], (11700, 11600, 500)),   # nine blocks
], ids=str)
@pytest.mark.parametrize("small_cap", [False, True])  # with the cap below the products they cannot be stored
def test_units_of_all_products_of_a_tile(lib, algs, shape, small_cap):
    """Every schedule adds the same products in the same order: the ab type's bits."""
    m, n, k = shape
    plan = rt.Plan.from_levels(algs, [1])
    gen = torch.Generator(device="cuda").manual_seed(k)
    A, B, C = (rt.colmajor(r, c, device="cuda").uniform_(-1, 1, generator=gen) for r, c in ((m, k), (k, n), (m, n)))
    want = C.clone(memory_format=torch.preserve_format)
    rt.fmm_gemm(plan, A, B, want, "ab")
    sums = rt.last_workspace_bytes()
    prev = rt.set_workspace_limit(sums + 1024) if small_cap else None
    try:
        rt.fmm_gemm(plan, A, B, C, "abc")
    finally:
        if small_cap:
            rt.set_workspace_limit(prev)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    assert torch.equal(C, want)
    plan.close()
