"""What calls allocate: the cap on one call's operand workspace."""
import pytest

torch = pytest.importorskip("torch")

from fmm_gen_b200 import algebra, build, runtime as rt  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return rt.load_library()


def uniform(rows, cols, gen):
    return rt.colmajor(rows, cols, device="cuda").uniform_(-1, 1, generator=gen)


def one_product(plan, m, n, k):
    """Bytes of one product's operand sums: what a cap below them is exceeded by."""
    p = algebra.partition(m, n, k, plan.dims)
    return 8 * (p.ms + p.ns) * ((p.ks + 7) // 8 * 8)


@pytest.mark.parametrize("algs,shape,limit", [
    (["222"], (1024, 1024, 1024), 16 << 20),       # sums 21 MB, products 14.7 MB
    (["222"], (400, 380, 6001), 8 << 20),          # 65 MB, 2.1 MB; one product's sums are 9.3 MB
    (["222", "333"], (528, 528, 2000), 12 << 20),  # 76 MB, 10 MB
], ids=str)
def test_cap_holds_where_the_products_alone_would_fit(lib, algs, shape, limit):
    """Few tiles and deep k: the products fit the cap, their operand sums do not."""
    m, n, k = shape
    gen = torch.Generator(device="cuda").manual_seed(k)
    plan = rt.Plan.from_levels(algs, [1] * len(algs))
    A, B, C = uniform(m, k, gen), uniform(k, n, gen), uniform(m, n, gen)
    whole = C.clone(memory_format=torch.preserve_format)
    rt.fmm_gemm(plan, A, B, whole)
    assert rt.last_workspace_bytes() > limit
    prev = rt.set_workspace_limit(limit)
    try:
        rt.fmm_gemm(plan, A, B, C)
        assert 0 < rt.last_workspace_bytes() <= max(limit, one_product(plan.algebra, *shape))
    finally:
        rt.set_workspace_limit(prev)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    assert torch.equal(C, whole)
    plan.close()
