"""Products that update C in ticket order: progress beside another persistent kernel, and the waits' time limit.

Which tickets a call uses depends on its size; the shapes here are 222-1 calls whose products have more tiles than
CTAs run at a time (a ticket per tile) and calls in groups of two products below that (a ticket per tile and C block).
The launches are counted, so that a call that stores its products instead, where nothing waits, fails the test.
"""
import pytest

torch = pytest.importorskip("torch")

from fmm_gen_b200 import build, runtime as rt  # noqa: E402

pytestmark = pytest.mark.gpu
FMM_E_TIMEOUT = -7
FMM_DEBUG_WAIT_LIMIT_NS = 1
FMM_DEBUG_TICKET_FILL = 2

CALLS = [
    ((4096, 4096, 2048), None),      # blocks of 32 x 32 tiles of 64
    ((2048, 2048, 2048), 40 << 20),  # 16 x 16 tiles; two products' sums take 33.6 MB
]


@pytest.fixture(scope="module")
def lib():
    build.build()
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return rt.load_library()


def uniform(rows, cols, g):
    return rt.colmajor(rows, cols, device="cuda").uniform_(-1, 1, generator=g)


@pytest.mark.parametrize("shape,cap", CALLS, ids=["per tile", "per tile and block"])
def test_ticket_ordered_products_beside_a_persistent_kernel(lib, shape, cap):
    """Three split-BF16 launches (persistent, a CTA per SM) on one stream and FMM launches whose units wait for
    tickets on another: all finish, no wait times out, and the bits are those of the call run alone."""
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(k)
    A32 = rt.colmajor(4096, 4096, dtype=torch.float32, device="cuda").normal_(generator=g)
    B32 = rt.colmajor(4096, 4096, dtype=torch.float32, device="cuda").normal_(generator=g)
    Cs = rt.colmajor(4096, 4096, device="cuda").zero_()
    A, B, C0 = uniform(m, k, g), uniform(k, n, g), uniform(m, n, g)
    plan, p2 = rt.Plan.from_levels(["222"], [1]), rt.Plan.from_levels(["222"], [2])
    prev = rt.set_workspace_limit(cap) if cap else None
    try:
        alone = C0.clone(memory_format=torch.preserve_format)
        with rt.KernelTimer() as kt:
            rt.fmm_gemm(plan, A, B, alone, "abc")
        assert kt.count["fmm_products_kernel"] == (4 if cap else 1)
        assert not kt.count.get("fmm_combine_kernel") and not kt.count.get("fmm_scatter_kernel")
        mixed = C0.clone(memory_format=torch.preserve_format)
        s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
        s1.wait_stream(torch.cuda.current_stream())
        s2.wait_stream(torch.cuda.current_stream())
        for _ in range(3):
            with torch.cuda.stream(s1):
                rt.split_gemm(p2, A32, B32, Cs, stream=s1)
            with torch.cuda.stream(s2):
                mixed.copy_(C0)
                rt.fmm_gemm(plan, A, B, mixed, "abc", stream=s2)
        torch.cuda.synchronize()
    finally:
        if cap:
            rt.set_workspace_limit(prev)
    assert lib.fmm_device_status(1) == 0
    assert torch.equal(mixed, alone)


@pytest.mark.parametrize("shape", [(2800, 2816, 64), (600, 616, 264)], ids=["per tile", "per tile and block"])
def test_ticket_waits_run_out(lib, shape):
    """Tickets that nothing releases, of both kinds: the waits end at their limit, the status says so, and the next
    call is right."""
    m, n, k = shape
    g = torch.Generator(device="cuda").manual_seed(m)
    plan = rt.Plan.from_levels(["222"], [1])
    A, B, C = uniform(m, k, g), uniform(k, n, g), uniform(m, n, g)
    want = C.clone(memory_format=torch.preserve_format)
    rt.fmm_gemm(plan, A, B, want, "ab")
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    try:
        assert lib.fmm_debug_set(FMM_DEBUG_WAIT_LIMIT_NS, 50_000_000) == 0
        assert lib.fmm_debug_set(FMM_DEBUG_TICKET_FILL, 0xFF) == 0
        rt.fmm_gemm(plan, A, B, C.clone(memory_format=torch.preserve_format), "abc")
        torch.cuda.synchronize()
        assert lib.fmm_device_status(1) == FMM_E_TIMEOUT
    finally:
        assert lib.fmm_debug_set(FMM_DEBUG_TICKET_FILL, 0) == 0
        assert lib.fmm_debug_set(FMM_DEBUG_WAIT_LIMIT_NS, 0) == 0
    rt.fmm_gemm(plan, A, B, C, "abc")
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    assert torch.equal(C, want)
