"""Single calls in a CUDA graph (after a warm-up call, which uploads the plan's tables): every schedule replays
with the bits of the call itself."""
import pytest

torch = pytest.importorskip("torch")

from fmm_gen_b200 import build, runtime as rt  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return rt.load_library()


@pytest.mark.parametrize("algs,pack,shape,cap", [
    (None, "abc", (3000, 2901, 8), None),               # little k
    (None, "abc", (1409, 1407, 2048), None),            # two parts
    (["222"], "abc", (1024, 1024, 1024), None),         # stored products
    (["222"], "abc", (1024, 1024, 1024), 16 << 20),     # groups
    (["222"], "ab", (1031, 1017, 515), None),
    (["222"], "abc", (7700, 7713, 512), None),          # units of all products of a tile, fringes
    (["222"], "abc", (4096, 4096, 2048), None),         # tickets
], ids=str)
def test_graph_of_one_call(lib, algs, pack, shape, cap):
    m, n, k = shape
    plan = None if algs is None else rt.Plan.from_levels(algs, [1])
    gen = torch.Generator(device="cuda").manual_seed(k)
    A, B, C0 = (rt.colmajor(r, c, device="cuda").uniform_(-1, 1, generator=gen) for r, c in ((m, k), (k, n), (m, n)))

    def call(c):
        rt.plain_gemm(A, B, c) if plan is None else rt.fmm_gemm(plan, A, B, c, pack)

    prev = rt.set_workspace_limit(cap) if cap else None
    try:
        want = C0.clone(memory_format=torch.preserve_format)
        call(want)
        C = C0.clone(memory_format=torch.preserve_format)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(C)
    finally:
        if cap:
            rt.set_workspace_limit(prev)
    for _ in range(2):
        C.copy_(C0)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(C, want)
    assert lib.fmm_device_status(1) == 0
    del g
    if plan is not None:
        plan.close()
