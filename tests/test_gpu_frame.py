"""What the FP64 kernels write lies inside C: every element of C's buffer outside the matrix (its leading
dimension's padding, the elements before and after it) keeps its value, where tiles, fragments and parts end in
remainders and the stores are 16 or 8 bytes wide."""
import pytest

torch = pytest.importorskip("torch")

from fmm_gen_b200 import build, runtime as rt  # noqa: E402

pytestmark = pytest.mark.gpu
FMM_DEBUG_KSPLIT = 4


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return rt.load_library()


def run(lib, call, m, n, k, pad, off):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    A = rt.colmajor(m, k, device="cuda").uniform_(-1, 1, generator=gen)
    B = rt.colmajor(k, n, device="cuda").uniform_(-1, 1, generator=gen)
    front, ld = 64 + off, m + pad
    flat = torch.full((front + ld * n + 64,), float("nan"), dtype=torch.float64, device="cuda")
    C = torch.as_strided(flat, (m, n), (1, ld), front)
    C.zero_()
    call(A, B, C)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    assert torch.isfinite(C).all()
    assert int(torch.isnan(flat).sum()) == flat.numel() - m * n


FRAMES = [(0, 0), (1, 0), (2, 0), (2, 1), (1, 1)]


@pytest.mark.parametrize("pad,off", FRAMES)
@pytest.mark.parametrize("shape", [(1, 1, 1), (31, 33, 70), (65, 63, 65), (701, 503, 615), (2101, 1051, 257)], ids=str)
def test_plain(lib, shape, pad, off):
    run(lib, rt.plain_gemm, *shape, pad, off)


@pytest.mark.parametrize("pad,off", FRAMES)
@pytest.mark.parametrize("parts", [2, 3, 8])
def test_plain_in_parts(lib, parts, pad, off):
    assert lib.fmm_debug_set(FMM_DEBUG_KSPLIT, parts) == 0
    try:
        run(lib, rt.plain_gemm, 97, 41, 515, pad, off)
    finally:
        assert lib.fmm_debug_set(FMM_DEBUG_KSPLIT, 0) == 0


@pytest.mark.parametrize("pad,off", FRAMES)
@pytest.mark.parametrize("pack", ["abc", "ab"])
@pytest.mark.parametrize("alg,shape", [
    ("222", (17, 9, 3)), ("222", (129, 67, 31)), ("222", (1073, 1001, 301)),  # the last: row strips and every fringe
    ("333", (101, 121, 50)), ("222", (3001, 3101, 1061)),
    ("222", (2950, 1203, 999)),  # fringe strips of 4 and 8 k parts in one launch, 372 CTAs in clusters of 8
], ids=str)
def test_fmm(lib, alg, shape, pack, pad, off):
    plan = rt.Plan.from_levels([alg], [1])
    run(lib, lambda A, B, C: rt.fmm_gemm(plan, A, B, C, pack), *shape, pad, off)
    plan.close()


@pytest.mark.parametrize("pad,off", FRAMES)
def test_batch(lib, pad, off):
    plan = rt.Plan.from_levels(["222"], [1])
    run(lib, lambda A, B, C: rt.batch_submit([plan], [A], [B], [C]), 713, 509, 333, pad, off)
    plan.close()
