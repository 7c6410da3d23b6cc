"""Calls that follow one another on a stream without a synchronisation, each reading what the
one before wrote: kernels start while their predecessors still run, and must see all of it."""
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


@pytest.mark.parametrize("algo", [None, (["222"], [1]), (["222", "333"], [1, 1])], ids=str)
@pytest.mark.parametrize("form", ["abc", "naive", "submit"])
@pytest.mark.parametrize("n", [96, 421, 1200])
def test_c_of_one_call_is_the_operand_of_the_next(lib, algo, form, n):
    """C0 = A B, C1 = C0 B, C2 = B C1, ...: the same bits with and without waiting between the calls."""
    if algo is None and form == "naive":
        form = "abc"
    plan = None if algo is None else rt.Plan.from_levels(*algo)
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = rt.colmajor(n, n, device="cuda").uniform_(-1, 1, generator=gen)
    B = rt.colmajor(n, n, device="cuda").uniform_(-1, 1, generator=gen) / n ** 0.5

    def call(a, b, c):
        if form == "submit":
            rt.batch_submit([plan], [a], [b], [c])
        elif plan is None:
            rt.plain_gemm(a, b, c)
        else:
            rt.fmm_gemm(plan, a, b, c, form)

    def chain(wait):
        Cs = [rt.colmajor(n, n, device="cuda").zero_() for _ in range(8)]
        X = A
        for i, C in enumerate(Cs):
            call(*((X, B) if i % 2 == 0 else (B, X)), C)
            if wait:
                torch.cuda.synchronize()
            X = C
        torch.cuda.synchronize()
        return Cs

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(chain(False), want))
    assert lib.fmm_device_status(1) == 0


def test_split_operands_written_just_before(lib):
    n = 700
    plan = rt.Plan.from_levels(["222"], [1])
    gen = torch.Generator(device="cuda").manual_seed(n)
    A = rt.colmajor(n, n, dtype=torch.float32, device="cuda").normal_(generator=gen)
    B = rt.colmajor(n, n, dtype=torch.float32, device="cuda").normal_(generator=gen)

    def chain(wait):
        X, out = A, []
        for _ in range(6):
            C = rt.colmajor(n, n, device="cuda").zero_()
            rt.split_gemm(plan, X, B, C)
            if wait:
                torch.cuda.synchronize()
            X = rt.colmajor(n, n, dtype=torch.float32, device="cuda").copy_(C)
            X /= n ** 0.5
            out.append(C)
        torch.cuda.synchronize()
        return out

    want = chain(True)
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(chain(False), want))
    assert lib.fmm_device_status(1) == 0
