"""Admission counts the operand sums that the library forms."""
import pytest

from fmm_gen_b200 import serve, tuner

SHAPES = [
    # Strassen: 5 of 7 products have sums of A, 5 of B; blocks 32 x 32 x 32
    ("222-1", (64, 64, 64), 2 * 8 * 5 * 32 * 32),
    # blocks 32 x 32 x 33: every product's operands, k rounded up to 40
    ("222-1", (64, 64, 66), 2 * 8 * 7 * 32 * 40),
    # odd k: every product's operands (blocks 32 x 32 x 32)
    ("222-1", (64, 64, 65), 2 * 8 * 7 * 32 * 32),
    ("222-1", (1024, 1024, 1024), 2 * 8 * 5 * 512 * 512),
    ("222-1", (8, 64, 64), 0),  # no core
]


@pytest.mark.parametrize("alg,shape,want", SHAPES, ids=str)
def test_bytes_of_operand_sums(alg, shape, want):
    m, n, k = shape
    got = serve.request_bytes(serve.FP64, shape, alg) - 8 * (m * k + k * n + m * n) - 8 * (k + 1) * n * (k & 1)
    assert got == want
    assert serve.request_bytes(serve.FP64, shape, "classical") + want == serve.request_bytes(serve.FP64, shape, alg)


@pytest.mark.gpu
@pytest.mark.parametrize("alg", ["222-1", "222-2", "232-1", "333-1", "222-1_333-1"])
@pytest.mark.parametrize("shape", [(96, 96, 96), (384, 416, 1008), (1024, 1024, 1024), (1000, 1000, 1000)], ids=str)
def test_bytes_are_those_of_a_call(alg, shape):
    torch = pytest.importorskip("torch")
    from fmm_gen_b200 import build, ops, runtime as rt

    build.build()
    m, n, k = shape
    A, B, C = (rt.colmajor(r, c, device="cuda").zero_() for r, c in ((m, k), (k, n), (m, n)))
    rt.fmm_gemm(ops.plan_for(alg), A, B, C)
    torch.cuda.synchronize()
    assert rt.last_workspace_bytes() == serve.operand_sum_bytes(tuner.plan_of(alg), m, n, k)
