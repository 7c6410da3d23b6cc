"""Rounding of the FP64 paths against sums in 80-bit arithmetic, where a call's sums over k are made
of several parts.

Expected error, derived from the arithmetic: with entries of A and B independent and uniform in (-1, 1) a
partial sum of j products has variance j v, and an addition to x rounds with a variance of 0.18 u^2 x^2
(u = 2^-53, mantissas log-uniform).  A chain of d additions then has an error variance of 0.09 u^2 d^2 v,
K / d such chains and the additions of their results together 0.09 u^2 (d + K / d) K v.  A product of an FMM has
|U_r|^2 |V_r|^2 times that and reaches C with its W, so that relative to the result

    error^2 = 0.09 u^2 (d + K / d) * mean over C blocks of sum_r W^2 |U_r|^2 |V_r|^2 / (k blocks).

The limit is 1.1 times its root: measured errors scatter by about 1 %, a chain twice as deep has 1.4 times it.
"""
import numpy as np
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


def amplification(plan):
    """Mean over the C blocks of sum_r W^2 |U_r|^2 |V_r|^2, over the number of k blocks."""
    total = 0.0
    for p in plan.products:
        uv = sum(t.coef ** 2 for t in p.a) * sum(t.coef ** 2 for t in p.b)
        total += uv * sum(t.coef ** 2 for t in p.c)
    return total / (plan.dims[0] * plan.dims[2] * plan.dims[1])


def to_dev(x):
    t = rt.colmajor(x.shape[0], x.shape[1], device="cuda")
    t.copy_(torch.from_numpy(x))
    return t


# depth of the parts that a product's sum over k is made of (at most)
CASES = [
    ("single", None, (2048, 2048, 2048), 512),
    ("single", None, (1024, 2048, 4096), 512),
    ("single", None, (1500, 900, 1800), 608),
    ("single", (["222"], [1]), (2048, 2048, 2048), 512),
    ("single", (["222"], [1]), (1501, 1203, 999), 176),
    ("single", (["222"], [2]), (2048, 2048, 6144), 768),
    ("batch", None, (1500, 900, 1800), 608),
    ("batch", (["222"], [1]), (1501, 1203, 1999), 208),
    ("submit", (["222"], [1]), (2048, 2048, 2048), 512),
]


@pytest.mark.parametrize("form,algo,shape,depth", CASES, ids=str)
def test_rounding_of_sums_in_parts(form, algo, shape, depth):
    m, n, k = shape
    rng = np.random.default_rng(m + 3 * n + 5 * k)
    A, B, C = (rng.uniform(-1, 1, s) for s in ((m, k), (k, n), (m, n)))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C)
    plan = None if algo is None else rt.Plan.from_levels(*algo)
    if form == "batch":
        batch = rt.Batch([shape], [plan])
        batch.run([dA], [dB], [dC])
        torch.cuda.synchronize()
        batch.close()
    elif form == "submit":
        rt.batch_submit([plan], [dA], [dB], [dC])
    elif plan is None:
        rt.plain_gemm(dA, dB, dC)
    else:
        rt.fmm_gemm(plan, dA, dB, dC, "abc")
    torch.cuda.synchronize()
    assert rt.load_library().fmm_device_status(1) == 0
    rows = np.linspace(0, m - 1, 16).astype(int)
    want = C[rows].astype(np.longdouble) + A[rows].astype(np.longdouble) @ B.astype(np.longdouble)
    diff = dC.cpu().numpy()[rows].astype(np.longdouble) - want
    error = float(np.sqrt((diff * diff).sum() / (want * want).sum()))
    K = k if plan is None else k // plan.algebra.dims[1]
    amp = 1.0 if plan is None else amplification(plan.algebra)
    assert error <= 1.1 * 0.3 * U * np.sqrt((depth + K / depth) * amp)
    if plan is not None:
        plan.close()
