"""The small-tile FP64 kernels at the sizes where they can go wrong: edges of 32- and 64-row
tiles and 16-row / 8-column fragments, k around the 8- and 16-deep groups, every k part count,
operands whose columns do not start on 16 bytes (odd leading dimensions, bases 8 bytes off).

Tolerance: a sum of k products of |a|, |b| <= 1 added to c has error at most (k + 1) u per
unit of |A||B| + |c| in any order of additions; the result and the FP64 reference each have
that much.  An FMM adds its own factor, algebra.error_bound.
"""
import pytest

torch = pytest.importorskip("torch")

from fmm_gen_b200 import algebra, build, runtime as rt  # noqa: E402

pytestmark = pytest.mark.gpu
U = 2.0 ** -53
FMM_DEBUG_KSPLIT = 4


@pytest.fixture(scope="module", autouse=True)
def lib():
    build.build()
    if not torch.cuda.is_available():
        pytest.fail("GPU tests need a CUDA device")
    return rt.load_library()


def matrix(rows, cols, ld, off, gen):
    """Column-major rows x cols with leading dimension ld, its base `off` doubles past a
    16-byte boundary; NaN outside the matrix, so that a read past it shows."""
    flat = torch.full((off + ld * cols + 2,), float("nan"), dtype=torch.float64, device="cuda")
    v = torch.as_strided(flat, (rows, cols), (1, ld), off)
    v.copy_(torch.rand(rows, cols, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1)
    return v


def operands(m, n, k, pad, off, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (matrix(m, k, m + pad, off, gen), matrix(k, n, k + pad, off, gen), matrix(m, n, m + pad, off, gen))


def check(A, B, C0, C, extra=0.0):
    k = A.shape[1]
    want = C0 + A @ B
    scale = A.abs() @ B.abs() + C0.abs()
    assert torch.isfinite(C).all()
    over = (C - want).abs() - (2 * (k + 2) * U * scale + extra)
    assert over.max().item() <= 0, over.max().item()


SHAPES = [(1, 1, 1), (31, 33, 7), (32, 32, 16), (33, 31, 17), (64, 64, 64), (65, 63, 65), (16, 8, 129), (17, 9, 8),
          (240, 250, 600), (7, 700, 515), (700, 7, 515), (1000, 1100, 24), (2100, 1050, 129), (1601, 1500, 1501)]


@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (0, 1), (3, 1)])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_plain_edges(lib, shape, pad, off):
    A, B, C0 = operands(*shape, pad, off, sum(shape))
    _, _, C = operands(*shape, pad, off, sum(shape))
    rt.plain_gemm(A, B, C)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    check(A, B, C0, C)


@pytest.mark.parametrize("parts", range(1, 9))
@pytest.mark.parametrize("shape,pad", [((100, 70, 515), 0), ((97, 41, 64), 1), ((33, 65, 130), 0)], ids=str)
def test_plain_part_counts(lib, shape, pad, parts):
    A, B, C0 = operands(*shape, pad, 0, 5)
    _, _, C = operands(*shape, pad, 0, 5)
    batch_C = C0.clone(memory_format=torch.preserve_format)
    assert lib.fmm_debug_set(FMM_DEBUG_KSPLIT, parts) == 0
    try:
        rt.plain_gemm(A, B, C)
        batch = rt.Batch([shape])
        batch.run([A], [B], [batch_C])
        torch.cuda.synchronize()
        batch.close()
    finally:
        assert lib.fmm_debug_set(FMM_DEBUG_KSPLIT, 0) == 0
    assert lib.fmm_device_status(1) == 0
    check(A, B, C0, C)
    assert torch.equal(C, batch_C)  # a batch adds the same parts in the same order


@pytest.mark.parametrize("pack", ["abc", "ab", "naive"])
@pytest.mark.parametrize("alg,shape", [("222", (16, 8, 2)), ("222", (17, 9, 3)), ("222", (129, 67, 31)),
                                       ("222", (272, 264, 66)), ("333", (100, 120, 50)), ("232", (1300, 1200, 190)),
                                       ("222", (3000, 3100, 160))], ids=str)
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 1)])
def test_fmm_edges(lib, alg, shape, pack, pad, off):
    plan = rt.Plan.from_levels([alg], [1])
    A, B, C0 = operands(*shape, pad, off, sum(shape))
    _, _, C = operands(*shape, pad, off, sum(shape))
    rt.fmm_gemm(plan, A, B, C, pack)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    check(A, B, C0, C, algebra.error_bound(plan.algebra, *shape, 1.0, 1.0, 1.0))
    plan.close()


@pytest.mark.parametrize("algs,shape", [(["222"], (416, 400, 400)), (["222"], (413, 399, 401)), (["222"], (850, 402, 398)),
                                        (["222", "333"], (846, 852, 858)), (["222", "333"], (845, 851, 849))], ids=str)
@pytest.mark.parametrize("pad,off", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("pack", ["abc", "naive"])
def test_staged_operand_sums(lib, algs, shape, pad, off, pack):
    """Operand sums from staged blocks (at least one 128-pair chunk per SM): even and odd blocks, aligned
    and unaligned operands, only the sums or every product's operands."""
    plan = rt.Plan.from_levels(algs, [1] * len(algs))
    A, B, C0 = operands(*shape, pad, off, sum(shape))
    _, _, C = operands(*shape, pad, off, sum(shape))
    rt.fmm_gemm(plan, A, B, C, pack)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    check(A, B, C0, C, algebra.error_bound(plan.algebra, *shape, 1.0, 1.0, 1.0))
    plan.close()


@pytest.mark.parametrize("side", [2, 66, 336, 338])
def test_combine_units(lib, side):
    """36 C blocks in five groups: a group per unit below three tiles of 256 positions per SM (blocks of
    336 x 336 are the last on a 148-SM chip), every group of a tile in one unit from there on."""
    plan = rt.Plan.from_levels(["222", "333"], [1, 1])
    shape = (6 * side, 6 * side, 48)
    A, B, C0 = operands(*shape, 0, 0, side)
    _, _, C = operands(*shape, 0, 0, side)
    rt.fmm_gemm(plan, A, B, C, "abc")
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    check(A, B, C0, C, algebra.error_bound(plan.algebra, *shape, 1.0, 1.0, 1.0))
    plan.close()


@pytest.mark.parametrize("shape", [(1024, 1024, 256), (1072, 1000, 300), (1040, 1136, 264), (1504, 1216, 272)], ids=str)
def test_product_strips(lib, shape):
    """Stored products whose last 64 x 64 units run as 16-row strips (three to four units per SM on
    148 SMs, and 0.7 past five): whole tiles, tiles of 24 and 8 rows whose lower strips are empty, and partial columns."""
    plan = rt.Plan.from_levels(["222"], [1])
    A, B, C0 = operands(*shape, 0, 0, sum(shape))
    _, _, C = operands(*shape, 0, 0, sum(shape))
    rt.fmm_gemm(plan, A, B, C, "abc")
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    check(A, B, C0, C, algebra.error_bound(plan.algebra, *shape, 1.0, 1.0, 1.0))
    plan.close()


@pytest.mark.parametrize("alg", [None, "222"])
@pytest.mark.parametrize("shape,pad", [((1030, 1100, 300), 0), ((1024, 2100, 257), 3), ((701, 511, 90), 0), ((2049, 700, 33), 1)],
                         ids=str)
def test_host_calls_in_column_panels(lib, alg, shape, pad):
    """Host matrices whose copies run in column panels (C of at least 2^20 elements) or whole, dense
    and with a padded leading dimension."""
    m, n, k = shape
    dev = operands(m, n, k, 0, 0, 3 * m + n)

    def host(x):
        flat = torch.full((x.shape[1], x.shape[0] + pad), 7.0, dtype=torch.float64)
        flat[:, :x.shape[0]] = x.t().cpu()
        return flat.numpy().T[:x.shape[0]], flat

    (A, _), (B, _), (C, flat) = (host(x) for x in dev)
    if alg is None:
        rt.bl_dgemm_host(A, B, C)
        extra = 0.0
    else:
        plan = rt.Plan.from_levels([alg], [1])
        rt.fmm_gemm_host(plan, A, B, C)
        extra = algebra.error_bound(plan.algebra, m, n, k, 1.0, 1.0, 1.0)
    assert pad == 0 or bool((flat[:, m:] == 7.0).all())
    check(dev[0], dev[1], dev[2], torch.from_numpy(C.copy()).cuda(), extra)


def test_batch_reads_unaligned_operands_in_place(lib):
    """Operands no tensor copy can read (bases 8 bytes off) in a batch beside aligned ones."""
    shapes = [(130, 70, 33), (64, 64, 64), (300, 257, 100)]
    ops = [operands(*s, 2, i % 2, 7 + i) for i, s in enumerate(shapes)]
    single = [operands(*s, 2, i % 2, 7 + i)[2] for i, s in enumerate(shapes)]
    plan = rt.Plan.from_levels(["222"], [1])
    plans = [None, None, plan]
    for p, (A, B, _), C in zip(plans, ops, single):
        rt.plain_gemm(A, B, C) if p is None else rt.fmm_gemm(p, A, B, C)
    rt.batch_submit(plans, [o[0] for o in ops], [o[1] for o in ops], [o[2] for o in ops])
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    for (_, _, C), w in zip(ops, single):
        assert torch.equal(C, w)
    plan.close()
