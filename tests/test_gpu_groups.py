"""Operand sums in groups: batches and calls whose sums together exceed what may be, or can be, allocated run
their products a group at a time, with the results of the ungrouped call."""
import subprocess
import sys

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


def uniform(rows, cols, gen):
    return rt.colmajor(rows, cols, device="cuda").uniform_(-1, 1, generator=gen)


@pytest.mark.parametrize("form", ["batch", "submit"])
@pytest.mark.parametrize("limit", [64 << 10, 1 << 20])
def test_batch_in_groups_equals_single_calls(lib, form, limit):
    """A cap of a few sums' size; classical problems, every fringe and odd sizes among the FMM problems."""
    gen = torch.Generator(device="cuda").manual_seed(limit)
    plans = {n: rt.Plan.from_levels(*a) for n, a in
             [("s", (["222"], [1])), ("h", (["222", "333"], [1, 1])), ("t", (["232"], [1]))]}
    shapes = [(300, 280, 260), (301, 257, 129), (64, 64, 64), (500, 96, 700), (210, 410, 77), (96, 96, 96), (640, 512, 131)]
    names = ["s", "h", None, "t", "s", "h", "h"]
    ps = [plans.get(n) for n in names]
    As = [uniform(m, k, gen) for m, n, k in shapes]
    Bs = [uniform(k, n, gen) for m, n, k in shapes]
    Cs = [uniform(m, n, gen) for m, n, k in shapes]
    want = [c.clone(memory_format=torch.preserve_format) for c in Cs]
    for p, a, b, c in zip(ps, As, Bs, want):
        rt.plain_gemm(a, b, c) if p is None else rt.fmm_gemm(p, a, b, c)

    def run(cs):
        before = lib.fmm_kernel_launch_count()
        if form == "batch":
            batch = rt.Batch(shapes, ps)
            batch.run(As, Bs, cs)
            torch.cuda.synchronize()
            units = [batch.units(ph) for ph in (0, 1)]
            batch.close()
        else:
            rt.batch_submit(ps, As, Bs, cs)
            torch.cuda.synchronize()
            units = None
        return lib.fmm_kernel_launch_count() - before, units

    whole = [c.clone(memory_format=torch.preserve_format) for c in Cs]
    launches, units = run(whole)
    prev = rt.set_workspace_limit(limit)
    try:
        grouped = run(Cs)
    finally:
        rt.set_workspace_limit(prev)
    assert grouped[0] > launches and grouped[1] == units
    assert lib.fmm_device_status(1) == 0
    for w, x, y in zip(want, whole, Cs):
        assert torch.equal(w, x) and torch.equal(w, y)


def test_batch_of_more_sums_than_one_launch_takes(lib):
    """33 000 small FMM problems: 66 000 operand sums, more than a launch's z extent."""
    count, (m, n, k) = 33000, (16, 8, 6)
    gen = torch.Generator(device="cuda").manual_seed(1)
    plan = rt.Plan.from_levels(["222"], [1])

    def many(rows, cols):
        flat = torch.rand(count, cols, rows, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        return [x.t() for x in flat.unbind(0)], flat.transpose(1, 2)

    (As, A), (Bs, B), (Cs, C) = many(m, k), many(k, n), many(m, n)
    want = C + A @ B
    rt.batch_submit([plan] * count, As, Bs, Cs)
    torch.cuda.synchronize()
    assert lib.fmm_device_status(1) == 0
    # sums of at most 4 products per C block over k / 2, operands of at most 2 terms: 12 (k + 8) u, see algebra.error_bound
    assert (C - want).abs().max().item() <= 12 * (k + 8) * k * 2.0 ** -53


FULL = """
import torch
from fmm_gen_b200 import runtime as rt
lib = rt.load_library()
gen = torch.Generator(device="cuda").manual_seed(3)
def uniform(r, c):
    return rt.colmajor(r, c, device="cuda").uniform_(-1, 1, generator=gen)
form, room = {form!r}, {room}
algs, shape, count = {algs!r}, {shape}, {count}
m, n, k = shape
plan = rt.Plan.from_levels(algs[0], algs[1])
As, Bs, Cs = [[uniform(r, c) for _ in range(count)] for r, c in ((m, k), (k, n), (m, n))]
want = [c.clone(memory_format=torch.preserve_format) for c in Cs]
prev = rt.set_workspace_limit(128 << 20)  # groups: the pool stays small
for a, b, c in zip(As, Bs, want):
    rt.fmm_gemm(plan, a, b, c)
torch.cuda.synchronize()
rt.set_workspace_limit(prev)
filler = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
if form == "batch":
    batch = rt.Batch([shape] * count, [plan] * count)
    batch.run(As, Bs, Cs)
elif form == "submit":
    rt.batch_submit([plan] * count, As, Bs, Cs)
else:
    for a, b, c in zip(As, Bs, Cs):
        rt.fmm_gemm(plan, a, b, c, form)
        assert 0 < rt.last_workspace_bytes() < room + (256 << 20)
torch.cuda.synchronize()
assert lib.fmm_device_status(1) == 0
for w, c in zip(want, Cs):
    assert torch.equal(w, c)
print("equal")
"""


@pytest.mark.parametrize("form,algs,shape,count,room", [
    ("ab", (["222"], [2]), (512, 512, 100000), 1, 1 << 30),             # 2.2 GB of sums, 0.05 GB a product
    ("abc", (["222"], [2]), (512, 512, 100000), 1, 1 << 30),
    ("batch", (["222", "333"], [1, 1]), (360, 360, 30000), 4, 2 << 30),  # 0.8 GB of sums a problem
    ("submit", (["222", "333"], [1, 1]), (360, 360, 30000), 4, 2 << 30),
], ids=["ab", "abc", "batch", "submit"])
def test_sums_larger_than_the_free_memory(form, algs, shape, count, room):
    """A card that is almost full (in a process of its own, whose pools are empty)."""
    code = FULL.format(form=form, algs=algs, shape=shape, count=count, room=room)
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300, cwd=build.ROOT)
    assert r.returncode == 0 and "equal" in r.stdout, r.stdout + r.stderr
