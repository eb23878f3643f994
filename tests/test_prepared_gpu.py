"""The prepared form of the 3xTF32 families (operands split into scaled FP16 pairs first): every edge of its tiles and
splits against float64, and the operands it has to leave to the TF32 kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ERROR_FLOOR = 2.0 ** -24


@pytest.fixture(scope="module")
def gpu(capi):
    import gpu_support

    return gpu_support


def run(capi, gpu, kernel, a, b, c, alpha, beta, out=None):
    m, n = a.shape[0], b.shape[1]
    d = out if out is not None else torch.full((m, n), float("nan"), device="cuda")
    desc = capi.make_desc(gpu.operand(a), gpu.operand(b), gpu.operand(c) if c is not None else capi.null_operand(m, n),
                          gpu.operand(d), alpha, beta, 0)
    assert capi.platform_supports(kernel, desc) is None
    launch = capi.PlatformGemm(kernel, desc)
    workspace = torch.full((launch.workspace_bytes + 4,), 255, dtype=torch.uint8, device="cuda")
    launch.run(workspace.data_ptr() + 4, launch.workspace_bytes, gpu.current_stream())  # any alignment must do
    torch.cuda.synchronize()
    return d


def check(oracle, d, a, b, c, alpha, beta, what):
    exact = alpha * (a.double() @ b.double()) + (beta * c.double() if c is not None else 0.0)
    ours = oracle.scaled_error(d, exact, a * abs(alpha), b, c, beta)
    plain = oracle.scaled_error(oracle.torch_reference(a, b, c, alpha, beta), exact, a * abs(alpha), b, c, beta)
    assert torch.isfinite(d).all() and ours <= 2.0 * max(plain, ERROR_FLOOR), f"{what}: {ours:.3e} against {plain:.3e}"


@pytest.mark.parametrize("m,k,n", [
    (1, 256, 1),          # the smallest it takes: one row, one column
    (255, 257, 63),       # just under a tile, one K value over a block
    (257, 448, 257),      # one row and one column over a tile
    (300, 1003, 501),     # nothing aligned
    (1500, 512, 700),     # several tiles, a whole number of K blocks
    (129, 5000, 130),     # K slices
    (640, 2048, 4740),    # several waves of tiles on few rows
])
def test_shapes_and_layouts(capi, gpu, oracle, m, k, n):
    torch.manual_seed(m + k + n)
    a, b, c = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda"), torch.randn(m, n, device="cuda")
    a_t, b_t = a.t().contiguous().t(), b.t().contiguous().t()
    a_odd = torch.empty(m, k + 3, device="cuda")[:, 1:k + 1].copy_(a)        # unaligned rows
    b_wide = torch.empty(k, 2 * n, device="cuda")[:, ::2].copy_(b)          # no unit stride at all
    d_odd = torch.full((n, m + 1), float("nan"), device="cuda")[:, :m].t()  # D written through strides
    for kernel in (capi.KERNEL_FP16X3, capi.KERNEL_FP16X3_SPLITK):
        if kernel == capi.KERNEL_FP16X3_SPLITK and k < 512:
            continue
        check(oracle, run(capi, gpu, kernel, a, b, None, 1.0, 0.0), a, b, None, 1.0, 0.0, "plain")
        check(oracle, run(capi, gpu, kernel, a_t, b_t, c, 1.5, -0.25), a, b, c, 1.5, -0.25, "both transposed, C")
        check(oracle, run(capi, gpu, kernel, a_odd, b_wide, c, -1.0, 0.5, out=d_odd), a, b, c, -1.0, 0.5, "strided")
        in_place = c.clone()
        run(capi, gpu, kernel, a, b_t, in_place, 1.0, 2.0, out=in_place)
        check(oracle, in_place, a, b, c, 1.0, 2.0, "in place")
        again = run(capi, gpu, kernel, a, b, None, 1.0, 0.0)
        assert torch.equal(again, run(capi, gpu, kernel, a, b, None, 1.0, 0.0)), "results repeat bit for bit"


def test_scales_of_rows_and_columns(capi, gpu, oracle):
    """Rows of A and columns of B of very different size, and rows without a single nonzero. (Neighbouring columns that far
    apart share a scale, so this goes to the TF32 kernel; the test below stays in the FP16 one.)"""
    torch.manual_seed(1)
    m, k, n = 300, 700, 270
    a = torch.randn(m, k, device="cuda") * torch.exp2(torch.randint(-40, 40, (m, 1), device="cuda").float())
    b = torch.randn(k, n, device="cuda") * torch.exp2(torch.randint(-40, 40, (1, n), device="cuda").float())
    a[7], a[:, 3], b[:, 11] = 0.0, 0.0, 0.0
    d = run(capi, gpu, capi.KERNEL_FP16X3, a, b, None, 1.0, 0.0)
    exact = a.double() @ b.double()
    bound = (a.double().norm(dim=1, keepdim=True) * b.double().norm(dim=0, keepdim=True)) * 2.0 ** -22
    assert ((d.double() - exact).abs() <= bound).all() and (d[7] == 0).all() and (d[:, 11] == 0).all()


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("m,k,n", [(300, 1700, 285), (129, 5000, 130)])  # three slabs; K slices that begin inside a slab
def test_scales_of_slabs_rows_and_column_groups(capi, gpu, m, k, n, transposed):
    """Every row of A, and every 16 columns of B, of another size in every slab of 768, columns of a group up to 2^8 apart: the
    FP16 kernel itself has to find each scale. A scale taken from another row, group or slab is wrong by powers of two; the
    bound is that of 48 truncating additions in a row (2^-23 each) and a few roundings, of the sum of magnitudes."""
    torch.manual_seed(m)
    a, b = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
    b *= torch.exp2(torch.randint(-8, 1, (1, n), device="cuda").float())
    for first in range(0, k, 768):
        slab = slice(first, first + 768)
        a[:, slab] *= torch.exp2(torch.randint(-30, 30, (m, 1), device="cuda").float())
        b[slab] *= torch.exp2(torch.randint(-30, 30, (1, -(-n // 16)), device="cuda").float()).repeat_interleave(16, dim=1)[:, :n]
    a_view, b_view = (a.t().contiguous().t(), b.t().contiguous().t()) if transposed else (a, b)
    d = run(capi, gpu, capi.KERNEL_FP16X3, a_view, b_view, None, 1.0, 0.0)
    bound = 2.0 ** -17 * (a.double().abs() @ b.double().abs())
    assert ((d.double() - a.double() @ b.double()).abs() <= bound).all()
    assert not torch.equal(d, run(capi, gpu, capi.KERNEL_TF32X3, a_view, b_view, None, 1.0, 0.0)), "went to the TF32 kernel"


@pytest.mark.parametrize("exponent_a,exponent_b", [(-55, -55), (-57, -57), (-63, -63), (-90, -30), (-30, -90), (-98, 55)])
@pytest.mark.parametrize("m,k,n", [(300, 1600, 270), (129, 5000, 130)])  # without and with K slices
def test_products_of_small_magnitude(capi, gpu, m, k, n, exponent_a, exponent_b):
    """The inverse scales of a row and of a column may each be a normal number and their product not: the results are
    normal numbers all the same, also when a large alpha brings them to an ordinary size."""
    torch.manual_seed(k)
    a, b = torch.randn(m, k, device="cuda") * 2.0 ** exponent_a, torch.randn(k, n, device="cuda") * 2.0 ** exponent_b
    for alpha in (1.0, 2.0 ** 60):
        exact = alpha * (a.double() @ b.double())
        prepared, plain = (run(capi, gpu, kernel, a, b, None, alpha, 0.0) for kernel in (capi.KERNEL_FP16X3, capi.KERNEL_TF32X3))
        ours, other = (((d.double() - exact).norm() / exact.norm()).item() for d in (prepared, plain))
        assert ours <= 2.0 * max(other, ERROR_FLOOR), f"alpha {alpha}: {ours:.3e} against {other:.3e} of the TF32 form"
        assert not torch.equal(prepared, plain), "went to the TF32 kernel"


@pytest.mark.parametrize("k", [256, 512, 768, 1024, 1536, 2048, 3072, 4096, 8192])
@pytest.mark.parametrize("positive", ["normal", "uniform"])
def test_sums_of_one_sign(capi, gpu, k, positive):
    """The tensor core's sums truncate, which products of one sign add up to a bias: no more of it than in the TF32 form, whose chains are half
    as deep but take the small products, too (measured: 0.83 to 1.06 of its error)."""
    torch.manual_seed(k)
    m, n = 300, 520
    draw = (lambda *shape: torch.randn(*shape, device="cuda").abs()) if positive == "normal" else (lambda *shape: torch.rand(*shape, device="cuda"))
    a, b = draw(m, k), draw(k, n)
    exact = a.double() @ b.double()
    prepared, plain = (run(capi, gpu, kernel, a, b, None, 1.0, 0.0) for kernel in (capi.KERNEL_FP16X3, capi.KERNEL_TF32X3))
    ours, other = (((d.double() - exact).norm() / exact.norm()).item() for d in (prepared, plain))
    assert ours <= 1.25 * other, f"{ours:.3e} against {other:.3e} of the TF32 form"
    assert not torch.equal(prepared, plain), "went to the TF32 kernel"


@pytest.mark.parametrize("kind", ["depth", "pair", "sparse", "large", "tiny", "inf", "nan"])
def test_operands_left_to_the_tf32_kernel(capi, gpu, kind):
    """Magnitudes that spread too far for scaled FP16 pairs (or are not finite): the result is bit for bit that of
    the TF32 family -- also where C is D, which nothing may have written before the decision."""
    torch.manual_seed(2)
    m, k, n = 300, 1000, 270
    a, b = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
    if kind == "depth":  # A and B scaled against each other along K
        scale = torch.exp2(torch.randint(-30, 30, (k,), device="cuda").float())
        a, b = a * scale, b / scale[:, None]
    elif kind == "pair":  # one row of A and one column of B that meet in a pair of far smaller elements
        a[5], b[:, 9] = 0.0, 0.0
        a[5, 0], a[5, 1], b[0, 9], b[1, 9] = 2.0 ** 40, 1.0, 2.0 ** -40, 1.0
    elif kind == "sparse":  # hardly any elements of full size to hide the small ones behind
        a[:, 10:] *= 2.0 ** -30
        b[:, 10:] *= 2.0 ** -30
    elif kind == "large":
        a[3, 4] = 2.0 ** 110
    elif kind == "tiny":
        b[:, 5] *= 2.0 ** -120
    elif kind == "inf":
        a[3, 4] = float("inf")
    else:
        b[3, 4] = float("nan")
    c = torch.randn(m, n, device="cuda")
    for prepared, plain in ((capi.KERNEL_FP16X3, capi.KERNEL_TF32X3), (capi.KERNEL_FP16X3_SPLITK, capi.KERNEL_TF32X3_SPLITK)):
        one, other = c.clone(), c.clone()
        run(capi, gpu, prepared, a, b, one, 1.0, 0.5, out=one)
        run(capi, gpu, plain, a, b, other, 1.0, 0.5, out=other)
        assert torch.equal(one.view(torch.int32), other.view(torch.int32)), kind


@pytest.mark.parametrize("k", [768, 769, 775, 1536 + 64])
@pytest.mark.parametrize("transposed", [False, True])
def test_a_gray_element_concerns_its_own_slab_only(capi, gpu, oracle, k, transposed):
    """A tiny element among full ones does not cost the prepared form, however short the last slab is; it does where its
    slab holds too few full ones beside it."""
    torch.manual_seed(k)
    m, n = 520, 900
    a, b = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
    a[5, 3] = 2.0 ** -40
    a_view, b_view = (a.t().contiguous().t(), b.t().contiguous().t()) if transposed else (a, b)
    d = run(capi, gpu, capi.KERNEL_FP16X3, a_view, b_view, None, 1.0, 0.0)
    check(oracle, d, a, b, None, 1.0, 0.0, "tiny element")
    assert not torch.equal(d, run(capi, gpu, capi.KERNEL_TF32X3, a_view, b_view, None, 1.0, 0.0)), "went to the TF32 kernel"
    b[:700, 7] *= 2.0 ** -20  # ... and now a column has hardly any full element where the row's tiny one is
    b_view = b.t().contiguous().t() if transposed else b
    a[:, :700] *= torch.where(torch.arange(700, device="cuda") % 2 == 0, 1.0, 2.0 ** -20)
    a_view = a.t().contiguous().t() if transposed else a
    assert torch.equal(run(capi, gpu, capi.KERNEL_FP16X3, a_view, b_view, None, 1.0, 0.0),
                       run(capi, gpu, capi.KERNEL_TF32X3, a_view, b_view, None, 1.0, 0.0)), "kept the FP16 kernel"


@pytest.mark.parametrize("transposed", [False, True])
@pytest.mark.parametrize("kind", ["other slab", "sparse", "many"])
def test_sparse_rows_and_gray_elements(capi, gpu, oracle, kind, transposed):
    """A row with next to nothing in one slab and a tiny element in another slab have nothing to do with each other, and a few
    tiny elements ask for one position in common only; a row that is tiny but for ten elements asks for more than ten leave."""
    torch.manual_seed(5)
    m, k, n = 520, 2000, 900
    a, b = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
    if kind == "other slab":
        a[9, 2:768] = 0.0                # slab 0: two elements, fewer than the small ones of a column
        b[:768] = torch.where(b[:768].abs() < 0.01, 0.01, b[:768])
        b[0:2, 4] = 2.0 ** -14
        a[30, 1000] = b[1900, 17] = 2.0 ** -40   # slabs 1 and 2
    elif kind == "sparse":               # 95 % zeros, tiny elements everywhere
        a *= torch.rand(m, k, device="cuda") < 0.05
        a[::7, 100::500] = 2.0 ** -40
        b[50::300, ::5] = 2.0 ** -40
    else:
        a[9, 10:768] *= 2.0 ** -32
    a_view, b_view = (a.t().contiguous().t(), b.t().contiguous().t()) if transposed else (a, b)
    for kernel, plain in ((capi.KERNEL_FP16X3, capi.KERNEL_TF32X3), (capi.KERNEL_FP16X3_SPLITK, capi.KERNEL_TF32X3_SPLITK)):
        d = run(capi, gpu, kernel, a_view, b_view, None, 1.0, 0.0)
        check(oracle, d, a, b, None, 1.0, 0.0, kind)
        left = torch.equal(d, run(capi, gpu, plain, a_view, b_view, None, 1.0, 0.0))
        assert left == (kind == "many"), "went to the TF32 kernel" if left else "kept the FP16 kernel"


def test_a_plan_offers_both_forms(capi, gpu, oracle):
    """Index 0 asks for the prepared form's workspace, the same Primitive without it follows, and index 0 still
    runs with less."""
    torch.manual_seed(3)
    m = k = n = 2048
    a, b = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
    d = torch.empty(m, n, device="cuda")
    plan = gpu.make_plan(a, b, None, d)
    names = plan.primitive_names()
    assert names[0] == names[1] and plan.workspace_bytes(0) > plan.workspace_bytes(1)
    for index in (0, 1):
        gpu.run_plan(plan, index)
        check(oracle, d, a, b, None, 1.0, 0.0, f"index {index}")
    less = torch.empty(max(plan.workspace_bytes(1), 1), dtype=torch.uint8, device="cuda")
    plan.execute(0, less.data_ptr(), plan.workspace_bytes(1), gpu.current_stream())
    torch.cuda.synchronize()
    check(oracle, d, a, b, None, 1.0, 0.0, "index 0 with the minimum")


def test_grouped_plan_mixes_both_forms(capi, gpu, oracle):
    """Large groups through the prepared form, one of them with operands it has to leave to the TF32 kernel, small ones
    and an empty one through the one launch: index 0, the same without the workspace, and index 0 with less."""
    torch.manual_seed(4)
    rows, k, n = [1500, 0, 130, 1024, 40], 2048, 4096  # at n = 2048 the one launch is faster, and the Plan has that form only
    groups = len(rows)
    a, b = torch.randn(sum(rows), k, device="cuda"), torch.randn(groups * k, n, device="cuda")
    c, d = torch.randn(sum(rows), n, device="cuda"), torch.empty(sum(rows), n, device="cuda")
    a[7, 5] = 2.0 ** 110
    plan = capi.GroupedGemmBinding().make_plan(
        {"address": a.data_ptr(), "rows": rows, "cols": [k] * groups}, {"address": b.data_ptr(), "rows": [k] * groups, "cols": [n] * groups},
        {"address": c.data_ptr(), "rows": rows, "cols": [n] * groups}, {"address": d.data_ptr(), "rows": rows, "cols": [n] * groups}, 1.5, 0.5)
    names = plan.primitive_names()
    assert names[0] == names[1] == "GroupedFp32Gemm3xTf32" and plan.workspace_bytes(0) > plan.workspace_bytes(1) > 0
    workspace = torch.empty(plan.workspace_bytes(0), dtype=torch.uint8, device="cuda")
    for index, size in ((0, plan.workspace_bytes(0)), (1, plan.workspace_bytes(1)), (0, plan.workspace_bytes(1))):
        d.fill_(float("nan"))
        plan.execute(index, workspace.data_ptr(), size, gpu.current_stream())
        torch.cuda.synchronize()
        first = 0
        for g, m in enumerate(rows):
            part = slice(first, first + m)
            first += m
            if m != 0:
                check(oracle, d[part], a[part], b[g * k:(g + 1) * k], c[part], 1.5, 0.5, f"group {g}, index {index}, {size} bytes")


def test_grouped_plan_of_large_groups_only(capi, gpu, oracle):
    """Nothing is left for the one TF32 launch."""
    torch.manual_seed(6)
    rows, k, n = [2048, 2000], 1024, 2048
    a, b = torch.randn(sum(rows), k, device="cuda"), torch.randn(2 * k, n, device="cuda")
    d = torch.full((sum(rows), n), float("nan"), device="cuda")
    plan = capi.GroupedGemmBinding().make_plan(
        {"address": a.data_ptr(), "rows": rows, "cols": [k] * 2}, {"address": b.data_ptr(), "rows": [k] * 2, "cols": [n] * 2},
        {"address": 0, "rows": rows, "cols": [n] * 2}, {"address": d.data_ptr(), "rows": rows, "cols": [n] * 2}, 1.0, 0.0)
    names = plan.primitive_names()
    assert names[0] == names[1] and plan.workspace_bytes(0) > plan.workspace_bytes(1)
    gpu.run_plan(plan, 0)
    torch.cuda.synchronize()
    check(oracle, d[:rows[0]], a[:rows[0]], b[:k], None, 1.0, 0.0, "first group")
    check(oracle, d[rows[0]:], a[rows[0]:], b[k:], None, 1.0, 0.0, "second group")
