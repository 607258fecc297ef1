"""fp32 products (the choice left open) against float64: tiles and their edges, ranges of input features, every kind of segment,
groups.  Up to 16 rows take the kernel for few rows (one row from 16 input features on), more with at least 128 input features the tensor cores, everything else (fewer input
features, rows of experts) the tiles of the CUDA cores."""
import numpy as np
import pytest
import torch

from tests.kv_util import make_ctx
from tests.test_gpu_linear import close, glu, rnd, run, wrap

pytestmark = pytest.mark.gpu

F32 = torch.float32


def bounded(got, x, w, add=0.0):
    """Each of the K products and sums rounds once, a residual's once more: at most (K + 1) * 2^-24 of the sum of magnitudes, in any order."""
    want, size = x.double() @ w.double() + add, x.double().abs() @ w.double().abs() + abs(add)
    assert ((got.double() - want).abs() <= (x.shape[1] + 1) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("rows", [1, 4, 5, 8, 9, 16, 17, 63, 64, 65, 200])
@pytest.mark.parametrize("K,cols", [(4, (4, 0)), (36, (64, 68)), (128, (128, 4)), (260, (96, 164)), (2052, (32, 100)), (1040, (2048, 32))])
def test_store_and_residual(pkg, rows, K, cols):
    from llm_experiments_b200 import projection as proj

    ctx, (a, b) = make_ctx(pkg), cols
    x, w = rnd((rows, K + 8), F32, 1)[:, 4:4 + K], rnd((K, a + b + 4), F32, 2, K ** -0.5)[:, :a + b]
    out = torch.full((rows + 1, a + 5), 7.0, dtype=F32, device="cuda")
    res = rnd((rows, b + 3), F32, 3)
    keep = res.clone()
    segments = [proj.OutputSegment(a, proj.SEG_STORE, wrap(pkg, out[:, :a]))]
    if b:
        segments.append(proj.OutputSegment(a + b, proj.SEG_F32, wrap(pkg, res)))
    run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, segments, residual=wrap(pkg, res) if b else None)
    bounded(out[:rows, :a], x, w[:, :a])
    bounded(res[:, :b], x, w[:, a:], keep[:, :b].double())
    assert (out[rows] == 7).all() and (out[:, a:] == 7).all() and torch.equal(res[:, b:], keep[:, b:])


@pytest.mark.parametrize("splits", [1, 2, 4, 8])
@pytest.mark.parametrize("rows,K", [(3, 2048), (16, 1000), (70, 1040), (64, 64)])
def test_ranges_of_input_features(pkg, rows, K, splits):
    """Any number of ranges, also more than there are steps: of the kernel for few rows and, at 70 rows, of the tensor cores (64 rows of
    64 input features go to a kernel without ranges, which leaves the knob alone)."""
    from llm_experiments_b200 import _native
    from llm_experiments_b200 import projection as proj

    ctx = make_ctx(pkg)
    x, w, bias = rnd((rows, K), F32, 4), rnd((K, 132), F32, 5, K ** -0.5), rnd((132,), F32, 6)
    out = torch.empty((rows, 132), dtype=F32, device="cuda")
    _native.tune("matmul_splits", splits)
    try:
        run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(132, proj.SEG_STORE, wrap(pkg, out))],
            bias=pkg.gpu.GPUBuffer1D(buffer=bias, shape=(132,), size=132))
    finally:
        _native.tune("matmul_splits", 0)
    bounded(out, x, w, bias.double())


@pytest.mark.parametrize("splits", [3, 5, 6, 7])
@pytest.mark.parametrize("rows,K", [(17, 384), (70, 1040), (300, 452)])
def test_any_number_of_ranges_on_the_tensor_cores(pkg, rows, K, splits):
    """Clusters of any size share rows that they do not divide, with a step or two of input features each, or none."""
    test_ranges_of_input_features(pkg, rows, K, splits)


@pytest.mark.parametrize("rows", [6, 90])
@pytest.mark.parametrize("kind", ["SEG_GLU_SILU", "SEG_GLU_CLAMP", "SEG_RELU2", "SEG_SOFTCAP", "SEG_DECAY"])
def test_kinds(pkg, rows, kind):
    from llm_experiments_b200 import projection as proj

    ctx, code, K, n, limit = make_ctx(pkg), getattr(proj, kind), 256, 136, 1.5
    x, w = rnd((rows, K), F32, 7), rnd((K, n), F32, 8, 2 * K ** -0.5)
    prod = x.double() @ w.double()
    pair = kind.startswith("SEG_GLU")
    want = glu(code, prod[:, ::2], prod[:, 1::2], limit, proj) if pair else dict(
        SEG_RELU2=prod.clamp(min=0) ** 2, SEG_SOFTCAP=limit * torch.tanh(prod / limit),
        SEG_DECAY=torch.exp(torch.nn.functional.logsigmoid(prod) / limit))[kind]
    out = torch.full((rows + 1, want.shape[1] + 1), 7.0, dtype=F32, device="cuda")
    run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(n, code, wrap(pkg, out[:, :-1]))], limit=limit)
    close(out[:rows, :-1], want, F32)
    assert (out[rows] == 7).all() and (out[:, -1] == 7).all()


@pytest.mark.parametrize("counts,K", [((3, 0, 16, 1), 132), ((0, 130, 64, 1, 0), 132), ((0, 130, 64, 1, 0), 1044), ((65, 700), 16), ((17, 1), 516)])
def test_rows_of_experts(pkg, counts, K):
    from llm_experiments_b200 import projection as proj

    ctx, n = make_ctx(pkg), 140
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    x, w = rnd((sum(counts), K), F32, 9), rnd((len(counts) * K, n), F32, 10, K ** -0.5)
    out = torch.empty((sum(counts), n), dtype=F32, device="cuda")
    run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, out))], groups=len(counts),
        group_w=K * n, group_rows=torch.from_numpy(offs).cuda(), max_group_rows=max(counts))
    for e in range(len(counts)):
        bounded(out[offs[e]:offs[e + 1]], x[offs[e]:offs[e + 1]], w[e * K:(e + 1) * K])


@pytest.mark.parametrize("rows", [2, 40])
def test_heads(pkg, rows):
    from llm_experiments_b200 import projection as proj

    ctx, heads, k, n = make_ctx(pkg), 3, 20, 132
    x, w = rnd((rows, heads * k), F32, 11), rnd((heads * k, n), F32, 12, k ** -0.5)
    out = torch.empty((rows, heads * n), dtype=F32, device="cuda")
    run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), k, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, out), group=n)], groups=heads,
        group_x=k, group_w=k * n)
    for h in range(heads):
        bounded(out[:, h * n:(h + 1) * n], x[:, h * k:(h + 1) * k], w[h * k:(h + 1) * k])


@pytest.mark.parametrize("K", [128, 1028])
def test_numbers_that_have_no_parts(pkg, K):
    """What is not finite, or rounds to nothing finite in bf16, in either operand: as with plain multiply-adds, and nowhere else."""
    from llm_experiments_b200 import projection as proj

    ctx, rows, n = make_ctx(pkg), 150, 200
    x, w = rnd((rows, K), F32, 13), rnd((K, n), F32, 14)
    x[3, 5], x[140, K - 1], w[11, 13], w[7, 190], x[9, 11] = float("inf"), float("nan"), 3.4e38, -float("inf"), 0.0
    got = {}
    for path in (0, 1):
        got[path] = torch.empty((rows, n), dtype=F32, device="cuda")
        run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, got[path]))], path=path)
    assert torch.equal(got[0].isnan(), got[1].isnan()) and torch.equal(got[0].isinf(), got[1].isinf())
    plain = torch.ones((rows, n), dtype=torch.bool, device="cuda")
    plain[[3, 140]] = False
    plain[:, [13, 190]] = False
    torch.testing.assert_close(got[0][plain].double(), (x.double() @ w.double())[plain], rtol=1e-4, atol=1e-3)


def product(pkg, ctx, x, w, path=0):
    from llm_experiments_b200 import projection as proj

    out = torch.empty((x.shape[0], w.shape[1]), dtype=F32, device="cuda")
    run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), x.shape[1], [proj.OutputSegment(w.shape[1], proj.SEG_STORE, wrap(pkg, out))], path=path)
    return out


@pytest.mark.parametrize("splits", [0, 3])
@pytest.mark.parametrize("odd", [float("nan"), float("inf"), 3.4e38, 1e-37])
def test_rows_beside_one_that_has_no_parts_keep_their_bits(pkg, odd, splits):
    """A row of x and a column of w with a number that three bf16 parts do not hold: nothing else in their tile changes, and they are
    what plain multiply-adds make of them."""
    from llm_experiments_b200 import _native

    ctx, rows, K, n = make_ctx(pkg), 200, 516, 260
    x, w = rnd((rows, K), F32, 15), rnd((K, n), F32, 16)
    _native.tune("matmul_splits", splits)
    try:
        plain = product(pkg, ctx, x, w)
        x[77, K - 3], w[130, 201] = odd, odd
        got = product(pkg, ctx, x, w)
    finally:
        _native.tune("matmul_splits", 0)
    want = product(pkg, ctx, x, w, path=1)
    mine = torch.zeros((rows, n), dtype=torch.bool, device="cuda")
    mine[77], mine[:, 201] = True, True
    assert torch.equal(got[~mine], plain[~mine])
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    finite = mine & want.isfinite()
    size = x.double().abs() @ w.double().abs()
    assert ((got.double() - want.double()).abs() <= 2 * (K + 1) * 2.0 ** -24 * size)[finite].all()  # (both are off by their sums)


@pytest.mark.parametrize("splits", [0, 3])
@pytest.mark.parametrize("K", [128, 1028])
def test_finite_operands_whose_products_overflow(pkg, K, splits):
    """A sum beyond the range is infinite of the sign that the sums in order have, not a difference of infinities of parts or of ranges."""
    from llm_experiments_b200 import _native

    ctx, rows, n = make_ctx(pkg), 140, 132
    x, w = rnd((rows, K), F32, 17), rnd((K, n), F32, 18)
    x[3, 7], w[7, 5], x[9], w[:, 11] = 1e30, -1e30, rnd((K,), F32, 19, 1e20), rnd((K,), F32, 20, 1e19)
    _native.tune("matmul_splits", splits)
    try:
        got = product(pkg, ctx, x, w)
    finally:
        _native.tune("matmul_splits", 0)
    want = product(pkg, ctx, x, w, path=1)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    assert got[3, 5] == -float("inf") and got.isinf().sum() >= 2


@pytest.mark.parametrize("sx,sw", [(1e-33, 1e10), (1e-36, 1e10), (1e15, 1e-38), (1e-41, 1e25), (1e-30, 1e-3), (1e18, 1e18)])
@pytest.mark.parametrize("rows,K", [(130, 256), (17, 1028)])
def test_operands_of_any_size(pkg, rows, K, sx, sw):
    """Down to subnormal numbers, whose parts bf16 does not hold: the bound of fp32 sums."""
    x, w = rnd((rows, K), F32, 21, sx), rnd((K, 200), F32, 22, sw)
    bounded(product(pkg, make_ctx(pkg), x, w), x, w)


@pytest.mark.parametrize("rows,K,n", [(693, 768, 3072), (1300, 1040, 644), (130, 16388, 388), (2100, 132, 2500), (257, 6404, 388)])
def test_parts_made_ahead_have_the_same_bits(pkg, rows, K, n):
    """With scratch memory the operands of large products are laid out by a kernel ahead: the same numbers, also where some have no parts,
    and in a scratch that another product left full of its own."""
    from llm_experiments_b200 import projection as proj

    ctx = make_ctx(pkg)
    x, w, bias = rnd((rows, K + 4), F32, 21)[:, :K], rnd((K, n + 4), F32, 22, K ** -0.5)[:, :n], rnd((n,), F32, 23)
    scratch = {"linear": torch.full((1 << 27,), 0x7f, dtype=torch.uint8, device="cuda")}
    for odd in (False, True):
        if odd:
            x[5, 7], x[rows - 1, K - 1], w[3, n - 1], w[K - 1, 0], x[9, 11] = float("inf"), 1e-39, float("nan"), 3.4e38, -2e-36
        out = [torch.full((rows + 1, n + 1), 7.0, dtype=F32, device="cuda") for _ in range(2)]
        for o, s in zip(out, (None, scratch)):
            run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, o[:, :n]))], scratch=s,
                bias=pkg.gpu.GPUBuffer1D(buffer=bias, shape=(n,), size=n))
        assert torch.equal(out[0].view(torch.int32), out[1].view(torch.int32))
        if not odd:
            bounded(out[1][:rows, :n], x, w, bias.double())


@pytest.mark.parametrize("ahead", [False, True])
def test_a_wait_that_runs_out_is_reported(pkg, ahead):
    """The warps that take sums out behave as if their first wait had run out.  The other warps run out of their own bounded waits (about two
    seconds), what is under way ends first, the status says so, and the next product is right."""
    from llm_experiments_b200 import projection as proj

    ctx, native, (rows, K, n) = make_ctx(pkg), pkg._native, (700, 1024, 1300)
    x, w, out = rnd((rows, K), F32, 31), rnd((K, n), F32, 32, K ** -0.5), torch.full((rows, n), 7.0, dtype=F32, device="cuda")
    scratch = {} if ahead else None
    ctx.config.check_device_status = True

    def product():
        run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, out))], scratch=scratch)

    native.tune("linear_test_expire", 1)
    try:
        with pytest.raises(RuntimeError, match="bounded wait"):
            product()
    finally:
        native.tune("linear_test_expire", 0)
    assert (out == 7).all() and bool(scratch) == ahead
    product()
    bounded(out, x, w)


def test_scratch_grows_and_is_left_alone_where_it_is_of_no_use(pkg):
    from llm_experiments_b200 import projection as proj

    ctx, scratch, sizes = make_ctx(pkg), {}, []
    for rows, K, n in ((100, 1024, 1024), (300, 256, 64), (1200, 1024, 1024), (1100, 1024, 1024), (2000, 1024, 1024)):
        x, w = rnd((rows, K), F32, 24), rnd((K, n), F32, 25, K ** -0.5)
        out = torch.empty((rows, n), dtype=F32, device="cuda")
        run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, out))], scratch=scratch)
        bounded(out, x, w)
        sizes.append(scratch["linear"].numel() if scratch else 0)
    assert sizes[0] == sizes[1] == 0 and 0 < sizes[2] == sizes[3] < sizes[4]


@pytest.mark.parametrize("rows", [17, 31, 33, 200, 1100, 9000])
@pytest.mark.parametrize("K,n", [(4, 4), (16, 384), (20, 260), (32, 100)])
@pytest.mark.parametrize("kind", ["SEG_STORE", "SEG_F32", "SEG_DECAY", "SEG_SOFTCAP", "SEG_GLU_SILU"])
def test_few_input_features_have_the_bits_of_the_tiles(pkg, rows, K, n, kind):
    """Input features that are zero change no bit of a sum in order, and 36 of them take the tiles."""
    from llm_experiments_b200 import projection as proj

    ctx, kind = make_ctx(pkg), getattr(proj, kind)
    x, w, bias, res = torch.zeros((rows, 36), dtype=F32, device="cuda"), torch.zeros((36, n), dtype=F32, device="cuda"), rnd((n,), F32, 6), rnd((rows, n), F32, 7)
    x[:, :K], w[:K] = rnd((rows, K), F32, 8), rnd((K, n), F32, 9)
    outs, cols = [], n // 2 if kind == proj.SEG_GLU_SILU else n
    for k in (K, 36):
        out = res.clone() if kind == proj.SEG_F32 else torch.full((rows, n), 7.0, dtype=F32, device="cuda")
        run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), k, [proj.OutputSegment(n, kind, wrap(pkg, out[:, :cols]))], limit=3.0,
            bias=pkg.gpu.GPUBuffer1D(buffer=bias, shape=(n,), size=n), residual=wrap(pkg, out) if kind == proj.SEG_F32 else None)
        assert (out[:, cols:] == 7).all()
        outs.append(out)
    if kind == proj.SEG_STORE:
        bounded(outs[0], x[:, :K], w[:K], bias.double())
    assert torch.equal(outs[0], outs[1])
