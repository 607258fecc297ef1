"""Tiled products whose output columns ask for every width of tile there is, by CTA pairs (300 rows) and by single CTAs (200 rows),
against float64: the sizes fill the places of one wave at that width and no narrower one."""
import pytest
import torch

from tests.kv_util import make_ctx
from tests.test_gpu_linear import close, rnd, run, wrap

pytestmark = pytest.mark.gpu

BF = torch.bfloat16
TILED = 3


@pytest.mark.parametrize("cols", [64, 96, 128, 160, 192, 224, 256])
@pytest.mark.parametrize("rows,tiles", [(300, 37), (200, 74)])
def test_every_width(pkg, rows, tiles, cols):
    from llm_experiments_b200 import projection as proj

    ctx, K, n, a = make_ctx(pkg), 200, tiles * cols - 24, 32
    x, w, res = rnd((rows, K), BF, 1), rnd((K, n), BF, 2, K ** -0.5), rnd((rows, n - a), torch.float32, 3)
    head, body = torch.full((rows + 1, a), 7.0, dtype=BF, device="cuda"), torch.full((rows + 1, n - a), 7.0, device="cuda")
    body[:rows] = res
    run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(a, proj.SEG_STORE, wrap(pkg, head)), proj.OutputSegment(n, proj.SEG_F32, wrap(pkg, body))],
        residual=wrap(pkg, body), path=TILED)
    want = x.double() @ w.double()
    close(head[:rows], want[:, :a], BF)
    close(body[:rows], want[:, a:] + res.double(), torch.float32)
    assert (head[rows] == 7).all() and (body[rows] == 7).all()


@pytest.mark.parametrize("cols", [64, 96, 160, 224])
@pytest.mark.parametrize("rows,tiles", [(300, 37), (200, 74)])
def test_matmul_with_everything_behind_it(pkg, rows, tiles, cols):
    ctx, K, n = make_ctx(pkg), 72, tiles * cols - 24
    ctx.config.check_device_status = True
    x, w, res, bias = rnd((rows, K), BF, 4), rnd((K, n), BF, 5, K ** -0.5), rnd((rows, n), BF, 6), rnd((n,), BF, 7)
    out = torch.full((rows + 1, n), 7.0, dtype=BF, device="cuda")
    pkg.gpu.batch_begin(ctx)
    from llm_experiments_b200 import projection

    projection.matmul(ctx, wrap(pkg, x), wrap(pkg, w), wrap(pkg, out[:rows]), residual=wrap(pkg, res),
                      bias=pkg.gpu.GPUBuffer1D(buffer=bias, shape=(n,), size=n), activation="gelu")
    pkg.gpu.batch_commit(ctx)
    z = x.double() @ w.double() + bias.double()
    close(out[:rows], z * torch.sigmoid(1.702 * z) + res.double(), BF)
    assert (out[rows] == 7).all()


@pytest.mark.parametrize("counts,starts", [((300, 1, 513), (700, 0, 40)), ((129, 128), (3, 3)), ((5, 0, 900, 17), (10, 20, 30, 931))])
def test_runs_of_rows_anywhere_with_one_matrix(pkg, counts, starts):
    """Groups whose rows of x start anywhere, also where others lie, or end with x."""
    import numpy as np

    from llm_experiments_b200 import projection as proj

    ctx, K, n = make_ctx(pkg), 136, 520
    x, w = rnd((948 if starts[-1] == 931 else 1100, K), BF, 8), rnd((K, n), BF, 9, K ** -0.5)
    offs = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
    out = torch.full((sum(counts) + 1, n), 7.0, dtype=BF, device="cuda")
    run(pkg, ctx, wrap(pkg, x), wrap(pkg, w), K, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, out[:-1]))], groups=len(counts), group_w=0,
        group_rows=torch.from_numpy(offs).cuda(), max_group_rows=max(counts),
        group_x_rows=torch.tensor(starts, dtype=torch.int32, device="cuda"), rows=sum(counts))
    want = torch.cat([x[s:s + c].double() @ w.double() for s, c in zip(starts, counts)])
    close(out[:-1], want, BF)
    assert (out[-1] == 7).all()


@pytest.mark.parametrize("kind", ["SEG_GLU_SILU", "SEG_GLU_CLAMP"])
def test_gated_outputs_have_the_bits_of_the_product_for_few_rows(pkg, kind):
    """Rows of the identity pick the weights as sums, the same in both kernels; gates of all sizes, up to where the denominator is no
    normal number's reciprocal any more, and infinity."""
    from llm_experiments_b200 import projection as proj

    ctx, n = make_ctx(pkg), 4096
    w = rnd((128, n), BF, 11, 30.0)
    w[1, ::2], w[2, ::2] = torch.linspace(-88.5, -86, n // 2, device="cuda"), torch.linspace(-52, -50, n // 2, device="cuda")
    w[1:3, 1::2] = 3e4
    w[3, 0], w[4, 2], w[5, 4], w[6, 6] = float("inf"), -float("inf"), -3e38, 3e38
    got = []
    for path in (2, TILED):
        got.append(torch.empty((128, n // 2), dtype=BF, device="cuda"))
        run(pkg, ctx, wrap(pkg, torch.eye(128, dtype=BF, device="cuda")), wrap(pkg, w), 128,
            [proj.OutputSegment(n, getattr(proj, kind), wrap(pkg, got[-1]))], limit=1e30, path=path)
    assert torch.equal(got[0].view(torch.int16), got[1].view(torch.int16))
    assert (got[1][1 if kind == "SEG_GLU_SILU" else 2] != 0).all()


def test_gelu_where_the_denominator_is_large(pkg):
    """z sigmoid(1.702 z) is a normal number of bf16 at z = -52; nothing of it is lost before the rounding."""
    from llm_experiments_b200 import projection

    ctx, n = make_ctx(pkg), 2048
    z = torch.linspace(-52, 3, 200 * n, device="cuda").view(200, n).to(BF)
    out = torch.empty((200, n), dtype=BF, device="cuda")
    pkg.gpu.batch_begin(ctx)
    projection.matmul(ctx, wrap(pkg, torch.eye(200, dtype=BF, device="cuda")), wrap(pkg, z), wrap(pkg, out), activation="gelu")
    pkg.gpu.batch_commit(ctx)
    want = z.double() * torch.sigmoid(1.702 * z.double())
    seen = want.abs() > 1.2e-38
    torch.testing.assert_close(out.double()[seen], want[seen], rtol=2.0 ** -8 + 2.0 ** -16, atol=0)  # bf16, and __expf of 90: 2^-16.5
    assert seen.sum() > 200 * n * 0.95


@pytest.mark.parametrize("by_linear", [False, True])
@pytest.mark.parametrize("rows", [256, 1024, 2048])
def test_a_product_used_as_a_weight_right_away(pkg, rows, by_linear):
    """The output of a tiled product is the second operand of the next one, of few rows, which reads its first tiles ahead of everything
    else: it finds what was written, call after call, and not what lay there before."""
    from llm_experiments_b200 import projection as proj

    ctx, K, n = make_ctx(pkg), 2048, 1024
    a, x = rnd((rows, K), BF, 21), rnd((8, rows), BF, 22)
    weights = [rnd((K, n), BF, 23 + i, K ** -0.5) for i in range(6)]
    c, out = torch.zeros((rows, n), dtype=BF, device="cuda"), [torch.empty((8, n), dtype=BF, device="cuda") for _ in weights]
    pkg.gpu.batch_begin(ctx)
    for w, o in zip(weights, out):
        if by_linear:
            proj.linear(ctx, wrap(pkg, a), wrap(pkg, w), K, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, c))])
            proj.linear(ctx, wrap(pkg, x), wrap(pkg, c), rows, [proj.OutputSegment(n, proj.SEG_STORE, wrap(pkg, o))])
        else:
            proj.matmul(ctx, wrap(pkg, a), wrap(pkg, w), wrap(pkg, c))
            proj.matmul(ctx, wrap(pkg, x), wrap(pkg, c), wrap(pkg, o))
    pkg.gpu.batch_commit(ctx)
    for w, o in zip(weights, out):
        want = x.double() @ (a.double() @ w.double()).to(BF).double()
        # c rounds once more or less at a tie: half a bf16 step of each of the terms at most, which are rows of order one
        torch.testing.assert_close(o.double(), want, rtol=2.0 ** -7, atol=2.0 ** -8 * rows ** 0.5)
