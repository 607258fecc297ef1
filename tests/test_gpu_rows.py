"""Row operations around the 32-bit residual stream against float64: one row, as many as fit the device together and more, widths around
what a thread keeps in registers, odd ones and views with a pitch; the rotations and norms of latent rows by a CTA each and by a warp each."""
import pytest
import torch

from tests.kv_util import make_ctx
from tests.test_gpu_linear import rnd, wrap

pytestmark = pytest.mark.gpu

F32, BF = torch.float32, torch.bfloat16


def b1(pkg, t):
    return pkg.gpu.GPUBuffer1D(buffer=t, shape=tuple(t.shape), size=t.numel())


def norm_close(got, want, dtype):
    """fp32 sums of at most 8200 squares in any order, one rounding of the result."""
    tol = dict(rtol=1e-5, atol=1e-5) if dtype == F32 else dict(rtol=2.0 ** -8, atol=2.0 ** -8)
    torch.testing.assert_close(got.double(), want, **tol)


@pytest.mark.parametrize("dtype", [F32, BF])
@pytest.mark.parametrize("rows,size", [(1, 4), (7, 30), (64, 1024), (5, 1028), (3001, 36), (2500, 1023), (1700, 2048), (2, 4096), (700, 4100), (3, 8196)])
def test_norms_of_any_number_of_rows(pkg, dtype, rows, size):
    ctx = make_ctx(pkg)
    x, w, b = rnd((rows + 3, size + 4), F32, 1)[:, :size] * 3 + 1, rnd((size,), F32, 2), rnd((size,), F32, 3)
    index = torch.randperm(rows + 3, device="cuda")[:rows].to(torch.int32)
    rms, ln, res = (torch.full((rows + 1, size + 4), 7.0, dtype=d, device="cuda") for d in (dtype, dtype, F32))
    before = res[:rows, :size].normal_().double()
    pkg.gpu.batch_begin(ctx)
    pkg.gpu.rms_norm(ctx, wrap(pkg, x), b1(pkg, w), wrap(pkg, rms[:rows, :size]), 1e-5, weight_offset=1.0, row_index=index)
    pkg.gpu.layernorm_rows(ctx, wrap(pkg, x), b1(pkg, w), b1(pkg, b), 1e-5, x=wrap(pkg, res[:rows, :size]), output=wrap(pkg, ln[:rows, :size]), row_index=index)
    pkg.gpu.batch_commit(ctx)
    y = x[index.long()].double()
    norm_close(rms[:rows, :size], y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5) * (w.double() + 1), dtype)
    want = before + torch.nn.functional.layer_norm(y, (size,), w.double(), b.double(), 1e-5)
    norm_close(res[:rows, :size], want, F32)
    norm_close(ln[:rows, :size], want, dtype)
    assert all((t[rows] == 7).all() and (t[:, size:] == 7).all() for t in (rms, ln, res))


@pytest.mark.parametrize("dtype", [F32, BF])
@pytest.mark.parametrize("rows,dim", [(1, 4), (9, 36), (300, 2048), (3, 30), (1500, 1028)])
def test_embedding_rows_of_any_width(pkg, dtype, rows, dim):
    ctx = make_ctx(pkg)
    table, ids = rnd((50, dim), dtype, 4), torch.randint(0, 50, (rows,), device="cuda", dtype=torch.int32)
    out, copy = torch.empty((rows, dim), device="cuda"), torch.empty((rows, dim), dtype=dtype, device="cuda")
    pkg.gpu.batch_begin(ctx)
    pkg.gpu.embedding_rows(ctx, wrap(pkg, table), ids, wrap(pkg, out), scale=1.5, copy=wrap(pkg, copy))
    pkg.gpu.batch_commit(ctx)
    want = table[ids.long()].float() * 1.5
    assert torch.equal(out, want) and torch.equal(copy, want.to(dtype))


@pytest.mark.parametrize("dtype", [F32, BF])
@pytest.mark.parametrize("H,rot,dims,rank,own", [(3, 64, 64, 512, True), (16, 32, 16, 72, True), (5, 128, 128, 1096, True), (2, 64, 48, 64, False)])
def test_latent_rows_by_warps_and_by_ctas(pkg, dtype, H, rot, dims, rank, own):
    """As many rows as take a warp each against the same ones in portions that take a CTA each: rotations and copies bit for bit."""
    from llm_experiments_b200 import latent

    ctx, rows, dim = make_ctx(pkg), 917, 24
    ctx.config.check_device_status = True
    shape = latent.LatentShape(H, dim, rot, dims, 8, rank, 0, 1.0)
    y = rnd((rows, H * (dim + rot) + rank + rot + 8), dtype, 5)
    w, inv = rnd((rank,), F32, 6) + 1, b1(pkg, 10000.0 ** (-torch.arange(dims // 2, device="cuda") / (dims // 2)))
    pos, got = torch.randperm(1000, device="cuda")[:rows].to(torch.int32), []
    for step in (rows, 200):
        cache = pkg.gpu.kv_cache_create(ctx, pkg.gpu.KVCacheConfig(batch_size=1, max_seq_len=1000, n_layers=1, n_heads=1, head_dim=rot, v_head_dim=rank,
                                                                   dtype=dtype, ragged=True))
        mine = y.clone()
        for r in range(0, rows, step):
            part = mine[r:r + step]
            pkg.gpu.batch_begin(ctx)
            pkg.gpu.latent_append(ctx, wrap(pkg, part), shape, inv, latent.RowPlaces(torch.zeros(len(part), dtype=torch.int32, device="cuda"), pos[r:r + step]), cache,
                                  b1(pkg, w) if own else None, 1e-5)
            pkg.gpu.batch_commit(ctx)
        got.append((mine, cache.layers[0].k_cache.buffer, cache.layers[0].v_cache.buffer))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    if own:
        lat = y[:, H * (dim + rot):][:, :rank].double()
        want = lat / torch.sqrt((lat * lat).mean(-1, keepdim=True) + 1e-5) * w.double()
        for _, _, v in got:
            norm_close(v.view(1000, rank)[pos.long()], want, dtype)
    else:
        assert not got[0][2].any()


@pytest.mark.parametrize("dtype", [F32, BF])
@pytest.mark.parametrize("rank", [8, 72, 264, 512, 1096])
def test_latents_do_not_depend_on_the_rows_of_a_step(pkg, dtype, rank):
    """A token's latent has the same bits in a step of 1200 rows, of 200, and alone."""
    from llm_experiments_b200 import latent

    ctx, rows, rot = make_ctx(pkg), 1200, 16
    y, w, inv = rnd((rows, 24 + rot + rank + rot), dtype, 8), rnd((rank,), F32, 9) + 1, b1(pkg, torch.ones(rot // 2, device="cuda"))
    got = []
    for step in (rows, 200, 1):
        cache = pkg.gpu.kv_cache_create(ctx, pkg.gpu.KVCacheConfig(batch_size=1, max_seq_len=rows, n_layers=1, n_heads=1, head_dim=rot, v_head_dim=rank,
                                                                   dtype=dtype, ragged=True))
        mine = y.clone()
        for r in range(0, rows, step)[:20]:
            pos = torch.arange(r, r + step, dtype=torch.int32, device="cuda")
            pkg.gpu.batch_begin(ctx)
            pkg.gpu.latent_append(ctx, wrap(pkg, mine[r:r + step]), latent.LatentShape(1, 24, rot, rot, 8, rank, 0, 1.0), inv,
                                  latent.RowPlaces(torch.zeros_like(pos), pos), cache, b1(pkg, w), 1e-5)
            pkg.gpu.batch_commit(ctx)
        got.append(cache.layers[0].v_cache.buffer.view(rows, rank))
    assert torch.equal(got[0], got[1]) and torch.equal(got[0][:20], got[2][:20])


def test_a_position_outside_the_cache_is_reported_among_many_rows(pkg):
    from llm_experiments_b200 import latent

    ctx, rows = make_ctx(pkg), 900
    ctx.config.check_device_status = True
    cache = pkg.gpu.kv_cache_create(ctx, pkg.gpu.KVCacheConfig(batch_size=1, max_seq_len=rows, n_layers=1, n_heads=1, head_dim=16, v_head_dim=64, dtype=BF, ragged=True))
    y, pos = rnd((rows, 40 + 80), BF, 7), torch.arange(rows, dtype=torch.int32, device="cuda")
    pos[300] = rows
    pkg.gpu.batch_begin(ctx)
    pkg.gpu.latent_append(ctx, wrap(pkg, y), latent.LatentShape(1, 24, 16, 16, 8, 64, 0, 1.0), b1(pkg, torch.ones(8, device="cuda")),
                          latent.RowPlaces(torch.zeros(rows, dtype=torch.int32, device="cuda"), pos), cache, b1(pkg, torch.ones(64, device="cuda")), 1e-5)
    with pytest.raises(RuntimeError, match="position"):
        pkg.gpu.batch_commit(ctx)
    filled = cache.layers[0].v_cache.buffer.view(rows, 64).any(dim=1)
    assert not filled[300] and filled.sum() == rows - 1


@pytest.mark.parametrize("rows", [2047, 2048, 2049, 2079, 3000])
@pytest.mark.parametrize("experts,groups,keep,top", [(64, 1, 1, 6), (64, 8, 3, 6), (8, 1, 1, 2), (96, 1, 1, 9), (60, 1, 1, 6)])
def test_choices_of_many_rows_are_counted(pkg, rows, experts, groups, keep, top):
    """A CTA of 32 rows counts for itself: the choices and scores of the same rows a few at a time, and every expert's count."""
    native = pkg._native
    g = torch.Generator(device="cuda").manual_seed(rows + experts)
    logits = torch.randn(rows, experts + 4, generator=g, device="cuda")
    logits[5] = float("nan")

    def route(first, n):
        idx, score = torch.full((n, top), -7, dtype=torch.int32, device="cuda"), torch.full((n, top), -7.0, device="cuda")
        counts = torch.full((2 * experts,), 9, dtype=torch.int32, device="cuda")
        native.check(native.lib.b2kv_route(logits[first:].data_ptr(), experts + 4, n, experts, groups, keep, top, idx.data_ptr(), score.data_ptr(),
                                           counts.data_ptr(), torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert torch.equal(counts[:experts].long(), torch.bincount(idx.view(-1).long(), minlength=experts)) and not counts[experts:].any()
        return idx, score

    idx, score = route(0, rows)
    few = [route(i, min(300, rows - i)) for i in range(0, rows, 300)]
    assert torch.equal(idx, torch.cat([i for i, _ in few])) and torch.equal(score, torch.cat([s for _, s in few]))


@pytest.mark.parametrize("rank", [8, 264, 512])
@pytest.mark.parametrize("span", [300, 700, 3000, 9000])
def test_shares_of_latent_rows_at_any_place(pkg, rank, span):
    """Rows in a few shares and in dozens, some of them empty, merged from and to memory by pairs of elements and, one element off, by elements."""
    native = pkg._native
    g = torch.Generator(device="cuda").manual_seed(rank + span)
    H, dim, rot, n = 20, 16, 8, 4
    bf = lambda *s: torch.randn(s, generator=g, device="cuda").bfloat16()  # noqa: E731
    ql, q, key, lat = bf(n, H, rank), bf(n, H * (dim + rot)), bf(n, span, rot), bf(n, span, rank)
    pos = torch.tensor([span - 1, 0, span // 2, 65], dtype=torch.int32, device="cuda")
    nbytes = native.lib.b2kv_latent_decode_workspace_bytes(n, H, rank, span, native.DTYPE_BF16)
    assert nbytes > 0
    scale = (dim + rot) ** -0.5
    ws, outs = torch.empty(nbytes + 16, dtype=torch.uint8, device="cuda"), []
    for off_ws, off_out in ((0, 0), (4, 0), (0, 1)):
        out = torch.full((n * H * rank + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
        native.check(native.lib.b2kv_latent_decode(ql.data_ptr(), q.data_ptr(), H * (dim + rot), dim, key.data_ptr(), lat.data_ptr(),
                                                   out[off_out:].data_ptr(), None, pos.data_ptr(), n, span, n, H, rank, rot, 0, span, scale,
                                                   native.DTYPE_BF16, 2, ws[off_ws:].data_ptr(), nbytes, None,
                                                   torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert (out[:off_out] == 7).all() and (out[off_out + n * H * rank:] == 7).all()
        outs.append(out[off_out:off_out + n * H * rank].view(n, H, rank))
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    for i, p in enumerate(pos.tolist()):
        l, k = lat[i, :p + 1].double(), key[i, :p + 1].double()
        s = ql[i].double() @ l.T + q[i].double().view(H, dim + rot)[:, dim:] @ k.T
        want = torch.softmax(s * scale, 1) @ l
        # weights and outputs are rounded to bf16: 2^-9 of the output, and of every weight's share of it
        assert ((outs[0][i].double() - want).abs() <= 2.0**-8 * want.abs() + 2.0**-8 * l.abs().amax(0)).all()
