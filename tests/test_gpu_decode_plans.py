"""How a decode launch cuts its work: a CTA per (sequence, head) for short sequences, a lane per sequence for up to 32 of them, the general way
for the rest.  Every launch is compared with attention in float64 and with the same launch cut the general way (a merge kernel behind it)."""
from __future__ import annotations

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _decode(native, case, merge_kernel):
    q, k, v, lens, table, block, t_upper = case
    B, H, D = q.shape
    code = native.DTYPE_BF16 if q.dtype == torch.bfloat16 else native.DTYPE_F32
    ws = torch.empty(native.lib.b2kv_decode_workspace_bytes(B, H, D, t_upper, code), dtype=torch.uint8, device="cuda")
    out = torch.full_like(q, 7)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    native.tune("decode_merge_kernel", int(merge_kernel))
    try:
        if table is None:  # [B, T, H, D]
            T = k.shape[1]
            rc = native.lib.b2kv_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lens.data_ptr(), 0, 0, B, H, D, t_upper,
                                        T * H * D, H * D, D, code, ws.data_ptr(), ws.numel(), status.data_ptr(), stream)
        else:  # pool [n_blocks, block, H, D]
            rc = native.lib.b2kv_decode_paged(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lens.data_ptr(), 0, 0, table.data_ptr(),
                                              table.shape[1], block, k.shape[0], B, H, D, t_upper, block * H * D, H * D, D, code, ws.data_ptr(),
                                              ws.numel(), status.data_ptr(), stream)
    finally:
        native.tune("decode_merge_kernel", 0)
    native.check(rc)
    torch.cuda.synchronize()
    assert status.item() == 0
    return out


def _reference(q, k, v, lens):
    """Attention in float64, and what fp32 sums may move it by: a score is off by at most D 2^-24 sum |q k| / sqrt(D), a weight by a factor
    of one and twice that, an output by that much of the largest |v|; the sums over tokens add as many roundings as there are tokens."""
    B, H, D = q.shape
    want, slack = torch.zeros(B, H, D, dtype=torch.float64, device="cuda"), torch.zeros(B, H, 1, dtype=torch.float64, device="cuda")
    for b, n in enumerate(lens.tolist()):
        if n == 0:
            continue
        kb, vb, qb = k[b, :n].double(), v[b, :n].double(), q[b].double()
        want[b] = torch.einsum("ht,thd->hd", torch.softmax(torch.einsum("hd,thd->ht", qb, kb) / math.sqrt(D), 1), vb)
        size = torch.einsum("hd,thd->ht", qb.abs(), kb.abs()).amax(1) / math.sqrt(D)
        slack[b] = ((2 * D * size + 2 * n) * 2.0**-24 * vb.abs().amax()).unsqueeze(1)
    return want, slack


@pytest.mark.parametrize("paged", [False, True])
@pytest.mark.parametrize("dtype,D", [(torch.bfloat16, 128), (torch.bfloat16, 64), (torch.float32, 64), (torch.float32, 16), (torch.bfloat16, 256)])
@pytest.mark.parametrize("B,H", [(1, 1), (3, 5), (32, 2), (33, 2), (40, 16)])
@pytest.mark.parametrize("tiles", [1, 4, 5, 11])
def test_decode_plans(pkg, paged, dtype, D, B, H, tiles):
    row = D * (4 if dtype == torch.float32 else 2)
    tile = 64 if row == 256 else min(128, max(8, 8192 // row))
    t_upper = tiles * tile
    g = torch.Generator(device="cuda").manual_seed(D + B * H + tiles)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for shape in ((B, H, D), (B, t_upper, H, D), (B, t_upper, H, D)))
    lens = torch.randint(1, t_upper + 1, (B,), generator=g, device="cuda", dtype=torch.int32)
    lens[0] = t_upper
    if B > 2:
        lens[1], lens[B - 1] = 0, 1
    want, slack = _reference(q, k, v, lens)
    table, block = None, 8
    if paged:
        per = t_upper // block
        table = torch.randperm(B * per, generator=g, device="cuda").to(torch.int32).view(B, per)
        pools = []
        for t in (k, v):
            pool = torch.empty(B * per, block, H, D, dtype=dtype, device="cuda")
            pool[table.long().view(-1)] = t.reshape(B * per, block, H, D)
            pools.append(pool)
        k, v = pools
    case = (q, k, v, lens, table, block, t_upper)
    rounding = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-23
    for merge_kernel in (False, True):
        got = _decode(pkg._native, case, merge_kernel).double()
        assert ((got - want).abs() <= rounding * want.abs() + slack).all()
        assert (got[lens == 0] == 0).all()


def test_a_decode_in_a_graph_follows_the_lengths(pkg):
    """A captured launch keeps its plan; its lengths come from memory: short ones, none, the longest."""
    native = pkg._native
    g = torch.Generator(device="cuda").manual_seed(5)
    for B, t_upper in ((4, 200), (9, 900)):
        q, k, v = (torch.randn(s, generator=g, device="cuda").to(torch.bfloat16) for s in ((B, 4, 128), (B, t_upper, 4, 128), (B, t_upper, 4, 128)))
        lens = torch.full((B,), t_upper, dtype=torch.int32, device="cuda")
        ws = torch.empty(native.lib.b2kv_decode_workspace_bytes(B, 4, 128, t_upper, native.DTYPE_BF16), dtype=torch.uint8, device="cuda")
        out = torch.empty_like(q)

        def launch():
            native.check(native.lib.b2kv_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lens.data_ptr(), 0, 0, B, 4, 128, t_upper,
                                                t_upper * 512, 512, 128, native.DTYPE_BF16, ws.data_ptr(), ws.numel(), None,
                                                torch.cuda.current_stream().cuda_stream))

        launch()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            launch()
        for values in ([t_upper] * B, [0] * B, list(range(1, B + 1)), [t_upper - 7 * b for b in range(B)]):
            lens.copy_(torch.tensor(values, dtype=torch.int32))
            graph.replay()
            torch.cuda.synchronize()
            want, slack = _reference(q, k, v, lens)
            assert ((out.double() - want).abs() <= 2.0**-8 * want.abs() + slack).all()
