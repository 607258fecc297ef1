"""Gated linear attention against float64: token after token and sixteen tokens at a time, any cut of a sequence, strong and
vanishing decays, states carried from call to call, places used again, sizes that fill no tile."""
import numpy as np
import pytest
import torch

from oracle import bamasun_oracle as bo
from tests.kv_util import make_ctx

pytestmark = pytest.mark.gpu

F32, BF = torch.float32, torch.bfloat16
STEP, CHUNK = 1, 2


def wrap(pkg, t):
    return pkg.gpu.GPUBuffer2D(buffer=t, shape=tuple(t.shape), size=t.numel())


class Layer:
    """Rows of random queries, keys, values, gates and decays, and what the equations make of them."""

    def __init__(self, pkg, heads, dim, vdim, tau, dtype, z_mean=3.0, z_std=2.0, seed=0):
        from llm_experiments_b200 import recurrent

        self.pkg, self.ctx, self.dtype = pkg, make_ctx(pkg), dtype
        self.ctx.config.check_device_status = True
        self.shape = recurrent.GlaShape(heads, dim, vdim, tau)
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        pad = lambda n: (n + 7) // 8 * 8  # noqa: E731
        nk, nv = heads * dim, heads * vdim
        self.cols = (0, pad(nk), 2 * pad(nk), 2 * pad(nk) + pad(nv))
        self.width = 2 * pad(nk) + 2 * pad(nv)
        self.norm = torch.randn(vdim, generator=self.gen, device="cuda") * 0.3 + 1
        self.z_mean, self.z_std = z_mean, z_std

    def rows(self, n):
        y = torch.randn((n, self.width), generator=self.gen, device="cuda").to(self.dtype)
        z = torch.randn((n, self.shape.heads * self.shape.dim), generator=self.gen, device="cuda") * self.z_std + self.z_mean
        return y, (torch.sigmoid(z.double()) ** (1 / self.shape.tau)).float()

    def states(self, slots):
        from llm_experiments_b200 import recurrent

        s = recurrent.gla_state_create(self.ctx, self.shape, slots)
        s.fill_(float("nan"))  # a run that starts at position 0 takes nothing over
        return s

    def run(self, y, al, segments, pos, state, path, eps=1e-4):
        """``segments``: (row0, n, slot)."""
        from llm_experiments_b200 import recurrent
        from llm_experiments_b200.serving import RowSegments

        pkg, sh = self.pkg, self.shape
        out = torch.full((len(y) + 1, sh.heads * sh.vdim + 8), 7.0, dtype=self.dtype, device="cuda")
        seg = RowSegments(torch.tensor(segments, dtype=torch.int32, device="cuda"), len(segments), max(n for _, n, _ in segments))
        pkg.gpu.batch_begin(self.ctx)
        recurrent.gated_linear_attention(self.ctx, wrap(pkg, y), self.cols, wrap(pkg, al), sh,
                                         pkg.gpu.GPUBuffer1D(buffer=self.norm, shape=(sh.vdim,), size=sh.vdim), eps, seg,
                                         torch.tensor(pos, dtype=torch.int32, device="cuda"), state, wrap(pkg, out[:len(y)]), path=path)
        pkg.gpu.batch_commit(self.ctx)
        torch.cuda.synchronize()
        assert (out[len(y)] == 7).all() and (out[:, sh.heads * sh.vdim:] == 7).all()
        return out[:len(y), :sh.heads * sh.vdim].double().cpu().numpy()

    def want(self, y, al, state=None, eps=1e-4):
        """Output and last state of one sequence, float64."""
        sh = self.shape
        n = len(y)
        y, alpha = y.double().cpu().numpy(), al.double().cpu().numpy().reshape(n, sh.heads, sh.dim)
        part = lambda c, d: y[:, c:c + sh.heads * d].reshape(n, sh.heads, d)  # noqa: E731
        q, k = part(self.cols[0], sh.dim) * sh.dim ** -0.5, part(self.cols[1], sh.dim)
        v, g = part(self.cols[2], sh.vdim), part(self.cols[3], sh.vdim)
        outs, states = [], []
        for h in range(sh.heads):
            o, s = bo.recurrence(q[:, h], k[:, h], v[:, h], alpha[:, h], None if state is None else state[h])
            outs.append(bo.rms_norm(o, self.norm.double().cpu().numpy(), eps))
            states.append(s)
        return (np.stack(outs, 1) * g * bo.sigmoid(g)).reshape(n, -1), np.stack(states)


def close(got, want, dtype, what=""):
    """The state and the output before rounding are fp32 whatever the storage type."""
    assert np.isfinite(got).all(), what
    tol = 3e-5 if dtype == F32 else 8e-3
    np.testing.assert_allclose(got, want, rtol=tol, atol=tol * max(1.0, np.abs(want).std()), err_msg=str(what))


def state_close(state, want, rtol=1e-4):
    got = state.double().cpu().numpy()
    assert np.abs(got - want).max() <= rtol * np.abs(want).max()


CASES = [(STEP, F32, 3, 5, 7), (STEP, BF, 2, 9, 33), (STEP, F32, 2, 48, 300), (STEP, BF, 4, 128, 256),
         (CHUNK, BF, 5, 40, 24), (CHUNK, BF, 1, 8, 8), (CHUNK, BF, 3, 24, 72), (CHUNK, BF, 2, 64, 160), (CHUNK, BF, 2, 128, 256),
         (CHUNK, BF, 2, 104, 104), (CHUNK, BF, 3, 128, 64)]


@pytest.mark.parametrize("path,dtype,heads,dim,vdim", CASES)
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 33, 100])
def test_whole_sequences(pkg, path, dtype, heads, dim, vdim, n):
    layer = Layer(pkg, heads, dim, vdim, 4.0, dtype, seed=n)
    y, al = layer.rows(n)
    state = layer.states(2)
    got = layer.run(y, al, [(0, n, 1)], range(n), state, path)
    want, last = layer.want(y, al)
    close(got, want, dtype, n)
    state_close(state[1], last)
    assert torch.isnan(state[0]).all()


@pytest.mark.parametrize("heads,dim,vdim", [(2, 4, 4), (3, 12, 36), (1, 32, 32), (2, 36, 20), (2, 64, 128), (1, 128, 68)])
@pytest.mark.parametrize("lens", [(2,), (7, 1, 8), (9, 17, 33), (100, 24, 25)])
def test_fp32_runs_with_the_state_in_registers(pkg, heads, dim, vdim, lens):
    """Lengths around the eight tokens of a step and the ring of three, several runs at a time, continued once."""
    layer = Layer(pkg, heads, dim, vdim, 4.0, F32, seed=sum(lens))
    state, pos = layer.states(len(lens)), np.concatenate([np.arange(n) for n in lens])
    segments, rows, last = [(sum(lens[:i]), n, len(lens) - 1 - i) for i, n in enumerate(lens)], sum(lens), {}
    for again in (0, 1):
        y, al = layer.rows(rows)
        got = layer.run(y, al, segments, pos + again * np.repeat(lens, lens), state, 0)
        for r0, n, slot in segments:
            want, last[slot] = layer.want(y[r0:r0 + n], al[r0:r0 + n], last.get(slot))
            close(got[r0:r0 + n], want, F32, (r0, n, again))
            state_close(state[slot], last[slot])


@pytest.mark.parametrize("dim,vdim", [(4, 8), (36, 20), (64, 64), (100, 36)])
def test_fp32_values_that_are_not_finite(pkg, dim, vdim):
    """An infinite value stays in its column of the state, whatever the key channels are rounded up to; the head's other columns are
    divided by an infinite norm, in registers as token after token."""
    layer = Layer(pkg, 2, dim, vdim, 4.0, F32, seed=13)
    y, al = layer.rows(21)
    y.abs_()
    y[9, layer.cols[2] + 3] = float("inf")
    got, state = {}, {}
    for path in (0, STEP):
        state[path] = layer.states(1)
        got[path] = layer.run(y, al, [(0, 21, 0)], range(21), state[path], path)
    assert np.array_equal(np.isnan(got[0]), np.isnan(got[STEP])) and np.isnan(got[0]).sum() == 12
    assert torch.equal(state[0].isinf(), state[STEP].isinf()) and not state[0].isnan().any()
    finite = ~np.isnan(got[0])
    np.testing.assert_allclose(got[0][finite], got[STEP][finite], rtol=1e-5, atol=1e-6)


@pytest.mark.parametrize("heads,dim,vdim", [(10, 24, 256), (10, 64, 248), (8, 128, 256)])
def test_a_sequence_does_not_depend_on_its_company(pkg, heads, dim, vdim):
    """Alone and among five others: the same bits, and those of the equations."""
    layer = Layer(pkg, heads, dim, vdim, 4.0, BF, seed=11)
    lens = (100, 17, 40, 33, 64, 16)
    y, al = layer.rows(sum(lens))
    segments, pos = [(sum(lens[:i]), n, i) for i, n in enumerate(lens)], np.concatenate([np.arange(n) for n in lens])
    state = layer.states(len(lens))
    got = layer.run(y, al, segments, pos, state, CHUNK)
    for r0, n, slot in segments:
        alone = layer.states(1)
        assert np.array_equal(layer.run(y[r0:r0 + n], al[r0:r0 + n], [(0, n, 0)], range(n), alone, CHUNK), got[r0:r0 + n]), n
        assert torch.equal(alone[0], state[slot]), n
        want, last = layer.want(y[r0:r0 + n], al[r0:r0 + n])
        close(got[r0:r0 + n], want, BF, n)
        state_close(state[slot], last)


@pytest.mark.parametrize("path,dtype,heads,dim,vdim", [(STEP, F32, 3, 5, 7), (CHUNK, BF, 5, 56, 40), (0, BF, 2, 128, 128), (0, BF, 2, 64, 64)])
def test_portions_carry_the_state(pkg, path, dtype, heads, dim, vdim):
    """Any cut gives the outputs of the whole, with two sequences in unequal portions per call and the rows of a call in any
    order; both kernels take turns when the choice is left open."""
    layer = Layer(pkg, heads, dim, vdim, 8.0, dtype, seed=3)
    (ya, ala), (yb, alb) = layer.rows(143), layer.rows(90)
    wa, sa = layer.want(ya, ala)
    wb, sb = layer.want(yb, alb)
    state = layer.states(3)
    at = [0, 0]
    for na, nb in [(2, 40), (30, 1), (1, 2), (64, 16), (17, 31), (29, 0)]:
        ra, rb = slice(at[0], at[0] + na), slice(at[1], at[1] + nb)
        y, al = torch.cat([yb[rb], ya[ra]]), torch.cat([alb[rb], ala[ra]])
        segs = ([(0, nb, 2)] if nb else []) + [(nb, na, 0)]
        pos = list(range(rb.start, rb.stop)) + list(range(ra.start, ra.stop))
        got = layer.run(y, al, segs, pos, state, path)
        if nb:
            close(got[:nb], wb[rb], dtype, (na, nb))
        close(got[nb:], wa[ra], dtype, (na, nb))
        at = [ra.stop, rb.stop]
    assert at == [143, 90]
    state_close(state[0], sa)
    state_close(state[2], sb)


@pytest.mark.parametrize("path,dtype", [(STEP, F32), (STEP, BF), (CHUNK, BF)])
@pytest.mark.parametrize("z_mean,z_std,tau", [(-30.0, 5.0, 1.0), (-3.0, 30.0, 0.5), (60.0, 1.0, 16.0), (0.0, 200.0, 1.0), (-100.0, 1.0, 16.0)])
def test_strong_and_vanishing_decays(pkg, path, dtype, z_mean, z_std, tau):
    """Channels that forget everything at once, that forget nothing, and both in turn: nothing overflows and nothing is lost."""
    layer = Layer(pkg, 2, 40, 48, tau, dtype, z_mean, z_std, seed=5)
    y, al = layer.rows(75)
    state = layer.states(1)
    got = layer.run(y, al, [(0, 75, 0)], range(75), state, path)
    want, last = layer.want(y, al)
    close(got, want, dtype)
    state_close(state[0], last)


@pytest.mark.parametrize("path,dtype", [(STEP, F32), (CHUNK, BF)])
def test_a_far_token_is_remembered_for_hundreds_of_tokens(pkg, path, dtype):
    """Without decay the value written at token 3 is read back by the only query that matches its key, 500 tokens later."""
    layer = Layer(pkg, 1, 16, 32, 1.0, dtype, z_mean=80.0, z_std=0.0, seed=7)
    y, al = layer.rows(520)
    c = layer.cols
    y[:, c[0]:c[0] + 16], y[:, c[1]:c[1] + 16] = 0, 0
    y[:, c[1] + 1] = 1.0         # every key is unit vector 1 ...
    y[3, c[1]:c[1] + 16] = 0
    y[3, c[1] + 9] = 1.0         # ... but token 3's is unit vector 9
    y[503, c[0] + 9] = 4.0
    got = layer.run(y, al, [(0, 520, 0)], range(520), layer.states(1), path)
    v, g = (y[r, k:k + 32].double().cpu().numpy() for r, k in ((3, c[2]), (503, c[3])))
    close(got[503], bo.rms_norm(v, layer.norm.double().cpu().numpy(), 1e-4) * g * bo.sigmoid(g), dtype)
    assert np.abs(got[502]).max() == 0  # (a query of zeros)


def test_a_decode_step_takes_one_row_per_sequence(pkg):
    """Without a table row i is the next token of sequence i, at positions of their own."""
    from llm_experiments_b200 import recurrent
    from llm_experiments_b200.serving import RowSegments

    layer = Layer(pkg, 4, 64, 96, 16.0, BF, seed=9)
    state = torch.randn((3, 4, 64, 96), generator=layer.gen, device="cuda")
    before = state.double().cpu().numpy()
    y, al = layer.rows(3)
    out = torch.empty((3, 4 * 96), dtype=BF, device="cuda")
    pos = torch.tensor([12, 0, 1], dtype=torch.int32, device="cuda")
    pkg.gpu.batch_begin(layer.ctx)
    recurrent.gated_linear_attention(layer.ctx, wrap(pkg, y), layer.cols, wrap(pkg, al), layer.shape,
                                     pkg.gpu.GPUBuffer1D(buffer=layer.norm, shape=(96,), size=96), 1e-4, RowSegments(None, 3, 1), pos, state,
                                     wrap(pkg, out))
    pkg.gpu.batch_commit(layer.ctx)
    for i in range(3):
        want, last = layer.want(y[i:i + 1], al[i:i + 1], None if i == 1 else before[i])
        close(out[i:i + 1].double().cpu().numpy(), want, BF, i)
        state_close(state[i], last)


def test_segments_outside_the_buffers_are_refused(pkg):
    layer = Layer(pkg, 2, 16, 16, 2.0, BF)
    y, al = layer.rows(20)
    for path in (STEP, CHUNK):
        for seg in ((0, 21, 0), (5, 16, 0), (0, 20, 1), (-1, 4, 0)):
            with pytest.raises(RuntimeError, match="position"):
                layer.run(y, al, [seg], range(20), layer.states(1), path)


@pytest.mark.parametrize("heads,dim,vdim", [(2, 24, 40), (3, 128, 256), (2, 64, 72)])
def test_spans_of_chunks(pkg, heads, dim, vdim):
    """Lengths around 256 tokens and 512, in the company of each other and of short ones, then each continued by a portion
    of another length: the outputs and states of the equations, and alone the same bits."""
    layer = Layer(pkg, heads, dim, vdim, 16.0, BF, z_mean=2.0, z_std=1.0, seed=17)
    first, then = (255, 256, 257, 511, 513, 30, 770), (300, 17, 256, 1, 273, 520, 16)
    state, alone, last = layer.states(len(first)), [layer.states(1) for _ in first], [None] * len(first)
    for lens, start in ((first, [0] * len(first)), (then, first)):
        y, al = layer.rows(sum(lens))
        segments = [(sum(lens[:i]), n, i) for i, n in enumerate(lens)]
        got = layer.run(y, al, segments, np.concatenate([s + np.arange(n) for s, n in zip(start, lens)]), state, CHUNK)
        for (r0, n, i), s in zip(segments, start):
            part = slice(r0, r0 + n)
            assert np.array_equal(layer.run(y[part], al[part], [(0, n, 0)], s + np.arange(n), alone[i], CHUNK), got[part]), (n, s)
            assert torch.equal(alone[i][0], state[i]), (n, s)
            want, last[i] = layer.want(y[part], al[part], last[i])
            close(got[part], want, BF, (n, s))
            state_close(state[i], last[i])


def test_spans_over_slices_of_a_bounded_workspace(pkg):
    """Many sequences of several hundred tokens, which one slice of the workspace does not hold: the bits of each alone."""
    layer = Layer(pkg, 8, 128, 256, 16.0, BF, z_mean=2.0, z_std=1.0, seed=19)
    lens = (700, 513, 300) * 8
    y, al = layer.rows(sum(lens))
    segments, pos = [(sum(lens[:i]), n, i) for i, n in enumerate(lens)], np.concatenate([np.arange(n) for n in lens])
    state = layer.states(len(lens))
    got = layer.run(y, al, segments, pos, state, CHUNK)
    for r0, n, slot in segments[:3] + segments[-3:]:
        alone = layer.states(1)
        assert np.array_equal(layer.run(y[r0:r0 + n], al[r0:r0 + n], [(0, n, 0)], range(n), alone, CHUNK), got[r0:r0 + n]), n
        assert torch.equal(alone[0], state[slot]), n


def test_portions_of_whole_chunks_change_no_bit(pkg):
    """A sequence in one run, and cut at multiples of sixteen tokens: one chain of chunks either way."""
    layer = Layer(pkg, 3, 128, 256, 16.0, BF, z_mean=2.0, z_std=1.0, seed=41)
    y, al = layer.rows(1000)
    whole, parts = layer.states(1), layer.states(1)
    want = layer.run(y, al, [(0, 1000, 0)], range(1000), whole, CHUNK)
    for a, b in ((0, 160), (160, 512), (512, 1000)):
        assert np.array_equal(layer.run(y[a:b], al[a:b], [(0, b - a, 0)], range(a, b), parts, CHUNK), want[a:b]), a
    assert torch.equal(whole, parts)


def test_an_infinite_state_is_not_turned_into_nan_by_a_span(pkg):
    """Decays whose product over some hundred tokens is below the smallest number: what is infinite stays so."""
    layer = Layer(pkg, 1, 16, 32, 1.0, BF, z_mean=-0.7, z_std=0.0, seed=23)
    y, al = layer.rows(600)
    state = torch.ones((1, 1, 16, 32), device="cuda")
    state[0, 0, 3, 5] = float("inf")
    layer.run(y, al, [(0, 600, 0)], 10 + np.arange(600), state, CHUNK)
    assert torch.isinf(state[0, 0, 3, 5]) and torch.isfinite(state).sum() == 16 * 32 - 1


@pytest.mark.parametrize("heads,dim,vdim", [(2, 20, 40), (3, 128, 256), (2, 64, 72), (1, 4, 4), (5, 64, 256)])
def test_spans_of_tokens_in_fp32(pkg, heads, dim, vdim):
    """As for chunks, with spans of 64 tokens of segments of more than 192 (heads of up to 64 key channels); the decays of half of the channels
    multiply up to nothing over a span."""
    layer = Layer(pkg, heads, dim, vdim, 4.0, F32, z_mean=2.0, z_std=4.0, seed=29)
    first, then = (63, 64, 192, 193, 129, 5, 400), (256, 17, 64, 2, 200, 320, 16)
    state, last = layer.states(len(first)), [None] * len(first)
    for lens, start in ((first, [0] * len(first)), (then, first)):
        y, al = layer.rows(sum(lens))
        segments, was = [(sum(lens[:i]), n, i) for i, n in enumerate(lens)], state.clone()
        got = layer.run(y, al, segments, np.concatenate([s + np.arange(n) for s, n in zip(start, lens)]), state, 0)
        for (r0, n, i), s in zip(segments, start):
            part = slice(r0, r0 + n)
            assert np.array_equal(layer.run(y[part], al[part], [(0, n, 0)], s + np.arange(n), was[i:i + 1], 0), got[part]), (n, s)
            assert torch.equal(was[i], state[i]), (n, s)
            want, last[i] = layer.want(y[part], al[part], last[i])
            close(got[part], want, F32, (n, s))
            state_close(state[i], last[i])


def test_spans_of_tokens_over_slices_of_a_bounded_workspace(pkg):
    layer = Layer(pkg, 8, 64, 128, 16.0, F32, z_mean=2.0, z_std=1.0, seed=31)
    lens = (16300, 64, 200, 16256)  # 255 spans of four segments, 254 at a time
    y, al = layer.rows(sum(lens))
    segments, pos = [(sum(lens[:i]), n, i) for i, n in enumerate(lens)], np.concatenate([np.arange(n) for n in lens])
    state = layer.states(len(lens))
    got = layer.run(y, al, segments, pos, state, 0)
    for r0, n, slot in segments:
        alone = layer.states(1)
        assert np.array_equal(layer.run(y[r0:r0 + n], al[r0:r0 + n], [(0, n, 0)], range(n), alone, 0), got[r0:r0 + n]), n
        assert torch.equal(alone[0], state[slot]), n


def test_an_infinite_state_is_not_turned_into_nan_by_a_span_of_tokens(pkg):
    layer = Layer(pkg, 1, 16, 32, 1.0, F32, z_mean=-1.5, z_std=0.0, seed=37)  # 0.18 ** 64 is below the smallest number
    y, al = layer.rows(300)
    state = torch.ones((1, 1, 16, 32), device="cuda")
    state[0, 0, 3, 5] = float("inf")
    layer.run(y, al, [(0, 300, 0)], 10 + np.arange(300), state, 0)
    assert torch.isinf(state[0, 0, 3, 5]) and torch.isfinite(state).sum() == 16 * 32 - 1
