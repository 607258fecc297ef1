"""Host-side behaviour of the reference API mirror, on CPU tensors: the same checks, texts
and state changes as simple-llm/src/gpu/gpu_kv_cache.py and gpu_ops.py, exercised up to (not
including) the kernel launch."""
import pytest
import torch


@pytest.fixture()
def ctx(pkg):
    gpu = pkg.gpu
    return gpu.GPUContext(device=torch.device("cpu"), config=gpu.GPUConfig(), batch_state=None)


def _cfg(gpu, **kw):
    base = dict(batch_size=2, max_seq_len=8, n_layers=2, n_heads=2, head_dim=16)
    base.update(kw)
    return gpu.KVCacheConfig(**base)


def test_create_validates_dimensions_like_the_reference(pkg, ctx):
    gpu = pkg.gpu
    for field in ["batch_size", "max_seq_len", "n_layers", "n_heads", "head_dim"]:
        with pytest.raises(ValueError, match=f"{field} must be > 0, got 0"):
            gpu.kv_cache_create(ctx, _cfg(gpu, **{field: 0}))
    with pytest.raises(ValueError, match="layout"):
        gpu.kv_cache_create(ctx, _cfg(gpu, layout="htbd"))


def test_create_shapes_and_zero_fill(pkg, ctx):
    gpu = pkg.gpu
    cache = gpu.kv_cache_create(ctx, _cfg(gpu))
    assert len(cache.layers) == 2 and cache.current_len == 0
    assert cache.layers[0].k_cache.shape == (2 * 8, 2 * 16)  # [B*T_max, H*D] as the reference
    assert float(cache.layers[1].v_cache.buffer.abs().sum()) == 0.0
    bhtd = gpu.kv_cache_create(ctx, _cfg(gpu, layout="bhtd", dtype=torch.bfloat16))
    assert bhtd.layers[0].k_cache.shape == (2 * 2 * 8, 16) and bhtd.layers[0].k_cache.buffer.dtype == torch.bfloat16
    paged = gpu.kv_cache_create(ctx, _cfg(gpu, block_size=4, n_blocks=10, ragged=True))
    assert paged.block_table.shape == (2, 2) and paged.layers[0].k_cache.shape == (10 * 2 * 4, 16)
    assert paged.seq_lens.tolist() == [0, 0]
    with pytest.raises(ValueError, match="n_blocks"):
        gpu.kv_cache_create(ctx, _cfg(gpu, block_size=4, n_blocks=3))


def test_reset_and_set_lengths(pkg, ctx):
    gpu = pkg.gpu
    cache = gpu.kv_cache_create(ctx, _cfg(gpu, ragged=True))
    cache.current_len = 5
    gpu.kv_cache_reset(cache)
    assert cache.current_len == 0
    gpu.kv_cache_set_lengths(cache, [3, 7])
    assert cache.current_len == 7 and cache.seq_lens.tolist() == [3, 7]
    with pytest.raises(ValueError):
        gpu.kv_cache_set_lengths(cache, [3, 9])


def test_update_checks_fire_before_the_launch(pkg, ctx):
    gpu = pkg.gpu
    cache = gpu.kv_cache_create(ctx, _cfg(gpu))
    good = gpu.gpu_buffer_2d_create(ctx, 2, 32)
    with pytest.raises(ValueError, match=r"layer_idx 2 out of range \[0, 2\)"):
        gpu.kv_cache_update(ctx, cache, 2, good, good)
    cache.current_len = 8
    with pytest.raises(ValueError, match="Cache is full: current_len=8, max_seq_len=8"):
        gpu.kv_cache_update(ctx, cache, 0, good, good)
    cache.current_len = 0
    bad = gpu.gpu_buffer_2d_create(ctx, 2, 16)
    with pytest.raises(ValueError, match="new_k shape mismatch"):
        gpu.kv_cache_update(ctx, cache, 0, bad, good)
    with pytest.raises(ValueError, match="new_v shape mismatch"):
        gpu.kv_cache_update(ctx, cache, 0, good, bad)
    # no open batch: the operation is refused on the host
    with pytest.raises(RuntimeError, match="batch_begin"):
        gpu.kv_cache_update(ctx, cache, 0, good, good)
    assert cache.current_len == 0


def test_attention_checks(pkg, ctx):
    gpu = pkg.gpu
    cache = gpu.kv_cache_create(ctx, _cfg(gpu, max_seq_len=512))
    q = gpu.gpu_buffer_2d_create(ctx, 2, 32)
    with pytest.raises(ValueError, match="Cache is empty: current_len=0"):
        gpu.attention_with_kv_cache(ctx, cache, 0, q, q)
    cache.current_len = 3
    with pytest.raises(ValueError, match="out of range"):
        gpu.attention_with_kv_cache(ctx, cache, -1, q, q)
    with pytest.raises(ValueError, match="q_new shape mismatch"):
        gpu.attention_with_kv_cache(ctx, cache, 0, gpu.gpu_buffer_2d_create(ctx, 2, 31), q)
    with pytest.raises(ValueError, match="output shape mismatch"):
        gpu.attention_with_kv_cache(ctx, cache, 0, q, gpu.gpu_buffer_2d_create(ctx, 1, 32))
    # the reference's 256-token limit is opt-in
    cache.current_len = 300
    ctx.config.enforce_reference_decode_limit = True
    with pytest.raises(ValueError, match=r"current_len \(300\) exceeds maximum supported"):
        gpu.attention_with_kv_cache(ctx, cache, 0, q, q)


def test_flash_attention_checks(pkg, ctx):
    gpu = pkg.gpu
    mk = lambda r, c: gpu.gpu_buffer_2d_create(ctx, r, c)  # noqa: E731
    Q = mk(8, 32)
    L = gpu.gpu_buffer_1d_create(ctx, 16)
    ctx.config.flash_attn_max_head_dim = 8
    with pytest.raises(ValueError, match="head_dim 16 exceeds maximum supported by config: 8"):
        gpu.flash_attention(ctx, Q, Q, Q, Q, L, L, 2, 4, 2, 16)
    ctx.config.flash_attn_max_head_dim = 128
    with pytest.raises(ValueError, match="Invalid dimensions"):
        gpu.flash_attention(ctx, Q, Q, Q, Q, L, L, 0, 4, 2, 16)
    with pytest.raises(ValueError, match="K shape mismatch"):
        gpu.flash_attention(ctx, Q, mk(8, 16), Q, Q, L, L, 2, 4, 2, 16)
    with pytest.raises(ValueError, match="L shape mismatch"):
        gpu.flash_attention(ctx, Q, Q, Q, Q, gpu.gpu_buffer_1d_create(ctx, 8), L, 2, 4, 2, 16)


def test_batch_rules(pkg, ctx):
    gpu = pkg.gpu
    with pytest.raises(RuntimeError, match="Batch already submitted or not initialized"):
        gpu.batch_commit(ctx)


def test_buffer_helpers(pkg, ctx):
    import numpy as np

    gpu = pkg.gpu
    with pytest.raises(ValueError, match="Buffer dimensions must be positive"):
        gpu.gpu_buffer_2d_create(ctx, 0, 4)
    with pytest.raises(ValueError, match="Buffer size must be positive"):
        gpu.gpu_buffer_1d_create(ctx, 0)
    with pytest.raises(ValueError, match="doesn't match buffer shape"):
        gpu.gpu_buffer_2d_create(ctx, 2, 2, np.zeros((2, 3), dtype=np.float32))
    with pytest.raises(ValueError, match="Unsupported dtype"):
        gpu.gpu_buffer_2d_create(ctx, 2, 2, np.zeros((2, 2), dtype=np.float64))
    buf = gpu.gpu_buffer_2d_create(ctx, 2, 2, np.arange(4, dtype=np.float32).reshape(2, 2))
    assert buf.shape == (2, 2) and buf.size == 4


def test_perf_monitor_mirrors_the_reference(pkg):
    """simple-llm/src/gpu/gpu_device.py:569-608: record, count, aggregate, reset."""
    gpu = pkg.gpu
    mon = gpu.perf_monitor_create()
    gpu.perf_monitor_kernel_time_record(mon, "kv_cache_update", 0.5)
    gpu.perf_monitor_kernel_time_record(mon, "kv_cache_update", 1.5)
    gpu.perf_monitor_kernel_time_record(mon, "flash_attention", 2.0)
    gpu.perf_monitor_submission_record(mon)
    stats = gpu.perf_monitor_stats_get(mon)
    assert stats.total_submissions == 1
    upd = stats.kernel_times["kv_cache_update"]
    assert (upd.count, upd.total_ms, upd.avg_ms, upd.min_ms, upd.max_ms) == (2, 2.0, 1.0, 0.5, 1.5)
    assert stats.kernel_times["flash_attention"].count == 1
    gpu.perf_monitor_reset(mon)
    assert gpu.perf_monitor_stats_get(mon).total_submissions == 0 and not mon.kernel_times


def test_embedding_checks_like_the_reference(pkg, ctx):
    """simple-llm/src/gpu/gpu_pass_forward.py:110-128."""
    gpu = pkg.gpu
    table = gpu.gpu_buffer_2d_create(ctx, 10, 16)
    pos = gpu.gpu_buffer_2d_create(ctx, 6, 16)
    ids = gpu.gpu_buffer_1d_create(ctx, 8, dtype=torch.int32)
    out = gpu.gpu_buffer_2d_create(ctx, 8, 16)
    with pytest.raises(ValueError, match="Invalid batch_size=0 or seq_len=4"):
        gpu.embedding(ctx, table, pos, ids, out, 0, 4)
    with pytest.raises(ValueError, match="Embedding dimension mismatch: table has 16, pos_encoding has 8"):
        gpu.embedding(ctx, table, gpu.gpu_buffer_2d_create(ctx, 6, 8), ids, out, 2, 4)
    with pytest.raises(ValueError, match="Sequence length 7 exceeds context size 6"):
        gpu.embedding(ctx, table, pos, ids, out, 2, 7)
    with pytest.raises(ValueError, match="input_ids shape mismatch"):
        gpu.embedding(ctx, table, pos, gpu.gpu_buffer_1d_create(ctx, 7, dtype=torch.int32), out, 2, 4)
    with pytest.raises(ValueError, match="output shape mismatch"):
        gpu.embedding(ctx, table, pos, ids, gpu.gpu_buffer_2d_create(ctx, 8, 8), 2, 4)
    with pytest.raises(RuntimeError, match="batch_begin"):
        gpu.embedding(ctx, table, pos, ids, out, 2, 4)


def test_decoder_state_and_graphed_step_checks(pkg, ctx):
    """model.py on CPU tensors: shapes of the state, and the checks that fire before anything is launched."""
    import numpy as np

    from llm_experiments_b200 import model

    cfg = model.DecoderConfig(vocab_size=64, context_size=32, embedding_dim=128, n_heads=1, n_layers=2)
    pe = model.positional_encoding(cfg.context_size, cfg.embedding_dim)
    assert pe.shape == (32, 128) and pe[0, 0] == 0.0 and pe[0, 1] == 1.0  # sin(0), cos(0) interleaved
    E, V = cfg.embedding_dim, cfg.vocab_size
    z = lambda *shape: np.zeros(shape, dtype=np.float32)  # noqa: E731
    layer = dict(ln1_gamma=z(E), ln1_beta=z(E), wq=z(E, E), wk=z(E, E), wv=z(E, E), wo=z(E, E), ln2_gamma=z(E),
                 ln2_beta=z(E), w1=z(E, 4 * E), b1=z(4 * E), w2=z(4 * E, E), b2=z(E))
    params = dict(embedding=z(V, E), pos_encoding=pe, layers=[layer, layer], lnf_gamma=z(E), lnf_beta=z(E),
                  out_proj=z(E, V))
    weights = model.weights_from_numpy(ctx, cfg, params)
    assert weights.out_proj.shape == (E, V) and weights.layers[1].w1.buffer.dtype == torch.bfloat16
    state = model.decoder_state_create(ctx, cfg, weights, batch_size=3)
    assert len(state.caches) == 2 and state.logits.shape == (3, V) and state.caches[0].layout == "bhtd"
    assert model.launches_per_decode_step(cfg) == 1 + 8 * 2 + 3
    with pytest.raises(ValueError, match="exceeds context size"):
        model.decoder_state_create(ctx, cfg, weights, batch_size=3, max_seq_len=33)
    with pytest.raises(ValueError, match="ragged=True"):
        model.GraphedDecodeStep(ctx, state)  # lengths must live on the device
    tok = pkg.gpu.gpu_buffer_1d_create(ctx, 3, dtype=torch.int32)
    with pytest.raises(RuntimeError, match="batch_begin"):
        model.decode_step(ctx, state, tok)
    for cache in state.caches:
        cache.current_len = 32
    with pytest.raises(ValueError, match="Cache is full"):
        model.decode_step(ctx, state, tok)


@pytest.mark.parametrize("heads,dim,vdim,max_n", [(8, 64, 256, 100), (3, 128, 64, 1000), (16, 32, 256, 5000), (1, 128, 8, 40)])
def test_a_recurrence_workspace_is_enough_for_fewer_segments(pkg, heads, dim, vdim, max_n):
    """A program may ask for its workspace once, for the most segments and tokens of a step."""
    size = lambda n, t: pkg._native.lib.b2kv_gla_workspace_bytes(heads, dim, vdim, n, t, pkg._native.DTYPE_BF16, 0)  # noqa: E731
    sizes = [size(n, max_n) for n in range(1, 65)]
    assert sizes == sorted(sizes) and 0 < size(7, max_n // 2) <= size(7, max_n)


def test_memory_of_a_captured_step_stays_when_it_is_replaced(pkg, ctx, monkeypatch):
    """A graph knows a step's scratch memory by its address: what later steps replace is not given back, and nothing else is kept."""
    import types
    import weakref

    from llm_experiments_b200 import batch, serving

    class State(serving.SequenceState):
        def run(self, ctx, step):
            self.rows("x", step.rows, 4, torch.float32)
            self.scratch["linear"] = batch.scratch(self.scratch.get("linear"), 100 * step.rows, torch.device("cpu"))
            for c in self.caches:
                c.workspace = batch.scratch(c.workspace, 10 * step.rows, torch.device("cpu"))

    cache = pkg.gpu.kv_cache_create(ctx, _cfg(pkg.gpu, n_layers=1, ragged=True))
    lens = types.SimpleNamespace(is_cuda=True, device=torch.device("cpu"), data_ptr=lambda: 0)
    state = State(batch_size=2, max_seq_len=8, dtype=torch.float32, owned={0: cache}, seq_lens=lens, lengths=[0, 0])
    monkeypatch.setattr(serving, "_lib", types.SimpleNamespace(b2kv_advance_lengths=lambda *a: 0))
    monkeypatch.setattr(serving, "batch_op_begin", lambda ctx: 0)
    capturing = [False]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: capturing[0])
    alive = []

    def step(rows):
        state.run(ctx, types.SimpleNamespace(rows=rows))
        alive.append([weakref.ref(t) for t in (state.scratch["x"], state.scratch["linear"], cache.workspace)])

    token = types.SimpleNamespace(buffer=None)
    serving.decode_step(ctx, state, token)
    step(2)
    step(5)
    assert [r() is None for r in alive[0]] == [True] * 3  # (no graph yet)
    capturing[0] = True
    serving.decode_step(ctx, state, token)
    capturing[0] = False
    assert state.captured
    for rows in (9, 17):
        step(rows)
    assert [r() is None for r in alive[1]] == [False] * 3  # the captured step's
    assert [r() is None for r in alive[2]] == [True] * 3  # what came behind it and was too small in its turn
    assert state.scratch["linear"].numel() == 1700 and state.scratch["x"].shape == (17, 4)


def test_memory_of_recurrent_layers_is_not_shared_by_two_models(pkg, ctx, monkeypatch):
    """Two states of one context may have steps under way on two streams: each brings its own memory, and a call that brings none does not
    write to what another fp32 call may still use."""
    import types

    from llm_experiments_b200 import recurrent
    from llm_experiments_b200.serving import RowSegments

    seen = []
    lib = types.SimpleNamespace(b2kv_gla_workspace_bytes=lambda *a: 1000, b2kv_gla=lambda a, status, stream: seen.append(a._obj.workspace) or 0)
    monkeypatch.setattr(recurrent, "_native", types.SimpleNamespace(lib=lib, check=lambda rc: None, GlaArgs=pkg._native.GlaArgs))
    monkeypatch.setattr(recurrent, "batch_op_begin", lambda ctx: 0)
    monkeypatch.setattr(recurrent, "dev_status_ptr", lambda ctx: 0)
    two = lambda t: pkg.gpu.GPUBuffer2D(buffer=t, shape=tuple(t.shape), size=t.numel())  # noqa: E731
    kept = [{}, {}, None, None]
    alive = []  # (so that no address comes twice)
    real = torch.empty
    monkeypatch.setattr(torch, "empty", lambda *a, **kw: alive.append(real(*a, **kw)) or alive[-1])
    for again in range(2):
        for scratch in kept:
            y = two(torch.zeros((300, 64)))
            recurrent.gated_linear_attention(ctx, y, (0, 16, 32, 48), two(torch.zeros((300, 16))), recurrent.GlaShape(1, 16, 16, 1.0),
                                             pkg.gpu.GPUBuffer1D(buffer=torch.zeros(16), shape=(16,), size=16), 1e-5, RowSegments(None, 1, 300),
                                             torch.zeros(300, dtype=torch.int32), torch.zeros((1, 1, 16, 16)), two(torch.zeros((300, 16))), scratch=scratch)
    assert len(set(seen[:4])) == 4 and seen[4:6] == seen[:2] and len(set(seen)) == 6 and ctx.recurrent_workspace is None


def test_few_long_runs_have_a_table_of_their_own(pkg):
    """One long run among many single rows does not make them all reserve its memory; what goes row by row stays with the kernel of runs."""
    from llm_experiments_b200 import serving

    size = lambda runs, most: pkg._native.lib.b2kv_gla_workspace_bytes(6, 64, 128, len(runs), most, 0, 0) if runs else 0  # noqa: E731
    singles = [(i, 1, i) for i in range(64)]
    runs = singles + [(64, 2000, 64), (2064, 192, 65)]
    rest, long, most = serving.split_runs(runs)
    assert rest == singles + [(2064, 192, 65)] and long == [(64, 2000, 64)] and most == 192
    assert size(rest, most) == 0 and 0 < 20 * size(long, 2000) < size(runs, 2000)
    assert serving.split_runs(singles + [(64, 193, 64)])[1:] == ([(64, 193, 64)], 2)
    from llm_experiments_b200 import recurrent

    kinds = [((6, 64, 128), torch.float32), ((6, 64, 128), torch.bfloat16), ((4, 128, 256), torch.float32), ((16, 64, 256), torch.float32)]
    assert [recurrent.cuts_runs(recurrent.GlaShape(*shape, 16.0), dtype) for shape, dtype in kinds] == [True, False, False, False]
    for together in (singles, singles[:15] + [(15, 400, 15)], singles[:20] + [(20 + 300 * i, 300, 20 + i) for i in range(7)], [(0, 5, 1)], []):
        assert serving.split_runs(together) == (together, [], max((n for _, n, _ in together), default=0))


def test_memory_of_fp32_products_has_a_ceiling(pkg):
    """Rows and columns around the edges of the rule, and products whose parts would take gigabytes."""
    native = pkg._native

    def size(rows, k, n, groups=1):
        return native.lib.b2kv_linear_workspace_bytes(native.linear_args(256, 256, 0, 0, 0, k, 0, n, 0, 0, [(256, n, 0, n, 0)], rows, k, n, groups, 0, 0, 0, 0.0))

    assert size(256, 4096, 4096) == 0 < size(257, 1024, 4096)  # three rows of tiles
    assert size(384, 1024, 5461 // 4 * 4) > 0 == size(384, 1024, 5464)  # w's parts: 32 MB,
    assert size(512, 1024, 19112) > 0 == size(512, 1024, 19116)  # 112 MB,
    assert size(513, 1024, 27304) > 0 == size(513, 1024, 27308)  # 160 MB
    assert size(257, 64, 384 * 128) == size(693, 64, 64) == size(1000, 4096, 4096, 2) == 0
    for rows, k, n in ((2048, 2048, 32768), (4096, 4096, 131072), (100000, 4096, 1024), (20000, 4096, 4096)):
        assert size(rows, k, n) == 0
    assert max(size(r, k, n) for r in (300, 1000, 5000, 14000) for k in (768, 4096) for n in (768, 4096, 6400)) <= 512 << 20
