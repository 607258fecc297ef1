"""Workloads that stand for what users of this framework have it do, through its public entry points.

Kinds of case:

* ``token``: one step of a decoding loop at the level of the operators (``kv_cache_update``, ``attention_with_kv_cache``) over a
  cache that already holds ``lo`` .. ``hi`` tokens per sequence (``lo == hi``: one shared length), in both storage types, in the
  reference's cache layout, the native one and paged;
* ``prompt``: causal attention over whole prompts (``flash_attention``) with its statistics and, with ``cache``, the cache write;
* ``gpt``, ``gigezen``, ``bamasun``: models.  ``phase="step"`` generates one token for each of ``B`` sequences with a captured
  step (``GraphedDecodeStep``), ``phase="mixed"`` is a step of a server: ``P`` new prompts of ``lo`` .. ``hi`` tokens beside ``S``
  sequences that hold ``past`` tokens or fewer and go on by one.

Everything a case computes from is drawn from its seed on the GPU, weights included.  Decoding loops let their sequences grow and
give them back after ``GROW`` tokens, as a program does whose sequences end.
"""
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parent.parent
GROW = 64
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def package():
    name = "llm_experiments_b200"  # the folder's name has a hyphen
    if name not in sys.modules:
        folder = ROOT / "llm-experiments_b200"
        spec = importlib.util.spec_from_file_location(name, folder / "__init__.py", submodule_search_locations=[str(folder)])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


_CTX = []


def context():
    if not _CTX:
        _CTX.append(package().gpu.context_create(0))
        _CTX[0].config.flash_attn_max_head_dim = 256
    return _CTX[0]


# ---------------------------------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------------------------------

def listed():
    return [
        # The reference's own small model (4 heads of 64, fp32, batch of one, its cache layout) in the middle of a generation: the
        # smallest call there is, nothing but latency.
        dict(name="token_one_f32", kind="token", B=1, H=4, D=64, dtype="f32", layout="bthd", block=0, lo=160, hi=160),
        # A handful of conversations with short histories.
        dict(name="token_few_bf16", kind="token", B=8, H=32, D=128, dtype="bf16", layout="bhtd", block=0, lo=128, hi=1024),
        # The benchmark's batch: 64 sequences of 512 .. 8192 tokens.
        dict(name="token_batch_bf16", kind="token", B=64, H=32, D=128, dtype="bf16", layout="bhtd", block=0, lo=512, hi=8192),
        # A server with a block table: 16-token blocks anywhere in a pool, odd numbers of sequences, smaller heads.
        dict(name="token_paged_bf16", kind="token", B=13, H=24, D=64, dtype="bf16", layout="bhtd", block=16, lo=301, hi=5003),
        # A shape of the reference's own attention test: short prompts, fp32.
        dict(name="prompt_short_f32", kind="prompt", B=8, N=32, H=8, D=64, dtype="f32", cache="none"),
        # Prompts in the reference's storage type, of a length that fills no tile, into its cache.
        dict(name="prompt_f32", kind="prompt", B=2, N=1000, H=12, D=64, dtype="f32", cache="bthd"),
        # The benchmark's prompts.
        dict(name="prompt_batch_bf16", kind="prompt", B=8, N=4096, H=32, D=128, dtype="bf16", cache="bhtd"),
        # A model whose step is made of many short kernels: few sequences, short contexts.
        dict(name="gpt_step", kind="gpt", phase="step", E=4096, heads=32, layers=4, vocab=32768, B=8, lo=128, hi=1024),
        # Latent attention and mixtures of experts, the benchmark's batch.
        dict(name="gigezen_step", kind="gigezen", phase="step", dtype="bf16", width=4096, heads=32, ff=10880, experts=64, top=6,
             expert_ff=1408, window=4096, layers=4, vocab=32768, B=64, lo=512, hi=8192),
        # A server's step: three new prompts of odd lengths beside five running sequences.
        dict(name="gigezen_mixed", kind="gigezen", phase="mixed", dtype="bf16", width=2048, heads=16, ff=5440, experts=64, top=6,
             expert_ff=1408, window=1024, layers=2, vocab=32768, P=3, S=5, lo=203, hi=1777, past=900),
        # Grouped attention and gated linear attention over prompts.
        dict(name="bamasun_mixed", kind="bamasun", phase="mixed", dtype="bf16", width=2048, heads=16, kv_heads=4, gla_heads=8, dim=128,
             gla_vdim=256, ff=8192, layers=2, vocab=32768, P=2, S=4, lo=1500, hi=2048, past=700),
        # The same design in fp32, the size of model that is run in that type.
        dict(name="bamasun_mixed_f32", kind="bamasun", phase="mixed", dtype="f32", width=768, heads=12, kv_heads=4, gla_heads=6, dim=64,
             gla_vdim=128, ff=3072, layers=2, vocab=4096, P=3, S=3, lo=60, hi=400, past=200),
    ]


def spread(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["token", "token", "prompt", "prompt", "gpt", "gigezen", "bamasun", "bamasun"])
    dtype = rng.choice(["bf16", "bf16", "f32"])
    if kind == "token":
        layout, block = rng.choice([("bthd", 0), ("bhtd", 0), ("bhtd", 0), ("bhtd", 16), ("bhtd", 64)])
        c = dict(kind=kind, B=spread(rng, 1, 64), H=spread(rng, 2, 64), D=rng.choice([32, 64, 64, 128, 128]), dtype=dtype, layout=layout,
                 block=block, lo=0, hi=spread(rng, 32, 8192))
        while c["B"] * c["H"] * c["D"] * c["hi"] > 6e8:
            c["B" if c["B"] > 4 else "hi"] //= 2
        c["lo"] = rng.choice([c["hi"], max(1, c["hi"] // 16), max(1, c["hi"] // 16)])
        return c
    if kind == "prompt":
        c = dict(kind=kind, B=spread(rng, 1, 16), N=spread(rng, 17, 4096), H=spread(rng, 2, 32), D=rng.choice([32, 64, 64, 128, 128]),
                 dtype=dtype, cache=rng.choice(["none", "bthd", "bhtd", "paged"]))
        most = 4e11 if dtype == "bf16" and c["D"] > 32 else 1e11 if c["D"] > 32 else 3e10
        while c["B"] * c["H"] * c["D"] * 2.0 * c["N"] ** 2 > most:
            key = "B" if c["B"] > 1 else "H" if c["H"] > 4 else "N"
            c[key] = -(-c[key] // 2)
        return c
    if kind == "gpt":
        heads, hi = rng.choice([4, 8, 16, 24, 32]), spread(rng, 64, 2048)
        return dict(kind=kind, phase="step", E=heads * 128, heads=heads, layers=rng.randint(1, 4), vocab=rng.choice([4096, 32768]),
                    B=spread(rng, 8, 64), lo=max(1, hi // 8), hi=hi)
    heads = rng.choice([4, 8, 12, 16])
    if kind == "gigezen":
        c = dict(kind=kind, phase=rng.choice(["step", "mixed"]), dtype="bf16", width=128 * heads, heads=heads, ff=32 * rng.randint(24, 160),
                 experts=rng.choice([16, 32, 64]), top=rng.choice([2, 4, 6]), expert_ff=16 * rng.randint(16, 88), window=spread(rng, 128, 4096),
                 layers=2, vocab=rng.choice([4096, 32768]))
    else:
        dim = 128 if dtype == "bf16" else 64
        c = dict(kind=kind, phase=rng.choice(["step", "mixed"]) if dtype == "bf16" else "mixed", dtype=dtype, width=dim * heads, heads=heads,
                 kv_heads=heads // rng.choice([1, 2, 4]), gla_heads=heads // 2, dim=dim, gla_vdim=rng.choice([dim, 2 * dim]),
                 ff=32 * rng.randint(24, 200 if dtype == "bf16" else 96), layers=2, vocab=rng.choice([4096, 32768]))
    if c["phase"] == "step":
        hi = spread(rng, 128, 8192)
        c.update(B=spread(rng, 8, 64), lo=max(1, hi // 16), hi=hi)
    else:
        hi = spread(rng, 40, 2048 if c["dtype"] == "bf16" else 400)
        c.update(P=rng.randint(1, 4), S=rng.randint(0, 8), lo=max(17, hi // 4), hi=hi, past=spread(rng, 16, 2048 if c["dtype"] == "bf16" else 400))
    return c


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------

def generator(seed, salt):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + salt)


def normal(gen, shape, dtype, scale=1.0, mean=0.0):
    t = torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=gen)
    return t if scale == 1.0 and mean == 0.0 else t.mul_(scale).add_(mean)


def lengths(seed, n, lo, hi):
    return np.random.default_rng(int(seed)).integers(lo, hi + 1, size=n).tolist()


def token_inputs(c, seed):
    """Lengths, cache buffers as the framework lays them out, block table, and the step's rows."""
    dt, gen = DTYPES[c["dtype"]], generator(seed, 1)
    B, H, D, T, block = c["B"], c["H"], c["D"], c["hi"] + GROW + 1, c["block"]
    blocks = -(-T // block) if block else 0
    rows = (B * T, H * D) if c["layout"] == "bthd" else (B * H * T, D) if not block else (B * blocks * H * block, D)
    k, v = normal(gen, rows, dt), normal(gen, rows, dt)
    table = torch.randperm(B * blocks, generator=gen, device="cuda").to(torch.int32).view(B, blocks) if block else None
    q, nk, nv = (normal(gen, (B, H * D), dt) for _ in range(3))
    return lengths(seed, B, c["lo"], c["hi"]), T, k, v, table, q, nk, nv


def prompt_inputs(c, seed):
    gen, shape = generator(seed, 2), (c["B"] * c["N"], c["H"] * c["D"])
    return [normal(gen, shape, DTYPES[c["dtype"]]) for _ in range(3)]


def gpt_tensors(c, seed):
    """Matrices N(0, 1 / fan_in), norms near the identity, by the framework's names; interleaved sine and cosine positions."""
    E, V, T, gen, bf = c["E"], c["vocab"], c["hi"] + GROW + 1, generator(seed, 3), torch.bfloat16
    mat = lambda a, b: normal(gen, (a, b), bf, a ** -0.5)  # noqa: E731
    vec = lambda n, mean=0.0: normal(gen, (n,), bf, 0.1, mean)  # noqa: E731
    angle = torch.arange(T, dtype=torch.float64)[:, None] * torch.exp(torch.arange(0, E, 2, dtype=torch.float64) * -(math.log(10000.0) / E))
    pos = torch.stack([angle.sin(), angle.cos()], dim=-1).view(T, E).to("cuda").to(bf)
    layers = [dict(ln1_gamma=vec(E, 1.0), ln1_beta=vec(E), wq=mat(E, E), wk=mat(E, E), wv=mat(E, E), wo=mat(E, E), ln2_gamma=vec(E, 1.0),
                   ln2_beta=vec(E), w1=mat(E, 4 * E), b1=vec(4 * E), w2=mat(4 * E, E), b2=vec(E)) for _ in range(c["layers"])]
    return dict(embedding=normal(gen, (V, E), bf), pos_encoding=pos, layers=layers, lnf_gamma=vec(E, 1.0), lnf_beta=vec(E), out_proj=mat(E, V))


def gigezen_config(c):
    """Dense layers with latents of their own and mixtures that read them, in turn."""
    layers = []
    for i in range(c["layers"]):
        mixer = dict(heads=c["heads"], dim=128, rot_dim=64, vdim=128, kv_rank=512, scale=192 ** -0.5, rot=dict(base=10000.0, dims=64),
                     mask=dict(size=c["window"]))
        mlp = dict(kind="dense", ff=c["ff"], limit=7.0)
        if i % 2:
            mixer["kv_from"] = i - 1
            mlp = dict(kind="moe", expert=dict(ff=c["expert_ff"]),
                       router=dict(experts=c["experts"], top=c["top"], groups=dict(count=8, keep=4)))
        layers.append(dict(type="latent_attention", mixer=mixer, mlp=mlp))
    return dict(architecture="Gigezen", layers=layers, vocab=c["vocab"], width=c["width"], norm=dict(eps=1e-6))


def bamasun_config(c):
    """Attention and recurrence in turn; the third layer, where there is one, reads the first one's keys and values."""
    layers = []
    for i in range(c["layers"]):
        mlp = dict(kind="dense", ff=c["ff"])
        if i % 2:
            layers.append(dict(type="gla", mixer=dict(heads=c["gla_heads"], dim=c["dim"], vdim=c["gla_vdim"], tau=16.0), mlp=mlp))
            continue
        mixer = dict(heads=c["heads"], kv_heads=c["kv_heads"], dim=c["dim"], vdim=c["dim"], scale=c["dim"] ** -0.5,
                     q_temp=dict(coef=0.1, every=2048))
        if i == 2:
            mixer["kv_from"] = 0
        layers.append(dict(type="attention", mixer=mixer, mlp=mlp))
    return dict(architecture="Bamasun", layers=layers, vocab=c["vocab"], width=c["width"], embedding=dict(scale=1.0), logit_softcap=30.0,
                norm=dict(eps=1e-5))


def served_tensors(c, cfg, seed):
    """Checkpoint tensors ([out, in] matrices N(0, 1 / fan_in)); the router's scores are spread as a trained one's."""
    gen, width, t, bf = generator(seed, 4), cfg["width"], {}, torch.bfloat16

    def mat(name, out, inp, bias=False, gain=1.0):
        t[name] = normal(gen, (out, inp), bf, gain * inp ** -0.5)
        if bias:
            t[name + ".b"] = normal(gen, (out,), bf, 0.1)

    def vec(name, n, mean, bias=False):
        t[name] = normal(gen, (n,), bf, 0.1, mean)
        if bias:
            t[name + ".b"] = normal(gen, (n,), bf, 0.1)

    t["embed"] = normal(gen, (cfg["vocab"], width), bf)
    mat("head", cfg["vocab"], width)
    gigezen = c["kind"] == "gigezen"
    vec("final.norm", width, 0.0 if gigezen else 1.0, not gigezen)
    for i, layer in enumerate(cfg["layers"]):
        p, m, mlp = "l%d." % i, layer["mixer"], layer["mlp"]
        vec(p + "norm1", width, 0.0 if gigezen else 1.0, not gigezen)
        if gigezen:
            mat(p + "mix.q", m["heads"] * (m["dim"] + m["rot_dim"]), width)
            if "kv_from" not in m:
                mat(p + "mix.dkv", m["kv_rank"] + m["rot_dim"], width)
                vec(p + "mix.dkv.norm", m["kv_rank"], 1.0)
            mat(p + "mix.uk", m["heads"] * m["dim"], m["kv_rank"])
            mat(p + "mix.uv", m["heads"] * m["vdim"], m["kv_rank"])
            mat(p + "mix.o", width, m["heads"] * m["vdim"])
            moe = mlp["kind"] == "moe"
            for name, ff in [("%smlp.e%d." % (p, e), mlp["expert"]["ff"]) for e in range(mlp["router"]["experts"])] if moe else [(p + "mlp.", mlp["ff"])]:
                mat(name + "gate", ff, width)
                mat(name + "up", ff, width)
                mat(name + "down", width, ff)
            if moe:
                mat(p + "mlp.router", mlp["router"]["experts"], width, gain=3.0)
            continue
        if layer["type"] == "attention":
            mat(p + "mix.q", m["heads"] * m["dim"], width, True)
            vec(p + "mix.q.norm", m["heads"] * m["dim"], 1.0)
            if "kv_from" not in m:
                mat(p + "mix.k", m["kv_heads"] * m["dim"], width, True)
                mat(p + "mix.v", m["kv_heads"] * m["vdim"], width, True)
                vec(p + "mix.k.norm", m["kv_heads"] * m["dim"], 1.0)
        else:
            nk, nv = m["heads"] * m["dim"], m["heads"] * m["vdim"]
            for name, n in (("q", nk), ("k", nk), ("v", nv), ("g", nv), ("a1", 16)):
                mat(p + "mix." + name, n, width)
            mat(p + "mix.a2", nk, 16)
            t[p + "mix.a2.b"] = normal(gen, (nk,), bf, 1.0, 2.0)
            vec(p + "mix.norm", m["vdim"], 1.0)
        mat(p + "mix.o", width, m["heads"] * m["vdim"])
        vec(p + "norm2", width, 1.0, True)
        mat(p + "mlp.up", mlp["ff"], width)
        mat(p + "mlp.down", width, mlp["ff"])
    return t


def served_batch(c, seed):
    """(tokens held by each sequence, new tokens of each sequence)."""
    rng = np.random.default_rng(int(seed) + 17)
    if c["phase"] == "step":
        held, new = lengths(seed, c["B"], c["lo"], c["hi"]), [1] * c["B"]
    else:
        held = [0] * c["P"] + lengths(seed, c["S"], max(1, c["past"] // 4), c["past"])
        new = lengths(seed + 1, c["P"], c["lo"], c["hi"]) + [1] * c["S"]
    return held, [rng.integers(0, c["vocab"], size=n).astype(np.int32) for n in new]


def served_room(c):
    return c["hi"] + GROW + 1 if c["phase"] == "step" else max(c["hi"], c["past"] + 1) + 7


def held_rows(c, seed, i, shape, dtype):
    """What a layer's cache (or its recurrent state) holds at the start."""
    return normal(generator(seed, 1000 + i), shape, dtype)


# ---------------------------------------------------------------------------------------------------------------------
# preparing and running a pass
# ---------------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    c, ctx, gpu = case, context(), package().gpu
    two = lambda t: gpu.GPUBuffer2D(buffer=t, shape=tuple(t.shape), size=t.numel())  # noqa: E731
    one = lambda t: gpu.GPUBuffer1D(buffer=t, shape=tuple(t.shape), size=t.numel())  # noqa: E731
    s = dict(case=c, ctx=ctx, gpu=gpu, grown=0)
    if c["kind"] == "token":
        lens, T, k, v, table, q, nk, nv = token_inputs(c, seed)
        cache = gpu.kv_cache_create(ctx, gpu.KVCacheConfig(batch_size=c["B"], max_seq_len=T, n_layers=1, n_heads=c["H"], head_dim=c["D"],
                                                           dtype=DTYPES[c["dtype"]], layout=c["layout"], block_size=c["block"],
                                                           ragged=c["lo"] != c["hi"]))
        cache.layers[0].k_cache.buffer.copy_(k)
        cache.layers[0].v_cache.buffer.copy_(v)
        if table is not None:
            cache.block_table.copy_(table)
        s.update(cache=cache, lens=lens, q=two(q), nk=two(nk), nv=two(nv), out=two(torch.empty_like(q)))
        reset_token(s)
    elif c["kind"] == "prompt":
        q, k, v = prompt_inputs(c, seed)
        cache, B, N, H, D = None, c["B"], c["N"], c["H"], c["D"]
        if c["cache"] != "none":
            paged = c["cache"] == "paged"
            cache = gpu.kv_cache_create(ctx, gpu.KVCacheConfig(batch_size=B, max_seq_len=N + 16, n_layers=1, n_heads=H, head_dim=D,
                                                               dtype=q.dtype, layout="bhtd" if paged else c["cache"],
                                                               block_size=16 if paged else 0))
            if paged:
                at = torch.randperm(cache.block_table.numel(), generator=generator(seed, 5), device="cuda")
                cache.block_table.copy_(at.to(torch.int32).view_as(cache.block_table))
        stat = lambda: one(torch.empty(B * N * H, device="cuda"))  # noqa: E731
        s.update(q=two(q), k=two(k), v=two(v), o=two(torch.empty_like(q)), l=stat(), m=stat(), cache=cache)
    elif c["kind"] == "gpt":
        from llm_experiments_b200 import model

        cfg = model.DecoderConfig(vocab_size=c["vocab"], context_size=c["hi"] + GROW + 1, embedding_dim=c["E"], n_heads=c["heads"], n_layers=c["layers"])
        t = gpt_tensors(c, seed)
        wrap = lambda x: one(x) if x.dim() == 1 else two(x)  # noqa: E731
        layers = [model.DecoderLayerWeights(**{k: wrap(v) for k, v in layer.items()}) for layer in t.pop("layers")]
        state = model.decoder_state_create(ctx, cfg, model.DecoderWeights(layers=layers, **{k: wrap(v) for k, v in t.items()}), c["B"], ragged=True)
        s["lens"] = lengths(seed, c["B"], c["lo"], c["hi"])
        for i, cache in enumerate(state.caches):
            b = cache.layers[0]
            b.k_cache.buffer.copy_(held_rows(c, seed, 2 * i, tuple(b.k_cache.buffer.shape), torch.bfloat16))
            b.v_cache.buffer.copy_(held_rows(c, seed, 2 * i + 1, tuple(b.v_cache.buffer.shape), torch.bfloat16))
            gpu.kv_cache_set_lengths(cache, s["lens"])
        s.update(state=state, step=model.GraphedDecodeStep(ctx, state))
        s["step"].token_ids.buffer.copy_(torch.from_numpy(np.concatenate(served_batch(c, seed)[1])))
        s["step"].capture()
    else:
        from llm_experiments_b200 import bamasun, gigezen, model, serving

        design = gigezen if c["kind"] == "gigezen" else bamasun
        config = gigezen_config(c) if c["kind"] == "gigezen" else bamasun_config(c)
        dt = DTYPES[c["dtype"]]
        cfg = (gigezen.GigezenConfig if c["kind"] == "gigezen" else bamasun.BamasunConfig).from_json(config)
        weights = design.prepare_weights(ctx, cfg, served_tensors(c, config, seed), dt)
        held, tokens = served_batch(c, seed)
        state = design.state_create(ctx, cfg, weights, len(held), served_room(c), dt)
        for i, cache in state.owned.items():
            b = cache.layers[0]
            b.k_cache.buffer.copy_(held_rows(c, seed, 2 * i, tuple(b.k_cache.buffer.shape), dt))
            b.v_cache.buffer.copy_(held_rows(c, seed, 2 * i + 1, tuple(b.v_cache.buffer.shape), dt))
        for i, rec in state.recurrent.items():
            rec.copy_(held_rows(c, seed, 2 * i, tuple(rec.shape), torch.float32))
        serving.state_set_lengths(state, held)
        s.update(serving=serving, state=state, held=held)
        if c["phase"] == "step":
            s["step"] = model.GraphedDecodeStep(ctx, state, step_fn=serving.decode_step)
            s["step"].token_ids.buffer.copy_(torch.from_numpy(np.concatenate(tokens)))
            s["step"].capture()
        else:
            s["entries"] = [(b, t, [len(t) - 1]) for b, t in enumerate(tokens)]
    return s


def reset_token(s):
    if s["case"]["lo"] == s["case"]["hi"]:
        s["cache"].current_len = s["case"]["hi"]
    else:
        s["gpu"].kv_cache_set_lengths(s["cache"], s["lens"])


def run(s):
    c, ctx, gpu = s["case"], s["ctx"], s["gpu"]
    if s["grown"] == GROW:  # the sequences end and others of the first lengths take their places
        s["grown"] = 0
        if c["kind"] == "token":
            reset_token(s)
        elif c["kind"] == "gpt":
            for cache in s["state"].caches:
                gpu.kv_cache_set_lengths(cache, s["lens"])
        else:
            s["serving"].state_set_lengths(s["state"], s["held"])
    if c["kind"] == "token":
        s["grown"] += 1
        gpu.batch_begin(ctx)
        gpu.kv_cache_update(ctx, s["cache"], 0, s["nk"], s["nv"])
        gpu.attention_with_kv_cache(ctx, s["cache"], 0, s["q"], s["out"])
        gpu.batch_commit(ctx)
        return dict(out=s["out"].buffer, **kept(s["cache"]))
    if c["kind"] == "prompt":
        gpu.batch_begin(ctx)
        gpu.flash_attention(ctx, s["q"], s["k"], s["v"], s["o"], s["l"], s["m"], c["B"], c["N"], c["H"], c["D"], cache=s["cache"])
        gpu.batch_commit(ctx)
        return dict(out=s["o"].buffer, l=s["l"].buffer, m=s["m"].buffer, **(kept(s["cache"]) if s["cache"] else {}))
    state = s["state"]
    if c["phase"] == "step":
        s["grown"] += 1
        s["step"].step()
        logits, tokens = state.logits.buffer, {"next": s["step"].next_ids.buffer}
    else:
        s["serving"].state_set_lengths(state, s["held"])
        logits, tokens = s["serving"].forward(ctx, state, s["entries"]), {}
    out = dict(logits=logits, **tokens)
    if c["kind"] == "gpt":
        out["caches"] = [kept(cache) for cache in state.caches]
    else:
        out["caches"] = [kept(state.owned[i]) for i in sorted(state.owned)]
        out["recurrent"] = [state.recurrent[i] for i in sorted(state.recurrent)]
    return out


def kept(cache):
    return dict(k=cache.layers[0].k_cache.buffer, v=cache.layers[0].v_cache.buffer)


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------

def work(case):
    c = case
    es = {"f32": 4, "bf16": 2}[c.get("dtype", "bf16")]
    if c["kind"] == "token":
        seen, row = c["B"] * ((c["lo"] + c["hi"]) / 2 + 1), c["H"] * c["D"]
        return {"bytes": es * row * (2 * seen + 6 * c["B"]), "flops": 4.0 * row * seen}
    if c["kind"] == "prompt":
        rows, row = c["B"] * c["N"], c["H"] * c["D"]
        return {"bytes": es * rows * row * (4 if c["cache"] == "none" else 6) + 8.0 * rows * c["H"], "flops": 2.0 * rows * (c["N"] + 1) * row}
    if c["kind"] == "gpt":
        E, rows = c["E"], c["B"]
        seen = rows * ((c["lo"] + c["hi"]) / 2 + 1)
        params = c["layers"] * 12 * E * E + E * c["vocab"]
        return {"bytes": 2.0 * (params + c["layers"] * 2 * seen * E + rows * c["vocab"]),
                "flops": 2.0 * rows * params + c["layers"] * 4.0 * seen * E}
    held, new = ([(c["lo"] + c["hi"]) / 2] * c["B"], [1] * c["B"]) if c["phase"] == "step" else \
        ([0] * c["P"] + [c["past"] * 0.625] * c["S"], [(c["lo"] + c["hi"]) / 2] * c["P"] + [1] * c["S"])
    rows, width, n_bytes, flops = sum(new), c["width"], 0.0, 0.0
    for i in range(c["layers"]):
        if c["kind"] == "gigezen":
            H, R, win = c["heads"], 512, c["window"]
            params = width * H * 192 + H * 256 * R + width * H * 128 + (0 if i % 2 else width * (R + 64))
            n_bytes += es * sum(min(h + n, win + n) for h, n in zip(held, new)) * (R + 64)
            pairs = sum(n * min(h + n / 2, win) for h, n in zip(held, new))
            flops += 2.0 * pairs * H * (192 + 128)
            if i % 2:
                expert = 3 * width * c["expert_ff"]
                n_bytes += es * expert * c["experts"] * (1 - (1 - c["top"] / c["experts"]) ** rows)
                flops += 2.0 * rows * c["top"] * expert
                params += width * c["experts"]
            else:
                params += 3 * width * c["ff"]
        elif i % 2:
            H, d, v = c["gla_heads"], c["dim"], c["gla_vdim"]
            params = width * (2 * H * d + 2 * H * v + 16) + 16 * H * d + H * v * width + 2 * width * c["ff"]
            n_bytes += 4.0 * H * d * v * (len(new) + sum(h > 0 for h in held))
            flops += 4.0 * rows * H * d * v
        else:
            H, G, d = c["heads"], c["kv_heads"], c["dim"]
            params = width * (H + (2 * G if i == 0 else 0)) * d + H * d * width + 2 * width * c["ff"]
            n_bytes += es * 2 * sum(h + n for h, n in zip(held, new)) * G * d
            flops += 4.0 * sum(n * (h + n / 2) for h, n in zip(held, new)) * H * d
        n_bytes += es * params
        flops += 2.0 * rows * params
    n_bytes += es * (width * c["vocab"] + rows * width) + 4.0 * len(new) * c["vocab"]
    return {"bytes": n_bytes, "flops": flops + 2.0 * len(new) * width * c["vocab"]}


def tolerance(case):
    """About four times what the results are off 64 bits (2-norm, relative)."""
    c = case
    f32 = c.get("dtype", "bf16") == "f32"
    if c["kind"] == "token":  # fp32 sums 2e-7; the rounding of bf16 outputs 1.7e-3
        return {"rel": 1e-6 if f32 else 8e-3}
    if c["kind"] == "prompt":  # fp32 operands as two bf16 halves 5.6e-6; bf16 probabilities and outputs 2.0e-3
        return {"rel": 2.4e-5 if f32 else 8e-3}
    if f32:  # 1.4e-6
        return {"rel": 8e-6}
    # 5e-3; rounding may tip the choice of an expert, or a token between two logits that are nearly the same
    return {"rel": 2e-2, "differ": 0.35}


# ---------------------------------------------------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------------------------------------------------

def exact(case, seed):
    c = case
    with torch.no_grad():
        return {"token": exact_token, "prompt": exact_prompt, "gpt": exact_gpt}.get(c["kind"], exact_served)(c, seed)


def attend(q, k, v, scale, first, bias=None, window=0):
    """Causal attention per head: q [H, n, d] at positions first .., k [H, t, d], v [H, t, e]."""
    s = (q @ k.transpose(1, 2)) * scale
    dist = (torch.arange(q.shape[1], device="cuda") + first)[:, None] - torch.arange(k.shape[1], device="cuda")[None, :]
    if bias is not None:
        s = s - bias[:, None, None] * dist
    seen = dist >= 0
    if window:
        seen &= dist < window
    s = s.masked_fill(~seen, -math.inf)
    m = s.amax(dim=-1, keepdim=True)
    e = (s - m).exp_()
    total = e.sum(dim=-1, keepdim=True)
    return (e / total) @ v, total[..., 0], m[..., 0]


def exact_token(c, seed):
    lens, T, k, v, table, q, nk, nv = token_inputs(c, seed)
    B, H, D, block = c["B"], c["H"], c["D"], c["block"]
    out = torch.empty(B, H * D, dtype=torch.float64, device="cuda")
    for b in range(B):
        n = lens[b]

        def rows(buf, new):  # [n + 1, H, D] of this sequence, the new row written to its place first
            if block:
                pool = buf.view(-1, H, block, D)
                pool[int(table[b, n // block]), :, n % block] = new[b].view(H, D)
                return pool[table[b].long()].permute(0, 2, 1, 3).reshape(-1, H, D)[:n + 1]
            view = buf.view(B, T, H, D)[b] if c["layout"] == "bthd" else buf.view(B, H, T, D)[b].transpose(0, 1)
            view[n] = new[b].view(H, D)
            return view[:n + 1]

        kb, vb = rows(k, nk), rows(v, nv)
        for h in range(0, H, 8):
            o = attend(q[b].view(H, 1, D)[h:h + 8].double(), kb[:, h:h + 8].double().transpose(0, 1), vb[:, h:h + 8].double().transpose(0, 1), D ** -0.5, n)[0]
            out[b, h * D:h * D + o.numel()] = o.flatten()
    return dict(out=out, k=k, v=v)


def exact_prompt(c, seed):
    B, N, H, D = c["B"], c["N"], c["H"], c["D"]
    q, k, v = prompt_inputs(c, seed)
    out = torch.empty(B, N, H, D, dtype=torch.float64, device="cuda")
    lm = torch.empty(2, B, N, H, dtype=torch.float64, device="cuda")
    head = lambda t, b, h: t.view(B, N, H, D)[b, :, h:h + 4].transpose(0, 1).double()  # noqa: E731
    for b in range(B):
        for h in range(0, H, 4):
            o, total, m = attend(head(q, b, h), head(k, b, h), head(v, b, h), D ** -0.5, 0)
            out[b, :, h:h + 4] = o.transpose(0, 1)
            lm[0, b, :, h:h + 4], lm[1, b, :, h:h + 4] = total.t(), m.t()
    r = dict(out=out.view(B * N, H * D), l=lm[0].flatten(), m=lm[1].flatten())
    if c["cache"] == "paged":
        blocks = -(-(N + 16) // 16)
        at = torch.randperm(B * blocks, generator=generator(seed, 5), device="cuda").view(B, blocks)

        def pool(t):
            rows = torch.zeros(B, blocks * 16, H, D, dtype=t.dtype, device="cuda")
            rows[:, :N] = t.view(B, N, H, D)
            p = torch.zeros(B * blocks, H, 16, D, dtype=t.dtype, device="cuda")
            p[at.flatten()] = rows.view(B * blocks, 16, H, D).transpose(1, 2)
            return p.view(-1, D)
    elif c["cache"] != "none":
        def pool(t):
            rows = torch.zeros(B, N + 16, H, D, dtype=t.dtype, device="cuda")
            rows[:, :N] = t.view(B, N, H, D)
            return rows.view(-1, H * D) if c["cache"] == "bthd" else rows.transpose(1, 2).reshape(-1, D)
    else:
        return r
    return dict(r, k=pool(k), v=pool(v))


def layer_norm(x, w, b, eps):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w.double(), b.double(), eps)


def rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps) * w


def times(x, w):
    """x @ w in 64 bits, w a slice at a time."""
    return torch.cat([x @ w[:, i:i + 4096].double() for i in range(0, w.shape[1], 4096)], dim=1)


def exact_gpt(c, seed):
    t, B, H, E, T = gpt_tensors(c, seed), c["B"], c["heads"], c["E"], c["hi"] + GROW + 1
    D, lens = E // H, lengths(seed, B, c["lo"], c["hi"])
    ids = torch.from_numpy(np.concatenate(served_batch(c, seed)[1])).cuda().long()
    x = t["embedding"][ids].double() + t["pos_encoding"][torch.tensor(lens, device="cuda")].double()
    caches = []
    for i, w in enumerate(t["layers"]):
        k, v = (held_rows(c, seed, 2 * i + j, (B * H * T, D), torch.bfloat16) for j in (0, 1))
        h = layer_norm(x, w["ln1_gamma"], w["ln1_beta"], 1e-5)
        q, nk, nv = (times(h, w[n]).view(B, H, D) for n in ("wq", "wk", "wv"))
        a = torch.empty(B, E, dtype=torch.float64, device="cuda")
        for b, n in enumerate(lens):
            kb, vb = k.view(B, H, T, D)[b], v.view(B, H, T, D)[b]
            a[b] = attend(q[b][:, None], torch.cat([kb[:, :n].double(), nk[b][:, None]], 1), torch.cat([vb[:, :n].double(), nv[b][:, None]], 1), D ** -0.5, n)[0].flatten()
            kb[:, n], vb[:, n] = nk[b].to(k.dtype), nv[b].to(v.dtype)
        caches.append(dict(k=k, v=v))
        x = x + times(a, w["wo"])
        z = times(layer_norm(x, w["ln2_gamma"], w["ln2_beta"], 1e-5), w["w1"]) + w["b1"].double()
        x = x + times(z * torch.sigmoid(1.702 * z), w["w2"]) + w["b2"].double()
    return dict(logits=times(layer_norm(x, t["lnf_gamma"], t["lnf_beta"], 1e-5), t["out_proj"]), next=None, caches=caches)


def turn(x, pos, base):
    """Rotary positions on the last axis of x [n, ..., dims]: element i is paired with i + dims / 2."""
    half = x.shape[-1] // 2
    freq = base ** (-torch.arange(half, dtype=torch.float64, device="cuda") / half)
    angle = (pos[:, None].double() * freq).view(len(pos), *([1] * (x.dim() - 2)), half)
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * angle.cos() - v * angle.sin(), v * angle.cos() + u * angle.sin()], dim=-1)


def mixture(h, t, p, mlp):
    r = mlp["router"]
    score = torch.softmax(times(h, t[p + "router"].t()), dim=-1)
    best = score.view(len(h), r["groups"]["count"], -1).amax(dim=-1).topk(r["groups"]["keep"], dim=-1).indices
    allowed = torch.zeros(len(h), r["groups"]["count"], dtype=torch.bool, device="cuda").scatter_(1, best, True)
    allowed = allowed.repeat_interleave(r["experts"] // r["groups"]["count"], dim=1)
    idx = score.masked_fill(~allowed, -1.0).topk(r["top"], dim=-1).indices
    y = torch.zeros_like(h)
    for e in range(r["experts"]):
        rows = (idx == e).any(dim=1).nonzero()[:, 0]
        if len(rows):
            g, u = (times(h[rows], t["%se%d.%s" % (p, e, n)].t()) for n in ("gate", "up"))
            y[rows] += score[rows, e, None] * times(g * torch.sigmoid(g) * u, t["%se%d.down" % (p, e)].t())
    return y


def exact_served(c, seed):
    cfg = gigezen_config(c) if c["kind"] == "gigezen" else bamasun_config(c)
    t, (held, tokens) = served_tensors(c, cfg, seed), served_batch(c, seed)
    gig, eps, T, B, dt = c["kind"] == "gigezen", cfg["norm"]["eps"], served_room(c), len(held), DTYPES[c["dtype"]]
    ids = torch.from_numpy(np.concatenate(tokens)).cuda().long()
    ends = np.cumsum([len(n) for n in tokens])
    runs = [(int(e) - len(n), int(e), h) for e, n, h in zip(ends, tokens, held)]  # first and last row, tokens held before
    pos = torch.cat([torch.arange(b - a, device="cuda") + h for a, b, h in runs])
    x = t["embed"][ids].double()
    k_of, v_of, recurrent = {}, {}, []
    for i, layer in enumerate(cfg["layers"]):
        p, m = "l%d." % i, layer["mixer"]
        get = lambda n: t[p + n].double()  # noqa: E731, B023
        h = rms(x, 1.0 + get("norm1"), eps) if gig else x
        prod = lambda n: times(h, t[p + "mix." + n].t()) + (get("mix." + n + ".b") if p + "mix." + n + ".b" in t else 0.0)  # noqa: E731, B023
        H, src = m["heads"], m.get("kv_from", i)
        n_out = H * m["vdim"]
        a = torch.empty(len(x), n_out, dtype=torch.float64, device="cuda")
        if layer["type"] == "gla":
            d, e = m["dim"], m["vdim"]
            state = held_rows(c, seed, 2 * i, (B, H, d, e), torch.float32).double()
            q, k, v, g = prod("q").view(-1, H, d) * d ** -0.5, prod("k").view(-1, H, d), prod("v").view(-1, H, e), prod("g")
            z = times(times(h, t[p + "mix.a1"].t()), t[p + "mix.a2"].t()) + get("mix.a2.b")
            fade = torch.exp(torch.nn.functional.logsigmoid(z) / m["tau"]).view(-1, H, d)
            o = torch.empty(len(x), H, e, dtype=torch.float64, device="cuda")
            for b, (r0, r1, n) in enumerate(runs):
                s = state[b] if n else torch.zeros_like(state[b])
                for r in range(r0, r1):
                    s = fade[r][:, :, None] * s + k[r][:, :, None] * v[r][:, None, :]
                    o[r] = (q[r][:, :, None] * s).sum(dim=1)
                state[b] = s
            recurrent.append(state)
            a = rms(o, get("mix.norm"), eps).view(-1, n_out) * g * torch.sigmoid(g)
        elif gig:
            d, rot, R, base = m["dim"], m["rot_dim"], m["kv_rank"], m["rot"]["base"]
            if src == i:
                k_of[i], v_of[i] = held_rows(c, seed, 2 * i, (B * T, rot), dt).double(), held_rows(c, seed, 2 * i + 1, (B * T, R), dt).double()
                down = prod("dkv")
                at = torch.cat([torch.arange(r1 - r0, device="cuda") + b * T + n for b, (r0, r1, n) in enumerate(runs)])
                k_of[i][at], v_of[i][at] = turn(down[:, R:], pos, base), rms(down[:, :R], get("mix.dkv.norm"), eps)
            q = prod("q").view(-1, H, d + rot)
            q = torch.cat([q[..., :d], turn(q[..., d:], pos, base)], dim=-1)
            for b, (r0, r1, n) in enumerate(runs):
                end = n + r1 - r0
                first = max(0, n + 1 - m["mask"]["size"])
                lat, kr = v_of[src].view(B, T, R)[b, first:end], k_of[src].view(B, T, rot)[b, first:end]
                kk = torch.cat([times(lat, t[p + "mix.uk"].t()).view(-1, H, d), kr[:, None].expand(-1, H, rot)], dim=-1)
                vv = times(lat, t[p + "mix.uv"].t()).view(-1, H, m["vdim"])
                for j in range(0, H, 4):
                    o = attend(q[r0:r1, j:j + 4].transpose(0, 1), kk[:, j:j + 4].transpose(0, 1), vv[:, j:j + 4].transpose(0, 1), m["scale"], n - first, window=m["mask"]["size"])[0]
                    a.view(-1, H, m["vdim"])[r0:r1, j:j + 4] = o.transpose(0, 1)
        else:
            G, d, e = m["kv_heads"], m["dim"], m["vdim"]
            if src == i:
                k_of[i], v_of[i] = held_rows(c, seed, 2 * i, (B * T, G * d), dt).double(), held_rows(c, seed, 2 * i + 1, (B * T, G * e), dt).double()
                at = torch.cat([torch.arange(r1 - r0, device="cuda") + b * T + n for b, (r0, r1, n) in enumerate(runs)])
                k_of[i][at], v_of[i][at] = rms(prod("k"), get("mix.k.norm"), eps), prod("v")
            warm = 1.0 + m["q_temp"]["coef"] * torch.log((pos + 1) // m["q_temp"]["every"] + 1.0).double()
            q = (rms(prod("q"), get("mix.q.norm"), eps) * warm[:, None]).view(-1, H, d)
            slopes = torch.exp2(-8.0 * torch.arange(1, H + 1, dtype=torch.float64, device="cuda") / H)
            for b, (r0, r1, n) in enumerate(runs):
                kk, vv = k_of[src].view(B, T, G, d)[b, :n + r1 - r0], v_of[src].view(B, T, G, e)[b, :n + r1 - r0]
                for j in range(G):
                    hs = slice(j * (H // G), (j + 1) * (H // G))
                    o = attend(q[r0:r1, hs].transpose(0, 1), kk[None, :, j], vv[None, :, j], m["scale"], n, bias=slopes[hs])[0]
                    a.view(-1, H, e)[r0:r1, hs] = o.transpose(0, 1)
        y = times(a, t[p + "mix.o"].t())
        mlp = layer["mlp"]
        if gig:
            if mlp["kind"] == "moe":
                y = y + mixture(h, t, p + "mlp.", mlp)
            else:
                g, u = times(h, t[p + "mlp.gate"].t()).clamp(max=mlp["limit"]), times(h, t[p + "mlp.up"].t()).clamp(-mlp["limit"], mlp["limit"])
                y = y + times(g * torch.sigmoid(1.702 * g) * (u + 1.0), t[p + "mlp.down"].t())
            x = x + y
        else:
            x = x + layer_norm(y, t[p + "norm1"], t[p + "norm1.b"], eps)
            y = times(times(x, t[p + "mlp.up"].t()).clamp(min=0.0).square(), t[p + "mlp.down"].t())
            x = x + layer_norm(y, t[p + "norm2"], t[p + "norm2.b"], eps)
    last = x[torch.from_numpy(ends - 1).cuda()]
    if gig:
        logits = times(rms(last, 1.0 + t["final.norm"].double(), eps), t["head"].t())
    else:
        logits = times(layer_norm(last, t["final.norm"], t["final.norm.b"], eps), t["head"].t())
        logits = cfg["logit_softcap"] * torch.tanh(logits / cfg["logit_softcap"])
    out = dict(logits=logits, caches=[dict(k=k_of[i], v=v_of[i]) for i in sorted(k_of)], recurrent=recurrent)
    return dict(out, next=None) if c["phase"] == "step" else out
