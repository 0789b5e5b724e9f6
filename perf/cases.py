"""The work this engine is timed on: steps and whole generations through its public entry points.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges.  A case is one of three kinds:

* ``"step"``: one ``ModelRunner.step`` of a Qwen3 model: ``decode`` requests that bring one token each to ``context`` cached keys
  (all of that length, or spread between an eighth of it and all of it when ``ragged``), beside ``prompts`` portions of ``prompt``
  tokens behind ``prefix`` tokens that are cached already;
* ``"tokens"``: one ``LLMEngine.generate`` of several requests, token ids in and token ids out;
* ``"generation"``: prompts of several requests in one step, then ``new`` decode steps with given tokens (as the trace replay runs
  them), of one of the designs with recurrent layers.

The layer sizes are those of the benchmark (``bench.py``); models have seeded random weights, caches random keys and values.
``exact`` restates the models in 64-bit arithmetic with torch alone.
"""
import math
import zlib

import torch

from spyinfer_b200 import LLMEngine, SamplingParams, config_from_json
from spyinfer_b200.config import EngineConfig
from spyinfer_b200.engine.batch import StepEntry
from spyinfer_b200.engine.model import Model
from spyinfer_b200.engine.runner import ModelRunner

PAGE = 16
#: decode steps that a batch goes on for before its requests end and others of the first length take their places
STEPS_A_LIFE = 64

#: layer sizes of the benchmark's Qwen3 shapes; the vocabulary is 151,936 in all of them
SHAPES = {
    "8b": dict(hidden=4096, heads=32, kv_heads=8, head_dim=128, ff=12288, depth=36),
    "14b": dict(hidden=5120, heads=40, kv_heads=8, head_dim=128, ff=17408, depth=40),
    "32b": dict(hidden=5120, heads=64, kv_heads=8, head_dim=128, ff=25600, depth=64),
}
VOCAB = 151936


def _step(name, shape, dtype, layers, decode=0, context=0, ragged=False, prompts=0, prompt=0, prefix=0, window=0, tied=False):
    case = dict(kind="step", shape=shape, dtype=dtype, layers=layers, decode=decode, context=context, ragged=ragged, prompts=prompts, prompt=prompt,
                prefix=prefix, window=window, tied=tied)
    return case if name is None else dict(name=name, **case)


def listed():
    return [
        # the smallest calls: a test-sized model through the whole engine (scheduler, chunked prompts, sampling), bound by launches and the host
        dict(name="tokens_tiny_f32", kind="tokens", dtype="float32", requests=4, longest=31, new=12, chunk=5),
        # one user's reply: every weight is read for one token
        _step("decode_b1_ctx640", "8b", "bfloat16", 36, decode=1, context=640),
        # the benchmark's step: a small batch with long contexts
        _step("decode_b8_ctx8192", "8b", "bfloat16", 36, decode=8, context=8192),
        # a full batch of replies to prompts of 512 tokens, at every stage of theirs
        _step("decode_b64_ragged1216", "8b", "bfloat16", 36, decode=64, context=1216, ragged=True),
        # a question's prompt, of no round length
        _step("prompt_37", "8b", "bfloat16", 36, prompts=1, prompt=37),
        # the benchmark's prompt
        _step("prompt_2048", "8b", "bfloat16", 36, prompts=1, prompt=2048),
        # a step of the mixed continuous batch: replies going on beside the rest of a prompt, odd sizes
        _step("mixed_14b", "14b", "bfloat16", 40, decode=47, context=2176, ragged=True, prompts=1, prompt=1501, prefix=512),
        # a long document on the largest layers: attention weighs as much as anywhere
        _step("prompt_8192_32b", "32b", "bfloat16", 8, prompts=1, prompt=8192),
        # the 32-bit path, replying and reading a prompt
        _step("decode_f32_b4", "8b", "float32", 12, decode=4, context=700, ragged=True),
        _step("prompt_f32_300", "8b", "float32", 12, prompts=1, prompt=300),
        # designs with recurrent layers: a batch of replies, and a long prompt
        dict(name="daronex_replies", kind="generation", design="daronex", dtype="bfloat16", width=4096, layers=6, requests=8, longest=400, new=24),
        dict(name="nezolorn_prompt", kind="generation", design="nezolorn", dtype="bfloat16", width=4096, layers=6, requests=1, longest=2047, new=4),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "prompt", "mixed", "mixed", "decode32", "prompt32", "tokens", "daronex", "nezolorn"])
    shape = rng.choice(["8b", "8b", "14b", "32b"])
    layers = {"8b": 24, "14b": 16, "32b": 12}[shape]
    window = rng.choice([0, 0, 0, 1024])
    tied = rng.random() < 0.2
    if what == "decode":
        batch = log(1, 256)
        return _step(None, shape, "bfloat16", layers, decode=batch, context=log(100, min(8192, 200000 // batch)), ragged=rng.random() < 0.7, window=window, tied=tied)
    if what == "prompt":
        total = log(8, 4096)
        prompts = min(rng.choice([1, 1, 1, 2, 5]), total // 8)
        return _step(None, shape, "bfloat16", layers, prompts=prompts, prompt=total // prompts, prefix=rng.choice([0, 0, 0, log(16, 4096)]), window=window, tied=tied)
    if what == "mixed":
        batch = log(1, 128)
        return _step(None, shape, "bfloat16", layers, decode=batch, context=log(100, min(8192, 200000 // batch)), ragged=True, prompts=1, prompt=log(16, 2000),
                     prefix=rng.choice([0, log(16, 2048)]), window=window, tied=tied)
    if what == "decode32":
        batch = log(1, 32)
        return _step(None, shape, "float32", 6, decode=batch, context=log(64, min(4096, 40000 // batch)), ragged=True, tied=tied)
    if what == "prompt32":
        return _step(None, shape, "float32", 4, prompts=rng.choice([1, 1, 3]), prompt=log(8, 400), tied=tied)
    if what == "tokens":
        return dict(kind="tokens", dtype="float32", requests=rng.randint(1, 8), longest=rng.randint(8, 60), new=rng.randint(4, 16), chunk=rng.choice([0, 5, 16]))
    return dict(kind="generation", design=what, dtype="bfloat16", width=rng.choice([2048, 4096]), layers=6, requests=rng.choice([1, 2, 4, 8, 16]),
                longest=log(16, 1024), new=rng.randint(2, 24))


# ---- models: configurations, tensors, seeded weights ----------------------------------------------------------

def _qwen3(case):
    if case["kind"] == "tokens":
        return {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": 3, "hidden_size": 96, "num_attention_heads": 8, "num_key_value_heads": 2,
                "head_dim": 32, "intermediate_size": 224, "vocab_size": 384, "rope_theta": 1000000.0, "rms_norm_eps": 1e-5, "tie_word_embeddings": False,
                "max_position_embeddings": 4096, "eos_token_id": -1}
    s = SHAPES[case["shape"]]
    cfg = {"architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": case["layers"], "hidden_size": s["hidden"], "num_attention_heads": s["heads"],
           "num_key_value_heads": s["kv_heads"], "head_dim": s["head_dim"], "intermediate_size": s["ff"], "vocab_size": VOCAB, "rope_theta": 1000000.0,
           "rms_norm_eps": 1e-6, "tie_word_embeddings": case["tied"], "max_position_embeddings": 40960, "eos_token_id": -1}
    if case["window"]:                                    # the second half of the layers attends to a window
        cfg.update(use_sliding_window=True, sliding_window=case["window"], max_window_layers=case["layers"] // 2)
    return cfg


def _qwen3_shapes(cfg):
    H, I, V, hd = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["head_dim"]
    nq, nk = cfg["num_attention_heads"] * hd, cfg["num_key_value_heads"] * hd
    out = {"model.embed_tokens.weight": (V, H), "model.norm.weight": (H,)}
    if not cfg["tie_word_embeddings"]:
        out["lm_head.weight"] = (V, H)
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        out.update({p + "input_layernorm.weight": (H,), p + "post_attention_layernorm.weight": (H,), p + "self_attn.q_norm.weight": (hd,),
                    p + "self_attn.k_norm.weight": (hd,), p + "self_attn.q_proj.weight": (nq, H), p + "self_attn.k_proj.weight": (nk, H),
                    p + "self_attn.v_proj.weight": (nk, H), p + "self_attn.o_proj.weight": (H, nq), p + "mlp.gate_proj.weight": (I, H),
                    p + "mlp.up_proj.weight": (I, H), p + "mlp.down_proj.weight": (H, I)})
    return out


def _qwen3_rule(name, shape, cfg):
    """(mean, standard deviation) of a tensor's values: 0.02, and as a model is initialised for training what a sublayer adds to the stream
    is divided by the root of their number."""
    if name == "model.embed_tokens.weight":
        return 0.0, 1.0
    if name.endswith(("o_proj.weight", "down_proj.weight")):
        return 0.0, 0.02 * (2 * cfg["num_hidden_layers"]) ** -0.5
    return (1.0, 0.05) if len(shape) == 1 else (0.0, 0.02)


def _daronex(case):
    z = {2048: dict(ff=8192, dim=64, q_rank=768, gla=8), 4096: dict(ff=12288, dim=128, q_rank=1536, gla=16)}[case["width"]]

    def latent(windowed):
        m = {"heads": 16, "dim": z["dim"], "rot_dim": 32, "vdim": z["dim"], "q_rank": z["q_rank"], "kv_rank": 96, "scale": (z["dim"] + 32) ** -0.5,
             "rot": {"base": 500000.0, "dims": 32}}
        if windowed:
            m["mask"] = {"size": 1024}
        return {"type": "latent_attention_2" if windowed else "latent_attention", "mlp": {"kind": "dense", "ff": z["ff"]}, "mixer": m}

    gla = {"type": "gla", "mlp": {"kind": "dense", "ff": z["ff"]}, "mixer": {"heads": z["gla"], "dim": 128, "vdim": 256, "tau": 16.0, "decay_rank": 64}}
    return {"architecture": "Daronex", "vocab": 32000, "width": case["width"], "norm": {"eps": 1e-6}, "logit_scale": 1.0,
            "layers": [(latent(False), latent(True), gla)[i % 3] for i in range(case["layers"])]}


def _daronex_shapes(cfg):
    W, V = cfg["width"], cfg["vocab"]
    out = {"embed": (V, W), "final.norm": (W,), "head": (V, W)}
    for i, layer in enumerate(cfg["layers"]):
        m, p, ff = layer["mixer"], f"l{i}.mix.", layer["mlp"]["ff"]
        out.update({f"l{i}.norm1": (W,), f"l{i}.norm2": (W,), f"l{i}.mlp.up": (ff, W), f"l{i}.mlp.down": (W, ff)})
        if layer["type"] == "gla":
            H, d, vd, r = m["heads"], m["dim"], m["vdim"], m["decay_rank"]
            out.update({p + "q": (H * d, W), p + "k": (H * d, W), p + "v": (H * vd, W), p + "g": (H * vd, W), p + "o": (W, H * vd), p + "norm": (vd,),
                        p + "a1": (r, W), p + "a2": (H * d, r), p + "a2.b": (H * d,)})
        else:
            H, d, rd, vd, qr, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["q_rank"], m["kv_rank"]
            out.update({p + "dq": (qr, W), p + "dq.norm": (qr,), p + "uq": (H * (d + rd), qr), p + "uk": (H * d, r), p + "uv": (H * vd, r), p + "o": (W, H * vd),
                        p + "dkv": (r + rd, W), p + "dkv.norm": (r,)})
            if layer["type"] == "latent_attention_2":
                out[p + "g"] = (H * vd, W)
    return out


def _daronex_rule(name, shape, cfg):
    if name == "embed":
        return 0.0, 1.0
    if name.endswith(".b"):
        return 1.0, 0.5                                   # decays mostly near one, as a trained model's
    if name.endswith(("dq.norm", "dkv.norm", "mix.norm")):
        return 1.0, 0.1
    return (0.0, 0.1) if len(shape) == 1 else (0.0, shape[1] ** -0.5)


def _nezolorn(case):
    z = {2048: dict(heads=16, kv=4, ff=8192), 4096: dict(heads=32, kv=8, ff=12288)}[case["width"]]
    left = {"heads": z["heads"], "kv_heads": z["kv"], "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": 1024, "pool": 64},
            "rot": {"base": 500000.0, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}}
    right = {"heads": z["kv"], "dim": 128, "vdim": 256, "gate_cap": 15.0}
    par = {"type": "parallel", "mlp": {"kind": "dense", "ff": z["ff"]}, "mixer": {"left": left, "right": right, "left_scale": 1.0, "right_scale": 1.0}}
    delta = {"type": "general_delta", "mlp": {"kind": "dense", "ff": z["ff"]}, "mixer": {"heads": case["width"] // 128, "dim": 64, "decay_rank": 64}}
    return {"architecture": "Nezolorn", "vocab": 32000, "width": case["width"], "residual_mult": 0.5, "norm": {"eps": 1e-6},
            "embedding": {"scale": 1.0, "bigram": {"buckets": 65521, "mul_prev": 31, "mul_cur": 7}},
            "layers": [par if i % 3 != 2 else delta for i in range(case["layers"])]}


def _nezolorn_shapes(cfg):
    W, V = cfg["width"], cfg["vocab"]
    out = {"embed": (V, W), "head": (V, W), "final.norm": (W,), "bigram": (cfg["embedding"]["bigram"]["buckets"] + 1, W)}
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        out.update({p + "norm1": (W,), p + "norm2": (W,), p + "mlp.gate": (ff, W), p + "mlp.up": (ff, W), p + "mlp.down": (W, ff)})
        if layer["type"] == "parallel":
            a, b = m["left"], m["right"]
            n, H, dk, dv = a["heads"] * a["dim"], b["heads"], b["dim"], b["vdim"]
            out.update({p + "mix.left.q": (n, W), p + "mix.left.k": (a["kv_heads"] * a["dim"], W), p + "mix.left.o": (W, n)})
            out.update({p + "mix.right." + k: (rows, W) for k, rows in (("q", H * dk), ("k", H * dk), ("v", H * dv), ("g", H * dv), ("i", H), ("f", H))})
            out.update({p + "mix.right.i.b": (H,), p + "mix.right.f.b": (H,), p + "mix.right.norm": (H * dv,), p + "mix.right.o": (W, H * dv)})
        else:
            n, R = m["heads"] * m["dim"], m["decay_rank"]
            out.update({p + "mix." + k: (n, W) for k in ("r", "k", "v", "g", "a")})
            out.update({p + "mix.a.b": (n,), p + "mix.w0": (n,), p + "mix.w1": (R, W), p + "mix.w2": (n, R), p + "mix.norm": (n,), p + "mix.o": (W, n)})
    return out


def _nezolorn_rule(name, shape, cfg):
    if name in ("embed", "bigram"):
        return 0.0, 1.0 if name == "embed" else 0.5
    if name.endswith("f.b"):
        return 2.0, 0.5
    if name.endswith((".b", "w0")):
        return 0.0, 0.5
    if len(shape) == 1:
        return 1.0, 0.1
    size = 2.0 if name.endswith(("left.q", "left.k")) else 4.0 if name.endswith("w2") else 0.4 if name.endswith((".o", ".down")) else 1.0
    return 0.0, size * shape[1] ** -0.5


DESIGNS = {"qwen3": (_qwen3, _qwen3_shapes, _qwen3_rule), "daronex": (_daronex, _daronex_shapes, _daronex_rule),
           "nezolorn": (_nezolorn, _nezolorn_shapes, _nezolorn_rule)}


def _generator(seed, *what):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(repr((int(seed),) + what).encode()))


class Weights:
    """A model's tensors by name, each made from the seed and its name when it is asked for, in bfloat16."""

    def __init__(self, case, seed):
        cfg, shapes, self.rule = DESIGNS[case.get("design", "qwen3")]
        self.cfg = cfg(case)
        self.shapes, self.seed = shapes(self.cfg), seed

    def __contains__(self, name):
        return name in self.shapes

    def __getitem__(self, name):
        shape = self.shapes[name]
        mean, std = self.rule(name, shape, self.cfg)
        return torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(mean, std, generator=_generator(self.seed, name))

    def wide(self, name):
        return self[name].double()

    def matrices(self):
        """Parameters of the matrices that a step multiplies by (tables that it gathers rows from are left out)."""
        tables = ("embed", "bigram") + (() if self.cfg.get("tie_word_embeddings") else ("model.embed_tokens.weight",))
        return sum(s[0] * s[1] for n, s in self.shapes.items() if len(s) == 2 and n not in tables)


# ---- what a case's requests bring --------------------------------------------------------------------------------

def _tokens(seed, what, count, vocab):
    return torch.randint(0, vocab, (count,), generator=torch.Generator().manual_seed(zlib.crc32(repr((seed, what)).encode()))).tolist()


def _contexts(case):
    """Cached keys of the decoding requests."""
    n, c = case["decode"], case["context"]
    return [c if not case["ragged"] else max(1, c // 8 + (c - c // 8) * ((7 * i + 3) % n) // max(1, n - 1)) for i in range(n)]


def _prompt_lengths(case):
    """Prompts of a generation: the first has the stated length, the others down to a quarter of it."""
    n, c = case["requests"], case["longest"]
    return [max(1, c - (3 * c // 4) * ((5 * i) % n) // n) for i in range(n)]


def _requests(case, seed):
    """[(name, cached tokens, tokens of each of the passes)] of a step."""
    out = [(f"d{i}", c, _tokens(seed, ("d", i), STEPS_A_LIFE, VOCAB)) for i, c in enumerate(_contexts(case))]
    return out + [(f"p{i}", case["prefix"], _tokens(seed, ("p", i), case["prompt"], VOCAB)) for i in range(case["prompts"])]


def _cached(case, cfg, seed, layer, name, length, dtype):
    """Keys and values [2, kv heads, length, head size] that a request has in a layer's cache."""
    shape = (2, cfg["num_key_value_heads"], length, cfg["head_dim"])
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, 1.0, generator=_generator(seed, "cache", layer, name))


def _dtype(case):
    return torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32


# ---- a case's state ------------------------------------------------------------------------------------------------

def _runner(case, W, max_num_seqs, max_model_len, pages, step_tokens):
    config = EngineConfig(dtype=case["dtype"], max_num_seqs=max_num_seqs, max_model_len=max_model_len, kvcache_block_size=PAGE, num_kvcache_blocks=pages,
                          max_num_batched_tokens=step_tokens)
    spec = config_from_json(W.cfg).to_spec()
    config.clamp_to_model(spec.max_position)
    model = Model(spec, _dtype(case), config.device, config.max_model_len)
    model.bind(W)
    return ModelRunner(model, config)


def _pages(tokens):
    return -(-tokens // PAGE) + 1


def prepare(case, seed):
    if case["kind"] == "tokens":
        return _prepare_tokens(case, seed)
    W = Weights(case, seed)
    if case["kind"] == "generation":
        lengths, vocab = _prompt_lengths(case), W.cfg["vocab"]
        prompts = [_tokens(seed, ("prompt", i), n, vocab) for i, n in enumerate(lengths)]
        later = [_tokens(seed, ("later", i), case["new"], vocab) for i in range(len(lengths))]
        most = max(lengths) + case["new"] + 1
        runner = _runner(case, W, max(8, len(lengths)), most + PAGE, len(lengths) * _pages(most) + 1, max(sum(lengths), 512))
        state = dict(case=case, runner=runner, prompts=prompts, later=later)
        for _ in range(2):                                # a program that serves has run such steps before: graphs are captured
            run(state)
        return state
    requests = _requests(case, seed)
    most = [cached + (STEPS_A_LIFE if name[0] == "d" else case["prompt"]) + 1 for name, cached, _ in requests]
    step_tokens = case["decode"] + case["prompts"] * case["prompt"]
    runner = _runner(case, W, max(8, len(requests)), max(most) + PAGE, sum(_pages(m) for m in most) + 1, max(step_tokens, 512))
    state = dict(case=case, runner=runner, requests=requests, at=0)
    for k in range(3):                                    # a program that serves has run such steps before: graphs are captured
        runner.step(_entries(state, k))
        for name, _, _ in requests[0 if k == 2 else case["decode"]:]:
            runner.finish(name)
    _admit(state, requests)
    cache, dtype = runner.cache, _dtype(case)
    for layer in range(case["layers"]):
        view = cache.view(layer)
        for name, cached, _ in requests:
            if cached:
                kv = _cached(case, W.cfg, seed, layer, name, cached, dtype)
                n = -(-cached // PAGE)
                table = torch.from_numpy(cache.block_table(name, view.group)[:n].copy())
                kv = torch.nn.functional.pad(kv, (0, 0, 0, n * PAGE - cached)).unflatten(2, (n, PAGE)).permute(2, 0, 1, 3, 4)
                held = (table >= 0).nonzero()[:, 0]       # a window has given its early pages back
                view.pages[table[held].long().cuda()] = kv[held.cuda()]
    return state


def _admit(state, requests):
    cache = state["runner"].cache
    portion = 512 if state["case"]["window"] else 1 << 30  # a window's pool holds the window and a step
    for name, cached, _ in requests:
        if cached:
            cache.add_request(name)
        for done in [*range(portion, cached, portion), cached] if cached else []:
            cache.reserve(name, done)
            cache.commit(name, done)


def _entries(state, k):
    return [StepEntry(name, [tokens[k]], [0]) if name[0] == "d" else StepEntry(name, tokens, [len(tokens) - 1]) for name, _, tokens in state["requests"]]


def run(state):
    case = state["case"]
    if case["kind"] == "tokens":
        return state["engine"].generate(state["prompts"], state["sampling"])
    runner = state["runner"]
    if case["kind"] == "generation":
        rids = list(range(len(state["prompts"])))
        out = [runner.step([StepEntry(r, p, [len(p) - 1]) for r, p in zip(rids, state["prompts"])]).clone()]
        for k in range(case["new"]):
            out.append(runner.step([StepEntry(r, [t[k]], [0]) for r, t in zip(rids, state["later"])]).clone())
        for r in rids:
            runner.finish(r)
        return out
    logits = runner.step(_entries(state, state["at"]))
    state["at"] = (state["at"] + 1) % STEPS_A_LIFE
    # a prompt's request is over; the decoding ones go on, until all of them end and others take their places
    over = [r for r in state["requests"] if r[0][0] == "p" or state["at"] == 0]
    for name, _, _ in over:
        runner.finish(name)
    _admit(state, over)
    return logits


def _prepare_tokens(case, seed):
    W = Weights(case, seed)
    lengths = [max(1, case["longest"] * (i + 1) ** 2 // case["requests"] ** 2) for i in range(case["requests"])]
    engine = LLMEngine(model_config=config_from_json(W.cfg), seed=0, dtype=case["dtype"], max_num_seqs=8, max_model_len=256, kvcache_block_size=8,
                       num_kvcache_blocks=256, max_num_batched_tokens=128, chunk_size=case["chunk"] or None)
    engine.model.bind(W)
    prompts = [_tokens(seed, ("prompt", i), n, W.cfg["vocab_size"]) for i, n in enumerate(lengths)]
    # half the requests take the likeliest token, a quarter sample from all and a quarter from the 40 likeliest
    sampling = [SamplingParams(max_new_tokens=case["new"], ignore_eos=True, **({}, dict(temperature=0.8, seed=seed + i), {}, dict(temperature=0.7, top_k=40, seed=seed + i))[i % 4])
                for i in range(case["requests"])]
    state = dict(case=case, engine=engine, prompts=prompts, sampling=sampling)
    for _ in range(2):
        run(state)
    return state


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

def work(case):
    W = Weights(case, 0)
    cfg, params = W.cfg, W.matrices()
    if case["kind"] == "tokens":
        lengths = [max(1, case["longest"] * (i + 1) ** 2 // case["requests"] ** 2) for i in range(case["requests"])]
        head = cfg["vocab_size"] * cfg["hidden_size"]
        tokens = sum(lengths) + case["requests"] * (case["new"] - 1)
        return {"bytes": 2.0 * params * case["new"], "flops": 2.0 * (params - head) * tokens + 2.0 * head * case["requests"] * case["new"]}
    if case["kind"] == "generation":
        lengths = _prompt_lengths(case)
        n, steps = len(lengths), case["new"] + 1
        head = cfg["vocab"] * cfg["width"]
        return {"bytes": 2.0 * params * steps + 4.0 * cfg["vocab"] * n * steps,
                "flops": 2.0 * (params - head) * (sum(lengths) + n * case["new"]) + 2.0 * head * n * steps}
    elt = 2 if case["dtype"] == "bfloat16" else 4
    brought = [(c, 1) for c in _contexts(case)] + [(case["prefix"], case["prompt"])] * case["prompts"]
    tokens, rows = sum(n for _, n in brought), len(brought)
    head = VOCAB * cfg["hidden_size"]
    row = 2 * cfg["num_key_value_heads"] * cfg["head_dim"] * elt
    bytes_, flops = 2.0 * params + 4.0 * VOCAB * rows, 2.0 * (params - head) * tokens + 2.0 * head * rows
    for layer in range(case["layers"]):
        window = case["window"] if case["window"] and layer >= case["layers"] // 2 else 1 << 30
        for cached, n in brought:
            bytes_ += row * (min(cached, window) + n)
            seen = sum(min(p + 1, window) for p in range(cached, cached + n))
            flops += 4.0 * seen * cfg["num_attention_heads"] * cfg["head_dim"]
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    if case["kind"] == "tokens":
        return "exact"
    # measured: the logits of the 32-bit path are 4e-6 to 5e-6 from the 64-bit ones, those of the bfloat16 path 5e-3 to 8e-3
    return {"rel": 2.5e-5} if case["dtype"] == "float32" else {"rel": 0.025, "max": 0.25}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------

def exact(case, seed):
    if case["kind"] == "tokens":
        return None                                       # whole numbers
    W = Weights(case, seed)
    if case["kind"] == "generation":
        forward = _exact_daronex if case["design"] == "daronex" else _exact_nezolorn
        per_request = []
        for i, n in enumerate(_prompt_lengths(case)):
            tokens = _tokens(seed, ("prompt", i), n, W.cfg["vocab"]) + _tokens(seed, ("later", i), case["new"], W.cfg["vocab"])
            per_request.append(forward(W, W.cfg, tokens, n - 1))
        return list(torch.stack(per_request, 1))
    return _exact_qwen3(case, W, seed)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _angles(positions, freq):
    a = positions.double()[:, None] * freq[None, :]
    return torch.cos(a)[:, None], torch.sin(a)[:, None]


def _halves(x, c, s):
    r = c.shape[-1]
    u, v = x[..., :r], x[..., r:2 * r]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * r:]], -1)


def _attend(q, k, v, scale, window, first):
    """q [n, H, d] at positions first.. over k, v [keys, G, d]; a few heads at a time."""
    n, H, d = q.shape
    G = k.shape[1]
    i, j = torch.arange(first, first + n, device="cuda")[:, None], torch.arange(k.shape[0], device="cuda")[None]
    hidden = (j > i) | (j <= i - window)
    out = torch.empty(n, H, v.shape[2], dtype=torch.float64, device="cuda")
    for g in range(G):
        for h0 in range(g * H // G, (g + 1) * H // G, 4):
            hs = slice(h0, min(h0 + 4, (g + 1) * H // G))
            s = (torch.einsum("nhd,kd->hnk", q[:, hs], k[:, g]) * scale).masked_fill(hidden, -math.inf)
            out[:, hs] = torch.einsum("hnk,kd->nhd", torch.softmax(s, -1), v[:, g])
    return out


def _exact_qwen3(case, W, seed):
    cfg = W.cfg
    eps, H, G, d = cfg["rms_norm_eps"], cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"]
    requests = [(name, cached, tokens[:1] if name[0] == "d" else tokens) for name, cached, tokens in _requests(case, seed)]
    ids = torch.tensor([t for _, _, tokens in requests for t in tokens], device="cuda")
    spans, at = [], 0
    for name, cached, tokens in requests:
        spans.append((name, cached, at, at + len(tokens)))
        at += len(tokens)
    positions = torch.cat([torch.arange(c, c + b - a, device="cuda") for _, c, a, b in spans])
    freq = cfg["rope_theta"] ** (-torch.arange(d // 2, dtype=torch.float64, device="cuda") / (d // 2))
    cos, sin = _angles(positions, freq)
    x = W["model.embed_tokens.weight"][ids].double()
    for layer in range(case["layers"]):
        p = f"model.layers.{layer}."
        window = case["window"] if case["window"] and layer >= case["layers"] // 2 else 1 << 40
        h = _rms(x, eps) * W.wide(p + "input_layernorm.weight")
        q, k, v = ((h @ W.wide(p + f"self_attn.{n}_proj.weight").T).unflatten(1, (-1, d)) for n in "qkv")
        q = _halves(_rms(q, eps) * W.wide(p + "self_attn.q_norm.weight"), cos, sin)
        k = _halves(_rms(k, eps) * W.wide(p + "self_attn.k_norm.weight"), cos, sin)
        o = torch.empty_like(q)
        for name, cached, a, b in spans:
            ks, vs = k[a:b], v[a:b]
            if cached:
                old = _cached(case, cfg, seed, layer, name, cached, _dtype(case)).double()
                ks, vs = torch.cat([old[0].transpose(0, 1), ks]), torch.cat([old[1].transpose(0, 1), vs])
            o[a:b] = _attend(q[a:b], ks, vs, d ** -0.5, window, cached)
        x = x + o.flatten(1) @ W.wide(p + "self_attn.o_proj.weight").T
        h = _rms(x, eps) * W.wide(p + "post_attention_layernorm.weight")
        g = h @ W.wide(p + "mlp.gate_proj.weight").T
        x = x + (g * torch.sigmoid(g) * (h @ W.wide(p + "mlp.up_proj.weight").T)) @ W.wide(p + "mlp.down_proj.weight").T
    x = _rms(x[[b - 1 for _, _, _, b in spans]], eps) * W.wide("model.norm.weight")
    head = W["model.embed_tokens.weight" if cfg["tie_word_embeddings"] else "lm_head.weight"]
    return torch.cat([x @ part.double().T for part in head.split(16384)], 1)


def _pairs(x, c, s):
    out = x.clone()
    u, v = x[..., 0::2], x[..., 1::2]
    out[..., 0::2], out[..., 1::2] = u * c - v * s, v * c + u * s
    return out


def _exact_daronex(W, cfg, tokens, first):
    """Logits of the tokens from the place `first` on."""
    eps, T = cfg["norm"]["eps"], len(tokens)
    positions = torch.arange(T, device="cuda")
    x = W["embed"][torch.tensor(tokens, device="cuda")].double()

    def lin(h, name):
        return h @ W.wide(name).T

    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix.", layer["mixer"]
        H, d, vd = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "gla":
            q, k, v = (lin(x, p + n).unflatten(1, (H, -1)) for n in "qkv")
            q = q * d ** -0.5
            z = lin(lin(x, p + "a1"), p + "a2") + W.wide(p + "a2.b")
            alpha = torch.sigmoid(z).pow(1.0 / m["tau"]).unflatten(1, (H, d))
            S, o = torch.zeros(H, d, vd, dtype=torch.float64, device="cuda"), torch.empty_like(v)
            for t in range(T):
                S = alpha[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
                o[t] = torch.einsum("hdv,hd->hv", S, q[t])
            g = lin(x, p + "g")
            y = lin((_rms(o, eps) * W.wide(p + "norm")).flatten(1) * g * torch.sigmoid(g), p + "o")
        else:
            windowed = layer["type"] == "latent_attention_2"
            rd, r = m["rot_dim"], m["kv_rank"]
            freq = m["rot"]["base"] ** (-2.0 * torch.arange(rd // 2, dtype=torch.float64, device="cuda") / rd)
            c, s = _angles(positions, freq)
            turn = _halves if windowed else _pairs
            q = lin(_rms(lin(x, p + "dq"), eps) * W.wide(p + "dq.norm"), p + "uq").unflatten(1, (H, d + rd))
            both = lin(x, p + "dkv")
            latent, kr = _rms(both[:, :r], eps) * W.wide(p + "dkv.norm"), turn(both[:, None, r:], c, s)
            q = torch.cat([q[..., :d], turn(q[..., d:], c, s)], -1)
            k = torch.cat([lin(latent, p + "uk").unflatten(1, (H, d)), kr.expand(T, H, rd)], -1)
            v = lin(latent, p + "uv").unflatten(1, (H, vd))
            o = _attend(q, k, v, m["scale"], m["mask"]["size"] if windowed else 1 << 40, 0).flatten(1)
            y = lin(o * torch.sigmoid(lin(x, p + "g")) if windowed else o, p + "o")
        x = x + _rms(y, eps) * (1.0 + W.wide(f"l{i}.norm1"))
        a = torch.relu(lin(x, f"l{i}.mlp.up"))
        x = x + _rms(lin(a * a, f"l{i}.mlp.down"), eps) * (1.0 + W.wide(f"l{i}.norm2"))
    return lin(_rms(x[first:], eps) * (1.0 + W.wide("final.norm")), "head") * cfg["logit_scale"]


def _layer_norm(x, w, eps):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _nezolorn_frequencies(rot):
    out = []
    sc = rot["scaling"]
    for j in range(rot["dims"] // 2):
        f = rot["base"] ** (-2.0 * j / rot["dims"])
        wave = 2.0 * math.pi / f
        s = min(1.0, max(0.0, (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])))
        out.append((1.0 - s) * f / sc["factor"] + s * f)
    return torch.tensor(out, dtype=torch.float64, device="cuda")


def _exact_nezolorn(W, cfg, tokens, first):
    """Logits of the tokens from the place `first` on."""
    eps, T, F = cfg["norm"]["eps"], len(tokens), torch.nn.functional
    positions = torch.arange(T, device="cuda")
    b = cfg["embedding"]["bigram"]
    rows = [b["buckets"]] + [(u * b["mul_prev"] + v * b["mul_cur"]) % b["buckets"] for u, v in zip(tokens, tokens[1:])]
    x = W["embed"][torch.tensor(tokens, device="cuda")].double() * cfg["embedding"]["scale"] + W["bigram"][torch.tensor(rows, device="cuda")].double()

    def lin(h, name):
        return h @ W.wide(name).T

    def pooled_attention(h, p, m):
        H, G, d, window, pool = m["heads"], m["kv_heads"], m["dim"], m["mask"]["size"], m["mask"]["pool"]
        q, v = lin(h, p + "q").unflatten(1, (H, d)), lin(h, p + "k").unflatten(1, (G, d))
        c, s = _angles(positions, _nezolorn_frequencies(m["rot"]))
        q, k = _halves(q, c, s), _halves(v, c, s)
        n = T // pool
        ks = torch.cat([k[:n * pool].unflatten(0, (n, pool)).mean(1), k])
        vs = torch.cat([v[:n * pool].unflatten(0, (n, pool)).mean(1), v])
        i, j, blk = positions[:, None], positions[None], torch.arange(n, device="cuda")[None]
        seen = torch.cat([(blk + 1) * pool - 1 <= i - window, (j <= i) & (i - j < window)], 1)
        o = torch.empty_like(q)
        for hh in range(H):
            s = (q[:, hh] @ ks[:, hh * G // H].T * m["scale"]).masked_fill(~seen, -math.inf)
            o[:, hh] = torch.softmax(s, -1) @ vs[:, hh * G // H]
        return lin(o.flatten(1), p + "o")

    def memory(h, p, m):
        H, d, cap = m["heads"], m["dim"], m["gate_cap"]
        q, k, v = (lin(h, p + n).unflatten(1, (H, -1)) for n in "qkv")
        q = q * d ** -0.5
        ig = cap * torch.tanh((lin(h, p + "i") + W.wide(p + "i.b")) / cap)
        fg = F.logsigmoid(cap * torch.tanh((lin(h, p + "f") + W.wide(p + "f.b")) / cap))
        S, n = torch.zeros(H, d, v.shape[2], dtype=torch.float64, device="cuda"), torch.zeros(H, d, dtype=torch.float64, device="cuda")
        big, o = torch.zeros(H, dtype=torch.float64, device="cuda"), torch.empty_like(v)
        for t in range(T):
            new = torch.maximum(fg[t] + big, ig[t])
            a, c = torch.exp(fg[t] + big - new)[:, None], torch.exp(ig[t] - new)[:, None]
            S = a[:, :, None] * S + (c * k[t])[:, :, None] * v[t][:, None, :]
            n, big = a * n + c * k[t], new
            den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-big)) + 1e-6
            o[t] = torch.einsum("hdv,hd->hv", S, q[t]) / den[:, None]
        return lin(_rms(o, eps).flatten(1) * W.wide(p + "norm") * torch.sigmoid(lin(h, p + "g")), p + "o")

    def delta(h, p, m):
        H, d = m["heads"], m["dim"]
        r, k, v = (lin(h, p + n).unflatten(1, (H, d)) for n in "rkv")
        decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(lin(torch.tanh(lin(h, p + "w1")), p + "w2") + W.wide(p + "w0"))).unflatten(1, (H, d))
        rate = torch.sigmoid(lin(h, p + "a") + W.wide(p + "a.b")).unflatten(1, (H, d))
        u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        S, o = torch.zeros(H, d, d, dtype=torch.float64, device="cuda"), torch.empty_like(v)
        for t in range(T):
            S = decay[t][:, :, None] * S - (rate[t] * u[t])[:, :, None] * torch.einsum("hd,hdv->hv", u[t], S)[:, None, :] + k[t][:, :, None] * v[t][:, None, :]
            o[t] = torch.einsum("hdv,hd->hv", S, r[t])
        return lin(_rms(o, eps).flatten(1) * W.wide(p + "norm") * torch.sigmoid(lin(h, p + "g")), p + "o")

    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        h = _layer_norm(x, W.wide(p + "norm1"), eps)
        if layer["type"] == "parallel":
            y = m["left_scale"] * pooled_attention(h, p + "mix.left.", m["left"]) + m["right_scale"] * memory(h, p + "mix.right.", m["right"])
        else:
            y = delta(h, p + "mix.", m)
        x = x + cfg["residual_mult"] * y
        h = _layer_norm(x, W.wide(p + "norm2"), eps)
        x = x + cfg["residual_mult"] * lin(F.silu(lin(h, p + "mlp.gate")) * lin(h, p + "mlp.up"), p + "mlp.down")
    return lin(_layer_norm(x[first:], W.wide("final.norm"), eps), "head")
