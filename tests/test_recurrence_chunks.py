"""Runs of tokens walked in chunks (csrc/recurrence.cu) against the token-by-token walk and against 64-bit arithmetic."""
import math

import pytest
import torch

gpu = pytest.mark.gpu
HEADS = 2
SHAPES = {"memory": [(64, 32), (128, 48)], "linear": [(64, 16), (128, 48)], "delta": [(64, 64)]}
CASES = [(kind, dk, dv) for kind, sizes in SHAPES.items() for dk, dv in sizes]


def inputs(kind, dk, dv, T, seed, hard=False):
    """Columns [q | k | v | x1 | x2] and the decay's pre-activation; ``hard``: decays near nothing as well as near one."""
    g = torch.Generator().manual_seed(seed)
    n, nv = HEADS * dk, HEADS * dv
    x1 = n if kind == "delta" else 4
    x = torch.randn(T, 2 * n + nv + 2 * x1, generator=g)
    if kind == "memory":
        x[:, -2 * x1:] *= 4.0
    pre = torch.randn(T, n, generator=g) * (20.0 if hard else 2.0)
    return x, pre, torch.randn(n, generator=g) + 1.0, torch.randn(n, generator=g)


def exact(kind, dk, dv, x, pre, b1, b2):
    """Outputs of one request's tokens in 64-bit."""
    H, n, nv = HEADS, HEADS * dk, HEADS * dv
    x = x.double()
    q, k, v = x[:, :n].view(-1, H, dk), x[:, n:2 * n].view(-1, H, dk), x[:, 2 * n:2 * n + nv].view(-1, H, dv)
    S = torch.zeros(H, dk, dv, dtype=torch.float64)
    out = []
    if kind == "memory":
        ig = 6.0 * torch.tanh((x[:, 2 * n + nv:2 * n + nv + H] + b1[:H].double()) / 6.0)
        fg = torch.nn.functional.logsigmoid(6.0 * torch.tanh((x[:, 2 * n + nv + 4:2 * n + nv + 4 + H] + b2[:H].double()) / 6.0))
        N, m = torch.zeros(H, dk, dtype=torch.float64), torch.zeros(H, dtype=torch.float64)
        for t in range(x.shape[0]):
            new = torch.maximum(fg[t] + m, ig[t])
            a, b = torch.exp(fg[t] + m - new), torch.exp(ig[t] - new)
            S = a[:, None, None] * S + b[:, None, None] * k[t][:, :, None] * v[t][:, None, :]
            N = a[:, None] * N + b[:, None] * k[t]
            m = new
            qs = q[t] * dk ** -0.5
            out.append(torch.einsum("hij,hi->hj", S, qs) / (torch.maximum((N * qs).sum(1).abs(), torch.exp(-m)) + 1e-6)[:, None])
    elif kind == "linear":
        a = torch.sigmoid(pre.double() + b2.double()).pow(1 / 16.0).view(-1, H, dk)
        for t in range(x.shape[0]):
            S = a[t][:, :, None] * S + k[t][:, :, None] * v[t][:, None, :]
            out.append(torch.einsum("hij,hi->hj", S, q[t] * dk ** -0.5))
    else:
        rate = torch.sigmoid(x[:, 2 * n + nv:3 * n + nv] + b1.double()).view(-1, H, dk)
        w = torch.exp(-math.exp(-0.5) * torch.sigmoid(pre.double() + b2.double())).view(-1, H, dk)
        for t in range(x.shape[0]):
            u = k[t] / torch.sqrt((k[t] ** 2).sum(1, keepdim=True) + 1e-6)
            S = w[t][:, :, None] * S - (rate[t] * u)[:, :, None] * torch.einsum("hij,hi->hj", S, u)[:, None, :] + k[t][:, :, None] * v[t][:, None, :]
            out.append(torch.einsum("hij,hi->hj", S, q[t]))
    return torch.stack(out).reshape(-1, nv)


def distance(kind, got, want, dv):
    """Relative 2-norm.  The matrix memory's outputs are divided by a sum that nearly cancels at some tokens, whose errors would be all that the norm
    shows: there the median of the tokens' own distances, each head's alone."""
    if kind != "memory":
        return float((got.double() - want).norm() / want.norm())
    d, w = (got.double() - want).view(-1, dv), want.view(-1, dv)
    return float((d.norm(dim=1) / w.norm(dim=1)).median())


def run(kind, dk, dv, xs, pres, b1, b2, state, slots, pad, **kw):
    """One step of several requests; ``pad`` columns ahead of q: with one, no row starts on a 16-byte border and every request is walked
    token by token."""
    from spyinfer_b200 import kernels

    n, nv = HEADS * dk, HEADS * dv
    x = torch.cat(xs)
    x = torch.cat([torch.zeros(len(x), pad), x, torch.zeros(len(x), -(x.shape[1] + pad) % 4)], 1).contiguous().cuda()
    pre = torch.cat(pres).cuda()
    starts = torch.tensor([0] + [len(p) for p in xs]).cumsum(0).to(torch.int32).cuda()
    where = torch.tensor(slots, dtype=torch.int32, device="cuda")
    out = torch.full((len(x), nv), 9.0, device="cuda")
    offs = [pad, pad + n, pad + 2 * n, pad + 2 * n + nv, pad + 2 * n + nv + 4]
    if kind == "memory":
        kernels.mlstm_scan(x, offs, b1[:HEADS].cuda(), b2[:HEADS].cuda(), state, starts, where, len(xs), out, HEADS, dk, dv, dk ** -0.5, 6.0, **kw)
    elif kind == "linear":
        kernels.gla_scan(x, offs[:3], pre, b2.cuda(), 16.0, state, starts, where, len(xs), out, HEADS, dk, dv, dk ** -0.5, **kw)
    else:
        kernels.delta_scan(x, offs[:4], pre, b1.cuda(), b2.cuda(), state, starts, where, len(xs), out, HEADS, dk, **kw)
    return out.cpu()


def new_state(kind, dk, dv, slots):
    from spyinfer_b200 import kernels

    return torch.zeros((slots, HEADS * (kernels.mlstm_record(dk, dv) if kind == "memory" else dk * dv)), device="cuda")


@gpu
@pytest.mark.parametrize("hard", [False, True])
@pytest.mark.parametrize("kind,dk,dv", CASES)
def test_chunks_carry_the_state_through_portions_as_the_walk_by_tokens_does(kind, dk, dv, hard):
    """Portions around the chunks' lengths and the least ones, short ones beside them, slots out of order, and a state that the one
    form leaves and the other goes on from."""
    portions = [[96, 64, 3, 231], [165, 1, 163, 128], [160, 95, 200, 159]]      # [step][request]
    slots = [4, 0, 3, 2]
    total = [sum(step[r] for step in portions) for r in range(4)]
    data = [inputs(kind, dk, dv, total[r], 10 * r + dk, hard) for r in range(4)]
    b1, b2 = data[0][2], data[0][3]
    want = [exact(kind, dk, dv, data[r][0], data[r][1], b1, b2) for r in range(4)]
    errors = {}
    for name, pads in {"chunks": [0, 0, 0], "tokens": [1, 1, 1], "in turns": [0, 1, 0]}.items():
        state, at, got = new_state(kind, dk, dv, 5), [0] * 4, [[] for _ in range(4)]
        state[1] = 7.0
        for step, pad in zip(portions, pads):
            out = run(kind, dk, dv, [data[r][0][at[r]:at[r] + step[r]] for r in range(4)], [data[r][1][at[r]:at[r] + step[r]] for r in range(4)], b1, b2,
                      state, slots, pad)
            for r, part in enumerate(out.split(step)):
                got[r].append(part)
                at[r] += step[r]
        assert bool((state[1] == 7.0).all())
        errors[name] = max(distance(kind, torch.cat(got[r]), want[r], dv) for r in range(4))
    print(f"\n  {kind} {dk} x {dv}{' hard' if hard else ''}: error against 64 bits {errors}")
    # 32-bit sums of up to 128 terms over some hundred tokens: a few roundings of 6e-8 each.  The chunks may not be the less exact form: 1.03 is what
    # the largest of four requests' errors, each over thousands of outputs, may scatter by
    assert errors["tokens"] < 1e-6, errors
    assert max(errors.values()) < 1.03 * errors["tokens"], errors


@gpu
@pytest.mark.parametrize("kind,dk,dv", CASES)
def test_chunks_of_a_long_prompt_are_as_exact_as_the_walk_by_tokens(kind, dk, dv):
    """2,047 tokens, 32 or 64 chunks of them: what one chunk rounds off does not grow through the others."""
    x, pre, b1, b2 = inputs(kind, dk, dv, 2047, 3)
    want = exact(kind, dk, dv, x, pre, b1, b2)
    errors = [distance(kind, run(kind, dk, dv, [x], [pre], b1, b2, new_state(kind, dk, dv, 1), [0], pad), want, dv) for pad in (0, 1)]
    print(f"\n  {kind} {dk} x {dv}, 2,047 tokens: error against 64 bits in chunks {errors[0]:.3g}, by tokens {errors[1]:.3g}")
    assert errors[0] < 1.03 * errors[1], errors


@gpu
@pytest.mark.parametrize("where", ["q", "k", "v", "decay"])
@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3e20])
@pytest.mark.parametrize("kind,dk,dv", [("memory", 64, 32), ("linear", 64, 16), ("delta", 64, 64)])
def test_requests_with_numbers_out_of_range_are_walked_by_tokens(kind, dk, dv, value, where):
    """A number that is none, or a huge one: the head's outputs are those of the walk by tokens bit for bit (nothing of it reaches an
    earlier token), its neighbour's are finite."""
    xs, pres = [], []
    for r in range(2):
        x, pre, b1, b2 = inputs(kind, dk, dv, 200, r)
        xs.append(x)
        pres.append(pre)
    n = HEADS * dk
    if where == "decay":
        if kind == "memory":
            xs[1][170, -8] = value
        else:
            pres[1][170, 5] = value
    else:
        xs[1][170, {"q": 5, "k": n + 5, "v": 2 * n + 5}[where]] = value
    outs = [run(kind, dk, dv, xs, pres, b1, b2, new_state(kind, dk, dv, 2), [1, 0], pad) for pad in (0, 1)]
    assert bool(outs[0][:200].isfinite().all()) and torch.allclose(outs[0][:200], outs[1][:200], rtol=1e-4, atol=1e-4)
    assert bool(outs[0][200:370].isfinite().all())
    h = slice(0, dv)                                                         # the head that holds the number
    if math.isnan(value) or where != "decay":
        assert torch.equal(outs[0][200:, h].nan_to_num(nan=1.25, posinf=2.5, neginf=-2.5), outs[1][200:, h].nan_to_num(nan=1.25, posinf=2.5, neginf=-2.5))
    else:
        assert torch.allclose(outs[0][200:, h], outs[1][200:, h], rtol=1e-4, atol=1e-4)     # a saturated gate is an ordinary one


@gpu
@pytest.mark.parametrize("kind,dk,dv", [("memory", 64, 32), ("linear", 64, 16), ("delta", 64, 64)])
def test_long_requests_anywhere_among_short_ones_take_the_same_chunks(kind, dk, dv):
    """Long requests between requests of one token, of a few and of none: every token once, as the walk by tokens has it; and the same bits whatever
    is said of the batch (the long requests counted, an upper bound as in a replayed step, nothing), and alone without the others."""
    from spyinfer_b200 import kernels

    name = {"memory": "matrix memory", "linear": "linear attention", "delta": "delta rule"}[kind]
    least = kernels.scan_chunk_min(name)
    for order in ([1, 1, least, 2, least + 1, 0, 300, 1], [1] * 70 + [0, 257, 1, least + 64, 0], [257] + [1] * 40 + [5, 200, least], [0, 300, 0, 1]):
        data = [inputs(kind, dk, dv, n, r)[:2] for r, n in enumerate(order)]
        _, _, b1, b2 = inputs(kind, dk, dv, 1, 99)
        xs, pres, slots = [d[0] for d in data], [d[1] for d in data], list(range(len(order)))[::-1]
        runs = (sum(n >= least for n in order), max(order))
        outs, states = [], []
        for pad, kw in ((0, dict(runs=runs)), (0, dict(runs=runs, replayed=True)), (0, {}), (1, {})):
            state = new_state(kind, dk, dv, len(order))
            outs.append(run(kind, dk, dv, xs, pres, b1, b2, state, slots, pad, **kw))
            states.append(state.cpu())
        for k in (1, 2):
            assert torch.equal(outs[0], outs[k]) and torch.equal(states[0], states[k])
        assert torch.allclose(outs[0], outs[3], rtol=2e-3, atol=2e-4) and torch.allclose(states[0], states[3], rtol=2e-4, atol=2e-5)
        assert not torch.equal(outs[0], outs[3])                                # chunks were taken
        at = 0
        for r, n in enumerate(order):
            if n >= 257:                                                        # long enough to take chunks alone
                alone = run(kind, dk, dv, [xs[r]], [pres[r]], b1, b2, new_state(kind, dk, dv, 1), [0], 0, runs=(1, n))
                assert torch.equal(alone, outs[0][at:at + n])
            at += n


@gpu
@pytest.mark.parametrize("kind,dk,dv,heads", [("linear", 128, 256, 16), ("delta", 64, 64, 32)])
def test_chunks_of_many_heads_are_the_walks_by_tokens(kind, dk, dv, heads, monkeypatch):
    """The heads of the large layers: every head and column tile, against the walk by tokens (whose distance from 64 bits is the same)."""
    monkeypatch.setitem(globals(), "HEADS", heads)
    x, pre, b1, b2 = inputs(kind, dk, dv, 300, 7)
    states, outs = [], []
    for pad in (0, 1):
        state = new_state(kind, dk, dv, 1)
        outs.append(run(kind, dk, dv, [x], [pre], b1, b2, state, [0], pad))
        states.append(state.cpu())
    assert not torch.equal(outs[0], outs[1])
    for a, b in (outs, states):
        assert float((a - b).norm() / b.norm()) < 4e-7                        # the two forms' distances from 64 bits, 1.7e-7 each at most


@gpu
@pytest.mark.parametrize("kind", ["memory", "linear", "delta"])
def test_a_step_without_long_requests_asks_for_no_scratch(kind):
    from spyinfer_b200 import kernels

    name = {"memory": "matrix memory", "linear": "linear attention", "delta": "delta rule"}[kind]
    least, sizes = kernels.scan_chunk_min(name), (2, 64, 64)
    proj = torch.empty((8 * (least - 1), 4), device="cuda")

    def asks(tokens, runs, **kw):
        return kernels._scan_chunk_work(name, proj[:tokens], 8, tokens, runs, kw.get("replayed", False), *sizes)

    assert asks(8 * (least - 1), (0, least - 1)) == (None, 0, 0)                 # many tokens, no request long enough
    work, floats, walks = asks(7 + 300, (1, 300))                                # one portion beside seven replies
    assert work.numel() == floats > 0 and walks == 1
    assert asks(7 + 300, (1, 300), replayed=True)[2] == (7 + 300) // least       # a replayed step: as many as there can be


@gpu
@pytest.mark.parametrize("design", ["nezolorn", "daronex"])
def test_models_take_chunks_whole_in_portions_and_replayed_beside_replies(design):
    """A matrix memory, a delta rule and a linear attention of sizes that take chunks, in whole models: prompts of some 200 tokens at once and in portions
    around the least length, then portions beside replies at one padded size, launched, captured and replayed for batches of other shapes
    and for one whose requests are all too short (which has a graph of its own)."""
    import importlib

    import numpy as np
    from spyinfer_b200 import config_from_json
    from spyinfer_b200.config import EngineConfig
    from spyinfer_b200.engine.batch import StepEntry
    from spyinfer_b200.engine.model import Model
    from spyinfer_b200.engine.runner import ModelRunner

    plain = importlib.import_module("plain_" + design)
    if design == "nezolorn":
        cfg = {"architecture": "Nezolorn", "vocab": 211, "width": 128, "residual_mult": 0.5, "norm": {"eps": 1e-6}, "embedding": {"scale": 1.0}, "layers": [
            {"type": "parallel", "mlp": {"kind": "dense", "ff": 96}, "mixer": {"left_scale": 1.0, "right_scale": 1.0,
             "left": {"heads": 2, "kv_heads": 1, "dim": 32, "vdim": 32, "scale": 0.2, "mask": {"size": 40, "pool": 8}, "rot": {"base": 1000.0, "dims": 32}},
             "right": {"heads": 2, "dim": 64, "vdim": 32, "gate_cap": 10.0}}},
            {"type": "general_delta", "mlp": {"kind": "dense", "ff": 80}, "mixer": {"heads": 2, "dim": 64, "decay_rank": 8}}]}
    else:
        cfg = {"architecture": "Daronex", "vocab": 211, "width": 128, "norm": {"eps": 1e-6}, "logit_scale": 1.0, "layers": [
            {"type": "latent_attention", "mlp": {"kind": "dense", "ff": 96}, "mixer": {"heads": 2, "dim": 16, "rot_dim": 8, "vdim": 24, "q_rank": 24, "kv_rank": 24,
                                                                                      "scale": 0.3, "rot": {"base": 500.0, "dims": 8}}},
            {"type": "gla", "mlp": {"kind": "dense", "ff": 80}, "mixer": {"heads": 2, "dim": 64, "vdim": 32, "tau": 16.0, "decay_rank": 8}}]}
    weights = plain.random_weights(cfg, 3)
    config = EngineConfig(dtype="float32", kvcache_block_size=16, num_kvcache_blocks=200, max_num_seqs=8, max_model_len=400, max_num_batched_tokens=512)
    model = Model(config_from_json(cfg).to_spec(), torch.float32, config.device, config.max_model_len)
    model.bind({k: v.cuda() for k, v in weights.items()})
    runner = ModelRunner(model, config)
    rng = np.random.default_rng(5)
    tokens = {r: rng.integers(0, 211, 340 if r in "ij" else 240).tolist() for r in "abcdefghij"}
    want = {r: plain.forward(weights, cfg, t).numpy() for r, t in tokens.items()}

    def close(got, ref):
        return float(np.abs(got - ref).max() / np.abs(ref).max())

    cuts = {}
    for name, sizes in {"whole": [240], "two": [200, 40], "least": [95, 145], "mixed": [1, 163, 5, 71]}.items():
        rows, at = [], 0
        for n in sizes:
            rows.append(runner.step([StepEntry("a", tokens["a"][at:at + n], list(range(n)))]).float().cpu().numpy().copy())
            at += n
        runner.finish("a")
        cuts[name] = np.concatenate(rows)
        assert close(cuts[name], want["a"]) < 2e-4 and close(cuts[name], cuts["whole"]) < 2e-6, name
    done = {r: 0 for r in tokens}

    def step(shares):
        entries = [StepEntry(r, tokens[r][done[r]:done[r] + n], [n - 1]) for r, n in shares]
        got = runner.step(entries).float().cpu().numpy()
        for (r, n), row in zip(shares, got):
            done[r] += n
            assert close(row, want[r][done[r] - 1]) < 2e-4, (shares, r)

    step([("a", 60), ("b", 60)])
    before = len(runner._graphs)
    for shares in ([("c", 200), ("a", 1), ("b", 1)], [("a", 1), ("d", 196), ("b", 1)], [("e", 12), ("f", 222), ("b", 5)], [("g", 195), ("h", 3), ("a", 40)]):
        step(shares)
    assert len(runner._graphs) - before == 1 and runner.graph_steps > 0
    step([("h", 90), ("a", 70), ("b", 50)])                                      # the same padded sizes, no request long enough
    assert len(runner._graphs) - before == 2
    for r in "abcdefgh":
        runner.finish(r)
    # one portion alone, too short to take chunks by itself, the next as long beside another that is: the other form goes on from the state
    n = 100 if design == "nezolorn" else 165
    assert not any(model.choices(runner.build_batch([StepEntry("i", tokens["i"][:n], [])]), 16))
    step([("i", n)])
    assert any(model.choices(runner.build_batch([StepEntry("i", tokens["i"][n:2 * n], []), StepEntry("j", tokens["j"][:n], [])]), 16))
    step([("i", n), ("j", n)])
    step([("i", 10), ("j", 1)])
    runner.check_status()


def test_which_sizes_take_chunks():
    """The rule of the entry point: scratch for the sizes that are served, none for others (the library answers without a device)."""
    import ctypes

    from spyinfer_b200.csrc import build

    f = build.load("recurrence").spy_scan_chunk_floats
    f.restype = ctypes.c_longlong
    # (mode, tokens, long requests, the longest, heads, dk, dv); one long request from 112, 128 and 192 tokens on, two from 96, 128 and 160
    assert f(0, 112, 1, 112, 8, 128, 256) > 0 and f(2, 2000, 8, 400, 16, 128, 256) > 0 and f(1, 2047, 1, 2047, 32, 64, 64) > 0
    assert f(0, 111, 1, 111, 8, 128, 256) == 0 and f(0, 192, 2, 96, 8, 128, 256) > 0 and f(2, 191, 1, 191, 16, 128, 256) == 0 and f(2, 320, 2, 160, 16, 128, 256) > 0
    assert f(0, 112, 1, 112, 8, 96, 256) == 0 and f(0, 112, 1, 112, 8, 128, 250) == 0 and f(1, 128, 1, 128, 8, 128, 128) == 0
    assert f(0, 8000, 0, 95, 8, 128, 256) == 0 and f(0, 8000, 1, 1000, 8, 128, 256) > 0           # short requests, many or beside a long one
    assert f(1, 3000, 2, 1000, 16, 64, 64) > 0 and f(1, 3000, 2, 1000, 32, 64, 64) == 0           # enough pairs for the walk by tokens
    assert f(0, 1 << 19, 1, 1 << 19, 8, 128, 256) == 0                                            # more scratch than the limit
    assert f(0, 4096, 1, 4096, 1, 64, 16 * 65536) == 0                                            # more columns than a grid takes
    # places run with a request's first token: those of long requests never meet, whatever lies ahead of them
    for mode, least, C, place in ((0, 96, 64, lambda t: 3 * t // 128), (1, 128, 32, lambda t: 5 * t // 128), (2, 160, 64, lambda t: 4 * t // 192)):
        assert build.load("recurrence").spy_scan_chunk_min(mode) == least
        for n in range(least, least + 4 * C + 1):
            assert all(place(t + n) - place(t) >= -(-n // C) for t in range(384))
        for T in (256, 1000, 4097):
            per_place = 2 * (f(mode, T, 1, T, 2, 64, 64) // (2 * place(T)))
            assert f(mode, T, 1, T, 2, 64, 64) == per_place * place(T)


def test_the_page_pool_leaves_room_for_the_chunks_scratch(monkeypatch):
    """A pool sized from the free memory (told by a stand-in): with steps of so many tokens that the linear attention's chunks need some hundred MB, the
    pool is smaller by as much."""
    from spyinfer_b200 import config_from_json, kernels
    from spyinfer_b200.config import EngineConfig
    from spyinfer_b200.engine.model import Model
    from spyinfer_b200.engine.runner import ModelRunner

    cfg = {"architecture": "Daronex", "vocab": 211, "width": 128, "norm": {"eps": 1e-6}, "logit_scale": 1.0, "layers": [
        {"type": "latent_attention", "mlp": None, "mixer": {"heads": 2, "dim": 16, "rot_dim": 8, "vdim": 24, "q_rank": 24, "kv_rank": 24, "scale": 0.3,
                                                            "rot": {"base": 500.0, "dims": 8}}},
        {"type": "gla", "mlp": None, "mixer": {"heads": 8, "dim": 128, "vdim": 256, "tau": 16.0, "decay_rank": 8}}]}
    monkeypatch.setattr(torch.cuda, "mem_get_info", lambda device=None: (60 << 30, 180 << 30))
    pages = {}
    for tokens in (100, 16384):
        config = EngineConfig(dtype="float32", kvcache_block_size=16, max_num_seqs=64, max_model_len=1 << 24, max_num_batched_tokens=tokens)
        runner = object.__new__(ModelRunner)
        runner.model, runner.config, runner.device = Model(config_from_json(cfg).to_spec(), torch.float32, None, 1 << 24), config, None
        needs, _ = runner.model.cache_needs()
        pages[tokens] = runner._pages_from_free_memory(needs)
    per_page = 16 * 32 * 4
    scratch = 4 * kernels.scan_chunk_floats("linear attention", 16384, 1, 16384, 8, 128, 256)
    assert scratch > 50 << 20 and pages[100] < 64 * (1 << 20)                    # the free memory, not the requests, sets the pool
    assert pages[100] - pages[16384] in (scratch // per_page, scratch // per_page + 1)
