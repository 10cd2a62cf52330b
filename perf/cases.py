"""The work a user of this backend has it do, as cases that can be prepared, run and checked.

Four kinds of calls, all through the package's public entry points:

* ``layer``  one MoE layer (router, experts, ordered combine) on device rows (``MoeLayer.forward_dev``)
             or, blocking, on host rows (``MoeLayer.forward``);
* ``group``  the engine's hot call on host rows, ``expert_group`` (or ``expert_group_reduce`` with the
             combine on the device);
* ``gemm``   one resident int4 matrix on device rows (``coli_cuda_pipe_gemm``: dense FFN, lm_head);
* ``stack``  greedy steps of an attention-free decode stack (``DeviceStack.decode``), logits included.

Weights are int4 in the container format (group scales or one scale per row), activations fp32; the
format's arithmetic quantises activation rows to int8, so ``exact`` does that in fp32 as the format
says and everything that follows in 64 bits.
"""
import ctypes
import math
import random

import numpy as np
import torch

from peregrine_b200 import cuda, stack, synth

DEV = 0
DISTINCT = 3  # different expert matrices of a layer; the other experts are copies with memory of their own

# The layer of the benchmark's decode, small-batch and prefill configurations, and its CPU-sized one.
FULL = dict(D=6144, I=2048, E=256, k=8)
SMALL = dict(D=2048, I=1024, E=64, k=4)


def listed():
    return [
        # one new token of one sequence: the latency of interactive decoding
        dict(name="layer_decode_1", kind="layer", host=False, m=1, gs=32, **FULL),
        # the same through the blocking host call, at the smallest configuration: launches and host work
        dict(name="layer_small_host_1", kind="layer", host=True, m=1, gs=32, **SMALL),
        # verification of an 8-node draft tree
        dict(name="layer_verify_8", kind="layer", host=False, m=8, gs=32, **FULL),
        # per-row scales (the engine's default int4 residency), a small serving batch
        dict(name="layer_rowscale_16", kind="layer", host=False, m=16, gs=0, **FULL),
        # a decode batch of 32 sequences
        dict(name="layer_batch_32", kind="layer", host=False, m=32, gs=32, **FULL),
        # a short prompt of odd length, hidden and inter off every tile size
        dict(name="layer_ragged_301", kind="layer", host=False, m=301, gs=64, D=1416, I=616, E=48, k=6),
        # a prompt chunk, and the longest one
        dict(name="layer_prefill_1000", kind="layer", host=False, m=1000, gs=32, **FULL),
        dict(name="layer_prefill_4096", kind="layer", host=False, m=4096, gs=32, **FULL),
        # the scheduler's GPU lane: the resident experts of one decode batch, host rows in and out
        dict(name="group_decode_24", kind="group", reduce=False, experts=24, rows_max=6, fmt="row", gs=0, D=6144,
             I=2048, tokens=0),
        # the same lane in a prompt, with the combine on the device
        dict(name="group_prompt_16", kind="group", reduce=True, experts=16, rows_max=120, fmt="grouped", gs=32,
             D=2048, I=1024, tokens=256),
        # lm_head of a prompt's scored positions
        dict(name="gemm_lm_head_100", kind="gemm", S=100, K=6144, O=32000, gs=32),
        # greedy decoding of a whole (small) stack
        dict(name="stack_decode_32", kind="stack", batch=32, steps=2, layers=4, dense=1, dense_I=4096, vocab=8192,
             gs=32, **SMALL),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))


def draw(rng: random.Random):
    kind = rng.choice(["layer"] * 5 + ["group", "group", "gemm", "gemm", "stack"])
    gs = rng.choice([32, 32, 32, 64, 128, 256, 0])
    if kind == "layer":
        shape = rng.choice([FULL, FULL, SMALL, None])
        if shape is None:  # any other model: 8-element multiples, not tile multiples
            E = rng.choice([8, 16, 40, 48, 64, 100])
            shape = dict(D=8 * _log_int(rng, 48, 400), I=8 * _log_int(rng, 16, 200), E=E,
                         k=rng.randint(1, min(8, E - 1)))
        m = _log_int(rng, 1, 4000)
        return dict(kind="layer", host=rng.random() < 0.25, m=m, gs=gs, **shape)
    if kind == "group":
        fmt = rng.choice(["row", "row", "grouped", "f32"])
        if fmt == "f32":
            D, I, n, r = 8 * rng.randint(32, 200), 8 * rng.randint(16, 100), rng.randint(1, 16), _log_int(rng, 1, 24)
        else:
            D, I = rng.choice([(6144, 2048), (2048, 1024), (8 * rng.randint(60, 500), 8 * rng.randint(30, 200))])
            n, r = rng.randint(1, 40), _log_int(rng, 1, 150)
        reduce = rng.random() < 0.5
        return dict(kind="group", reduce=reduce, experts=n, rows_max=r, fmt=fmt, gs=(gs or 32) if fmt == "grouped" else 0,
                    D=D, I=I, tokens=rng.randint(r, 2 * r + 8) if reduce else 0)
    if kind == "gemm":
        return dict(kind="gemm", S=_log_int(rng, 1, 1200), K=8 * _log_int(rng, 32, 768), O=_log_int(rng, 200, 33000), gs=gs)
    return dict(kind="stack", batch=_log_int(rng, 1, 40), steps=2, layers=rng.randint(2, 5), dense=1,
                dense_I=256 * rng.randint(4, 16), vocab=8 * rng.randint(100, 1200), gs=gs or 32, **SMALL)


# ------------------------------------------------------------------------------------ inputs
def _matrix(rng, o, i, gs, std=0.02):
    rb = (i + 1) // 2
    q = rng.integers(0, 256, size=o * rb, dtype=np.uint8)
    if i % 2:
        q.reshape(o, rb)[:, -1] &= 0x0F
    ng = -(-i // gs) if gs else 1
    s = np.abs(rng.standard_normal(o * ng, dtype=np.float32)) * np.float32(std)
    return synth.SynthMatrix(q, np.maximum(s, np.float32(std * 5e-5)).astype(np.float32), i, o, gs)


def _expert(rng, D, I, gs, std=0.02):
    return synth.SynthExpert(_matrix(rng, I, D, gs, std), _matrix(rng, I, D, gs, std), _matrix(rng, D, I, gs, std))


def _router(case, rng):
    """Router rows and a selection bias that makes some experts popular: Zipf(1.1) for decode batches,
    Dirichlet(0.5) for prompts (the bias only affects which experts are chosen, not their weights)."""
    E, D = case["E"], case["D"]
    w = rng.standard_normal((E, D), dtype=np.float32) * np.float32(0.02)
    if case.get("m", 1) <= 64:
        p = (rng.permutation(E) + 1.0) ** -1.1
    else:
        p = np.maximum(rng.dirichlet(np.full(E, 0.5)), 1e-30)
    return w, np.maximum(0.35 * (np.log(p) - np.log(p.max())), -4.0).astype(np.float32)


def _layer_host(case, rng, std=0.02):
    w, b = _router(case, rng)
    some = [_expert(rng, case["D"], case["I"], case["gs"], std) for _ in range(min(DISTINCT, case["E"]))]
    layer = synth.SynthLayer(case["D"], case["I"], case["E"], case["k"], case["gs"], True, 2.5, w, b)
    layer.experts = [some[e % len(some)] for e in range(case["E"])]
    layer.shared = _expert(rng, case["D"], case["I"], case["gs"], std)
    return layer


def _layer_inputs(case, seed):
    rng = np.random.default_rng(seed)
    layer = _layer_host(case, rng)
    return layer, rng.standard_normal((case["m"], case["D"]), dtype=np.float32)


def _group_inputs(case, seed):
    # the row counts belong to the case, the values to the seed
    rows = np.random.default_rng(case["experts"]).integers(1, case["rows_max"] + 1, case["experts"]).astype(np.int32)
    rows[0] = case["rows_max"]
    rng = np.random.default_rng(seed)
    D, I = case["D"], case["I"]
    if case["fmt"] == "f32":
        experts = [tuple(rng.standard_normal((o, i), dtype=np.float32) * np.float32(0.05)
                         for o, i in ((I, D), (I, D), (D, I))) for _ in range(case["experts"])]
    else:
        some = [_expert(rng, D, I, case["gs"]) for _ in range(min(DISTINCT, case["experts"]))]
        experts = [some[e % len(some)] for e in range(case["experts"])]
    total = int(rows.sum())
    x = rng.standard_normal((total, D), dtype=np.float32)
    dst = rw = None
    if case["reduce"]:
        dst = np.concatenate([np.sort(rng.permutation(case["tokens"])[:r]) for r in rows])
        rw = rng.uniform(0.05, 1.0, total).astype(np.float32)
    return experts, rows, x, dst, rw


def _gemm_inputs(case, seed):
    rng = np.random.default_rng(seed)
    return _matrix(rng, case["O"], case["K"], case["gs"]), rng.standard_normal((case["S"], case["K"]), dtype=np.float32)


def _stack_inputs(case, seed):
    rng = np.random.default_rng(seed)
    D, std = case["D"], 0.002  # scales small enough for the ids to keep depending on the tokens
    st = stack.SynthStack(D, case["vocab"], 1e-5, rng.standard_normal((case["vocab"], D), dtype=np.float32),
                          [(1.0 + 0.1 * rng.standard_normal(D)).astype(np.float32) for _ in range(case["layers"])],
                          (1.0 + 0.1 * rng.standard_normal(D)).astype(np.float32),
                          _matrix(rng, case["vocab"], D, case["gs"]))
    for li in range(case["layers"]):
        st.layers.append(_expert(rng, D, case["dense_I"], case["gs"], std) if li < case["dense"]
                         else _layer_host(case, rng, std))
    return st, rng.integers(0, case["vocab"], case["batch"]).astype(np.int32)


# ----------------------------------------------------------------------------------- prepare, run
def _init():
    if cuda.device_count() == 0 and cuda.init([DEV]) < 1:
        raise RuntimeError("the backend could not initialise its device")


def _upload(ex, D, I):
    g, u, d = ((m.q, m.scale) for m in (ex.gate, ex.up, ex.down))
    if ex.gate.gs:
        return cuda.GpuExpert.upload_int4_grouped(DEV, g, u, d, D, I, ex.gate.gs)
    return cuda.GpuExpert.upload_int4(DEV, g, u, d, D, I)


def _upload_all(experts, D, I):
    first, out = {}, []
    for ex in experts:
        known = first.get(id(ex))
        out.append(known.clone() if known else first.setdefault(id(ex), _upload(ex, D, I)))
    return out


class _Stack:
    def __init__(self, case, st):
        self.ds = stack.DeviceStack(DEV, st, case["batch"], case["steps"], repeats="clone")

    def __del__(self):
        self.ds.free()


def prepare(case, seed):
    _init()
    kind = case["kind"]
    if kind == "layer":
        layer, x = _layer_inputs(case, seed)
        ml = cuda.MoeLayer(DEV, case["D"], case["I"], case["E"], case["k"], True, 2.5, layer.router_w, layer.router_bias)
        for e, ge in enumerate(_upload_all(layer.experts, case["D"], case["I"])):
            ml.set_expert(e, ge)
        ml.set_shared(_upload(layer.shared, case["D"], case["I"]))
        if case["host"]:
            return dict(kind=kind, layer=ml, x=x, out=np.empty_like(x), host=True)
        s = dict(kind=kind, layer=ml, x=torch.from_numpy(x).to("cuda:%d" % DEV), host=False, m=case["m"])
        s["out"] = torch.empty_like(s["x"])
    elif kind == "group":
        experts, rows, x, dst, rw = _group_inputs(case, seed)
        D, I = case["D"], case["I"]
        ge = ([cuda.GpuExpert.upload(DEV, *e, D, I) for e in experts] if case["fmt"] == "f32"
              else _upload_all(experts, D, I))
        s = dict(kind=kind, experts=ge, rows=rows, x=x, D=D, tokens=case["tokens"], reduce=case["reduce"], rw=rw,
                 lay=cuda.ReduceLayout.build(dst, case["tokens"]) if case["reduce"] else None)
    elif kind == "gemm":
        w, x = _gemm_inputs(case, seed)
        t = (cuda.Tensor.upload_grouped(DEV, w.q, w.scale, w.i_n, w.o_n, w.gs) if w.gs
             else cuda.Tensor.upload(DEV, w.q, w.scale, 2, w.i_n, w.o_n))
        s = dict(kind=kind, t=t, x=torch.from_numpy(x).to("cuda:%d" % DEV), S=case["S"])
        s["y"] = torch.empty((case["S"], case["O"]), dtype=torch.float32, device="cuda:%d" % DEV)
    else:
        st, ids = _stack_inputs(case, seed)
        s = dict(kind=kind, stack=_Stack(case, st), ids=ids, steps=case["steps"], shape=(case["batch"], case["vocab"]))
    torch.cuda.synchronize()  # the backend works on a stream of its own
    return s


def run(s):
    kind = s["kind"]
    if kind == "layer":
        if s["host"]:
            return s["layer"].forward(s["x"], s["out"])
        s["layer"].forward_dev(s["out"].data_ptr(), s["x"].data_ptr(), s["m"])
        return s["out"]
    if kind == "group":
        if s["reduce"]:
            return cuda.expert_group_reduce(s["experts"], s["rows"], s["x"], s["D"], s["lay"], s["rw"], s["tokens"])
        return cuda.expert_group(s["experts"], s["rows"], s["x"], s["D"])
    if kind == "gemm":
        if cuda.lib().coli_cuda_pipe_gemm(s["t"].handle, ctypes.c_void_p(s["y"].data_ptr()),
                                          ctypes.c_void_p(s["x"].data_ptr()), s["S"]) != 1:
            raise RuntimeError("pipe_gemm failed")
        return s["y"]
    ds = s["stack"].ds
    ids = ds.decode(s["ids"], s["steps"])
    return {"logits": ds.logits.download(s["shape"], np.float32), "ids": ids}


# ------------------------------------------------------------------------------- work, tolerance
def _wbytes(o, i, gs, f32=False):
    return o * i * 4 if f32 else o * ((i + 1) // 2) + o * (-(-i // gs) if gs else 1) * 4


def _pick(x, w, b, k):
    """ids [m, k] and normalised gate weights of the router (dtype of x)."""
    s = torch.sigmoid(x @ w.T)
    ids = torch.topk(s + b, k, dim=1).indices
    g = torch.gather(s, 1, ids)
    return ids, g / (g.sum(1, keepdim=True) + 1e-20) * 2.5


def _layer_work(case, m, touched):
    D, I, gs = case["D"], case["I"], case["gs"]
    we = 2 * _wbytes(I, D, gs) + _wbytes(D, I, gs)
    return ((touched + 1) * we + case["E"] * D * 4 + 2 * m * D * 4,
            2 * 3 * D * I * m * (case["k"] + 1) + 2 * m * case["E"] * D)


def work(case):
    kind = case["kind"]
    if kind == "layer":  # the experts that a batch like this one touches
        rng = np.random.default_rng(0)
        w, b = (torch.from_numpy(a) for a in _router(case, rng))
        m = min(case["m"], 512)
        ids, _ = _pick(torch.from_numpy(rng.standard_normal((m, case["D"]), dtype=np.float32)), w, b, case["k"])
        n, f = _layer_work(case, case["m"], int(ids.unique().numel()))
    elif kind == "group":
        D, I, gs, f32 = case["D"], case["I"], case["gs"], case["fmt"] == "f32"
        total = case["experts"] * (case["rows_max"] + 1) // 2
        n = case["experts"] * (2 * _wbytes(I, D, gs, f32) + _wbytes(D, I, gs, f32))
        n += total * D * 4 + (case["tokens"] if case["reduce"] else total) * D * 4
        f = 2 * 3 * D * I * total
    elif kind == "gemm":
        n = _wbytes(case["O"], case["K"], case["gs"]) + case["S"] * (case["K"] + case["O"]) * 4
        f = 2 * case["S"] * case["K"] * case["O"]
    else:
        D, b = case["D"], case["batch"]
        touched = case["E"] * (1 - (1 - case["k"] / case["E"]) ** b)
        n, f = _layer_work(case, b, touched)
        n, f = n * (case["layers"] - case["dense"]), f * (case["layers"] - case["dense"])
        n += case["dense"] * (2 * _wbytes(case["dense_I"], D, case["gs"]) + _wbytes(D, case["dense_I"], case["gs"]))
        n += _wbytes(case["vocab"], D, case["gs"]) + b * (D + case["vocab"]) * 4
        f += 2 * 3 * D * case["dense_I"] * b * case["dense"] + 2 * D * case["vocab"] * b
        n, f = n * case["steps"], f * case["steps"]
    return {"bytes": float(n), "flops": float(f)}


def tolerance(case):
    """One matrix is an fp32 sum.  A layer quantises the hidden row to int8 between its matrices: a last-bit
    difference there moves a few of its elements by a whole step, now and then."""
    if case["kind"] == "gemm" or case.get("fmt") == "f32":
        return {"rel": 2e-6, "max": 2e-5}
    if case["kind"] == "stack":
        return {"rel": 6e-3, "max": 0.2, "differ": 0.01}
    return {"rel": 6e-4, "max": 0.03}


# --------------------------------------------------------------------------------------- exact
def _dense(m):
    """The matrix in 64 bits, [o, i]."""
    q = torch.from_numpy(m.q).cuda().reshape(m.o_n, -1)
    w = torch.stack([q & 15, q >> 4], dim=2).reshape(m.o_n, -1)[:, :m.i_n].double() - 8.0
    s = torch.from_numpy(m.scale).cuda().double().reshape(m.o_n, -1)
    return w * (torch.repeat_interleave(s, m.gs, dim=1)[:, :m.i_n] if m.gs else s)


def _quantised(x):
    """Rows as the format's int8 rows stand for them: fp32 scale max / 127, rounded to nearest."""
    x = x.float()
    s = torch.clamp(x.abs().amax(1, keepdim=True) / np.float32(127.0), min=1e-12)
    return torch.round(x * (1.0 / s)).double() * s.double()


def _ffn(x, ex, dense=None):
    g, u, d = dense or tuple(_dense(m) for m in (ex.gate, ex.up, ex.down))
    xq = _quantised(x)
    return _quantised(torch.nn.functional.silu(xq @ g.T) * (xq @ u.T)) @ d.T


def _exact_layer(layer, x):
    ids, g = _pick(x, torch.from_numpy(layer.router_w).cuda().double(), torch.from_numpy(layer.router_bias).cuda().double(),
                   layer.k)
    out = _ffn(x, layer.shared)
    some = list({id(e): e for e in layer.experts}.values())
    for j, ex in enumerate(some):
        tok, pick = torch.nonzero(ids % len(some) == j, as_tuple=True)
        if tok.numel():
            out.index_add_(0, tok, _ffn(x[tok], ex) * g[tok, pick][:, None])
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "layer":
        layer, x = _layer_inputs(case, seed)
        out = _exact_layer(layer, torch.from_numpy(x).cuda().double())
        return out.cpu().numpy() if case["host"] else out
    if kind == "group":
        experts, rows, x, dst, rw = _group_inputs(case, seed)
        x = torch.from_numpy(x).cuda().double()
        y, at = torch.empty_like(x), 0
        for ex, r in zip(experts, rows):
            xs = x[at:at + r]
            if case["fmt"] == "f32":
                g, u, d = (torch.from_numpy(a).cuda().double() for a in ex)
                y[at:at + r] = (torch.nn.functional.silu(xs @ g.T) * (xs @ u.T)) @ d.T
            else:
                y[at:at + r] = _ffn(xs, ex)
            at += r
        if case["reduce"]:
            out = torch.zeros((case["tokens"], case["D"]), dtype=torch.float64, device="cuda")
            y = out.index_add_(0, torch.from_numpy(dst).cuda(), y * torch.from_numpy(rw).cuda().double()[:, None])
        return y.cpu().numpy()
    if kind == "gemm":
        w, x = _gemm_inputs(case, seed)
        return _quantised(torch.from_numpy(x).cuda()) @ _dense(w).T
    st, ids = _stack_inputs(case, seed)

    def norm(x, w):
        return x / torch.sqrt((x * x).mean(1, keepdim=True) + st.eps) * torch.from_numpy(w).cuda().double()

    picked = []
    for _ in range(case["steps"]):
        x = torch.from_numpy(st.embed[ids]).cuda().double()
        for layer, w in zip(st.layers, st.norms):
            n = norm(x, w)
            x = x + (_exact_layer(layer, n) if isinstance(layer, synth.SynthLayer) else _ffn(n, layer))
        logits = _quantised(norm(x, st.final_norm)) @ _dense(st.lm_head).T
        ids = logits.argmax(1).cpu().numpy().astype(np.int32)
        picked.append(ids)
    return {"logits": logits.cpu().numpy(), "ids": None}
