"""The attention steps whose speed is tracked, as a serving program runs them through the package's public objects.

A case is one step of a batch through ``layers`` full-attention layers: the step's metadata (``GQA.prepare``, which every
step needs because positions move), then per layer the front stage and the attention.  ``front`` says which entry points
a layer uses:

    append      append_attend: K/V rows into their pages and attention, one call
    norm        norm_rope_append, then attend (q, k, v as three projections)
    gated       projection_norm_rope_append with gates, then attend_gated (one fused projection per layer)
    draft       attend_partial over the history, block_partial over the draft block, combine (DSpark composite)
    host        step_host: the whole step from and to pinned host buffers

Every layer has pages, inputs and outputs of its own, so a pass leaves nothing of an earlier layer or pass in a cache it
would not find there in a real model.  Context lengths are the evenly spaced quantiles of the case's distribution: the
seed orders the requests, places their pages and draws the values (N(0, 1), as the parity tests do).
"""
import math
import sys

import numpy as np
import torch

from __graft_entry__ import load_package

pkg = load_package()

_DTYPES = {"f32": (pkg.F32, torch.float32, 4), "bf16": (pkg.BF16, torch.bfloat16, 2), "f16": (pkg.F16, torch.float16, 2)}


def _case(name, dtype, heads, head_dim, page, requests, ctx, run=(1, 1), spread="even", front="append", layers=1,
          chunk=0, chunk_share=0.0, replay=False, ids_per_block=1):
    case = dict(dtype=dtype, q_heads=heads[0], kv_heads=heads[1], head_dim=head_dim, page=page, requests=requests,
                ctx_lo=ctx[0], ctx_hi=ctx[1], run_lo=run[0], run_hi=run[1], spread=spread, front=front, layers=layers,
                chunk=chunk, chunk_share=chunk_share, replay=replay, ids_per_block=ids_per_block)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # One chat user, the next token: nothing but latency, replayed as a graph (40/8 heads, 8-token pages).
        _case("decode-one", "bf16", (40, 8), 128, 8, 1, (777, 777), front="norm", layers=6, replay=True),
        # The everyday decode batch of the sparse 35B profile: gated attention, contexts of 1k to 8k.
        _case("decode-batch", "bf16", (16, 2), 256, 16, 32, (1024, 8192), front="gated", layers=4),
        # Four very long documents, one token each.
        _case("decode-long", "bf16", (16, 2), 256, 16, 4, (262144, 262144), ids_per_block=128),
        # Speculative decoding with one drafted token per request (dense 27B profile), a full batch.
        _case("verify-pair", "bf16", (24, 4), 256, 16, 64, (4096, 32768), run=(2, 2), spread="log", front="norm"),
        # Verification of a seven-token draft: eight query tokens per request on the 14B profile.
        _case("verify-block", "bf16", (40, 8), 128, 8, 16, (512, 16384), run=(8, 8), spread="log", front="norm", layers=2),
        # The drafter's own step: seven draft tokens per request see the history and, both ways, their block.
        _case("draft-block", "bf16", (40, 8), 128, 8, 12, (512, 12288), run=(7, 7), spread="log", front="draft", layers=2),
        # New prompts, nothing cached: ragged lengths, gated projection (dense 27B profile).
        _case("prompt", "bf16", (24, 4), 256, 16, 3, (0, 0), run=(611, 2500), front="gated", layers=2),
        # Continuous batching: long prompts arrive in 512-token chunks between the decode rows of everybody else.
        _case("mixed", "bf16", (16, 2), 256, 16, 96, (128, 131072), spread="zipf", chunk=512, chunk_share=0.3,
              ids_per_block=128),
        # A float32 model, the reference's other data type: its bench profile with a batch of long contexts.
        _case("decode-f32", "f32", (32, 8), 128, 16, 16, (4096, 12288)),
        # A small float16 model with narrow heads.
        _case("decode-narrow", "f16", (16, 4), 64, 16, 32, (1024, 8192), layers=4),
        # A head size that is no multiple of 64, and pages of twelve tokens.
        _case("decode-odd", "bf16", (24, 8), 96, 12, 24, (300, 6000)),
        # A host program that keeps its tensors in pinned host memory: the decode batch in one blocking call.
        _case("host-step", "bf16", (16, 2), 256, 16, 32, (1024, 8192), front="host"),
    ]


# What draw() varies: profile (dtype, heads, head_dim, page), fronts, and the ranges of requests, contexts and runs.
_PROFILES = [("bf16", (40, 8), 128, 8), ("bf16", (16, 2), 256, 16), ("bf16", (24, 4), 256, 16), ("bf16", (32, 8), 128, 16),
             ("bf16", (16, 2), 256, 8), ("f16", (4, 1), 128, 16), ("f16", (16, 4), 64, 16), ("bf16", (32, 8), 64, 16)]
_MOST_BYTES, _MOST_FLOPS = 2.2e9, 2.5e12


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        kind = rng.choice(["decode", "decode", "verify", "draft", "prompt", "mixed", "plain", "host"])
        dtype, heads, head_dim, page = rng.choice(_PROFILES)
        hi = log(64, 65536)
        ctx = (max(1, log(max(1, hi // 16), hi)), hi)
        front = rng.choice(["append", "norm", "gated"])
        spread, ids = rng.choice(["even", "log"]), rng.choice([1, 128])
        if kind == "decode":
            case = _case(None, dtype, heads, head_dim, page, log(1, 64), ctx, spread=spread, front=front,
                         layers=rng.randint(1, 6), ids_per_block=ids, replay=rng.random() < 0.3)
        elif kind == "verify":
            run = rng.randint(2, 9)
            case = _case(None, dtype, heads, head_dim, page, log(1, 64), ctx, run=(run, run), spread=spread, front=front,
                         layers=rng.randint(1, 3), ids_per_block=ids)
        elif kind == "draft":
            run = rng.randint(3, 8)
            case = _case(None, dtype, heads, head_dim, page, log(1, 24), ctx, run=(run, run), spread=spread, front="draft",
                         layers=rng.randint(1, 3), ids_per_block=ids)
        elif kind == "prompt":
            longest = log(48, 4096)
            case = _case(None, dtype, heads, head_dim, page, log(1, 6), (0, 0), run=(max(1, longest // 4), longest),
                         front=front, layers=rng.randint(1, 3), ids_per_block=ids)
        elif kind == "mixed":
            case = _case(None, dtype, heads, head_dim, page, log(4, 96), (128, log(4096, 131072)), spread="zipf",
                         front=front, chunk=rng.choice([128, 256, 512]), chunk_share=rng.uniform(0.1, 0.4), ids_per_block=128)
        elif kind == "plain":
            dtype, heads, head_dim, page = rng.choice([("f32", (32, 8), 128, 16), ("f32", (16, 2), 256, 16),
                                                       ("bf16", (24, 8), 96, 12), ("bf16", (32, 8), 80, 16)])
            case = _case(None, dtype, heads, head_dim, page, log(1, 32), (max(1, ctx[0] // 4), max(1, hi // 4)), spread=spread,
                         front="append", layers=rng.randint(1, 2))
        else:
            case = _case(None, dtype, heads, head_dim, page, log(1, 64), ctx, spread=spread, front="host")
        need = work(case)
        if need["bytes"] <= _MOST_BYTES and need["flops"] <= _MOST_FLOPS:
            return case


# ---- sizes -----------------------------------------------------------------------------------------------------------
def _quantiles(lo, hi, n, spread):
    if n == 1 or lo == hi:
        return np.full(n, hi, dtype=np.int64)
    u = (np.arange(n) + 0.5) / n
    if spread == "zipf":  # density x ** -1.1 on [lo, hi]
        a, b = lo ** -0.1, hi ** -0.1
        x = (a + u * (b - a)) ** -10.0
    elif spread == "log":
        x = lo * (hi / lo) ** u
    else:
        x = lo + (hi - lo) * u
    return np.clip(np.rint(x), lo, hi).astype(np.int64)


def _lengths(case):
    """(cached tokens, query tokens) of every request, shortest context first."""
    n = case["requests"]
    ctx = _quantiles(case["ctx_lo"], case["ctx_hi"], n, case["spread"])
    run = _quantiles(case["run_lo"], case["run_hi"], n, "even")
    if case["chunk"]:
        share = case["chunk_share"]
        at = np.arange(n)
        run = np.where(np.floor((at + 1) * share) > np.floor(at * share), case["chunk"], run)
    return ctx, run


def work(case):
    """Bytes: the cached K/V once, every input and output tensor of the step once, a table entry per page."""
    ctx, run = _lengths(case)
    esz = _DTYPES[case["dtype"]][2]
    hq, hkv, d, layers = case["q_heads"], case["kv_heads"], case["head_dim"], case["layers"]
    tokens, front = int(run.sum()), case["front"]
    q_row, kv_row = hq * d * esz, 2 * hkv * d * esz
    per_token = 2 * q_row + kv_row                      # q, k, v in, out
    if front == "draft":
        per_token += 2 * hq * (d + 2) * 4               # the two partials the composite hands out
        keys = int((run * (ctx + run)).sum())
        pages = -(-ctx // case["page"])
    else:
        per_token += kv_row                             # rows into their pages
        per_token += {"norm": q_row, "gated": 3 * q_row}.get(front, 0)  # normalised q (and gates in, gates out)
        keys = int((run * ctx + run * (run + 1) // 2).sum())
        pages = -(-(ctx + run) // case["page"])
    nbytes = int(ctx.sum()) * kv_row + tokens * per_token + int(pages.sum()) * 4
    return {"bytes": nbytes * layers, "flops": 4 * d * hq * keys * layers}


def tolerance(case):
    """Relative error of another summation order and split of the same step: about four times what was measured.

    Tensor-core kernels against the CUDA-core kernel (f32 products and weights throughout), two plans against each other,
    and single requests against a float64 softmax gave 1.4e-6 in f32, 2.9e-4 in f16 and 2.4e-3 in bf16, where P and the
    output are rounded to the data type."""
    return {"rel": {"f32": 6e-6, "f16": 1.2e-3, "bf16": 1e-2}[case["dtype"]]}


# ---- one case on the GPU ---------------------------------------------------------------------------------------------
_context = None


def _shared_context():
    """The one context (device and stream) of this process: a serving program's steps follow one another on it."""
    global _context
    if _context is None:
        _context = pkg.Context(0)
    return _context


class _Inputs:
    """What the seed draws for a case: requests in their order, the arena's values, which pages each row owns, and the
    step's tensors.  Needs no object of the package, so that ``exact`` starts from the same numbers."""

    def __init__(self, case, seed):
        dtype, esz = _DTYPES[case["dtype"]][1:]
        hq, hkv, d, page, layers = (case[k] for k in ("q_heads", "kv_heads", "head_dim", "page", "layers"))
        front = case["front"]
        rng = np.random.default_rng(seed)
        gen = torch.Generator(device="cuda").manual_seed(int(seed))
        order = rng.permutation(case["requests"])
        self.ctx, self.run = ctx, run = [x[order] for x in _lengths(case)]
        n, self.tokens = len(ctx), int(run.sum())

        def normal(*shape):
            return torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=gen)

        held = ctx if front == "draft" else ctx + run
        self.pages_of = -(-held // page)
        total = int(self.pages_of.sum()) * layers
        self.num_pages = total + total // 8 + 1
        self.page_bytes = 2 * hkv * page * d * esz
        self.arena = normal(self.num_pages, self.page_bytes // esz)
        pool, at = rng.permutation(self.num_pages).astype(np.uint32), 0
        self.rows = {}
        for slot in range(n):
            for layer in range(layers):
                self.rows[slot, layer] = pool[at:at + int(self.pages_of[slot])]
                at += int(self.pages_of[slot])
        self.shape_q, self.shape_kv = (layers, self.tokens, hq, d), (layers, self.tokens, hkv, d)
        if front == "gated":
            self.projection = normal(layers, self.tokens, (2 * hq + 2 * hkv) * d)
        else:
            self.q, self.k, self.v = normal(*self.shape_q), normal(*self.shape_kv), normal(*self.shape_kv)
        if front in ("norm", "gated"):
            # the 256-wide profiles rotate a quarter of the head, the others all of it
            self.rope_dim, self.eps, self.theta = 64 if d == 256 else d, 1e-6, 1e6
            self.weights = [(1.0 + 0.1 * torch.from_numpy(rng.standard_normal(d))).to(torch.bfloat16) for _ in range(2)]


class _Step:
    """Arena, page table, component and buffers of one case: what a serving program keeps between steps."""

    def __init__(self, case, seed):
        self.case = case
        code, dtype = _DTYPES[case["dtype"]][:2]
        hq, hkv, d, layers = (case[k] for k in ("q_heads", "kv_heads", "head_dim", "layers"))
        front = self.front = case["front"]
        given = _Inputs(case, seed)
        ctx, run, n, tokens = given.ctx, given.run, len(given.ctx), given.tokens
        self.context = _shared_context()
        self.arena = given.arena
        torch.cuda.synchronize()
        self.pages = pkg.PageArena(self.context, given.num_pages, given.page_bytes, device_ptr=self.arena)
        ids = case["ids_per_block"]
        layout = pkg.GQAPageTableLayout(n, layers, -(-int(given.pages_of.max()) // ids), ids)
        self.table = pkg.GQARequestPageTable(self.context, layout)
        for (slot, layer), row in given.rows.items():
            self.table.write_row(slot, layer, row)
        self.gqa = pkg.GQA(self.context, pkg.GQAConfig(hq, hkv, d, 1.0 / math.sqrt(d), given.page_bytes, code, layout, tokens))

        slots = np.arange(n, dtype=np.uint32)
        if front == "draft":  # every draft token is a row of its own at the last history position
            self.block = int(run[0])
            self.batch = (np.repeat(slots, run), np.repeat(ctx - 1, run).astype(np.uint32),
                          np.arange(tokens + 1, dtype=np.uint32))
        else:
            self.batch = (slots, ctx.astype(np.uint32), np.concatenate([[0], np.cumsum(run)]).astype(np.uint32))
        self.tokens = tokens
        shape_q = given.shape_q
        zeros = lambda shape, kind=dtype: torch.zeros(shape, dtype=kind, device="cuda")  # noqa: E731
        self.out = zeros(shape_q)
        self.answer = {"out": self.out}
        if front == "host":
            self.q, self.k, self.v = (x[0].cpu().pin_memory() for x in (given.q, given.k, given.v))
            self.out = torch.zeros(shape_q[1:], dtype=dtype).pin_memory()
            self.answer = {"out": self.out}
        elif front == "gated":
            self.projection = given.projection
            self.q, self.gates = zeros(shape_q), zeros(shape_q)
            self.answer.update(q=self.q, gates=self.gates)
        else:
            self.q_in, self.k, self.v = given.q, given.k, given.v
            self.q = self.q_in
            if front == "norm":
                self.q = zeros(shape_q)
                self.answer["q"] = self.q
            if front == "draft":
                self.parts = [[zeros(s, torch.float32) for s in (shape_q, shape_q[:3], shape_q[:3])] for _ in range(2)]
                self.answer["history"], self.answer["local"] = self.parts
        if front not in ("draft",):
            self.answer["pages"] = self.arena
        if front in ("norm", "gated"):
            rope = pkg.NormRopeConfig(given.rope_dim, given.eps, given.theta, 0, 1.0, 1.0, 32.0, 1.0, 1, 0)
            self.gqa.set_norm_rope(rope, *(w.view(torch.int16).numpy().view(np.uint16) for w in given.weights))
        self.layers = list(range(layers))
        torch.cuda.synchronize()
        self.graph = None
        if case["replay"]:
            self.gqa.reserve_replay()
            self._plan()
            self._launch()  # once eagerly: kernels configure themselves outside a capture
            self.context.sync()
            self.context.capture_begin()
            self._launch()
            self.graph = self.context.capture_end()
            self.out.zero_()
            torch.cuda.synchronize()

    def _plan(self):
        if self.case["replay"]:
            self.gqa.prepare_bucketed_with_token_capacity(*self.batch, self.tokens)
        else:
            self.gqa.prepare(*self.batch)

    def _launch(self):
        g, pages, table, front = self.gqa, self.pages, self.table, self.front
        for layer in self.layers:
            out, q = self.out[layer], self.q[layer]
            if front == "append":
                g.append_attend(pages, table, layer, self.k[layer], self.v[layer], q, out)
            elif front == "norm":
                g.norm_rope_append(pages, table, layer, self.q_in[layer], self.k[layer], self.v[layer], q)
                g.attend(pages, table, layer, q, out)
            elif front == "gated":
                gates = self.gates[layer]
                g.projection_norm_rope_append(pages, table, layer, self.projection[layer], True, q, gates)
                g.attend_gated(pages, table, layer, q, gates, out)
            else:
                history, local = ([x[layer] for x in part] for part in self.parts)
                g.attend_partial(pages, table, layer, q, *history)
                g.block_partial(q, self.k[layer], self.v[layer], self.tokens, self.block, *local)
                g.combine(*zip(history, local), self.tokens, out)

    def step(self):
        if self.front == "host":
            self.gqa.step_host(self.pages, self.table, 0, *self.batch, self.k, self.v, self.q, self.out)
        else:
            self._plan()
            if self.graph is not None:
                self.graph.launch()
            else:
                self._launch()
        return self.answer

    def __del__(self):
        if sys.is_finalizing():
            return
        torch.cuda.synchronize()
        for name in ("graph", "gqa", "table", "pages"):
            held = getattr(self, name, None)
            if held is not None:
                held.close()


def prepare(case, seed):
    return _Step(case, seed)


def run(state):
    return state.step()


# ---- the same step in 64 bits ----------------------------------------------------------------------------------------
def _norm_rope(x, weight, positions, given):
    """RMSNorm over the head and RoPE of its first ``rope_dim`` dims, x [tokens][heads][D] in float64."""
    x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + given.eps) * weight
    half = given.rope_dim // 2
    inverse = given.theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    angle = (positions[:, None] * inverse)[:, None]
    a, b = x[..., :half], x[..., half:2 * half]
    return torch.cat([a * angle.cos() - b * angle.sin(), a * angle.sin() + b * angle.cos(), x[..., 2 * half:]], -1)


def _softmax_values(q, k, v, group, scale, first=None):
    """(o, m, l) of q [rows][Hq][D] over k, v [keys][Hkv][D]; with `first`, row i sees keys [0, first + i]."""
    parts = []
    for head in range(q.shape[1]):
        s = q[:, head] @ k[:, head // group].T * scale
        if first is not None:
            keys = torch.arange(k.shape[0], device=q.device)
            s.masked_fill_(keys[None] > first + torch.arange(q.shape[0], device=q.device)[:, None], -math.inf)
        m = s.max(-1).values
        w = torch.exp(s - m[:, None])
        parts.append(((w @ v[:, head // group]) / w.sum(-1, keepdim=True), m, w.sum(-1)))
    return [torch.stack(x, 1) for x in zip(*parts)]


def exact(case, seed):
    """What ``run`` returns for these inputs, by plain torch in float64.  The arena comes back where the step computes
    rows of it (norm and RoPE) and it is small; elsewhere its rows are copies."""
    if work(case)["flops"] > 4e11:
        return None
    given = _Inputs(case, seed)
    hq, hkv, d, page, front = (case[k] for k in ("q_heads", "kv_heads", "head_dim", "page", "front"))
    group, scale = hq // hkv, 1.0 / math.sqrt(d)
    tokens, layers = given.tokens, case["layers"]
    starts = np.concatenate([[0], np.cumsum(given.run)])
    positions = torch.from_numpy(np.concatenate([c + np.arange(r) for c, r in zip(given.ctx, given.run)])).to("cuda", torch.float64)
    arena = given.arena.view(-1, 2, hkv, page, d)
    computed = front in ("norm", "gated")
    full = arena.double() if computed and arena.numel() <= 1 << 27 else None
    names = ["out"] + (["q"] if computed else []) + (["gates"] if front == "gated" else [])
    answer = {name: torch.zeros(given.shape_q, dtype=torch.float64, device="cuda") for name in names}
    parts = [[torch.zeros(s, dtype=torch.float64, device="cuda") for s in (given.shape_q, given.shape_q[:3], given.shape_q[:3])]
             for _ in range(2)]
    for layer in range(layers):
        if front == "gated":
            pair, k, v = given.projection[layer].double().split([2 * hq * d, hkv * d, hkv * d], -1)
            q, gates = pair.view(tokens, hq, 2, d).unbind(2)
            k, v = k.view(tokens, hkv, d), v.view(tokens, hkv, d)
            answer["gates"][layer] = gates
        else:
            q, k, v = (x[layer].double() for x in (given.q, given.k, given.v))
        if computed:
            q, k = (_norm_rope(x, w.to("cuda", torch.float64), positions, given) for x, w in zip((q, k), given.weights))
            answer["q"][layer] = q
        for slot in range(len(given.ctx)):
            ctx, run = int(given.ctx[slot]), int(given.run[slot])
            at = slice(int(starts[slot]), int(starts[slot]) + run)
            ids = torch.from_numpy(given.rows[slot, layer].astype(np.int64)).cuda()
            old = arena[ids[:-(-ctx // page)]].permute(1, 0, 3, 2, 4).reshape(2, -1, hkv, d)[:, :ctx].double()
            if front == "draft":
                both = [_softmax_values(q[at], old[0], old[1], group, scale), _softmax_values(q[at], k[at], v[at], group, scale)]
                for part, found in zip(parts, both):
                    for whole, x in zip(part, found):
                        whole[layer, at] = x
                top = torch.maximum(both[0][1], both[1][1])
                mass = [x[2] * torch.exp(x[1] - top) for x in both]
                answer["out"][layer, at] = sum(x[0] * w[..., None] for x, w in zip(both, mass)) / sum(mass)[..., None]
                continue
            out = _softmax_values(q[at], torch.cat([old[0], k[at]]), torch.cat([old[1], v[at]]), group, scale, ctx)[0]
            answer["out"][layer, at] = out * torch.sigmoid(gates[at]) if front == "gated" else out
            if full is not None:
                place = torch.arange(ctx, ctx + run, device="cuda")
                full[ids[place // page], 0, :, place % page] = k[at]
                full[ids[place // page], 1, :, place % page] = v[at]
    if front == "host":
        answer["out"] = answer["out"][0]
    if front == "draft":
        answer["history"], answer["local"] = parts
    else:
        answer["pages"] = None if full is None else full.view(given.arena.shape)
    return answer
