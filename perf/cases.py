"""The work that programs built on this library have it do, as cases that can be timed and compared.

A case is one of

  prompt   one or several prompts ingested into free slots of a batch, each up to the logits its first token is chosen from
  step     decode steps of a batch of requests that stand in the middle of their contexts, the emitted tokens read after
           every step as a serving loop does
  matmul   the quantised product behind the operator interface, as a host that brings its own executor calls it

over the three model families (the qwen35 hybrid with Q8_0 weights, and the layered Kezilix and Figonex with bfloat16 weights
or in 32 bits).  Sizes are those of the package's configurations: the 27B shape and slices of it, and the 8-layer models at
widths 2048, 4096 and 5120.
"""
import ctypes
import importlib.util
import os
import random
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    name = "kvmem_qw3_b200"
    if name not in sys.modules:
        pkg = os.path.join(_ROOT, "kvmem-qw3_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(pkg, "__init__.py"), submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


FF = {2048: 6144, 4096: 12288, 5120: 17408}
VOCAB = {"qwen27b": 151936, "qwen35": 32768, "kezilix": 32768, "figonex": 32768}


# ---- the cases ---------------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the product's own headline: one request of the 27B model, context 2048, three drafts per step, the tokens of each
        # step read before the next (the accepted counts follow the benchmark's 2.55 tokens per step)
        _step("step_27b", "qwen27b", layers=64, ctx=2048, k=3, steps=4),
        # time to first token of the same model for a prompt of 2048 tokens
        _prompt("prompt_27b", "qwen27b", layers=64, tokens=2048, k=3),
        # a full server: 32 requests of unequal lengths, 128 verify rows per step
        _step("step_batch32", "qwen27b", layers=8, ctx=500, seqs=32, k=3, steps=8),
        # one long document: the K/V cache is as much of the step as the weights
        _step("step_long", "qwen27b", layers=8, ctx=30011, k=3, steps=6),
        # admission of short, ragged requests between the steps of others
        _prompt("prompt_ragged", "qwen27b", layers=8, tokens=331, requests=4, k=3),
        # the smallest call: one plain step of one short request on the smallest model of the range
        _step("step_small", "qwen35", width=2048, ctx=17, steps=1),
        # a whole prompt, and a batch of requests, on the latent-attention family
        _prompt("prompt_kezilix", "kezilix", width=4096, tokens=2048),
        _step("step_kezilix32", "kezilix", width=4096, ctx=1024, seqs=32, steps=8),
        # a prompt that ends off every tile, and a single request, on the shared-key/value family
        _prompt("prompt_figonex", "figonex", width=5120, tokens=1531),
        _step("step_figonex", "figonex", width=2048, ctx=777, steps=8),
        # a short prompt with every product and activation in 32 bits (the traces that a conversion is checked with)
        _prompt("prompt_f32", "kezilix", width=2048, tokens=100, dtype="float32"),
        # the feed-forward input product at the row count of a middling batch, through the operator interface
        _matmul("matmul_q8", 34816, 5120, 100),
    ]


def _step(name, model, layers=8, width=5120, ctx=1, seqs=1, k=0, steps=1, dtype="bfloat16"):
    return dict(name=name, kind="step", model=model, layers=layers, width=width, ctx=ctx, seqs=seqs, k=k, steps=steps, dtype=dtype)


def _prompt(name, model, layers=8, width=5120, tokens=1, requests=1, k=0, dtype="bfloat16"):
    return dict(name=name, kind="prompt", model=model, layers=layers, width=width, tokens=tokens, requests=requests, k=k, dtype=dtype)


def _matmul(name, rows, cols, m):
    return dict(name=name, kind="matmul", rows=rows, cols=cols, m=m)


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["prompt", "prompt", "step", "step", "step", "matmul"])
    if kind == "matmul":
        rows, cols = rng.choice([(34816, 5120), (5120, 17408), (16480, 5120), (14336, 5120), (5120, 6144), (5120, 10240), (24576, 4096), (4096, 12288)])
        case = _matmul("", rows, cols, _log(rng, 1, 600))
    else:
        model = rng.choice(["qwen27b", "qwen35", "kezilix", "figonex"])
        width = 5120 if model == "qwen27b" else rng.choice(sorted(FF))
        if kind == "prompt":
            f32 = model in ("kezilix", "figonex") and rng.random() < 0.15
            requests = rng.choice([1, 1, 1, 2, 3, 5])
            case = _prompt("", model, width=width, tokens=_log(rng, 5, 120 if f32 else 3000 // requests), requests=requests,
                           k=rng.choice([0, 1, 3, 5]) if model == "qwen27b" else 0, dtype="float32" if f32 else "bfloat16")
        else:
            seqs = _log(rng, 1, 32)
            case = _step("", model, width=width, ctx=_log(rng, 9, 12000 // seqs), seqs=seqs,
                         k=rng.choice([0, 1, 2, 3, 4, 5]) if model == "qwen27b" else 0, steps=rng.choice([2, 3, 4, 6]))
    del case["name"]
    return case


def _lengths(longest, n):
    """Unequal lengths of n requests, the longest first: down to a quarter of it, odd ones among them."""
    return [max(1, longest - (longest * 3 * i) // (4 * n) - (i % 2 if longest > 8 else 0)) for i in range(n)]


# ---- models and states ---------------------------------------------------------------------------------------------------------
_held = {}


class _Model:
    """A model of the library, freed with its last user.  The seeded weights stand for the checkpoint that a server loads once."""

    def __init__(self, case):
        qb = _package()
        if "ctx" not in _held:
            _held["ctx"] = qb.Context(0)
        ctx, c = _held["ctx"], qb.configs
        if case["model"] == "qwen27b":
            self.m = qb.Model(ctx, c.qwen27b(case["layers"]), c.MODEL_SEED)
        elif case["model"] == "qwen35":
            self.m = qb.Model(ctx, c.qwen35_bench(case["width"], FF[case["width"]], case["layers"]), c.MODEL_SEED)
        else:
            make = c.kezilix_bench if case["model"] == "kezilix" else c.figonex_bench
            self.m = qb.Model.layered_synth(ctx, make(case["width"], FF[case["width"]], case["layers"]), c.MODEL_SEED, case["dtype"])

    def __del__(self):
        self.m.close()


def _model(case):
    key = (case["model"], case["layers"], case["width"], case["dtype"])
    if _held.get("key") != key:
        _held.pop("model", None)
        _held["model"], _held["key"] = _Model(case), key
    return _held["model"]


class _State:
    """A batch with what its program keeps beside it; the batch's device memory goes back with the object."""

    def __init__(self, case, n_seqs, max_ctx, logit_rows):
        self.case, self.model = case, _model(case)
        self.snap = None
        self.batch = _package().Batch(self.model.m, n_seqs, max_ctx, case["k"])
        self.vocab = VOCAB[case["model"]]
        self.logits = torch.empty((logit_rows, self.vocab), dtype=torch.float32, pin_memory=True)

    def read_logits(self, first, rows):
        """The logits of the last forward's rows, to pinned memory."""
        qb, n = _package(), ctypes.c_uint32()
        qb.binding.check(qb.lib().qb_debug_last_logits(self.batch.ctx.h, self.batch.h, ctypes.c_void_p(self.logits[first:].data_ptr()), rows, ctypes.byref(n)))

    def __del__(self):
        if self.snap is not None:
            self.batch.free_snapshot(self.snap)
        self.batch.close()


# At this temperature the distribution is flat, so the caller's draw alone decides the token: the steps replay a given
# continuation, the same for every implementation of the arithmetic.
FLAT = 1e6


def prepare(case, seed):
    rs = np.random.RandomState(seed % (1 << 32))
    if case["kind"] == "matmul":
        return _prepare_matmul(case, rs)
    V = VOCAB[case["model"]]
    if case["kind"] == "prompt":
        lens = _lengths(case["tokens"], case["requests"])
        s = _State(case, len(lens), max(lens) + 8, len(lens))
        s.prompts = [rs.randint(0, V, n).astype(np.int32) for n in lens]
        return s
    n, k, steps = case["seqs"], case["k"], case["steps"]
    lens = _lengths(case["ctx"], n)
    s = _State(case, n, max(lens) + (k + 1) * (steps + 1), n * (k + 1))
    for i, m in enumerate(lens):
        s.batch.prefill_sampled(i, rs.randint(0, V, m).astype(np.int32), (rs.randint(0, V) + 0.5) / V, FLAT)
    s.snap = s.batch.snapshot()
    # draws of every step: plain steps take one per request; a speculative step accepts `a` drafts (a draw of 0 accepts, one
    # near 1 rejects), then takes its last token by the draw behind
    s.draws = (rs.randint(0, V, (steps, n, k + 1)) + 0.5) / V
    s.drafts = torch.from_numpy(rs.randint(0, V, (steps, n, max(k, 1))).astype(np.int32)).pin_memory().numpy()
    for t in range(steps if k else 0):
        for i in range(n):
            a = min(k, [0, 3, 1, 3, 2, 3, 0, 1][(t + i) % 8])
            s.draws[t, i, :a] = 0.0
            if a < k:
                s.draws[t, i, a] = 0.999
    s.batch.ctx.sync()
    return s


def run(s):
    if isinstance(s, dict):
        return _run_matmul(s)
    b, case = s.batch, s.case
    if case["kind"] == "prompt":
        for i, p in enumerate(s.prompts):
            b.reset(i)
            b.prefill(i, p)
            s.read_logits(i, 1)
        return s.logits
    b.restore(s.snap)
    tokens = []
    for t in range(case["steps"]):
        if case["k"]:
            b.mtp_draft()
            b.mtp_set_drafts(s.drafts[t])
            b.mtp_verify()
            b.mtp_sample_rows(s.draws[t], FLAT)
            b.mtp_accept_commit()
        else:
            b.sampled_step(s.draws[t], FLAT)
        tokens.append(b.read_output())
    s.read_logits(0, case["seqs"] * (case["k"] + 1))
    return {"logits": s.logits, "tokens": np.array([t for step in tokens for seq in step for t in seq], np.int64)}


# ---- the quantised product -----------------------------------------------------------------------------------------------------
def _matmul_inputs(case, rs):
    """Q8_0 blocks [rows][cols / 32] of a weight with values N(0, 0.02^2), and activations N(0, 1) with a few large columns."""
    g = torch.Generator(device="cuda").manual_seed(int(rs.randint(1 << 31)))
    w = torch.randn((case["rows"], case["cols"] // 32, 32), generator=g, device="cuda") * 0.02
    d = (w.abs().amax(2) / 127.0).half()
    q = torch.clamp(torch.round(w / d.float().unsqueeze(2)), -127, 127).to(torch.int8)
    x = torch.randn((case["m"], case["cols"]), generator=g, device="cuda")
    x[:, torch.randint(0, case["cols"], (8,), generator=g, device="cuda")] *= 20.0
    return d, q, x


def _prepare_matmul(case, rs):
    qb = _package()
    if "ctx" not in _held:
        _held["ctx"] = qb.Context(0)
    d, q, x = _matmul_inputs(case, rs)
    blocks = torch.cat([d.unsqueeze(2).view(torch.int8), q], dim=2).cpu().numpy().view(np.uint8)
    y = torch.empty((case["m"], case["rows"]), device="cuda")
    torch.cuda.synchronize()
    return {"case": case, "w": qb.Weight.from_blocks(_held["ctx"], blocks, case["rows"], case["cols"]), "x": x, "y": y}


def _run_matmul(s):
    qb, c = _package(), s["case"]
    qb.binding.check(qb.lib().qb_q8_0_matmul(_held["ctx"].h, s["w"].h, ctypes.c_void_p(s["x"].data_ptr()), c["m"], c["cols"], ctypes.c_void_p(s["y"].data_ptr()),
                                             c["rows"], 0, 0))
    return s["y"]


def exact(case, seed):
    """The product on the quantised operands in 64 bits.  A model's logits have no such value here: its seeded weights exist in
    the library's device layout only."""
    if case["kind"] != "matmul":
        return None
    d, q, x = _matmul_inputs(case, np.random.RandomState(seed % (1 << 32)))
    # activations as the operator defines them: per block of 32, whole numbers of 127ths of the largest magnitude, in 32 bits
    xb = x.view(case["m"], -1, 32)
    big = xb.abs().amax(2, keepdim=True)
    inv = torch.where(big > 0, 127.0 / big, torch.zeros_like(big))
    xq = torch.round(xb * inv).double() * torch.where(inv > 0, 1.0 / inv, torch.zeros_like(inv)).double()
    xq = xq.view(case["m"], -1)
    y = torch.empty((case["m"], case["rows"]), dtype=torch.float64, device="cuda")
    for r in range(0, case["rows"], 4096):
        w = (q[r:r + 4096].double() * d[r:r + 4096].double().unsqueeze(2)).view(-1, case["cols"])
        y[:, r:r + 4096] = xq @ w.T
    return y


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def _shape(case):
    """(weights of the layers, weights of the head, K/V bytes per token, state bytes per request, attention FLOPs per row and
    key, recurrence FLOPs per row, bytes per weight) of a case's model."""
    model, L, W = case["model"], case["layers"], case["width"]
    F = FF[W]
    V = VOCAB[model]
    n_attn = L // 4
    n_rec = L - n_attn
    if model in ("qwen27b", "qwen35"):
        if model == "qwen27b":
            heads, kv, nk, nv = 24, 4, 16, 48
        else:
            heads, kv, nk, nv = W // 256, 4 if W % 1024 == 0 else 2, W // 128, W // 128
        attn = (2 * heads * 256 + 2 * kv * 256) * W + W * heads * 256 + 3 * W * F
        rec = (2 * nk * 128 + 2 * nv * 128 + 2 * nv) * W + W * nv * 128 + 3 * W * F
        return (n_attn * attn + n_rec * rec, V * W, n_attn * kv * 256 * 4, n_rec * nv * 128 * 128 * 4, n_attn * heads * 256 * 4,
                n_rec * nv * 128 * 128 * 8, 34 / 32)
    H = W // 128
    if model == "kezilix":
        attn = H * 192 * W + 576 * W + H * 256 * 512 + W * W + 3 * W * F
        rec = 5 * W * W + 3 * W * F
        per_token, state, aflops = n_attn * 576 * 2, n_rec * H * 128 * 128 * 4, n_attn * H * (192 + 128) * 2
        layers, rflops = n_attn * attn + n_rec * rec, n_rec * H * 128 * 128 * 6
    else:
        n_mls = sum(1 for i in range(L) if i % 4 == 1)
        n_lig = n_rec - n_mls
        layers = int((2.25 * n_attn + 4 * n_mls + 5 * n_lig) * W * W) + L * 3 * W * F
        per_token = n_attn * (H // 4) * 324
        state = n_lig * H * 128 * 128 * 4 + n_mls * (W // 256) * 128 * 256 * 4
        aflops = n_attn * H * 128 * 4
        rflops = n_lig * H * 128 * 128 * 6 + n_mls * (W // 256) * 128 * 256 * 6
    return layers, V * W, per_token, state, aflops, rflops, 2


def work(case):
    if case["kind"] == "matmul":
        n, c, m = case["rows"], case["cols"], case["m"]
        return {"bytes": n * c * 34 / 32 + m * c * 4 + m * n * 4, "flops": 2 * n * c * m}
    layers, head, per_token, state, aflops, rflops, wb = _shape(case)
    if case["kind"] == "prompt":
        lens = _lengths(case["tokens"], case["requests"])
        nbytes = flops = 0
        for n in lens:
            nbytes += (layers + head) * wb + n * per_token + state
            flops += 2 * layers * n + 2 * head + aflops * n * n / 2 + rflops * n
        return {"bytes": nbytes, "flops": flops}
    k, n = case["k"], case["seqs"]
    lens = _lengths(case["ctx"], n)
    nbytes = (layers + head) * wb + sum(lens) * per_token + n * state * (2 + k)
    flops = (2 * (layers + head) + rflops) * n * (k + 1) + aflops * sum(lens) * (k + 1)
    if k:       # the draft layer of the hybrid: one attention layer, the product that joins its two inputs, the head
        W, F = 5120, 17408
        draft = (2 * 24 * 256 + 8 * 256) * W + W * 24 * 256 + 3 * W * F + 2 * W * W
        nbytes += k * ((draft + head) * wb + sum(lens) * 4096)
        flops += k * n * 2 * (draft + head)
    return {"bytes": case["steps"] * nbytes, "flops": case["steps"] * flops}


def tolerance(case):
    if case["kind"] == "matmul":
        # 32-bit sums of up to 544 scaled block products: 2e-7 from the 64-bit value
        return {"rel": 2e-6, "max": 1e-4}
    if case["model"] in ("qwen27b", "qwen35"):
        # the network rounds its activations to 8 bits before every product: one unit in the last place of one norm's gains
        # moves the logits of the 4-layer slice by 1.6 to 2.6 percent
        return {"rel": 0.03, "max": 0.3}
    # the same prompts ingested in other portions (other sums, other blocks of the recurrences): 4e-6 in 32 bits, 8e-3 on the
    # latent-attention family (expanded or absorbed form, bfloat16 latents), 5e-4 on the shared-key/value family
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 1e-4}
    return {"rel": 0.03, "max": 0.13} if case["model"] == "kezilix" else {"rel": 0.01, "max": 0.05}
