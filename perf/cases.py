"""The work this framework is timed on, case by case.

Each case is one call a program makes through the public entry points: a training step or a generation through
`gradcraft_b200.trainer.Trainer`, or a group of operators through the C ABI (`gradcraft_b200.capi.Context`) on buffers that
the program owns.  `listed()` gives the fixed cases, `draw()` further ones of the same ranges; everything a case works on is
made from its seed by `prepare()`, and `run()` makes one pass.
"""
import math

import numpy as np
import torch

from gradcraft_b200 import capi, synth
from gradcraft_b200.trainer import Trainer

HYPER = dict(lr=3e-4, beta1=0.9, beta2=0.95, wd=0.1, eps=1e-5, norm_eps=1e-5, ce_eps=1e-5)
CLIP = 1.0


def model(arch, V, T, C, H, L, F=0):
    """A GPT of either architecture: vocabulary, longest sequence, width, heads, layers, hidden width (RMSNorm + SwiGLU: 3 C)."""
    return dict(arch=arch, V=V, T=T, C=C, H=H, L=L, F=F if arch == "lngelu" else 3 * C)


def listed():
    tiny = model("lngelu", 512, 64, 128, 4, 2, 512)
    mid = model("rmsswiglu", 1024, 256, 256, 4, 2)
    gpt180m = model("lngelu", 32768, 1024, 1024, 16, 12, 4096)
    return [
        # ---- training steps: zero_grad, forward, backward, clip, AdamW; token ids from pinned host memory, the loss read back
        # the two-layer model a user tries things out on: every kernel is short, launches and host work are what counts
        dict(tiny, name="train_tiny", kind="train", B=4, accum=1),
        # a corpus whose tokenizer and document lengths came out odd: no size is a multiple of four but the width
        dict(model("rmsswiglu", 5003, 331, 384, 6, 4), name="train_odd_sizes", kind="train", B=5, accum=1),
        # the model with the sizes that GPTConfig has by default
        dict(model("rmsswiglu", 8192, 512, 768, 12, 11), name="train_default_config", kind="train", B=8, accum=1),
        # 90M parameters, gradient accumulation over two micro-batches
        dict(model("lngelu", 16384, 512, 768, 12, 12, 3072), name="train_90m_accumulating", kind="train", B=32, accum=2),
        # 180M parameters, the headline training step
        dict(gpt180m, name="train_180m", kind="train", B=32, accum=1),
        # ---- generation: greedy decoding from a prompt (sampling adds host work only, and what it picks hangs on the last bit of
        # every logit, through the order in which std::nth_element leaves its candidates)
        # a few words with the small model
        dict(tiny, name="generate_tiny", kind="generate", prompt=8, new=40, seqs=1, context=64),
        # several samples side by side, running past the context window
        dict(mid, name="generate_past_window", kind="generate", prompt=50, new=70, seqs=4, context=96),
        # one continuation of a long prompt with the large model
        dict(gpt180m, name="generate_180m", kind="generate", prompt=385, new=48, seqs=1, context=1024),
        # ---- operators through the C ABI, forward and backward, as a program with its own graph calls them
        # softmax + cross-entropy over a 32k vocabulary
        dict(name="loss_32k", kind="loss", rows=16384, V=32768, i32=True),
        # LayerNorm of a residual stream, its gradient accumulated into the stream's
        dict(name="norm_16k_rows", kind="norm", norm="layernorm", rows=16384, C=1024, accumulate=True),
        # embedding gather and gradient scatter of one batch of Zipf tokens
        dict(name="embedding_zipf", kind="embedding", n=32768, V=32768, C=1024, i32=False),
        # a linear layer with sizes that are no multiple of anything
        dict(name="linear_odd_sizes", kind="linear", M=1023, K=771, N=1029),
    ]


# ---- drawing further cases ------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _draw_model(rng):
    D = rng.choice([16, 24, 32, 40, 64, 64, 96])
    H = rng.randint(2, 16)
    arch = rng.choice(["lngelu", "rmsswiglu"])
    C = D * H
    return model(arch, _log_int(rng, 97, 32768), 0, C, H, rng.randint(1, 12), C * rng.randint(2, 4) + rng.choice([0, 0, 4, 20]))


def _affordable(c):
    """Drawn cases stay below the largest listed one, in work and in what preparing them takes."""
    if c["kind"] == "train":
        return _params(c) < 6e7 and work(c)["flops"] < 1e13 and c["B"] * c["H"] * c["T"] ** 2 * c["L"] < 4e9 and c["B"] * c["T"] * c["V"] < 2e9
    again = c["new"] * min(c["context"], c["prompt"] + c["new"]) * c["seqs"]  # token positions if every step forwards its whole context
    return _params(c) < 6e7 and 2 * _params(c) * again < 1e13


def draw(rng):
    kind = rng.choice(["train", "train", "train", "generate", "generate", "loss", "norm", "embedding", "linear"])
    if kind == "train":
        while True:
            c = dict(_draw_model(rng), kind=kind, B=_log_int(rng, 1, 32), accum=rng.choice([1, 1, 1, 2, 3]))
            c["T"] = _log_int(rng, 16, 1024)
            if rng.random() < 0.5:  # half of the sequences have a length that is a multiple of 64, as most configurations do
                c["T"] = max(64, c["T"] // 64 * 64)
            if _affordable(c):
                return c
    if kind == "generate":
        while True:
            c = dict(_draw_model(rng), kind=kind, prompt=_log_int(rng, 1, 512), new=_log_int(rng, 8, 96), seqs=rng.choice([1, 1, 2, 3, 4, 8]))
            c["T"] = c["context"] = _log_int(rng, 16, 1024)
            if _affordable(c):
                return c
    if kind == "loss":
        V = _log_int(rng, 97, 50021)
        return dict(kind=kind, rows=_log_int(rng, 16, max(16, min(32768, 500_000_000 // V))), V=V, i32=rng.random() < 0.5)
    if kind == "norm":
        C = _log_int(rng, 64, 4096)
        if rng.random() < 0.7:
            C = max(64, C // 32 * 32)
        return dict(kind=kind, norm=rng.choice(["layernorm", "rmsnorm"]), rows=_log_int(rng, 64, min(65536, 40_000_000 // C)), C=C, accumulate=rng.random() < 0.5)
    if kind == "embedding":
        C = _log_int(rng, 64, 1536) // 4 * 4
        return dict(kind=kind, n=_log_int(rng, 64, min(65536, 50_000_000 // C)), V=_log_int(rng, 97, 50021), C=C, i32=rng.random() < 0.5)
    while True:
        c = dict(kind=kind, M=_log_int(rng, 16, 16384), K=_log_int(rng, 16, 4096), N=_log_int(rng, 16, 8192))
        if rng.random() < 0.3:
            c = dict(c, **{d: max(32, c[d] // 32 * 32) for d in ("M", "K", "N")})
        if c["M"] * c["K"] * c["N"] < 1e11:
            return c


# ---- state ----------------------------------------------------------------------------------------------------------------
class _Model:
    """A trainer with seeded weights (matrices N(0, 0.02), biases 0, gains 1), closed when the last holder lets go of it."""

    def __init__(self, case, seed):
        self.tr = Trainer(*(case[k] for k in ("arch", "V", "T", "C", "H", "L", "F")), clip=CLIP, **HYPER)
        g = torch.Generator(device="cuda").manual_seed(seed)
        shapes = synth.gpt_param_shapes(case["arch"], *(case[k] for k in ("V", "T", "C", "H", "L", "F")))
        weights = {}
        for name, (shape, kind) in shapes.items():
            if kind == "matrix":
                weights[name] = (torch.randn(shape, generator=g, device="cuda") * 0.02).cpu().numpy()
            else:
                weights[name] = np.full(shape, 1.0 if kind == "gamma" else 0.0, np.float32)
        self.tr.load(weights)

    def __del__(self):
        self.tr.close()


class _Trained(dict):
    """What a training step leaves: the loss, and the updated weights and the gradients, which stay on the device, where a
    training program leaves them, and are read back when somebody looks at them."""

    def __init__(self, loss, holder):
        super().__init__(loss=loss, weights=None, gradients=None)
        self._holder = holder

    def __getitem__(self, key):
        if key == "loss":
            return super().__getitem__(key)
        got = self._holder.tr.get("param" if key == "weights" else "grad")
        return np.concatenate([got[name] for name, _, _ in self._holder.tr.params()])


class _Operators:
    """A C ABI context on torch's stream and the buffers that a program keeps for it."""

    def __init__(self, **buffers):
        self.ctx = capi.Context()
        self.__dict__.update(buffers)

    def __del__(self):
        self.ctx.close()


def _tokens(case, seed, count):
    return torch.from_numpy(synth.zipf_tokens(seed, count, case["V"]))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        B, T = case["B"], case["T"]
        batches = torch.from_numpy(synth.token_batches(seed, case["accum"], B, T, case["V"])).pin_memory()
        return dict(case=case, model=_Model(case, seed), batches=[(b[0], b[1]) for b in batches])
    if kind == "generate":
        return dict(case=case, model=_Model(case, seed), prompt=_tokens(case, seed, case["prompt"]).numpy())
    g = torch.Generator(device="cuda").manual_seed(seed)

    def randn(*shape, std=1.0):
        return torch.randn(shape, generator=g, device="cuda") * std

    def empty(*shape):
        return torch.empty(shape, device="cuda")

    if kind == "loss":
        M, V = case["rows"], case["V"]
        targets = torch.randint(0, V, (M,), generator=g, device="cuda", dtype=torch.int32 if case["i32"] else torch.int64)
        ops = _Operators(logits=randn(M, V), targets=targets, probs=empty(M, V), dlogits=empty(M, V), loss=empty(1))
    elif kind == "norm":
        M, C = case["rows"], case["C"]
        ops = _Operators(x=randn(M, C), dy=randn(M, C, std=1e-2), gamma=1.0 + randn(C, std=0.1), beta=randn(C, std=0.05), y=empty(M, C), dx=randn(M, C, std=1e-2), mean=empty(M), rstd=empty(M),
                         dgamma=empty(C), dbeta=empty(C))
    elif kind == "embedding":
        n, V, C = case["n"], case["V"], case["C"]
        idx = _tokens(case, seed, n).to("cuda", torch.int32 if case["i32"] else torch.int64)
        ops = _Operators(idx=idx, table=randn(V, C, std=0.02), out=empty(n, C), dy=randn(n, C, std=1e-2), dtable=randn(V, C, std=1e-2))
    else:
        M, K, N = case["M"], case["K"], case["N"]
        ops = _Operators(x=randn(M, K), W=randn(K, N, std=0.02), b=randn(N, std=0.02), y=empty(M, N), dy=randn(M, N, std=1e-2), dx=empty(M, K), dW=empty(K, N), db=empty(N))
        if K >= 128 and N >= 128 and N % 4 == 0:  # as Module::to does with every weight matrix
            ops.ctx.weight_twins_register(ops.W, K, N)
    return dict(case=case, ops=ops)


# ---- one pass -------------------------------------------------------------------------------------------------------------
def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "train":
        loss = state["model"].tr.train_step(state["batches"])
        return _Trained(loss, state["model"])
    if kind == "generate":
        return state["model"].tr.generate(state["prompt"], c["prompt"] + c["new"], num_sequences=c["seqs"], context_length=c["context"])
    o = state["ops"]
    ctx = o.ctx
    if kind == "loss":
        M, V, it = c["rows"], c["V"], capi.IDX_I32 if c["i32"] else capi.IDX_I64
        ctx.softmax_ce_fwd_f32(o.loss, o.probs, o.logits, o.targets, it, M, V, 1e-5)
        ctx.softmax_ce_bwd_f32(o.dlogits, o.probs, o.targets, it, 1.0, M, V, 0)
        return [o.loss, o.probs, o.dlogits]
    if kind == "norm":
        M, C, acc = c["rows"], c["C"], int(c["accumulate"])
        if c["norm"] == "layernorm":
            ctx.layernorm_fwd_f32(o.y, o.mean, o.rstd, o.x, o.gamma, o.beta, M, C, 1e-5)
            ctx.layernorm_bwd_f32(o.dx, o.dgamma, o.dbeta, o.dy, o.x, o.gamma, o.mean, o.rstd, M, C, acc, 0)
            return [o.y, o.mean, o.rstd, o.dx, o.dgamma, o.dbeta]
        ctx.rmsnorm_fwd_f32(o.y, o.rstd, o.x, o.gamma, M, C, 1e-5)
        ctx.rmsnorm_bwd_f32(o.dx, o.dgamma, o.dy, o.x, o.gamma, o.rstd, M, C, acc, 0)
        return [o.y, o.rstd, o.dx, o.dgamma]
    if kind == "embedding":
        n, V, C, it = c["n"], c["V"], c["C"], capi.IDX_I32 if c["i32"] else capi.IDX_I64
        ctx.embed_f32(o.out, o.idx, it, o.table, n, C, V)
        ctx.scatter_add_f32(o.dtable, o.idx, it, o.dy, n, C, V)
        return [o.out, o.dtable]
    M, K, N = c["M"], c["K"], c["N"]
    ctx.gemm_f32(capi.OP_N, capi.OP_N, M, N, K, 1.0, o.x, K, o.W, N, 0.0, o.y, N, o.b)
    ctx.gemm_f32(capi.OP_N, capi.OP_T, M, K, N, 1.0, o.dy, N, o.W, N, 0.0, o.dx, K, None)
    ctx.gemm_colsum_f32(capi.OP_T, K, N, M, 1.0, o.x, K, o.dy, 0.0, o.dW, N, o.db, 0)
    return [o.y, o.dx, o.dW, o.db]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------
def _matrices(c):
    """Weights of one layer's linear maps."""
    C, F = c["C"], c["F"]
    return 4 * C * C + (2 if c["arch"] == "lngelu" else 3) * C * F


def _params(c):
    return c["L"] * _matrices(c) + (c["V"] + c["T"]) * c["C"]


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        tokens = c["B"] * c["T"] * c["accum"]
        # weights and both moments in and out, gradients out, ids in; causal attention: half of the square
        return dict(bytes=28 * _params(c) + 16 * tokens, flops=tokens * (6 * (c["L"] * _matrices(c) + c["C"] * c["V"]) + 6 * c["L"] * c["T"] * c["C"]))
    if kind == "generate":
        # every new token waits for the one before it, so each reads the weights once; a position is forwarded once while the
        # window still holds the whole text, and the whole window is once its positions have shifted
        flops = 0
        for step in range(c["prompt"], c["prompt"] + c["new"]):
            fresh = step if step == c["prompt"] else 1
            if step > c["context"] or fresh > c["context"]:
                fresh = c["context"]
            flops += c["seqs"] * (2 * fresh * c["L"] * (_matrices(c) + c["C"] * min(step, c["context"])) + 2 * c["C"] * c["V"])
        return dict(bytes=4 * c["new"] * (c["L"] * _matrices(c) + c["V"] * c["C"]) + 8 * c["seqs"] * (c["prompt"] + c["new"]), flops=flops)
    if kind == "loss":  # logits in, probabilities out and in, their gradient out
        n = c["rows"] * c["V"]
        return dict(bytes=16 * n + c["rows"] * (8 if c["i32"] else 16), flops=8 * n)
    if kind == "norm":  # x in, y out; x and dy in, dx out (in as well where it is accumulated into)
        n = c["rows"] * c["C"]
        return dict(bytes=(20 + 4 * int(c["accumulate"])) * n, flops=20 * n)
    if kind == "embedding":  # the rows that occur in, n rows out; n gradient rows in, the rows that occur in and out
        p = np.diff(synth.zipf_cdf(c["V"]), prepend=0.0)
        hit = float(np.sum(1.0 - np.exp(c["n"] * np.log1p(-p))))
        return dict(bytes=4 * c["C"] * (2 * c["n"] + 3 * hit) + 2 * c["n"] * (4 if c["i32"] else 8), flops=c["n"] * c["C"])
    M, K, N = c["M"], c["K"], c["N"]
    return dict(bytes=4 * (3 * M * K + 3 * M * N + 3 * K * N), flops=6 * M * K * N)


def tolerance(case):
    if case["kind"] == "train":  # 32-bit products and sums through every layer and back; one AdamW step on top
        return {"rel": 1e-4}
    if case["kind"] == "generate":  # token ids; a tie between two logits may fall either way
        return {"rel": 0.0, "differ": 0.01}
    return {"rel": 1e-5}
