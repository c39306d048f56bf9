"""What this library's speed is measured on: the work its users have it do, through its public entry points.

A user trains the decoder (a step, a validation loss), generates with it (a prompt pass, greedy or sampled
continuation), or calls the kernels from a training program of their own (a linear layer's forward pass and both
gradients, causal attention forward and backward, a matrix product on host arrays).  Each kind of work has its range of
sizes here: `listed` holds fixed points of it, `draw` gives any other.  Sizes are those of this repository's benchmark,
its tests and the model it is built for (12 layers of width 384 and a vocabulary of 31,769), and sizes between.
"""
import numpy as np
import torch

from turkce_llm_b200 import lib
from turkce_llm_b200.decode import Decoder
from turkce_llm_b200.gpu_train import ADAM_M, ADAM_V, GRADS, PARAMS, AdamState, GpuTrainer

# V, D, H, L, F: the model of the benchmark, its 24-layer and 2-layer forms, and the tests' narrow models
MODELS = {
    "base": (31769, 384, 6, 12, 1024),
    "deep": (31769, 384, 6, 24, 1024),
    "shallow": (31769, 384, 6, 2, 1024),
    "wide": (500, 256, 4, 3, 1024),
    "small": (300, 64, 2, 2, 128),
}
EPS = 1e-5
PRECISIONS = {"bf16": lib.PREC_BF16, "tf32": lib.PREC_TF32, "fp32": lib.PREC_FP32}
# (in, out) of the model's four linear layers
LAYERS = ((384, 1152), (384, 384), (384, 2048), (1024, 384))


def listed():
    return [
        # a step of a test-sized model: nothing but launches and host work
        {"name": "train_small", "kind": "train", "model": "small", "batch": 4, "context": 64, "precision": "bf16"},
        # the first production run of the reference's GPU trainer: 28 windows of 128 tokens, here with TF32 operands
        {"name": "train_28x128_tf32", "kind": "train", "model": "base", "batch": 28, "context": 128, "precision": "tf32"},
        # the benchmark's training step
        {"name": "train_8x1024", "kind": "train", "model": "base", "batch": 8, "context": 1024, "precision": "bf16"},
        # the reference's largest run: 24 layers, 14 windows of 1024 tokens
        {"name": "train_deep_14x1024", "kind": "train", "model": "deep", "batch": 14, "context": 1024, "precision": "bf16"},
        # validation loss on windows of a length that is no multiple of anything
        {"name": "eval_5x777", "kind": "eval", "model": "base", "batch": 5, "context": 777, "precision": "bf16"},
        # a batch of long prompts scored: next token and its logits
        {"name": "prompt_16x700", "kind": "prompt", "model": "base", "seqs": 16, "prompt": 700},
        # the benchmark's batched generation
        {"name": "generate_64", "kind": "generate", "model": "base", "seqs": 64, "prompt": 128, "new": 128, "temperature": 0.0},
        # a chat: one sequence, a short prompt, sampled
        {"name": "generate_1_sampled", "kind": "generate", "model": "base", "seqs": 1, "prompt": 37, "new": 80, "temperature": 0.8},
        # the QKV projection of 4 x 256 tokens on float32 matrices at float32 precision, as the reference stores them
        {"name": "linear_1024_fp32", "kind": "linear", "rows": 1024, "inner": 384, "outer": 1152, "precision": "fp32"},
        # the gate|up projection of 8 x 1024 tokens on bf16 matrices
        {"name": "linear_8192_native", "kind": "linear", "rows": 8192, "inner": 384, "outer": 2048, "precision": "native"},
        # the benchmark's attention
        {"name": "attention_16x1024", "kind": "attention", "batch": 16, "heads": 6, "context": 1024, "head_dim": 64},
        # a product of host arrays, copies included
        {"name": "host_matmul_1024", "kind": "matmul", "m": 1024, "k": 1024, "n": 1024, "precision": "fp32"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    kind = rng.choice(["train", "train", "eval", "prompt", "generate", "generate", "linear", "linear", "attention", "matmul"])
    if kind in ("train", "eval"):
        context = _log_int(rng, 12, 1024)
        tokens = _log_int(rng, max(64, context), 8192)
        return {"kind": kind, "model": rng.choice(["base", "base", "shallow", "wide", "small"]), "batch": max(1, tokens // context),
                "context": context, "precision": rng.choice(["bf16", "bf16", "tf32"])}
    if kind == "prompt":
        prompt = _log_int(rng, 3, 1000)
        return {"kind": kind, "model": rng.choice(["base", "base", "shallow", "wide", "small"]),
                "seqs": min(_log_int(rng, 1, 64), max(1, 12000 // prompt)), "prompt": prompt}
    if kind == "generate":
        return {"kind": kind, "model": rng.choice(["base", "base", "base", "shallow", "wide", "small"]), "seqs": _log_int(rng, 1, 64),
                "prompt": _log_int(rng, 3, 128), "new": _log_int(rng, 8, 128), "temperature": rng.choice([0.0, 0.0, 0.8])}
    if kind == "linear":
        precision = rng.choice(["native", "bf16", "tf32", "fp32"])
        rows = _log_int(rng, 16, 8192)
        if precision == "native" or rng.random() < 0.5:
            inner, outer = rng.choice(LAYERS)
        else:
            inner, outer = _log_int(rng, 40, 1100), _log_int(rng, 40, 2048)
        return {"kind": kind, "rows": rows, "inner": inner, "outer": outer, "precision": precision}
    if kind == "attention":
        context = _log_int(rng, 12, 1024)
        return {"kind": kind, "batch": _log_int(rng, 1, 16), "heads": rng.choice([1, 2, 3, 6]), "context": context,
                "head_dim": rng.choice([16, 32, 64, 64, 64])}
    return {"kind": "matmul", "m": _log_int(rng, 16, 1024), "k": _log_int(rng, 16, 1024), "n": _log_int(rng, 16, 1024),
            "precision": rng.choice(["bf16", "tf32", "fp32"])}


# ---------------------------------------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(gen, *shape, std=1.0):
    return torch.randn(shape, device="cuda", generator=gen) * std


def _zipf(gen, count, vocab):
    """Token ids, Zipf(1.1) over the vocabulary."""
    cdf = torch.cumsum(torch.arange(1, vocab + 1, device="cuda", dtype=torch.float64) ** -1.1, 0)
    u = torch.rand(count, device="cuda", dtype=torch.float64, generator=gen) * cdf[-1]
    return torch.searchsorted(cdf, u).clamp_(max=vocab - 1).cpu().numpy().astype(np.uint32)


def _weights(gen, model, embedding_std):
    """Flat parameters: N(0, 0.02) matrices, norm weights and biases a little off one and zero, as after some training."""
    V, D, _, L, F = MODELS[model]
    parts = [_normal(gen, V * D, std=embedding_std)]
    for _ in range(L):
        parts += [1 + _normal(gen, D, std=0.05), _normal(gen, D * 3 * D, std=0.02), _normal(gen, 3 * D, std=0.02),
                  _normal(gen, D * D, std=0.02), _normal(gen, D, std=0.02), 1 + _normal(gen, D, std=0.05),
                  _normal(gen, D * 2 * F, std=0.02), _normal(gen, 2 * F, std=0.02), _normal(gen, F * D, std=0.02),
                  _normal(gen, D, std=0.02)]
    parts.append(1 + _normal(gen, D, std=0.05))
    return torch.cat(parts).cpu().numpy()


class _DeviceView:
    """A flat buffer of a trainer as torch sees it, without a copy; keeps the trainer alive as long as the tensor."""

    def __init__(self, trainer, which):
        self.trainer = trainer
        self.__cuda_array_interface__ = {"shape": (trainer.total,), "typestr": "<f4", "data": (trainer.device_ptr(which), False),
                                         "version": 2}


def _view(trainer, which):
    return torch.as_tensor(_DeviceView(trainer, which), device="cuda")


def prepare(case, seed):
    lib.init(0)
    gen = _generator(seed)
    s = {"kind": case["kind"], "case": case}
    if case["kind"] in ("train", "eval"):
        V, D, H, L, F = MODELS[case["model"]]
        T, B = case["context"], case["batch"]
        g = GpuTrainer(V, D, H, L, F, T, B, EPS, precision=PRECISIONS[case["precision"]])
        g.upload(_weights(gen, case["model"], 0.02))
        tokens = _zipf(gen, B * (T + 1), V).reshape(B, T + 1)
        s.update(trainer=g, opt=AdamState(lr=3e-4), ids=np.ascontiguousarray(tokens[:, :-1]).reshape(-1),
                 targets=np.ascontiguousarray(tokens[:, 1:]).reshape(-1))
        if case["kind"] == "train":
            s["views"] = {"params": _view(g, PARAMS), "grads": _view(g, GRADS), "adam_m": _view(g, ADAM_M), "adam_v": _view(g, ADAM_V)}
    elif case["kind"] in ("prompt", "generate"):
        V, D, H, L, F = MODELS[case["model"]]
        S, T = case["seqs"], case["prompt"]
        new = case.get("new", 1)
        d = Decoder(V, D, H, L, F, S, T + new + 1, EPS)
        # a trained model prefers some token clearly; among the near-equal logits of small random embeddings the choice
        # would hang on the last bit of a sum
        d.upload(_weights(gen, case["model"], 0.25))
        if case.get("temperature", 0.0) > 0.0:
            d.set_sampling(case["temperature"], 4242, 7 + int(seed))
        s.update(decoder=d, prompts=_zipf(gen, S * T, V).reshape(S, T), new=new)
    elif case["kind"] == "linear":
        M, K, N = case["rows"], case["inner"], case["outer"]
        native = case["precision"] == "native"
        dt = torch.bfloat16 if native else torch.float32
        s.update(x=_normal(gen, M, K).to(dt), w=_normal(gen, K, N, std=0.02).to(dt), bias=_normal(gen, N, std=0.02),
                 dy=_normal(gen, M, N).to(dt), y=torch.empty(M, N, device="cuda", dtype=dt),
                 dx=torch.empty(M, K, device="cuda"), dw=torch.zeros(K, N, device="cuda"),
                 precision=None if native else PRECISIONS[case["precision"]])
    elif case["kind"] == "attention":
        B, H, T, hd = case["batch"], case["heads"], case["context"], case["head_dim"]
        for name in ("q", "k", "v"):
            s[name] = _normal(gen, B * H, T, hd).to(torch.bfloat16)
        s.update(datt=_normal(gen, B * T, H * hd).to(torch.bfloat16), delta=torch.empty(B * H, T, device="cuda"))
        s["out"] = {"att": torch.empty(B * T, H * hd, device="cuda", dtype=torch.bfloat16), "lse": torch.empty(B * H, T, device="cuda"),
                    "dq": torch.empty(B * H, T, hd, device="cuda"), "dk": torch.empty(B * H, T, hd, device="cuda"),
                    "dv": torch.empty(B * H, T, hd, device="cuda")}
    else:
        M, K, N = case["m"], case["k"], case["n"]
        s.update(a=_normal(gen, M, K).cpu().numpy(), b=_normal(gen, K, N, std=0.02).cpu().numpy(), c=np.zeros((M, N), np.float32),
                 precision=PRECISIONS[case["precision"]])
    return s


# ---------------------------------------------------------------------------------------------- one pass

def run(s):
    case = s["case"]
    if s["kind"] == "train":
        # one iteration of the training loop: forward, backward, clip, Adam; loss and norm come back
        loss, norm = s["trainer"].train_step(s["ids"], s["targets"], s["opt"], 1.0)
        return {"loss": loss, "norm": norm, **s["views"]}
    if s["kind"] == "eval":
        return s["trainer"].eval_loss(s["ids"], s["targets"])
    if s["kind"] == "prompt":
        s["decoder"].prefill(s["prompts"])
        return {"token": s["decoder"].tokens(1), "logits": s["decoder"].logits()}
    if s["kind"] == "generate":
        s["decoder"].prefill(s["prompts"])
        s["decoder"].generate(s["new"] - 1)
        return s["decoder"].tokens(s["new"])
    if s["kind"] == "linear":
        M, K, N = case["rows"], case["inner"], case["outer"]
        if s["precision"] is None:
            # forward with bias, input gradient, weight gradient added to what the step has gathered so far
            lib.gemm_bf16(lib.NN, s["x"], s["w"], M, N, K, K, N, C16=s["y"], ldc16=N, bias=s["bias"])
            lib.gemm_bf16(lib.NT, s["dy"], s["w"], M, K, N, N, N, C32=s["dx"], ldc32=K)
            lib.gemm_bf16(lib.TN, s["x"], s["dy"], K, N, M, K, N, C32=s["dw"], ldc32=N, beta=1.0)
        else:
            lib.gemm_bias_f32(s["x"], s["w"], s["bias"], None, s["y"], M, N, K, precision=s["precision"])
            lib.gemm_f32(lib.NT, s["dy"], s["w"], s["dx"], M, K, N, N, N, K, precision=s["precision"])
            lib.gemm_f32(lib.TN, s["x"], s["dy"], s["dw"], K, N, M, K, N, N, beta=1.0, precision=s["precision"])
        return {"y": s["y"], "dx": s["dx"], "dw": s["dw"]}
    if s["kind"] == "attention":
        B, H, T, hd = case["batch"], case["heads"], case["context"], case["head_dim"]
        o, scale = s["out"], float(hd) ** -0.5
        lib.attention_fwd(s["q"], s["k"], s["v"], o["att"], o["lse"], B, H, T, hd, scale)
        lib.attention_bwd(s["q"], s["k"], s["v"], o["att"], s["datt"], o["lse"], s["delta"], o["dq"], o["dk"], o["dv"], B, H, T, hd, scale)
        return o
    lib.matmul_host(s["a"], s["b"], s["c"], case["m"], case["k"], case["n"], s["precision"])
    return s["c"]


# ---------------------------------------------------------------------------------------------- what a pass cannot do without

def _linear_scalars(model):
    V, D, _, L, F = MODELS[model]
    return L * (D * 3 * D + D * D + D * 2 * F + F * D), V * D


def work(case):
    if case["kind"] in ("train", "eval"):
        V, D, H, L, F = MODELS[case["model"]]
        T, N = case["context"], case["context"] * case["batch"]
        layers, table = _linear_scalars(case["model"])
        total = layers + table + L * (2 * D + 3 * D + D + 2 * F + D) + D
        # causal attention: two triangular products forward, four more backward
        attention = 2.0 * N * T * D * L
        if case["kind"] == "eval":
            weight = 2 if case["precision"] == "bf16" else 4
            return {"bytes": weight * total + 8 * N, "flops": 2.0 * N * (layers + table) + attention}
        # every parameter with both moments read and written, its gradient written
        return {"bytes": 28 * total + 8 * N, "flops": 6.0 * N * (layers + table) + 3 * attention}
    if case["kind"] in ("prompt", "generate"):
        V, D, H, L, F = MODELS[case["model"]]
        S, T, steps = case["seqs"], case["prompt"], case.get("new", 1) - 1
        layers, table = _linear_scalars(case["model"])
        row = 4 * D * L                                          # key and value of one position, bf16, all layers
        flops = 2.0 * S * (T + steps) * layers + 2.0 * S * (1 + steps) * table + 2.0 * S * T * T * D * L
        read = sum(T + i + 1 for i in range(steps))              # cache positions the steps attend to
        flops += 4.0 * S * read * D * L
        move = 2 * (layers + table) * (1 + steps) + S * (T + steps) * row + S * read * row + 4 * S * (T + 1 + steps)
        return {"bytes": move + (4 * S * V if case["kind"] == "prompt" else 0), "flops": flops}
    if case["kind"] == "linear":
        M, K, N = case["rows"], case["inner"], case["outer"]
        size = 2 if case["precision"] == "native" else 4
        # x, w, dy in; y and dx out, dw read and written
        return {"bytes": size * (M * K + K * N + 2 * M * N) + 4 * (M * K + 2 * K * N + N), "flops": 6.0 * M * N * K}
    if case["kind"] == "attention":
        B, H, T, hd = case["batch"], case["heads"], case["context"], case["head_dim"]
        rows = B * H * T
        return {"bytes": rows * hd * (5 * 2 + 3 * 4) + 4 * rows, "flops": 6.0 * rows * T * hd}
    M, K, N = case["m"], case["k"], case["n"]
    return {"bytes": 4 * (M * K + K * N + M * N), "flops": 2.0 * M * N * K}


def tolerance(case):
    if case["kind"] == "train":
        # bf16 operands and a bf16 attention core; the squared gradients of Adam's second moment count twice
        return {"rel": 5e-3, "max": 0.3}
    if case["kind"] == "eval":
        return {"rel": 1e-4}
    if case["kind"] == "prompt":
        return {"rel": 1e-2, "differ": 0.005}
    if case["kind"] == "generate":
        return {"rel": 0.0, "differ": 0.005}
    if case["kind"] == "attention":
        return {"rel": 1e-2}
    if case.get("precision") == "native":
        return {"rel": 5e-3}                                     # y leaves as bf16
    # operands of 8, 11 and 24 bits; sums in float32
    return {"rel": {"bf16": 2e-5, "tf32": 1e-3, "fp32": 1e-5}[case["precision"]]}
