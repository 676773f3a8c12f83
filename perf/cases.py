"""What is measured when this framework is made faster: the work its users have it do, through its public entry points.

Five kinds of work, each with its forward and its backward direction:

* ``train``      one optimizer step of a model through ``Trainer.train_step`` (dense Llama and GPT families);
* ``attention``  packed variable-length attention, ``pymha_varlen_fwd`` and ``pymha_varlen_bwd``;
* ``linear``     one linear layer, ``gemm_fwd`` and ``gemm_bwd`` (data gradient, weight gradient added to fp32);
* ``head``       LM head and cross entropy, logits to gradients, through ``gemm_*`` and ``cross_entropy_*``;
* ``moe``        the routed expert MLP of one layer, as the layer program's ops run it.

Sizes are those of the presets in ``dhellam_b200/config.py`` (the whole layer, or one GPU's share of it under tensor
parallelism), of the smoke run in ``__graft_entry__.py`` and of the tests, with fewer layers so that a pass stays short,
or generic ones in between.
"""
import math
import random

import torch

from dhellam_b200 import gemm_bwd, gemm_fwd, pymha_varlen_bwd, pymha_varlen_fwd
from dhellam_b200.config import ModelConfig, ParallelConfig, TrainConfig
from dhellam_b200.core.engine import Env
from dhellam_b200.core.modules import DSLLM
from dhellam_b200.data import synthetic_step_batches
from dhellam_b200.models.transformer import build_layer_program
from dhellam_b200.ops.loss import cross_entropy_bwd, cross_entropy_fwd
from dhellam_b200.ops.moe_native import DeviceMoE
from dhellam_b200.parallel import state as PS
from dhellam_b200.sched.ir import LayerRun
from dhellam_b200.trainer import Trainer

DEV = "cuda"
D = 128                                        # head size of every preset

MOE_FWD = ("router_mlp", "dispatch_mlp", "gemm_expert_c", "act_expert", "gemm_expert_l", "combine_mlp")
MOE_BWD = ("combine_mlp_bwd", "gemm_dgrad_expert_l", "gemm_wgrad_expert_l", "act_expert_bwd", "gemm_dgrad_expert_c",
           "gemm_wgrad_expert_c", "dispatch_mlp_bwd", "router_mlp_bwd")


# --------------------------------------------------------------------------- the cases
def _train(layers, hidden, ffn, heads, kv_heads, vocab, seq, micro_batch, global_batch, family="llama", dropout=0.0,
           label_smoothing=0.0):
    return dict(kind="train", family=family, layers=layers, hidden=hidden, ffn=ffn, heads=heads, kv_heads=kv_heads, vocab=vocab,
                seq=seq, micro_batch=micro_batch, global_batch=global_batch, dropout=dropout, label_smoothing=label_smoothing)


def _attention(q_lengths, k_lengths, heads, kv_heads, causal=True, offsets="host"):
    return dict(kind="attention", q_lengths=" ".join(map(str, q_lengths)), k_lengths=" ".join(map(str, k_lengths)), heads=heads,
                kv_heads=kv_heads, causal=causal, offsets=offsets)


def _linear(tokens, n_in, n_out):
    return dict(kind="linear", tokens=tokens, n_in=n_in, n_out=n_out)


def _head(tokens, hidden, vocab, label_smoothing=0.0):
    return dict(kind="head", tokens=tokens, hidden=hidden, vocab=vocab, label_smoothing=label_smoothing)


def _moe(tokens, hidden, ffn, experts, top_k):
    return dict(kind="moe", tokens=tokens, hidden=hidden, ffn=ffn, experts=experts, top_k=top_k)


RAGGED = [977, 64, 2048, 311, 1500, 128, 733, 3071, 45, 1024, 260, 1888, 17, 610, 4000, 419]


def listed():
    return [
        # the smoke run's model: a step of a model this small is launches and host work (debugging, unit runs, sweeps of small models)
        dict(name="train-small", **_train(2, 512, 1024, 4, 2, 2048, 256, 2, 4)),
        # two layers of the 8B preset with its whole vocabulary, the ordinary pre-training step on one GPU
        dict(name="train-llama-8b", **_train(2, 4096, 14336, 32, 8, 128256, 4096, 1, 2)),
        # two layers of the 70B preset, one GPU's half of the heads, FFN and vocabulary under two-way tensor parallelism: the largest GEMMs
        dict(name="train-llama-70b-half", **_train(2, 8192, 14336, 32, 4, 64128, 4096, 1, 4)),
        # long context: a quarter of the 8B preset's heads on 32k tokens, where attention is most of the step
        dict(name="train-long-context", **_train(2, 4096, 3584, 8, 2, 32064, 32768, 1, 1)),
        # the GPT preset: layer norm, GeLU, dropout, as many KV heads as query heads, a sequence length that fills no tile
        dict(name="train-gpt-13b", **_train(2, 5120, 20480, 40, 40, 50304, 1900, 2, 4, family="gpt", dropout=0.1)),
        # a packed batch of documents of unequal length (fine-tuning), GQA
        dict(name="attention-packed", **_attention(RAGGED, RAGGED, 32, 8)),
        # two short sequences, offsets on the device as the reference's callers hold them: the smallest attention call
        dict(name="attention-short", **_attention([200, 200], [200, 200], 4, 2, offsets="device")),
        # one context-parallel chunk of queries against the keys before it
        dict(name="attention-chunk", **_attention([2048], [14336], 16, 4)),
        # a few hundred tokens through the 8B preset's QKV projection (short fine-tuning samples)
        dict(name="linear-few-tokens", **_linear(300, 4096, 6144)),
        # the headline benchmark's FC1 on one of eight GPUs
        dict(name="linear-many-tokens", **_linear(16384, 8192, 7168)),
        # LM head and loss with label smoothing, GPT vocabulary
        dict(name="head-gpt", **_head(4096, 5120, 50304, 0.1)),
        # the Mixtral-style expert MLP
        dict(name="moe-mixtral", **_moe(4096, 4096, 14336, 8, 2)),
    ]


def _log(rng, lo, hi, multiple=1):
    """A size between lo and hi, spread over its logarithm, rounded to a multiple."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(multiple, int(round(v / multiple)) * multiple)


def draw(rng: random.Random):
    kind = rng.choice(["train", "train", "attention", "attention", "linear", "linear", "head", "moe"])
    if kind == "train":
        while True:
            kv = rng.choice([1, 2, 4, 8])
            heads = kv * rng.choice([1, 2, 4, 8])
            family = rng.choice(["llama", "llama", "gpt"])
            micro = rng.choice([1, 1, 2, 4])
            case = _train(2 * rng.choice([1, 1, 2]), _log(rng, 512, 8192, 128), _log(rng, 1024, 20480, 64), min(heads, 40),
                          heads if family == "gpt" else kv, _log(rng, 2048, 65536, 8), _log(rng, 100, 16384), micro,
                          micro * rng.choice([1, 2, 3]), family=family, dropout=0.1 if family == "gpt" else 0.0,
                          label_smoothing=rng.choice([0.0, 0.0, 0.1]))
            if heads <= 40 and work(case)["flops"] <= 1.0e14 and _params(case) <= 1.2e9:
                return case
    if kind == "attention":
        while True:
            kv = rng.choice([1, 2, 4, 8])
            heads = kv * rng.choice([1, 2, 4, 8])
            n = _log(rng, 1, 24)
            shape = rng.choice(["equal", "ragged", "ragged", "prefix"])
            if shape == "equal":
                q = [_log(rng, 64, 8192)] * n
            else:
                q = [_log(rng, 16, 8192) for _ in range(n)]
            k = [a + _log(rng, 16, 16384) for a in q] if shape == "prefix" else q
            case = _attention(q, k, heads, kv, causal=rng.random() < 0.8, offsets=rng.choice(["host", "host", "device"]))
            if heads <= 64 and sum(k) <= 65536 and work(case)["flops"] <= 1.0e13:
                return case
    if kind == "linear":
        while True:
            case = _linear(_log(rng, 8, 32768), _log(rng, 512, 28672, 8), _log(rng, 512, 28672, 8))
            if work(case)["flops"] <= 1.2e13:
                return case
    if kind == "head":
        while True:
            case = _head(_log(rng, 64, 16384), _log(rng, 512, 8192, 8), _log(rng, 2048, 131072, 8), rng.choice([0.0, 0.0, 0.1]))
            if work(case)["flops"] <= 1.0e13:
                return case
    while True:
        experts = rng.choice([4, 8, 16])
        case = _moe(_log(rng, 64, 16384), _log(rng, 512, 5120, 256), _log(rng, 512, 14336, 128), experts, rng.choice([1, 2, 2, 4]))
        if work(case)["flops"] <= 1.5e13 and _params(case) <= 3.2e9:
            return case


# --------------------------------------------------------------------------- inputs, plans and weights
def _model_config(c):
    gpt = c["family"] == "gpt"
    return ModelConfig(name="measured", num_layers=c["layers"], hidden_size=c["hidden"], ffn_hidden_size=c["ffn"],
                       num_attention_heads=c["heads"], num_query_groups=c["kv_heads"], head_dim=D, vocab_size=c["vocab"],
                       seq_length=c["seq"], norm="layernorm" if gpt else "rmsnorm", activation="gelu" if gpt else "swiglu",
                       rope_theta=10000.0 if gpt else 500000.0, hidden_dropout=c["dropout"])


def _moe_config(c):
    return ModelConfig(name="measured-moe", num_layers=2, hidden_size=c["hidden"], ffn_hidden_size=c["ffn"], num_attention_heads=4,
                       num_query_groups=2, head_dim=D, vocab_size=1024, seq_length=c["tokens"], num_experts=c["experts"],
                       moe_top_k=c["top_k"])


def _params(c):
    """Parameters that the case's state holds."""
    return (_model_config(c) if c["kind"] == "train" else _moe_config(c)).total_params()


def _lengths(c):
    return [int(x) for x in c["q_lengths"].split()], [int(x) for x in c["k_lengths"].split()]


def _offsets(lengths, where):
    out = [0]
    for n in lengths:
        out.append(out[-1] + n)
    t = torch.tensor(out, dtype=torch.int32)
    return t.to(DEV) if where == "device" else t


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(*shape, scale=1.0, dtype=torch.bfloat16):
        return (torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * scale).to(dtype)

    kind = case["kind"]
    if kind == "train":
        cfg = _model_config(case)
        train = TrainConfig(micro_batch_size=case["micro_batch"], global_batch_size=case["global_batch"], seed=seed,
                            label_smoothing=case["label_smoothing"])
        PS.set_state(None)
        trainer = Trainer(cfg, ParallelConfig(), train, device=DEV)
        return dict(kind=kind, trainer=trainer, batches=synthetic_step_batches(cfg, train, trainer.ps, 0, DEV))
    if kind == "attention":
        ql, kl = _lengths(case)
        tq, tk, h, hk = sum(ql), sum(kl), case["heads"], case["kv_heads"]
        return dict(kind=kind, q=normal(tq, h, D), k=normal(tk, hk, D), v=normal(tk, hk, D), dout=normal(tq, h, D),
                    cu_q=_offsets(ql, case["offsets"]), cu_k=_offsets(kl, case["offsets"]), max_q=max(ql), max_k=max(kl),
                    causal=case["causal"])
    if kind == "linear":
        t, n_in, n_out = case["tokens"], case["n_in"], case["n_out"]
        return dict(kind=kind, x=normal(t, n_in), w=normal(n_out, n_in, scale=0.02), dy=normal(t, n_out, scale=0.01),
                    main_grad=torch.zeros(n_out, n_in, dtype=torch.float32, device=DEV))
    if kind == "head":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        labels = torch.randint(0, v, (t,), generator=g, device=DEV)
        return dict(kind=kind, x=normal(t, h), w=normal(v, h, scale=0.02), labels=labels,
                    dloss=torch.full((t,), 1.0 / t, dtype=torch.float32, device=DEV), smoothing=case["label_smoothing"],
                    main_grad=torch.zeros(v, h, dtype=torch.float32, device=DEV))
    cfg = _moe_config(case)
    train = TrainConfig(micro_batch_size=1, global_batch_size=1, seed=seed)
    PS.set_state(None)
    ps = PS.initialize_model_parallel(ParallelConfig())
    model = DSLLM(cfg, ps, train, device=DEV)
    env = Env(cfg, ps, train, DEV, model.dtype)
    env.moe_dev = DeviceMoE(ps, cfg, train, DEV, case["tokens"])
    return dict(kind=kind, model=model, env=env, program=build_layer_program(cfg), x=normal(case["tokens"], case["hidden"]),
                dout=normal(case["tokens"], case["hidden"], scale=0.01))


# --------------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "train":
        tr = state["trainer"]
        loss = tr.train_step(state["batches"])
        opt = tr.optimizer
        return dict(loss=loss, grad_norm=tr.last_grad_norm, grads=tr.model.flat_grad, params=tr.model.flat_param, master=opt.master,
                    exp_avg=opt.exp_avg, exp_avg_sq=opt.exp_avg_sq)
    if kind == "attention":
        s = state
        packed = (s["cu_q"], s["cu_k"], s["max_q"], s["max_k"])
        out, lse = pymha_varlen_fwd(s["q"], s["k"], s["v"], *packed, is_causal=s["causal"])
        dq, dk, dv = pymha_varlen_bwd(s["dout"], s["q"], s["k"], s["v"], out, lse, *packed, is_causal=s["causal"])
        return dict(out=out, lse=lse, dq=dq, dk=dk, dv=dv)
    if kind == "linear":
        y, _ = gemm_fwd(None, state["x"], state["w"])
        dx, dw, _, _ = gemm_bwd(None, state["dy"], state["w"], state["x"], None, state["main_grad"], grad_accumulate=True)
        return dict(y=y, dx=dx, dw=dw)
    if kind == "head":
        logits, _ = gemm_fwd(None, state["x"], state["w"])
        ctx = cross_entropy_fwd({"vocab_parallel_logits": logits, "target": state["labels"]}, label_smoothing=state["smoothing"])
        dlogits = cross_entropy_bwd(ctx, state["dloss"])
        dx, dw, _, _ = gemm_bwd(None, dlogits, state["w"], state["x"], None, state["main_grad"], grad_accumulate=True)
        return dict(loss=ctx["loss"], dlogits=dlogits, dx=dx, dw=dw)
    env, program = state["env"], state["program"]
    params = state["model"].blocks[0][0]
    env.moe_aux = []
    fwd = LayerRun(params, {}, None, env, {"ln2": state["x"]})
    for name in MOE_FWD:
        program.op(name).fn(fwd)
    bwd = LayerRun(params, fwd.acts, None, env, {"d_fc2": state["dout"]})
    for name in MOE_BWD:
        program.op(name).fn(bwd)
    return dict(out=fwd.v["fc2"], aux=env.moe_aux[0], dx=bwd.v["d_ln2"], d_router=params.router_weight.main_grad,
                d_column=params.expert_column_weight.main_grad, d_linear=params.expert_linear_weight.main_grad)


# --------------------------------------------------------------------------- what a pass cannot do without
def _visible(nq, nk, causal):
    """Query-key pairs of one sequence; causal rows are aligned at the end."""
    if not causal:
        return nq * nk
    first = nk - nq + 1                        # keys that the first query sees
    return nq * first + nq * (nq - 1) // 2 if first >= 0 else nk * (nk + 1) // 2


def work(case):
    kind = case["kind"]
    if kind == "train":
        cfg = _model_config(case)
        tokens = case["seq"] * case["global_batch"]
        # weights and optimizer state read and written, gradients written, token ids and labels read
        return dict(bytes=32.0 * cfg.total_params() + 8.0 * tokens, flops=cfg.flops_per_token() * tokens)
    if kind == "attention":
        ql, kl = _lengths(case)
        pairs = sum(_visible(a, b, case["causal"]) for a, b in zip(ql, kl))
        tq, tk, h, hk = sum(ql), sum(kl), case["heads"], case["kv_heads"]
        # q, k, v, dout read and out, lse, dq, dk, dv written; two products forward, five backward
        return dict(bytes=2.0 * D * (4 * tq * h + 4 * tk * hk) + 4.0 * tq * h, flops=14.0 * D * h * pairs)
    if kind == "linear":
        t, a, b = case["tokens"], case["n_in"], case["n_out"]
        return dict(bytes=2.0 * (2 * t * a + 2 * t * b + a * b) + 8.0 * a * b, flops=6.0 * t * a * b)
    if kind == "head":
        t, h, v = case["tokens"], case["hidden"], case["vocab"]
        # x, w, labels read; dlogits, dx, loss written; the fp32 weight gradient read and written
        return dict(bytes=2.0 * (2 * t * h + h * v + t * v) + 8.0 * h * v + 16.0 * t, flops=6.0 * t * h * v)
    t, h, f, e, k = case["tokens"], case["hidden"], case["ffn"], case["experts"], case["top_k"]
    return dict(bytes=8.0 * t * h + (2.0 + 8.0) * 3 * e * h * f, flops=18.0 * t * k * h * f)


def tolerance(case):
    """About four times what the library composition of the same ops (cuBLAS, flash-attn 2, PyTorch elementwise ops; same
    precision, other sums and other roundings between ops) was seen to differ by on the listed cases:
    train 0.006 to 0.019 (second moments; gradients 0.006 to 0.016), single elements up to 0.7; attention 0.0031, single
    elements up to 0.10; moe 0.0026 and 0.021; head 0.0017 and 0.0078; linear: bf16 results equal in the library's order of
    sums, another order moves a few percent of them by one bf16 step (0.0078 of the value)."""
    return {"train": {"rel": 0.03, "max": 0.99},
            "attention": {"rel": 0.012, "max": 0.4},
            "linear": {"rel": 0.003, "max": 0.016},
            "head": {"rel": 0.007, "max": 0.03},
            "moe": {"rel": 0.01, "max": 0.08}}[case["kind"]]


# --------------------------------------------------------------------------- the same in 64 bits
def _exact_attention(case, s):
    """Sequence by sequence, KV head by KV head, 1024 queries at a time."""
    ql, kl = _lengths(case)
    h, hk, causal = case["heads"], case["kv_heads"], case["causal"]
    g, scale = h // hk, 1.0 / math.sqrt(D)
    f = dict(dtype=torch.float64, device=DEV)
    out, dq = torch.zeros(sum(ql), h, D, **f), torch.zeros(sum(ql), h, D, **f)
    dk, dv = torch.zeros(sum(kl), hk, D, **f), torch.zeros(sum(kl), hk, D, **f)
    lse = torch.full((len(ql), h, max(ql)), float("-inf"), **f)
    q0 = k0 = 0
    for i, (nq, nk) in enumerate(zip(ql, kl)):
        for c in range(hk):
            k, v = s["k"][k0:k0 + nk, c].double(), s["v"][k0:k0 + nk, c].double()
            for a in range(0, nq, 1024):
                n = min(1024, nq - a)
                rows, hs = slice(q0 + a, q0 + a + n), slice(c * g, (c + 1) * g)
                q = s["q"][rows, hs].double().transpose(0, 1).reshape(g * n, D)
                do = s["dout"][rows, hs].double().transpose(0, 1).reshape(g * n, D)
                p = q @ k.t() * scale
                if causal:
                    last = torch.arange(a, a + n, device=DEV).repeat(g)[:, None] + (nk - nq)
                    p.masked_fill_(torch.arange(nk, device=DEV)[None] > last, float("-inf"))
                l = torch.logsumexp(p, dim=1, keepdim=True)
                p = torch.exp(p - l)
                o = p @ v
                ds = p * (do @ v.t() - (do * o).sum(1, keepdim=True)) * scale
                out[rows, hs] = o.view(g, n, D).transpose(0, 1)
                dq[rows, hs] = (ds @ k).view(g, n, D).transpose(0, 1)
                dk[k0:k0 + nk, c] += ds.t() @ q
                dv[k0:k0 + nk, c] += p.t() @ do
                lse[i, hs, a:a + n] = l.view(g, n)
        q0, k0 = q0 + nq, k0 + nk
    return dict(out=out, lse=None if min(ql) < max(ql) else lse, dq=dq, dk=dk, dv=dv)


def _exact_head(case, s):
    """512 tokens at a time; the loss with label smoothing as ``dhellam_b200/ops/loss.py`` states it."""
    t, v = case["tokens"], case["vocab"]
    smooth = case["label_smoothing"] * v / (v - 1)
    w = s["w"].double()
    loss, dlogits, dx, dw = [], [], [], torch.zeros_like(w)
    for a in range(0, t, 512):
        x, labels = s["x"][a:a + 512].double(), s["labels"][a:a + 512, None]
        logits = x @ w.t()
        lse = torch.logsumexp(logits, dim=1, keepdim=True)
        loss.append(((1 - smooth) * (lse - logits.gather(1, labels)) - smooth * (logits.mean(1, keepdim=True) - lse)).squeeze(1))
        d = torch.exp(logits - lse) - smooth / v
        d.scatter_add_(1, labels, torch.full_like(d[:, :1], smooth - 1))
        d *= s["dloss"][a:a + 512, None].double()
        dlogits.append(d.float())
        dx.append(d @ w)
        dw += d.t() @ x
    return dict(loss=torch.cat(loss), dlogits=torch.cat(dlogits), dx=torch.cat(dx), dw=dw)


def exact(case, seed):
    """No value for a training step (every layer rounds to bf16 what the next one reads) nor for the experts (tokens whose
    routes are nearly tied go elsewhere in 64 bits)."""
    if case["kind"] not in ("attention", "linear", "head"):
        return None
    s = prepare(case, seed)
    if case["kind"] == "attention":
        return _exact_attention(case, s)
    if case["kind"] == "head":
        return _exact_head(case, s)
    x, w, dy = s["x"].double(), s["w"].double(), s["dy"].double()
    return dict(y=x @ w.t(), dx=dy @ w, dw=dy.t() @ x)
