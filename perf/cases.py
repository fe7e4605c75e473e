"""Performance cases: the work a user of this framework has it do on one GPU, through its public entry points.

Four kinds of case:

* ``step``: one optimizer step of a ``Trainer`` (``Trainer.train_step``: pinned copies of the micro-batches, forward, loss,
  manual backward, gradient norm, AdamW) on seeded synthetic tokens and random-init weights, bf16 with fp32 master weights.
* ``attention``: one direction of the causal GQA attention op of the op table, on the packed QKV activation; the backward
  is the one a training step calls, with the RoPE backward folded in.
* ``head``: final projection, fused cross-entropy and both of its backward products, the vocabulary width ragged or a shard.
* ``ffn``: the FFN half of a decoder layer, forward and backward, in bf16 or with block-scaled MXFP8 products.

``listed()`` holds twelve fixed cases, ``draw(rng)`` gives further ones from the same ranges.
"""
from __future__ import annotations

import math

import torch

import forge_train_harness_b200 as fth
from forge_train_harness_b200.ops import get_ops, rope_table
from forge_train_harness_b200.ops.mxfp8 import Mxfp8Ops

DEV = "cuda:0"
EPS = 1e-6


def _step(name, layers, hidden, ffn, heads, kv, head_dim, vocab, seq, mbs, accum, tied=True, mtp=0, qk_norm=False, fp8=False):
    return dict(name=name, kind="step", layers=layers, hidden=hidden, ffn=ffn, heads=heads, kv=kv, head_dim=head_dim, vocab=vocab,
                seq=seq, mbs=mbs, accum=accum, tied=tied, mtp=mtp, qk_norm=qk_norm, fp8=fp8)


def listed():
    return [
        # the tiny model of the tests and the CPU config: a step is a hundred small launches, so this is launch and host latency
        _step("step tiny", 2, 256, 1024, 4, 2, 64, 8192, 256, 2, 1),
        # short sequences (fine-tuning data, gate runs with cut layers) and rows that fill no whole tile: 3 x 640 tokens
        _step("step short sequences", 6, 1024, 4096, 16, 2, 64, 73448, 640, 3, 4),
        # the flagship pre-training step, with two micro-batches instead of the benchmark's sixteen
        _step("step 0.5b", 24, 1024, 4096, 16, 2, 64, 73448, 4096, 4, 2),
        # 1B with the MTP branch: untied tables, two losses, a large optimizer share at one micro-batch per step
        _step("step 1b mtp", 24, 1536, 4608, 16, 2, 128, 130560, 4096, 1, 1, tied=False, mtp=1),
        # the q/k-norm family: head_dim 128 with 8 KV heads and the widest vocabulary
        _step("step qwen3 0.6b", 28, 1024, 3072, 16, 8, 128, 151936, 4096, 2, 1, qk_norm=True),
        # the 8B width cut to two layers, block-scaled fp8 linears
        _step("step 8b width mxfp8", 2, 4096, 16384, 32, 2, 128, 73448, 4096, 1, 2, tied=False, fp8=True),
        # the flagship's attention, each direction
        dict(name="attention fwd d64 4x4096", kind="attention", backward=False, batch=4, seq=4096, heads=16, kv=2, head_dim=64),
        dict(name="attention bwd d64 4x4096", kind="attention", backward=True, batch=4, seq=4096, heads=16, kv=2, head_dim=64),
        # a small call: three short sequences, 384 is an odd number of 128-row tiles
        dict(name="attention fwd d128 3x384", kind="attention", backward=False, batch=3, seq=384, heads=16, kv=8, head_dim=128),
        # the 8B attention backward
        dict(name="attention bwd d128 1x4096", kind="attention", backward=True, batch=1, seq=4096, heads=32, kv=2, head_dim=128),
        # the LM head on one TP-4 vocabulary shard (18362 columns: not a multiple of 8) with an odd number of tokens
        dict(name="head shard 1500x18362", kind="head", tokens=1500, hidden=4096, vocab=18362),
        # an FFN on a ragged number of tokens at the 1B width
        dict(name="ffn 776x1536x4608", kind="ffn", tokens=776, hidden=1536, ffn=4608, fp8=False),
    ]


def _log_int(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / multiple)) * multiple))


def _draw_one(rng):
    kind = rng.choices(["step", "attention", "head", "ffn"], [40, 30, 15, 15])[0]
    if kind == "attention":
        d = rng.choice([64, 128])
        kv = rng.choice([1, 2, 4, 8])
        return dict(kind=kind, backward=rng.random() < 0.5, batch=rng.randint(1, 8), seq=_log_int(rng, 128, 4096, 128),
                    heads=kv * rng.choice([1, 2, 4, 8]), kv=kv, head_dim=d)
    if kind == "head":
        return dict(kind=kind, tokens=_log_int(rng, 64, 8192), hidden=_log_int(rng, 256, 4096, 8), vocab=_log_int(rng, 1000, 151936))
    if kind == "ffn":
        fp8 = rng.random() < 0.4
        m = 32 if fp8 else 8
        return dict(kind=kind, tokens=_log_int(rng, 64, 16384, m), hidden=_log_int(rng, 256, 4096, m), ffn=_log_int(rng, 512, 16384, m),
                    fp8=fp8)
    d = rng.choice([64, 128])
    hidden = _log_int(rng, 256, 2048, 64)
    kv = rng.choice([1, 2, 4, 8])
    group = max(1, min(16, hidden // d // kv))
    variant = rng.choice(["plain", "plain", "mtp", "qk_norm", "fp8"])
    seq = _log_int(rng, 128, 4096, 128)
    return dict(kind=kind, layers=rng.randint(1, 8), hidden=hidden, ffn=_log_int(rng, 512, 8192, 32), heads=kv * group, kv=kv,
                head_dim=d, vocab=_log_int(rng, 1000, 151936, 8), seq=seq, mbs=rng.randint(1, max(1, min(8, 16384 // seq))),
                accum=rng.randint(1, 4), tied=variant != "mtp" and rng.random() < 0.5, mtp=int(variant == "mtp"),
                qk_norm=variant == "qk_norm", fp8=variant == "fp8")


def _floor_s(case):
    w = work(case)
    return max(w["bytes"] / 6.4e12, w["flops"] / 1.4e15)


def draw(rng):
    limit = max(_floor_s(c) for c in listed())
    while True:
        c = _draw_one(rng)
        if _floor_s(c) <= limit:
            return c


# ---------------------------------------------------------------------------------------------------------------------

def _model(c):
    return fth.ModelConfig(name="case", num_layers=c["layers"], hidden_size=c["hidden"], ffn_hidden_size=c["ffn"],
                           num_attention_heads=c["heads"], num_query_groups=c["kv"], head_dim=c["head_dim"], seq_length=c["seq"],
                           padded_vocab_size=c["vocab"], norm_epsilon=EPS, init_method_std=0.02, tie_embeddings=c["tied"],
                           mtp_num_layers=c["mtp"], mtp_loss_weight=0.3 if c["mtp"] else 0.0, qk_norm=c["qk_norm"],
                           use_mup=not c["qk_norm"])


def _n_params(c):
    H, F, q, kv = c["hidden"], c["ffn"], c["heads"] * c["head_dim"], c["kv"] * c["head_dim"]
    layer = H * (q + 2 * kv) + q * H + 3 * F * H + 2 * H + (2 * c["head_dim"] if c["qk_norm"] else 0)
    return (c["layers"] + c["mtp"]) * layer + c["vocab"] * H * (1 if c["tied"] else 2) + H + c["mtp"] * (2 * H * H + 3 * H)


class _TrainState:
    """A running training job: the trainer after its first step (which captures the micro-batch graph)."""

    def __init__(self, case, seed):
        cfg = fth.RunConfig(
            model=_model(case),
            optim=fth.OptimConfig(lr=1e-3, min_lr=1e-4, lr_warmup_iters=2000, lr_decay_iters=100_000, lr_schedule="cosine",
                                  weight_decay=0.1, adam_beta1=0.9, adam_beta2=0.95, clip_grad=1.0),
            parallel=fth.ParallelConfig(fp8="mxfp8" if case["fp8"] else "off"),
            train=fth.TrainConfig(micro_batch_size=case["mbs"], grad_accum_steps=case["accum"], seed=seed % (1 << 30), dtype="bf16"),
            data=fth.DataConfig(data_loader="synthetic", synthetic_seed=seed % (1 << 30)))
        self.trainer = fth.Trainer(cfg, device=DEV, init_mode="device", quiet=True)
        self.trainer.train_step()

    def __del__(self):
        if hasattr(self, "trainer"):
            self.trainer.close()


def _randn(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float32).mul_(std).to(dtype)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        return dict(case=case, job=_TrainState(case, seed))
    gen = torch.Generator(device=DEV).manual_seed(seed)
    ops = get_ops(DEV)
    st = dict(case=case, ops=ops)
    if kind == "attention":
        g, d, S = case["heads"] // case["kv"], case["head_dim"], case["seq"]
        M = case["batch"] * S
        st["qkv"] = _randn(gen, M, case["kv"] * (g + 2) * d)
        st["geo"] = (S, case["kv"], g, d)
        if case["backward"]:
            st["dout"] = _randn(gen, M, case["heads"] * d, std=1e-2)
            st["out"], st["lse"] = ops.attention_fwd(st["qkv"], *st["geo"])
            st["table"] = rope_table(S, d, 10000.0, DEV)
    elif kind == "head":
        M, H, V = case["tokens"], case["hidden"], case["vocab"]
        st["x"], st["w"] = _randn(gen, M, H), _randn(gen, V, H, std=0.1)
        st["labels"] = torch.randint(0, V, (M,), generator=gen, device=DEV, dtype=torch.int32)
        st["mask"] = torch.ones(M, device=DEV)
        st["gw"] = torch.zeros(V, H, device=DEV)
        st["alpha"] = 256.0 / H
    else:
        M, H, F = case["tokens"], case["hidden"], case["ffn"]
        if case["fp8"]:
            st["ops"] = Mxfp8Ops(ops)
        st["h"], st["a"], st["g"] = _randn(gen, M, H), _randn(gen, M, H), _randn(gen, M, H, std=1e-2)
        st["wn"] = torch.ones(H, device=DEV, dtype=torch.bfloat16)
        st["w1"], st["w2"] = _randn(gen, 2 * F, H, std=0.02), _randn(gen, H, F, std=0.02)
        st["gwn"] = torch.zeros(H, device=DEV)
        st["gw1"], st["gw2"] = torch.zeros(2 * F, H, device=DEV), torch.zeros(H, F, device=DEV)
    return st


def run(st):
    kind = st["case"]["kind"]
    if kind == "step":
        tr = st["job"].trainer
        res = tr.train_step()
        return {"loss": res["loss"], "grad_norm": res["grad_norm"], "grad": tr.store.flat_grad, "param": tr.store.flat_param,
                "master": tr.opt.master, "exp_avg": tr.opt.m, "exp_avg_sq": tr.opt.v}
    ops = st["ops"]
    if kind == "attention":
        if not st["case"]["backward"]:
            return ops.attention_fwd(st["qkv"], *st["geo"])
        return ops.attention_rope_bwd(st["dout"], st["qkv"], st["out"], st["lse"], st["table"], *st["geo"])
    if kind == "head":
        st["gw"].zero_()
        logits = ops.linear_fwd(st["x"], st["w"], st["alpha"])
        nll = ops.cross_entropy_fwd_bwd(logits, st["labels"], st["mask"])
        ops.linear_wgrad(logits, st["x"], st["gw"], st["alpha"])
        return {"nll": nll, "dlogits": logits, "dx": ops.linear_dgrad(logits, st["w"], st["alpha"]), "dw": st["gw"]}
    ds = 0.25
    for k in ("gwn", "gw1", "gw2"):
        st[k].zero_()
    r, n, rstd = ops.residual_rmsnorm_fwd(st["h"], st["a"], ds, st["wn"], EPS)
    gu = ops.linear_fwd(n, st["w1"])
    inter = ops.swiglu_fwd(gu)
    m = ops.linear_fwd(inter, st["w2"])
    d_inter = ops.linear_dgrad(st["g"], st["w2"], ds)
    ops.linear_wgrad(st["g"], inter, st["gw2"], ds)
    d_gu = ops.swiglu_bwd(d_inter, gu)
    ops.linear_wgrad(d_gu, n, st["gw1"])
    d_n = ops.linear_dgrad(d_gu, st["w1"])
    dx = ops.rmsnorm_bwd(d_n, r, st["wn"], rstd, st["gwn"], st["g"])
    return {"m": m, "dx": dx, "dw_norm": st["gwn"], "dw1": st["gw1"], "dw2": st["gw2"]}


def work(case):
    kind = case["kind"]
    if kind == "step":
        tokens = case["mbs"] * case["seq"] * case["accum"]
        # weights 2 B and fp32 master / two moments 12 B read and written, the fp32 gradient written; ids, labels and mask read
        return {"bytes": 32.0 * _n_params(case) + 12.0 * tokens, "flops": _model(case).flops_per_token() * tokens}
    if kind == "attention":
        rows, nq, kv, d, S = case["batch"] * case["seq"], case["heads"], case["kv"], case["head_dim"], case["seq"]
        qkv, o, stat = 2.0 * rows * (nq + 2 * kv) * d, 2.0 * rows * nq * d, 4.0 * rows * nq
        pairs = case["batch"] * nq * S * (S + 1) / 2.0
        if case["backward"]:
            return {"bytes": 2 * qkv + 2 * o + stat + 4.0 * S * d, "flops": 10.0 * pairs * d}
        return {"bytes": qkv + o + stat, "flops": 4.0 * pairs * d}
    M, H = case["tokens"], case["hidden"]
    if kind == "head":
        V = case["vocab"]
        return {"bytes": 4.0 * M * H + 2.0 * M * V + 6.0 * V * H + 12.0 * M, "flops": 6.0 * M * V * H}
    F = case["ffn"]
    return {"bytes": 10.0 * M * H + 18.0 * F * H + 6.0 * H, "flops": 18.0 * M * F * H}


def tolerance(case):
    # bf16 results of long sums: 1e-2.  A step's gradient went through every layer in bf16 twice: the same step on the plain
    # PyTorch ops differs by 0.4e-2 to 1.6e-2 (28 layers), and single elements, sums of cancelling terms, by up to their own
    # size.  An MXFP8 product rounds to 3 mantissa bits: a last-bit difference of an activation moves such a rounding by up to
    # 2^-4 of the element, and the two-layer step then differs by 2.2e-2.
    if case.get("fp8"):
        return {"rel": 3e-2, "max": 0.9}
    if case["kind"] == "step":
        return {"rel": 2e-2, "max": 0.9}
    return {"rel": 1e-2}
