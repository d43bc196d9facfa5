"""The work that this framework is used for, as cases that can be timed and compared.

A case is one pass of a user's program through the public entry points on one GPU: a training step of a sharded
dense decoder or of a sharded mixture-of-experts decoder (forward, backward, optimizer), an evaluation pass, forward
and backward of a block's projections whose weights travel and multiply in FP8, or a Muon optimizer step. The listed cases take the repository's own configurations (the benchmark's and the examples'
widths, with fewer layers so that several states fit one card) and generic sizes between them; ``draw`` spreads over
the same ranges.
"""
from __future__ import annotations

import math

import torch

from flex_shard_b200 import BucketSpec, MixedPrecisionPolicy, flex_shard, relayout_bucket
from flex_shard_b200.dist_muon import build_local_dist_muon
from flex_shard_b200.models.deepseek_v3 import DeepSeekV3, DeepSeekV3Config, deepseek_buckets
from flex_shard_b200.models.llama import Llama, LlamaConfig, llama_buckets
from flex_shard_b200.ops import attention
from flex_shard_b200.ops.gemm import linear
from flex_shard_b200.optim.adamw import FusedAdamW
from flex_shard_b200.placements import (Shard, make_bucketed_owned_full_param_placement_fn,
                                        make_fp8_bucketed_block_shard_placement_fn,
                                        make_mxfp8_bucketed_block_shard_placement_fn)
from flex_shard_b200.placements.mixed_bucket import make_mixed_placement_fn
from flex_shard_b200.utils.training import clip_grad_norm_

GPU = torch.device("cuda")
HEAD = 128                                   # head width of the dense decoder
MLA = {"full": (128, 64, 128), "half": (64, 32, 64)}   # latent attention: no-position, rotary and value widths of a head


# --------------------------------------------------------------------------- the cases
def dense(name, **kw):
    """A dense decoder. ``ordered``: bitwise reproducible attention backward."""
    case = dict(kind="dense", heads=32, kv_heads=8, ffn=14336, vocab=128256, layers=1, batch=1, seq=8192, ordered=False)
    case.update(kw)
    return dict(case, name=name) if name else case


def projections(name, **kw):
    """The four projections of a decoder block, each with an input of its own, whose weights are gathered and multiplied
    as FP8 128x128 blocks or MXFP8. (Not a chain of them: a quantiser turns the last bit of its input into a step of its
    coarse grid, so the outputs of a whole quantised model say little about whether a part of it is right.)"""
    case = dict(kind="projections", heads=32, kv_heads=8, ffn=14336, batch=1, seq=8192, gather="fp8")
    case.update(kw)
    return dict(case, name=name) if name else case


def moe(name, **kw):
    """A mixture-of-experts decoder with latent attention: one dense block, then ``layers - 1`` expert blocks.
    ``recompute``: activation checkpointing per block; ``documents``: packed documents of about that many tokens
    (0: one document per row); ``balance``: the router's balance loss."""
    case = dict(kind="moe", width=2048, heads=16, q_rank=1536, kv_rank=512, mla="full", dense_ffn=10944, experts=64,
                expert_ffn=1408, top_k=6, vocab=102400, layers=2, batch=2, seq=4096, recompute=True, documents=0,
                balance=False)
    case.update(kw)
    return dict(case, name=name) if name else case


SMALL_MOE = dict(width=256, heads=2, q_rank=128, kv_rank=64, mla="half", dense_ffn=512, experts=8, expert_ffn=128,
                 top_k=2, vocab=2048)


def listed():
    return [
        # the smallest training job (the smoke step's sizes): launches and host work decide
        dense("dense_step_tiny", heads=4, kv_heads=2, ffn=1024, vocab=4096, layers=2, batch=2, seq=256),
        # an ordinary experiment: a billion-parameter width, an odd batch of rows that are no power of two
        dense("dense_step_mid", heads=16, kv_heads=4, ffn=5632, vocab=32000, layers=3, batch=3, seq=1152),
        # the benchmark's widths, vocabulary and sequence length, three of its layers: the largest step
        dense("dense_step_8b", layers=3),
        # the same widths with reproducible gradients asked for, shorter rows
        dense("dense_step_ordered", layers=2, seq=3072, vocab=32000, ordered=True),
        # the benchmark's quantised configuration: weights gathered as FP8 128x128 blocks
        projections("projections_fp8"),
        # the same widths in MXFP8, an odd batch of shorter rows
        projections("projections_mxfp8", batch=3, seq=1920, gather="mxfp8"),
        # evaluation between training steps: forward only, an odd batch of short rows
        dict(dense("dense_eval", layers=4, seq=640, batch=5), kind="eval"),
        # the expert example's smoke sizes
        moe("moe_step_small", **SMALL_MOE, layers=2, batch=2, seq=512, recompute=False),
        # the expert example's widths and batch: its defaults recompute every block
        moe("moe_step_16b"),
        # packed documents with the balance loss, activations kept, a row length that no tile divides
        moe("moe_step_documents", batch=1, seq=3000, documents=700, balance=True, recompute=False),
        # a Muon step of whole matrices (one decoder layer of the benchmark's Muon configuration)
        dict(dense("muon_step_dense", layers=1, vocab=32000), kind="muon_dense"),
        # a Muon step of many small matrices: attention heads and experts
        dict(moe("muon_step_moe", layers=2, vocab=32000), kind="muon_moe"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _multiple(x, m, least=1):
    return max(least, round(x / m)) * m


def _draw_block(rng):
    heads = rng.choice([4, 6, 8, 12, 16, 20, 24, 32])
    groups = [g for g in (1, 2, 4, 8) if heads % g == 0]
    seq = _multiple(_log(rng, 128, 8192), 128)
    return dict(heads=heads, kv_heads=heads // rng.choice(groups), ffn=_multiple(heads * HEAD * rng.uniform(2.0, 4.0), 128),
                batch=max(1, min(rng.choice([1, 1, 2, 3, 5]), 8192 // seq)), seq=seq)


def _draw_dense(rng, **kw):
    return dense(None, **_draw_block(rng), vocab=_multiple(_log(rng, 4096, 128256), 8), layers=rng.choice([1, 2, 3]), **kw)


def _draw_moe(rng, **kw):
    if rng.random() < 0.25:
        sizes = dict(SMALL_MOE, experts=rng.choice([4, 8, 12]), expert_ffn=_multiple(rng.uniform(96, 512), 8),
                     top_k=rng.choice([1, 2, 3]), vocab=_multiple(_log(rng, 1024, 8192), 8))
    else:
        width = rng.choice([1024, 1536, 2048])
        sizes = dict(width=width, heads=width // 128, q_rank=_multiple(width * 0.75, 64), kv_rank=rng.choice([256, 512]),
                     mla="full", dense_ffn=_multiple(width * rng.uniform(3.0, 5.3), 16), experts=rng.choice([16, 24, 48, 64]),
                     expert_ffn=_multiple(rng.uniform(512, 1408), 8), top_k=rng.choice([2, 4, 6, 8]),
                     vocab=_multiple(_log(rng, 8192, 102400), 8))
    seq = _multiple(_log(rng, 200, 4096), 8)
    batch = max(1, min(rng.choice([1, 2, 3]), 8192 // seq))
    documents = rng.choice([0, 0, int(_log(rng, 64, 2048))])
    return moe(None, **sizes, batch=batch, seq=seq, recompute=rng.random() < 0.5, documents=documents,
               balance=rng.random() < 0.3, **kw)


def draw(rng):
    kind = rng.choice(["dense", "dense", "projections", "ordered", "eval", "moe", "moe", "muon_dense", "muon_moe"])
    if kind == "projections":
        return projections(None, **_draw_block(rng), gather=rng.choice(["fp8", "mxfp8"]))
    if kind == "ordered":
        return _draw_dense(rng, ordered=True)
    if kind in ("dense", "eval", "muon_dense"):
        return dict(_draw_dense(rng), kind=kind)
    return dict(_draw_moe(rng), kind=kind)


# --------------------------------------------------------------------------- what a user's program has in hand
def _generator(seed):
    return torch.Generator(device=GPU).manual_seed(seed)


@torch.no_grad()
def _init(model, layers, g):
    """Random weights of a model at work: token embeddings that outweigh what a block adds to them (the projections
    back into the residual stream shrink with depth), so that tokens stay distinct from layer to layer."""
    for n, p in model.named_parameters():
        if n.endswith("norm"):
            p.fill_(1.0).add_(torch.randn(p.shape, generator=g, device=GPU) * 0.02)
        elif n.startswith("tok_embeddings"):
            p.normal_(0.0, 1.0, generator=g)
        else:
            p.normal_(0.0, 1.0 / math.sqrt(p.shape[-1] * (2 * layers if n.endswith(("wo", "w2")) else 1)), generator=g)


@torch.no_grad()
def _specialise_router(model, case, g):
    """Gives the tokens of a fresh model the decided routing of a trained one, where the experts a token goes to
    depend mostly on which token it is: every vocabulary entry leans towards ``top_k`` experts of its own, some
    experts being more popular than others."""
    E, k, V, D = case["experts"], case["top_k"], case["vocab"], case["width"]
    lean = torch.linalg.qr(torch.randn(D, E, generator=g, device=GPU))[0].t().contiguous()      # [E, D]
    popular = 1.0 + torch.rand(E, generator=g, device=GPU)
    score = torch.rand(V, E, generator=g, device=GPU).log() / popular
    chosen = torch.zeros(V, E, device=GPU).scatter_(1, score.topk(k, dim=1).indices, 1.0)
    chosen *= 0.4 * math.sqrt(D) * (1.0 + 0.7 * torch.rand(V, E, generator=g, device=GPU))
    model.tok_embeddings.weight.add_((chosen @ lean).to(model.tok_embeddings.weight.dtype))
    for m in model.moe_layers():
        m.gate.copy_(7.0 / math.sqrt(D) * lean + 0.1 / D * torch.randn(E, D, generator=g, device=GPU))


class Projections(torch.nn.Module):
    def __init__(self, shapes):
        super().__init__()
        for i, (rows, cols) in enumerate(shapes):
            self.register_parameter(f"w{i}", torch.nn.Parameter(torch.empty(rows, cols, dtype=torch.bfloat16, device=GPU)))

    def forward(self, *inputs):
        return tuple(linear(x, w) for x, w in zip(inputs, self._parameters.values()))


def _dense_model(case, g):
    cfg = LlamaConfig(vocab_size=case["vocab"], d_model=case["heads"] * HEAD, n_layers=case["layers"],
                      n_heads=case["heads"], n_kv_heads=case["kv_heads"], ffn_hidden=case["ffn"], max_seq_len=case["seq"])
    model = Llama(cfg, dtype=torch.bfloat16, device=GPU)
    _init(model, case["layers"], g)
    return model


def _moe_model(case, g):
    nope, rope, v = MLA[case["mla"]]
    cfg = DeepSeekV3Config(vocab_size=case["vocab"], d_model=case["width"], n_layers=case["layers"], n_heads=case["heads"],
                           q_lora_rank=case["q_rank"], kv_lora_rank=case["kv_rank"], qk_nope_dim=nope, qk_rope_dim=rope,
                           v_dim=v, dense_hidden=case["dense_ffn"], n_experts=case["experts"],
                           expert_hidden=case["expert_ffn"], top_k=case["top_k"], max_seq_len=case["seq"],
                           activation_checkpointing=case["recompute"], aux_loss_coeff=1e-3 if case["balance"] else 0.0)
    model = DeepSeekV3(cfg, dtype=torch.bfloat16, device=GPU)
    _init(model, case["layers"], g)
    _specialise_router(model, case, g)
    return model


def _positions(case, g):
    """Positions of tokens inside packed documents of uneven lengths (a document starts where the position is 0)."""
    B, S, length = case["batch"], case["seq"], case["documents"]
    starts = torch.rand(B, S, generator=g, device=GPU) < 1.0 / length
    starts[:, 0] = True
    at = torch.arange(S, device=GPU).expand(B, S)
    return at - torch.where(starts, at, torch.zeros_like(at)).cummax(dim=1).values


def _gradients(model, g):
    for p in model.parameters():
        p.grad = (torch.randn(p.shape, generator=g, device=GPU) * 1e-3).to(p.dtype)


def prepare(case, seed):
    g = _generator(seed)
    kind = case["kind"]
    state = {"case": case}
    if kind in ("dense", "eval"):
        model = _dense_model(case, g)
        for p in model.parameters():
            p.grad_dtype = torch.float32
        flex_shard(model, llama_buckets(model))
        if kind == "dense":
            opt = FusedAdamW(model.parameters(), lr=1e-4, betas=(0.9, 0.95), weight_decay=0.1)
            opt.fuse_into_backward(model)
            state["opt"] = opt
    elif kind == "projections":
        model = Projections(_dense_matrices(case))
        _init(model, 1, g)
        for p in model.parameters():
            p.grad_dtype = torch.float32
        place = (make_fp8_bucketed_block_shard_placement_fn() if case["gather"] == "fp8"
                 else make_mxfp8_bucketed_block_shard_placement_fn())
        mp = MixedPrecisionPolicy(param_dtype=torch.bfloat16, reduce_dtype=torch.float32)
        flex_shard(model, [BucketSpec(["w*"], mp_policy=mp, placement_fn=place)])
        T = case["batch"] * case["seq"]
        draw_rows = lambda cols: torch.randn(T, cols, generator=g, device=GPU).to(torch.bfloat16)  # noqa: E731
        state["inputs"] = [draw_rows(c).requires_grad_() for _, c in _dense_matrices(case)]
        state["output_gradients"] = [draw_rows(r) * 1e-3 for r, _ in _dense_matrices(case)]
    elif kind == "moe":
        model = _moe_model(case, g)
        flex_shard(model, deepseek_buckets(model))
        state["opt"] = FusedAdamW(model.parameters(), lr=1e-4, betas=(0.9, 0.95), weight_decay=0.1)
        state["positions"] = _positions(case, g) if case["documents"] else None
    elif kind == "muon_dense":
        model = _dense_model(case, g)
        owned = make_bucketed_owned_full_param_placement_fn(carry_loads=True)

        def layer_fn(named, mesh):
            out = dict(owned([(n, p) for n, p in named if p.dim() >= 2], mesh))
            out.update({n: Shard(0) for n, p in named if p.dim() < 2})
            return out

        mp = MixedPrecisionPolicy(param_dtype=torch.bfloat16, reduce_dtype=torch.float32)
        flex_shard(model, [BucketSpec(["tok_embeddings"], mp_policy=mp)]
                   + [BucketSpec([f"layers.{i}"], mp_policy=mp, placement_fn=make_mixed_placement_fn(layer_fn))
                      for i in range(case["layers"])]
                   + [BucketSpec(["head"], mp_policy=mp)])
        is_matrix = lambda n, p: n.startswith("layers.") and p.dim() >= 2  # noqa: E731
        state["muon"] = build_local_dist_muon(model, is_muon_param=is_matrix, lr=0.02, momentum=0.95, weight_decay=0.0)
        state["opt"] = FusedAdamW([p for n, p in model.named_parameters() if not is_matrix(n, p)], lr=3e-4,
                                  betas=(0.9, 0.95), weight_decay=0.1)
        _gradients(model, g)
    else:
        model = _moe_model(case, g)
        flex_shard(model, deepseek_buckets(model))
        owned = make_bucketed_owned_full_param_placement_fn(carry_loads=True)
        for st in list(model.sharded_bucket_storages):
            if st.name.startswith("layers.") and ".moe" not in st.name:
                relayout_bucket(model, st, owned)
        nope, rope, v = MLA[case["mla"]]
        is_matrix = lambda n, p: p.dim() >= 2 and not (  # noqa: E731
            n.startswith("tok_embeddings") or n == "output" or n.endswith(".gate"))
        state["muon"] = build_local_dist_muon(model, is_muon_param=is_matrix, lr=0.02, momentum=0.95, weight_decay=0.1,
                                              block_rows_by_fqn={"wq_b": nope + rope, "wkv_b": nope + v},
                                              adjust_lr_fn="match_rms_adamw")
        state["opt"] = FusedAdamW([p for n, p in model.named_parameters() if not is_matrix(n, p)], lr=3e-4,
                                  betas=(0.9, 0.95), weight_decay=0.1)
        _gradients(model, g)
    state["model"] = model
    if kind in ("dense", "eval", "moe"):
        state["tokens"] = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), generator=g, device=GPU)
    return state


# --------------------------------------------------------------------------- one pass
def run(state):
    case, model = state["case"], state["model"]
    kind = case["kind"]
    if kind == "eval":
        with torch.no_grad():
            return model(state["tokens"][:, :-1])
    if kind == "projections":
        for t in (*model.parameters(), *state["inputs"]):
            t.grad = None
        outs = model(*state["inputs"])
        torch.autograd.backward(outs, state["output_gradients"])
        return {"outputs": [y.detach() for y in outs], "input_gradients": [x.grad for x in state["inputs"]],
                "gradients": [p.grad for p in model.parameters()]}
    opt = state["opt"]
    if kind.startswith("muon"):
        muon = state["muon"]
        muon.step()
        opt.step()
        return {"weights": [p.detach() for p in model.parameters()],
                "momentum": [muon.state[p]["momentum_buffer"] for gr in muon.param_groups for p in gr["params"]]}
    tokens = state["tokens"]
    opt.zero_grad(set_to_none=True)
    if kind == "dense":
        if case["ordered"]:
            attention.set_deterministic(True)
        loss = model.loss(tokens[:, :-1], tokens[:, 1:])
        loss.backward()
        if case["ordered"]:
            attention.set_deterministic(None)
    else:
        loss = model.loss(tokens[:, :-1], tokens[:, 1:], loss_is_root=False, positions=state["positions"])
        loss.backward()
        clip_grad_norm_(model, 1.0)
        for m in model.moe_layers():
            m.update_expert_bias()
    opt.step()
    return {"loss": loss.detach(), "gradients": [p.grad for p in model.parameters()],
            "weights": [p.detach() for p in model.parameters()]}


# --------------------------------------------------------------------------- what a pass cannot do without
def _dense_matrices(case):
    d, f = case["heads"] * HEAD, case["ffn"]
    return [((case["heads"] + 2 * case["kv_heads"]) * HEAD, d), (d, d), (2 * f, d), (d, f)]


def _moe_matrices(case, expert_block):
    """(count, rows, columns, how many of them a token passes) of a block's matrices."""
    nope, rope, v = MLA[case["mla"]]
    d, H = case["width"], case["heads"]
    out = [(1, case["q_rank"], d, 1), (H, nope + rope, case["q_rank"], H), (1, case["kv_rank"] + rope, d, 1),
           (H, nope + v, case["kv_rank"], H), (1, d, H * v, 1)]
    if expert_block:
        e, E, k = case["expert_ffn"], case["experts"], case["top_k"]
        return out + [(E, 2 * e, d, k), (E, d, e, k), (1, 2 * e, d, 1), (1, d, e, 1)]
    return out + [(1, 2 * case["dense_ffn"], d, 1), (1, d, case["dense_ffn"], 1)]


def _polar_flops(n, rows, cols, steps=5):
    s, long = min(rows, cols), max(rows, cols)
    return n * steps * (3.0 * s * s * long + s ** 3)     # the two symmetric products counted by halves


def work(case):
    kind = case["kind"]
    T = case["batch"] * case["seq"]
    if kind == "projections":
        mats = _dense_matrices(case)
        return {"bytes": sum(r * c * (2 + 4) + 2.0 * T * 2 * (r + c) for r, c in mats),
                "flops": sum(6.0 * T * r * c for r, c in mats)}
    L, V = case["layers"], case["vocab"]
    if kind in ("dense", "eval", "muon_dense"):
        d = case["heads"] * HEAD
        mats = [(1, r, c, 1) for r, c in _dense_matrices(case)] * L
        attention_fwd = L * 2.0 * T * case["seq"] * d        # causal: half of the square, two products
    else:
        nope, rope, v = MLA[case["mla"]]
        d = case["width"]
        mats = _moe_matrices(case, False) + _moe_matrices(case, True) * (L - 1)
        span = min(case["seq"], case["documents"] or case["seq"])
        attention_fwd = L * 1.0 * T * span * case["heads"] * (nope + rope + v)
    params = sum(n * r * c for n, r, c, _ in mats) + 2.0 * V * d
    active = sum(used * r * c for _, r, c, used in mats)
    if kind.startswith("muon"):
        matrix_params = params - 2.0 * V * d
        return {"bytes": matrix_params * (2 + 2 + 2 + 8) + 2.0 * V * d * (2 + 2 + 2 + 16),
                "flops": sum(_polar_flops(n, r, c) for n, r, c, _ in mats)}
    if kind == "eval":
        return {"bytes": 2.0 * (params - V * d) + 2.0 * T * V, "flops": 2.0 * T * (active + V * d) + attention_fwd}
    grad = 4 if kind == "dense" else 2
    return {"bytes": params * (2 + 2 + grad + 16), "flops": 6.0 * T * (active + V * d) + 3.0 * attention_fwd}


def tolerance(case):
    """About four times what was measured between this path and the same model with the library's attention or the
    library's matrix products in place of the kernels here, over one and two passes: bf16 gradients through up to three
    blocks 0.010 (single elements 0.32), logits 0.005 (0.03), weights after Muon steps 0.007 (0.08). Quantised products
    sum exact 8-bit products in fp32 and round once: single bf16 roundings may fall the other way."""
    if case["kind"] == "projections":
        return {"rel": 0.004, "max": 0.03}
    if case["kind"] == "eval":
        return {"rel": 0.02, "max": 0.15}
    return {"rel": 0.03, "max": 0.3 if case["kind"].startswith("muon") else 0.95}
