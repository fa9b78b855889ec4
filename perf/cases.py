"""The decode workloads whose speed this repository looks after, from the smallest calls to the largest.

A case is one pass a serving program makes: one decode step of a model at some context (one sequence or a batch), a
short prompt fed and continued greedily, the host-buffer token loop, or one stand-alone GEMV.  Models have the shapes of
the bundled configurations with fewer layers (every layer of a model does the same work, so a few stand for all), random
weights and a random-filled KV cache of the values a prefill leaves.

Weights: linear layers ~ N(0, 0.02) as the random-init configurations; so that a deep stack behaves like a trained model
(the residual stream large against one layer's update, a peaked router, a clear next token) the embedding has unit
variance, the matrices that write to the residual stream are scaled by 0.1, the router by 3, and the row of the lm_head
for a token is the embedding of the token before it.
"""
import math
import random

import numpy as np
import torch

import etx_megakernel_b200  # noqa: F401
from etx_megakernel_b200 import ops
from etx_megakernel_b200.frontends import cuda_link
from etx_megakernel_b200.importer import argblock
from etx_megakernel_b200.ir import Graph
from etx_megakernel_b200.machine import load_machine
from etx_megakernel_b200.models import batched as BT
from etx_megakernel_b200.models import decode as D
from etx_megakernel_b200.models import dsv2 as M
from etx_megakernel_b200.models import qwen as Q
from etx_megakernel_b200.passes import compile_graph
from etx_megakernel_b200.runtime import Session, op_launch

DEV = 0


def listed():
    return [
        # the headline: one sequence of a mixture-of-experts model, one token at a context of about a thousand positions
        {"name": "moe-1seq-ctx1k", "kind": "step", "model": "qwen3-30b-a3b", "layers": 12, "ctx": 1037},
        # the same model deep into a long conversation: the attention phase reads 17 MB per layer
        {"name": "moe-1seq-ctx8k", "kind": "step", "model": "qwen3-30b-a3b", "layers": 6, "ctx": 8150},
        # a dense model: two thirds of the step are long weight rows
        {"name": "dense-1seq-ctx1k", "kind": "step", "model": "qwen3-8b", "layers": 12, "ctx": 1031},
        # a small dense model with biases, tied embeddings, 6 query heads per kv head and a hidden size that is no power of two
        {"name": "small-dense-1seq-ctx600", "kind": "step", "model": "dense-1536", "layers": 10, "ctx": 601},
        # latent attention and shared experts
        {"name": "mla-1seq-ctx1k", "kind": "step", "model": "deepseek-v2-lite", "layers": 9, "ctx": 1043},
        # batches: the two sizes of the benchmark and a ragged one at a short context
        {"name": "moe-8seq-ctx1k", "kind": "batch", "batch": 8, "layers": 8, "ctx": 1033},
        {"name": "moe-32seq-ctx1k", "kind": "batch", "batch": 32, "layers": 6, "ctx": 1045},
        {"name": "moe-13seq-ctx333", "kind": "batch", "batch": 13, "layers": 6, "ctx": 333},
        # a request from its first token: a short prompt fed token by token, then greedy tokens, through generate()
        {"name": "moe-request-19+8", "kind": "request", "model": "qwen3-30b-a3b", "layers": 4, "prompt": 19, "new": 8},
        # the host-buffer token loop of a tiny model: launch and hand-off latency, no bytes to speak of
        {"name": "tiny-host-loop-12", "kind": "host", "H": 512, "NH": 8, "NKV": 2, "E": 16, "TOPK": 4, "MI": 128, "V": 1024, "layers": 2, "tokens": 12},
        # the stand-alone GEMV sweep: one token (one-grid plan) and eight tokens (column-batched kernel)
        {"name": "gemv-1x4096x12288", "kind": "gemv", "M": 1, "K": 4096, "N": 12288},
        {"name": "gemv-8x4096x12288", "kind": "gemv", "M": 8, "K": 4096, "N": 12288},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "batch", "batch", "request", "host", "gemv"])
    if kind == "step":
        model = rng.choice(["qwen3-30b-a3b", "qwen3-8b", "dense-1536", "deepseek-v2-lite"])
        top = {"qwen3-30b-a3b": 8190, "qwen3-8b": 8190, "dense-1536": 8190, "deepseek-v2-lite": 4090}[model]
        return {"kind": "step", "model": model, "layers": rng.randint(2, 7), "ctx": _log_int(rng, 5, top)}
    if kind == "batch":
        return {"kind": "batch", "batch": _log_int(rng, 2, 64), "layers": rng.randint(2, 3), "ctx": _log_int(rng, 20, 1500)}
    if kind == "request":
        c = {"kind": "request", "model": rng.choice(["qwen3-30b-a3b", "qwen3-8b", "dense-1536"]), "layers": rng.randint(2, 3),
             "prompt": _log_int(rng, 3, 60), "new": rng.randint(2, 20)}
        while work(c)["bytes"] > 26e9:                                  # no longer than the listed request
            c["prompt"], c["new"] = max(3, c["prompt"] * 2 // 3), max(2, c["new"] * 2 // 3)
        return c
    if kind == "host":
        nkv = rng.choice([1, 2, 4])
        E = rng.choice([8, 16, 24, 32, 64])
        return {"kind": "host", "H": 64 * rng.randint(4, 16), "NH": nkv * rng.choice([1, 2, 4, 8]), "NKV": nkv, "E": E, "TOPK": rng.choice([2, 4, 8]),
                "MI": 64 * rng.randint(1, 6), "V": 8 * rng.randint(64, 1000), "layers": rng.randint(2, 4), "tokens": rng.randint(3, 24)}
    Mt = rng.choice([1, 1, 2, 4, 8])
    K = 8 * _log_int(rng, 32, 1536 if Mt < 8 else 1200)
    return {"kind": "gemv", "M": Mt, "K": K, "N": min(_log_int(rng, 64, 151936), 620_000_000 // K)}


# ------------------------------------------------------------------------------------------------ shapes
# 28 layers of this shape make a 1.5-billion-parameter dense model with attention biases and tied embeddings
DENSE_1536 = {"hidden_size": 1536, "intermediate_size": 8960, "num_attention_heads": 12, "num_key_value_heads": 2, "num_hidden_layers": 28,
              "vocab_size": 151936, "rms_norm_eps": 1e-06, "rope_theta": 1000000.0, "tie_word_embeddings": True, "model_type": "qwen2"}


def _dims(case):
    kind = case["kind"]
    if kind == "host":
        return Q.Dims(name="tiny", H=case["H"], NH=case["NH"], NKV=case["NKV"], HD=128, INTER=0, L=case["layers"], V=case["V"], qk_norm=True, moe=True,
                      E=case["E"], TOPK=case["TOPK"], MI=case["MI"], norm_topk=True)
    model = case.get("model", "qwen3-30b-a3b")
    if model == "deepseek-v2-lite":
        return M.load_dims(model, layers=case["layers"])
    return Q.load_dims(DENSE_1536 if model == "dense-1536" else model, layers=case["layers"], name=model)


def _positions(case):
    """Positions a pass touches: the cache and the tables are sized for them."""
    kind = case["kind"]
    n = case["ctx"] + 1 if kind in ("step", "batch") else case["prompt"] + case["new"] if kind == "request" else case["tokens"] + 1
    return -(-(n + 2) // 16) * 16


def _like_trained(w):
    emb = w["embed"]
    emb.mul_(50.0)
    for name, t in w.items():
        leaf = name.rsplit(".", 1)[-1]
        if leaf in ("wo", "w2", "wd"):
            t.mul_(0.1)
        elif leaf == "wr":
            t.mul_(3.0)
    if "lm_head" in w:
        torch.mul(torch.roll(emb, 1, 0), 0.02, out=w["lm_head"])
    return w


# ------------------------------------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    dev = torch.device("cuda", DEV)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    ids = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "gemv":
        return _prepare_gemv(case, dev, gen)
    d, maxlen = _dims(case), _positions(case)
    if isinstance(d, M.MlaDims):
        prog = M.MlaProgram(d, _like_trained(M.random_weights(d, maxlen, dev, seed=seed)), device=DEV, maxlen=maxlen)
        prog.buf["ckv"].normal_(0.0, 1.0, generator=gen)               # normed latents and rotated keys have unit variance
    else:
        w = _like_trained(D.random_packed_weights(d, maxlen, dev, seed=seed))
        prog = BT.BatchProgram(d, w, case["batch"], device=DEV, maxlen=maxlen, steps=8) if kind == "batch" else D.DecodeProgram(d, w, device=DEV, maxlen=maxlen)
        if kind in ("step", "batch"):
            prog.buf["kc"].normal_(0.0, 1.0, generator=gen)             # (k rows are normed, v rows are W x of a normed x)
            prog.buf["vc"].normal_(0.0, 0.9, generator=gen)
    if kind in ("step", "batch"):
        tok = prog.buf["token_in"]
        tok[0] = torch.from_numpy(np.atleast_1d(ids.integers(0, d.V, tok[0].shape)).astype(np.int32)).to(dev).view(tok[0].shape)
    return {"case": dict(case), "prog": prog, "prompt": ids.integers(0, d.V, case.get("prompt", 1)).astype(np.int32)}


def _prepare_gemv(case, dev, gen):
    Mt, K, N = case["M"], case["K"], case["N"]
    W = torch.empty((N, K), dtype=torch.bfloat16, device=dev).normal_(0.0, 0.02, generator=gen)
    x = torch.empty((Mt, K), dtype=torch.bfloat16, device=dev).normal_(0.0, 1.0, generator=gen)
    out = torch.zeros((Mt, N), dtype=torch.bfloat16, device=dev)
    m = load_machine("b200")
    tasks, rpt = m.gemv_tasks(N, waves=4 if N > 65536 else 1)          # the split of the repository's own sweep
    blob = argblock.pack_named(ops.all_entries()["dsl_gemv"], (tasks, 1, 1), W=W.data_ptr(), x=x.data_ptr(), out=out.data_ptr(), M=N, K=K, rpt=rpt,
                               tpe=1, nb=Mt, sx=K, sout=N)
    session = None
    if Mt == 1:
        g = Graph(f"gemv_{K}x{N}")
        g.tensor("impargs", (len(blob),), role="weight", bytes_per_elem=1)
        g.etensor("E_done", (1,), wait_count=tasks)
        g.call_device("gemv", (tasks,), cuda_link("", "etx_tile_dsl_gemv", stream_after=""), args=["impargs"], consts=(0,), out_edges={"E_done": "i->(0)"})
        session = Session(compile_graph(g, m, {}), {}, blob, DEV)
    return {"case": dict(case), "session": session, "blob": blob, "tasks": tasks, "W": W, "x": x, "out": out}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "gemv":
        if state["session"] is not None:
            state["session"].launch()
        else:
            op_launch("gemv", state["blob"], state["tasks"])
        return {"out": state["out"]}
    prog = state["prog"]
    tokens = None
    if kind in ("step", "batch"):
        prog.step(0, case["ctx"], write_next=False, wait=False)         # steps are queued back to back, as the token loop does
    elif kind == "request":
        tokens = prog.generate(state["prompt"], case["new"])
    else:
        tokens, _ = prog.generate_host(state["prompt"], case["tokens"])
    out = {"logits": prog.buf["logits"]}
    out.update({"ckv": prog.buf["ckv"]} if "ckv" in prog.buf else {"kc": prog.buf["kc"], "vc": prog.buf["vc"]})
    if tokens is not None:
        out["tokens"] = tokens
    return out


# ------------------------------------------------------------------------------------------------ work / tolerance
def _layer_bytes(d, B):
    """Weight bytes one step of B sequences reads per layer: each dense matrix once, each expert some sequence selects once
    (expected number under uniform routing)."""
    if isinstance(d, M.MlaDims):
        raise TypeError("latent-attention models have their own ledger")
    attn = 2 * d.H * (d.NQKV + d.NH * d.HD)
    if not d.moe:
        return attn + 2 * 3 * d.INTER * d.H
    experts = d.E * (1.0 - (1.0 - d.TOPK / d.E) ** B)
    return attn + 2 * d.E * d.H + experts * 2 * 3 * d.MI * d.H


def work(case):
    kind = case["kind"]
    if kind == "gemv":
        Mt, K, N = case["M"], case["K"], case["N"]
        return {"bytes": 2 * (N * K + Mt * K + Mt * N), "flops": 2.0 * Mt * N * K}
    d = _dims(case)
    if isinstance(d, M.MlaDims):
        b = M.step_bytes(d, case["ctx"])["total"]
        return {"bytes": b, "flops": float(b)}
    B = case.get("batch", 1)
    if kind in ("step", "batch"):
        steps, ctx = 1, case["ctx"]
    else:
        steps = case["prompt"] + case["new"] - 1 if kind == "request" else case["tokens"]
        ctx = steps / 2
    kv = 2 * 2 * d.NKV * d.HD * (ctx + 1) * B
    per_token = d.L * (2 * d.H * (d.NQKV + d.NH * d.HD) + (2 * 3 * d.H * (d.MI * d.TOPK if d.moe else d.INTER))) + 2 * d.V * d.H
    return {"bytes": steps * (d.L * (_layer_bytes(d, B) + kv) + 2 * d.V * d.H + 2 * B * (d.H + d.V)),
            "flops": float(steps * B * (per_token + d.L * 4 * d.NH * d.HD * ctx))}


def tolerance(case):
    # bf16 results of fp32 sums.  A GEMV compared with fp64 sums: 1.7e-3, the rounding of the result itself; two correct ones
    # round a few results in a thousand to neighbouring values.  Steps with the sums of the attention phase, or of every
    # matrix of a batch, in another order: 2e-3 .. 4e-3 after the layers of a case, up to 9e-3 for the dense models, whose
    # wide MLP passes a change of a rounding on more strongly.
    if case["kind"] == "gemv":
        return {"rel": 1e-3, "max": 0.01}
    dense = case.get("model") in ("qwen3-8b", "dense-1536")
    return {"rel": 0.03 if dense else 0.012, "max": 0.15 if dense else 0.12}
