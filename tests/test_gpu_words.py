"""The one-token step's hand-off as words (bf16 value and step flag in 4 bytes) against the same step through bf16 vectors and events; the way the
consumer warps share a GEMV task's rows at the edges of its rules, against 64-bit sums; contexts that one task takes whole at the edge of the limit."""
import functools

import numpy as np
import pytest
import torch

from etx_megakernel_b200.models import decode as D
from etx_megakernel_b200.models import qwen as Q

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dims(H, moe, MI, NH=4, NKV=2, bias=False, L=2):
    return Q.Dims(name="words", H=H, NH=NH, NKV=NKV, HD=128, INTER=0 if moe else MI, L=L, V=1000, qk_norm=not bias, bias=bias, moe=moe,
                  E=16 if moe else 0, TOPK=4 if moe else 0, MI=MI if moe else 0, norm_topk=True)


def steps(d, w, maxlen, positions, full=False, **kw):
    """Logits and caches after single steps at `positions` over a random cache."""
    prog = D.DecodeProgram(d, w, device=0, maxlen=maxlen, **kw)
    if full:
        prog.session.set_option("full_kernel", 1)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(5)
    prog.buf["kc"].normal_(0, 1, generator=gen)
    prog.buf["vc"].normal_(0, 1, generator=gen)
    out = []
    for i, pos in enumerate(positions):
        prog.buf["token_in"][0] = 17 + i
        prog.step(0, pos, write_next=False)
        out.append({n: prog.read(n).copy() for n in ("logits", "attn_out", "resid", "moe_out")})
    out.append({"kc": prog.read("kc"), "vc": prog.read("vc")})
    prog.close()
    return out


@pytest.mark.parametrize("H,moe,MI,bias", [(512, True, 128, False), (1024, False, 1432, True), (2048, True, 96, False), (4096, False, 2056, False), (8192, False, 264, False)])
def test_words_give_the_bits_of_the_vectors(monkeypatch, H, moe, MI, bias):
    """Powers of two: the norm fold sums its squares in the same order either way, everything else is the same arithmetic.  Rows of 7, 8 and
    16 vectors a lane, down rows of one and of several slots, lean and full kernel."""
    d = dims(H, moe, MI, bias=bias)
    w = D.random_packed_weights(d, 300, DEV, seed=3)
    pos = [0, 1, 130, 290]
    got, full = steps(d, w, 300, pos), steps(d, w, 300, pos, full=True)
    monkeypatch.setattr(Q, "build_graph", functools.partial(lambda build, *a, **k: build(*a, **{**k, "words": False}), Q.build_graph))
    want = steps(d, w, 300, pos)
    for g, f, e in zip(got, full, want):
        for n in e:
            assert np.array_equal(g[n], e[n]), n
            assert np.array_equal(f[n], e[n]), n


def test_words_of_a_width_that_is_no_power_of_two(monkeypatch):
    """1096 values: eight and a half blocks of 128.  The squares are summed in another order than without words: 32-bit sums, so z and x differ by a
    rounding to bf16 here and there (2^-8 relative)."""
    d = dims(1096, False, 520, L=1)
    w = D.random_packed_weights(d, 64, DEV, seed=4)
    got = steps(d, w, 64, [0, 40])
    monkeypatch.setattr(Q, "build_graph", functools.partial(lambda build, *a, **k: build(*a, **{**k, "words": False}), Q.build_graph))
    want = steps(d, w, 64, [0, 40])
    for g, e in zip(got[:2], want[:2]):
        for n in e:
            assert np.linalg.norm(g[n] - e[n]) <= 2.0 ** -8 * np.linalg.norm(e[n]), n


@pytest.mark.parametrize("K", [64, 1024, 1096, 1536, 2880, 8184, 8192])
def test_the_norms_mean_to_fp32(K):
    """The norm fold of a grid that writes words, against 64-bit sums: a value of the normed vector may differ from the one rounded from 64 bits only where it
    lies within the fp32 roundings of the boundary between two.  Those of 1 / sqrt(mean + eps): a square, 15 + 3 + 6 sums, the mean and its eps, all
    halved by the root, then root, division and product: 17, so 20 units of 2^-24."""
    from etx_megakernel_b200 import ops
    from etx_megakernel_b200.frontends import cuda_link
    from etx_megakernel_b200.importer import argblock
    from etx_megakernel_b200.ir import Graph
    from etx_megakernel_b200.ops import gemv
    from etx_megakernel_b200.passes import compile_graph
    from etx_megakernel_b200.runtime import Session
    gen = torch.Generator(device=DEV)
    gen.manual_seed(K)
    z = torch.empty(K, dtype=torch.bfloat16, device=DEV).normal_(0, 1.5, generator=gen)
    ln, W = torch.ones(K, dtype=torch.bfloat16, device=DEV), torch.zeros((8, K), dtype=torch.bfloat16, device=DEV)
    x, out = torch.zeros_like(z), torch.zeros(8, dtype=torch.bfloat16, device=DEV)
    words = torch.zeros(K + 8, dtype=torch.int32, device=DEV)
    blob = gemv.words_block(argblock.pack_named(ops.all_entries()["dsl_gemv_fold"], (1, 1, 1), W=W.data_ptr(), x=x.data_ptr(), out=out.data_ptr(), M=8, K=K, rpt=8, tpe=1,
                                                rows=0, resid_in=z.data_ptr(), resid_out=0, ln=ln.data_ptr(), R=0, eps=1e-6, mode=gemv.MODE_NORM | gemv.MODE_WORDS_OUT, nb=1),
                            out=words.data_ptr() + 4 * K, x=words.data_ptr())
    g = Graph("norm")
    g.tensor("impargs", (len(blob),), role="weight", bytes_per_elem=1)
    g.etensor("E_done", (1,), wait_count=1)
    g.call_device("norm", (1,), cuda_link("", "etx_tile_dsl_gemv_fold", stream_after=""), args=["impargs"], consts=(0,), out_edges={"E_done": "i->(0)"})
    s = Session(compile_graph(g, "b200", {}), {}, blob, 0)
    s.run(5.0)
    s.close()
    v = z.double() / torch.sqrt((z.double() ** 2).mean() + float(np.float32(1e-6)))
    d = 20 * 2.0 ** -24
    lo, hi = ((v * (1 + t * torch.sign(v))).float().bfloat16().float() for t in (-d, d))
    lo, hi = torch.minimum(lo, hi), torch.maximum(lo, hi)
    assert bool(((x.float() >= lo) & (x.float() <= hi)).all())
    assert torch.equal(x.view(torch.int16).int() & 0xffff, words[:K] & 0xffff)


@pytest.mark.parametrize("K,N", [(8, 5), (264, 37), (1792, 900), (2048, 1), (2048, 2000), (2056, 300), (3072, 700), (4096, 1500), (6152, 777), (8960, 100), (12288, 640), (64, 310000)])
def test_rows_shared_by_the_warps(K, N):
    """One-grid plans: a few rows and many, rows of a lane's one vector to 48, several warps a row, more rows per task than the results' place holds.
    fp32 sums of K products: 1e-6 of the terms' size, then one rounding to bf16."""
    from etx_megakernel_b200 import ops
    from etx_megakernel_b200.frontends import cuda_link
    from etx_megakernel_b200.importer import argblock
    from etx_megakernel_b200.ir import Graph
    from etx_megakernel_b200.machine import load_machine
    from etx_megakernel_b200.passes import compile_graph
    from etx_megakernel_b200.runtime import Session
    gen = torch.Generator(device=DEV)
    gen.manual_seed(K + N)
    W = torch.empty((N, K), dtype=torch.bfloat16, device=DEV).normal_(0, 1, generator=gen)
    x = torch.empty((1, K), dtype=torch.bfloat16, device=DEV).normal_(0, 1, generator=gen)
    out = torch.zeros((1, N), dtype=torch.bfloat16, device=DEV)
    m = load_machine("b200")
    tasks, rpt = m.gemv_tasks(N)
    blob = argblock.pack_named(ops.all_entries()["dsl_gemv"], (tasks, 1, 1), W=W.data_ptr(), x=x.data_ptr(), out=out.data_ptr(), M=N, K=K, rpt=rpt, tpe=1, nb=1)
    g = Graph("rows")
    g.tensor("impargs", (len(blob),), role="weight", bytes_per_elem=1)
    g.etensor("E_done", (1,), wait_count=tasks)
    g.call_device("gemv", (tasks,), cuda_link("", "etx_tile_dsl_gemv", stream_after=""), args=["impargs"], consts=(0,), out_edges={"E_done": "i->(0)"})
    s = Session(compile_graph(g, m, {}), {}, blob, 0)
    for _ in range(2):
        out.zero_()
        torch.cuda.synchronize()
        s.run(5.0)
    s.close()
    want = (W.double() @ x[0].double()).cpu().numpy()
    got = out[0].double().cpu().numpy()
    assert np.all(np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-6 * np.sqrt(K))


@pytest.mark.parametrize("NH,NKV", [(4, 2), (3, 1)])
def test_contexts_taken_whole(monkeypatch, NH, NKV):
    """One layer at contexts around one, two and three partitions, with the limit and without: the same sums in another order, 2 bf16 ulps."""
    from etx_megakernel_b200.ops import attn
    d = dims(512, True, 128, NH=NH, NKV=NKV, L=1)
    w = D.random_packed_weights(d, 500, DEV, seed=6)
    pos = [0, 14, 127, 128, 143, 254, 255, 256, 383, 480]
    assert attn.GQ_LIM == 2
    got = steps(d, w, 500, pos)
    monkeypatch.setattr(attn, "GQ_LIM", 0)
    want = steps(d, w, 500, pos)
    for g, e in zip(got[:-1], want[:-1]):
        a, b = g["attn_out"], e["attn_out"]
        assert np.all(np.abs(a - b) <= 2 * np.maximum(np.abs(b) * 2.0 ** -7, np.abs(b).max() / 4096)) and np.mean(a == b) >= 0.9
    assert np.array_equal(got[-1]["kc"], want[-1]["kc"]) and np.array_equal(got[-1]["vc"], want[-1]["vc"])


def test_words_are_refused_where_nobody_flags_them():
    """A single-tile launch has no step, so a block that names words is refused before it reaches the device."""
    from etx_megakernel_b200 import ops
    from etx_megakernel_b200.importer import argblock
    from etx_megakernel_b200.ops import gemv
    from etx_megakernel_b200.runtime import op_launch
    from etx_megakernel_b200.runtime.lib import EtxbError
    t = torch.zeros(4096, dtype=torch.int32, device=DEV)
    blob = argblock.pack_named(ops.all_entries()["dsl_gemv"], (1, 1, 1), W=t.data_ptr(), x=t.data_ptr(), out=t.data_ptr(), M=4, K=64, rpt=4, tpe=1, nb=1,
                               mode=gemv.MODE_WORDS_IN | gemv.MODE_WORDS_OUT)
    with pytest.raises(EtxbError, match="words"):
        op_launch("gemv", gemv.words_block(blob, out=t.data_ptr()), 1)


def test_a_reader_of_vectors_behind_words_is_refused():
    """A grid that hands words over does not wait for its bf16 stores: a plan whose next grid reads the bf16 vector does not run."""
    from etx_megakernel_b200 import ops
    from etx_megakernel_b200.frontends import cuda_link
    from etx_megakernel_b200.importer import argblock
    from etx_megakernel_b200.ir import Graph
    from etx_megakernel_b200.ops import gemv
    from etx_megakernel_b200.passes import compile_graph
    from etx_megakernel_b200.runtime import Session
    from etx_megakernel_b200.runtime.lib import EtxbError
    W = torch.zeros((64, 64), dtype=torch.bfloat16, device=DEV)
    x, y, z = (torch.zeros(64, dtype=torch.bfloat16, device=DEV) for _ in range(3))
    words = torch.zeros(64, dtype=torch.int32, device=DEV)
    f = dict(W=W.data_ptr(), M=64, K=64, rpt=64, tpe=1, nb=1)
    first = gemv.words_block(argblock.pack_named(ops.all_entries()["dsl_gemv"], (1, 1, 1), x=x.data_ptr(), out=y.data_ptr(), mode=gemv.MODE_WORDS_OUT, **f), out=words.data_ptr())

    def session(second):
        g = Graph("readers")
        g.tensor("impargs", (len(first) + len(second),), role="weight", bytes_per_elem=1)
        g.etensor("E_a", (1,), wait_count=1)
        g.etensor("E_b", (1,), wait_count=1)
        g.call_device("a", (1,), cuda_link("", "etx_tile_dsl_gemv", stream_after=""), args=["impargs"], consts=(0,), out_edges={"E_a": "i->(0)"})
        g.call_device("b", (1,), cuda_link("", "etx_tile_dsl_gemv", stream_after=""), args=["impargs"], consts=(len(first),), in_edges={"E_a": "i->(0)"}, out_edges={"E_b": "i->(0)"})
        return Session(compile_graph(g, "b200", {}), {}, first + second, 0)
    ent = ops.all_entries()["dsl_gemv"]
    for at in (y, y[8:]):                                           # the vector, and a part of it
        s = session(argblock.pack_named(ent, (1, 1, 1), x=at.data_ptr(), out=z.data_ptr(), **{**f, "K": at.numel()}))
        with pytest.raises(EtxbError, match="words"):
            s.run(5.0)
        s.close()
    s = session(gemv.words_block(argblock.pack_named(ent, (1, 1, 1), x=words.data_ptr(), out=z.data_ptr(), mode=gemv.MODE_WORDS_IN, **f)))
    s.run(5.0)
    s.close()
    s = session(argblock.pack_named(ent, (1, 1, 1), x=x.data_ptr(), out=z.data_ptr(), **f))       # (another vector)
    s.run(5.0)
    s.close()


def test_latent_attention_words_give_the_bits_of_the_vectors(monkeypatch):
    """Two layers (dense, experts) of the latent-attention model; 11 partitions are two rounds of the finishing tasks."""
    from etx_megakernel_b200.models import dsv2 as M
    d = M.load_dims("deepseek-v2-lite", layers=2)
    w = M.random_weights(d, 1400, torch.device(DEV), seed=2)

    def run():
        prog = M.MlaProgram(d, w, device=0, maxlen=1400)
        gen = torch.Generator(device=DEV)
        gen.manual_seed(7)
        prog.buf["ckv"].normal_(0, 1, generator=gen)
        out = []
        for i, pos in enumerate([0, 127, 300, 1279, 1290]):
            prog.buf["token_in"][0] = 11 + i
            prog.step(0, pos, write_next=False)
            out += [prog.read(n).copy() for n in ("logits", "attn_out", "resid", "moe_out")]
        out.append(prog.read("ckv"))
        prog.close()
        return out
    got = run()
    monkeypatch.setattr(M, "build_graph", functools.partial(lambda build, *a, **k: build(*a, **{**k, "words": False}), M.build_graph))
    for g, e in zip(got, run()):
        assert np.array_equal(g, e)


@pytest.mark.parametrize("E", [16, 128, 200])
@pytest.mark.parametrize("logits", ["spread", "equal", "tiny", "far"])
def test_expert_ids_by_logit_are_those_by_probability(E, logits):
    """Router rows that make logits equal, closer than the probabilities tell apart, or so far below the largest that their probabilities are 0: the
    program whose streams take the ids from the logits against the one whose top-k is a grid of its own (softmax, then ids from memory)."""
    d = Q.Dims(name="ids", H=512, NH=4, NKV=2, HD=128, INTER=0, L=2, V=1000, qk_norm=True, moe=True, E=E, TOPK=8, MI=64, norm_topk=True)
    w = D.random_packed_weights(d, 32, DEV, seed=9)
    for L in range(d.L):
        wr = w[f"{L}.wr"]
        if logits == "equal":
            wr[1::3] = wr[0]
            wr[2::3] = 0
        elif logits == "tiny":
            wr.mul_(1e-5)
        elif logits == "far":
            wr.mul_(2000.0)
    got, want = steps(d, w, 32, [0, 1, 2, 3, 20]), steps(d, w, 32, [0, 1, 2, 3, 20], fold_topk=False)
    for g, e in zip(got, want):
        for n in e:
            assert np.array_equal(g[n], e[n]), n
