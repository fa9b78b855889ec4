"""Sessions over the same buffers, one step after the other: no step takes what another session's step left in the hand-off's words or among the partial
results of the attention phase, nor what the memory held before."""
import numpy as np
import pytest
import torch

from etx_megakernel_b200.models import decode as D
from etx_megakernel_b200.models import qwen as Q
from etx_megakernel_b200.runtime import Session

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
MAXLEN, POS = 720, 641                  # six partitions, the last of two positions: its task merges while others still publish theirs


def dims(moe):
    return Q.Dims(name="shared", H=512, NH=4, NKV=1, HD=128, INTER=0 if moe else 512, L=2, V=1000, qk_norm=True, moe=moe, E=16 if moe else 0,
                  TOPK=4 if moe else 0, MI=128 if moe else 0, norm_topk=True)


def program(d, w, workers):
    prog = D.DecodeProgram(d, w, device=0, maxlen=MAXLEN, workers=workers)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(2)
    prog.buf["kc"].normal_(0, 1, generator=gen)
    prog.buf["vc"].normal_(0, 1, generator=gen)
    return prog


def another_session(prog):
    s, b, d = Session(prog.plan, {"vl": prog.vl}, prog.pool.bytes(), 0), prog.buf, prog.d
    s.set_step(tok=0, pos=0, write_next=0, H=d.H, V=d.lm_rows, nrep=1, embed=prog.w["embed"], resid=b["resid"], positions=b["positions"],
               seq_lens=b["seq_lens"], slot_mapping=b["slot_mapping"], logits=b["logits"], token_in=b["token_in"], token_out=b["token_out"],
               token_time=b["token_time"])
    return s


def step(prog, session, token):
    prog.buf["token_in"][0] = token
    torch.cuda.synchronize()
    session.set_step(tok=0, pos=POS, write_next=0)
    session.run(10.0)
    return prog.read("logits").copy()


def alone(d, w, tokens, workers=None):
    prog = program(d, w, workers)
    out = [step(prog, prog.session, t) for t in tokens]
    prog.close()
    return out


@pytest.mark.parametrize("workers", [None, 2, 3])
@pytest.mark.parametrize("moe", [True, False])
def test_sessions_take_turns(moe, workers):
    """Equal step numbers, other tokens; then a session that comes when another has closed."""
    d = dims(moe)
    w = D.random_packed_weights(d, MAXLEN, DEV, seed=1)
    tokens = list(range(3, 3 + 12))
    want = alone(d, w, tokens, workers)
    prog = program(d, w, workers)
    other = another_session(prog)
    got = [step(prog, (prog.session, other)[i % 2], t) for i, t in enumerate(tokens[:8])]
    other.close()
    for t in tokens[8:]:
        other = another_session(prog)
        got.append(step(prog, other, t))
        other.close()
    prog.close()
    for i, (g, e) in enumerate(zip(got, want)):
        assert np.array_equal(g, e), i


def test_a_merge_does_not_take_another_sessions_partials():
    """A queue with the merging task in front of one of its partitions: in a session of its own it runs out of time (tests/test_gpu_attn_groups.py), and it must
    when a session before it has left partials of the same step number in the buffer."""
    from etx_megakernel_b200 import ops
    from etx_megakernel_b200.frontends import cuda_link
    from etx_megakernel_b200.importer import argblock
    from etx_megakernel_b200.ir import Graph
    from etx_megakernel_b200.passes import compile_graph
    from etx_megakernel_b200.runtime.lib import EtxbError
    parts = 3
    maxlen = 128 * parts
    t = lambda dt, *shape: torch.zeros(shape, dtype=dt, device=DEV)                    # noqa: E731
    qkv, cs, out = t(torch.bfloat16, 3, 128), t(torch.bfloat16, maxlen, 128), t(torch.bfloat16, 1, 128)
    kc, vc = t(torch.bfloat16, maxlen // 16, 1, 16, 16, 8), t(torch.bfloat16, maxlen // 16, 1, 128, 16)
    bt, tmp, stat = torch.arange(maxlen // 16, dtype=torch.int32, device=DEV), t(torch.float32, parts, ops.attn.GQ_PARTIAL_FLOATS), t(torch.float32, parts)
    seq, pos, cnt = torch.tensor([maxlen - 3], dtype=torch.int32, device=DEV), torch.tensor([maxlen - 4], device=DEV), t(torch.int32, 1)
    p = lambda x: x.data_ptr()                                                         # noqa: E731
    blob = argblock.pack_named(ops.all_entries()["attn_fused"], (parts, 1, 1), qkv=p(qkv), cos_sin=p(cs), kc=p(kc), vc=p(vc), block_tables=p(bt),
                               seq_lens=p(seq), positions=p(pos), slot_mapping=p(pos), exp_sums=p(stat), max_logits=p(stat), tmp_out=p(tmp), out=p(out),
                               counters=p(cnt), scale=0.1, eps=1e-6, NH=1, NKV=1, HD=128, BS=16, X=8, max_parts=parts, gq=1, part_len=128)
    g = Graph("partials")
    g.tensor("impargs", (len(blob),), role="weight", bytes_per_elem=1)
    g.etensor("E_done", (1,), wait_count=parts)
    g.call_device("attn", (parts,), cuda_link("", "etx_tile_attn_fused"), args=["impargs"], consts=(0, 0), out_edges={"E_done": "i->(0)"})
    first = Session(compile_graph(g, "b200", {}), {}, blob, 0)
    first.run(5.0)
    first.close()
    plan = compile_graph(g, "b200", {})
    queues = [k for k, q in plan.static_queues.items() if q]
    for k in queues:
        plan.static_queues[k] = []
    plan.static_queues[queues[0]] = [parts - 1, 0]
    plan.static_queues[queues[1]] = [1]
    second = Session(plan, {}, blob, 0)
    second.set_option("timeout_ms", 200)
    with pytest.raises(EtxbError, match="TIMEOUT"):
        second.run(5.0)
    second.close()


@pytest.mark.parametrize("moe", [True, False])
def test_words_that_look_current_before_the_first_step(moe):
    """Memory that holds the first step's flag everywhere, with values of its own."""
    d = dims(moe)
    w = D.random_packed_weights(d, MAXLEN, DEV, seed=1)
    want = alone(d, w, [5])[0]
    prog = program(d, w, None)
    prog.buf["words"].fill_(-0x7ffec080)                            # 0x80013f80: 1.0 of step 1
    got = step(prog, prog.session, 5)
    prog.close()
    assert np.array_equal(got, want)
