"""Grouped attention where the q heads per kv head are no power of two (the size of a group divides them), at the edges of a
partition of 128 positions; and the rule that picks the group size."""
import pytest

torch = pytest.importorskip("torch")

import etx_megakernel_b200  # noqa: E402,F401
from etx_megakernel_b200.machine import load_machine  # noqa: E402


@pytest.mark.parametrize("G", [1, 2, 3, 4, 5, 6, 7, 8, 12, 16])
@pytest.mark.parametrize("NKV,maxlen", [(1, 128), (2, 608), (4, 1072), (8, 8192)])
def test_group_size_divides_the_heads_of_a_kv_head(G, NKV, maxlen):
    m = load_machine("b200")
    gq, plen, parts = m.attention_groups(G * NKV, NKV, 128, 16, maxlen)
    assert gq in (1, 2, 4, 8) and G % gq == 0 and plen == 128 and parts == -(-maxlen // 128)
    smaller = [g for g in (1, 2, 4, 8) if g < gq and G % g == 0]
    assert all(G * NKV // g * parts > m.workers() for g in smaller)          # no smaller group would have given every task its own SM
    assert m.attention_groups(G * NKV, NKV, 64, 16, maxlen) == (0, 0, 0)     # other head sizes: the general tile


@pytest.mark.gpu
@pytest.mark.parametrize("NH,NKV,qk_norm,seq,gq", [(12, 2, False, 1, 1), (12, 2, False, 127, 2), (12, 2, False, 128, 1), (12, 2, True, 129, 2),
                                                   (12, 2, False, 1700, 2), (6, 2, True, 300, 1), (12, 1, False, 257, 4),
                                                   (28, 4, False, 385, 1), (15, 1, True, 256, 1), (16, 1, False, 300, 8)])
def test_grouped_phase_with_other_head_counts(NH, NKV, qk_norm, seq, gq):
    from tests.test_gpu_ops import test_attention_phase_fused as phase
    phase(NH, NKV, 128, qk_norm, seq, gq)


@pytest.mark.gpu
@pytest.mark.parametrize("parts", [2, 14])
def test_a_merge_whose_partition_never_comes_reports_the_flags(parts):
    """The task of the first partition is queued BEHIND the merging one on the same worker (a plan that the host-side verifier
    rejects; built here by hand), so the merge can only end by its deadline, with the partials in registers (2 partitions) or
    in rounds (14): the status names the flag it needed and the one it saw, and the context stays usable."""
    from etx_megakernel_b200 import ops
    from etx_megakernel_b200.frontends import cuda_link
    from etx_megakernel_b200.importer import argblock
    from etx_megakernel_b200.ir import Graph
    from etx_megakernel_b200.passes import compile_graph
    from etx_megakernel_b200.runtime import Session
    from etx_megakernel_b200.runtime.lib import EtxbError
    dev, maxlen = "cuda:0", 128 * parts
    b16 = lambda *shape: torch.zeros(shape, dtype=torch.bfloat16, device=dev)          # noqa: E731
    qkv, cs, kc, vc, out = b16(3, 128), b16(maxlen, 128), b16(maxlen // 16, 1, 16, 16, 8), b16(maxlen // 16, 1, 128, 16), b16(1, 128)
    bt = torch.arange(maxlen // 16, dtype=torch.int32, device=dev)
    seq, pos = torch.tensor([maxlen - 3], dtype=torch.int32, device=dev), torch.tensor([maxlen - 4], dtype=torch.int64, device=dev)
    tmp = torch.zeros((parts, ops.attn.GQ_PARTIAL_FLOATS), dtype=torch.float32, device=dev)
    stat, cnt = torch.zeros(parts, dtype=torch.float32, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    p = lambda t: t.data_ptr()                                                         # noqa: E731
    blob = argblock.pack_named(ops.all_entries()["attn_fused"], (parts, 1, 1), qkv=p(qkv), cos_sin=p(cs), kc=p(kc), vc=p(vc), block_tables=p(bt),
                               seq_lens=p(seq), positions=p(pos), slot_mapping=p(pos), exp_sums=p(stat), max_logits=p(stat), tmp_out=p(tmp), out=p(out),
                               counters=p(cnt), scale=0.1, eps=1e-6, NH=1, NKV=1, HD=128, BS=16, X=8, max_parts=parts, gq=1, part_len=128)
    g = Graph("merge_deadline")
    g.tensor("impargs", (len(blob),), role="weight", bytes_per_elem=1)
    g.etensor("E_done", (1,), wait_count=parts)
    g.call_device("attn", (parts,), cuda_link("", "etx_tile_attn_fused"), args=["impargs"], consts=(0, 0), out_edges={"E_done": "i->(0)"})
    plan = compile_graph(g, "b200", {})
    queues = [k for k, q in plan.static_queues.items() if q]
    assert sorted(t for q in plan.static_queues.values() for t in q) == list(range(parts))
    for k in queues:
        plan.static_queues[k] = []
    plan.static_queues[queues[0]] = [parts - 1, 0]
    for t in range(1, parts - 1):
        plan.static_queues[queues[t]] = [t]
    s = Session(plan, {}, blob, 0)
    s.set_option("timeout_ms", 200)
    with pytest.raises(EtxbError) as e:
        s.run(5.0)
    st = s.status()
    assert e.value.status == "E_TIMEOUT" and st.stuck_event == -3 and st.stuck_value == 0
    assert st.stuck_target & 0xffffffff == 0x80000000 | (1 << 8)                       # the first step's flag
    s.close()
    healthy = Session(compile_graph(g, "b200", {}), {}, blob, 0)
    healthy.run(5.0)
    healthy.close()
