"""The grouped attention tile inside a plan, where its K / V units come through the ring and the merge is shared out: contexts that end
inside, at and behind a unit of 16 positions, more tasks than workers, the whole-context form with fewer and more units than warps,
cache slots beyond the context that hold NaN."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import etx_megakernel_b200  # noqa: E402,F401
from etx_megakernel_b200 import ops  # noqa: E402
from etx_megakernel_b200.frontends import cuda_link  # noqa: E402
from etx_megakernel_b200.importer import argblock  # noqa: E402
from etx_megakernel_b200.ir import Graph  # noqa: E402
from etx_megakernel_b200.models import qwen as Q  # noqa: E402
from etx_megakernel_b200.passes import compile_graph  # noqa: E402
from etx_megakernel_b200.runtime import Session  # noqa: E402
from oracle import ref_decode as O  # noqa: E402
from tests.test_gpu_ops import dev_bf16, host  # noqa: E402

DEV, HD = "cuda:0", 128


@pytest.mark.parametrize("NH,NKV,seq,gq,whole", [
    (8, 1, 15, 8, False), (8, 1, 16, 8, False), (8, 1, 17, 8, False), (8, 1, 128, 8, False), (16, 2, 1041, 8, False),
    (32, 4, 8150, 8, False), (12, 2, 1200, 2, False), (4, 4, 300, 1, False),
    (8, 1, 1, 8, True), (16, 4, 16, 4, True), (8, 1, 130, 8, True), (16, 2, 257, 8, True), (8, 1, 2400, 8, True)])
def test_units_through_the_ring_and_shared_merge(NH, NKV, seq, gq, whole):
    rng = np.random.default_rng(NH + seq)
    G, pos = NH // NKV, seq - 1
    parts = -(-seq // 128) + (0 if whole else 1)                              # one partition more than the context fills: idle tasks
    maxlen = parts * 128
    K = O.bfr(rng.standard_normal((maxlen, NKV, HD), dtype=np.float32) * np.float32(0.5))
    V = O.bfr(rng.standard_normal((maxlen, NKV, HD), dtype=np.float32))
    qkv = O.bfr(rng.standard_normal((NH + 2 * NKV, HD), dtype=np.float32))
    cos, sin = O.rope_tables(1e6, HD, maxlen)
    q = np.stack([O.apply_rope(h, cos[pos], sin[pos]) for h in qkv[:NH]])
    k = np.stack([O.apply_rope(h, cos[pos], sin[pos]) for h in qkv[NH:NH + NKV]])
    Kref, Vref = K.copy(), V.copy()
    Kref[pos], Vref[pos] = k, qkv[NH + NKV:]
    K[pos:], V[pos:] = np.nan, np.nan                                         # the new position's slot and everything behind it
    scale = np.float32(1.0 / np.sqrt(HD))
    want = np.zeros((NH, HD))
    for h in range(NH):
        s = (Kref[:seq, h // G].astype(np.float64) @ q[h].astype(np.float64)) * float(scale)
        p = np.exp(s - s.max())
        want[h] = (p / p.sum()) @ Vref[:seq, h // G].astype(np.float64)
    nblk = maxlen // 16
    table = rng.permutation(nblk).astype(np.int32)                            # any block order
    kc0, vc0 = O.paged_from_contig(K, V, nblk)
    inv = np.argsort(table)
    kc, vc = dev_bf16(kc0[inv]), dev_bf16(vc0[inv])
    cs = torch.from_numpy(Q.rope_table(1e6, HD, maxlen).view(np.int16)).to(DEV).view(torch.bfloat16)
    t = {"qkv": dev_bf16(qkv), "cos_sin": cs, "kc": kc, "vc": vc, "block_tables": torch.from_numpy(table).to(DEV),
         "seq_lens": torch.tensor([seq], dtype=torch.int32, device=DEV), "positions": torch.tensor([pos], dtype=torch.int64, device=DEV),
         "slot_mapping": torch.tensor([int(table[pos // 16]) * 16 + pos % 16], dtype=torch.int64, device=DEV),
         "tmp_out": torch.zeros((NH, parts, ops.attn.GQ_PARTIAL_FLOATS), dtype=torch.float32, device=DEV),
         "out": torch.zeros((NH, HD), dtype=torch.bfloat16, device=DEV)}
    ntask = NH // gq * (1 if whole else parts)
    blob = argblock.pack_named(ops.all_entries()["attn_fused"], (ntask, 1, 1), **{n: x.data_ptr() for n, x in t.items()}, scale=float(scale), eps=1e-6,
                               NH=NH, NKV=NKV, HD=HD, BS=16, X=8, max_parts=parts, gq=gq, part_len=ops.attn.tagged_part_len(3, whole))
    g = Graph("attn")
    g.tensor("impargs", (len(blob),), role="weight", bytes_per_elem=1)
    g.etensor("E_done", (1,), wait_count=ntask)
    g.call_device("attn", (ntask,), cuda_link("", "etx_tile_attn_fused"), args=["impargs"], consts=(0, 0), out_edges={"E_done": "i->(0)"})
    s = Session(compile_graph(g, "b200", {}), {}, blob, 0)
    for _ in range(2):                                                        # the second step finds the first one's partials and cache row
        t["out"].zero_()
        s.run(10.0)
        got = host(t["out"]).astype(np.float64)
        # the bf16 rounding of the result (2^-9 of it), and fp32 sums of up to 8150 terms with probabilities exact to 2^-17
        err = np.abs(got - want)
        assert np.all(err <= 2.0 ** -8 * np.abs(want) + np.abs(want).max() * 2.0 ** -13), float(err.max() / np.abs(want).max())
        assert np.linalg.norm(got - want) <= 2.0e-3 * np.linalg.norm(want)
    s.close()
    slot = int(t["slot_mapping"].item())
    row = host(kc)[slot // 16, :, :, slot % 16].reshape(NKV, HD)
    assert np.array_equal(row, k) and np.array_equal(host(vc)[slot // 16, :, :, slot % 16], qkv[NH + NKV:])
