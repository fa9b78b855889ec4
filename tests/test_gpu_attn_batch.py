"""The grouped attention tile in plans of several sequences (one argument block each) and of long contexts: what a column gets may not depend
on its place in the batch, on the other columns or on how large the cache is."""
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

DEV, HD, SCALE = "cuda:0", 128, float(np.float32(1.0 / np.sqrt(128)))


def run(NH, NKV, K, V, qkv, maxlen, gq, whole=False, scale=SCALE, rotary=True, behind=None, norm=None, seqs=None, pos=None, lim=0):
    """One attention grid over B sequences.  K, V: per sequence [seq][NKV][HD], the last position being the new one (its cache row holds NaN and comes from qkv
    [B][NH + 2 NKV][HD] instead).  Returns (out [B][NH][HD] bf16 values, the cached k rows at the new positions [B][NKV][HD], the partials
    [B][NH][partitions][128 sums, maximum, sum of the probabilities]).  behind: a second grid of one empty task that waits for the first attention task
    alone, and the queues of the plan as a function of the attention tasks' and its number.  norm: weights of the q and k norms.  seqs, pos: sequence
    lengths and new positions where the new one is not the last (its cache row and all rows behind the length hold NaN)."""
    B, nblk, parts = len(K), maxlen // 16, -(-maxlen // 128)
    seq = np.array(seqs if seqs is not None else [len(k) for k in K])
    pos = np.array(pos) if pos is not None else seq - 1
    pools = []
    for b in range(B):
        kv = np.full((2, maxlen, NKV, HD), np.nan, np.float32)
        kv[0, :seq[b]], kv[1, :seq[b]] = K[b][:seq[b]], V[b][:seq[b]]
        kv[:, pos[b]] = np.nan
        pools.append(O.paged_from_contig(kv[0], kv[1], nblk))
    table = np.random.default_rng(1).permutation(B * nblk).astype(np.int32)                # any block order
    inv = np.argsort(table)
    kc, vc = (dev_bf16(np.concatenate([p[i] for p in pools])[inv]) for i in (0, 1))
    tab = Q.rope_table(1e6, HD, maxlen).view(np.int16)
    if not rotary:
        tab = np.concatenate([O.f32_to_bf16_bits(np.ones((maxlen, HD // 2), np.float32)).view(np.int16), np.zeros((maxlen, HD // 2), np.int16)], 1)
    t = {"qkv": dev_bf16(qkv), "cos_sin": torch.from_numpy(tab).to(DEV).view(torch.bfloat16), "kc": kc, "vc": vc,
         "block_tables": torch.from_numpy(table).to(DEV), "seq_lens": torch.from_numpy(seq.astype(np.int32)).to(DEV),
         "positions": torch.from_numpy(pos.astype(np.int64)).to(DEV), "tmp_out": torch.zeros((B, NH, parts, ops.attn.GQ_PARTIAL_FLOATS), dtype=torch.float32, device=DEV),
         "slot_mapping": torch.from_numpy(np.array([int(table[b * nblk + p // 16]) * 16 + p % 16 for b, p in enumerate(pos)], np.int64)).to(DEV),
         "out": torch.zeros((B, NH, HD), dtype=torch.bfloat16, device=DEV)}
    if norm is not None:
        t["qw"], t["kw"] = (dev_bf16(w) for w in norm)
    step = {"qkv": (NH + 2 * NKV) * HD * 2, "block_tables": nblk * 4, "seq_lens": 4, "positions": 8, "slot_mapping": 8,
            "tmp_out": NH * parts * ops.attn.GQ_PARTIAL_FLOATS * 4, "out": NH * HD * 2}
    ntask = NH // gq * (1 if whole else parts)
    blobs = b"".join(argblock.pack_named(ops.all_entries()["attn_fused"], (ntask, 1, 1), **{n: x.data_ptr() + b * step.get(n, 0) for n, x in t.items()}, scale=scale,
                                         eps=1e-6, NH=NH, NKV=NKV, HD=HD, BS=16, X=8, max_parts=parts, gq=gq, part_len=ops.attn.tagged_part_len(3, whole, lim=lim)) for b in range(B))
    g = Graph("attn")
    g.tensor("impargs", (len(blobs),), role="weight", bytes_per_elem=1)
    if behind is None:
        g.etensor("E_done", (1,), wait_count=ntask * B)
        g.call_device("attn", (ntask, B), cuda_link("", "etx_tile_attn_fused"), args=["impargs"], consts=(0, ops.attn.F_ARG_BYTES), out_edges={"E_done": "ij->(0)"})
    else:
        g.etensor("E_done", (ntask, B), wait_count=1)
        g.etensor("E_empty", (1,), wait_count=1)
        g.call_device("attn", (ntask, B), cuda_link("", "etx_tile_attn_fused"), args=["impargs"], consts=(0, ops.attn.F_ARG_BYTES), out_edges={"E_done": "ij->ij"})
        g.call_device("empty", (1,), cuda_link("", "nop"), args=["impargs"], consts=(0, 0), in_edges={"E_done": "i->(0)(0)"}, out_edges={"E_empty": "i->(0)"})
    plan = compile_graph(g, "b200", {})
    if behind is not None:
        queues = behind([i for i, t in enumerate(plan.tasks) if t.grid == "attn"], [i for i, t in enumerate(plan.tasks) if t.grid == "empty"][0])
        plan.static_queues = {(0, w): queues[w] if w < len(queues) else [] for w in range(plan.workers_per_device())}
    s = Session(plan, {}, blobs, 0)
    outs = []
    for _ in range(2):
        t["out"].zero_()
        s.run(10.0)
        outs.append(host(t["out"]).copy())
    s.close()
    assert np.array_equal(outs[0], outs[1], equal_nan=True)
    slot = host(t["slot_mapping"])
    tmp = host(t["tmp_out"]).reshape(B, NH, parts, ops.attn.GQ_PARTIAL_FLOATS // 2, 2)[..., :HD + 2, 0]
    return outs[0], np.stack([host(kc)[s // 16, :, :, s % 16].reshape(NKV, HD) for s in slot]), tmp


@pytest.mark.parametrize("seq,gq,B", [(1030, 8, 10), (1030, 2, 10), (900, 8, 10), (4200, 8, 10), (1000, 8, 40)])
def test_equal_columns_get_equal_bits_wherever_they_stand(seq, gq, B):
    """Ten equal sequences, 9 partitions: the numbers of tasks that share a group's merge differ between the columns; 40 sequences: more groups than workers,
    some with no worker's last task among theirs; one sequence, and three in a larger cache: other numbers again.  V alternates by partition, so that the sum over the partitions is small beside its terms and
    another order of them would show."""
    NH, NKV, G = 32, 4, 8
    rng = np.random.default_rng(seq)
    V = O.bfr(rng.standard_normal((seq, NKV, HD), dtype=np.float32) + np.where(np.arange(seq) // 128 % 2, -900.0, 900.0).astype(np.float32)[:, None, None])
    K = O.bfr(rng.standard_normal((seq, NKV, HD), dtype=np.float32) * np.float32(0.3))
    qkv = O.bfr(rng.standard_normal((NH + 2 * NKV, HD), dtype=np.float32))
    maxlen = -(-seq // 128) * 128
    one, _, _ = run(NH, NKV, [K], [V], qkv[None], maxlen, gq)
    many, _, _ = run(NH, NKV, [K] * B, [V] * B, np.stack([qkv] * B), maxlen, gq)
    large, _, _ = run(NH, NKV, [K] * 3, [V] * 3, np.stack([qkv] * 3), maxlen + 640, gq)
    assert np.isfinite(one).all() and np.abs(one).max() < 900
    for b in range(B):
        assert np.array_equal(many[b], one[0]), f"column {b}: {np.mean(many[b] != one[0]):.4f} of the values differ"
    for b in range(3):
        assert np.array_equal(large[b], one[0]), f"larger cache, column {b}: {np.mean(large[b] != one[0]):.4f} of the values differ"


def test_a_merge_waits_for_nothing_that_waits_for_its_task():
    """Eight partitions of one group, 64 partials.  The first worker has the first attention task alone; the second one an empty task that waits for it, then the other
    attention tasks.  If the first task, the last of its worker, waited for the others' partials, they would wait for it too."""
    rng = np.random.default_rng(3)
    K, V, qkv = (O.bfr(rng.standard_normal(s, dtype=np.float32)) for s in ((1000, 1, HD), (1000, 1, HD), (10, HD)))
    want, _, _ = run(8, 1, [K], [V], qkv[None], 1024, 8)
    got, _, _ = run(8, 1, [K], [V], qkv[None], 1024, 8, behind=lambda attn, empty: [attn[:1], [empty] + attn[1:]])
    assert np.array_equal(got, want)


def chains(terms, n=32):
    """Sum over the last axis in fp32: chains of n terms (each step rounded once), their results added one by one."""
    out = None
    for c in range(0, terms.shape[-1], n):
        acc = np.zeros(terms.shape[:-1], np.float32)
        for i in range(c, min(c + n, terms.shape[-1])):
            acc = (acc.astype(np.float64) + terms[..., i]).astype(np.float32)
        out = acc if out is None else (out + acc).astype(np.float32)
    return out


@pytest.mark.parametrize("seq,NH,NKV,gq", [(1030, 8, 1, 8), (334, 12, 2, 1), (2100, 8, 2, 4)])
def test_partials_are_as_exact_as_fp32_chains(seq, NH, NKV, gq):
    """What the tasks publish, put together in 64 bits, against attention in 64 bits: no further off than fp32 arithmetic in chains of 32 terms (scores over 32
    dims, outputs over 32 positions), which is what the products ran in before they went to the tensor cores.  The rounding of the result to
    bf16 hides all of it, so the partials are looked at."""
    G, got, plain = NH // NKV, [], []
    for seed in range(3):
        rng = np.random.default_rng(100 * seed + seq)
        K, V, qkv = (O.bfr(rng.standard_normal(s, dtype=np.float32)) for s in ((seq, NKV, HD), (seq, NKV, HD), (NH + 2 * NKV, HD)))
        cos, sin = O.rope_tables(1e6, HD, seq)
        q = np.stack([O.apply_rope(h, cos[-1], sin[-1]) for h in qkv[:NH]])
        _, _, tmp = run(NH, NKV, [K], [V], qkv[None], -(-seq // 128) * 128, gq)
        K[-1], V[-1] = np.stack([O.apply_rope(h, cos[-1], sin[-1]) for h in qkv[NH:NH + NKV]]), qkv[NH + NKV:]
        for h in range(NH):
            k, v = K[:, h // G].astype(np.float64), V[:, h // G].astype(np.float64)
            s = k @ q[h].astype(np.float64) * SCALE
            p = np.exp(s - s.max())
            want = p @ v / p.sum()
            pr = tmp[0, h].astype(np.float64)
            w = np.exp(pr[:, HD] - pr[:, HD].max())
            got.append((w @ pr[:, :HD] / (w @ pr[:, HD + 1]) - want) / np.linalg.norm(want))
            sf = chains(k * q[h].astype(np.float64)) * np.float32(SCALE)
            o, l, m = [], [], []
            for a in range(0, seq, 128):
                sp = sf[a:a + 128]
                pf = np.exp(sp - sp.max()).astype(np.float32)
                o.append(chains((pf[:, None].astype(np.float64) * v[a:a + 128]).T)); l.append(pf.astype(np.float64).sum()); m.append(sp.max())
            w = np.exp(np.float64(m) - np.max(m))
            plain.append((w @ np.float64(o) / (w @ l) - want) / np.linalg.norm(want))
    got, plain = np.sqrt(np.mean(np.square(got)) * HD), np.sqrt(np.mean(np.square(plain)) * HD)
    print(f"{seq} positions, gq {gq}: {got:.3e}, fp32 chains {plain:.3e}")
    assert got <= plain


def third_parts(NH):
    """NH differences of scores whose probability has a third bf16 part of 2^-19 of it and more, and the probability with its parts."""
    d = np.arange(1, 4096, dtype=np.float32) / np.float32(1024)                          # bf16-exact differences of the scores, the third parts largest
    d = d[O.bfr(d) == d]
    p = np.exp(-d.astype(np.float64)).astype(np.float32)
    first = O.bfr(p)
    second = O.bfr(p - first)
    third = p - first - second
    best = np.argsort(-np.abs(third) / p)[:NH]
    d, first, second, third, p = (x[best].astype(np.float64) for x in (d, first, second, third, p))
    assert np.all(np.abs(third) / p > 2.0 ** -19)
    return d, first, second, third, p


@pytest.mark.parametrize("whole", [True, False])
def test_the_new_position_keeps_all_bits_of_its_probability(whole):
    """Two cached positions of probability 1 take away the first two bf16 parts of the new position's, so what is left of the sum is its third part (2^-18
    of it and less): 0 if that part were not multiplied.  A difference of two units in the last place of exp() is 2^-5 of what is left."""
    NH, gq = 8, 8
    d, first, second, third, p = third_parts(NH)
    K, V, qkv = np.zeros((3, 1, HD), np.float32), np.zeros((3, 1, HD), np.float32), np.zeros((NH + 2, HD), np.float32)
    K[:2, 0, 0], qkv[:NH, 0] = 1.0, d                                                    # score of a cached position: d of the head, of the new one: 0
    V[0, 0, :NH], V[1, 0, :NH], qkv[NH + 1, :NH] = -first, -second, 1.0
    out, _, _ = run(NH, 1, [K], [V], qkv[None], 128, gq, whole=whole, scale=1.0, rotary=False)
    want = third / (2.0 + p)
    got = out[0, np.arange(NH), np.arange(NH)]
    assert np.all(np.abs(got - want) <= 2.0 ** -4 * np.abs(want)), (got, want)


@pytest.mark.parametrize("whole,lim,all_bits", [(False, 0, True), (False, 2, True), (True, 1, True), (True, 0, False)])
def test_a_cached_position_keeps_all_bits_of_its_probability(whole, lim, all_bits):
    """The same with the third of the three in the cache, in a unit of 16 positions that the new one is not in (its probability and those of the others are
    below 2^-100): partitions and contexts up to the limit keep 24 bits, whole contexts where the block asks for them, else 17."""
    NH, gq, seq = 8, 8, 40
    d, first, second, third, p = third_parts(NH)
    K, V, qkv = np.zeros((seq, 1, HD), np.float32), np.zeros((seq, 1, HD), np.float32), np.zeros((NH + 2, HD), np.float32)
    K[:2, 0, 0], K[3:, 0, 1], qkv[NH, 1] = 1.0, -128.0, -128.0
    qkv[:NH, 0], qkv[:NH, 1] = d, 1.0                                                    # scores: d, d, 0, then -128
    V[0, 0, :NH], V[1, 0, :NH], V[2, 0, :NH] = -first, -second, 1.0
    out, _, _ = run(NH, 1, [K], [V], qkv[None], 128, gq, whole=whole, scale=1.0, rotary=False, lim=lim)
    want = third / (2.0 + p)
    got = out[0, np.arange(NH), np.arange(NH)]
    assert np.all(np.abs(got - want) <= 2.0 ** -4 * np.abs(want)) == all_bits, (got, want)


@pytest.mark.parametrize("seq,NH,NKV,gq,whole", [(300, 8, 2, 4, False), (40, 8, 1, 8, False), (300, 8, 2, 4, True)])
def test_infinite_values_in_the_cache_stay_infinite(seq, NH, NKV, gq, whole):
    """V rows that overflowed bf16: the sum of an infinite value and finite ones is that value, in its dim alone; values of both signs give NaN.  A key row of
    minus infinity (against positive q values) takes its position out."""
    rng = np.random.default_rng(seq)
    K, V, qkv = (O.bfr(rng.standard_normal(s, dtype=np.float32)) for s in ((seq, NKV, HD), (seq, NKV, HD), (NH + 2 * NKV, HD)))
    qkv = np.abs(qkv)
    K[5, :, 7] = -np.inf
    V[5], V[3, :, 10], V[seq // 2, :, 11] = 3.0, np.inf, -np.inf
    V[2, :, 12], V[9, :, 12] = np.inf, -np.inf
    qkv[NH + NKV:, 13] = np.inf                                                           # the new position's own row
    out, _, _ = run(NH, NKV, [K], [V], qkv[None], -(-seq // 128) * 128, gq, whole=whole, rotary=False)
    K[-1], V[-1] = qkv[NH:NH + NKV], qkv[NH + NKV:]
    for h in range(NH):
        k, v = K[:, h * NKV // NH].astype(np.float64), V[:, h * NKV // NH].astype(np.float64)
        s = k @ qkv[h].astype(np.float64) * SCALE
        assert s[5] == -np.inf
        p = np.exp(s - s.max())
        want = np.where(p[:, None] > 0, p[:, None] * v, 0.0).sum(0) / p.sum()
        fin = np.isfinite(want)
        assert np.array_equal(np.flatnonzero(~fin), [10, 11, 12, 13])
        assert np.array_equal(out[0, h, ~fin], want[~fin].astype(np.float32), equal_nan=True), out[0, h, ~fin]
        assert np.all(np.abs(out[0, h, fin] - want[fin]) <= 2.0 ** -8 * np.abs(want[fin]) + np.abs(want[fin]).max() * 2.0 ** -13)


@pytest.mark.parametrize("norm", [True, False])
@pytest.mark.parametrize("whole", [False, True])
def test_sequences_of_different_lengths_in_a_large_cache(norm, whole):
    """One plan over sequences of 1 to 1000 positions (1 to 8 partitions of 8 q heads: both sides of the number of partials from which the merge is shared) in a cache of
    1280, most of whose tasks have nothing to do; with and without the q / k norms; positions that are not the last of their sequence -- inside it, where the
    cached row is replaced, behind it in its last block, and in a block behind that."""
    NH, NKV, gq, maxlen = 16, 2, 8, 1280
    seqs, pos = (1, 16, 129, 700, 1000, 890, 333, 97, 100, 100), (0, 15, 128, 699, 999, 889, 200, 0, 105, 125)
    rng = np.random.default_rng(7)
    nw, kw = (O.bfr(1 + 0.1 * rng.standard_normal(HD, dtype=np.float32)) for _ in range(2))
    K, V = ([O.bfr(rng.standard_normal((max(s, p + 1), NKV, HD), dtype=np.float32)) for s, p in zip(seqs, pos)] for _ in range(2))
    qkv = O.bfr(rng.standard_normal((len(seqs), NH + 2 * NKV, HD), dtype=np.float32))
    out, rows, _ = run(NH, NKV, K, V, qkv, maxlen, gq, whole=whole, norm=(nw, kw) if norm else None, seqs=seqs, pos=pos)
    cos, sin = O.rope_tables(1e6, HD, maxlen)
    for b, (s, p) in enumerate(zip(seqs, pos)):
        x = qkv[b]
        q, k = (np.stack([O.rmsnorm(h, w, 1e-6) for h in y]) if norm else y for y, w in ((x[:NH], nw), (x[NH:NH + NKV], kw)))
        q, k = (np.stack([O.apply_rope(h, cos[p], sin[p]) for h in y]) for y in (q, k))
        assert np.array_equal(rows[b], k), f"column {b}: the cached k row"
        used = sorted(set(range(s)) | {p})
        for h in range(NH):
            kk, vv = K[b][:, h * NKV // NH].astype(np.float64), V[b][:, h * NKV // NH].astype(np.float64)
            kk[p], vv[p] = k[h * NKV // NH], x[NH + NKV + h * NKV // NH]
            sc = kk[used] @ q[h].astype(np.float64) * SCALE
            w = np.exp(sc - sc.max())
            want = w @ vv[used] / w.sum()
            # the bf16 rounding of the result (2^-9 of it), and fp32 sums with probabilities exact to 2^-17
            assert np.all(np.abs(out[b, h] - want) <= 2.0 ** -8 * np.abs(want) + np.abs(want).max() * 2.0 ** -13), (b, h)


def test_shared_and_single_merges_give_the_same_bits():
    """64 partials of a group, merged by eight tasks, by the last ones of two workers, and by the last partition's task alone (a queue that is not in ascending order)."""
    rng = np.random.default_rng(11)
    V = O.bfr(rng.standard_normal((1000, 1, HD), dtype=np.float32) + np.where(np.arange(1000) // 128 % 2, -900.0, 900.0).astype(np.float32)[:, None, None])
    K, qkv = (O.bfr(rng.standard_normal(s, dtype=np.float32) * np.float32(0.3)) for s in ((1000, 1, HD), (10, HD)))
    eight, _, _ = run(8, 1, [K], [V], qkv[None], 1024, 8)
    two, _, _ = run(8, 1, [K], [V], qkv[None], 1024, 8, behind=lambda attn, empty: [attn[4:], attn[:4] + [empty]])
    alone, _, _ = run(8, 1, [K], [V], qkv[None], 1024, 8, behind=lambda attn, empty: [attn[4:], attn[3::-1] + [empty]])
    assert np.array_equal(two, eight) and np.array_equal(alone, eight)
