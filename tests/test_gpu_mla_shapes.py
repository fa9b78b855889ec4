"""The latent-attention tile at other widths than the bundled model's: W_UK and the cached rows come through the ring as many whole rows to a stage as fit,
so the widths decide where a stage ends; cached rows whose score is minus infinity."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import etx_megakernel_b200  # noqa: E402,F401
from etx_megakernel_b200 import ops  # noqa: E402
from etx_megakernel_b200.importer import argblock  # noqa: E402
from etx_megakernel_b200.models import dsv2 as M  # noqa: E402
from etx_megakernel_b200.ops import mla as op_mla  # noqa: E402
from etx_megakernel_b200.runtime import op_launch  # noqa: E402
from oracle import ref_mla as R  # noqa: E402
from oracle.ref_decode import bfr  # noqa: E402
from tests.test_gpu_mla import BF16_REL, DEV, dev_bf16, host  # noqa: E402
from tests.test_mla_host import oracle_dims  # noqa: E402


def setup(NH, C, DN, DR, DV, ctx):
    d = M.MlaDims(name="t", H=NH * DV, NH=NH, C=C, DN=DN, DR=DR, DV=DV, MI=128, E=4, TOPK=2, NS=0, DENSE_LAYERS=0, DENSE_INTER=0, L=1, V=256)
    od = oracle_dims(d)
    lw = R.synthetic_layer(od, seed=10 + ctx)
    lw.o_proj = np.eye(d.H, dtype=np.float32)                 # the oracle's attention() then returns bf16(out) itself
    rng = np.random.default_rng(ctx)
    cos, sin = R.yarn_tables(od, ctx + 8)
    cache = np.zeros((ctx + 8, d.ROW), np.float32)
    for t in range(ctx):
        R.attention(od, lw, bfr(rng.standard_normal(d.H).astype(np.float32)), cache, t, cos, sin)
    return d, od, lw, cache, bfr(rng.standard_normal(d.H).astype(np.float32)), cos, sin


def tile(d, lw, x, cache, ctx):
    """One launch of the tile: (output [NH * DV], cache afterwards)."""
    maxlen = cache.shape[0]
    xn = R.rmsnorm2(x, lw.input_layernorm, d.eps)
    t = {"qkv": dev_bf16(np.concatenate([bfr(lw.q_proj @ xn), bfr(lw.kv_a_proj_with_mqa @ xn)])), "kvln": dev_bf16(lw.kv_a_layernorm), "wkvb": dev_bf16(lw.kv_b_proj),
         "cos_sin": torch.from_numpy(M.yarn_table(d, maxlen)).to(DEV), "cache": dev_bf16(cache), "positions": torch.tensor([ctx], dtype=torch.int64, device=DEV),
         "out": torch.zeros(d.NH * d.DV, dtype=torch.bfloat16, device=DEV), "tmp": torch.zeros((op_mla.tmp_pairs(d.NH, d.C, maxlen), 2), dtype=torch.float32, device=DEV)}
    nparts = op_mla.partitions(maxlen)
    tasks = d.NH * (nparts + op_mla.FINISHERS)
    op_launch("mla_attn", argblock.pack_named(ops.all_entries()["mla_attn"], (tasks, 1, 1), **{n: v.data_ptr() for n, v in t.items()}, NH=d.NH, C=d.C, DN=d.DN, DR=d.DR, DV=d.DV,
                                              maxlen=maxlen, scale=d.scale, eps=d.eps, max_parts=nparts, tag=3), tasks)
    return host(t["out"]), host(t["cache"])


@pytest.mark.parametrize("NH,C,DN,DR,DV,ctx", [(3, 96, 40, 16, 48, 140), (4, 256, 100, 32, 64, 270), (2, 512, 192, 64, 128, 129), (5, 8, 1, 8, 8, 37), (2, 256, 64, 64, 200, 300)])
def test_other_widths_against_the_oracle(NH, C, DN, DR, DV, ctx):
    d, od, lw, cache, x, cos, sin = setup(NH, C, DN, DR, DV, ctx)
    before = cache.copy()
    want = R.attention(od, lw, x, cache, ctx, cos, sin)
    got, after = tile(d, lw, x, before, ctx)
    # (the latent norm sums in numpy's order where C is a power of two from 128 on, else to fp32 rounding)
    assert np.abs(after[ctx] - cache[ctx]).max() <= 2.0 ** -7 * np.abs(cache[ctx]).max()
    assert np.array_equal(after[:ctx], before[:ctx]) and not after[ctx + 1:].any()
    err = np.abs(got - want).max() / np.abs(want).max()
    assert err <= BF16_REL and np.mean(got == want) >= 0.9, (err, np.mean(got == want))


def test_rows_whose_score_is_minus_infinity_take_no_part():
    """The first row that every warp takes has a key of minus infinity against the query: probability 0, as in any other place.  (Of plus infinity: NaN.)"""
    d, od, lw, cache, x, cos, sin = setup(1, 256, 64, 32, 64, 150)
    finite = 0
    for key in (-np.inf, np.inf):                             # one of them, by the sign of the query in this dim
        before = cache.copy()
        before[:16, d.C + 3] = key
        with np.errstate(invalid="ignore"):
            want = R.attention(od, lw, x, before.copy(), 150, cos, sin)
        got, _ = tile(d, lw, x, before, 150)
        if np.isfinite(want).all():
            finite += 1
            assert np.abs(got - want).max() <= BF16_REL * np.abs(want).max()
        else:
            assert np.isnan(want).all() and np.isnan(got).all()
    assert finite == 1


@pytest.mark.parametrize("ctx", [5, 1043, 1290, 4095, 8150])
def test_long_contexts_to_fp32(ctx):
    """Weighted means to 32 bits, through the bf16 output: latent columns that hold one constant c_j at every position have c_j as their mean whatever the
    weights are, and an output row c_k o_j - c_j o_k leaves the errors of the sums alone.  The roundings in a mean: 8 positions a warp, 16 warps,
    the partitions, once more for the sum of the weights, the division and the product."""
    NH, C, DN, DR, DV, maxlen = 2, 512, 128, 64, 128, ctx + 9
    d = M.MlaDims(name="t", H=NH * DV, NH=NH, C=C, DN=DN, DR=DR, DV=DV, MI=128, E=4, TOPK=2, NS=0, DENSE_LAYERS=0, DENSE_INTER=0, L=1, V=256)
    rng = np.random.default_rng(ctx)
    const = rng.integers(4, 16, 480).astype(np.float32) / 8                            # (short mantissas: c_k o_j rounds once)
    cache = np.zeros((maxlen, d.ROW), np.float32)
    cache[:ctx, :480] = const
    cache[:ctx, 480:] = bfr(rng.standard_normal((ctx, d.ROW - 480), dtype=np.float32))
    cache[:ctx, 480] = bfr(8 * np.arange(ctx, dtype=np.float32) / ctx)                 # the partitions' maxima differ, most grow
    wkvb = np.zeros((NH, DN + DV, C), np.float32)
    wkvb[:, :DN, 480:] = bfr(0.3 * rng.standard_normal((NH, DN, 32), dtype=np.float32))
    pair = rng.permuted(np.tile(np.arange(480), (NH * DV, 1)), axis=1)[:, :2].reshape(NH, DV, 2)
    for h in range(NH):
        for v in range(DV):
            j, k = pair[h, v]
            wkvb[h, DN + v, j], wkvb[h, DN + v, k] = const[k], -const[j]
    qkv = np.concatenate([bfr(rng.standard_normal(NH * (DN + DR), dtype=np.float32)), np.ones(C, np.float32), bfr(rng.standard_normal(DR, dtype=np.float32))])
    ln = np.concatenate([const, np.ones(32, np.float32)])                              # the new position's normed latent: the constants again
    nparts = op_mla.partitions(maxlen)
    tasks = NH * (nparts + op_mla.FINISHERS)
    t = {"qkv": dev_bf16(qkv), "kvln": dev_bf16(ln), "wkvb": dev_bf16(wkvb.reshape(-1, C)), "cos_sin": torch.from_numpy(M.yarn_table(d, maxlen)).to(DEV),
         "cache": dev_bf16(cache), "positions": torch.tensor([ctx], dtype=torch.int64, device=DEV), "out": torch.zeros(NH * DV, dtype=torch.bfloat16, device=DEV),
         "tmp": torch.zeros((op_mla.tmp_pairs(NH, C, maxlen), 2), dtype=torch.float32, device=DEV)}
    op_launch("mla_attn", argblock.pack_named(ops.all_entries()["mla_attn"], (tasks, 1, 1), **{n: v.data_ptr() for n, v in t.items()}, NH=NH, C=C, DN=DN, DR=DR, DV=DV,
                                              maxlen=maxlen, scale=d.scale, eps=d.eps, max_parts=nparts, tag=3), tasks)
    got = host(t["out"]).reshape(NH, DV)
    assert np.array_equal(host(t["cache"])[ctx, :480], const)
    size = const[pair[..., 0]] * const[pair[..., 1]]
    roundings = 2 * (8 + 16 + -(-(ctx + 1) // 128)) + 2
    assert np.isfinite(got).all() and np.abs(got).max() > 0 or ctx < 10
    assert (np.abs(got) <= 2 * roundings * 2.0 ** -24 * size).all(), np.abs(got / size).max()
