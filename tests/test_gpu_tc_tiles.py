"""The tensor-core tiles of a batched step on their own, at the sizes where a run of 64-row units, a prefill for the next expert
or a window of K can go wrong: rows that end inside a unit, neighbouring experts whose token counts cross 8 and 32 (another
number of weight stages on either side of the prefill), an expert that takes two passes behind one that takes one, fewer
k-chunks than stages, K in windows."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import etx_megakernel_b200  # noqa: E402,F401
from etx_megakernel_b200 import ops  # noqa: E402
from etx_megakernel_b200.frontends import cuda_link  # noqa: E402
from etx_megakernel_b200.importer import argblock  # noqa: E402
from etx_megakernel_b200.ir import Graph  # noqa: E402
from etx_megakernel_b200.passes import compile_graph  # noqa: E402
from etx_megakernel_b200.runtime import Session  # noqa: E402
from oracle import ref_decode as O  # noqa: E402
from tests.test_gpu_ops import assert_bf16_close, dev_bf16, host  # noqa: E402

ENT = ops.all_entries()
DEV = "cuda:0"


def run_grid(export, tasks, **fields):
    blob = argblock.pack_named(ENT[export], (tasks, 1, 1), **fields)
    g = Graph(f"one_{export}")
    g.tensor("impargs", (len(blob),), role="weight", bytes_per_elem=1)
    g.etensor("E_done", (1,), wait_count=tasks)
    g.call_device("grid", (tasks,), cuda_link("", f"etx_tile_{export}"), args=["impargs"], consts=(0, 0), out_edges={"E_done": "i->(0)"})
    s = Session(compile_graph(g, "b200", {}), {}, blob, 0)
    assert s.status().kernel_variant == 11
    for _ in range(2):                                        # twice: the barriers' phases carry on inside a launch only
        s.run(10.0)
    s.close()


def matmul(W, X):
    """[rows][K] . [tokens][K] -> [tokens][rows], fp64 sums of bf16 values rounded once."""
    return O.bfr((X.astype(np.float64) @ W.astype(np.float64).T).astype(np.float32))


@pytest.mark.parametrize("M,K", [(77, 64), (320, 2112), (200, 4160)])
@pytest.mark.parametrize("nb", [9, 40])
def test_dense_tile_with_ragged_rows_passes_and_windows(M, K, nb):
    rng = np.random.default_rng(M + K + nb)
    W, x = O.bfr(rng.standard_normal((M, K), dtype=np.float32) * np.float32(0.02)), O.bfr(rng.standard_normal((nb, K), dtype=np.float32))
    Wd, xd, out = dev_bf16(W), dev_bf16(x), torch.zeros((nb + 1, M), dtype=torch.bfloat16, device=DEV)
    run_grid("gemv_tc", -(-M // 256), W=Wd.data_ptr(), x=xd.data_ptr(), out=out.data_ptr(), M=M, K=K, rpt=256, tpe=1, nb=nb, sx=K, sout=M)
    # fp32 sums against fp64 sums: a result near a rounding boundary may go to the neighbouring bf16 value
    assert_bf16_close(host(out)[:nb], matmul(W, x), f"M={M} K={K} nb={nb}", min_exact=0.97)
    assert not host(out)[nb:].any()                           # nothing behind the last column


def routing(nb, E):
    """Two slots per column: slot 0 is expert 3 for everybody (40 tokens: two passes), slot 1 gives the experts 0, 1, 2, 4 and 6
    1, 9, 8, 5 and 17 tokens; 5 and 7 have none."""
    slot1 = np.repeat([0, 1, 2, 4, 6], [1, 9, 8, 5, 17])
    assert nb == len(slot1) == 40 and E == 8
    return np.stack([np.full(nb, 3), np.random.default_rng(7).permutation(slot1)], 1).astype(np.int32)


@pytest.mark.parametrize("M,K", [(64, 128), (100, 2112), (200, 512)])
@pytest.mark.parametrize("tasks", [1, 3, 148])
def test_expert_tiles_across_experts_of_different_token_counts(M, K, tasks):
    """One task that walks all experts, three, and one per worker (most of them with less than a unit)."""
    nb, R, E = 40, 2, 8
    rng = np.random.default_rng(M + K)
    ids = routing(nb, E)
    wts = O.bfr(rng.random((nb, R), dtype=np.float32))
    x = O.bfr(rng.standard_normal((nb, K), dtype=np.float32))
    w13 = O.bfr(rng.standard_normal((E, 2 * M, K), dtype=np.float32) * np.float32(0.02))
    idd, wtd = torch.from_numpy(ids).to(DEV), torch.from_numpy(wts).to(DEV)
    xd, wd = dev_bf16(x), dev_bf16(w13)
    act, active = torch.zeros((nb * R + 1, M), dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    run_grid("moe_up_tc", tasks, E=E, W=wd.data_ptr(), x=xd.data_ptr(), out=act.data_ptr(), estride=2 * M * K, M=M, K=K, rpt=128, tpe=-(-M // 128),
             ids=idd.data_ptr(), resid_out=active.data_ptr(), nb=nb, R=R, sx=K)
    got = host(act)
    assert int(active) == 2 * 6 and not got[nb * R:].any()    # six experts with tokens, counted in both runs
    g, u = (np.stack([matmul(w13[e, h * M:(h + 1) * M], x[c:c + 1])[0] for c in range(nb) for e in ids[c]]) for h in (0, 1))
    want = O.bfr(O.bfr(O.silu(g)) * u)
    # three roundings that may each go to the neighbouring bf16 value (2^-7 of the value at most), the gate's amplified by silu's
    # slope (at most 1.1), and the silu of the device against numpy's
    d = np.abs(got[:nb * R] - want)
    assert np.all(d <= 4 * 2.0 ** -7 * np.abs(want) + np.abs(want).max() / 4096) and np.mean(d == 0) >= 0.95
    # down: its own rows per (column, slot), each scaled by the routing weight
    a = O.bfr(rng.standard_normal((nb * R, K), dtype=np.float32))
    w2 = O.bfr(rng.standard_normal((E, M, K), dtype=np.float32) * np.float32(0.02))
    ad, w2d, out = dev_bf16(a), dev_bf16(w2), torch.zeros((nb * R + 1, M), dtype=torch.bfloat16, device=DEV)
    run_grid("moe_down_tc", tasks, E=E, W=w2d.data_ptr(), x=ad.data_ptr(), out=out.data_ptr(), wts=wtd.data_ptr(), estride=M * K, M=M, K=K, rpt=256,
             tpe=-(-M // 256), ids=idd.data_ptr(), nb=nb, R=R)
    flat = ids.reshape(-1)
    want = O.bfr(np.stack([matmul(w2[flat[i]], a[i:i + 1])[0] for i in range(nb * R)]) * wts.reshape(-1, 1))
    assert_bf16_close(host(out)[:nb * R], want, f"down M={M} K={K} tasks={tasks}", min_exact=0.95)
    assert not host(out)[nb * R:].any()
