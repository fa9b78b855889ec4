"""One plan that holds tcgen05 tiles and streamed GEMVs: the tensor-core tiles take the weight ring's memory for their own tokens and weights, so a later
task's rows may not be copied into it while one of them runs."""
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

DEV = "cuda:0"


@pytest.mark.parametrize("K,nb", [(2048, 4), (4096, 40)])
def test_streamed_rows_wait_for_the_tensor_core_tile(K, nb):
    """Every worker's queue: GEMV, tcgen05 tile, narrow tile (tasks of the first workers), GEMV, tcgen05 tile -- no edges between them, static weights, so that only
    the queue keeps the copies of one from the memory of the other."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(K)
    W = 148
    pool, grids, checks = b"", [], []
    for name, export, M, rpt, S in (("g0", "dsl_gemv", W * 9, 9, 1), ("t0", "gemv_tc", W * 256, 256, 1), ("n0", "gemv_tc", 2048, 256, 8), ("g1", "dsl_gemv", W * 11, 11, 1),
                                    ("t1", "gemv_tc", W * 64, 64, 1)):
        b = nb if export == "gemv_tc" else 1
        w = torch.empty((M, K), device=DEV).normal_(0.0, 0.02, generator=gen).to(torch.bfloat16)
        x = torch.empty((b, K), device=DEV).normal_(0.0, 1.0, generator=gen).to(torch.bfloat16)
        out, word = torch.zeros((b, M), dtype=torch.bfloat16, device=DEV), torch.zeros(64, device=DEV)
        tasks = -(-M // rpt) * S
        grids.append((name, export, tasks, len(pool)))
        pool += argblock.pack_named(ops.all_entries()[export], (tasks, 1, 1), W=w.data_ptr(), x=x.data_ptr(), out=out.data_ptr(), M=M, K=K, rpt=rpt, tpe=S, nb=b, sx=K, sout=M,
                                    rows=word.data_ptr(), resid_in=word.data_ptr())
        checks.append((name, w, x, out, word))
    g = Graph("mixed")
    g.tensor("impargs", (len(pool),), role="weight", bytes_per_elem=1)
    for name, export, tasks, off in grids:
        g.etensor("E_" + name, (1,), wait_count=tasks)
        g.call_device(name, (tasks,), cuda_link("", "etx_tile_" + export, stream_after=""), args=["impargs"], consts=(off, 0), out_edges={"E_" + name: "i->(0)"})
    s = Session(compile_graph(g, "b200", {}), {}, pool, 0)
    assert s.status().kernel_variant == 0
    for _ in range(4):
        for _, _, _, out, _ in checks:
            out.zero_()
        torch.cuda.synchronize()
        s.run(10.0)
        for name, w, x, out, _ in checks:
            want = x.double() @ w.double().T
            # the result's rounding to bf16 (2^-9 of it) and fp32 sums of K products
            assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -18 * want.abs().max()).all()), name
    s.close()
