"""The dense tiles of a batched step that share a block of rows (split > 1): 16, 32, 64 and 128 rows a task and more than one sub-block,
rows that end inside a sub-block, chunks of K that fill a ring stage or not, tokens in one window and in several, two passes of tokens."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import ref_decode as O  # noqa: E402
from tests.test_gpu_ops import assert_bf16_close, dev_bf16, host  # noqa: E402
from tests.test_gpu_tc_tiles import DEV, run_grid  # noqa: E402


@pytest.mark.parametrize("M,K,rpt,S", [(128, 2048, 128, 8), (77, 1024, 128, 8), (700, 512, 256, 8), (1000, 448, 256, 7), (320, 4096, 256, 4), (520, 256, 256, 2),
                                       (900, 384, 512, 2)])
@pytest.mark.parametrize("nb", [1, 8, 13, 32, 40])
def test_rows_shared_between_tasks(M, K, rpt, S, nb):
    rng = np.random.default_rng(M + K + nb)
    W, x = O.bfr(rng.standard_normal((M, K), dtype=np.float32) * np.float32(0.02)), O.bfr(rng.standard_normal((nb, K), dtype=np.float32))
    bias = O.bfr(rng.standard_normal(M, dtype=np.float32))
    Wd, xd, bd, out = dev_bf16(W), dev_bf16(x), dev_bf16(bias), torch.zeros((nb + 1, M), dtype=torch.bfloat16, device=DEV)
    word = torch.zeros(64, dtype=torch.float32, device=DEV)
    run_grid("gemv_tc", -(-M // rpt) * S, W=Wd.data_ptr(), x=xd.data_ptr(), out=out.data_ptr(), M=M, K=K, rpt=rpt, tpe=S, nb=nb, sx=K, sout=M,
             rows=word.data_ptr(), resid_in=word.data_ptr(), wts=bd.data_ptr(), mode=0x200)
    # fp32 sums against fp64 sums: a result near a rounding boundary may go to the neighbouring bf16 value
    want = O.bfr((x.astype(np.float64) @ W.astype(np.float64).T + bias).astype(np.float32))
    assert_bf16_close(host(out)[:nb], want, f"M={M} K={K} nb={nb}", min_exact=0.97)
    assert not host(out)[nb:].any() and not word.any()        # nothing behind the last column, no partial sums


@pytest.mark.parametrize("nb", [5, 33])
def test_token_and_result_rows_further_apart_than_their_length(nb):
    M, K, rpt, S, sx, sout = 300, 512, 256, 4, 520, 311
    rng = np.random.default_rng(nb)
    W, x = O.bfr(rng.standard_normal((M, K), dtype=np.float32) * np.float32(0.02)), np.full((nb, sx), np.nan, np.float32)
    x[:, :K] = O.bfr(rng.standard_normal((nb, K), dtype=np.float32))
    Wd, xd, out = dev_bf16(W), dev_bf16(x), torch.full((nb, sout), 7.0, dtype=torch.bfloat16, device=DEV)
    word = torch.zeros(64, dtype=torch.float32, device=DEV)
    run_grid("gemv_tc", -(-M // rpt) * S, W=Wd.data_ptr(), x=xd.data_ptr(), out=out.data_ptr(), M=M, K=K, rpt=rpt, tpe=S, nb=nb, sx=sx, sout=sout,
             rows=word.data_ptr(), resid_in=word.data_ptr())
    want = O.bfr((x[:, :K].astype(np.float64) @ W.astype(np.float64).T).astype(np.float32))
    assert_bf16_close(host(out)[:, :M], want, f"nb={nb}", min_exact=0.97)
    assert (host(out)[:, M:] == 7.0).all()                    # nothing between the columns' rows
