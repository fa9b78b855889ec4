"""The one-token GEMV at the edges of its rule for sharing a stage between the warps (rows at once, warps per stage): the
widest row of each class, the next one, rows that fill a stage exactly or not, and several tasks behind each other on a
worker so that a stage changes hands between groups."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from oracle import ref_decode as O  # noqa: E402
from tests.test_gpu_ops import assert_bf16_close, gemv_case  # noqa: E402
from tests.test_gpu_ops import test_moe_block_grouped_slots_and_summed_down as moe_block_grouped  # noqa: E402


# K: 4 rows at once up to 1792 (7 vectors per lane), 3 up to 2048, one above; 24 KB stages hold 1536 / 6 / 3 / 1 of the rows
@pytest.mark.parametrize("K", [8, 512, 1536, 1792, 1800, 2048, 2056, 2736, 4096, 4104, 12288])
@pytest.mark.parametrize("N,tasks", [(3, 3), (148 * 7 + 3, 148), (148 * 37, 148 * 3 + 5)])
def test_rows_per_warp_classes(K, N, tasks):
    got, want = gemv_case(1, K, N, seed=K + N, tasks=tasks)
    # fp32 sums of K products in another order: a result may round to the neighbouring bf16 value when it lies within
    # the fp32 error of a rounding boundary, one in a few hundred
    assert_bf16_close(got, want, f"K={K} N={N} tasks={tasks}", min_exact=0.97 if N > 100 else 0.6)
    if N == 3:
        # too few for a share: each against its fp64 sum, half a bf16 ulp (2^-8 of the value at most) and the bound of a lane's
        # chain of K / 32 fp32 steps with the butterfly behind it
        rng = np.random.default_rng(K + N)
        W, x = O.bfr(rng.standard_normal((N, K), dtype=np.float32) * np.float32(0.02)), O.bfr(rng.standard_normal((1, K), dtype=np.float32))
        terms = W.astype(np.float64) * x.astype(np.float64)
        assert np.all(np.abs(got[0] - terms.sum(1)) <= 2.0 ** -8 * np.abs(terms.sum(1)) + (K / 32 + 8) * 2.0 ** -24 * np.abs(terms).sum(1))


# each slot with its own activation vector: 4 rows at once (short rows) and one (2048 and more), slots that straddle stages
@pytest.mark.parametrize("MI,slots", [(256, 4), (1792, 4), (2048, 2)])
def test_rows_with_a_vector_per_slot(MI, slots):
    moe_block_grouped(16, slots, MI, 512, slots)
