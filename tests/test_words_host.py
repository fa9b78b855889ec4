"""Programs that hand their vectors over as words: which bf16 vectors their grids still write."""
import pytest

from etx_megakernel_b200.models import dsv2 as M
from etx_megakernel_b200.models import qwen as Q


class Addresses:
    """name -> an address of its own"""

    def __init__(self):
        self.at = {}

    def __call__(self, name):
        return self.at.setdefault(name, 0x7a0000000000 + (len(self.at) << 28))


def uses(pool, at, name):
    return pool.count(at(name).to_bytes(8, "little"))


@pytest.mark.parametrize("model", ["moe", "dense", "latent"])
def test_one_grid_writes_each_vector(model):
    """Nothing orders the stores of two layers behind relaxed arrivals, so a buffer that the caller reads when the step is over has one writer: the last
    layer's grid, or the lm_head's norm fold."""
    at = Addresses()
    if model == "latent":
        d = M.load_dims("deepseek-v2-lite", layers=4)
        pool = M.build_graph(d, at, 300, words=True)[1].bytes()
    else:
        d = Q.Dims(name="w", H=512, NH=8, NKV=2, HD=128, INTER=0 if model == "moe" else 768, L=4, V=1000, qk_norm=True, moe=model == "moe", E=16 if model == "moe" else 0,
                   TOPK=4 if model == "moe" else 0, MI=128 if model == "moe" else 0, norm_topk=True)
        pool = Q.build_graph(d, at, 300, words=True)[1].bytes()
    for name in ("qkv", "attn_out", "o", "resid2", "o_norm", "mc2", "moe_out", "hn", "logits"):
        assert uses(pool, at, name) == 1, name
    if model != "dense":
        assert uses(pool, at, "rlog") == 1
    assert uses(pool, at, "resid") == 2                             # (the first layer reads what the prologue wrote, the lm_head's fold writes)
