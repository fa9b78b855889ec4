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
                                                   (12, 2, False, 1700, 2), (6, 2, True, 300, 1), (12, 1, False, 257, 4)])
def test_grouped_phase_with_other_head_counts(NH, NKV, qk_norm, seq, gq):
    from tests.test_gpu_ops import test_attention_phase_fused as phase
    phase(NH, NKV, 128, qk_norm, seq, gq)
