"""The host-buffer token loop when a step in the middle of it fails: the call ends with the step's error, the tokens before it are there, and the session can
be used again."""
import numpy as np
import pytest
import torch

from etx_megakernel_b200.models import decode as D
from etx_megakernel_b200.models import qwen as Q
from etx_megakernel_b200.runtime import Session
from etx_megakernel_b200.runtime import lib as L

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
DIMS = Q.Dims(name="loop", H=512, NH=4, NKV=1, HD=128, INTER=0, L=2, V=1000, qk_norm=True, moe=True, E=16, TOPK=4, MI=128, norm_topk=True)


def loop(session, tokens_in, n_total, start):
    """The C call: (status, tokens of the steps that ran, device ms per step)."""
    import ctypes as C
    tin, out, ms = np.asarray(tokens_in, np.int32), np.full(n_total, -7, np.int32), np.zeros(n_total, np.float32)
    rc = session.lib.etxb_decode_host(session._h, tin.ctypes.data_as(C.c_void_p), len(tin), n_total, start, out.ctypes.data_as(C.c_void_p), ms.ctypes.data_as(C.c_void_p))
    return L.STATUS[rc], out, ms


def test_a_step_that_runs_out_of_time(monkeypatch):
    """From 257 positions on a merge waits for the partitions' partials; here its task stands before one of theirs in a queue.  The first two steps are of 255
    and 256 positions, the third waits until the device's time limit."""
    w = D.random_packed_weights(DIMS, 400, DEV, seed=9)
    prog = D.DecodeProgram(DIMS, w, device=0, maxlen=400)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1)
    prog.buf["kc"].normal_(0, 1, generator=gen)
    prog.buf["vc"].normal_(0, 1, generator=gen)
    kc, vc = prog.buf["kc"].clone(), prog.buf["vc"].clone()

    def refill():
        prog.buf["kc"].copy_(kc)
        prog.buf["vc"].copy_(vc)
        torch.cuda.synchronize()
    status, want, _ = loop(prog.session, [5, 6], 6, 254)
    assert status == "OK" and (want >= 0).all()
    refill()
    status, early, _ = loop(prog.session, [5, 6], 4, 20)
    assert status == "OK"

    plan = prog.plan
    tasks = [i for i, t in enumerate(plan.tasks) if t.grid == "attn_0"]
    assert len(tasks) % 4 == 0                                      # four partitions of the same groups, in order
    queue = {t: k for k, q in plan.static_queues.items() for t in q}
    first, merging = tasks[0], tasks[2 * (len(tasks) // 4)]
    plan.static_queues[queue[merging]].remove(merging)
    q = plan.static_queues[queue[first]]
    q.insert(q.index(first), merging)
    s, b = Session(plan, {"vl": prog.vl}, prog.pool.bytes(), 0), prog.buf
    s.set_step(tok=0, pos=0, write_next=0, H=DIMS.H, V=DIMS.lm_rows, nrep=1, embed=prog.w["embed"], resid=b["resid"], positions=b["positions"],
               seq_lens=b["seq_lens"], slot_mapping=b["slot_mapping"], logits=b["logits"], token_in=b["token_in"], token_out=b["token_out"],
               token_time=b["token_time"])
    s.set_option("timeout_ms", 200)
    for _ in range(2):
        refill()
        status, got, ms = loop(s, [5, 6], 6, 254)
        assert status == "E_TIMEOUT" and "step" in L.load().etxb_last_error().decode()
        assert got[:2].tolist() == want[:2].tolist() and (got[2:] == -7).all() and (ms[:1] > 0).all()
        refill()
        status, got, ms = loop(s, [5, 6], 4, 20)                   # (short contexts: no merge)
        assert status == "OK" and got.tolist() == early.tolist() and (ms > 0).all() and (ms < 100).all()
        s.set_step(tok=0, pos=20, write_next=0)                    # the session's own slots, as after any step
        b["token_in"][0] = 5
        torch.cuda.synchronize()
        s.run(5.0)
        assert int(b["token_out"][0]) == int(early[0])
    s.close()
    prog.close()
