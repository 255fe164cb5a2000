"""A round's statistics are whole once the round is over, whatever ends the rounds: the last one asked for or a
cancellation that the next one meets."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

from cartogenesis_gb300 import ErosionConfig, StageRounds, abi, synthetic
from cartogenesis_gb300.api import P, default_context

pytestmark = pytest.mark.gpu

TIMES = ["ms_total", "ms_cut", "ms_fill", "ms_route", "ms_tree", "ms_incise", "ms_relax"]


def check(stats):
    for s in stats:
        assert all(getattr(s, t) > 0.0 for t in TIMES), (s.round, [getattr(s, t) for t in TIMES])
        assert s.ms_total < 1e4


@pytest.mark.parametrize("profile", [0, 3])
def test_cancelled(profile):
    W, H, rounds, seed = 512, 256, 400, 5
    h, up, rk = synthetic.world(W, H, seed)
    cfg = ErosionConfig(W, H, seed, sea_level=0.70, hydraulic_rounds=rounds, profile=profile)
    ctx = default_context()
    out = np.empty((H, W), np.float32)
    inputs, outputs = abi.Inputs(P(h), P(up), P(rk), None, None), abi.Outputs(height=P(out))
    stats = (abi.RoundStats * rounds)()
    status = []
    with ctx.lock:
        stage = threading.Thread(target=lambda: status.append(
            ctx.lib.cg_erode_stage(ctx.handle, C.byref(cfg.params), C.byref(inputs), C.byref(outputs),
                                   C.cast(stats, C.c_void_p))))
        stage.start()
        until = time.monotonic() + 60.0
        while stats[2].kernel_launches == 0 and stage.is_alive() and time.monotonic() < until:
            pass
        ctx.lib.cg_cancel(ctx.handle)
        stage.join()
    assert status == [abi.CG_CANCELLED]
    run = [s for s in stats if s.kernel_launches > 0]
    assert 3 <= len(run) < rounds
    check(run)


@pytest.mark.parametrize("ends", [(1, 2, 5), (5,)])
def test_every_round_asked_for(ends):
    W, H, seed = 256, 128, 5
    h, up, rk = synthetic.world(W, H, seed)
    cfg = ErosionConfig(W, H, seed, sea_level=0.70, hydraulic_rounds=5)
    run = StageRounds(cfg, h, up, rk)
    for end in ends:
        first = run.next_round
        stats = run.rounds(end)
        assert [s["round"] for s in stats] == list(range(first, end))
        for s in stats:
            assert all(s[t] > 0.0 for t in TIMES)
