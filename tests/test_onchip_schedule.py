"""The on-chip CG solves' schedule (hf_plan_jobs): which blocks solve which scenes, against a plain restatement of the rule, and
what forming it costs on the host."""
import ctypes as C
import time

import numpy as np
import pytest


def _plan(edges, active=None, options=0, flags=0):
    from heatflow_mpm import _lib
    host = (_lib.Scene * len(edges))()
    for i, n in enumerate(edges):
        host[i].n = n
        host[i].flags = (_lib.HF_FLAG_ACTIVE if active is None or active[i] else 0) | flags
    plan = _lib.Plan()
    plan.num_scenes = len(edges)
    plan.scenes_host = C.cast(host, C.c_void_p)
    plan.options = options
    return plan, host


def _jobs(edges, sms=148, **kw):
    from heatflow_mpm import _lib
    plan, host = _plan(edges, **kw)
    out = (C.c_int32 * (4 * len(edges)))()
    count = _lib.load().hf_plan_jobs(C.byref(plan), sms, out)
    assert count >= 0
    return [tuple(out[4 * q:4 * q + 4]) for q in range(count)]


def _most(T, blocks):
    units = min(T, 148)
    first = [T * (units * b // blocks) // units for b in range(blocks + 1)]
    return max(b - a for a, b in zip(first, first[1:]))


def _restated(edges, sms, active):
    """As few blocks as hold each scene (15 tiles a block, else 36); when all fit side by side the rest goes, one by one, to the
    scene with the most tiles a block; then the largest first, each where the blocks are free the soonest."""
    from heatflow_mpm import _lib
    L, blocks = _lib.load(), min(sms, 148)
    tiles = {s: L.hf_tiles_for(n) for s, n in enumerate(edges) if active[s]}
    for cap in (15, 36):
        want = {}
        for s, T in tiles.items():
            nb = -(-T // cap)
            while nb <= min(blocks, T) and _most(T, nb) > cap:
                nb += 1
            want[s] = nb
        if tiles and all(nb <= min(blocks, tiles[s]) for s, nb in want.items()):
            break
    else:
        return []
    while sum(want.values()) < blocks:
        room = [s for s in want if want[s] < min(blocks, tiles[s])]
        if not room:
            break
        most = room[0]
        for s in room[1:]:
            if tiles[s] * want[most] > tiles[most] * want[s]:
                most = s
        want[most] += 1
    until, out = np.zeros(blocks), []
    for s in sorted(want, key=lambda s: -tiles[s]):
        free = [until[f:f + want[s]].max() for f in range(blocks - want[s] + 1)]
        at, most = int(np.argmin(free)), _most(tiles[s], want[s])
        until[at:at + want[s]] = free[at] + edges[s] * (1.6 + 0.35 * most)
        out.append((s, at, want[s], most))
    return out


@pytest.mark.parametrize("edges", [(2,), (96,), (128,), (129,), (168,), (169,), (20, 33, 47), (96, 96), (120, 120), (136, 40, 88),
                                   (168, 2), (170, 12)], ids=str)
def test_schedule_is_the_rules(edges):
    assert _jobs(edges) == _restated(edges, 148, [True] * len(edges))


def test_schedule_of_batches_is_the_rules():
    rng = np.random.default_rng(2)
    for count in (5, 12, 64, 200):
        for top in (24, 64, 128, 168):
            edges = [int(n) for n in rng.integers(2, top + 1, count)]
            active = [bool(a) for a in rng.random(count) < 0.8]
            sms = int(rng.choice([148, 132, 160, 40]))
            assert _jobs(edges, sms, active=active) == _restated(edges, sms, active), (edges, active, sms)


def test_plans_that_stream_have_no_jobs():
    from heatflow_mpm import _lib
    assert _jobs((96, 32)) and not _jobs((96, 32), options=_lib.HF_PLAN_STREAMING_CG)
    assert not _jobs((96, 32), flags=_lib.HF_FLAG_DEFECT_CORRECTION)
    assert not _jobs((0, 32)) and not _jobs((96, 200)) and _jobs((96, 200), active=(True, False))
    assert _lib.load().hf_plan_jobs(None, 148, None) == -1


def test_schedule_costs_little_on_the_host():
    """Direct launches form the teams twice a substep, and every upload the whole schedule: 1024 scenes took 8 ms, most of it
    in the search for free blocks, which is linear in the blocks now (a few ns for each scene and block)."""
    from heatflow_mpm import _lib
    L = _lib.load()
    edges = [int(n) for n in np.random.default_rng(3).choice([32, 48, 64, 96, 128], 1024)]
    plan, host = _plan(edges)
    out = (C.c_int32 * (4 * len(edges)))()
    best = 1.0
    for _ in range(9):
        t0 = time.perf_counter()
        assert L.hf_plan_jobs(C.byref(plan), 148, out) == 1024
        best = min(best, time.perf_counter() - t0)
    assert best < 4e-3, best
