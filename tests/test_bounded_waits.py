"""Every device-side wait made to run out on its own: the context's limit is set to
one poll around the one call whose kernel waits, never around the calls that
prepare it. A call whose wait gives up fails with PG_ERR_TIMEOUT after its copies have
landed, and the next call with the built-in limit is right. The one-launch build's grid
barriers are the exception: the build returns before its kernel has run, so a barrier
that is given up on sends the table to the exact build and no call fails."""
import numpy as np
import pytest

from oracle import oracle as orc
from pythia_gb300 import datagen as dg
from pythia_gb300 import gpu

pytestmark = pytest.mark.gpu

PG_ERR_TIMEOUT = 4


def _case(ctx, op):
    """(call, check of its result, knobs that pick the kernel)."""
    if op in ("tile_sort", "one_launch_sort"):
        rows = dg.uniform_keys(300_000, 1 << 40, dg.seed_for(401))
        want = np.sort(rows[:, 0])
        return (lambda: ctx.sort(rows), lambda got: np.array_equal(got[:, 0], want),
                dict(sort_path=2 if op == "tile_sort" else 0))
    if op in ("partition_16", "partition_24"):
        rows = dg.uniform_keys(300_000, 1 << 40, dg.seed_for(402))
        if op == "partition_24":
            rows = np.ascontiguousarray(np.concatenate([rows, rows[:, 1:]], axis=1))
        want, _ = orc.partition(rows, orc.hashcfg("parammodulo", 256))
        return (lambda: ctx.partition(rows, gpu.hashcfg("parammodulo", 256))[0],
                lambda got: np.array_equal(got.view(np.uint8), want.view(np.uint8)), {})
    if op in ("filter", "project"):
        rows = dg.uniform_keys(1_000_003, 1000, dg.seed_for(403))
        if op == "filter":
            want = rows[rows[:, 0] < 300]
            return (lambda: ctx.filter(rows, [("long", "<", 0, 300)]), lambda got: np.array_equal(got, want), {})
        return (lambda: ctx.project(rows, [(8, 8)]),
                lambda got: np.array_equal(np.ascontiguousarray(got).view(np.int64)[:, 0], rows[:, 1]), {})
    R = dg.build_relation(70_000, dg.seed_for(404))
    S = dg.probe_uniform(500_000, R, dg.seed_for(405))
    t = ctx.build_table(R)
    t.probe(S[:10])                                     # built and settled
    want, _, _ = orc.hashjoin(R, S, hash=orc.hashcfg("modulo", 1 << 16))
    want = orc.canonical(want)
    return (lambda: t.probe(S)[0], lambda got: np.array_equal(orc.canonical(got), want), dict(probe_variant=1))


@pytest.mark.parametrize("op", ["tile_sort", "one_launch_sort", "partition_16", "partition_24", "filter", "project",
                                "staged_probe"])
def test_each_wait_gives_up_and_the_next_call_succeeds(ctx, op):
    call, right, knobs = _case(ctx, op)
    ctx.tune(spin_limit=1, **knobs)
    try:
        with pytest.raises(gpu.PgError) as err:
            call()
        assert err.value.code == PG_ERR_TIMEOUT
        ctx.tune(spin_limit=0)
        assert right(call())
    finally:
        ctx.tune(spin_limit=0, **{k: 0 for k in knobs})


@pytest.mark.parametrize("n", [2048, 2049, 3000, 70_001, 1 << 20])
@pytest.mark.parametrize("case", ["dense", "far", "repeated", "wide"])
def test_a_build_that_gives_up_on_its_barriers_is_made_again(ctx, n, case):
    R = dg.build_relation(n, dg.seed_for(406))
    S = dg.probe_uniform(2000, R, dg.seed_for(407))
    if case == "far":
        R[:, 0] *= -7046029254386353131
        S[:, 0] *= -7046029254386353131
    elif case == "repeated":
        R[n // 2:, 0] = R[: n - n // 2, 0]
    elif case == "wide":
        R[0, 1] = -5
    order = np.argsort(R[:, 0], kind="stable")
    keys, vals = R[order, 0], R[order, 1].astype(np.uint64)
    lo, hi = np.searchsorted(keys, S[:, 0], "left"), np.searchsorted(keys, S[:, 0], "right")
    pre = np.concatenate([np.zeros(1, np.uint64), np.cumsum(vals, dtype=np.uint64)])
    want = (int((hi - lo).sum()), int((pre[hi] - pre[lo]).sum(dtype=np.uint64).astype(np.int64)))
    ctx.tune(spin_limit=1)
    try:
        t = ctx.build_table(R)
        ctx.sync()
        assert gpu.lib().pg_device_status(ctx.h) == 0   # no other call is failed for it
    finally:
        ctx.tune(spin_limit=0)
    try:
        for _ in range(2):
            _, count, total = t.probe(S, flags=gpu.JOIN_COUNT | gpu.JOIN_SUM, sum_col=1)
            assert (count, total) == want
    finally:
        t.free()
