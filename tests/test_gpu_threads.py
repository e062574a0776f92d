"""Calls from several threads: one thread builds the graphs of GPU_LOOP contexts and
of batches, others destroy contexts, free cached memory and synchronise the device
meanwhile. Every result is the single-threaded one."""
import threading

import numpy as np
import pytest

import gdp
import gdpgen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _answer(lb, ub, st):
    return lb.tobytes(), ub.tobytes(), st["rounds"]


def test_graphs_are_built_while_others_synchronise():
    mips = [gdpgen.random_mip(0, seed=1, m=m, n=3 * m // 4) for m in (30, 400, 2_000)]
    mips.append(gdpgen.random_mip(1, seed=2, m=3_000, n=2_200))
    expect = []
    for p in mips:
        with gdp.Context(p, sync_type=gdp.MEGAKERNEL) as ctx:
            expect.append(_answer(*ctx.propagate()))
    x = np.random.default_rng(0).normal(size=(1000, 16)).astype(np.float32)
    z = gdp.Mlp(seed=3).forward(x)
    stop, wrong = threading.Event(), []

    def guard(f):
        def run(*a):
            try:
                f(*a)
            except Exception as e:  # a thread's failure is the test's
                wrong.append(repr(e))
        return run

    @guard
    def graphs(first):
        for k in range(40):
            i = (first + k) % len(mips)
            with gdp.Context(mips[i], sync_type=gdp.GPU_LOOP) as ctx:
                if _answer(*ctx.propagate()) != expect[i]:
                    wrong.append(("loop", i))
            batch = gdp.Batch.instances([mips[i], mips[0]])
            lbs, ubs, sts, _ = batch.propagate([mips[i].lb, mips[0].lb], [mips[i].ub, mips[0].ub])
            if not batch.uses_graph or _answer(lbs[0], ubs[0], sts[0]) != expect[i]:
                wrong.append(("batch", i))
            batch.close()

    @guard
    def contexts():
        while not stop.is_set():
            for i, p in enumerate(mips):
                if _answer(*gdp.propagate(p)) != expect[i]:
                    wrong.append(("call", i))
            gdp.release_cached_memory()

    @guard
    def others():
        m = gdp.Mlp(seed=3)
        while not stop.is_set():
            torch.cuda.synchronize()
            if not np.array_equal(m.forward(x), z):
                wrong.append("forward")

    back = [threading.Thread(target=f) for f in (contexts, contexts, others, others)]
    front = [threading.Thread(target=graphs, args=(k,)) for k in range(3)]
    for t in back + front:
        t.start()
    for t in front:
        t.join()
    stop.set()
    for t in back:
        t.join()
    assert not wrong, wrong[:5]
