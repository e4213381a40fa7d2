"""The resident kernels on a device that holds fewer of their blocks than the
whole part (a partition), in launches of few sweeps (a level that needs several),
and with a barrier whose wait runs out (other work holds blocks back: the class
kernels take over).  The limits are set on the host; no result depends on them.
Bar: the oracle's run bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(a, b):
    assert (a["level_sizes"] == b["level_sizes"]).all() and a["iterations"] == b["iterations"]
    assert (a["trace"] == b["trace"]).all() and a["modularity"] == b["modularity"]
    assert (a["assignment"] == b["assignment"]).all()


@pytest.fixture(scope="module")
def graphs(O):
    hub = O.csr_from_pairs(5001, np.zeros(5000, np.int64), np.arange(1, 5001))
    gs = [O.gen_sbm(20011, 40, 12.0, 0.7, seed=5), O.gen_rmat(12, seed=3), O.gen_sbm(300, 3, 9.0, 0.8, seed=1), hub]
    return gs, [O.louvain(g) for g in gs]


@pytest.fixture
def limited(ctx):
    yield ctx
    ctx.resident_limits()


def _check(ctx, graphs):
    gs, refs = graphs
    launches = []
    for g, ref in zip(gs, refs):
        dg = ctx.graph_from_csr(g.n, g.offsets, g.cols, g.weights)
        a = dg.louvain()
        _same(a, ref)
        launches.append(a["kernel_launches"])
        dg.close()
    b = ctx.batch_from_csr([(g.n, g.offsets, g.cols, g.weights) for g in gs])
    r = b.run()
    b.close()
    for i, ref in enumerate(refs):
        assert r["graphs"]["modularity"][i] == ref["modularity"] and r["graphs"]["iterations"][i] == ref["iterations"]
        assert (r["assignments"][i] == ref["assignment"]).all()
    return launches, r["kernel_launches"]


@pytest.mark.parametrize("sms", [0, 1, 2, 3, 7, 8, 9, 20, 100, 147, 148, 1000])
def test_few_sms(limited, graphs, sms):
    whole = _check(limited, graphs)
    limited.resident_limits(sms=sms)
    part = _check(limited, graphs)
    if sms == 0:  # the class kernels: launches for every sweep
        assert all(a < b for a, b in zip(whole[0], part[0])) and whole[1] < part[1]
    else:
        assert whole[0] == part[0]


@pytest.mark.parametrize("sweeps", [1, 2, 7])
def test_few_sweeps_per_launch(limited, graphs, sweeps):
    whole = _check(limited, graphs)
    limited.resident_limits(sweeps=sweeps)
    part = _check(limited, graphs)
    assert whole[0][0] < part[0][0] and whole[1] < part[1]


def test_more_sweeps_than_a_launch_holds(O, ctx):
    g = O.gen_sbm(40009, 30, 10.0, 0.6, seed=13)
    ref = O.louvain(g)
    phase = ref["trace"][:, 0]
    assert max((phase == p).sum() for p in np.unique(phase)) > 48
    dg = ctx.graph_from_csr(g.n, g.offsets, g.cols, None)
    _same(dg.louvain(), ref)
    dg.close()


@pytest.mark.parametrize("polls", [1, 3])
def test_barrier_wait_runs_out(limited, graphs, polls):
    limited.resident_limits(polls=polls)
    _check(limited, graphs)
    limited.resident_limits()
    _check(limited, graphs)
