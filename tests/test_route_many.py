"""FlowRouter.route_many: a sequence of DEMs routed with the copies of neighbouring
DEMs overlapped on copy streams gives, for every DEM, exactly the results of the
plain call sequence."""
import numpy as np
import pytest

from pyfastflow_b200 import synthetic


@pytest.mark.gpu
def test_route_many_matches_single_calls(cuda):
    torch = cuda
    import pyfastflow_b200 as pf

    n = 256
    dems = [synthetic.routing_lakes(n, seed=s)["z"] for s in (3, 4, 5, 3)]
    ws = [synthetic.lognormal_weights(n * n, 10 + k) for k in range(4)]
    r = pf.flow.FlowRouter(n, n, 30.0, boundary_mode="periodic_EW")
    zh = [torch.from_numpy(d.ravel().copy()).pin_memory() for d in dems]
    wh = [torch.from_numpy(w.copy()).pin_memory() for w in ws]
    qh = [torch.empty(n * n, dtype=torch.float32).pin_memory() for _ in dems]
    ch = [torch.empty(n * n, dtype=torch.int32).pin_memory() for _ in dems]
    r.route_many(zh, wh, qh, ch)
    torch.cuda.synchronize()
    for k, d in enumerate(dems):
        r1 = pf.flow.FlowRouter(n, n, 30.0, boundary_mode="periodic_EW")
        r1.set_z(d)
        r1.compute_receivers()
        r1.reroute_flow()
        r1.accumulate_weighted_Q(ws[k])
        torch.cuda.synchronize()
        assert np.array_equal(qh[k].numpy().view(np.uint32), r1.Q.cpu().numpy().view(np.uint32)), k
        assert np.array_equal(ch[k].numpy(), r1.counts.cpu().numpy()), k


@pytest.mark.gpu
@pytest.mark.parametrize("failing", [(0,), (1, 2), (0, 1, 2, 3, 4)])
@pytest.mark.parametrize("weighted", [False, True])
def test_route_many_repeats_a_refused_accumulation(cuda, failing, weighted):
    """A nonzero status after the next DEM's fields are queued: the results are still those
    of every DEM's own seeds, bit for bit.  The status is made up on the host."""
    torch = cuda
    import pyfastflow_b200 as pf

    n = 96
    dems = [synthetic.routing_lakes(n, seed=s)["z"] for s in (3, 4, 5, 6, 7)]
    zh = [torch.from_numpy(d.ravel().copy()).pin_memory() for d in dems]
    wh = [torch.from_numpy(synthetic.lognormal_weights(n * n, 10 + k)).pin_memory() for k in range(5)]

    def run(fail):
        qh = [torch.empty(n * n, dtype=torch.float32).pin_memory() for _ in dems]
        ch = [torch.empty(n * n, dtype=torch.int32).pin_memory() for _ in dems]
        r = pf.flow.FlowRouter(n, n, 30.0)
        begin, calls = r._accumulate_begin, []

        def refused():
            calls.append(0)
            if len(calls) - 1 not in fail:
                return begin()
            r.counts.fill_(-1)
            return lambda: 4

        r._accumulate_begin = refused
        r.route_many(zh, wh if weighted else None, qh, ch)
        torch.cuda.synchronize()
        return qh, ch

    for a, b in zip(run(()), run(failing)):
        for k in range(5):
            assert torch.equal(a[k].view(torch.int32), b[k].view(torch.int32)), k


@pytest.mark.gpu
def test_route_many_with_seeds_the_tree_refuses(cuda):
    """An infinite weight: the results of the plain call, and no second tree pass."""
    torch = cuda
    import pyfastflow_b200 as pf
    from pyfastflow_b200 import _lib

    n = 96
    zh = [torch.from_numpy(synthetic.routing_lakes(n, seed=s)["z"].ravel().copy()).pin_memory() for s in (3, 4, 5)]
    wh = [torch.from_numpy(synthetic.lognormal_weights(n * n, 10 + k)).pin_memory() for k in range(3)]
    wh[1][n * 7 + 5] = float("inf")
    qh = [torch.empty(n * n).pin_memory() for _ in zh]
    ch = [torch.empty(n * n, dtype=torch.int32).pin_memory() for _ in zh]
    r = pf.flow.FlowRouter(n, n, 30.0)
    r.route_many(zh, wh, qh, ch)
    torch.cuda.synchronize()
    for k in range(3):
        r1 = pf.flow.FlowRouter(n, n, 30.0)
        r1.set_z(zh[k])
        r1.compute_receivers()
        r1.reroute_flow()
        r1.accumulate_weighted_Q(wh[k])
        assert torch.equal(qh[k].view(torch.int32), r1.Q.cpu().view(torch.int32)), k
        assert torch.equal(ch[k], r1.counts.cpu()), k
    assert torch.isinf(qh[1]).any()

    def launches(f, *a, **kw):
        l0 = _lib.load().pff_launch_count()
        f(*a, **kw)
        return _lib.load().pff_launch_count() - l0

    rounds = launches(r1.accumulate_weighted_Q, wh[1], exact_order=True)
    plain = launches(r.route_many, zh[1:2], wh[:1], qh[:1], ch[:1])
    assert launches(r.route_many, zh[1:2], wh[1:2], qh[:1], ch[:1]) == plain + rounds


@pytest.mark.gpu
def test_route_many_delivers_nothing_of_a_failed_accumulation(cuda):
    """A status read that raises (made on the host): that DEM's buffers stay as they were."""
    torch = cuda
    import pyfastflow_b200 as pf
    from pyfastflow_b200 import _lib

    n = 96
    zh = [torch.from_numpy(synthetic.routing_lakes(n, seed=s)["z"].ravel().copy()).pin_memory() for s in (3, 4, 5)]
    qh = [torch.full((n * n,), -1.0).pin_memory() for _ in zh]
    r = pf.flow.FlowRouter(n, n, 30.0)
    begin, calls = r._accumulate_begin, []

    def failing():
        calls.append(0)
        read = begin()
        if len(calls) < 2:
            return read

        def fail():
            raise _lib.PFFError("made up")

        return fail

    r._accumulate_begin = failing
    with pytest.raises(_lib.PFFError, match="made up"):
        r.route_many(zh, None, qh)
    torch.cuda.synchronize()
    assert (qh[0] >= 1).all() and (qh[1] == -1).all() and (qh[2] == -1).all()
