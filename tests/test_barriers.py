"""Barriers between the blocks of a cooperative launch that give up: the call reports it,
nothing is taken for a result, and the next call works.  The waits run out because one
more block is awaited than there is, or because their limit is about as long as the blocks
are apart."""
import numpy as np
import pytest

from pyfastflow_b200 import synthetic

REROUTE, LABELS, TREE, ROUNDS = 1, 2, 4, 8


@pytest.fixture
def barrier_test():
    from pyfastflow_b200 import _lib

    yield lambda *a: _lib.call("pff_barrier_test", *a)
    _lib.call("pff_barrier_test", 0, 0, 0)


def test_barrier_test_arguments():
    from pyfastflow_b200 import _lib

    lib = _lib.load()
    for bad in ((-1, 0, 1), (16, 0, 1), (1, 2, 1), (1, -1, 1), (1, 0, 0), (1, 0, 2000001)):
        assert lib.pff_barrier_test(*bad) == 1, bad
    assert lib.pff_barrier_test(0, 0, 0) == 0


def router(nx, ny):
    from pyfastflow_b200.flow import FlowRouter

    r = FlowRouter(nx, ny, 30.0)
    r.set_z(synthetic.spectral_dem(nx, ny, 1, relief=300.0, npits=nx * ny // 400, pit_scale=0.1))
    return r


def chain(r, exact):
    r.compute_receivers()
    r.reroute_flow()
    r.accumulate_constant_Q(1.0, exact_order=exact)


def results(r):
    return [t.cpu().numpy().copy() for t in (r.receivers, r.Q, r.counts)]


# one launch of several blocks, and the four launches of larger grids
@pytest.mark.gpu
@pytest.mark.parametrize("nx,ny", [(300, 200), (600, 601)])
@pytest.mark.parametrize("kernels,exact", [(REROUTE, False), (TREE, False), (ROUNDS, True)])
def test_a_barrier_that_gives_up_is_an_error(cuda, barrier_test, nx, ny, kernels, exact):
    from pyfastflow_b200._lib import PFFError

    r = router(nx, ny)
    chain(r, exact)
    want = results(r)
    r.counts.zero_()
    barrier_test(kernels, 1, 1000)
    with pytest.raises(PFFError, match="status 3"):
        chain(r, exact)
    barrier_test(0, 0, 0)
    chain(r, exact)
    for a, b in zip(want, results(r)):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_labels_that_give_up_end_the_reroute(cuda, barrier_test):
    """The labels are a launch of their own on larger grids: the saddle pass and the loop behind
    it must not run on what an earlier call left.  The receivers stay as they were."""
    from pyfastflow_b200._lib import PFFError

    r = router(600, 601)
    chain(r, False)
    want = results(r)
    r.compute_receivers()
    before = r.receivers.cpu().numpy().copy()
    barrier_test(LABELS, 1, 1000)
    with pytest.raises(PFFError, match="status 3"):
        r.reroute_flow()
    assert np.array_equal(before, r.receivers.cpu().numpy())
    barrier_test(0, 0, 0)
    chain(r, False)
    for a, b in zip(want, results(r)):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_tree_status_reports_a_barrier_given_up(cuda, barrier_test):
    """pff_accumulate_tree and its status call apart, as FlowRouter.route_many makes them."""
    torch = cuda
    from pyfastflow_b200._lib import PFFError

    r = router(300, 200)
    z = [r.z.cpu().pin_memory() for _ in range(3)]
    q = [torch.full((r.N,), -1.0).pin_memory() for _ in z]
    r.route_many(z, None, q)
    torch.cuda.synchronize()
    want = q[0].clone()
    barrier_test(TREE, 1, 1000)
    with pytest.raises(PFFError, match="status 3"):
        r.route_many(z, None, q)
    barrier_test(0, 0, 0)
    r.route_many(z, None, q)
    torch.cuda.synchronize()
    assert all(torch.equal(want, t) for t in q)


@pytest.mark.gpu
@pytest.mark.parametrize("graph", [False, True])
def test_batch_status_reports_a_barrier_given_up(cuda, barrier_test, graph):
    from pyfastflow_b200._lib import PFFError
    from pyfastflow_b200.flow import RaggedRouter

    shapes = [(60 + 9 * k, 150 - 11 * k) for k in range(8)]
    rr = RaggedRouter(shapes, 30.0, "normal")
    rr.set_z([synthetic.spectral_dem(nx, ny, k, relief=300.0, npits=20, pit_scale=0.1)
              for k, (ny, nx) in enumerate(shapes)])
    rr.seed_constant()
    rr.route()
    want = [t.cpu().numpy().copy() for t in (rr.receivers, rr.Q, rr.counts)]
    barrier_test(ROUNDS, 1, 1000)
    with pytest.raises(PFFError, match="status 32"):
        rr.route(graph=graph)
    rr._graph = None  # it holds the launch made for the test
    barrier_test(0, 0, 0)
    rr.route(graph=graph)
    for a, b in zip(want, (rr.receivers, rr.Q, rr.counts)):
        assert np.array_equal(a, b.cpu().numpy())


# limits around the blocks' distance: some waits end in time and others do not
@pytest.mark.gpu
@pytest.mark.parametrize("n,kernels,exact", [(380, REROUTE, False), (600, LABELS, False), (380, TREE, False),
                                             (380, ROUNDS, True)])
def test_blocks_agree_on_a_barrier_given_up(cuda, barrier_test, n, kernels, exact):
    """Every call is an error or gives the usual results."""
    from pyfastflow_b200._lib import PFFError

    r = router(n, n + 10)
    chain(r, exact)
    want = results(r)
    ended = []
    for k in range(120):
        r.counts.zero_()
        barrier_test(kernels, 0, 1 + 2 * (k % 30))
        try:
            chain(r, exact)
        except PFFError as e:
            assert "status 3" in str(e)
            ended.append(False)
            continue
        ended.append(True)
        for a, b in zip(want, results(r)):
            assert np.array_equal(a, b), k
    barrier_test(0, 0, 0)
    chain(r, exact)
    for a, b in zip(want, results(r)):
        assert np.array_equal(a, b)
    print(kernels, sum(ended), "of", len(ended), "calls ended in time")
