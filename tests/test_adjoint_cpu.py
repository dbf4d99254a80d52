"""The binomial checkpoint schedule of the adjoint (host logic, no GPU): every step is
reversed exactly once, in order N-1 .. 0, from its own state; no more snapshots are
live than allowed; the forward steps match the binomial optimum."""
import numpy as np
import pytest
import torch

from geoswe_b200.adjoint import Treeverse, binomial_beta, interp_weights, snapshot_chain, treeverse_split


def _run(N, S, pre_stored=True):
    snaps = {0: 0}
    cur = {"n": None}

    def store(n):
        assert cur["n"] == n
        snaps[n] = n

    def restore(n):
        cur["n"] = snaps[n]

    def advance(n0, n1):
        assert cur["n"] == n0
        cur["n"] = n1

    def free(n):
        snaps.pop(n)

    def reverse(n):
        assert cur["n"] == n, (cur["n"], n)

    chain = snapshot_chain(N, S) if pre_stored else []
    for m in chain:
        snaps[m] = m
    tv = Treeverse(N, S, store, restore, advance, free, reverse, stored=chain)
    tv.run()
    return tv


@pytest.mark.parametrize("N,S", [(1, 3), (2, 1), (7, 2), (100, 3), (200, 10), (1000, 20), (3000, 55), (50, 0)])
def test_every_step_reversed_once_in_order(N, S):
    tv = _run(N, S)
    assert tv.order == list(range(N - 1, -1, -1))
    assert tv.max_live <= S


@pytest.mark.parametrize("N,S", [(100, 3), (200, 10), (1000, 20), (3000, 55)])
def test_forward_steps_binomial_optimum(N, S):
    tv = _run(N, S)
    t = 0
    while binomial_beta(S, t) < N:
        t += 1
    optimum = t * N - binomial_beta(S + 1, t - 1)
    assert tv.forward_steps + N <= optimum + 1          # + the recording pass


def test_split_keeps_recomputation_count():
    for N in (10, 57, 300, 3000):
        for S in (1, 4, 55):
            m = treeverse_split(N, S)
            assert 1 <= m <= N - 1


def test_interp_weights_reproduce_numpy():
    rng = np.random.default_rng(0)
    xp = np.sort(rng.uniform(0, 100, 9))
    fp = rng.normal(size=9)
    t = np.concatenate([rng.uniform(-10, 110, 50), xp])
    assert np.allclose(interp_weights(t, xp) @ fp, np.interp(t, xp, fp), rtol=0, atol=1e-12)


@pytest.mark.parametrize("code", [-1, -2, -3, -5])
@pytest.mark.parametrize("failing", ["gsw_dt_finalize", "gsw_flat_step", "gsw_adj_flat_step"])
def test_a_failing_launch_keeps_its_status(monkeypatch, failing, code):
    """The launchers of a recording pass and of a reverse sweep raise GswError with the status
    the library returned (no GPU: the entry points are stubs)."""
    from geoswe_b200 import _lib as L
    from geoswe_b200 import adjoint as A

    class Lib:
        def __getattr__(self, name):
            if name == "gsw_last_error":
                return lambda: b"stub"
            fn = lambda *a: code if name == failing else L.OK  # noqa: E731
            fn.__name__ = name
            return fn

    stub = Lib()
    monkeypatch.setattr(L, "lib", lambda: stub)
    monkeypatch.setattr(A, "_stream", lambda: None)
    monkeypatch.setattr(A, "_ptr", lambda x: None)
    adj = object.__new__(A.FlatAdjoint)
    adj.inlet, adj.G, adj.code, adj.adj_min_blocks, adj.kernel_launches = None, 0, L.F32, 8, 0
    adj.dev, adj._buf, adj._state = torch.device("cpu"), [[None] * 3] * 2, None
    adj._lam, adj._rbar, adj.n_bar, adj.rate_bar = [[None] * 3, [None] * 3], [None] * 3, None, None
    adj._state_tab = torch.zeros((2, 128), dtype=torch.uint8)
    adj._flat_args = lambda *a: L.GswFlatArgs()
    p = L.GswDtParams()
    with pytest.raises(L.GswError) as e:
        if failing == "gsw_adj_flat_step":
            adj._reverser(p)(0, 0)
        else:
            adj._stepper(p, False)(0)
    assert e.value.code == code and failing in str(e.value)
    if failing == "gsw_dt_finalize":
        with pytest.raises(L.GswError) as e:
            adj._reverser(p)(0, 0)
        assert e.value.code == code
