"""The iteration graphs of planc_gpu_run: a run asked for a second time is
captured and later ones replay it. Replayed runs of every update give the bits
of the same run launched kernel by kernel (under timing no graph is used), and
launch nothing but the first leave-one-out product."""
import numpy as np
import pytest

from helpers import cp_tensor, init_factors

pytestmark = pytest.mark.gpu

ALGOS = ["hals", "mu", "anlsbpp", "aoadmm", "nesterov"]


def _ctx(gpu, prec, X):
    c = gpu.Context(0, prec)
    c.set_tensor(X if prec == "fp64" else X.astype(np.float32))
    return c


def _run(c, F0, algo, iters, dimtree=True):
    c.set_factors(F0)
    c.reset_update_state()
    before = c.launch_count()
    errs = c.run(algo, iters, dimtree=dimtree)
    launched = c.launch_count() - before
    F, lam = c.get_factors()
    return launched, [errs, lam] + F


def _same(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("prec,dimtree", [("fp64", True), ("fp64", False), ("bf16", True)])
@pytest.mark.parametrize("algo", ALGOS)
def test_replayed_runs_give_the_bits_of_direct_ones(gpu, algo, prec, dimtree):
    X, _ = cp_tensor((33, 26, 21), 5, noise=0.01, seed=31)
    F0 = init_factors(X.shape, 5, seed=32)
    # a remainder (11), a divisor (20), one graph (8), shorter than it (3, 1),
    # captured at once (45)
    lengths = [11, 20, 8, 3, 1, 45, 8]
    with _ctx(gpu, prec, X) as c:
        c.set_timing(True)
        direct = {n: _run(c, F0, algo, n, dimtree)[1] for n in set(lengths)}
    with _ctx(gpu, prec, X) as c:
        for n in lengths:
            for _ in range(3):
                launched, got = _run(c, F0, algo, n, dimtree)
                assert _same(got, direct[n]), n
            assert launched == 1, (n, launched)


def test_longer_runs_than_before(gpu):
    X, _ = cp_tensor((24, 20, 16), 4, noise=0.01, seed=33)
    F0 = init_factors(X.shape, 4, seed=34)
    with _ctx(gpu, "fp64", X) as c:
        c.set_timing(True)
        direct = {n: _run(c, F0, "hals", n)[1] for n in (5, 20, 300)}
    with _ctx(gpu, "fp64", X) as c:
        for n in (5, 5, 20):  # 20: four graphs of five, the error buffer holds it
            launched, got = _run(c, F0, "hals", n)
            assert _same(got, direct[n])
        assert launched == 1
        for n in (300, 300, 20, 20, 20):  # 300: the error buffer moves
            launched, got = _run(c, F0, "hals", n)
            assert _same(got, direct[n])
        assert launched == 1


def test_alternating_configurations_replay(gpu):
    X, _ = cp_tensor((24, 20, 16), 4, noise=0.01, seed=35)
    F0 = init_factors(X.shape, 4, seed=36)
    with _ctx(gpu, "fp64", X) as c:
        first = {a: _run(c, F0, a, 6)[1] for a in ALGOS}
        for _ in range(2):
            got = {a: _run(c, F0, a, 6) for a in ALGOS}
        assert all(_same(got[a][1], first[a]) for a in ALGOS)
        assert all(got[a][0] == 1 for a in ALGOS)


def test_more_lengths_than_graphs_are_kept(gpu):
    X, _ = cp_tensor((24, 20, 16), 4, noise=0.01, seed=37)
    F0 = init_factors(X.shape, 4, seed=38)
    with _ctx(gpu, "fp64", X) as c:
        first = {}
        for _ in range(3):
            for algo in ("hals", "mu", "anlsbpp"):
                for n in range(1, 9):
                    got = _run(c, F0, algo, n)[1]
                    assert _same(got, first.setdefault((algo, n), got))
