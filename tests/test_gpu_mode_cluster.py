"""The one-launch end of a factor step (HALS / MU update up to rank 16,
normalisation, Grams, error) at the edges of its shapes, against the CPU oracle: one row and
one past a CTA's rows, the largest factor it takes and one past it (the
separate launches), ranks either side of the lane groups. FP64, 3 iterations,
1e-10 relative as the other FP64 parity tests."""
import pytest

from helpers import cp_tensor, init_factors, rel

pytestmark = pytest.mark.gpu
TOL = 1e-10


@pytest.mark.parametrize("algo", ["hals", "mu"])
@pytest.mark.parametrize("dims,k", [((1, 5, 4), 1), ((2, 33, 9), 3), ((31, 32, 33), 15), ((65, 64, 17), 16),
                                    ((66, 20, 19), 17), ((513, 24, 9), 9), ((70, 66, 40), 32),
                                    ((80, 49, 48), 33), ((90, 70, 64), 64), ((4096, 6, 5), 5),
                                    ((4097, 6, 5), 5), ((12, 11, 600, 3), 6)])
def test_mode_cluster_shapes(gpu, oracle_lib, algo, dims, k):
    X, _ = cp_tensor(dims, k, noise=0.01, seed=81)
    F0 = init_factors(dims, k, seed=82)
    Fo, lamo, eo = oracle_lib.ntf_run(X, F0, algo, 3, dimtree=True)
    with gpu.Context(0, "fp64") as c:
        c.set_tensor(X)
        c.set_factors(F0)
        e = c.run(algo, 3)
        F, lam = c.get_factors()
    assert rel(e, eo) < TOL
    assert rel(lam, lamo) < TOL
    for a, b in zip(F, Fo):
        assert rel(a, b) < TOL
