"""sfx_powq returns sfx_pow's bits at the large exponents 2 / (gamma - 1) and
2 gamma / (gamma - 1) of nearly isothermal gas: the logarithm's error is multiplied by the
exponent, and the rounding test's margin has to follow it."""
import numpy as np
import pytest

from test_powq import _exponents, differing  # noqa: F401 (fixture)


@pytest.mark.parametrize("gamma", [1.1, 1.05, 1.01, 1.001, 1.0001])
def test_equal_at_large_exponents(differing, gamma):  # noqa: F811
    rng = np.random.default_rng(17)
    for y in _exponents(gamma):
        # |y ln x| up to 21, inside the quick path's range
        x = np.exp(21 * (2 * rng.random(2_000_000) - 1) / max(abs(y), 1.0))
        assert differing(x, y)[0] == 0


def test_equal_at_a_known_argument(differing):  # noqa: F811
    # differed in the last bit under a margin of 2^-68 whatever the exponent
    assert differing(0.91426448344632838, 2 * 1.01 / (1.01 - 1))[0] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("gamma", [1.05, 1.001])
def test_riemann_solver_of_nearly_isothermal_gas(cuda_ok, oracle, gamma):
    """the device's exact solver against the oracle, bit for bit: receding states, whose guess
    and fans take the large powers"""
    from oracle.oracle import Params
    from shadowfax_b200.hydro import Context, RiemannSolverFactory
    rng = np.random.default_rng(31)
    n = 400_000
    W = [np.stack([np.exp(rng.uniform(-1, 1, n)), v, rng.uniform(-0.1, 0.1, n),
                   np.exp(rng.uniform(-1, 1, n))], 1)
         for v in (rng.uniform(-6, 0, n), rng.uniform(0, 6, n))]
    normal = np.tile([1.0, 0.0], (n, 1))
    ctx = Context(2, RiemannSolverFactory.generate("Exact", gamma=gamma), 0)
    half, flux, code = ctx.riemann(*W, normal)
    ohalf, oflux, ocode = oracle.riemann(2, Params(solver="Exact", gamma=gamma), *W, normal)
    assert np.array_equal(code, ocode)
    assert np.array_equal(half, ohalf) and np.array_equal(flux, oflux)
    ctx.close()
