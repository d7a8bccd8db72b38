"""The rate kernels' own exponential, logarithm and quotient, slot by slot against the oracle: temperatures
from where most rates underflow to where the fits end, both sides of one in F_cent, pressures from the
low to the high end of the fall-off, empty and negative third bodies, and arguments outside every range."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle.oracle import Oracle  # noqa: E402
from tiger_nga_b200 import capi  # noqa: E402
from tiger_nga_b200.mechanism import load  # noqa: E402

pytestmark = pytest.mark.gpu
P = 101325.0


def slot_rates(mech, sol):
    _, rates = capi.FiniteChem(mech, "fp64").compute_rhs_rates(torch.from_numpy(sol).cuda(), P)
    torch.cuda.synchronize()
    return rates.cpu().numpy(), Oracle(mech).rates_batch(sol, P)


def cells(ns, T, rho, seed):
    g = np.random.default_rng(seed)
    y = 10.0 ** g.uniform(-12, 0, (ns, len(T)))
    rho = np.broadcast_to(rho, T.shape)
    sol = np.empty((ns + 1, len(T)))
    sol[:ns] = rho * y / y.sum(axis=0)
    sol[ns] = sol[:ns].sum(axis=0) * T
    return np.ascontiguousarray(sol)


@pytest.mark.parametrize("mech", ["hydrogen", "grimech30", "dme39"])
@pytest.mark.parametrize("lo,hi", [(100.0, 300.0), (300.0, 4000.0), (4000.0, 3.0e4)])
def test_slot_rates_over_temperature_and_density(mech, lo, hi):
    ns = load(mech).ns
    n = 3001
    g = np.random.default_rng(7)
    sol = cells(ns, np.exp(g.uniform(np.log(lo), np.log(hi), n)), 10.0 ** g.uniform(-8, 4, n), 8)
    sol[:ns, 5] = 0.0  # an empty cell but for one species; a cell of negative densities
    sol[0, 5], sol[ns, 5] = 1e-3, 0.5 * (lo + hi) * 1e-3
    sol[:, 6] *= -1.0
    W, Wo = slot_rates(mech, sol)
    big = np.abs(Wo) > 1e-280
    # |ln W| < 645 and ln A, n ln T below 100 each: four roundings of sums up to 850, 4 * 850 * 1.1e-16 on
    # either side, and a few units in the last place for the functions and products
    assert np.isfinite(W).all()
    assert (np.abs(W - Wo)[big] / np.abs(Wo)[big]).max() <= 1e-12
    assert np.abs(W[~big]).max(initial=0.0) <= 1e-270


@pytest.mark.parametrize("mech", ["grimech30", "dme39"])
def test_arguments_outside_the_exponentials_range(mech):
    """Underflow gives zero, overflow a non-finite rate, a NaN temperature NaN, from the bound on T
    (0.047 K for GRI) on; below it the argument stays at its value there."""
    m = load(mech)
    T = np.array([0.05, 0.3, 1.0, 20.0, np.nan])
    sol = cells(m.ns, T, 1.0, 9)
    W, Wo = slot_rates(mech, sol)
    plain = [i for i, s in enumerate(m.slots) if s.kind != "falloff" and s.arr.E is not None]
    for i in plain:
        a, b = W[i, :-1], Wo[i, :-1]
        gone, over = np.abs(b) < 1e-300, np.isinf(b)
        assert (np.abs(a[gone]) <= 1e-290).all()
        assert not np.isfinite(a[over]).any()
        assert np.isfinite(a[~over & ~np.isnan(b)]).all()
        assert np.isnan(W[i, -1])


@pytest.mark.parametrize("mech", ["hydrogen", "grimech30", "dme39"])
def test_arguments_stay_in_range_at_any_temperature(mech):
    """Temperatures of states that have gone wrong (a density near zero, an infinity): the exponentials' arguments
    are held in the tables' range, so a rate that is finite comes out as the oracle's, one that vanishes vanishes
    and one that overflows is not finite."""
    m = load(mech)
    T = np.concatenate([10.0 ** np.linspace(8.0, 14.0, 1500), [0.0, np.inf]])
    sol = cells(m.ns, T, 1.0, 10)
    W, Wo = slot_rates(mech, sol)
    emax = max(abs(a.E) for s in m.slots for a in ((s.k0, s.kinf) if s.kind == "falloff" else (s.arr,)) if a.E is not None)
    for i, s in enumerate(m.slots):
        a, b = W[i], Wo[i]
        finite = np.isfinite(b) & np.isfinite(T) & (np.abs(b) > 1e-280) & (T > 0.0)
        # |ln W| < 645, n ln T below 600: the roundings of sums up to 1,400 on either side
        assert (np.abs(a[finite] - b[finite]) <= 2e-12 * np.abs(b[finite])).all(), s.index
        if s.kind == "falloff" or abs(s.arr.n or 0.0) < 0.1 or abs(s.arr.E or 0.0) < 1e-3 * emax:
            continue  # small exponents need not have saturated at the bounds
        assert (np.abs(a[b == 0.0]) <= 1e-290).all(), s.index
        assert not np.isfinite(a[np.isinf(b)]).any(), s.index
