"""The post-processing of a prediction for every element count the built-in mechanisms have (3, 4 and 5,
each with kernels of its own), on ragged cell counts: mass, elements and enthalpy are conserved to
rounding whatever the network says.

Tolerances: the projection accepts normal equations whose pivots are above 1e-8 of the diagonal, so its solve
is off by at most some 2^-53 / 1e-8 = 1.1e-8 times the handful of constraints, below 1e-7 of an element's mass;
a cell with smaller pivots is rejected. The temperature's Newton iteration stops at 1e-9."""
import struct

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from tiger_nga_b200 import capi, states  # noqa: E402
from tiger_nga_b200.mechanism import load  # noqa: E402
from tiger_nga_b200.train_surrogate import state_batch  # noqa: E402

pytestmark = pytest.mark.gpu
P = 101325.0


@pytest.mark.parametrize("mech,nel", [("hydrogen", 3), ("dme39", 4), ("grimech30", 5)])
@pytest.mark.parametrize("post_mode", [0, 1])
def test_prediction_conserves(mech, nel, post_mode):
    m = load(mech)
    assert len(m.elements) == nel
    chem = capi.FiniteChem(mech, "fp64")
    sol, dts = state_batch(mech, 4096, 31, side=0)
    s0, d = torch.from_numpy(sol).cuda(), torch.from_numpy(dts).cuda()
    s1 = s0.clone()
    chem.substep(s1, d, P)
    sur = capi.Surrogate(chem, judge_cells=16, post_mode=post_mode)
    sur.train(s0, s1, d, P, epochs=6, batch=256, lr=2e-3)
    for n in (1, 127, 129, 3000):
        out, reason, ind = sur.predict(s0[:, :n].contiguous(), d[:n].contiguous(), P)
        torch.cuda.synchronize()
        a, b = sol[:, :n], out.cpu().numpy()
        ok = np.isfinite(ind.cpu().numpy()[:, 0])
        assert n < 1000 or ok.mean() > 0.9
        Ya, Yb = a[:-1] / a[:-1].sum(0), b[:-1] / b[:-1].sum(0)
        assert np.all(b[:-1] >= 0.0)
        assert np.max(np.abs(b[:-1].sum(0) / a[:-1].sum(0) - 1.0)) <= 1e-12
        E = m.elem / m.wmol
        dE = np.abs(E @ Yb - E @ Ya) / np.maximum(E @ Ya, 1e-3 * (E @ Ya).max(0))
        assert np.max(dE[:, ok], initial=0.0) <= 1e-7
        Ta, Tb = a[-1] / a[:-1].sum(0), b[-1] / b[:-1].sum(0)
        ha, hb = (Ya * states.thermo_h(m, Ta)).sum(0), (Yb * states.thermo_h(m, Tb)).sum(0)
        cp = (Yb * states.thermo_cp(m, Tb)).sum(0)
        assert np.max(np.abs(hb - ha)[ok] / (cp * Tb)[ok]) <= 1e-7
    sur.close()
    chem.close()


def fixed_prediction(chem, path, target):
    """A model file whose networks answer (relative temperature change, mass-fraction changes) = target, whatever
    the cell: zero weights, the answer in the targets' means."""
    sur = capi.Surrogate(chem, members=1, layers=1, judge_cells=0, post_mode=0)
    ns, m = chem.nspecies, sur
    with open(path, "wb") as f:
        f.write(b"TNGSUR3\0" + chem.mechanism.encode().ljust(32, b"\0"))
        f.write(struct.pack("<10i", ns, m.n_in, m.n_out, 256, 1, 0, 0, 1, 0, 0) + struct.pack("<q", m.nparam))
        for v in (np.zeros(m.n_in), np.ones(m.n_in), np.full(m.n_in, -1e30), np.full(m.n_in, 1e30), target, np.ones(m.n_out)):
            f.write(np.asarray(v, dtype=np.float64).tobytes())
        f.write(np.zeros(m.nparam, dtype=np.float32).tobytes())
    sur.load(str(path))
    return sur


def test_nearly_dependent_elements_are_rejected(tmp_path):
    """Steam in nitrogen, a little oxygen that the network overdraws, and traces of the rest: the oxygen that is
    missing has to come from the traces, and the smaller they are, the closer the rows of H and O of the normal
    equations come to each other. Whatever is not rejected conserves the elements; traces of 1e-5 are enough."""
    m = load("hydrogen")
    chem = capi.FiniteChem("hydrogen", "fp64")
    at = {s: i for i, s in enumerate(m.species)}
    trace = np.concatenate([10.0 ** np.linspace(-15.0, -4.0, 500), np.zeros(13)])
    Y = np.tile(trace, (m.ns, 1))
    Y[at["H2O"]], Y[at["O2"]] = 0.25, 0.01
    Y[at["N2"]] += 1.0 - Y.sum(0)
    rho = 0.5
    sol = np.vstack([rho * Y, np.full((1, trace.size), rho * 1500.0)])
    target = np.zeros(m.ns + 1)
    target[1 + at["O2"]] = -0.02
    sur = fixed_prediction(chem, tmp_path / "fixed.tngs", target)
    out, _, ind = sur.predict(torch.from_numpy(np.ascontiguousarray(sol)).cuda(), 1e-6, P)
    torch.cuda.synchronize()
    b = out.cpu().numpy()
    ok = np.isfinite(ind.cpu().numpy()[:, 0])
    E = m.elem / m.wmol
    dE = np.abs(E @ (b[:-1] / b[:-1].sum(0)) - E @ Y) / np.maximum(E @ Y, 1e-3 * (E @ Y).max(0))
    assert np.max(dE[:, ok]) <= 1e-7
    assert ok[trace >= 1e-5].all() and not ok[trace <= 1e-12].any()
    sur.close()
    chem.close()
