"""Wilke's viscosity on the tensor cores at the edges of its tiles: cell counts around the 32 cells of a
warp and the 8 of a matrix product, species counts that fill the 8 x 4 fragments or do not (9, 36, 39),
masked cells, and cells that hold absent, negative or non-finite mass fractions next to sound ones.

Tolerance: sums of at most 40 terms of one sign, a dozen roundings each: 40 * 12 * 2^-53 = 5e-14."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle.oracle import Oracle  # noqa: E402
from tiger_nga_b200 import capi  # noqa: E402

pytestmark = pytest.mark.gpu
P = 101325.0


def cells(ns, n, seed):
    rng = np.random.default_rng(seed)
    Y = 10.0 ** rng.uniform(-12, 0, (ns, n))
    Y[rng.random((ns, n)) < 0.2] = 0.0
    Y[0] += 0.1
    return Y / Y.sum(0), rng.uniform(40.0, 5100.0, n)


@pytest.mark.parametrize("mech", ["hydrogen", "grimech30", "dme39"])
@pytest.mark.parametrize("n", [1, 7, 9, 31, 33, 64, 65, 4099])
def test_viscosity_and_diffusivity_at_tile_edges(mech, n):
    chem, o = capi.FiniteChem(mech, "fp64"), Oracle(mech)
    Y, T = cells(chem.nspecies, n, n)
    want = o.props_batch(Y, T, p_thermo=P)
    sc = torch.from_numpy(np.vstack([Y, T[None]])).cuda()
    for kw in (dict(visc=True, diff=True), dict(visc=True), dict(diff=True)):
        got = chem.mixture_props(sc, **kw)
        torch.cuda.synchronize()
        for k, v in got.items():
            assert np.max(np.abs(v.cpu().numpy() - want[k]) / np.abs(want[k])) <= 5e-14, (kw, k)


def test_masked_and_unsound_cells_leave_their_neighbours_alone():
    chem, o = capi.FiniteChem("grimech30", "fp64"), Oracle("grimech30")
    ns, nx, ny, nz = chem.nspecies, 7, 5, 6
    n = nx * ny * nz
    Y, T = cells(ns, n, 3)
    Y[4, 10], Y[5, 20], T[30], Y[:, 40] = np.nan, np.inf, np.nan, 0.0
    Y[7, 50] = -1e-3
    mask = np.zeros((nx, ny), dtype=np.int32, order="F")
    mask[2, 1] = mask[6, 4] = 1
    off = np.broadcast_to((mask == 1)[:, :, None], (nx, ny, nz)).reshape(-1, order="F")
    SC = np.zeros((nx, ny, nz, ns + 1), order="F")
    SC[..., :ns] = Y.T.reshape(nx, ny, nz, ns, order="F")
    SC[..., ns] = T.reshape(nx, ny, nz, order="F")
    VISC, DIFF = np.full((nx, ny, nz), -7.0, order="F"), np.full(SC.shape, -9.0, order="F")
    ext = dict(imino=1, imaxo=nx, jmino=1, jmaxo=ny, kmino=1, kmaxo=nz, imin=1, imax=nx, jmin=1, jmax=ny, kmin=1,
               kmax=nz, nscalar=ns + 1, isc_sc=1, isc_T=ns + 1, isc_H2O=0, isc_CO=0, isc_CO2=0)
    chem.transport(SC, ext, VISC=VISC, DIFF=DIFF, mask=mask)
    v, d = VISC.reshape(-1, order="F"), DIFF.reshape(n, ns + 1, order="F")
    assert np.all(v[off] == -7.0) and np.all(d[off] == -9.0)
    want = o.props_batch(Y, T, p_thermo=P)
    sound = ~off
    sound[[10, 20, 30, 40]] = False
    assert np.max(np.abs(v[sound] - want["visc"][sound]) / np.abs(want["visc"][sound])) <= 5e-14
    assert np.max(np.abs(d[sound].T - want["diff"][:, sound]) / np.abs(want["diff"][:, sound])) <= 5e-13
    assert np.isnan(v[10]) and np.isnan(d[10]).all()  # (a NaN temperature is clipped to the fits' range)


@pytest.mark.parametrize("mech", ["hydrogen", "grimech30", "dme39"])
def test_diffusivities_beside_the_viscosity_are_those_of_the_division(mech):
    """The call for both takes the species viscosities from the reciprocal square root, the call for the
    diffusivities alone from a division. The corrected quotient is the correctly rounded one unless the exact
    one lies within 2^-100 of a tie, so the two calls agree bit for bit."""
    chem = capi.FiniteChem(mech, "fp64")
    Y, T = cells(chem.nspecies, 20_011, 9)
    sc = torch.from_numpy(np.vstack([Y, T[None]])).cuda()
    both, alone = chem.mixture_props(sc, visc=True, diff=True), chem.mixture_props(sc, diff=True)
    torch.cuda.synchronize()
    assert torch.equal(both["diff"], alone["diff"])


def device_transport(chem, sc, visc, diff, mask, nx, ny, nz):
    """tng_chem_transport on device arrays of a padded block (species at 1..N, T at N+1)."""
    ns = chem.nspecies
    e = capi.Extent(imino=1, imaxo=nx, jmino=1, jmaxo=ny, kmino=1, kmaxo=nz, imin=1, imax=nx, jmin=1, jmax=ny, kmin=1,
                    kmax=nz, nscalar=ns + 1, isc_sc=1, isc_T=ns + 1, isc_H2O=0, isc_CO=0, isc_CO2=0)
    capi._check(chem.lib.tng_chem_transport(chem.h, visc.data_ptr(), diff.data_ptr(), sc.data_ptr(), mask.data_ptr(),
                                            ctypes.byref(e), None, 0, capi.TNG_DEVICE_PTRS), "tng_chem_transport")


def test_masked_warps_do_no_work():
    """A block whose masked cells fill whole warps: the others are those of the unmasked call, the masked ones keep
    their values, and a block that is masked throughout takes the time of reading its mask (a twentieth of the
    whole block's time or less; the bound leaves a factor of four)."""
    chem = capi.FiniteChem("grimech30", "fp64")
    nx, ny, nz = 96, 64, 64
    n = nx * ny * nz
    Y, T = cells(chem.nspecies, n, 11)
    sc = torch.from_numpy(np.vstack([Y, T[None]])).cuda()
    time = {}
    for name in ("none", "half", "all"):
        mask = torch.zeros(ny, nx, dtype=torch.int32, device="cuda")
        mask[:, 32:] = 1 if name == "all" else 0
        mask[:, :32] = 0 if name == "none" else 1
        visc, diff = torch.full((n,), -7.0, device="cuda").double(), torch.full_like(sc, -9.0)
        torch.cuda.synchronize()
        for _ in range(3):
            device_transport(chem, sc, visc, diff, mask, nx, ny, nz)
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(chem.torch_stream()):
            a.record()
            for _ in range(20):
                device_transport(chem, sc, visc, diff, mask, nx, ny, nz)
            b.record()
        chem.sync()
        time[name] = a.elapsed_time(b)
        off = (mask == 1).expand(nz, ny, nx).reshape(-1)
        if name == "none":
            want = visc, diff
        assert bool((visc[off] == -7.0).all()) and bool((diff[:, off] == -9.0).all())
        assert torch.equal(visc[~off], want[0][~off]) and torch.equal(diff[:, ~off], want[1][:, ~off])
    assert time["all"] <= 0.2 * time["none"], time
