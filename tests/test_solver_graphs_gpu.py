"""The solver's captured graphs hold addresses of the handle's scratch, which grows with the batch: a call whose
graph was captured before a larger call made the scratch grow has to capture again, not replay the old
addresses. Every call is compared bit for bit with the same call on a handle that sees nothing else."""
import pytest

torch = pytest.importorskip("torch")

from tiger_nga_b200 import capi  # noqa: E402
from tiger_nga_b200.train_surrogate import state_batch  # noqa: E402

pytestmark = pytest.mark.gpu
P = 101325.0


def call(chem, x0, x, d, cnt):
    """tng_substep_batch in the caller's own buffers, so that a repeated call repeats every argument."""
    x.copy_(x0)
    torch.cuda.synchronize()
    capi._check(chem.lib.tng_substep_batch(chem.h, x.data_ptr(), x.shape[1], x.shape[1], d.data_ptr(), 0.0, P,
                                           capi.TNG_DEVICE_PTRS, cnt[0].data_ptr(), cnt[1].data_ptr(),
                                           cnt[2].data_ptr(), None), "tng_substep_batch")
    chem.sync()
    return x.clone(), cnt.clone()


@pytest.mark.parametrize("mech", ["hydrogen", "grimech30"])
@pytest.mark.parametrize("cfg", [dict(), dict(pass_budget=16, max_passes=4)])
def test_growth_captures_again(mech, cfg):
    sizes = (300, 2000, 300, 9000, 300, 2000)
    buf = {}
    for n in set(sizes):
        sol, dts = state_batch(mech, n, n, side=0)
        x0 = torch.from_numpy(sol).cuda()
        buf[n] = (x0, torch.empty_like(x0), torch.from_numpy(dts).cuda(),
                  torch.zeros((3, n), dtype=torch.int32, device="cuda"))
    want = {n: call(capi.FiniteChem(mech, "fp64", **cfg), *buf[n]) for n in buf}
    chem = capi.FiniteChem(mech, "fp64", **cfg)
    for n in sizes:
        got = call(chem, *buf[n])
        assert torch.equal(got[0], want[n][0]) and torch.equal(got[1], want[n][1]), n


def test_scratch_that_a_one_pass_call_leaves_behind():
    """A large one-pass call grows the counters but not the saved histories; budgeted calls after it grow those
    between two equal calls whose other buffers stay where they are."""
    buf = {}
    for n in (300, 2000, 9000):
        sol, dts = state_batch("hydrogen", n, n, side=0)
        x0 = torch.from_numpy(sol).cuda()
        buf[n] = (x0, torch.empty_like(x0), torch.from_numpy(dts).cuda(),
                  torch.zeros((3, n), dtype=torch.int32, device="cuda"))

    def tuned(chem, n, budget):
        capi._check(chem.lib.tng_chem_set_tuning(chem.h, -1, 0, 8, budget), "tng_chem_set_tuning")
        return call(chem, *buf[n])

    chem = capi.FiniteChem("hydrogen", "fp64")
    for n, budget in ((9000, 0), (300, 16), (2000, 16), (300, 16), (9000, 16), (300, 16)):
        got, want = tuned(chem, n, budget), tuned(capi.FiniteChem("hydrogen", "fp64"), n, budget)
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]), (n, budget)
