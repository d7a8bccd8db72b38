"""The pooled solver kernel (12 warps per SM, factors in global memory, matrix areas shared by the
block's warps) does the arithmetic of the other launch shapes: bit-identical states and step counts, for
one cell, for fewer and more cells than a block has warps, and for more than the card has."""
import pytest

torch = pytest.importorskip("torch")

from tiger_nga_b200 import capi  # noqa: E402
from tiger_nga_b200.train_surrogate import state_batch  # noqa: E402

pytestmark = pytest.mark.gpu
P = 101325.0


@pytest.mark.parametrize("mech", ["grimech30", "dme39"])  # 37 and 40 unknowns: a short last group of eight and none
@pytest.mark.parametrize("precision,n", [("fp64", 1), ("fp64", 13), ("mixed", 150), ("fp64", 1800)])
def test_pooled_kernel_equals_the_eight_warp_kernel(mech, precision, n):
    sol, dts = state_batch(mech, n, 77 + n, side=0)
    x0, d = torch.from_numpy(sol).cuda(), torch.from_numpy(dts).cuda()
    got = []
    for warps in (0, 12, 8):
        x = x0.clone()
        stats, cnt = capi.FiniteChem(mech, precision, solver_warps=warps).substep(x, d, P, cell_counts=True)
        assert stats["cells_failed"] == 0
        got.append((x, cnt["nst"], cnt["nni"]))
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
    # a step budget (passes that save and resume cells) and the call that allocates nothing
    x = x0.clone()
    capi.FiniteChem(mech, precision, pass_budget=32, max_passes=4).substep(x, d, P)
    y = x0.clone()
    assert capi.FiniteChem(mech, precision).substep_static(y, d, P) == 0
    torch.cuda.synchronize()
    assert torch.equal(y, got[0][0])
    z = x0.clone()
    capi.FiniteChem(mech, precision, pass_budget=32, max_passes=4, solver_warps=8).substep(z, d, P)
    torch.cuda.synchronize()
    assert torch.equal(x, z)


def test_failed_cells_give_their_matrix_area_back():
    """Cells that stop early (step limit, non-finite state) leave the pool whole for those after them."""
    sol, dts = state_batch("grimech30", 600, 5, side=0)
    sol[3, ::7] = float("nan")
    x0, d = torch.from_numpy(sol).cuda(), torch.from_numpy(dts).cuda()
    got = []
    for warps in (0, 8):
        x = x0.clone()
        _, cnt = capi.FiniteChem("grimech30", "fp64", solver_warps=warps, max_steps=40).substep(x, d, P, cell_counts=True)
        got.append((x, cnt["status"]))
    assert torch.equal(got[0][1], got[1][1]) and torch.equal(got[0][0].nan_to_num(), got[1][0].nan_to_num())
    assert int((got[0][1] == 4).sum()) == 86 and int((got[0][1] == 1).sum()) > 100


def solver_kernels_of(call):
    """Device time in us of the solver's kernels in one call, pooled and not."""
    from torch.profiler import ProfilerActivity, profile

    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    k = [(e.name, e.device_time) for e in prof.events() if "k_bdf<" in e.name]
    return sum(t for n, t in k if ", 12, 1," in n), sum(t for n, t in k if ", 12, 1," not in n)


def test_cells_counted_on_the_device_get_the_kernel_for_their_number():
    """A surrogate's fallback list has the batch's capacity, but few cells: they run on the 8-warp kernel, as a batch of
    that size does; a list of many runs on the pooled one."""
    import os

    chem = capi.FiniteChem("grimech30", "fp64")
    sur = capi.Surrogate(chem, judge_cells=0)
    sur.load(os.path.join(os.path.dirname(capi.__file__), "models", "grimech30.tngs"))
    sol, dts = state_batch("grimech30", 8_000, 3, side=0)
    x0, d = torch.from_numpy(sol).cuda(), torch.from_numpy(dts).cuda()
    x, stats = torch.empty_like(x0), {}

    def call():
        x.copy_(x0)
        stats.update(sur.substep(x, d, P))

    pooled, eight = solver_kernels_of(call)
    n = stats["cells"] - stats["accepted"]
    assert 20 < n < 1480 and pooled < 50.0 < 500.0 < eight, (n, pooled, eight)
    sur.set_gate_tol(1e-9)  # every cell falls back
    pooled, eight = solver_kernels_of(call)
    assert stats["accepted"] == 0 and eight < 50.0 < 500.0 < pooled, (pooled, eight)
    # and the batch of all cells is solved as the list was
    chem.substep(x0, d, P)
    torch.cuda.synchronize()
    assert torch.equal(x, x0)
    sur.close()
