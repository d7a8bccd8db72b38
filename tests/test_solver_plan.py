"""The rule that picks the implicit solver's launch shape (csrc/solver_plan.h), compiled for the host with a
stand-in for the occupancy query."""
import json
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tiger_nga_b200", "csrc")
SMS, SM_BYTES, OPTIN = 148, 233_472, 232_448  # B200: shared memory of an SM and of a block

PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "solver_plan.h"
using namespace tng;
int main(int argc, char** argv) {
  long long v[17];
  for (int i = 0; i < 17; ++i) v[i] = i + 1 < argc ? std::atoll(argv[i + 1]) : 0;
  const SolverSizes z{(size_t)v[0], (size_t)v[1], (size_t)v[2], (size_t)v[3], (size_t)v[4], (size_t)v[5]};
  auto resident = [&](int kernel, int threads, size_t smem) {  // by shared memory and by registers
    const long long by_smem = v[10] / (long long)(smem + 2048), by_regs = 65536 / (v[11 + kernel] * threads);
    return (int)(by_smem < by_regs ? by_smem : by_regs);
  };
  SolverShape s;
  if (solver_shape(z, (int)v[6], (int)v[7], v[8], 148, v[9] != 0, resident, &s) < 0) return 1;
  std::printf("{\"kernel\": %d, \"warps\": %d, \"stages\": %d, \"cold\": %d, \"per_sm\": %d, \"smem\": %zu, \"factors\": %zu, \"from\": %d}",
              s.kernel, s.warps, s.stages, s.cold, s.per_sm, s.smem, s.factors, s.from);
}
"""
K2, K4, K8, K8X2, POOLED = range(5)
REGS = (255, 255, 178, 128, 168)  # registers of a thread by kernel


@pytest.fixture(scope="module")
def shape(tmp_path_factory):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.check_call([gxx, "-std=c++17", "-I", CSRC, str(d / "plan.cpp"), "-o", str(d / "plan")])

    def call(sizes, ncells, warps=0, occupancy=0, scratch=True, regs=REGS):
        args = [*sizes, warps, occupancy, ncells, int(scratch), SM_BYTES, *regs]
        return json.loads(subprocess.check_output([str(d / "plan"), *map(str, args)]))

    return call


def sizes(ns, hot=30_000, cold=10_000, slots=400, factors=0):
    """Bytes as the layout gives them, for ns species and a typical set of tables."""
    nv = ns + 1
    rs = nv + 1 if nv % 2 == 0 else nv
    return 8 * (slots + 4 * ns + 300), 8 * (nv * rs + 4 * ns), hot, cold, OPTIN, factors


FACTORS = 8 * (32 + 8) * 40  # a warp of the pooled kernel


@pytest.mark.parametrize("regs", [168, 80])  # one or two blocks of 12 warps by registers
def test_factors_cover_every_resident_warp(shape, regs):
    z = (4_000, 1_500, 10_000, 4_000, OPTIN, FACTORS)
    s = shape(z, 100_000, regs=REGS[:4] + (regs,))
    assert s["kernel"] == POOLED and s["warps"] == 12 and s["per_sm"] == (1 if regs == 168 else 2)
    assert s["factors"] == FACTORS * s["warps"] * s["per_sm"] * SMS


def test_lines_between_the_shapes(shape):
    big, small = sizes(36, factors=FACTORS), sizes(9, hot=6_000, cold=2_000, slots=50)
    assert [shape(big, n)["kernel"] for n in (1, 8 * SMS, 10 * SMS, 10 * SMS + 1)] == [K8, K8, K8, POOLED]
    assert [shape(small, n)["kernel"] for n in (1, 8 * SMS, 8 * SMS + 1)] == [K8, K8, K8X2]
    assert shape(big, 10**6, scratch=False)["kernel"] == K8
    assert [shape(big, 10**6, warps=w)["kernel"] for w in (2, 4, 8, 12)] == [K2, K4, K8, POOLED]
    assert shape(small, 10**6, warps=12)["kernel"] == K8


@pytest.mark.parametrize("ns", [9, 20, 31, 40, 42])
def test_two_blocks_per_sm_only_where_both_are_resident(shape, ns):
    s = shape(sizes(ns), 10**6)
    assert (s["kernel"] == K8X2) == (ns <= 20)  # the others' matrices leave no room for a second block
    assert s["per_sm"] == (2 if s["kernel"] == K8X2 else 1)
    # as configured where the caller says so
    assert shape(sizes(ns), 10**6, warps=8, occupancy=2)["kernel"] == K8X2
    assert shape(sizes(ns), 10**6, warps=8)["kernel"] == K8


def test_configured_occupancy_is_honoured(shape):
    """A caller that sets the blocks per SM and leaves the warps to the default gets the 8-warp kernels."""
    for z in (sizes(36, factors=FACTORS), sizes(9, hot=6_000, cold=2_000, slots=50)):
        assert [shape(z, 10**6, occupancy=o)["kernel"] for o in (1, 2)] == [K8, K8X2]


def test_line_of_the_default_shapes(shape):
    """Where only the device knows the number of cells both sides of the line are launched: each gets the cells that
    the rule gives it."""
    for z in (sizes(36, factors=FACTORS), sizes(9, hot=6_000, cold=2_000, slots=50), sizes(31)):
        at = shape(z, 10**6)["from"]
        for n in (1, at - 1, at, 10**5):
            few = n < at
            assert shape(z, max(n, 1))["kernel"] == shape(z, 1 if few else 10**6)["kernel"]
    assert [shape(sizes(36, factors=FACTORS), 10**6, **kw)["from"] for kw in (dict(warps=12), dict(occupancy=2))] == [0, 0]
    assert shape(sizes(31), 10**6)["from"] == 0  # one block resident: one shape


def test_every_status_is_documented_and_leaves_an_accepted_state():
    """The statuses of the kernel are those the public header lists, and an exit between a step's prediction and
    its acceptance takes the prediction back first (the cell's state is written as it then is)."""
    def read(*p):
        with open(os.path.join(CSRC, *p)) as f:
            return f.read()

    enum = re.search(r"enum \{ (ST_OK[^}]*)\}", read("solver.cuh")).group(1)
    codes = {int(v): k for k, v in re.findall(r"(ST_\w+) = (\d+)", enum) if k != "ST_PENDING"}
    doc = " ".join(read("..", "..", "include", "tiger_chem.h").replace("\n *", " ").split())
    listed = re.search(r"status \((0 ok, .*?)\)", doc).group(1)
    assert [int(v) for v in re.findall(r"(?:^|, )(\d) ", listed)] == sorted(codes)
    kernel = read("bdf_kernel.cuh")
    attempt = kernel[kernel.index("z_predict<two>(z, q);"):kernel.index("// accept\n")]
    failing = [m.start() for m in re.finditer(r"\bfail = true;", attempt)]
    assert failing
    for at in failing:
        block = attempt[attempt.rindex("if (uni(", 0, at) - 250:at]
        assert "z_retract<two>(z, q);" in block, block
