"""What the loops with gradients queue (csrc/quad_loop.cu), walked on the CPU: a kernel that may start while the one ahead of it still runs
must not read, before it has waited, what that one writes. On a GPU the mistake would show as a race, if at all."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "gridnet_b200", "csrc")
OUTER = 4


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("queue") / "loop_queue")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", exe, os.path.join(HERE, "loop_queue.cu"),
                    os.path.join(CSRC, "quad_loop.cu")], check=True)
    return exe


def walk(program, form, sets, border, kept):
    out = subprocess.run([program, form, str(sets), str(OUTER), str(border), str(kept)], check=True, capture_output=True, text=True).stdout
    return [(name, set(ahead.split()), set(writes.split())) for name, ahead, writes in (line.split(";") for line in out.splitlines())]


@pytest.mark.parametrize("kept", [0b1111, 0b1100, 0b1010, 0])
@pytest.mark.parametrize("border", [0, 1])
@pytest.mark.parametrize("form,sets", [("plain", 1), ("plain", OUTER), ("residual", 1), ("residual", OUTER), ("gated", 1)])
def test_nothing_is_read_ahead_that_the_kernel_before_writes(program, form, sets, border, kept):
    kernels = walk(program, form, sets, border, kept)
    for (before, _, writes), (name, ahead, _) in zip(kernels, kernels[1:]):
        assert not writes & ahead, f"{name} reads ahead what {before} writes"
    # the order that the rest of this test takes for granted
    names = [name for name, _, _ in kernels]
    assert names.count("reverse") + names.count("gated_reverse") == names.count("wgrad") == OUTER
    assert names.count("prepare") == 2 * sets


@pytest.mark.parametrize("form,sets,late", [("plain", 1, 0), ("plain", OUTER, OUTER - 1), ("residual", 1, 1), ("residual", OUTER, OUTER), ("gated", 1, 0)])
def test_parameters_are_loaded_ahead_wherever_they_may_be(program, form, sets, late):
    """Only a reverse sweep queued right behind the re-ordering of its parameters waits before it loads them (sums in the border pass, all
    iterations kept)."""
    kernels = walk(program, form, sets, 1, (1 << OUTER) - 1)
    behind = sum(before == "prepare" and name.endswith("reverse") for (before, _, _), (name, _, _) in zip(kernels, kernels[1:]))
    assert behind == late
    assert sum(name.endswith("reverse") and not ahead for name, ahead, _ in kernels) == late


def longest_quarter(items, quads, quarters, unit):
    """Cycles of an iteration, times the rounds that the slowest quarter needs: two warps share a region, a lone one is faster than two."""
    worst = 0
    for w in range(quarters):
        at, end = items // unit * w // quarters * unit, items // unit * (w + 1) // quarters * unit
        cost = 0
        while at < end:
            here = min(end, (at // quads + 1) * quads) - at  # of one region
            cost += here // 2 * 2 * 2820 + here % 2 * 3100
            at += here
        worst = max(worst, cost)
    return worst


def test_items_are_split_so_that_the_longest_quarter_is_shortest(program):
    """The rule against a walk through every quarter, on a GPU of 6 SMs: grids of up to 40 regions, batches of up to 18 quads. In pairs or
    one by one, whichever is over first."""
    out = subprocess.run([program, "split", "40", "6", "18"], check=True, capture_output=True, text=True).stdout
    units = set()
    for line in out.splitlines():
        regions, quads, ctas, unit = map(int, line.split())
        items = regions * quads
        assert unit == 1 or (unit == 2 and quads % 2 == 0), line
        one = longest_quarter(items, quads, 4 * ctas, 1)
        best = min(one, longest_quarter(items, quads, 4 * ctas, 2)) if quads % 2 == 0 else one
        assert longest_quarter(items, quads, 4 * ctas, unit) == best, line
        units.add(unit)
    assert units == {1, 2}
