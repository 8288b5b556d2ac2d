"""Stages are launched as programmatic dependents: up to three are resident at once, and the
buffer one of them reads is the one the next writes.  So a kernel that may be launched that
way reads the states and the LSRK register by coherent loads behind its wait, and only tables
that no kernel writes through the read-only path.

The rule is about which loads the source asks for, so this is checked on the source; the
GPU test runs the chains in which the launches overlap most."""
import glob
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nekwave_b200", "csrc")
# arrays that are written before the first launch and never again
TABLES = r"(&?Gp->|P\.(fplus|fnrm|flift|conn|met_n)\b)"


def source(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def overlapped_sources():
    """Every file with kernels that launch_overlapped() launches, and their headers."""
    files = sorted(glob.glob(os.path.join(CSRC, "stage_*.cu*")) + glob.glob(os.path.join(CSRC, "batch.cu*")))
    assert len(files) >= 10
    return files


@pytest.mark.parametrize("path", overlapped_sources(), ids=os.path.basename)
def test_read_only_loads_take_tables_only(path):
    for arg in re.findall(r"__ldg\(([^;]*)", source(path)):
        assert re.match(TABLES, arg.replace("reinterpret_cast<const double2*>(", "")), arg


def test_probe_kernel_reads_the_state_coherently():
    text = source(os.path.join(CSRC, "diag_kernels.cu"))
    kernel = re.search(r"\bprobe_kernel\(.*?\n}\n", text, re.S).group(0)
    assert not re.search(r"__restrict__\s+u\b", kernel) and "__ldg" not in kernel


@pytest.mark.gpu
@pytest.mark.parametrize("N", range(2, 11))
def test_queued_steps_equal_waited_ones(gpu, N):
    """150 queued steps of a small box, with probes read between, and the same steps waited
    for one by one: the same bits."""
    from nekwave_b200 import DgSolver
    pulses = [(1.0 - 0.2 * c, 0.4, 0.6, 0.5, 0.2 + 0.05 * c) for c in range(6)]

    def run(waits):
        s = DgSolver("fp64")
        s.initializeBox(N, (4, 4, 4), (0, 0, 0), (1, 1, 1), 1.0)
        s.initPulse(pulses)
        s.probeSetup([0, 63 * N ** 3], np.full((2, N ** 3), 1.0 / N ** 3))
        seen = []
        for _ in range(3):
            for n in [1] * 50 if waits else [50]:
                s.steps(1e-4, n, sync=waits)
            seen.append(s.probeRead())
        state = s.downloadState()
        s.finalize()
        return np.array(seen), state

    for a, b in zip(run(False), run(True)):
        np.testing.assert_array_equal(a, b)
