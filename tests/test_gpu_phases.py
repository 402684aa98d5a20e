"""The phase counter: the clocked call returns the plain call's bits, and takes about its time, so that its shares of
the cycles are the plain call's."""

import numpy as np
import pytest
import torch

from maxichem_b200 import abi, synthetic
from maxichem_b200.solver import CudaSolver

pytestmark = pytest.mark.gpu


def milliseconds(call) -> float:
    times = []
    for _ in range(6):  # the first one warms up
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        call()
        e1.record()
        torch.cuda.synchronize()
        times.append(e0.elapsed_time(e1))
    return min(times[1:])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["cho41", "chno69"])  # 2 and 4 warps a cell
def test_the_clocked_call_stands_for_the_plain_one(gpu, networks, name, precision):
    net = networks(name)
    w = synthetic.workload(net, "column", 2048, seed=6)
    args = [torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=gpu) for a in (w.x, w.T, w.P, w.dt, w.h)]
    J = torch.as_tensor(w.J, dtype=torch.float64, device=gpu)
    cycles = torch.zeros(8, dtype=torch.int64, device=gpu)
    with CudaSolver(net, gpu, photo=True, precision=precision) as solver:
        plain = solver.launch(*args, J=J)
        fast = milliseconds(lambda: solver.launch(*args, J=J))
        assert abi.library().mx_set_phase_counter(solver._handle, cycles.data_ptr()) == 0
        clocked = solver.launch(*args, J=J)
        slow = milliseconds(lambda: solver.launch(*args, J=J))
        assert abi.library().mx_set_phase_counter(solver._handle, None) == 0
    assert all(torch.equal(a, b) for a, b in zip(plain, clocked, strict=True))
    assert bool((cycles > 0).all())
    # a clock read a phase costs a few of its thousands of cycles, its sums some registers
    assert slow <= 1.2 * fast, (slow, fast, (cycles / cycles.sum()).tolist())
    print(name, precision, f"{fast:.3f} {slow:.3f} ms", [round(v, 3) for v in (cycles / cycles.sum()).tolist()])
