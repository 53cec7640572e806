"""Calls that run out of device memory half-way report it and leave the context
usable: the same call succeeds once there is memory again. The memory is taken
by this process, up to a few MB that are left for the call to start with.
"""
import numpy as np
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import cases
from pfem2_b200.solver import Pfem2Error, Solver

pytestmark = pytest.mark.gpu

MB = 1 << 20


class NoMemory:
    """all device memory but about `left` bytes"""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch

        torch.cuda.synchronize()
        self.held = []
        size = torch.cuda.mem_get_info()[0] - self.left
        while size >= 2 * MB:  # (what is free is not one piece)
            try:
                self.held.append(torch.empty(size // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:
                size //= 2
            size = min(size, torch.cuda.mem_get_info()[0] - self.left)

    def __exit__(self, *exc):
        import torch

        self.held.clear()
        torch.cuda.empty_cache()


def test_mesh_elasticity():
    sp = cases.channel_disk(h=float(np.sqrt(4.0 / 30000)))

    def solve(s):
        s.problem_of_elasticity(1.0, 1.0, (1, 2, 4), 3, (0.0, 0.002), rtol=1e-10)
        return s.field(A.FIELD_DISP_X), s.field(A.FIELD_DISP_Y)

    first = Solver(sp, precision=A.PREC_FP64, moving_mesh=True)
    want = solve(first)
    failed = []
    for left in range(2, 62, 4):
        s = Solver(sp, precision=A.PREC_FP64, moving_mesh=True)
        with NoMemory(left * MB):
            try:
                solve(s)
            except Pfem2Error as e:
                assert e.status == A.CUDA_ERROR and "cudaMalloc" in str(e)
                failed.append(left)
        for x, y in zip(solve(s), want):
            assert np.array_equal(x, y), left
        s.close()
    first.close()
    assert len(failed) >= 2, failed  # at more than one of the call's allocations


def test_seed():
    """a context that cannot hold the particles asked for has none"""
    sp = cases.channel_disk(h=float(np.sqrt(4.0 / 30000)))
    kw = dict(precision=A.PREC_FP64, particles_only=True)
    first = Solver(sp, **kw)
    first.seed_particles((5, 5), 1, 0.1)
    first.step()
    want = first.particles()
    failed = []
    for left in range(6, 166, 20):
        s = Solver(sp, **kw)
        s.seed_particles((1, 1), 1, 0.1)
        s.step()
        with NoMemory(left * MB):
            try:
                s.seed_particles((5, 5), 1, 0.1)
            except Pfem2Error as e:
                assert e.status == A.CUDA_ERROR
                failed.append(left)
                for call in (s.step, s.move_particles, s.particles):
                    with pytest.raises(Pfem2Error) as e:
                        call()
                    assert e.value.status == A.BAD_STATE
        s.seed_particles((5, 5), 1, 0.1)
        s.step()
        for x, y in zip(s.particles(), want):
            assert np.array_equal(x, y), left
        s.close()
    first.close()
    assert len(failed) >= 2, failed
