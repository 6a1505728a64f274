"""CPU tests of what the engine does when device memory is short: the calls that
can do without scratch fall back to the fused kernel, and scratch kept between
calls is bounded and given back (tests/fake_cudart.cpp; no kernel runs)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import golden_sk
from fake_cuda import GLOBAL_CAPTURE, Fake  # noqa: F401
from test_host_streams import built, fake, mixed  # noqa: F401


def scratch_calls(fake, eng, key, sizes):  # noqa: F811
    """Calls that take scratch when they can have it."""
    cmd = fake.cmd
    for n in sizes:
        yield lambda: cmd.decrypt_device(eng, key, 0x1000, n, 0x1000, 0x1000)
        yield lambda: cmd.decrypt_positions_device(eng, key, 0x1000, n, 0x1000)
    for n in sizes[:-1]:  # (the work lists of the largest would have to grow)
        yield lambda: mixed(fake, eng, [key], np.zeros(n), 0)


@pytest.mark.parametrize("grown", [False, True])
def test_a_full_gpu_leaves_the_fused_kernel(fake, grown):  # noqa: F811
    """cudaMalloc fails although the budget would allow the scratch: the budget is a
    share of what was free when the engine was created."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, 6960119, golden_sk(6960119))
        mixed(fake, eng, [key], np.zeros(40000), 0)  # work lists
        for job in scratch_calls(fake, eng, key, (10000, 70000) if grown else (3000, 5000, 70000)):
            fake.rt.fake_largest_malloc(2 ** 63)
            if grown:  # the scratch is there but has to grow, and loses what it had
                cmd.decrypt_device(eng, key, 0x1000, 4000, 0x1000)
            used = eng.memory()[0]
            fake.rt.fake_largest_malloc(0)
            fake.rt.fake_clear()
            job()
            assert [o.name for o in fake.ops() if "k_fused" in o.name]
            assert eng.memory()[0] <= used
        key.free()
