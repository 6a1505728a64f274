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


def test_a_mixed_batchs_scratch_is_bounded(fake):  # noqa: F811
    """By that of four parts of a single-key batch, however many keys cut the batch
    into partly filled tiles; the passes over the scratch follow one another."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        keys = [cmd.Key(eng, s, golden_sk(s)) for s in (348864, 6960119, 8192128)]
        cmd.decrypt_device(eng, keys[2], 0x1000, 1 << 20, 0x1000)
        single = eng.memory()[0]
        n = 20000
        fake.rt.fake_clear()
        mixed(fake, eng, [keys[i % 3] for i in range(n)], np.arange(n), 0)  # a key each
        assert eng.memory()[0] <= single + (4 << 20)  # the work lists
        synd, nets = ([o for o in fake.ops() if name in o.name] for name in ("k_synd_table", "k_net_rows"))
        assert len(synd) == len(nets) == 5  # 8192128, 6960119; the rest, 348864; the rest
        for i, o in enumerate(synd):
            # ordered after the rows of every earlier pass, beside those of its own
            done = [j for j, net in enumerate(nets) if o.after(net)]
            assert done == list(range((0, 0, 2, 2, 4)[i])), i
        for k in keys:
            k.free()


def keys_that_fit(fake, eng):  # noqa: F811
    cmd, keys = fake.cmd, []
    try:
        while True:
            keys.append(cmd.Key(eng, 8192128, golden_sk(8192128)))
    except cmd.CmdError as e:
        assert e.code == cmd.CMD_E_BUDGET
    n = len(keys)
    for k in keys:
        k.free()
    return n


def test_kept_scratch_is_given_back(fake):  # noqa: F811
    """To what the budget or the device would otherwise refuse: keys, a server, key
    generation, decapsulation, the buffers of a host batch."""
    cmd = fake.cmd

    def engine():
        eng = cmd.Engine(0, hbm_budget=200 << 20)
        return eng, cmd.Key(eng, 8192128, golden_sk(8192128))

    def warm(eng, key):  # staged scratch of 100 MB and more
        mixed(fake, eng, [key], np.zeros(75000), 0)
        assert eng.memory()[0] > 100 << 20

    eng, key = engine()
    fits = keys_that_fit(fake, eng)
    warm(eng, key)
    assert keys_that_fit(fake, eng) >= fits - 2  # the mixed batch's work lists, 2 MB, stay
    key.free()
    eng.close()
    host = np.zeros((65535, 208), np.uint8)
    for job in (lambda e, k: cmd.Server(e, max_batch=16384, slots=4).close(),
                lambda e, k: cmd.lib().cmd_stage_synd_fft(e.handle, k.handle, 0x1000, 250000, 0x1000, None),
                lambda e, k: cmd.decrypt(e, k, host, path="fused"),
                lambda e, k: cmd.kem_decap(e, k, host)):
        eng, key = engine()
        job(eng, key)  # fits
        key.free()
        eng.close()
        eng, key = engine()
        warm(eng, key)
        job(eng, key)
        assert eng.memory()[0] <= 200 << 20
        key.free()
        eng.close()
    # the device's memory rather than the budget
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, 8192128, golden_sk(8192128))
        warm(eng, key)
        fake.rt.fake_total(fake.rt.fake_allocated() + (1 << 20))
        more = cmd.Key(eng, 8192128, golden_sk(8192128))
        cmd.prepare_decap(eng, more)
        assert eng.memory()[0] < 100 << 20
        key.free()
        more.free()
