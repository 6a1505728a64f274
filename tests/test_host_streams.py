"""CPU tests of the host side's stream ordering: calls in flight on several
streams share buffers of the engine only in order, whatever the streams' timing
(tests/fake_cudart.cpp records who waits for whom; no kernel runs)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import golden_sk
from fake_cuda import GLOBAL_CAPTURE, Fake


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    return Fake(str(tmp_path_factory.mktemp("fake")))


@pytest.fixture
def fake(built):
    built.reset()
    yield built
    built.reset()


def mixed(fake, eng, keys, key_idx, stream):
    cmd = fake.cmd
    key_idx = np.asarray(key_idx, np.uint32)
    ct = np.array([k.info.ct_bytes for k in keys], np.uint64)[key_idx]
    nw = np.array([k.info.err_words for k in keys], np.uint64)[key_idx]
    off = lambda n: (np.cumsum(n) - n).astype(np.uint64)
    cmd.decrypt_mixed_device(eng, keys, key_idx, 0x1000, off(ct), 0x1000, off(nw), 0, stream)


# 148 SMs: up to 3,552 ciphertexts the per-ciphertext kernels, from 28,417 to
# 47,360 the fused kernel, the staged ones between and above
@pytest.mark.parametrize("first,then", [(10000, 40000), (40000, 10000), (40000, 30000), (1000, 40000), (50000, 5000)])
def test_mixed_lists_are_rewritten_after_their_last_use(fake, first, then):
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        keys = [cmd.Key(eng, s, golden_sk(s)) for s in (348864, 6960119)]
        streams = [fake.stream() for _ in range(2)]
        for i, count in enumerate((then, first, then)):  # the first of them: buffers grown
            fake.call(i)
            mixed(fake, eng, keys, np.arange(count) % 2, streams[i % 2])
        ops = fake.ops()
        kernels = [o for o in ops if o.call == 1 and not o.bytes]
        wrote = [o for o in ops if o.call == 1 and o.name == "h2d"]
        assert kernels and wrote
        for o in ops:
            if o.call == 2 and any(o.writes(w) for w in wrote):
                assert all(o.after(k) for k in kernels), (o.name, o.dst)
        for k in keys:
            k.free()


@pytest.mark.parametrize("count", [1, 3000, 5000, 30000, 70000])
def test_auto_is_captured_after_a_warm_up_of_its_own(fake, count):
    """In the default capture mode, where an allocation would end the capture."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key, s = cmd.Key(eng, 348864, golden_sk(348864)), fake.stream()
        cmd.decrypt_device(eng, key, 0x1000, count, 0x1000, 0x1000, s)
        fake.begin_capture(s, GLOBAL_CAPTURE)
        cmd.decrypt_device(eng, key, 0x1000, count, 0x1000, 0x1000, s)
        cmd.decrypt_positions_device(eng, key, 0x1000, count, 0x1000, s)
        assert fake.end_capture(s) == 0
        key.free()
