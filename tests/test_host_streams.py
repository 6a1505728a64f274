"""CPU tests of the host side's stream ordering: calls in flight on several
streams share buffers of the engine only in order, whatever the streams' timing
(tests/fake_cudart.cpp records who waits for whom; no kernel runs)."""
from __future__ import annotations

import threading
import time

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


def fused_calls(fake, eng, key, stream):
    """Every kind of call that may take the fused kernel, one after the other."""
    cmd = fake.cmd
    yield lambda: cmd.decrypt_device(eng, key, 0x1000, 30000, 0x1000, 0, stream)
    yield lambda: cmd.decrypt_device(eng, key, 0x1000, 500, 0x1000, 0, stream, "fused")
    yield lambda: cmd.decrypt_positions_device(eng, key, 0x1000, 37888, 0x1000, stream)
    yield lambda: mixed(fake, eng, [key], np.zeros(40000), stream)


def test_a_fused_launch_has_its_work_counter_to_itself(fake):
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, 348864, golden_sk(348864))
        n = 0
        for i in range(30):
            for job in fused_calls(fake, eng, key, fake.stream()):
                fake.call(n := n + 1)
                job()
        ops = fake.ops()
        zeroed = [o for o in ops if o.name == "memset"]
        kernel = {o.call: o for o in ops if "k_fused" in o.name}
        assert len(zeroed) == n == len(kernel)
        for i, m in enumerate(zeroed):
            for before in zeroed[:i]:
                assert not m.writes(before) or m.after(kernel[before.call]), (before.call, m.call)
        # launches on different streams do not wait for one another needlessly
        assert not zeroed[4].after(kernel[1])
        key.free()


def test_a_captured_launch_keeps_its_work_counter(fake):
    """A graph zeroes its counter at every replay: no other launch may use it."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, 348864, golden_sk(348864))
        streams, live = [fake.stream() for _ in range(2)], 0
        for i in range(2000):
            s = streams[i % 2]
            fake.call(i % 2)
            if i % 2:
                fake.begin_capture(s, GLOBAL_CAPTURE)
                cmd.decrypt_device(eng, key, 0x1000, 5000, 0x1000, 0, s)
                assert fake.end_capture(s) == 0
            else:
                cmd.decrypt_device(eng, key, 0x1000, 30000, 0x1000, 0, s)
        zeroed = [o for o in fake.ops() if o.name == "memset"]
        captured = {o.dst for o in zeroed if o.call == 1}
        assert len(captured) == 1000 and not captured & {o.dst for o in zeroed if o.call == 0}
        key.free()


@pytest.mark.parametrize("first", ["decap", "plain", "tile", "tile_small", "synd"])
@pytest.mark.parametrize("then", ["decap", "plain", "tile", "tile_small", "synd"])
def test_the_engines_scratch_is_reused_after_its_last_use(fake, first, then):
    """Error rows of a decapsulation, intermediates of the plain and tile paths."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, 348864, golden_sk(348864))
        cmd.prepare_decap(eng, key)
        jobs = {"decap": lambda s: cmd.kem_decap_device(eng, key, 0x1000, 20000, 0x1000, 0x1000, s),
                "plain": lambda s: cmd.decrypt_device(eng, key, 0x1000, 300, 0x1000, 0, s, "plain"),
                "tile": lambda s: cmd.decrypt_device(eng, key, 0x1000, 5000, 0x1000, 0, s, "tile"),
                "tile_small": lambda s: cmd.decrypt_device(eng, key, 0x1000, 100, 0x1000, 0, s, "tile"),
                "synd": lambda s: cmd.lib().cmd_stage_synd_fft(eng.handle, key.handle, 0x1000, 40, 0x1000, s)}
        a, b = fake.stream(), fake.stream()
        jobs["tile"](a)  # grown: no call below moves it
        jobs["decap"](a)
        fake.call(1)
        jobs[first](a)
        fake.call(2)
        jobs[then](b)
        ops = fake.ops()
        one, two = ([o for o in ops if o.call == i] for i in (1, 2))
        assert one and two
        assert all(o.after(one[-1]) for o in two)
        key.free()


def test_an_older_tuners_file_is_tuned_again(fake, tmp_path, monkeypatch):
    """Its crossover was against the fused kernel; today's is against the staged ones."""
    cmd = fake.cmd
    path = tmp_path / "tune.json"
    path.write_text('{\n  "host test|348864": {"wpb": 4, "balanced": 0, "ns_per_ct": 50.0, "tile_below": 8192}\n}\n')
    monkeypatch.setenv("CMD_TUNE_CACHE", str(path))
    for tuned in (False, True):
        with cmd.Engine(0) as eng:
            key = cmd.Key(eng, 348864, golden_sk(348864))
            fake.rt.fake_clear()
            assert cmd.tune(eng, key)["tile_below"] == 0  # equal times: not faster
            assert bool(fake.ops()) != tuned  # the second engine reads what the first one wrote
            fake.rt.fake_clear()
            cmd.decrypt_device(eng, key, 0x1000, 5000, 0x1000)
            assert any("k_bm_tile" in o.name for o in fake.ops())
            key.free()


def test_host_decapsulations_of_two_threads_take_turns(fake):
    """From the copy of the ciphertexts to that of the keys: both use the same
    device buffers."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, 348864, golden_sk(348864))
        cts = np.zeros((100, key.info.ct_bytes), np.uint8)
        cmd.kem_decap(eng, key, cts)
        fake.rt.fake_clear()
        fake.rt.fake_pause(300)

        def work(i):
            for j in range(20):
                fake.call(1 + 2 * j + i)
                cmd.kem_decap(eng, key, cts)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        calls = [o.call for o in fake.ops()]
        assert len(set(calls)) == 40
        assert sum(a != b for a, b in zip(calls, calls[1:])) == 39  # each call's operations in one run
        key.free()


@pytest.mark.parametrize("job", ["plain", "tile", "synd", "decap", "graph"])
def test_scratch_in_a_graph_outlives_its_growth(fake, job):
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key, s = cmd.Key(eng, 348864, golden_sk(348864)), fake.stream()
        cmd.prepare_decap(eng, key)
        cmd.decrypt_device(eng, key, 0x1000, 1 << 20, 0x1000)  # all the scratch a decapsulation's decrypt takes
        jobs = {"plain": lambda n: cmd.decrypt_device(eng, key, 0x1000, n, 0x1000, 0, s, "plain"),
                "tile": lambda n: cmd.decrypt_device(eng, key, 0x1000, n, 0x1000, 0, s, "tile"),
                "synd": lambda n: cmd.lib().cmd_stage_synd_fft(eng.handle, key.handle, 0x1000, n, 0x1000, s),
                "decap": lambda n: cmd.kem_decap_device(eng, key, 0x1000, n, 0x1000, 0x1000, s)}
        if job == "graph":
            cmd.Graph(eng, key, 0x1000, 5000, 0x1000, path="plain")
        else:
            jobs[job](5000)
            fake.begin_capture(s, GLOBAL_CAPTURE)
            jobs[job](5000)
            assert fake.end_capture(s) == 0
        held = fake.blocks()
        for n in (200000, 300000):
            jobs["decap"](n)
            jobs["plain"](n)
        later = fake.blocks()
        assert held <= later  # what the graph may use
        jobs["decap"](1000000)
        assert held <= fake.blocks() and not later <= fake.blocks()  # and no more than that
        key.free()


def test_a_captured_mixed_batch_keeps_its_work_lists(fake):
    """On the device: a copy in the graph would read the call's host vectors at every
    replay, and the engine's own lists are rewritten by the next batch."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        keys, s = [cmd.Key(eng, x, golden_sk(x)) for x in (348864, 6960119)], fake.stream()
        for warm in (False, True):
            fake.rt.fake_clear()
            fake.begin_capture(s, GLOBAL_CAPTURE)
            mixed(fake, eng, keys, np.arange(1000) % 2, s)
            assert fake.end_capture(s) == 0
            ops = fake.ops()
            kernel = next(o for o in ops if "k_fused" in o.name)
            lists = [o for o in ops if o.name == "h2d"]
            assert lists and not [o for o in lists if o.stream == kernel.stream]
            assert any(o.dst == kernel.arg[0] for o in lists)  # FusedArgs::tiles
            held = fake.blocks()
            fake.rt.fake_clear()
            mixed(fake, eng, keys, np.arange(47000) % 2, s)
            assert not [o for o in fake.ops() if any(o.writes(x) for x in lists)]
            assert held <= fake.blocks()
        for k in keys:
            k.free()


def test_server_batches_take_their_kernels_by_what_is_in_flight(fake):
    """The per-ciphertext kernels do more work for a ciphertext than the tile kernels:
    they are for a GPU with few ciphertexts on it, not for one batch of many."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng, cmd.Server(eng, max_batch=2000, slots=16, max_wait_us=0) as srv:
        kid = srv.add_key(348864, golden_sk(348864))
        cts, rows = np.zeros((2000, 208), np.uint8), np.zeros((2000, 1024), np.uint8)

        def batch():
            fake.rt.fake_clear()
            before = srv.stats()["batches"]
            srv.submit_many(np.full(2000, kid, np.uint32), cts, rows)
            until = time.monotonic() + 20
            while srv.stats()["batches"] == before and time.monotonic() < until:
                time.sleep(0.001)
            names = [o.name for o in fake.ops() if "k_" in o.name]
            assert any("k_ct" in n for n in names) != any("k_tile_bm" in n for n in names)
            return any("k_ct" in n for n in names)

        assert batch()  # (expands the key)
        srv.drain()
        fake.rt.fake_hold(1)
        try:
            kinds = [batch() for _ in range(10)]
        finally:
            fake.rt.fake_hold(0)
        assert kinds[0] and not kinds[-1] and kinds == sorted(kinds, reverse=True)
        srv.drain()
        assert batch()
        srv.drain()


@pytest.mark.parametrize("count,sets", [(1, 2), (44, 2), (45, 1), (74, 1), (300, 1)])
def test_seed_chains_of_a_key_generation(fake, count, sets):
    """A second set of chains ahead of the rounds, while their slots leave the GPU room."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        cmd.kem_keypair_batch(eng, 348864, np.zeros((count, 32), np.uint8))
        names = [o.name for o in fake.ops()]
        first = next(i for i, n in enumerate(names) if "k_kg_fill" in n)
        assert sum("k_kg_expand" in n for n in names[:first]) == sets


def test_scratch_grows_beside_another_streams_capture(fake):
    """In the default mode an allocation by any thread would end that capture."""
    cmd = fake.cmd
    with cmd.Engine(0) as eng:
        key, a, b = cmd.Key(eng, 348864, golden_sk(348864)), fake.stream(), fake.stream()
        cmd.decrypt_device(eng, key, 0x1000, 30000, 0x1000, 0, b)
        fake.begin_capture(a, GLOBAL_CAPTURE)
        for n in (3000, 5000, 100000):
            cmd.decrypt_device(eng, key, 0x1000, n, 0x1000, 0, b)
            cmd.decrypt_positions_device(eng, key, 0x1000, n, 0x1000, b)
            mixed(fake, eng, [key], np.zeros(n), b)
        assert fake.end_capture(a) == 0
        key.free()
