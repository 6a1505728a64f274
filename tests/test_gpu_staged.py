"""The staged kernels (CMD_PATH_AUTO above the small batches): every batch size at
which their launches change shape, against the fused kernel (itself checked
against the oracle), bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import cm_decrypt__b200 as cmd
from conftest import golden_sk
from test_gpu_small_batches import degenerate

pytestmark = pytest.mark.gpu

# tiles of 32 an SM (148 SMs): 1, 2, 4, 6 (fused up to 8), then two and more parts
EDGES = (3553, 4736, 4737, 9472, 9473, 18944, 18945, 28416, 28417, 37889, 45000, 45001, 45089, 131072, 131073)


def batch(s: int, count: int) -> tuple[cmd.SetInfo, torch.Tensor]:
    info = cmd.set_info(s)
    valid, _, _ = cmd.PubKey(s, golden_sk(s)).ciphertexts(seed=41, count=4000, malformed_permille=80)
    cts = torch.from_numpy(np.concatenate([degenerate(info), valid])).cuda()
    g = torch.Generator(device="cuda").manual_seed(7)
    return info, cts[torch.randint(0, cts.shape[0], (count,), generator=g, device="cuda")].contiguous()


def run(engine, key, cts, path, first=0, count=None, stream=0):
    info, n = key.info, count or cts.shape[0] - first
    err = torch.full((n, info.err_words), -1, dtype=torch.int32, device="cuda")
    w = torch.full((n,), -1, dtype=torch.int16, device="cuda")
    torch.cuda.synchronize()
    cmd.decrypt_device(engine, key, cts.data_ptr() + first * info.ct_bytes, n, err.data_ptr(), w.data_ptr(), stream,
                       path)
    return err, w


@pytest.mark.parametrize("s", [348864, 460896, 6960119, 8192128])
def test_staged_sizes_match_fused(engine, s):
    info, cts = batch(s, max(EDGES) + 5)
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        want, want_w = run(engine, key, cts, "fused")
        torch.cuda.synchronize()
        for count in EDGES:
            for first in (0, 5):  # the second: ciphertexts not 16-byte aligned
                err, w = run(engine, key, cts, "auto", first, count)
                torch.cuda.synchronize()
                assert torch.equal(err, want[first:first + count]), (count, first)
                assert torch.equal(w, want_w[first:first + count]), (count, first)
        count = 50001
        pos = torch.zeros((count, info.t + 1), dtype=torch.int16, device="cuda")
        cmd.decrypt_positions_device(engine, key, cts.data_ptr(), count, pos.data_ptr())
        torch.cuda.synchronize()
        rows = want[:count].cpu().numpy().view(np.uint8)[:, :info.err_bytes]
        assert np.array_equal(pos.cpu().numpy().view(np.uint16)[-2000:], cmd.positions_from_errors(s, rows[-2000:]))
    finally:
        key.free()


def test_staged_streams_and_capture(engine):
    """Batches in flight on two streams share the engine's scratch, and under
    stream capture CMD_PATH_AUTO keeps to the fused kernel."""
    s = 348864
    info, cts = batch(s, 60000)
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        want, want_w = run(engine, key, cts, "fused")
        streams = [torch.cuda.Stream() for _ in range(2)]
        sizes = [60000, 5000, 50000, 20000]
        outs = [(torch.zeros((n, info.err_words), dtype=torch.int32, device="cuda"),
                 torch.zeros(n, dtype=torch.int16, device="cuda")) for n in sizes]
        torch.cuda.synchronize()
        for i, (n, (err, w)) in enumerate(zip(sizes, outs)):
            cmd.decrypt_device(engine, key, cts.data_ptr(), n, err.data_ptr(), w.data_ptr(), streams[i % 2].cuda_stream)
        torch.cuda.synchronize()
        for n, (err, w) in zip(sizes, outs):
            assert torch.equal(err, want[:n]) and torch.equal(w, want_w[:n]), n
        err = torch.zeros((5000, info.err_words), dtype=torch.int32, device="cuda")
        graph = torch.cuda.CUDAGraph()
        side = torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=side):
            cmd.decrypt_device(engine, key, cts.data_ptr(), 5000, err.data_ptr(), 0, side.cuda_stream)
        assert not err.any()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(err, want[:5000])
    finally:
        key.free()


def test_mixed_sizes_match_plain(engine):
    """Mixed batches at the sizes where the kernels change (one launch, three
    launches, staged), keys of all sets, ciphertexts at odd offsets, against the
    plain path key by key."""
    sets = [348864, 460896, 6688128, 6960119, 8192128, 348864, 6960119]
    keys, pool, want = [], [], []
    rng = np.random.default_rng(5)
    try:
        for i, s in enumerate(sets):
            sk = cmd.synth_key(s, golden_sk(s), 1000 + i)
            keys.append(cmd.Key(engine, s, sk))
            cts, _, _ = cmd.PubKey(s, sk).ciphertexts(seed=50 + i, count=300, malformed_permille=100)
            pool.append(np.concatenate([degenerate(keys[-1].info), cts]))
            want.append(cmd.decrypt(engine, keys[-1], pool[-1], path="plain"))
        for count in (1, 64, 65, 1000, 3552, 3553, 20011):
            ki = rng.integers(0, len(sets) if count != 65 else 1, count).astype(np.uint32)
            which = np.array([rng.integers(0, len(pool[k])) for k in ki])
            sizes = np.array([pool[k].shape[1] for k in ki])
            off = np.concatenate([[3], 3 + np.cumsum(sizes + 1)]).astype(np.uint64)  # a byte between them
            buf = np.zeros(int(off[-1]), np.uint8)
            for c, (k, j) in enumerate(zip(ki, which)):
                buf[int(off[c]):int(off[c]) + sizes[c]] = pool[k][j]
            words = np.array([keys[k].info.err_words for k in ki])
            eoff = np.concatenate([[0], np.cumsum(words)]).astype(np.uint64)
            d, err = torch.from_numpy(buf).cuda(), torch.full((int(eoff[-1]),), -1, dtype=torch.int32, device="cuda")
            w = torch.full((count,), -1, dtype=torch.int16, device="cuda")
            torch.cuda.synchronize()
            cmd.decrypt_mixed_device(engine, keys, ki, d.data_ptr(), off[:-1], err.data_ptr(), eoff[:-1], w.data_ptr())
            torch.cuda.synchronize()
            got, got_w = err.cpu().numpy().view(np.uint8), w.cpu().numpy().view(np.uint16)
            for c, (k, j) in enumerate(zip(ki, which)):
                row = got[4 * int(eoff[c]):4 * int(eoff[c + 1])]
                nb = keys[k].info.err_bytes
                assert np.array_equal(row[:nb], want[k][0][j]) and not row[nb:].any(), (count, c)
                assert got_w[c] == want[k][1][j], (count, c)
    finally:
        for k in keys:
            k.free()


def test_small_batches_on_two_streams(engine):
    """Small batches in flight on two streams at once share the scratch between
    their kernels' launches in order, beside a larger batch."""
    s = 460896
    info, cts = batch(s, 8000)
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        want, want_w = run(engine, key, cts, "plain")
        streams = [torch.cuda.Stream() for _ in range(2)]
        jobs = [(first, n) for n in (3000, 100, 8000, 65, 3552) for first in (0, 31) if first + n <= 8000] * 4
        outs = [(torch.zeros((n, info.err_words), dtype=torch.int32, device="cuda"),
                 torch.zeros(n, dtype=torch.int16, device="cuda")) for _, n in jobs]
        torch.cuda.synchronize()
        for i, ((first, n), (err, w)) in enumerate(zip(jobs, outs)):
            cmd.decrypt_device(engine, key, cts.data_ptr() + first * info.ct_bytes, n, err.data_ptr(), w.data_ptr(),
                               streams[i % 2].cuda_stream)
        torch.cuda.synchronize()
        for (first, n), (err, w) in zip(jobs, outs):
            assert torch.equal(err, want[first:first + n]) and torch.equal(w, want_w[first:first + n]), (first, n)
    finally:
        key.free()


def test_mixed_batches_on_two_streams(engine):
    """Mixed batches in flight on two streams, of the sizes of all three kinds of
    kernels, each with its own order of the keys, rewrite the work lists in turn."""
    sets = [348864, 6960119, 460896]
    keys = [cmd.Key(engine, s, golden_sk(s)) for s in sets]
    try:
        pool = [batch(s, 300)[1] for s in sets]
        want = [run(engine, k, c, "plain") for k, c in zip(keys, pool)]
        torch.cuda.synchronize()
        rng = np.random.default_rng(11)
        jobs = []
        for n in (20000, 40000, 3000, 40000, 10000, 30000):
            ki = rng.integers(0, 3, n).astype(np.uint32)
            at = torch.from_numpy(rng.integers(0, 300, n)).cuda()
            ct = np.array([k.info.ct_bytes for k in keys], np.uint64)[ki]
            nw = np.array([k.info.err_words for k in keys], np.uint64)[ki]
            off, eoff = (np.cumsum(ct) - ct).astype(np.uint64), (np.cumsum(nw) - nw).astype(np.uint64)
            buf = torch.zeros(int(ct.sum()), dtype=torch.uint8, device="cuda")
            expect = torch.zeros(int(nw.sum()), dtype=torch.int32, device="cuda")
            for k in range(3):
                m = ki == k
                rows = at[torch.from_numpy(m).cuda()]
                for dst, src, o in ((buf, pool[k], off), (expect, want[k][0], eoff)):
                    w = torch.arange(src.shape[1], device="cuda")
                    dst[(torch.from_numpy(o[m].astype(np.int64)).cuda()[:, None] + w).reshape(-1)] = src[rows].reshape(-1)
            jobs.append((ki, buf, off, torch.full_like(expect, -1), eoff, expect))
        streams = [torch.cuda.Stream() for _ in range(2)]
        torch.cuda.synchronize()
        for i, (ki, buf, off, err, eoff, _) in enumerate(jobs):
            cmd.decrypt_mixed_device(engine, keys, ki, buf.data_ptr(), off, err.data_ptr(), eoff, 0,
                                     streams[i % 2].cuda_stream)
        torch.cuda.synchronize()
        for i, job in enumerate(jobs):
            assert torch.equal(job[3], job[5]), i
    finally:
        for k in keys:
            k.free()


@pytest.mark.parametrize("count", [40, 5000])
def test_capture_after_an_auto_warm_up_only(count):
    """On an engine of its own, so that no other call has prepared anything."""
    s = 348864
    info, cts = batch(s, count)
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, s, golden_sk(s))
        try:
            want, _ = run(eng, key, cts, "auto")
            err = torch.zeros_like(want)
            torch.cuda.synchronize()
            graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.graph(graph, stream=side):
                cmd.decrypt_device(eng, key, cts.data_ptr(), count, err.data_ptr(), 0, side.cuda_stream)
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(err, want)
            del graph
        finally:
            key.free()


def test_fused_batches_on_two_streams(engine):
    """Batches of the sizes that CMD_PATH_AUTO gives to the fused kernel, and a
    captured one, each with its own work counter."""
    s = 348864
    info, cts = batch(s, 60000)
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        want, want_w = run(engine, key, cts, "plain")
        streams = [torch.cuda.Stream() for _ in range(3)]
        jobs = [(n, path) for n, path in ((30000, "auto"), (37888, "auto"), (500, "fused"), (60000, "auto"))] * 6
        outs = [(torch.zeros((n, info.err_words), dtype=torch.int32, device="cuda"),
                 torch.zeros(n, dtype=torch.int16, device="cuda")) for n, _ in jobs]
        graph_err = torch.zeros((5000, info.err_words), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=streams[2]):
            cmd.decrypt_device(engine, key, cts.data_ptr(), 5000, graph_err.data_ptr(), 0, streams[2].cuda_stream)
        torch.cuda.synchronize()
        for i, ((n, path), (err, w)) in enumerate(zip(jobs, outs)):
            cmd.decrypt_device(engine, key, cts.data_ptr(), n, err.data_ptr(), w.data_ptr(), streams[i % 2].cuda_stream,
                               path)
            if i % 4 == 0:
                with torch.cuda.stream(streams[2]):
                    graph.replay()
        torch.cuda.synchronize()
        for (n, path), (err, w) in zip(jobs, outs):
            assert torch.equal(err, want[:n]) and torch.equal(w, want_w[:n]), (n, path)
        assert torch.equal(graph_err, want[:5000])
    finally:
        key.free()


@pytest.mark.parametrize("s,n", [(348864, 20000), (6688128, 3000)])
def test_decapsulations_on_two_streams(engine, s, n):
    """Beside one another and beside tile- and plain-path batches, which use the
    same scratch; also the 6688128 set at staged sizes."""
    info, cts = batch(s, 2 * n)
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        want = cmd.kem_decap(engine, key, cts.cpu().numpy())
        rows, _ = run(engine, key, cts, "fused")
        streams = [torch.cuda.Stream() for _ in range(2)]
        outs = [(torch.zeros((n, 32), dtype=torch.uint8, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda"))
                for _ in range(6)]
        errs = [torch.zeros((700, info.err_words), dtype=torch.int32, device="cuda") for _ in range(6)]
        torch.cuda.synchronize()
        for i in range(6):
            half = cts[i % 2 * n:]
            cmd.kem_decap_device(engine, key, half.data_ptr(), n, outs[i][0].data_ptr(), outs[i][1].data_ptr(),
                                 streams[i % 2].cuda_stream)
            cmd.decrypt_device(engine, key, half.data_ptr(), 700, errs[i].data_ptr(), 0, streams[i % 2].cuda_stream,
                               "plain" if i % 3 else "tile")
        torch.cuda.synchronize()
        for i, ((k, a), err) in enumerate(zip(outs, errs)):
            at = i % 2 * n
            assert np.array_equal(k.cpu().numpy(), want[0][at:at + n]), i
            assert np.array_equal(a.cpu().numpy(), want[1][at:at + n]), i
            assert torch.equal(err, rows[at:at + 700]), i
        assert want[1].any() and not want[1].all()
    finally:
        key.free()


def test_budget_without_room_for_scratch(engine):
    """The staged and small-batch scratch refused: the same results from the fused
    kernel, within the budget."""
    s = 6960119
    info, cts = batch(s, 50000)
    key = cmd.Key(engine, s, golden_sk(s))
    want, want_w = run(engine, key, cts, "fused")
    pos = torch.zeros((50000, info.t + 1), dtype=torch.int16, device="cuda")
    cmd.decrypt_positions_device(engine, key, cts.data_ptr(), 50000, pos.data_ptr())
    torch.cuda.synchronize()
    key.free()
    with cmd.Engine(0, hbm_budget=3 << 20) as eng:
        key = cmd.Key(eng, s, golden_sk(s))
        try:
            for n in (3000, 5000, 50000):
                err, w = run(eng, key, cts, "auto", 0, n)
                got = torch.zeros_like(pos[:n])
                cmd.decrypt_positions_device(eng, key, cts.data_ptr(), n, got.data_ptr())
                torch.cuda.synchronize()
                assert torch.equal(err, want[:n]) and torch.equal(w, want_w[:n]), n
                assert torch.equal(got, pos[:n]), n
            for n in (3000, 5000):
                err = torch.full((n, info.err_words), -1, dtype=torch.int32, device="cuda")
                step = np.arange(n, dtype=np.uint64)
                cmd.decrypt_mixed_device(eng, [key], np.zeros(n, np.uint32), cts.data_ptr(), step * info.ct_bytes,
                                         err.data_ptr(), step * info.err_words)
                torch.cuda.synchronize()
                assert torch.equal(err, want[:n]), n
            assert eng.memory()[0] <= eng.memory()[1]
        finally:
            key.free()


def test_mixed_batch_of_many_keys(engine):
    """A ciphertext or two a key: more tiles than one pass over the scratch holds."""
    sets = [348864, 6960119, 8192128]
    keys = [cmd.Key(engine, s, golden_sk(s)) for s in sets]
    try:
        pool = [batch(s, 200)[1] for s in sets]
        want = [run(engine, k, c, "plain") for k, c in zip(keys, pool)]
        n = 9500
        many = [keys[i % 3] for i in range(n - 500)]
        ki = np.arange(n, dtype=np.uint32) % (n - 500)
        ct = np.array([k.info.ct_bytes for k in many], np.uint64)[ki]
        nw = np.array([k.info.err_words for k in many], np.uint64)[ki]
        off, eoff = (np.cumsum(ct) - ct).astype(np.uint64), (np.cumsum(nw) - nw).astype(np.uint64)
        rows = np.arange(n) // 3 % 200
        host = [c.cpu().numpy() for c in pool]
        buf = torch.from_numpy(np.concatenate([host[k % 3][r] for k, r in zip(ki, rows)])).cuda()
        err = torch.full((int(nw.sum()),), -1, dtype=torch.int32, device="cuda")
        w = torch.full((n,), -1, dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        cmd.decrypt_mixed_device(engine, many, ki, buf.data_ptr(), off, err.data_ptr(), eoff, w.data_ptr())
        torch.cuda.synchronize()
        e, got_w = [x[0].cpu().numpy() for x in want], w.cpu().numpy()
        assert np.array_equal(err.cpu().numpy(), np.concatenate([e[k % 3][r] for k, r in zip(ki, rows)]))
        we = [x[1].cpu().numpy() for x in want]
        assert np.array_equal(got_w, np.array([we[k % 3][r] for k, r in zip(ki, rows)]))
    finally:
        for k in keys:
            k.free()


def test_captured_batches_outlive_larger_calls():
    """A mixed batch, a plain-path batch and a decapsulation captured on an engine of
    their own, replayed after larger calls have replaced its buffers."""
    sets = [348864, 460896]
    with cmd.Engine(0) as eng:
        keys = [cmd.Key(eng, s, golden_sk(s)) for s in sets]
        try:
            pool = [batch(s, 40000)[1] for s in sets]
            info, n = keys[0].info, 600
            cmd.prepare_decap(eng, keys[0])
            want = [run(eng, k, c, "plain", 0, n)[0] for k, c in zip(keys, pool)]
            session, accept = cmd.kem_decap(eng, keys[0], pool[0][:n].cpu().numpy())
            buf = torch.cat([c[:n].reshape(-1) for c in pool])
            err = torch.zeros(n * sum(k.info.err_words for k in keys), dtype=torch.int32, device="cuda")
            plain = torch.zeros((n, info.err_words), dtype=torch.int32, device="cuda")
            k32, acc = (torch.zeros((n, m), dtype=torch.uint8, device="cuda") for m in (32, 1))
            torch.cuda.synchronize()
            graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
            with torch.cuda.graph(graph, stream=side):
                ki = np.repeat(np.arange(2, dtype=np.uint32), n)
                ct = np.array([k.info.ct_bytes for k in keys], np.uint64)[ki]
                nw = np.array([k.info.err_words for k in keys], np.uint64)[ki]
                off, eoff = (np.cumsum(ct) - ct).astype(np.uint64), (np.cumsum(nw) - nw).astype(np.uint64)
                cmd.decrypt_mixed_device(eng, keys, ki, buf.data_ptr(), off, err.data_ptr(), eoff, 0, side.cuda_stream)
                cmd.decrypt_device(eng, keys[0], pool[0].data_ptr(), n, plain.data_ptr(), 0, side.cuda_stream, "plain")
                cmd.kem_decap_device(eng, keys[0], pool[0].data_ptr(), n, k32.data_ptr(), acc.data_ptr(), side.cuda_stream)
            for x in (ki, ct, nw, off, eoff):
                x.fill(2 ** 31)
            big = cmd.kem_decap(eng, keys[0], pool[0].cpu().numpy())
            assert np.array_equal(big[0][:n], session)
            run(eng, keys[1], pool[1], "plain")
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(err, torch.cat([w.reshape(-1) for w in want]))
            assert torch.equal(plain, want[0])
            assert np.array_equal(k32.cpu().numpy(), session) and np.array_equal(acc.cpu().numpy()[:, 0], accept)
            del graph
        finally:
            for k in keys:
                k.free()


def test_staged_edges_of_the_largest_t(engine):
    """6688128 (t = 128 at n < 2^13) at the sizes where the launches change shape."""
    s = 6688128
    info, cts = batch(s, max(EDGES))
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        want, want_w = run(engine, key, cts, "fused")
        for count in EDGES:
            err, w = run(engine, key, cts, "auto", 0, count)
            torch.cuda.synchronize()
            assert torch.equal(err, want[:count]) and torch.equal(w, want_w[:count]), count
    finally:
        key.free()


def test_growth_beside_another_streams_capture():
    """A larger batch on one stream, for which the scratch grows, while another
    stream is captured in the default mode."""
    s = 348864
    info, cts = batch(s, 100000)
    with cmd.Engine(0) as eng:
        key = cmd.Key(eng, s, golden_sk(s))
        try:
            want, _ = run(eng, key, cts, "fused")
            run(eng, key, cts, "auto", 0, 4000)
            err, small = torch.zeros_like(want), torch.zeros((5000, info.err_words), dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            graph, side, other = torch.cuda.CUDAGraph(), torch.cuda.Stream(), torch.cuda.Stream()
            with torch.cuda.graph(graph, stream=side):
                cmd.decrypt_device(eng, key, cts.data_ptr(), 5000, small.data_ptr(), 0, side.cuda_stream)
                cmd.decrypt_device(eng, key, cts.data_ptr(), 100000, err.data_ptr(), 0, other.cuda_stream)
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(err, want) and torch.equal(small, want[:5000])
            del graph
        finally:
            key.free()
