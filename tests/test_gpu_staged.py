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
