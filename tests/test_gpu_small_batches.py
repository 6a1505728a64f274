"""The per-ciphertext kernels (small batches): every batch size at which their
launches change shape, against the plain per-stage path (itself checked against
the oracle), with valid, malformed and degenerate ciphertexts."""
from __future__ import annotations

import numpy as np
import pytest

import cm_decrypt__b200 as cmd
from conftest import SETS, golden_sk, rng

pytestmark = pytest.mark.gpu


def degenerate(info) -> np.ndarray:
    """No bit, one bit (first, last), two bits, every syndrome bit set: long
    zero runs and late length changes in Berlekamp-Massey."""
    c = np.zeros((5, info.ct_bytes), np.uint8)
    c[1, 0] = 1
    c[2, (info.m * info.t - 1) // 8] = 1 << ((info.m * info.t - 1) % 8)
    c[3, 3] = 0x81
    c[4] = 0xFF
    return c


@pytest.mark.parametrize("s", SETS)
def test_small_batch_shapes_match_plain(engine, s):
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        info = key.info
        valid, planted, ok = cmd.PubKey(s, golden_sk(s)).ciphertexts(seed=31, count=3700, malformed_permille=60)
        cts = np.concatenate([degenerate(info), rng(s).integers(0, 256, (3, info.ct_bytes), dtype=np.uint8), valid])
        want, want_w = cmd.decrypt(engine, key, cts, path="plain")
        good = np.nonzero(ok)[0]
        assert np.array_equal(want[8 + good], planted[good])
        # one launch up to 64; three up to an SM each (148 on a B200) and above;
        # the 32-ciphertext tile kernels above 24 an SM (3,552)
        for count in (1, 2, 8, 63, 64, 65, 147, 148, 149, 593, 3552, 3553):
            for first in (0, 5):
                got, got_w = cmd.decrypt(engine, key, cts[first:first + count], path="tile")
                assert np.array_equal(got, want[first:first + count]), (count, first)
                assert np.array_equal(got_w, want_w[first:first + count]), (count, first)
    finally:
        key.free()


@pytest.mark.parametrize("s", [348864, 6960119])
def test_auto_positions_and_decap_small(engine, s):
    """Small batches of the calls without a path argument: positions against
    the fused kernel's rows, decapsulation against the keys of a large batch."""
    key = cmd.Key(engine, s, golden_sk(s))
    try:
        info = key.info
        valid, _, _ = cmd.PubKey(s, golden_sk(s)).ciphertexts(seed=32, count=9000, malformed_permille=60)
        cts = np.concatenate([degenerate(info), valid])
        rows, _ = cmd.decrypt(engine, key, cts, path="fused")
        large_k, large_a = cmd.kem_decap(engine, key, cts)
        for count in (1, 64, 65, 3552, 3553, 8191, 8192):
            assert np.array_equal(cmd.decrypt_positions(engine, key, cts[:count]),
                                  cmd.positions_from_errors(s, rows[:count])), count
            assert np.array_equal(cmd.decrypt(engine, key, cts[:count])[0], rows[:count]), count
            k, a = cmd.kem_decap(engine, key, cts[:count])
            assert np.array_equal(k, large_k[:count]) and np.array_equal(a, large_a[:count]), count
    finally:
        key.free()
