"""Measured cases of the decryption engine, through its public Python API.

Each case is one call (or one submit-and-drain) that a program using the
engine makes: device batches of one key from a single ciphertext up to 2^20,
a host-buffer batch, a mixed batch of many keys and parameter sets, KEM
decapsulation, error positions, the serving loop and key generation.  Keys
come from the engine's own key generation, seeded by the case's seed;
ciphertexts are encryptions of uniform weight-t error vectors under them (made
on the GPU), a stated share replaced by random strings where the real traffic
has malformed ones.

Every output is whole bytes or integers, so there is no rounding to bound and
``exact`` has no value to give.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cm_decrypt__b200 as cmd

# set: (m, n, t, ciphertext bytes)
SETS = {348864: (12, 3488, 64, 96), 460896: (13, 4608, 96, 156), 6688128: (13, 6688, 128, 208),
        6960119: (13, 6960, 119, 194), 8192128: (13, 8192, 128, 208)}
# Shares of the five sets in traffic that mixes them.
MIX = {348864: 0.30, 460896: 0.15, 6688128: 0.20, 6960119: 0.20, 8192128: 0.15}


def listed():
    return [
        # One message decrypted on its own: the smallest call, pure latency.
        {"name": "one", "kind": "device", "set": 6960119, "count": 1, "path": "auto", "malformed": 0},
        # A small group through the small-batch kernels, a ragged second tile.
        {"name": "few", "kind": "device", "set": 348864, "count": 37, "path": "tile", "malformed": 0},
        # An ordinary small batch that fills part of the GPU.
        {"name": "small", "kind": "device", "set": 460896, "count": 2500, "path": "auto", "malformed": 0},
        # The flagship batch: 65,536 ciphertexts resident on the device.
        {"name": "batch", "kind": "device", "set": 6960119, "count": 65536, "path": "auto", "malformed": 0},
        # The largest parameter set at a size that does not fill whole rounds,
        # with some corrupted ciphertexts.
        {"name": "ragged", "kind": "device", "set": 8192128, "count": 50000, "path": "auto", "malformed": 20},
        # Bulk decryption: 2^20 ciphertexts of the smallest set.
        {"name": "bulk", "kind": "device", "set": 348864, "count": 1 << 20, "path": "auto", "malformed": 0},
        # A file-sized host batch in pinned buffers, copies included.
        {"name": "host", "kind": "host", "set": 6960119, "count": 100003, "malformed": 0},
        # Error positions instead of error rows (the compact output).
        {"name": "positions", "kind": "positions", "set": 460896, "count": 12345, "malformed": 0},
        # KEM decapsulation: decrypt, re-encoding check, session keys.
        {"name": "decap", "kind": "decap", "set": 6688128, "count": 20000, "malformed": 10},
        # A mixed batch over 64 keys of all five sets, 10 % malformed.
        {"name": "mixed", "kind": "mixed", "keys": 64, "count": 65536, "malformed": 100},
        # The serving loop: a burst of requests over many resident keys.
        {"name": "serve", "kind": "serve", "keys": 64, "count": 1000, "malformed": 50},
        # Key generation for a handful of users.
        {"name": "keygen", "kind": "keygen", "set": 6960119, "count": 8},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["device", "device", "device", "device", "host", "positions", "decap", "mixed", "serve",
                       "keygen"])
    if kind == "mixed":
        return {"kind": kind, "keys": size(5, 100), "count": size(100, 100000), "malformed": rng.choice([0, 50, 100])}
    if kind == "serve":
        return {"kind": kind, "keys": size(5, 100), "count": size(1, 4000), "malformed": rng.choice([0, 50])}
    s = rng.choice(sorted(SETS))
    if kind == "keygen":
        return {"kind": kind, "set": s, "count": size(1, 16)}
    case = {"kind": kind, "set": s, "count": size(1, 200000), "malformed": rng.choice([0, 0, 10, 50])}
    if kind == "device":
        case["path"] = "tile" if case["count"] <= 4096 and rng.random() < 0.5 else "auto"
    return case


# One engine per process, as a program has it; created on first use.
_engine = None


def _eng() -> cmd.Engine:
    global _engine
    if _engine is None:
        _engine = cmd.Engine(0)
    return _engine


def _rngs(seed: int):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return np.random.default_rng(seed), g


def _parity_check(set_id: int, pk: bytes) -> torch.Tensor:
    """[I | T] as a bf16 matrix [n, mt] on the GPU, from the public key bytes."""
    m, n, t, _ = SETS[set_id]
    mt = m * t
    rows = np.frombuffer(pk, np.uint8).reshape(mt, (n - mt + 7) // 8)
    d = torch.from_numpy(rows.copy()).cuda()
    bits = (d.unsqueeze(-1) >> torch.arange(8, device="cuda", dtype=torch.uint8)) & 1
    # a row's bytes are the last (n - mt + 7) / 8 of n/8 row bytes (bit 0 first)
    T = bits.reshape(mt, -1)
    h = torch.zeros((mt, n), dtype=torch.bfloat16, device="cuda")
    h[:, n - T.shape[1]:] = T.to(torch.bfloat16)
    h[:, :mt] = torch.eye(mt, dtype=torch.bfloat16, device="cuda")
    return h.t().contiguous()


def _positions(g, count: int, n: int, t: int) -> torch.Tensor:
    """count uniform t-subsets of [0, n): the first t distinct of more draws."""
    k = t + 48
    v = torch.randint(0, n, (count, k), generator=g, device="cuda")
    order = torch.sort(v * k + torch.arange(k, device="cuda"), dim=1).values
    val, idx = order // k, order % k
    first = torch.ones_like(val, dtype=torch.bool)
    first[:, 1:] = val[:, 1:] != val[:, :-1]
    keep = torch.zeros_like(first).scatter_(1, idx, first)
    rank = torch.cumsum(keep, 1)
    take = keep & (rank <= t)
    return v[take].reshape(count, t)


def _encrypt(set_id: int, h: torch.Tensor, g, count: int, malformed: int) -> torch.Tensor:
    """Ciphertexts uint8 [count, ct] on the GPU: C = [I | T] e, a share random."""
    m, n, t, ct = SETS[set_id]
    mt = m * t
    out = torch.zeros((count, ct), dtype=torch.uint8, device="cuda")
    weights = (1 << torch.arange(8, device="cuda", dtype=torch.int32))
    for c0 in range(0, count, 32768):
        c = min(32768, count - c0)
        e = torch.zeros((c, n), dtype=torch.bfloat16, device="cuda")
        e.scatter_(1, _positions(g, c, n, t), 1.0)
        s = torch.zeros((c, 8 * ct), dtype=torch.int32, device="cuda")
        s[:, :mt] = (e @ h).to(torch.int32) & 1
        if malformed:
            bad = torch.rand(c, generator=g, device="cuda") < malformed / 1000
            r = torch.randint(0, 2, (c, mt), generator=g, device="cuda", dtype=torch.int32)
            s[:, :mt] = torch.where(bad[:, None], r, s[:, :mt])
        out[c0:c0 + c] = (s.reshape(c, ct, 8) * weights).sum(2).to(torch.uint8)
    return out


class _State:
    """What the program keeps; frees its keys and server when dropped."""

    def __init__(self, **kw):
        self.__dict__.update(kw)

    def __del__(self):
        torch.cuda.synchronize()
        if hasattr(self, "server"):
            self.server.close()
        for k in getattr(self, "keys", []):
            k.free()


def _keyring(case, rng):
    """Secret and public keys of `keys` users, their sets drawn from MIX."""
    ids = sorted(SETS)
    sets = ids + list(rng.choice(ids, case["keys"] - len(ids), p=[MIX[s] for s in ids]))
    ring = []
    for s in ids:
        seeds = rng.integers(0, 256, (sets.count(s), 32), dtype=np.uint8)
        pks, sks, _ = cmd.kem_keypair_batch(_eng(), s, seeds)
        ring += [(s, pks[i].tobytes(), sks[i].tobytes()) for i in range(len(seeds))]
    return ring


def _mixed_cts(case, ring, rng, g):
    """Key index per ciphertext and each key's ciphertexts, batch order random."""
    by_set = {s: [i for i, k in enumerate(ring) if k[0] == s] for s in SETS}
    ids = sorted(SETS)
    ends = np.round(np.cumsum([MIX[s] for s in ids]) * case["count"]).astype(int)
    sets = rng.permutation(np.repeat(ids, np.diff(ends, prepend=0)))
    key_idx = np.zeros(case["count"], np.uint32)
    for s in ids:
        at = np.nonzero(sets == s)[0]
        key_idx[at] = rng.choice(by_set[s], at.size)
    cts = {}
    for i, (s, pk, _) in enumerate(ring):
        mine = int((key_idx == i).sum())
        if mine:
            cts[i] = _encrypt(s, _parity_check(s, pk), g, mine, case["malformed"])
    return key_idx, cts


def prepare(case, seed):
    eng = _eng()
    rng, g = _rngs(seed)
    kind = case["kind"]
    if kind == "keygen":
        m, n, t, _ = SETS[case["set"]]
        count, mt = case["count"], m * t
        seeds = rng.integers(0, 256, (count, 32), dtype=np.uint8)
        pk = torch.zeros((count, mt * ((n - mt + 7) // 8)), dtype=torch.uint8).pin_memory()
        sk = torch.zeros((count, cmd.set_info(case["set"]).sk_bytes), dtype=torch.uint8).pin_memory()
        return _State(kind=kind, set=case["set"], seeds=seeds, pk=pk, sk=sk)
    if kind == "mixed":
        ring = _keyring(case, rng)
        keys = [cmd.Key(eng, s, sk) for s, _, sk in ring]
        key_idx, per_key = _mixed_cts(case, ring, rng, g)
        ctb = np.array([SETS[s][3] for s, _, _ in ring], np.uint64)
        nw = np.array([(SETS[s][1] + 31) // 32 for s, _, _ in ring], np.uint64)
        ct_off = np.concatenate([[0], np.cumsum(ctb[key_idx])]).astype(np.uint64)
        err_off = np.concatenate([[0], np.cumsum(nw[key_idx])]).astype(np.uint64)
        buf = torch.zeros(int(ct_off[-1]), dtype=torch.uint8, device="cuda")
        for i, c in per_key.items():
            at = torch.from_numpy(ct_off[:-1][key_idx == i].astype(np.int64)).cuda()
            buf[(at[:, None] + torch.arange(c.shape[1], device="cuda")).reshape(-1)] = c.reshape(-1)
        err = torch.zeros(int(err_off[-1]), dtype=torch.int32, device="cuda")
        w = torch.zeros(case["count"], dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        return _State(kind=kind, keys=keys, key_idx=key_idx, cts=buf, ct_off=ct_off[:-1].copy(),
                      err_off=err_off[:-1].copy(), err=err, weight=w)
    if kind == "serve":
        ring = _keyring(case, rng)
        key_idx, per_key = _mixed_cts(case, ring, rng, g)
        server = cmd.Server(eng, record_completions=False)
        kids = np.array([server.add_key(s, sk) for s, _, sk in ring], np.uint32)
        cts = np.zeros((case["count"], 208), np.uint8)
        for i, c in per_key.items():
            cts[np.nonzero(key_idx == i)[0], :c.shape[1]] = c.cpu().numpy()
        rows = np.zeros((case["count"], 1024), np.uint8)
        server.register_rows(rows)
        return _State(kind=kind, server=server, key_ids=kids[key_idx], cts=cts, rows=rows)
    m, n, t, ct = SETS[case["set"]]
    count = case["count"]
    pk, sk, _ = cmd.kem_keypair(eng, case["set"], rng.bytes(32))
    key = cmd.Key(eng, case["set"], sk)
    cts = _encrypt(case["set"], _parity_check(case["set"], pk), g, count, case["malformed"])
    st = _State(kind=kind, keys=[key], key=key, count=count, cts=cts, path=case.get("path", "auto"))
    if kind == "device":
        st.err = torch.zeros((count, (n + 31) // 32), dtype=torch.int32, device="cuda")
        st.weight = torch.zeros(count, dtype=torch.int16, device="cuda")
    elif kind == "positions":
        st.pos = torch.zeros((count, t + 1), dtype=torch.int16, device="cuda")
    elif kind == "decap":
        cmd.prepare_decap(eng, key)
        st.session = torch.zeros((count, 32), dtype=torch.uint8, device="cuda")
        st.accept = torch.zeros(count, dtype=torch.uint8, device="cuda")
    else:
        st.cts = cts.cpu().pin_memory()
        st.err = torch.zeros((count, n // 8), dtype=torch.uint8).pin_memory()
        st.weight = torch.zeros(count, dtype=torch.int16).pin_memory()
    torch.cuda.synchronize()
    return st


def run(state):
    eng, s = _eng(), state
    if s.kind == "device":
        cmd.decrypt_device(eng, s.key, s.cts.data_ptr(), s.count, s.err.data_ptr(), s.weight.data_ptr(), path=s.path)
        return s.err, s.weight
    if s.kind == "host":
        cmd.decrypt_into(eng, s.key, s.cts.numpy(), s.err.numpy(), s.weight.numpy().view(np.uint16))
        return s.err, s.weight
    if s.kind == "positions":
        cmd.decrypt_positions_device(eng, s.key, s.cts.data_ptr(), s.count, s.pos.data_ptr())
        return s.pos
    if s.kind == "decap":
        cmd.kem_decap_device(eng, s.key, s.cts.data_ptr(), s.count, s.session.data_ptr(), s.accept.data_ptr())
        return s.session, s.accept
    if s.kind == "mixed":
        cmd.decrypt_mixed_device(eng, s.keys, s.key_idx, s.cts.data_ptr(), s.ct_off, s.err.data_ptr(), s.err_off,
                                 s.weight.data_ptr())
        return s.err, s.weight
    if s.kind == "serve":
        s.server.submit_many(s.key_ids, s.cts, s.rows)
        s.server.drain()
        return s.rows
    pk, sk, attempts = cmd.kem_keypair_batch(eng, s.set, s.seeds, pk_out=s.pk.numpy(), sk_out=s.sk.numpy())
    return pk, sk, attempts.astype(np.int64)


def _decrypt_ops(set_id: int) -> float:
    """32-bit logic operations of one decryption: syndrome rows four at a time,
    Berlekamp-Massey's 3 t^2 field products, an additive FFT over the field
    (a bitsliced product: m^2 AND-XORs and the reduction, 1/32 of each per
    element)."""
    m, n, t, ct = SETS[set_id]
    mul = (m * m + (22 if m == 12 else 48)) / 32
    depth = math.ceil(math.log2(t + 1))
    return 2 * ct * (2 * t * m / 32) + 3 * t * t * mul + depth * 2 ** (m - 1) * mul


def work(case):
    kind, count = case["kind"], case["count"]
    if kind in ("mixed", "serve"):
        per = [(MIX[s], SETS[s][3] + SETS[s][1] / 8, _decrypt_ops(s)) for s in SETS]
        return {"bytes": count * sum(p * b for p, b, _ in per), "flops": count * sum(p * o for p, _, o in per)}
    m, n, t, ct = SETS[case["set"]]
    if kind == "keygen":
        mt = m * t
        pk = mt * ((n - mt + 7) // 8)
        # a reduced row echelon form over GF(2), about 3.5 random attempts
        return {"bytes": count * (32 + pk + n), "flops": count * 3.5 * mt * mt * n / 32}
    out = {"positions": 2 * (t + 1), "decap": 33}.get(kind, n / 8 + 2)
    ops = _decrypt_ops(case["set"])
    if kind == "decap":
        ops += (n - m * t) * m * t / 32
    return {"bytes": count * (ct + out), "flops": count * ops}


def exact(case, seed):
    return None  # whole numbers and bytes: equal, with nothing to round
