"""Batches on both sides of the line (2,048 instances, HASH_WARP_MAX in csrc/ops.h) up to which a warp
hashes an instance and past which a thread does: keypair, expand-sk, sign and the shared-key calls,
whose ragged messages are ordered by their length past it, against the oracle byte for byte.  The
batches repeat a few dozen distinct keys and messages."""
import hashlib
import json
import os
import re

import numpy as np
import pytest

from cumayo_b200 import Mayo, MayoError
from oracle import oracle as O

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = os.path.join(ROOT, "tests", "golden")
N = 53
LINE = 2048
BATCHES = (LINE, LINE + 1, 2501)


def _dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a).copy()).cuda()


def test_the_line():
    ops = open(os.path.join(ROOT, "cumayo_b200", "csrc", "ops.h")).read()
    assert int(re.search(r"HASH_WARP_MAX = (\d+);", ops).group(1)) == LINE


@pytest.fixture(scope="module", params=[1, 2, 3, 5])
def case(request, cuda):
    s = request.param
    rng = np.random.default_rng(1300 + s)
    seeds = rng.integers(0, 256, (N, Mayo(s).sizes.sk_bytes), dtype=np.uint8)
    seeds[0] = np.frombuffer(O.keypair(s, 0, 0)[0], np.uint8)
    return s, rng, seeds, O.expandsk_batch(s, seeds), O.keypair_from_seed_batch(s, seeds)


def _messages(s, rng):
    """Of 0 to 9 SHAKE256 blocks (the order's last bin holds 7 and more), around every block's end; two
    whose first attempt under the counter key 0 is singular."""
    lens = [max(0, 136 * b + d) for b in range(10) for d in (-1, 0, 1, 8)] + list(rng.integers(0, 1400, N))
    msgs = [rng.integers(0, 256, int(n), dtype=np.uint8).tobytes() for n in lens[:N]]
    g = json.load(open(os.path.join(GOLDEN, f"ref_mayo{s}.json")))["rejection"]
    for q, idx in enumerate(g["indices"][:2]):
        msgs[11 * q] = hashlib.shake_256(f"reject-search/{s}/{idx}".encode()).digest(32)
    return msgs


def _ragged(msgs, pick):
    lens = np.array([len(x) for x in msgs], np.uint32)
    start = np.concatenate([[0], np.cumsum(lens[:-1])]).astype(np.int64)
    return dict(msgs=_dev(np.frombuffer(b"".join(msgs), np.uint8)), msg_off=_dev(start[pick]),
                msg_len=_dev(lens[pick].view(np.int32)))


@pytest.mark.parametrize("n", BATCHES)
def test_keypair_and_expandsk(case, n):
    import torch
    s, _, seeds, esk, cpk = case
    m = Mayo(s)
    z = m.sizes
    at = (z.sk_bytes + 127) // 128 * 128
    pick = (np.arange(n) * 7 + 3) % N
    d_seed, d_pick = _dev(seeds[pick]), _dev(pick)
    rows = torch.zeros(n, z.pitch_keypair, dtype=torch.uint8, device="cuda")
    rows[:, : z.sk_bytes] = d_seed
    m.crypto_sign_keypair_from_seed(rows.view(-1), z.pitch_keypair, n)
    assert torch.equal(rows[:, at: at + z.pk_bytes], _dev(cpk)[d_pick])
    # seeds of the counter, whose keys are all different
    rows.zero_()
    m.crypto_sign_keypair(rows.view(-1), z.pitch_keypair, n, rand_index=9)
    torch.cuda.synchronize()
    for i in (0, 1, 31, 32, LINE - 1, n - 1):
        sk, pk = O.keypair(s, 9, i)
        assert rows[i, : z.sk_bytes].cpu().numpy().tobytes() == sk, i
        assert rows[i, at: at + z.pk_bytes].cpu().numpy().tobytes() == pk, i
    assert len(set(map(bytes, rows[:, : z.sk_bytes].cpu().numpy()))) == n
    del rows
    rows = torch.zeros(n, z.esk_bytes, dtype=torch.uint8, device="cuda")
    rows[:, : z.sk_bytes] = d_seed
    m.crypto_sign_expandsk(rows.view(-1), z.esk_bytes, n)
    assert torch.equal(rows, _dev(esk)[d_pick])


@pytest.mark.parametrize("n", BATCHES)
def test_sign_of_distinct_keys(case, n):
    import torch
    s, rng, _, esk, _ = case
    m = Mayo(s)
    z = m.sizes
    msgs = _messages(s, rng)
    sig, attempts = O.sign_batch(s, esk, msgs)
    assert attempts[0] > 1
    pick = (np.arange(n) * 5 + 1) % N
    out = torch.zeros(n + 1, z.sig_bytes, dtype=torch.uint8, device="cuda")
    ws = torch.zeros(n * m.sign_ws_bytes(), dtype=torch.uint8, device="cuda")
    m.sign_many(_dev(esk)[_dev(pick)], sig=out, ws=ws, batch=n, esk_stride=z.esk_bytes, **_ragged(msgs, pick))
    torch.cuda.synchronize()
    assert (out[:n].cpu().numpy() == sig[pick]).all() and not out[n].any()


@pytest.mark.parametrize("n", BATCHES)
def test_one_key_and_ragged_messages(case, n):
    """sign_shared and verify_shared with every block shape's hash CTA, an odd batch among them."""
    import torch
    s, rng, _, esk, cpk = case
    m = Mayo(s)
    z = m.sizes
    msgs = _messages(s, rng)
    sig, attempts = O.sign_batch(s, esk[:1], msgs, shared_key=True)
    assert attempts[0] > 1
    pick = (np.arange(n) * 3 + 2) % N
    io = _ragged(msgs, pick)
    bad = sig[pick].copy()
    bad[::7, 3] ^= 1
    d_esk, d_epk, d_bad = _dev(esk[0]), _dev(np.frombuffer(O.expandpk(s, cpk[0].tobytes()), np.uint8)), _dev(bad)
    ws = torch.zeros(max(m.sign_shared_ws_bytes(n), m.verify_shared_ws_bytes(n)), dtype=torch.uint8, device="cuda")
    try:
        for h, g, p in ((0, 0, 0), (32, 2, 1), (128, 4, 1), (256, 1, 1), (64, 1, 2)):
            try:
                m.set_shared_shape(h, g, p)
            except MayoError:  # there is no CTA of four MAYO_5 signatures
                assert s == 5 and g == 4
                continue
            out = torch.zeros(n + 1, z.sig_bytes, dtype=torch.uint8, device="cuda")
            m.sign_shared(d_esk, sig=out, ws=ws, batch=n, **io)
            torch.cuda.synchronize()
            assert int(ws[:4].cpu().numpy().view(np.uint32)[0]) == 0, ("product gave up", h, g, p)
            assert (out[:n].cpu().numpy() == sig[pick]).all() and not out[n].any(), (h, g, p)
            res = torch.full((n + 1,), 0xEE, dtype=torch.uint8, device="cuda")
            m.verify_shared(d_epk, sig=d_bad, result=res, ws=ws, batch=n, **io)
            torch.cuda.synchronize()
            assert int(ws[:4].cpu().numpy().view(np.uint32)[0]) == 0, ("product gave up", h, g, p)
            assert (res[:n].cpu().numpy() == (np.arange(n) % 7 == 0)).all() and res[n] == 0xEE, (h, g, p)
    finally:
        m.set_shared_shape(0, 0, 0)
