"""Per-instance keypair, expand-sk, sign and verify at the edges of their launch rule (one CTA per instance, or a
cluster of two, four or eight where the batch is small), with keys at every alignment, against the
oracle byte for byte.  Instance 0 signs a message whose first attempt is singular."""
import hashlib
import json
import os

import numpy as np
import pytest

from cumayo_b200 import Mayo
from oracle import oracle as O

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden")
N = 73
BATCHES = (1, 12, 13, 32, 33, 72, 73)


@pytest.fixture(scope="module", params=[1, 2, 3, 5])
def case(request, cuda):
    s = request.param
    rng = np.random.default_rng(700 + s)
    z = Mayo(s).sizes
    seeds = rng.integers(0, 256, (N, z.sk_bytes), dtype=np.uint8)
    sk0, _ = O.keypair(s, 0, 0)
    seeds[0] = np.frombuffer(sk0, np.uint8)
    esk = O.expandsk_batch(s, seeds)
    cpk = O.keypair_from_seed_batch(s, seeds)
    epk = O.expandpk_batch(s, cpk)
    g = json.load(open(os.path.join(GOLDEN, f"ref_mayo{s}.json")))["rejection"]
    msgs = [rng.integers(0, 256, 32, dtype=np.uint8).tobytes() for _ in range(N)]
    msgs[0] = hashlib.shake_256(f"reject-search/{s}/{g['indices'][0]}".encode()).digest(32)
    sig, attempts = O.sign_batch(s, esk, msgs)
    assert attempts[0] > 1
    return s, seeds, esk, epk, np.frombuffer(b"".join(msgs), np.uint8).reshape(N, 32), sig, cpk


def _rows(a, stride, off):
    """Rows of `a` at `stride` bytes from byte `off` of a device buffer that ends with the last row."""
    import torch
    host = np.zeros(off + (len(a) - 1) * stride + a.shape[1], np.uint8)
    for i, r in enumerate(a):
        host[off + i * stride: off + i * stride + a.shape[1]] = r
    return torch.from_numpy(host).cuda()[off:]


@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_sign_verify_launch_edges(case, off):
    import torch
    s, _, esk, epk, msgs, sig, _ = case
    m = Mayo(s)
    z = m.sizes
    es, ps = z.esk_bytes + 3 * off, z.epk_bytes + off
    d_esk, d_epk, d_msg = _rows(esk, es, off), _rows(epk, ps, off), torch.from_numpy(msgs.copy()).cuda()
    bad = sig.copy()
    bad[1::3, 5] ^= 0x10
    d_bad = torch.from_numpy(bad).cuda()
    want = np.zeros(N, np.uint8)
    want[1::3] = 1
    ws = torch.zeros(N * m.sign_ws_bytes(), dtype=torch.uint8, device="cuda")
    for b in BATCHES if off == 0 else (1, 13, 73):
        out = torch.zeros(N, z.sig_bytes, dtype=torch.uint8, device="cuda")
        m.sign_many(d_esk, d_msg, out, ws, b, msg_stride=32, mlen=32, esk_stride=es)
        res = torch.full((N,), 0xEE, dtype=torch.uint8, device="cuda")
        m.verify_many(d_epk, d_msg, d_bad, res, b, msg_stride=32, mlen=32, epk_stride=ps)
        torch.cuda.synchronize()
        assert (out[:b].cpu().numpy() == sig[:b]).all() and not out[b:].any(), b
        assert (res[:b].cpu().numpy() == want[:b]).all() and (res[b:] == 0xEE).all(), b


def test_sign_more_than_a_wave(case):
    """More signatures than CTAs fit the GPU at once; singular first attempts at the start, in the
    middle and at the end of the batch."""
    import torch
    s, _, esk, _, msgs, sig, _ = case
    m = Mayo(s)
    z = m.sizes
    n = 148 * {1: 3, 2: 6, 3: 2, 5: 1}[s] + 37
    pick = np.arange(n) % N  # 0: singular
    pick[[1, 149, n - 1, n - 2]] = 0
    d_esk = torch.from_numpy(esk[pick]).cuda()
    d_msg = torch.from_numpy(msgs[pick]).cuda()
    ws = torch.zeros(n * m.sign_ws_bytes(), dtype=torch.uint8, device="cuda")
    for b in (n, n - 1, 149):
        out = torch.zeros(n, z.sig_bytes, dtype=torch.uint8, device="cuda")
        m.sign_many(d_esk, d_msg, out, ws, b, msg_stride=32, mlen=32, esk_stride=z.esk_bytes)
        torch.cuda.synchronize()
        assert (out[:b].cpu().numpy() == sig[pick[:b]]).all() and not out[b:].any(), b


@pytest.mark.parametrize("off", [0, 1, 2, 3])
def test_keypair_expandsk_launch_edges(case, off):
    import torch
    s, seeds, esk, _, _, _, cpk = case
    m = Mayo(s)
    z = m.sizes
    kp, ep = z.pitch_keypair + off, z.esk_bytes + off
    at = (z.sk_bytes + 127) // 128 * 128
    for b in BATCHES if off == 0 else (1, 13, 73):
        pool = torch.zeros(off + N * kp, dtype=torch.uint8, device="cuda")[off:]  # ends with the last row
        rows = pool.view(N, kp)
        rows[:, : z.sk_bytes] = torch.from_numpy(seeds).cuda()
        m.crypto_sign_keypair_from_seed(pool, kp, b)
        epool = torch.zeros(off + N * ep, dtype=torch.uint8, device="cuda")[off:]
        erows = epool.view(N, ep)
        erows[:, : z.sk_bytes] = torch.from_numpy(seeds).cuda()
        m.crypto_sign_expandsk(epool, ep, b)
        torch.cuda.synchronize()
        assert (rows[:b, at: at + z.pk_bytes].cpu().numpy() == cpk[:b]).all() and not rows[b:, at:].any(), b
        assert (erows[:b, : z.esk_bytes].cpu().numpy() == esk[:b]).all() and not erows[b:, z.sk_bytes:].any(), b
        assert not erows[:, z.esk_bytes:].any(), b


@pytest.mark.parametrize("n", [74, 75, 148, 149])
def test_keypair_keys_derived_or_hashed_first(case, n):
    """Around the batches from which a hash kernel runs before the expansion (148 SMs: one item each)."""
    import torch
    s, seeds, esk, _, _, _, cpk = case
    m = Mayo(s)
    z = m.sizes
    at = (z.sk_bytes + 127) // 128 * 128
    pick = np.arange(n) % N
    d_seed = torch.from_numpy(seeds[pick]).cuda()
    rows = torch.zeros(n, z.pitch_keypair, dtype=torch.uint8, device="cuda")
    rows[:, : z.sk_bytes] = d_seed
    m.crypto_sign_keypair_from_seed(rows.view(-1), z.pitch_keypair, n)
    erows = torch.zeros(n, z.esk_bytes, dtype=torch.uint8, device="cuda")
    erows[:, : z.sk_bytes] = d_seed
    m.crypto_sign_expandsk(erows.view(-1), z.esk_bytes, n)
    # seeds of the counter: the same keypair alone, from the seed that it wrote
    drawn = torch.zeros(n, z.pitch_keypair, dtype=torch.uint8, device="cuda")
    m.crypto_sign_keypair(drawn.view(-1), z.pitch_keypair, n, rand_index=5)
    again = torch.zeros_like(drawn)
    again[:, : z.sk_bytes] = drawn[:, : z.sk_bytes]
    m.crypto_sign_keypair_from_seed(again.view(-1), z.pitch_keypair, n)
    other = torch.zeros(300, z.pitch_keypair, dtype=torch.uint8, device="cuda")
    m.crypto_sign_keypair(other.view(-1), z.pitch_keypair, 300, rand_index=5)
    torch.cuda.synchronize()
    assert (rows[:, at: at + z.pk_bytes].cpu().numpy() == cpk[pick]).all()
    assert (erows.cpu().numpy() == esk[pick]).all()
    assert torch.equal(drawn, again) and torch.equal(drawn, other[:n])


@pytest.fixture(scope="module")
def ragged(case):
    s, _, esk, _, _, _, _ = case
    rng = np.random.default_rng(900 + s)
    msgs = [rng.integers(0, 256, int(n), dtype=np.uint8).tobytes() for n in rng.integers(0, 200, N)]
    return msgs, O.sign_batch(s, esk, msgs)[0]


@pytest.mark.parametrize("rest", [1, 12, 13, 32, 33, 72, 73])
def test_full_waves_and_a_remainder(case, ragged, rest):
    """Sign and verify of messages at offsets, keypair and expand-sk: 148 or 296 instances and a remainder."""
    import torch
    s, seeds, esk, epk, _, _, cpk = case
    msgs, sig = ragged
    m = Mayo(s)
    z = m.sizes
    lens = np.array([len(x) for x in msgs], np.uint32)
    start = np.concatenate([[0], np.cumsum(lens[:-1])]).astype(np.uint64)
    blob = torch.from_numpy(np.frombuffer(b"".join(msgs), np.uint8).copy()).cuda()
    at = (z.sk_bytes + 127) // 128 * 128
    for full in {1: (444,), 2: (296, 888), 3: (148, 296), 5: (148, 296)}[s]:
        n = full + rest
        pick = (np.arange(n) * 5 + 1) % N
        d_off, d_len = torch.from_numpy(start[pick]).cuda(), torch.from_numpy(lens[pick]).cuda()
        out = torch.zeros(n + 1, z.sig_bytes, dtype=torch.uint8, device="cuda")
        ws = torch.zeros(n * m.sign_ws_bytes(), dtype=torch.uint8, device="cuda")
        m.sign_many(torch.from_numpy(esk[pick]).cuda(), blob, out, ws, n, msg_off=d_off, msg_len=d_len,
                    esk_stride=z.esk_bytes)
        bad = sig[pick].copy()
        bad[::7, 3] ^= 1
        res = torch.full((n + 1,), 0xEE, dtype=torch.uint8, device="cuda")
        m.verify_many(torch.from_numpy(epk[pick]).cuda(), blob, torch.from_numpy(bad).cuda(), res, n, msg_off=d_off,
                      msg_len=d_len, epk_stride=z.epk_bytes)
        rows = torch.zeros(n, z.pitch_keypair, dtype=torch.uint8, device="cuda")
        rows[:, : z.sk_bytes] = torch.from_numpy(seeds[pick]).cuda()
        m.crypto_sign_keypair_from_seed(rows.view(-1), z.pitch_keypair, n)
        erows = torch.zeros(n, z.esk_bytes, dtype=torch.uint8, device="cuda")
        erows[:, : z.sk_bytes] = rows[:, : z.sk_bytes]
        m.crypto_sign_expandsk(erows.view(-1), z.esk_bytes, n)
        torch.cuda.synchronize()
        assert (out[:n].cpu().numpy() == sig[pick]).all() and not out[n:].any()
        assert (res[:n].cpu().numpy() == (np.arange(n) % 7 == 0)).all() and (res[n:] == 0xEE).all()
        assert (rows[:, at: at + z.pk_bytes].cpu().numpy() == cpk[pick]).all()
        assert (erows.cpu().numpy() == esk[pick]).all()
