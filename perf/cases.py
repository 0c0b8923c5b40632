"""Performance cases: what users of this library have it do, through its public entry points.

Every case is one call of the batched API (``cumayo_b200.Mayo``) or one run of the work queue on
operands that are already on the GPU: distinct random keys (unless the case is a batch under one
resident key), random messages, and for verification signatures made by the matching secret keys,
one in ten of them corrupted.  Outputs are bytes (keys, signatures, verify results).
"""
import math

import numpy as np
import torch

from cumayo_b200 import A128, Mayo
from cumayo_b200.queue import Queue, SetOperands, items_array

SETS = (1, 2, 3, 5)
MIXED_KEYS = 64  # resident expanded keys per parameter set in the mixed queue


def listed():
    return [
        # one interactive signature from a compact key (latency)
        dict(name="sign_one", op="signWithesk", set=1, batch=1, mlen=32, var=False),
        # a handful of certificates to check, as one request of a service brings them
        dict(name="verify_few", op="verifyWithepk", set=3, batch=7, mlen=300, var=False),
        # the reference benchmark's three operations for MAYO_1 at a batch of 1,024
        dict(name="keypair_batch", op="keypair", set=1, batch=1024, mlen=0, var=False),
        dict(name="sign_batch", op="signWithesk", set=1, batch=1024, mlen=32, var=False),
        dict(name="verify_batch", op="verifyWithepk", set=1, batch=1024, mlen=32, var=False),
        # the largest parameter set at an odd batch
        dict(name="keypair_large_set", op="keypair", set=5, batch=777, mlen=0, var=False),
        # the reference benchmark's own batch of 20,000 signatures from compact keys
        dict(name="sign_bulk", op="signWithesk", set=2, batch=20000, mlen=32, var=False),
        # a resident directory of expanded public keys, every signature under its own key
        dict(name="verify_directory", op="verify", set=3, batch=16384, mlen=32, var=False),
        # pre-expanded secret keys of many tenants, ragged messages
        dict(name="sign_tenants", op="sign_many", set=5, batch=301, mlen=777, var=True),
        # one service key: sign and verify a large batch of messages of 32 to 1,024 bytes
        dict(name="sign_service_key", op="sign_shared", set=2, batch=65536, mlen=1024, var=True),
        dict(name="verify_service_key", op="verify_shared", set=2, batch=65536, mlen=1024, var=True),
        # a serving batch: keypairs, signatures and verifications of all four sets in one queue run
        dict(name="mixed_queue", op="queue", set=0, batch=16384, mlen=64, var=False),
    ]


# largest drawn batch of each operation for MAYO_1, 2, 3, 5 (no dearer than the largest listed case)
_MOST = {
    "keypair": (12000, 16000, 6000, 2400),
    "signWithesk": (6000, 12000, 2400, 1000),
    "verifyWithepk": (12000, 20000, 5000, 2400),
    "sign": (12000, 16000, 6000, 2400),
    "verify": (16384, 20000, 12000, 6000),
    "sign_many": (12000, 16000, 6000, 2400),
    "verify_many": (16384, 20000, 12000, 6000),
    "sign_shared": (40000, 65536, 16384, 8192),
    "verify_shared": (40000, 65536, 16384, 8192),
    "queue": (16384,),
}


def draw(rng):
    op = rng.choice(sorted(_MOST))
    i = rng.randrange(len(_MOST[op]))
    most = _MOST[op][i]
    least = 64 if op in ("queue", "sign_shared", "verify_shared") else 1
    batch = int(round(math.exp(rng.uniform(math.log(least), math.log(most)))))
    batch = min(max(batch, least), most)
    var = op in ("sign_many", "verify_many", "sign_shared", "verify_shared") and rng.random() < 0.7
    mlen = 0 if op == "keypair" else int(round(math.exp(rng.uniform(math.log(32), math.log(1024)))))
    return dict(op=op, set=0 if op == "queue" else SETS[i], batch=batch, mlen=mlen, var=var)


def _random_bytes(rng, *shape):
    return torch.from_numpy(rng.integers(0, 256, size=shape, dtype=np.uint8)).cuda()


def _pool(m, kind, batch, mlen=0):
    pool, pitch = m.alloc_pool(kind, batch, mlen)
    return pool, pitch, pool.view(batch, pitch)


def _keys(m, rng, batch):
    """Random secret seeds and the compact public keys that belong to them."""
    z = m.sizes
    sk = _random_bytes(rng, batch, z.sk_bytes)
    pool, pitch, rows = _pool(m, "keypair", batch)
    rows[:, :z.sk_bytes] = sk
    m.crypto_sign_keypair_from_seed(pool, pitch, batch)
    at = A128(z.sk_bytes)
    return sk, rows[:, at:at + z.pk_bytes].clone()


def _expanded_sk(m, sk):
    pool, pitch, rows = _pool(m, "expandsk", sk.shape[0])
    rows[:, :sk.shape[1]] = sk
    m.crypto_sign_expandsk(pool, pitch, sk.shape[0])
    return rows, pitch


def _expanded_pk(m, pk):
    pool, pitch, rows = _pool(m, "expandpk", pk.shape[0])
    at = m.sizes.p_bytes - 16
    rows[:, at:at + pk.shape[1]] = pk
    m.crypto_sign_expandpk(pool, pitch, pk.shape[0])
    return rows, pitch


def _messages(rng, case):
    """Messages back to back, and with `var` their device offsets and lengths (uniform 32..mlen)."""
    batch, mlen = case["batch"], case["mlen"]
    if not case["var"]:
        return dict(msgs=_random_bytes(rng, batch, mlen), msg_stride=mlen, mlen=mlen)
    lens = rng.integers(32, max(mlen, 32) + 1, size=batch).astype(np.int32)
    off = np.concatenate([[0], np.cumsum(lens.astype(np.int64))])
    return dict(msgs=_random_bytes(rng, int(off[-1])), msg_off=torch.from_numpy(off[:-1].copy()).cuda(),
                msg_len=torch.from_numpy(lens).cuda())


def _signatures(m, rows, pitch, msg, batch):
    """Signatures with the expanded secret keys in `rows` (one row: the same key for all)."""
    sig = torch.zeros(batch, m.sizes.sig_bytes, dtype=torch.uint8, device="cuda")
    ws = torch.zeros(batch * m.sign_ws_bytes() + 16, dtype=torch.uint8, device="cuda")
    m.sign_many(rows, sig=sig, ws=ws, batch=batch, esk_stride=0 if rows.shape[0] == 1 else pitch, **msg)
    return sig


def _corrupt(rng, sig):
    """Flip one nibble of one signature in ten."""
    bad = rng.random(sig.shape[0]) < 0.1
    at = rng.integers(0, sig.shape[1], size=sig.shape[0])
    i = torch.from_numpy(np.nonzero(bad)[0]).cuda()
    sig[i, torch.from_numpy(at[bad]).cuda()] ^= 0x05
    return sig


def _prepare_queue(case, rng):
    n, mlen = case["batch"], case["mlen"]
    ops = rng.permutation(np.arange(n) % 12)  # every (set, operation) alike, shuffled
    count = np.bincount(ops, minlength=12)
    seen = np.zeros(12, dtype=np.int64)
    entries = []
    for o in ops:
        entries.append((int(o % 3), SETS[o // 3], int(seen[o])))
        seen[o] += 1
    q = Queue(n + n // 8 + 64)
    out = {}
    for si, s in enumerate(SETS):
        m = Mayo(s)
        z = m.sizes
        nk, ns, nv = (int(c) for c in count[3 * si:3 * si + 3])
        sk, pk = _keys(m, rng, MIXED_KEYS)
        esk = _expanded_sk(m, sk)[0][:, :z.esk_bytes].contiguous()
        epk = _expanded_pk(m, pk)[0][:, :z.epk_bytes].contiguous()
        key = rng.integers(0, MIXED_KEYS, size=(2, max(ns, nv, 1))).astype(np.int32)
        sg_msg, vf_msg = _random_bytes(rng, max(ns, 1), mlen), _random_bytes(rng, max(nv, 1), mlen)
        vf_key = torch.from_numpy(key[1, :max(nv, 1)].copy()).cuda()
        vf_sig = torch.zeros(max(nv, 1), z.sig_bytes, dtype=torch.uint8, device="cuda")
        ws = torch.zeros(max(nv, 1) * m.sign_ws_bytes() + 16, dtype=torch.uint8, device="cuda")
        rows = esk.index_select(0, vf_key.long())
        m.sign_many(rows, vf_msg, vf_sig, ws, max(nv, 1), msg_stride=mlen, mlen=mlen, esk_stride=z.esk_bytes)
        _corrupt(rng, vf_sig)
        o = SetOperands(
            kp_seed=_random_bytes(rng, max(nk, 1), z.sk_bytes),
            kp_pk=torch.zeros(max(nk, 1), z.pk_bytes, dtype=torch.uint8, device="cuda"), kp_count=nk,
            sg_esk=esk, sg_nkeys=MIXED_KEYS, sg_key=torch.from_numpy(key[0, :max(ns, 1)].copy()).cuda(), sg_msg=sg_msg,
            sg_mlen=mlen, sg_sig=torch.zeros(max(ns, 1), z.sig_bytes, dtype=torch.uint8, device="cuda"), sg_count=ns,
            vf_epk=epk, vf_nkeys=MIXED_KEYS, vf_key=vf_key, vf_msg=vf_msg, vf_mlen=mlen, vf_sig=vf_sig,
            vf_res=torch.zeros(max(nv, 1), dtype=torch.uint8, device="cuda"), vf_count=nv)
        q.set_operands(s, o)
        out[s] = (o.kp_pk, o.sg_sig, o.vf_res)
    q.load(items_array(entries))
    return dict(case=case, queue=q, out=out)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    op, batch, mlen = case["op"], case["batch"], case["mlen"]
    if op == "queue":
        return _prepare_queue(case, rng)
    m = Mayo(case["set"])
    z = m.sizes
    st = dict(case=case, mayo=m)
    if op == "keypair":
        pool, pitch, rows = _pool(m, "keypair", batch)
        rows[:, :z.sk_bytes] = _random_bytes(rng, batch, z.sk_bytes)
        at = A128(z.sk_bytes)
        st.update(pool=pool, pitch=pitch, out=[rows[:, at:at + z.pk_bytes], rows[:, :z.sk_bytes]])
    elif op == "signWithesk":
        pool, pitch, rows = _pool(m, "signWithesk", batch, mlen)
        rows[:, :z.sk_bytes] = _random_bytes(rng, batch, z.sk_bytes)
        at = A128(z.esk_bytes)
        rows[:, at:at + mlen] = _random_bytes(rng, batch, mlen)
        at += A128(mlen)
        st.update(pool=pool, pitch=pitch, out=rows[:, at:at + z.sig_bytes])
    elif op == "sign":
        sk = _random_bytes(rng, batch, z.sk_bytes)
        pool, pitch, rows = _pool(m, "sign", batch, mlen)
        rows[:, :z.esk_bytes] = _expanded_sk(m, sk)[0][:, :z.esk_bytes]
        rows[:, z.esk_bytes:z.esk_bytes + mlen] = _random_bytes(rng, batch, mlen)
        at = z.esk_bytes + mlen
        st.update(pool=pool, pitch=pitch, out=rows[:, at:at + z.sig_bytes])
    elif op in ("verify", "verifyWithepk"):
        sk, pk = _keys(m, rng, batch)
        msg = _messages(rng, case)
        esk, esk_pitch = _expanded_sk(m, sk)
        sig = _corrupt(rng, _signatures(m, esk, esk_pitch, msg, batch))
        del esk
        pool, pitch, rows = _pool(m, op, batch, mlen)
        if op == "verify":
            rows[:, :z.epk_bytes] = _expanded_pk(m, pk)[0][:, :z.epk_bytes]
        at = A128(z.epk_bytes)
        rows[:, at:at + mlen] = msg["msgs"]
        at += A128(mlen)
        rows[:, at:at + z.sig_bytes] = sig
        at += A128(z.sig_bytes)
        st.update(pool=pool, pitch=pitch, pk=pk, pk_slot=rows[:, z.p_bytes - 16:z.p_bytes - 16 + z.pk_bytes],
                  out=rows[:, at])
    else:  # sign_many, verify_many, sign_shared, verify_shared
        shared = op.endswith("_shared")
        sk, pk = _keys(m, rng, 1 if shared else batch)
        msg = _messages(rng, case)
        esk, esk_pitch = _expanded_sk(m, sk)
        if op.startswith("sign"):
            sig = torch.zeros(batch, z.sig_bytes, dtype=torch.uint8, device="cuda")
            nws = m.sign_shared_ws_bytes(batch) if shared else batch * m.sign_ws_bytes() + 16
            st.update(key=esk, key_stride=esk_pitch, sig=sig)
        else:
            sig = _corrupt(rng, _signatures(m, esk, esk_pitch, msg, batch))
            nws = m.verify_shared_ws_bytes(batch) if shared else 0
            epk, epk_pitch = _expanded_pk(m, pk)
            st.update(key=epk, key_stride=epk_pitch, sig=sig,
                      res=torch.zeros(batch, dtype=torch.uint8, device="cuda"))
        st.update(msg=msg, ws=torch.zeros(nws, dtype=torch.uint8, device="cuda"))
    return st


def run(st):
    case = st["case"]
    op, batch, mlen = case["op"], case["batch"], case["mlen"]
    if op == "queue":
        st["queue"].run()
        return st["out"]
    m = st["mayo"]
    if op == "keypair":
        m.crypto_sign_keypair_from_seed(st["pool"], st["pitch"], batch)
        return st["out"]
    if op == "signWithesk":
        m.crypto_sign_signWithesk(st["pool"], mlen, st["pitch"], batch)
        return st["out"]
    if op == "sign":
        m.crypto_sign_sign(st["pool"], mlen, st["pitch"], batch)
        return st["out"]
    if op == "verify":
        m.crypto_sign_verify(st["pool"], mlen, st["pitch"], batch)
        return st["out"]
    if op == "verifyWithepk":
        st["pk_slot"].copy_(st["pk"])  # the expansion overwrites the compact keys in the pool
        m.crypto_sign_verifyWithepk(st["pool"], mlen, st["pitch"], batch)
        return st["out"]
    if op == "sign_many":
        m.sign_many(st["key"], sig=st["sig"], ws=st["ws"], batch=batch, esk_stride=st["key_stride"], **st["msg"])
        return st["sig"]
    if op == "sign_shared":
        m.sign_shared(st["key"], sig=st["sig"], ws=st["ws"], batch=batch, **st["msg"])
        return st["sig"]
    if op == "verify_many":
        m.verify_many(st["key"], sig=st["sig"], result=st["res"], batch=batch, epk_stride=st["key_stride"], **st["msg"])
        return st["res"]
    m.verify_shared(st["key"], sig=st["sig"], result=st["res"], ws=st["ws"], batch=batch, **st["msg"])
    return st["res"]


def _work_one(op, s, mlen, shared):
    """Bytes and GF(16) multiply-adds (two operations each) of one instance."""
    z = Mayo(s).sizes
    n, m, o, k = z.n, z.m, z.o, z.k
    v = n - o
    e1, e3 = v * (v + 1) // 2, o * (o + 1) // 2
    p3 = m * (e1 * o + v * o * (o + 1) // 2)
    expand_l = m * v * (v - 1) * o
    sign = m * (k * e1 + v * k * (k + 1) // 2 + k * v * o) + m * m * (k * o + 1)
    verify = m * (k * n * (n + 1) // 2 + n * k * (k + 1) // 2)
    if op == "keypair":
        return z.sk_bytes + z.pk_bytes, p3
    if op == "signWithesk":
        return z.sk_bytes + mlen + z.sig_bytes, expand_l + sign
    if op == "verifyWithepk":
        return z.pk_bytes + mlen + z.sig_bytes + 1, verify
    if op.startswith("sign"):
        return (0 if shared else z.esk_bytes) + mlen + z.sig_bytes, sign
    return (0 if shared else z.epk_bytes) + mlen + z.sig_bytes + 1, verify


def work(case):
    op, s, batch, mlen = case["op"], case["set"], case["batch"], case["mlen"]
    if op == "queue":
        each = [_work_one(o, s, mlen, True) for s in SETS for o in ("keypair", "sign", "verify")]
        keys = sum(Mayo(s).sizes.esk_bytes + Mayo(s).sizes.epk_bytes for s in SETS) * MIXED_KEYS
        return {"bytes": keys + batch * sum(b for b, _ in each) / 12, "flops": 2 * batch * sum(f for _, f in each) / 12}
    shared = op.endswith("_shared")
    mean = (32 + max(mlen, 32)) / 2 if case["var"] else mlen
    b, f = _work_one(op, s, mean, shared)
    z = Mayo(s).sizes
    key = (z.esk_bytes if op.startswith("sign") else z.epk_bytes) if shared else 0
    return {"bytes": key + batch * b, "flops": 2 * batch * f}


def exact(case, seed):
    """Outputs are bytes of a fixed format (keys, signatures, verify results): they are compared as
    they are, so there is no 64-bit value beside them."""
    return None
