"""Per-instance verify of messages on both sides of the length past which a CTA takes a group of instances
(VerifyLong in csrc/op_verify.cu), in batches of one wave and one instance more, of full and partial
groups, against the oracle's signatures."""
import os
import re

import numpy as np
import pytest

from cumayo_b200 import Mayo
from oracle import oracle as O

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N = 13  # distinct keys and messages: no multiple of a group
LIMIT = {1: 3328, 2: 3328, 3: 3072, 5: 7168}
BATCHES = {1: (444, 445, 1335, 1775, 1777), 2: (900,), 3: (148, 149, 1183, 1185), 5: (148, 149, 299, 1185)}


def test_the_limits():
    src = open(os.path.join(ROOT, "cumayo_b200", "csrc", "op_verify.cu")).read()
    assert re.search(r"len = SET == 1 \? (\d+) : .*SET == 3 \? (\d+) : (\d+);", src).groups() == tuple(
        str(LIMIT[s]) for s in (1, 3, 5))


@pytest.mark.parametrize("extra", [0, 1, 137])
@pytest.mark.parametrize("s", [1, 2, 3, 5])
def test_verify_long_messages(cuda, s, extra):
    import torch
    m = Mayo(s)
    z = m.sizes
    mlen = LIMIT[s] + extra
    rng = np.random.default_rng(1700 + 10 * s + extra)
    seeds = rng.integers(0, 256, (N, z.sk_bytes), dtype=np.uint8)
    msgs = rng.integers(0, 256, (N, mlen + 3), dtype=np.uint8)  # three bytes that belong to no message
    sig, _ = O.sign_batch(s, O.expandsk_batch(s, seeds), [x[:mlen].tobytes() for x in msgs])
    epk = O.expandpk_batch(s, O.keypair_from_seed_batch(s, seeds))
    d_epk = torch.from_numpy(epk).cuda()
    for n in BATCHES[s]:
        pick = (np.arange(n) * 5 + 1) % N
        bad, at = sig[pick].copy(), pick.copy()
        bad[::7, 3] ^= 1
        at[4::11] = (at[4::11] + 1) % N  # another message
        want = (np.arange(n) % 7 == 0) | (at != pick)
        d_pick = torch.from_numpy(pick).cuda()
        res = torch.full((n + 1,), 0xEE, dtype=torch.uint8, device="cuda")
        m.verify_many(d_epk[d_pick], torch.from_numpy(msgs[at]).cuda(), torch.from_numpy(bad).cuda(), res, n,
                      msg_stride=mlen + 3, mlen=mlen, epk_stride=z.epk_bytes)
        torch.cuda.synchronize()
        assert (res[:n].cpu().numpy() == want).all() and res[n] == 0xEE, n
