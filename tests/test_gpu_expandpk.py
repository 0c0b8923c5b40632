"""Expand-pk around the batches where the key's split over CTAs changes and where the blocks that hold the
key come from a launch of their own, at every alignment, against the oracle."""
import numpy as np
import pytest

from cumayo_b200 import Mayo
from oracle import oracle as O

pytestmark = pytest.mark.gpu
N = 19


@pytest.mark.parametrize("off", [0, 1, 2, 3])
@pytest.mark.parametrize("s", [1, 2, 3, 5])
def test_expandpk_split_edges(cuda, s, off):
    import torch
    m = Mayo(s)
    z = m.sizes
    rng = np.random.default_rng(1900 + 4 * s + off)
    cpk = O.keypair_from_seed_batch(s, rng.integers(0, 256, (N, z.sk_bytes), dtype=np.uint8))
    epk = torch.from_numpy(O.expandpk_batch(s, cpk)).cuda()
    at, pitch = z.p_bytes - 16, z.epk_bytes + off  # the compact key lies where P ends
    assert at + z.pk_bytes <= pitch
    for n in (1, 7, 28, 32, 40, 48, 49, 50, 52, 74, 75, 148, 149):
        pick = (np.arange(n) * 4 + 1) % N
        pool = torch.zeros(off + n * pitch, dtype=torch.uint8, device="cuda")[off:]  # ends with the last row
        rows = pool.view(n, pitch)
        rows[:, at: at + z.pk_bytes] = torch.from_numpy(cpk[pick]).cuda()
        m.crypto_sign_expandpk(pool, pitch, n)
        assert torch.equal(rows[:, : z.epk_bytes], epk[torch.from_numpy(pick).cuda()]), n
        assert not rows[:, z.epk_bytes:].any(), n
