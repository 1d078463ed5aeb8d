"""The one-launch sorts at the edges of their shapes: the bitonic block, one
block of radix passes and several, slices
that fill and that do not, warps without a pair, blocks without a pair, the
largest count it takes and the first one it does not, counts below the
estimate, digits that all keys share, and many equal keys (stability)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ag(native):
    return native


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 64, 65, 1023, 1024, 1025, 2049, 4095, 4096, 4097, 16383, 16385,
                               60001, 65535, 65536, 65537])
@pytest.mark.parametrize("key_bits,used", [(64, 63), (64, 18), (21, 21), (8, 3), (1, 1), (0, 5)])
def test_matches_stable_argsort(ag, n, key_bits, used):
    import torch
    from astro_gb300.radix_sort import RadixSort

    rng = np.random.default_rng(n + key_bits)
    keys = rng.integers(0, 1 << used, n, dtype=np.uint64)
    keys[rng.integers(0, n, n // 3)] = keys[0]
    idx = rng.permutation(n).astype(np.int32)
    room = n + n % 7
    pad = np.full(room - n, 0x7FFFFFFFFFFFFFFF, np.uint64)
    dk = torch.from_numpy(np.concatenate([keys, pad]).view(np.int64)).cuda()
    di = torch.from_numpy(np.concatenate([idx, np.zeros(room - n, np.int32)])).cuda()
    order = np.argsort(keys & np.uint64((1 << key_bits) - 1 if key_bits < 64 else 2**64 - 1), kind="stable")
    for counted, iota in ((False, False), (True, False), (True, True)):
        m = room if counted else n
        ok = torch.full((room,), -1, dtype=torch.int64, device="cuda")
        oi = torch.full((room,), -1, dtype=torch.int32, device="cuda")
        count = torch.tensor([n], dtype=torch.int32, device="cuda") if counted else None
        s = RadixSort(room, key_bits)
        s.sort(dk, None if iota else di, ok, oi, m, count)
        s.status()
        assert np.array_equal(ok[:n].cpu().numpy().view(np.uint64), keys[order])
        assert np.array_equal(oi[:n].cpu().numpy(), order if iota else idx[order])
        assert (ok[n:] == -1).all() and (oi[n:] == -1).all()


def test_count_of_zero_writes_nothing(ag):
    import torch
    from astro_gb300.radix_sort import RadixSort

    keys = torch.arange(5000, 0, -1, device="cuda")
    out = torch.full((5000,), -7, device="cuda")
    oi = torch.full((5000,), -7, dtype=torch.int32, device="cuda")
    RadixSort(5000).sort(keys, None, out, oi, 5000, torch.zeros(1, dtype=torch.int32, device="cuda"))
    assert (out == -7).all() and (oi == -7).all()
