"""Where large sorts ask whether the top digits suffice: below 1,572,864 pairs
they do not, since keys that do not qualify would pay for the question. Counter
word 10 of the scratch holds from bit 8 the top digits sorted by."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,top", [(1400000, 0), (1572863, 0), (1572864, 3)])
def test_question_asked_from(native, n, top):
    import torch

    from astro_gb300.radix_sort import RadixSort

    gen = torch.Generator(device="cuda").manual_seed(n)
    keys = torch.randint(0, (1 << 48) - 1, (n,), device="cuda", generator=gen, dtype=torch.int64)
    index = torch.arange(n, device="cuda", dtype=torch.int32)
    keys_out, index_out = torch.full_like(keys, -1), torch.full_like(index, -1)
    sorter = RadixSort(n, 48)
    sorter.sort(keys, index, keys_out, index_out, n)
    want, order = torch.sort(keys, stable=True)
    assert torch.equal(keys_out, want) and torch.equal(index_out.long(), order)
    assert int(sorter.temp[40:44].view(torch.int32)) >> 8 == top
