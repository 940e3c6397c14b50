"""The row, search, routing, optimizer and attention kernels at the sizes where they can go wrong: edges of tiles and chunks,
remainders, the smallest and largest of a range, every branch of a dispatch - against the PyTorch statements."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp(min=1e-30)).item()


# ------------------------------------------------------------------------------------------------ keys and locks
def _share0_words(T, count):
    """Words whose 1-gram key belongs to share 0 of a text of T words: they overflow that share's table."""
    shares, out, mask, w = T // 256 + 1, [], (1 << 64) - 1, 0
    while len(out) < count:
        k = w * 0x9E3779B97F4A7C15 & mask
        k ^= k >> 29
        h = (k * 0xBF58476D1CE4E5B9 & mask) >> 32
        if h * shares >> 32 == 0:
            out.append(w)
        w += 1
    return torch.tensor(out)


@pytest.mark.parametrize("text", ["zipf", "same", "pair", "distinct", "overflow"])
@pytest.mark.parametrize("B,T,n_keys", [(1, 1, 3), (3, 2, 2), (2, 5, 3), (3, 127, 1), (2, 128, 3), (2, 257, 3), (2, 4099, 3), (1, 30000, 3), (1, 30001, 3)])
def test_lock_find_tables_and_scan(text, B, T, n_keys):
    from memarch_b200.ops import anchors, ref
    g = torch.Generator().manual_seed(T)
    V = 1 << 20
    if text == "zipf":
        x = (torch.exp(torch.rand(B, T, generator=g) * 8).long() - 1)
    elif text == "same":
        x = torch.full((B, T), V - 1)
    elif text == "pair":
        x = (torch.arange(T)[None] % 2 + torch.arange(B)[:, None]).long()
    elif text == "distinct":
        x = torch.stack([torch.randperm(max(T, 8), generator=g)[:T] for _ in range(B)])
    else:
        words = _share0_words(T, 700)
        x = words[torch.randint(0, 700, (B, T), generator=g)]
    bucket = torch.randint(0, 9, (1000,), generator=g)
    for lb in (None, bucket):
        got = anchors.find_locks(x.cuda(), V, n_keys, None if lb is None else lb.cuda())
        want = ref.find_locks(x, V, max(n_keys, 2), lb)
        for a, b, per_key in zip(got, want, (True, True, False, True)):
            if per_key and n_keys == 1:
                continue                                        # the statement has at least two key lengths
            assert torch.equal(a.cpu(), b)
    if n_keys == 1:
        got, want = anchors.find_locks(x.cuda(), V, 1, None), ref.find_locks(x, V, 2, None)
        assert torch.equal(got[0][..., 0].cpu(), want[0][..., 0]) and torch.equal(got[3][..., 0].cpu(), want[3][..., 0])
