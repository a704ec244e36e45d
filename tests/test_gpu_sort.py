"""The frontier dedupe's radix sort (cz_sort_pairs) against a stable reference sort: below 2^22 keys one launch
per 8-bit digit pass with decoupled look-back, from 2^22 keys per-tile histograms, a scan and the same staged
scatter per pass. The dedupe relies on stability (equal class keys keep the
order of their child indices) and on the bit ranges it sorts by: the top 32 bits of the class key, and the low
bytes of the child index when the kept classes are put back in order."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    import cheese_b200 as cz
    e = cz.Engine(0)
    yield e
    e.close()


def stable_reference(keys, vals, lo, hi):
    """(keys, vals) stably sorted by bits [lo, hi) of the key, with torch on the device"""
    import torch
    k = keys.clone()
    if hi - lo < 64:
        k = (k >> lo) & ((1 << (hi - lo)) - 1) if hi - lo < 63 else (k >> lo)
    u = k ^ torch.iinfo(torch.int64).min if hi - lo == 64 else k      # unsigned order of the full 64-bit key
    _, order = torch.sort(u, stable=True)
    return keys[order], vals[order]


@pytest.mark.parametrize("n,lo,hi,spread", [
    (2, 0, 64, 64), (2047, 32, 64, 64), (2048, 32, 64, 64), (2049, 32, 64, 64), (100000, 32, 64, 64),
    (100000, 32, 64, 3), (300001, 0, 64, 64), (1 << 20, 0, 24, 24), (3 << 20, 32, 64, 9), (1 << 22, 32, 64, 12),
    (5000000, 32, 64, 64), (9000001, 0, 40, 64)])
def test_sort_matches_stable_reference(engine, n, lo, hi, spread):
    """few distinct keys (spread = random bits in the key) exercise long equal runs across many tiles"""
    import torch
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(n + lo + spread)
    r = torch.randint(0, 1 << 62, (n,), dtype=torch.int64, device=dev, generator=g)
    keys = (r & ((1 << spread) - 1)) << (64 - spread) if spread < 64 else r * 4 + (r >> 60)
    vals = torch.arange(n, dtype=torch.int32, device=dev)
    want_k, want_v = stable_reference(keys, vals, lo, hi)
    k, v = keys.clone(), vals.clone()
    torch.cuda.synchronize()                  # the sort runs on the engine's stream, not torch's
    engine.sort_pairs(k.data_ptr(), v.data_ptr(), n, lo, hi)
    torch.cuda.synchronize()
    assert torch.equal(v, want_v)
    assert torch.equal(k, want_k)


def test_sort_refuses_partial_bytes(engine):
    import torch
    k = torch.zeros(4, dtype=torch.int64, device="cuda")
    v = torch.zeros(4, dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError):
        engine.sort_pairs(k.data_ptr(), v.data_ptr(), 4, 0, 12)


@pytest.mark.parametrize("lo,hi", [(32, 64), (0, 8), (0, 64), (24, 64)])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 1023, 1025, 8191, 8192, 8193, 8193 + 2048])
def test_counted_and_digit_sorts_meet(engine, n, lo, hi):
    """sorts of up to 8192 pairs are placed by counting, larger ones by digit passes: block and tile edges on both
    sides, 32-bit and 64-bit digits, half of the keys equal"""
    import torch
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(7 * n + lo + hi)
    keys = torch.randint(-(1 << 62), 1 << 62, (n,), dtype=torch.int64, device=dev, generator=g) * 2
    keys[::2] = keys[0].clone()
    vals = torch.arange(n, dtype=torch.int32, device=dev)
    want_k, want_v = stable_reference(keys, vals, lo, hi)
    torch.cuda.synchronize()
    engine.sort_pairs(keys.data_ptr(), vals.data_ptr(), n, lo, hi)
    torch.cuda.synchronize()
    assert torch.equal(vals, want_v)
    assert torch.equal(keys, want_k)


@pytest.mark.parametrize("n", [4095, 4096, 4097, 6144])
def test_one_byte_sorts_meet(engine, n):
    """one digit pass is counted only up to 4096 pairs: both sides of that line, equal keys in their order"""
    import torch
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(n)
    keys = torch.randint(-(1 << 62), 1 << 62, (n,), dtype=torch.int64, device=dev, generator=g) * 2
    vals = torch.arange(n, dtype=torch.int32, device=dev)
    for lo in (0, 32, 56):
        want_k, want_v = stable_reference(keys, vals, lo, lo + 8)
        k, v = keys.clone(), vals.clone()
        torch.cuda.synchronize()
        engine.sort_pairs(k.data_ptr(), v.data_ptr(), n, lo, lo + 8)
        torch.cuda.synchronize()
        assert torch.equal(v, want_v)
        assert torch.equal(k, want_k)
