"""GPU: the stable pair sort at the edges of its one-block form (8192 pairs) and
of its skipped passes, against numpy's stable argsort."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 255, 257, 4095, 8191, 8192, 8193, 12289, 1 << 20, (1 << 20) + 1])
@pytest.mark.parametrize("kind", ["random", "few", "one", "low", "ordered"])
def test_sort_edges(engine, n, kind):
    import torch
    rng = np.random.default_rng(n)
    k = {"random": lambda: rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2) + np.uint64(1),
         "few": lambda: rng.integers(0, 3, n).astype(np.uint64) * np.uint64(0x0123456789abcdef),
         "one": lambda: np.full(n, 2 ** 64 - 1, dtype=np.uint64),
         "low": lambda: rng.integers(0, 1 << 9, n).astype(np.uint64),
         "ordered": lambda: np.arange(n, dtype=np.uint64)[::-1].copy() << np.uint64(20)}[kind]()
    keys = torch.from_numpy(k.view(np.int64)).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    engine.sort_pairs_u64(keys.data_ptr(), vals.data_ptr(), n)
    torch.cuda.synchronize()
    order = np.argsort(k, kind="stable")
    assert np.array_equal(vals.cpu().numpy().view(np.uint32), order.astype(np.uint32))
    assert np.array_equal(keys.cpu().numpy().view(np.uint64), k[order])


@pytest.mark.parametrize("bits", [8, 11])
@pytest.mark.parametrize("n", [8193, 8223, 12287, 12289, 40_001])
def test_largest_keys_in_partial_tiles(engine, n, bits):
    """Keys equal to what fills a tile past the end, beside ones that share some
    of its digits."""
    import torch
    rng = np.random.default_rng(n)
    k = rng.integers(0, 1 << 63, n, dtype=np.uint64) * np.uint64(2)
    k[rng.random(n) < 0.3] = np.uint64(2 ** 64 - 1)
    top = rng.random(n) < 0.3
    k[top] |= np.uint64(0xffffffff00000000)
    k[-40:] = np.uint64(2 ** 64 - 1)
    keys = torch.from_numpy(k.view(np.int64)).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    try:
        engine.set_tuning(radix_bits=bits)
        engine.sort_pairs_u64(keys.data_ptr(), vals.data_ptr(), n)
    finally:
        engine.set_tuning()
    torch.cuda.synchronize()
    order = np.argsort(k, kind="stable")
    assert np.array_equal(vals.cpu().numpy().view(np.uint32), order.astype(np.uint32))
    assert np.array_equal(keys.cpu().numpy().view(np.uint64), k[order])
