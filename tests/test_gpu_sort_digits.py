"""GPU: the stable pair sort where a digit's counter passes from lane to lane of
a warp between two rounds: 1 to 256 distinct digits, so that the lane that
updates a counter is another one in the next round, against numpy's stable
argsort.  One-block and multi-tile forms, both digit widths."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [8, 11])
@pytest.mark.parametrize("n", [8191, 8192, 8193, 70_001])
@pytest.mark.parametrize("digits", [1, 2, 3, 31, 33, 256])
def test_counters_between_rounds(engine, n, digits, bits):
    import torch
    rng = np.random.default_rng(digits * 7 + bits)
    # position p holds digit (p + p // 32) % digits in every byte: the first lane
    # with a digit moves by one each round; a third of the keys are random
    p = np.arange(n, dtype=np.uint64)
    d = (p + p // np.uint64(32)) % np.uint64(digits)
    mix = rng.random(n) < 0.33
    d[mix] = rng.integers(0, digits, int(mix.sum())).astype(np.uint64)
    k = d * np.uint64(0x0101010101010101)
    keys = torch.from_numpy(k.view(np.int64).copy()).cuda()
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
