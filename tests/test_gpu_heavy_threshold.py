"""GPU: the heavy-record threshold of the unions: 0 is the automatic one and is
reported as 0, any other value is used as given -- 64 too, which leaves records of
8 to 63 colors without a bitmap."""
import numpy as np
import pytest

from cdbg_gpu import native

pytestmark = pytest.mark.gpu


def _batch(colors):
    """One block between different flanks, every sequence in 10 to 40 of 40 colors, so
    that every record, also one of several sequences, has 10 to 40."""
    rng = np.random.default_rng(colors)
    dna = lambda n: rng.choice(np.frombuffer(b"ACGT", dtype=np.uint8), size=n).tobytes()  # noqa: E731
    block, flat = dna(40), []
    for _ in range(12):
        s = dna(9) + block + dna(9)
        for c in rng.choice(np.linspace(0, colors - 1, 40).astype(int), size=int(rng.integers(10, 41)), replace=False):
            flat.append((int(c), s))
    flat.sort()  # genome by genome, as the reader delivers them
    return native.host_batch([s for _, s in flat], [c for c, _ in flat])


def _run(e, b, colors):
    e.profile(True)
    r = e.build(b, 31, 4, colors)
    out = native.result_frag_bytes(r), native.result_class_words(r).tobytes(), native.result_class_offsets(r).tobytes()
    ks = e.kernel_stats()
    e.profile(False)
    return out, "k_heavy_bitmaps" in ks


@pytest.mark.parametrize("colors,auto", [(60, True), (256, True), (257, False)])
def test_threshold_is_used_as_given(colors, auto):
    b = _batch(colors)
    with native.Engine(0) as e:
        assert e.tuning()["heavy_colors"] == 0
        want, used = _run(e, b, colors)
        assert used == auto
        for v, bitmaps in ((8, True), (64, False), (41, False), (10, True), (0, auto)):
            e.set_tuning(heavy_colors=v)
            assert e.tuning()["heavy_colors"] == v
            got, used = _run(e, b, colors)
            assert got == want and used == bitmaps, v
