"""GPU: even k, where a k-mer can be its own reverse complement: at the end of a
chain (its one neighbour lies on both of its sides), inside one, next to another
and in tandem repeats, with the fragments of the CPU oracle."""
import numpy as np
import pytest

from test_gpu_edges import _check, _dna

pytestmark = pytest.mark.gpu


def _rc(s):
    return s.translate(bytes.maketrans(b"ACGT", b"TGCA"))[::-1]


@pytest.mark.parametrize("k", [4, 6, 10, 20, 30, 32, 62])
@pytest.mark.parametrize("seed", [0, 1, 2])
def test_own_reverse_complements(oracle, engine, tmp_path, k, seed):
    rng = np.random.default_rng(100 * k + seed)
    pal = lambda: (lambda h: h + _rc(h))(_dna(rng, k // 2))  # noqa: E731
    n = 40 if k < 8 else 300
    g0 = [_dna(rng, n) + pal(), pal() + _dna(rng, n), _dna(rng, n) + pal() + _dna(rng, n), pal(), _dna(rng, n)]
    g1 = [pal() + _dna(rng, n // 3) + pal(), b"AT" * k, b"ACGT" * k, g0[0][-2 * k:], _rc(g0[1])[-k - 3:]]
    g2 = [(lambda h: h + _rc(h))(_dna(rng, 2 * k)), g0[2][n - 5: n + k + 5], _dna(rng, 5 * k)]
    for B in (1, 9):
        d = tmp_path / str(B)
        d.mkdir()
        _check(oracle, engine, d, [g0, g1, g2], k, B)
