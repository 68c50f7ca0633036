"""GPU: k-mers in many records -- neighbours with the same records, with as many
but other ones, with one more -- around the list lengths where a lane, then the
warp, compares them, against the CPU oracle."""
import numpy as np
import pytest

from test_gpu_edges import _check, _dna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [31, 63])
@pytest.mark.parametrize("n", [2, 7, 8, 9, 31, 32, 33, 127, 128, 129, 300])
def test_neighbours_records(oracle, engine, tmp_path, k, n):
    rng = np.random.default_rng(n + k)
    colors = 12
    seqs = []  # (color, sequence)
    for _ in range(3):  # three blocks, each between other flanks in every carrier
        x = _dna(rng, k + 4)
        own = [int(c) for c in rng.integers(0, colors, n)]
        seqs += [(c, _dna(rng, 5) + x + _dna(rng, 5)) for c in own]                        # all five k-mers
        for extra in range(2):  # as many carriers of the first two k-mers as of the last two
            seqs.append((extra, _dna(rng, 6) + x[: k + 1] + _dna(rng, 6)))
            seqs.append((extra + 2, _dna(rng, 6) + x[3:] + _dna(rng, 6)))
    genomes = [[] for _ in range(colors)]
    for c, s in seqs:
        genomes[c].append(s)
    for g in genomes:
        g.append(_dna(rng, k + 9))
    for B in (1, 7):
        d = tmp_path / str(B)
        d.mkdir()
        _check(oracle, engine, d, genomes, k, B)
