"""The graph generator at the edges of its turns (1,024 candidates), masks (32) and rows
(truncation, padding, p = 0 and 1) against its CPU restatement, bit for bit."""
import numpy as np
import pytest

import oracle
from spice_b200 import Layout, Snn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pops,conns", [
    ([40, 1023], [(0, 1, 0.1), (1, 0, 0.9)]),
    ([40, 1024], [(0, 1, 0.3)]),
    ([40, 1025], [(0, 1, 0.1), (0, 0, 0.5)]),
    ([33, 31, 32], [(0, 1, 1.0), (0, 2, 0.5), (1, 0, 1.0), (2, 2, 0.01)]),
    ([50, 2049], [(0, 1, 1.0), (1, 1, 0.0005)]),
    ([3000], [(0, 0, 0.02)]),   # rows of mean 60 cut at 96: some are truncated
    ([64, 5], [(0, 1, 0.0), (0, 0, 1.0)]),
])
def test_generator_edges(pops, conns):
    lay = Layout(pops, conns)
    for seed in (1, 2 ** 40 + 17):
        edges, width = Snn("synth", lay, delay=1, graph_seed=seed).adj()
        ref, ref_width = oracle.generate(pops, conns, seed, graph="philox")
        assert width == ref_width and np.array_equal(edges, ref)
