"""The batch autotuner times satisfaction shapes; the chunk of a solve's start
is not one of them and stays as asked for, from trials and from the cache."""
import pytest

import gsc_b200 as G
import gsc_cases as C

pytestmark = pytest.mark.gpu


def test_autotuned_batch_keeps_its_chunk():
    cases = [C.random_instance(77, i, n_hi=(24, 24, 20, 18)) for i in range(3)]
    with G.Context(0) as ctx:
        for chunk, used in ((512, 512), (0, 2048)):
            b = G.Batch(ctx, cases, autotune=True, chunk_words=chunk)
            rep = b.report()
            assert rep["tuned"] in (1, 2) and rep["chunk_words"] == used
            b.solve(graph=True)
            assert b.read(0)["iterations"] > 0
            b.close()
