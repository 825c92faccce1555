"""Kernels at the sizes where their tiling can go wrong -- edges of tiles and
passes, remainders, the smallest and largest of a range -- against the oracle
(bit for bit) or a plain restatement of the same operation."""
import numpy as np
import pytest

from helpers import make_queries, oracle_of, tiny_index
from mvr import SEM_BASIC, SEM_PP, Index

pytestmark = pytest.mark.gpu


def gpu_index(ix):
    return Index.from_arrays(ix["item_n_vec"], ix["centroid"], ix["vq_code"], ix["ivf_off"],
                             ix["ivf_size"], ix["ivf_ids"], ix["weight"], ix["n_bit"],
                             ix["residual"])


# doc lengths around the exact rerank's 32-token rows and 128-token tiles
LENGTHS = [1, 2, 31, 32, 33, 63, 64, 65, 127, 128, 129, 160, 255, 256, 257, 300]


@pytest.mark.parametrize("n_bit", [1, 2, 4, 8])
def test_exact_rerank_edges(n_bit):
    """Query widths around the 16- and 32-token passes, shortlists around the
    docs-per-CTA windows (4 to 64), one query and enough for the widest window."""
    ix = tiny_index(n_doc=160, n_centroid=32, n_bit=n_bit, seed=50 + n_bit,
                    lengths=(LENGTHS * 10)[:160])
    o = oracle_of(ix)
    with gpu_index(ix) as g:
        for nq, sem in ((1, SEM_PP), (15, SEM_PP), (16, SEM_BASIC), (17, SEM_PP), (32, SEM_BASIC),
                        (33, SEM_PP), (48, SEM_PP), (49, SEM_BASIC), (64, SEM_PP)):
            q, off = make_queries(ix, 2, nq, seed=nq)
            for ptk in (3, 4, 9, 65, 160):
                r = o.search(q, off, 3, 8, ptk, sem)
                s, i = g.search(q, 3, 8, ptk, tok_off=off, semantics=sem)
                np.testing.assert_array_equal(i, r[1])
                np.testing.assert_array_equal(s, r[0])
        q, off = make_queries(ix, 700, (1, 64), seed=3)
        r = o.search(q, off, 3, 8, 130)
        s, i = g.search(q, 3, 8, 130, tok_off=off)
        np.testing.assert_array_equal(i, r[1])
        np.testing.assert_array_equal(s, r[0])
