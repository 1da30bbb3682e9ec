"""The CSR sort at its tile edges: item counts one below, at and above whole
tiles (8,192 items), whole warps of a tile (512) and whole rounds (32), for
digits of 8 and 9 bits, and keys that repeat through a whole round."""
import numpy as np
import pytest

import _oracle as orc

pytestmark = pytest.mark.gpu

# d = 1 with the clique seed has exactly n - 1 items
COUNTS = [31, 32, 33, 511, 512, 513, 8191, 8192, 8193, 16383, 16384, 16385, 70000, 300001]


@pytest.mark.parametrize("p", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("items", COUNTS)
def test_csr_item_counts(pa, cuda_ok, items, p):
    n = items + 1
    prm = pa.make_params(n, 1, p, seed=items, id_bits=32)
    edges, _ = pa.generate(prm)
    assert edges.shape[0] == items
    rowptr, col = pa.build_csr(prm, edges)
    want_rp, want_col = orc.csr(orc.generate(n, 1, p, items, orc.SEED_CLIQUE), orc.SEED_CLIQUE)
    assert (rowptr.cpu().numpy() == want_rp).all()
    assert (col.cpu().numpy().astype(np.int64) == want_col).all()


@pytest.mark.parametrize("n,d,p", [(200000, 1, 0.0), (200000, 1, 0.1), (150000, 2, 0.05),
                                   (100001, 3, 0.0), (33000, 32, 1.0), (40, 1, 0.5), (3, 1, 0.5)])
def test_csr_rows_without_in_edges(pa, cuda_ok, n, d, p):
    """Long runs of rows without in-edges beside rows with most of them: the shares of
    rows and items a warp of the rowptr pass takes end inside both."""
    prm = pa.make_params(n, d, p, seed=n + d, id_bits=64)
    edges, _ = pa.generate(prm)
    rowptr, col = pa.build_csr(prm, edges)
    want_rp, want_col = orc.csr(orc.generate(n, d, p, n + d, orc.SEED_CLIQUE), orc.SEED_CLIQUE)
    assert (rowptr.cpu().numpy() == want_rp).all()
    assert (col.cpu().numpy() == want_col).all()
