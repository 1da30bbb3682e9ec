"""The CSR sort's two kernels at the edges of their tiles: 8,192 items (long lists, and
lists whose look-back words find no room otherwise) and 2,048 items (short ones), with
8-bit and 9-bit digits; item counts one below, at and above whole tiles, and on both
sides of the line between the kernels (148 tiles of 8,192)."""
import numpy as np
import pytest

import _oracle as orc

pytestmark = pytest.mark.gpu

LARGE, SMALL, LINE = 8192, 2048, 148 * 8192


def digits(n):
    """(bits of a digit, passes): the fewest passes of 8 or 9 bits; on a tie of three, 9."""
    bits = max(1, (n - 1).bit_length())
    eight, nine = -(-bits // 8), -(-bits // 9)
    return (9, nine) if nine < eight or (nine == eight and eight == 3) else (8, eight)


def tile(n, m, id_bits):
    words = (8 << digits(n)[0]) * -(-m // SMALL)
    return SMALL if m <= LINE and words <= (8 * m if id_bits == 64 else 8 * (n + 1)) else LARGE


def rows_for(d, items):
    """The least number of rows for which a clique-seeded graph has `items` mod LARGE
    items (d odd)."""
    return (items - d * (d + 1) // 2) * pow(d, -1, LARGE) % LARGE


CASES = []
for off in (-1, 0, 1):
    # (d, rows, id bits, tile, digit bits)
    CASES += [(11, rows_for(11, off), 32, LARGE, 8), (31, rows_for(31, off), 32, LARGE, 8)]
    CASES += [(9, 65536 + LARGE + rows_for(9, off), 32, LARGE, 9)]
    CASES += [(1, 149 * LARGE + off - 1, b, LARGE, 9) for b in (32, 64)]
    CASES += [(1, LINE + off - 1, b, SMALL if off < 1 else LARGE, 9) for b in (32, 64)]
    CASES += [(1, k * SMALL + off - 1, b, SMALL, 8) for k in (1, 2, 20) for b in (32, 64)]
    CASES += [(1, 100 * SMALL + off - 1, b, SMALL, 9) for b in (32, 64)]


@pytest.mark.parametrize("d,rows,bits,want_tile,want_digits", CASES)
def test_csr_at_tile_edges(pa, cuda_ok, d, rows, bits, want_tile, want_digits):
    n = rows + d + 1
    for p in (0.0, 0.5):
        prm = pa.make_params(n, d, p, seed=rows, id_bits=bits)
        m = pa.edge_count(prm)
        assert (tile(n, m, bits), digits(n)[0]) == (want_tile, want_digits), (n, m)
        assert pa.csr_launches(prm) == 4 + digits(n)[1]
        edges, _ = pa.generate(prm)
        rowptr, col = pa.build_csr(prm, edges)
        want_rp, want_col = orc.csr(orc.generate(n, d, p, rows, orc.SEED_CLIQUE), orc.SEED_CLIQUE)
        assert (rowptr.cpu().numpy() == want_rp).all()
        assert (col.cpu().numpy().astype(np.int64) == want_col).all()
