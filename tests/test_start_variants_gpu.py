"""The start kernel's variants (1, 2 or 4 warp passes per tile, 32, 40 or 48
warps per SM), chosen by the number of nodes and the chance of a direct pick: sizes on
both sides of the lines (2^20, 2^22 and 2^24 nodes), last tiles cut short, both layouts and id
widths, d with idle lanes, against the oracle."""
import numpy as np
import pytest

import _oracle as orc

pytestmark = pytest.mark.gpu

EDGE = [(2 ** 20 + d + 1 + x, d) for d in (1, 3) for x in (-1, 0, 1)] + \
       [(2 ** 22 + d + 1 + x, d) for d in (1, 2) for x in (-1, 0, 5)] + \
       [(2 ** 24 + 2 + x, 1) for x in (0, 1)]


@pytest.mark.parametrize("p", [0.0, 0.3, 0.8, 1.0])
@pytest.mark.parametrize("n,d", EDGE)
def test_variants_match_oracle(pa, cuda_ok, n, d, p):
    slots = (n + d) % 2
    bits = 64 if n % 3 == 0 else 32
    prm = pa.make_params(n, d, p, seed=n, id_bits=bits, layout=slots)
    edges, st = pa.generate(prm)
    G, retries = orc.generate(n, d, p, n, orc.SEED_CLIQUE, with_retries=True)
    assert st.retries == retries
    got = edges.cpu().numpy()
    want = G[d + 1:] if slots else orc.pairs_slot_order(G, orc.SEED_CLIQUE)
    assert (got.astype(np.int64) == want).all()


@pytest.mark.parametrize("p", [0.1, 0.3])
@pytest.mark.parametrize("n,d", [(2 ** 21 + 5 + x, 4) for x in (-1, 0)] + [(2 ** 21 + 6, 5)])
def test_variants_by_slots(pa, cuda_ok, n, d, p):
    """The lines at 2^23 slots, 2^21 nodes and p = 1/4."""
    test_variants_match_oracle(pa, cuda_ok, n, d, p)


def test_ba_above_the_lines(pa, cuda_ok):
    for n in (2 ** 20 + 9, 2 ** 22 + 9):
        prm = pa.make_params(n, 2, 0.0, seed=5, id_bits=64, seed_mode=pa.PA_SEED_STAR_REF,
                             model=pa.PA_MODEL_BA)
        edges, st = pa.generate(prm)
        G, retries = orc.generate_ba(n, 2, 5, with_retries=True)
        assert st.retries == retries
        assert (edges.cpu().numpy() == orc.pairs_slot_order(G, orc.SEED_STAR_REF)).all()


def test_batch_in_the_scratch_of_coarse_levels(pa, cuda_ok):
    """A caller's scratch too small for the tables of many small levels gets fewer
    levels and the same graphs; one too small for those is refused."""
    import ctypes
    import torch
    prms = [pa.make_params(n, d, 0.4, seed=i) for i, (n, d) in
            enumerate([(30000, 4), (1000, 32), (70001, 3), (9, 8), (5000, 17)])]
    b = pa.Batch(prms)
    b.generate()
    assert b.finish().status == 0
    want = [b.graph(i).clone() for i in range(len(prms))]
    full, least = b.scratch.numel(), None
    for size in range(full, 0, -256):
        b.scratch = torch.empty(size, dtype=torch.uint8, device="cuda")
        for i in range(len(prms)):
            b.graph(i).zero_()
        try:
            b.generate()
        except pa.CuppaError as e:
            assert e.status == pa.PA_ERR_CAPACITY
            break
        least = size
        assert b.finish().status == 0
        assert all(torch.equal(b.graph(i), w) for i, w in enumerate(want))
    assert least is not None and least < full


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("bits", [32, 64])
def test_one_launch_set_up(pa, cuda_ok, bits, layout):
    """The control block, the claim counters and the region around a small graph's
    edges: seed edges of odd counts (ragged region ends), a scratch and a buffer full of
    other bytes, two generations in a row on one stream, sizes around the largest
    region that is filled by the same launch (32 MB)."""
    import torch
    slot = (1 if layout else 2) * bits // 8
    for n, d in [(50, 1), (1000, 3), (1001, 5), (3000, 40),
                 ((32 << 20) // slot // 4 + 5, 4), ((32 << 20) // slot // 4 + 6, 4)]:
        prm = pa.make_params(n, d, 0.5, seed=n, id_bits=bits, layout=layout)
        G = orc.generate(n, d, 0.5, n, orc.SEED_CLIQUE)
        want = G[d + 1:] if layout else orc.pairs_slot_order(G, orc.SEED_CLIQUE)
        edges, scratch = pa.alloc_buffers(prm)
        for byte in (0, 7):
            edges.fill_(byte)
            scratch.fill_(byte)
            pa.generate_into(prm, edges, scratch)
            pa.generate_into(prm, edges, scratch)
            assert pa.finish(scratch).status == 0
            assert (edges.cpu().numpy().astype(np.int64) == want).all()
