"""pa_degrees against the oracle and a plain count: sizes around the shared
counters (8,192 ids), chunk edges (1,024 .. 8,192 pairs), 32-bit counts and their
in-place widening (above 2^22 nodes), d = 1 and d > 32, both layouts and id widths, lists in another order
than generated, lists with ids outside the graph, and a list that is aligned to
its ids but not to its pairs."""
import ctypes

import numpy as np
import pytest

import _oracle as orc

pytestmark = pytest.mark.gpu

SIZES = [(2, 1), (3, 2), (8191, 1), (8192, 1), (8193, 1), (8194, 3), (16385, 2), (16386, 1),
         (40000, 7), (30000, 32), (3000, 40), (600, 555),
         (2 ** 22, 1), (2 ** 22 + 1, 2), (2 ** 22 + 8193, 1)]


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n,d", SIZES)
def test_degrees_match_oracle(pa, cuda_ok, n, d, bits, layout):
    for mode, p in ((orc.SEED_CLIQUE, 0.4), (orc.SEED_STAR_REF, 0.1)):
        prm = pa.make_params(n, d, p, seed=n, id_bits=bits, seed_mode=mode, layout=layout)
        edges, _ = pa.generate(prm)
        if edges.numel() == 0:
            continue   # SLOTS of a seed graph alone: no array to hand over
        want = orc.degrees(orc.generate(n, d, p, n, mode), mode)
        assert (pa.degrees(prm, edges).cpu().numpy() == want).all()


def counted(pairs, n):
    ok = ((pairs >= 0) & (pairs < n)).all(axis=1)
    return np.bincount(pairs[ok].ravel(), minlength=n)


@pytest.mark.parametrize("bits", [32, 64])
def test_degrees_of_other_lists(pa, cuda_ok, bits):
    import torch
    n, d = 20000, 5
    prm = pa.make_params(n, d, 0.3, seed=3, id_bits=bits)
    edges, _ = pa.generate(prm)
    gen = torch.Generator().manual_seed(1)
    shuffled = edges[torch.randperm(edges.shape[0], generator=gen).cuda()].contiguous()
    flipped = edges.flip(1).contiguous()
    broken = edges.clone()
    broken[1000:3000:7, 0] = n
    broken[2000:9000:11, 1] = -1
    broken[5000:9000:13, 1] = 2 ** 31 - 1
    for lst in (shuffled, flipped, broken):
        got = pa.degrees(prm, lst).cpu().numpy()
        assert (got == counted(lst.cpu().numpy().astype(np.int64), n)).all()
    # the same list one id further on: aligned to an id only
    raw = torch.empty(edges.numel() + 1, dtype=edges.dtype, device="cuda")
    raw[1:] = edges.reshape(-1)
    deg = torch.empty(n, dtype=torch.int64, device="cuda")
    s = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    pa.check(pa.lib().pa_degrees(ctypes.byref(prm), ctypes.c_void_p(raw.data_ptr() + bits // 8),
                                 ctypes.c_void_p(deg.data_ptr()), s), "pa_degrees")
    assert (deg.cpu().numpy() == counted(edges.cpu().numpy().astype(np.int64), n)).all()
