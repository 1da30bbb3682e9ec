"""pa_degrees where the seed graph is a large part of the list: seed edges by the
thousand and the million, seed ids on both sides of the counters in shared memory
(8,192), both seed graphs and layouts, ids outside the graph among them; and no slower
for it than for as many pairs of generated nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _seed_pairs(d, star):
    if star:
        return np.stack([np.full(d, d), np.arange(d)], axis=1)
    v, j = np.tril_indices(d + 1, -1)
    return np.stack([v, j], axis=1)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("star", [False, True])
@pytest.mark.parametrize("d,rows", [(1, 0), (1, 1), (127, 2), (128, 3), (1000, 0), (1000, 5), (8190, 3),
                                    (8192, 2), (9001, 1)])
def test_degrees_of_seed_graphs(pa, cuda_ok, d, rows, star, bits):
    import torch
    n = d + 1 + rows
    mode = pa.PA_SEED_STAR_REF if star else pa.PA_SEED_CLIQUE
    dt = torch.int64 if bits == 64 else torch.int32
    rng = np.random.default_rng(d + rows)
    targets = rng.integers(0, d + 1, size=(rows, d))
    seeds = _seed_pairs(d, star)
    pairs = np.concatenate([seeds, np.stack([np.repeat(np.arange(d + 1, n), d), targets.ravel()],
                                            axis=1)])
    want = np.bincount(pairs.ravel(), minlength=n)
    prm = pa.make_params(n, d, 0.5, id_bits=bits, seed_mode=mode)
    assert pa.edge_count(prm) == len(pairs)
    got = pa.degrees(prm, torch.from_numpy(pairs).to("cuda", dt))
    assert (got.cpu().numpy() == want).all()
    # in another order, and with ids outside the graph: such a pair counts at neither end
    broken = rng.permutation(pairs)
    broken[::5, 0] = n
    broken[::7, 1] = -1
    ok = ((broken >= 0) & (broken < n)).all(axis=1)
    got = pa.degrees(prm, torch.from_numpy(broken).to("cuda", dt))
    assert (got.cpu().numpy() == np.bincount(broken[ok].ravel(), minlength=n)).all()
    if rows:
        prm = pa.make_params(n, d, 0.5, id_bits=bits, seed_mode=mode, layout=pa.PA_LAYOUT_SLOTS)
        got = pa.degrees(prm, torch.from_numpy(targets).to("cuda", dt))
        assert (got.cpu().numpy() == want).all()


def test_seed_edges_take_no_longer_than_others(pa, cuda_ok):
    import torch

    def ms(prm, edges):
        best = None
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            pa.degrees(prm, edges)
            b.record()
            torch.cuda.synchronize()
            best = min(best or 1e9, a.elapsed_time(b))
        return best

    d = 8000
    seeds = pa.make_params(d + 1, d, 0.5)      # the clique alone, 3.2 * 10^7 pairs
    a, _ = pa.generate(seeds)
    others = pa.make_params(a.shape[0] // 32 + 16, 32, 0.5)
    b, _ = pa.generate(others)
    assert abs(a.shape[0] - b.shape[0]) < 1000
    # both read the list once; one block for all seed edges takes 60 times as long
    assert ms(seeds, a) < 8 * ms(others, b)
