"""Graphs of 2 GB and more with p near 1/2, generated by the start kernel in launches
that draw copied slots again instead of reading them: the same edges and retries as
from the tile kernels, whose start region (start_nodes) ends early.  The sizes
leave the last tile and the last launch ragged; d = 5 leaves lanes idle."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,p,bits,slots,model", [
    (2 ** 25 + 37, 4, 0.5, 64, 0, 0),
    (2 ** 23 + 45, 32, 0.4, 64, 1, 0),
    (2 ** 22 + 41, 32, 0.45, 64, 0, 0),
    (2 ** 25 + 2 ** 21 + 1, 9, 0.6, 32, 0, 0),
    (100000103, 5, 0.0, 32, 1, 1),
])
def test_hop_launches_match_tile_kernels(pa, cuda_ok, n, d, p, bits, slots, model):
    import torch
    mode = pa.PA_SEED_STAR_REF if model else pa.PA_SEED_CLIQUE
    kw = dict(seed=n, id_bits=bits, model=model, seed_mode=mode)
    a, sa = pa.generate(pa.make_params(n, d, p, layout=slots, **kw))
    b, sb = pa.generate(pa.make_params(n, d, p, start_nodes=2 ** 20, **kw))
    assert a.numel() * a.element_size() >= 2_000_000_000
    if slots:   # only the start kernel writes this layout
        b = b[-(n - d - 1) * d:, 1].view(n - d - 1, d)
    assert torch.equal(a, b)
    assert sa.retries == sb.retries


def test_hop_launches_captured_prefilled_and_on_few_blocks(pa, cuda_ok):
    """The same graph from a replayed plan into dirty scratch, from a buffer filled
    beforehand, and from grids of 3 and 500 blocks."""
    import torch
    kw = dict(seed=3, id_bits=64)
    n, d, p = 2 ** 25 + 3, 4, 0.5
    want, st = pa.generate(pa.make_params(n, d, p, **kw))
    prm = pa.make_params(n, d, p, **kw)
    edges, scratch = pa.alloc_buffers(prm)
    scratch.fill_(0xab)
    plan = pa.Plan(prm, edges, scratch)
    for _ in range(2):
        edges.zero_()
        plan.launch()
        assert pa.finish(scratch).status == 0
        assert torch.equal(edges[: want.shape[0]], want)
    plan.close()
    for extra in (dict(flags=pa.PA_FLAG_PREFILLED), dict(blocks=3), dict(blocks=500)):
        q = pa.make_params(n, d, p, **kw, **extra)
        edges.zero_()
        scratch.fill_(0xcd)
        if "flags" in extra:
            pa.fill(q, edges)
        pa.generate_into(q, edges, scratch)
        assert pa.finish(scratch).status == 0
        assert torch.equal(edges[: want.shape[0]], want)
