"""A call that the CUDA runtime refuses leaves nothing behind: the next call of the same
thread, valid in itself, succeeds."""
import ctypes

import pytest

import _oracle as orc

pytestmark = pytest.mark.gpu

TOO_MANY = 0xffffffff   # blocks: the runtime refuses a grid of 2^31 and more


def test_calls_after_a_refused_launch(pa, cuda_ok):
    import torch
    good = pa.make_params(5000, 4, 0.5, seed=3)
    want = orc.pairs_slot_order(orc.generate(5000, 4, 0.5, 3, orc.SEED_CLIQUE), orc.SEED_CLIQUE)
    edges, scratch = pa.alloc_buffers(good)
    spare, spare_scratch = pa.alloc_buffers(good)   # set up, and the launch then refused

    def refuse():
        bad = pa.make_params(5000, 4, 0.5, seed=3, blocks=TOO_MANY)
        with pytest.raises(pa.CuppaError) as e:
            pa.generate_into(bad, spare, spare_scratch)
        assert e.value.status == pa.PA_ERR_CUDA
        assert pa.lib().pa_last_cuda_error() != 0

    refuse()
    pa.generate_into(good, edges, scratch)
    assert pa.finish(scratch).status == 0
    assert (edges.cpu().numpy() == want).all()
    refuse()
    assert int(pa.degrees(good, edges).sum()) == 2 * len(want)
    refuse()
    rowptr, _ = pa.build_csr(good, edges)
    assert int(rowptr[-1]) == 2 * len(want)
    refuse()
    edges.zero_()
    plan = pa.Plan(good, edges, scratch)
    plan.launch()
    assert pa.finish(scratch).status == 0
    assert (edges.cpu().numpy() == want).all()
    plan.close()
    # and a refused capture
    handle = ctypes.c_void_p()
    bad = pa.make_params(5000, 4, 0.5, seed=3, blocks=TOO_MANY)
    rc = pa.lib().pa_plan_create(ctypes.byref(bad), ctypes.c_void_p(spare.data_ptr()),
                                 ctypes.c_uint64(spare.numel() * spare.element_size()),
                                 ctypes.c_void_p(spare_scratch.data_ptr()),
                                 ctypes.c_uint64(spare_scratch.numel()),
                                 ctypes.byref(handle))
    assert rc == pa.PA_ERR_CUDA
    pa.generate_into(good, edges, scratch)
    assert pa.finish(scratch).status == 0
    assert torch.equal(edges.cpu(), torch.from_numpy(want).to(edges.dtype))
