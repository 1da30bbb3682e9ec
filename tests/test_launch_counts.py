"""pa_generate_launches and pa_csr_launches: the kernels of a call, counted by the library
that launches them; against the nodes of a captured generation on the GPU."""
import pytest

# n, d, p, further parameters, kernels of the generation
GEN = [
    (5, 4, 0.5, {}, 1),                                      # the seed graph alone: tile kernel
    (5, 4, 0.5, dict(layout=1), 0),
    (1000, 4, 0.5, {}, 2),                                   # set-up, start kernel
    (300, 40, 0.5, {}, 2),                                   # set-up, wide kernel
    (100_000, 4, 0.5, dict(start_nodes=1000), 2),            # start kernel, tile kernel
    (100_000, 4, 0.5, dict(start_nodes=2 ** 64 - 1), 1),     # PA_START_NONE: tile kernel
    (2 ** 22 + 41, 32, 0.45, dict(id_bits=64), 1 + 3),       # 2.1 GB: to 2^21, 2^22, the end
    (2 ** 22 + 41, 32, 0.39, dict(id_bits=64), 2),           # p outside the rule
    (2 ** 25 + 37, 4, 0.5, dict(id_bits=64), 1 + 6),         # to 2^21 .. 2^25, the end
]
BIG = [(2 ** 30, 4, 0.5, dict(id_bits=64), 1 + 10), (2 ** 31 + 2 ** 20, 4, 0.5, dict(id_bits=64), 2)]
CSR = [(100, 3, 6 - 1), (2 ** 9, 2, 5), (2 ** 16, 4, 6), (2 ** 18, 4, 6), (2 ** 18 + 1, 4, 7),
       (2 ** 27, 4, 7), (2 ** 27 + 1, 4, 8), (2 ** 30, 4, 8), (3000, 40, 6), (41, 40, 5)]


@pytest.mark.parametrize("n,d,p,kw,want", GEN + BIG)
def test_generate_launches(pa, n, d, p, kw, want):
    assert pa.generate_launches(pa.make_params(n, d, p, **kw)) == want


@pytest.mark.parametrize("n,d,want", CSR)
def test_csr_launches(pa, n, d, want):
    assert pa.csr_launches(pa.make_params(n, d, 0.5, id_bits=64)) == want


@pytest.mark.gpu
@pytest.mark.parametrize("n,d,p,kw,want", GEN[2:])
def test_captured_generation_has_that_many_kernels(pa, cuda_ok, n, d, p, kw, want):
    import torch
    from cuda.bindings import runtime as rt

    def ok(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1] if len(r) == 2 else r[1:]

    prm = pa.make_params(n, d, p, **kw)
    edges, scratch = pa.alloc_buffers(prm)
    stream = torch.cuda.Stream()
    ok(rt.cudaStreamBeginCapture(stream.cuda_stream,
                                 rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
    pa.generate_into(prm, edges, scratch, stream)
    graph = ok(rt.cudaStreamEndCapture(stream.cuda_stream))
    _, count = ok(rt.cudaGraphGetNodes(graph, 0))
    nodes, _ = ok(rt.cudaGraphGetNodes(graph, count))
    kinds = [ok(rt.cudaGraphNodeGetType(x)) for x in nodes]
    ok(rt.cudaGraphDestroy(graph))
    assert kinds.count(rt.cudaGraphNodeType.cudaGraphNodeTypeKernel) == want, kinds
