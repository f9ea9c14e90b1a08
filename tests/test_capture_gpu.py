"""Steps and orthogonalisations captured into CUDA graphs: a replay computes what the call computes, on the inputs that
lie in the buffers when it runs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
NS = (3.4445, -4.7750, 2.0315)


@pytest.mark.parametrize("nbytes", [16, 3984, 4000, 4016, 64 * 4000, 64 * 4000 + 16])
@pytest.mark.parametrize("captured", [False, True])
def test_upload(cuda_device, nbytes, captured):
    """Both ways of an upload, and a host buffer that changes as soon as the call returns."""
    from gefen_b200 import _lib

    host = np.random.default_rng(nbytes).integers(0, 256, nbytes, dtype=np.uint8)
    want = torch.from_numpy(host.copy())
    dst = torch.zeros(nbytes + 16, dtype=torch.uint8, device=cuda_device)

    def upload():
        _lib.check(_lib.load().gefen_b200_upload(_lib.ptr(dst), host.ctypes.data, nbytes, _lib.current_stream(cuda_device)))

    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                upload()
            host[:] = 0
            graph.replay()
        else:
            upload()
            host[:] = 0
    stream.synchronize()
    assert torch.equal(dst[:nbytes].cpu(), want) and not bool(dst[nbytes:].any())


def test_captured_orthogonalisation(cuda_device):
    from gefen_b200 import newton_schulz as ns

    shapes = [(64, 200), (300, 96), (33, 50)]
    gen = torch.Generator(device=cuda_device).manual_seed(0)
    inputs = [torch.randn(s, generator=gen, device=cuda_device) for s in shapes]
    for x in inputs:
        ns.zeropower_via_newtonschulz(x, NS, 5, 1e-7)   # (kernels loaded, status word allocated)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = [ns.zeropower_via_newtonschulz(x, NS, 5, 1e-7) for x in inputs]
    for _ in range(2):
        for x in inputs:
            x.copy_(torch.randn(x.shape, generator=gen, device=cuda_device))
        graph.replay()
        for x, got in zip(inputs, out):
            assert torch.equal(got, ns.zeropower_via_newtonschulz(x, NS, 5, 1e-7))
    ns.check_status(cuda_device)


@pytest.mark.parametrize("kind,count", [("gefen", 3), ("gefen", 30), ("muon", 4), ("muon", 30)])
def test_captured_step(cuda_device, kind, count):
    """Two eager steps, then a third one: from a graph on one side, called on the other. 30 tensors: more than the
    kernel parameters hold."""
    from gefen_b200 import Gefen, GefenMuon

    shapes = [(96 + 8 * (i % 5), 64 + 4 * (i % 3)) for i in range(count)]
    gen = torch.Generator(device=cuda_device).manual_seed(1)
    start = [torch.randn(s, generator=gen, device=cuda_device) * 0.02 for s in shapes]
    scale = [torch.exp(torch.randn(s[0], 1, generator=gen, device=cuda_device)) for s in shapes]
    grads = [[torch.randn(s, generator=gen, device=cuda_device) * 1e-3 * f for s, f in zip(shapes, scale)] for _ in range(3)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    sides = []
    with torch.cuda.stream(stream):
        for captured in (False, True):
            params = [torch.nn.Parameter(p.bfloat16()) for p in start]
            opt = Gefen(params, lr=1e-3, weight_decay=0.1) if kind == "gefen" else GefenMuon(params, lr=1e-2, weight_decay=0.1)
            for p in params:
                p.grad = torch.zeros_like(p)
            for step, of_step in enumerate(grads):
                for p, g in zip(params, of_step):
                    p.grad.copy_(g)
                if captured and step == 2:
                    graph = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(graph, stream=stream):
                        opt.step()
                    graph.replay()
                else:
                    opt.step()
            stream.synchronize()
            opt.check()
            sides.append([p.detach().clone() for p in params] +
                         [opt.state[p][key].clone() for p in params for key in ("m_codebook", "m_magnitude")])
    for a, b in zip(*sides):
        assert torch.equal(a, b)
