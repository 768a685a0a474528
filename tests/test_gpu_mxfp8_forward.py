"""GPU: the MXFP8 forward without a backward (quantising SwiGLU epilogue, no pad rows) against the training forward."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one token, experts without rows, 32-row blocks with and without live rows, more than one row tile an expert; d_model 128 takes
# the single-CTA kernel for the down product
@pytest.mark.parametrize("T,H,I,E,k", [(1, 128, 128, 8, 1), (33, 256, 384, 16, 2), (64, 512, 256, 8, 2), (2000, 256, 128, 8, 2)])
def test_mxfp8_forward_without_gradient_equals_the_training_forward(pkg, T, H, I, E, k):
    torch.manual_seed(T)
    layer = pkg.MoELayer(H, I, E, top_k=k, precision="mxfp8").to(DEV).to(torch.bfloat16)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    torch.empty(64 << 20, dtype=torch.uint8, device=DEV).fill_(255)      # pad rows that nobody writes hold NaN codes and scales
    with torch.no_grad():
        quiet = layer(x)
    trained = layer(x)          # quantises the weights both ways after the row-wise copies were kept
    with torch.no_grad():
        again = layer(x)
    pkg.check_status()
    assert torch.isfinite(quiet).all()
    assert torch.equal(quiet, trained.detach()) and torch.equal(again, quiet)
    trained.float().sum().backward()
    assert torch.isfinite(layer.gate_up_proj.grad).all()


def test_forward_without_gradient_keeps_only_the_row_wise_copies(pkg):
    """Trainable parameters and a trainable input under no_grad: no transposed copy is made or kept; the next training
    forward adds them."""
    from importlib import import_module
    mx = import_module(pkg.__name__ + ".mxfp8")
    layer = pkg.MoELayer(256, 128, 8, top_k=2, precision="mxfp8").to(DEV).to(torch.bfloat16)
    x = torch.randn(40, 256, device=DEV).to(torch.bfloat16).requires_grad_()
    kept = lambda: [len(mx._QUANTISED[id(p)][4]) for p in (layer.gate_up_proj, layer.down_proj)]     # noqa: E731
    with torch.no_grad():
        quiet = layer(x)
    assert kept() == [2, 2]
    trained = layer(x)
    assert kept() == [4, 4] and torch.equal(quiet, trained.detach())
    trained.float().sum().backward()
    with torch.no_grad():
        assert torch.equal(layer(x), quiet)
    pkg.check_status()


def test_kept_copies_are_complete_on_another_stream(pkg):
    """Copies that a busy stream has only queued, read at once by a call on another stream; then freed while that call runs."""
    g = torch.Generator().manual_seed(8)
    idx = torch.stack([torch.randperm(8, generator=g)[:2] for _ in range(64)]).to(DEV)
    x = torch.randn(64, 256, generator=g).to(torch.bfloat16).to(DEV)
    w, codes = torch.rand(64, 2, generator=g).to(DEV), torch.zeros(8, dtype=torch.int32, device=DEV)
    dn = (torch.randn(8, 256, 512, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    side = torch.cuda.Stream()
    for fn, dtype in ((pkg.moe_mxfp8, torch.bfloat16), (pkg.moe, torch.float32)):
        gu = (torch.randn(8, 1024, 256, generator=g) * 0.1).to(dtype).to(DEV)
        args = lambda: (x.to(dtype), idx, w, gu, dn.to(dtype), codes)     # noqa: E731
        with torch.no_grad():
            want = fn(*args())
            for maker in (torch.cuda.current_stream(), torch.cuda.Stream()) * 2:
                a = args()
                torch.cuda.synchronize()
                with torch.cuda.stream(maker):
                    gu.mul_(1.0)                       # another version: new copies, of the same values
                    torch.cuda._sleep(20_000_000)      # the stream is busy for about 10 ms
                    fn(*a)
                with torch.cuda.stream(side):
                    got = fn(*a)
                with torch.cuda.stream(maker):
                    gu.mul_(1.0)
                    fn(*a)                             # the old copies go; new ones are written on the same stream
                torch.cuda.synchronize()
                assert torch.equal(got, want)
    pkg.check_status()


def test_captured_passes_use_the_weights_of_the_replay(pkg):
    """Training passes captured after eager ones (whose copies are kept): replays after an update of the weights give what an eager
    pass on the new weights gives.  A forward captured on new weights leaves eager calls before its first replay right."""
    torch.manual_seed(4)
    layer = pkg.MoELayer(256, 128, 8, top_k=2, precision="mxfp8").to(DEV).to(torch.bfloat16)
    x = torch.randn(96, 256, device=DEV).to(torch.bfloat16).requires_grad_()
    params = [x, *layer.parameters()]

    def step():
        for p in params:
            p.grad = None
        out = layer(x)
        out.backward(out.detach())
        return [out.detach()] + [p.grad for p in params]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        res = step()
    for scale in (-1.5, 0.5):
        with torch.no_grad():
            for p in layer.parameters():
                p.mul_(scale)
        graph.replay()
        got = [t.clone() for t in res]
        assert all(torch.equal(a, b) for a, b in zip(got, step()))
    with torch.no_grad():
        layer.gate_up_proj.mul_(2.0)
        layer.down_proj.mul_(0.25)
        forward = torch.cuda.CUDAGraph()
        with torch.cuda.graph(forward):
            out = layer(x)
        eager = layer(x).clone()
        forward.replay()
        assert torch.equal(out, eager) and eager.abs().max() > 0
    pkg.check_status()
