"""Small launches may be set up while the kernel before them runs: a chain of
them on one stream, every input and output buffer reused by the next step, with
ordinary launches in between, gives what the same steps give one at a time, and
so does a captured graph of them (nerf/core/model.py:57-125)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _points(n, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000 + k)
    return (torch.rand(n, 3, device="cuda", generator=g) * 4 - 2,
            torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1))


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
@pytest.mark.parametrize("n", [61, 1000, 9000])
def test_chain_on_reused_buffers(ng, cuda, precision, n):
    mlp = ng.get_coarse_or_fine_model("fine", params=ng.weights.glorot_blob(8), precision=precision)
    steps = [_points(n, k) for k in range(12)]
    want = []
    for x, d in steps:
        rgb, sig = mlp((x, d))
        torch.cuda.synchronize()
        want.append((rgb.clone(), sig.clone()))
    X, D = torch.empty_like(steps[0][0]), torch.empty_like(steps[0][1])
    rgb, sig = torch.empty(n, 3, device="cuda"), torch.empty(n, 1, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def forward(x, d):
        ng._lib.call("nerfgb_mlp_forward", mlp.packed().data_ptr(), ng.model.PRECISIONS[precision], x.data_ptr(),
                     d.data_ptr(), n, 1, rgb.data_ptr(), sig.data_ptr(), mlp.err_word.data_ptr(), st)

    for rounds in range(3):
        got = []
        for k, (x, d) in enumerate(steps):
            if (k + rounds) % 2:  # an ordinary kernel writes the input
                X.copy_(x)
                D.copy_(d)
                forward(X, D)
            else:  # one small launch behind another
                forward(*steps[(k + 5) % 12])
                forward(x, d)
            got.append((rgb.clone(), sig.clone()))
        for (r, s), (wr, ws) in zip(got, want):
            assert torch.equal(r, wr) and torch.equal(s, ws)
    mlp.check_device_errors()


def test_small_render_repeated_and_captured(ng, cuda):
    params = ng.make_params()
    nerf = ng.NeRF(params, precision="bf16")
    rays = [torch.from_numpy(v).cuda() for v in ng.synthetic.sphere_rays(61, 3)]
    once = {k: v.clone() for k, v in nerf.render(*rays, seed=5).items() if torch.is_tensor(v)}
    torch.cuda.synchronize()
    for _ in range(20):
        out = nerf.render(*rays, seed=5)
    for k, v in once.items():
        assert torch.equal(out[k], v), k
    x, d = _points(700, 1)
    mlp = nerf.fine_model
    want = [v.clone() for v in mlp((x, d))]
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        mlp((x, d))
    torch.cuda.current_stream().wait_stream(side)
    with torch.cuda.graph(graph):
        a = mlp((x, d))
        b = mlp((x, d))
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for got in (a, b):
        assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
