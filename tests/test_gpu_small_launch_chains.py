"""Small launches set up while the kernel before them runs (csrc/common.cuh,
after_previous), over changing inputs: a kernel that read its inputs too early
would find the step before's in the buffers that all steps share. The samplers,
the network and the compositor op by op (nerf/core/model.py:88-123), renders
plain and gated, and two streams of them at a time, against each step by itself
with the device idle before it."""
import pytest
import torch

pytestmark = pytest.mark.gpu
SC, SF, STEPS = 64, 128, 10


def _rays(ng, R, k):
    return [torch.from_numpy(v).cuda() for v in ng.synthetic.sphere_rays(R, 100 + k)]


def _draws(R, k):
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    return torch.rand(R, SC, device="cuda", generator=g), torch.rand(R, SF, device="cuda", generator=g)


class Ops:
    """NeRF.forward's chain over buffers that every step shares; the fine maps
    go to buffers of the step's own."""

    def __init__(self, ng, mlp, precision, R):
        f = lambda *s: torch.empty(*s, device="cuda")  # noqa: E731
        self.ng, self.mlp, self.prec, self.R = ng, mlp, ng.model.PRECISIONS[precision], R
        S = SC + SF
        self.b = {"xyz": f(R * S, 3), "dirs": f(R * S, 3), "t_c": f(R, SC), "edges": f(R, SC + 1), "width": f(R, SC),
                  "rgb": f(R * S, 3), "sigma": f(R * S, 1), "w": f(R, SC), "t_f": f(R, S), "w_f": f(R, S),
                  "map_rgb": f(R, 3), "map_d": f(R), "map_a": f(R)}
        self.packed = mlp.packed(precision)

    def __call__(self, rays, u, out):
        b, call, R = {k: v.data_ptr() for k, v in self.b.items()}, self.ng._lib.call, self.R
        o, d, near, far = (x.data_ptr() for x in rays)
        st = torch.cuda.current_stream().cuda_stream

        def network(S):
            call("nerfgb_mlp_forward", self.packed.data_ptr(), self.prec, b["xyz"], b["dirs"], R * S, 1, b["rgb"],
                 b["sigma"], self.mlp.err_word.data_ptr(), st)

        call("nerfgb_coarse_sample", o, d, near, far, u[0].data_ptr(), R, SC, 1, 0, b["xyz"], b["dirs"], b["t_c"],
             b["edges"], b["width"], st)
        network(SC)
        call("nerfgb_composite", b["rgb"], b["sigma"], b["t_c"], R, SC, 0, 1, b["w"], b["map_rgb"], b["map_d"],
             b["map_a"], st)
        call("nerfgb_fine_sample", o, d, b["w"], b["edges"], SC + 1, b["width"], b["t_c"], u[1].data_ptr(), R, SC, SF,
             b["xyz"], b["dirs"], b["t_f"], None, None, st)
        network(SC + SF)
        call("nerfgb_composite", b["rgb"], b["sigma"], b["t_f"], R, SC + SF, 1, 1, b["w_f"],
             *(v.data_ptr() for v in out), st)


def _maps(R):
    return [torch.full(s, -1.0, device="cuda") for s in ((R, 3), (R,), (R,))]


@pytest.mark.parametrize("precision", ["bf16", "fp8", "fp32"])
@pytest.mark.parametrize("R", [5, 61, 150])
def test_ops_chained_over_changing_inputs(ng, cuda, precision, R):
    mlp = ng.get_coarse_or_fine_model("fine", params=ng.synthetic.sparse_scene_blob(3), precision=precision)
    ops = Ops(ng, mlp, precision, R)
    steps = [(_rays(ng, R, k), _draws(R, k)) for k in range(STEPS)]
    want = []
    for rays, u in steps:
        torch.cuda.synchronize()
        out = _maps(R)
        torch.cuda.synchronize()
        ops(rays, u, out)
        torch.cuda.synchronize()
        want.append(out)
    assert any(not torch.equal(want[0][0], w[0]) for w in want[1:])
    for _ in range(5):
        got = [_maps(R) for _ in range(STEPS)]
        torch.cuda.synchronize()
        for (rays, u), out in zip(steps, got):
            ops(rays, u, out)  # nothing but the library's launches in between
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
    mlp.check_device_errors()


def _render(ng, nerf, rays, k, proposal):
    out = nerf.render(*rays, seed=k, proposal=proposal, proposal_mode="gate")
    return [out[m] for m in ("rgb", "depth", "acc")]


@pytest.mark.parametrize("precision", ["bf16", "fp8", "fp32"])
@pytest.mark.parametrize("gated", [False, True])
def test_renders_chained_over_changing_inputs(ng, cuda, precision, gated):
    scene = ng.synthetic.sparse_scene_blob(3)
    nerf = ng.NeRF(ng.make_params(), precision=precision, coarse_params=scene, fine_params=scene)
    proposal = ng.ProposalNetwork(seed=7) if gated else None
    for R in (7, 61):
        rays = [_rays(ng, R, k) for k in range(STEPS)]
        want = []
        for k in range(STEPS):
            torch.cuda.synchronize()
            want.append([v.clone() for v in _render(ng, nerf, rays[k], k, proposal)])
        for _ in range(4):
            torch.cuda.synchronize()
            got = [_render(ng, nerf, rays[k], k, proposal) for k in range(STEPS)]
            for a, b in zip(got, want):
                assert all(torch.equal(x, y) for x, y in zip(a, b))
    nerf.fine_model.check_device_errors()


@pytest.mark.parametrize("gated", [False, True])
def test_two_streams_of_small_renders(ng, cuda, gated):
    scene = ng.synthetic.sparse_scene_blob(3)
    nerf = ng.NeRF(ng.make_params(), precision="bf16", coarse_params=scene, fine_params=scene)
    proposal = ng.ProposalNetwork(seed=7) if gated else None
    rays = [_rays(ng, 40 + 11 * k, k) for k in range(STEPS)]
    want = []
    for k in range(STEPS):
        torch.cuda.synchronize()
        want.append([v.clone() for v in _render(ng, nerf, rays[k], k, proposal)])
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for rounds in range(4):
        got = []
        for k in range(STEPS):
            with torch.cuda.stream(streams[(k + rounds) % 2]):
                got.append(_render(ng, nerf, rays[k], k, proposal))
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert all(torch.equal(x, y) for x, y in zip(a, b))
    nerf.fine_model.check_device_errors()
