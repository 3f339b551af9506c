"""Workloads of the render and training path, each through the entry points a
program calls.

A case's "kind" names the path:

* ``render``: ``NeRF.render``, the hierarchical coarse -> fine render of a
  batch of rays (a whole 800x800 frame, or the few pixels of a probe), plain
  or with the proposal network gating the samples.
* ``train``: one optimisation step's loss and gradients,
  ``autograd.render_with_grad`` + ``autograd.mse`` + ``backward()``.
* ``mlp``: one coarse or fine network on a batch of points.
* ``mlp_grad``: one network's training forward and its backward.
* ``rays``: the samplers and the compositor of one ray batch, op by op
  (``create_input_batch_coarse_model``, ``post_process_model_output``,
  ``create_input_batch_fine_model``).
* ``proposal``: the proposal network's forward and backward on a batch of
  points.

Inputs are synthetic and come from the seed alone: rays of a pinhole camera
or of random cameras on the radius-4 sphere (near 2, far 6), Glorot-initialised
networks with small biases, and for rendering a network whose density sits in
sparse blobs, as a trained scene's does.
"""
import importlib
import math

import numpy as np
import torch

ng = importlib.import_module("nerf-tf2_gb300")

NEAR, FAR = 2.0, 6.0
MLP_MACS = 593_408  # multiply-adds of one network on one sample
PROP_MACS = 39 * 64 + 64 * 64 + 64
PARAM_BYTES = 4 * ng.weights.PARAM_COUNT
LAYERS = ng.weights.LAYERS


def listed():
    return [
        # an 800x800 frame of the render loop: BF16 networks, a trained
        # proposal skipping the empty samples (the fastest way to a frame)
        {"name": "frame_gated_bf16", "kind": "render", "precision": "bf16", "mode": "gate", "rays": 640_000,
         "coarse": 64, "fine": 128},
        # a few pixels under the cursor of a viewer: latency, not throughput
        {"name": "probe_bf16", "kind": "render", "precision": "bf16", "mode": "plain", "rays": 61, "coarse": 64,
         "fine": 128},
        # the reference's training batch (4096 rays) on tensor cores
        {"name": "train_bf16", "kind": "train", "precision": "bf16", "rays": 4096, "coarse": 64, "fine": 128},
        # a smaller batch at the default precision
        {"name": "train_fp32", "kind": "train", "precision": "fp32", "rays": 1024, "coarse": 64, "fine": 128},
        # the fine pass of one 4096-ray render chunk, per tensor-core precision
        {"name": "mlp_bf16_fine", "kind": "mlp", "precision": "bf16", "rows": 786_432, "per_dir": 192},
        {"name": "mlp_fp8_fine", "kind": "mlp", "precision": "fp8", "rows": 786_432, "per_dir": 192},
        # a handful of points queried one by one
        {"name": "mlp_bf16_points", "kind": "mlp", "precision": "bf16", "rows": 1000, "per_dir": 1},
        # density and colour of a scattered point set at the default precision
        {"name": "mlp_fp32_points", "kind": "mlp", "precision": "fp32", "rows": 100_003, "per_dir": 1},
        # the coarse network's forward and backward in a 4096-ray step
        {"name": "mlp_grad_bf16", "kind": "mlp_grad", "precision": "bf16", "rows": 262_144, "per_dir": 64},
        # the same at the default precision on a ragged batch
        {"name": "mlp_grad_fp32", "kind": "mlp_grad", "precision": "fp32", "rows": 50_007, "per_dir": 1},
        # samplers and compositing of one chunk, as NeRF.forward calls them
        {"name": "rays_4096", "kind": "rays", "rays": 4096, "coarse": 64, "fine": 128},
        # the proposal's share of one of its training steps (4096 rays x 64)
        {"name": "proposal_262144", "kind": "proposal", "rows": 262_144},
    ]


def _size(rng, low, high):
    """Spread over the logarithm; rarely round."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["render", "render", "train", "mlp", "mlp", "mlp", "mlp_grad", "mlp_grad", "rays", "proposal"])
    if kind == "render":
        mode = rng.choice(["plain", "gate"])
        precision = rng.choice(["bf16", "bf16", "fp8", "fp32"])
        most = 8192 if precision == "fp32" else 300_000
        return {"kind": kind, "precision": precision, "mode": mode, "rays": _size(rng, 16, most),
                "coarse": rng.choice([32, 64, 64, 96]), "fine": rng.choice([64, 100, 128, 128])}
    if kind == "train":
        precision = rng.choice(["bf16", "bf16", "fp32"])
        return {"kind": kind, "precision": precision, "rays": _size(rng, 64, 1024 if precision == "fp32" else 4096),
                "coarse": rng.choice([32, 64, 64]), "fine": rng.choice([64, 128, 128])}
    if kind == "mlp":
        precision = rng.choice(["bf16", "bf16", "fp8", "fp32"])
        return {"kind": kind, "precision": precision,
                "rows": _size(rng, 100, 200_000 if precision == "fp32" else 786_432),
                "per_dir": rng.choice([1, 64, 192])}
    if kind == "mlp_grad":
        precision = rng.choice(["bf16", "bf16", "fp32"])
        return {"kind": kind, "precision": precision,
                "rows": _size(rng, 1000, 65_536 if precision == "fp32" else 400_000),
                "per_dir": rng.choice([1, 64, 192])}
    if kind == "rays":
        return {"kind": kind, "rays": _size(rng, 100, 16_384), "coarse": rng.choice([32, 48, 64, 64, 96]),
                "fine": rng.choice([64, 100, 128, 128, 192])}
    return {"kind": kind, "rows": _size(rng, 4096, 400_000)}


def _rng(case, seed):
    return np.random.default_rng([int(seed), sum(map(ord, case["kind"]))])


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()


def _random(rng):
    """A torch generator on the GPU, for the large inputs."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(rng.integers(1 << 31)))
    return g


def _points(rng, n, per_dir):
    """Points of the scene's box and unit directions, one per `per_dir`."""
    g = _random(rng)
    xyz = torch.rand(n, 3, generator=g, device="cuda") * 4 - 2
    d = torch.randn((n + per_dir - 1) // per_dir, 3, generator=g, device="cuda")
    return xyz, torch.nn.functional.normalize(d, dim=1)


def _blob(rng):
    """A network some way into training: Glorot kernels, small biases, and a
    density that is positive at most points (a random sigma head can be
    negative, and its gradient zero, everywhere)."""
    blob = ng.weights.glorot_blob(int(rng.integers(1 << 31)))
    for name, (_, bias, _, out) in ng.weights.offsets().items():
        blob[bias:bias + out] = rng.normal(scale=0.05, size=out) + (0.5 if name == "sigma" else 0.0)
    return blob


def _proposal_blob():
    """A proposal that has learned the extent of an object at the origin, by
    hand: density softplus(11.2 - 4 |x|_1) within |x|_1 < 2.3, falling to
    none by 2.4, from the six rectified coordinates and a step of two ramps."""
    W1, b1 = np.zeros((39, 64), np.float32), np.zeros(64, np.float32)
    W2, b2 = np.zeros((64, 64), np.float32), np.zeros(64, np.float32)
    W3, b3 = np.zeros(64, np.float32), np.full(1, -24.0, np.float32)
    for c in range(3):
        W1[c, 2 * c], W1[c, 2 * c + 1] = 1.0, -1.0
    W2[:6, 0] = W2[:6, 1] = -1.0
    b2[0], b2[1] = 2.4, 2.3
    W3[0], W3[1] = 260.0, -256.0
    return np.concatenate([a.reshape(-1) for a in (W1, b1, W2, b2, W3, b3)])


def _sphere_rays(rng, n):
    return [_dev(x) for x in ng.synthetic.sphere_rays(n, int(rng.integers(1 << 31)), near=NEAR, far=FAR)]


def prepare(case, seed):
    rng = _rng(case, seed)
    kind = case["kind"]
    s = {"case": case}
    if kind in ("render", "train", "rays"):
        R, Sc, Sf = case["rays"], case["coarse"], case["fine"]
        s["params"] = ng.make_params(N_coarse=Sc, N_fine=Sf)
        if kind == "render" and R == 640_000:
            s["rays"] = [_dev(x) for x in ng.synthetic.frame_rays(int(rng.integers(1 << 31)), 800, 800)]
        else:
            s["rays"] = _sphere_rays(rng, R)
    if kind == "render":
        scene = ng.synthetic.sparse_scene_blob(int(rng.integers(1 << 31)), max_freq_log2=5)
        s["nerf"] = ng.NeRF(s["params"], precision=case["precision"], coarse_params=scene, fine_params=scene)
        s["proposal"] = ng.ProposalNetwork(params=_proposal_blob()) if case["mode"] == "gate" else None
        s["draws"] = int(rng.integers(1 << 31))
        if R < 640_000:
            g = _random(rng)
            s["u"] = (torch.rand(R, Sc, generator=g, device="cuda"), torch.rand(R, Sf, generator=g, device="cuda"))
        else:
            s["u"] = (None, None)
    elif kind == "train":
        s["blobs"] = _blob(rng), _blob(rng)
        s["nerf"] = ng.NeRF(s["params"], precision=case["precision"], coarse_params=s["blobs"][0],
                            fine_params=s["blobs"][1])
        g = _random(rng)
        s["u"] = (torch.rand(R, Sc, generator=g, device="cuda"), torch.rand(R, Sf, generator=g, device="cuda"))
        s["target"] = 0.5 + 0.5 * torch.sin(3 * s["rays"][1] + torch.rand(3, generator=g, device="cuda"))
    elif kind in ("mlp", "mlp_grad"):
        s["blob"] = _blob(rng)
        s["model"] = ng.get_coarse_or_fine_model("fine", params=s["blob"], precision=case["precision"])
        s["xyz"], s["dirs"] = _points(rng, case["rows"], case["per_dir"])
        if kind == "mlp_grad":
            g = _random(rng)
            s["d_rgb"] = torch.randn(case["rows"], 3, generator=g, device="cuda") / case["rows"]
            s["d_sigma"] = torch.randn(case["rows"], generator=g, device="cuda") / case["rows"]
    elif kind == "rays":
        g = _random(rng)
        s["u"] = (torch.rand(R, Sc, generator=g, device="cuda"), torch.rand(R, Sf, generator=g, device="cuda"))
        # what a trained network gives: mostly empty space, some solid runs
        for k, S in (("c", Sc), ("f", Sc + Sf)):
            s["sigma_" + k] = torch.relu(6 * torch.randn(R * S, 1, generator=g, device="cuda") - 4)
            s["rgb_" + k] = torch.rand(R * S, 3, generator=g, device="cuda")
    else:
        s["blob"] = ng.proposal.glorot_blob(int(rng.integers(1 << 31)))
        s["proposal"] = ng.ProposalNetwork(params=s["blob"])
        s["xyz"], _ = _points(rng, case["rows"], 1)
        s["d_sigma"] = torch.randn(case["rows"], generator=_random(rng), device="cuda") / case["rows"]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "render":
        return s["nerf"].render(*s["rays"], u_coarse=s["u"][0], u_fine=s["u"][1], seed=s["draws"],
                                proposal=s["proposal"], proposal_mode="gate")
    if kind == "train":
        nerf = s["nerf"]
        nerf.coarse_model.params.grad = nerf.fine_model.params.grad = None
        rgb_c, rgb_f = ng.autograd.render_with_grad(nerf, *s["rays"], u_coarse=s["u"][0], u_fine=s["u"][1])
        loss = ng.autograd.mse(rgb_c, s["target"]) + ng.autograd.mse(rgb_f, s["target"])
        loss.backward()
        return {"loss": loss, "rgb_c": rgb_c, "rgb_f": rgb_f, "grad_c": nerf.coarse_model.params.grad,
                "grad_f": nerf.fine_model.params.grad}
    if kind == "mlp":
        return s["model"]((s["xyz"], s["dirs"]), rows_per_dir=case["per_dir"])
    if kind == "mlp_grad":
        rgb, sigma, tape = s["model"].forward_train(s["xyz"], s["dirs"], rows_per_dir=case["per_dir"],
                                                    precision=case["precision"])
        grad = torch.zeros(ng.weights.PARAM_COUNT, device="cuda")
        return rgb, sigma, s["model"].backward(tape, s["d_rgb"], s["d_sigma"], grad)
    if kind == "rays":
        p, (o, d, near, far) = s["params"], s["rays"]
        c = ng.create_input_batch_coarse_model(p, o, d, near, far, u_vals=s["u"][0])
        maps_c = ng.post_process_model_output(s["rgb_c"], s["sigma_c"], c["t_vals"])
        f = ng.create_input_batch_fine_model(p, o, d, maps_c["weights"], c["bin_data"], c["t_vals"],
                                             u_vals=s["u"][1])
        maps_f = ng.post_process_model_output(s["rgb_f"], s["sigma_f"], f["t_vals"], white_bg=True)
        return {"xyz_c": c["xyz_inputs"], "dir_c": c["dir_inputs"], "t_c": c["t_vals"], "maps_c": maps_c,
                "xyz_f": f["xyz_inputs"], "dir_f": f["dir_inputs"], "t_f": f["t_vals"], "maps_f": maps_f}
    sigma = s["proposal"](s["xyz"])
    return sigma, s["proposal"].backward(s["xyz"], s["d_sigma"])


def work(case):
    kind = case["kind"]
    if kind == "render":
        R, Sc, S = case["rays"], case["coarse"], case["coarse"] + case["fine"]
        rows, flops = R * (Sc + S), 0
        if case["mode"] == "gate":
            # about this share of the samples is left by the proposal
            rows, flops = int(0.42 * rows), 2 * PROP_MACS * R * Sc
        return {"bytes": R * (8 + 5) * 4 + 2 * PARAM_BYTES, "flops": flops + 2 * MLP_MACS * rows}
    if kind == "train":
        R, rows = case["rays"], case["rays"] * (2 * case["coarse"] + case["fine"])
        return {"bytes": R * (8 + 3 + 6 + case["coarse"] + case["fine"]) * 4 + 4 * PARAM_BYTES,
                "flops": 6 * MLP_MACS * rows}
    if kind in ("mlp", "mlp_grad"):
        n, nd = case["rows"], -(-case["rows"] // case["per_dir"])
        if kind == "mlp":
            return {"bytes": (7 * n + 3 * nd) * 4 + PARAM_BYTES, "flops": 2 * MLP_MACS * n}
        return {"bytes": (11 * n + 3 * nd) * 4 + 2 * PARAM_BYTES, "flops": 6 * MLP_MACS * n}
    if kind == "rays":
        R, Sc, S = case["rays"], case["coarse"], case["coarse"] + case["fine"]
        floats = R * (8 + Sc + case["fine"])             # rays, uniforms
        floats += R * (Sc + S) * (4 + 1 + 7) + 10 * R    # rgb and sigma in; weights, t, points, directions, maps out
        return {"bytes": 4 * floats, "flops": 40 * R * (Sc + S)}
    n = case["rows"]
    return {"bytes": 4 * (5 * n + 2 * ng.proposal.PARAM_COUNT), "flops": 2 * PROP_MACS * n * 4}


# --- 64 bits, in plain torch --------------------------------------------------

def _encode64(x, L):
    a = x[:, :, None] * (2.0 ** torch.arange(L, dtype=torch.float64, device=x.device) * math.pi)
    return torch.cat([x, torch.stack([torch.sin(a), torch.cos(a)], dim=-1).reshape(len(x), -1)], dim=1)


def _mlp64(params, xyz, dirs):
    """The network on float64 points; params: the flat blob."""
    w, at = {}, 0
    for name, i, o in LAYERS:
        w[name] = params[at:at + i * o].reshape(i, o), params[at + i * o:at + i * o + o]
        at += i * o + o

    def dense(name, h):
        return torch.addmm(w[name][1], h, w[name][0])

    e, h = _encode64(xyz, 10), None
    for k in range(8):
        h = torch.relu(dense("dense_%d" % k, e if k == 0 else torch.cat([h, e], 1) if k == 5 else h))
    sigma = torch.relu(dense("sigma", h))
    h = torch.cat([dense("dense_8", h), _encode64(dirs, 4)], 1)
    return torch.sigmoid(dense("rgb", torch.relu(dense("dense_9", h)))), sigma


def _coarse64(o, d, near, far, u):
    S = u.shape[1]
    i = torch.arange(S + 1, dtype=torch.float64, device=u.device)[None, :]
    edges = 1.0 / (1.0 / near + (1.0 / far - 1.0 / near) / S * i)
    width = edges[:, 1:] - edges[:, :-1]
    return edges, width, edges[:, :-1] + u * width


def _composite64(rgb, sigma, t, white=False):
    R, S = t.shape
    delta = torch.cat([t[:, 1:] - t[:, :-1], torch.full((R, 1), 1e10, dtype=torch.float64, device=t.device)], 1)
    alpha = 1 - torch.exp(-sigma.reshape(R, S) * delta)
    left = torch.cumprod((1 - alpha) + 1e-10, dim=1)
    w = alpha * torch.cat([torch.ones_like(left[:, :1]), left[:, :-1]], 1)
    acc = w.sum(1)
    m = (w[:, :, None] * rgb.reshape(R, S, 3)).sum(1)
    return {"acc_map": acc, "weights": w, "pred_rgb": m + (1 - acc)[:, None] if white else m,
            "pred_depth": (w * t).sum(1)}


def _fine64(weights, edges, width, t_c, u):
    w = weights + 1e-5
    pdf = w / (w * width).sum(1, keepdim=True)
    cdf = torch.cat([torch.zeros_like(t_c[:, :1]), torch.cumsum(pdf * width, 1)], 1)
    k = torch.searchsorted(cdf[:, 1:-1].contiguous(), u, right=True)
    p = pdf.gather(1, k)
    t = (u - cdf.gather(1, k)) / p.clamp(min=1e-8) * (p >= 1e-8) + edges[:, :-1].gather(1, k)
    return torch.sort(torch.cat([t_c, t], 1), dim=1).values


def _along(o, d, t):
    return (o[:, None] + t[:, :, None] * d[:, None]).reshape(-1, 3)


def _forward64(pc, pf, o, d, near, far, uc, uf):
    edges, width, t_c = _coarse64(o, d, near, far, uc)
    rgb, sigma = _mlp64(pc, _along(o, d, t_c), d.repeat_interleave(t_c.shape[1], 0))
    maps_c = _composite64(rgb, sigma, t_c)
    t_f = _fine64(maps_c["weights"].detach(), edges, width, t_c, uf)
    rgb, sigma = _mlp64(pf, _along(o, d, t_f), d.repeat_interleave(t_f.shape[1], 0))
    return maps_c, _composite64(rgb, sigma, t_f)


def _proposal64(params, xyz):
    W1, b1, W2, b2, W3, b3 = torch.split(params, [39 * 64, 64, 64 * 64, 64, 64, 1])
    h = torch.relu(torch.addmm(b1, _encode64(xyz, 6), W1.reshape(39, 64)))
    h = torch.relu(torch.addmm(b2, h, W2.reshape(64, 64)))
    return torch.nn.functional.softplus(h @ W3 + b3)[:, None]


def exact(case, seed):
    kind = case["kind"]
    if kind == "render" and (case["mode"] == "gate" or case["rays"] > 8192):
        return None  # which samples the gate skips has no value in 64 bits; a large render takes minutes
    s = prepare(case, seed)
    if kind == "rays":
        o, d, near, far = (x.double() for x in s["rays"])
        u = [x.double() for x in s["u"]]
        edges, width, t_c = _coarse64(o, d, near, far, u[0])
        maps_c = _composite64(s["rgb_c"].double(), s["sigma_c"].double(), t_c)
        t_f = _fine64(maps_c["weights"], edges, width, t_c, u[1])
        maps_f = _composite64(s["rgb_f"].double(), s["sigma_f"].double(), t_f, white=True)
        return {"xyz_c": _along(o, d, t_c), "dir_c": d.repeat_interleave(t_c.shape[1], 0), "t_c": t_c,
                "maps_c": maps_c, "xyz_f": _along(o, d, t_f), "dir_f": d.repeat_interleave(t_f.shape[1], 0),
                "t_f": t_f, "maps_f": maps_f}
    if kind == "proposal":
        p = torch.from_numpy(s["blob"]).double().cuda().requires_grad_(True)
        out = _proposal64(p, s["xyz"].double())
        (out[:, 0] * s["d_sigma"].double()).sum().backward()
        return out.detach(), p.grad
    if kind in ("mlp", "mlp_grad"):
        p = torch.from_numpy(s["blob"]).double().cuda().requires_grad_(kind == "mlp_grad")
        n, per, step = case["rows"], case["per_dir"], 32_768
        got = []
        for a in range(0, n, step):
            b = min(n, a + step)
            row = torch.arange(a, b, device="cuda") // per
            rgb, sigma = _mlp64(p, s["xyz"][a:b].double(), s["dirs"][row].double())
            if kind == "mlp_grad":
                ((rgb * s["d_rgb"][a:b]).sum() + (sigma[:, 0] * s["d_sigma"][a:b]).sum()).backward()
            got.append((rgb.detach(), sigma.detach()))
        out = tuple(torch.cat(x) for x in zip(*got))
        return out + (p.grad,) if kind == "mlp_grad" else out
    R, step = case["rays"], 256
    models = s["nerf"].coarse_model, s["nerf"].fine_model
    pc, pf = (m.params.detach().double().requires_grad_(kind == "train") for m in models)
    got = []
    for a in range(0, R, step):
        part = [x[a:a + step].double() for x in (*s["rays"], *s["u"])]
        maps_c, maps_f = _forward64(pc, pf, *part)
        if kind == "train":
            y = s["target"][a:a + step].double()
            ((maps_c["pred_rgb"] - y).square().sum() + (maps_f["pred_rgb"] - y).square().sum()).div(3 * R).backward()
        got.append((maps_c["pred_rgb"].detach(), *(maps_f[k].detach() for k in ("pred_rgb", "pred_depth", "acc_map"))))
    rgb_c, rgb_f, depth, acc = (torch.cat(x) for x in zip(*got))
    if kind == "render":
        return {"rgb": rgb_f, "depth": depth, "acc": acc}
    y = s["target"].double()
    return {"loss": (rgb_c - y).square().mean() + (rgb_f - y).square().mean(), "rgb_c": rgb_c, "rgb_f": rgb_f,
            "grad_c": pc.grad, "grad_f": pf.grad}
