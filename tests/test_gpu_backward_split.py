"""FP32 backward products on the tensor cores (an FP32 value as three BF16
values, six products, FP32 sums per 64 rows): gradients against the same
backward in 64-bit arithmetic from the same activation tape, at row counts
around a 64-row stage and where the stages split over the pairs
(nerf/core/model.py:148-170, 366-387)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(ng, n, seed):
    rng = np.random.default_rng(seed)
    blob = ng.weights.glorot_blob(3)
    for name, (w, b, i, o) in ng.weights.offsets().items():
        blob[b:b + o] = rng.normal(scale=0.05, size=o) + (0.3 if name == "sigma" else 0.0)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="fp32")
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    xyz = torch.rand(n, 3, device="cuda", generator=g) * 4 - 2
    dirs = torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1)
    acts = mlp.forward_train(xyz, dirs)[2]
    d_rgb = torch.randn(n, 3, device="cuda", generator=g)
    d_sigma = torch.randn(n, 1, device="cuda", generator=g)
    return blob, mlp, acts, d_rgb, d_sigma


def _gradient64(ng, blob, acts, d_rgb, d_sigma):
    p = ng.weights.offsets()
    w = {k: torch.from_numpy(blob[a:a + i * o].reshape(i, o)).cuda().double() for k, (a, _, i, o) in p.items()}
    bias = {k: torch.from_numpy(blob[b:b + o]).cuda().double() for k, (_, b, _, o) in p.items()}
    out = torch.zeros(len(blob), dtype=torch.float64, device="cuda")
    a = acts.double()
    h = [a[:, 64 + 256 * g:64 + 256 * (g + 1)] for g in range(9)] + [a[:, 2400:2528]]
    enc_xyz, enc_dir = a[:, :63], a[:, 2368:2395]

    def put(name, x, dz):
        k, b, i, o = p[name]
        out[k:k + i * o] += (x.T @ dz).reshape(-1)
        out[b:b + o] += dz.sum(0)

    s = torch.sigmoid(h[9] @ w["rgb"] + bias["rgb"])
    dz = d_rgb.double() * s * (1 - s)
    put("rgb", h[9], dz)
    ds = d_sigma.double() * ((h[7] @ w["sigma"] + bias["sigma"]) > 0)
    put("sigma", h[7], ds)
    dz = (dz @ w["rgb"].T) * (h[9] > 0)
    put("dense_9", torch.cat([h[8], enc_dir], 1), dz)
    dz = dz @ w["dense_9"][:256].T
    put("dense_8", h[7], dz)
    dz = (dz @ w["dense_8"].T + ds @ w["sigma"].T) * (h[7] > 0)
    for g in range(7, 0, -1):
        put(f"dense_{g}", h[g - 1] if g != 5 else torch.cat([h[4], enc_xyz], 1), dz)
        dz = (dz @ w[f"dense_{g}"][:256].T) * (h[g - 1] > 0)
    put("dense_0", enc_xyz, dz)
    return out


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 129, 257, 1000, 76 * 64 + 1, 20_000, 77_824 + 65])
def test_gradient_against_64_bits(ng, cuda, n):
    blob, mlp, acts, d_rgb, d_sigma = _case(ng, n, 40 + n % 13)
    got = torch.zeros(len(blob), device="cuda")
    mlp.backward(acts, d_rgb, d_sigma, got)
    want = _gradient64(ng, blob, acts, d_rgb, d_sigma)
    # a layer's dZ is a sum of 256 products rounded to 24 bits as it grows:
    # sqrt(256) 2^-25 = 4.8e-7 of its norm, 1.5e-6 over ten layers; the sum
    # over the rows adds as much again
    for name, (w, b, i, o) in ng.weights.offsets().items():
        for lo, hi in ((w, w + i * o), (b, b + o)):
            err, norm = (float(v.norm()) for v in (got[lo:hi].double() - want[lo:hi], want[lo:hi]))
            assert err <= 3e-6 * norm, (name, lo == b, err, norm)  # (a single row's sigma may be off: 0 <= 0)
    # accumulates: a second call adds the same again
    mlp.backward(acts, d_rgb, d_sigma, got)
    assert float((got.double() - 2 * want).norm() / want.norm()) < 6e-6


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_what_is_not_finite_stays_so(ng, cuda, bad):
    blob, mlp, acts, d_rgb, d_sigma = _case(ng, 300, 5)
    d_rgb[130, 1] = bad
    got = torch.zeros(len(blob), device="cuda")
    mlp.backward(acts, d_rgb, d_sigma, got)
    w, b, i, o = ng.weights.offsets()["dense_9"]
    live = acts[130, 2400:2528] > 0
    assert not bool(torch.isfinite(got[b:b + o][live]).any())
    assert bool(torch.isfinite(got[b:b + o][~live]).all())
