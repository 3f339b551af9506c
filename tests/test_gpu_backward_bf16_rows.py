"""The BF16 backward over many rows, all with a gradient (csrc/mlp_bwd_tc.cu,
gemm_tc.cu): pairs with one 256-row sub-tile and with two, several tiles and an
odd last one, the weight gradients' ring and its windows of 64, 128 and 256 rows.
Every layer's kernel and bias against the same chain in 64 bits from the same
tape with its BF16 roundings: W, each product's result and each dZ
(nerf/core/model.py:148-170, 366-387)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gradient(ng, blob, tape, d_rgb, d_sigma):
    off = ng.weights.offsets()
    w = {k: torch.from_numpy(blob[a:a + i * o].reshape(i, o)).cuda() for k, (a, _, i, o) in off.items()}
    bias = {k: torch.from_numpy(blob[b:b + o]).cuda().double() for k, (_, b, _, o) in off.items()}
    low = lambda x: x.bfloat16().double()  # noqa: E731
    out = torch.zeros(len(blob), dtype=torch.float64, device="cuda")

    def put(name, x, dz, z):
        k, b, i, o = off[name]
        out[k:k + i * o] += (x.T @ dz).reshape(-1)
        out[b:b + o] += z.sum(0)

    for r in range(0, len(tape), 32_768):
        a = tape[r:r + 32_768].view(torch.bfloat16).double()
        h = [a[:, 64 + 256 * g:64 + 256 * (g + 1)] for g in range(9)] + [a[:, 2400:2528]]
        enc_xyz, enc_dir = a[:, :63], a[:, 2368:2395]
        s = torch.sigmoid(h[9] @ w["rgb"].double() + bias["rgb"])
        dz = d_rgb[r:r + 32_768].double() * s * (1 - s)
        put("rgb", h[9], dz, dz)
        ds = d_sigma[r:r + 32_768, None].double() * ((h[7] @ w["sigma"].double() + bias["sigma"]) > 0)
        put("sigma", h[7], ds, ds)
        z = (dz @ w["rgb"].double().T) * (h[9] > 0)
        dz = low(z)
        put("dense_9", torch.cat([h[8], enc_dir], 1), dz, z)
        z = dz = low(dz @ low(w["dense_9"][:256]).T)
        put("dense_8", h[7], dz, z)
        z = (low(dz @ low(w["dense_8"]).T) + ds @ w["sigma"].double().T) * (h[7] > 0)
        dz = low(z)
        for g in range(7, 0, -1):
            put(f"dense_{g}", h[g - 1] if g != 5 else torch.cat([h[4], enc_xyz], 1), dz, z)
            z = dz = low(dz @ low(w[f"dense_{g}"][:256]).T) * (h[g - 1] > 0)
        put("dense_0", enc_xyz, dz, z)
    return out


@pytest.mark.parametrize("n", [255, 511, 20_000, 40_001, 100_003, 250_001])
def test_every_layer_over_many_rows(ng, cuda, n):
    blob = ng.weights.glorot_blob(3)
    rng = np.random.default_rng(4)
    off = ng.weights.offsets()
    for name, (_, b, _, o) in off.items():
        blob[b:b + o] = rng.normal(scale=0.05, size=o) + (0.3 if name == "sigma" else 0.0)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="bf16")
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.rand(n, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1)
    dr, ds = torch.randn(n, 3, device="cuda", generator=g), torch.randn(n, device="cuda", generator=g)
    tape = mlp.forward_train(x, d, precision="bf16")[2]
    got = torch.zeros(len(blob), device="cuda")
    mlp.backward(tape, dr, ds, got)
    mlp.check_device_errors()
    want = _gradient(ng, blob, tape, dr, ds)
    # What is left are sums that FP32 puts on the other side of a BF16 rounding
    # than 64 bits: an error of ~3e-7 of a sum against roundings 2^-8 apart, so
    # about one in 10^4, each 2^-8 of its value off, 4e-5 of a layer's norm and a
    # little more with every layer below; 256 rows taken from the wrong place
    # would be sqrt(256 / n) >= 3e-2 of it.
    for name, (k, b, i, o) in off.items():
        for lo, hi in ((k, k + i * o), (b, b + o)):
            err = float((got[lo:hi].double() - want[lo:hi]).norm() / want[lo:hi].norm())
            assert err < 1e-3, (name, lo == b, err)
