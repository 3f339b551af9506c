"""The FP32 backward of a single row (nerf/core/model.py:148-170): a Dense
layer's kernel gradient is then one product per weight, input times dZ, and dZ
is the layer's bias gradient, so that the rounding of a product can be seen by
itself, without the longer sums of other tests over it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 200])  # 200: all but one without a gradient
def test_products_are_rounded_to_nearest(ng, cuda, rows):
    blob = ng.weights.glorot_blob(3)
    rng = np.random.default_rng(4)
    off = ng.weights.offsets()
    for name, (_, b, _, o) in off.items():
        blob[b:b + o] = rng.normal(scale=0.05, size=o) + (0.3 if name == "sigma" else 0.0)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="fp32")
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    x = torch.rand(rows, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(rows, 3, device="cuda", generator=g), dim=1)
    acts = mlp.forward_train(x, d)[2]
    dr, ds = torch.zeros(rows, 3, device="cuda"), torch.zeros(rows, 1, device="cuda")
    live = rows // 2
    dr[live], ds[live] = torch.tensor([0.7, -1.3, 0.4], device="cuda"), 0.9
    got = torch.zeros(len(blob), device="cuda")
    mlp.backward(acts, dr, ds, got)
    a = acts[live].double()
    h = [a[64 + 256 * k:64 + 256 * (k + 1)] for k in range(9)]
    enc_xyz, enc_dir = a[:63], a[2368:2395]
    for k in range(10):
        inp = {0: enc_xyz, 5: torch.cat([h[4], enc_xyz]), 9: torch.cat([h[8], enc_dir])}.get(k, h[max(k - 1, 0)])
        w, b, i, o = off[f"dense_{k}"]
        want = torch.outer(inp, got[b:b + o].double())
        some = want != 0
        assert int(some.sum()) > 3000 and bool((got[w:w + i * o].reshape(i, o)[~some] == 0).all()), k
        e = (got[w:w + i * o].reshape(i, o).double() - want)[some] / want[some]
        # a product rounded to nearest is off by half a unit at most: RMS 2^-24
        # sqrt(E[1 / m^2] / 3) = 2.53e-8 for significands m spread evenly over
        # their logarithm, no mean; what the split leaves out (two products of
        # 2^-9.5 by 2^-18.5) adds 5e-9 to the RMS. (Cut off instead of rounded:
        # RMS 5e-8, mean -4.3e-8.)
        rms, mean = float(e.square().mean().sqrt()), float(e.mean())
        assert rms < 2.9e-8 and abs(mean) < 3e-9, (k, rms, mean)
