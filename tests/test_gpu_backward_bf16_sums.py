"""The BF16 backward's weight gradients as sums (nerf/core/model.py:148-170):
each row's dZ by itself from a backward of that row alone (a layer's bias
gradient is then its dZ, rounded to BF16 for the product), the sums of input
times dZ over the rows in 64 bits from those, against the gradient of all rows
at once."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _blob(ng):
    blob = ng.weights.glorot_blob(3)
    rng = np.random.default_rng(4)
    for name, (_, b, _, o) in ng.weights.offsets().items():
        blob[b:b + o] = rng.normal(scale=0.05, size=o) + (0.3 if name == "sigma" else 0.0)
    return blob


@pytest.mark.parametrize("one_sign", [False, True])
@pytest.mark.parametrize("n", [257, 1000, 3001])
def test_sums_over_few_rows(ng, cuda, n, one_sign):
    blob = _blob(ng)
    off = ng.weights.offsets()
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="bf16")
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.rand(n, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1)
    dr, ds = torch.randn(n, 3, device="cuda", generator=g), torch.randn(n, device="cuda", generator=g)
    if one_sign:
        dr, ds = dr.abs(), ds.abs()
    tape = mlp.forward_train(x, d, precision="bf16")[2]
    got = torch.zeros(len(blob), device="cuda")
    mlp.backward(tape, dr, ds, got)
    dz = [torch.empty(n, off[f"dense_{k}"][3], dtype=torch.float64, device="cuda") for k in range(10)]
    for r in range(n):
        one = torch.zeros(len(blob), device="cuda")
        mlp.backward(tape[r:r + 1], dr[r:r + 1], ds[r:r + 1], one)
        for k in range(10):
            _, b, _, o = off[f"dense_{k}"]
            dz[k][r] = one[b:b + o].bfloat16().double()
    mlp.check_device_errors()
    a = tape.view(torch.bfloat16).double()
    h = [a[:, 64 + 256 * k:64 + 256 * (k + 1)] for k in range(9)]
    for k in range(10):
        inp = {0: a[:, :63], 5: torch.cat([h[4], a[:, :63]], 1),
               9: torch.cat([h[8], a[:, 2368:2395]], 1)}.get(k, h[max(k - 1, 0)])
        w, _, i, o = off[f"dense_{k}"]
        want = inp.T @ dz[k]
        err = float((got[w:w + i * o].reshape(i, o).double() - want).norm() / want.norm())
        # An accumulator takes 64 rows in four steps and is cut off after each:
        # 0.36 2^-23 of it on average (significands spread evenly over their
        # logarithm), the four partial sums together 2.5 times the last: at most
        # 1.07e-7 if all cuts went one way (256 rows per accumulator: up to
        # 3.6e-7, 1.1e-7 - 1.9e-7 at 1,000 to 5,000 rows). The few additions of
        # the accumulators round off 2^-25 of the sum each.
        assert err < 1.07e-7, (k, err)


@pytest.mark.parametrize("repeats", [33, 8192, 24_576])
def test_bias_sums_over_many_rows(ng, cuda, repeats):
    blob = _blob(ng)
    off = ng.weights.offsets()
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="bf16")
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    x = torch.rand(32, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(32, 3, device="cuda", generator=g), dim=1)
    dr, ds = torch.randn(32, 3, device="cuda", generator=g), torch.randn(32, 1, device="cuda", generator=g)

    def grads(k):
        tape = mlp.forward_train(x.repeat(k, 1), d.repeat(k, 1), precision="bf16")[2]
        out = torch.zeros(len(blob), device="cuda")
        mlp.backward(tape, dr.repeat(k, 1), ds.repeat(k, 1), out)
        return out

    got, want = grads(repeats), grads(1).double() * repeats
    mlp.check_device_errors()
    # A CTA adds the sums of 32 rows (a warp's) one after another, at most 216 of
    # them here (2^20 rows over 152 CTAs); all terms alike, every addition may
    # round the same way, half a unit of the sum so far: 216 / 2 * 2^-24 = 6.4e-6
    # at the most. (Added to the gradient itself, 24,576 of them: 1.9e-4.)
    for k in range(9):
        _, b, _, o = off[f"dense_{k}"]
        err = float((got[b:b + o].double() - want[b:b + o]).norm() / want[b:b + o].norm())
        assert err < 6.4e-6, (k, err)
