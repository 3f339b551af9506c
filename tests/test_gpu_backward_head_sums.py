"""The heads' gradients (and, in BF16, dense_9's bias gradient) as sums over many
rows and several chunks (nerf/core/model.py:148-170, 374-387): rows that repeat
a few, against those few times their number."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,repeats", [("fp32", 3), ("fp32", 2000), ("fp32", 9000), ("bf16", 3),
                                               ("bf16", 8192), ("bf16", 34_000)])
def test_head_sums_over_many_rows(ng, cuda, precision, repeats):
    blob = ng.weights.glorot_blob(3)
    rng = np.random.default_rng(4)
    off = ng.weights.offsets()
    for name, (_, b, _, o) in off.items():
        blob[b:b + o] = rng.normal(scale=0.05, size=o) + (0.3 if name == "sigma" else 0.0)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision=precision)
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    x = torch.rand(32, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(32, 3, device="cuda", generator=g), dim=1)
    dr, ds = torch.randn(32, 3, device="cuda", generator=g), torch.randn(32, 1, device="cuda", generator=g)

    def grads(k):
        tape = mlp.forward_train(x.repeat(k, 1), d.repeat(k, 1), precision=precision)[2]
        out = torch.zeros(len(blob), device="cuda")
        mlp.backward(tape, dr.repeat(k, 1), ds.repeat(k, 1), out)
        return out

    got, want = grads(repeats), grads(1).double() * repeats
    mlp.check_device_errors()
    # A lane adds at most 2 rows of 2^20 / (2 * 152 * 8 * 2) rounds, 432 alike
    # terms, and a block its eight warps' sums: every addition may round the same
    # way, half a unit of the sum so far, (432 + 8) / 2 * 2^-24 = 1.3e-5 for a
    # chunk of 2^20 rows and (32 + 8) / 2 * 2^-24 = 1.2e-6 for one of 77,824; the
    # chunks (2 to 4) add 2^-24 each.
    bound = (1.2e-6 if precision == "fp32" or repeats < 3 else 1.3e-5) + 4 * 2.0**-24
    parts = [off["rgb"][:2], (off["rgb"][1], off["rgb"][1] + 3), off["sigma"][:2],
             (off["sigma"][1], off["sigma"][1] + 1)]
    if precision == "bf16":
        parts.append((off["dense_9"][1], off["dense_9"][1] + 128))
    for lo, hi in parts:
        err = float((got[lo:hi].double() - want[lo:hi]).norm() / want[lo:hi].norm())
        print(precision, repeats, lo, f"{err:.2e}")
        assert err < bound, (lo, hi, err)
