"""The FP32 backward at counts around its tiles (csrc/gemm_fp32_tc.cu: 256-row
tiles of the dX chain, two at a time per CTA pair, 64-row stages of the weight
gradients): against the same backward in 64 bits from the same tape
(nerf/core/model.py:148-170, 366-387)."""
import pytest
import torch

from test_gpu_backward_split import _case, _gradient64

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 255, 256, 511, 512, 513, 76 * 256, 76 * 256 + 1, 2 * 76 * 256 + 257,
                               3 * 76 * 256 - 1])
def test_counts_around_the_tiles(ng, cuda, n):
    blob, mlp, acts, d_rgb, d_sigma = _case(ng, n, 60 + n % 11)
    got = torch.zeros(len(blob), device="cuda")
    mlp.backward(acts, d_rgb, d_sigma, got)
    mlp.check_device_errors()
    want = _gradient64(ng, blob, acts, d_rgb, d_sigma)
    # a product rounds off 2^-25, a layer's dZ is four sums of 64 of them added
    # with rounding (four to eight roundings, 2^-24 of its norm), ten layers
    # deep 2e-7, and the sums over the rows, of either sign, one addition per 64
    # rows and pair: 0.29 2^-23 sqrt(n / 64 / 2), 7e-7 for 58,000 rows. All of it
    # of what a sum of such terms comes to, which a layer's kernel does and its
    # bias (one number of the sigma head, three of the rgb head) need not: there of
    # the root of the sum of the terms' squares.
    w, b, i, o = ng.weights.offsets()["sigma"]
    ds = d_sigma.double().reshape(-1) * ((acts[:, 64 + 7 * 256:64 + 8 * 256].double()
                                          @ torch.from_numpy(blob[w:w + i]).cuda().double() + float(blob[b])) > 0)
    for name, (w, b, i, o) in ng.weights.offsets().items():
        for lo, hi in ((w, w + i * o), (b, b + o)):
            err, norm = (float(v.norm()) for v in (got[lo:hi].double() - want[lo:hi], want[lo:hi]))
            if name == "sigma" and lo == b:
                norm = float(ds.norm())
            elif name == "rgb" and lo == b:
                norm = max(norm, 0.05 * float(d_rgb.norm()))  # y (1 - y) is 0.25 at the most, above 0.05 for y in [.05, .95]
            assert err <= 1.2e-6 * norm, (name, lo == b, err / norm)
