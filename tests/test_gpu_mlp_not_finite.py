"""What the BF16 MLP gives for a row with a NaN coordinate
(nerf/core/model.py:334-394): every layer's activations are NaN up to the
heads, whose FP32 ReLU (fmaxf) takes NaN for 0, so that sigma and rgb are those
of the heads' biases; the tape keeps the NaN; the other rows are untouched."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 300, 77_000])  # a sub-tile alone, two, pairs of them
def test_nan_reaches_the_heads_in_bf16(ng, cuda, n):
    blob = ng.weights.glorot_blob(8)
    rng = np.random.default_rng(2)
    for name, (_, b, _, o) in ng.weights.offsets().items():
        blob[b:b + o] = rng.normal(scale=0.05, size=o) + (0.3 if name == "sigma" else 0.0)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="bf16")
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    x = torch.rand(n, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1)
    rgb, sig = mlp((x, d))
    bad = torch.tensor(sorted({0, n // 2, n - 1}), device="cuda")
    y = x.clone()
    y[bad, torch.arange(len(bad), device="cuda") % 3] = float("nan")
    r, s = mlp((y, d))
    rt, st, tape = mlp.forward_train(y, d, precision="bf16")
    mlp.check_device_errors()
    assert torch.equal(r, rt) and torch.equal(s, st)
    keep = torch.ones(n, dtype=torch.bool, device="cuda")
    keep[bad] = False
    assert torch.equal(r[keep], rgb[keep]) and torch.equal(s[keep], sig[keep])
    off = ng.weights.offsets()
    b_rgb, b_sig = (torch.from_numpy(blob[off[k][1]:off[k][1] + off[k][3]]).cuda() for k in ("rgb", "sigma"))
    # the sums are exactly 0: what is left is the sigmoid's own rounding (expf and a division)
    assert float((r[bad] - torch.sigmoid(b_rgb)).abs().max()) < 1e-6
    assert torch.equal(s[bad], torch.relu(b_sig).expand(len(bad), 1))
    acts = tape[bad].view(torch.bfloat16).float()
    assert bool(torch.isnan(acts[:, 64:64 + 9 * 256]).all()) and bool(torch.isnan(acts[:, 2400:]).all())
