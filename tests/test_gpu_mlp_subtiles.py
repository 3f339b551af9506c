"""The tensor-core MLP's deal of 256-row sub-tiles (128 rows per CTA of a
pair): row counts around a sub-tile, a whole tile of two and the point from
which pairs take more than one. Each row's outputs depend on that row alone,
so a count's outputs are the first rows of a larger count's, bit for bit; the
small counts are also held to the oracle's emulation of the BF16 and FP8
arithmetic (nerf/core/model.py:334-394)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F32 = np.float32


def _points(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-2, 2, (n, 3)).astype(F32)
    d = rng.normal(size=(n, 3))
    return x, (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F32)


@pytest.mark.parametrize("precision", ["bf16", "fp8"])
def test_counts_around_the_subtiles(ng, oracle, cuda, precision):
    pairs = torch.cuda.get_device_properties(0).multi_processor_count // 2
    full = 2 * 256 * pairs + 700
    x, d = _points(full, 31)
    X, D = torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda()
    blob = ng.weights.glorot_blob(8)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision=precision)
    rgb, sig = mlp((X, D))
    mlp.check_device_errors()
    counts = [1, 127, 128, 129, 255, 256, 257, 511, 512, 513, 256 * pairs - 1, 256 * pairs, 256 * pairs + 1,
              512 * pairs, 512 * pairs + 257]
    for n in counts:
        r, s = mlp((X[:n], D[:n]))
        mlp.check_device_errors()
        assert torch.equal(r, rgb[:n]) and torch.equal(s, sig[:n]), n
        # through a device-side count, fewer rows than the launch was made for
        rows = torch.arange(full, dtype=torch.int32, device="cuda")
        cnt = torch.tensor([n], dtype=torch.int32, device="cuda")
        r2, s2 = torch.full_like(rgb, -1.0), torch.full_like(sig, -1.0)
        ng._lib.call("nerfgb_mlp_forward_mapped", mlp.packed().data_ptr(), ng.model.PRECISIONS[precision],
                     X.data_ptr(), D.data_ptr(), full, 1, rows.data_ptr(), cnt.data_ptr(), r2.data_ptr(),
                     s2.data_ptr(), mlp.err_word.data_ptr(), torch.cuda.current_stream().cuda_stream)
        mlp.check_device_errors()
        assert torch.equal(r2[:n], rgb[:n]) and torch.equal(s2[:n], sig[:n]), n
        assert bool((r2[n:] == -1.0).all()) and bool((s2[n:] == -1.0).all()), n
        if precision == "bf16" and n <= 20_000:
            r3, s3, _ = mlp.forward_train(X[:n], D[:n], precision="bf16")
            mlp.check_device_errors()
            assert torch.equal(r3, r) and torch.equal(s3, s), n
    # the emulation rounds the same operands; what is left is the FP32
    # summation order, and an activation within that of a rounding boundary
    # (one BF16 step 2^-8, one E4M3 step 2^-3 relative): the bounds of
    # test_mlp_lowp_vs_emulation
    want_rgb, want_sig = oracle.mlp_forward_lowp(oracle.unpack_params(blob, F32), x[:600], d[:600], precision)
    tol = {"bf16": 2e-3, "fp8": 3e-2}[precision]
    assert np.abs(rgb[:600].cpu().numpy() - want_rgb).max() < tol
    assert np.abs(sig[:600].cpu().numpy() - want_sig).max() < tol * max(1.0, float(np.abs(want_sig).max()))


def test_fp8_relu_of_not_a_number(ng, cuda):
    """ReLU on packed E4M3 words is max(x, 0) of the FP32 value, NaN included
    (fmaxf(NaN, 0) = 0): rows with a NaN coordinate give what a zero dense_0
    and dense_5 give, finite and the same for each such row of one direction,
    and leave the other rows alone."""
    x, d = _points(600, 32)
    X, D = torch.from_numpy(x).cuda(), torch.from_numpy(np.repeat(d[:1], 600, 0)).cuda()
    mlp = ng.get_coarse_or_fine_model("fine", params=ng.weights.glorot_blob(8), precision="fp8")
    rgb, sig = mlp((X, D))
    bad = torch.tensor([0, 3, 127, 128, 300, 599], device="cuda")
    Y = X.clone()
    Y[bad, torch.arange(6, device="cuda") % 3] = float("nan")
    r, s = mlp((Y, D))
    mlp.check_device_errors()
    keep = torch.ones(600, dtype=torch.bool, device="cuda")
    keep[bad] = False
    assert torch.equal(r[keep], rgb[keep]) and torch.equal(s[keep], sig[keep])
    assert bool(torch.isfinite(r[bad]).all()) and bool(torch.isfinite(s[bad]).all())
    assert bool((r[bad] == r[bad[0]]).all()) and bool((s[bad] == s[bad[0]]).all())
