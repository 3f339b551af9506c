"""The FP32 MLP's tile sizes (64, 56, 48, 32 or 16 rows, chosen by the row
count): each row's outputs depend on that row alone, so a count's outputs are
the first rows of a larger count's, bit for bit, with and without the tape and
through a row map (nerf/core/model.py:334-394)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_every_tile_size_gives_the_same_rows(ng, oracle, cuda):
    sms = torch.cuda.get_device_properties(0).multi_processor_count

    def rows_of_tile(n):  # the rule
        def half_waves(tiles):
            rest = tiles % (2 * sms)
            return tiles // (2 * sms) * 2 + (0 if rest == 0 else 1 if tiles <= sms or rest <= sms // 2 else 2)

        return min((8, 7, 6, 4, 2), key=lambda r: half_waves(-(-n // (8 * r))) * (r + 3)) * 8

    counts = [1, 15, 16, 17, 1000, 16 * sms, 16 * sms + 1, 32 * sms - 5, 32 * sms + 1, 48 * sms, 48 * sms + 1,
              56 * sms - 1, 64 * sms, 64 * sms + 1, 112 * sms, 128 * sms, 140 * sms]
    assert {rows_of_tile(n) for n in counts} == {16, 32, 48, 56, 64}
    full = max(counts) + 777
    rng = np.random.default_rng(77)
    x = rng.uniform(-2, 2, (full, 3)).astype(np.float32)
    d = rng.normal(size=(full, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)
    X, D = torch.from_numpy(x).cuda(), torch.from_numpy(d).cuda()
    blob = ng.weights.glorot_blob(8)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="fp32")
    rgb, sig = mlp((X, D))
    for n in counts:
        r, s = mlp((X[:n], D[:n]))
        assert torch.equal(r, rgb[:n]) and torch.equal(s, sig[:n]), n
        perm = torch.randperm(n, device="cuda").int()
        r2, s2 = torch.full_like(rgb, -1.0), torch.full_like(sig, -1.0)
        ng._lib.call("nerfgb_mlp_forward_mapped", mlp.packed().data_ptr(), ng.model.PRECISIONS["fp32"], X.data_ptr(),
                     D.data_ptr(), n, 1, perm.data_ptr(), None, r2.data_ptr(), s2.data_ptr(), None,
                     torch.cuda.current_stream().cuda_stream)
        assert torch.equal(r2[:n], rgb[:n]) and torch.equal(s2[:n], sig[:n]), n
        assert bool((r2[n:] == -1.0).all()), n
        r3, s3, acts = mlp.forward_train(X[:n], D[:n])
        assert torch.equal(r3, r) and torch.equal(s3, s), n
        if n == counts[0]:
            first = acts[0].clone()
        assert torch.equal(acts[0], first), n
    # the bounds of test_mlp_fp32_vs_oracle
    want_rgb, want_sig = oracle.mlp_forward(oracle.unpack_params(blob, np.float32), x[:300], d[:300], np.float32)
    np.testing.assert_allclose(rgb[:300].cpu().numpy(), want_rgb, atol=2e-5, rtol=0)
    np.testing.assert_allclose(sig[:300].cpu().numpy(), want_sig, atol=1e-4, rtol=1e-4)
