"""The FP32 MLP backward's row tiles, slices and chunks (csrc/mlp_train.cu):
64-row tiles of the chain, 16-row stages of the weight gradient, 77,824-row
chunks. Against the oracle's float64 chain on the same tape (the gradient
tf.GradientTape takes at nerf/core/model.py:148-170) at small counts; a count
past one chunk against the rows by themselves."""
import numpy as np
import pytest
import torch

from test_gpu_backward import biased_blob, compare, dev, flat_grads, host

pytestmark = pytest.mark.gpu
F32, F64 = np.float32, np.float64
CHUNK = 4 * 2 * 152 * 64


def _inputs(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.uniform(-3, 3, (n, 3)).astype(F32)
    d = rng.normal(size=(n, 3))
    d = (d / np.linalg.norm(d, axis=1, keepdims=True)).astype(F32)
    return x, d, rng.normal(size=(n, 3)).astype(F32), rng.normal(size=(n,)).astype(F32)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 63, 64, 65, 257])
def test_small_counts_vs_oracle(ng, oracle, cuda, n):
    blob = biased_blob(ng, 21)
    x, d, dr, ds = _inputs(n, n)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob)
    _, _, acts = mlp.forward_train(dev(x), dev(d))
    g = torch.zeros(ng.weights.PARAM_COUNT, device="cuda")
    mlp.backward(acts, dev(dr), dev(ds), g)
    tape = oracle.acts_from_tape(acts.cpu().numpy().astype(F64))
    want = flat_grads(ng, oracle.mlp_backward_cached(oracle.unpack_params(blob, F64), tape, dr.astype(F64),
                                                     ds.astype(F64)))
    # FP32 sums of at most 320 products per layer, ten layers deep
    compare(ng, host(g), want, rel=1e-4, norm=True)


def test_rows_past_one_chunk(ng, cuda):
    n = CHUNK + 130
    x, d, dr, ds = (dev(a) for a in _inputs(n, 5))
    mlp = ng.get_coarse_or_fine_model("fine", params=biased_blob(ng, 22))
    _, _, acts = mlp.forward_train(x, d)
    # only the rows on both sides of the chunk's end carry a gradient
    lo = CHUNK - 70
    dr[:lo] = 0
    ds[:lo] = 0
    g = torch.zeros(ng.weights.PARAM_COUNT, device="cuda")
    mlp.backward(acts, dr, ds, g)
    w = torch.zeros_like(g)
    mlp.backward(acts[lo:].contiguous(), dr[lo:].contiguous(), ds[lo:].contiguous(), w)
    # the same FP32 products, summed in another grouping: 200 rows' terms
    assert float((g - w).norm() / w.norm()) < 1e-5


@pytest.mark.parametrize("n", [1, 63, 64, 65, 127, 128, 129, 255, 256, 257, 513])
def test_bf16_small_counts_vs_oracle(ng, oracle, cuda, n):
    """The BF16 chain's 256-row sub-tiles and the weight gradient's 64-row
    chunks (csrc/mlp_bwd_tc.cu, csrc/gemm_tc.cu)."""
    blob = biased_blob(ng, 23)
    x, d, dr, ds = _inputs(n, 100 + n)
    mlp = ng.get_coarse_or_fine_model("fine", params=blob, precision="bf16")
    _, _, acts = mlp.forward_train(dev(x), dev(d), precision="bf16")
    g = torch.zeros(ng.weights.PARAM_COUNT, device="cuda")
    mlp.backward(acts, dev(dr), dev(ds), g)
    mlp.check_device_errors()
    tape = oracle.acts_from_tape(acts.view(torch.bfloat16).float().cpu().numpy().astype(F64))
    want = flat_grads(ng, oracle.mlp_backward_cached(oracle.unpack_params(blob, F64), tape, dr.astype(F64),
                                                     ds.astype(F64)))
    # dZ and W rounded to BF16 for every product (2^-9 relative each), ten layers deep
    compare(ng, host(g), want, rel=3e-2, norm=True)


def test_bf16_rows_past_one_chunk(ng, cuda):
    chunk = 1 << 20
    n = chunk + 130
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.rand(n, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(n, 3, device="cuda", generator=g), dim=1)
    dr = torch.randn(n, 3, device="cuda", generator=g)
    ds = torch.randn(n, device="cuda", generator=g)
    mlp = ng.get_coarse_or_fine_model("fine", params=biased_blob(ng, 24), precision="bf16")
    _, _, acts = mlp.forward_train(x, d, precision="bf16")
    lo = chunk - 70  # only the rows on both sides of the chunk's end carry a gradient
    dr[:lo] = 0
    ds[:lo] = 0
    got = torch.zeros(ng.weights.PARAM_COUNT, device="cuda")
    mlp.backward(acts, dr, ds, got)
    want = torch.zeros_like(got)
    mlp.backward(acts[lo:].contiguous(), dr[lo:].contiguous(), ds[lo:].contiguous(), want)
    mlp.check_device_errors()
    # the same BF16 products, summed in FP32 in another grouping: 200 rows' terms
    assert float((got - want).norm() / want.norm()) < 1e-5
