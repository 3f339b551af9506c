"""The failure path of the backward's tensor-core kernels (csrc/gemm_fp32_tc.cu,
mlp_bwd_tc.cu, gemm_tc.cu): every wait is bounded; when one runs out the kernel
reports NERFGB_E_TIMEOUT in the error word and returns, the FP32 gradient is NaN
throughout, and the context stays usable. A diagnostic entry point shortens the
limit and leaves a copy or an arrival out, so that a wait runs out; the reference
has no counterpart (it surfaces TensorFlow's errors)."""
import ctypes
import time

import pytest
import torch

pytestmark = pytest.mark.gpu
N = 20_000  # one to two 256-row tiles and ~50 64-row stages per CTA pair


@pytest.fixture(scope="module", params=["fp32", "bf16"])
def case(request, ng, cuda):
    precision = request.param
    mlp = ng.get_coarse_or_fine_model("fine", seed=4, precision=precision)
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    x = torch.rand(N, 3, device="cuda", generator=g) * 4 - 2
    d = torch.nn.functional.normalize(torch.randn(N, 3, device="cuda", generator=g), dim=1)
    tape = mlp.forward_train(x, d, precision=precision)[2]
    dr, ds = torch.randn(N, 3, device="cuda", generator=g), torch.randn(N, device="cuda", generator=g)
    want = mlp.backward(tape, dr, ds, torch.zeros(ng.weights.PARAM_COUNT, device="cuda"))
    mlp.check_device_errors()
    return precision, mlp, tape, dr, ds, want


def _run(ng, case, wait_ns, withhold, n=N):
    precision, mlp, tape, dr, ds, want = case
    lib = ng._lib.lib()
    size = lib.nerfgb_mlp_backward_workspace_bytes if precision == "fp32" else \
        lib.nerfgb_mlp_backward_bf16_workspace_bytes
    ws = torch.empty(int(size(N)), dtype=torch.uint8, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    grad = torch.zeros_like(want)
    t0 = time.perf_counter()
    rc = lib.nerfgb_mlp_backward_wait_test(mlp.packed("fp32").data_ptr(), ng.model.PRECISIONS[precision],
                                           tape.data_ptr(), n, dr.data_ptr(), ds.data_ptr(), grad.data_ptr(),
                                           ws.data_ptr(), err.data_ptr(), ctypes.c_ulonglong(wait_ns), withhold,
                                           torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    return rc, int(err.item()), grad, time.perf_counter() - t0


def _close(a, b):
    # the same products, added in another order: FP32 sums of up to 20,000 terms
    return float((a - b).norm() / b.norm()) < 1e-5


def test_short_limit_alone(ng, case):
    rc, code, grad, _ = _run(ng, case, 10_000_000, 0)
    assert rc == ng._lib.OK and code == 0 and _close(grad, case[5])


@pytest.mark.parametrize("withhold", [1, 2])
def test_wait_runs_out_and_the_next_call_is_clean(ng, case, withhold):
    precision, mlp, tape, dr, ds, want = case
    rc, code, grad, secs = _run(ng, case, 2_000_000, withhold)
    assert rc == ng._lib.OK and secs < 5.0
    assert code == ng._lib.E_TIMEOUT, ng._lib.status_name(code)
    if precision == "fp32":
        assert bool(torch.isnan(grad).all())
    for _ in range(2):
        again = mlp.backward(tape, dr, ds, torch.zeros_like(want))
        mlp.check_device_errors()
        assert _close(again, want)


def test_the_model_reports(ng, cuda):
    """NerfMLP.backward's error word is the one check_device_errors reads, in
    either precision (the entry points take it)."""
    lib = ng._lib.lib()
    assert lib.nerfgb_mlp_backward_checked(None, None, 5, None, None, None, None, None, None) == ng._lib.E_INVALID_ARG
    assert lib.nerfgb_mlp_backward_checked(None, None, 0, None, None, None, None, None, None) == ng._lib.OK
    mlp = ng.get_coarse_or_fine_model("fine", seed=4)
    mlp.err_word.fill_(ng._lib.E_TIMEOUT)
    with pytest.raises(ng.NerfgbError):
        mlp.check_device_errors()
    mlp.check_device_errors()


def test_bad_arguments(ng, case):
    for wait_ns, withhold in ((10, 0), (10**11, 0), (10**7, 3), (10**7, -1)):
        assert _run(ng, case, wait_ns, withhold)[0] == ng._lib.E_INVALID_ARG
