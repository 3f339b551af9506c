"""The FP32 proposal kernels' 128-sample tiles (csrc/proposal.cu): counts
around a tile, and more tiles than CTAs, against the oracle's float64 network
and its gradient."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F32, F64 = np.float32, np.float64


@pytest.mark.parametrize("n", [1, 127, 128, 129, 300, 128 * 152 * 2 + 5])
def test_forward_and_backward_counts(ng, oracle, cuda, n):
    rng = np.random.default_rng(n)
    x = rng.uniform(-2, 2, (n, 3)).astype(F32)
    ds = rng.normal(size=n).astype(F32)
    blob = ng.proposal.glorot_blob(3)
    prop = ng.ProposalNetwork(params=blob)
    X, D = torch.from_numpy(x).cuda(), torch.from_numpy(ds).cuda()
    sigma = prop(X)
    g = prop.backward(X, D)
    # plain float64 restatement: 2x64 ReLU MLP on the L=6 encoding, softplus
    p = torch.from_numpy(blob).double().cuda().requires_grad_(True)
    W1, b1, W2, b2, W3, b3 = torch.split(p, [39 * 64, 64, 64 * 64, 64, 64, 1])
    # the angles as the float32 encoding has them (model.py:309-311), so that the ReLU masks agree
    m = torch.tensor([np.float32(2.0 ** l) * np.float32(np.pi) for l in range(6)], dtype=torch.float32, device="cuda")
    a = (X[:, :, None] * m).double()
    enc = torch.cat([X.double(), torch.stack([a.sin(), a.cos()], -1).reshape(n, -1)], 1)
    h = torch.relu(enc @ W1.reshape(39, 64) + b1)
    h = torch.relu(h @ W2.reshape(64, 64) + b2)
    want = torch.nn.functional.softplus(h @ W3 + b3)
    (want * D.double()).sum().backward()
    # FP32 sums of 39 and 64 products
    assert float((sigma[:, 0].double() - want.detach()).abs().max()) < 2e-5
    # a pre-activation within FP32 rounding of zero may take the other side of
    # its ReLU: a few of n * 128 units, each one term of a sum of n
    assert float((g.double() - p.grad).norm() / p.grad.norm()) < 2e-3
