"""The half kick and the drift in one launch round as the two launches do."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 5000])
def test_kick_drift_equals_kick_then_drift(n, dtype):
    from tsb import ops  # noqa: F401

    g = torch.Generator(device="cuda").manual_seed(n)
    q, p, f = (torch.randn(n, 3, generator=g, device="cuda", dtype=dtype) for _ in range(3))
    m = torch.rand(n, generator=g, device="cuda", dtype=dtype) + 0.5
    f[0, 1], p[-1, 2] = float("inf"), float("nan")
    idx = torch.arange(n, device="cuda") * 3 // n
    dt = torch.tensor([1e-3, 0.1, 7e-7], device="cuda", dtype=torch.float64)
    a, b = (q.clone(), p.clone()), (q.clone(), p.clone())
    torch.ops.tsb.md_kick_(a[1], f, idx, dt, 0.5)
    torch.ops.tsb.md_drift_(a[0], a[1], m, idx, dt, 1.0)
    torch.ops.tsb.md_kick_drift_(*b, f, m, idx, dt, 0.5, 1.0)
    for x, y in zip(a, b, strict=True):
        torch.testing.assert_close(x, y, rtol=0, atol=0, equal_nan=True)
