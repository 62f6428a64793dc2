"""Chains of kernels that start before their predecessor has finished: the same results as with every launch waited for."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 128, 1000, 4096])
@pytest.mark.parametrize("graph", [False, True])
def test_chain_over_two_buffers_keeps_its_order(rows, graph):
    """Every kernel reads what the one before wrote and overwrites what it read: a kernel that did not wait for its
    predecessor would see stale rows or destroy rows that are still being read."""
    import torch
    from splitrpc_b200 import ops

    torch.cuda.set_device(0)
    g = torch.Generator(device="cuda").manual_seed(rows)
    h = 768
    w = [(torch.randn(h, h, device="cuda", generator=g) / h ** 0.5).bfloat16() for _ in range(3)]
    gamma, beta = torch.ones(h, device="cuda"), torch.zeros(h, device="cuda")
    x0 = torch.randn(rows, h, device="cuda", generator=g).bfloat16()
    x, y = x0.clone(), torch.empty_like(x0)
    skinny = torch.empty(rows, 40, device="cuda")

    def chain(wait):
        def step(f, *a, **k):
            f(*a, **k)
            if wait:
                torch.cuda.synchronize()

        x.copy_(x0)
        for i in range(6):
            step(ops.gemm, x, w[i % 3], residual=x, act="gelu", out=y)
            step(ops.layernorm, y, gamma, beta, out=x)
            step(ops.gemm, x, w[(i + 1) % 3], out=y)
            step(ops.layernorm, y, gamma, beta, residual=x, out=x)
        step(ops.fc_skinny, x, w[0][:40], out=skinny)

    chain(True)
    want, want_s = x.clone(), skinny.clone()
    if graph:
        s = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s):
            chain(False)
        run = s.replay
    else:
        run = lambda: chain(False)
    for _ in range(5):
        x.zero_(), y.zero_(), skinny.zero_()
        run()
        torch.cuda.synchronize()
        ops.check_status()
        assert torch.equal(x, want) and torch.equal(skinny, want_s)
