"""The surrogate's reductions: bias gradients (column sums of a bf16 matrix, which
add one row after another in FP32 like numpy's accumulate) at the edges of their
batches of 32 rows, and the squared-error loss with its gradient against float64,
for odd sizes and unaligned bases.

The loss is FP64: n * 2^-53 of it. The gradient is one bf16 rounding of
scale * 2 d."""
import ctypes as C

import numpy as np
import pytest

import bellhopcuda_b200 as B

pytestmark = pytest.mark.gpu


def ptr(t):
    return C.c_void_p(t.data_ptr())


def stream():
    import torch
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


@pytest.mark.parametrize("M", [1, 31, 32, 33, 256, 4100])
@pytest.mark.parametrize("N,shift", [(1, 0), (8, 0), (63, 0), (64, 1), (66, 0), (512, 0)])
def test_colsum(M, N, shift):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N)
    dy = torch.randn(M * N + shift, device="cuda", generator=g).bfloat16()[shift:].view(M, N)
    db = torch.full((N + 1,), 7.0, device="cuda")
    assert B.load_library().bhcb_nn_colsum(ptr(dy), M, N, ptr(db), stream()) == 0
    ref = np.add.accumulate(dy.float().cpu().numpy(), axis=0)[-1]
    assert np.array_equal(db[:N].cpu().numpy(), ref) and db[N].item() == 7.0


@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (255, 1), (1024, 0), (1027, 0), (2097155, 0), (300000, 1)])
def test_mse(n, shift):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    p, t = (torch.randn(n + shift, device="cuda", generator=g)[shift:] for _ in range(2))
    grad = torch.zeros(n + 1, device="cuda", dtype=torch.bfloat16)
    loss = torch.full((1,), 0.25, device="cuda", dtype=torch.float64)
    assert B.load_library().bhcb_nn_mse(ptr(p), ptr(t), n, 0.37, ptr(grad), ptr(loss), stream()) == 0
    d = p - t
    ref = 0.25 + (d.double() ** 2).sum().item()
    assert abs(loss.item() - ref) <= n * 2.0 ** -53 * ref
    s = torch.tensor(0.37, device="cuda") * 2.0
    assert torch.equal(grad[:n], (s * d).bfloat16()) and grad[n].item() == 0.0
