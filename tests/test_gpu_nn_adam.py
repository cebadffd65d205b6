"""The optimiser's kernel with its bf16 copies, plain and transposed, and the transposed
weights of a layer.

The update is a dozen FP32 operations, each within 2^-24 of its result, of terms no
larger than the weight and lr (1 + wd |w|): 16 x 2^-24 of those bounds it. The copies are
bf16 roundings of the same value, so they are equal to the bit."""
import ctypes as C

import pytest

import bellhopcuda_b200 as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(1, 1), (33, 8), (128, 257)])
@pytest.mark.parametrize("wd", [0.0, 0.1])
def test_adam(rows, cols, wd):
    import torch
    g = torch.Generator(device="cuda").manual_seed(rows + cols)
    rnd = lambda: torch.randn(rows, cols, device="cuda", generator=g)
    w, gr, m, v = rnd(), rnd(), rnd(), rnd().abs()
    w0, m0, v0 = (t.double() for t in (w, m, v))
    wb = torch.empty((rows, cols), device="cuda", dtype=torch.bfloat16)
    wt = torch.empty((cols, rows), device="cuda", dtype=torch.bfloat16)
    p = lambda t: C.c_void_p(t.data_ptr())
    lr, b1, b2, eps, step = 1e-2, 0.9, 0.999, 1e-8, 3
    assert B.load_library().bhcb_nn_adam(p(w), p(gr), p(m), p(v), rows, cols, lr, b1, b2, eps, step, wd, p(wb), p(wt),
                                         C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    f = lambda x: float(torch.tensor(x, dtype=torch.float32))
    lr, b1, b2, eps, wd = map(f, (lr, b1, b2, eps, wd))
    d = gr.double()
    m1, v1 = b1 * m0 + (1 - b1) * d, b2 * v0 + (1 - b2) * d * d
    up = lr * (m1 / (1 - b1 ** step)) / ((v1 / (1 - b2 ** step)).sqrt() + eps)
    ref = w0 * (1 - lr * wd) - up
    terms = lr * (b1 * m0.abs() + (1 - b1) * d.abs()) / (1 - b1 ** step) / ((v1 / (1 - b2 ** step)).sqrt() + eps)
    # 1 - beta^step loses log2(1 / (1 - beta^step)) = 9 bits of FP32 to cancellation
    bound = 16 * 2.0 ** -24 * (w0.abs() + terms) + 2.0 ** -14 * terms
    assert bool(((w.double() - ref).abs() <= bound).all())
    assert torch.equal(wb, w.bfloat16()) and torch.equal(wt, w.bfloat16().T.contiguous())


def test_layer_transposed_weights():
    import torch
    from bellhopcuda_b200 import surrogate as S
    m = S.Surrogate(seed=2)
    for layer in m.branch.layers + m.trunk.layers:
        assert torch.equal(layer.wt, layer.w.bfloat16().T.contiguous())
