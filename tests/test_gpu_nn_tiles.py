"""Every epilogue of the surrogate's GEMM on both tile widths, at the edges of
tiles and of the rule between them (148 tiles of 128 x 32), with K blocks that
end early, widths and bases that rule out 16-byte accesses, against float64.

The accumulator adds K products, each addition within 2^-23 of the sum of their
magnitudes (it truncates): K 2^-23 |A| |B|^T. A bf16 result adds 2^-8 of itself,
tanhf and the products of the GELUs at most 1e-6; |gelu'| <= 1.13."""
import ctypes as C

import pytest

import bellhopcuda_b200 as B

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 8), (129, 33, 72), (128, 32, 128), (130, 160, 200), (512, 1184, 136), (512, 1185, 136), (77, 2400, 64)]


def gelu(x):
    import torch
    return 0.5 * x * (1.0 + torch.tanh(0.7978845608028654 * (x + 0.044715 * x ** 3)))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("epi", [0, 1, 2, 3])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_epilogues(M, N, K, epi, shift):
    """shift: C, bias and the auxiliary matrix start one element past an aligned base"""
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    A, Bm = rnd(M, K).bfloat16(), (rnd(N, K) / K ** 0.5).bfloat16()
    dt = torch.float32 if epi == 0 else torch.bfloat16
    out = torch.full((M * N + 2,), 5.0, device="cuda", dtype=dt)
    bias = rnd(N + 1)[shift:]
    aux = torch.full((M * N + 2,), 5.0, device="cuda", dtype=torch.bfloat16)
    if epi == 3:
        aux[shift:shift + M * N] = rnd(M * N).bfloat16()
    p = lambda t, n: C.c_void_p(t.data_ptr() + n * t.element_size())
    lib = B.load_library()
    assert lib.bhcb_nn_gemm(p(A, 0), p(Bm, 0), p(out, shift), M, N, K, epi, p(bias, 0) if epi < 3 else None,
                            p(aux, shift) if epi == 3 else None, p(aux, shift) if epi == 2 else None,
                            C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    err = C.c_int32()
    assert lib.bhcb_nn_status(C.byref(err), 1) == 0 and err.value == 0
    a, b = A.double(), Bm.double()
    acc, bound = a @ b.T, K * 2.0 ** -23 * (a.abs() @ b.abs().T)
    view = lambda t: t[shift:shift + M * N].view(M, N).double()
    pre = acc + bias[:N].double()
    small = 2.0 ** -23 * (acc.abs() + pre.abs())
    if epi == 3:
        x = view(aux).requires_grad_(True)
        gelu(x).sum().backward()
        ref, bound = acc * x.grad, 1.13 * bound + 1e-6 * (1.0 + acc.abs())
    elif epi == 2:
        ref, bound = gelu(pre), 1.13 * (bound + small) + 1e-6 * (1.0 + pre.abs())
        assert bool(((view(aux) - pre).abs() <= bound + 2.0 ** -8 * pre.abs()).all())
    else:
        ref, bound = pre, bound + small
    if epi:
        bound = bound * 1.01 + 2.0 ** -8 * ref.abs()
    assert bool(((view(out) - ref).abs() <= bound).all())
    for t in [out] + ([aux] if epi == 2 else []):   # nothing written beside the matrix
        assert t[shift + M * N].item() == 5.0 and (shift == 0 or t[0].item() == 5.0)
