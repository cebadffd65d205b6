"""The surrogate's GEMM with operands stored transposed, against the same product
of transposed copies: equal to the bit, since the tensor cores see the same
operands in the same order of K. Both tile widths, ragged M, N and K, every
epilogue; and the column sums that a transposed A brings along, which add one row
after another in FP32 like numpy's accumulate."""
import ctypes as C

import numpy as np
import pytest

import bellhopcuda_b200 as B

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 8), (64, 32, 64), (136, 40, 72), (72, 200, 128), (512, 512, 4104), (512, 128, 264), (640, 1000, 200),
          (2048, 1032, 72), (2056, 40, 1000)]


@pytest.mark.parametrize("a_t,b_t", [(1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_transposed_operands(M, N, K, a_t, b_t):
    import torch
    lib = B.load_library()
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()
    A, Bm, aux = rnd(M, K), rnd(N, K), rnd(M, N)
    As, Bs = A.T.contiguous() if a_t else A, Bm.T.contiguous() if b_t else Bm
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    bias = torch.randn(N, device="cuda", generator=g)
    for epi in range(4):
        new = lambda: torch.full((M, N), 3.0, device="cuda", dtype=torch.float32 if epi == 0 else torch.bfloat16)
        ref, out = new(), new()
        pre = [torch.zeros_like(aux) if epi == 2 else None for _ in range(2)]
        ai = aux if epi == 3 else None
        sums = torch.full((M + 1,), 7.0, device="cuda") if a_t else None
        assert lib.bhcb_nn_gemm(p(A), p(Bm), p(ref), M, N, K, epi, p(bias), p(ai), p(pre[0]), st) == 0
        assert lib.bhcb_nn_gemm_t(p(As), p(Bs), p(out), M, N, K, a_t, b_t, epi, p(bias), p(ai), p(pre[1]), p(sums),
                                  st) == 0
        err = C.c_int32()
        assert lib.bhcb_nn_status(C.byref(err), 1) == 0 and err.value == 0
        assert torch.equal(ref, out)
        assert epi != 2 or torch.equal(pre[0], pre[1])
        if a_t:
            seq = np.add.accumulate(As.float().cpu().numpy(), axis=0)[-1]
            assert np.array_equal(sums[:M].cpu().numpy(), seq) and sums[M].item() == 7.0


def test_refused():
    """K, and the row of a transposed operand, that TMA cannot step over; sums without a transposed A"""
    import torch
    lib = B.load_library()
    x = torch.zeros(64 * 64, device="cuda", dtype=torch.bfloat16)
    o = torch.zeros(64 * 64, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr()) if t is not None else None
    call = lambda M, N, K, a, b, s: lib.bhcb_nn_gemm_t(p(x), p(x), p(o), M, N, K, a, b, 0, None, None, None, p(s), None)
    assert call(16, 16, 12, 1, 1, None) != 0
    assert call(12, 16, 16, 1, 0, None) != 0
    assert call(16, 12, 16, 0, 1, None) != 0
    assert call(16, 16, 16, 0, 0, o) != 0
    assert call(12, 12, 16, 0, 0, None) == 0
    torch.cuda.synchronize()
