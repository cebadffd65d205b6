"""Large results on their way to the host, on both sides of the size (32 MB) from
which threads share the copy to pageable memory: the same bytes as the plain copy
to pinned memory, and again the same when repeated."""
import ctypes as C
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile import EnvSpec, write_env
from bellhopcuda_b200.workloads import munk_c

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrz,nrr", [(2001, 2003), (2101, 1999), (3001, 2003), (501, 101)])   # 32.1, 33.6, 48.1, 0.4 MB
def test_large_field(nrz, nrr, tmp_path):
    import torch
    z = np.linspace(0.0, 1500.0, 31)
    s = EnvSpec(title="copy", freq=50.0, ssp_type="C", top_bc="V", atten_unit="W", ssp_z=z, ssp_cp=munk_c(z * 3.0),
                bot_bc="R", bot_hs=(1500.0, 1600.0, 0.0, 1.5, 0.0, 0.0), nsz=1, sz=(700.0,), nrz=nrz, rz=(0.0, 1500.0),
                nrr=nrr, rr_km=(0.0, 15.0), run_type="CG RR ", nalpha=31, alpha=(-20.0, 20.0), deltas=0.0,
                box_z=1600.0, box_r_km=15.2)
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup(write_env(s, os.path.join(str(tmp_path), "e"))).run()
        first = t.field()
        assert first.size == nrz * nrr and np.abs(first).max() > 0
        pinned = torch.zeros(first.size * 2, dtype=torch.float32, pin_memory=True)
        lib = B.load_library()
        assert lib.bhcb_copy_field(t._h, 0, 0, C.c_void_p(pinned.data_ptr()), first.nbytes) == 0
        assert np.array_equal(pinned.numpy().view(np.complex64), first.ravel())
        assert np.array_equal(t.field(), first)
