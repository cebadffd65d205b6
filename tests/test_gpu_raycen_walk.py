"""Ray-centred geometric beams: the influence kernel's walk over records and depths
(slabs of 1 to 32 depths a warp, chosen by the number of depths) against
 * eigenray runs, whose gather takes every record and depth by itself: as many
   contributions as hits, at receivers where the field is not zero;
 * itself with one depth at a time, the narrowest slab: both add the same FP64
   contributions to FP32 in another order, n < 1e3 additions of rounding 6e-8, so
   1e-4 of the largest pressure."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile import EnvSpec, write_env
from bellhopcuda_b200.workloads import munk_c

pytestmark = pytest.mark.gpu


def spec(run, depths, **kw):
    z = np.linspace(0.0, 1500.0, 31)
    s = EnvSpec(title="walk", freq=120.0, ssp_type="C", top_bc="V", atten_unit="W", ssp_z=z, ssp_cp=munk_c(z * 3.0),
                bot_bc="A", bot_hs=(1500.0, 1650.0, 0.0, 1.7, 0.5, 0.0), nsz=2, sz=(430.0, 900.0), nrz=len(depths),
                rz=depths, nrr=41, rr_km=(0.0, 15.0), run_type=run, nalpha=61, alpha=(-50.0, 50.0), deltas=0.0,
                box_z=1600.0, box_r_km=14.0)
    for k, v in kw.items():
        setattr(s, k, v)
    return s


WALLS = dict(bty_r=np.array([0.0, 3.0, 3.001, 6.0, 8.0, 8.002, 11.0, 16.0]), bty_type="LS",
             bty_z=np.array([1500.0, 1400.0, 700.0, 760.0, 1300.0, 900.0, 1450.0, 1400.0]))


def run(s, root):
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup(write_env(s, root)).run()
        if s.run_type[0] == "E":
            return t.eigen_hits(), t.stats()
        return t.field(), t.stats()


@pytest.mark.parametrize("nz", [1, 2, 9, 16, 17, 33, 70])
@pytest.mark.parametrize("beam,kw", [("b", {}), ("g", WALLS), ("b", dict(nrr=1, rr_km=(5.0, 5.0))),
                                     ("g", dict(rr_km=(-3.0, 40.0)))])
def test_walk(beam, kw, nz, tmp_path):
    depths = tuple(np.linspace(20.0, 1480.0, nz)) if nz > 1 else (700.0,)
    root = os.path.join(str(tmp_path), "e")
    field, st = run(spec("C%s RR " % beam, depths, **kw), root)
    hits, est = run(spec("E%s RR " % beam, depths, **kw), root + "h")
    assert st["steps"] == est["steps"] and st["evals"] == len(hits)
    got = np.abs(field).astype(np.float64)
    for iz in sorted({0, nz // 2, nz - 1}):
        one, _ = run(spec("C%s RR " % beam, (float(np.float32(depths[iz])),), **kw), root + "one")
        assert np.abs(field[:, iz] - one[:, 0]).max() <= 1e-4 * max(got.max(), 1e-30)
