"""Packed-segment rays of ray and eigenray runs and of the beams in ray
coordinates, against the general step: a batch that also holds an environment
with volume attenuation takes the general step for all of it, a run of the
environment alone the packed one.

Both do the same FP64 operations in the same order, so the trajectories are
equal to the bit, and so are the step and contribution counts. Fields sum equal
contributions to FP32 in another order, n < 1e3 additions of rounding 6e-8:
1e-4 of the largest pressure. The fans sit on both sides of the sizes at which
a warp takes a second and a fourth ray (888 and 1776 on 148 SMs)."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile import EnvSpec, write_env
from bellhopcuda_b200.workloads import munk_c

pytestmark = pytest.mark.gpu


def spec(kind, run, nalpha, **kw):
    z = np.linspace(0.0, 1500.0, 31)
    return EnvSpec(title="lanes", freq=120.0, ssp_type=kind, top_bc="V", atten_unit="W", ssp_z=z,
                   ssp_cp=munk_c(z * 3.0), bot_bc="A", bot_hs=(1500.0, 1650.0, 0.0, 1.7, 0.5, 0.0), nsz=1, sz=(430.0,),
                   nrz=5, rz=(10.0, 1400.0), nrr=31, rr_km=(0.5, 15.0), run_type=run, nalpha=nalpha,
                   alpha=(-40.0, 40.0), deltas=0.0, box_z=1600.0, box_r_km=15.2, **kw)


def walls():
    r = np.array([0.0, 3.0, 3.001, 6.0, 8.0, 8.002, 11.0, 16.0])
    return dict(bty_r=r, bty_z=np.array([1500.0, 1400.0, 700.0, 760.0, 1300.0, 900.0, 1450.0, 1400.0]), bty_type="LS")


def run(specs, root):
    with B.Tracer(precision=B.PREC_FP64) as t:
        for i, s in enumerate(specs):
            path = write_env(s, root + str(i))
            if s.run_type[1] in "RC":
                with open(root + str(i) + ".env", "a") as f:
                    f.write("'MS' 1.0 50.0\n1 5 'P'\n")
            t.add_env(path)
        t.run()
        rays = t.rays() if specs[0].run_type[0] in "RE" else None
        field = t.field(0) if rays is None else None
        return rays, field, t.stats()


@pytest.mark.parametrize("kind,nalpha", [("C", 1), ("S", 888), ("P", 889), ("C", 1777)])
@pytest.mark.parametrize("beam", ["RG RR ", "EG RR ", "Cb RR ", "Cg RR ", "CS RR ", "CR RR ", "CC RR "])
def test_rays_equal_the_general_step(beam, kind, nalpha, tmp_path):
    s = spec(kind, beam, nalpha, **(walls() if nalpha != 888 else {}))
    other = spec("C", beam, 1, ssp_ap=np.full(31, 0.02))
    root = os.path.join(str(tmp_path), "e")
    rays, field, st = run([s], root)
    grays, gfield, gst = run([s, other], root + "g")
    _, _, ost = run([other], root + "o")
    for k in ("steps", "evals", "segments"):
        assert st[k] + ost[k] == gst[k], k
    if rays is None:
        # a simple Gaussian beam's amplitude is NaN when its fan has one beam (no beam spacing)
        assert np.array_equal(np.isnan(field), np.isnan(gfield))
        field, gfield = np.nan_to_num(field), np.nan_to_num(gfield)
        assert np.abs(field - gfield).max() <= 1e-4 * np.abs(gfield).max()
        return
    key = lambda r: (r["alpha"], len(r["rz"]), r["ntop"], r["nbot"])   # eigenrays come in any order
    rays, grays = sorted(rays, key=key), sorted(grays, key=key)
    assert len(rays) == len(grays)
    for a, b in zip(rays, grays):
        assert key(a) == key(b) and np.array_equal(a["rz"], b["rz"])
