"""The packed-segment ray step (profiles of types C, S and P without
attenuation) against the oracle where it can go wrong: two-node profiles (one
segment), sources on a profile node and on the axis of launch, boundaries that
leave no rectangle free of tests (steep walls, curvilinear nodes), altimetry,
segment-wise halfspaces, the smallest fans, and the rule that sends a batch of
several profile types, or one with attenuation, to the general step.

FP64 rays: step and contribution counts equal the oracle's. Fields: both sides
add the same FP64 contributions to FP32 accumulators in another order, n
additions of rounding 6e-8 each; n is below 1e3 for these grids, so 1e-4 of the
largest pressure bounds the difference."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile import EnvSpec, write_env
from bellhopcuda_b200.workloads import munk_c
import oracle_ctypes

pytestmark = pytest.mark.gpu


def spec(**kw):
    z = np.linspace(0.0, 1500.0, 31)
    s = EnvSpec(title="segments", freq=120.0, ssp_type="C", top_bc="V", atten_unit="W", ssp_z=z,
                ssp_cp=munk_c(z * 3.0), bot_bc="A", bot_hs=(1500.0, 1650.0, 0.0, 1.7, 0.5, 0.0), nsz=1, sz=(430.0,),
                nrz=23, rz=(0.0, 1500.0), nrr=61, rr_km=(0.0, 15.0), run_type="CB RR ", nalpha=61,
                alpha=(-40.0, 40.0), deltas=0.0, box_z=1600.0, box_r_km=15.2)
    for k, v in kw.items():
        setattr(s, k, v)
    return s


def walls(kind):
    r = np.array([0.0, 3.0, 3.001, 6.0, 8.0, 8.002, 11.0, 16.0])
    z = np.array([1500.0, 1400.0, 700.0, 760.0, 1300.0, 900.0, 1450.0, 1400.0])
    return dict(bty_r=r, bty_z=z, bty_type=kind + "S")


CASES = {
    "node_source_%s" % t: dict(ssp_type=t, sz=(500.0,), nalpha=61) for t in "CSP"
}
CASES.update({"walls_%s" % t: dict(ssp_type=t, run_type="CG RR ", **walls("L")) for t in "CSP"})
CASES.update({
    "two_nodes": dict(ssp_z=np.array([0.0, 1500.0]), ssp_cp=np.array([1480.0, 1525.0]), run_type="CG RR "),
    "curvilinear": dict(ssp_type="P", bty_r=np.linspace(0.0, 16.0, 9), bty_type="CS",
                        bty_z=1200.0 + 250.0 * np.cos(np.linspace(0.0, 9.0, 9))),
    "altimetry": dict(ssp_type="S", ati_r=np.array([0.0, 5.0, 9.0, 16.0]), ati_z=np.array([0.0, 30.0, 5.0, 20.0]),
                      ati_type="LS", sz=(200.0,)),
    "long_halfspaces": dict(bty_r=np.array([0.0, 7.0, 16.0]), bty_z=np.array([1400.0, 1200.0, 1500.0]), bty_type="LL",
                            bty_geo=[(1600.0, 0.0, 1.5, 0.4, 0.0), (1800.0, 400.0, 2.0, 0.6, 0.2),
                                     (1550.0, 0.0, 1.3, 0.2, 0.0)]),
    "one_beam": dict(single_beam=True, isingle=7, nalpha=21),
    "three_rays": dict(nalpha=3, ssp_type="P"),
    "attenuation": dict(ssp_ap=np.full(31, 0.02), ssp_type="S"),   # complex speed: the general step
})


def check(got, st, o):
    assert st["steps"] == o["nsteps"] and st["evals"] == o["nevals"]
    ref = o["field"]
    assert np.abs(got - ref).max() <= 1e-4 * np.abs(ref).max()


@pytest.mark.parametrize("case", sorted(CASES))
def test_steps_equal_the_oracle(case, tmp_path):
    s = spec(**CASES[case])
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup(write_env(s, os.path.join(str(tmp_path), "e"))).run()
        check(t.field(), t.stats(), oracle_ctypes.run(s))


def test_batch_of_several_profile_types(tmp_path):
    """C, S and P together run the general step, three of one type the packed one."""
    for types in ("CSP", "PPP"):
        specs = [spec(ssp_type=k, sz=(300.0 + 150.0 * i,), nalpha=31 + 7 * i) for i, k in enumerate(types)]
        runs = [oracle_ctypes.run(s) for s in specs]
        with B.Tracer(precision=B.PREC_FP64) as t:
            for i, s in enumerate(specs):
                t.add_env(write_env(s, os.path.join(str(tmp_path), "%s%d" % (types, i))))
            t.run()
            st = t.stats()
            assert st["steps"] == sum(o["nsteps"] for o in runs)
            assert st["evals"] == sum(o["nevals"] for o in runs)
            for i, o in enumerate(runs):
                assert np.abs(t.field(i) - o["field"]).max() <= 1e-4 * np.abs(o["field"]).max()
