"""The 3-D influence kernel's rules for the bearings and depths a beam can
reach, at the fans where they differ: a closed circle of bearings, one that
does not divide it, open fans under and over half the circle (the latter takes
every bearing), uneven and single bearings, two receiver depths, receivers at
the source's range and behind it, a beam wider than the fan.

The rules only drop receivers that the beam-window test rejects, so a fan
evaluated at once and bearing by bearing (a single bearing takes no rule for
bearings) has the same contributions: their numbers are equal. The fields add
the same FP64 contributions to FP32 sums in another order, n of them at 6e-8
each; n is below 1e3 here, so 1e-4 of the largest pressure bounds the rest."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile3d import env_text, write_files

pytestmark = pytest.mark.gpu

FANS = {
    "closed_12": [30.0 * i for i in range(12)],
    "closed_7": [360.0 / 7 * i for i in range(7)],
    "open_60": [10.0 * i for i in range(7)],
    "open_negative": [-40.0 + 20.0 * i for i in range(5)],
    "open_300": [30.0 * i for i in range(11)],
    "uneven": [0.0, 7.0, 30.0, 110.0, 200.0],
}


def run(tmp_path, theta, run_type, precision, **kw):
    args = dict(title="reach", freq=80.0, ssp_opt="CVW", depth=1200.0, ssp=[(0.0, 1520.0), (500.0, 1490.0), (1200.0, 1505.0)],
                bot=("A", 1650.0, 1.6, 0.5), sx=[0.3], sy=[-0.2], sz=[300.0], rz=None, rr_km=None, theta=theta,
                run_type=run_type + "   3", alpha=(25, -25.0, 25.0), beta=(25, 0.0, 360.0), step=100.0, box_km=(9.0, 9.0),
                box_z=1300.0, nrz_range=(2, 150.0, 1100.0), rr_range=(33, 0.0, 8.0))
    args.update(kw)
    root = write_files({".env": env_text(**args)}, os.path.join(str(tmp_path), "e"))
    with B.Tracer(precision=precision) as t:
        t.setup3d(root).run()
        return t.field3d()[0, 0, 0], t.stats()["evals"]


@pytest.mark.parametrize("precision", [B.PREC_FP64, B.PREC_MIXED], ids=["fp64", "mixed"])
@pytest.mark.parametrize("run_type", ["CB", "IG"])
@pytest.mark.parametrize("fan", sorted(FANS))
def test_fan_equals_its_bearings(fan, run_type, precision, tmp_path):
    theta = FANS[fan]
    whole, n = run(tmp_path, theta, run_type, precision)
    assert n > 0
    one = [run(tmp_path, [a], run_type, precision) for a in theta]
    assert n == sum(k for _, k in one)
    for i, (f, _) in enumerate(one):
        assert np.abs(whole[i] - f[0]).max() <= 1e-4 * np.abs(whole).max()


def test_beam_wider_than_the_fan(tmp_path):
    """Three launch bearings: each beam covers many receiver bearings."""
    kw = dict(beta=(4, 0.0, 360.0), nrz_range=(9, 100.0, 1100.0))
    whole, n = run(tmp_path, FANS["closed_12"], "CB", B.PREC_FP64, **kw)
    assert n == sum(run(tmp_path, [a], "CB", B.PREC_FP64, **kw)[1] for a in FANS["closed_12"])
