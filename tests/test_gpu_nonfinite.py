"""Beams whose spreading is not a finite number: a receiver test that compares with
NaN or infinity keeps the receiver, and so must every rule that leaves out work.

Beams in ray-centred coordinates and N x 2-D beams against eigenray runs, whose
gathers take every record and receiver by itself: as many contributions as hits. The
step over kept cells against the general step, which a batch of both kinds of ocean
takes: contributions of the batch are the sum of those of its environments alone."""
import os
import random

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile import EnvSpec, write_env
from bellhopcuda_b200.envfile3d import env_text, grid_text, hex_ssp_text, write_files

pytestmark = pytest.mark.gpu


def run(s, root):
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup(write_env(s, root)).run()
        return (t.eigen_hits() if s.run_type[0] == "E" else t.field()), t.stats()


@pytest.mark.parametrize("beam", "gb")
def test_raycen_beam_shift_without_loss(beam, tmp_path):
    """The displacement of a beam at total reflection off a lossless bottom has NaN q."""
    s = EnvSpec(title="nan", freq=400.0, ssp_type="C", top_bc="R", atten_unit="W", ssp_z=np.linspace(0.0, 120.0, 6),
                ssp_cp=np.array([1509.3, 1504.7, 1496.0, 1497.3, 1499.3, 1506.7]), bot_bc="A",
                bot_hs=(120.0, 1600.0, 0.0, 1.7, 0.0, 0.0), nsz=1, sz=(24.0,), nrz=16, rz=(12.0, 114.0), nrr=31,
                rr_km=(-0.24, 1.2), run_type="C%s RR S" % beam, nalpha=2, alpha=(-20.0, 20.0), deltas=0.0, box_z=132.0,
                box_r_km=1.212)
    root = os.path.join(str(tmp_path), "e")
    field, st = run(s, root)
    s.run_type = "E%s RR S" % beam
    hits, _ = run(s, root)
    assert st["evals"] == len(hits) > 0
    assert np.isnan(field).any()


BOTTOM = [(-1.0, 3080.76622911), (3.41496, 2705.46346941), (3.98412, 2778.14218172), (5.1408, 2534.57457607),
          (8.86788, 2793.5918653), (9.01476, 3286.31065653), (18.9, 3110.45643377)]
SPEEDS = [1510.12842095, 1507.46967454, 1506.6479501, 1503.86137494, 1504.2264313, 1499.65926978, 1502.06426914,
          1500.98318806, 1499.90210698, 1498.82102589, 1497.28074557, 1494.74556774, 1495.57778265, 1493.50869379,
          1492.86381948, 1492.38595148, 1490.77940815, 1490.17237725, 1490.63031007, 1491.98978492, 1493.070866,
          1494.18462547, 1495.23302816, 1496.27469847, 1497.99938253, 1498.73608054, 1498.78162588, 1501.16364204,
          1501.61146881, 1504.72987296, 1504.72713614, 1504.96275789, 1506.88222121, 1507.22807957, 1508.20600113,
          1509.28708221, 1512.70123607, 1510.99714923]


@pytest.mark.parametrize("run_type", ["CG", "CB", "IG"])
def test_infinite_spreading(run_type, tmp_path):
    """A ray caught in a hollow of a curvilinear bottom, whose q grows until it is
    infinite: such a beam reaches every depth of the range it passes, and since its
    amplitude is 0 there and its width infinite, the whole column is not a number."""
    r, z = np.array(BOTTOM).T
    s = EnvSpec(title="inf", freq=50.0, ssp_type="S", top_bc="V", atten_unit="W", ssp_z=np.linspace(0.0, 4500.0, 38),
                ssp_cp=np.array(SPEEDS), bot_bc="A", bot_hs=(4500.0, 1600.0, 500.0, 1.7, 0.6, 0.0), nsz=1,
                sz=(121.62162162162163,), nrz=16, rz=(450.0, 4275.0), nrr=31, rr_km=(0.0, 18.0),
                run_type=run_type + " RR S", nalpha=301, single_beam=True, isingle=74, alpha=(-80.0, 48.0), deltas=0.0,
                box_z=4950.0, box_r_km=18.18, bty_r=r, bty_z=z, bty_type="CS")
    field, _ = run(s, os.path.join(str(tmp_path), "e"))
    bad = np.isnan(field[0])
    assert bad.any() and np.array_equal(bad.any(axis=0), bad.all(axis=0))


def hollows(seed, run_type):
    """A curvilinear bottom of hollows under N x 2-D rays."""
    r = random.Random(seed)
    xy = np.linspace(-5.0, 5.0, r.choice([5, 7, 9]))
    bty = np.array([[r.uniform(300.0, 980.0) for _ in xy] for _ in xy])
    if r.random() < 0.5:
        bty = np.repeat(bty[:, :1], len(xy), axis=1)
    hexa = r.random() < 0.4
    z = np.linspace(0.0, 1000.0, r.choice([2, 4, 9]))
    c = 1500.0 - 10.0 * np.sin(z / 300.0)
    beam = r.choice(["CG", "CB", "IG"])
    f = {".bty": grid_text(xy, xy, np.round(bty, 2), "C")}
    f[".env"] = env_text(title="hollows", freq=100.0, ssp_opt=("H" if hexa else r.choice("CSPN")) + r.choice("RV") + "W",
                         depth=1000.0, ssp=list(zip(z, c)), bot=(r.choice("RV") + "~",), sx=[0.0], sy=[0.0], sz=[250.0],
                         rz=None, rr_km=None, theta=[0.0, 60.0, 90.0, 180.0], run_type=(run_type or beam[0]) + beam[1] + "   2",
                         alpha=(41, -80.0, 80.0), beta=(9, 0.0, 360.0), step=100.0, box_km=(4.2, 4.2), box_z=1100.0,
                         nrz_range=(9, 100.0, 900.0), rr_range=(81, 0.0, 4.0))
    if hexa:
        h = np.linspace(-5.0, 5.0, 3)
        X, _, Z = np.meshgrid(h, h, z, indexing="ij")
        f[".ssp"] = hex_ssp_text(h, h, z, np.interp(Z, z, c) + (3.0 * np.sin(X) if r.random() < 0.5 else 0.0))
    return f


@pytest.mark.parametrize("seed", [20, 21, 7])
def test_nx2d_spreading_not_a_number(seed, tmp_path):
    """Rays caught in hollows: q grows until it is infinite, and then is not a number."""
    root = os.path.join(str(tmp_path), "e")
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup3d(write_files(hollows(seed, None), root)).run()
        field, evals = t.field3d(), t.stats()["evals"]
    with B.Tracer(precision=B.PREC_FP64) as t:
        t.setup3d(write_files(hollows(seed, "E"), root)).run()
        assert t.stats()["evals"] == evals
    assert np.isnan(field).any()


def test_nx2d_step_past_all_numbers(tmp_path):
    """p changes by 0 q where the ocean has no depth curvature: nothing, until q is infinite."""
    def evals(roots):
        with B.Tracer(precision=B.PREC_FP64) as t:
            for r in roots:
                t.add_env3d(r)
            t.run()
            return t.stats()["steps"], t.stats()["evals"]
    flat = env_text(title="flat", freq=100.0, ssp_opt="CVW", depth=1000.0, ssp=[(0.0, 1500.0), (1000.0, 1510.0)],
                    bot=("R",), sx=[0.0], sy=[0.0], sz=[250.0], rz=None, rr_km=None, theta=[0.0, 90.0], run_type="CB   2",
                    alpha=(5, -20.0, 20.0), beta=(9, 0.0, 360.0), step=100.0, box_km=(4.2, 4.2), box_z=1100.0,
                    nrz_range=(9, 100.0, 900.0), rr_range=(81, 0.0, 4.0))
    a = write_files(hollows(11, None), os.path.join(str(tmp_path), "a"))
    b = write_files({".env": flat}, os.path.join(str(tmp_path), "b"))
    (sa, ea), (sb, eb) = evals([a]), evals([b])
    assert evals([a, b]) == (sa + sb, ea + eb)


def trap():
    """A horizontal ray along an interface of a hexahedral ocean: it is caught in small
    steps, and its p is 5e304 when the half step, whose length is still the full one,
    takes q past all numbers."""
    x, y = np.linspace(-20.8, 20.8, 2), np.linspace(-20.8, 20.8, 5)
    bty = np.array([[2708.02, 3189.64, 3012.39, 2980.44, 2837.09], [2577.44, 3844.82, 3221.02, 3408.98, 2474.34]])
    ati = np.array([[65.89, 132.56, 14.16, 111.71, 165.63], [146.13, 23.79, 68.95, 113.63, 67.39]])
    z = np.array([0.0, 2000.0, 4000.0])
    c = [1492.1967, 1497.4665, 1494.9830, 1492.4996, 1497.7694, 1491.8159, 1497.0857, 1494.6023, 1492.1188, 1497.3886,
         1494.9378, 1500.2077, 1497.7242, 1495.2407, 1500.5106, 1491.8159, 1497.0857, 1494.6023, 1492.1188, 1497.3886,
         1492.1967, 1497.4665, 1494.9830, 1492.4996, 1497.7694, 1492.1039, 1497.3737, 1494.8902, 1492.4068, 1497.6766,
         1491.7231, 1496.9929, 1494.5095, 1492.0260, 1497.2958, 1494.8450, 1500.1149, 1497.6314, 1495.1479, 1500.4178,
         1491.7231, 1496.9929, 1494.5095, 1492.0260, 1497.2958, 1492.1039, 1497.3737, 1494.8902, 1492.4068, 1497.6766,
         1509.3154, 1514.5853, 1512.1018, 1509.6183, 1514.8882, 1508.9346, 1514.2045, 1511.7210, 1509.2375, 1514.5074,
         1512.0566, 1517.3265, 1514.8430, 1512.3595, 1517.6294, 1508.9346, 1514.2045, 1511.7210, 1509.2375, 1514.5074,
         1509.3154, 1514.5853, 1512.1018, 1509.6183, 1514.8882]
    env = env_text(title="trap", freq=30.0, ssp_opt="HVW ~", depth=4000.0, ssp=[(0.0, 1495.72), (2000.0, 1495.63),
                   (4000.0, 1512.84)], bot=("A~", 1650.0, 1.6, 0.5), sx=[-0.3], sy=[-0.25], sz=[2000.0],
                   rz=[651.57, 838.87, 1858.87, 1996.95, 2487.69, 2955.4, 3655.58], rr_km=[0.0319, 0.2021, 0.2545],
                   theta=[90.0], run_type="CB   3", alpha=(3, -60.0, 60.0), beta=(9, -30.0, 40.0), step=1333.33,
                   box_km=(16.8, 12.8), box_z=3200.0)
    # the file holds one record of x values per (z, y)
    c = np.array(c).reshape(3, 5, 5).transpose(2, 1, 0)
    return {".env": env, ".bty": grid_text(x, y, bty, "R"), ".ati": grid_text(x, y, ati, "R"),
            ".ssp": hex_ssp_text(y, y, z, c)}


def test_half_step_past_all_numbers(tmp_path):
    """As test_nx2d_step_past_all_numbers, in 3-D, for q at the half step."""
    def evals(roots):
        with B.Tracer(precision=B.PREC_FP64) as t:
            for r in roots:
                t.add_env3d(r)
            t.run()
            return t.stats()["steps"], t.stats()["evals"]
    flat = env_text(title="flat", freq=100.0, ssp_opt="CVW", depth=1000.0, ssp=[(0.0, 1500.0), (1000.0, 1510.0)],
                    bot=("R",), sx=[0.0], sy=[0.0], sz=[250.0], rz=[300.0], rr_km=[3.0], theta=[0.0], run_type="CB   3",
                    alpha=(3, -20.0, 20.0), beta=(4, 0.0, 360.0), step=100.0, box_km=(4.2, 4.2), box_z=1100.0)
    a = write_files(trap(), os.path.join(str(tmp_path), "a"))
    b = write_files({".env": flat}, os.path.join(str(tmp_path), "b"))
    (sa, ea), (sb, eb) = evals([a]), evals([b])
    assert evals([a, b]) == (sa + sb, ea + eb) and sa > 100000
