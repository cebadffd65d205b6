"""The 3-D ray step over Walk3 (walk3d.cuh) against the general step, at the
places where it can go wrong: sources on a cell face, on a cell diagonal and on
a profile interface, rays launched along the axes (a tangent component exactly
zero) and straight down, boundary cells smaller than a step, a steep wall (no
box without tests), curvilinear and altimetry grids, every 1-D profile type,
attenuation, the hexahedral grid, and beam boxes cutting a cell.

A batch that mixes a hexahedral environment with a 1-D one takes the general
step, so each case runs once alone (Walk3) and once beside the other kind: step
and contribution counts of the pair are the sums of the single ones, and the
field differs by the order of FP32 sums only (n additions of the same FP64
contributions at 6e-8 each; n is below 1e3, so 1e-4 of the largest pressure)."""
import os

import numpy as np
import pytest

import bellhopcuda_b200 as B
from bellhopcuda_b200.envfile3d import env_text, grid_text, hex_ssp_text, write_files

pytestmark = pytest.mark.gpu

PROFILE = [(0.0, 1520.0), (200.0, 1500.0), (400.0, 1485.0), (700.0, 1490.0), (1000.0, 1502.0)]
XY = np.linspace(-6.0, 6.0, 9)


def bowl(scale=1.0, wall=0.0):
    X, Y = np.meshgrid(XY, XY, indexing="ij")
    return 1000.0 - scale * (40.0 * np.cos(X) + 30.0 * np.sin(1.3 * Y)) - 70.0 - wall * (X > 2.9) * 600.0


def files(ssp_opt="CVW", bty=None, ati=None, kind="R", hexa=False, **kw):
    args = dict(title="walk", freq=90.0, ssp_opt=ssp_opt, depth=1000.0, ssp=PROFILE, bot=("A", 1650.0, 1.6, 0.5),
                sx=[0.0], sy=[0.0], sz=[310.0], rz=None, rr_km=None, theta=[0.0, 45.0, 90.0, 200.0], run_type="CB   3",
                alpha=(13, -30.0, 30.0), beta=(9, 0.0, 360.0), step=100.0, box_km=(5.0, 5.0), box_z=1100.0,
                nrz_range=(7, 100.0, 900.0), rr_range=(21, 0.0, 4.5))
    args.update(kw)
    f = {".env": env_text(**args)}
    if bty is not None:
        f[".env"] = f[".env"].replace("'A' 0.0", "'A~' 0.0")
        f[".bty"] = grid_text(XY, XY, bty, kind)
    if ati is not None:
        f[".env"] = f[".env"].replace("'%s'" % ssp_opt, "'%s ~'" % ssp_opt, 1)
        f[".ati"] = grid_text(XY, XY, ati, kind)
    if hexa:
        z = np.array([p[0] for p in PROFILE])
        X, Y, Z = np.meshgrid(XY, XY, z, indexing="ij")
        f[".ssp"] = hex_ssp_text(XY, XY, z, np.interp(Z, z, [p[1] for p in PROFILE]) + 3.0 * np.sin(X) + 2.0 * np.cos(Y))
    return f


CASES = {"profile_" + t: dict(ssp_opt=t + "VW", bty=bowl()) for t in "CNSP"}
CASES.update({
    "attenuation": dict(ssp_opt="SVWT", bty=bowl()),
    "flat": dict(),
    "axes_and_interface": dict(sz=[400.0], alpha=(3, -20.0, 20.0), beta=(5, 0.0, 360.0)),
    "straight_down": dict(alpha=(3, -90.0, 90.0), bty=bowl()),
    "wall": dict(bty=bowl(wall=1.0)),
    "small_cells": dict(bty=bowl(), step=2500.0),
    "curvilinear": dict(bty=bowl(), kind="C"),
    "altimetry": dict(bty=bowl(), ati=bowl(0.2) - 910.0),
    "off_centre": dict(sx=[1.5], sy=[-0.75], bty=bowl(), box_km=(3.2, 2.9)),
    "hex": dict(ssp_opt="HVW", hexa=True, bty=bowl()),
    "hex_on_face": dict(ssp_opt="HVW", hexa=True, sx=[1.5], sy=[1.5], sz=[400.0], bty=bowl(), box_km=(3.4, 3.4)),
    "hex_hat_incoherent": dict(ssp_opt="HVW", hexa=True, bty=bowl(), run_type="IG   3"),
})
# the same ocean as N x 2-D rays (trace_nx_kernel); not the displaced sources, whose planes leave the grid
CASES.update({"nx2d_" + k: dict(v, run_type=v.get("run_type", "CB   3").replace("3", "2")) for k, v in CASES.items()
              if k not in ("off_centre", "hex_on_face")})


def run(roots):
    with B.Tracer(precision=B.PREC_FP64) as t:
        for r in roots:
            t.add_env3d(r)
        t.run()
        st = t.stats()
        return [t.field3d(i) for i in range(len(roots))], st["steps"], st["evals"]


@pytest.mark.parametrize("case", sorted(CASES))
def test_alone_equals_general_step(case, tmp_path):
    other = dict() if "hex" in case else dict(ssp_opt="HVW", hexa=True)
    if CASES[case].get("run_type", "")[-1:] == "2":
        other["run_type"] = "CB   2"
    if "IG" in CASES[case].get("run_type", ""):   # a batch has one beam type and coherence
        other["run_type"] = CASES[case]["run_type"]
    a = write_files(files(**CASES[case]), os.path.join(str(tmp_path), "a"))
    b = write_files(files(alpha=(5, -10.0, 10.0), **other), os.path.join(str(tmp_path), "b"))
    (fa,), sa, ea = run([a])
    (fb,), sb, eb = run([b])
    (ga, gb), s, e = run([a, b])
    assert sa > 0
    assert (s, e) == (sa + sb, ea + eb)
    for x, y in ((fa, ga), (fb, gb)):
        x, y = np.nan_to_num(x), np.nan_to_num(y)
        assert np.abs(x - y).max() <= 1e-4 * np.abs(x).max()
