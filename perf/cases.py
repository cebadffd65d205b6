"""The work a user has this library do, as cases to be timed and compared.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (an environment set up in a context, or a network and its batch),
``run`` makes one pass through the public entry points and returns its whole
outputs, ``work`` says what a pass cannot do without, and ``exact`` gives the
same outputs from plain 64-bit torch where that is quick enough.

Families (key ``kind``):

* ``sweep``     a new in-memory environment per pass: described, run, copied to
                the host (inversions and parameter sweeps: latency counts)
* ``munk``      2-D TL of a deep Munk channel, flat boundaries
* ``rd``        2-D TL, PCHIP profile over 200-point bathymetry, one or more
                frequencies per environment
* ``batch``     many uneven spline-profile environments in one run
* ``arrivals``  2-D arrivals (AddArr order), counts and records on the host
* ``eigen``     2-D eigenray hits and the re-traced rays
* ``beams``     2-D TL with the beam types other than Cartesian geometric
* ``tl3d``      3-D TL, hexahedral profile over gridded bathymetry
* ``arr3d``     3-D arrivals of the same ocean
* ``nx2d``      Nx2D TL: 2-D rays in each receiver bearing's plane
* ``train`` / ``infer``  the TL surrogate's training step and inference
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import bellhopcuda_b200 as B
from bellhopcuda_b200 import surrogate as S
from bellhopcuda_b200 import workloads as W
from bellhopcuda_b200.envfile import write_env

FAN_3D = (361, 144)                 # elevations, bearings of the full 3-D fan
GRID_3D = (36, 101, 501)            # bearings, depths, ranges of its receivers


def listed():
    return [
        # the smallest call: a coarse field of a new environment, host to host
        dict(name="sweep_hat_201", kind="sweep", precision="mixed", beam="G", nalpha=201, nrz=51, nrr=201),
        # the ordinary single field: 2001 hat beams, 201 x 1001 receivers
        dict(name="munk_hat_2001", kind="munk", precision="mixed", run="CG", nalpha=2001, nrz=201, nrr=1001),
        # the benchmark's own: 20001 Gaussian beams, 501 x 2001 receivers, 10 frequencies
        dict(name="rd_gauss_10f", kind="rd", precision="mixed", run="CB", nalpha=20001, nrz=501, nrr=2001, nfreq=10),
        # one field in double precision, incoherent, odd sizes
        dict(name="rd_incoherent_fp64", kind="rd", precision="fp64", run="IB", nalpha=7001, nrz=251, nrr=1003,
             nfreq=1),
        # a batch of short uneven environments in one launch
        dict(name="batch_spline_24", kind="batch", precision="mixed", n=24, scale=0.25,
             env_seed=1003),
        # arrivals on a receiver grid, merged as the reference merges them
        dict(name="arrivals_gauss", kind="arrivals", precision="fp64", beam="B", nalpha=1001, nrz=41, nrr=101,
             merge=True),
        # eigenrays to a handful of receivers
        dict(name="eigen_hat", kind="eigen", precision="fp64", beam="G", nalpha=5001, nrz=5, nrr=11),
        # Gaussian beams in ray-centred coordinates, odd sizes
        dict(name="raycen_gauss", kind="beams", precision="fp64", beam="b", nalpha=801, nrz=101, nrr=403),
        # the largest field: 51,984 rays through a 3-D ocean
        dict(name="tl3d_full", kind="tl3d", precision="mixed", run="CB", fan=1.0, grid=1.0),
        # 3-D arrivals on a coarser fan and grid
        dict(name="arr3d", kind="arr3d", precision="fp64", run="aB", fan=0.5, grid=0.3),
        # 36 bearings of 361 rays each
        dict(name="nx2d_gauss", kind="nx2d", precision="fp64", run="CB", nalpha=361, ntheta=36, nrz=101, nrr=501),
        # one optimiser step of the surrogate at its training batch
        dict(name="train_256", kind="train", batch=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "munk", "rd", "batch", "arrivals", "eigen", "beams", "tl3d", "arr3d", "nx2d",
                       "train", "infer"])
    prec = rng.choice(["mixed", "fp64"])
    if kind == "sweep":
        return dict(kind=kind, precision=prec, beam=rng.choice("GB"), nalpha=_log(rng, 51, 801),
                    nrz=_log(rng, 11, 101), nrr=_log(rng, 51, 401))
    if kind == "munk":
        return dict(kind=kind, precision=prec, run=rng.choice("CIS") + rng.choice("GB"), nalpha=_log(rng, 301, 4001),
                    nrz=_log(rng, 21, 301), nrr=_log(rng, 101, 1501))
    if kind == "rd":
        return dict(kind=kind, precision=prec, run=rng.choice("CI") + rng.choice("GB"),
                    nalpha=_log(rng, 1001, 20001), nrz=_log(rng, 101, 501), nrr=_log(rng, 401, 2001),
                    nfreq=rng.randint(1, 10) if prec == "mixed" else rng.randint(1, 3))
    if kind == "batch":
        return dict(kind=kind, precision=prec, n=_log(rng, 4, 32), scale=round(rng.uniform(0.05, 0.2), 3),
                    env_seed=rng.randint(1, 9999))
    if kind == "arrivals":
        return dict(kind=kind, precision=prec, beam=rng.choice("GB"), nalpha=_log(rng, 101, 2001),
                    nrz=_log(rng, 5, 61), nrr=_log(rng, 11, 151), merge=rng.random() < 0.7)
    if kind == "eigen":
        return dict(kind=kind, precision="fp64", beam="G", nalpha=_log(rng, 501, 10001), nrz=_log(rng, 1, 5),
                    nrr=_log(rng, 1, 11))
    if kind == "beams":
        return dict(kind=kind, precision=prec, beam=rng.choice("gbRCS"), nalpha=_log(rng, 201, 1501),
                    nrz=_log(rng, 11, 151), nrr=_log(rng, 51, 601))
    if kind == "tl3d":
        return dict(kind=kind, precision=prec, run=rng.choice("CI") + rng.choice("GB"),
                    fan=round(math.exp(rng.uniform(math.log(0.1), 0.0)), 3),
                    grid=round(math.exp(rng.uniform(math.log(0.1), math.log(0.8))), 3))
    if kind == "arr3d":
        return dict(kind=kind, precision="fp64", run="a" + rng.choice("GB"), fan=round(rng.uniform(0.1, 0.6), 3),
                    grid=round(rng.uniform(0.08, 0.3), 3))
    if kind == "nx2d":
        return dict(kind=kind, precision="fp64", run=rng.choice("CI") + rng.choice("GB"), nalpha=_log(rng, 61, 721),
                    ntheta=_log(rng, 4, 72), nrz=_log(rng, 11, 151), nrr=_log(rng, 51, 601))
    if kind == "train":
        return dict(kind=kind, batch=8 * _log(rng, 4, 64))
    return dict(kind=kind, batch=_log(rng, 1, 4096))


# ------------------------------------------------------------------ inputs
def _munk(case, seed, run):
    """The Munk channel with the profile, source and frequency of one seed."""
    r = np.random.Generator(np.random.PCG64([seed, 11]))
    s = W.munk_tl(nalpha=case["nalpha"], nrz=case["nrz"], nrr=case["nrr"], freq=float(r.uniform(45.0, 75.0)))
    s.ssp_cp = s.ssp_cp + np.cumsum(r.normal(0.0, 0.05, len(s.ssp_cp)))
    s.sz = (float(r.uniform(600.0, 1400.0)),)
    s.run_type = run + " RR "
    return s


def _rd(case, seed, run):
    s = W.rd_gauss(seed=2000 + seed, nalpha=case["nalpha"], nrz=case["nrz"], nrr=case["nrr"])
    s.run_type = run + " RR "
    return s


def _beams(case, seed):
    s = _munk(case, seed, "C" + case["beam"])
    s.rr_km, s.box_r_km = (0.0, 50.0), 51.0
    s.alpha = (-20.0, 20.0)
    return s


def _files_3d(case, seed):
    run = case["run"]
    if case["kind"] == "nx2d":
        return W.c4_3d(seed=3000 + seed, run_type=run + "   2", nalpha=case["nalpha"], nbeta=8,
                       ntheta=case["ntheta"], nrz=case["nrz"], nrr=case["nrr"])
    na, nb = FAN_3D
    nt, nz, nr = GRID_3D
    g = case["grid"]
    return W.c4_3d(seed=3000 + seed, run_type=run + "   3", nalpha=max(11, int(na * case["fan"])) | 1,
                   nbeta=max(8, int(nb * case["fan"])), ntheta=max(2, int(nt * g)), nrz=max(5, int(nz * g)),
                   nrr=max(11, int(nr * g)))


def _batch(case, seed):
    """Environments whose sizes are the case's own; profiles and sources vary with the seed."""
    r = np.random.Generator(np.random.PCG64([seed, 13]))
    envs = W.batch_envs(case["n"], seed=case["env_seed"], scale=case["scale"])
    for s in envs:
        s.ssp_cp = s.ssp_cp + r.normal(0.0, 0.3, len(s.ssp_cp))
        s.sz = (s.sz[0] * float(r.uniform(0.9, 1.05)),)
    return envs


HITS_PER_RECEIVER, POINTS_PER_HIT = 40, 1500      # room of an eigenray program's output arrays


class _State:
    pass


def prepare(case, seed):
    st = _State()
    st.case = case
    kind = case["kind"]
    if kind in ("train", "infer"):
        st.model = S.Surrogate(seed=seed)
        g = torch.Generator(device="cuda").manual_seed(seed)
        P = W.c5_params(case["batch"], seed=seed)
        st.x = torch.tensor(S.features(P, range(case["batch"])), device="cuda").bfloat16()
        if kind == "train":
            st.y = torch.randn((case["batch"], S.NP), device="cuda", generator=g)
            st.grad = torch.empty((case["batch"], S.NP), dtype=torch.bfloat16, device="cuda")
            st.loss = torch.zeros(1, dtype=torch.float64, device="cuda")
        return st
    t = st.tracer = B.Tracer(precision=B.PREC_FP64 if case["precision"] == "fp64" else B.PREC_MIXED)
    with tempfile.TemporaryDirectory() as d:
        root = os.path.join(d, "env")
        if kind == "sweep":
            st.spec = _munk(case, seed, "C" + case["beam"])
            st.desc = B.EnvDescription(write_env(st.spec, root))
        elif kind == "munk":
            st.spec = _munk(case, seed, case["run"])
            t.setup(write_env(st.spec, root))
        elif kind == "rd":
            t.setup(write_env(_rd(case, seed, case["run"]), root))
            t.set_frequencies(0, W.rd_gauss_freqs()[:case["nfreq"]])
        elif kind == "batch":
            for i, s in enumerate(_batch(case, seed)):
                t.add_env(write_env(s, root + str(i)))
        elif kind == "arrivals":
            t.set_arrival_options(60, case["merge"])
            t.setup(write_env(_munk(case, seed, "a" + case["beam"]), root))
        elif kind == "eigen":
            t.setup(write_env(_rd(case, seed, "E" + case["beam"]), root))
            room = HITS_PER_RECEIVER * case["nrz"] * case["nrr"]
            st.hits = np.full((room, len(B.EIGEN_HIT_DTYPE)), -1, np.int32)
            st.rz, st.points = np.zeros((room * POINTS_PER_HIT, 2)), 0
        elif kind == "beams":
            write_env(_beams(case, seed), root)
            if case["beam"] in "RC":   # Cerveny beams read their width options after the beam box
                with open(root + ".env", "a") as f:
                    f.write("'MS' 1.0 50.0\n1 5 'P'\n")
            t.setup(root)
        else:
            for suffix, text in _files_3d(case, seed).items():
                with open(root + suffix, "w") as f:
                    f.write(text)
            if kind == "arr3d":
                t.set_arrival_options(58, True)
            t.setup3d(root)
    return st


# -------------------------------------------------------------------- pass
class _OnDevice:
    """A device buffer of a context's, as torch.as_tensor takes it: the tensor
    keeps this object, and with it the context that owns the memory."""

    def __init__(self, tracer, ptr, shape):
        self.tracer = tracer
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<c8", "data": (ptr, False), "version": 3}


def run(st):
    case, kind = st.case, st.case["kind"]
    if kind == "train":
        m = st.model
        pred = m.forward(st.x, keep=True)
        st.loss.zero_()
        m.ops.mse(pred, st.y, st.grad, st.loss, 1.0 / float(pred.numel()))
        m.backward(st.grad)
        grads = [[l.gw, l.gb] for l in m.branch.layers + m.trunk.layers]
        m.step(1e-3)
        return {"pred": pred, "loss": st.loss, "grads": grads, "pbias": m.gpb}
    if kind == "infer":
        return {"pred": st.model.forward(st.x), "error": st.model.predict_error(st.x)}
    t = st.tracer
    if kind == "sweep":
        t.clear()
        t.add_env_desc(st.desc)
        t.run()
        return t.field()
    t.run()
    if kind in ("arrivals", "arr3d"):
        narr, arr = t.arrivals()
        return {"narr": narr, **{k: arr[k] for k in B.ARRIVAL_DTYPE.names}}
    if kind == "eigen":
        hits, rays = t.eigen_hits(), t.rays()
        st.hits[:len(hits)] = hits.view("<i4").reshape(len(hits), st.hits.shape[1])
        st.hits[len(hits):] = -1
        n = 0
        for r in rays:
            st.rz[n:n + len(r["rz"])] = r["rz"]
            n += len(r["rz"])
        st.rz[n:st.points] = 0.0
        st.points = n
        return {"nhits": len(hits), "hits": st.hits, "rz": st.rz}
    if kind in ("tl3d", "nx2d"):
        return torch.as_tensor(_OnDevice(t, t.field_device_ptr(), t.field_shape3d()), device="cuda")
    if kind == "batch":
        return [_field(t, e, 0) for e in range(case["n"])]
    return [_field(t, 0, i) for i in range(case.get("nfreq", 1))]


def _field(t, env, ifreq):
    return torch.as_tensor(_OnDevice(t, t.field_device_ptr(env, ifreq), t.field_shape(env)[1:]), device="cuda")


# -------------------------------------------------------------------- work
# Operations of one ray step (2-D; 3-D) and of one applied contribution, and
# the bytes of a receiver's complex pressure. Steps and contributions per ray
# are those the workloads above take, rounded.
F_STEP, F_STEP3, F_INFL = 320.0, 900.0, 40.0


def work(case):
    kind = case["kind"]
    if kind in ("train", "infer"):
        b = case["batch"]
        branch = S.N_IN * 1024 + 3 * 1024 * 1024 + 1024 * 512
        trunk = S.N_TRUNK_IN * 512 + 2 * 512 * 512 + 512 * 512
        mac = b * branch + S.NP * trunk + b * S.NP * 512
        if kind == "infer":
            return {"bytes": 4.0 * b * S.NP + 2.0 * (branch + trunk), "flops": 2.0 * mac}
        n = branch + trunk + S.NP
        return {"bytes": 8.0 * b * S.NP + 28.0 * n, "flops": 6.0 * mac}
    if kind in ("tl3d", "arr3d"):
        rays = max(11, FAN_3D[0] * case["fan"]) * max(8, FAN_3D[1] * case["fan"])
        cells = math.prod(max(2, n * case["grid"]) for n in GRID_3D)
        contrib = rays * cells * (266e6 / (51984 * 1821636))
        return {"bytes": 8.0 * cells + 2.0e6, "flops": rays * 930 * F_STEP3 + contrib * 60}
    if kind == "nx2d":
        rays, cells = case["nalpha"] * case["ntheta"], case["nrz"] * case["nrr"] * case["ntheta"]
        return {"bytes": 8.0 * cells + 2.0e6, "flops": rays * 930 * F_STEP + rays * case["nrr"] * 0.09 * case["nrz"] * F_INFL}
    if kind == "batch":
        rays, cells = 10250 * case["scale"] * case["n"], 330000 * case["scale"] ** 2 * case["n"]
        return {"bytes": 8.0 * cells, "flops": rays * 4300 * F_STEP + rays * 56000 * case["scale"] ** 2 * F_INFL}
    rays, cells, nf = case["nalpha"], case["nrz"] * case["nrr"], case.get("nfreq", 1)
    steps = 1050 if kind in ("rd", "eigen") else 480
    # a ray's beam covers about a sixteenth (Gaussian) or a hundredth (hat) of each receiver column
    gauss = "B" in case.get("run", case.get("beam", "")) or case.get("beam") in ("b", "R", "C", "S")
    contrib = rays * cells * (0.032 if gauss else 0.005)
    out = 4.0 * 44 if kind == "arrivals" else 8.0
    return {"bytes": out * cells * nf, "flops": rays * steps * F_STEP + contrib * nf * F_INFL}


# ------------------------------------------------------- 64-bit counterparts
def exact(case, seed):
    """Plain 64-bit torch: the surrogate's step from its own formulas, and the
    2-D field of a channel with flat boundaries and a c-linear profile. The
    other families' outputs are records in the order of a sequential program,
    or fields that plain torch takes minutes for."""
    kind = case["kind"]
    if kind in ("train", "infer"):
        return _exact_surrogate(case, seed)
    if kind == "sweep":
        return _exact_field(_munk(case, seed, "C" + case["beam"])).cpu().numpy()
    if kind == "munk" and case["run"][0] in "CI":
        return [_exact_field(_munk(case, seed, case["run"]))]
    return None


def _exact_surrogate(case, seed):
    """Forward (and backward) of the network in float64 from the same weights,
    rounded once to bf16 as the layers hold them for their products."""
    st = prepare(case, seed)
    m = st.model
    layers = m.branch.layers + m.trunk.layers
    w = [l.wb.double().requires_grad_() for l in layers]
    b = [l.b.double().requires_grad_() for l in layers]
    pbias = m.pbias.double().requires_grad_()

    def mlp(x, lo, hi):
        for k in range(lo, hi):
            x = torch.nn.functional.linear(x, w[k], b[k])
            if layers[k].gelu:
                x = torch.nn.functional.gelu(x, approximate="tanh")
        return x

    nb = len(m.branch.layers)
    pred = mlp(st.x.double(), 0, nb) @ mlp(m.phi.double(), nb, len(layers)).T + pbias
    if case["kind"] == "infer":
        h = st.x.double()
        for l in m.err_head.layers:
            h = torch.nn.functional.linear(h, l.wb.double(), l.b.double())
            h = torch.nn.functional.gelu(h, approximate="tanh") if l.gelu else h
        return {"pred": pred.detach(), "error": h.detach()[:, 0].exp()}
    d = pred - st.y.double()
    loss = (d * d).sum()
    (loss / d.numel()).backward()
    return {"pred": pred.detach(), "loss": loss.detach().reshape(1),
            "grads": [[x.grad, y.grad] for x, y in zip(w, b)], "pbias": pbias.grad}


def _exact_field(s):
    """The pressure of one source in a c-linear channel with a vacuum surface
    and a fluid halfspace bottom, both flat: the modified polygon steps of
    every ray in lockstep, then the geometric beams' contributions."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def t64(v):
        return torch.tensor(np.asarray(v, dtype=np.float64), device=dev)

    tiny, dmax = 2.0 ** -52, float(np.finfo(np.float64).max)
    gauss, coherent = s.run_type[1] == "B", s.run_type[0] == "C"
    z, c = t64(s.ssp_z), t64(s.ssp_cp)
    cz = (c[1:] - c[:-1]) / (z[1:] - z[:-1])
    depth = float(s.ssp_z[-1])
    steplen = depth / 10.0
    hmin = 1e-6 * steplen
    na, omega = s.nalpha, 2.0 * math.pi * s.freq
    al = s.alpha[0] + np.arange(na) * ((s.alpha[1] - s.alpha[0]) / (na - 1))
    al = al * (math.pi / 180.0)
    dalpha = (al[-1] - al[0]) / (na - 1)
    z0, dz = np.float32(s.rz[0]), (np.float32(s.rz[1]) - np.float32(s.rz[0])) / np.float32(max(1, s.nrz - 1))
    rz = t64((np.float64(z0) + np.arange(s.nrz) * np.float64(dz)).astype(np.float32))
    rr = t64((s.rr_km[0] + np.arange(s.nrr) * ((s.rr_km[1] - s.rr_km[0]) / max(1, s.nrr - 1))) * 1000.0)
    cb, rho_b, att = s.bot_hs[1], s.bot_hs[3], s.bot_hs[4]
    cp_bot = complex(cb, att * s.freq / (8.6858896 * cb) * cb * cb / omega)
    box_x, box_z = s.box_r_km * 1000.0, s.box_z

    n = na
    alive = torch.arange(n, device=dev)

    def segment(x, tz):         # the profile interval a ray moves in
        up = torch.clamp(torch.searchsorted(z, x, right=True) - 1, 0, len(z) - 2)
        down = torch.clamp(torch.searchsorted(z, x, right=False) - 1, 0, len(z) - 2)
        return torch.where(tz >= 0, up, down)

    def speed(x, i):
        return c[i] + (x - z[i]) * cz[i], cz[i]

    zs = float(np.float32(s.sz[0]))
    x, y = torch.zeros(n, dtype=torch.float64, device=dev), torch.full((n,), zs, dtype=torch.float64, device=dev)
    ca, sa = t64(np.cos(al)), t64(np.sin(al))
    iz = segment(y, sa)
    c0, _ = speed(y, iz)
    tx, tz = ca / c0, sa / c0
    rcpq = dalpha / c0
    zero = torch.zeros_like(x)
    p, q = torch.ones_like(x), zero.clone()
    tau, amp, phase = zero.clone(), torch.ones_like(x), zero.clone()
    caus, qold, xold = zero.clone(), zero.clone(), zero.clone()
    cc = c0.clone()
    ratio = torch.sqrt(torch.abs(t64(np.cos(al)))) / (math.sqrt(2.0 * math.pi) if gauss else 1.0)
    dtop, dbot = y.clone(), depth - y
    segs = []

    def reduce(h, x0, y0, ux, uy, i):
        xe, ye = x0 + h * ux, y0 + h * uy
        za, zb = z[i], z[i + 1]
        big = torch.full_like(h, dmax)
        moving = torch.abs(uy) > tiny
        hs = torch.where(moving & (za > ye), (za - y0) / uy, torch.where(moving & (zb < ye), (zb - y0) / uy, big))
        h1 = torch.where(torch.abs(xe) >= box_x, (box_x - torch.abs(x0)) / torch.abs(ux), big)
        h2 = torch.where(torch.abs(ye) >= box_z, (box_z - torch.abs(y0)) / torch.abs(uy), big)
        h3 = torch.where(ye <= 0.0, -y0 / uy, big)
        h4 = torch.where(ye >= depth, (depth - y0) / uy, big)
        for v in (hs, h1, h2, h3, h4):
            h = torch.minimum(h, v)
        return torch.clamp(h, min=hmin)

    def record(x0, y0, x1, y1, tau0, tau1, q0, q1, c0_, c1, amp1, ph0, ph1, who, caus, qold, xold):
        """The carried state of the influence along the ray, and the segment's columns."""
        length = torch.sqrt((x1 - x0) ** 2 + (y1 - y0) ** 2)
        real = length >= 1.0e3 * torch.abs(torch.nextafter(x1, torch.zeros_like(x1)) - x1)
        turn = ((q0 <= 0) & (qold > 0)) | ((q0 >= 0) & (qold < 0))
        caus = torch.where(real & turn, caus + math.pi / 2, caus)
        qold = torch.where(real, q0, qold)
        lo = torch.searchsorted(rr, xold, right=False)
        hi = torch.searchsorted(rr, x1, right=False)
        use = real & (hi > lo)
        if bool(use.any()):
            k = use.nonzero()[:, 0]
            segs.append(torch.stack([v[k] for v in (
                x0, y0, x1, y1, tau0, tau1, q0, q1, c0_, ratio[who] * torch.sqrt(c1) * amp1,
                (ph1 if gauss else ph0) + caus, caus + math.pi / 2, rcpq[who], lo.double(), hi.double())]))
        return caus, qold, torch.where(real, x1, xold)

    for _ in range(100000):
        if not len(alive):
            break
        iz = segment(y, tz)
        s0 = iz
        ca0, g0 = speed(y, iz)
        ux, uy = ca0 * tx, ca0 * tz
        h = reduce(torch.full_like(x, steplen), x, y, ux, uy, s0)
        half = 0.5 * h
        y1, t1z = y + half * uy, tz - half * g0 / (ca0 * ca0)
        q1 = q + half * (ca0 * p)
        p1 = p
        i1 = segment(y1, t1z)
        c1, g1 = speed(y1, i1)
        vx, vy = c1 * tx, c1 * t1z
        h = reduce(h, x, y, vx, vy, s0)
        w1 = h / (2.0 * half)
        w0 = 1.0 - w1
        wx, wy = w0 * ux + w1 * vx, w0 * uy + w1 * vy
        xe, ye = x + h * wx, y + h * wy
        # land on an interface, the box or a boundary
        za, zb = z[s0], z[s0 + 1]
        moving = torch.abs(wy) > tiny
        above, below = moving & (za > ye), moving & (zb < ye)
        for hit, to in ((above, za), (below & ~above, zb)):
            h = torch.where(hit, (to - y) / wy, h)
            xe, ye = torch.where(hit, x + h * wx, xe), torch.where(hit, to, ye)
        out = torch.abs(xe) >= box_x
        h = torch.where(out, (box_x - torch.abs(x)) / torch.abs(wx), h)
        xe, ye = torch.where(out, torch.full_like(xe, box_x), xe), torch.where(out, y + h * wy, ye)
        top = ye < 1e-6
        h = torch.where(top, -y / wy, h)
        xe, ye = torch.where(top, x + h * wx, xe), torch.where(top, torch.zeros_like(ye), ye)
        bot = ye > depth - 1e-6
        h = torch.where(bot, (depth - y) / wy, h)
        xe, ye = torch.where(bot, x + h * wx, xe), torch.where(bot, torch.full_like(ye, depth), ye)
        top = top & ~bot
        short = h < hmin
        h = torch.where(short, torch.full_like(h, hmin), h)
        xe, ye = torch.where(short, x + h * wx, xe), torch.where(short, y + h * wy, ye)
        top, bot = torch.where(short, -ye > tiny, top), torch.where(short, ye - depth > tiny, bot)
        top = top & ~bot
        hw0, hw1 = h * w0, h * w1
        t2z = tz - hw0 * g0 / (ca0 * ca0) - hw1 * g1 / (c1 * c1)
        tau2 = tau + hw0 / ca0 + hw1 / c1
        pn = p
        qn = q + hw0 * (ca0 * p) + hw1 * (c1 * p1)
        i2 = segment(ye, t2z)
        c2, g2 = speed(ye, i2)
        # curvature jump across a profile node
        jump = i2 != s0
        gj = g2 - g0
        n2x, n2z = -t2z, tx
        rm = tx / t2z
        rn = rm * (2.0 * gj * n2z - rm * gj * t2z) / c2
        pn = torch.where(jump, pn - rn * qn, pn)
        caus, qold, xold = record(x, y, xe, ye, tau, tau2, q, qn, cc, c2, amp, phase, phase, alive, caus, qold, xold)
        # reflections
        t3z, i3 = t2z.clone(), i2
        amp3, ph3 = amp.clone(), phase.clone()
        two = top | bot
        if bool(two.any()):
            th = torch.where(bot, t2z, -t2z)             # along the outward normal
            t3z = torch.where(two, -t2z, t2z)
            # unit tangent vectors before and after, and the jumps of the gradient along and across
            rtx, rtz = c2 * tx, c2 * t2z
            rnx, rnz = -rtz, rtx
            rtz_t = c2 * t3z
            rnx_t, rnz_t = rtz_t, -rtx
            cn = -(g2 * (rnz_t - rnz))
            cs = -(g2 * (rtz_t - rtz))
            cn = torch.where(top, -cn, cn)
            rm = tx / th
            rn = rm * (2.0 * cn - rm * cs) / (c2 * c2)
            pn = torch.where(two, pn + rn * qn, pn)
            ph3 = torch.where(top, phase + math.pi, phase)
            kx, kz = omega * tx, omega * t2z
            kzp = torch.sqrt((kx * kx).to(torch.complex128) - (omega / cp_bot) ** 2)
            kzp = torch.where((torch.abs(kzp.real) < tiny) & (kzp.imag < 0), -kzp, kzp)
            jkg = 1j * kz * rho_b
            r = -(kzp - jkg) / (kzp + jkg)
            mag = torch.abs(r)
            amp3 = torch.where(bot, torch.where(mag < float(np.float32(1e-5)), torch.zeros_like(amp), mag * amp), amp)
            ph3 = torch.where(bot & (mag >= float(np.float32(1e-5))), phase + torch.angle(r), ph3)
        x, y, tau, q, p, tz, cc, iz = xe, ye, tau2, qn, pn, t3z, c2, i3
        amp, phase = amp3, ph3
        etop, ebot = y, depth - y
        gone = (torch.abs(x) >= box_x) | (torch.abs(y) >= box_z) | (amp < float(np.float32(0.005)))
        gone |= ((dtop < 0) & (etop < 0)) | ((dbot < 0) & (ebot < 0))
        dtop, dbot = etop, ebot
        if bool(gone.any()):
            k = (~gone).nonzero()[:, 0]
            alive, x, y, tx, tz, tau, q, p, cc, iz, amp, phase, caus, qold, xold, dtop, dbot = (
                v[k] for v in (alive, x, y, tx, tz, tau, q, p, cc, iz, amp, phase, caus, qold, xold, dtop, dbot))

    field = torch.zeros((s.nrr, s.nrz), dtype=torch.complex128 if coherent else torch.float64, device=dev)
    if segs:
        rec = torch.cat(segs, 1)
        ncol = (rec[14] - rec[13]).long()
        per = max(1, 30_000_000 // s.nrz)
        ends = torch.cumsum(ncol, 0).cpu().numpy()
        a = 0
        while a < rec.shape[1]:
            done = ends[a - 1] if a else 0
            b = max(a + 1, int(np.searchsorted(ends, done + per, "right")))
            _add_segments(field, rec[:, a:b], ncol[a:b], rr, rz, omega, s.freq, gauss, coherent)
            a = b
    u = (field if coherent else torch.sqrt(field).to(torch.complex128)).T
    scale = torch.where(torch.abs(rr) < tiny, torch.zeros_like(rr), -1.0 / torch.sqrt(torch.clamp(rr, min=tiny)))
    return (u * scale).contiguous()[None]


def _add_segments(field, rec, ncol, rr, rz, omega, freq, gauss, coherent):
    """Contributions of segments to every depth of the receiver columns they span."""
    r = rec.repeat_interleave(ncol, 1)[:, :, None]
    first = torch.cumsum(ncol, 0) - ncol
    off = torch.arange(int(ncol.sum()), device=rec.device) - first.repeat_interleave(ncol)
    col = r[13, :, 0].long() + off
    x0, y0, x1, y1, tau0, tau1, q0, q1, c0, num, ph_a, ph_b, rcpq = r[:13]
    length = torch.sqrt((x1 - x0) ** 2 + (y1 - y0) ** 2)
    ex, ez = (x1 - x0) / length, (y1 - y0) / length
    dx, dz = rr[col][:, None] - x0, rz[None, :] - y0
    at = (dx * ex + dz * ez) / length
    off_n = torch.abs(dz * ex - dx * ez)
    qf = q0 + at * (q1 - q0)
    sig0 = torch.abs(qf * rcpq)
    sig, edge = sig0, torch.maximum(torch.abs(q0), torch.abs(q1)) * rcpq / torch.abs(ex)
    window = 1.0
    if gauss:
        floor = torch.minimum(float(np.float32(0.2)) * freq * tau1, math.pi * c0 / freq)
        sig, edge, window = torch.maximum(sig0, floor), torch.maximum(edge, floor), 4.0
    steep = torch.abs(ex) <= float(np.float32(0.50001))
    inside = steep | ((rz[None, :] >= torch.minimum(y0, y1) - window * edge)
                      & (rz[None, :] <= torch.maximum(y0, y1) + window * edge))
    inside = inside & (off_n < window * sig)
    amp = num / torch.sqrt(torch.abs(qf))
    wgt = torch.exp(-0.5 * (off_n / sig) ** 2) * (sig0 / sig) if gauss else (sig - off_n) / sig
    if coherent:
        caustic = ((qf <= 0) & (q0 > 0)) | ((qf >= 0) & (q0 < 0))
        ang = omega * (tau0 + at * (tau1 - tau0)) - torch.where(caustic, ph_b, ph_a)
        v = torch.polar(torch.where(inside, amp * wgt, torch.zeros_like(ang)), -ang)
    else:
        v = torch.where(inside, amp * amp * wgt * (math.sqrt(2.0 * math.pi) if gauss else 1.0), torch.zeros_like(amp))
    field.index_add_(0, col, v)
