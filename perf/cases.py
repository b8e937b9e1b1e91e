"""The work a user of this package has it do, as timed cases.

Four kinds of calls, each through the public Python entry points:

* ``run``: the reference's own loop body, one tilt at a time: ``Session.upload``
  of a tilt's arrays, then ``Session.run`` (per-position updates of volume,
  probe and scan positions).  What a MEX caller does with 'upload' and
  'run_mset' / 'run_sset'.
* ``batch``: one step of the batched method on a tilt series the session
  holds: ``BatchSession.gradient``, ``apply``, and the updated state read back.
* ``iterate``: whole reconstruction iterations (rotate, pass, rotate back,
  update, TV) from a given volume: ``set_rec``, ``iterate``, ``get_rec``.
* ``rotate``: ``Session.rotate_volume`` of a host volume, as the reference's
  loop does before and after each tilt.

Specimens are fcc lattices of Gaussian atoms, measured patterns are Poisson
counts of the specimen's diffraction patterns at the stated dose, and the
state is a mid-reconstruction one (half the true potential).
"""
import math

import numpy as np
import torch

from mset_b200 import MSET_ADJOINT_EXACT, MSET_ADJOINT_REF, MSET_MODE_MSET, MSET_MODE_SSET
from mset_b200.batch import BatchSession
from mset_b200.session import Session

WINDOWS = (24, 32, 48, 64, 96, 128, 160, 256)  # windows the package supports


def _case(kind, n, **kw):
    """A case with every option named: nz voxels of dx Angstrom in slabs of
    `binning`, scan of scan_x x scan_y positions `scan_step` pixels apart."""
    c = dict(kind=kind, n=n, nz=n, dx=0.3, binning=1, sset=False, exact_adjoint=False, scan_x=8, scan_y=8,
             scan_step=2.0, tilts=1, tilt_max=0.0, dose=1e4, defocus=0.0, jitter=0.0, bf16=False, ckpt=0)
    c.update(kw)
    return c


def listed():
    return [
        # one tilt of the reference's example dataset: 24^2 patterns, 24x24 scan
        _case("run", 24, dx=0.5, scan_x=24, scan_y=24, scan_step=1.0, dose=333.0, name="run_24"),
        # one tilt of the small configuration
        _case("run", 64, nz=24, dx=0.4, scan_x=12, scan_y=12, name="run_64"),
        # the mid configuration's slabs through the reference-semantics pass
        _case("run", 128, binning=2, scan_x=10, scan_y=10, scan_step=3.0, jitter=0.5, name="run_128"),
        # a wide window with thin slabs, an odd scan and the exact adjoint
        _case("run", 160, nz=95, scan_x=5, scan_y=5, scan_step=4.0, dose=3e4, exact_adjoint=True, name="run_160"),
        # the small configuration's five tilts as one batched step
        _case("batch", 64, nz=24, dx=0.4, scan_x=12, scan_y=12, tilts=5, tilt_max=30.0, name="batch_64"),
        # two tilts of an uneven series: 96 thin slabs, exact adjoint
        _case("batch", 96, scan_x=20, scan_y=20, scan_step=3.0, tilts=2, tilt_max=40.0, dose=1e5,
              exact_adjoint=True, name="batch_96"),
        # three tilts of the mid configuration
        _case("batch", 128, binning=2, scan_x=32, scan_y=32, scan_step=3.0, tilts=3, tilt_max=60.0, name="batch_128"),
        # a 160^2 series with its waves checkpointed (memory shared with other work)
        _case("batch", 160, nz=96, scan_x=24, scan_y=24, scan_step=4.0, dose=3e4, ckpt=8, name="batch_160"),
        # one tilt of the large configuration, counts stored as BF16
        _case("batch", 256, nz=192, dx=0.25, binning=2, scan_x=32, scan_y=32, scan_step=4.0, bf16=True,
              name="batch_256"),
        # the small configuration's whole iteration with TV-FISTA
        _case("iterate", 64, nz=24, dx=0.4, scan_x=12, scan_y=12, tilts=5, tilt_max=30.0, edge=24, niter=4,
              tv_lambda=1e-3, tv_iter=300, fista=True, name="iterate_64"),
        # the mid configuration's reconstruction on a few tilts and a coarse scan
        _case("iterate", 128, binning=2, scan_x=12, scan_y=12, scan_step=8.0, tilts=5, tilt_max=60.0, edge=128,
              niter=2, tv_lambda=1e-3, tv_iter=300, fista=True, name="iterate_128"),
        # a tilt rotation of the mid configuration's volume
        _case("rotate", 128, n1=128, n2=128, n3=128, phi=0.0, theta=48.0, psi=0.0, inverse=True, name="rotate_128"),
    ]


def _slabs(c):
    return 1 if c["sset"] else -(-c["nz"] // c["binning"])


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("run", "run", "batch", "batch", "batch", "iterate", "rotate"))
    if kind == "rotate":
        sides = (24, 32, 48, 64, 96, 128, 160)
        n1 = rng.choice(sides)
        cubic = rng.random() < 0.5
        n2, n3 = (n1, n1) if cubic else (rng.choice(sides), rng.choice(sides))
        return _case("rotate", n1, n1=n1, n2=n2, n3=n3, phi=round(rng.uniform(-20, 20), 2),
                     theta=round(rng.uniform(-70, 70), 2), psi=round(rng.uniform(-20, 20), 2),
                     inverse=rng.random() < 0.5)
    n = rng.choice(WINDOWS)
    edge = None
    if kind == "iterate":
        n = rng.choice((24, 32, 48, 64, 96, 128))
        edge = rng.choice([e for e in (24, 32, 48, 64, 96, 128) if e <= n])
    nz = edge if edge else _log(rng, 8, min(n, 128))
    if edge and rng.random() < 0.3:
        nz = rng.choice((24, 32, 48, 64, 96))  # a reconstruction of unequal sides
    binning = rng.choice((1, 1, 2, 3, 4))
    sset = kind != "iterate" and rng.random() < 0.1
    c = _case(kind, n, nz=nz, dx=rng.choice((0.25, 0.3, 0.4)), binning=binning, sset=sset,
              exact_adjoint=rng.random() < 0.4, scan_step=rng.choice((1.0, 2.0, 3.0)),
              dose=float(rng.choice((1e3, 1e4, 1e5))), defocus=rng.choice((0.0, 0.0, 50.0)),
              jitter=rng.choice((0.0, 0.5)))
    ns = _slabs(c)
    scale = (max(n, 48) / 128.0) ** 2
    if kind == "run":
        most = max(2, int(1500 / (ns * scale)))
        p = _log(rng, 1, min(most, 300))
    else:
        c["tilts"] = rng.randint(1, 5)
        c["tilt_max"] = float(rng.choice((30, 50, 70))) if c["tilts"] > 1 else 0.0
        most = max(2, int(100000 / (ns * scale * c["tilts"])))
        p = _log(rng, 4, min(most, 1024))
        if kind == "batch":
            c["bf16"] = rng.random() < 0.25
            c["ckpt"] = rng.choice((0, 0, 0, 4, 8))
        else:
            c.update(edge=edge, niter=rng.randint(1, 3), tv_lambda=rng.choice((0.0, 1e-3, 1e-2)),
                     tv_iter=rng.choice((50, 100, 300)), fista=rng.random() < 0.7)
    c["scan_x"] = max(1, int(math.sqrt(p)))
    c["scan_y"] = max(1, p // c["scan_x"])
    return c


# ---- inputs -----------------------------------------------------------------
E0 = 300e3
_ME, _QE, _CL, _PH = 9.109383e-31, 1.602177e-19, 299792458.0, 6.62607e-34
LAM = _PH / math.sqrt(2 * _ME * _QE * E0) / math.sqrt(1 + _QE * E0 / 2 / _ME / _CL ** 2) * 1e10
SIGMA = (2 * math.pi / LAM / E0) * (_ME * _CL ** 2 + _QE * E0) / (2 * _ME * _CL ** 2 + _QE * E0)


def _atoms(extent, seed):
    """fcc lattice in a box of `extent` Angstrom (x, y, z): positions, peaks"""
    rng = np.random.default_rng([7, seed])
    a = 3.8
    k = [np.arange(-int(e / a) // 2 - 2, int(e / a) // 2 + 3) for e in extent]
    g = np.stack(np.meshgrid(*k, indexing="ij"), -1).reshape(-1, 1, 3)
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    pos = (g + base).reshape(-1, 3) * a
    pos = pos + rng.normal(0, 0.05, pos.shape)
    pos = pos[np.all(np.abs(pos) < np.asarray(extent) / 2 - 0.6, axis=1)]
    return pos, rng.uniform(1.0, 3.0, len(pos))


def _voxels(pos, peak, shape, dx):
    """[nz][ny][nx] sum of Gaussian atoms (sigma 0.3 Angstrom)"""
    p = torch.as_tensor(pos, dtype=torch.float64, device="cuda")
    ax = [(torch.arange(m, device="cuda", dtype=torch.float64) - m // 2) * dx for m in shape]
    gz, gy, gx = (torch.exp(-(a[None] - p[:, 2 - i:3 - i]) ** 2 / (2 * 0.09)).float() for i, a in enumerate(ax))
    gx = gx * torch.as_tensor(peak, dtype=torch.float32, device="cuda")[:, None]
    out = torch.empty(shape, device="cuda")
    for z0 in range(0, shape[0], 8):
        zy = gz[:, z0:z0 + 8, None] * gy[:, None, :]
        out[z0:z0 + 8] = torch.tensordot(zy, gx, dims=([0], [0]))
    return out


def _pad(v, n):
    """[nz][ny][nx] centred laterally in the n x n window"""
    oy, ox = (n - v.shape[1]) // 2, (n - v.shape[2]) // 2
    return torch.nn.functional.pad(v, (ox, n - v.shape[2] - ox, oy, n - v.shape[1] - oy))


def _q2(n, dx):
    q = (np.arange(n) - n // 2) / (n * dx)
    return q[:, None] ** 2 + q[None, :] ** 2


def _probe(c):
    """20 mrad aperture with the case's defocus, sum |F probe|^2 = dose"""
    n, q2 = c["n"], _q2(c["n"], c["dx"])
    chi = math.pi * LAM * q2 * -c["defocus"]
    p = np.fft.fftshift(np.fft.fft2(np.fft.ifftshift((q2 < (0.02 / LAM) ** 2) * np.exp(-1j * chi))))
    return (p * math.sqrt(c["dose"] / np.sum(np.abs(np.fft.fft2(p)) ** 2))).astype(np.complex64)


def _inputs(c, seed):
    """Host arrays of the case, from the seed alone."""
    n, nz, dx, b = c["n"], c["nz"], c["dx"], c["binning"]
    rng = np.random.default_rng([11, seed])
    edge = c.get("edge")
    shape = (nz, edge, edge) if edge else (nz, n, n)
    pos, peak = _atoms((shape[2] * dx, shape[1] * dx, nz * dx), seed)
    th = np.linspace(-c["tilt_max"], c["tilt_max"], c["tilts"]) if c["tilts"] > 1 else np.zeros(1)
    d = dict(angles=np.stack([0 * th, th, 0 * th], 1).astype(np.float32), probe=_probe(c))
    d["prop"] = np.exp(-1j * np.pi * LAM * dx * b * _q2(n, dx)).astype(np.complex64)
    nsx, nsy = c["scan_x"], c["scan_y"]
    cen = n // 2 + 1
    X, Y = np.meshgrid(cen + (np.arange(nsx) - (nsx - 1) / 2) * c["scan_step"],
                       cen + (np.arange(nsy) - (nsy - 1) / 2) * c["scan_step"])
    d["sx"], d["sy"] = X.reshape(-1).astype(np.float32), Y.reshape(-1).astype(np.float32)
    j = rng.uniform(-1, 1, (2, X.size)) * c["jitter"]  # true positions off the nominal ones
    prb, prp = (torch.as_tensor(d[k], device="cuda") for k in ("probe", "prop"))
    tx = torch.as_tensor(d["sx"] + j[0], dtype=torch.float32, device="cuda")
    ty = torch.as_tensor(d["sy"] + j[1], dtype=torch.float32, device="cuda")
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000003 * seed + 17)
    d["meas"], d["vol"] = [], []
    for t in np.deg2rad(th):
        R = np.array([[math.cos(t), 0, -math.sin(t)], [0, 1, 0], [math.sin(t), 0, math.cos(t)]])
        v = _pad(_voxels(pos @ R.T, peak, shape, dx), n)
        T = _transmission(c, v)
        m = torch.cat([torch.poisson(_forward(c, T, torch.fft.ifft2(prb), prp, tx[i:i + 256], ty[i:i + 256])[1]
                                     .abs() ** 2, generator=gen) for i in range(0, tx.numel(), 256)])
        d["meas"].append(torch.fft.fftshift(m, dim=(1, 2)).cpu().numpy())
        d["vol"].append((0.5 * v).cpu().numpy())
    if edge:
        d["rec"] = (0.5 * _voxels(pos, peak, shape, dx)).cpu().numpy()
    # damped steps (a few percent of the state per pass) from the loss's
    # curvature in the volume, the probe and the positions
    per = c["dose"] / n ** 2
    npos = X.size * (1 if c["kind"] == "run" else c["tilts"] if edge else 1)
    cover = per * npos / (X.size * max(1.0, c["scan_step"]) ** 2)
    d["step"] = (0.02 / (SIGMA * dx * nz * max(cover, per / 40)), 0.1 / X.size, 0.02 / per)
    return d


def _rot_volume(c, seed):
    sh = (c["n3"], c["n2"], c["n1"])
    pos, peak = _atoms([0.7 * s * c["dx"] for s in sh[::-1]], seed)
    return _voxels(pos, peak, sh, c["dx"]).cpu().numpy()


def _modes(c):
    return (MSET_MODE_SSET if c["sset"] else MSET_MODE_MSET,
            MSET_ADJOINT_EXACT if c["exact_adjoint"] else MSET_ADJOINT_REF)


def prepare(case, seed):
    c = case
    if c["kind"] == "rotate":
        return dict(case=c, session=Session(0), vol=_rot_volume(c, seed))
    d = _inputs(c, seed)
    st = dict(case=c, d=d)
    if c["kind"] == "run":
        st["session"] = Session(0)
        return st
    method, adjoint = _modes(c)
    step = d["step"] if c["kind"] == "batch" else (d["step"][0], 0.0, 0.0)
    bs = BatchSession(n=c["n"], nz=c["nz"], npos=[d["sx"].size] * c["tilts"], prop=d["prop"], sigma=SIGMA,
                      potential_pixelsize=c["dx"], slice_binning=c["binning"], method=method, adjoint=adjoint,
                      step_size=step)
    if c["bf16"]:
        bs.set_amplitude_bf16(True)
    for j in range(c["tilts"]):
        bs.set_tilt(j, probe=d["probe"], scan_x=d["sx"], scan_y=d["sy"], measured=d["meas"][j], volume=d["vol"][j])
    if c["ckpt"]:
        bs.set_checkpoint(c["ckpt"])
    if c["kind"] == "iterate":
        bs.iteration_setup((c["nz"], c["edge"], c["edge"]), d["angles"], tv_lambda=c["tv_lambda"],
                           tv_iter=c["tv_iter"], tv_fista=c["fista"])
    st["session"] = bs
    return st


def run(state):
    c, s = state["case"], state["session"]
    if c["kind"] == "rotate":
        return s.rotate_volume(state["vol"], (c["phi"], c["theta"], c["psi"]), inverse=c["inverse"])
    d = state["d"]
    if c["kind"] == "run":
        mode, adjoint = _modes(c)
        s.upload(d["vol"][0], d["probe"], d["prop"], sigma=SIGMA, potential_pixelsize=c["dx"], scan_x=d["sx"],
                 scan_y=d["sy"], measured=d["meas"][0], step_size=d["step"], slice_binning=c["binning"],
                 n_scan_x=c["scan_x"], n_scan_y=c["scan_y"])
        return s.run(mode, adjoint)
    if c["kind"] == "batch":
        err = s.gradient(want=("err",))["err"]
        s.apply()
        return [float(e) for e in err], [s.get_tilt(j) for j in range(c["tilts"])]
    s.set_rec(d["rec"])
    err, _ = s.iterate(c["niter"])
    return s.get_rec(), [[float(e) for e in row] for row in err]


def work(case):
    c = case
    if c["kind"] == "rotate":
        vox = c["n1"] * c["n2"] * c["n3"]
        steps = math.floor(max(abs(c["theta"]), 1.0) / 11.0) + 1
        return {"bytes": 8.0 * vox, "flops": steps * 4 * 10.0 * vox * math.log2(c["n1"] * c["n2"])}
    n2, ns, p = c["n"] ** 2, _slabs(c), c["scan_x"] * c["scan_y"]
    fft = 5.0 * n2 * math.log2(n2)
    flops = c["tilts"] * p * ((4 * ns * fft if not c["sset"] else 0) + 32 * ns * n2 + 6 * fft + 40 * n2)
    meas = (2 if c["bf16"] else 4) * n2 * p
    if c["kind"] == "iterate":
        vox = c["nz"] * c["edge"] ** 2
        tv = 60.0 * vox * c["tv_iter"] if c["tv_lambda"] > 0 else 0.0
        return {"bytes": 8.0 * vox + c["niter"] * c["tilts"] * meas, "flops": c["niter"] * (flops + tv)}
    return {"bytes": float(c["tilts"] * (8 * n2 * c["nz"] + meas + 24 * n2)), "flops": flops}


# ---- the same in 64 bits (plain torch) ----------------------------------------
def _transmission(c, v):
    """[ns][n][n] slabs exp(i sigma dz sum V)"""
    b = c["nz"] if c["sset"] else c["binning"]
    s = torch.stack([v[z:z + b].sum(0) for z in range(0, v.shape[0], b)]) * (SIGMA * c["dx"])
    return torch.polar(torch.ones_like(s), s)


def _shift(sx, sy, n):
    """Fourier shift factors [P][n][n] of scan coordinates"""
    k = torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=sx.dtype)
    a = 2 * 3.1415926 / n * k  # pi as the reference's shift factor has it
    ey, ex = (a[None] * (t - (n // 2 + 1))[:, None] for t in (sy, sx))
    return torch.polar(torch.ones_like(ey), ey)[:, :, None] * torch.polar(torch.ones_like(ex), ex)[:, None, :]


def _forward(c, T, Q, prop, sx, sy, keep=None):
    """incident waves and far fields [P][n][n]; keep: list of the waves before
    the first slab and after each"""
    P = torch.fft.ifftshift(prop)
    fs = _shift(sx, sy, c["n"])
    psi0 = torch.fft.fft2(Q * fs)
    w = psi0
    if keep is not None:
        keep.append(w)
    for t in T:
        w = torch.fft.fft2(w * t)
        if c["sset"]:
            return psi0, w, fs
        w = torch.fft.ifft2(w * P)
        if keep is not None:
            keep.append(w)
    return psi0, torch.fft.fft2(w), fs


def _adjoint(c, T, Q, prop, sx, sy, M):
    """of P positions: per-slab gradient sum, probe direction (spectral) sum,
    position directions, error sum; M = sqrt of the patterns, FFT order"""
    n, waves = c["n"], []
    psi0, far, fs = _forward(c, T, Q, prop, sx, sy, waves)
    A = torch.sqrt(far.abs() ** 2 + 1e-30)
    err = ((A - M) ** 2).sum()
    chi = far * (1 - M / A)
    Pc = torch.fft.ifftshift(prop).conj()
    chi = torch.fft.ifft2(chi if c["sset"] else chi * Pc)
    G = torch.empty(T.shape, device="cuda", dtype=M.dtype)
    for s in range(len(T) - 1, -1, -1):
        W = waves[s if c["sset"] or c["exact_adjoint"] else s + 1]
        chi = chi * T[s].conj()
        G[s] = -(chi * W.conj()).imag.sum(0)
        if s:
            chi = torch.fft.ifft2(torch.fft.fft2(chi) * Pc)
    back = torch.fft.ifft2(chi)
    if c["exact_adjoint"]:
        k = 2 * 3.1415926 / n * torch.fft.fftfreq(n, 1.0 / n, device="cuda", dtype=M.dtype)
        X = 1j * Q * fs
        d = [-((X * kk).conj() * back).real.sum((1, 2)) * n * n for kk in (k[None, None, :], k[None, :, None])]
    else:
        d = [(torch.gradient(psi0, dim=ax)[0].conj() * chi).real.sum((1, 2)) for ax in (2, 1)]
    return G, (back * fs.conj()).sum(0), torch.stack(d, 1), err


def _f64(a):
    t = torch.as_tensor(a, device="cuda")
    return t.to(torch.complex128 if t.is_complex() else torch.float64)


def _bf16(m):
    return m.to(torch.bfloat16).to(m.dtype)


def _pass(c, V, probe, prop, sx, sy, meas):
    """batched pass over one tilt, in chunks of positions"""
    T, Q = _transmission(c, V), torch.fft.ifft2(probe)
    G = q = e = 0
    pd = []
    step = max(1, int(6e9 / (16 * (len(T) + 8) * c["n"] ** 2)))
    for i in range(0, sx.numel(), step):
        m = _f64(meas[i:i + step])
        M = torch.sqrt(torch.fft.ifftshift(_bf16(m) if c["bf16"] else m, dim=(1, 2)))
        g, dq, d, err = _adjoint(c, T, Q, prop, sx[i:i + step], sy[i:i + step], M)
        G, q, e = G + g, q + dq, e + err
        pd.append(d)
    return G, q, torch.cat(pd), e


def _spread(c, G):
    """slab gradient on every voxel"""
    return G.repeat_interleave(c["nz"] if c["sset"] else c["binning"], 0)[:c["nz"]]


def _host(t):
    return t.cpu().numpy()


def exact(case, seed):
    c = case
    if c["kind"] == "rotate":
        return _host(_rotate(_f64(_rot_volume(c, seed)), (c["phi"], c["theta"], c["psi"]), c["inverse"]))
    d = _inputs(c, seed)
    step = [float(np.float32(s)) for s in d["step"]]
    probe, prop, sx, sy = (_f64(d[k]) for k in ("probe", "prop", "sx", "sy"))
    if c["kind"] == "run":
        V, Q = _f64(d["vol"][0]), torch.fft.ifft2(probe)
        M = torch.sqrt(torch.fft.ifftshift(_f64(d["meas"][0]), dim=(1, 2)))
        err = 0.0
        for p in range(sx.numel()):
            g, q, pd, e = _adjoint(c, _transmission(c, V), Q, prop, sx[p:p + 1], sy[p:p + 1], M[p:p + 1])
            V += step[0] * _spread(c, g)
            Q = Q - step[1] * q
            sx[p] += step[2] * pd[0, 0]
            sy[p] += step[2] * pd[0, 1]
            err = err + e
        return (_host(V), _host(torch.fft.fft2(Q)), _host(sx), _host(sy),
                float(err) / (c["scan_x"] * c["scan_y"]) / c["n"] ** 2)
    if c["kind"] == "batch":
        errs, tilts = [], []
        for j in range(c["tilts"]):
            V = _f64(d["vol"][j])
            G, q, pd, e = _pass(c, V, probe, prop, sx, sy, d["meas"][j])
            errs.append(float(e))
            tilts.append((_host(V + step[0] * _spread(c, G)),
                          _host(torch.fft.fft2(torch.fft.ifft2(probe) - step[1] * q)),
                          _host(sx + step[2] * pd[:, 0]), _host(sy + step[2] * pd[:, 1])))
        return errs, tilts
    rec, errs = _f64(d["rec"]), []
    o, m = (c["n"] - c["edge"]) // 2, c["edge"]
    for _ in range(c["niter"]):
        acc, row = torch.zeros_like(rec), []
        for j in range(c["tilts"]):
            an = [float(x) for x in d["angles"][j]]
            V = _pad(_rotate(rec, an, True), c["n"])
            G, _, _, e = _pass(c, V, probe, prop, sx, sy, d["meas"][j])
            acc += _rotate(_spread(c, G)[:, o:o + m, o:o + m].contiguous(), an, False)
            row.append(float(e))
        errs.append(row)
        rec = (rec + step[0] * acc).clamp_min(0)
        if c["tv_lambda"] > 0:
            top = rec.max()
            rec = _tv(rec / top, c["tv_lambda"], c["tv_iter"], c["fista"]) * top
    return _host(rec), errs


def _tv(u, lam, niter, fista):
    """dual projected gradient (FISTA momentum), periodic differences"""
    ax = (2, 1, 0)

    def div(P):
        return sum(P[k] - torch.roll(P[k], 1, ax[k]) for k in range(3))

    P = torch.zeros((3,) + u.shape, dtype=u.dtype, device="cuda")
    Y, t = P, 1.0
    for _ in range(niter):
        src = Y if fista else P
        D = div(src) - u / lam
        q = src + torch.stack([torch.roll(D, -1, a) - D for a in ax]) / 12.0
        new = q / torch.sqrt((q ** 2).sum(0).clamp_min(1.0))
        t0, t = t, (1 + math.sqrt(1 + 4 * t * t)) / 2
        Y = new + (t0 - 1) / t * (new - P)
        P = new
    return u - lam * div(P)


def _turn(axis, deg):
    """rotation matrix of the unit quaternion with vector part -axis sin(deg/2)"""
    h = math.radians(deg) / 2
    w, (x, y, z) = math.cos(h), (-math.sin(h) * a for a in axis)
    return np.array([[1 - 2 * y * y - 2 * z * z, 2 * x * y + 2 * w * z, 2 * x * z - 2 * w * y],
                     [2 * x * y - 2 * w * z, 1 - 2 * x * x - 2 * z * z, 2 * y * z + 2 * w * x],
                     [2 * x * z + 2 * w * y, 2 * y * z - 2 * w * x, 1 - 2 * x * x - 2 * y * y]])


def _four_shears(v, w, perm, backward):
    """the four shears (axis, coefficient, coefficient) of the rotation with
    quaternion (v, w), the axes permuted by perm, and their coefficients' sum"""
    x, y, z = (v[(i + perm) % 3] for i in range(3))
    w = -w if backward else w
    yzxw, xyzw = y * z - x * w, x * y - z * w
    if abs(yzxw) > 1e-5 and abs(xyzw) > 1e-5:
        co = [(x * x + y * y) / yzxw, (y * y - z * z) / xyzw - 2 * y * z * (x * x + y * y) / xyzw / yzxw,
              2 * y * z / xyzw, -2 * yzxw, 2 * xyzw, -2 * x * y / yzxw,
              (x * x - y * y) / yzxw + 2 * x * y * (y * y + z * z) / xyzw / yzxw, (x * x + w * w - 1) / xyzw]
    elif abs(y) < 1e-6:
        co = [-x / w, z / w, 0, 2 * x * w, -2 * z * w, 0, -x / w, z / w]
    else:
        return math.inf, None
    ax = [(perm + 1) % 3, perm % 3, (perm + 2) % 3, (perm + 1) % 3]
    if backward:
        sh = [(ax[0], -co[0], -co[1]), (ax[2], -co[2], -co[3]), (ax[1], -co[4], -co[5]), (ax[3], -co[6], -co[7])]
    else:
        sh = [(ax[0], co[6], co[7]), (ax[1], co[4], co[5]), (ax[2], co[2], co[3]), (ax[3], co[0], co[1])]
    return sum(abs(x) for x in co), sh


def _rotate(vol, angles, inverse):
    """Fourier-shear rotation of a [n3][n2][n1] volume: sub-rotations of at
    most 11 degrees, four shears each"""
    if all(abs(a) <= 0.5 for a in angles):
        return vol
    M = (_turn((0, 0, 1), angles[0]) @ _turn((0, 1, 0), angles[1]) @ _turn((1, 0, 0), angles[2])).T
    M = np.linalg.inv(M) if inverse else M
    s = math.sqrt(np.trace(M) + 1) * 2  # below 120 degrees the trace term stays positive
    q = np.array([M[2, 1] - M[1, 2], M[0, 2] - M[2, 0], M[1, 0] - M[0, 1]]) / s
    ang = math.degrees(2 * math.acos(0.25 * s))
    steps = int(ang // 11) + 1
    h = math.radians(ang / steps) / 2
    v, w = -math.sin(h) * q / np.linalg.norm(q), math.cos(h)
    best = [min((_four_shears(v, w, p, b) for p in (1, 2, 3)), key=lambda r: r[0]) for b in (False, True)]
    shears = (best[0] if best[0][0] < best[1][0] else best[1])[1]
    S = torch.fft.ifftshift(vol).to(torch.complex128)
    grid = []
    for ax in range(3):  # 0: x (fastest)
        m = vol.shape[2 - ax]
        g = torch.fft.fftfreq(m, 1.0 / m, device="cuda", dtype=torch.float64)
        nyq = torch.arange(m, device="cuda") == m // 2
        sh = [1, 1, 1]
        sh[2 - ax] = m
        grid.append((g.masked_fill(nyq, 0).reshape(sh), nyq.reshape(sh)))
    for _ in range(steps):
        for k, (d, ca, cb) in enumerate(shears):
            a, b = ((1, 2), (2, 0), (0, 1))[d]  # ca goes with axis a, cb with axis b
            ph = 2 * math.pi / vol.shape[2 - d] * grid[d][0] * (ca * grid[a][0] + cb * grid[b][0])
            ph = ph.masked_fill(grid[0][1] | grid[1][1] | grid[2][1], 0)
            dims = (2 - a, 2 - b)
            S = torch.fft.ifftn(torch.fft.fftn(S, dim=dims) * torch.polar(torch.ones_like(ph), ph), dim=dims)
            if k == 3:
                S = S.real.to(torch.complex128)
    return torch.fft.fftshift(S.real)
