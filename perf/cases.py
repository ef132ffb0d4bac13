"""Performance cases of the tilt framework: what its users run, over the range of sizes they run it at.

Every case goes through the public Python binding of libtiltgpu: a resident session (`Session`),
many series together (`Batch`), the request loop (`Server`), the one-call host form
(`reconstruct`) and the CTF correction that precedes a reconstruction (`ctf_phaseflip`).
Widths, view counts and thicknesses are those of the benchmark's workloads (a 512-wide and a
2048-wide weighted back-projection, a 1024-wide SIRT run, series of uneven size) and of detectors
whose width is not a power of two.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "imod-rs_b200"))
import tiltgpu as T  # noqa: E402

RELAX = 0.3  # the relaxation the benchmark's SIRT workload runs at (1.0 diverges on thick volumes)


def _series(name, kind, nx, ny, nz, thickness, storage, **more):
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "thickness": thickness, "storage": storage,
         "width": nx, "log": False, "sirt": 0, "xtilt": 0.0, "fill": "mean", "cubic": False, "half_range": 60.0}
    c.update(more)
    return c


def listed():
    return [
        # a trial reconstruction of a few slices, to look at before the whole series is run: launches and latency
        _series("trial_rows_fp32", "session", 256, 16, 41, 128, "fp32"),
        # the one-call form, host array in and host array out, at the size of the reference's own benchmark table
        _series("oneshot_host_256_fp32", "oneshot", 256, 256, 41, 128, "fp32"),
        # an ordinary binned series, weighted back-projection, in the reference's precision and in the half staging form
        _series("wbp_512_fp32", "session", 512, 512, 61, 200, "fp32"),
        _series("wbp_512_fp16", "session", 512, 512, 61, 200, "fp16"),
        # a binned detector of odd width: counts to be log'd, cubic stretch, edge fill, a ragged output
        _series("wbp_odd_1023_bf16", "session", 1023, 717, 77, 187, "bf16", width=1001, log=True, cubic=True,
                fill="edge", half_range=55.0),
        # a full-size series from counts, both forms of the benchmark's large workload
        _series("wbp_2048_fp32", "session", 2048, 2048, 121, 800, "fp32", log=True),
        _series("wbp_2048_fp16", "session", 2048, 2048, 121, 800, "fp16", log=True),
        # SIRT in the reference's precision without x-tilt
        _series("sirt_512_fp32", "session", 512, 512, 61, 200, "fp32", sirt=10),
        # the benchmark's SIRT workload: log, x-tilt, 20 iterations, half staging
        _series("sirt_1024_xtilt_bf16", "session", 1024, 1024, 61, 400, "bf16", sirt=20, log=True, xtilt=1.5),
        # several resident series of uneven size run together, WBP and SIRT(10) at 3:1
        _series("batch_uneven_fp16", "batch", 512, 384, 61, 200, "fp16", sirt=10, count=8),
        # requests with host input and output through the server, WBP and SIRT at 3:1
        _series("serve_mixed_fp16", "serve", 384, 256, 41, 128, "fp16", sirt=10, count=8),
        # the step before a reconstruction: CTF phase flip of a stack, host to host
        _series("ctf_512_host", "ctf", 512, 512, 41, 0, "fp32"),
    ]


def draw(rng):
    kind = rng.choice(["session"] * 7 + ["batch", "serve", "oneshot", "ctf"])

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def width(lo, hi):  # half of them powers of two and 3 * 2^k, half any integer
        if rng.random() < 0.5:
            return rng.choice([w for w in (128, 192, 256, 384, 512, 768, 1024, 1536, 2048) if lo <= w <= hi])
        return log_int(lo, hi)

    storage = rng.choice(["fp32", "fp32", "fp16", "bf16"])
    nz = rng.randint(31, 121)
    half = rng.uniform(50.0, 65.0)
    if kind == "ctf":
        c = _series("", kind, width(256, 1024), width(256, 1024), rng.randint(11, 61), 0, "fp32", half_range=half)
        return {k: v for k, v in c.items() if k != "name"}
    if kind in ("batch", "serve"):
        c = _series("", kind, width(192, 512), log_int(128, 384), rng.randint(31, 61), log_int(64, 200),
                    rng.choice(["fp16", "fp32"]), sirt=rng.choice([5, 10]), count=rng.randint(4, 8), half_range=half)
        return {k: v for k, v in c.items() if k != "name"}
    sirt = rng.choice([0, 0, 0, 3, 10]) if kind == "session" else 0
    top = 2e9 if kind == "oneshot" else 6e10 / (1 + 2 * sirt)
    while True:
        nx, ny = width(128, 2048), log_int(16, 1536)
        thick = log_int(32, 400 if sirt else 800)
        out = nx if rng.random() < 0.7 else max(64, int(nx * rng.uniform(0.6, 1.1)))
        if 1e6 <= float(out) * ny * thick * nz <= top:
            break
    c = _series("", kind, nx, ny, nz, thick, storage, width=out, log=rng.random() < 0.5, sirt=sirt,
                xtilt=rng.choice([0.0, 0.0, round(rng.uniform(-3.0, 3.0), 2)]), fill=rng.choice(["mean", "mean", "zero", "edge"]),
                cubic=rng.random() < 0.2, half_range=half)
    return {k: v for k, v in c.items() if k != "name"}


# ---- inputs ----

def _angles(nz, half_range, rng):
    """A tilt scheme with the goniometer's jitter (degrees)."""
    a = np.linspace(-half_range, half_range, nz) + rng.normal(0.0, 0.1, nz)
    return a.astype(np.float32)


def _stack(nx, ny, angles, counts, seed):
    """Projections [view][row][x] on the GPU: structure at several scales that grows with the path through the
    specimen, plus noise; counts: Poisson counts of a transmitted beam, to be log'd."""
    nz = len(angles)
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    out = torch.empty((nz, ny, nx), dtype=torch.float32, device="cuda")
    base = []
    for cell in (64, 16, 5):
        h, w = max(2, ny // cell + 2), max(2, nx // cell + 2)
        base.append(torch.randn((1, 2, h, w), generator=g, device="cuda"))
    for v in range(nz):
        t = math.radians(float(angles[v]))
        s = torch.zeros((1, 1, ny, nx), device="cuda")
        for b in base:  # the features move and change with the tilt
            f = (b[:, 0:1] * math.cos(t) + b[:, 1:2] * math.sin(t))
            s += torch.nn.functional.interpolate(f, size=(ny, nx), mode="bilinear", align_corners=True)
        path = (1.0 + 0.25 * s[0, 0]) / max(0.2, math.cos(t))
        if counts:
            out[v] = torch.poisson(20000.0 * torch.exp(-0.4 * path.clamp_(min=0.0)), generator=g)
        else:
            out[v] = path + 0.5 * torch.randn((ny, nx), generator=g, device="cuda")
    return out


def _members(case, seed):
    """The single series of a case: a batch or a served mix is several, uneven, every fourth one SIRT."""
    if case["kind"] not in ("batch", "serve"):
        return [case]
    rng = np.random.default_rng([int(case["nx"]), int(case["ny"]), int(case["count"])])  # shapes do not go with the seed
    out = []
    for i in range(case["count"]):
        m = dict(case)
        m["nx"] = m["width"] = int(case["nx"] * rng.choice([0.5, 0.75, 1.0, 1.0, 1.5]))
        m["ny"] = int(case["ny"] * rng.uniform(0.6, 1.1))
        m["nz"] = int(case["nz"] * rng.uniform(0.7, 1.3))
        m["thickness"] = int(case["thickness"] * rng.uniform(0.6, 1.3))
        m["half_range"] = float(rng.uniform(50.0, 65.0))
        m["sirt"] = case["sirt"] if i % 4 == 3 else 0
        out.append(m)
    return out


def _inputs(m, seed):
    rng = np.random.default_rng(int(seed) + 1)
    ang = _angles(m["nz"], m["half_range"], rng)
    return ang, _stack(m["nx"], m["ny"], ang, m["log"], seed)


def _options(m):
    o = dict(width=m["width"], thickness=m["thickness"], radial=(0.35, 0.035), storage=m["storage"], log=m["log"],
             fill_mode=m["fill"], cosine_interp="cubic" if m["cubic"] else "linear")
    if m["sirt"]:
        o.update(sirt=m["sirt"], sirt_relax=RELAX)
    if m["xtilt"]:
        o["xtilt"] = np.full(m["nz"], m["xtilt"], np.float32)
    return o


class _DeviceVolume:
    """A session's resident volume for torch, without a copy (the session lives as long as its volume is in use)."""

    def __init__(self, s):
        self.session = s
        self.__cuda_array_interface__ = {"shape": tuple(s.out_shape), "typestr": "<f4", "data": (s.volume_ptr(), False),
                                         "version": 3}


def _session(m, seed):
    ang, proj = _inputs(m, seed)
    s = T.Session(m["nx"], m["ny"], m["nz"], ang, **_options(m))
    torch.cuda.synchronize()
    s.set_device(proj.data_ptr(), proj.numel())
    s.synchronize()
    return s, torch.as_tensor(_DeviceVolume(s), device="cuda")


def _pinned(t):
    p = torch.empty(t.shape, dtype=torch.float32, pin_memory=True)
    p.copy_(t)
    return p.numpy()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "session":
        s, vol = _session(case, seed)
        return {"kind": kind, "session": s, "volume": vol}
    if kind == "batch":
        b, vols = T.Batch(), []
        for i, m in enumerate(_members(case, seed)):
            s, vol = _session(m, seed * 100 + i)
            b.add(s)
            vols.append(vol)
        return {"kind": kind, "batch": b, "volumes": vols}
    if kind == "serve":
        jobs = []
        for i, m in enumerate(_members(case, seed)):
            ang, proj = _inputs(m, seed * 100 + i)
            out = torch.empty((m["ny"], m["thickness"], m["width"]), dtype=torch.float32, pin_memory=True).numpy()
            jobs.append((_pinned(proj), ang, out, _options(m)))
        return {"kind": kind, "server": T.Server(budget_bytes=8 << 30), "jobs": jobs}
    ang, proj = _inputs(case, seed)
    state = {"kind": kind, "proj": proj.cpu().numpy(), "angles": ang}
    if kind == "oneshot":
        state["options"] = _options(case)
    return state


def run(state):
    kind = state["kind"]
    if kind == "session":
        s = state["session"]
        s.reconstruct()
        st = s.stats()
        return {"volume": state["volume"], "amin": st["amin"], "amax": st["amax"], "amean": st["amean"]}
    if kind == "batch":
        state["batch"].reconstruct()
        return state["volumes"]
    if kind == "serve":
        sv = state["server"]
        ids = [sv.submit(proj, ang, out=out, **o) for proj, ang, out, o in state["jobs"]]
        for i in ids:
            if sv.wait(i)["status"] != 0:
                raise RuntimeError("a served job failed")
            sv.release(i)
        return [job[2] for job in state["jobs"]]
    if kind == "oneshot":
        vol, st = T.reconstruct(state["proj"], state["angles"], **state["options"])
        return {"volume": vol, "amin": st["amin"], "amax": st["amax"], "amean": st["amean"]}
    out, st = T.ctf_phaseflip(state["proj"], state["angles"], pixel_size=_PIXEL, strip_width=256)
    return {"stack": out, "amin": st["amin"], "amax": st["amax"], "amean": st["amean"]}


# ---- the work of a pass ----

def work(case):
    if case["kind"] == "ctf":
        n = float(case["nx"]) * case["ny"] * case["nz"]
        return {"bytes": 8.0 * n, "flops": 4.0 * 2.5 * n * math.log2(max(2.0, case["ny"] * 256.0))}
    b = f = 0.0
    for m in _members(case, 0):
        n_in, n_out = float(m["nx"]) * m["ny"] * m["nz"], float(m["width"]) * m["ny"] * m["thickness"]
        b += 4.0 * (n_in + n_out)
        # one interpolation (a product and a sum for each of two samples) per voxel and view and pass
        f += 4.0 * n_out * m["nz"] * (1 + 2 * m["sirt"]) + (1 + m["sirt"]) * 5.0 * n_in * math.log2(m["nx"])
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits, in plain torch ----
# The sample positions are formed in 32-bit floats in the reference's order, as its sampling decisions (which pair of
# samples, inside or outside a row) are part of what is computed; all data and weights are 64-bit.

_F = np.float32
_PIXEL = 3.4


def _view_geometry(deg, xdeg):
    rad = _F(_F(_F(deg) * _F(math.pi)) / _F(180.0))
    xrad = _F(_F(_F(xdeg) * _F(math.pi)) / _F(180.0))
    return _F(math.cos(rad)), _F(math.sin(rad)), _F(math.cos(xrad)), _F(math.sin(xrad))


def _filter(rows):
    n = rows.shape[-1]
    i = torch.arange(n, device="cuda")
    fb = torch.where(i <= n // 2, i, n - i).double()
    w = fb / (n // 2 + 1)
    cut, fall = float(_F(0.35)), float(_F(0.035))
    wt = torch.where(w <= cut, w, w * torch.exp(-(w - cut) ** 2 / (2.0 * fall * fall)))
    return torch.fft.ifft(torch.fft.fft(rows, dim=-1) * wt, dim=-1).real


def _stretch(rows, deg, cubic):
    """rows [row][x] of one view, as its cosine stretch leaves them."""
    if abs(_F(deg)) > _F(80.0):
        return rows
    n = rows.shape[-1]
    cos_t = _view_geometry(deg, 0.0)[0]
    center = torch.tensor(n / 2.0, dtype=torch.float32, device="cuda")
    x = (torch.arange(n, device="cuda", dtype=torch.float32) - center) * float(_F(1.0) / cos_t) + center
    k = torch.floor(x)
    f = (x - k).double()
    k = k.long()
    at = lambda j: rows[:, j.clamp(0, n - 1)]  # noqa: E731
    lin = at(k) * (1.0 - f) + at(k + 1) * f
    if cubic:
        p0, p1, p2, p3 = at(k - 1), at(k), at(k + 1), at(k + 2)
        a = -0.5 * p0 + 1.5 * p1 - 1.5 * p2 + 0.5 * p3
        b = p0 - 2.5 * p1 + 2.0 * p2 - 0.5 * p3
        c = -0.5 * p0 + 0.5 * p2
        lin = torch.where((k >= 1) & (k + 2 < n), ((a * f + b) * f + c) * f + p1, lin)
    lin = torch.where(k + 1 < n, lin, at(k))
    return torch.where((k >= 0) & (k < n), lin, torch.zeros_like(lin))


class _Geometry:
    """Sampling of one view over the output plane, and of its rows along the columns (x-tilt)."""

    def __init__(self, m, deg):
        c, s, cx, sx = _view_geometry(deg, m["xtilt"])
        nx, onx, onz = m["nx"], m["width"], m["thickness"]
        dx = torch.arange(onx, device="cuda", dtype=torch.float32) - float(_F(onx) / _F(2.0))
        dz = torch.arange(onz, device="cuda", dtype=torch.float32) - float(_F(onz) / _F(2.0))
        x = ((dx * float(c)) * float(cx))[None, :] + (dz * float(s))[:, None] + float(_F(nx) / _F(2.0))
        k = torch.floor(x)
        self.f = (x - k).double().reshape(-1, 1)
        k = k.long().reshape(-1)
        self.inside = ((k >= 0) & (k + 1 < nx)).reshape(-1, 1)
        self.left = (k < 0).reshape(-1, 1)
        self.k = k.clamp(0, nx - 2)


def _rows_of_columns(m):
    """Per (column, slice): the two rows it takes and the weights of both (x-tilt shared by all views)."""
    ny, onx = m["ny"], m["width"]
    sx = _view_geometry(0.0, m["xtilt"])[3]
    dx = torch.arange(onx, device="cuda", dtype=torch.float32) - float(_F(onx) / _F(2.0))
    off = (dx * float(sx))[:, None]
    y = torch.arange(ny, device="cuda", dtype=torch.float32)[None, :] + off
    k = torch.floor(y)
    f = (y - k).double()
    k = k.long()
    two = (k >= 0) & (k + 1 < ny) & (off.abs() > 1e-6)
    one = (k >= 0) & (k < ny) & ~two
    w0 = torch.where(two, 1.0 - f, one.double())
    w1 = torch.where(two, f, torch.zeros_like(f))
    return k.clamp(0, ny - 1), (k + 1).clamp(0, ny - 1), w0, w1


def _backproject(m, ang, rows, means, geometry):
    """rows [view][row][x] to the volume [z * x][row], 1/views applied."""
    ny, onx, onz = m["ny"], m["width"], m["thickness"]
    vol = torch.zeros((onz * onx, ny), dtype=torch.float64, device="cuda")
    for v in range(m["nz"]):
        g = geometry(v)
        r = rows[v].t().contiguous()
        val = r[g.k] * (1.0 - g.f) + r[g.k + 1] * g.f
        if m["fill"] == "edge":
            out = torch.where(g.left, r[0:1], r[-1:])
        else:
            out = torch.full((1, 1), float(means[v]) if m["fill"] == "mean" else 0.0, dtype=torch.float64, device="cuda")
        vol += torch.where(g.inside, val, out)
    vol /= m["nz"]
    if m["xtilt"]:
        k0, k1, w0, w1 = _rows_of_columns(m)
        p = vol.view(onz, onx, ny)
        vol = (p.gather(2, k0.expand(onz, -1, -1)) * w0 + p.gather(2, k1.expand(onz, -1, -1)) * w1).view(onz * onx, ny)
    return vol


def _project(m, vol, geometry):
    ny, onx, onz = m["ny"], m["width"], m["thickness"]
    if m["xtilt"]:
        k0, k1, w0, w1 = _rows_of_columns(m)
        p, q = vol.view(onz, onx, ny), torch.zeros_like(vol).view(onz, onx, ny)
        q.scatter_add_(2, k0.expand(onz, -1, -1), p * w0)
        q.scatter_add_(2, k1.expand(onz, -1, -1), p * w1)
        vol = q.view(onz * onx, ny)
    out = torch.empty((m["nz"], ny, m["nx"]), dtype=torch.float64, device="cuda")
    for v in range(m["nz"]):
        g = geometry(v)
        s = torch.zeros((m["nx"], ny), dtype=torch.float64, device="cuda")
        s.index_add_(0, g.k, torch.where(g.inside, vol * (1.0 - g.f), 0.0))
        s.index_add_(0, g.k + 1, torch.where(g.inside, vol * g.f, 0.0))
        out[v] = s.t()
    return out


def _reconstruct64(m, seed):
    ang, proj = _inputs(m, seed)
    p = proj.double()
    if m["log"]:
        p = torch.log10(p.clamp(min=float(_F(0.001))))
    means = p.mean(dim=(1, 2)).tolist()
    geometry = lambda v: _Geometry(m, ang[v])  # noqa: E731
    rows = _filter(p)
    rows = torch.stack([_stretch(rows[v], ang[v], m["cubic"]) for v in range(m["nz"])])
    vol = _backproject(m, ang, rows, means, geometry)
    del rows
    for _ in range(m["sirt"]):
        vol += float(_F(RELAX)) * _backproject(m, ang, _filter(p - _project(m, vol, geometry)), means, geometry)
    vol = vol.view(m["thickness"], m["width"], m["ny"]).permute(2, 0, 1).contiguous()
    return vol


def _ctf64(case, seed):
    ang, stack = _inputs(case, seed)
    nx, ny = case["nx"], case["ny"]
    kv, cs_a, amp, defocus = 300.0 * 1000.0, float(_F(2.7)) * 1e7, float(_F(0.07)), -3000.0 * 10.0
    m0, e, c, h = 9.10938e-31, 1.60218e-19, 2.99792e8, 6.62607e-34
    wl = h / math.sqrt(2.0 * m0 * e * kv * (1.0 + e * kv / (2.0 * m0 * c * c))) * 1e10
    pixel = float(_F(_PIXEL))
    sw = min(256, int(max(pixel / (wl * (abs(defocus) / nx)), 16.0)))
    out = stack.double()
    res = out.clone()
    for v in range(case["nz"]):
        tilt = float(_F(ang[v])) * float(_F(math.pi)) / 180.0
        for k in range(-(-nx // sw)):
            lo, hi = k * sw, min(nx, (k + 1) * sw)
            center = -nx / 2.0 + (k + 0.5) * sw
            f = torch.fft.fft2(out[v, :, lo:hi])
            fx = torch.fft.fftfreq(hi - lo, device="cuda", dtype=torch.float64).abs() / pixel
            fy = torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64).abs() / pixel
            s2 = fx[None, :] ** 2 + fy[:, None] ** 2
            chi = math.pi * wl * s2 * (defocus + center * pixel * math.sin(tilt) - 0.5 * cs_a * wl * wl * s2)
            ctf = -torch.sin(chi) * math.sqrt(1.0 - amp * amp) + torch.cos(chi) * amp
            val = torch.fft.ifft2(torch.where(ctf < 0.0, -f, f)).real
            x = torch.arange(lo, hi, device="cuda", dtype=torch.float64) - nx / 2.0
            weighs = (1.0 - ((x - center) / (sw / 2.0)).abs()) > 1e-10
            res[v, :, lo:hi] = torch.where(weighs[None, :], val, out[v, :, lo:hi])
    return res


def exact(case, seed):
    kind = case["kind"]
    members = _members(case, seed)
    if kind == "ctf":
        r = _ctf64(case, seed)
        return {"stack": r, "amin": r.min().item(), "amax": r.max().item(), "amean": r.mean().item()}
    updates = [float(m["width"]) * m["ny"] * m["thickness"] * m["nz"] * (1 + 2 * m["sirt"]) for m in members]
    if sum(updates) > 1.2e11:
        return None
    if kind in ("batch", "serve"):
        return [_reconstruct64(m, seed * 100 + i) for i, m in enumerate(members)]
    vol = _reconstruct64(case, seed)
    return {"volume": vol, "amin": vol.min().item(), "amax": vol.max().item(), "amean": vol.mean().item()}
