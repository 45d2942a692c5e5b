"""What the advection step is timed on: whole calls through the public entry
points, from one small tracer domain to a 63-million-cell one, in the default
bit-exact kernels and in the single-pass fast ones, the standard scheme, the
batched form, the step with host-resident species, the wind balance and the
simple microphysics.

A pass of the advection cases is one coupling interval of a program whose
other physics keeps the species in its own device arrays: hand the species to
the handle, advance `steps` time steps (boundary update, advection, clipping
where the program asks for it), take them back.

`exact` restates the schemes in float64 torch, array statement by array
statement, from the same inputs.
"""
import ctypes as C
import math

import torch

from hicar_b200 import (AdvOptions, Domain, Options, Parameters, PhysicsOptions, TimeOptions, _lib, advect,
                        balance_uvw, compute_dt, kADV_MPDATA, kADV_STD, kMP_SB04, mp, precipitation, step, step_host,
                        synth)
from hicar_b200.batch import Batch

# species in the order a program adds them: vapour and temperature, then the
# simple scheme's hydrometeors, then the rest of a two-moment set
SPECIES = ("qv", "theta", "qc", "qr", "qs", "qi", "qg", "nr", "ni", "ns", "ng", "nc")


def _case(name, kind, nx, ny, nz, species=1, steps=1, **kw):
    c = {"name": name, "kind": kind, "nx": nx, "ny": ny, "nz": nz, "species": species, "steps": steps, "path": 0,
         "fct": True, "forced": False, "limits": False, "adv_den": False, "real": True, "rk3": False, "flux_corr": 0,
         "h_order": 1, "v_order": 1, "members": 1}
    c.update(kw)
    return c


def listed():
    return [
        # a single call on a small odd-sized nest: launches and latency
        _case("mpdata_call", "mpdata", 67, 45, 16, 4, 1, forced=True),
        # the plain single-tracer domain (128 x 128 x 20), ten steps per coupling interval
        _case("mpdata_tracer", "mpdata", 128, 128, 20, 1, 10, real=False),
        # an ordinary regional domain with the full species set, boundary relaxation and clipping
        _case("mpdata_region", "mpdata", 250, 210, 40, 12, 2, forced=True, limits=True),
        # the full-species benchmark domain on the default (bit-exact) kernels
        _case("mpdata_full", "mpdata", 512, 512, 40, 12, 2, forced=True),
        # the same domain on the fast kernels (the benchmark's headline)
        _case("fast_full", "mpdata", 512, 512, 40, 12, 4, forced=True, path=3),
        # ragged extents, five species, fast kernels
        _case("fast_ragged", "mpdata", 187, 301, 33, 5, 4, forced=True, path=3),
        # a large single domain
        _case("fast_large", "mpdata", 1024, 1024, 60, 12, 1, path=3),
        # the model's default setting: RK3, 5th/3rd order, monotonic flux correction
        _case("std_monotone", "std", 256, 256, 40, 5, 2, forced=True, rk3=True, flux_corr=1, h_order=5, v_order=3),
        # an uneven ensemble advanced together
        _case("ensemble", "batch", 64, 384, 50, 12, 2, members=8, real=False, path=3, forced=True),
        # species in host memory between steps (host physics), page-locked arrays
        _case("host_step", "host", 200, 180, 40, 12, 1, forced=True),
        # wind balance and stable time step, once per forcing update
        _case("winds", "winds", 512, 512, 40, 1, 1, adv_den=True),
        # simple microphysics with its precipitation read back
        _case("microphysics", "mp", 384, 320, 40, 5, 4),
    ]


def draw(rng):
    """Another case of the same ranges: horizontal extents 16..640 (odd ones
    included), 8..60 levels, 1..12 species, any of the kinds."""
    lg = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    kind = rng.choice(["mpdata", "mpdata", "mpdata", "mpdata", "std", "std", "batch", "host", "winds", "mp"])
    nx, ny, nz, s, n = lg(16, 640), lg(16, 640), rng.randint(8, 60), rng.randint(1, 12), rng.randint(1, 4)
    kw = {"forced": rng.random() < 0.7, "limits": rng.random() < 0.3, "real": rng.random() < 0.6,
          "adv_den": rng.random() < 0.3}
    if kind == "mpdata":
        kw.update(path=rng.choice([0, 0, 3]), fct=rng.random() < 0.85)
    elif kind == "std":
        kw.update(rk3=rng.random() < 0.6, flux_corr=int(rng.random() < 0.6), h_order=rng.choice([1, 3, 5]))
        kw["v_order"] = rng.choice([v for v in (1, 3, 5) if v <= kw["h_order"]])
    elif kind == "batch":
        kw.update(path=rng.choice([0, 3, 3]), members=rng.randint(2, 8), forced=True, limits=False)
        nx, ny, nz = rng.randint(24, 96), rng.randint(100, 320), rng.randint(20, 50)
    elif kind == "host":
        nx, ny, n = min(nx, 256), min(ny, 256), 1
        kw.update(path=rng.choice([0, 3]))
    elif kind == "winds":
        s, n = 1, 1
        kw.update(adv_den=rng.random() < 0.5, forced=False, limits=False)
    else:
        s = 5
        kw.update(forced=False, limits=False)
    # no dearer than the largest listed cases
    most = 7e8 if kw.get("path") == 3 else 2e8
    n = max(1, min(n, int(most / (nx * ny * nz * s))))
    s = s if kind == "mp" else max(1, min(s, int(most / (nx * ny * nz * n))))
    return {k: v for k, v in _case("", kind, nx, ny, nz, s, n, **kw).items() if k != "name"}


# ------------------------------------------------------------------ inputs
def _sizes(case, seed):
    """Extents of every domain of the case; ensemble members vary between
    nx and ny in both directions and between 20 and nz levels."""
    if case["kind"] != "batch":
        return [(case["nx"], case["ny"], case["nz"])]
    lo, hi, m = case["nx"], case["ny"], case["members"]
    out = []
    for i in range(m):  # fixed by the case, so that every seed has the same work
        a, b, c = (math.modf((i + 1) * f)[0] for f in (0.618034, 0.754878, 0.569840))
        out.append((int(lo + a * (hi - lo)), int(lo + b * (hi - lo)), int(20 + c * (case["nz"] - 20))))
    return out


def _inputs(case, size, seed):
    """Device fields (Fortran layout) and the time step of one domain: the
    full-species workload's distributions (fractal terrain, 15 m/s westerly
    with 5 % smooth noise, 1 km cells, 4 s) or the ridge workload's (10 m/s,
    4 km, 20 s)."""
    nx, ny, nz = size
    names = SPECIES[: case["species"]]
    if case["real"]:
        f, dt = synth.device_member(nx, ny, nz, seed, dx=1000.0, dz=max(500.0, 20000.0 / nz), species=names,
                                    terrain_kind="fractal", U=15.0, noise=0.05, dt=4.0, rms=600.0, hmax=3000.0)
        dx = 1000.0
    else:
        f, dt = synth.device_member(nx, ny, nz, seed, dx=4000.0, dz=500.0, species=names, U=10.0, noise=0.02, dt=20.0)
        dx = 4000.0
    if case["kind"] == "mp":
        z = -8500.0 * torch.log(f["density"].double() / 1.225)
        p = 101325.0 * torch.exp(-z / 8000.0)
        f["pressure"] = p.float()
        f["exner"] = ((p / 100000.0) ** (287.058 / 1004.5)).float()
        f["dz_mass"] = (f["advection_dz"] * f["jacobian"]).contiguous()
        f["species"]["qv"] = (f["species"]["qv"] * 1.5).contiguous()
    return f, dx, dt


def _options(case):
    return Options(physics=PhysicsOptions(advection=kADV_STD if case["kind"] == "std" else kADV_MPDATA,
                                          microphysics=kMP_SB04 if case["kind"] == "mp" else 0),
                   adv_options=AdvOptions(MPDATA_FCT=case["fct"], flux_corr=case["flux_corr"], h_order=case["h_order"],
                                          v_order=case["v_order"]),
                   time_options=TimeOptions(RK3=case["rk3"]),
                   parameters=Parameters(advect_density=case["adv_den"]))


def prepare(case, seed):
    opts = _options(case)
    st = {"case": case, "opts": opts, "domains": [], "dts": [], "q": [], "out": []}
    for i, size in enumerate(_sizes(case, seed)):
        f, dx, dt = _inputs(case, size, seed + 7919 * i)
        d = Domain.create_on_device(f, *size, dx, opts, forcing=case["forced"])
        d._device_fields = None          # the handle holds its own copies
        if case["path"]:
            d.set_path(case["path"])
        st["domains"].append(d)
        st["dts"].append(dt)
        st["q"].append(f["species"])
        if case["kind"] == "winds":
            st["out"].append({"w": torch.empty_like(f["w"])})
            st["dz_levels"] = f["advection_dz"][0, :, 0].cpu().numpy()
        else:
            st["out"].append({k: torch.empty_like(v) for k, v in f["species"].items()})
    if case["kind"] == "batch":
        # the whole ensemble's state, one array per field, each member fetched into its part
        st["all"] = {k: torch.empty(sum(o[k].numel() for o in st["out"]), device=v.device)
                     for k, v in st["out"][0].items()}
        at = 0
        for o in st["out"]:
            n = next(iter(o.values())).numel()
            for k in o:
                o[k] = st["all"][k][at:at + n]
            at += n
        st["batch"] = Batch(0)
        if case["path"]:
            st["batch"].set_path(case["path"])
        for d, dt in zip(st["domains"], st["dts"]):
            st["batch"].add(d, dt)
    if case["kind"] == "host":
        st["keep"] = [{k: v.cpu().pin_memory() for k, v in st["q"][0].items()},
                      {k: torch.empty(v.shape, pin_memory=True) for k, v in st["q"][0].items()}]
        st["host_in"], st["host_out"] = ({k: v.numpy() for k, v in t.items()} for t in st["keep"])
    torch.cuda.synchronize()
    return st


def _hand_over(d, q):
    lib = _lib.load()
    for k, t in q.items():
        _lib.check(lib.icar_adv_set_field_device(d.handle, _lib.SPECIES_IDS[k], C.c_void_p(t.data_ptr())), d.handle)


def run(state):
    case, opts, doms = state["case"], state["opts"], state["domains"]
    d, dt, q, out = doms[0], state["dts"][0], state["q"][0], state["out"][0]
    if case["kind"] == "host":
        return step_host(d, opts, dt, state["host_in"], state["host_out"], enforce_limits=case["limits"])
    if case["kind"] == "winds":
        balance_uvw(d, opts)
        dt = compute_dt(d, opts, state["dz_levels"])
        d.fetch_device("w", out["w"])
        return {"w": out["w"], "dt": dt}
    if case["kind"] == "mp":
        _hand_over(d, q)
        _lib.check(_lib.load().icar_adv_set_precipitation(d.handle, None, None), d.handle)
        for _ in range(case["steps"]):
            mp(d, opts, dt)
        for k in q:
            d.fetch_device(k, out[k])
        rain, snow = precipitation(d)
        return {**out, "rain": rain, "snow": snow}
    if case["kind"] == "batch":
        for d, q in zip(doms, state["q"]):
            _hand_over(d, q)
        for _ in range(case["steps"]):
            state["batch"].step()
        for d, o in zip(doms, state["out"]):
            for k in o:
                d.fetch_device(k, o[k])
        return state["all"]
    _hand_over(d, q)
    for _ in range(case["steps"]):
        if case["forced"] or case["limits"]:
            step(d, opts, dt, enforce_limits=case["limits"])
        else:
            advect(d, opts, dt)
    for k in q:
        d.fetch_device(k, out[k])
    return out


def work(case):
    """Compulsory traffic and arithmetic.  A step reads the nine wind and
    metric fields and reads and writes every species once (RK3 reads and
    writes it three times); the operation counts are the schemes' own."""
    cells = sum(x * y * z for x, y, z in _sizes(case, 0))
    s, n = case["species"], case["steps"]
    if case["kind"] == "winds":
        return {"bytes": 4.0 * cells * (7 + 1 + 3), "flops": 35.0 * cells}
    if case["kind"] == "mp":
        return {"bytes": n * 4.0 * cells * 14, "flops": n * 250.0 * cells}
    stages = 3 if case["rk3"] else 1
    per = 330.0 if case["kind"] != "std" else 80.0 * stages + (160.0 if case["flux_corr"] else 0.0)
    if case["kind"] != "std" and not case["fct"]:
        per = 230.0
    return {"bytes": n * 4.0 * cells * (9 + 2 * s * stages), "flops": n * per * cells * s}


# ------------------------------------------------------- float64 restatement
def _flux(l, r, U):
    return torch.where(U > 0, l, r) * U


def _sh(a, d, lo, hi):
    return a.narrow(d, lo, hi - lo)


def _upwind64(q, U, V, W, Wtop, G, DJ):
    """Donor-cell update of the interior columns; W has nz-1 inner faces."""
    fx = _flux(q[:, :, :-1], q[:, :, 1:], U[:, :, 1:-1])
    fy = _flux(q[:-1], q[1:], V[1:-1])
    fz = _flux(q[:, :-1], q[:, 1:], W)
    I = (slice(1, -1), slice(None), slice(1, -1))
    top = torch.cat([fz, (q[:, -1] * Wtop)[:, None]], 1)
    bot = torch.cat([torch.zeros_like(fz[:, :1]), fz], 1)
    new = q.clone()
    new[I] = q[I] - ((fx[1:-1, :, 1:] - fx[1:-1, :, :-1]) + (fy[1:] - fy[:-1])[:, :, 1:-1]) / G[I] \
        - ((top - bot) / DJ)[I]
    return new


def _ratio(p, m):
    return (p - m) / (p + m + 1e-10)


def _pseudo64(q, U, V, Wp, G, dz):
    """Antidiffusive velocities on the faces (zero on the outermost)."""
    ny, nz, nx = q.shape
    k = slice(1, nz - 1)
    # x faces 1..nx-1
    l, r, u = q[:, :, :-1], q[:, :, 1:], U[:, :, 1:-1]
    Gs = G[:, :, 1:] + G[:, :, :-1]
    a = u.abs() * (1 - 2 * u.abs() / Gs) * (r - l) / (r + l + 1e-10)
    sx = q[:, :, 1:] + q[:, :, :-1]
    vx = V[:-1] + V[1:]
    vx = vx[:, :, 1:] + vx[:, :, :-1]
    a[1:-1] -= 0.5 * u[1:-1] * 0.25 * vx[1:-1] * _ratio(sx[2:], sx[:-2]) / Gs[1:-1]
    wz = Wp.clone()
    wz[:, 1:] = Wp[:, 1:] + Wp[:, :-1]
    wx = wz[:, :, 1:] + wz[:, :, :-1]
    a[:, k] -= 0.5 * u[:, k] * 0.25 * wx[:, k] * _ratio(sx[:, 2:], sx[:, :-2]) / Gs[:, k]
    u2 = torch.zeros_like(U)
    u2[:, :, 1:-1] = 0.5 * a
    # y faces 1..ny-1
    l, r, v = q[:-1], q[1:], V[1:-1]
    Gs = G[1:] + G[:-1]
    a = v.abs() * (1 - 2 * v.abs() / Gs) * (r - l) / (r + l + 1e-10)
    sy = q[1:] + q[:-1]
    uy = U[1:] + U[:-1]
    uy = uy[:, :, 1:] + uy[:, :, :-1]
    i = slice(1, nx - 1)
    a[:, :, i] -= 0.5 * v[:, :, i] * 0.25 * uy[:, :, i] * _ratio(sy[:, :, 2:], sy[:, :, :-2]) / Gs[:, :, i]
    wy = wz[1:] + wz[:-1]
    a[:, k] -= 0.5 * v[:, k] * 0.25 * wy[:, k] * _ratio(sy[:, 2:], sy[:, :-2]) / Gs[:, k]
    v2 = torch.zeros_like(V)
    v2[1:-1] = 0.5 * a
    # top faces of levels 0..nz-2, interior columns
    I = (slice(1, -1), slice(None), slice(1, -1))
    l, r, w = q[:, :-1], q[:, 1:], Wp[:, :-1]
    Gs = G[:, 1:] + G[:, :-1]
    a = w.abs() * (1 - 2 * w.abs() / Gs) * (r - l) / (r + l + 1e-10)
    sz = q[:, 1:] + q[:, :-1]
    uz = U[:, :, 1:] + U[:, :, :-1]
    uz = uz[:, 1:] + uz[:, :-1]
    vz = V[1:] + V[:-1]
    vz = vz[:, 1:] + vz[:, :-1]
    a = a[I] - 0.5 * w[I] * 0.25 * (uz[I] * _ratio(sz[1:-1, :, 2:], sz[1:-1, :, :-2]) +
                                    vz[I] * _ratio(sz[2:, :, 1:-1], sz[:-2, :, 1:-1])) / Gs[I]
    w2 = torch.zeros_like(w)
    w2[I] = 0.5 * a * dz[:, :-1][I]
    return u2, v2, w2


def _limit64(q0, q1, f2, d, wline):
    """Limited velocities on the inner faces of direction d."""
    n = q1.shape[d]
    f = _flux(_sh(q1, d, 0, n - 1), _sh(q1, d, 1, n), f2)
    z = torch.zeros_like(_sh(f, d, 0, 1))
    fl, fr = torch.cat([z, f], d), torch.cat([f, z], d)
    lo, hi = torch.cat([_sh(q1, d, 0, 1), _sh(q1, d, 0, n - 1)], d), torch.cat([_sh(q1, d, 1, n), _sh(q1, d, n - 1, n)], d)
    # the last cell's bounds leave its own old value out
    p0 = torch.cat([_sh(q0, d, 0, n - 1), _sh(q0, d, n - 2, n - 1)], d)
    l0, h0 = torch.cat([_sh(p0, d, 0, 1), _sh(p0, d, 0, n - 1)], d), torch.cat([_sh(p0, d, 1, n), _sh(p0, d, n - 1, n)], d)
    h0 = torch.cat([_sh(h0, d, 0, n - 2), _sh(q0, d, n - 1, n), _sh(p0, d, n - 1, n)], d)
    six = (lo, q1, hi, l0, p0, h0)
    qmax, qmin = six[0], six[0]
    for a in six[1:]:
        qmax, qmin = torch.maximum(qmax, a), torch.minimum(qmin, a)
    fin, fout = fl.clamp(min=0) - fr.clamp(max=0), fr.clamp(min=0) - fl.clamp(max=0)
    first, last = _sh(fin, d, 0, 1), _sh(fin, d, n - 1, n)
    if wline:
        g = _sh(f, d, n - 2, n - 1).abs()
        last.copy_(g)
        _sh(fout, d, n - 1, n).copy_(g)
    else:
        for t in (first, last, _sh(fout, d, 0, 1), _sh(fout, d, n - 1, n)):
            t.zero_()
    bi, bo = (qmax - q1) / (fin + 1e-15), (q1 - qmin) / (fout + 1e-15)
    il, ir, ol, orr = _sh(bi, d, 0, n - 1), _sh(bi, d, 1, n), _sh(bo, d, 0, n - 1), _sh(bo, d, 1, n)
    return torch.where(f2 > 0, torch.minimum(ir, ol).clamp(max=1), torch.minimum(il, orr).clamp(max=1)) * f2


def _mpdata64(q, P, fct):
    q1 = _upwind64(q, P["U"], P["V"], P["W"][:, :-1], P["W"][:, -1], P["G"], P["DJ"])
    u2, v2, w2 = _pseudo64(q1, P["U"], P["V"], P["W"] / P["dz"], P["G"], P["dz"])
    if fct:
        u2[:, :, 1:-1] = _limit64(q, q1, u2[:, :, 1:-1], 2, False)
        v2[1:-1] = _limit64(q, q1, v2[1:-1], 0, False)
        w2 = _limit64(q, q1, w2, 1, True)
    return _upwind64(q1, u2, v2, w2, torch.zeros_like(q1[:, -1]), P["G"], P["DJ"])


def _filter64(nx, ny, hs, dev):
    """Relaxation weights of a single-image domain (its north and west
    sides, as the model builds them when all four sides are boundaries)."""
    w = [0.9, 0.75, 0.6, 0.5, 0.4, 0.25, 0.1]
    n = min(7, nx - 1 - hs, ny - 1 - hs)
    f = [[0.0] * nx for _ in range(ny)]

    def put(i, j, v):
        if 0 <= i < nx and 0 <= j < ny:
            f[j][i] = v
    for j in range(ny):
        for i in range(hs):
            put(i, j, 1.0)
    for j in range(ny - hs - 2, ny):
        for i in range(nx):
            put(i, j, 1.0)
    for j in range(ny - hs):
        for m in range(n):
            put(hs + m, j, w[m])
    for i in range(hs, nx):
        for m in range(n):
            put(i, ny - hs - n + m, w[6 - m])
    for i in range(n):
        for k in range(n):
            put(hs + i, ny - hs - 1 - k, w[min(i, k)])
    return torch.tensor(f, dtype=torch.float32, device=dev).double()[:, None, :]


def _winds64(f, dx, dt, adv_den, std):
    g = {k: v.double() for k, v in f.items() if k != "species"}
    rho = g["density"] if adv_den else torch.ones_like(g["density"])
    U, V, W = (g[a] * dt * g["jacobian_" + a] for a in "uvw")
    U, V = U / dx, V / dx
    U[:, :, 1:-1] *= 0.5 * (rho[:, :, 1:] + rho[:, :, :-1])
    V[1:-1] *= 0.5 * (rho[1:] + rho[:-1])
    U[:, :, 0] = U[:, :, -1] = 0
    V[0] = V[-1] = 0
    dz = g["advection_dz"]
    if std:
        W[:, :-1] *= (rho[:, :-1] * dz[:, :-1] + rho[:, 1:] * dz[:, 1:]) / (dz[:, :-1] + dz[:, 1:])
    else:
        W[:, :-1] *= 0.5 * (rho[:, :-1] + rho[:, 1:])
    W[:, -1] *= rho[:, -1]
    G = g["jacobian"] * (rho if std else g["density"])
    return {"U": U, "V": V, "W": W, "dz": dz, "G": G, "DJ": dz * G}


def _hflux64(q, U, order, d, a, b):
    """Fluxes through faces a..b of direction d (face f between f-1 and f)."""
    R = lambda o: _sh(q, d, a + o, b + 1 + o)
    u = _sh(U, d, a, b + 1)
    if order == 1:
        return _flux(R(-1), R(0), u)
    if order == 3:
        return u * (7 * (R(0) + R(-1)) - (R(1) + R(-2))) / 12 - u.abs() / 12 * (3 * (R(0) - R(-1)) - (R(1) - R(-2)))
    return u * (37 * (R(0) + R(-1)) - 8 * (R(1) + R(-2)) + (R(2) + R(-3))) / 60 - \
        u.abs() / 60 * (10 * (R(0) - R(-1)) - 5 * (R(1) - R(-2)) + (R(2) - R(-3)))


def _vflux64(q, W, order, top=1.0):
    """Fluxes through the nz+1 horizontal faces."""
    nz = q.shape[1]
    f = torch.zeros_like(torch.cat([q, q[:, :1]], 1))
    f[:, 1:nz] = _flux(q[:, :-1], q[:, 1:], W[:, :-1])
    Wf = torch.cat([torch.zeros_like(W[:, :1]), W], 1)
    if order >= 3 and nz >= 4:
        f[:, 2:nz - 1] = _hflux64(q, Wf, 3, 1, 2, nz - 2)
    if order == 5 and nz >= 6:
        f[:, 3:nz - 2] = _hflux64(q, Wf, 5, 1, 3, nz - 3)
    f[:, nz] = q[:, -1] * W[:, -1] * top
    return f


def _std_stage64(qf, qo, P, tf, hord, vord, hs, corr):
    ny, nz, nx = qo.shape
    e = 1 if corr else 0
    is_, ie, js, je = hs - e, nx - 1 - hs + e, hs - e, ny - 1 - hs + e
    X, Y = slice(is_, ie + 1), slice(js, je + 1)
    U, V, W, G, DJ = P["U"], P["V"], P["W"], P["G"], P["DJ"]

    def fluxes(q, ho, vo, t):
        return (_hflux64(q[Y], U[Y] * t, ho, 2, is_, ie + 1), _hflux64(q[:, :, X], V[:, :, X] * t, ho, 0, js, je + 1),
                _vflux64(q[Y, :, X], W[Y, :, X] * t, vo))

    def div(F):
        return ((F[0][:, :, 1:] - F[0][:, :, :-1]) + (F[1][1:] - F[1][:-1])) / G[Y, :, X] + \
            (F[2][:, 1:] - F[2][:, :-1]) / DJ[Y, :, X]
    F = fluxes(qf, hord, vord, tf)
    if not corr:
        new = qo.clone()
        new[Y, :, X] = qo[Y, :, X] - div(F)
        return new
    up = fluxes(qo, 1, 1, 0.5)
    dq = qo.clone()
    dq[Y, :, X] = qo[Y, :, X] - div(up)
    up = [a + b for a, b in zip(up, fluxes(dq, 1, 1, 0.5))]
    M = [a - b for a, b in zip(F, up)]
    low = qo[Y, :, X] - div(up)
    pos, neg = [m.clamp(min=0) for m in M], [m.clamp(max=0) for m in M]

    def sums(a, b):  # a through the far faces minus b through the near ones
        return ((a[0][:, :, 1:] - b[0][:, :, :-1]) + (a[1][1:] - b[1][:-1])) / G[Y, :, X] + \
            (a[2][:, 1:] - b[2][:, :-1]) / DJ[Y, :, X]
    fin, fout = -sums(neg, pos), sums(pos, neg)
    q = qo[Y, :, X]
    mx, mn = q, q

    def bound(mask, val):
        nonlocal mx, mn
        mx, mn = torch.where(mask, torch.maximum(mx, val), mx), torch.where(mask, torch.minimum(mn, val), mn)
    Uw, Ue = U[Y, :, is_:ie + 1] > 0, U[Y, :, is_ + 1:ie + 2] < 0
    bound(Uw, qo[Y, :, is_ - 1:ie])
    bound(~Uw & Ue, qo[Y, :, is_ + 1:ie + 2])
    Vs, Vn = V[js:je + 1, :, X] > 0, V[js + 1:je + 2, :, X] < 0
    bound(Vs, qo[js - 1:je, :, X])
    bound(~Vs & Vn, qo[js + 1:je + 2, :, X])
    w = W[Y, :, X]
    dn, un = torch.cat([q[:, :1], q[:, :-1]], 1), torch.cat([q[:, 1:], q[:, -1:]], 1)
    wb = torch.cat([torch.zeros_like(w[:, :1]), w[:, :-1]], 1)
    bound(wb > 0, dn)
    bound(w < 0, un)
    si = torch.where(fin > mx - low, ((mx - low) / (fin + 1e-15)).clamp(min=0), torch.ones_like(q))
    so = torch.where(fout > low - mn, ((low - mn) / (fout + 1e-15)).clamp(min=0), torch.ones_like(q))
    out = []
    for m, u, d in ((M[0], up[0], 2), (M[1], up[1], 0), (M[2], up[2], 1)):
        n = q.shape[d]
        inner = _sh(m, d, 1, n)
        s = torch.where(inner > 0, torch.minimum(_sh(si, d, 1, n), _sh(so, d, 0, n - 1)),
                        torch.minimum(_sh(so, d, 1, n), _sh(si, d, 0, n - 1)))
        m = m.clone()
        _sh(m, d, 1, n).mul_(s)
        out.append(m + u)
    new = qo.clone()
    T = (slice(1, -1), slice(None), slice(1, -1))
    new[hs:ny - hs, :, hs:nx - hs] = (q - div(out))[T]
    return new


def _std64(q, P, case, hs):
    st = lambda qf, tf, c: _std_stage64(qf, q, P, tf, case["h_order"], case["v_order"], hs, c)
    if not case["rk3"]:
        return st(q, 1.0, case["flux_corr"] == 1)
    return st(st(st(q, 0.333, False), 0.5, False), 1.0, case["flux_corr"] == 1)


def _halo(case):
    if case["kind"] != "std":
        return 2
    return (max(case["h_order"], case["v_order"]) + (2 if case["flux_corr"] else 0) + 1) // 2


def _advance64(case, size, seed):
    f, dx, dt = _inputs(case, size, seed)
    hs = _halo(case)
    std = case["kind"] == "std"
    P = _winds64(f, dx, dt, case["adv_den"], std)
    flt = _filter64(size[0], size[1], hs, P["U"].device) if case["forced"] else None
    out = {}
    for k, t in f["species"].items():
        q0 = q = t.double()
        for _ in range(case["steps"]):
            if flt is not None:
                q = torch.where(flt == 1, q0, q + flt * dt / 3600.0 * (q0 - q))
            q = _std64(q, P, case, hs) if std else _mpdata64(q, P, case["fct"])
            if case["limits"]:
                q = q.clamp(min=0)
        out[k] = q
    return out


def _balance64(case, size, seed):
    f, dx, dt = _inputs(case, size, seed)
    g = {k: v.double() for k, v in f.items() if k != "species"}
    nx, ny, nz = size
    um, vm, rho, dz, jw = g["u"] * g["jacobian_u"], g["v"] * g["jacobian_v"], g["density"], g["advection_dz"], g["jacobian_w"]
    if case["adv_den"]:
        um[:, :, 1:-1] *= 0.5 * (rho[:, :, 1:] + rho[:, :, :-1])
        um[:, :, 0] *= 1.5 * rho[:, :, 0] - 0.5 * rho[:, :, 1]
        um[:, :, -1] *= 1.5 * rho[:, :, -1] - 0.5 * rho[:, :, -2]
        vm[1:-1] *= 0.5 * (rho[1:] + rho[:-1])
        vm[0] *= 1.5 * rho[0] - 0.5 * rho[1]
        vm[-1] *= 1.5 * rho[-1] - 0.5 * rho[-2]
    div = ((um[:, :, 1:] - um[:, :, :-1]) + (vm[1:] - vm[:-1])) / dx
    ri = torch.ones_like(rho)
    if case["adv_den"]:
        ri[:, :-1] = (rho[:, :-1] * dz[:, :-1] + rho[:, 1:] * dz[:, 1:]) / (dz[:, :-1] + dz[:, 1:])
        ri[:, -1] = rho[:, -1]
    w = -torch.cumsum(div * dz, 1) / (jw * ri)
    keep = torch.zeros_like(w)
    I = (slice(1, ny - 1), slice(None), slice(1, nx - 1))    # one column beyond the tile on each side (halo 2)
    keep[I] = w[I]
    w = keep
    wb = torch.cat([w[:, :1], w[:, :-1]], 1)
    T = (slice(2, ny - 2), slice(None), slice(2, nx - 2))
    u, v = g["u"].abs(), g["v"].abs()
    rate = torch.maximum(torch.maximum(u[:, :, 1:], u[:, :, :-1]) / dx, torch.maximum(v[1:], v[:-1]) / dx)
    rate = torch.maximum(rate, torch.maximum(w.abs(), wb.abs()) / dz[:1, :, :1])
    return {"w": w, "dt": 0.9 / float(rate[T].max())}


def _satmr64(T, p):
    ice = T < 273.15
    a, b = torch.where(ice, 21.8745584, 17.2693882).double(), torch.where(ice, 7.66, 35.86).double()
    e = 610.78 * torch.exp(a * (T - 273.16) / (T - b))
    e = torch.where(p - e <= 0, p * 0.99999, e)
    return 0.6219907 * e / (p - e)


def _change64(on, T, q1, qmax, q2, heat, rate):
    d = (qmax - q2) * rate
    d = torch.minimum(torch.minimum(d, q1), (qmax - q2) * 0.99)
    d = torch.where(on, d, torch.zeros_like(d))
    return T + d * heat / 1006.0, (q1 - d).clamp(min=0), q2 + d


def _microphysics64(case, size, seed):
    f, dx, dt = _inputs(case, size, seed)
    hs = 2
    I = (slice(hs, size[1] - hs), slice(None), slice(hs, size[0] - hs))
    full = {k: v.double() for k, v in f["species"].items()}
    p, ex, rho, dz = (f[k].double()[I] for k in ("pressure", "exner", "density", "dz_mass"))
    th, qv, qc, qr, qs = (full[k][I].clone() for k in ("theta", "qv", "qc", "qr", "qs"))
    c2s, c2r, tiny = math.exp(-dt / 2000.0), math.exp(-dt / 500.0), 1e-30
    rain, snow = torch.zeros_like(th[:, 0]), torch.zeros_like(th[:, 0])
    nz = size[2]
    for _ in range(case["steps"]):
        T = th * ex
        evap = -(2.26e6 + (373.15 - T) * 2400.0)
        v2t, T0, v0, c0 = -evap / 1006.0, T, qv, qc
        last, sat = qv + 2e-4, torch.zeros_like(qv)
        it = torch.zeros_like(qv, dtype=torch.int32)
        for n in range(15):
            on = (last - qv).abs() > 1e-4
            if not bool(on.any()):
                break
            it += on.int()
            last = torch.where(on, qv, last)
            sat = torch.where(on, _satmr64(T, p), sat)
            ex1 = torch.where(on & (qv > sat), (qv - sat) * 0.5, torch.zeros_like(qv))
            lack = torch.where(on & ~(qv > sat) & (qc > 0), torch.minimum((sat - qv) * 0.5, qc), torch.zeros_like(qv))
            T, qv, qc = T + (ex1 - lack) * v2t, qv - ex1 + lack, qc + ex1 - lack
        bad = it == 15
        qv, T, qc = torch.where(bad, _satmr64(T0, p), qv), torch.where(bad, T0, T), torch.where(bad, c0, qc).clamp(min=0)
        any_ = (qc + qr + qs) > tiny
        cloud = any_ & (qc > tiny)
        warm, cold = cloud & (T > 273.15), cloud & ~(T > 273.15)
        d = torch.where(qc > 1e-4, qc * (1 - c2r), torch.zeros_like(qc))
        d = torch.where(warm, d, torch.zeros_like(d))
        qr = qr + d
        d2 = torch.where(cold & (qc > 1e-4), qc * (1 - c2s), torch.zeros_like(qc))
        qc, qs = qc - d - d2, qs + d2
        T, qs, qr = _change64(warm & (qs > tiny), T, qs, 100.0, qr, -3.34e5, c2r)
        dry = any_ & (qv < sat)
        T, qr, qv = _change64(dry & (qr > tiny), T, qr, sat, qv, evap, c2r / 2)
        T, qs, qv = _change64(dry & (qs > tiny), T, qs, sat, qv, evap - 3.34e5, c2s / 2)
        for which in (0, 1):
            q, fall, c = (qr, 10.0, c2r) if which == 0 else (qs, 1.5, c2s)
            on = q.amax(1) > tiny
            cfl = torch.ceil((dt / dz * fall).amax(1))
            for sub in range(int(cfl.max())):
                act = (on & (sub < cfl))[:, None]
                amount = torch.where(act, (dt * fall / cfl)[:, None] * q * rho, torch.zeros_like(q))
                q = q - amount / (rho * dz)
                q[:, :-1] += amount[:, 1:] / (rho * dz)[:, :-1]
                rain = rain + amount[:, 0]
                if which:
                    snow = snow + amount[:, 0]
                sat2 = _satmr64(T, p)
                heat = -(2.26e6 + (373.15 - T) * 2400.0) - (3.34e5 if which else 0.0)
                T, q, qv = _change64(act & (q > tiny) & (qv < sat2), T, q, sat2, qv, heat, (c / (2 * cfl))[:, None])
            if which == 0:
                qr = q
            else:
                qs = q
        th = T / ex
    for k, v in zip(("theta", "qv", "qc", "qr", "qs"), (th, qv, qc, qr, qs)):
        full[k][I] = v
    acc = []
    for a in (rain, snow):
        t = torch.zeros(size[1], size[0], dtype=torch.float64, device=a.device)
        t[hs:size[1] - hs, hs:size[0] - hs] = a
        acc.append(t)
    return {**full, "rain": acc[0], "snow": acc[1]}


def exact(case, seed):
    sizes = _sizes(case, seed)
    if sum(x * y * z for x, y, z in sizes) * case["species"] > 2e8:
        return None
    if case["kind"] == "winds":
        return _balance64(case, sizes[0], seed)
    if case["kind"] == "mp":
        return _microphysics64(case, sizes[0], seed)
    outs = [_advance64(case, size, seed + 7919 * i) for i, size in enumerate(sizes)]
    if case["kind"] == "batch":
        return {k: torch.cat([o[k].reshape(-1) for o in outs]) for k in outs[0]}
    return outs[0]
