"""Workloads of the LES time step on the GPU, with their inputs, outputs and
64-bit values.

Every case is something a program that uses this library does in its time
loop, through the entry points it would call:

  step      one time step of a device-resident domain (GpuLes.step); the
            state stays on the device and is read there (GpuLes.field);
  refined   the same with the FP64-refined pressure solve;
  coupled   one step of a host-coupled run: the inflow profile goes up, the
            step runs, the halo ring of the seven combined arrays goes down
            and back up through page-locked buffers, the step record is read;
  ensemble  one step of several uneven domains (Ensemble.step);
  gradient  the checkpointed gradient of the resolved TKE over a few steps
            (tke_gradient): forward steps, recomputation, step adjoints;
  press     the drop-in pressure routine on host arrays (les_press_).

The inputs are a flow in mid-run: a logarithmic inflow over a block terrain
with smooth random eddies, made from the seed on the GPU.  exact() evaluates
the reference's Fortran statements in FP64 with torch, materialised ghosts
and all.
"""
import ctypes as C
import math

import numpy as np
import torch

import les_halo_b200 as lh
from les_halo_b200 import abi

NMAXP = 50  # SOR iteration cap, press.f95:108
PJUGE = 0.0001
ALPHA, BETA, RO, CS0 = -10.0, -1.0, 1.1763, 0.1
VN = 15.83e-6
GRAD = ("u", "v", "w", "p", "usum", "f", "fold", "gold", "hold")
STATE = ("u", "v", "w", "p", "usum", "vsum", "wsum", "f", "g", "h", "fold", "gold", "hold", "sm")


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest domain in use (smoke runs, unit set-ups): latency
        {"name": "step_24x20x16", "kind": "step", "ip": 24, "jp": 20, "kp": 16, "dx": 4.0, "dt": 0.05},
        # a small ragged domain, nothing a multiple of anything
        {"name": "step_61x47x35", "kind": "step", "ip": 61, "jp": 47, "kp": 35, "dx": 5.0, "dt": 0.05},
        # the reference's own domain and spacing
        {"name": "step_150x150x90", "kind": "step", "ip": 150, "jp": 150, "kp": 90, "dx": 20.0, "dt": 0.2},
        # a mid-size domain with odd extents
        {"name": "step_257x203x61", "kind": "step", "ip": 257, "jp": 203, "kp": 61, "dx": 4.0, "dt": 0.05},
        # four times the reference's area: the step of a district
        {"name": "step_300x300x120", "kind": "step", "ip": 300, "jp": 300, "kp": 120, "dx": 4.0, "dt": 0.05},
        # the headline domain
        {"name": "step_600x600x120", "kind": "step", "ip": 600, "jp": 600, "kp": 120, "dx": 4.0, "dt": 0.05},
        # a step whose pressure is solved to FP64 rounding
        {"name": "refined_300x300x90", "kind": "refined", "ip": 300, "jp": 300, "kp": 90, "dx": 4.0, "dt": 0.05},
        # a domain coupled to a host model through its halo
        {"name": "coupled_200x200x80", "kind": "coupled", "ip": 200, "jp": 200, "kp": 80, "dx": 4.0, "dt": 0.05},
        # a parameter study: domains of different sizes advanced together
        {"name": "ensemble_8", "kind": "ensemble", "members": 8, "lo": 96, "hi": 256, "kp": 80, "pick": 3,
         "dx": 4.0, "dt": 0.05},
        # sensitivities: forward and backward in time
        {"name": "gradient_96x96x48", "kind": "gradient", "ip": 96, "jp": 96, "kp": 48, "nt": 4, "ckpt": 2,
         "dx": 4.0, "dt": 0.05},
        # a Fortran host that calls the pressure routine on its own arrays
        {"name": "press_150x150x90", "kind": "press", "ip": 150, "jp": 150, "kp": 90, "dx": 20.0, "dt": 0.2},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def even(lo, hi):
        """An extent the spectral solve takes: even, prime factors up to 13."""
        n = 2 * size(lo // 2, hi // 2)
        while True:
            m = n
            for q in (2, 3, 5, 7, 11, 13):
                while m % q == 0:
                    m //= q
            if m == 1:
                return n
            n -= 2

    kind = rng.choice(["step"] * 6 + ["refined", "coupled", "ensemble", "gradient", "press"])
    c = {"kind": kind, "dx": rng.choice([4.0, 5.0, 20.0])}
    c["dt"] = 0.2 if c["dx"] == 20.0 else 0.05
    if kind == "ensemble":
        c.update(members=rng.randint(2, 8), lo=rng.randint(48, 128), hi=rng.randint(160, 256), kp=rng.randint(30, 90),
                 pick=rng.randint(0, 10 ** 6))
    elif kind == "gradient":
        c.update(ip=size(24, 128), jp=size(20, 128), kp=size(16, 60), nt=rng.randint(2, 4))
        c["ckpt"] = rng.randint(1, c["nt"])
    elif kind == "refined":
        c.update(ip=even(40, 320), jp=even(40, 320), kp=size(20, 120))
    elif kind == "press":
        c.update(ip=size(24, 200), jp=size(20, 200), kp=size(16, 100))
    elif kind == "coupled":
        c.update(ip=size(32, 300), jp=size(32, 300), kp=size(20, 100))
    else:
        c.update(ip=size(20, 600), jp=size(16, 600))
        c["kp"] = size(12, min(140, 43200000 // (c["ip"] * c["jp"])))
    return c


def _members(case):
    """(ip, jp, kp) of an ensemble's members."""
    r = np.random.RandomState(case["pick"] % (2 ** 31))
    return [(int(r.randint(case["lo"], case["hi"] + 1)), int(r.randint(case["lo"], case["hi"] + 1)), case["kp"])
            for _ in range(case["members"])]


def work(case):
    """A step reads u v w p, the sums, f g h, fold gold hold and three masks
    and writes all but the masks, and sm; about 430 operations a cell beside
    the SOR's 19 a cell and iteration."""
    step_b, step_f, press_f = 4.0 * (16 + 14), 430.0 + 19.0 * NMAXP, 20.0 + 19.0 * NMAXP
    kind = case["kind"]
    if kind == "ensemble":
        n = sum(a * b * c for a, b, c in _members(case))
        return {"bytes": step_b * n, "flops": step_f * n}
    n = float(case["ip"] * case["jp"] * case["kp"])
    if kind == "press":  # u v w f g h p in, f g h p rhs out
        return {"bytes": 4.0 * (7 + 5) * n, "flops": press_f * n}
    if kind == "gradient":  # the state in, its adjoint out; a step and about twice its work back, each step
        return {"bytes": 2 * 4.0 * 13 * n, "flops": 3 * step_f * n * case["nt"]}
    if kind == "refined":  # beside the step: residual, transforms and line solves in FP64
        return {"bytes": step_b * n, "flops": (step_f + 250.0) * n}
    return {"bytes": step_b * n, "flops": step_f * n}


# --------------------------------------------------------------------------
# inputs (plain torch; boxes are [k][j][i] with index -1 first, two planes
# past the end)
# --------------------------------------------------------------------------
def _grid(case):
    """The 1-D tables in FP32 (grid.f95:22-82, init.f95:82-107): uniform x
    and y, 5% stretching in z up to 16 m."""
    ip, jp, kp = case["ip"], case["jp"], case["kp"]
    one = np.float32
    dz = np.empty(kp + 2, one)
    dz[0] = 2.5 if case["dx"] == 20.0 else 2.0
    for k in range(1, kp + 2):
        dz[k] = min(one(dz[k - 1] * one(1.05)), one(16.0))
    dzn = np.zeros(kp + 4, one)  # -1..kp+2
    dzn[2:kp + 2] = dz[:kp]
    dzn[kp + 2:] = dz[kp - 1]
    dzn[:2] = dz[0]
    dzs = np.zeros(kp + 4, one)
    dzs[1:kp + 2] = dzn[2:kp + 3] / one(2) + dzn[1:kp + 2] / one(2)
    dzs[kp + 2:] = dzs[kp + 1]
    dzs[0] = dzs[1]
    z2 = np.zeros(kp + 2, one)  # 1..kp+2
    z2[0] = dzn[2]
    for k in range(1, kp + 2):
        z2[k] = z2[k - 1] + dzn[k + 2]
    d = one(case["dx"])
    t = {"dx1": np.full(ip + 3, d), "dy1": np.full(jp + 2, d), "dxs": np.full(ip + 1, d), "dys": np.full(jp + 1, d),
         "dzn": dzn, "dzs": dzs, "z2": z2}
    for a, s, lo in (("2", t["dxs"], 0), ("3", t["dys"], 0), ("4", dzs[1:kp + 2], 0)):
        t["cn%ss" % a] = one(2) / (s[:-1] * (s[:-1] + s[1:]))
        t["cn%sl" % a] = one(2) / (s[1:] * (s[:-1] + s[1:]))
    return t


def _fields(case, seed, grid, dev):
    """FP32 state boxes, masks and inflow profile of a flow in mid-run."""
    ip, jp, kp = case["ip"], case["jp"], case["kp"]
    gen = torch.Generator(device=dev).manual_seed(int(seed) * 7919 + ip * 31 + jp * 17 + kp)
    r = np.random.RandomState((int(seed) * 104729 + ip + 1000 * jp) % (2 ** 31))
    z = torch.tensor(grid["z2"][:kp] + 0.5 * grid["dzn"][2:kp + 2], device=dev)
    i = torch.arange(-1, ip + 3, device=dev, dtype=torch.float32).view(1, 1, -1)
    j = torch.arange(-1, jp + 3, device=dev, dtype=torch.float32).view(1, -1, 1)
    k = torch.arange(-1, kp + 3, device=dev, dtype=torch.float32).view(-1, 1, 1)

    def eddies(amp):
        a = torch.zeros((kp + 4, jp + 4, ip + 4), device=dev)
        for _ in range(3):  # periodic in j
            kx, ky, kz = r.uniform(0.05, 0.5), 2 * math.pi * r.randint(1, max(2, jp // 12)) / jp, r.uniform(0.05, 0.5)
            a += torch.sin((kx * i + r.uniform(0, 6.28)) + ky * j) * torch.cos(kz * k + r.uniform(0, 6.28))
        a += 0.1 * torch.randn(a.shape, generator=gen, device=dev)
        return a.mul_(amp)

    # block terrain: about 30% of the area built, heights up to half the domain
    top = float(grid["z2"][kp - 1])
    zbm = np.zeros((jp, ip), np.float32)
    margin = max(2, ip // 16)
    for _ in range(int(0.30 * ip * jp / 16) + 1):
        wx, wy = r.randint(2, 7), r.randint(2, 7)
        i0 = r.randint(margin, max(margin + 1, ip - margin - wx))
        rows = (r.randint(0, jp) + np.arange(wy)) % jp
        cols = np.arange(i0, min(i0 + wx, ip - margin))
        hgt = min(max(20.0 * math.exp(0.5 * r.randn() - 0.125), 4.0), 0.5 * top)
        zbm[np.ix_(rows, cols)] = np.maximum(zbm[np.ix_(rows, cols)], np.float32(hgt))
    built = torch.zeros((kp + 4, jp + 4, ip + 4), device=dev)
    built[2:kp + 2, 2:jp + 2, 2:ip + 2] = (torch.tensor(zbm, device=dev)[None] > z.view(-1, 1, 1)).float()
    prof = (0.3 / 0.4) * torch.log(z / 0.1)
    wind = prof.view(-1, 1) * (1 + 0.02 * (2 * torch.rand((kp, jp), generator=gen, device=dev) - 1))
    full = torch.cat([prof[:1], prof[:1], prof, prof[-1:], prof[-1:]]).view(-1, 1, 1)
    A = {"bmask1": built, "wind_profile": wind.float()}
    A["u"] = (full * (1 + eddies(0.08))) * (1 - 0.9 * built)
    A["v"] = eddies(0.3) * (1 - 0.9 * built)
    A["w"] = eddies(0.2) * (1 - 0.9 * built)
    A["p"] = eddies(0.3)
    for n in ("f", "g", "h", "fold", "gold", "hold"):
        A[n] = eddies(0.02)
    for n in ("usum", "vsum", "wsum"):
        A[n] = eddies(0.05) * built
    p = A["p"]  # the ghosts press leaves (boundp.f95)
    _boundp1(p, ip, jp)
    _boundp2(p, kp)
    return A


_LO = {"u": (0, -1, 0), "v": (0, -1, 0), "w": (0, -1, -1), "p": (0, 0, 0), "fold": (1, 1, 1), "gold": (1, 1, 1),
       "hold": (1, 1, 1), "bmask1": (-1, 0, 0), "cmask1": (0, -1, 0), "dmask1": (0, 0, 0)}
_HI = {"u": (1, 1, 1), "v": (1, 1, 1), "w": (1, 1, 1), "p": (2, 2, 1), "bmask1": (1, 1, 1), "cmask1": (1, 1, 1),
       "dmask1": (1, 1, 1)}


def _host(case, A, names):
    """Fortran-layout host arrays (bounds of main_ocl.f95:41-167) of boxes."""
    out = {}
    for n in names:
        (li, lj, lk), (hi, hj, hk) = _LO.get(n, (0, 0, 0)), _HI.get(n, (0, 0, 0))
        b = A["bmask1" if n in ("cmask1", "dmask1") else n]
        v = b[lk + 1:case["kp"] + hk + 2, lj + 1:case["jp"] + hj + 2, li + 1:case["ip"] + hi + 2]
        out[n] = v.contiguous().cpu().numpy().transpose(2, 1, 0)
    return out


def _les_case(case, seed, nmaxp=NMAXP, pjuge=PJUGE):
    """The LesCase a program would hold (host arrays), ready for GpuLes."""
    grid = _grid(case)
    A = _fields(case, seed, grid, "cuda")
    prm = lh.default_params(case["ip"], case["jp"], case["kp"], dt=case["dt"], inflow="external", nmaxp=nmaxp)
    prm.pjuge = pjuge
    arr = _host(case, A, ["u", "v", "w", "p", "usum", "vsum", "wsum", "f", "g", "h", "fold", "gold", "hold",
                          "bmask1", "cmask1", "dmask1"])
    arr["wind_profile"] = A["wind_profile"].cpu().numpy().T
    arr.update({n: np.ascontiguousarray(t) for n, t in grid.items()})
    return lh.LesCase(case["ip"], case["jp"], case["kp"], prm, arr)


class _Device:
    """A device pointer as a CUDA array; keeps the context that owns it."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


def _views(gpu, names):
    """The interiors of state fields, on the device, [k][j][i]."""
    c, out = gpu.case, {}
    for n in names:
        ptr, ox, si, sj, sk = gpu.field(n)
        box = torch.as_tensor(_Device(gpu, ptr, (sk, sj, si)), device="cuda")
        out[n] = box[2:c.kp + 2, 2:c.jp + 2, ox + 1:ox + 1 + c.ip]
    return out


# --------------------------------------------------------------------------
# what a program has in hand, and one pass
# --------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        mem = []
        for q, (ip, jp, kp) in enumerate(_members(case)):
            mem.append(lh.GpuLes(_les_case(dict(case, ip=ip, jp=jp, kp=kp), seed + 100 * q)))
        return {"kind": kind, "n": 2, "members": mem, "ens": lh.Ensemble(mem),
                "views": [_views(m, ("u", "v", "w", "p")) for m in mem]}
    if kind == "press":
        grid = _grid(case)
        A = _fields(case, seed, grid, "cuda")
        arr = _host(case, A, ["u", "v", "w", "p", "f", "g", "h"])
        arr.update({n: np.ascontiguousarray(t) for n, t in grid.items()})
        ip, jp, kp = case["ip"], case["jp"], case["kp"]
        arr["rhs"] = np.zeros((ip + 2, jp + 2, kp + 2), np.float32, order="F")
        arr["cn1"] = np.asfortranarray(_cn1(grid, np.float32))
        arr["p0"] = arr["p"].copy(order="F")
        ints = {n: C.c_int(v) for n, v in (("km", kp), ("jm", jp), ("im", ip), ("n", 2), ("nmax", 200), ("it", 0))}
        return {"kind": kind, "arr": arr, "ints": ints, "dt": C.c_float(case["dt"])}
    if kind == "gradient":
        lc = _les_case(case, seed, nmaxp=NMAXP, pjuge=-1.0)
        gpu = lh.GpuLes(lc)
        nck = -(-case["nt"] // case["ckpt"])
        adj = lh.GpuAdjoint(gpu, nck + case["ckpt"] + 1, NMAXP)
        adj.save(nck + case["ckpt"])
        return {"kind": kind, "gpu": gpu, "adj": adj, "slot": nck + case["ckpt"], "nt": case["nt"],
                "ckpt": case["ckpt"], "box": _box(case)}
    gpu = lh.GpuLes(_les_case(case, seed))
    s = {"kind": kind, "gpu": gpu, "n": 2, "views": _views(gpu, STATE)}
    if kind == "refined":
        gpu.press_refine_fp64(2, 0, 1e-9)
        s["views"] = _views(gpu, ("u", "v", "w", "p", "f", "g", "h"))
    if kind == "coupled":
        s["halo"] = [torch.zeros(abi.lib().les_ctx_halo_floats(gpu.ctx, w), dtype=torch.float32, pin_memory=True)
                     for w in range(7)]
        s["wind"] = gpu.case.a("wind_profile").copy(order="F")
    return s


def _box(case):
    return ((2, case["ip"] // 2), (2, case["jp"] // 2), (1, max(2, case["kp"] // 3)))


def run(state):
    kind = state["kind"]
    if kind == "ensemble":
        state["ens"].step(state["n"])
        state["n"] += 1
        return state["views"]
    if kind == "press":
        a, q = state["arr"], state["ints"]
        np.copyto(a["p"], a["p0"])  # the step's pressure, changed in place

        def P(n):
            return a[n].ctypes.data

        abi.check(abi.lib().les_press_(
            C.byref(q["km"]), C.byref(q["jm"]), C.byref(q["im"]), P("rhs"), P("u"), P("dx1"), P("v"), P("dy1"), P("w"),
            P("dzn"), P("f"), P("g"), P("h"), C.byref(state["dt"]), P("cn1"), P("cn2l"), P("p"), P("cn2s"), P("cn3l"),
            P("cn3s"), P("cn4l"), P("cn4s"), C.byref(q["n"]), C.byref(q["nmax"]), C.byref(q["it"])))
        return {"p": a["p"][1:-2, 1:-2, 1:-1], "rhs": a["rhs"][1:-1, 1:-1, 1:-1], "iters": q["it"].value}
    gpu = state["gpu"]
    if kind == "gradient":
        state["adj"].load(state["slot"])
        J, grad = lh.tke_gradient(gpu, state["adj"], 2, state["nt"], state["box"], state["ckpt"])
        c, out = gpu.case, {"J": J, "wp": grad["wp"]}
        for n in GRAD:
            i, j, k = (1 - lo for lo in _LO.get(n, (0, 0, 0)))
            out[n] = grad["state"][n][i:i + c.ip, j:j + c.jp, k:k + c.kp]
        return out
    if kind == "coupled":
        gpu.set_wind_profile(state["wind"])
    gpu.step(state["n"])
    state["n"] += 1
    if kind != "coupled":
        return state["views"]
    L, bufs = abi.lib(), state["halo"]
    for w in range(7):
        abi.check(L.les_ctx_halo_read(gpu.ctx, w, bufs[w].data_ptr()))
    for w in range(7):
        abi.check(L.les_ctx_halo_write(gpu.ctx, w, bufs[w].data_ptr()))
    m = gpu.metrics()
    return {"state": state["views"], "halo": bufs, "uout": m["uout"], "rhsav": m["rhsav"], "iters": m["sor_iters"]}


# --------------------------------------------------------------------------
# the same in 64 bits: the reference's Fortran statements on torch boxes
# --------------------------------------------------------------------------
def _cn1(g, dtype):
    """cn1(1:ip,1:jp,1:kp), init.f95:87-93."""
    dxs, dys, dzs = (np.asarray(g[n], dtype) for n in ("dxs", "dys", "dzs"))
    dzs = dzs[1:-2]
    a, b, c = (dtype(2) / (s[:-1] * s[1:]) for s in (dxs, dys, dzs))
    return dtype(1) / (a[:, None, None] + b[None, :, None] + c[None, None, :])


def _r(a, I, J, K):
    """a(I, J, K) over inclusive Fortran ranges."""
    return a[K[0] + 1:K[1] + 2, J[0] + 1:J[1] + 2, I[0] + 1:I[1] + 2]


def _boundp1(p, im, jm):
    """boundp.f95:23-44 (the copies' clones keep torch's reverse mode)."""
    p[:, :, 1] = p[:, :, 2].clone()
    p[:, :, im + 2] = p[:, :, im + 1].clone()
    p[:, 1, :] = p[:, jm + 1, :].clone()
    p[:, jm + 2, :] = p[:, 2, :].clone()


def _boundp2(p, km):
    """boundp.f95:5-21."""
    p[1] = p[2].clone()
    p[km + 2] = p[km + 1].clone()


class _Step64:
    """One time step (main_ocl.f95:264-299) on FP64 boxes."""

    def __init__(self, case, grid, dev, nmaxp, pjuge):
        self.c, self.nmaxp, self.pjuge = case, nmaxp, pjuge
        T = lambda n: torch.tensor(np.asarray(grid[n], np.float64), device=dev)  # noqa: E731
        self.t = {n: T(n) for n in ("dx1", "dy1", "dzn", "dzs", "dxs", "dys", "cn2l", "cn2s", "cn3l", "cn3s", "cn4l",
                                    "cn4s")}
        # the Poisson tables are FP32 inputs; cn1 is their FP32 combination
        self.cn1 = torch.tensor(_cn1(grid, np.float32).astype(np.float64), device=dev).permute(2, 1, 0)
        self.dev = dev
        f = np.float32
        self.dt, self.ro, self.vn, self.cs0 = float(f(case["dt"])), float(f(RO)), float(f(VN)), float(f(CS0))

    def x(self, n, lo, rng):
        return self.t[n][rng[0] - lo:rng[1] - lo + 1].view(1, 1, -1)

    def y(self, n, lo, rng):
        return self.t[n][rng[0] - lo:rng[1] - lo + 1].view(1, -1, 1)

    def z(self, n, lo, rng):
        return self.t[n][rng[0] - lo:rng[1] - lo + 1].view(-1, 1, 1)

    def __call__(self, A, wind):
        A = {n: a.clone() for n, a in A.items()}
        self.velnw(A)
        self.bondv1(A, wind)
        D, Cv = self.vel2(A)
        self.velfg(A, D, Cv)
        del Cv
        self.feedbf(A)
        self.les(A, D)
        del D
        self.adam(A)
        self.press(A)
        return A

    def velnw(self, A):
        c = self.c
        I, J, K = (1, c["ip"]), (1, c["jp"]), (1, c["kp"])
        K1 = (1, c["kp"] - 1)
        p, dt = A["p"], self.dt
        P = lambda di, dj, dk, K=K: _r(p, (1 + di, I[1] + di), (1 + dj, J[1] + dj), (1 + dk, K[1] + dk))  # noqa: E731
        pc = P(0, 0, 0)
        du = dt * (_r(A["f"], I, J, K) - (P(1, 0, 0) - pc) / self.ro / self.x("dxs", 0, I))
        dv = dt * (_r(A["g"], I, J, K) - (P(0, 1, 0) - pc) / self.ro / self.y("dys", 0, J))
        dw = dt * (_r(A["h"], I, J, K1) - (P(0, 0, 1, K1) - P(0, 0, 0, K1)) / self.ro / self.z("dzs", -1, K1))
        _r(A["u"], I, J, K).add_(du)
        _r(A["v"], I, J, K).add_(dv)
        _r(A["w"], I, J, K1).add_(dw)

    def bondv1(self, A, wind):
        c, dt = self.c, self.dt
        im, jm, km = c["ip"], c["jp"], c["kp"]
        J, K = (1, jm), (1, km)
        u, v, w = A["u"], A["v"], A["w"]
        for i in (0, 1):
            _r(u, (i, i), J, K).copy_(wind.unsqueeze(2))
            _r(v, (i, i), J, K).zero_()
            _r(w, (i, i), J, K).zero_()
        face = _r(u, (im, im), J, K).clone()
        zero = torch.zeros((), dtype=u.dtype, device=u.device)
        a = dt * (torch.maximum(face.max(), zero) + torch.minimum(face.min(), zero)) / 2.0 / self.t["dxs"][im]
        e = (im, im)
        _r(u, e, J, K).copy_(_r(u, e, J, K) - a * (_r(u, e, J, K) - _r(u, (im - 1, im - 1), J, K)))
        e1 = (im + 1, im + 1)
        for q in (v, w):
            _r(q, e1, J, K).copy_(_r(q, e1, J, K) - a * (_r(q, e1, J, K) - _r(q, e, J, K)))
        I = (0, im + 1)
        for q, k1 in ((u, km + 1), (v, km + 1), (w, km)):
            _r(q, I, (0, 0), (0, k1)).copy_(_r(q, I, (jm, jm), (0, k1)).clone())
            _r(q, I, (jm + 1, jm + 1), (0, k1)).copy_(_r(q, I, (1, 1), (0, k1)).clone())
        Jg = (0, jm + 1)
        for q in (u, v):
            _r(q, I, Jg, (0, 0)).copy_(-_r(q, I, Jg, (1, 1)))
            _r(q, I, Jg, (km + 1, km + 1)).copy_(_r(q, I, Jg, (km, km)).clone())
        _r(w, I, (-1, jm + 1), (0, 0)).zero_()
        _r(w, I, (-1, jm + 1), (km, km)).zero_()
        # the loop's i = -1 aliases onto these (bondv1.f95:132-137)
        _r(w, e1, (jm + 1, jm + 1), (-1, -1)).zero_()
        _r(w, e1, (jm + 1, jm + 1), (km - 1, km - 1)).zero_()

    def vel2(self, A):
        c = self.c
        im, jm, km = c["ip"], c["jp"], c["kp"]
        I, J = (1, im), (1, jm)
        shape = A["u"].shape
        X = lambda r: self.x("dx1", -1, r)  # noqa: E731
        Y = lambda r: self.y("dy1", 0, r)  # noqa: E731
        Z = lambda r: self.z("dzn", -1, r)  # noqa: E731
        sh = lambda r, d: (r[0] + d, r[1] + d)  # noqa: E731
        D, Cv = {}, {}

        def face(n, K, nou, diu):
            d = torch.zeros(shape, dtype=A["u"].dtype, device=self.dev)
            cv = torch.zeros_like(d)
            dv = diu(K)
            _r(d, I, J, K).copy_(dv)
            _r(cv, I, J, K).copy_(nou(K) * dv)
            D[n], Cv[n] = d, cv

        def at(q):
            return lambda K, di=0, dj=0, dk=0: _r(A[q], sh(I, di), sh(J, dj), sh(K, dk))

        U, V, W = at("u"), at("v"), at("w")
        sx, sxm = X(sh(I, 1)) + X(I), X(sh(I, -1)) + X(I)
        sy, sym = Y(sh(J, 1)) + Y(J), Y(sh(J, -1)) + Y(J)
        mx = lambda q, K, dj, dk: (X(sh(I, 1)) * q(K, 0, dj, dk) + X(I) * q(K, 1, dj, dk)) / sx  # noqa: E731
        my = lambda q, K, di, dk: (Y(sh(J, 1)) * q(K, di, 0, dk) + Y(J) * q(K, di, 1, dk)) / sy  # noqa: E731

        def mz(q, K, di, dj):
            return (Z(sh(K, 1)) * q(K, di, dj, 0) + Z(K) * q(K, di, dj, 1)) / (Z(K) + Z(sh(K, 1)))

        K0, Kp, Km = (1, km), (1, km + 1), (1, km - 1)
        face(1, K0, lambda K: (U(K, -1) + U(K)) / 2, lambda K: (U(K) - U(K, -1)) / X(I))
        face(5, K0, lambda K: (V(K, 0, -1) + V(K)) / 2, lambda K: (V(K) - V(K, 0, -1)) / Y(J))
        face(9, K0, lambda K: (W(K, 0, 0, -1) + W(K)) / 2, lambda K: (W(K) - W(K, 0, 0, -1)) / Z(K))
        face(2, K0, lambda K: mx(V, K, -1, 0), lambda K: 2 * (U(K) - U(K, 0, -1)) / sym)
        zs = lambda K: self.z("dzs", -1, sh(K, -1))  # noqa: E731
        face(3, Kp, lambda K: mx(W, K, 0, -1), lambda K: (U(K) - U(K, 0, 0, -1)) / zs(K))
        face(4, K0, lambda K: my(U, K, -1, 0), lambda K: 2 * (V(K) - V(K, -1)) / sxm)
        face(6, Kp, lambda K: my(W, K, 0, -1), lambda K: (V(K) - V(K, 0, 0, -1)) / zs(K))
        face(7, Km, lambda K: mz(U, K, -1, 0), lambda K: 2 * (W(K) - W(K, -1)) / sxm)
        face(8, Km, lambda K: mz(V, K, 0, -1), lambda K: 2 * (W(K) - W(K, 0, -1)) / sym)
        # boundary copies, vel2.f95:125-188
        e, e1 = (im, im), (im + 1, im + 1)
        for n, K in ((1, K0), (4, K0), (7, Km)):
            for B in (D, Cv):
                _r(B[n], e1, J, K).copy_(_r(B[n], e, J, K).clone())
        for n, K in ((2, K0), (5, K0), (8, Km)):
            for B in (D, Cv):
                _r(B[n], I, (0, 0), K).copy_(_r(B[n], I, (jm, jm), K).clone())
                _r(B[n], I, (jm + 1, jm + 1), K).copy_(_r(B[n], I, (1, 1), K).clone())
        for n in (2, 3):
            _r(D[n], e1, (1, jm + 1), Kp).copy_(_r(D[n], e, (1, jm + 1), Kp).clone())
        for n in (4, 6):
            _r(D[n], (1, im + 1), (0, 0), Kp).copy_(_r(D[n], (1, im + 1), (jm, jm), Kp).clone())
        return D, Cv

    def _cells(self, K=None):
        c = self.c
        I, J = (1, c["ip"]), (1, c["jp"])
        K = K or (1, c["kp"])
        return I, J, K, lambda a, di=0, dj=0, dk=0: _r(a, (I[0] + di, I[1] + di), (J[0] + dj, J[1] + dj),
                                                       (K[0] + dk, K[1] + dk))

    def velfg(self, A, D, Cv):
        for K, parts in (((1, self.c["kp"]), "fg"), ((1, self.c["kp"] - 1), "h")):
            I, J, K, at = self._cells(K)
            sh = lambda r, d: (r[0] + d, r[1] + d)  # noqa: E731
            x0, x1 = self.x("dx1", -1, I), self.x("dx1", -1, sh(I, 1))
            y0, y1 = self.y("dy1", 0, J), self.y("dy1", 0, sh(J, 1))
            z0, z1, zs = self.z("dzn", -1, K), self.z("dzn", -1, sh(K, 1)), self.z("dzs", -1, K)
            if "f" in parts:
                cov = ((x1 * at(Cv[1]) + x0 * at(Cv[1], 1)) / (x0 + x1) + (at(Cv[2]) + at(Cv[2], 0, 1)) / 2 +
                       (at(Cv[3]) + at(Cv[3], 0, 0, 1)) / 2)
                dfu = (2 * (at(D[1], 1) - at(D[1])) / (x0 + x1) + (at(D[2], 0, 1) - at(D[2])) / y0 +
                       (at(D[3], 0, 0, 1) - at(D[3])) / z0)
                at(A["f"]).copy_(self.vn * dfu - cov)
                cov = ((at(Cv[4]) + at(Cv[4], 1)) / 2 + (y1 * at(Cv[5]) + y0 * at(Cv[5], 0, 1)) / (y0 + y1) +
                       (at(Cv[6]) + at(Cv[6], 0, 0, 1)) / 2)
                dfv = ((at(D[4], 1) - at(D[4])) / x0 + 2 * (at(D[5], 0, 1) - at(D[5])) / (y0 + y1) +
                       (at(D[6], 0, 0, 1) - at(D[6])) / z0)
                at(A["g"]).copy_(self.vn * dfv - cov)
            else:
                cov = ((at(Cv[7]) + at(Cv[7], 1)) / 2 + (at(Cv[8]) + at(Cv[8], 0, 1)) / 2 +
                       (z1 * at(Cv[9]) + z0 * at(Cv[9], 0, 0, 1)) / (z0 + z1))
                dfw = ((at(D[7], 1) - at(D[7])) / x0 + (at(D[8], 0, 1) - at(D[8])) / y0 +
                       (at(D[9], 0, 0, 1) - at(D[9])) / zs)
                at(A["h"]).copy_(self.vn * dfw - cov)

    def feedbf(self, A):
        _, _, _, at = self._cells()
        m = at(A["bmask1"])
        for s, q, f in (("usum", "u", "f"), ("vsum", "v", "g"), ("wsum", "w", "h")):
            at(A[s]).copy_((at(A[s]) + at(A[q])) * m)
            at(A[f]).add_(ALPHA * at(A[s]) * self.dt + BETA * at(A[q]) * m)

    def les(self, A, D):
        c = self.c
        im, jm, km = c["ip"], c["jp"], c["kp"]
        I, J, K, at = self._cells()
        sh = lambda r, d: (r[0] + d, r[1] + d)  # noqa: E731
        X = lambda d: self.x("dx1", -1, sh(I, d))  # noqa: E731
        Y = lambda d: self.y("dy1", 0, sh(J, d))  # noqa: E731
        Z = lambda d: self.z("dzn", -1, sh(K, d))  # noqa: E731
        a = (at(D[2], -1) + at(D[2], -1, 1) + at(D[2]) + at(D[2], 0, 1) + at(D[4]) + at(D[4], 0, -1) + at(D[4], 1) +
             at(D[4], 1, -1)) * 0.25
        b = (at(D[8]) + at(D[8], 0, 0, -1) + at(D[8], 0, 1) + at(D[8], 0, 1, -1) + at(D[6], 0, -1) +
             at(D[6], 0, -1, 1) + at(D[6]) + at(D[6], 0, 0, 1)) * 0.25
        e = (at(D[3], -1) + at(D[3], -1, 0, 1) + at(D[3]) + at(D[3], 0, 0, 1) + at(D[7]) + at(D[7], 0, 0, -1) +
             at(D[7], 1) + at(D[7], 1, 0, -1)) * 0.25
        q = 2 * (at(D[1]) ** 2 + at(D[5]) ** 2 + at(D[9]) ** 2) + a * a + b * b + e * e
        root = torch.where(q > 0, torch.sqrt(torch.where(q > 0, q, torch.ones_like(q))), torch.zeros_like(q))
        del a, b, e, q
        cd = self.cs0 * (self.t["dx1"][1] * self.t["dy1"][0] * Z(0)) ** (1.0 / 3.0)
        if "sm" not in A:
            A["sm"] = torch.zeros_like(A["u"])
        sm = A["sm"]
        at(sm).copy_(cd * cd * root)
        # boundsm.f95:13-32
        _r(sm, (0, 0), (-1, jm + 1), (0, km + 1)).copy_(_r(sm, (1, 1), (-1, jm + 1), (0, km + 1)).clone())
        _r(sm, (im + 1, im + 1), (-1, jm + 1), (0, km + 1)).copy_(_r(sm, (im, im), (-1, jm + 1), (0, km + 1)).clone())
        Ig = (0, im + 1)
        _r(sm, Ig, (jm + 1, jm + 1), (0, km + 1)).copy_(_r(sm, Ig, (jm, jm), (0, km + 1)).clone())
        _r(sm, Ig, (0, 0), (0, km + 1)).copy_(_r(sm, Ig, (1, 1), (0, km + 1)).clone())
        _r(sm, Ig, (-1, jm + 1), (0, 0)).copy_(-_r(sm, Ig, (-1, jm + 1), (1, 1)))
        _r(sm, Ig, (-1, jm + 1), (km + 1, km + 1)).copy_(_r(sm, Ig, (-1, jm + 1), (km, km)).clone())
        S = lambda di=0, dj=0, dk=0: at(sm, di, dj, dk)  # noqa: E731
        # x average between i+d and i+d+1, y average alike
        ax = lambda d, dj, dk: (X(d + 1) * S(d, dj, dk) + X(d) * S(d + 1, dj, dk)) / (X(d) + X(d + 1))  # noqa: E731
        ay = lambda d, di, dk: (Y(d + 1) * S(di, d, dk) + Y(d) * S(di, d + 1, dk)) / (Y(d) + Y(d + 1))  # noqa: E731
        zz = lambda lo, hi, d: (Z(d + 1) * lo + Z(d) * hi) / (Z(d) + Z(d + 1))  # noqa: E731
        yy = lambda lo, hi: (Y(1) * lo + Y(0) * hi) / (Y(0) + Y(1))  # noqa: E731
        T = {n: (lambda n: lambda di=0, dj=0, dk=0: at(D[n], di, dj, dk))(n) for n in D}
        sxy = lambda di=0, dj=0: T[2](di, dj + 1) + T[4](di + 1, dj)  # noqa: E731
        ez = zz(ax(0, 0, 0), ax(0, 0, 1), 0)
        ez0 = zz(ax(0, 0, -1), ax(0, 0, 0), -1)
        exy = yy(ax(0, 0, 0), ax(0, 1, 0))
        vf = (S(1) * 2 * T[1](1) - S() * 2 * T[1]()) / X(0)
        vf = vf + (exy * sxy() - yy(ax(0, -1, 0), ax(0, 0, 0)) * (T[2]() + T[4](1, -1))) / Y(0)
        vf = vf + (ez * (T[3](0, 0, 1) + T[7](1)) - ez0 * (T[3]() + T[7](1, 0, -1))) / Z(0)
        at(A["f"]).add_(vf)
        vf = (exy * sxy() - yy(ax(-1, 0, 0), ax(-1, 1, 0)) * (T[2](-1, 1) + T[4]())) / X(0)
        vf = vf + (S(0, 1) * 2 * T[5](0, 1) - S() * 2 * T[5]()) / Y(0)
        vf = vf + (ez * (T[6](0, 0, 1) + T[8](0, 1)) - ez0 * (T[6]() + T[8](0, 1, -1))) / Z(0)
        at(A["g"]).add_(vf)
        vf = (ez * (T[3](0, 0, 1) + T[7](1)) - zz(ax(-1, 0, 0), ax(-1, 0, 1), 0) * (T[3](-1, 0, 1) + T[7]())) / X(0)
        vf = vf + (zz(ay(0, 0, 0), ay(0, 0, 1), 0) * (T[6](0, 0, 1) + T[8](0, 1)) -
                   zz(ay(-1, 0, 0), ay(-1, 0, 1), 0) * (T[6](0, -1, 1) + T[8]())) / Y(0)
        vf = vf + (S(0, 0, 1) * 2 * T[9](0, 0, 1) - S() * 2 * T[9]()) / Z(0)
        at(A["h"]).add_(vf)

    def adam(self, A):
        _, _, _, at = self._cells()
        for f, o in (("f", "fold"), ("g", "gold"), ("h", "hold")):
            now = at(A[f]).clone()
            at(A[f]).copy_(1.5 * now - 0.5 * at(A[o]))
            at(A[o]).copy_(now)

    def rhs(self, A):
        """press.f95:49-82: bondfg, rhs and its volume mean removed."""
        c = self.c
        jm, km = c["jp"], c["kp"]
        I, J, K, at = self._cells()
        f, g, h = A["f"], A["g"], A["h"]
        _r(f, (0, 0), J, K).copy_(_r(f, (1, 1), J, K).clone())
        _r(g, I, (0, 0), K).copy_(_r(g, I, (jm, jm), K).clone())
        _r(h, I, J, (0, 0)).zero_()
        _r(h, I, J, (km, km)).zero_()
        x, y, z = self.x("dx1", -1, I), self.y("dy1", 0, J), self.z("dzn", -1, K)
        div = lambda a, b, e: ((at(a) - at(a, -1)) / x + (at(b) - at(b, 0, -1)) / y +  # noqa: E731
                               (at(e) - at(e, 0, 0, -1)) / z)
        r = div(f, g, h) + div(A["u"], A["v"], A["w"]) / self.dt
        self.vol = x * y * z
        self.area = self.vol.expand(r.shape).sum()
        self.av = (r * self.vol).sum() / self.area
        self.raw = r
        return r - self.av

    def sweep(self, A, r):
        """press.f95:87-115: the red-black SOR with its ghosts."""
        c = self.c
        I, J, K, at = self._cells()
        p = A["p"]
        cl = [self.x("cn2l", 1, I), self.x("cn2s", 1, I), self.y("cn3l", 1, J), self.y("cn3s", 1, J),
              self.z("cn4l", 1, K), self.z("cn4s", 1, K)]
        ii, jj, kk = (torch.arange(1, n + 1, device=self.dev) for n in (c["ip"], c["jp"], c["kp"]))
        par = (ii.view(1, 1, -1) + jj.view(1, -1, 1) + kk.view(-1, 1, 1)) & 1
        black = [(par == 1).to(r.dtype), (par == 0).to(r.dtype)]  # colour nrd sweeps i+j+k+nrd odd
        self.iters = 0
        for _ in range(self.nmaxp):
            sor = 0.0
            for nrd in (0, 1):
                rel = (cl[0] * at(p, 1) + cl[1] * at(p, -1) + cl[2] * at(p, 0, 1) + cl[3] * at(p, 0, -1) +
                       cl[4] * at(p, 0, 0, 1) + cl[5] * at(p, 0, 0, -1) - r)
                rel = (self.cn1 * rel - at(p)) * black[nrd]
                at(p).add_(rel)
                if self.pjuge >= 0:
                    sor += float((rel * rel).sum())
                _boundp1(p, c["ip"], c["jp"])
            _boundp2(p, c["kp"])
            self.iters += 1
            if self.pjuge >= 0 and sor < self.pjuge:
                break

    def press(self, A):
        c = self.c
        r = self.rhs(A)
        self.sweep(A, r)
        at = self._cells()[3]
        p = A["p"]
        at(p).sub_((at(p) * self.vol).sum() / self.area)
        _boundp1(p, c["ip"], c["jp"])
        _boundp2(p, c["kp"])
        A["rhs"] = r

    def solve(self, A):
        """p of the refined press: A p = rhs - mu solved exactly, its volume
        mean removed (A the sweeps' operator with the diagonal that makes
        its rows sum to 0, mu the mean of rhs weighted by its left null
        vector).  x and y are uniform, so A's eigenvectors along them are
        those of two symmetric matrices; z is symmetrised by its weights."""
        def matrix(lo, hi, wrap):
            n = lo.numel()
            m = torch.zeros((n, n), dtype=torch.float64, device=self.dev)
            for q in range(n):
                for s, co in ((q - 1, lo[q]), (q + 1, hi[q])):
                    s = s % n if wrap else min(max(s, 0), n - 1)
                    m[q, s] += co
                    m[q, q] -= co
            return m

        t = {n: self.t[n].cpu() for n in ("cn2l", "cn2s", "cn3l", "cn3s", "cn4l", "cn4s")}
        dev, self.dev = self.dev, "cpu"
        mx, my = matrix(t["cn2s"], t["cn2l"], False), matrix(t["cn3s"], t["cn3l"], True)
        mz = matrix(t["cn4s"], t["cn4l"], False)
        self.dev = dev
        mx, my, mz = mx.to(dev), my.to(dev), mz.to(dev)
        w = torch.ones(mz.shape[0], dtype=torch.float64, device=dev)  # w(q+1) cs(q+1) = w(q) cl(q)
        for q in range(1, w.numel()):
            w[q] = w[q - 1] * self.t["cn4l"][q - 1] / self.t["cn4s"][q]
        s = w.sqrt()
        sz = s.view(-1, 1) * mz / s.view(1, -1)
        lx, vx = torch.linalg.eigh((mx + mx.T) / 2)
        ly, vy = torch.linalg.eigh((my + my.T) / 2)
        lz, vz = torch.linalg.eigh((sz + sz.T) / 2)
        b = self.raw
        mu = (b * w.view(-1, 1, 1)).sum() / (w.sum() * b.shape[1] * b.shape[2])
        b = (b - mu) * s.view(-1, 1, 1)
        b = torch.einsum("kji,ia->kja", b, vx)
        b = torch.einsum("kja,jb->kba", b, vy)
        b = torch.einsum("kba,kc->cba", b, vz)
        lam = lz.view(-1, 1, 1) + ly.view(1, -1, 1) + lx.view(1, 1, -1)
        null = lam.abs().argmin()
        b = b / lam
        b.view(-1)[null] = 0.0
        b = torch.einsum("cba,kc->kba", b, vz)
        b = torch.einsum("kba,jb->kja", b, vy)
        b = torch.einsum("kja,ia->kji", b, vx) / s.view(-1, 1, 1)
        b = b - (b * self.vol).sum() / self.area
        self._cells()[3](A["p"]).copy_(b)


def _inputs64(case, seed, dev):
    grid = _grid(case)
    A = _fields(case, seed, grid, dev)
    wind = A.pop("wind_profile").double()
    return grid, {n: a.double() for n, a in A.items()}, wind


def exact(case, seed):
    dev, kind = "cuda", case["kind"]
    inner = lambda c, a: a[2:c["kp"] + 2, 2:c["jp"] + 2, 2:c["ip"] + 2]  # noqa: E731
    if kind == "ensemble":
        out = []
        for q, (ip, jp, kp) in enumerate(_members(case)):
            c = dict(case, ip=ip, jp=jp, kp=kp)
            grid, A, wind = _inputs64(c, seed + 100 * q, dev)
            A = _Step64(c, grid, dev, NMAXP, PJUGE)(A, wind)
            out.append({n: inner(c, A[n]).clone() for n in ("u", "v", "w", "p")})
        return out
    grid, A, wind = _inputs64(case, seed, dev)
    if kind == "press":
        s = _Step64(case, grid, dev, NMAXP, PJUGE)
        s.press(A)
        return {"p": inner(case, A["p"]).permute(2, 1, 0), "rhs": A["rhs"].permute(2, 1, 0), "iters": None}
    if kind == "gradient":
        return _gradient64(case, grid, A, wind, dev)
    s = _Step64(case, grid, dev, NMAXP, PJUGE)
    A = s(A, wind)
    if kind == "refined":
        s.solve(A)
        return {n: inner(case, A[n]) for n in ("u", "v", "w", "p", "f", "g", "h")}
    out = {n: inner(case, A[n]) for n in STATE}
    if kind == "coupled":
        return {"state": out, "halo": [None] * 7, "uout": None, "rhsav": float(s.av), "iters": None}
    return out


def _gradient64(case, grid, A, wind, dev):
    """J and its gradient by torch's reverse mode through the FP64 steps."""
    leaves = {n: a.clone().requires_grad_(n != "bmask1") for n, a in A.items()}
    wl = wind.clone().requires_grad_(True)
    s = _Step64(case, grid, dev, NMAXP, -1.0)
    (i0, i1), (j0, j1), (k0, k1) = _box(case)
    S, J = leaves, 0.0
    for _ in range(case["nt"]):
        S = s(S, wl)
        S.pop("rhs")
        c = lambda q, di, dj, dk: _r(S[q], (i0 - di, i1 - di), (j0 - dj, j1 - dj), (k0 - dk, k1 - dk))  # noqa: E731
        e = sum(((c(q, 0, 0, 0) + c(q, *d)) / 2) ** 2 for q, d in (("u", (1, 0, 0)), ("v", (0, 1, 0)), ("w", (0, 0, 1))))
        J = J + 0.5 * e.mean() / case["nt"]
    J.backward()
    inner = lambda a: a[2:case["kp"] + 2, 2:case["jp"] + 2, 2:case["ip"] + 2].permute(2, 1, 0)  # noqa: E731
    out = {n: inner(leaves[n].grad) for n in GRAD}
    out.update(J=float(J), wp=wl.grad.T)
    return out
