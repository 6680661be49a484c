"""The work that programs give this framework, as measurable cases.

A simulation program makes a model, sets a field, advances it some steps and reads
the field back; a parameter sweep advances many small fields together; an
optimisation runs steps forward and their adjoint backward; a program with its own
spectral method calls the transform.  Each case is one such call sequence through
the Python entry points, on sizes from the configurations, tests and benchmark of
this repository:

  kind      plain / filtered / tungsten / aluminum   set_psi, step(steps), sync, get_psi
            ensemble                                 step(steps), sync, get_psi of every member
            adjoint                                  PfcEvolve forward and its backward
            fft                                      forward, backward
  n0 n1 n2  grid (x fastest); ensembles have `members` cubes instead
  f64       FP64 arithmetic and buffers (else FP32)
  numpy     fields pass through numpy float64 arrays, as in the documented Python example
            (else CUDA tensors of the compute precision)
  tuned     the program calls autotune() when it starts
"""
import math
import random

import numpy as np
import torch

import openpfc_b200 as ob
from openpfc_b200.autograd import PfcEvolve

PI4 = math.pi / 4
TUNGSTEN_DX = 1.1107207345395915
SIDES = (32, 48, 64, 80, 96)  # ensemble members
# axis lengths: N0 = 2 M with M a transform length, N1 and N2 transform lengths
X_LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 256, 512, 1024)
YZ_LENGTHS = (16, 24, 32, 40, 48, 64, 80, 96, 128, 256, 512, 1024)


def listed():
    return [
        # the headline workload: one large grid, FP32, tuned at start-up
        dict(name="plain-512-f32-tuned", kind="plain", n0=512, n1=512, n2=512, f64=False, steps=20, numpy=False, tuned=True),
        # the same model at reference precision on an ordinary grid
        dict(name="plain-256-f64", kind="plain", n0=256, n1=256, n2=256, f64=True, steps=20, numpy=False, tuned=False),
        # a small grid: launches and latency count
        dict(name="plain-64-f32", kind="plain", n0=64, n1=64, n2=64, f64=False, steps=100, numpy=False, tuned=False),
        # axes that are no powers of two, a box that is no cube
        dict(name="plain-192x96x80-f32", kind="plain", n0=192, n1=96, n2=80, f64=False, steps=50, numpy=False, tuned=False),
        # the documented Python example: numpy in, 100 steps, numpy out
        dict(name="plain-256-f32-numpy", kind="plain", n0=256, n1=256, n2=256, f64=False, steps=100, numpy=True, tuned=False),
        # mean-field-filtered model on a box with the long axis of the 1024-point configuration
        dict(name="filtered-256x256x1024-f32", kind="filtered", n0=256, n1=256, n2=1024, f64=False, steps=10, numpy=False, tuned=False),
        # the Tungsten application in its default precision (two real fields a step)
        dict(name="tungsten-256-f64", kind="tungsten", n0=256, n1=256, n2=256, f64=True, steps=10, numpy=False, tuned=False),
        # directional solidification: moving temperature gradient along x (three real fields a step)
        dict(name="aluminum-256x64x64-f64", kind="aluminum", n0=256, n1=64, n2=64, f64=True, steps=20, numpy=False, tuned=False),
        # a parameter sweep: independent cubes of uneven sides, read out every 200 steps
        dict(name="ensemble-64-f32", kind="ensemble", members=64, f64=False, steps=200),
        # gradient of a loss on the end state through 40 steps, snapshots every 20
        dict(name="adjoint-128-f32", kind="adjoint", n0=128, n1=128, n2=128, f64=False, steps=40),
        # the transform alone, forward and backward, at the reference's precision
        dict(name="fft-256-f64", kind="fft", n0=256, n1=256, n2=256, f64=True),
        # a small ragged transform
        dict(name="fft-96x80x48-f32", kind="fft", n0=96, n1=80, n2=48, f64=False),
    ]


def _cells(c):
    return c["n0"] * c["n1"] * c["n2"]


def draw(rng):
    kind = rng.choice(("plain", "plain", "plain", "filtered", "filtered", "tungsten", "aluminum", "ensemble", "adjoint", "fft", "fft"))
    f64 = rng.random() < 0.5
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(4, 64), f64=f64, steps=rng.choice((50, 100)) if f64 else rng.choice((50, 100, 200)))
    most = {"adjoint": 2 ** 22, "aluminum": 2 ** 22}.get(kind, 2 ** 25)
    # the cell count is spread over its logarithm; the box is the drawn one closest to it
    want = math.exp(rng.uniform(math.log(2 ** 14), math.log(most)))
    boxes = [(rng.choice(X_LENGTHS), rng.choice(YZ_LENGTHS), rng.choice(YZ_LENGTHS)) for _ in range(60)]
    n = min((b for b in boxes if b[0] * b[1] * b[2] <= most), key=lambda b: abs(math.log(b[0] * b[1] * b[2] / want)))
    c = dict(kind=kind, n0=n[0], n1=n[1], n2=n[2], f64=f64)
    if kind == "fft":
        return c
    # the filtered configuration's dynamics are unstable: FP32 overflows after some 50 steps
    c["steps"] = {"adjoint": rng.choice((20, 40)), "filtered": 10}.get(kind) or rng.choice((10, 20) if want > 2 ** 22 else (10, 20, 50))
    if kind != "adjoint":
        c["numpy"] = rng.random() < 0.2 and _cells(c) <= 2 ** 24
        c["tuned"] = kind in ("plain", "filtered") and rng.random() < 0.2
    return c


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _noise(c, seed, mean, amp, dtype):
    u = torch.rand((c["n2"], c["n1"], c["n0"]), generator=_gen(seed), device="cuda", dtype=dtype)
    return u.mul_(2 * amp).add_(mean - amp)


BCC = [(1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 0, -1), (1, -1, 0), (0, 1, -1)]
FCC = [(-1, 1, 1), (1, -1, 1), (1, 1, -1), (1, 1, 1)]


def _with_seeds(psi, seed, dx, count, radius, inside, amp, lattice):
    """Spheres of a one-mode crystal (radius in cells, centres from the seed) in the field psi."""
    n2, n1, n0 = psi.shape
    rng = random.Random(seed)
    norm = math.sqrt(sum(q * q for q in lattice[0]))
    ax = [torch.arange(n, device="cuda", dtype=torch.float64) for n in (n0, n1, n2)]
    for _ in range(count):
        centre = [rng.random() * n for n in (n0, n1, n2)]
        d = [(a - x + n / 2) % n - n / 2 for a, x, n in zip(ax, centre, (n0, n1, n2))]  # nearest image
        at = [torch.nonzero(t.abs() <= radius).flatten() for t in d]
        X, Y, Z = d[0][at[0]][None, None, :], d[1][at[1]][None, :, None], d[2][at[2]][:, None, None]
        u = torch.full((), inside, device="cuda", dtype=torch.float64)
        for q in lattice:
            u = u + 2 * amp * torch.cos((q[0] * X + q[1] * Y + q[2] * Z) * (dx / norm))
        box = (at[2][:, None, None], at[1][None, :, None], at[0][None, None, :])
        hit = X * X + Y * Y + Z * Z < radius * radius
        psi[box] = torch.where(hit, u, psi[box].double()).to(psi.dtype)
    return psi


def _field(c, seed, dtype):
    kind, small = c["kind"], min(c["n0"], c["n1"], c["n2"])
    if kind == "filtered":
        return _with_seeds(_noise(c, seed, -0.10, 0.001, dtype), seed, PI4, 8, min(20.0, small / 4), -0.10, 0.1, BCC)
    if kind == "tungsten":
        return _with_seeds(_noise(c, seed, -0.40, 0.001, dtype), seed, TUNGSTEN_DX, 1, small / 3, -0.047, 0.215936, BCC)
    if kind == "aluminum":
        return _with_seeds(_noise(c, seed, -0.006, 0.001, dtype), seed, 1.0, 4, small / 6, -0.036, 0.4, FCC)
    return _noise(c, seed, -0.285, 0.01, dtype)


ALUMINUM = dict(n0=-0.0060, alpha=0.20, n_sol=-0.036, n_vap=-1.297, T_const=980.0, T_min=780.0, T_max=1280.0, T0=89285.0,
                Bx=0.817900686921996, G_grid=2.0, V_grid=0.5, x_initial=4.0, m_xpos=5.0, alpha_farTol=0.001, tau_const=0.3,
                lambda_=0.22, stabP=0.05, shift_u=1.0, shift_s=0.0, p2_bar=0.8286531831, p3_bar=-0.04204863, p4_bar=0.007533,
                q20_bar=0.016531729105214, q21_bar=5.467, q30_bar=1.7152418049986, q31_bar=0.45, q40_bar=0.787482,
                q4_bar=0.787482)
ALUMINUM_DT, ALUMINUM_T = 1e-2, 0.3
FILTERED = dict(r=-0.3, alpha=0.5, p2=-0.1, p3=-0.5, p4=0.3)


def _spacing(c):
    return {"tungsten": TUNGSTEN_DX, "aluminum": 1.0}.get(c["kind"], PI4)


def _members(c, seed):
    """Sides and r of the sweep (the case's own), mean densities (the seed's)."""
    rng, by_seed = random.Random(c["members"]), random.Random(seed)
    return [dict(n=(s, s, s), dx=(PI4,) * 3, r=rng.uniform(-0.35, -0.10), n0=by_seed.uniform(-0.35, -0.20))
            for s in (rng.choice(SIDES) for _ in range(c["members"]))]


def _member_fields(c, seed):
    rng = np.random.default_rng(seed)
    return [m["n0"] + rng.uniform(-0.01, 0.01, (m["n"][2], m["n"][1], m["n"][0])) for m in _members(c, seed)]


def prepare(case, seed):
    c = case
    prec, dtype = (ob.FP64, torch.float64) if c["f64"] else (ob.FP32, torch.float32)
    if c["kind"] == "ensemble":
        e = ob.Ensemble(_members(c, seed), precision=prec)
        e.initialize(0.5)
        for i, p in enumerate(_member_fields(c, seed)):
            e.set_psi(i, p)
        return dict(case=c, model=e)
    n, dx = (c["n0"], c["n1"], c["n2"]), (_spacing(c),) * 3
    if c["kind"] == "fft":
        shape = (c["n2"], c["n1"], c["n0"] // 2 + 1, 2)
        x = torch.randn((c["n2"], c["n1"], c["n0"]), generator=_gen(seed), device="cuda", dtype=dtype)
        return dict(case=c, model=ob.B200Fft(n, precision=prec), x=x, hat=torch.empty(shape, device="cuda", dtype=dtype),
                    back=torch.empty_like(x))
    if c["kind"] == "filtered":
        m = ob.FilteredB200(n, dx, precision=prec, **FILTERED)
    elif c["kind"] == "tungsten":
        m = ob.TungstenB200(n, dx, precision=prec)
    elif c["kind"] == "aluminum":
        p = ob.AluminumParams()
        for k, v in ALUMINUM.items():
            setattr(p, k, v)
        m = ob.AluminumB200(n, dx, p, precision=prec)
    else:
        m = ob.PfcB200(n, dx, r=-0.25, precision=prec)
    m.initialize(ALUMINUM_DT if c["kind"] == "aluminum" else 1.0 if c["kind"] == "tungsten" else 0.5)
    if c.get("tuned"):
        m.autotune()
    if c["kind"] == "adjoint":
        psi0 = _field(c, seed, dtype)
        w = _weight(psi0)
        r = torch.tensor(-0.25, dtype=torch.float64, requires_grad=True)
        return dict(case=c, model=m, psi0=psi0.requires_grad_(), r=r, w=w)
    psi0 = _field(c, seed, dtype)
    if c["numpy"]:
        return dict(case=c, model=m, psi0=psi0.double().cpu().numpy())
    return dict(case=c, model=m, psi0=psi0, out=torch.empty_like(psi0))


def _weight(psi0):
    """dLoss/dpsi_T of the adjoint case: how much of the initial pattern the end state holds."""
    return psi0 - psi0.mean()


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------

def run(state):
    c, m = state["case"], state["model"]
    if c["kind"] == "ensemble":
        m.step(c["steps"])
        m.sync()
        return [m.get_psi(i) for i in range(c["members"])]
    if c["kind"] == "fft":
        m.forward(state["x"], state["hat"])
        m.backward(state["hat"], state["back"])
        return state["hat"], state["back"]
    if c["kind"] == "adjoint":
        psi = PfcEvolve.apply(state["psi0"], state["r"], m, c["steps"], 20)
        g, dr = torch.autograd.grad(psi, (state["psi0"], state["r"]), state["w"])
        return psi.detach(), g, dr
    m.set_psi(state["psi0"])
    if c["kind"] == "aluminum":
        m.set_time(ALUMINUM_T, ALUMINUM_DT)
    m.step(c["steps"])
    m.sync()
    return m.get_psi() if c["numpy"] else m.get_psi(state["out"])


# --------------------------------------------------------------------------
# what a pass cannot do without
# --------------------------------------------------------------------------

def work(case):
    """A step is two 3D transforms of each field around pointwise work.  Between the
    z transforms and the xy transforms every mode has to pass through memory (L2 for
    small grids): the state in and out of the update once, each field's spectrum
    written and read once between update and xy part, N_hat written and read once
    on the way back.  2.5 N log2 N operations a real transform."""
    c = case
    rs = 8 if c["f64"] else 4
    if c["kind"] == "ensemble":
        sides = [m["n"][0] for m in _members(c, 0)]
        return dict(bytes=sum(c["steps"] * 6 * (s // 2 + 1) * s * s * 2 * rs + s ** 3 * 8 for s in sides),
                    flops=sum(c["steps"] * (5 * s ** 3 * math.log2(s ** 3) + 10 * s ** 3) for s in sides))
    n = _cells(c)
    real, hat = n * rs, (c["n0"] // 2 + 1) * c["n1"] * c["n2"] * 2 * rs
    one = 2.5 * n * math.log2(n)
    if c["kind"] == "fft":  # x -> between the axes -> hat, and back
        return dict(bytes=2 * (real + 2 * hat + hat), flops=2 * one)
    fields = {"tungsten": 2, "aluminum": 3}.get(c["kind"], 1)
    step_bytes, step_flops = (2 + 2 * fields + 2) * hat, (1 + fields) * one + 20 * n
    if c["kind"] == "adjoint":
        # forward, recomputation, and a reverse step: lambda_hat out of and two fields into the xy part, u read
        return dict(bytes=c["steps"] * (2 * step_bytes + 6 * hat + 3 * real) + 3 * real,
                    flops=c["steps"] * (2 * step_flops + 3 * one + 20 * n))
    io = 2 * (8 * n if c["numpy"] else real)
    return dict(bytes=c["steps"] * step_bytes + io, flops=c["steps"] * step_flops + 2 * one)


def tolerance(case):
    """About four times the largest distance from exact() seen over these cases and drawn ones."""
    c = case
    if c["f64"]:
        return {"rel": {"fft": 4e-15, "adjoint": 4e-14, "ensemble": 4e-14}.get(c["kind"], 4e-15)}
    return {"rel": {"fft": 1e-6, "adjoint": 1e-4, "ensemble": 1.8e-4}.get(c["kind"], 2e-6)}


# --------------------------------------------------------------------------
# the same in plain torch, 64 bits
# --------------------------------------------------------------------------

def _k2(n, dx):
    n0, n1, n2 = n
    k = [2 * math.pi * torch.fft.fftfreq(n2, dx, dtype=torch.float64, device="cuda")[:, None, None],
         2 * math.pi * torch.fft.fftfreq(n1, dx, dtype=torch.float64, device="cuda")[None, :, None],
         2 * math.pi * torch.fft.rfftfreq(n0, dx, dtype=torch.float64, device="cuda")[None, None, :]]
    return k[0] ** 2 + k[1] ** 2 + k[2] ** 2


def _etd(k2, r, dt):
    """opL, opN of the conserved plain model."""
    L = -k2 * (r + (1 - k2) ** 2)
    safe = torch.where(L.abs() > 1e-14, L, torch.ones_like(L))
    return torch.exp(L * dt), torch.where(L.abs() > 1e-14, torch.expm1(safe * dt) / safe * -k2, -dt * k2)


def _plain(psi, dx, r, dt, steps):
    n = psi.shape[::-1]
    opl, opn = _etd(_k2(n, dx), r, dt)
    hat = torch.fft.rfftn(psi)
    for _ in range(steps):
        hat = opl * hat + opn * torch.fft.rfftn(torch.fft.irfftn(hat, s=psi.shape, dim=(0, 1, 2)) ** 3)
    return torch.fft.irfftn(hat, s=psi.shape, dim=(0, 1, 2))


def _filtered(psi, steps, dt=0.5):
    p = FILTERED
    k2 = _k2(psi.shape[::-1], PI4)
    opl, opn = _etd(k2, p["r"], dt)
    chi = torch.exp(-k2 / (2 * p["alpha"] ** 2))
    hat = torch.fft.rfftn(psi)
    for _ in range(steps):
        v = torch.fft.irfftn(chi * hat, s=psi.shape, dim=(0, 1, 2))
        hat = opl * hat + opn * torch.fft.rfftn(v * v * (p["p2"] / 2 + p["p3"] / 3 * v + p["p4"] / 4 * v * v))
    return torch.fft.irfftn(hat, s=psi.shape, dim=(0, 1, 2))


def _tungsten(psi, steps, dt=1.0):
    T, T0, Bx, alpha, far, high = 3300.0, 156000.0, 0.8582, 0.50, 0.001, 4
    lam, stab, su, ss = 0.22, 0.2, 0.3341, 0.1898
    p2, p3, p4, q20, q21, q30, q31, q40 = 1.0, -0.5, 0.333333333, -0.0037, 1.0, -12.4567, 20.0, 45.0
    tau = T / T0
    p2b, p3b, p4b = p2 + 2 * ss * p3 + 3 * ss ** 2 * p4, su * (p3 + 3 * ss * p4), su ** 2 * p4
    q2b = (q21 + 2 * ss * q31) * tau + q20 + 2 * ss * q30 + 3 * ss ** 2 * q40
    q3b, q4b = su * q31 * tau + su * (q30 + 3 * ss * q40), su ** 2 * q40
    lap = -_k2(psi.shape[::-1], TUNGSTEN_DX)
    chi = torch.exp(lap / (2 * lam ** 2))
    kv, a2 = torch.sqrt(-lap) - 1, 2 * alpha ** 2
    rtol = -a2 * math.log(far) - 1
    near = torch.exp(-(kv ** 2 + rtol * kv ** high) / a2)
    L = lap * (stab + p2b - Bx * math.exp(-tau) * torch.where(kv < 0, near, 1 - kv ** 2 / a2) + q2b * chi)
    safe = torch.where(L.abs() < 1e-12, torch.ones_like(L), L)
    opl, opn = torch.exp(L * dt), lap * torch.where(L.abs() < 1e-12, dt + L * dt * dt / 2, torch.expm1(safe * dt) / safe)
    hat = torch.fft.rfftn(psi)
    for _ in range(steps):
        u = torch.fft.irfftn(hat, s=psi.shape, dim=(0, 1, 2))
        v = torch.fft.irfftn(chi * hat, s=psi.shape, dim=(0, 1, 2))
        hat = opl * hat + opn * torch.fft.rfftn(p3b * u ** 2 + p4b * u ** 3 + q3b * v ** 2 + q4b * v ** 3 - stab * u)
    return torch.fft.irfftn(hat, s=psi.shape, dim=(0, 1, 2))


def _aluminum(psi, steps, dt=ALUMINUM_DT):
    p = ALUMINUM
    n0 = psi.shape[2]
    lap = -_k2(psi.shape[::-1], 1.0)
    chi = torch.exp(lap / (2 * p["lambda_"] ** 2))
    k, a2 = torch.sqrt(-lap), 2 * p["alpha"] ** 2
    peak = torch.maximum(torch.exp(-(k - 1) ** 2 / a2), torch.exp(-(k - 2 / math.sqrt(3)) ** 2 / a2))
    pf = p["Bx"] * math.exp(-p["tau_const"]) * peak
    ck = p["stabP"] + p["p2_bar"] - pf  # q2_bar_L = 0
    opl = torch.exp(lap * ck * dt)
    opn = torch.where(ck == 0, lap * dt, (opl - 1) / ck)
    x = torch.arange(n0, dtype=torch.float64, device="cuda")
    dist = x + math.floor(p["m_xpos"] / n0) * n0 - torch.where(x > math.fmod(p["m_xpos"], n0), float(n0), 0.0)
    hat = torch.fft.rfftn(psi)
    for s in range(steps):
        u, v, w = (torch.fft.irfftn(f * hat, s=psi.shape, dim=(0, 1, 2)) for f in (1.0, chi, pf))
        tv = p["G_grid"] * (dist - p["x_initial"] - p["V_grid"] * (ALUMINUM_T + s * ALUMINUM_DT))
        N = (p["p3_bar"] * u ** 2 + p["p4_bar"] * u ** 3 + p["q21_bar"] * tv / p["T0"] * v
             + (p["q31_bar"] * (p["T_const"] + tv) / p["T0"] + p["q30_bar"]) * v ** 2 + p["q4_bar"] * v ** 3
             + (1 - torch.exp(-tv / p["T0"])) * w - p["stabP"] * u)
        hat = opl * hat + opn * torch.fft.rfftn(N)
    return torch.fft.irfftn(hat, s=psi.shape, dim=(0, 1, 2))


def exact(case, seed):
    c = case
    dtype = torch.float64 if c["f64"] else torch.float32
    if c["kind"] == "ensemble":
        return [_plain(torch.from_numpy(p).cuda(), PI4, m["r"], 0.5, c["steps"]).cpu().numpy()
                for m, p in zip(_members(c, seed), _member_fields(c, seed))]
    if c["kind"] == "fft":
        x = torch.randn((c["n2"], c["n1"], c["n0"]), generator=_gen(seed), device="cuda", dtype=dtype).double()
        return torch.view_as_real(torch.fft.rfftn(x)).contiguous(), x
    psi = _field(c, seed, dtype)
    if c["kind"] == "adjoint":
        w = _weight(psi).double()
        psi = psi.double().requires_grad_()
        r = torch.tensor(-0.25, dtype=torch.float64, device="cuda", requires_grad=True)
        end = _plain(psi, PI4, r, 0.5, c["steps"])
        g, dr = torch.autograd.grad(end, (psi, r), w)
        return end.detach(), g, dr.cpu()
    psi = psi.double()
    if c["kind"] == "filtered":
        out = _filtered(psi, c["steps"])
    elif c["kind"] == "tungsten":
        out = _tungsten(psi, c["steps"])
    elif c["kind"] == "aluminum":
        out = _aluminum(psi, c["steps"])
    else:
        out = _plain(psi, PI4, -0.25, 0.5, c["steps"])
    return out.cpu().numpy() if c["numpy"] else out
