"""What a user of this framework has it do: field evaluations, RK4 and RKDP54 runs, multilayered and
batched systems, and the discrete adjoint, from a 512-cell film (launch latency) to the 4.2 M-cell film
of the benchmark and the three-mesh stack of 2.6 M cells, in mixed precision and FP64.

Every pass goes through the public API (boris2_b200.Context and the C ABI of include/boris_b200.h):
the state arrives (bm_set_m_device, or Context.set_m for host arrays), the steps run, the state or the
field comes back whole. Contexts are set up in prepare(), as a program does once per simulation.

exact() restates each pass in plain torch FP64 (Newell tensor, padded FFT convolution, stencils, LLG,
Runge-Kutta stages, autograd for the adjoint); it uses none of the package's code.
"""
import ctypes
import math

import numpy as np
import torch
import torch.utils.checkpoint

import boris2_b200 as bm

MU0 = 1.256637061435916e-6
GAMMA = 2.212761569e5
NM = 1e-9
# largest RKDP54 step of the cases: the controller runs at every step and doubles the first ones up to
# this limit, below the step at which its factor hangs on the last digits of a mixed-precision estimate
DT_MAX = 1e-14


# ------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # the demag field of a small element for a host program that keeps its vectors on the GPU (the
        # Boris-side module): one field evaluation, all launch latency
        _field("demag_film_32x16", 32, 16, 1, 5, 5, 3),
        # the 128 x 64 permalloy film of the standard problem: thousands of RK4 steps on few cells
        _run("rk4_film_128x64", 128, 64, 1, 5, 5, 3, "RK4", 100, 1e-13, Ms=8e5, A=1.3e-11, alpha=0.5, Hx=1e3),
        # a square in-plane periodic film (PBC images along x and y) with anisotropy under RK4
        _run("rk4_pbc_film_192x192", 192, 192, 1, 4, 4, 3, "RK4", 40, 1e-13, Ms=8e5, A=1.3e-11, alpha=0.02, K1=1e5,
             pbc=3),
        # a 3D box of odd cell counts, all field terms of the interfacial-DMI film, RK4
        _run("rk4_box_97x61x23", 97, 61, 23, 4, 4, 3, "RK4", 20, 5e-14, Ms=1.1e6, A=1.5e-11, alpha=0.1, K1=5e5,
             D=1.5e-3),
        # plain FP64 demag field and energy of an odd box (validation runs use the FP64 form)
        _field("demag_fp64_200x150x12", 200, 150, 12, 4, 4, 3, prec="fp64", energy=True),
        # Python front end on host arrays: set M, read the effective field back (relaxed-state analysis)
        _heff("heff_host_256x256x4", 256, 256, 4, 4, 4, 3),
        # inverse design: gradients of a final-state loss through RK4 steps of a 256 x 256 film
        _adjoint("adjoint_film_256x256", 256, 256, 200, 50),
        # many independent uneven films advanced together (a parameter study), the benchmark's size set
        _batch("batch_24_films", 24, 2),
        # the benchmark film, RKDP54 with adaptive steps, mixed precision: the headline workload
        _run("rkdp54_film_512x512x16", 512, 512, 16, 2, 2, 2, "RKDP54", 4, 5e-15, Ms=1.1e6, A=1.5e-11, alpha=0.1,
             K1=5e5, D=1.5e-3, tol=1e-5),
        # the same film in plain FP64
        _run("rkdp54_fp64_film_512x512x16", 512, 512, 16, 2, 2, 2, "RKDP54", 2, 5e-15, Ms=1.1e6, A=1.5e-11, alpha=0.1,
             K1=5e5, D=1.5e-3, tol=1e-5, prec="fp64"),
        # the same film under RK4 with the demag field extrapolated quadratically between steps
        _run("rk4_speedup_film_512x512x16", 512, 512, 16, 2, 2, 2, "RK4", 6, 1e-14, Ms=1.1e6, A=1.5e-11, alpha=0.1,
             K1=5e5, D=1.5e-3, es=3),
        # three stacked meshes of different cellsizes under one multilayered convolution
        _stack("multilayer_stack3", 1024, 1024, 2),
    ]


def _film(name, kind, nx, ny, nz, hx, hy, hz, prec):
    d = dict(kind=kind, nx=nx, ny=ny, nz=nz, hx=float(hx), hy=float(hy), hz=float(hz), prec=prec)
    if name:
        d["name"] = name
    return d


def _field(name, nx, ny, nz, hx, hy, hz, prec="mixed", energy=False):
    return dict(_film(name, "field", nx, ny, nz, hx, hy, hz, prec), energy=energy, Ms=8e5)


def _heff(name, nx, ny, nz, hx, hy, hz, prec="mixed"):
    return dict(_film(name, "heff", nx, ny, nz, hx, hy, hz, prec), Ms=8e5, A=1.3e-11, K1=1e5, D=0.0, Hx=1e3, pbc=0)


def _run(name, nx, ny, nz, hx, hy, hz, ode, steps, dt, Ms, A, alpha, K1=0.0, D=0.0, Hx=0.0, tol=0.0, es=0, pbc=0,
         prec="mixed"):
    return dict(_film(name, "run", nx, ny, nz, hx, hy, hz, prec), ode=ode, steps=steps, dt=dt, Ms=Ms, A=A, alpha=alpha,
                K1=K1, D=D, Hx=Hx, tol=tol, es=es, pbc=pbc)


def _adjoint(name, nx, ny, steps, every, prec="mixed"):
    return dict(_film(name, "adjoint", nx, ny, 1, 4, 4, 3, prec), steps=steps, every=every, dt=1e-13, A=1.3e-11,
                alpha=0.02)


def _batch(name, count, steps, prec="mixed", sizes=3):
    d = dict(kind="batch", count=count, steps=steps, dt=5e-14, sizes=sizes, prec=prec)
    if name:
        d["name"] = name
    return d


def _stack(name, nx, ny, steps, same=False, prec="mixed"):
    """same: three equal one-cell-thick films; otherwise the benchmark's stack, the middle mesh on a
    coarser grid (mesh transfer) and the cells of unequal thickness."""
    d = dict(kind="stack", nx=nx, ny=ny, steps=steps, same=same, prec=prec)
    if name:
        d["name"] = name
    return d


def draw(rng):
    """One more case: sizes over the logarithm of 12 .. 512 cells per in-plane axis (odd and ragged ones
    among them), 1 .. 24 cells thick, every kind, precision and option of the listed cases."""
    def size(lo, hi):
        v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return max(lo, min(hi, v))

    def thick():
        return 1 if rng.random() < 0.35 else size(2, 24)

    prec = "fp64" if rng.random() < 0.25 else "mixed"
    kind = rng.choice(["field", "field", "run", "run", "run", "run", "heff", "adjoint", "batch", "stack"])
    nx, ny, nz = size(12, 512), size(12, 512), thick()
    while nx * ny * nz > 2000000:
        nz = max(1, nz // 2)
    hx = rng.choice([2.0, 4.0, 5.0])
    hz = rng.choice([2.0, 3.0])
    if kind == "field":
        return _field(None, nx, ny, nz, hx, hx, hz, prec, rng.random() < 0.5)
    if kind == "heff":
        return _heff(None, nx, ny, min(nz, 8), hx, hx, hz, prec)
    if kind == "adjoint":
        every = rng.choice([4, 5, 8])
        return _adjoint(None, size(24, 256), size(24, 256), every * rng.choice([2, 3, 4]), every, prec)
    if kind == "batch":
        return _batch(None, size(4, 24), rng.choice([1, 2, 3]), prec, rng.choice([2, 3, 5, 7]))
    if kind == "stack":
        same = rng.random() < 0.6
        n = 4 * size(16, 160)
        return _stack(None, n if not same else n + rng.choice([0, 1, 3]), 4 * size(16, 160), rng.choice([1, 2, 3]), same,
                      prec)
    ode = rng.choice(["RK4", "RK4", "RKDP54"])
    es = rng.choice([0, 0, 2, 3]) if ode == "RK4" else 0
    pbc = rng.choice([0, 0, 0, 2]) if nz <= 8 and max(nx, ny) <= 256 else 0
    steps = rng.choice([4, 6, 8])
    return _run(None, nx, ny, nz, hx, hx, hz, ode, steps, 5e-14 if ode == "RK4" else 5e-15, Ms=rng.choice([8e5, 1.1e6]),
                A=1.3e-11, alpha=rng.choice([0.02, 0.1, 0.5]), K1=rng.choice([0.0, 1e5, 5e5]),
                D=rng.choice([0.0, 1.5e-3]), Hx=rng.choice([0.0, 1e3]), tol=1e-5 if ode == "RKDP54" else 0.0, es=es,
                pbc=pbc, prec=prec)


# ------------------------------------------------------------------------------------ inputs
def _h(case):
    return case["hx"] * NM, case["hy"] * NM, case["hz"] * NM


def _n(case):
    return case["nx"], case["ny"], case["nz"]


def _batch_systems(case):
    """Uneven films as the batching benchmark draws them, the set of sizes fixed by the case."""
    rng = np.random.default_rng(case["sizes"])
    sizes = [64, 96, 128, 192, 256, 384, 512]
    out = []
    for _ in range(case["count"]):
        n = (int(rng.choice(sizes)), int(rng.choice(sizes)), int(rng.choice([1, 2, 4])))
        out.append(dict(n=n, h=(4 * NM, 4 * NM, 3 * NM), o=(0.0, 0.0, 0.0), Ms=float(rng.uniform(4e5, 1.4e6)), K1=0.0,
                        A=float(rng.uniform(0.8e-11, 2e-11)), alpha=float(rng.uniform(0.01, 0.5)), modules=1 | 2))
    return out


def _stack_meshes(case):
    nx, ny = case["nx"], case["ny"]
    if case["same"]:
        return [dict(n=(nx, ny, 1), h=(2 * NM, 2 * NM, 1 * NM), o=(0, 0, z * NM), Ms=Ms, K1=0.0, A=1.5e-11, alpha=0.05,
                     modules=1 | 2) for z, Ms in ((0, 1.4e6), (2, 6e5), (5, 1.1e6))]
    return [dict(n=(nx, ny, 1), h=(2 * NM, 2 * NM, 1 * NM), o=(0, 0, 0), Ms=1.4e6, K1=0.0, A=1.5e-11, alpha=0.05,
                 modules=1 | 2),
            dict(n=(nx // 2, ny // 2, 2), h=(4 * NM, 4 * NM, 2 * NM), o=(0, 0, 2 * NM), Ms=6e5, K1=0.0, A=1.5e-11,
                 alpha=0.05, modules=1 | 2),
            dict(n=(nx, ny, 1), h=(2 * NM, 2 * NM, 1.5 * NM), o=(0, 0, 7 * NM), Ms=1.1e6, K1=3e5, A=1.5e-11, alpha=0.05,
                 modules=1 | 2 | 8)]


def _directions(n, rng, tilt):
    """Unit vectors per cell: tilted up to 15 degrees from +z, or uniform over the sphere."""
    if tilt:
        th = np.deg2rad(rng.uniform(0.0, 15.0, n))
        ph = rng.uniform(0.0, 2 * np.pi, n)
        return np.stack([np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)], axis=1)
    v = rng.standard_normal((n, 3))
    return v / np.linalg.norm(v, axis=1)[:, None]


def _m0(case, seed):
    """Initial M (A/m, FP64 host arrays) of every mesh, rounded to the precision that the pass receives."""
    rng = np.random.default_rng(seed)
    if case["kind"] in ("batch", "stack"):
        meshes = _batch_systems(case) if case["kind"] == "batch" else _stack_meshes(case)
        out = [_directions(int(np.prod(m["n"])), rng, case["kind"] == "stack") * m["Ms"] for m in meshes]
    else:
        tilt = case["kind"] == "run" and (case["D"] != 0.0 or case["ode"] == "RKDP54")
        out = [_directions(case["nx"] * case["ny"] * case["nz"], rng, tilt) * case["Ms"]]
    if case["prec"] == "mixed" and case["kind"] != "heff":
        out = [m.astype(np.float32).astype(np.float64) for m in out]
    return out


def _adjoint_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = case["nx"] * case["ny"]
    g = rng.standard_normal((case["ny"], case["nx"]))
    kx = 2 * np.pi * np.fft.fftfreq(case["nx"], d=case["hx"])
    ky = 2 * np.pi * np.fft.fftfreq(case["ny"], d=case["hy"])
    g = np.real(np.fft.ifft2(np.fft.fft2(g) * np.exp(-(ky[:, None] ** 2 + kx[None, :] ** 2) * 20.0 ** 2 / 4)))
    g = (g - g.mean()) / g.std()
    Ms = 8e5 * (1 + 0.1 * np.clip(g, -4, 4).reshape(-1))
    return dict(Ms=Ms, K1=rng.uniform(0, 2e5, n), Ha=rng.normal(0, 5e3, 3), m0=_directions(n, rng, True),
                target=_directions(n, rng, False))


# ------------------------------------------------------------------------------------ prepare and run
def _check(rc):
    if rc != 0:
        raise RuntimeError("boris_b200 error %d: %s" % (rc, bm.lib().bm_last_error().decode()))


def _context(case, meshes):
    c = bm.Context(device=0, precision=bm.FP64 if case["prec"] == "fp64" else bm.MIXED)
    for q, m in enumerate(meshes):
        c.add_mesh(m["n"], m["h"], m["o"])
        c.set_material(q, Ms=m["Ms"], A=m["A"], alpha=m["alpha"], K1=m["K1"], ea=(0, 0, 1), D=m.get("D", 0.0))
        c.set_modules(q, m["modules"])
        c.set_field(q, m.get("Ha", (0.0, 0.0, 0.0)))
        if m.get("pbc"):
            c.set_pbc(q, (m["pbc"], m["pbc"], 0))
    return c


def _mesh(case):
    modules = bm.DEMAG
    if case["kind"] != "field":
        modules |= bm.IDMI if case["D"] else bm.EXCH
        modules |= bm.ZEEMAN if case["Hx"] else 0
        modules |= bm.ANIUNI if case["K1"] else 0
    return dict(n=_n(case), h=_h(case), o=(0.0, 0.0, 0.0), Ms=case["Ms"], A=case.get("A", 0.0),
                alpha=case.get("alpha", 0.1), K1=case.get("K1", 0.0), D=case.get("D", 0.0), modules=modules,
                Ha=(case.get("Hx", 0.0), 0.0, 0.0), pbc=case.get("pbc", 0))


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda")
    dtype = torch.float64 if case["prec"] == "fp64" else torch.float32
    s = dict(case=case)
    if kind == "adjoint":
        p = _adjoint_inputs(case, seed)
        c = bm.Context(device=0, precision=bm.FP64 if case["prec"] == "fp64" else bm.MIXED)
        c.add_mesh(_n(case), _h(case))
        c.set_material(0, Ms=8e5, A=case["A"], alpha=case["alpha"], ea=(0, 0, 1))
        c.set_material_maps(0, Ms_map=p["Ms"], K1_map=p["K1"])
        c.set_modules(0, bm.DEMAG | bm.EXCH | bm.ANIUNI | bm.ZEEMAN)
        c.set_field(0, p["Ha"])
        c.setode("RK4", case["dt"])
        c.set_m(p["m0"] * p["Ms"][:, None])
        c.prepare()
        s.update(c=c, target=p["target"], m=torch.from_numpy(p["m0"] * p["Ms"][:, None]).to(dev, dtype))
        return s
    m0 = _m0(case, seed)
    if kind == "batch":
        meshes = _batch_systems(case)
        c = _context(case, meshes)
        c.set_batched(True)
        c.setode("RK4", case["dt"])
    elif kind == "stack":
        meshes = _stack_meshes(case)
        c = _context(case, meshes)
        c.multiconvolution(bm.ML_3D)
        c.setode("RKDP54", 5e-15)
        c.astepctrl(1e-5, 2.0, 1e-15, DT_MAX)
    else:
        meshes = [_mesh(case)]
        c = _context(case, meshes)
        if kind == "run":
            c.setode(case["ode"], case["dt"])
            if case["ode"] == "RKDP54":
                c.astepctrl(case["tol"], 2.0, 1e-15, DT_MAX)
            if case["es"]:
                c.evalspeedup(case["es"])
    for q, m in enumerate(m0):
        c.set_m(m, q)
    c.prepare()
    s["c"] = c
    if kind == "heff":
        s["m"] = m0[0]
        return s
    s["m"] = [torch.from_numpy(m).to(dev, dtype) for m in m0]
    s["out"] = [torch.empty_like(m) for m in s["m"]]
    if kind in ("run", "batch"):
        s["dt"] = case["dt"]
    elif kind == "stack":
        s["dt"] = 5e-15
    return s


def run(s):
    case, c = s["case"], s["c"]
    kind, h, L = case["kind"], s["c"]._h, bm.lib()
    eb = 8 if case["prec"] == "fp64" else 4
    if kind == "field":
        e = ctypes.c_double(0.0)
        _check(L.bm_demag_field_device(h, 0, s["m"][0].data_ptr(), s["out"][0].data_ptr(), eb, 0,
                                       ctypes.byref(e) if case["energy"] else None, None))
        return (s["out"][0], e.value) if case["energy"] else s["out"][0]
    if kind == "heff":
        c.set_m(s["m"])
        return c.update_field()
    if kind == "adjoint":
        _check(L.bm_set_m_device(h, 0, s["m"].data_ptr(), eb, None))
        loss, dMs, dK1, dHa, _ = c.adjoint_rk4(s["target"], case["steps"], case["every"], True)
        return loss, dMs, dK1, dHa
    c.setdt(s["dt"])   # every pass starts from the same step
    for q, m in enumerate(s["m"]):
        _check(L.bm_set_m_device(h, q, m.data_ptr(), eb, None))
    c.run(case["steps"])
    for q, m in enumerate(s["out"]):
        _check(L.bm_get_m_device(h, q, m.data_ptr(), eb, None))
    return s["out"]


# ------------------------------------------------------------------------------------ work and tolerance
def _nice(n):
    b = 1
    while b < n:
        b *= 2
    t = 3
    while t < b:
        if t >= n:
            return t
        t *= 2
    return b


def _eval_work(n, p):
    """(bytes, flops) of one effective-field evaluation: M read, the field or rhs written, the six (2D:
    four) real kernel components read once; six padded real transforms, the 3 x 3 product, the stencils."""
    cells = n[0] * n[1] * n[2]
    N = [2 * _nice(v) if v > 1 else 1 for v in n]
    spec = (N[0] // 2 + 1) * (N[1] // 2 + 1) * (N[2] // 2 + 1)
    tot = N[0] * N[1] * N[2]
    return 6 * p * cells + (6 if n[2] > 1 else 4) * p * spec, 15.0 * tot * math.log2(max(tot, 2)) + 30.0 * tot / 2 + 100.0 * cells


def work(case):
    p = 8 if case["prec"] == "fp64" else 4
    kind = case["kind"]
    if kind == "batch":
        meshes = _batch_systems(case)
    elif kind == "stack":
        meshes = _stack_meshes(case)
    else:
        meshes = [dict(n=_n(case))]
    evals = 1
    if kind == "run":
        per = 6 if case["ode"] == "RKDP54" else 4
        evals = per * case["steps"]
        if case["es"]:
            # full fields until es are saved, then one per step
            evals = per * (case["es"] - 1) + max(0, case["steps"] - case["es"] + 1)
    elif kind == "batch":
        evals = 4 * case["steps"]
    elif kind == "stack":
        evals = 6 * case["steps"]
    elif kind == "adjoint":
        evals = 3 * 4 * case["steps"]   # forward, recompute, transposed
    by = fl = 0.0
    for m in meshes:
        b, f = _eval_work(m["n"], p)
        by += b * evals
        fl += f * evals
    return {"bytes": by, "flops": fl}


def tolerance(case):
    # FP32 fields and states are within 4e-7 of FP64 (fields 2e-7, M after 100 steps 4e-7), the adjoint's
    # gradients, sums of many such terms, within 3e-6; two FP64 orders of summation differ by 1e-13
    if case["prec"] == "fp64":
        return {"rel": 1e-11, "max": 1e-9}
    return {"rel": 1.2e-5, "max": 1e-3} if case["kind"] == "adjoint" else {"rel": 1.6e-6, "max": 1e-4}


# ------------------------------------------------------------------------------------ exact
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _newell_f(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    R = torch.sqrt(x2 + y2 + z2)
    one = torch.ones_like(R)
    rxz, rxy = torch.sqrt(x2 + z2), torch.sqrt(x2 + y2)
    out = (2 * x2 - y2 - z2) * R / 6
    out = out + 0.5 * y * (z2 - x2) * torch.asinh(y / torch.where(rxz > 0, rxz, one)) * (rxz > 0)
    out = out + 0.5 * z * (y2 - x2) * torch.asinh(z / torch.where(rxy > 0, rxy, one)) * (rxy > 0)
    den = x * R
    return out - x * y * z * torch.atan(y * z / torch.where(den != 0, den, one)) * (den != 0)


def _newell_g(x, y, z):
    x2, y2, z2 = x * x, y * y, z * z
    R = torch.sqrt(x2 + y2 + z2)
    one = torch.ones_like(R)

    def div(a, b):
        return a / torch.where(b != 0, b, one) * (b != 0)

    rxy, ryz, rxz = torch.sqrt(x2 + y2), torch.sqrt(y2 + z2), torch.sqrt(x2 + z2)
    out = -x * y * R / 3 + x * y * z * torch.asinh(div(z, rxy))
    out = out + y * (3 * z2 - y2) * torch.asinh(div(x, ryz)) / 6 + x * (3 * z2 - x2) * torch.asinh(div(y, rxz)) / 6
    out = out - z2 * z * torch.atan(div(x * y, z * R)) / 6 - y2 * z * torch.atan(div(x * z, y * R)) / 2
    return out - x2 * z * torch.atan(div(y * z, x * R)) / 2


def _newell(x, y, z, h):
    """-N of two cells of size h at the offset (x, y, z): the 27-point second differences."""
    f = [0, 0, 0, 0, 0, 0]
    cw = (-1.0, 2.0, -1.0)
    for a in (-1, 0, 1):
        for b in (-1, 0, 1):
            for c in (-1, 0, 1):
                X, Y, Z = x + a * h[0], y + b * h[1], z + c * h[2]
                w = -cw[a + 1] * cw[b + 1] * cw[c + 1] / (4 * math.pi * h[0] * h[1] * h[2])
                v = (_newell_f(X, Y, Z), _newell_f(Y, X, Z), _newell_f(Z, Y, X), _newell_g(X, Y, Z), _newell_g(X, Z, Y),
                     _newell_g(Y, Z, X))
                f = [p + w * q for p, q in zip(f, v)]
    return f


def _far(x, y, z, h):
    """The same far from the origin: the dipole tensor under the three-point Gauss rule of the double
    cell average's triangular weight per axis."""
    f = [0, 0, 0, 0, 0, 0]
    a = math.sqrt(0.4)
    rule = ((-a, 5.0 / 24), (0.0, 7.0 / 12), (a, 5.0 / 24))
    for qx, wx in rule:
        for qy, wy in rule:
            for qz, wz in rule:
                X, Y, Z = x + qx * h[0], y + qy * h[1], z + qz * h[2]
                r2 = X * X + Y * Y + Z * Z
                r5 = r2 ** -2.5 * (wx * wy * wz * h[0] * h[1] * h[2] / (4 * math.pi))
                v = (3 * X * X - r2, 3 * Y * Y - r2, 3 * Z * Z - r2, 3 * X * Y, 3 * X * Z, 3 * Y * Z)
                f = [p + q * r5 for p, q in zip(f, v)]
    return f


NEAR = 16   # cells per axis within which the tensor is the Newell form


def _octant(n, h, z0=0.0):
    """The tensor at the offsets (i hx, j hy, z0 + k hz), i < n[0] and so on: six arrays [k][j][i]."""
    hm = max(h)
    g = [v / hm for v in h]
    ax = [torch.arange(v, dtype=torch.float64, device=_dev()) * s for v, s in zip(n, g)]
    ax[2] = ax[2] + z0 / hm
    x, y, z = ax[0][None, None, :], ax[1][None, :, None], ax[2][:, None, None]
    shape = (n[2], n[1], n[0])
    far = [v.expand(shape).clone() for v in _far(x, y, torch.where(z.abs() + x + y == 0, z + 1.0, z), g)]
    k = [min(v, NEAR) for v in n]
    if z0 / hm < NEAR * g[2]:
        near = _newell(x[:, :, :k[0]], y[:, :k[1]], z[:k[2]], g)
        for p, q in zip(far, near):
            p[:k[2], :k[1], :k[0]] = q
    return far


ODD = ((0, 0, 0), (0, 0, 0), (0, 0, 0), (1, 1, 0), (1, 0, 1), (0, 1, 1))   # xx, yy, zz, xy, xz, yz: odd along x, y, z


def _padded(octant, n, N):
    """Offsets -(n-1) .. n-1 of the octant on the N grid, by the parity of each component."""
    out = []
    for D, odd in zip(octant, ODD):
        for axis, dim in ((0, 2), (1, 1), (2, 0)):
            L = N[axis]
            if L == 1:
                continue
            P = torch.zeros([L if d == dim else D.shape[d] for d in range(3)], dtype=D.dtype, device=D.device)
            m = n[axis]
            P.narrow(dim, 0, m).copy_(D)
            if m > 1:
                P.narrow(dim, L - m + 1, m - 1).copy_(D.narrow(dim, 1, m - 1).flip(dim) * (-1.0 if odd[axis] else 1.0))
            D = P
        out.append(D)
    return out


def _pbc_octant(n, h, images):
    """Octant of the image-summed tensor along x and y (period n): sum over the images of the tensor made
    even or odd about the origin, the two ends of the range with half weight."""
    X = images
    big = _octant(((X + 2) * n[0], (X + 2) * n[1], n[2]), h)
    out = []
    for D, odd in zip(big, ODD):
        for axis, dim in ((0, 2), (1, 1)):
            m = n[axis]
            i0 = torch.arange(m, device=D.device)
            S = 0
            for q in range(-X - 1, X + 1):
                off = q * m + i0
                w = torch.where((off.new_tensor(q) == -X - 1) | (off.new_tensor(q) == X), 0.5, 1.0)
                wv = torch.full((m,), 1.0, dtype=D.dtype, device=D.device) * w
                wv[0] = 0.0 if q == -X - 1 else 1.0
                sign = torch.where(off < 0, -1.0 if odd[axis] else 1.0, 1.0).to(D.dtype) * wv
                shape = [1, 1, 1]
                shape[dim] = m
                S = S + D.index_select(dim, off.abs()) * sign.reshape(shape)
            if odd[axis]:
                S.narrow(dim, 0, 1).zero_()
            D = S
        out.append(D)
    return out


class _Demag:
    """Open or periodic demag field of M [3][nz][ny][nx] by the padded FFT convolution."""

    def __init__(self, n, h, pbc=0, octant=None):
        self.n = n
        self.N = [2 * v if v > 1 else 1 for v in n]
        oc = octant if octant is not None else _pbc_octant(n, h, pbc) if pbc else _octant(n, h)
        self.S = [float(oc[c][0, 0, 0]) for c in range(3)]
        self.K = [torch.fft.rfftn(P) for P in _padded(oc, n, self.N)]
        self.real = octant is None

    def __call__(self, M):
        N, n = self.N, self.n
        F = torch.fft.rfftn(M, s=(N[2], N[1], N[0]), dim=(1, 2, 3))
        k = self.K
        G = torch.stack([k[0] * F[0] + k[3] * F[1] + k[4] * F[2], k[3] * F[0] + k[1] * F[1] + k[5] * F[2],
                         k[4] * F[0] + k[5] * F[1] + k[2] * F[2]])
        return torch.fft.irfftn(G, s=(N[2], N[1], N[0]), dim=(1, 2, 3))[:, :n[2], :n[1], :n[0]]


def _axis(M, dim, h, bd, wrap):
    """Second and first derivative along one axis: central inside; at a face the missing neighbour is the
    far side (wrap) or given by the boundary slope bd."""
    m = M.shape[dim]
    if m == 1:
        return torch.zeros_like(M), torch.zeros_like(M)
    up, dn = torch.roll(M, -1, dim), torch.roll(M, 1, dim)
    if wrap:
        return (up + dn - 2 * M) / h ** 2, (up - dn) / (2 * h)
    idx = torch.arange(m, device=M.device)
    shape = [1] * M.dim()
    shape[dim] = m
    lo, hi = (idx == 0).reshape(shape), (idx == m - 1).reshape(shape)
    d2 = torch.where(lo, (up - M - bd * h) / h ** 2, torch.where(hi, (dn - M + bd * h) / h ** 2, (up + dn - 2 * M) / h ** 2))
    g = torch.where(lo, 0.5 * ((up - M) / h + bd), torch.where(hi, 0.5 * ((M - dn) / h + bd), (up - dn) / (2 * h)))
    return d2, g


def _local(M, h, Ms, A, K1, D, Ha, pbc):
    """Exchange (interfacial DMI), uniaxial anisotropy along z and the applied field; Ms, K1 numbers or maps."""
    H = Ha.reshape(3, 1, 1, 1) + torch.zeros_like(M)
    z = torch.zeros_like(M[0])
    rr = D / (2 * A) if D else 0.0
    bx = torch.stack([rr * M[2], z, -rr * M[0]])
    by = torch.stack([z, rr * M[2], -rr * M[1]])
    dx, gx = _axis(M, 3, h[0], bx, pbc)
    dy, gy = _axis(M, 2, h[1], by, pbc)
    dz, _ = _axis(M, 1, h[2], torch.zeros_like(M), False)
    H = H + (2 * A / MU0) / Ms ** 2 * (dx + dy + dz)
    if D:
        H = H - (2 * D / MU0) / Ms ** 2 * torch.stack([gx[2], gy[2], -gx[0] - gy[1]])
    aniso = (2 / MU0) * K1 * M[2] / Ms ** 2
    return H + torch.stack([z, z, aniso])


def _llg(M, H, Ms, alpha):
    mxh = torch.linalg.cross(M, H, dim=0)
    return -GAMMA / (1 + alpha ** 2) * (mxh + (alpha / Ms) * torch.linalg.cross(M, mxh, dim=0))


def _renorm(M, Ms):
    return M * (Ms / torch.sqrt((M * M).sum(0, keepdim=True)))


def _rk4(M, f, Ms, dt, steps):
    for _ in range(steps):
        # one step at a time is kept for the gradients, and its inside recomputed
        M = (torch.utils.checkpoint.checkpoint(_rk4_step, M, f, Ms, dt, use_reentrant=False) if M.requires_grad
             else _rk4_step(M, f, Ms, dt))
    return M


def _rk4_step(M, f, Ms, dt):
    k1 = f(M, 0)
    k2 = f(M + 0.5 * dt * k1, 1)
    k3 = f(M + 0.5 * dt * k2, 2)
    k4 = f(M + dt * k3, 3)
    return _renorm(M + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4), Ms)


A54 = ((0.2,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9), (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
       (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
       (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
B54 = ((0, 5179 / 57600), (2, 7571 / 16695), (3, 393 / 640), (4, -92097 / 339200), (5, 187 / 2100))


def _rkdp54(Ms_list, fs, Ms, dt, tol, steps):
    """Adaptive Dormand-Prince steps of several meshes with one step size. Ms_list: their M."""
    M, base, k, primed, done, tries = list(Ms_list), None, None, False, 0, 0
    while done < steps and tries < 20 * steps:
        tries += 1
        k0 = fs(M)
        if primed:
            lte = 0.0
            for q in range(len(M)):
                pred = base[q] + dt * (sum(b * k[i][q] for i, b in B54) + k0[q] / 40)
                e = torch.sqrt(((M[q] - pred) ** 2).sum(0)) / torch.sqrt((M[q] ** 2).sum(0))
                lte = max(lte, float(e.max()))
            c = (0.8 * tol / lte) ** (1 / 6) if lte > 0 else 2.0
            if lte > tol and dt > 1e-15:
                M, primed, done = base, False, done - 1
                dt = max(dt * max(c, 0.01), 1e-15)
                continue
            dt = min(max(dt * max(min(c, 2.0), 0.01), 1e-15), DT_MAX)
        primed, base, k = True, M, [k0]
        for s in range(6):
            M = [base[q] + dt * sum(a * k[i][q] for i, a in enumerate(A54[s]) if a) for q in range(len(base))]
            if s < 5:
                k.append(fs(M))
        M = [_renorm(m, ms) for m, ms in zip(M, Ms)]
        done += 1
    return M


def _planes(aos, n):
    return torch.as_tensor(aos, dtype=torch.float64, device=_dev()).reshape(n[2], n[1], n[0], 3).permute(3, 0, 1, 2).contiguous()


def _aos(M):
    return M.permute(1, 2, 3, 0).reshape(-1, 3)


class _Speedup:
    """Demag field saved at the first evaluation of every step (without the self term), extrapolated by
    Lagrange weights at the others once `level` are saved."""

    def __init__(self, demag, level, dt):
        self.d, self.K, self.dt, self.t, self.saved = demag, level, dt, 0.0, []
        self.S = torch.tensor(demag.S, dtype=torch.float64, device=_dev()).reshape(3, 1, 1, 1)

    def __call__(self, M, stage):
        if stage == 0:
            H = self.d(M)
            self.saved = (self.saved + [(self.t, H - self.S * M)])[-self.K:]
            self.t0, self.t = self.t, self.t + self.dt
            return H
        if len(self.saved) < self.K:
            return self.d(M)
        t = self.t0 + (0.0, 0.5, 0.5, 1.0)[stage] * self.dt
        H = self.S * M
        for i, (ti, Hi) in enumerate(self.saved):
            w = 1.0
            for j, (tj, _) in enumerate(self.saved):
                if j != i:
                    w *= (t - tj) / (ti - tj)
            H = H + w * Hi
        return H


def _exact_adjoint(case, seed):
    n, h, p = _n(case), _h(case), _adjoint_inputs(case, seed)
    d, dev = _Demag(n, h), _dev()
    Ms = torch.as_tensor(p["Ms"], device=dev).reshape(n[2], n[1], n[0]).clone().requires_grad_()
    K1 = torch.as_tensor(p["K1"], device=dev).reshape(n[2], n[1], n[0]).clone().requires_grad_()
    Ha = torch.as_tensor(p["Ha"], device=dev).clone().requires_grad_()
    M = Ms * _planes(p["m0"], n)
    f = lambda X, s: _llg(X, d(X) + _local(X, h, Ms, case["A"], K1, 0.0, Ha, False), Ms, case["alpha"])  # noqa: E731
    M = _rk4(M, f, Ms, case["dt"], case["steps"])
    loss = ((M / Ms - _planes(p["target"], n)) ** 2).sum() / (n[0] * n[1] * n[2])
    loss.backward()
    return (float(loss.detach()), Ms.grad.reshape(-1).cpu().numpy(), K1.grad.reshape(-1).cpu().numpy(),
            Ha.grad.reshape(1, 3).cpu().numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    m0 = _m0(case, seed)
    if kind == "batch":
        out = []
        for m, a in zip(_batch_systems(case), m0):
            d = _Demag(m["n"], m["h"])
            zero = torch.zeros(3, dtype=torch.float64, device=_dev())
            f = lambda X, s: _llg(X, d(X) + _local(X, m["h"], m["Ms"], m["A"], 0.0, 0.0, zero, False),  # noqa: E731
                                  m["Ms"], m["alpha"])
            out.append(_aos(_rk4(_planes(a, m["n"]), f, m["Ms"], case["dt"], case["steps"])))
        return out
    if kind == "stack":
        return _exact_stack(case, m0) if case["same"] else None   # the mesh transfer's weights are the package's own rule
    n, h, Ms = _n(case), _h(case), case["Ms"]
    M = _planes(m0[0], n)
    d = _Demag(n, h, case.get("pbc", 0))
    if kind == "field":
        H = d(M)
        e = -MU0 * float((M * H).sum()) / (2.0 * n[0] * n[1] * n[2])
        return (_aos(H), e) if case["energy"] else _aos(H)
    Ha = torch.tensor([case["Hx"], 0.0, 0.0], dtype=torch.float64, device=_dev())
    local = lambda X: _local(X, h, Ms, case["A"], case["K1"], case["D"], Ha, case["pbc"] > 0)  # noqa: E731
    if kind == "heff":
        return _aos(d(M) + local(M)).cpu().numpy()
    if case["ode"] == "RK4":
        hd = _Speedup(d, case["es"], case["dt"]) if case["es"] else lambda X, s: d(X)
        f = lambda X, s: _llg(X, hd(X, s) + local(X), Ms, case["alpha"])  # noqa: E731
        return [_aos(_rk4(M, f, Ms, case["dt"], case["steps"]))]
    fs = lambda Xs: [_llg(Xs[0], d(Xs[0]) + local(Xs[0]), Ms, case["alpha"])]  # noqa: E731
    return [_aos(_rkdp54([M], fs, [Ms], case["dt"], case["tol"], case["steps"])[0])]


def _exact_stack(case, m0):
    """Layers on one grid: the demag field of a layer is the sum over the layers of 2D convolutions with
    the tensor at their distance in z."""
    meshes = _stack_meshes(case)
    n, h = meshes[0]["n"], meshes[0]["h"]
    kernels = {}
    for a in meshes:
        for b in meshes:
            dz = a["o"][2] - b["o"][2]
            key = round(abs(dz) / NM, 6)
            if key not in kernels:
                kernels[key] = _Demag(n, h, octant=_octant(n, h, abs(dz)))
    zero = torch.zeros(3, dtype=torch.float64, device=_dev())
    flip = torch.tensor([1.0, 1.0, -1.0], dtype=torch.float64, device=_dev()).reshape(3, 1, 1, 1)

    def fs(Ms_):
        out = []
        for a, X in zip(meshes, Ms_):
            H = 0
            for b, Y in zip(meshes, Ms_):
                dz = a["o"][2] - b["o"][2]
                k = kernels[round(abs(dz) / NM, 6)]
                # below the source the components odd in z change sign: mirror M and H in z
                H = H + (k(Y) if dz >= 0 else flip * k(flip * Y))
            out.append(_llg(X, H + _local(X, h, a["Ms"], a["A"], a["K1"], 0.0, zero, False), a["Ms"], a["alpha"]))
        return out

    M = _rkdp54([_planes(m, n) for m in m0], fs, [m["Ms"] for m in meshes], 5e-15, 1e-5, case["steps"])
    return [_aos(m) for m in M]
