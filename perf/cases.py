"""The work that users of this framework have it do, as measurable cases.

Each case is a dict of plain values; ``prepare`` makes what a user's program
holds before the call, ``run`` is one call through the public entry points,
``exact`` the same result in plain float64 numpy / torch where there is one.
Arrays on the device are laid out as the library takes them: a (rows, cols)
column-major matrix is a contiguous (cols, rows) tensor, so the first index
is x and the second z.
"""
import ctypes
import math

import numpy as np
import torch

import xcore_gb300 as xc
import xcore_gb300.learned as learned

EPS = 2.0 ** -52
DEV = "cuda"


def listed():
    return [
        # one field of the 100^2 box (100 steps of it is the parity run): the
        # smallest grid a stencil is called on, where a call's latency counts
        dict(name="advect_weno5_100", kind="advect", scheme="weno5", Nz=100, Nx=100),
        # the same call on the 1024^2 grid of the mixed-precision workload
        dict(name="advect_weno5_1024", kind="advect", scheme="weno5", Nz=1024, Nx=1024),
        # diffusion of a halo'd field with its face fluxes on a grid that no
        # tile divides
        dict(name="diffus_1000x517", kind="diffus", Nz=1000, Nx=517),
        # phase evolution (two advections, one diffusion, the implicit update)
        # of the 400^2 box with QUICK
        dict(name="phsevo_quick_400", kind="phsevo", scheme="quick", Nz=400, Nx=400),
        # the Ornstein-Uhlenbeck noise of a second or later Picard sweep on a
        # grid whose sides are no powers of two
        dict(name="noise_300x231", kind="noise", Nz=300, Nx=231),
        # the constitutive update of the 1024^2 workload
        dict(name="update_1024", kind="update", Nz=1024, Nx=1024),
        # one Stokes solve at the largest side of the ensemble, viscosity
        # contrast 1e4, FP32 iterations inside FP64 refinement
        dict(name="stokes_mixed_512", kind="stokes", solver="mixed", Nz=512, Nx=512, etacntr=1e4),
        # whole time steps (three Picard sweeps): the smallest ensemble
        # member, the 100^2 box with the plain FP64 solver (the API's default),
        # and the 1024^2 workload of the benchmark
        dict(name="step_mixed_64", kind="step", solver="mixed", Nz=64, Nx=64, etacntr=1e4, onediv=1),
        dict(name="step_fp64_100", kind="step", solver="fgmres64", Nz=100, Nx=100, etacntr=1e2, onediv=0),
        dict(name="step_mixed_1024", kind="step", solver="mixed", Nz=1024, Nx=1024, etacntr=1e4, onediv=1),
        # the widest layer of the preconditioner network on a training batch
        dict(name="conv_128_8x32x32", kind="conv", direction="fwd", B=8, H=32, W=32, Cin=128, Cout=128),
        # loss and gradients of the network on a training batch (8 images of 256^2)
        dict(name="unet_grad_8x256", kind="unet", B=8, N=256),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["advect", "diffus", "phsevo", "noise", "update", "stokes", "step", "conv", "unet"])
    c = dict(kind=kind)
    if kind in ("advect", "diffus", "phsevo"):
        if kind != "diffus":
            c["scheme"] = rng.choice(["weno5", "quick"])
        c.update(Nz=_side(rng, 64, 1024), Nx=_side(rng, 64, 1024))
    elif kind == "noise":
        c.update(Nz=_side(rng, 64, 600), Nx=_side(rng, 64, 600))
    elif kind == "update":
        c.update(Nz=_side(rng, 64, 1024), Nx=_side(rng, 64, 1024))
    elif kind in ("stokes", "step"):
        # the solver's grids: sides are multiples of 16 in every configuration
        # but the 100^2 and 400^2 boxes
        c.update(solver=rng.choice(["mixed", "mixed", "fgmres64"]), Nz=16 * rng.randint(4, 24),
                 Nx=16 * rng.randint(4, 24), etacntr=10.0 ** rng.randint(2, 4))
        if kind == "step":
            c["onediv"] = rng.randint(0, 1)
            if c["solver"] == "fgmres64":
                c.update(Nz=16 * rng.randint(4, 8), Nx=16 * rng.randint(4, 8))
    elif kind == "conv":
        W = rng.choice([16, 32, 64, 128, 256])
        c.update(direction=rng.choice(["fwd", "wgrad"]), B=rng.randint(1, 8), W=W,
                 H=max(1, 128 // W) * rng.randint(1, 128 // max(1, 128 // W)), Cin=rng.choice([16, 32, 64, 128]),
                 Cout=rng.choice([16, 32, 64, 128]))
    else:
        c.update(B=rng.randint(1, 8), N=rng.choice([128, 256]))
    return c


# ---------------------------------------------------------------------------
# inputs (numpy, from the seed alone; arrays are [x, z])
# ---------------------------------------------------------------------------
def _smooth(g, shape, width):
    """Unit-RMS random field smoothed over `width` cells."""
    z = g.standard_normal(shape)
    k = np.fft.fftfreq(shape[0])[:, None] ** 2 + np.fft.rfftfreq(shape[1])[None, :] ** 2
    z = np.fft.irfft2(np.fft.rfft2(z) * np.exp(-2.0 * (math.pi * width) ** 2 * k), s=shape)
    return z / np.sqrt(np.mean(z * z))


def _constants(Nz, Nx):
    """Grid and scales of a 10 m deep box (L0 = l0 = 3h, as every configuration has)."""
    D = 10.0
    h = D / Nz
    L0 = 3 * h
    return dict(Nz=Nz, Nx=Nx, D=D, h=h, L=Nx * h, L0=L0, l0=L0, L0h=(L0 + h) / 2, l0h=(L0 + h) / 2, D0=D / 10,
                bnd_w=L0 / 2 + D / 100, txi0=3200.0 * 1e-4 / 18 / 10.0, G0=1e-3, dt0=0.1 * h)


PHYS = dict(rhom0=2700.0, rhox0=3200.0, d0=0.01, g0=10.0, etam0=10.0, etax0=1e18, Xi=0.5, Ptop=1e5, alpha=0.9,
            etacntr=1e4, AA=((0.72, 0.19), (0.81, 0.20)), BB=((0.63, 0.37), (0.999, 0.001)),
            CC=((2.09, 0.09), (0.37, 1.45)))


def _state(k, scheme="weno5"):
    par = xc.Parameters(D=k["D"], N=k["Nz"], L=k["L"], x0=0.1, Da=0.0, L0=k["L0"], l0=k["l0"], ADVN=scheme, **PHYS)
    grid = xc.Grid(Nx=k["Nx"], Nz=k["Nz"], h=k["h"], D=k["D"], L=k["L"])
    return xc.State(par, grid=grid, scales={n: k[n] for n in ("L0", "l0", "L0h", "l0h", "D0", "txi0", "G0", "bnd_w",
                                                              "dt0")})


def _bind(st, names):
    """The fields `names` of a State as the caller's own tensors."""
    out = {}
    for n in names:
        (rows, cols), _ = st.shape(n)
        out[n] = torch.empty((cols, rows), dtype=torch.float64, device=DEV)
        out[n].copy_(torch.from_numpy(np.ascontiguousarray(st[n].T)))
    torch.cuda.synchronize()
    for n, t in out.items():
        st.bind(n, t)
    return out


def _fields(case, seed):
    """Host inputs of the stencil, phase-evolution, noise and update cases."""
    g = np.random.default_rng(seed)
    Nz, Nx, kind = case["Nz"], case["Nx"], case["kind"]
    k = _constants(Nz, Nx)
    C, ZF, XF, W, U, P = (Nx, Nz), (Nx, Nz + 1), (Nx + 1, Nz), (Nx + 2, Nz + 1), (Nx + 1, Nz + 2), (Nx + 2, Nz + 2)

    def crystals():   # lognormal crystal fraction, median 0.1
        return np.clip(np.exp(np.log(0.1) + 0.5 * (0.8 * _smooth(g, C, 4.0) + 0.6 * g.standard_normal(C))), 0.0, 0.4)

    def speed(shape):   # velocities of both signs, in metres per second
        return 1e-2 * (_smooth(g, shape, 12.0) + 0.1 * g.standard_normal(shape))

    def positive(shape, median):
        return median * np.exp(0.5 * _smooth(g, shape, 4.0))
    if kind == "advect":
        return k, dict(f=3000.0 * crystals(), u=speed(XF), w=speed(ZF))
    if kind == "diffus":
        return k, dict(f=crystals(), k=positive(C, 1e-3))
    if kind == "phsevo":
        x = crystals()
        m = 1.0 - x
        rho = 1.0 / (m / 2700.0 + x / 3200.0)
        X = rho * x
        zc = (np.arange(1, Nz + 1) - 0.5) * k["h"]
        return k, dict(x=x, m=m, rho=rho, X=X, M=rho - X, chi=x * rho / 3200.0, kx=positive(C, 1e-4),
                       Wx=speed(W), Wm=speed(W), Ux=speed(U), Um=speed(U), Xo=X * (1 + 1e-3 * _smooth(g, C, 3.0)),
                       Xoo=X * (1 + 1e-3 * _smooth(g, C, 3.0)), dXdto=_smooth(g, C, 3.0), dXdtoo=_smooth(g, C, 3.0),
                       bndshape=np.broadcast_to(np.exp((-zc + k["h"] / 2) / k["bnd_w"]), C).copy())
    if kind == "noise":
        x = crystals()
        return k, dict(V=positive(C, 1e-2), vx=positive(C, 1e-4), fReL=1.0 / (1.0 + positive(C, 0.5)),
                       ke=positive(C, 1e-3), ks=positive(C, 1e-5), chi=x, psieo=1e-3 * _smooth(g, C, 1.0),
                       psixo=1e-4 * _smooth(g, C, 1.0), psiso=1e-5 * _smooth(g, C, 1.0), re=g.standard_normal(C),
                       rs=g.standard_normal(C), chiw=np.clip(0.1 + 0.05 * _smooth(g, W, 3.0), 0.0, 1.0),
                       muw=np.clip(0.9 + 0.05 * _smooth(g, W, 3.0), 0.0, 1.0),
                       chiu=np.clip(0.1 + 0.05 * _smooth(g, U, 3.0), 0.0, 1.0),
                       muu=np.clip(0.9 + 0.05 * _smooth(g, U, 3.0), 0.0, 1.0))
    x = crystals()
    return k, dict(x=x, m=1.0 - x, W=speed(W), U=speed(U), P=1e2 * _smooth(g, P, 8.0), wx=1e-2 * speed(W),
                   wm=1e-3 * speed(W), eta=positive(C, 20.0), etas=positive(C, 20.0))


PHSEVO_OUT = ("X", "M", "x", "m", "advn_X", "advn_M", "advn_rho", "dffn_X", "Gx", "dXdt", "qx_advn_X", "qz_advn_X",
              "qx_advn_M", "qz_advn_M", "qx_dffn_X", "qz_dffn_X")
NOISE_OUT = ("psie", "psix", "psis", "xieu", "xiew", "xixu", "xixw", "xisu", "xisw", "xie", "xix", "xis")
UPDATE_OUT = ("rho", "rhow", "rhou", "chi", "mu", "chiw", "muu", "etamix", "eII", "V", "vx", "Div_V", "eta", "etae",
              "etas", "etat", "etaco", "etasw", "ke", "ks", "kx", "fReL", "ReL", "ReD", "fRel", "Red", "Rc", "Ra",
              "txx", "txz", "tII", "Drho", "Pl", "Pt")
STEP_OUT = ("W", "U", "P", "X", "M", "x", "rho", "eta", "kx", "psie", "psix", "psis", "Wx", "Ux")

# iterative solves end on a residual: these are the tolerances at which their
# results agree to rounding from one order of operations to another
RTOL = {"mixed": 1e-13, "fgmres64": 1e-12}


def _solver(case):
    if case["solver"] == "mixed":   # the benchmark's settings
        return dict(solver="mixed", rtol=RTOL["mixed"], maxit=400, inner_rtol=5e-2, inner_maxit=30, pressure_sweeps=1)
    return dict(solver="fgmres64", rtol=RTOL["fgmres64"])


def _workload(case, seed, onediv=0):
    """A State of the lognormal workload's physics after initialize!."""
    D = 10.0
    Nz, Nx = case["Nz"], case["Nx"]
    h = D / Nz
    par = xc.Parameters(D=D, N=Nz, L=Nx * h, etam0=10.0, x0=0.1, Da=0.0, L0=3 * h, l0=3 * h,
                        etacntr=float(case["etacntr"]), ADVN="weno5", TINT="bd2im")
    st = xc.State(par, weno_weights=onediv)
    g = np.random.default_rng(seed)
    x0 = np.clip(np.exp(np.log(0.1) + 0.5 * g.standard_normal((Nz, Nx))), 0.0, 0.4)
    st.initialize(x0, g.standard_normal((Nz, Nx)), g.standard_normal((Nz, Nx)))
    return st, g


# the network of the learned preconditioner: (input channels, output channels) per layer
NET = ((16, 16), (16, 16), (16, 32), (32, 32), (32, 64), (64, 64), (64, 128), (128, 128), (128, 64), (64, 64),
       (64, 32), (32, 32), (32, 16), (16, 16), (16, 16))


def _net_params(seed):
    g = np.random.default_rng(seed)
    parts = []
    for L, (ci, co) in enumerate(NET):
        fan = 9 * (4 if L == 0 else ci)
        parts.append(g.standard_normal(9 * ci * co) * math.sqrt(2.0 / fan))
        parts.append(0.05 * g.standard_normal(co))
    return np.concatenate(parts).astype(np.float32)


def _conv_inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    B, H, W, ci, co = (case[n] for n in ("B", "H", "W", "Cin", "Cout"))
    x = torch.randn((B, H, W, ci), generator=gen, device=DEV).to(torch.bfloat16)
    if case["direction"] == "fwd":
        w = (torch.randn((co, 9, ci), generator=gen, device=DEV) / (3 * ci ** 0.5)).to(torch.bfloat16)
        return x, w, torch.randn((co,), generator=gen, device=DEV)
    return x, torch.randn((B, H, W, co), generator=gen, device=DEV).to(torch.bfloat16), None


def _unet_inputs(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    B, N = case["B"], case["N"]
    inp = torch.randn((B, N, N, 4), generator=gen, device=DEV)
    inp[..., 3] = inp[..., 3].abs()      # the log-viscosity channel
    return inp, torch.randn((B, N, N, 3), generator=gen, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("advect", "diffus"):
        k, f = _fields(case, seed)
        Nz, Nx = case["Nz"], case["Nx"]
        s["h"] = k["h"]
        s["adv"] = torch.empty((Nx, Nz), dtype=torch.float64, device=DEV)
        s["qx"] = torch.empty((Nx + 1, Nz + 2), dtype=torch.float64, device=DEV)
        s["qz"] = torch.empty((Nx + 2, Nz + 1), dtype=torch.float64, device=DEV)
        if kind == "diffus":   # the caller's halo'd arrays
            f = {n: np.pad(np.pad(a, ((1, 1), (0, 0)), mode="wrap"), ((0, 0), (1, 1)), mode="edge")
                 for n, a in f.items()}
        s.update({n: torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for n, a in f.items()})
    elif kind in ("phsevo", "noise", "update"):
        k, f = _fields(case, seed)
        st = _state(k, case.get("scheme", "weno5"))
        for n, a in f.items():
            st[n] = a.T
        s.update(st=st, coefs=xc.time_coefs("bd2im", 3), dt=k["dt0"],
                 out=_bind(st, {"phsevo": PHSEVO_OUT, "noise": NOISE_OUT, "update": UPDATE_OUT}[kind]))
    elif kind == "stokes":
        st, _ = _workload(case, seed)
        coefs, dt = xc.time_coefs("bd2im", 1), st.scales["dt0"]
        st.store_previous()
        st.store_noise()
        st.snapshot()
        st.phsevo(coefs, dt)
        out = _bind(st, ("W", "U", "P", "MFS"))
        s.update(st=st, coefs=coefs, dt=dt, out=out, start={n: t.clone() for n, t in out.items()},
                 stream=torch.cuda.ExternalStream(st.stream_handle()), opts=_solver(case))
    elif kind == "step":
        st, g = _workload(case, seed, case["onediv"])
        Nz, Nx = case["Nz"], case["Nx"]
        draws = []
        for _ in range(6):   # white noise in pinned memory, (Nz, Nx) column-major
            t = torch.empty((Nx, Nz), dtype=torch.float64).pin_memory()
            t.copy_(torch.from_numpy(g.standard_normal((Nx, Nz))))
            draws.append(t.numpy().T)
        s.update(st=st, dt=st.scales["dt0"], k=0, draws=draws, out=_bind(st, STEP_OUT), opts=_solver(case))
    elif kind == "conv":
        x, w, b = _conv_inputs(case, seed)
        B, H, W, ci, co = (case[n] for n in ("B", "H", "W", "Cin", "Cout"))
        y = torch.empty((B, H, W, co), dtype=torch.bfloat16, device=DEV) if b is not None else \
            torch.empty((co, 9, ci), dtype=torch.float32, device=DEV)
        s.update(x=x, w=w, b=b, y=y)
    else:
        net = learned.Network(case["N"], case["N"], case["B"])
        net.set_params(_net_params(seed))
        inp, tgt = _unet_inputs(case, seed)
        s.update(net=net, inp=inp, tgt=tgt, grads=np.empty(net.nparams, dtype=np.float32))
    torch.cuda.synchronize()
    return s


def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _ok(status):
    if status != 0:
        raise RuntimeError(xc.lib().xc_last_error().decode())


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "advect":
        xc.advect_centered_with_flux(s["adv"], s["qx"], s["qz"], s["f"], s["u"], s["w"], s["h"], case["scheme"])
        return [s["adv"], s["qx"], s["qz"]]
    if kind == "diffus":
        xc.diffus_with_flux(s["adv"], s["qx"], s["qz"], s["f"], s["k"], s["h"])
        return [s["adv"], s["qx"], s["qz"]]
    if kind == "phsevo":
        s["st"].phsevo(s["coefs"], s["dt"])
        return s["out"]
    if kind == "noise":
        s["st"].noise(s["dt"], first_iter=False)
        return s["out"]
    if kind == "update":
        s["st"].update()
        return s["out"]
    if kind == "stokes":   # from the same initial guess each time
        with torch.cuda.stream(s["stream"]):
            for n, t in s["out"].items():
                t.copy_(s["start"][n])
        s["st"].fluidmech(s["coefs"], s["dt"], **s["opts"])
        return s["out"]
    if kind == "step":   # the next step of the run
        d = s["draws"]
        k = s["k"]
        info = s["st"].step(k + 1, s["dt"], d[2 * k % 6], d[(2 * k + 1) % 6], sweeps=3, **s["opts"])
        s["dt"], s["k"] = info["dt_next"], k + 1
        return dict(s["out"], dt=s["dt"])
    if kind == "conv":
        B, H, W, ci, co = (case[n] for n in ("B", "H", "W", "Cin", "Cout"))
        if case["direction"] == "fwd":
            _ok(xc.lib().xc_nn_conv3x3(_p(s["x"]), _p(s["w"]), _p(s["b"]), _p(s["y"]), None, B, H, W, ci, co, 1, None))
        else:
            _ok(xc.lib().xc_nn_conv3x3_wgrad(_p(s["x"]), _p(s["w"]), _p(s["y"]), B, H, W, ci, co, None))
        return s["y"]
    loss = ctypes.c_float()
    _ok(xc.lib().xc_nn_loss_grad(s["net"].h, _p(s["inp"]), _p(s["tgt"]), ctypes.byref(loss), None))
    _ok(xc.lib().xc_nn_get_grads(s["net"].h, s["grads"].ctypes.data))
    return dict(loss=loss.value, grads=s["grads"].copy())


def work(case):
    kind = case["kind"]
    if kind == "conv":
        px, ci, co = case["B"] * case["H"] * case["W"], case["Cin"], case["Cout"]
        out = 2 * px * co if case["direction"] == "fwd" else 36 * ci * co
        rest = 18 * ci * co if case["direction"] == "fwd" else 2 * px * co
        return dict(bytes=2 * px * ci + out + rest, flops=18.0 * px * ci * co)
    if kind == "unet":
        px = case["B"] * case["N"] ** 2
        level = (0, 0, 1, 1, 2, 2, 3, 3, 3, 2, 2, 1, 1, 0, 0)
        fwd = sum(18.0 * ci * co * px / 4 ** lv for (ci, co), lv in zip(NET, level))
        return dict(bytes=28 * px + 8 * sum(9 * a * b + b for a, b in NET), flops=3 * fwd)
    n = float(case["Nz"] * case["Nx"])
    # 8-byte fields read plus written per cell, and operations per cell
    fields = dict(advect=6, diffus=5, phsevo=32, noise=27, update=50, stokes=22, step=130)[kind]
    flops = dict(advect=150, diffus=22, phsevo=340, noise=400, update=600, stokes=2000, step=10000)[kind]
    return dict(bytes=8 * fields * n, flops=flops * n)


# ---------------------------------------------------------------------------
# the same results in plain float64
# ---------------------------------------------------------------------------
def _upwind(s, v, scheme):
    """Flux through the face between s[2] and s[3] of six neighbouring cells."""
    def weno5(a, b, c, d, e):
        p = ((2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6)
        be = (13 / 12 * (a - 2 * b + c) ** 2 + (a - 4 * b + 3 * c) ** 2 / 4,
              13 / 12 * (b - 2 * c + d) ** 2 + (b - d) ** 2 / 4,
              13 / 12 * (c - 2 * d + e) ** 2 + (3 * c - 4 * d + e) ** 2 / 4)
        w = [q / (EPS + t) ** 2 for q, t in zip((0.1, 0.6, 0.3), be)]
        return sum(x * y for x, y in zip(w, p)) / sum(w)
    if scheme == "weno5":
        pos, neg = weno5(*s[:5]), weno5(*s[:0:-1])
    else:
        pos, neg = (2 * s[3] + 5 * s[2] - s[1]) / 6, (2 * s[2] + 5 * s[3] - s[4]) / 6
    return np.maximum(v, 0) * pos + np.minimum(v, 0) * neg


def _padded_fluxes(fx, fz):
    """Face fluxes with the copied boundary rows (closed z) and columns (periodic x)."""
    return np.pad(fx, ((0, 0), (1, 1)), mode="edge"), np.pad(fz, ((1, 1), (0, 0)), mode="wrap")


def _advect(f, u, w, h, scheme):
    a = np.pad(np.pad(f, ((3, 3), (0, 0)), mode="wrap"), ((0, 0), (3, 3)), mode="edge")
    Nx, Nz = f.shape
    fx = _upwind([a[k:k + Nx + 1, 3:-3] for k in range(6)], u, scheme)
    fz = _upwind([a[3:-3, k:k + Nz + 1] for k in range(6)], w, scheme)
    return (fx[1:] - fx[:-1] + fz[:, 1:] - fz[:, :-1]) / h, fx, fz


def _diffuse(f, k, h):
    """Of halo'd f, k."""
    fx = -(k[1:, 1:-1] + k[:-1, 1:-1]) / 2 * (f[1:, 1:-1] - f[:-1, 1:-1]) / h
    fz = -(k[1:-1, 1:] + k[1:-1, :-1]) / 2 * (f[1:-1, 1:] - f[1:-1, :-1]) / h
    return -(fx[1:] - fx[:-1] + fz[:, 1:] - fz[:, :-1]) / h, fx, fz


def _halo(a):
    return np.pad(np.pad(a, ((1, 1), (0, 0)), mode="wrap"), ((0, 0), (1, 1)), mode="edge")


def _exact_phsevo(case, seed):
    k, f = _fields(case, seed)
    h, dt = k["h"], k["dt0"]
    scheme = case["scheme"]
    aX, fxX, fzX = _advect(f["X"], f["Ux"][:, 1:-1], f["Wx"][1:-1], h, scheme)
    aM, fxM, fzM = _advect(f["M"], f["Um"][:, 1:-1], f["Wm"][1:-1], h, scheme)
    d, fxd, fzd = _diffuse(_halo(f["chi"]), _halo(f["X"] * f["kx"]), h)
    G = k["G0"] * (1 - f["x"]) * f["bndshape"]
    r = -aX + d + G
    res = 1.5 * f["X"] - 2 * f["Xo"] + 0.5 * f["Xoo"] - r * dt
    X = np.clip(f["X"] - PHYS["alpha"] * res / 1.5, f["rho"] * EPS, f["rho"] * (1 - EPS))
    M = f["rho"] - X
    o = dict(X=X, M=M, x=X / f["rho"], m=M / f["rho"], advn_X=aX, advn_M=aM, advn_rho=aX + aM, dffn_X=d, Gx=G, dXdt=r)
    for n, fx, fz in (("advn_X", fxX, fzX), ("advn_M", fxM, fzM), ("dffn_X", fxd, fzd)):
        o["qx_" + n], o["qz_" + n] = _padded_fluxes(fx, fz)
    return o


def _exact_noise(case, seed):
    k, f = _fields(case, seed)
    h, dt, Xi, s = k["h"], k["dt0"], PHYS["Xi"], k["L0h"]
    te, ts = s / (2 * (f["V"] + EPS)), s / (2 * (f["vx"] + EPS))
    St = k["txi0"] / (te + EPS)
    sg = (Xi * np.sqrt(f["fReL"] * f["ke"] / te), Xi * np.sqrt(f["chi"] * f["fReL"] * f["ke"] / te * St / (1 + St * St)),
          Xi * np.sqrt(f["chi"] * f["ks"] / ts))
    amp = 2 / math.sqrt(1 - math.exp(-h * h / (2 * s * s)))
    o, flt = {}, []
    Nx, Nz = f["V"].shape
    pad = 4 * math.ceil(s / h)
    kz, kx = 2 * np.pi * np.fft.fftfreq(Nz + pad, h), 2 * np.pi * np.fft.fftfreq(Nx, h)
    spec = np.exp(-s * s * (kz[None, :] ** 2 + kx[:, None] ** 2))
    for n, t, a, r in (("psie", te, sg[0], "re"), ("psix", te, sg[1], "re"), ("psis", ts, sg[2], "rs")):
        F = np.exp(-dt / (1 / (1 / t + 1 / (100 * dt)) + dt))
        p = F * f[n + "o"] + np.sqrt(1 - F * F) * a * amp * f[r]
        o[n] = p
        q = np.fft.ifft2(np.fft.fft2(np.pad(p, ((0, 0), (0, pad)))) * spec).real[:, :Nz]
        flt.append((q - q.mean()) * (p.std(ddof=1) / q.std(ddof=1)) + p.mean())
    e, x, z = (_halo(q) for q in flt)
    co = (e[:-1, :-1] + e[1:, :-1] + e[:-1, 1:] + e[1:, 1:]) / 4
    o["xieu"] = np.pad(co[:, 1:] - co[:, :-1], ((0, 0), (1, 1)), mode="edge")
    o["xiew"] = np.pad(-(co[1:] - co[:-1]), ((1, 1), (0, 0)), mode="wrap")

    def taper(c, m):
        return (1 - np.exp(-c / 1e-4)) * (1 - np.exp(-np.maximum(0, m - 0.4) / 0.05))
    tu, tw = taper(f["chiu"], f["muu"]), taper(f["chiw"], f["muw"])
    for n, q in (("xix", x), ("xis", z)):
        o[n + "u"], o[n + "w"] = -(q[1:] - q[:-1]) * tu, -(q[:, 1:] - q[:, :-1]) * tw
    for n in ("xie", "xix", "xis"):
        w, u = o[n + "w"], o[n + "u"]
        o[n] = np.hypot((w[1:-1, :-1] + w[1:-1, 1:]) / 2, (u[:-1, 1:-1] + u[1:, 1:-1]) / 2)
    return o


def _exact_update(case, seed):
    k, f = _fields(case, seed)
    h, p = k["h"], PHYS
    x, m, W, U = f["x"], f["m"], f["W"], f["U"]
    rho = 1 / (m / p["rhom0"] + x / p["rhox0"])
    chi, mu = (np.clip(v * rho / r, EPS, 1 - EPS) for v, r in ((x, p["rhox0"]), (m, p["rhom0"])))
    f2, ee = (chi, mu), (p["etax0"], p["etam0"])
    S = [[(f2[b] / p["BB"][a][b]) ** (1 / p["CC"][a][b]) for b in (0, 1)] for a in (0, 1)]
    etamix = 0
    for a in (0, 1):
        Sf = [v / (S[a][0] + S[a][1]) for v in S[a]]
        w = p["AA"][a][0] * Sf[0] + p["AA"][a][1] * Sf[1]
        Xf = [w * f2[b] + (1 - w) * Sf[b] for b in (0, 1)]
        etamix = etamix + f2[a] * ee[a] * (ee[1 - a] / ee[a]) ** Xf[1 - a]
    ext = _halo

    def zavg(v):
        v = np.pad(v, ((0, 0), (1, 1)), mode="edge")
        return (v[:, 1:] + v[:, :-1]) / 2

    def xavg(v):
        v = np.pad(v, ((1, 1), (0, 0)), mode="wrap")
        return (v[1:] + v[:-1]) / 2
    rhow = zavg(rho)
    o = dict(rho=rho, rhow=rhow, rhou=xavg(rho), chi=chi, mu=mu, chiw=zavg(np.pad(chi, ((1, 1), (0, 0)), mode="wrap")),
             muu=xavg(np.pad(mu, ((0, 0), (1, 1)), mode="edge")), etamix=etamix)
    ref = rhow.mean(axis=0)
    t = ref[:-1] * p["g0"] * h
    pl = np.cumsum(np.concatenate(([t[0] / 2 + p["Ptop"]], t[1:])))
    o["Drho"] = rhow - ref
    o["Pl"] = np.broadcast_to(pl, rho.shape).copy()
    o["Pt"] = np.maximum(p["Ptop"] / 100, pl + f["P"][1:-1, 1:-1])
    exz = ((U[:, 1:] - U[:, :-1]) / h + (W[1:] - W[:-1]) / h) / 2
    du, dw = (U[1:, 1:-1] - U[:-1, 1:-1]) / h, (W[1:-1, 1:] - W[1:-1, :-1]) / h
    o["Div_V"] = du + dw
    exx, ezz = du - (du + dw) / 3, dw - (du + dw) / 3

    def four(a):
        return (a[:-1, :-1] + a[:-1, 1:] + a[1:, :-1] + a[1:, 1:]) / 4
    o["eII"] = np.sqrt(EPS + (exx ** 2 + ezz ** 2) / 2 + four(exz ** 2))
    V = np.hypot((W[1:-1, 1:] + W[1:-1, :-1]) / 2, (U[1:, 1:-1] + U[:-1, 1:-1]) / 2)
    vx = np.sqrt(((f["wx"][1:-1, 1:] + f["wx"][1:-1, :-1]) / 2) ** 2 + EPS)
    ke = o["eII"] * k["L0"] ** 2
    ReL = V * k["L0"] / (etamix / rho)
    fReL = -np.expm1(-ReL)
    etae = fReL * ke * rho
    ei = etamix + etae
    eta = 0.5 / (1 / (ei.min() * p["etacntr"]) + 1 / ei) + 0.5 * f["eta"]
    fRel = -np.expm1(-(vx * k["l0"] / (etamix / rho)))
    ks = vx * k["l0"]
    etat = fRel * ks * rho
    es = etamix + etat
    etas = 0.5 / (1 / (es.min() * p["etacntr"]) + 1 / es) + 0.5 * f["etas"]
    kx = ks + fReL * ke
    e = ext(eta)
    etaco = (e[:-1, :-1] * e[1:, :-1] * e[:-1, 1:] * e[1:, 1:]) ** 0.25
    s = np.pad(etas, ((0, 0), (1, 1)), mode="edge")
    txz, txx, tzz = etaco * exz, eta * exx, eta * ezz
    o.update(V=V, vx=vx, eta=eta, etae=etae, etas=etas, etat=etat, etaco=etaco, etasw=np.sqrt(s[:, 1:] * s[:, :-1]),
             ke=ke, ks=ks, kx=kx, fReL=fReL, ReL=ReL, ReD=V * k["D0"] / (eta / rho), fRel=fRel,
             Red=vx * p["d0"] / (etas / rho), Rc=V / np.maximum(vx, EPS), Ra=V * k["D0"] / kx, txx=txx, txz=txz,
             tII=np.sqrt(EPS + (txx ** 2 + tzz ** 2) / 2 + four(txz ** 2)))
    return o


def _conv64(x, w, b):
    """3x3 convolution in float64 of NCHW x with w [Cout][9][Cin]."""
    co, _, ci = w.shape
    return torch.nn.functional.conv2d(x, w.reshape(co, 3, 3, ci).permute(0, 3, 1, 2), b, padding=1)


def _exact_unet(case, seed):
    F = torch.nn.functional
    inp, tgt = _unet_inputs(case, seed)
    flat = torch.from_numpy(_net_params(seed)).to(DEV).double().requires_grad_(True)
    p, off = [], 0
    for ci, co in NET:
        p.append((flat[off:off + 9 * ci * co].reshape(co, 9, ci), flat[off + 9 * ci * co:off + 9 * ci * co + co]))
        off += 9 * ci * co + co

    def c(L, x):
        y = _conv64(x, *p[L])
        return y if L in (8, 10, 12, 14) else torch.relu(y)
    x = F.pad(inp.double().permute(0, 3, 1, 2), (0, 0, 0, 0, 0, 12))
    x0 = c(1, c(0, x))
    x1 = c(3, c(2, F.avg_pool2d(x0, 2)))
    x2 = c(5, c(4, F.avg_pool2d(x1, 2)))
    x3 = c(7, c(6, F.avg_pool2d(x2, 2)))

    def up(v):
        return F.interpolate(v, scale_factor=2, mode="nearest")
    y2 = c(9, up(c(8, x3)) + x2)
    y1 = c(11, up(c(10, y2)) + x1)
    y0 = c(13, up(c(12, y1)) + x0)
    d = c(14, y0)[:, :3] - tgt.double().permute(0, 3, 1, 2)
    loss = (d * d).sum() / (case["B"] * case["N"] ** 2)
    loss.backward()
    return dict(loss=loss.item(), grads=flat.grad.detach())


def exact(case, seed):
    kind = case["kind"]
    if kind == "advect":
        k, f = _fields(case, seed)
        a, fx, fz = _advect(f["f"], f["u"], f["w"], k["h"], case["scheme"])
        return [a, *_padded_fluxes(fx, fz)]
    if kind == "diffus":
        k, f = _fields(case, seed)
        a, fx, fz = _diffuse(_halo(f["f"]), _halo(f["k"]), k["h"])
        return [a, *_padded_fluxes(fx, fz)]
    if kind == "phsevo":
        return _exact_phsevo(case, seed)
    if kind == "noise":
        return _exact_noise(case, seed)
    if kind == "update":
        return _exact_update(case, seed)
    if kind == "conv":
        x, w, b = _conv_inputs(case, seed)
        xd = x.double().permute(0, 3, 1, 2)
        if b is not None:
            return torch.relu(_conv64(xd, w.double(), b.double())).permute(0, 2, 3, 1).contiguous()
        xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1))
        B, H, W, ci = x.shape
        d = w.double().reshape(-1, w.shape[-1])
        return torch.stack([d.T @ xp[:, t // 3:t // 3 + H, t % 3:t % 3 + W].reshape(-1, ci) for t in range(9)], dim=1)
    if kind == "unet":
        return _exact_unet(case, seed)
    return None   # whole solves and steps: a direct solve of these grids takes minutes
