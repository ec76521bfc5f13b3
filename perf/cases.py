"""Workloads that stand for what programs ask of this library, for timing them.

Every case goes through the Python front-end as a user's program does:

  matvec     Solver.matvec on device vectors: inside a caller's own Krylov method or
             design loop; FP64 or FP32, A or its transpose.  Grid sides 24 to 2048.
  solve      Solver.solve of a seeded GFIEM system (a thresholded Gaussian random field
             in the central 75 % square, plane wave), from host or device arrays.
  batch      solve_batch: a sweep of independent systems with uneven grid sides.
  gradient   topopt.Problem.value_and_gradient of two binary designs: per design the
             operator set-up, a forward solve, a transposed solve and one product
             with the Green's matrix.
  fno        learned.FNO.forward: the network as initial guess for a batch of systems.
  fno_grad   learned.FNO.loss_grad: one gradient of the network's training.

`listed` holds the named cases, `draw` gives further ones of the same ranges.
"""
import math

import numpy as np
import torch

import cugmres_b200 as cg
from cugmres_b200 import learned, topopt

SIDES = (96, 128, 192, 256, 384, 512)  # grid sides of the sweep

# the network's sizes: channels, features, hidden width, kept row and column modes, layers
CH, NIN, HID, M1, M2, LAYERS = 32, 4, 128, 16, 16, 4


def listed():
    return [
        # the smallest product: a caller's own iteration on a small grid, bound by latency
        dict(name="matvec_fp64_64", kind="matvec", N=64, precision="fp64", transpose=False),
        # an odd side whose transform length is well above 2N - 1, the adjoint's direction
        dict(name="matvec_fp64_t_385", kind="matvec", N=385, precision="fp64", transpose=True),
        # the product of the 1024 x 1024 benchmark system
        dict(name="matvec_fp64_1024", kind="matvec", N=1024, precision="fp64", transpose=False),
        # the largest grid, in the precision of its mixed-precision cycles
        dict(name="matvec_fp32_2048", kind="matvec", N=2048, precision="fp32", transpose=False),
        # plain unrestarted GMRES of a small system from NumPy arrays, to tolerance
        dict(name="solve_fp64_64", kind="solve", N=64, eps=2.25, lh=20.0, restart=500, max_iter=500, tol=1e-10,
             precision="fp64", ortho="dcgs2", transpose=False, host=True),
        # the default scheme on an ordinary grid, a restarted solve that its budget ends
        dict(name="solve_fp64_512", kind="solve", N=512, eps=4.0, lh=20.0, restart=100, max_iter=300, tol=1e-10,
             precision="fp64", ortho="dcgs2", transpose=False, host=False),
        # the 1024 x 1024 benchmark solve: s-step GMRES(100), 1000 steps
        dict(name="solve_sstep_1024", kind="solve", N=1024, eps=4.0, lh=20.0, restart=100, max_iter=1000, tol=1e-10,
             precision="fp64", ortho="sstep", transpose=False, host=False),
        # mixed precision on the largest grid: a scatterer of a few wavelengths, finely sampled, to tolerance
        dict(name="solve_mixed_2048", kind="solve", N=2048, eps=2.25, lh=2048 / 6.0, restart=50, max_iter=500,
             tol=1e-11, precision="mixed", ortho="dcgs2", transpose=False, host=False),
        # a sweep over designs and wavelengths on uneven grids
        dict(name="batch_sweep_10", kind="batch", nsys=10, sides="96,128,192,256,384,512", restart=50, max_iter=200),
        # two evaluations of a design search on a small grid
        dict(name="gradient_96", kind="gradient", N=96, eps=4.0, lh=20.0),
        # the initial guesses of a few systems on the network's training grid
        dict(name="fno_forward_256", kind="fno", N=256, batch=4),
        # one training gradient on the small grids that training runs on
        dict(name="fno_grad_64", kind="fno_grad", N=64, batch=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["matvec", "solve", "batch", "gradient", "fno", "fno_grad"], [8, 7, 2, 2, 2, 2])[0]
    lh = round(rng.uniform(15.0, 30.0), 2)
    if kind == "matvec":
        return dict(kind=kind, N=_log(rng, 24, 2048), precision=rng.choice(["fp64", "fp64", "fp32"]),
                    transpose=rng.random() < 0.3)
    if kind == "solve":
        # sizes at which a fixed number of steps gives an iterate that rounding hardly moves
        ortho = rng.choice(["dcgs2", "dcgs2", "sstep", "cgs2"])
        if rng.random() < 0.3:  # to tolerance: few wavelengths across the grid
            N = _log(rng, 48, 1024)
            return dict(kind=kind, N=N, eps=round(rng.uniform(1.5, 2.5), 2), lh=round(N / rng.uniform(3.0, 6.0), 2),
                        restart=rng.choice([50, 100, 200]), max_iter=500, tol=1e-11,
                        precision=rng.choice(["fp64", "mixed"]), ortho="dcgs2", transpose=rng.random() < 0.3,
                        host=rng.random() < 0.5)
        restart = 8 * rng.randint(3, 13)
        return dict(kind=kind, N=_log(rng, 256 if ortho == "sstep" else 128, 768), eps=round(rng.uniform(3.0, 12.0), 2), lh=lh, restart=restart,
                    max_iter=restart * rng.randint(1, 3), tol=1e-10, precision="fp64", ortho=ortho,
                    transpose=rng.random() < 0.3, host=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind=kind, nsys=rng.randint(2, 16),
                    sides=",".join(str(v) for v in sorted(rng.sample(SIDES, rng.randint(1, 3)))),
                    restart=rng.choice([30, 50, 75]), max_iter=rng.choice([100, 150, 200]))
    if kind == "gradient":
        return dict(kind=kind, N=rng.randint(48, 160), eps=round(rng.uniform(2.0, 6.0), 2), lh=lh)
    if kind == "fno":
        return dict(kind=kind, N=rng.choice([_log(rng, 32, 512), 1024]), batch=rng.randint(1, 6))
    return dict(kind=kind, N=_log(rng, 32, 160), batch=rng.randint(1, 16))


# ------------------------------------------------------------------ inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed, salt=0):
    return torch.Generator().manual_seed(1000003 * int(seed) + salt)


def _cnormal(shape, seed, salt):
    """Complex normal values, complex128, on the device."""
    v = torch.randn(*shape, 2, generator=_gen(seed, salt), dtype=torch.float64)
    return torch.view_as_complex(v).to(_device())


def _filter(N, corr):
    f = torch.fft.fftfreq(N, dtype=torch.float64, device=_device())
    return torch.exp(-2.0 * (math.pi * corr) ** 2 * (f[:, None] ** 2 + f[None, :] ** 2))


def _system(N, eps, lh, seed, salt=0):
    """Contrast, wavenumber, cell size and plane wave of one GFIEM system (wavelength 1)."""
    w = torch.randn(N, N, generator=_gen(seed, salt), dtype=torch.float64).to(_device())
    field = torch.fft.ifft2(torch.fft.fft2(w) * _filter(N, 4.0)).real
    lo = int(round(N / 8.0))
    chi = torch.zeros(N, N, dtype=torch.float64, device=_device())
    chi[lo:N - lo, lo:N - lo] = torch.where(field[lo:N - lo, lo:N - lo] > 0, eps - 1.0, 0.0)
    k0, h = 2.0 * math.pi, 1.0 / lh
    phase = k0 * h * (torch.arange(N, dtype=torch.float64, device=_device()) + 0.5)
    b = torch.polar(torch.ones_like(phase), phase)[:, None].repeat(1, N).contiguous()
    return dict(N=N, chi=chi, k0=k0, h=h, b=b)


def _sweep(case, seed):
    """The systems of one sweep: side, contrast and sampling drawn per system."""
    rng = np.random.default_rng(seed)
    sides = [int(v) for v in case["sides"].split(",")]
    out = []
    for i in range(case["nsys"]):
        # the sides take turns, so that the work does not depend on the seed
        out.append(_system(sides[i % len(sides)], float(rng.uniform(2.0, 12.0)), float(rng.uniform(15.0, 30.0)), seed,
                           salt=i + 1))
    return out


def _designs(case, seed):
    """Two binary designs in the central square of a grid, and two target cells outside it."""
    N = case["N"]
    lo, hi = N // 4, N - N // 4
    design = np.zeros((N, N), bool)
    design[lo:hi, lo:hi] = True
    xs = []
    for k in range(2):
        w = torch.randn(N, N, generator=_gen(seed, 11 + k), dtype=torch.float64).to(_device())
        field = torch.fft.ifft2(torch.fft.fft2(w) * _filter(N, 4.0)).real.cpu().numpy()
        xs.append(np.where(design & (field > 0), 1.0, 0.0))
    targets = [(N - 1 - N // 8, N // 2), (N // 2, N - 1 - N // 8)]
    return design, xs, targets


def _net_inputs(case, seed):
    """Parameters with activations of order one, and a batch (chi, k0 h, r, x)."""
    N, B = case["N"], case["batch"]
    rng = np.random.default_rng(seed)
    parts = [rng.standard_normal((CH, NIN)) / 2.0, 0.1 * rng.standard_normal(CH)]
    for _ in range(LAYERS):
        parts += [rng.standard_normal((2 * M1, M2, CH, CH, 2)) / 8.0, rng.standard_normal((CH, CH)) / math.sqrt(CH),
                  0.1 * rng.standard_normal(CH)]
    parts += [rng.standard_normal((HID, CH)) / math.sqrt(CH), 0.1 * rng.standard_normal(HID),
              rng.standard_normal((2, HID)) / math.sqrt(HID), 0.1 * rng.standard_normal(2)]
    params = np.concatenate([p.reshape(-1) for p in parts]).astype(np.float32)
    sysd = [_system(N, float(rng.uniform(2.0, 12.0)), float(rng.uniform(15.0, 30.0)), seed, salt=i + 1)
            for i in range(B)]
    chi = torch.stack([s["chi"] for s in sysd]).float()
    k0h = np.asarray([s["k0"] * s["h"] for s in sysd], np.float32)

    def smooth(salt, corr):
        v = torch.fft.ifft2(torch.fft.fft2(_cnormal((B, N, N), seed, salt)) * _filter(N, corr))
        return v / v.abs().square().mean(dim=(1, 2), keepdim=True).sqrt()

    x = smooth(101, 2.0)
    r = x + 0.5 * smooth(102, 1.0)
    return params, chi.contiguous(), k0h, r.to(torch.complex64).contiguous(), x.to(torch.complex64).contiguous()


def prepare(case, seed):
    kind, N = case["kind"], case.get("N")
    if kind == "matvec":
        p = _system(N, 4.0, 20.0, seed)
        s = cg.Solver(0).set_operator_green(N, p["chi"], p["k0"] ** 2, k0=p["k0"], h=p["h"])
        x = _cnormal((N, N), seed, 5)
        return dict(case=case, solver=s, x=x if case["precision"] == "fp64" else x.to(torch.complex64))
    if kind == "solve":
        p = _system(N, case["eps"], case["lh"], seed)
        s = cg.Solver(0).set_operator_green(N, p["chi"], p["k0"] ** 2, k0=p["k0"], h=p["h"])
        return dict(case=case, solver=s, b=p["b"].cpu().numpy() if case["host"] else p["b"])
    if kind == "batch":
        return dict(case=case, systems=[dict(chi=p["chi"].cpu().numpy(), chi_scale=p["k0"] ** 2, k0=p["k0"], h=p["h"],
                                             b=p["b"].cpu().numpy()) for p in _sweep(case, seed)])
    if kind == "gradient":
        p = _system(N, case["eps"], case["lh"], seed)
        design, xs, targets = _designs(case, seed)
        prob = topopt.Problem(cg.green_block("helmholtz", N, p["k0"], p["h"]), np.zeros((N, N)), design,
                              case["eps"] - 1.0, p["k0"] ** 2, p["b"].cpu().numpy())
        return dict(case=case, prob=prob, xs=xs, targets=targets)
    params, chi, k0h, r, x = _net_inputs(case, seed)
    net = learned.FNO(0, seed=0)
    net.set_params(params)
    net.set_params(params)  # again: the BF16 copies of the weights come from a vector that has surely arrived
    if kind == "fno":
        return dict(case=case, net=net, chi=chi, k0h=k0h, r=r)
    # training batches are picked from NumPy arrays
    return dict(case=case, net=net, chi=chi.cpu().numpy(), k0h=k0h, r=r.cpu().numpy(), x=x.cpu().numpy())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "matvec":
        return state["solver"].matvec(state["x"], precision=case["precision"], transpose=case["transpose"])
    if kind == "solve":
        x, _ = state["solver"].solve(state["b"], restart=case["restart"], max_iter=case["max_iter"], tol=case["tol"],
                                     precision=case["precision"], ortho=case["ortho"], transpose=case["transpose"])
        return x
    if kind == "batch":
        xs, _ = cg.solve_batch(state["systems"], restart=case["restart"], max_iter=case["max_iter"], tol=1e-10)
        return xs
    if kind == "gradient":
        return [state["prob"].value_and_gradient(x, state["targets"]) for x in state["xs"]]
    if kind == "fno":
        return state["net"].forward(state["chi"], state["k0h"], state["r"])
    return state["net"].loss_grad(state["chi"], state["k0h"], state["r"], state["x"])


# ------------------------------------------------------------------ work
def _matvec_work(N, e):
    """Two transforms of an embedding of side 2N, with the rows and columns that are zero or
    cropped left out; the vector, the contrast and the Green's block read, the result written."""
    L = 2 * N
    line = 5.0 * L * math.log2(L)
    return dict(bytes=3.5 * e * N * N, flops=6.0 * N * line + 6.0 * L * L)


def _solve_work(N, steps, restart, e):
    """One product per Arnoldi step, each new vector orthogonalised against its cycle's basis:
    the basis read once per step, 16 flops per entry; one residual product and update per cycle."""
    n, mv = float(N * N), _matvec_work(N, e)
    cycles = max(1, -(-steps // restart))
    m = min(steps, restart)
    basis = cycles * m * (m + 1) / 2.0
    return dict(bytes=(steps + cycles) * mv["bytes"] + basis * n * e,
                flops=(steps + cycles) * mv["flops"] + 16.0 * basis * n)


def _steps(case):
    """Arnoldi steps of a solve: its budget, or about what few wavelengths take to tolerance."""
    return 40 if case["max_iter"] == 500 else case["max_iter"]


def work(case):
    kind, N = case["kind"], case.get("N")
    if kind == "matvec":
        return _matvec_work(N, 16 if case["precision"] == "fp64" else 8)
    if kind == "solve":
        return _solve_work(N, _steps(case), case["restart"], 16 if case["precision"] == "fp64" else 8)
    if kind == "batch":
        sides = [int(v) for v in case["sides"].split(",")]
        each = [_solve_work(sides[i % len(sides)], case["max_iter"], case["restart"], 16) for i in range(case["nsys"])]
        return dict(bytes=sum(w["bytes"] for w in each), flops=sum(w["flops"] for w in each))
    if kind == "gradient":
        w = _solve_work(N, 60, 200, 16)
        return dict(bytes=4 * w["bytes"], flops=4 * w["flops"])
    cells = float(case["batch"] * N * N)
    modes = 2 * M1 * M2
    # lift, four layers (channel mixing, truncated column transforms both ways, mode mixing), projection
    fwd = cells * (2.0 * NIN * CH + LAYERS * (2.0 * CH * CH + 2 * 4.0 * CH * M2) + 2.0 * CH * HID + 4.0 * HID)
    fwd += LAYERS * case["batch"] * modes * (8.0 * CH * CH + 2 * 8.0 * CH * N)
    if kind == "fno":
        return dict(bytes=cells * (4 + 8 + 8), flops=fwd)
    params = LAYERS * (2.0 * modes * CH * CH + CH * CH + CH) + CH * (NIN + 1) + HID * (CH + 1) + 2 * (HID + 1)
    return dict(bytes=cells * (4 + 8 + 8) + 8 * params, flops=3.0 * fwd)


# ------------------------------------------------------------------ 64-bit answers in plain torch
def _hankel(order, z):
    """H0 or H1 of the first kind: Hankel's integral (DLMF 10.9.9 and 10.9.11 in the form
    sqrt(2 / (pi z)) e^{i(z - phase)} / Gamma * int_0^inf e^-t t^(order -+ 1/2) (1 + i t / 2z)^(order -+ 1/2) dt)
    with t = u^2 by the trapezoidal rule, which converges like exp(-2 pi sqrt(z) / step)."""
    step = min(0.25, 2.0 * math.pi * math.sqrt(float(z.min())) / 42.0)
    w = torch.complex(torch.zeros_like(z), 0.5 / z)
    acc = torch.full_like(w, 0.5 if order == 0 else 0.0)
    for i in range(1, int(6.4 / step) + 1):
        u2 = (i * step) ** 2
        f = torch.sqrt(1.0 + w * u2)
        acc += math.exp(-u2) * (f.reciprocal() if order == 0 else u2 * f)
    gamma = math.sqrt(math.pi) * (1.0 if order == 0 else 0.5)
    amp = torch.sqrt(2.0 / (math.pi * z)) * (2.0 * step / gamma)
    return torch.polar(amp, z - math.pi * (0.25 + 0.5 * order)) * acc


class _Operator:
    """A = I - G diag(c) by torch's FFT, complex128; G the GFIEM block of k0 and h."""

    def __init__(self, N, chi, k0, h):
        dev = _device()
        d = torch.arange(N, dtype=torch.float64, device=dev)
        z = k0 * h * torch.sqrt(d[:, None] ** 2 + d[None, :] ** 2)
        z[0, 0] = k0 * h
        g = _hankel(0, z) * (0.25j * h * h)
        a = h / math.sqrt(math.pi)
        h1 = complex(_hankel(1, torch.tensor([k0 * a], dtype=torch.float64)))
        g[0, 0] = complex(0.0, math.pi * a / (2.0 * k0)) * h1 - 1.0 / (k0 * k0)
        full = torch.zeros(2 * N, 2 * N, dtype=torch.complex128, device=dev)
        full[:N, :N] = g
        full[N + 1:, :N] = g[1:].flip(0)
        full[:, N + 1:] = full[:, 1:N].flip(1)
        self.N, self.spectrum, self.c = N, torch.fft.fft2(full), chi * (k0 * k0)

    def green(self, v):
        L = 2 * self.N
        w = torch.fft.fft(v, n=L, dim=1)
        w = torch.fft.ifft(torch.fft.fft(w, n=L, dim=0) * self.spectrum, dim=0)[:self.N]
        return torch.fft.ifft(w, dim=1)[:, :self.N]

    def apply(self, v, transpose=False):
        return v - (self.c * self.green(v) if transpose else self.green(self.c * v))


def _gmres(op, b, restart, max_iter, tol, transpose=False):
    """Restarted GMRES from zero: the iterate after max_iter steps, or, once the relative
    residual reaches tol, the solution (continued to 1e-13)."""
    N = op.N
    x = torch.zeros_like(b)
    nb = float(torch.linalg.norm(b))
    left, target = max_iter, tol
    for _ in range(1000):
        r = b - op.apply(x, transpose)
        beta = float(torch.linalg.norm(r))
        if beta <= target * nb and target > 1e-13:
            left, target = 10 * restart, 1e-13  # reached: go on to the solution
        if beta <= target * nb or left <= 0:
            break
        m = min(restart, left)
        V = torch.empty(m + 1, N * N, dtype=torch.complex128, device=b.device)
        V[0] = r.reshape(-1) / beta
        H = np.zeros((m + 1, m), np.complex128)
        R = np.zeros((m, m), np.complex128)
        cs, sn = np.zeros(m, np.complex128), np.zeros(m)
        g = np.zeros(m + 1, np.complex128)
        g[0], k = beta, 0
        for j in range(m):
            w = op.apply(V[j].view(N, N), transpose).reshape(-1)
            h = torch.zeros(j + 1, dtype=torch.complex128, device=b.device)
            for _ in range(2):
                d = torch.mv(V[:j + 1], w.conj()).conj()
                w = w - torch.mv(V[:j + 1].t(), d)
                h = h + d
            nrm = torch.linalg.norm(w)
            V[j + 1] = w / nrm
            H[:j + 1, j], H[j + 1, j] = h.cpu().numpy(), float(nrm)
            col = H[:j + 2, j].copy()
            for i in range(j):
                t = np.conj(cs[i]) * col[i] + sn[i] * col[i + 1]
                col[i + 1] = -sn[i] * col[i] + cs[i] * col[i + 1]
                col[i] = t
            rho = math.sqrt(abs(col[j]) ** 2 + abs(col[j + 1]) ** 2)
            cs[j], sn[j] = col[j] / rho, col[j + 1].real / rho
            R[:j, j], R[j, j] = col[:j], rho
            g[j + 1], g[j] = -sn[j] * g[j], np.conj(cs[j]) * g[j]
            k = j + 1
            if abs(g[k]) <= target * nb:
                break
        y = np.linalg.solve(R[:k, :k], g[:k])
        x = x + torch.mv(V[:k].t(), torch.from_numpy(y).to(b.device)).view(N, N)
        left -= k
        del V
    return x


def _gelu(v):
    return 0.5 * v * (1.0 + torch.erf(v / math.sqrt(2.0)))


def _net(params, chi, k0h, r):
    """(M(r), the network's outputs, 1 / rms) in float64 for a leaf vector of parameters."""
    at = 0

    def take(*shape):
        nonlocal at
        n = math.prod(shape)
        at += n
        return params[at - n:at].reshape(shape)

    B, H, W = r.shape
    s = r.abs().square().mean(dim=(1, 2)).sqrt()
    u = r / s[:, None, None]
    f = torch.stack([0.1 * chi, k0h[:, None, None].expand(B, H, W), u.real, u.imag], dim=-1)
    P, p = take(CH, NIN), take(CH)
    v = f @ P.t() + p
    rows = list(range(M1)) + list(range(H - M1, H))
    for layer in range(LAYERS):
        R = torch.view_as_complex(take(2 * M1, M2, CH, CH, 2).contiguous())
        Wl, bl = take(CH, CH), take(CH)
        modes = torch.fft.rfft2(v.permute(0, 3, 1, 2))[:, :, rows, :M2]
        full = torch.zeros(B, CH, H, W // 2 + 1, dtype=torch.complex128, device=v.device)
        full[:, :, rows, :M2] = torch.einsum("bcij,ijco->boij", modes, R)
        z = v @ Wl.t() + bl + torch.fft.irfft2(full, s=(H, W)).permute(0, 2, 3, 1)
        v = _gelu(z) if layer < LAYERS - 1 else z
    Q1, q1, Q2, q2 = take(HID, CH), take(HID), take(2, HID), take(2)
    o = _gelu(v @ Q1.t() + q1) @ Q2.t() + q2
    return r + s[:, None, None] * torch.view_as_complex(o.contiguous()), o, s


def exact(case, seed):
    kind, N = case["kind"], case.get("N")
    if kind == "matvec":
        p = _system(N, 4.0, 20.0, seed)
        x = _cnormal((N, N), seed, 5)
        if case["precision"] != "fp64":
            x = x.to(torch.complex64).to(torch.complex128)
        return _Operator(N, p["chi"], p["k0"], p["h"]).apply(x, case["transpose"])
    if kind == "solve":
        p = _system(N, case["eps"], case["lh"], seed)
        op = _Operator(N, p["chi"], p["k0"], p["h"])
        x = _gmres(op, p["b"], case["restart"], case["max_iter"], case["tol"], case["transpose"])
        return x.cpu().numpy() if case["host"] else x
    if kind == "batch":
        return [_gmres(_Operator(p["N"], p["chi"], p["k0"], p["h"]), p["b"], case["restart"], case["max_iter"],
                       1e-10).cpu().numpy() for p in _sweep(case, seed)]
    if kind == "gradient":
        p = _system(N, case["eps"], case["lh"], seed)
        _, xs, targets = _designs(case, seed)
        out = []
        for x in xs:
            op = _Operator(N, torch.from_numpy(x).to(_device()) * (case["eps"] - 1.0), p["k0"], p["h"])
            E = _gmres(op, p["b"], 200, 20000, 1e-11)
            q = torch.zeros_like(E)
            for i, j in targets:
                q[i, j] = E[i, j].conj()
            w = op.green(_gmres(op, q, 200, 20000, 1e-11, transpose=True))
            F = sum(float(E[i, j].abs() ** 2) for i, j in targets)
            out.append((F, (2.0 * p["k0"] ** 2 * (w * E).real).cpu().numpy(), E.cpu().numpy()))
        return out
    params, chi, k0h, r, x = _net_inputs(case, seed)
    leaf = torch.from_numpy(params).double().to(_device()).requires_grad_(kind == "fno_grad")
    r = r.to(torch.complex128)
    z, o, s = _net(leaf, chi.double(), torch.from_numpy(k0h).double().to(_device()), r)
    if kind == "fno":
        return z.detach().cpu().numpy()
    t = torch.view_as_real(((x.to(torch.complex128) - r) / s[:, None, None]).contiguous())
    loss = ((o - t).square().sum(dim=(1, 2, 3)) / t.square().sum(dim=(1, 2, 3))).mean()
    loss.backward()
    return float(loss.detach()), leaf.grad.cpu().numpy()
