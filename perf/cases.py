"""Performance cases of the solver library: what a user's program has it do.

Each case goes through the package's public Python entry points
(``isg.Solver``, ``isg.multi.MultiSolver``) on seeded inputs of the kind the
path meets: random lossy ellipses as contrast, plane waves or line sources as
incidence.  ``exact`` gives the same results in 64 bits from the dense
discretised operator, applied by FFT convolution in plain torch.

Sides are 8 times a power of two (the tree's leaves are 8 x 8 pixels); batches
are any number of right-hand sides.
"""
from __future__ import annotations

import math
import os
import sys

import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "inverse-solver-gpu_b200"))

import isg  # noqa: E402
from isg.multi import MultiSolver  # noqa: E402

K0, RES = 2 * math.pi, 0.1  # background wavenumber (wavelength 1) and pixel size
ENGINES = {"plain": isg.ENGINE_SIMT, "tensor": isg.ENGINE_TENSOR}
ORDERS = {"tree": isg.ORDER_TREE, "raster": isg.ORDER_RASTER, "blocked": isg.ORDER_BLOCKED}
DEV = "cuda"


# ---- the cases ----

def operator(side, nrhs, engine, order, adjoint=False, own_contrast=False):
    """y = x - G(g x) or its adjoint: one application of the operator."""
    return {"do": "operator", "side": side, "nrhs": nrhs, "engine": engine, "order": order, "adjoint": adjoint,
            "own_contrast": own_contrast}


def solve(side, nrhs, engine, order, eps, adjoint=False, line=False, stream=True, check=4):
    """BiCGSTAB to 1e-5 for every right-hand side."""
    return {"do": "solve", "side": side, "nrhs": nrhs, "engine": engine, "order": order, "eps": eps,
            "adjoint": adjoint, "line": line, "stream": stream, "check": check}


def mixed(problems, max_rhs):
    """Independent problems of several grid sizes, "<side>x<transmitters>" each."""
    return {"do": "mixed", "problems": problems, "max_rhs": max_rhs, "eps": 1.8}


def receivers(side, nrhs, numrx, near):
    """Receiver samples of fields and the back-projection of samples."""
    return {"do": "receivers", "side": side, "nrhs": nrhs, "numrx": numrx, "near": near}


def invert(side, ntx, numrx, near, iterations):
    """The distorted-Born inversion loop."""
    return {"do": "invert", "side": side, "ntx": ntx, "numrx": numrx, "near": near, "iterations": iterations}


def network(side, nrhs, batch, train):
    """The warm-start network: its output, or the loss and gradient of a training step."""
    return {"do": "network", "side": side, "nrhs": nrhs, "batch": batch, "train": train}


def listed():
    return [
        # one application on the smallest grid that a program sets up in earnest: call latency
        dict(operator(64, 1, "plain", "tree"), name="apply 64 x1 plain"),
        # the adjoint of an ordinary batch, every right-hand side with its own contrast, image order
        dict(operator(256, 9, "tensor", "raster", adjoint=True, own_contrast=True), name="adjoint 256 x9"),
        # the operator alone at the headline's grid
        dict(operator(1024, 16, "tensor", "tree"), name="apply 1024 x16"),
        # the largest grid, in the library's own order
        dict(operator(4096, 2, "tensor", "blocked"), name="apply 4096 x2"),
        # the call with every default: one transmitter, the plain engine, the current stream
        dict(solve(128, 1, "plain", "tree", 1.5, stream=False, check=1), name="solve 128 x1 plain"),
        # the small problem of the reference: 32 line sources at once
        dict(solve(128, 32, "tensor", "tree", 1.5, line=True), name="solve 128 x32"),
        # the adjoint solves of an inversion, an odd number of transmitters
        dict(solve(512, 33, "tensor", "tree", 1.5, adjoint=True), name="adjoint solve 512 x33"),
        # the headline problem (lossy, eps_r up to 2), a quarter of its transmitters
        dict(solve(1024, 64, "tensor", "tree", 2.0), name="solve 1024 x64"),
        # many independent problems of uneven size
        dict(mixed("128x16,128x37,256x21,256x16,512x19", 64), name="mixed sizes"),
        # near-field receivers: the dense receiver operator and its adjoint
        dict(receivers(512, 64, 256, near=True), name="receivers near 512 x64"),
        # the inversion loop with far-field receivers
        dict(invert(256, 16, 64, near=False, iterations=2), name="invert 256 x16"),
        # a training step of the warm-start network
        dict(network(256, 8, 4, train=True), name="train 256 x8"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["operator"] * 4 + ["solve"] * 4 + ["mixed", "receivers", "receivers", "invert", "network"])
    order = rng.choice(sorted(ORDERS))
    if kind == "operator":
        side = 2 ** rng.randint(5, 12)
        engine = rng.choice(["plain", "tensor", "tensor"])
        most = (2 ** 25 if engine == "tensor" else 2 ** 22) // side ** 2
        nrhs = _log_int(rng, 1, min(256, max(1, most)))
        own = bool(rng.randint(0, 1)) and nrhs > 1
        return operator(side, nrhs, engine, order, bool(rng.randint(0, 1)), own)
    if kind == "solve":
        engine = rng.choice(["plain", "tensor", "tensor"])
        side = 2 ** rng.randint(5, 10 if engine == "tensor" else 9)
        most = (2 ** 25 if engine == "tensor" else 2 ** 21) // side ** 2
        nrhs = _log_int(rng, 1, min(256, most))
        return solve(side, nrhs, engine, order, rng.choice([1.5, 2.0]), bool(rng.randint(0, 1)),
                     bool(rng.randint(0, 1)), bool(rng.randint(0, 1)), rng.choice([1, 2, 4]))
    if kind == "mixed":
        parts = ["%dx%d" % (2 ** rng.randint(6, 9), rng.randint(3, 40)) for _ in range(rng.randint(2, 6))]
        return mixed(",".join(parts), rng.choice([32, 64, 100]))
    if kind == "receivers":
        near = bool(rng.randint(0, 1))
        side = 2 ** rng.randint(6, 9 if near else 10)
        nrhs = _log_int(rng, 1, min(160, 2 ** 24 // side ** 2))
        return receivers(side, nrhs, rng.randint(16, 256), near)
    if kind == "invert":
        side = 2 ** rng.randint(6, 8)
        return invert(side, rng.randint(4, 16), rng.randint(16, 64), bool(rng.randint(0, 1)), rng.randint(1, 2))
    return network(2 ** rng.randint(6, 8), rng.randint(1, 12), rng.randint(1, 6), bool(rng.randint(0, 1)))


# ---- inputs, in raster order (row 0 at the top) until the last step ----

def _gen(seed):
    g = torch.Generator(device="cpu")
    g.manual_seed(1_000_003 * seed + 17)
    return g


def _rand(gen, lo, hi, n=1):
    v = torch.rand(n, generator=gen, dtype=torch.float64) * (hi - lo) + lo
    return v.tolist() if n > 1 else v.item()


def _cgauss(gen, *shape):
    """Complex normal numbers, made on the GPU from one number of `gen`."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(torch.randint(0, 2 ** 62, (1,), generator=gen).item()))
    return torch.complex(torch.randn(*shape, generator=g, device=DEV), torch.randn(*shape, generator=g, device=DEV))


def _axes(side):
    c = (torch.arange(side, device=DEV, dtype=torch.float64) + 0.5) * RES - side * RES / 2
    return c, -c  # x of the columns, y of the rows


def _ellipses(gen, side, eps_max):
    """Contrast eps_r - 1 of random ellipses, semi-axes 1 to 3 wavelengths; lossy above eps_r 1.5."""
    x, y = _axes(side)
    d = side * RES
    chi = torch.zeros(side, side, dtype=torch.complex128, device=DEV)
    for _ in range(max(3, side // 50)):
        a, b = (min(v, d / 3) for v in _rand(gen, 1.0, 3.0, 2))
        m = max(a, b)
        cx, cy = (m - d / 2 + (d - 2 * m) * v for v in _rand(gen, 0.0, 1.0, 2))
        th, eps = _rand(gen, 0.0, math.pi), _rand(gen, 1.1, eps_max)
        tan = _rand(gen, 0.0, 0.1) if eps_max > 1.5 else 0.0
        px, py = x[None, :] - cx, y[:, None] - cy
        u = (math.cos(th) * px + math.sin(th) * py) / a
        v = (-math.sin(th) * px + math.cos(th) * py) / b
        chi[u * u + v * v <= 1.0] = complex(eps - 1.0, eps * tan)
    return chi.reshape(-1)


def _incident(gen, side, n, line):
    """n fields: plane waves, or line sources on a circle outside the domain, from equally spaced angles."""
    x, y = _axes(side)
    first, out = _rand(gen, 0.0, 2 * math.pi), torch.empty(n, side * side, dtype=torch.complex64, device=DEV)
    radius = 1.5 * side * RES
    for j in range(n):
        a = first + 2 * math.pi * j / n
        if line:
            f = _hankel(torch.hypot(x[None, :] - radius * math.cos(a), y[:, None] - radius * math.sin(a)))
        else:
            f = torch.exp(1j * K0 * (math.cos(a) * x[None, :] + math.sin(a) * y[:, None]))
        out[j] = f.reshape(-1)
    return out


def _place(side, order):
    """For every raster pixel its index in `order`."""
    r = torch.arange(side * side, device=DEV)
    row, col = r // side, r % side
    if order == "raster":
        return r
    ly, lx, leaf = row // 8, col // 8, torch.zeros_like(r)
    if order == "blocked":
        leaf = ly * (side // 8) + lx
    else:  # the tree's quadrants are numbered 2 * row + column at every level
        for bit in range((side // 8).bit_length() - 1):
            leaf |= ((lx >> bit) & 1) << (2 * bit) | ((ly >> bit) & 1) << (2 * bit + 1)
    return leaf * 64 + (row % 8) * 8 + col % 8


def _to(v, side, order):
    if order == "raster":
        return v
    out = torch.empty_like(v)
    out[..., _place(side, order)] = v
    return out


def _from(v, side, order):
    return v if order == "raster" else v[..., _place(side, order)]


def _inputs(case, seed):
    """The inputs of a case as complex64 (contrasts as complex128), in raster order."""
    gen, do = _gen(seed), case["do"]
    if do == "operator":
        n, side = case["nrhs"], case["side"]
        g = [K0 ** 2 * _ellipses(gen, side, 2.0) for _ in range(min(n, 4) if case["own_contrast"] else 1)]
        g = torch.stack([g[j % len(g)] * (1 - 0.01 * (j // len(g))) for j in range(n)]) if case["own_contrast"] else g[0]
        return {"g": g.to(torch.complex64), "x": _cgauss(gen, n, side * side)}
    if do == "solve":
        return {"g": (K0 ** 2 * _ellipses(gen, case["side"], case["eps"])).to(torch.complex64),
                "b": _incident(gen, case["side"], case["nrhs"], case["line"])}
    if do == "mixed":
        return {"problems": [((K0 ** 2 * _ellipses(gen, side, case["eps"])).to(torch.complex64),
                              _incident(gen, side, n, False)) for side, n in _sizes(case)]}
    if do == "receivers":
        return {"x": _cgauss(gen, case["nrhs"], case["side"] ** 2), "r": _cgauss(gen, case["nrhs"], case["numrx"])}
    if do == "invert":
        side = case["side"]
        chi, inc = 0.5 * _ellipses(gen, side, 1.5), _incident(gen, side, case["ntx"], case["near"])
        g, b = K0 ** 2 * chi, inc.to(torch.complex128)
        u = _solve64(_Dense(side), g, b, 1e-6, False)
        mes = _receive64(g * u, side, case["numrx"], _radius(case)).to(torch.complex64)
        return {"inc": inc, "mes": mes}
    side, n = case["side"], case["nrhs"]
    g = torch.stack([K0 ** 2 * _ellipses(gen, side, 1.5) for _ in range(n)]).to(torch.complex64)
    b = _incident(gen, side, n, True)
    b = b / b.abs().mean()
    u = _solve64(_Dense(side), g.to(torch.complex128), b.to(torch.complex128), 1e-5, False).to(torch.complex64)
    return {"g": g, "b": b, "u": u, "p": _parameters(gen)}


def _sizes(case):
    return [tuple(int(v) for v in p.split("x")) for p in case["problems"].split(",")]


def _level(side):
    return (side // 8).bit_length()


def _radius(case):
    return case["side"] * RES if case["near"] else 0.0


# ---- what a program has in hand, and one pass ----

def prepare(case, seed):
    """The inputs on the GPU and the set-up solver that a program keeps across its calls."""
    do, v = case["do"], _inputs(case, seed)
    order = case.get("order", "tree")
    state = {"case": case, "stream": torch.cuda.Stream()}
    if do == "mixed":
        state["ms"] = MultiSolver(max_rhs=case["max_rhs"])
        state["problems"] = [(_to(g, s, order), _to(b, s, order)) for (g, b), (s, _) in zip(v["problems"], _sizes(case))]
        for side, _ in _sizes(case):
            state["ms"].solver(_level(side))
        torch.cuda.synchronize()
        return state
    side = case["side"]
    for k in ("g", "x", "b", "inc", "u"):
        if k in v:
            state[k] = _to(v[k], side, order)
    for k in ("r", "mes", "p"):
        if k in v:
            state[k] = v[k]
    state["solver"] = isg.Solver(_level(side), numrx=case.get("numrx", 32),
                                 max_rhs=case.get("ntx", case.get("nrhs")))
    state["solver"].setup_gpu()
    if case.get("near"):
        state["solver"].set_nearfield_receivers(_radius(case))
    if do == "solve":
        state["x"] = torch.zeros_like(state["b"])
    if do == "network":
        state["solver"].fno_create(batch=case["batch"])
        state["solver"].fno_set_params(state["p"].numpy())
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    do = case["do"]
    if do == "mixed":
        return [x for x, _ in state["ms"].solve(state["problems"], tol=1e-5)]
    s, order = state["solver"], ORDERS[case.get("order", "tree")]
    if do == "operator":
        return s.matvec(state["x"], state["g"], hermitian=case["adjoint"], order=order, engine=ENGINES[case["engine"]])
    if do == "solve":
        s.bicgs(state["x"], state["g"], state["b"], hermitian=case["adjoint"], order=order, tol=1e-5, maxit=1000,
                engine=ENGINES[case["engine"]], check_every=case["check"],
                stream=state["stream"] if case["stream"] else None)
        return state["x"]
    if do == "receivers":
        if case["near"]:
            return s.receive(state["x"]), s.receiveh(state["r"])
        return s.aggregate(state["x"]), s.aggregateh(state["r"])
    if do == "invert":
        return s.dbim(state["inc"], state["mes"], iterations=case["iterations"], tol=1e-5, maxit=1000,
                      engine=isg.ENGINE_TENSOR, check_every=2, stream=state["stream"])[0]
    if case["train"]:
        loss = s.fno_grad(state["g"], state["b"], state["u"])
        return {"loss": loss, "grad": s.fno_params(1)}
    return s.fno_apply(state["g"], state["b"])


def _iterations(side, eps):
    """BiCGSTAB iterations to 1e-5, about: 15 at 128 pixels and eps_r 1.5, 116 at 1024 and 2."""
    return 15 * math.sqrt(side / 128) * (2 * (eps - 1)) ** 1.46


def work(case):
    """An application reads its vector and contrast, writes its result and takes 6.9 kflop per
    pixel (near field, tree and leaves); a BiCGSTAB iteration is two of them and reads or writes
    its vectors 16 times besides; receivers take one complex product per pixel and receiver, or
    the leaves of the tree; the network's layers read and write their channels."""
    do, px = case["do"], 8.0
    if do == "mixed":
        parts = [work(solve(s, n, "tensor", "tree", case["eps"])) for s, n in _sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    U = float(case["side"] ** 2)
    if do == "operator":
        n = case["nrhs"]
        return {"bytes": px * U * (2 * n + (n if case["own_contrast"] else 1)), "flops": 6900 * U * n}
    if do in ("solve", "invert"):
        n, solves, eps = (case["nrhs"], 1, case["eps"]) if do == "solve" else (case["ntx"], 1 + 3 * case["iterations"], 1.25)
        its = _iterations(case["side"], eps) * solves
        return {"bytes": px * U * n * its * (2 * 2 + 16), "flops": 2 * 6900 * U * n * its}
    if do == "receivers":
        n = case["nrhs"]
        # two directions; the dense operator (8 bytes an entry) is larger than the vectors
        per_px = 8.0 * case["numrx"] if case["near"] else 8.0 * 68
        return {"bytes": 2 * px * U * (n + (case["numrx"] if case["near"] else 0)), "flops": 2 * per_px * U * n}
    n, c, layers = case["nrhs"], 32, 4
    dirs = 3 if case["train"] else 1
    return {"bytes": dirs * layers * 3 * 4.0 * c * U * n, "flops": dirs * layers * 2.0 * c * (c + 2 * 24) * U * n}


# ---- the same results in 64 bits ----

def _hankel(d):
    return torch.special.bessel_j0(K0 * d) + 1j * torch.special.bessel_y0(K0 * d)


def _green(d):
    """(i/4) H0(k0 d) over a pixel's area, the pixel taken as a point."""
    return 0.25j * RES ** 2 * _hankel(d)


class _Dense:
    """G on side x side pixels: the convolution with the sampled Green's function, whose own-pixel
    entry integrates the logarithm over the square."""

    def __init__(self, side):
        self.side = side
        i = torch.arange(2 * side, device=DEV)
        i = torch.minimum(i, 2 * side - i).to(torch.float64) * RES
        k = torch.empty(2 * side, 2 * side, dtype=torch.complex128, device=DEV)
        for r0 in range(0, 2 * side, 512):
            k[r0:r0 + 512] = _green(torch.hypot(i[r0:r0 + 512, None], i[None, :]).clamp_min(RES / 2))
        log_area = RES ** 2 * (math.log(RES ** 2 / 2) - 3 + math.pi / 2)  # of log(x^2 + y^2)
        y0 = 2 / math.pi * (RES ** 2 * (0.5772156649015329 + math.log(K0 / 2)) + log_area / 2)
        k[0, 0] = 0.25j * complex(RES ** 2, y0)
        self.hat = torch.fft.fft2(k)

    def __call__(self, x):
        n, out = self.side, torch.empty_like(x)
        step = max(1, 2 ** 24 // n ** 2)
        for j in range(0, x.shape[0], step):
            v = torch.fft.fft2(x[j:j + step].reshape(-1, n, n), s=(2 * n, 2 * n))
            v = torch.fft.ifft2(v.mul_(self.hat))[:, :n, :n]
            out[j:j + step] = v.reshape(-1, n * n)
        return out


def _apply64(G, x, g, adjoint):
    return x - (g * G(x.conj())).conj() if adjoint else x - G(g * x)


def _solve64(G, g, b, tol, adjoint, most=1500):
    """BiCGSTAB in complex128, all right-hand sides at once."""
    dot = lambda a, c: (a.conj() * c).sum(1, keepdim=True)  # noqa: E731
    x, r = torch.zeros_like(b), b.clone()
    rt, p, bn = r.clone(), r.clone(), torch.linalg.vector_norm(b, dim=1, keepdim=True)
    rho, done = dot(rt, r), torch.zeros(b.shape[0], 1, dtype=torch.bool, device=DEV)
    bn = torch.where(bn > 0, bn, torch.ones_like(bn))
    div = lambda a, c: torch.where(done, torch.zeros_like(a), a / torch.where(c == 0, torch.ones_like(c), c))  # noqa: E731
    for it in range(most):
        v = _apply64(G, p, g, adjoint)
        alpha = div(rho, dot(rt, v))
        s = r - alpha * v
        t = _apply64(G, s, g, adjoint)
        omega = div(dot(t, s), dot(t, t))
        x += alpha * p + omega * s
        r = torch.where(done, r, s - omega * t)
        done = torch.linalg.vector_norm(r, dim=1, keepdim=True) < tol * bn
        if it % 4 == 3 and bool(done.all()):
            break
        new = dot(rt, r)
        p = r + div(new, rho) * div(alpha, omega) * (p - omega * v)
        rho = new
    return x


def _directions(numrx):
    a = 2 * math.pi * torch.arange(numrx, device=DEV, dtype=torch.float64) / numrx
    return torch.cos(a), torch.sin(a)


def _rows(side, numrx, radius):
    """The receivers' operator, a slab of pixel rows at a time: (slice, (numrx, pixels))."""
    x, y = _axes(side)
    cx, cy = _directions(numrx)
    step = max(1, 2 ** 24 // (numrx * side))
    for r0 in range(0, side, step):
        yy = y[r0:r0 + step]
        if radius:
            k = _green(torch.hypot(x[None, None, :] - radius * cx[:, None, None],
                                   yy[None, :, None] - radius * cy[:, None, None]))
        else:
            ph = cx[:, None, None] * x[None, None, :] + cy[:, None, None] * yy[None, :, None]
            k = RES ** 2 * torch.exp(-1j * K0 * ph)
        yield slice(r0 * side, (r0 + len(yy)) * side), k.reshape(numrx, -1)


def _receive64(x, side, numrx, radius):
    out = torch.zeros(x.shape[0], numrx, dtype=torch.complex128, device=DEV)
    for at, k in _rows(side, numrx, radius):
        out += x[:, at] @ k.T
    return out


def _receiveh64(r, side, numrx, radius):
    out = torch.empty(r.shape[0], side * side, dtype=torch.complex128, device=DEV)
    for at, k in _rows(side, numrx, radius):
        out[:, at] = r @ k.conj()
    return out


def _invert64(case, inc, mes):
    """Polak-Ribiere iterations from the empty domain with the Born-linearised step."""
    side, radius, nrx = case["side"], _radius(case), case["numrx"]
    G, k2 = _Dense(side), K0 ** 2
    rec = lambda x: _receive64(x, side, nrx, radius)  # noqa: E731
    chi = torch.zeros(side * side, dtype=torch.complex128, device=DEV)
    tot, mis = inc.clone(), -mes

    def gradient():
        g, y = k2 * chi, _receiveh64(mis, side, nrx, radius)
        x = _solve64(G, g, g.conj() * y, 1e-10, True)
        return (tot.conj() * (y + G(x.conj()).conj())).sum(0)

    od = gradient()
    ot = od.clone()
    for _ in range(case["iterations"]):
        y = tot * (k2 * ot)
        x = _solve64(G, k2 * chi, G(y), 1e-10, False)
        d = rec(y + k2 * chi * x)
        chi -= ((mis.conj() * d).sum().real / d.abs().square().sum()) * ot
        tot = _solve64(G, k2 * chi, inc, 1e-10, False)
        mis, old = rec(k2 * chi * tot) - mes, od
        od = gradient()
        ot = od + (od * (od - old).conj()).sum() / old.abs().square().sum() * ot
    return chi


WIDTH, MODES, LAYERS = 32, 12, 4  # the network's defaults


def _layout():
    """Name, shape and offset of each block of the flat parameters (blocks begin at multiples of 4)."""
    shapes = [("Wl", (WIDTH, 10)), ("bl", (WIDTH,))]
    for l in range(LAYERS):
        shapes += [("R%d" % l, (2 * MODES * MODES, WIDTH, WIDTH, 2)), ("W%d" % l, (WIDTH, WIDTH)), ("b%d" % l, (WIDTH,))]
    shapes += [("Wp", (2, WIDTH)), ("Ws", (2, 10)), ("bp", (2,))]
    at = 0
    for name, shape in shapes:
        n = math.prod(shape)
        yield name, shape, at, n
        at += (n + 3) // 4 * 4
    yield "", (), at, 0


def _parameters(gen):
    """Parameters of the scale that training starts from (on the host, as a program loads them)."""
    p = torch.zeros(list(_layout())[-1][2], dtype=torch.float32)
    limits = {"Wl": 10 ** -0.5, "W": WIDTH ** -0.5, "Wp": 0.1 * WIDTH ** -0.5, "Ws": 0.1 * 10 ** -0.5}
    for name, _, at, n in _layout():
        if name.startswith("R"):
            p[at:at + n] = torch.rand(n, generator=gen) / WIDTH ** 2
        elif name:
            p[at:at + n] = (2 * torch.rand(n, generator=gen) - 1) * limits.get(name, limits["W"] if name[0] == "W" else 0.01)
    return p


def _network64(p, g, b, s1, side):
    """x0 = b + N(g, b) of every sample."""
    d = {name: p[at:at + n].reshape(shape) for name, shape, at, n in _layout() if name}
    chi = g / K0 ** 2
    feats = torch.stack([f for z in (chi, b, chi * b, s1, chi * s1) for f in (z.real, z.imag)], 1)
    inp = feats.reshape(-1, 10, side, side)
    mix = lambda w, v: torch.einsum("oc,scyx->soyx", w, v)  # noqa: E731
    rows = list(range(MODES)) + list(range(side - MODES, side))
    weight = torch.full((MODES,), 2.0, dtype=torch.float64, device=DEV)
    weight[0] = 1.0
    v = mix(d["Wl"], inp) + d["bl"][:, None, None]
    for l in range(LAYERS):
        R = torch.view_as_complex(d["R%d" % l]).reshape(2 * MODES, MODES, WIDTH, WIDTH)
        X = torch.fft.fft2(v)[:, :, rows, :MODES]
        Y = torch.einsum("rkoc,scrk->sork", R, X) * weight
        full = torch.zeros(v.shape, dtype=torch.complex128, device=DEV)
        full[:, :, rows, :MODES] = Y
        h = mix(d["W%d" % l], v) + d["b%d" % l][:, None, None] + torch.fft.ifft2(full).real
        v = torch.nn.functional.gelu(h) if l + 1 < LAYERS else h
    out = (mix(d["Wp"], v) + mix(d["Ws"], inp) + d["bp"][:, None, None]).reshape(-1, 2, side * side)
    return b + torch.complex(out[:, 0], out[:, 1])


def exact(case, seed):
    do, v, c128 = case["do"], _inputs(case, seed), torch.complex128
    if do == "mixed":
        return [_to(_solve64(_Dense(s), g.to(c128), b.to(c128), 1e-10, False), s, "tree")
                for (g, b), (s, _) in zip(v["problems"], _sizes(case))]
    side, order = case["side"], case.get("order", "tree")
    if do == "operator":
        return _to(_apply64(_Dense(side), v["x"].to(c128), v["g"].to(c128), case["adjoint"]), side, order)
    if do == "solve":
        if case["nrhs"] * side ** 2 * _iterations(side, case["eps"]) > 2 ** 33.2:
            return None
        return _to(_solve64(_Dense(side), v["g"].to(c128), v["b"].to(c128), 1e-9, case["adjoint"]), side, order)
    if do == "receivers":
        r = (side, case["numrx"], _radius(case))
        return _receive64(v["x"].to(c128), *r), _to(_receiveh64(v["r"].to(c128), *r), side, order)
    if do == "invert":
        return _to(_invert64(case, v["inc"].to(c128), v["mes"].to(c128)), side, order)
    g, b, u = (v[k].to(c128) for k in ("g", "b", "u"))
    p = v["p"].to(DEV).to(torch.float64).requires_grad_(case["train"])
    s1 = _Dense(side)(g * b)
    if not case["train"]:
        return _to(_network64(p, g, b, s1, side), side, order)
    e = _network64(p, g, b, s1, side) - u
    loss = (e.abs().square().sum(1) / u.abs().square().sum(1)).mean()
    loss.backward()
    return {"loss": loss.item(), "grad": p.grad.cpu().numpy()}
