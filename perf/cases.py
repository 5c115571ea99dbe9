"""What users of the engine have it do, as timed cases.

Every case works on a population that is near the solution of its pattern
(the state of a reconstruction after its first generations): there the
iterations are well conditioned, so that a pass can be compared with 64-bit
arithmetic.  The patterns have the geometry of the benchmark's workloads: an
object about 0.23 of the side across with densities in [0.3, 1] and a phase
noise of 0.2 rad, Poisson noise, a masked beamstop with upper amplitude
bounds on its rim, and two detector gaps.  (A bright exposure and a few
iterations a call: with the noise of a faint one HIO and RAAR amplify a
rounding difference tenfold every few iterations.)

Operations (`op`):
  iterate    HIO / RAAR / ER through the engine handle, population resident
  sequence   one op list with shrink-wrap through the drop-in Solver, on one
             individual, density and support read back at the end
  evaluate   error metrics of every individual
  shrinkwrap support update by blurred threshold (SW) or area (SWA)
  crossover  one child per individual: alignment of the parents, mixing,
             gating
  lossgrad   far-field loss and its gradient through torch autograd
  refine     fused Adam steps on the far-field loss
"""
import math

import numpy as np
import torch

from s_spi_spring_gb300 import _lib
from s_spi_spring_gb300.refine import farfield_loss, population_tensors, refine
from s_spi_spring_gb300.spring_core.phase_retrieval import Reconstruction, Solver

DEV = "cuda"
PHOTONS = 1e11
SPREAD = 0.05  # of the starting individuals about the object
METRICS = ("error", "error_fourier", "error_real", "reality", "modulesum", "complexsum", "symmetry")
COMPILED = (16, 32, 64, 128, 256, 384, 512, 768, 1024, 2048)


def listed():
    return [
        # one reconstruction of a small pattern, start to end through the front
        # end: many short launches, where latency counts
        {"name": "sequence_128_p1", "op": "sequence", "n": 128, "p": 1, "iters": 20, "er": 10, "beta": 0.9,
         "sigma": 2.0, "threshold": 0.1},
        # a few individuals polished by error reduction
        {"name": "er_512_p4", "op": "iterate", "alg": "er", "n": 512, "p": 4, "iters": 20, "beta": 0.0},
        # the front end's default population on its example pattern's side
        {"name": "raar_256_p128", "op": "iterate", "alg": "raar", "n": 256, "p": 128, "iters": 20, "beta": 0.87},
        # the headline workload: one RAAR step of a 512^2 population
        {"name": "raar_512_p64", "op": "iterate", "alg": "raar", "n": 512, "p": 64, "iters": 10, "beta": 0.87},
        # the HIO part of the gradient-refinement workload's epochs
        {"name": "hio_1024_p32", "op": "iterate", "alg": "hio", "n": 1024, "p": 32, "iters": 8, "beta": 0.9},
        # the large population (17 GB on the device)
        {"name": "raar_2048_p128", "op": "iterate", "alg": "raar", "n": 2048, "p": 128, "iters": 8, "beta": 0.87},
        # the reference's example patterns, 1054 x 1024 cropped to a square: a
        # side without a compiled plan (2 x 17 x 31)
        {"name": "raar_1054_p16", "op": "iterate", "alg": "raar", "n": 1054, "p": 16, "iters": 8, "beta": 0.87},
        # a generation's evaluation, support update and crossover
        {"name": "evaluate_512_p64", "op": "evaluate", "n": 512, "p": 64},
        {"name": "shrinkwrap_512_p64", "op": "shrinkwrap", "n": 512, "p": 64, "area": False, "sigma": 3.0,
         "threshold": 0.1},
        {"name": "crossover_512_p64", "op": "crossover", "n": 512, "p": 64, "crossft": 1.0, "average": 0.0},
        # gradient refinement: an autograd step of a user's own optimiser, and
        # the fused optimiser
        {"name": "lossgrad_1024_p32", "op": "lossgrad", "n": 1024, "p": 32, "loss": "poisson"},
        {"name": "refine_512_p64", "op": "refine", "n": 512, "p": 64, "loss": "poisson", "steps": 10},
    ]


def _largest_prime(n):
    f, big = 2, 1
    while n > 1:
        if n % f == 0:
            big, n = f, n // f
        else:
            f += 1
    return big


def draw(rng):
    """A case of the same operations: compiled sides and any other side (odd
    and prime ones among them), populations from one individual up."""
    op = rng.choice(["iterate"] * 6 + ["sequence", "evaluate", "shrinkwrap", "crossover", "lossgrad", "refine"])
    if rng.random() < 0.65:
        n = rng.choice(COMPILED[2:] if op != "sequence" else COMPILED[2:6])
        pixels = 2.0 ** 27 if op == "iterate" else 2.0 ** 25
    else:
        n = int(round(math.exp(rng.uniform(math.log(50), math.log(1200)))))
        while n in COMPILED or _largest_prime(n) > 300:
            n += 1
        pixels = 2.0 ** 24 if op == "iterate" else 2.0 ** 23
    lo = 4 if op == "crossover" else 1
    top = max(lo, min(1024, int(pixels / (n * n))))
    p = int(round(math.exp(rng.uniform(math.log(lo), math.log(top)))))
    if op == "iterate":
        alg = rng.choice(["hio", "raar", "er"])
        return {"op": op, "alg": alg, "n": n, "p": p, "iters": rng.randint(4, 20) if alg == "er" else rng.randint(4, 10),
                "beta": 0.0 if alg == "er" else round(rng.uniform(0.8, 0.95), 3)}
    if op == "sequence":
        return {"op": op, "n": n, "p": 1, "iters": rng.randint(10, 30), "er": rng.randint(5, 15),
                "beta": round(rng.uniform(0.8, 0.95), 3), "sigma": 2.0, "threshold": 0.1}
    if op == "shrinkwrap":
        return {"op": op, "n": n, "p": p, "area": rng.random() < 0.5, "sigma": round(rng.uniform(1.5, 3.0), 2),
                "threshold": round(rng.uniform(0.05, 0.15), 3)}
    if op == "crossover":
        return {"op": op, "n": n, "p": p, "crossft": rng.choice([0.0, 0.5, 1.0]),
                "average": rng.choice([0.0, 0.5, -0.5])}
    if op == "lossgrad":
        return {"op": op, "n": n, "p": p, "loss": rng.choice(["poisson", "amplitude"])}
    if op == "refine":
        return {"op": op, "n": n, "p": p, "loss": rng.choice(["poisson", "amplitude"]), "steps": rng.randint(5, 10)}
    return {"op": op, "n": n, "p": p}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _ellipse(n, a, b, t):
    r = torch.arange(n, device=DEV, dtype=torch.float64) - n // 2
    y, x = r[:, None], r[None, :]
    u, v = x * math.cos(t) + y * math.sin(t), -x * math.sin(t) + y * math.cos(t)
    return (u / a) ** 2 + (v / b) ** 2 <= 1.0


def _inputs(case, seed):
    """Amplitudes (DC at [0, 0]; negative: unknown, at most -2: upper bound
    -A - 2), starting densities and supports of the case's population."""
    n, p = case["n"], case["p"]
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    r = torch.rand(3, generator=g, device=DEV, dtype=torch.float64).tolist()
    a = max(3.0, 0.115 * n * (0.85 + 0.15 * r[0]))
    b = max(3.0, 0.115 * n * (0.65 + 0.15 * r[1]))
    inside = _ellipse(n, a, b, math.pi * r[2])
    dens = 0.3 + 0.7 * torch.rand(n, n, generator=g, device=DEV, dtype=torch.float64)
    phase = 0.2 * torch.randn(n, n, generator=g, device=DEV, dtype=torch.float64)
    obj = torch.where(inside, torch.polar(dens, phase), 0)
    intensity = torch.fft.ifft2(obj).mul_(n * n).abs().square_()
    scale = PHOTONS / float(intensity.sum())
    counts = torch.poisson(intensity * scale, generator=g)
    amp = counts.sqrt().to(torch.float32)
    k = torch.fft.fftfreq(n, device=DEV, dtype=torch.float64) * n
    radius = torch.sqrt(k[:, None] ** 2 + k[None, :] ** 2)
    if case["op"] != "sequence":  # (the Solver encodes the mask itself there)
        rim = (radius > max(1.0, n / 64)) & (radius <= max(1.0, n / 64) + 1)
        amp = torch.where(rim, -1.2 * amp - 2.0, amp)
    stop = radius <= max(1.0, n / 64)
    gap = max(1, n // 128)
    rows = (k >= n // 8) & (k < n // 8 + gap)
    cols = (k >= -(n // 8)) & (k < -(n // 8) + gap)
    amp = torch.where(stop | rows[:, None] | cols[None, :], -1.0, amp)
    start = (obj * math.sqrt(scale)).to(torch.complex64)
    rho = torch.randn(p, n, n, generator=g, device=DEV, dtype=torch.complex64)
    rho.mul_(SPREAD).add_(1.0).mul_(start)
    supp = _ellipse(n, 1.1 * a + 1, 1.1 * b + 1, math.pi * r[2]).to(torch.int32)
    if case["op"] == "crossover":  # individuals that the alignment has to move
        rho = torch.stack([torch.roll(rho[i], (i % 5 - 2, i % 3 - 1), (0, 1)) for i in range(p)])
        supp = torch.stack([torch.roll(supp, (i % 5 - 2, i % 3 - 1), (0, 1)) for i in range(p)])
    else:
        supp = supp.expand(p, n, n)
    return amp, rho, supp


def prepare(case, seed):
    n, p, op = case["n"], case["p"], case["op"]
    amp, rho, supp = _inputs(case, seed)
    state = {"case": case}
    if op == "sequence":
        img = torch.fft.fftshift(torch.where(amp >= 0, amp.double() ** 2, -1.0)).to(torch.float32).cpu().numpy()
        solver = Solver(img, use_bounds=False, seed=int(seed) & 0x7FFFFFFF)
        solver.set_sequence([("HIO", [case["iters"], case["beta"]]), ("SW", [case["sigma"], case["threshold"]]),
                             ("ER", [case["er"]])])
        state["solver"] = solver
        state["rec"] = Reconstruction(rho[0].cpu().numpy(), supp[0].cpu().numpy())
        return state
    engine = _lib.Engine(n, 0)
    engine.set_amplitudes(amp.cpu().numpy())
    engine.seed(int(seed) & 0x7FFFFFFF)
    state["engine"] = engine
    if op == "lossgrad":
        engine.reserve(p)
        state["density"] = rho.requires_grad_(True)
        state["support"] = supp.contiguous()
        return state
    children = op == "crossover"
    engine.reserve(2 * p + 2 if children else p)
    density, support = population_tensors(engine, 0, engine.capacity, torch.device(DEV, 0))
    density[:p].copy_(rho)
    support[:p].copy_(supp)
    if children:
        # slot 2p: the best individual, slot 2p + 1: the average
        density[2 * p].copy_(rho[0])
        support[2 * p].copy_(supp[0])
        density[2 * p + 1].copy_(rho.mean(dim=0))
        support[2 * p + 1].copy_(supp.amax(dim=0))
        g = torch.Generator()
        g.manual_seed(int(seed))
        state["errors"] = torch.rand(p, generator=g).numpy()
    state["density"], state["support"] = density, support
    if op == "shrinkwrap":
        state["area"] = int(supp[0].sum())
    torch.cuda.synchronize()
    return state


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _metric_arrays(metrics):
    return {k: np.array([m[k] for m in metrics], np.float32) for k in METRICS}


def run(state):
    case = state["case"]
    op, p = case["op"], case["p"]
    if op == "sequence":
        rec = state["solver"].Sequence(state["rec"])
        return {"density": rec.get_density(), "support": rec.get_support(),
                "metrics": _metric_arrays([{"error": rec.get_error(), "error_fourier": rec.get_fourier_error(),
                                            "error_real": rec.get_real_error(), "reality": rec.get_reality(),
                                            "modulesum": rec.get_module_sum(), "complexsum": rec.get_complex_sum(),
                                            "symmetry": rec.get_symmetry()}])}
    engine = state["engine"]
    if op == "iterate":
        if case["alg"] == "hio":
            engine.hio(0, p, case["iters"], case["beta"])
        elif case["alg"] == "raar":
            engine.raar(0, p, case["iters"], case["beta"])
        else:
            engine.er(0, p, case["iters"])
        return {"density": state["density"]}
    if op == "evaluate":
        return {"metrics": _metric_arrays(engine.evaluate(0, p))}
    if op == "shrinkwrap":
        if case["area"]:
            engine.swa(0, p, case["sigma"], state["area"])
        else:
            engine.sw(0, p, case["sigma"], case["threshold"])
        return {"support": state["support"]}
    if op == "crossover":
        engine.crossover(0, p, state["errors"], 2 * p, 2 * p + 1, p, 0.6, 0.4, crossft=case["crossft"],
                         use_average=case["average"])
        return {"density": state["density"][p:2 * p], "support": state["support"][p:2 * p]}
    if op == "lossgrad":
        rho = state["density"]
        rho.grad = None
        loss = farfield_loss(rho, state["support"], engine, case["loss"], 1e-6)
        loss.sum().backward()
        return {"loss": loss.detach(), "gradient": rho.grad}
    losses = refine(engine, 0, p, steps=case["steps"], lr=1e-3, loss=case["loss"], eps=1e-6,
                    device=state["density"].device)
    return {"losses": np.array(losses), "density": state["density"]}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    n, p, op = case["n"], case["p"], case["op"]
    px = float(n) * n * p
    fft = 5.0 * px * math.log2(float(n) * n)  # one 2D transform of the population
    amp = 4.0 * n * n
    if op == "iterate":
        return {"bytes": 20 * px + amp, "flops": (2 * case["iters"] + 2) * fft}
    if op == "sequence":
        return {"bytes": 24 * px + amp, "flops": (2 * (case["iters"] + case["er"] + 2) + 4 + 5) * fft}
    if op == "evaluate":
        return {"bytes": 12 * px + amp, "flops": 5 * fft}
    if op == "shrinkwrap":
        return {"bytes": 12 * px + amp, "flops": 4 * fft}
    if op == "crossover":
        ft = case["crossft"]
        return {"bytes": 24 * px + amp, "flops": (1 + 8 + 1 + 6 * ft) * fft}
    if op == "lossgrad":
        return {"bytes": 20 * px + amp, "flops": 2 * fft}
    return {"bytes": 20 * px + amp, "flops": 2 * case["steps"] * fft}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _forward(x):
    return torch.fft.ifft2(x) * (x.shape[-1] * x.shape[-1])


def _back(F):
    return torch.fft.fft2(F) / (F.shape[-1] * F.shape[-1])


def _project(F, amp):
    m = F.abs()
    unit = F / torch.where(m > 0, m, 1.0)
    known = torch.where(m > 0, unit, 1.0) * amp
    bound = -amp - 2.0
    return torch.where(amp >= 0, known, torch.where((amp < -1.5) & (m > bound), unit * bound, F))


def _iterate(rho, supp, amp, alg, iters, beta):
    s = supp.to(torch.float64)
    for _ in range(iters):
        rp = _back(_project(_forward(rho), amp))
        if alg == "er":
            rho = rp * s
        elif alg == "hio":
            rho = rp * s + (rho - beta * rp) * (1 - s)
        else:
            rho = torch.where(supp == 0, beta * rho + (1 - 2 * beta) * rp, rp)
    return _back(_project(_forward(rho), amp))


def _blur(rho, amp, sigma):
    n = rho.shape[-1]
    r = torch.arange(n, device=DEV, dtype=torch.float64)
    r = torch.where(r >= n // 2, r - n, r)
    sft = n / sigma / math.pi
    F = _forward(_back(_project(_forward(rho), amp)).abs().to(torch.complex128))
    return _back(F * torch.exp(-(r[:, None] ** 2 + r[None, :] ** 2) / sft ** 2)).abs()


def _symmetry(rho, amp):
    n = rho.shape[-1]
    r = torch.arange(n, device=DEV, dtype=torch.float64)
    r = torch.where(r >= n // 2, r - n, r)
    radius = torch.sqrt(r[:, None] ** 2 + r[None, :] ** 2)
    low, top = 1e-12, n / 2.0
    lo = radius - 0.9 * low
    hi = radius - 0.9 * top
    w = torch.where(lo > 0, 1 - torch.exp(-(lo / (0.1 * low)) ** 2), 0.0)
    w = (w * torch.where(hi > 0, torch.exp(-(hi / (0.1 * top)) ** 2), 1.0)) ** 2
    w = torch.where(amp < 0, 0.0, w)
    D = _forward(rho.abs().to(torch.complex128))
    peak = [torch.fft.fft2(c * w).abs().flatten(1).amax(dim=1) for c in (D.conj() * D, D * D)]
    return peak[1] / peak[0]


def _evaluate(rho, supp, amp):
    s = supp.to(torch.float64)
    inside = rho * s
    F = _forward(inside)
    m = F.abs()
    known = (amp >= 0).to(torch.float64)
    sums = lambda x: x.flatten(1).sum(dim=1)  # noqa: E731
    ef = torch.sqrt(sums(known * (amp - m) ** 2) / (known * amp ** 2).sum())
    back = _back(_project(F, amp))
    er = torch.sqrt(sums(torch.where(supp == 0, back.imag ** 2, 0.0)) / sums(back.abs() ** 2))
    modulesum, complexsum = sums(inside.abs()), m.flatten(1).amax(dim=1)
    reality = 1 - complexsum / modulesum
    return dict(zip(METRICS, (ef, ef, er, reality, modulesum, complexsum, _symmetry(rho, amp))))


def _loss(rho, supp, amp, kind, eps):
    """Loss per individual and its gradient (2 dL / d conj(rho))."""
    s = (supp > 0).to(torch.float64)
    F = _forward(rho * s)
    known = amp >= 0
    if kind == "amplitude":
        m = F.abs()
        loss = torch.where(known, (m - amp) ** 2, 0.0)
        g = torch.where(known & (m > 0), 2 * (m - amp) / torch.where(m > 0, m, 1.0), 0.0) * F
    else:
        m2 = F.abs() ** 2
        loss = torch.where(known, m2 - amp ** 2 * torch.log(m2 + eps), 0.0)
        g = torch.where(known, 2 * (1 - amp ** 2 / (m2 + eps)), 0.0) * F
    return loss.flatten(1).sum(dim=1), s * torch.fft.fft2(g)


def exact(case, seed):
    op, p, n = case["op"], case["p"], case["n"]
    if op in ("shrinkwrap", "crossover"):
        # a support is whole numbers; a crossover's outcome hangs on the
        # engine's random draws
        return None
    amp, rho, supp = _inputs(case, seed)
    amp = amp.double()
    step = max(1, 2 ** 24 // (n * n))
    beta = float(np.float32(case.get("beta", 0.0)))
    parts = []
    for i in range(0, p, step):
        r, s = rho[i:i + step].to(torch.complex128), supp[i:i + step]
        if op == "iterate":
            parts.append(_iterate(r, s, amp, case["alg"], case["iters"], beta))
        elif op == "evaluate":
            parts.append(_evaluate(r, s, amp))
        elif op == "lossgrad":
            parts.append(_loss(r, s, amp, case["loss"], float(np.float32(1e-6))))
        elif op == "sequence":
            r = _iterate(r, s, amp, "hio", case["iters"], beta)
            M = _blur(r, amp, case["sigma"])
            s = (M >= M.amax() * case["threshold"]).to(torch.int32)
            r = _iterate(r, s, amp, "er", case["er"], 0.0)
            return {"density": r[0], "support": None, "metrics": _evaluate(r, s, amp)}
        else:
            m, v, losses = torch.zeros_like(r), torch.zeros(r.shape + (2,), device=DEV, dtype=torch.float64), []
            b1, b2, lr = 0.9, 0.999, 1e-3
            for t in range(1, case["steps"] + 1):
                loss, grad = _loss(r, s, amp, case["loss"], float(np.float32(1e-6)))
                losses.append(loss.sum())
                m = b1 * m + (1 - b1) * grad
                v = b2 * v + (1 - b2) * torch.view_as_real(grad) ** 2
                den = torch.sqrt(v / (1 - b2 ** t)) + 1e-8
                r = r - lr / (1 - b1 ** t) * torch.view_as_complex(torch.view_as_real(m) / den)
            parts.append((torch.stack(losses), r))
    if op == "iterate":
        return {"density": torch.cat(parts)}
    if op == "evaluate":
        return {"metrics": {k: torch.cat([part[k] for part in parts]) for k in METRICS}}
    if op == "lossgrad":
        return {"loss": torch.cat([a for a, _ in parts]), "gradient": torch.cat([b for _, b in parts])}
    return {"losses": sum(a for a, _ in parts), "density": torch.cat([b for _, b in parts])}
