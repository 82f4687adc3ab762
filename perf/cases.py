"""The measured cases of chaos_b200: what a user of the engine has it do, through its public calls, from one small
ensemble to the largest workloads of bench.py.

A case is a dict of plain values; `kind` picks the call:

  propagate    `propagate(sys, x0, N, k=, tau=, reducers=)`: host arrays in, the full result back
  frames       `propagate_frames` with two frames on one orbit (Lyapunov spectrum | GALI + SALI)
  ensemble     `propagate_ensemble` of uneven lattice classes with an escape stop
  record       the study recorder, grid rows
  predict      the screen network's inference pass on device-resident features
  train        one training step of the screen network

`propagate` and the recorders take and return host (numpy) arrays, as the reference's call does, so the copies and
the host's own records are part of a pass.
"""
import math

import numpy as np
import torch

from chaos_b200 import (FLI, GALI, MEGNO, MGS, SALI, FrameSpec, FroeschleMap, Gauss, GivensQR, HenonHeilesFlow,
                        HouseholderQR, IntegratorMap, KahanLi, QRSpectrum, StandardMap, StandardMapChain,
                        WrappedFroeschleMap, WrappedStandardMap, propagate, propagate_frames, random_energy_starts,
                        record)
from chaos_b200.ensemble import lattice_workload, propagate_ensemble
from chaos_b200.mlp import MLP

TWO_PI = 2 * math.pi


def listed():
    return [
        # a first look at one map: a few hundred orbits, where launches, copies and host work count most
        dict(name="standard_small", kind="propagate", system="standard", chain="mgs", n=257, N=1000, tau=1),
        # the reference's own chaos-indicator benchmark size (2e4 orbits x 1e3 steps, K = 2 pi), three indicators at once
        dict(name="standard_indicators", kind="propagate", system="standard", chain="megno-fli-sali", n=20001, N=1000,
             tau=1),
        # Chirikov's map on the torus at the parity configuration's ensemble, K = 6, renormalised every step
        dict(name="wrapped_spectrum", kind="propagate", system="wrapped", chain="mgs", n=4096, N=20000, tau=1),
        # the coupled-maps workload in the default precision (Float64 throughout)
        dict(name="coupled_fp64", kind="frames", system="froeschle", precision="fp64", n=65536, N=10000, tau=10),
        # the same workload at its full length in the precision made for it (bench.py's default workload)
        dict(name="coupled_split", kind="frames", system="froeschle", precision="mixed-ind64", n=65536, N=100000,
             tau=10),
        # Henon-Heiles by Gauss-Legendre collocation with its exact tangent, three reducers in a chain
        dict(name="henon_gauss", kind="propagate", system="gauss", chain="megno-fli-givens", n=16384, N=1000, tau=10),
        # Henon-Heiles by an 18-stage symplectic splitting
        dict(name="henon_kahanli", kind="propagate", system="kahanli", chain="megno-fli-givens", n=16384, N=10000,
             tau=10),
        # uneven lattices d = 2, 4, 8, 16 with per-orbit lengths and an escape stop, one call
        dict(name="lattice_ensemble", kind="ensemble", precision="mixed", n=40000, N=100000),
        # a lattice of 8 sites, d = 16, eight exponents of a modest ensemble
        dict(name="lattice_spectrum", kind="propagate", system="chain8", chain="householder", n=2048, N=2000, tau=10),
        # the study recorder: log-spaced grid rows of every orbit
        dict(name="record_rows", kind="record", system="wrapped", n=4099, N=10000, tau=1, rows=80),
        # the screen network: every orbit of a 512 x 512 grid at once
        dict(name="screen_predict", kind="predict", rows=262144),
        # the screen network: one training step at the pipeline's batch
        dict(name="screen_train", kind="train", rows=4096),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# kind, system, chains, orbits, orbit-steps at most (about the listed case's time)
_PROPAGATE = (
    ("standard", ("mgs", "householder", "megno-fli-sali", "sali", "megno", "fli"), (64, 65536), 3e7),
    ("wrapped", ("mgs", "householder", "megno-fli-sali", "sali"), (64, 16384), 8e7),
    ("gauss", ("megno-fli-givens",), (64, 16384), 1.2e7),
    ("kahanli", ("megno-fli-givens", "mgs"), (64, 16384), 1.2e8),
    ("chain8", ("householder", "mgs", "gali"), (64, 4096), 4e6),
    ("chain4", ("householder", "mgs", "gali"), (64, 16384), 1.2e7),
)


def draw(rng):
    kind = rng.choice(("propagate", "propagate", "propagate", "propagate", "frames", "frames", "ensemble", "record",
                       "predict", "train"))
    if kind == "propagate":
        system, chains, (lo, hi), most = rng.choice(_PROPAGATE)
        n = _spread(rng, lo, hi) | 1
        tau = 1 if system in ("standard", "wrapped") else rng.choice((1, 5, 10))
        N = _spread(rng, 200, max(400, min(20000, most / n)))
        return dict(kind=kind, system=system, chain=rng.choice(chains), n=n, N=max(1, N // tau) * tau, tau=tau)
    if kind == "frames":
        system, precision, most = rng.choice((("froeschle", "fp64", 6e8), ("froeschle", "mixed-ind64", 4e9),
                                              ("froeschle-torus", "fp64", 4e8)))
        n, tau = _spread(rng, 256, 65536) | 1, rng.choice((1, 5, 10, 20))
        N = _spread(rng, 200, max(400, min(50000, most * tau / 10 / n)))
        return dict(kind=kind, system=system, precision=precision, n=n, N=max(1, N // tau) * tau, tau=tau)
    if kind == "ensemble":
        return dict(kind=kind, precision=rng.choice(("mixed", "fp64")), n=4 * _spread(rng, 64, 4096),
                    N=_spread(rng, 2000, 30000))
    if kind == "record":
        n = _spread(rng, 64, 8192) | 1
        return dict(kind=kind, system=rng.choice(("wrapped", "standard")), n=n,
                    N=_spread(rng, 200, max(400, min(20000, 4e7 / n))), tau=1, rows=rng.randint(5, 90))
    if kind == "predict":
        return dict(kind=kind, rows=_spread(rng, 100, 262144) | 1)
    return dict(kind=kind, rows=128 * _spread(rng, 1, 64))


# ---- inputs --------------------------------------------------------------------------------------------------------

def _system(name):
    """(map, tangent dimension, deviation vectors of a full-spectrum chain)"""
    if name == "standard":
        return StandardMap(TWO_PI), 2, 2
    if name == "wrapped":
        return WrappedStandardMap(6.0), 2, 2
    if name == "froeschle":
        return FroeschleMap(1.5, 1.5, 0.05), 4, 4
    if name == "froeschle-torus":
        return WrappedFroeschleMap(1.5, 1.5, 0.05), 4, 4
    if name == "gauss":
        return IntegratorMap(Gauss(3, tol=1e-14), HenonHeilesFlow(), 0.01), 4, 2
    if name == "kahanli":
        return IntegratorMap(KahanLi(8), HenonHeilesFlow(), 0.05), 4, 2
    sites = int(name[5:])
    return StandardMapChain(sites, 1.2, 0.05), 2 * sites, min(2 * sites, 8)


def _starts(name, d, n, seed):
    if name in ("gauss", "kahanli"):
        return random_energy_starts(1 / 8, n, seed=seed)
    x = np.random.default_rng(seed).uniform(0, TWO_PI, (n, d))
    if name in ("wrapped", "froeschle-torus"):   # reduced coordinates and their winding counts, all zero
        return np.concatenate([x, np.zeros((n, d))], axis=1)
    return x


def _chain(name):
    return {"mgs": (QRSpectrum(MGS()),), "householder": (QRSpectrum(HouseholderQR()),), "gali": (GALI(),),
            "sali": (SALI(),), "megno": (MEGNO(),), "fli": (FLI(),),
            "megno-fli-sali": (MEGNO(replace=False), FLI(replace=False), SALI()),
            "megno-fli-givens": (MEGNO(replace=False), FLI(replace=False), QRSpectrum(GivensQR()))}[name]


def _identity(n, d, k):
    return np.ascontiguousarray(np.broadcast_to(np.eye(d)[:, :k], (n, d, k)))


def _features(rows, seed, device):
    """Screen features as the coupled-maps ensemble gives them: per window the column-1 stretch rate, log10 SALI / 8
    and Y / 4, then the four end-of-prefix columns; most rows chaotic, SALI falling to its floor."""
    g = torch.Generator(device=device).manual_seed(seed)
    def normal(*shape):
        return torch.randn(*shape, generator=g, device=device)
    w = torch.arange(1, 21, device=device, dtype=torch.float32)
    chaotic = (torch.rand(rows, 1, generator=g, device=device) < 0.9).float()
    rate = chaotic * (0.5 + 0.15 * normal(rows, 1)).abs() * (1 + 0.2 * normal(rows, 20) / w.sqrt())
    rate = rate + (1 - chaotic) * 0.03 / w * (1 + 0.3 * normal(rows, 20))
    lsal = torch.maximum(-rate * w * 100 / 2.3, torch.full_like(rate, -16.0)) / 8 + 0.02 * normal(rows, 20)
    Y = (chaotic * rate * 100 * w / 4 + (1 - chaotic) * (2 + 0.2 * normal(rows, 20))) / 4
    X = torch.zeros(rows, 64, device=device)
    X[:, 0:60:3], X[:, 1:60:3], X[:, 2:60:3] = rate, lsal, Y
    X[:, 60], X[:, 61], X[:, 62] = Y.mean(1), rate[:, -1], lsal[:, -1]
    return X.to(torch.bfloat16), chaotic[:, 0].contiguous(), rate[:, -1].contiguous()


def _network(seed, device):
    """A network in the middle of its training: nonzero biases, Adam moments of a few hundred steps."""
    net = MLP(torch, device, seed=seed)
    g = torch.Generator(device=device).manual_seed(seed + 1)
    for lay in net.layers:
        lay["b"].copy_(0.1 * torch.randn(lay["b"].shape, generator=g, device=device))
        for p in ("W", "b"):
            m = 1e-3 * torch.randn(lay[p].shape, generator=g, device=device)
            lay["m" + p].copy_(m)
            lay["v" + p].copy_(m * m + 1e-6)
    net.step = 300
    return net


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("predict", "train"):
        device = torch.device("cuda", torch.cuda.current_device())
        X, label, target = _features(case["rows"], seed, device)
        return dict(case=case, net=_network(seed, device), X=X, label=label, target=target)
    if kind == "ensemble":
        classes = lattice_workload(case["n"], seed=seed, n_max=case["N"], precision=case["precision"])
        return dict(case=case, classes=classes)
    sysm, d, k = _system(case["system"])
    st = dict(case=case, sys=sysm, x0=_starts(case["system"], d, case["n"], seed))
    if kind == "propagate":
        st["chain"] = _chain(case["chain"])
        st["k"] = k if case["chain"] in ("mgs", "householder", "gali") else 2
        st["W0"] = _identity(case["n"], d, st["k"])
    elif kind == "frames":
        W0 = _identity(case["n"], 4, 4)
        st["frames"] = [FrameSpec(4, (QRSpectrum(HouseholderQR()),), W0), FrameSpec(4, (GALI(), SALI()), W0)]
    else:
        st["chain"] = (QRSpectrum(MGS()),)
        rows = np.logspace(0, math.log10(case["N"]), case["rows"])
        st["grid"] = np.unique(np.round(rows / case["tau"]).clip(1).astype(np.int64) * case["tau"])
    return st


# ---- one pass ------------------------------------------------------------------------------------------------------

def _fields(states):
    """A structured array of reducer states as one array (a view) per field."""
    out = {}
    for r in states.dtype.names or ():
        sub = states[r]
        out[r] = {f: sub[f] for f in sub.dtype.names if not f.startswith("_")}
    return out


def _result(r):
    out = dict(x=r.x, W=r.W, code=r.code, hstep=r.hstep)
    if r.states is not None:
        out["states"] = _fields(r.states)
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "propagate":
        return _result(propagate(state["sys"], state["x0"], case["N"], k=state["k"], tau=case["tau"],
                                 reducers=state["chain"], W0=state["W0"]))
    if kind == "frames":
        return [_result(r) for r in propagate_frames(state["sys"], state["x0"], case["N"], state["frames"],
                                                     tau=case["tau"], precision=case["precision"], throw=False)]
    if kind == "ensemble":
        return [_result(r) for r in propagate_ensemble(state["classes"])]
    if kind == "record":
        r = record(state["sys"], state["x0"], case["N"], case["tau"], state["chain"][0], state["grid"])
        return dict(R=r.R, fail=r.fail, x=r.x, W=r.W, code=r.code, hstep=r.hstep, states=r.states)
    net = state["net"]
    if kind == "predict":
        return net.predict(state["X"])
    loss = net.train_step(state["X"], state["label"], state["target"], w_reg=1.0, lr=2e-3)
    return dict(loss=loss, W=[lay["W"] for lay in net.layers], b=[lay["b"] for lay in net.layers],
                gW=[lay["gW"] for lay in net.layers], gb=[lay["gb"] for lay in net.layers])


# ---- the work a pass cannot do without -----------------------------------------------------------------------------

# Operations of one map step (a sine or cosine counted as 16: its polynomial), of the tangent product per deviation
# vector, and of one handoff of a chain with k vectors of d entries.
_STEP = {"standard": 36, "wrapped": 44, "froeschle": 110, "froeschle-torus": 220, "gauss": 6 * 3 * 40 + 1200,
         "kahanli": 18 * 20}
_TANGENT = {"standard": 4, "wrapped": 4, "froeschle": 16, "froeschle-torus": 16, "gauss": 28, "kahanli": 18 * 12}


def _map_flops(system, k):
    if system.startswith("chain"):
        sites = int(system[5:])
        return sites * 70 + k * 9 * sites
    return _STEP[system] + k * _TANGENT[system]


def _handoff_flops(chain, d, k):
    logs = 30 * k
    if chain in ("mgs", "householder", "megno-fli-givens"):
        extra = 120 if "megno" in chain else 0
        return 4 * d * k * k + k ** 3 // 3 + logs + extra
    if chain == "gali":
        return 6 * d * k * k + logs
    return 12 * d + logs + (120 if "megno" in chain else 30)


def work(case):
    kind = case["kind"]
    if kind in ("predict", "train"):
        per = 2 * (64 * 256 + 2 * 256 * 256 + 256 * 2)
        weights = 64 * 256 + 2 * 256 * 256 + 256 * 2
        if kind == "predict":
            return dict(bytes=case["rows"] * (64 * 2 + 16 * 4) + 2 * weights, flops=case["rows"] * per)
        back = 2 * per - 2 * 64 * 256
        return dict(bytes=case["rows"] * (64 * 2 + 12) + 4 * 7 * weights, flops=case["rows"] * (per + back))
    if kind == "ensemble":
        per = case["n"] // 4
        mean = (case["N"] - 1e3) / math.log(case["N"] / 1e3)
        flops = bytes_ = 0
        for d, tau in ((2, 5), (4, 10), (8, 10), (16, 20)):
            k = min(d, 8)
            system = "standard" if d == 2 else f"chain{d // 2}"
            flops += per * mean * (_map_flops(system, k) + _handoff_flops("householder", d, k) / tau)
            bytes_ += per * (8 * (2 * d + 2 * d * k + 2 * k) + 100)
        return dict(bytes=bytes_, flops=flops)
    n, N, tau = case["n"], case["N"], case["tau"]
    _, d, kfull = _system(case["system"])
    s = 2 * d if case["system"] in ("wrapped", "froeschle-torus") else d
    if kind == "frames":
        hand = _handoff_flops("householder", 4, 4) + 4 * 8 + 30 * 4
        return dict(bytes=n * (16 * s + 4 * 128 + 17 * 8 + 25 * 8 + 18),
                    flops=n * N * (_map_flops(case["system"], 8) + hand / tau))
    chain = case.get("chain", "mgs")
    k = kfull if chain in ("mgs", "householder", "gali") else 2
    flops = n * N * (_map_flops(case["system"], k) + _handoff_flops(chain, d, k) / tau)
    bytes_ = n * (16 * s + 16 * d * k + 16 * k + 81)
    if kind == "record":
        flops += n * N * 20
        bytes_ += 8 * n * case["rows"] * (k + 7 + s)
    return dict(bytes=bytes_, flops=flops)


# ---- the same in plain 64-bit arithmetic ---------------------------------------------------------------------------

def _gauss_exact(case, seed):
    """x and W after the run, by the collocation equations solved to convergence in 64 bits: the starts lie on
    the E = 1/8 shell and 10 time units amplify rounding by less than a hundred, so they have such a value. The frame
    spans what the product of the steps' tangents spans, orthonormalised every tau steps with positive diagonals."""
    dev = torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")
    z = torch.tensor(_starts("gauss", 4, case["n"], seed), device=dev)
    h, r15 = 0.01, math.sqrt(15.0)
    A = torch.tensor([[5 / 36, 2 / 9 - r15 / 15, 5 / 36 - r15 / 30], [5 / 36 + r15 / 24, 2 / 9, 5 / 36 - r15 / 24],
                      [5 / 36 + r15 / 30, 2 / 9 + r15 / 15, 5 / 36]], dtype=torch.float64, device=dev)
    b = torch.tensor([5 / 18, 4 / 9, 5 / 18], dtype=torch.float64, device=dev)
    n = case["n"]
    W = torch.zeros(n, 4, 2, dtype=torch.float64, device=dev)
    W[:, 0, 0] = W[:, 1, 1] = 1.0

    def field(y):   # (..., 4) -> (..., 4)
        q1, q2 = y[..., 0], y[..., 1]
        return torch.stack([y[..., 2], y[..., 3], -(q1 + 2 * q1 * q2), -(q2 + q1 * q1 - q2 * q2)], -1)

    def jac_times(y, v):   # y (n, 3, 4), v (n, 3, 4, k)
        q1, q2 = y[..., 0, None], y[..., 1, None]
        a, c = v[..., 0, :], v[..., 1, :]
        return torch.stack([v[..., 2, :], v[..., 3, :], -((1 + 2 * q2) * a + 2 * q1 * c),
                            -(2 * q1 * a + (1 - 2 * q2) * c)], -2)

    for step in range(case["N"]):
        Y = z[:, None, :].expand(n, 3, 4)
        for _ in range(12):
            Y = z[:, None, :] + h * torch.einsum("ij,njc->nic", A, field(Y))
        V = W[:, None].expand(n, 3, 4, 2)
        for _ in range(12):
            V = W[:, None] + h * torch.einsum("ij,njck->nick", A, jac_times(Y, V))
        W = W + h * torch.einsum("i,nick->nck", b, jac_times(Y, V))
        z = z + h * torch.einsum("i,nic->nc", b, field(Y))
        if (step + 1) % case["tau"] == 0:
            q0 = W[:, :, 0] / W[:, :, 0].norm(dim=1, keepdim=True)
            u = W[:, :, 1] - (q0 * W[:, :, 1]).sum(1, keepdim=True) * q0
            u = u - (q0 * u).sum(1, keepdim=True) * q0
            W = torch.stack([q0, u / u.norm(dim=1, keepdim=True)], -1)
    return dict(x=z.cpu().numpy(), W=W.cpu().numpy(), code=None, hstep=None, states=None)


def _gelu(z):
    return 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))


def _network_exact(case, seed):
    st = prepare(case, seed)
    net = st["net"]
    params = [(lay["W"].double().requires_grad_(), lay["b"].double().requires_grad_()) for lay in net.layers]
    a = st["X"].double()
    for i, (W, b) in enumerate(params):
        z = a @ W.T + b
        a = _gelu(z) if i + 1 < len(params) else z
    if case["kind"] == "predict":
        return a.detach()
    t, lam = st["label"].double(), st["target"].double()
    loss = torch.nn.functional.binary_cross_entropy_with_logits(a[:, 0], t, reduction="none") + (a[:, 1] - lam) ** 2
    loss.mean().backward()
    out = dict(loss=loss.detach(), W=[], b=[], gW=[], gb=[])
    step = net.step + 1
    for lay, (W, b) in zip(net.layers, params):
        for p, v in (("W", W), ("b", b)):
            g = v.grad
            m = 0.9 * lay["m" + p].double() + 0.1 * g
            s = 0.999 * lay["v" + p].double() + 0.001 * g * g
            out[p].append(v.detach() - 2e-3 * (m / (1 - 0.9 ** step)) / ((s / (1 - 0.999 ** step)).sqrt() + 1e-8))
            out["g" + p].append(g)
    return out


def exact(case, seed):
    """The other propagation cases run chaotic orbits over hundreds to a hundred thousand steps: another rounding of
    one sine changes every digit, so their outputs have no value that plain 64-bit arithmetic would give again."""
    if case["kind"] in ("predict", "train"):
        return _network_exact(case, seed)
    if case["kind"] == "propagate" and case["system"] == "gauss" and case["n"] * case["N"] <= 2e7 \
            and case["N"] <= 2000:
        return _gauss_exact(case, seed)
    return None
