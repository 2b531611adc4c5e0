"""The work users have this package do, through its public entry points, at the sizes they use.

A wake simulation advances its particle field once per time step (vpm.nextstep, by the direct sum or
by the treecode), reads the state back for the host code that sheds the next particles, evaluates the
wake's velocity on probe points and the forces on bound particles, and runs its monitors.  Beside that
stand single U/∇U evaluations (verification in FP64, large fields on caller-owned device arrays) and
batches of independent fields.  Inputs follow the seeded workloads of flowunsteady_gb300.workloads.
"""
import ctypes
import math

import numpy as np
import torch

from flowunsteady_gb300 import _lib as L
from flowunsteady_gb300 import vpm
from flowunsteady_gb300.batch import FieldBatch
from flowunsteady_gb300.workloads import helical_wake, leapfrog_rings, uniform_box

_UJ = {"fp64": vpm.UJ_direct, "fp32c": vpm.UJ_gpu}
_KERNEL = {"gaussianerf": vpm.gaussianerf, "winckelmans": vpm.winckelmans}


def listed():
    return [
        # The first steps of a simulation: about a thousand particles shed so far, default options
        # (Gaussian-erf, FP32C, RK3, no SFS).  Latency and launches.
        _step("step_first_shedding", "wake", 1201, "fp32c", "none", 1e-4),
        # An ordinary rotor wake with the full method: dynamic SFS (the default finite-difference
        # procedure), core spreading and relaxation after the step.
        _step("step_rotor_sfs", "wake", 14003, "fp32c", "fd", 1e-4, relax=True),
        # A long wake on the default options, beyond the size from which pair passes run in Morton order.
        _step("step_long_wake", "wake", 81003, "fp32c", "none", 1e-3),
        # Two leapfrogging rings in the parity form: FP64 with dynamic SFS and core spreading.
        _step("step_rings_fp64", "rings", 7600, "fp64", "fd", 1e-3),
        # The default U/J evaluator of FLOWUnsteady is its FMM: a step by the treecode.
        _step("step_tree", "wake", 60007, "fp32c", "none", 1e-3, tree=True),
        # Verification: one FP64 U/J evaluation of the uniform box, read back.
        {"name": "uj_box_fp64", "kind": "uj", "field": "box", "n": 4096, "kernel": "winckelmans",
         "precision": "fp64", "tree": False},
        # A large field by the treecode, read back.
        {"name": "uj_tree_large", "kind": "uj", "field": "wake", "n": 500009, "kernel": "gaussianerf",
         "precision": "fp32c", "tree": True},
        # The benchmark's evaluation, on caller-owned device arrays.
        {"name": "uj_device_large", "kind": "device", "field": "wake", "n": 262144,
         "kernel": "gaussianerf", "precision": "fp32c"},
        # Velocity of the wake on the control points and probes of the lifting surfaces.
        {"name": "probes", "kind": "probes", "field": "wake", "n": 30011, "m": 2501,
         "kernel": "gaussianerf", "precision": "fp32c"},
        # Forces on bound particles from the free wake.
        {"name": "bound_forces", "kind": "forces", "field": "wake", "n": 30011, "m": 421,
         "kernel": "gaussianerf", "precision": "fp64"},
        # The monitors of a step: enstrophy, impulse, C_d statistics.
        {"name": "monitors", "kind": "monitors", "field": "wake", "n": 50021,
         "kernel": "gaussianerf", "precision": "fp32c"},
        # A parameter study: independent fields of uneven size, five steps with dynamic SFS
        # (analytic derivatives), then every field read back.
        {"name": "batch_study", "kind": "batch", "fields": 24, "lo": 512, "hi": 16384,
         "precision": "fp32c", "nsteps": 5, "dt": 1e-3},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step_small", "step", "step_long", "step_fp64", "step_tree", "uj_fp64",
                       "uj_tree", "device", "probes", "forces", "monitors", "batch"])
    kernel = rng.choice(["gaussianerf", "gaussianerf", "winckelmans"])
    if kind == "step_small":
        return _step(None, "wake", size(150, 5000), "fp32c", rng.choice(["none", "analytic"]), 1e-4,
                     relax=rng.random() < 0.3)
    if kind == "step":
        return _step(None, "wake", size(5000, 40000), "fp32c", rng.choice(["none", "fd", "analytic"]),
                     1e-4, relax=rng.random() < 0.5)
    if kind == "step_long":
        return _step(None, "wake", size(40000, 100000), "fp32c", rng.choice(["none", "analytic"]), 1e-3)
    if kind == "step_fp64":
        return _step(None, rng.choice(["wake", "box"]), size(500, 7600), "fp64",
                     rng.choice(["none", "fd", "analytic"]), 1e-3)
    if kind == "step_tree":
        return _step(None, "wake", size(8000, 250000), "fp32c", rng.choice(["none", "analytic"]), 1e-3,
                     tree=True)
    if kind == "uj_fp64":
        return {"kind": "uj", "field": rng.choice(["box", "wake"]), "n": size(500, 12000),
                "kernel": kernel, "precision": "fp64", "tree": False}
    if kind == "uj_tree":
        return {"kind": "uj", "field": "wake", "n": size(20000, 500000), "kernel": "gaussianerf",
                "precision": "fp32c", "tree": True}
    if kind == "device":
        return {"kind": "device", "field": rng.choice(["wake", "box"]), "n": size(1000, 230000),
                "kernel": kernel, "precision": "fp32c"}
    if kind == "probes":
        return {"kind": "probes", "field": "wake", "n": size(1000, 60000), "m": size(50, 4000),
                "kernel": kernel, "precision": rng.choice(["fp32c", "fp32c", "fp64"])}
    if kind == "forces":
        return {"kind": "forces", "field": "wake", "n": size(1000, 100000), "m": size(50, 2000),
                "kernel": kernel, "precision": "fp64"}
    if kind == "monitors":
        return {"kind": "monitors", "field": "wake", "n": size(1000, 150000), "kernel": kernel,
                "precision": "fp32c"}
    lo = size(200, 2000)
    return {"kind": "batch", "fields": rng.randint(3, 40), "lo": lo, "hi": lo * rng.randint(2, 16),
            "precision": "fp32c", "nsteps": rng.randint(1, 6), "dt": 1e-3}


def _step(name, field, n, precision, sfs, dt, relax=False, tree=False):
    c = {"kind": "step", "field": field, "n": n, "kernel": "gaussianerf", "precision": precision,
         "sfs": sfs, "nu": 0.0 if sfs == "none" else 1e-4, "relax": relax, "tree": tree, "dt": dt}
    return c if name is None else dict(c, name=name)


# ------------------------------------------------------------------ inputs --
def _field(case, seed):
    """X, Γ, σ of the case's particle field."""
    n = case["n"]
    if case["field"] == "box":
        return uniform_box(n, seed_index=seed, gamma_std=1e-2)
    if case["field"] == "rings":
        X, G, S = leapfrog_rings(nstations=n // 38)
        rng = np.random.default_rng(seed)
        return X + rng.normal(0.0, 2e-3, X.shape), G * rng.uniform(0.95, 1.05, (X.shape[0], 1)), S
    # The core size follows the particle spacing of a wake resolved by more or fewer particles.
    return helical_wake(n, turns=12 if n > 400000 else 4, seed_index=seed,
                        sigma=min(0.08, 0.03 * (262144.0 / n) ** (1.0 / 3.0)))


def _points(case, seed):
    rng = np.random.default_rng([seed, 1])
    th = rng.uniform(0.0, 2 * np.pi, case["m"])
    rad = rng.uniform(0.1, 1.1, case["m"])
    return np.stack([rad * np.cos(th), rad * np.sin(th), rng.uniform(-0.05, 0.9, case["m"])], axis=1)


def _bound(case, seed):
    rng = np.random.default_rng([seed, 2])
    return (_points(case, seed), rng.normal(0.0, 0.05, (case["m"], 3)),
            rng.uniform(0.02, 0.08, case["m"]))


def _memory(case, seed):
    rng = np.random.default_rng([seed, 3])
    C = np.zeros((case["n"], 3))
    C[:, 0] = np.where(rng.random(case["n"]) < 0.3, 0.0, rng.uniform(0.0, 1.0, case["n"]))
    C[:, 1:] = rng.normal(0.0, 1e-3, (case["n"], 2))
    return C


def _sizes(case):
    """Field sizes of a study, even and odd, spread over the logarithm of its range."""
    k = np.arange(case["fields"]) / max(case["fields"] - 1, 1)
    s = np.exp(np.log(case["lo"]) + k * np.log(case["hi"] / case["lo"])).astype(int)
    s[1::2] |= 1
    return [int(v) for v in s]


def _batch_fields(case, seed):
    rng = np.random.default_rng([seed, 4])
    return [uniform_box(n, seed_index=int(rng.integers(1 << 30)), gamma_std=1e-2)
            for n in _sizes(case)]


def _scheme(case):
    s = L.default_scheme()
    s.precision = {"fp64": L.PREC_FP64, "fp32c": L.PREC_FP32C}[case["precision"]]
    s.sfs = L.SFS_DYNAMIC
    s.sfs_flags = L.SFS_CLIP_BACKSCATTER | L.SFS_FORCE_POSITIVE | L.SFS_ANALYTIC_DSIGMA
    s.nu = 1e-4
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        b = FieldBatch(_sizes(case))
        for f, (X, G, S) in enumerate(_batch_fields(case, seed)):
            b.set_field(f, X, G, S)
        return {"case": case, "batch": b, "scheme": _scheme(case)}
    X, G, S = _field(case, seed)
    n = X.shape[0]
    if kind == "device":
        dev = torch.device("cuda:0")
        st = {"case": case, "n": n}
        st["X"] = torch.tensor(np.ascontiguousarray(X.T), device=dev)
        st["G"] = torch.tensor(np.ascontiguousarray(G.T), device=dev)
        st["S"] = torch.tensor(S, device=dev)
        st["U"] = torch.zeros((3, n), dtype=torch.float64, device=dev)
        st["J"] = torch.zeros((9, n), dtype=torch.float64, device=dev)
        return st
    sfs, viscous, relaxation = vpm.noSFS, None, None
    if case.get("sfs", "none") != "none":
        sfs, viscous = vpm.DynamicSFS(), vpm.CoreSpreading(case["nu"])
    if case.get("relax"):
        relaxation = vpm.pedrizzetti
    p = vpm.ParticleField(n + case.get("m", 0), kernel=_KERNEL[case["kernel"]],
                          UJ=_UJ[case["precision"]], SFS=sfs, viscous=viscous, relaxation=relaxation)
    if kind == "monitors":
        vpm.add_particle(p, X, G, S, C=_memory(case, seed))
        p.get_np()
    else:
        p.set_particles(X, G, S)
    st = {"case": case, "pfield": p}
    if kind == "probes":
        st["points"] = _points(case, seed)
    if kind == "forces":
        st["bound"] = _bound(case, seed)
    if kind == "uj" and case["tree"]:
        st["fmm"] = L.default_fmm()
    if kind == "step" and (case["tree"] or case["sfs"] == "analytic"):
        # Options that the scheme of the C ABI has beyond ParticleField's keywords.
        s = p.scheme()
        if case["tree"]:
            s.uj_method, s.fmm = L.UJ_TREE, L.default_fmm()
        if case["sfs"] == "analytic":
            s.sfs_flags |= L.SFS_ANALYTIC_DSIGMA
        st["scheme"] = s
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        b.step(case["dt"], state["scheme"], case["nsteps"])
        out = [b.get_field(f) for f in range(case["fields"])]
        # One array per quantity over all fields, as the study stores them.
        return {"X": np.concatenate([o[0] for o in out]), "G": np.concatenate([o[1] for o in out]),
                "S": np.concatenate([o[2] for o in out])}
    if kind == "device":
        n = state["n"]
        X, G, S, U, J = (state[k] for k in ("X", "G", "S", "U", "J"))
        k, prec = _KERNEL[case["kernel"]].id, _UJ[case["precision"]].precision
        L.check(L.lib().vpm_uj_device_async(
            k, prec, n, X.data_ptr(), G.data_ptr(), S.data_ptr(), n, n, None, n, U.data_ptr(),
            J.data_ptr(), n, torch.cuda.current_stream().cuda_stream))
        return {"U": U, "J": J}
    p = state["pfield"]
    if kind == "step":
        if "scheme" in state:
            L.check(L.lib().vpm_step(p._ctx, case["dt"], ctypes.byref(state["scheme"]), 1, 1),
                    p._ctx)
        else:
            vpm.nextstep(p, case["dt"], relax=case["relax"])
        X, G, S = p.state()
        return {"X": X, "G": G, "S": S}
    if kind == "uj":
        if case["tree"]:
            L.check(L.lib().vpm_eval_UJ_fmm(p._ctx, p.kernel.id, p.UJ.precision,
                                                 ctypes.byref(state["fmm"])), p._ctx)
        else:
            p.UJ(p)
        U, J = p.get_UJ()
        return {"U": U, "J": J}
    if kind == "probes":
        return vpm.Vvpm_on_Xs(p, state["points"])
    if kind == "forces":
        return vpm.Ffv_direct(p, *state["bound"])
    return p.diagnostics()


# -------------------------------------------------------------------- work --
def work(case):
    """Each input read once and each output written once; 60 flop per U/J pair, 66 more with the
    α-derivatives, 22 per ζ pair (44 with them), 45 per pair of a force evaluation.  A treecode
    evaluation cannot do with less than its near pairs: about 64 + 26·ncrit sources a target."""
    kind = case["kind"]
    if kind == "batch":
        sizes = _sizes(case)
        pairs = sum(float(s) ** 2 for s in sizes)
        return {"bytes": 112.0 * sum(sizes) * case["nsteps"],
                "flops": pairs * case["nsteps"] * (2 * (60 + 22) + (126 + 44))}
    n = float(case["n"])
    per = 1400.0 if case.get("tree") else n
    if kind == "step":
        stages = 3 * 60 + (60 if case["relax"] else 0)
        if case["sfs"] == "fd":
            stages += 3 * 22 + 60 + 22
        elif case["sfs"] == "analytic":
            stages += 2 * 22 + 66 + 44
        return {"bytes": 112.0 * n, "flops": n * per * stages}
    if kind in ("uj", "device"):
        return {"bytes": (56.0 + 96.0) * n, "flops": n * per * 60}
    if kind == "probes":
        return {"bytes": 56.0 * n + 48.0 * case["m"], "flops": case["m"] * n * 60}
    if kind == "forces":
        return {"bytes": 48.0 * n + 104.0 * case["m"], "flops": case["m"] * n * 45}
    return {"bytes": 64.0 * n, "flops": n * n * 22}


# ------------------------------------------------------------------- exact --
_INV4PI = 1.0 / (4.0 * math.pi)
_SQ2PI = math.sqrt(2.0 / math.pi)
_ALPHA = 0.999
_MOST_PAIRS = 2.5e10   # direct-sum pairs that torch takes well under 20 s for


def _zeta0(kernel):
    return 15.0 / (8.0 * math.pi) if kernel == "winckelmans" else (2.0 * math.pi) ** -1.5


def _gauss_h(x):
    """g/ρ³ and (ρg' - 3g)/ρ⁵ of the Gaussian-erf core at x = ρ²: series below 1, closed form above."""
    t, s1, s2, f = torch.clamp(x, max=1.0), torch.zeros_like(x), torch.zeros_like(x), 1.0
    for n in range(20):
        c = (-0.5) ** n / f
        s1 += (c / (2 * n + 3)) * t ** n
        s2 -= (c / (2 * n + 5)) * t ** n
        f *= n + 1
    y = torch.clamp(x, min=1.0)
    rho, e = torch.sqrt(y), torch.exp(-0.5 * y)
    g = torch.special.erf(rho * math.sqrt(0.5)) - _SQ2PI * rho * e
    h1 = g / (y * rho)
    h2 = (_SQ2PI * y * rho * e - 3.0 * g) / (y * y * rho)
    return torch.where(x < 1.0, _SQ2PI * s1, h1), torch.where(x < 1.0, _SQ2PI * s2, h2)


def _qp(kernel, r2, s, d=False):
    """q = g/r³ and q'/r of each pair (and their derivatives to a common scale of the cores)."""
    if kernel == "winckelmans":
        h = r2 + s * s
        q, p = (r2 + 2.5 * s * s) * h ** -2.5, -3.0 * (r2 + 3.5 * s * s) * h ** -3.5
        if d:
            return q, p, -7.5 * s ** 4 * h ** -3.5, 52.5 * s ** 4 * h ** -4.5
        return q, p
    x = r2 / (s * s)
    h1, h2 = _gauss_h(x)
    if d:
        e = _SQ2PI * torch.exp(-0.5 * x)
        return h1 / s ** 3, h2 / s ** 5, -e / s ** 3, e / s ** 5
    return h1 / s ** 3, h2 / s ** 5


def _chunks(m, n):
    step = max(1, (1 << 23) // max(n, 1))
    return [(a, min(m, a + step)) for a in range(0, m, step)]


def _pass_uj(kernel, T, X, G, S, d=False):
    """U, J (and dJ/dα) at the rows of T."""
    m = T.shape[0]
    U, J = T.new_zeros((m, 3)), T.new_zeros((m, 3, 3))
    DJ = T.new_zeros((m, 3, 3)) if d else None
    for a, b in _chunks(m, X.shape[0]):
        D = [T[a:b, None, k] - X[None, :, k] for k in range(3)]
        r2 = D[0] * D[0] + D[1] * D[1] + D[2] * D[2]
        off = (r2 > 0.0).to(r2.dtype)
        v = [w * off for w in _qp(kernel, r2, S[None], d)]
        g = [G[None, :, k] for k in range(3)]
        c = [D[1] * g[2] - D[2] * g[1], D[2] * g[0] - D[0] * g[2], D[0] * g[1] - D[1] * g[0]]
        for k in range(3):
            U[a:b, k] = -_INV4PI * (v[0] * c[k]).sum(1)
        for out, q, p in ((J, v[0], v[1]),) + (((DJ, v[2], v[3]),) if d else ()):
            w = [(q * g[k]).sum(1) for k in range(3)]
            for i in range(3):
                pc = p * c[i]
                for k in range(3):
                    out[a:b, i, k] = -_INV4PI * (pc * D[k]).sum(1)
            for i, k, l, sg in ((0, 1, 2, 1), (1, 2, 0, 1), (2, 0, 1, 1), (1, 0, 2, -1), (2, 1, 0, -1),
                                (0, 2, 1, -1)):
                out[a:b, i, k] += -_INV4PI * sg * w[l]
    return (U, J, DJ) if d else (U, J)


def _pass_zeta(kernel, X, G, S, V, W=None):
    """Σ ζ Γ and Σ ζ v at every particle without its own term (and their α-derivatives)."""
    n = X.shape[0]
    out = X.new_zeros((n, 6 if W is None else 12))
    z0 = _zeta0(kernel)
    for a, b in _chunks(n, n):
        r2 = sum((X[a:b, None, k] - X[None, :, k]) ** 2 for k in range(3))
        x = r2 / (S * S)[None]
        z = z0 / (S ** 3)[None] * ((x + 1.0) ** -3.5 if kernel == "winckelmans" else torch.exp(-0.5 * x))
        z = torch.where(r2 > 0.0, z, torch.zeros_like(z))
        out[a:b, :3], out[a:b, 3:6] = z @ G, z @ V
        if W is not None:
            dz = z * ((4.0 - 7.0 / (x + 1.0)) if kernel == "winckelmans" else (x - 3.0))
            out[a:b, 6:9], out[a:b, 9:12] = dz @ G, dz @ V + z @ W
    return out


def _stretch(J, v):
    return torch.einsum("iba,ib->ia", J, v)   # the transposed scheme


def _sfs_stage(kernel, X, G, S, C, mode, first):
    """U, J, E_str of a stage; the first one sets C_d (rlxf 1, positive, at most 1)."""
    z0 = _zeta0(kernel)
    if first and mode == "analytic":
        U, J, DJ = _pass_uj(kernel, X, X, G, S, True)
        o = _pass_zeta(kernel, X, G, S, _stretch(J, G), _stretch(DJ, G))
        E = _stretch(J, o[:, :3]) - o[:, 3:6]
        DE = _stretch(DJ, o[:, :3]) + _stretch(J, o[:, 6:9]) - o[:, 9:12]
        h = _ALPHA - 1.0
        num, den = h * (G * _stretch(DJ, G)).sum(1), h * (G * DE).sum(1)
    else:
        U, J = _pass_uj(kernel, X, X, G, S)
        o = _pass_zeta(kernel, X, G, S, _stretch(J, G))
        E = _stretch(J, o[:, :3]) - o[:, 3:6]
        if not first:
            return U, J, E, C
        _, Jt = _pass_uj(kernel, X, X, G, _ALPHA * S)
        o = _pass_zeta(kernel, X, G, _ALPHA * S, _stretch(Jt, G))
        Et = _stretch(Jt, o[:, :3]) - o[:, 3:6]
        num, den = (G * (_stretch(Jt, G) - _stretch(J, G))).sum(1), (G * (Et - E)).sum(1)
    num, den = num * (3.0 * _ALPHA - 2.0), den * S ** 3 / z0
    C = torch.where(den != 0.0, num / torch.where(den != 0.0, den, torch.ones_like(den)),
                    torch.zeros_like(den)).abs().clamp(max=1.0)
    return U, J, E, C


def _exact_steps(kernel, X, G, S, dt, nsteps, mode, nu, relax):
    """Low-storage RK3 steps of the reformulated method (f = 0, g = 1/5)."""
    z0 = _zeta0(kernel)
    for _ in range(nsteps):
        QX, QG, QS, QN, C = (torch.zeros_like(v) for v in (X, G, S, S, S))
        for k, (a, b) in enumerate(((0.0, 1 / 3), (-5 / 9, 15 / 16), (-153 / 128, 8 / 15))):
            if mode == "none":
                (U, J), E, cz = _pass_uj(kernel, X, X, G, S), torch.zeros_like(G), torch.zeros_like(S)
            else:
                U, J, E, C = _sfs_stage(kernel, X, G, S, C, mode, k == 0)
                C = torch.where(C * (G * E).sum(1) < 0.0, torch.zeros_like(C), C)
                cz = C * S ** 3 / z0
            s, gg = _stretch(J, G), (G * G).sum(1)
            Z = torch.where(gg > 0.0, 0.2 * (s * G).sum(1) / torch.where(gg > 0.0, gg, 1.0 + gg),
                            torch.zeros_like(gg))
            QX = a * QX + dt * U
            QG = a * QG + dt * (s - 3.0 * Z[:, None] * G - cz[:, None] * E)
            QS = a * QS - dt * S * Z
            X, G, S = X + b * QX, G + b * QG, S + b * QS
            if nu > 0.0:
                QN = a * QN + dt * 2.0 * nu
                S = torch.sqrt(S * S + b * QN)
        if relax:
            _, J = _pass_uj(kernel, X, X, G, S)
            w = torch.stack([J[:, 2, 1] - J[:, 1, 2], J[:, 0, 2] - J[:, 2, 0],
                             J[:, 1, 0] - J[:, 0, 1]], 1)
            r = 0.3
            G = (1.0 - r) * G + r * G.norm(dim=1, keepdim=True) * w / w.norm(dim=1, keepdim=True)
    return X, G, S


def exact(case, seed):
    dev = torch.device("cuda:0")
    t = lambda v: torch.tensor(np.ascontiguousarray(v), dtype=torch.float64, device=dev)  # noqa: E731
    kind = case["kind"]
    if kind == "batch":
        if sum(float(s) ** 2 for s in _sizes(case)) * 4.5 * case["nsteps"] > _MOST_PAIRS:
            return None
        outs = [_exact_steps("gaussianerf", t(X), t(G), t(S), case["dt"], case["nsteps"], "analytic",
                             1e-4, False) for X, G, S in _batch_fields(case, seed)]
        return {k: torch.cat([o[i] for o in outs]).cpu().numpy() for i, k in enumerate("XGS")}
    n, kernel = float(case["n"]), case["kernel"]
    passes = {"step": {"none": 3, "fd": 6, "analytic": 5}.get(case.get("sfs"), 3) + 1, "monitors": 0.4}
    if n * (case["m"] if "m" in case else n) * passes.get(kind, 1) > _MOST_PAIRS:
        return None
    X, G, S = (t(v) for v in _field(case, seed))
    if kind == "step":
        X, G, S = _exact_steps(kernel, X, G, S, case["dt"], 1, case["sfs"], case["nu"], case["relax"])
        return {"X": X.cpu().numpy(), "G": G.cpu().numpy(), "S": S.cpu().numpy()}
    if kind == "uj":
        U, J = _pass_uj(kernel, X, X, G, S)
        return {"U": U.cpu().numpy(), "J": J.cpu().numpy()}
    if kind == "device":
        U, J = _pass_uj(kernel, X, X, G, S)
        return {"U": U.T.contiguous(), "J": J.reshape(-1, 9).T.contiguous()}
    if kind == "probes":
        return _pass_uj(kernel, t(_points(case, seed)), X, G, S)[0].cpu().numpy()
    if kind == "forces":
        Xb, Gb, Sb = (t(v) for v in _bound(case, seed))
        M = Xb.new_zeros((case["m"], 6))
        for a, b in _chunks(case["m"], 4 * X.shape[0]):
            d = X[None] - Xb[a:b, None]
            r2 = (d * d).sum(2)
            q = torch.where(r2 > 0.0, _qp(kernel, r2, Sb[a:b, None])[0], torch.zeros_like(r2))
            gb, gf = Gb[a:b, None].expand_as(d), G[None].expand_as(d)
            u = -_INV4PI * q[..., None] * torch.linalg.cross(d, gb)
            M[a:b, :3] = torch.linalg.cross(u, gf).sum(1)
            M[a:b, 3:] = (_INV4PI * q[..., None] * torch.linalg.cross(d, torch.linalg.cross(gb, gf))).sum(1)
        return M.cpu().numpy()
    om = _pass_zeta(kernel, X, G, S, G)[:, :3] + (_zeta0(kernel) / S ** 3)[:, None] * G
    imp, gam = 0.5 * torch.linalg.cross(X, G).sum(0), G.sum(0)
    c = t(_memory(case, seed)[:, 0])
    nz = c[c != 0.0]
    mean = nz.mean()
    m2, m3, m4 = (((nz - mean) ** k).mean() for k in (2, 3, 4))
    return {k: float(v) for k, v in {
        "enstrophy": 0.5 * (G * om).sum(), "impulse_x": imp[0], "impulse_y": imp[1], "impulse_z": imp[2],
        "gamma_x": gam[0], "gamma_y": gam[1], "gamma_z": gam[2], "cd_mean": mean,
        "cd_std": m2.sqrt(), "cd_zero_ratio": 1.0 - nz.numel() / c.numel(), "cd_min": nz.min(),
        "cd_max": nz.max(), "sigma_mean": S.mean(), "nonfinite": 0.0, "cd_skew": m3 / m2 ** 1.5,
        "cd_kurt": m4 / (m2 * m2) - 3.0}.items()}
