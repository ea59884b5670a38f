"""Performance cases of the phaseless-AFQMC engine.

Each case is one call that a program using this package makes on its hot path: a block, a step, the
driver's block loop, the local energy, the population's QR, the differentiated run.  Hamiltonians follow the
synthetic recipe of ``ad_afqmc_prototype_gb300.synth`` (drawn on the GPU, so that large ones are quick).

``listed()`` holds sizes of this repository's workloads and odd ones between them, ``draw(rng)`` spreads
over the same ranges.  Step and energy cases are given their auxiliary fields (a run on common random
numbers); block, driver and gradient cases draw theirs from the engine's own stream.
"""
from __future__ import annotations

import math

import torch

from ad_afqmc_prototype_gb300 import walkers as wk
from ad_afqmc_prototype_gb300.core.ops import k_energy
from ad_afqmc_prototype_gb300.core.system import system
from ad_afqmc_prototype_gb300.driver import make_run_blocks
from ad_afqmc_prototype_gb300.grad import block_energies
from ad_afqmc_prototype_gb300.ham.chol import ham_chol
from ad_afqmc_prototype_gb300.meas.rhf import make_rhf_meas_ops
from ad_afqmc_prototype_gb300.prop.afqmc import afqmc_step, init_prop_state
from ad_afqmc_prototype_gb300.prop.blocks import afqmc_block
from ad_afqmc_prototype_gb300.prop.chol_afqmc_ops import make_chol_afqmc_ops
from ad_afqmc_prototype_gb300.prop.types import afqmc_params
from ad_afqmc_prototype_gb300.trial.rhf import get_rdm1, make_rhf_trial_ops, rhf_trial

F64, C128 = torch.float64, torch.complex128


def _case(name, op, n, o, g, w, precision="fp64", kind="restricted", steps=1, qr=0, blocks=1):
    return {"name": name, "op": op, "norb": n, "nocc": o, "nchol": g, "walkers": w, "precision": precision,
            "kind": kind, "steps": steps, "qr_every": qr, "blocks": blocks}


def listed():
    return [
        # a small molecule's block: 12 orbitals, 256 walkers, ten steps, QR every five; latency and launches
        _case("block_fp64_n12", "block", 12, 6, 48, 256, steps=10, qr=5),
        # the driver with its default 200 walkers and 50 steps a block (graph-replayed), default precision
        _case("driver_fp64_n30", "driver", 30, 7, 150, 200, steps=50, blocks=2),
        # unrestricted walkers (the only form they have is binary64), odd sizes
        _case("block_unrestricted_n61", "block", 61, 9, 301, 203, kind="unrestricted", steps=5),
        # one step at the 120-orbital workload, default precision
        _case("step_fp64_n120", "step", 120, 20, 600, 2048),
        # one step at the 200-orbital benchmark Hamiltonian with a quarter of its walkers, default precision
        _case("step_fp64_n200", "step", 200, 30, 1000, 1024),
        # the largest Hamiltonian of the workloads, few walkers, default precision
        _case("step_fp64_n400", "step", 400, 50, 2000, 128),
        # the measurement: local energies of a population, default precision
        _case("energy_fp64_n120", "energy", 120, 20, 600, 512),
        # the population's phase-fixed QR at the benchmark shape
        _case("qr_fp64_n200", "qr", 200, 30, 1, 4096),
        # dE/dh1: a differentiated run, forward and backward
        _case("gradient_fp64_n60", "gradient", 60, 10, 300, 256, steps=5, blocks=2),
        # the six-section mixed form, one step at the 120-orbital workload
        _case("step_mixed_n120", "step", 120, 20, 600, 2048, precision="mixed"),
        # the three-section form at odd sizes between the workloads
        _case("block_mixed_fast_n75", "block", 75, 13, 411, 777, precision="mixed_fast", steps=10, qr=5),
        # the benchmark block: 200 orbitals, 4096 walkers, ten steps, QR every five
        _case("block_mixed_fast_n200", "block", 200, 30, 1000, 4096, precision="mixed_fast", steps=10, qr=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _energy_fits(o, g):
    """The binary64 energy takes every nocc >= 7; below that only few Cholesky vectors fit its shared memory."""
    ng = min(g, max(1, 4096 // (o * o)))
    return 16 * (32 * o + 16 * ng * o + ng * o * o) <= 227 * 1024


def draw(rng):
    """A case of the same ranges: 8-400 orbitals, G = 3 n to 6 n, 8-4096 walkers, every form."""
    op, precision, kind = rng.choice([
        ("block", "fp64", "restricted"), ("driver", "fp64", "restricted"), ("block", "fp64", "unrestricted"),
        ("step", "fp64", "restricted"), ("step", "fp64", "restricted"), ("energy", "fp64", "restricted"),
        ("qr", "fp64", "restricted"), ("gradient", "fp64", "restricted"), ("step", "mixed", "restricted"),
        ("block", "mixed_fast", "restricted"), ("step", "mixed_fast", "restricted")])
    hi = {"gradient": 120, "driver": 120, "qr": 256}.get(op, 400)
    n = _log_int(rng, 12 if op == "gradient" else 8, hi)
    if precision != "fp64":
        n = max(n, 24)
    o = max(1, min(50, int(n * rng.uniform(0.1, 0.35))))
    if precision != "fp64" or op in ("gradient", "qr"):
        o = min(o, 32)
    g = 1 if op == "qr" else int(n * rng.uniform(3.0, 6.0))
    while not _energy_fits(o, g):
        o += 1
    steps = {"block": rng.choice([3, 5, 10]), "driver": rng.choice([10, 20, 50]), "gradient": rng.choice([2, 5])}.get(op, 1)
    blocks = {"driver": rng.choice([1, 2, 3]), "gradient": rng.choice([1, 2])}.get(op, 1)
    c = _case("", op, n, o, g, 1, precision, kind, steps, rng.choice([0, 5]) if op == "block" else 0, blocks)
    del c["name"]
    # binary64 passes up to 0.2 Tflop, the tensor-core forms up to 4 Tflop (the largest listed ones take more)
    per_walker = work(c)["flops"]
    top = 4e12 if precision != "fp64" else 2e11
    w_max = max(8, min(4096, int(top / per_walker)))
    c["walkers"] = _log_int(rng, 8, w_max)
    return c


# ----------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) % (2**62))


def _sym(b):
    return 0.5 * (b + b.transpose(-1, -2))


def _inputs(case, seed):
    """Hamiltonian, trial orbitals, walkers near the trial, weights and fields, all from the seed."""
    n, o, G, W = case["norb"], case["nocc"], case["nchol"], case["walkers"]
    gen = _gen(seed)
    rn = lambda *s: torch.randn(s, generator=gen, device="cuda", dtype=F64)  # noqa: E731
    off = _sym(0.1 * rn(n, n))
    h1 = torch.diag(torch.linspace(-2.0, 0.5, n, dtype=F64, device="cuda")) + off - torch.diag(torch.diag(off))
    chol = _sym(rn(G, n, n))
    chol *= (0.3 * 12.0 / n * torch.exp(-torch.arange(G, dtype=F64, device="cuda") * (4.0 / G)))[:, None, None]
    mo = torch.linalg.eigh(h1)[1][:, :o].contiguous()
    noise = 0.2 / math.sqrt(n)
    spins = 2 if case["kind"] == "unrestricted" else 1
    w = torch.complex(mo.expand(spins, W, n, o) + noise * rn(spins, W, n, o), noise * rn(spins, W, n, o))
    weights = 1.0 + 0.2 * torch.rand((W,), generator=gen, device="cuda", dtype=F64)
    fields = rn(W, G) if case["op"] == "step" else None
    return {"h1": h1, "chol": chol, "mo": mo, "w": w if spins == 2 else w[0], "weights": weights, "fields": fields}


def _params(case, seed):
    return afqmc_params(n_walkers=case["walkers"], n_prop_steps=case["steps"], qr_every=case["qr_every"],
                        precision=case["precision"], seed=int(seed) % 1000003)


def prepare(case, seed):
    x = _inputs(case, seed)
    if case["op"] == "qr":
        return {"case": case, "w": x["w"]}
    n, o, W = case["norb"], case["nocc"], case["walkers"]
    sys_ = system(norb=n, nelec=(o, o), walker_kind=case["kind"])
    params = _params(case, seed)
    ham = ham_chol(h0=0.0, h1=x["h1"], chol=x["chol"])
    trial = rhf_trial(x["mo"])
    t_ops, m_ops = make_rhf_trial_ops(sys_), make_rhf_meas_ops(sys_)
    p_ops = make_chol_afqmc_ops(ham, case["kind"])
    meas_ctx = m_ops.build_meas_ctx(ham, trial)
    kw = dict(params=params, ham_data=ham, trial_data=trial, meas_ops=m_ops, prop_ops=p_ops,
              prop_ctx=p_ops.build_prop_ctx(get_rdm1(trial), params.dt), meas_ctx=meas_ctx)
    walkers = (x["w"][0], x["w"][1]) if case["kind"] == "unrestricted" else x["w"]
    few = (walkers[0][:8], walkers[1][:8]) if case["kind"] == "unrestricted" else walkers[:8]
    e_est = m_ops.require_kernel(k_energy).batched(few, ham, meas_ctx, trial).real.mean()
    state = init_prop_state(sys=sys_, n_walkers=W, seed=params.seed, ham_data=ham, trial_ops_=t_ops, trial_data=trial,
                            meas_ops=m_ops, initial_walkers=walkers, initial_e_estimate=e_est)
    state = state._replace(weights=x["weights"])
    s = {"case": case, "state": state, "kw": kw, "sys": sys_, "fields": x["fields"]}
    if case["op"] == "driver":
        kwd = dict(kw, sys=sys_)
        s["run_blocks"] = make_run_blocks(lambda st: afqmc_block(st, **kwd), kwd)
    return s


def _state_out(st):
    w = st.walkers
    return {"walkers": list(w) if isinstance(w, (tuple, list)) else w, "weights": st.weights, "overlaps": st.overlaps,
            "shift": st.pop_control_ene_shift, "e_estimate": st.e_estimate}


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "qr":
        q, det = wk.orthogonalize(s["w"], "restricted")
        return {"q": q, "det": det}
    kw = s["kw"]
    if op == "step":
        return _state_out(afqmc_step(s["state"], fields=s["fields"], **kw))
    if op == "block":
        new, obs = afqmc_block(s["state"], sys=s["sys"], **kw)
        return dict(_state_out(new), **obs.scalars)
    if op == "driver":
        new, e, w = s["run_blocks"](s["state"], n_blocks=case["blocks"])
        return dict(_state_out(new), energies=e, block_weights=w)
    if op == "energy":
        return {"energy": wk.apply_chunked(s["state"].walkers, kw["meas_ops"].require_kernel(k_energy), 1,
                                           kw["ham_data"], kw["meas_ctx"], kw["trial_data"])}
    if op == "gradient":
        h1 = kw["ham_data"].h1.detach().requires_grad_(True)
        e, w = block_energies(h1, ham_data=kw["ham_data"], trial_data=kw["trial_data"], params=kw["params"],
                              state=s["state"], n_blocks=case["blocks"])
        ((w * e).sum() / w.sum()).backward()
        return {"energies": e.detach(), "weights": w.detach(), "h1_grad": h1.grad}
    raise ValueError(f"unknown op {op!r}")


def work(case):
    """Real flops and bytes of one pass: V-build 4 G n^2, Taylor and E_half 56 n^2 o, force bias 4 G o n,
    overlap and Green's function 12 n o^2 a step and walker; exchange 4 G o^2 n and QR 16 n o^2 a measurement."""
    n, o, G, W = case["norb"], case["nocc"], case["nchol"], case["walkers"]
    spins = 2 if case["kind"] == "unrestricted" else 1
    step = 4.0 * G * n * n + spins * (56.0 * n * n * o + 4.0 * G * o * n + 12.0 * n * o * o)
    meas = spins * (4.0 * G * o * o * n + 28.0 * n * o * o)
    walkers = 16.0 * W * spins * n * o
    ham = 8.0 * G * n * n + 8.0 * G * n * o
    op = case["op"]
    if op == "qr":
        return {"bytes": 2 * walkers, "flops": 16.0 * W * n * o * o}
    if op == "energy":
        return {"bytes": walkers + 8.0 * G * n * o, "flops": W * (4.0 * G * o * o * n + 12.0 * n * o * o)}
    if op == "step":
        return {"bytes": 2 * walkers + ham + 8.0 * W * G, "flops": W * step}
    run_ = case["blocks"] * (case["steps"] * step + meas) * W
    return {"bytes": 2 * walkers + ham, "flops": run_ * (3.0 if op == "gradient" else 1.0)}


# --------------------------------------------------- 64-bit values by torch
def _overlap_green(w, c):
    m = c.transpose(0, 1) @ w  # (W, o, o)
    g = torch.linalg.solve(m.transpose(1, 2), w.transpose(1, 2))  # (W, o, n)
    return torch.linalg.det(m) ** 2, g


def _exact_qr(w):
    q, r = torch.linalg.qr(w)
    d = torch.diagonal(r, dim1=1, dim2=2)
    ph = d / d.abs()
    return {"q": q * ph[:, None, :], "det": torch.prod(d.abs(), 1).to(C128) ** 2}


def _exact_energy(x, case):
    c, W, o = x["mo"].to(C128), case["walkers"], case["nocc"]
    _, g = _overlap_green(x["w"], c)
    rot_h1 = (x["mo"].T @ x["h1"]).to(C128)
    rot = torch.matmul(x["mo"].T, x["chol"])  # (G, o, n)
    e1 = 2.0 * (rot_h1 * g).sum((1, 2))
    e2 = torch.zeros((W,), dtype=C128, device="cuda")
    per = max(1, int(2e8 // (W * o * o)))
    for a in range(0, rot.shape[0], per):
        r = rot[a:a + per]
        f = torch.complex(torch.einsum("gin,wjn->wgij", r, g.real), torch.einsum("gin,wjn->wgij", r, g.imag))
        tr = torch.diagonal(f, dim1=2, dim2=3).sum(2)
        e2 += 2.0 * (tr * tr).sum(1) - (f * f.transpose(2, 3)).sum((1, 2, 3))
    return {"energy": e1 + e2}


def _exact_step(x, case, seed):
    p = _params(case, seed)
    n, G, W, dt = case["norb"], case["nchol"], case["walkers"], p.dt
    sq = math.sqrt(dt)
    c, w, L = x["mo"].to(C128), x["w"], x["chol"]
    rot = torch.matmul(x["mo"].T, L).reshape(G, -1)
    rdm = 2.0 * (x["mo"] @ x["mo"].T)
    mf = 1j * (L.reshape(G, -1) @ rdm.reshape(-1)).to(C128)
    h0p = -0.5 * (mf * mf).sum()
    v0 = 0.5 * (L.transpose(1, 2) @ L).sum(0)
    v1 = torch.tensordot((1j * mf).real, L, dims=1)
    e_half = torch.linalg.matrix_exp(-0.5 * dt * (x["h1"] - v0 - v1)).to(C128)
    ov, g = _overlap_green(w, c)
    gf = g.reshape(W, -1)
    fb = 2.0 * torch.complex(gf.real @ rot.T, gf.imag @ rot.T)
    fs = -sq * (1j * fb - mf)
    xs = x["fields"] - fs
    shift = (xs * mf).sum(1)
    fbt = (x["fields"] * fs - 0.5 * fs * fs).sum(1)
    out = torch.empty_like(w)
    per = max(1, int(1e8 // (n * n)))
    Lf = L.reshape(G, -1)
    for a in range(0, W, per):
        xa = xs[a:a + per]
        V = torch.complex(xa.real @ Lf, xa.imag @ Lf).reshape(-1, n, n)
        t = e_half @ w[a:a + per]
        acc = t.clone()
        for k in range(1, p.n_exp_terms + 1):
            t = (1j * sq / k) * (V @ t)
            acc += t
        out[a:a + per] = e_half @ acc
    ov_new = _overlap_green(out, c)[0]
    return out, ov, ov_new, shift, fbt, h0p


def exact(case, seed):
    """Restricted steps, energies and QRs in 64 bits by torch.  Whole blocks, driver runs and gradients draw
    from the engine's own stream, so they have no value without it."""
    op = case["op"]
    if op not in ("step", "energy", "qr"):
        return None
    x = _inputs(case, seed)
    if op == "qr":
        return _exact_qr(x["w"])
    if op == "energy":
        return _exact_energy(x, case)
    p = _params(case, seed)
    out, ov, ov_new, shift, fbt, h0p = _exact_step(x, case, seed)
    # e_estimate and the population shift start as the mean energy of the first eight walkers
    few = dict(case, walkers=min(8, case["walkers"]))
    e0 = _exact_energy(dict(x, w=x["w"][:8]), few)["energy"].real.mean()
    ratio = ov_new / ov
    sq, dt = math.sqrt(p.dt), p.dt
    imp = torch.exp(-sq * shift + fbt + dt * (e0 + h0p)) * ratio
    theta = torch.angle(torch.exp(-sq * shift) * ratio)
    ph = imp.abs() * torch.cos(theta)
    ph = torch.where(torch.isnan(ph) | (ph < p.weight_floor) | (ph > p.weight_cap), torch.zeros_like(ph), ph)
    weights = x["weights"] * ph
    weights = torch.where(weights > p.weight_cap, torch.zeros_like(weights), weights)
    shift_new = e0 - p.pop_control_damping * torch.log(weights.mean()) / dt
    return {"walkers": out, "weights": weights, "overlaps": ov_new, "shift": shift_new, "e_estimate": e0}
