"""What a user of this framework has it do, as cases that can be timed and checked.

Each case is one of these uses, through the package's public entry points:

* ``pass``     one nonlocal ladder pass, ``LadderPass.run`` on resident inputs, or ``run_e2e`` (host G(k) in, host
               Sigma out) where ``host`` is set, as a self-consistency loop calls it; ``mixed`` chooses the precision
* ``pair``     two passes of different orbital counts replayed as one CUDA graph (``serving.BatchedPasses``)
* ``pairing``  an FP64 pass that also writes the pairing box, and the gap-equation operators built from it
               (``EliashbergSolver``), the end of a calculation
* ``gap``      one application of both channels' gap-equation operators, the inner step of every eigen-solve
* ``local``    the local Schwinger-Dyson equation of one atom (``LocalSde``), the start of a calculation
* ``dense``    the FourPoint inversion summed over the last frequency, for a program that holds the matrix itself

Inputs come from a model with the value ranges of a Hubbard or t2g calculation (square-lattice dispersion, Hubbard-I
self-energy, an irreducible vertex of U plus a smooth frequency structure plus 1e-3 seeded noise), made on the GPU.
"""

import math

import numpy as np
import torch

from dgamore_b200 import four_point
from dgamore_b200.eliashberg_solver import EliashbergSolver
from dgamore_b200.local_sde import LocalSde
from dgamore_b200.pipeline import LadderPass
from dgamore_b200.serving import BatchedPasses

C128 = torch.complex128

# Hubbard, bilayer Hubbard and t2g square lattices: interaction, hoppings, temperature and filling
MODELS = {
    1: {"u": 8.0, "j": 0.0, "t": (1.0,), "tp": -0.25, "t_perp": 0.0, "n": 0.85, "beta": 12.5},
    2: {"u": 6.0, "j": 0.0, "t": (1.0, 1.0), "tp": 0.0, "t_perp": 0.8, "n": 1.8, "beta": 15.0},
    3: {"u": 2.3, "j": 0.4, "t": (0.5, 0.5, 0.1), "tp": 0.0, "t_perp": 0.0, "n": 1.0, "beta": 20.0},
}


def listed():
    return [
        # the plain one-band calculation on a small grid: about a dozen short launches, so latency counts
        {"name": "one_band_16_fp64", "use": "pass", "orb": 1, "nk": 16, "niw": 20, "niv": 20, "shell": 0, "mixed": False, "host": False},
        # a small two-orbital request as a self-consistency loop runs it: odd grid and box, shell frequencies, G(k)
        # from the host and Sigma back to it
        {"name": "bilayer_9_host_mixed", "use": "pass", "orb": 2, "nk": 9, "niw": 10, "niv": 9, "shell": 3, "mixed": True, "host": True},
        # the one-band calculation at scale: tens of thousands of small solves (N = 120), in both precisions
        {"name": "one_band_64_fp64", "use": "pass", "orb": 1, "nk": 64, "niw": 60, "niv": 60, "shell": 0, "mixed": False, "host": False},
        {"name": "one_band_64_mixed", "use": "pass", "orb": 1, "nk": 64, "niw": 60, "niv": 60, "shell": 0, "mixed": True, "host": False},
        # the three-orbital calculation (N = 720), the framework's headline workload, in both precisions
        {"name": "t2g_32_mixed", "use": "pass", "orb": 3, "nk": 32, "niw": 40, "niv": 40, "shell": 0, "mixed": True, "host": False},
        {"name": "t2g_32_fp64", "use": "pass", "orb": 3, "nk": 32, "niw": 40, "niv": 40, "shell": 0, "mixed": False, "host": False},
        # serving: a bilayer and a one-band request of different sizes as one graph
        {"name": "pair_48_32_mixed", "use": "pair", "orb": 2, "nk": 48, "niw": 30, "niv": 30, "shell": 0, "mixed": True, "nk1": 32, "niv1": 50},
        # superconductivity: the pass with the pairing vertex, and the operator that an eigen-solve applies
        {"name": "bilayer_48_pairing", "use": "pairing", "orb": 2, "nk": 48, "niw": 30, "niv": 30, "shell": 0, "mixed": False},
        {"name": "bilayer_48_gap", "use": "gap", "orb": 2, "nk": 48, "niw": 30, "niv": 30, "shell": 0, "mixed": False},
        # the local equation: the three-orbital box, and a one-band box with shell frequencies
        {"name": "local_t2g", "use": "local", "orb": 3, "niw": 40, "niv": 40, "shell": 0},
        {"name": "local_one_band", "use": "local", "orb": 1, "niw": 20, "niv": 20, "shell": 10},
        # a program that brings its own FourPoint matrices: two orbitals, a box that is no multiple of 32
        {"name": "dense_bilayer", "use": "dense", "orb": 2, "nq": 21, "niw": 20, "niv": 25},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _solves(c):
    """(number of compound solves, compound size) of a case's BSE."""
    n2 = c["orb"] ** 2
    nq = c["nq"] if "nq" in c else 1 if c["use"] == "local" else (c["nk"] // 2 + 1) * (c["nk"] // 2 + 2) // 2
    return (2 if c["use"] != "dense" else 1) * nq * (c["niw"] + 1), n2 * 2 * c["niv"]


def _cost(c):
    """Seconds of the case's solves at 10 TFLOP/s, a bound to keep drawn cases below the largest listed one."""
    items, n = _solves(c)
    rhs = c["orb"] ** 2
    if c["use"] == "local":
        rhs = 4 * n
    if c["use"] in ("pairing", "gap"):
        rhs = rhs * (1 + min(c["niw"] // 2, c["niv"] // 2))
    return items * (8 / 3 * n**3 + 8 * rhs * n**2) / 10e12


def draw(rng):
    while True:
        use = rng.choice(("pass", "pass", "pass", "pass", "pair", "pairing", "gap", "local", "dense"))
        orb = rng.choice((1, 2, 3))
        c = {"use": use, "orb": orb}
        top = {1: 60, 2: 40, 3: 40}[orb]
        if use == "dense":
            c |= {"nq": _log(rng, 2, 64), "niw": _log(rng, 2, 30), "niv": _log(rng, 4, top)}
            size = _solves(c)[0] * _solves(c)[1] ** 2 * 16
            if size > 2 << 30:
                continue
        elif use == "local":
            c |= {"niw": _log(rng, 4, top), "niv": _log(rng, 4, top), "shell": rng.choice((0, 0, 3, 10))}
        else:
            c |= {"nk": _log(rng, 8, 64), "niw": _log(rng, 6, top), "niv": _log(rng, 6, top), "shell": rng.choice((0, 0, 2, 5)), "mixed": rng.random() < 0.5}
            if use == "pair":
                c |= {"orb": rng.choice((2, 3)), "shell": 0, "nk1": _log(rng, 8, 48), "niv1": _log(rng, 8, 60)}
            if use in ("pairing", "gap"):
                c |= {"nk": min(c["nk"], 48), "shell": 0}
                box = c["orb"] ** 2 * 2 * min(c["niw"] // 2, c["niv"] // 2)
                if box > 160 or c["nk"] ** 2 * box**2 > 2304 * 120**2:
                    continue
            if use == "pairing":
                c["mixed"] = False
            if use == "pass":
                c["host"] = rng.random() < 0.25
            if c["orb"] == 3 and c["nk"] > 32:
                continue
        if _cost(c) < 0.7:
            return c


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _interaction(m, n):
    u = np.zeros((n,) * 4, dtype=np.complex128)
    for a in range(n):
        for b in range(n):
            u[a, b, a, b] = m["u"] - 2 * m["j"]
            u[a, b, b, a] = u[a, a, b, b] = m["j"]
    for a in range(n):
        u[a, a, a, a] = m["u"]
    return u


def _channel(u, ch):
    x = np.einsum("abcd->adcb", u)
    return 2 * u - x if ch == "dens" else -x


def _orbmat(x):
    """[..., a, b, c, d] -> [..., (a,b), (d,c)]."""
    n = x.shape[-1]
    return x.swapaxes(-1, -2).reshape(*x.shape[:-4], n * n, n * n)


def _wedge(nk):
    """Irreducible points of the square lattice's nk x nk grid: indices, map of every point, counts."""
    i = np.arange(nk)
    r = np.minimum(i, (-i) % nk)
    lo, hi = np.minimum(r[:, None], r[None, :]), np.maximum(r[:, None], r[None, :])
    _, ind, inv, count = np.unique(lo * nk + hi, return_index=True, return_inverse=True, return_counts=True)
    return ind, inv.reshape(-1), count


def _bands(m, n, nk):
    k = 2 * np.pi * np.arange(nk) / nk
    c = np.cos(k)[:, None] + np.cos(k)[None, :]
    e = np.zeros((nk, nk, n, n), dtype=np.complex128)
    for a in range(n):
        e[..., a, a] = -2 * m["t"][a] * c - 4 * m["tp"] * np.cos(k)[:, None] * np.cos(k)[None, :]
    if m["t_perp"]:
        e[..., 0, 1] = e[..., 1, 0] = -m["t_perp"]
    return torch.from_numpy(e.reshape(nk * nk, n, n)).cuda()


def _green(m, n, e, mu, niv):
    """G(k, nu) [Nk, n, n, 2 niv] with the Hubbard-I self-energy."""
    ns = m["n"] / (2 * n)
    iv = 1j * torch.pi / m["beta"] * (2 * torch.arange(-niv, niv, device="cuda", dtype=torch.float64) + 1)
    s = m["u"] * ns + m["u"] ** 2 * ns * (1 - ns) / (iv + mu - m["u"] * (1 - ns))
    a = (iv + mu - s)[:, None, None] * torch.eye(n, device="cuda") - e[:, None]
    return torch.linalg.inv(a).permute(0, 2, 3, 1)


def _chemical_potential(m, n):
    e = _bands(m, n, 12)
    lo, hi = -4 * m["u"] - 10, 4 * m["u"] + 10
    for _ in range(30):
        mu = 0.5 * (lo + hi)
        g = _green(m, n, e, mu, 48).mean(0)
        fill = float(2 * (0.5 + torch.diagonal(g).sum(0).real / m["beta"]).sum())
        lo, hi = (mu, hi) if fill < m["n"] else (lo, mu)
    return 0.5 * (lo + hi)


def _vertex(m, u, ch, niw, niv, gen):
    """Irreducible vertex [a,b,c,d,w >= 0,nu,nu'] with the nu <-> nu' and w = 0 symmetries."""
    n, beta, scale = u.shape[0], m["beta"], m["u"]
    u_r = _channel(u, ch)
    mat = _orbmat(u_r)
    shape = (mat @ mat / scale).reshape((n,) * 4).swapaxes(2, 3)
    nu = math.pi / beta * (2 * torch.arange(-niv, niv, device="cuda", dtype=torch.float64) + 1)
    om = 2 * math.pi / beta * torch.arange(niw + 1, device="cuda", dtype=torch.float64)
    d1 = (nu[:, None] - nu[None, :]) / scale
    d2 = (nu[:, None] + nu[None, :] + om[:, None, None]) / scale
    w = 1 / (1 + d1**2) + 0.5 / (1 + d2**2)
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    g = up(u_r)[..., None, None, None] + (0.3 if ch == "dens" else -0.3) * up(shape)[..., None, None, None] * w
    noise = torch.randn((*g.shape, 2), generator=gen, device="cuda", dtype=torch.float64)
    g = g + 1e-3 * scale * torch.view_as_complex(noise)
    g = 0.5 * (g + g.permute(2, 3, 0, 1, 4, 6, 5))
    g0 = g[..., 0, :, :].clone()
    g[..., 0, :, :] = 0.5 * (g0 + g0.flip((-1, -2)).conj())
    return g


def _local_bubble(g, niw, niv, beta):
    """chi0 [w, nu, (a,b), (d,c)] = -beta G_ad(nu) G_cb(nu - w), w >= 0."""
    n, mid = g.shape[0], g.shape[-1] // 2
    left = g[..., mid - niv : mid + niv]
    out = []
    for w in range(niw + 1):
        right = g[..., mid - niv - w : mid + niv - w]
        x = -beta * torch.einsum("adv,cbv->vabdc", left, right)
        out.append(x.reshape(2 * niv, n * n, n * n))
    return torch.stack(out)


def _compound(x):
    """[a,b,c,d,w,nu,nu'] -> [w, (a,b,nu), (d,c,nu')]."""
    n, w, v = x.shape[0], x.shape[4], x.shape[5]
    return x.permute(4, 0, 1, 5, 3, 2, 6).reshape(w, n * n * v, n * n * v)


def _four(x, n):
    """[w, (a,b,nu), (d,c,nu')] -> [a,b,c,d,w,nu,nu']."""
    w, v = x.shape[0], x.shape[1] // (n * n)
    return x.reshape(w, n, n, v, n, n, v).permute(1, 2, 5, 4, 0, 3, 6)


def _block_diag(c):
    """[..., nu, p, s] -> [..., (p,nu), (s,nu)], block diagonal in nu."""
    v, p = c.shape[-3], c.shape[-1]
    out = torch.zeros((*c.shape[:-3], p, v, p, v), dtype=c.dtype, device=c.device)
    i = torch.arange(v, device=c.device)
    out[..., :, i, :, i] = torch.movedim(c, -3, 0)
    return out.reshape(*c.shape[:-3], p * v, p * v)


def _local_ladder(c0, gamma, u_r, beta, with_f):
    """Local chi_r(w) [w,(a,b),(d,c)] and, where asked for, F_r [w, N, N] from the local bubble and vertex."""
    w, v, p = c0.shape[:3]
    c0i = torch.linalg.inv(c0)
    um = torch.from_numpy(np.ascontiguousarray(_orbmat(u_r))).cuda()
    chi_r, f = [], []
    for i in range(w):
        d = _block_diag(c0i[i])
        a = d + (_compound(gamma[..., i : i + 1, :, :])[0].reshape(p, v, p, v) - um[:, None, :, None]).reshape(p * v, p * v) / beta**2
        chi = torch.linalg.inv(a)
        aux = chi.reshape(p, v, p, v).sum((1, 3)) / beta**2
        chi_r.append(torch.linalg.inv(torch.linalg.inv(aux) + um))
        if with_f:
            f.append(beta**2 * (d - d @ chi @ d))
    return torch.stack(chi_r), torch.stack(f) if with_f else None


def _pass_inputs(c, seed):
    """The inputs of one nonlocal pass: G(k) and the interaction on the host, the vertices on the GPU."""
    orb, nk, niw, niv, shell = c["orb"], c["nk"], c["niw"], c["niv"], c["shell"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    m = dict(MODELS[orb])
    m["n"] *= 1 + 0.02 * (float(torch.rand(1, generator=gen, device="cuda")) - 0.5)
    beta, full = m["beta"], niv + shell
    ind, inv, count = _wedge(nk)
    u = _interaction(m, orb)
    e = _bands(m, orb, nk)
    g = _green(m, orb, e, _chemical_potential(m, orb), full + niw + 10)
    out = {
        "beta": beta, "niw": niw, "niv_core": niv, "niv_shell": shell, "nk": (nk, nk, 1), "irrk_ind": ind, "irrk_inv": inv,
        "irrk_count": count, "u": u, "v_q_irr": np.zeros((len(ind),) + (orb,) * 4, dtype=np.complex128),
        "g_k": g.reshape(nk, nk, 1, orb, orb, -1).cpu().numpy(),
    }
    c0 = _local_bubble(g.mean(0), niw, full, beta)
    core = c0[:, shell : shell + 2 * niv]
    for ch in ("dens", "magn"):
        gamma = _vertex(m, u, ch, niw, niv, gen)
        u_r = _channel(u, ch)
        out["gamma_" + ch] = gamma
        if orb == 1:
            s = _local_ladder(core, gamma, u_r, beta, False)[0].reshape(-1)
            if float((s[0] + 2 * s[1:].real.sum()).real) <= 0:  # past the model's instability: the bubble's sum
                s = core.sum(1).reshape(-1) / beta**2
            out["chi_loc_sum_" + ch] = complex((s.sum() + s[1:].conj().sum()) / beta)
        if ch == "magn":
            pad = torch.from_numpy(u_r).cuda()[..., None, None, None].expand(*gamma.shape[:5], 2 * full, 2 * full).clone()
            pad[..., shell : shell + 2 * niv, shell : shell + 2 * niv] = gamma
            f = _four(_local_ladder(c0, pad, u_r, beta, True)[1], orb)
            out["f_dc"] = 2 * f.permute(2, 1, 0, 3, 4, 5, 6)
    return out


def _local_inputs(c, seed):
    """g, G2 of both channels (w >= 0), u, beta and occupations of the local equation."""
    orb, niw, niv, shell = c["orb"], c["niw"], c["niv"], c["shell"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    m = dict(MODELS[orb])
    m["n"] *= 1 + 0.02 * (float(torch.rand(1, generator=gen, device="cuda")) - 0.5)
    beta, p = m["beta"], orb * orb
    u = _interaction(m, orb)
    g = _green(m, orb, _bands(m, orb, 8), _chemical_potential(m, orb), niv + shell + niw + 4).mean(0)
    c0 = _local_bubble(g, niw, niv + shell, beta)
    g2 = []
    for ch in ("dens", "magn"):
        u_r = _channel(u, ch)
        um = torch.from_numpy(np.ascontiguousarray(_orbmat(u_r))).cuda()
        tilde = _shell_bubble_inverse(c0, um, beta, niv, shell)
        gamma = _compound(_vertex(m, u, ch, niw, niv, gen))
        gm = (gamma.reshape(-1, p, 2 * niv, p, 2 * niv) - um[:, None, :, None]).reshape(gamma.shape)
        x = _four(torch.linalg.inv(tilde + gm / beta**2), orb) / beta
        if ch == "dens":
            gs = g[..., g.shape[-1] // 2 - niv : g.shape[-1] // 2 + niv]
            x[:, :, :, :, 0] += 2 * gs[:, :, None, None, :, None] * gs[None, None, :, :, None, :]
        g2.append(x.contiguous())
    occ = np.diag([m["n"] / (2 * orb)] * orb).astype(np.complex128)
    return g.contiguous(), g2[0], g2[1], u, beta, occ


def _shell_bubble_inverse(c0, um, beta, niv, shell):
    """[(chi0^-1 + U/beta^2 over the full box)^-1 cut to the core]^-1, [w, N, N]."""
    w, v, p = c0.shape[:3]
    if not shell:
        a = _block_diag(torch.linalg.inv(c0)).reshape(w, p, v, p, v)
        return (a + um[:, None, :, None] / beta**2).reshape(w, p * v, p * v)
    out = []
    for i in range(w):
        a = _block_diag(torch.linalg.inv(c0[i])).reshape(p, v, p, v) + um[:, None, :, None] / beta**2
        a = torch.linalg.inv(a.reshape(p * v, p * v)).reshape(p, v, p, v)[:, shell : shell + 2 * niv, :, shell : shell + 2 * niv]
        out.append(torch.linalg.inv(a.reshape(p * 2 * niv, -1)))
    return torch.stack(out)


def _dense_inputs(c, seed):
    """FourPoint matrices [q,a,b,c,d,w,nu,nu'] of chi0^-1 + (Gamma - U)/beta^2 with a q-dependent bubble."""
    orb, nq, niw, niv = c["orb"], c["nq"], c["niw"], c["niv"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    m = MODELS[orb]
    u = _interaction(m, orb)
    g = _green(m, orb, _bands(m, orb, 8), _chemical_potential(m, orb), niv + niw + 4).mean(0)
    c0i = torch.linalg.inv(_local_bubble(g, niw, niv, m["beta"]))
    ladder = _vertex(m, u, "magn", niw, niv, gen) - torch.from_numpy(_channel(u, "magn")).cuda()[..., None, None, None]
    x = torch.empty((nq, *ladder.shape), dtype=C128, device="cuda")
    for q in range(nq):
        a = _block_diag(c0i * (1 + 0.4 * math.cos(math.pi * q / nq) * float(torch.rand(1, generator=gen, device="cuda"))))
        x[q] = _four(a, orb) + ladder / m["beta"] ** 2
    return x, m["beta"]


# ------------------------------------------------------------------------------------------------
# preparing and running
# ------------------------------------------------------------------------------------------------
def _one_band(c):
    return {"use": "pass", "orb": 1, "nk": c["nk1"], "niw": c["niv1"], "niv": c["niv1"], "shell": 0}


def _gap_vectors(dim, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    x = torch.randn((2, dim, 2), generator=gen, device="cuda", dtype=torch.float64)
    x = torch.view_as_complex(x)
    return x / torch.linalg.vector_norm(x, dim=1, keepdim=True)


def prepare(case, seed):
    use = case["use"]
    if use == "dense":
        x, beta = _dense_inputs(case, seed)
        return {"use": use, "x": x, "beta": beta}
    if use == "local":
        g, d, m, u, beta, occ = _local_inputs(case, seed)
        return {"use": use, "sde": LocalSde(g, d, m, u, beta, case["niw"], case["niv"], case["shell"], occ)}
    precision = "mixed" if case["mixed"] else "fp64"
    if use == "pass":
        lp = LadderPass(_pass_inputs(case, seed), precision=precision, keep_intermediates=False)
        return {"use": use, "lp": lp, "host": case["host"]}
    if use == "pair":
        lps = [LadderPass(_pass_inputs(c, seed), precision=precision, keep_intermediates=False, own_bse_scratch=False)
               for c in (case, _one_band(case))]
        both = BatchedPasses(lps, precision)
        both.capture()
        return {"use": use, "lps": lps, "both": both}
    box = min(case["niw"] // 2, case["niv"] // 2)
    lp = LadderPass(_pass_inputs(case, seed), eliashberg_pp=box)
    if use == "pairing":
        return {"use": use, "lp": lp, "box": box}
    lp.run()
    es = EliashbergSolver(lp, box, precision=precision)
    return {"use": use, "es": es, "x": _gap_vectors(es.dim, seed)}


def _pass_outputs(lp):
    if lp.do_lambda:
        return {"sigma": lp.sigma, "chi": lp.chi_lam, "lambdas": lp.lambdas}
    return {"sigma": lp.sigma, "chi": lp.chi_phys}


def run(state):
    use = state["use"]
    if use == "dense":
        return four_point.invert_and_sum_over_last_vn(state["x"], state["beta"], return_device=True)
    if use == "local":
        s = state["sde"].run()
        return {"gamma": [s.gamma(0), s.gamma(1)], "f_dc": s.f_dc(), "chi": [s.chi(0), s.chi(1)], "vrg": [s.vrg_r(0), s.vrg_r(1)],
                "sigma": s.sigma_loc()}
    if use == "pass":
        lp = state["lp"]
        if state["host"]:
            return {"sigma": lp.run_e2e()}
        lp.run()
        return _pass_outputs(lp)
    if use == "pair":
        state["both"].replay()
        return [_pass_outputs(lp) for lp in state["lps"]]
    if use == "pairing":
        lp = state["lp"]
        lp.run()
        es = EliashbergSolver(lp, state["box"])
        return {"sigma": lp.sigma, "vertex": es.gamma_pp_irr, "operators": es.mat, "bubble": es.chi0pp}
    es, x = state["es"], state["x"]
    return {"sing": es.matvec("sing", x[0]), "trip": es.matvec("trip", x[1])}


# ------------------------------------------------------------------------------------------------
# work
# ------------------------------------------------------------------------------------------------
def _pass_work(c, box=0):
    """The G(k), vertices and F of a pass read once and Sigma written; its solves, the double-counting product, the
    bubble and the Sigma sums through fast transforms."""
    n, nk, niw, niv, full = c["orb"], c["nk"] ** 2, c["niw"], c["niv"], c["niv"] + c["shell"]
    n2, w = n * n, niw + 1
    items, size = _solves(c)
    nq = items // (2 * w)
    fft = 5 * nk * math.log2(nk)
    flops = items * (8 / 3 * size**3 + 8 * n2 * size**2)
    flops += w * 8.0 * nq * n2 * (n2 * 2 * full) * (n2 * 2 * niv)
    flops += n2 * n2 * w * 2 * full * fft + n2 * n2 * w * 2 * niv * (fft + 8 * nk)
    read = 16 * (nk * n2 * 2 * (full + niw) + 2 * w * size**2 + w * (n2 * 2 * full) * (n2 * 2 * niv))
    write = 16 * (nk * n2 * 2 * niv + 2 * nq * w * n2 * n2)
    if box:
        b = n2 * 2 * box
        flops += 2 * nq * 2 * box * 8.0 * b * size**2 + 2 * b * b * fft
        write += 16 * (2 * nq * b * b + 2 * nk * b * b)
    return read + write, flops


def work(case):
    use = case["use"]
    if use == "pass":
        b, f = _pass_work(case)
    elif use == "pair":
        (b, f), (b1, f1) = _pass_work(case), _pass_work(_one_band(case))
        b, f = b + b1, f + f1
    elif use == "pairing":
        b, f = _pass_work(case, min(case["niw"] // 2, case["niv"] // 2))
    elif use == "gap":
        m = case["orb"] ** 2 * 2 * min(case["niw"] // 2, case["niv"] // 2)
        nk = case["nk"] ** 2
        item = 8 if case["mixed"] else 16
        b = 2 * (nk * m * m * item + nk * m * case["orb"] ** 2 * 16 + 2 * nk * m * 16)
        f = 2 * (2 * 8.0 * nk * m * m + 2 * m * 5 * nk * math.log2(nk))
    elif use == "local":
        w, n = case["niw"] + 1, case["orb"] ** 2 * 2 * case["niv"]
        full = case["orb"] ** 2 * 2 * (case["niv"] + case["shell"])
        b = 2 * w * 16 * (2 * n * n) + w * 16 * full**2
        f = 2 * w * (8 / 3 * n**3 + 8.0 * n**3 + 8 / 3 * n**3 + 8 / 3 * full**3 + 8.0 * full**3)
    else:
        items, n = _solves(case)
        b = items * 16 * (n * n + n * case["orb"] ** 2)
        f = items * (8 / 3 * n**3 + 8 * case["orb"] ** 2 * n**2)
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------------------------------------
# the same results by plain torch in complex128
# ------------------------------------------------------------------------------------------------
def _small_zero(x):
    return torch.where((x.real.abs() < 1e-12) & (x.imag.abs() < 1e-12), torch.zeros_like(x), x)


def _lambda(chi, count, target, beta, nk):
    """The lambda-correction of one channel: chi [q, w >= 0] -> (corrected chi, lambda)."""
    full = torch.cat([chi[:, 1:].flip(1).conj(), chi], 1)
    w = torch.from_numpy(count.astype(np.float64)).cuda()[:, None]
    start = -float((1 / chi[:, 0].real).min())
    delta = 0.1
    lam = start + delta
    for _ in range(1000):
        x = 1 / (1 / full + lam)
        f = complex((w * x).sum() / beta / nk) - target
        fp = -complex((w * x * x).sum() / beta / nk)
        new = lam - (f / fp).real
        if abs(f.real) < 1e-7:
            lam = new
            break
        if new < lam:
            delta /= 2
            lam = start + delta
        else:
            lam = new
    return 1 / (1 / chi + lam), lam


def _exact_pass(inp, box=0):
    n, (nk, _, _), niw, niv, shell, beta = inp["u"].shape[0], inp["nk"], inp["niw"], inp["niv_core"], inp["niv_shell"], inp["beta"]
    p, full, n_w, nkt = n * n, niv + shell, niw + 1, nk * nk
    up = lambda x: torch.from_numpy(np.ascontiguousarray(x)).cuda()  # noqa: E731
    g = up(inp["g_k"]).reshape(nk, nk, n, n, -1)
    mid = g.shape[-1] // 2
    ind, inv = up(inp["irrk_ind"]), up(inp["irrk_inv"])
    nq = len(ind)
    gr = torch.fft.fftn(g, dim=(0, 1))
    rev = torch.roll(gr.flip((0, 1)), (1, 1), (0, 1))
    um = {ch: up(_orbmat(_channel(inp["u"], ch))) for ch in ("dens", "magn")}
    u_dc = up(_orbmat(np.einsum("abcd->adcb", inp["u"])))
    kernel = torch.empty((nq, n_w, 2 * niv, p, p), dtype=C128, device="cuda")
    c0i = torch.empty_like(kernel)
    x = {ch: torch.empty_like(kernel) for ch in um}
    chi = {ch: torch.empty((nq, n_w, p, p), dtype=C128, device="cuda") for ch in um}
    pp = {ch: torch.empty((nq, 2 * box, p * 2 * box, p * 2 * box), dtype=C128, device="cuda") for ch in um} if box else None
    sel = torch.eye(p, dtype=C128, device="cuda").repeat_interleave(2 * niv, 0)
    for w in range(n_w):
        left, right = gr[..., mid - full : mid + full], rev[..., mid - full - w : mid + full - w]
        c0 = torch.fft.ifftn(torch.einsum("xyadv,xycbv->xyvabdc", left, right), dim=(0, 1)).reshape(nkt, 2 * full, p, p)[ind]
        c0 = _small_zero(c0 * (-beta / nkt))
        f = _compound(inp["f_dc"][..., w : w + 1, :, :])[0].reshape(p, 2 * full, p, 2 * full)[..., shell : shell + 2 * niv]
        t = (u_dc @ c0 / beta**2).permute(0, 2, 3, 1).reshape(nq * p, p * 2 * full)
        kernel[:, w] = -(t @ f.reshape(p * 2 * full, -1)).reshape(nq, p, p, 2 * niv).permute(0, 3, 1, 2)
        core = c0[:, shell : shell + 2 * niv]
        c0i[:, w] = torch.linalg.inv(core)
        extra = (c0.sum(1) - core.sum(1)) / beta**2
        for ch in um:
            base = _compound(inp["gamma_" + ch][..., w : w + 1, :, :])[0].reshape(p, 2 * niv, p, 2 * niv)
            base = ((base - um[ch][:, None, :, None]) / beta**2).reshape(p * 2 * niv, -1)
            step = max(1, (1 << 27) // base.numel())
            for q in range(0, nq, step):
                a = _block_diag(c0i[q : q + step, w]) + base
                if box and w < 2 * box:
                    star = torch.linalg.inv(a)
                    y = star @ sel
                    star = star.reshape(-1, p, 2 * niv, p, 2 * niv)[:, :, niv - box : niv + box, :, niv - box : niv + box]
                    c = c0i[q : q + step, w, niv - box : niv + box]
                    star = torch.einsum("qvpm,qmvnu,quns->qpvsu", c, star, c)
                    pp[ch][q : q + step, w] = beta**2 * (_block_diag(c) - star.reshape(len(c), p * 2 * box, -1))
                else:
                    y = torch.linalg.solve(a, sel.expand(len(a), -1, -1))
                x[ch][q : q + step, w] = y.reshape(-1, p, 2 * niv, p).permute(0, 2, 1, 3) / beta
            aux = x[ch][:, w].sum(1) / beta
            chi[ch][:, w] = torch.linalg.inv(torch.linalg.inv(aux + extra) + um[ch])
    lambdas = []
    if n == 1:
        for ch in um:
            c, lam = _lambda(chi[ch].reshape(nq, n_w), inp["irrk_count"], inp["chi_loc_sum_" + ch], beta, nkt)
            chi[ch] = c.reshape(nq, n_w, 1, 1)
            lambdas.append(lam)
    gamma3 = {ch: beta * c0i @ x[ch] for ch in um}
    for ch in um:
        k = gamma3[ch] - gamma3[ch] @ (um[ch] @ chi[ch])[:, :, None]
        if ch == "magn":
            k = k - 2 / 3 * torch.eye(p, dtype=C128, device="cuda")
        kernel += (1 if ch == "dens" else 3) * (um[ch] @ k)
    # Sigma(R, nu > 0) over all w with K(-w, nu) = conj K(w, -nu - 1)
    sig = torch.zeros((nk, nk, n, n, niv), dtype=C128, device="cuda")
    for w in range(-niw, n_w):
        k = kernel[:, w, niv:] if w >= 0 else kernel[:, -w].flip(1)[:, niv:].conj()
        k = k[inv].reshape(nk, nk, niv, n, n, n, n)  # x y nu a b(i) d c(j) of K[a, i, j, d]
        k = torch.fft.fftn(k.conj(), dim=(0, 1)).conj()
        sig += torch.einsum("xyadv,xyvaidj->xyijv", gr[..., mid - w : mid + niv - w], k)
    sig = torch.fft.ifftn(sig * (-0.5 / beta / nkt), dim=(0, 1)).reshape(nkt, n, n, niv)
    out = {"sigma": torch.cat([sig.flip(-1).conj(), sig], -1), "chi": torch.stack([chi["dens"], chi["magn"]])}
    if n == 1:
        out["lambdas"] = torch.tensor(lambdas, dtype=torch.float64, device="cuda")
    if box:
        for ch in um:
            z = um[ch] - um[ch] @ chi[ch][:, : 2 * box] @ um[ch]
            g3 = gamma3[ch][:, : 2 * box, niv - box : niv + box]
            pp[ch] += torch.einsum("qwpm,qwvmn,qwuns->qwpvsu", z, g3, g3).reshape(pp[ch].shape)
        out["pp"] = pp
    return out


def _exact_pairing(inp, box):
    """Sigma, the pairing vertices [2][q][(a,b,nu)][(c,d,nu')] (Gamma[a,c,b,d]), their operators and chi0_pp."""
    n, (nk, _, _), v = inp["u"].shape[0], inp["nk"], 2 * box
    out = _exact_pass(inp, box)
    inv = torch.from_numpy(inp["irrk_inv"]).cuda()
    i = torch.arange(v, device="cuda")
    om = i[:, None] - i[None, :]
    f_pp = {}
    for ch, f in out["pp"].items():
        f = f.reshape(-1, v, n, n, v, n, n, v).permute(0, 2, 3, 6, 5, 1, 4, 7)  # q a b c d w nu nu'
        pos = f[..., om.clamp(min=0), i[:, None], (v - 1 - i)[None, :]]
        neg = f.conj()[..., (-om).clamp(min=0), (v - 1 - i)[:, None], i[None, :]]
        f_pp[ch] = -torch.where(om >= 0, pos, neg)
    sing, trip = 0.5 * f_pp["dens"] - 1.5 * f_pp["magn"], 0.5 * f_pp["dens"] + 0.5 * f_pp["magn"]
    mats = torch.stack([x.permute(0, 1, 3, 5, 2, 4, 6).reshape(len(x), n * n * v, n * n * v) for x in (sing, trip)])
    ops = []
    for x, sign in zip(mats, (1, -1)):
        full = x[inv].reshape(nk, nk, *x.shape[1:])
        ops.append(sign * torch.fft.fftn(full, dim=(0, 1)).reshape(nk * nk, *x.shape[1:]))
    g = torch.from_numpy(inp["g_k"]).cuda().reshape(nk * nk, n, n, -1)
    mid = g.shape[-1] // 2
    g = g[..., mid - box : mid + box]
    bubble = _small_zero(torch.einsum("kadv,kbcv->kvabcd", g, g.conj().transpose(1, 2)).reshape(nk * nk, v, n * n, n * n))
    return {"sigma": out["sigma"], "vertex": mats, "operators": torch.stack(ops), "bubble": bubble}


def _exact_gap(inp, box, x):
    n, (nk, _, _), v, beta = inp["u"].shape[0], inp["nk"], 2 * box, inp["beta"]
    ex = _exact_pairing(inp, box)
    bubble = ex["bubble"].reshape(nk * nk, v, n, n, n, n)
    res = []
    for st, sign in ((0, 1), (1, -1)):
        gap = x[st].reshape(nk * nk, n, n, v)
        gg = torch.einsum("kvabcd,kcdv->kabv", bubble, gap).reshape(nk, nk, n, n, v)
        gg = torch.fft.fftn(gg, dim=(0, 1))
        back = torch.roll(gg.flip((0, 1)), (1, 1), (0, 1))
        op = ex["operators"][st].reshape(nk, nk, n, n, v, n, n, v)  # a b nu c d nu' of Gamma[a, c, b, d]
        flip = torch.roll(op.flip((0, 1)), (1, 1), (0, 1)).flip(-1).permute(0, 1, 2, 3, 4, 6, 5, 7)
        new = torch.einsum("xyabvcdp,xycdp->xyabv", op, gg) + sign * torch.einsum("xyabvcdp,xycdp->xyabv", flip, back)
        res.append(torch.fft.ifftn(0.5 / (nk * nk) / beta * new, dim=(0, 1)).reshape(-1))
    return {"sing": res[0], "trip": res[1]}


def _exact_local(c, seed):
    orb, niw, niv, shell = c["orb"], c["niw"], c["niv"], c["shell"]
    g, g2d, g2m, u, beta, occ = _local_inputs(c, seed)
    p, full, n_w, v = orb * orb, niv + shell, niw + 1, 2 * niv
    mid = g.shape[-1] // 2
    gs = g[..., mid - niv : mid + niv]
    c0 = _small_zero(_local_bubble(g, niw, full, beta))
    core = c0[:, shell : shell + v]
    c0i = torch.linalg.inv(core)
    gammas, chis, vrgs, inner = [], [], [], 0
    for ch, g2 in (("dens", g2d), ("magn", g2m)):
        u_r = _channel(u, ch)
        um = torch.from_numpy(np.ascontiguousarray(_orbmat(u_r))).cuda()
        gchi = beta * g2
        if ch == "dens":
            gchi[:, :, :, :, 0] -= 2 * beta * gs[:, :, None, None, :, None] * gs[None, None, :, :, None, :]
        ub = um[:, None, :, None]
        gamma = beta**2 * (torch.linalg.inv(_compound(gchi)) - _shell_bubble_inverse(c0, um, beta, niv, shell))
        gamma = (gamma.reshape(n_w, p, v, p, v) + ub).reshape(n_w, p * v, p * v)
        gammas.append(_four(gamma, orb))
        if ch == "magn":
            gu = torch.zeros((n_w, p, 2 * full, p, 2 * full), dtype=C128, device="cuda") + ub
            gu[:, :, shell : shell + v, :, shell : shell + v] = gamma.reshape(n_w, p, v, p, v)
            gu = gu.reshape(n_w, p * 2 * full, -1)
            eye = torch.eye(p * 2 * full, dtype=C128, device="cuda")
            f = gu @ torch.linalg.inv(eye + _block_diag(c0) @ gu / beta**2)
            f_dc = 2 * _four(f, orb).permute(2, 1, 0, 3, 4, 5, 6)
        star = torch.linalg.inv(_block_diag(c0i) + (gamma.reshape(n_w, p, v, p, v) - ub).reshape(gamma.shape) / beta**2)
        x = star.reshape(n_w, p, v, p, v).sum(-1).permute(0, 2, 1, 3) / beta
        vr = beta * c0i @ x
        chi = torch.linalg.inv(torch.linalg.inv(x.sum(1) / beta + (c0.sum(1) - core.sum(1)) / beta**2) + um)
        inner = inner + (0.5 if ch == "dens" else -0.5) * (vr - vr @ (um @ chi)[:, None])
        vrgs.append(vr.reshape(n_w, v, orb, orb, orb, orb).permute(2, 3, 5, 4, 0, 1))
        chis.append(chi.reshape(n_w, orb, orb, orb, orb).permute(1, 2, 4, 3, 0))
    inner = inner.reshape(n_w, v, orb, orb, orb, orb).permute(2, 3, 5, 4, 0, 1)  # i l p o w nu
    inner = torch.cat([inner[..., 1:, :].flip((-2, -1)).conj(), inner], -2)
    gw = torch.stack([g[..., mid - niv - w : mid + niv - w] for w in range(-niw, n_w)], -2)
    um4 = torch.from_numpy(u).cuda()
    sigma = -1 / beta * torch.einsum("kjop,ilpowv,lkwv->ijv", um4, inner, gw)
    sigma = sigma + torch.einsum("abcd,dc->ab", torch.from_numpy(_channel(u, "dens")).cuda(), torch.from_numpy(occ).cuda())[..., None]
    return {"gamma": gammas, "f_dc": f_dc, "chi": chis, "vrg": vrgs, "sigma": sigma.reshape(1, 1, 1, orb, orb, v)}


def exact(case, seed):
    use = case["use"]
    if use == "dense":
        x, beta = _dense_inputs(case, seed)
        n, v = case["orb"], 2 * case["niv"]
        out = [torch.linalg.inv(_compound(a)).reshape(-1, n, n, v, n, n, v).sum(-1).permute(1, 2, 5, 4, 0, 3) / beta for a in x]
        return torch.stack(out)
    if use == "local":
        return _exact_local(case, seed)
    inp = _pass_inputs(case, seed)
    if use == "pair":
        return [{k: v for k, v in _exact_pass(_pass_inputs(c, seed)).items()} for c in (case, _one_band(case))]
    if use == "pass":
        out = _exact_pass(inp)
        return {"sigma": out["sigma"].cpu().numpy()} if case["host"] else out
    box = min(case["niw"] // 2, case["niv"] // 2)
    if use == "pairing":
        return _exact_pairing(inp, box)
    nk = case["nk"] ** 2
    return _exact_gap(inp, box, _gap_vectors(nk * case["orb"] ** 2 * 2 * box, seed))
