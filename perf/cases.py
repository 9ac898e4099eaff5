"""The work that programs built on nrcps_b200 have it do, as cases to measure.

One function per kind of call (the `KINDS` table at the end): how its inputs
are made, one pass through the public entry points, the bytes and operations
that pass cannot do without, and its result in 64 bits from plain torch.

Sizes are those of this repository's workloads, tests and benchmark: lattices
of 8 to 48 sites a side, Fermi seas of 7, 19 and 33 plane waves or a handful
of oscillator states, one configuration to a few thousand.

Results of FP32 orbitals carry single precision whatever type an entry point
hands them back in, and a program that runs in FP32 keeps them so: such cases
return complex64 and float32.
"""
import math

import numpy as np
import torch

import nrcps_b200 as nb

PI = math.pi
EXTENTS = (4, 6, 8, 12, 16, 24, 32, 48)      # lattice extents the transforms take
CUBES = (8, 12, 16, 24, 32, 48)
SITES = 1024 * 19 * 32 ** 3 // 4             # orbital entries of the largest block case


def listed():
    return [
        # one time slice of two particles in a small box through the class API: launches and latency
        dict(name="class_l8_f64", kind="class", X=8, Y=8, Z=8, N=2, precision="f64", trap=False, slices=1),
        # a small uneven box with a trap, FP32, two slices
        dict(name="class_box_trap_f32", kind="class", X=24, Y=12, Z=16, N=7, precision="f32", trap=True, slices=2),
        # the reference's own call structure at the production size: one configuration, FP64
        dict(name="class_l32_f64", kind="class", X=32, Y=32, Z=32, N=19, precision="f64", trap=False, slices=2),
        # transfer-matrix steps of a batch of configurations, fields of four slices at hand:
        # a few small ones
        dict(name="step_l16_z2_f32", kind="step", L=16, N=7, n_conf=24, precision="f32", field="z2", trap=False, slices=4),
        # the batched production step
        dict(name="step_l32_z2_f32", kind="step", L=32, N=19, n_conf=256, precision="f32", field="z2", trap=False, slices=4),
        # the trapped few-body step, an odd number of configurations
        dict(name="step_l48_trap_f32", kind="step", L=48, N=10, n_conf=51, precision="f32", field="z2", trap=True, slices=4),
        # double precision with a Gaussian field, as checks of the FP32 mode and small production runs have it
        dict(name="step_l24_gauss_f64", kind="step", L=24, N=19, n_conf=33, precision="f64", field="gauss", trap=False, slices=4),
        # re-orthonormalisation of live orbitals, every eighth slice of an FP32 run
        dict(name="qr_l32_f32", kind="qr", L=32, N=19, n_conf=256, precision="f32"),
        # the measurement of a trapped run: overlaps with dense sources, the pair matrix
        dict(name="overlap_l48_f32", kind="overlap", L=48, N=10, n_conf=128, precision="f32"),
        dict(name="pair_l48_f32", kind="pair", L=48, N=10, n_conf=128, precision="f32"),
        # the determinants of all leading minors, one slice of the production run
        dict(name="dets_n19", kind="dets", N=19, n_conf=4096, pair_sink=False),
        # a whole run of the batched production loop: fields, sources, steps, measurements, re-orthonormalisation
        dict(name="ensemble_l32_f32", kind="ensemble", L=32, N=19, n_conf=1024, T=16, precision="f32", qr_period=8),
    ]


def _log_int(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["class", "class", "step", "step", "step", "qr", "overlap", "pair", "dets", "ensemble"])
    precision = rng.choice(["f32", "f32", "f64"])
    n = rng.choice([1, 2, 3, 5, 7, 10, 13, 19, 19, 24, 33])
    L = rng.choice(CUBES)
    V = L ** 3
    if kind == "class":
        X, Y, Z = (rng.choice(EXTENTS) for _ in range(3))
        if rng.random() < 0.5:
            X = Y = Z = L
        n = max(1, min(n, 2 ** 21 // (X * Y * Z), X * Y * Z // 8))
        return dict(kind="class", X=X, Y=Y, Z=Z, N=n, precision=rng.choice(["f64", "f64", "f32"]),
                    trap=rng.random() < 0.4, slices=rng.choice([1, 2]))
    if kind == "step":
        field = rng.choice(["z2", "z2", "gauss", "table"])
        if field == "table":
            precision = "f32"
        most = SITES // (2 if precision == "f64" else 1) // (V * n)
        if field == "gauss":  # 16 bytes per site and slice of field beside the orbitals
            most = min(most, 2 ** 23 // V)
        return dict(kind="step", L=L, N=n, n_conf=_log_int(rng, 1, max(1, most)), precision=precision, field=field,
                    trap=field != "table" and rng.random() < 0.4, slices=rng.choice([2, 3, 4]))
    if kind in ("qr", "overlap", "pair"):
        most = SITES // (8 if precision == "f64" else 2) // (V * n)
        return dict(kind=kind, L=L, N=n, n_conf=_log_int(rng, 1, max(1, most)), precision=precision)
    if kind == "dets":
        return dict(kind="dets", N=rng.randint(2, 40), n_conf=_log_int(rng, 1, 4096), pair_sink=rng.random() < 0.4)
    T = rng.choice([4, 7, 12, 16])
    if L == 48:
        n = min(n, 10)
    most = 32 * SITES // (8 if precision == "f64" else 1) // (V * n) // T
    return dict(kind="ensemble", L=L, N=n, n_conf=_log_int(rng, 1, max(1, min(most, 4096))), T=T, precision=precision,
                qr_period=8 if precision == "f32" else 0)


# ------------------------------------------------------------------ inputs
def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _gen(seed, salt=0):
    return torch.Generator(device=_dev()).manual_seed(1000003 * salt + int(seed))


def _cdtype(precision):
    return torch.complex128 if precision == "f64" else torch.complex64


def _kept(t, precision):
    """A result as a program of that precision keeps it."""
    if precision == "f64":
        return t
    return t.to(torch.complex64 if t.is_complex() else torch.float32)


def _fold(n):
    """Site or momentum numbers folded to [-n/2, n/2)."""
    i = torch.arange(n, dtype=torch.float64, device=_dev())
    return torch.where(i >= n // 2, i - n, i)


def _grid(dims, f):
    """f of the three folded numbers, summed over the axes, as a flat table."""
    t = [f(_fold(n), n) for n in dims]
    return (t[0][:, None, None] + t[1][None, :, None] + t[2][None, None, :]).reshape(-1)


def _psq(dims):
    return _grid(dims, lambda i, n: (2 * PI * i / n) ** 2)


def _kinv(dims, dt=0.5):
    """1/xi(p) of the continuum dispersion, mass 1."""
    return torch.exp(-_psq(dims) * dt / 2)


def _trap(dims, kappa=0.005, dt=0.5):
    """exp(-dt kappa x^2 / 2) of the harmonic trap."""
    return torch.exp(-dt * kappa * _grid(dims, lambda i, n: i ** 2) / 2)


def _waves(dims, n):
    """Lattice indices of the n plane waves of lowest energy."""
    return torch.argsort(_psq(dims), stable=True)[:n]


def _normal(shape, gen, dtype):
    return torch.randn(shape, generator=gen, dtype=dtype, device=_dev())


def _orbitals(n_conf, n, dims, gen, dtype):
    """Orbitals in momentum space as some slices leave them: smooth, of norm
    about one, every one with a share of its predecessor."""
    V = math.prod(dims)
    shape = torch.exp(-_psq(dims) / 8)
    shape /= torch.linalg.vector_norm(shape)
    psi = _normal((n_conf, n, V), gen, dtype) * shape.to(dtype)
    for i in range(1, n):
        psi[:, i] += 0.5 * psi[:, i - 1]
    return psi


def _signs(bits, count):
    """+-1 of packed field bits."""
    b = torch.arange(32, dtype=torch.int32, device=bits.device)
    return (((bits[:, None] >> b) & 1).reshape(-1)[:count] * 2 - 1).to(torch.float64)


def _minors(S):
    """det of every leading minor of [.., N, N]."""
    return torch.stack([torch.linalg.det(S[..., :k, :k]) for k in range(1, S.shape[-1] + 1)], dim=-1)


def _fft(x, sign):
    return torch.fft.fftn(x, dim=(-3, -2, -1)) if sign < 0 else torch.fft.ifftn(x, dim=(-3, -2, -1), norm="forward")


def _esize(c):
    return 16 if c["precision"] == "f64" else 8


def _fft_flops(V):
    return 5 * V * math.log2(V)


# ------------------------------------------- the class API, one configuration
# Sources into the propagator, then per slice the Slater determinants, the
# interaction on the slice's field and the Hamiltonians one after the other.
def _class_inputs(c, seed):
    dims = (c["X"], c["Y"], c["Z"])
    V, N = math.prod(dims), c["N"]
    g = _gen(seed, 1)
    if c["trap"]:  # dense sources
        src = _orbitals(1, N, dims, g, torch.complex128)[0]
    else:  # plane waves, mixed a little so that no determinant is trivial
        src = 0.01 * _orbitals(1, N, dims, g, torch.complex128)[0]
        src[torch.arange(N, device=_dev()), _waves(dims, N)[:N]] += 1
    phi = torch.zeros((V, 2), dtype=torch.float64, device=_dev())
    phi[:, 0] = torch.randint(0, 2, (V,), generator=g, device=_dev()) * 2.0 - 1.0
    return dims, V, N, src, phi


def _class_prepare(c, seed):
    dims, V, N, src, phi = _class_inputs(c, seed)
    ctx = nb.default_context()
    lattice = nb.Lattice(dims, nb.Random("RANLXS2", 7), "ZTWO", ctx)
    lattice.get().copy_(phi)
    kinetic = nb.Kinetic(dims, ctx=ctx)
    interaction = nb.Interaction(lattice)
    h = [kinetic, interaction, kinetic]
    if c["trap"]:
        potential = nb.Potential(dims, 0.005, 0.5, "EXP", ctx)
        h = [kinetic, potential, interaction, potential, kinetic]
    sources = []
    for n in range(N):
        one = nb.OneBody(dims, ctx)
        one.get().copy_(src[n])
        sources.append(one)
    return dict(c=c, h=h, interaction=interaction, sources=sources, prop=nb.Propagator(N, dims, c["precision"], ctx))


def _class_run(s):
    prop, N = s["prop"], len(s["sources"])
    for n in range(N):
        prop.set(s["sources"][n].get(), n)
    dets = []
    for _ in range(s["c"]["slices"]):
        s["interaction"].initialize()
        prop.run(s["h"])
        slater = nb.SlaterDet(prop.get().b, s["sources"])
        dets.append([slater.run(n) for n in range(1, N + 1)])
    dets = np.array(dets)
    return {"psi": prop.get().b, "dets": dets if s["c"]["precision"] == "f64" else dets.astype(np.complex64)}


def _class_exact(c, seed):
    dims, V, N, src, phi = _class_inputs(c, seed)
    psi = src.to(_cdtype(c["precision"])).to(torch.complex128).reshape((N,) + dims)
    k, v = _kinv(dims).reshape(dims), _trap(dims).reshape(dims) / V
    # one constant coupling: c(p) = 1/(2 V), so the smeared field is (1 + phi/2)/V
    fld = ((1 + 0.5 * phi[:, 0]) / V).reshape(dims)
    dets = []
    for _ in range(c["slices"]):
        psi = k * psi
        for w in ([v, fld, v] if c["trap"] else [fld]):
            psi = _fft(w * _fft(psi, -1), +1)
        psi = k * psi
        dets.append(_minors(src.conj() @ psi.reshape(N, V).T))
    return {"psi": psi, "dets": torch.stack(dets).cpu().numpy()}


def _class_work(c):
    V, N, e = c["X"] * c["Y"] * c["Z"], c["N"], _esize(c)
    h = 5 if c["trap"] else 3
    per_slice = 2 * h * N * V * e + N * V * (16 + e) + 3 * 16 * V
    flops = (2 * (h - 2) * N + 2) * _fft_flops(V) + 8 * N * N * V + 8 * N ** 4 / 12
    return dict(bytes=N * V * (16 + e) + c["slices"] * per_slice, flops=c["slices"] * flops)


# ------------------------------------------------- steps of many configurations
# Every configuration starts from the same sources; its field of each slice is
# at hand, as an ensemble draws them ahead of its time loop.
def _step_inputs(c, seed):
    dims = (c["L"],) * 3
    V, count = c["L"] ** 3, c["n_conf"] * c["slices"] * c["L"] ** 3
    g = _gen(seed, 2)
    src = _orbitals(1, c["N"], dims, g, _cdtype(c["precision"]))[0]
    if c["field"] == "z2":
        a, mode = 0.5, 1
        field = torch.randint(-2 ** 31, 2 ** 31, ((count + 31) // 32,), generator=g, dtype=torch.int32, device=_dev())
    else:
        a, mode = 0.3, 2
        field = torch.zeros((count, 2), dtype=torch.float64, device=_dev())
        field[:, 0] = torch.randn(count, generator=g, dtype=torch.float64, device=_dev())
        if c["field"] == "table":
            mode, field = 3, ((1 + a * field[:, 0]) / V).to(torch.float32)
    return dims, V, src, a, mode, field, _trap(dims) if c["trap"] else None


def _step_prepare(c, seed):
    dims, V, src, a, mode, field, pos = _step_inputs(c, seed)
    ctx = nb.default_context()
    if ctx.fused_choice(c["precision"], c["L"])[0] >= 0:
        ctx.autotune(c["precision"], c["L"])
    psi = torch.empty((c["n_conf"] * c["N"],) + dims, dtype=src.dtype, device=_dev())
    return dict(c=c, V=V, src=src.reshape((c["N"],) + dims), psi=psi, kinv=_kinv(dims), a=a, mode=mode, field=field,
                pos=pos, ctx=ctx)


def _step_run(s):
    c, V = s["c"], s["V"]
    s["psi"].view((c["n_conf"],) + s["src"].shape).copy_(s["src"])
    for t in range(c["slices"]):
        nb.propagate(s["psi"], c["N"], s["kinv"], s["field"], s["a"], s["mode"], t * V, c["slices"] * V, s["pos"],
                     s["ctx"])
    return s["psi"]


def _step_exact(c, seed):
    dims, V, src, a, mode, field, pos = _step_inputs(c, seed)
    count = c["n_conf"] * c["slices"] * V
    if mode == 1:
        w = (1 + a * _signs(field, count)) / V
    else:
        w = (1 + a * field[:, 0]) / V if mode == 2 else field.to(torch.float64)
    w = w.reshape((c["n_conf"], c["slices"]) + dims)
    if pos is not None:
        w = w * pos.reshape(dims)
    k = _kinv(dims).reshape(dims)
    out = torch.empty((c["n_conf"], c["N"]) + dims, dtype=torch.complex128, device=_dev())
    for i in range(c["n_conf"]):
        psi = src.to(torch.complex128).reshape((c["N"],) + dims)
        for t in range(c["slices"]):
            psi = k * _fft(w[i, t] * _fft(k * psi, -1), +1)
        out[i] = psi
    return out.reshape((c["n_conf"] * c["N"],) + dims)


def _step_work(c):
    V, n = c["L"] ** 3, c["n_conf"] * c["N"]
    site = {"z2": 0.125, "gauss": 16, "table": 4}[c["field"]]
    moved = n * V * _esize(c) * (1 + 2 * c["slices"])
    return dict(bytes=moved + c["n_conf"] * c["slices"] * V * site,
                flops=c["slices"] * n * (2 * _fft_flops(V) + 6 * V))


# ------------------------------------------------------- re-orthonormalisation
# In place on orbitals that have grown since the last one; a pass takes them
# from where they were left, so that every pass meets the same.
def _qr_inputs(c, seed):
    return 20 * _orbitals(c["n_conf"], c["N"], (c["L"],) * 3, _gen(seed, 3), _cdtype(c["precision"]))


def _qr_prepare(c, seed):
    left = _qr_inputs(c, seed)
    return dict(c=c, left=left, psi=torch.empty_like(left), ctx=nb.default_context())


def _qr_run(s):
    s["psi"].copy_(s["left"])
    log_r = nb.reorthonormalise(s["psi"], None, s["ctx"])
    return {"psi": s["psi"], "log_r": _kept(log_r, s["c"]["precision"])}


def _qr_exact(c, seed):
    psi = _qr_inputs(c, seed)
    out = torch.empty(psi.shape, dtype=torch.complex128, device=_dev())
    log_r = torch.empty((c["n_conf"], c["N"]), dtype=torch.float64, device=_dev())
    for i in range(c["n_conf"]):
        p = psi[i].to(torch.complex128)
        low = torch.linalg.cholesky(p.conj() @ p.T)  # G = R^H R, R = low^H
        out[i] = torch.linalg.solve_triangular(low.conj(), p, upper=False)
        log_r[i] = torch.log(torch.diagonal(low).real)
    return {"psi": out, "log_r": log_r}


def _qr_work(c):
    size = c["n_conf"] * c["N"] * c["L"] ** 3
    return dict(bytes=4 * size * _esize(c), flops=8 * size * c["N"])


# ------------------------------------------- overlaps and pair matrices
def _overlap_inputs(c, seed):
    dims, g = (c["L"],) * 3, _gen(seed, 4)
    src = _orbitals(1, c["N"], dims, g, torch.complex128)[0]
    return src, _orbitals(c["n_conf"], c["N"], dims, g, _cdtype(c["precision"]))


def _overlap_prepare(c, seed):
    src, psi = _overlap_inputs(c, seed)
    return dict(c=c, src=src, psi=psi, ctx=nb.default_context())


def _overlap_run(s):
    return _kept(nb.overlap(s["src"], s["psi"], s["ctx"]), s["c"]["precision"])


def _overlap_exact(c, seed):
    src, psi = _overlap_inputs(c, seed)
    return torch.stack([src.conj() @ p.to(torch.complex128).T for p in psi])


def _overlap_work(c):
    V, n = c["L"] ** 3, c["N"]
    return dict(bytes=c["n_conf"] * n * V * _esize(c) + 16 * n * V + 16 * c["n_conf"] * n * n,
                flops=8 * c["n_conf"] * n * n * V)


def _pair_prepare(c, seed):
    dims = (c["L"],) * 3
    ctx = nb.default_context()
    psi = _orbitals(c["n_conf"], c["N"], dims, _gen(seed, 5), _cdtype(c["precision"]))
    return dict(c=c, psi=psi, two=nb.TwoBody(dims, "TGND", "STANDARD", 1.0, 0.176776695, 2.0, ctx))


def _pair_run(s):
    return _kept(s["two"].run_matrix(s["psi"], s["psi"]), s["c"]["precision"])


def _pair_weight(L, lam):
    """The trapped ground state's weight F(q)/q, q = |p| / (2 lambda), up to
    |p| = 2 pi; F: Dawson's integral by Rybicki's sampling (h = 0.4, six terms,
    three terms of the series below 0.2)."""
    psq = _psq((L,) * 3)
    q = torch.sqrt(psq) / (2 * lam)
    n0 = 2 * torch.floor(0.5 * q / 0.4 + 0.5)
    xp = q - n0 * 0.4
    total = torch.zeros_like(q)
    for i in range(6):
        m = 2 * i + 1
        total += math.exp(-(m * 0.4) ** 2) * (torch.exp(0.8 * m * xp) / (n0 + m) + torch.exp(-0.8 * m * xp) / (n0 - m))
    sampled = torch.exp(-xp ** 2) * total / math.sqrt(PI) / q.clamp(min=1e-300)
    series = 1 - 2 / 3 * q ** 2 * (1 - 0.4 * q ** 2 * (1 - 2 / 7 * q ** 2))
    return torch.where(psq > (2 * PI) ** 2, torch.zeros_like(q), torch.where(q < 0.2, series, sampled))


def _pair_exact(c, seed):
    L = c["L"]
    psi = _orbitals(c["n_conf"], c["N"], (L,) * 3, _gen(seed, 5), _cdtype(c["precision"]))
    w = _pair_weight(L, 0.176776695)
    i = (-torch.arange(L, device=_dev())) % L
    out = []
    for p in psi:
        p = p.to(torch.complex128).reshape((-1, L, L, L))
        q = p[:, i][:, :, i][:, :, :, i]
        out.append((p.reshape(c["N"], -1) * w) @ q.reshape(c["N"], -1).T)
    return torch.stack(out)


def _pair_work(c):
    V, n = c["L"] ** 3, c["N"]
    return dict(bytes=c["n_conf"] * n * V * _esize(c) + 12 * V + 16 * c["n_conf"] * n * n,
                flops=4 * c["n_conf"] * n * (n + 1) * V)


# ------------------------------------------------------------- determinants
def _dets_prepare(c, seed):
    g, n = _gen(seed, 6), c["N"]
    S = torch.eye(n, dtype=torch.complex128, device=_dev()) + 0.3 * _normal((c["n_conf"], n, n), g, torch.complex128)
    one = _normal((c["n_conf"], n, n), g, torch.complex128) if c["pair_sink"] else None
    return dict(c=c, S=S, one=one, ctx=nb.default_context())


def _dets_run(s):
    return nb.slater_dets(s["S"], s["one"], 1 if s["c"]["pair_sink"] else 0, False, s["ctx"])


def _dets_exact(c, seed):
    if c["pair_sink"]:  # which column is replaced by which is the driver's own convention
        return None
    return _minors(_dets_prepare(c, seed)["S"])


def _dets_work(c):
    n, m = c["N"], 2 if c["pair_sink"] else 1
    return dict(bytes=16 * c["n_conf"] * (m * n * n + m * n), flops=c["n_conf"] * m * 8 * sum(k ** 3 for k in range(1, n + 1)) / 3)


# ------------------------------------------------------------- whole runs
# Block after block of configurations, the fields drawn from the generator's
# stream; each configuration's determinants after every slice come back.
def _ensemble_prepare(c, seed):
    dims = (c["L"],) * 3
    job = nb.EnsembleJob(L=c["L"], T=c["T"], n_conf=c["n_conf"], seed=1 + int(seed) % 100000, precision=c["precision"],
                         qr_period=c["qr_period"])
    ens = nb.Ensemble(job, plane_wave_index=_waves(dims, c["N"]).cpu().numpy(), ctx=nb.default_context())
    return dict(c=c, ens=ens, first=0)


def _ensemble_run(s):
    dets = s["ens"].run(s["first"])
    s["first"] += s["c"]["n_conf"]
    return _kept(dets, s["c"]["precision"])


def _ensemble_exact(c, seed):
    return None  # the fields come from inside the run


def _ensemble_work(c):
    V, n = c["L"] ** 3, c["n_conf"] * c["N"]
    qr = (c["T"] - 1) // c["qr_period"] if c["qr_period"] else 0
    return dict(bytes=(2 * c["T"] + 2 * qr) * n * V * _esize(c) + c["n_conf"] * c["T"] * (V / 8 + 16 * c["N"]),
                flops=c["T"] * n * (2 * _fft_flops(V) + 6 * V) + qr * 8 * n * c["N"] * V)


KINDS = {
    "class": (_class_prepare, _class_run, _class_exact, _class_work),
    "step": (_step_prepare, _step_run, _step_exact, _step_work),
    "qr": (_qr_prepare, _qr_run, _qr_exact, _qr_work),
    "overlap": (_overlap_prepare, _overlap_run, _overlap_exact, _overlap_work),
    "pair": (_pair_prepare, _pair_run, _pair_exact, _pair_work),
    "dets": (_dets_prepare, _dets_run, _dets_exact, _dets_work),
    "ensemble": (_ensemble_prepare, _ensemble_run, _ensemble_exact, _ensemble_work),
}


def prepare(case, seed):
    return KINDS[case["kind"]][0](case, seed)


def run(state):
    return KINDS[state["c"]["kind"]][1](state)


def exact(case, seed):
    return KINDS[case["kind"]][2](case, seed)


def work(case):
    return KINDS[case["kind"]][3](case)
