"""The workloads whose speed is tracked: what users of this package have it do.

Each case is one pass through the public entry points: the propagator closures a
stage holds (``stage.propagator``), multi-step calls, the outputs of a due
diagnostic step, the spectrum helpers and a batched parameter sweep.  Sizes run
from 32^3 (a quick interactive solve) to 512^3, in both precisions, and take in
grid sides that are no power of two, as users choose dx and the box freely.

Units are the reference convention: kinetic factor exp(-i k^2 dt), local factor
exp(-i (V + beta |psi|^2) dt/2); the trap x^2 + 1.44 y^2 + 2.25 z^2 is the
harmonic trap (x^2 + 1.44 y^2 + 2.25 z^2)/2 of oscillator units.
"""

import math

import numpy as np
import torch

from gpe_simulator_b200 import helper, nk_extraction
from gpe_simulator_b200.batch import Batch, Instance
from gpe_simulator_b200.expressions import cuda_expression
from gpe_simulator_b200.plan import Beam
from gpe_simulator_b200.stage import stage as Stage

TRAP = (1.0, 1.44, 2.25)
N_ATOMS = 1.0e5
BOHR = 5.29177210544e-11

# op: "closure" one call of the stage's propagator; "run" `steps` steps in one call;
#     "output" what a stage writes at a due step; "spectrum" the FFT and k-space
#     helpers on a state the caller holds; "sweep" a batch of imaginary-time solves.
# potential: "trap" static formula; "beam" trap + rotating stirring beam; "walls" box
#     walls as an array (real time: with absorber and momentum cutoff) on top of the
#     trap; "shaken" trap + a formula in x, y, z, t.


def listed():
    return [
        # one step of an interactive ground-state search on a small grid: latency
        _case("step_32_c128", "closure", 32, "complex128", "imaginary", "trap", 1),
        # one step of a user's own Python time loop while stirring
        _case("step_stir_128_c64", "closure", 128, "complex64", "real", "beam", 1),
        # the plain 64^3 ground state in the reference's precision, between two log points
        _case("ground_64_c128", "run", 64, "complex128", "imaginary", "trap", 50),
        # a ground state on a grid side that is no power of two
        _case("ground_200_c64", "run", 200, "complex64", "imaginary", "trap", 6),
        # an odd grid side and a potential formula that moves in x, y and z
        _case("shaken_105_c128", "run", 105, "complex128", "real", "shaken", 5),
        # the large single solve: stirred 256^3 (the bench workload)
        _case("stir_256_c64", "run", 256, "complex64", "real", "beam", 10),
        # a trapped cloud in a box with absorbing edges and a cutoff, reference precision
        _case("walls_256_c128", "run", 256, "complex128", "real", "walls", 4),
        # the largest solves
        _case("stir_512_c64", "run", 512, "complex64", "real", "beam", 2),
        _case("stir_512_c128", "run", 512, "complex128", "real", "beam", 1),
        # scalars, n(k) in 256 bins and Lz of a running 256^3 solve
        _case("output_256_c64", "output", 256, "complex64", "real", "beam", 1),
        # FFTs and k-space reductions called by the user's own analysis
        _case("spectrum_128_c128", "spectrum", 128, "complex128", "imaginary", "trap", 1),
        # a parameter sweep of mixed grid sizes, two convergence checks of 10 steps
        dict(name="sweep_48_160_c64", op="sweep", count=10, dtype="complex64", steps=10, checks=2),
    ]


def _case(name, op, n, dtype, kind, potential, steps):
    return dict(name=name, op=op, n=n, dtype=dtype, kind=kind, potential=potential, steps=steps)


def draw(rng):
    op = rng.choice(["run", "run", "run", "run", "closure", "output", "spectrum", "sweep"])
    if op == "sweep":
        return dict(op=op, count=rng.randint(3, 14), dtype="complex64", steps=rng.choice([5, 10, 20]),
                    checks=rng.choice([1, 2]))
    n = _smooth(int(round(math.exp(rng.uniform(math.log(24), math.log(384))))))
    dtype = rng.choice(["complex64", "complex128"])
    kind = rng.choice(["imaginary", "real", "real"])
    potential = rng.choice(["trap", "walls"] if kind == "imaginary" else ["trap", "beam", "beam", "walls", "shaken"])
    # no more work than one step of the largest listed case (a formula in x, y, z and t
    # is evaluated twice per point and step)
    if potential == "shaken":
        n = min(n, 256)
    most = int(0.6 * 512 ** 3 / (n ** 3 * (5 if potential == "shaken" else 1)))
    steps = 1 if op != "run" else max(1, min(rng.choice([1, 2, 5, 10, 20, 50]), most))
    return dict(op=op, n=n, dtype=dtype, kind=kind, potential=potential, steps=steps)


def _smooth(n):
    """The nearest grid side from n on without a prime factor above 13."""
    while True:
        m = n
        for p in (2, 3, 5, 7, 11, 13):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


# ---------------------------------------------------------------- physics of a case
def _physics(case):
    n, kind = case["n"], case["kind"]
    L = 16.0 if n <= 64 else 20.0 if n <= 96 else 24.0
    beta = 1000.0 if n <= 96 else 2000.0 if n < 200 else 4000.0
    dt = (5e-4 if kind == "imaginary" else 2.5e-4) if n < 200 else 1.25e-4
    a = beta * 1e-6 / (8 * math.pi * N_ATOMS * BOHR)          # scattering length giving beta
    return dict(n=n, L=L, dt=dt, a=a, beta=8 * math.pi * N_ATOMS * (a * BOHR) / 1e-6)


def _axes(n, L):
    x = np.linspace(-L / 2, L / 2, n, endpoint=False)
    return x, 2 * np.pi * np.fft.fftfreq(n, L / n)


def _beam(dt):
    """Amplitude 20, width 0.5, orbit radius 2, rate ramped 0 -> 1 over 200 steps."""
    return dict(amp=20.0, width=0.5, radius=2.0, omega=1.0, t_ramp=200 * dt)


# a plug moved through the cloud along z and an axial modulation of the trap
SHAKEN = "8*exp(-(x**2+y**2+(z-1.5*sin(4*t))**2)/0.64)+0.3*sin(10*t)*z**2"
STEP0 = 60          # steps already taken by a real-time solve when the call is made


def _box(case, p):
    return dict(R=0.42 * p["L"], L=0.84 * p["L"], wall_thickness=0.6, trap_depth=60.0)


def _absorber(p):
    return dict(activation_distance=0.08 * p["L"], strength=15.0)


def _k_cut(p):
    return 0.8 * math.pi * p["n"] / p["L"]


def _state(n, L, beta, kind, dtype, seed):
    """A Gaussian (ground-state search) or a trapped cloud with the quadrupole flow that
    stirring drives (real time) times (1 + 0.01 complex noise), normalised, in the
    case's precision."""
    x = torch.from_numpy(_axes(n, L)[0]).cuda()
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    noise = torch.randn((n, n, n, 2), generator=g, device="cuda", dtype=torch.float64)
    X, Y, Z = x[:, None, None], x[None, :, None], x[None, None, :]
    if kind == "imaginary":
        psi = torch.exp(-(X * X + Y * Y + Z * Z) / 2)
    else:
        mu = (15 * beta * math.sqrt(TRAP[1] * TRAP[2]) / (8 * math.pi)) ** 0.4
        psi = torch.sqrt(torch.clamp(mu - (X * X + TRAP[1] * Y * Y + TRAP[2] * Z * Z), min=0.0) / beta)
        psi = psi * torch.polar(torch.ones_like(X * Y), 0.3 * X * Y)
    psi = psi * torch.complex(1 + 0.01 * noise[..., 0], 0.01 * noise[..., 1])
    dx = float(x[1] - x[0])
    psi = psi / torch.sqrt((psi.abs() ** 2).sum() * dx ** 3)
    return psi.to(getattr(torch, dtype)).contiguous()


def _sweep_instances(case, seed):
    """Sizes drawn as in the parameter sweep: 48^3 to 160^3 with their boxes."""
    sizes = [(48, 6.0), (64, 8.0), (96, 10.0), (128, 12.0), (160, 14.0)]
    shape = np.random.default_rng(case["count"])             # the grids belong to the case
    rng = np.random.default_rng(int(seed))                   # the physics to the inputs
    out = []
    for i in range(case["count"]):
        n, L = sizes[i] if i < 5 else sizes[shape.integers(5)]
        beta = 2 * float(math.exp(rng.uniform(math.log(100.0), math.log(5000.0))))
        ly, lz = (float(v) for v in rng.uniform(0.5, 2.0, 2))
        out.append(dict(n=n, L=2 * L, beta=beta, dt=5e-4, trap=(1.0, ly * ly, lz * lz), seed=int(seed) + i))
    return out


def _trap_expr(trap):
    return f"{trap[0]!r}*x**2+{trap[1]!r}*y**2+{trap[2]!r}*z**2"


# ---------------------------------------------------------------- what the program holds
def prepare(case, seed):
    if case["op"] == "sweep":
        insts = _sweep_instances(case, seed)
        batch = Batch([Instance(n=i["n"], simulation_range=i["L"], beta=i["beta"], dt=i["dt"],
                                static_expr=_trap_expr(i["trap"])) for i in insts],
                      dtype=getattr(torch, case["dtype"]))
        psis = [_state(i["n"], i["L"], i["beta"], "imaginary", case["dtype"], i["seed"]) for i in insts]
        batch.bind(psis)
        return dict(case=case, batch=batch, psis=psis)
    p = _physics(case)
    psi = _state(p["n"], p["L"], p["beta"], case["kind"], case["dtype"], seed)
    x, k = helper.get_grids(p["n"], p["L"])
    if case["op"] == "spectrum":
        return dict(case=case, psi=psi, x=x, k=k)
    pot, real = case["potential"], case["kind"] == "real"
    walls = pot == "walls"
    st = Stage(simulation_range=p["L"], x_array=x, k_array=k, N_grids=p["n"], type=case["kind"],
               steps=case["steps"], dt=p["dt"], initial_state=dict(type="continue"),
               box_params=dict(activate=walls, **_box(case, p)),
               absorber_params=dict(activate=walls and real, **_absorber(p)),
               noise_params=dict(activate=False), cloud_params=dict(a=p["a"], N_atom=N_ATOMS),
               monitor_params={}, save_params={},
               potential_params=dict(
                   static=dict(activate=True, expression=cuda_expression(_trap_expr(TRAP))),
                   dynamic=dict(activate=pot == "shaken", expression=cuda_expression(SHAKEN, time_dependent=True))),
               k_cut_params=dict(activate=walls and real, k_cut=_k_cut(p)),
               precision=case["dtype"], beam=Beam(**_beam(p["dt"])) if pot == "beam" else None,
               nk_bins=256 if case["op"] == "output" else 0)
    st.prepare(psi)
    state = dict(case=case, stage=st, t=STEP0 * p["dt"])
    if case["op"] == "output":
        state["plan"] = st.propagator.binding.plan(st)[0]
    return state


def run(state):
    case = state["case"]
    op = case["op"]
    if op == "sweep":
        b, count = state["batch"], case["count"]
        live, steps, last = np.ones(count, np.int32), np.zeros(count, np.int64), np.full(count, np.nan)
        diag = b.run(case["steps"], case["checks"], 0.0, 10 ** 6, live, steps, last)
        return dict(psi=state["psis"], diagnostics=diag, steps=steps)
    if op == "spectrum":
        psi, x, k = state["psi"], state["x"], state["k"]
        helper.normalise(psi, x)
        f = helper.fftn(psi, x)
        e = helper.get_E(f, x, k)
        nk = nk_extraction.nk_extraction(f, x, k)
        return dict(psi=psi, psi_k=f, back=helper.ifftn(f, x), N=helper.get_N(psi, x), E=e, Nk=nk["Nk"],
                    counts=nk["counts"])
    st = state["stage"]
    if op == "closure":
        return st.propagator(st, state["t"]) if st.propagator.dynamic else st.propagator(st)
    if op == "run":
        return st.propagator.run(st, case["steps"], STEP0 if case["kind"] == "real" else 0)
    plan = state["plan"]
    out = plan.diagnostics(st.psi, t=state["t"], nk=True)
    out["Lz"] = plan.angular_momentum(st.psi)
    return out


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    """Bytes: every step reads and writes the state once (and reads an array
    potential once); an output or a transform reads its state once and writes its
    results once.  Operations: 5 M log2 M per 3-D transform, 20 per point and local
    half-step or reduction, 12 per point and kinetic factor."""
    s = 8 if case["dtype"] == "complex64" else 16
    if case["op"] == "sweep":
        steps = case["steps"] * case["checks"]
        sizes = [i["n"] ** 3 for i in _sweep_instances(case, 0)]
        return dict(bytes=float(sum(m * s * (2 * steps + case["checks"]) for m in sizes)),
                    flops=float(sum((steps * 2 + case["checks"]) * _fft_ops(m) + 60.0 * m * steps for m in sizes)))
    m = case["n"] ** 3
    if case["op"] == "output":
        return dict(bytes=float(m * s), flops=5.0 / 3.0 * _fft_ops(m) + 60.0 * m)
    if case["op"] == "spectrum":
        return dict(bytes=float(m * s * 4), flops=2 * _fft_ops(m) + 40.0 * m)
    arrays = 0
    if case["potential"] == "walls":
        arrays = s // 2 if case["kind"] == "imaginary" else s
    per_point = 2 * 20.0 + 12.0 + (40.0 if case["potential"] == "shaken" else 0.0)
    return dict(bytes=float(case["steps"] * m * (2 * s + arrays)),
                flops=float(case["steps"] * (2 * _fft_ops(m) + per_point * m)))


def _fft_ops(m):
    return 5.0 * m * math.log2(m)


# ---------------------------------------------------------------- the same in 64 bits
def exact(case, seed):
    if case["op"] == "sweep":
        psis, diags = [], []
        for i in _sweep_instances(case, seed):
            psi = _state(i["n"], i["L"], i["beta"], "imaginary", case["dtype"], i["seed"]).to(torch.complex128)
            phys = dict(n=i["n"], L=i["L"], dt=i["dt"], beta=i["beta"])
            V, _ = _potential(phys, i["trap"], "trap", "imaginary", None, 0.0)
            for _ in range(case["steps"] * case["checks"]):
                psi = _step(psi, phys, V, None, "imaginary", None)
            psis.append(psi)
            diags.append(list(_scalars(psi, phys, V).values()))
        return dict(psi=psis, diagnostics=np.array(diags), steps=None)
    p = _physics(case)
    psi = _state(p["n"], p["L"], p["beta"], case["kind"], case["dtype"], seed).to(torch.complex128)
    x, k = _axes(p["n"], p["L"])
    dx = x[1] - x[0]
    if case["op"] == "spectrum":
        psi = psi / torch.sqrt((psi.abs() ** 2).sum() * dx ** 3)
        f = torch.fft.fftn(psi)
        Nk, e = _shells(f, p, 0)
        return dict(psi=psi, psi_k=f, back=psi, N=float((psi.abs() ** 2).sum() * dx ** 3), E=e, Nk=Nk, counts=None)
    pot, kind = case["potential"], case["kind"]
    if case["op"] == "output":
        V, _ = _potential(p, TRAP, pot, kind, case, STEP0 * p["dt"])
        out = _scalars(psi, p, V)
        out["Nk"], _ = _shells(torch.fft.fftn(psi), p, 256)
        out["counts"] = None
        out["Lz"] = _angular(psi, p)
        return out
    kc = _k_cut(p) if pot == "walls" and kind == "real" else None
    step0 = STEP0 if kind == "real" else 0
    for i in range(case["steps"]):
        V, G = _potential(p, TRAP, pot, kind, case, (step0 + i) * p["dt"] + p["dt"] / 2)
        psi = _step(psi, p, V, G, kind, kc)
    return psi


def _grid(v):
    v = torch.from_numpy(np.ascontiguousarray(v)).cuda()
    return v[:, None, None], v[None, :, None], v[None, None, :]


def _potential(p, trap, pot, kind, case, t):
    """(V, Gamma) on the grid at time t, Gamma the absorber's loss rate or None."""
    X, Y, Z = _grid(_axes(p["n"], p["L"])[0])
    V = trap[0] * X * X + trap[1] * Y * Y + trap[2] * Z * Z
    if pot == "beam":
        b = _beam(p["dt"])
        m = min(t, b["t_ramp"])
        th = b["omega"] * (m * m / (2 * b["t_ramp"]) + t - m)
        r2 = (X - b["radius"] * math.cos(th)) ** 2 + (Y - b["radius"] * math.sin(th)) ** 2
        V = V + b["amp"] * torch.exp(-r2 / b["width"] ** 2)
    elif pot == "shaken":
        V = V + 8 * torch.exp(-(X * X + Y * Y + (Z - 1.5 * math.sin(4 * t)) ** 2) / 0.64)
        V = V + 0.3 * math.sin(10 * t) * Z * Z
    elif pot == "walls":
        b = _box(case, p)
        tube = torch.exp(-(torch.sqrt(X ** 2 + Y ** 2) - b["R"]) ** 2 / (2 * b["wall_thickness"] ** 2))
        cap = torch.exp(-(torch.abs(Z) - b["L"] / 2) ** 2 / (2 * b["wall_thickness"] ** 2))
        V = V + torch.maximum(tube, cap) * b["trap_depth"]
        if kind == "real":
            a, half = _absorber(p), p["L"] / 2
            ramp = sum(torch.clamp(a["activation_distance"] - (half + s * q), min=0)
                       for q in (X, Y, Z) for s in (1, -1))
            return V, ramp * a["strength"]
    return V, None


def _local(psi, p, V, G, kind):
    h = p["dt"] / 2
    e = (V + p["beta"] * (psi.real ** 2 + psi.imag ** 2)) * h
    if kind == "imaginary":
        return psi * torch.exp(-e)
    a = torch.exp(-G * h) if G is not None else torch.ones_like(e)
    return psi * torch.polar(a.expand_as(e).contiguous(), -e)


def _step(psi, p, V, G, kind, k_cut):
    KX, KY, KZ = _grid(_axes(p["n"], p["L"])[1])
    psi = torch.fft.fftn(_local(psi, p, V, G, kind))
    if kind == "imaginary":
        for K in (KX, KY, KZ):
            psi *= torch.exp(-K * K * p["dt"])
    else:
        for K in (KX, KY, KZ):
            psi *= torch.polar(torch.ones_like(K), -K * K * p["dt"])
        if k_cut is not None:
            psi[KX * KX + KY * KY + KZ * KZ > k_cut * k_cut] = 0
    psi = _local(torch.fft.ifftn(psi), p, V, G, kind)
    if kind == "imaginary":
        psi /= torch.sqrt((psi.abs() ** 2).sum() * (p["L"] / p["n"]) ** 3)
    return psi


def _scalars(psi, p, V):
    dx3, M = (p["L"] / p["n"]) ** 3, p["n"] ** 3
    rho = psi.real ** 2 + psi.imag ** 2
    KX, KY, KZ = _grid(_axes(p["n"], p["L"])[1])
    f = torch.fft.fftn(psi)
    N = float(rho.sum()) * dx3
    kin = float(((KX * KX + KY * KY + KZ * KZ) * (f.real ** 2 + f.imag ** 2)).sum()) * dx3 / M
    e_pot = float((V * rho).sum()) * dx3
    e_int = 0.5 * p["beta"] * float((rho * rho).sum()) * dx3
    return dict(N=N, E_kin=kin, E_pot=e_pot, E_int=e_int, E=kin + e_pot + e_int,
                mu=(kin + e_pot + 2 * e_int) / N)


def _shells(f, p, bins):
    """Shell sums of the spectrum and its kinetic energy."""
    n, k = p["n"], _axes(p["n"], p["L"])[1]
    KX, KY, KZ = _grid(k)
    kk = KX * KX + KY * KY + KZ * KZ
    w = (f.real ** 2 + f.imag ** 2) * ((p["L"] / n) ** 3 / n ** 3)
    dk = abs(float(k[1] - k[0]))
    if bins:
        nb, width = bins, math.sqrt(3) * (n // 2) * dk / (bins - 1)
    else:
        nb, width = int(math.floor(math.sqrt(3) * (n // 2) + 0.5)) + 1, dk
    shell = torch.clamp(torch.floor(torch.sqrt(kk) / width + 0.5).long(), max=nb - 1)
    Nk = torch.zeros(nb, dtype=torch.float64, device="cuda")
    Nk.index_add_(0, shell.reshape(-1), w.reshape(-1))
    return Nk.cpu().numpy(), float((kk * w).sum())


def _angular(psi, p):
    x, k = _axes(p["n"], p["L"])
    X, Y, _ = _grid(x)
    KX, KY, _ = _grid(k)
    py = torch.fft.ifftn(KY * torch.fft.fftn(psi, dim=1), dim=1)
    lz = float((psi.conj() * X * py).sum().real)
    px = torch.fft.ifftn(KX * torch.fft.fftn(psi, dim=0), dim=0)
    return (lz - float((psi.conj() * Y * px).sum().real)) * (p["L"] / p["n"]) ** 3
