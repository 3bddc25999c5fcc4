"""Timed work of the KPM path through its public entry points.

Each case is one call (or one round of requests) as a TBTK user's program
makes it: a Hamiltonian on a square, honeycomb or Rashba lattice with spin,
t = 1, J = 0.5, on-site disorder drawn from [-1, 1], and

* ``greens``   PropertyExtractor.calculateGreensFunctions: one source, the
  Green's functions to a list of indices (one recursion in the reference's
  arithmetic, then the energy sums);
* ``ldos``     PropertyExtractor.calculateLDOS of a list of sites, at FP64
  (TBTK's own precision) or at the mixed precisions;
* ``spin``     PropertyExtractor.calculateSpinPolarizedLDOS;
* ``density``  a self-consistency step: the model has changed, so setModel
  with the new Hamiltonian, then calculateDensity of some sites;
* ``sums``     generateGreensFunction of coefficients in hand;
* ``server``   a round of LDOS and Green's-function requests for models of
  different sizes at one Server.

The sizes run from the 30x30 known-answer lattice to the 2048x2048 lattice
of the benchmark.  ``run`` returns what the call returns: host arrays.
"""
import math

import numpy as np
import torch

from tbtk_b200 import kpm

BROADENING = 1e-3
J, W, RASHBA = 0.5, 2.0, 0.3
PRECISIONS = {"fp64": kpm.FP64, "mixed": kpm.MIXED, "mixed_direct": kpm.MIXED_DIRECT}


# ------------------------------------------------------------------ cases
def listed():
    def case(name, call, lattice, Lx, Ly, M, E, sites, precision="fp64", periodic=True,
             scale=12.0, type="Retarded"):
        return dict(name=name, call=call, lattice=lattice, Lx=Lx, Ly=Ly, M=M, E=E, sites=sites,
                    precision=precision, periodic=periodic, scale=scale, type=type)

    return [
        # the smallest call: G(E) at one index of TBTK's 30x30 example
        case("greens_30x30", "greens", "square", 30, 30, 1000, 1000, 1, periodic=False, scale=10.0),
        # propagation from one source to 32 indices of a ragged honeycomb flake
        case("greens_honeycomb_23x31_32to", "greens", "honeycomb", 23, 31, 777, 500, 32,
             periodic=False, type="NonPrincipal"),
        # a line cut of the LDOS across the 30x30 lattice, at TBTK's precision
        case("ldos_fp64_30x30_30", "ldos", "square", 30, 30, 1000, 1000, 30, periodic=False,
             scale=10.0),
        # a few sites of a small disordered flake at the mixed precision
        case("ldos_mixed_honeycomb_45x37_12", "ldos", "honeycomb", 45, 37, 1024, 1000, 12, "mixed"),
        # an ordinary LDOS map: 64 sites of a 256x256 lattice, high resolution
        case("ldos_mixed_256x256_64", "ldos", "square", 256, 256, 2048, 1000, 64, "mixed"),
        # complex Hamiltonian (Rashba), 128 sites in one batch
        case("ldos_mixed_rashba_512x512_128", "ldos", "rashba", 512, 512, 1024, 1000, 128, "mixed"),
        # the plain form: one site of a large lattice, one vector per recursion
        case("ldos_fp64_1024x1024_1", "ldos", "square", 1024, 1024, 1000, 1000, 1),
        # the benchmark's lattice and batch at a shorter expansion
        case("ldos_mixed_2048x2048_64", "ldos", "square", 2048, 2048, 512, 2000, 64, "mixed"),
        # spin texture of a Rashba lattice of odd sides: 8 sites, 16 sources
        case("spin_fp64_rashba_301x203_8", "spin", "rashba", 301, 203, 1000, 500, 8),
        # a self-consistency step on a changed model
        case("density_fp64_200x200_4", "density", "square", 200, 200, 512, 1000, 4, periodic=False),
        # energy sums alone: 64 coefficient vectors at full resolution
        case("sums_64x4096x2000", "sums", "square", 3, 3, 4096, 2000, 64),
        # the LDOS service: 24 uneven models, L in [16, 256], M in {512, ..., 4096}
        dict(name="server_uneven_24", call="server", models=24, pick=4, Lmin=16, Lmax=256,
             Mmax=4096, E=1000, scale=12.0),
    ]


def draw(rng):
    """One more case of the listed ranges."""
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        call = rng.choice(["greens", "ldos", "ldos", "ldos", "ldos", "spin", "density", "sums",
                           "server"])
        if call == "server":
            Lmin = log(16, 64)
            case = dict(call=call, models=rng.randint(4, 24), pick=rng.randrange(1 << 20), Lmin=Lmin,
                        Lmax=log(Lmin + 8, 256), Mmax=rng.choice([1024, 2048, 4096]),
                        E=log(300, 1000), scale=12.0)
        else:
            lattice = rng.choice(["square", "honeycomb", "rashba"])
            if call == "spin":
                lattice = rng.choice(["square", "rashba"])
            precision = "fp64"
            if call == "ldos":
                precision = rng.choice(["fp64", "fp64", "mixed", "mixed", "mixed", "mixed_direct"])
            elif call in ("spin", "density"):
                precision = rng.choice(["fp64", "fp64", "mixed"])
            side = {"greens": 1024, "ldos": 2048, "spin": 512, "density": 400, "sums": 3}[call]
            L = 3 if call == "sums" else log(20, side)
            case = dict(call=call, lattice=lattice, Lx=max(3, int(L * rng.uniform(0.7, 1.3))), Ly=L,
                        M=log(200, 4096), E=log(300, 2000),
                        sites=log(1, {"greens": 64, "ldos": 128, "spin": 16, "density": 16,
                                      "sums": 64}[call]),
                        precision=precision, periodic=rng.random() < 0.5, scale=12.0,
                        type=rng.choice(["Retarded", "Advanced", "Principal", "NonPrincipal"]))
        if _cost(case) <= 0.4:
            return case


def _orbitals(case):
    return 4 if case["lattice"] == "honeycomb" else 2


def _sizes(case):
    """Rows, entries (as of a periodic lattice), sources and recursion steps."""
    N = case["Lx"] * case["Ly"] * _orbitals(case)
    nnz = N * {"square": 5, "rashba": 9, "honeycomb": 4}[case["lattice"]]
    B = {"greens": 1, "spin": 2 * case["sites"]}.get(case["call"], case["sites"])
    halved = case["call"] == "ldos" and case["precision"] == "mixed"
    return N, nnz, B, case["M"] // 2 if halved else case["M"] - 1


def _value_bytes(case):
    if case["precision"] == "fp64":
        return 16
    return 8 if case["lattice"] == "rashba" else 4


def _recursion_work(N, nnz, B, steps, vec, out_bytes, real):
    """A step reads the matrix once and moves three vectors of every source;
    a recursion whose matrix and two vectors fit the 126 MB cache needs them
    from memory only once."""
    matrix = nnz * ((8 if real else 16) + 4) + 4 * N
    state = matrix + 2 * N * B * vec
    if state <= 126e6:
        nbytes = matrix + out_bytes
    else:
        nbytes = steps * (matrix + 3 * N * B * vec) + out_bytes
    return nbytes, steps * B * (nnz * (2 if real else 8) + N * (1 if real else 2))


def _server_models(case):
    """(lattice, Lx, Ly, sites, M) of each model and whether its request asks
    for Green's functions."""
    r = np.random.Generator(np.random.PCG64(case["pick"]))
    out = []
    for i in range(case["models"]):
        lattice = ("square", "honeycomb", "square", "rashba")[i % 4]
        L = int(r.integers(case["Lmin"], case["Lmax"] + 1))
        Ms = [m for m in (512, 1024, 2048, 4096) if m <= case["Mmax"]]
        out.append((lattice, L, L + int(r.integers(0, 5)), int(r.integers(1, 17)), int(r.choice(Ms)),
                    i % 6 == 5))
    return out


def _model_case(case, model):
    lattice, Lx, Ly, sites, M, _ = model
    return dict(case, lattice=lattice, Lx=Lx, Ly=Ly, sites=sites, M=M, periodic=True, call="ldos",
                precision="mixed")


def work(case):
    if case["call"] == "server":
        nbytes = flops = 0
        for model in _server_models(case):
            N, nnz, B, steps = _sizes(_model_case(case, model))
            if model[5]:
                steps = model[4] - 1
            b, f = _recursion_work(N, nnz, B, steps, 4 if model[0] != "rashba" else 8,
                                   8 * B * case["E"], model[0] != "rashba")
            nbytes, flops = nbytes + b, flops + f + 2 * B * model[4] * case["E"]
        return {"bytes": nbytes, "flops": flops}
    M, E, K = case["M"], case["E"], case["sites"]
    if case["call"] == "sums":
        return {"bytes": 16 * (M * E + K * M + K * E), "flops": 4 * K * M * E}
    N, nnz, B, steps = _sizes(case)
    outs = 4 * K if case["call"] == "spin" else K
    real = case["lattice"] != "rashba" and case["precision"] != "fp64"
    nbytes, flops = _recursion_work(N, nnz, B, steps, _value_bytes(case),
                                    outs * (8 if case["call"] in ("ldos", "density") else 16) * E, real)
    if case["call"] == "density":
        nbytes += 20 * nnz  # the new Hamiltonian, from the host
    return {"bytes": nbytes, "flops": flops + outs * M * E * (2 if case["call"] == "ldos" else 4)}


def _cost(case):
    """Rough seconds of a pass, to keep drawn cases within the listed range."""
    if case["call"] == "sums":
        return 0.01
    if case["call"] == "server":
        models = [(_model_case(case, m), m) for m in _server_models(case)]
        return sum(_cost(dict(c, M=2 * m[4] if m[5] else m[4])) for c, m in models) / 4
    N, nnz, B, steps = _sizes(case)
    vec = _value_bytes(case)
    return steps * max(6e-6, (nnz * 20 + 3 * N * B * vec) / (3e12 if case["lattice"] == "rashba" else 4.5e12))


# ------------------------------------------------------------------ inputs
def _rng(seed, k=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * seed + k)
    return g


def _rows(case, seed):
    """The Hamiltonian by rows: columns ascending, [N][k] with absent entries
    last (column N), and its values."""
    Lx, Ly, kind, periodic = case["Lx"], case["Ly"], case["lattice"], case["periodic"]
    n_orb = _orbitals(case)
    N = Lx * Ly * n_orb
    b = torch.arange(N, device="cuda", dtype=torch.int64)
    s, cell = b % 2, b // n_orb
    x, y = cell // Ly, cell % Ly
    v = (torch.rand(N // 2, generator=_rng(seed), device="cuda", dtype=torch.float64) - 0.5) * W
    diag = -J * 2.0 * (0.5 - s) + v[b // 2]
    complex_ = kind == "rashba"
    dtype = torch.complex128 if complex_ else torch.float64
    cols, vals = [b], [diag.to(dtype)]

    def hop(dx, dy, orb, value):
        xx, yy = x + dx, y + dy
        col = ((xx % Lx) * Ly + yy % Ly) * n_orb + orb
        if not periodic:
            col = torch.where((xx >= 0) & (xx < Lx) & (yy >= 0) & (yy < Ly), col, N)
        cols.append(col)
        vals.append(value if isinstance(value, torch.Tensor) else torch.full((N,), value, device="cuda", dtype=dtype))

    if kind == "honeycomb":
        a = (b // 2) % 2
        other = (1 - a) * 2 + s
        d = torch.where(a == 0, -1, 1)
        hop(0, 0, other, -1.0)
        hop(d, 0, other, -1.0)
        hop(0, d, other, -1.0)
    else:
        for dx, dy in ((1, 0), (-1, 0), (0, 1), (0, -1)):
            hop(dx, dy, s, -1.0)
            if complex_:
                # i alpha (sigma x d)_z between opposite spins
                if dx:
                    f = torch.where(s == 0, float(dx), -float(dx)) * RASHBA
                    hop(dx, dy, 1 - s, f.to(dtype))
                else:
                    hop(dx, dy, 1 - s, complex(0.0, -dy * RASHBA))
    col, order = torch.sort(torch.stack(cols, 1), dim=1)
    return col, torch.gather(torch.stack(vals, 1), 1, order), N


def _csr(case, seed):
    """Host CSR as TBTK's getSparseMatrix gives it."""
    col, val, N = _rows(case, seed)
    keep = col < N
    rowptr = torch.zeros(N + 1, device="cuda", dtype=torch.int64)
    rowptr[1:] = torch.cumsum(keep.sum(1), 0)
    return (rowptr.to(torch.int32).cpu().numpy().view(np.uint32),
            col[keep].to(torch.int32).cpu().numpy().view(np.uint32),
            val[keep].to(torch.complex128).cpu().numpy())


def _sites(case, seed):
    """Distinct lattice sites, spin up."""
    n = case["Lx"] * case["Ly"] * _orbitals(case) // 2
    r = np.random.Generator(np.random.PCG64(seed + 17))
    return (2 * r.choice(n, size=case["sites"], replace=case["sites"] > n)).astype(np.uint32)


def _window(case):
    """Energies of the open grid (-s, s)."""
    s, E = case["scale"], case["E"]
    d = 2 * s / (E + 1)
    return -s + d, s - d


def _occupation(case):
    """Fermi function at mu = 0.1, kT = 0.05, at the window's energies."""
    lo, hi = _window(case)
    return 1.0 / (np.exp(np.clip((np.linspace(lo, hi, case["E"]) - 0.1) / 0.05, -700, 700)) + 1.0)


def _damping(M):
    lam = BROADENING * M
    return np.sinh(lam * (1 - np.arange(M) / M)) / np.sinh(lam)


def _coefficients(case, seed):
    """Damped coefficients with the decay of a disordered lattice's."""
    r = np.random.Generator(np.random.PCG64(seed + 29))
    K, M = case["sites"], case["M"]
    c = (r.standard_normal((K, M)) + 1j * r.standard_normal((K, M))) / np.sqrt(1.0 + np.arange(M))
    c[:, 0] = 1.0
    return c * _damping(M)


def prepare(case, seed):
    if case["call"] == "server":
        lo, hi = _window(case)
        srv = kpm.Server(case["Mmax"], np.linspace(lo, hi, case["E"]), hbm_budget=8 << 30)
        requests = []
        for i, model in enumerate(_server_models(case)):
            mc = _model_case(case, model)
            sites = _sites(mc, seed + i)
            lanes = 1 << (len(sites) - 1).bit_length()
            requests.append((srv.add_model(*_csr(mc, seed + 100 * i), case["scale"], lanes), sites,
                             model[4], model[5]))
        return {"case": case, "server": srv, "requests": requests}
    solver = kpm.ChebyshevExpander()
    solver.setScaleFactor(case["scale"])
    solver.setNumCoefficients(case["M"])
    solver.setBroadening(BROADENING)
    solver.setPrecision(PRECISIONS[case["precision"]])
    pe = kpm.PropertyExtractor(solver)
    pe.setEnergyWindow(*_window(case), case["E"])
    state = {"case": case, "solver": solver, "pe": pe}
    if case["call"] == "sums":
        state["coefficients"] = _coefficients(case, seed)
        return state
    state["csr"] = _csr(case, seed)
    solver.setModel(state["csr"])
    state["sites"] = _sites(case, seed)
    state["occupation"] = _occupation(case)
    return state


def run(state):
    case = state["case"]
    call = case["call"]
    if call == "server":
        srv = state["server"]
        ids = []
        for model, sites, M, greens in state["requests"]:
            if greens:
                ids.append(srv.submit_greens(model, sites, np.full_like(sites, sites[0]), M, BROADENING,
                                             "Retarded"))
            else:
                ids.append(srv.submit(model, sites, M, BROADENING))
        return [srv.wait(i)[0] for i in ids]
    solver, pe = state["solver"], state["pe"]
    if call == "sums":
        return solver.generateGreensFunction(state["coefficients"], case["type"])
    sites = state["sites"]
    if call == "greens":
        return pe.calculateGreensFunctions(sites, int(sites[0]), case["type"])
    if call == "ldos":
        return pe.calculateLDOS(sites)
    if call == "spin":
        return pe.calculateSpinPolarizedLDOS(sites, sites + 1)
    solver.setModel(state["csr"])
    return pe.calculateDensity(sites, state["occupation"])


# ------------------------------------------------------------------ in 64 bits
def _recursion(case, seed, sources, targets, M, doubling):
    """Moments [len(targets)][M] of pairs (to row, source number)."""
    col, val, N = _rows(case, seed)
    val = torch.where(col < N, val, torch.zeros((), device="cuda", dtype=val.dtype)) * (2 / case["scale"])
    col = torch.where(col < N, col, 0)
    K = len(targets)
    to = torch.tensor([t for t, _ in targets], device="cuda")
    own = torch.tensor([b for _, b in targets], device="cuda")
    mu = torch.zeros(M, K, device="cuda", dtype=torch.complex128)
    chunk = max(1, int(6e9 / (N * val.element_size())))
    for b0 in range(0, len(sources), chunk):
        src = torch.tensor(sources[b0:b0 + chunk], device="cuda")
        pick = torch.nonzero((own >= b0) & (own < b0 + len(src)))[:, 0]
        rows, cols = to[pick], own[pick] - b0
        prev = torch.zeros(N, len(src), device="cuda", dtype=val.dtype)
        prev[src, torch.arange(len(src), device="cuda")] = 1.0

        def apply(x, acc):
            for k in range(col.shape[1]):
                acc.addcmul_(x.index_select(0, col[:, k]), val[:, k, None])
            return acc

        mu[0, pick] = prev[rows, cols].to(torch.complex128)
        cur = apply(prev, torch.zeros_like(prev)).mul_(0.5)
        if M > 1:
            mu[1, pick] = cur[rows, cols].to(torch.complex128)
        if not doubling:
            for n in range(2, M):
                prev, cur = cur, apply(cur, prev.neg_())
                mu[n, pick] = cur[rows, cols].to(torch.complex128)
            continue

        def dot(a, b):
            return torch.linalg.vecdot(a, b, dim=0)[cols].to(torch.complex128)

        n = 1  # prev = j_{n-1}, cur = j_n
        while 2 * n < M:
            mu[2 * n, pick] = 2 * dot(cur, cur) - mu[0, pick]
            if 2 * n + 1 >= M:
                break
            prev, cur = cur, apply(cur, prev.neg_())
            n += 1
            mu[2 * n - 1, pick] = 2 * dot(cur, prev) - mu[1, pick]
    return mu.t().contiguous()


def _sum(case, mu, damped=False):
    """sum c_n cos(n theta)/(1 + delta_n0) and the sine sum, [K][E], and the
    prefactor 2/(s sin theta)."""
    M, s = mu.shape[1], case["scale"]
    lo, hi = _window(case)
    x = (lo + (hi - lo) / (case["E"] - 1) * torch.arange(case["E"], device="cuda", dtype=torch.float64)) / s
    c = mu if damped else mu * torch.from_numpy(_damping(M)).cuda()
    c = c.clone()
    c[:, 0] *= 0.5
    phase = torch.arange(M, device="cuda", dtype=torch.float64)[:, None] * torch.arccos(x)[None, :]
    cs, sn = torch.cos(phase), torch.sin(phase)
    mm = lambda t: torch.complex(c.real.contiguous() @ t, c.imag.contiguous() @ t)  # noqa: E731
    return mm(cs), mm(sn), 2.0 / (s * torch.sqrt(1 - x * x))


def _greens(case, mu, type, damped=False):
    C, S, a = _sum(case, mu, damped)
    if type == "Retarded":
        return -a * (S + 1j * C)
    if type == "Advanced":
        return -a * (S - 1j * C)
    return a * S if type == "Principal" else 1j * a * C


def exact(case, seed):
    if case["call"] == "server":
        out = []
        for i, model in enumerate(_server_models(case)):
            mc = _model_case(case, model)
            sites = [int(v) for v in _sites(mc, seed + i)]
            if model[5]:
                mu = _recursion(mc, seed + 100 * i, sites[:1], [(t, 0) for t in sites], model[4], False)
                out.append(_greens(mc, mu, "Retarded").cpu().numpy())
            else:
                mu = _recursion(mc, seed + 100 * i, sites, [(t, k) for k, t in enumerate(sites)],
                                model[4], True)
                out.append((_greens(mc, mu, "NonPrincipal").imag / math.pi).cpu().numpy())
        return out
    if case["call"] == "sums":
        c = torch.from_numpy(_coefficients(case, seed)).cuda()
        return _greens(case, c, case["type"], damped=True).cpu().numpy()
    sites, M = [int(v) for v in _sites(case, seed)], case["M"]
    if case["call"] == "greens":
        mu = _recursion(case, seed, sites[:1], [(t, 0) for t in sites], M, False)
        return _greens(case, mu, case["type"]).cpu().numpy()
    if case["call"] == "spin":
        sources = [s + d for s in sites for d in (0, 1)]
        targets = [(s + n // 2, 2 * k + n % 2) for k, s in enumerate(sites) for n in range(4)]
        mu = _recursion(case, seed, sources, targets, M, False)
        g = -1j * _greens(case, mu, "NonPrincipal") / math.pi
        return g.reshape(len(sites), 2, 2, case["E"]).permute(0, 3, 1, 2).contiguous().cpu().numpy()
    mu = _recursion(case, seed, sites, [(t, k) for k, t in enumerate(sites)], M, True)
    ldos = (_greens(case, mu, "NonPrincipal").imag / math.pi).cpu().numpy()
    if case["call"] == "ldos":
        return ldos
    lo, hi = _window(case)
    return (ldos * _occupation(case)).sum(1) * ((hi - lo) / (case["E"] - 1))
