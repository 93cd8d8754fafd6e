"""What is measured: the calls that a user of the field pipeline makes, each
through a public entry point, over grid levels J = 6 to 9 and catalogues of
1e4 to 4e6 points.

  project      SFCProjection.run() on host arrays: a catalogue to its field
  deposit      the same deposit for a catalogue that is on the GPU already
  window       field @ WindowFunc: smoothing of a field
  pcf          Corr_2PCF.run(): pair products and xi over a sampling grid
  terms        the (l, m) terms of the 3PCF multipoles of one field (the layer
               that a multipole run repeats): fields of all radii, all pairs
  zeta         Corr_3PCF_Multipole.run(): delta_ddd_l, rrr_l and zeta_l
  triplets     the Monte Carlo triplet sums of DDD(theta)
  density      the field's density at positions

The pair products, the summands, zeta_l, the triplet sums and the
interpolated densities are formed from float32 fields by float32 products, so
that is what they are kept in here, although some calls hand them over in
64-bit containers.
"""

import math

import numpy as np
import torch

BOX = 1000.0
DEV = "cuda"


# ---- the cases -------------------------------------------------------------
def listed():
    return [
        # the smallest full step of a study: a 200k-point sample projected at J = 7
        {"name": "project_J7", "kind": "project", "J": 7, "n": 200000, "weighted": True},
        # the deposit benchmark: 4e6 points on 512^3
        {"name": "deposit_J9", "kind": "deposit", "J": 9, "n": 4000000, "weighted": True},
        # smoothing at the largest level, and a top-hat at the default level
        {"name": "window_gaussian_J9", "kind": "window", "J": 9, "type": "gaussian", "R": 10.0, "d": 0.0},
        {"name": "window_sphere_J8", "kind": "window", "J": 8, "type": "sphere", "R": 8.0, "d": 0.0},
        # xi(s): 20 shells of a small sample, and the default 30 separations against a random catalogue
        {"name": "xi_s_J7", "kind": "pcf", "J": 7, "type": "shell", "na": 20, "nb": 1, "top": 150.0, "random": "uniform"},
        {"name": "xi_s_J9", "kind": "pcf", "J": 9, "type": "shell", "na": 30, "nb": 1, "top": 150.0, "random": "field"},
        # xi(s, mu) in 30 x 10 ring bins
        {"name": "xi_smu_J9", "kind": "pcf", "J": 9, "type": "ring", "na": 30, "nb": 10, "top": 150.0, "random": "uniform"},
        # one (l, m) term of the 15 x 15 shell run on 512^3
        {"name": "terms_J9", "kind": "terms", "J": 9, "l": 4, "m": 2, "nr": 15, "top": 160.0, "paired": False},
        # the reference's benchmark unit: one (r12, r13) sample at J = 8 up to l = 7
        {"name": "zeta_J8", "kind": "zeta", "J": 8, "lmax": 7, "nr": 2, "top": 90.0, "grid": False},
        # a 10 x 10 shell grid on a small box
        {"name": "zeta_J7", "kind": "zeta", "J": 7, "lmax": 4, "nr": 10, "top": 140.0, "grid": True},
        # DDD(theta): box-random centres x rotations for three angles
        {"name": "triplets_J9", "kind": "triplets", "J": 9, "nc": 200000, "n_rot": 100, "n_theta": 3, "r12": 20.0, "r13": 40.0},
        # densities at 1e6 positions (the counts-in-cells task's default)
        {"name": "density_J8", "kind": "density", "J": 8, "n": 1000000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["project", "deposit", "window", "window", "pcf", "pcf", "pcf", "terms", "terms", "zeta", "triplets",
                       "density"])
    J = rng.choice([6, 7, 8, 9])
    if kind == "project":
        return {"kind": kind, "J": J, "n": _log(rng, 10000, 1000000), "weighted": rng.random() < 0.5}
    if kind == "deposit":
        return {"kind": kind, "J": J, "n": _log(rng, 10000, 4000000), "weighted": rng.random() < 0.5}
    if kind == "window":
        t = rng.choice(["gaussian", "sphere", "shell", "thick_shell", "gaussian_shell", "cylinder"])
        return {"kind": kind, "J": J, "type": t, "R": round(rng.uniform(5.0, 60.0), 2), "d": round(rng.uniform(2.0, 15.0), 2)}
    if kind == "pcf":
        t = rng.choice(["shell", "shell", "thick_shell", "ring", "cylshell"])
        nb = 1 if t in ("shell", "thick_shell") else _log(rng, 4, 12)
        return {"kind": kind, "J": J, "type": t, "na": _log(rng, 5, 40), "nb": nb, "top": round(rng.uniform(60.0, 180.0), 1),
                "random": rng.choice(["uniform", "uniform", "field"])}
    if kind == "terms":
        l = rng.randint(0, 10)
        paired = rng.random() < 0.25
        return {"kind": kind, "J": J, "l": l - l % 2 if paired else l, "m": 0 if paired else rng.randint(0, l),
                "nr": rng.randint(2, 16), "top": round(rng.uniform(80.0, 180.0), 1), "paired": paired}
    if kind == "zeta":
        grid = rng.random() < 0.6
        return {"kind": kind, "J": min(J, 8), "lmax": rng.randint(1, 6), "nr": rng.randint(3, 12) if grid else 2,
                "top": round(rng.uniform(80.0, 160.0), 1), "grid": grid}
    if kind == "triplets":
        return {"kind": kind, "J": J, "nc": _log(rng, 5000, 200000), "n_rot": _log(rng, 20, 100), "n_theta": rng.randint(1, 3),
                "r12": round(rng.uniform(10.0, 60.0), 1), "r13": round(rng.uniform(20.0, 100.0), 1)}
    return {"kind": kind, "J": J, "n": _log(rng, 10000, 4000000)}


# ---- inputs ----------------------------------------------------------------
def _gen(seed, k=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 64 + k)
    return g


def _lognormal(L, g, kcut=0.5):
    """exp of a smooth Gaussian field, mean 1: a clustered density on L^3 cells."""
    white = torch.fft.rfftn(torch.randn((L, L, L), generator=g, device=DEV))
    kf = 2.0 * math.pi / BOX
    k1 = torch.fft.fftfreq(L, d=1.0 / L, device=DEV) * kf
    kz = torch.fft.rfftfreq(L, d=1.0 / L, device=DEV) * kf
    k = torch.sqrt(k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2)
    white *= torch.where(k > 0, k.clamp_min(1e-9) ** -0.75 * torch.exp(-0.5 * (k / kcut) ** 2), torch.zeros_like(k))
    f = torch.fft.irfftn(white, s=(L, L, L))
    f = torch.exp(f / f.std() - 0.5)
    return f / f.mean()


def _points(n, g, weighted):
    """n clustered positions in the box (float64) and their weights."""
    L = 128
    rho = _lognormal(L, g).reshape(-1).double()
    cdf = torch.cumsum(rho, 0)
    at = torch.searchsorted(cdf, torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * cdf[-1]).clamp_max(L ** 3 - 1)
    cell = torch.stack([at // (L * L), at // L % L, at % L], 1).double()
    pos = (cell + torch.rand((n, 3), generator=g, device=DEV, dtype=torch.float64)) * (BOX / L)
    w = torch.exp(0.3 * torch.randn(n, generator=g, device=DEV, dtype=torch.float64)) if weighted else \
        torch.ones(n, device=DEV, dtype=torch.float64)
    return pos.clamp(0.0, math.nextafter(BOX, 0.0)), w


def _eps(J, g, clustered=True):
    """Coefficients of a catalogue of about 0.03 points per cell (at least
    1e5): Poisson counts spread over three cells per axis as the scaling
    function spreads them, of unit sum."""
    L = 1 << J
    mean = max(0.03, 1e5 / L ** 3)
    lam = _lognormal(L, g) * mean if clustered else torch.full((L, L, L), mean, device=DEV)
    e = torch.poisson(lam, generator=g)
    for ax in range(3):
        e = 0.55 * e + 0.6 * torch.roll(e, -1, ax) - 0.15 * torch.roll(e, -2, ax)
    return (e / e.double().sum().item()).contiguous()


def _field(eps, J):
    """The field object that a projection hands over, around `eps`."""
    from pyhermes_gb300.phi import sample_scaling_function
    from pyhermes_gb300.sfc_field import SFCField

    L = 1 << J
    phi = sample_scaling_function("db2", 10)
    f = SFCField(threads=1, device=DEV)
    f.sfc_info = {"fin": {}, "particle_count": L ** 3 // 32, "catalog_weight_sum": 1.0, "catalog_weight_sq_sum": 1.0,
                  "raw_field_weighted_sum": 1.0, "field_integral": float(eps.double().sum().item()), "box_size": BOX,
                  "J": J, "L": L, "V": L ** 3, "scale_factor": L / BOX, "field_kind": "catalog_field",
                  "weight_normalization": "catalog", "particle_data_retrievable": False, "wavelet_mode": "db2",
                  "wavelet_level": 10, "phi_resolution": 1024, "particle_data_path": "", "particle_data_format": "",
                  "phi_support": 3, "phi_array": phi}
    f.format_sfc_params()
    f.epsilon_device = eps
    return f


def _window_len(case):
    t = case["type"]
    if t == "thick_shell":
        return {"R": case["R"], "delta_R": case["d"]}
    if t == "gaussian_shell":
        return {"R_shell": case["R"], "R_smooth": case["d"]}
    return {"R": case["R"], "H": case["d"]} if t == "cylinder" else {"R": case["R"]}


def _sampling(case):
    """The sampling grid of a pcf case: (names, first axis, second axis)."""
    a = np.linspace(case["top"] / case["na"], case["top"], case["na"])
    if case["type"] == "ring":
        return ("s", "mu"), a, np.linspace(0.0, 1.0, case["nb"])
    if case["type"] == "cylshell":
        return ("rp", "pi"), a, np.linspace(2.0, 40.0, case["nb"])
    return ("s",), a, None


def _radii(case):
    if case["kind"] == "zeta" and not case["grid"]:
        return [case["top"] * 5.0 / 9.0, case["top"]]
    return [float(r) for r in np.linspace(10.0 if case["J"] > 7 else 20.0, case["top"], case["nr"])]


def _triangles(case, seed):
    """[n_theta][n_rot, 6] offsets, in cells, of randomly turned triangles."""
    rng = np.random.default_rng(seed)
    sf = (1 << case["J"]) / BOX
    out = []
    for mu in np.linspace(-0.8, 0.9, case["n_theta"]):
        a = rng.normal(size=(case["n_rot"], 3))
        a /= np.linalg.norm(a, axis=1, keepdims=True)
        b = np.cross(a, rng.normal(size=a.shape))
        b /= np.linalg.norm(b, axis=1, keepdims=True)
        out.append(np.concatenate([case["r12"] * sf * a, case["r13"] * sf * (mu * a + math.sqrt(1 - mu * mu) * b)], 1))
    return out


def _inputs(case, seed):
    """The numbers of a case, without any of the package's objects."""
    g, J, kind = _gen(seed), case["J"], case["kind"]
    if kind in ("project", "deposit"):
        return dict(zip(("pos", "w"), _points(case["n"], g, case["weighted"])))
    d = {"eps": _eps(J, g)}
    if kind == "pcf" and case["random"] == "field":
        d["random"] = _eps(J, _gen(seed, 1), clustered=False)
    if kind == "density":
        d["pos"] = torch.rand((case["n"], 3), generator=g, device=DEV, dtype=torch.float64) * BOX
    if kind == "triplets":
        d["centers"] = torch.rand((case["nc"], 3), generator=g, device=DEV, dtype=torch.float64) * (1 << J)
        d["offsets"] = _triangles(case, seed)
    return d


def prepare(case, seed):
    from pyhermes_gb300 import kernels
    from pyhermes_gb300.phi import sample_scaling_function
    from pyhermes_gb300.window import WindowFunc

    d, J, kind = _inputs(case, seed), case["J"], case["kind"]
    s = {"case": case, "J": J}
    phi = sample_scaling_function("db2", 10)
    if kind == "project":
        s["params"] = {"SFCProjection": {"particle_pos": d["pos"].cpu().numpy(), "J": J, "box_size": BOX}}
        if case["weighted"]:
            s["params"]["SFCProjection"]["catalog_weight"] = d["w"].cpu().numpy()
        return s
    if kind == "deposit":
        s.update(pos=d["pos"], w=d["w"] / d["w"].sum(), phi=torch.as_tensor(phi, device=DEV),
                 ws=kernels.DepositWorkspace(DEV))
        return s
    s["field"] = _field(d["eps"], J)
    if kind == "window":
        s["window"] = WindowFunc({"type": case["type"], "len_args": _window_len(case)}, s["field"].sfc_info, device=DEV)
    elif kind == "pcf":
        names, a, b = _sampling(case)
        bw = {"type": case["type"]}
        if case["type"] == "thick_shell":
            bw["len_args"] = {"R": None, "delta_R": 5.0}
        elif case["type"] == "cylshell":
            bw["mapping"] = "rppi_to_RH"
        s["params"] = {"Corr_2PCF": {
            "sfc_field": s["field"], "random": _field(d["random"], J) if "random" in d else "uniform", "binning_window": bw,
            "sampling": dict(zip(names, (a.tolist(),) if b is None else (a.tolist(), b.tolist()))), "products": "xi"}}
    elif kind == "terms":
        s["phi"], s["radii"] = phi, _radii(case)
        s["lms"] = [(case["l"] + k, case["m"]) for k in range(2 if case["paired"] else 1)]
    elif kind == "zeta":
        r = _radii(case)
        samp = {"mode": "grid", "r12": r, "r13": r} if case["grid"] else {"mode": "paired", "r12": r[:1], "r13": r[1:]}
        s["params"] = {"Corr_3PCF_Multipole": {
            "sfc_field": s["field"], "random": "uniform",
            "binning_window12": {"type": "shell", "len_args": {}, "other_args": {}, "mapping": {"R": "r12"}},
            "binning_window13": {"type": "shell", "len_args": {}, "other_args": {}, "mapping": {"R": "r13"}},
            "sampling": samp, "l_min": 0, "l_max": case["lmax"], "products": "zeta_l"}}
    elif kind == "triplets":
        s.update(centers=d["centers"], offsets=d["offsets"], phi=torch.as_tensor(phi, device=DEV))
    else:
        s["pos"] = d["pos"]
    return s


def run(s):
    from pyhermes_gb300 import kernels, mc3pcf
    from pyhermes_gb300.corr2pcf import Corr_2PCF
    from pyhermes_gb300.multipole import Corr_3PCF_Multipole, MultipoleEngine
    from pyhermes_gb300.projection import SFCProjection

    case, J = s["case"], s["J"]
    kind = case["kind"]
    if kind == "project":
        return SFCProjection(s["params"]).run(save_result=False).epsilon_device
    if kind == "deposit":
        return kernels.deposit(s["pos"], s["w"], J, BOX, s["phi"], workspace=s["ws"])[0]
    if kind == "window":
        return (s["field"] @ s["window"]).epsilon_device
    if kind == "pcf":
        r = Corr_2PCF(s["params"]).run(save_result=False)
        return {k: np.float32(getattr(r, k)) for k in ("delta_dd", "rr", "xi")}
    if kind == "terms":
        e = s["field"].epsilon_device
        return MultipoleEngine(e, e, e, s["phi"], J, BOX).summands_shared(s["lms"], s["radii"]).astype(np.complex64)
    if kind == "zeta":
        r = Corr_3PCF_Multipole(s["params"]).run(save_result=False)
        return {k: np.float32(getattr(r, k)) for k in ("delta_ddd_l", "rrr_l", "zeta_l")}
    if kind == "triplets":
        e = s["field"].epsilon_device
        return np.array([mc3pcf.triplet_sum(e, e, e, J, s["centers"], o, s["phi"])[0] for o in s["offsets"]], dtype=np.float32)
    return s["field"].field_density_at_pos(s["pos"], value_unit="grid").astype(np.float32)


def work(case):
    """Inputs read once, outputs written once; the transforms at 2.5 N log2 N
    (real) or 5 N log2 N (complex) and the products that no order of the sums
    avoids."""
    J, kind = case["J"], case["kind"]
    N = 8 ** J
    lg = 3 * J
    if kind in ("project", "deposit"):
        return {"bytes": 32 * case["n"] + 4 * N, "flops": 60 * case["n"]}
    if kind == "window":
        return {"bytes": 8 * N, "flops": 5 * N * lg + 2 * N}
    if kind == "pcf":
        nf = 2 if case["random"] == "field" else 1
        return {"bytes": 4 * N * nf + 12 * case["na"] * case["nb"], "flops": nf * (2.5 * N * lg + 2 * N)}
    if kind in ("terms", "zeta"):
        nr = case["nr"]
        passes = 1 if kind == "terms" else (case["lmax"] + 1) * (case["lmax"] + 2) // 2
        pairs = nr * nr if kind == "terms" or case["grid"] else 1
        # per pass: one complex transform per radius, 63 real x complex products per cell and radius, 8 flops per cell and pair
        return {"bytes": 4 * N + 8 * pairs * passes,
                "flops": 2.5 * N * lg + passes * (nr * 5 * N * lg + 4 * 63 * nr * N + 8 * pairs * N)}
    if kind == "triplets":
        t = case["nc"] * case["n_rot"] * case["n_theta"]
        return {"bytes": 4 * N + 24 * case["nc"] + 48 * case["n_rot"] * case["n_theta"], "flops": 2 * 27 * 2 * t}
    return {"bytes": 4 * N + 28 * case["n"], "flops": 27 * 2 * case["n"]}


# ---- the same in 64 bits ----------------------------------------------------
def _phi64():
    """db2 scaling function sampled 1024 times per unit on [0, 3) (cascade)."""
    q = math.sqrt(3.0)
    h = np.array([1 + q, 3 + q, 3 - q, 1 - q]) / (4 * math.sqrt(2.0))
    c = np.array([math.sqrt(2.0) ** 10])
    for _ in range(10):
        up = np.zeros(2 * c.size + 2)
        for j in range(4):
            up[j:j + 2 * c.size:2] += c * h[j]
        c = up
    keep = 1
    for _ in range(10):
        keep = 2 * keep + 2
    left = (c.size - keep) // 2
    full = np.concatenate([[0.0], c[left:left + keep], np.zeros(max(0, 3073 - keep - 1))])
    return full[:3072]


def _power64(L):
    phi = _phi64()
    ph = np.exp(-2j * np.pi * (np.arange(L + 1) / L)[:, None] * (np.arange(3072) / 1024.0)[None, :])
    return torch.as_tensor(np.abs(ph @ phi / 1024.0) ** 2, device=DEV)


def _sinc(q):
    return torch.where(q == 0, torch.ones_like(q), torch.sin(q) / torch.where(q == 0, torch.ones_like(q), q))


def _sphere(q):
    p = torch.where(q < 0.05, torch.ones_like(q), q)
    s = 1 - q * q / 10 * (1 - q * q / 28 * (1 - q * q / 54))
    return torch.where(q < 0.05, s, 3 * (torch.sin(p) - p * torch.cos(p)) / p ** 3)


def _iso64(kind, a, b, L):
    """An isotropic window over |k|^2 = 0 .. 3 L^2 (lengths in cells)."""
    k = torch.sqrt(torch.arange(3 * L * L + 1, device=DEV, dtype=torch.float64)) * (2 * math.pi / L)
    if kind == "gaussian":
        return torch.exp(-0.5 * (k * a) ** 2)
    if kind == "sphere":
        return _sphere(k * a)
    if kind == "shell":
        return _sinc(k * a)
    if kind == "gaussian_shell":
        w = (b * b * torch.cos(k * a) + a * a * _sinc(k * a)) / (a * a + b * b)
        return w * torch.exp(-0.5 * (k * b) ** 2)
    ro, ri = a + 0.5 * b, max(a - 0.5 * b, 0.0)
    return (ro ** 3 * _sphere(k * ro) - ri ** 3 * _sphere(k * ri)) / (ro ** 3 - ri ** 3)


def _iso_kernel(tab, P, L, x):
    """The window's sum over the images of the planes x (rows) of the half grid."""
    y, z = torch.arange(L, device=DEV), torch.arange(L // 2 + 1, device=DEV)
    out = 0.0
    for a in (x, L - x):
        for b in (y, L - y):
            for c in (z, L - z):
                w = tab[(a * a)[:, None, None] + (b * b)[None, :, None] + (c * c)[None, None, :]]
                out = out + w * P[a][:, None, None] * P[b][None, :, None] * P[c][None, None, :]
    return out


def _cyl64(kind, P, L, R, H):
    """(A[x, y], B[z]) of a cylindrical window along z (lengths in cells)."""
    i, z = torch.arange(L, device=DEV), torch.arange(L // 2 + 1, device=DEV)
    A = 0.0
    for a in (i, L - i):
        for b in (i, L - i):
            q = torch.sqrt(((a * a)[:, None] + (b * b)[None, :]).double()) * (2 * math.pi * R / L)
            if kind == "cylinder":
                f = torch.where(q == 0, torch.ones_like(q), 2 * torch.special.bessel_j1(q) / torch.where(q == 0, torch.ones_like(q), q))
            else:
                f = torch.special.bessel_j0(q)
            A = A + f * P[a][:, None] * P[b][None, :]
    B = 0.0
    for c in (z, L - z):
        q = c.double() * (2 * math.pi * H / L)
        B = B + (torch.cos(q) if kind == "ring" else _sinc(q)) * P[c]
    return A, B


def _deposit64(pos, w, J):
    L = 1 << J
    phi = torch.as_tensor(_phi64(), device=DEV)
    s = pos * (L / BOX)
    c = torch.floor(s)
    f = ((s - c) * 1024).long()
    c = c.long()
    out = torch.zeros(L ** 3, device=DEV, dtype=torch.float64)
    for a in range(3):
        for b in range(3):
            for d in range(3):
                at = (((c[:, 0] - a) & (L - 1)) * L + ((c[:, 1] - b) & (L - 1))) * L + ((c[:, 2] - d) & (L - 1))
                out.index_add_(0, at, w * phi[f[:, 0] + 1024 * a] * phi[f[:, 1] + 1024 * b] * phi[f[:, 2] + 1024 * d])
    return out.view(L, L, L)


def _density64(eps, s):
    """`eps` interpolated at positions s (cells)."""
    L = eps.shape[0]
    phi = torch.as_tensor(_phi64(), device=DEV)
    c = torch.floor(s)
    f = ((s - c) * 1024).long()
    c = c.long()
    i = [[(c[:, k] - a) & (L - 1) for a in range(3)] for k in range(3)]
    p = [[phi[f[:, k] + 1024 * a] for a in range(3)] for k in range(3)]
    e, out = eps.reshape(-1), 0.0
    for a in range(3):
        for b in range(3):
            row, pab = (i[0][a] * L + i[1][b]) * L, p[0][a] * p[1][b]
            for d in range(3):
                out = out + e[row + i[2][d]].double() * (pab * p[2][d])
    return out


def _pcf64(case, d):
    J = case["J"]
    L = 1 << J
    P = _power64(L)
    eps = d["eps"].double()
    if "random" in d:
        rnd = d["random"].double()
        fields = {"delta_dd": eps - rnd, "rr": rnd}
    else:
        rho = float(eps.sum().item()) / L ** 3
        fields = {"delta_dd": eps - rho}
    _, a, b = _sampling(case)
    sf = L / BOX
    wz = torch.full((L // 2 + 1,), 2.0, device=DEV, dtype=torch.float64)
    wz[0] = wz[-1] = 1.0
    out = {}
    for name, f in fields.items():
        T = torch.fft.rfftn(f)
        T = (T.real ** 2 + T.imag ** 2) * wz
        if b is None:
            tabs = [_iso64(case["type"], s * sf, 5.0 * sf, L) for s in a]
            v = [0.0] * len(tabs)
            for x in torch.arange(L, device=DEV).split(32):
                for k, t in enumerate(tabs):
                    v[k] += float((_iso_kernel(t, P, L, x) * T[x]).sum().item())
            v = np.array(v)
        else:
            v = np.zeros((len(a), len(b)))
            for i, s in enumerate(a):
                for j, t in enumerate(b):
                    R, H = (s * math.sqrt(max(0.0, 1 - t * t)), s * t) if case["type"] == "ring" else (s, t)
                    A, B = _cyl64(case["type"], P, L, R * sf, H * sf)
                    v[i, j] = float((A * (T @ B)).sum().item())
        out[name] = v / float(L) ** 6 * sf ** 6
    if "rr" not in out:
        out["rr"] = np.full_like(out["delta_dd"], rho * rho * sf ** 6)
    out["xi"] = out["delta_dd"] / out["rr"]
    return out


def _jl64(l, x):
    """Spherical Bessel j_l: a series below 1, downward recurrence below
    l + 1, upward recurrence above."""
    x = x.double()
    small, mid = x < 1.0, x < l + 1.0
    xs = torch.where(small, x, torch.ones_like(x))
    t = torch.ones_like(x)
    for n in range(1, l + 1):
        t = t * xs / (2 * n + 1)
    series = torch.zeros_like(x)
    for n in range(14):
        series = series + t
        t = t * (-0.5 * xs * xs) / ((n + 1) * (2 * l + 2 * n + 3))
    xd = torch.where(small, torch.ones_like(x), torch.where(mid, x, torch.ones_like(x)))
    hi, cur, at = torch.zeros_like(x), torch.full_like(x, 1e-200), None
    j1 = None
    for n in range(l + 45, 0, -1):
        hi, cur = cur, (2 * n + 1) / xd * cur - hi
        if n - 1 == l:
            at = cur
        if n - 1 == 1:
            j1 = cur
    j1 = cur if j1 is None else j1
    s0, s1 = torch.sin(xd) / xd, torch.sin(xd) / xd ** 2 - torch.cos(xd) / xd
    down = torch.where(cur.abs() > j1.abs(), at * (s0 / cur), at * (s1 / j1))
    xu = torch.where(mid, torch.full_like(x, l + 1.0), x)
    p, c = torch.sin(xu) / xu, torch.sin(xu) / xu ** 2 - torch.cos(xu) / xu
    if l == 0:
        c = p
    for n in range(1, l):
        p, c = c, (2 * n + 1) / xu * c - p
    return torch.where(small, series, torch.where(mid, down, c))


def _ylm64(l, m, a, b, c):
    """Y_lm (m >= 0, Condon-Shortley) of integer vectors, and |k|^2."""
    n2 = a * a + b * b + c * c
    r = torch.sqrt(torch.where(n2 == 0, torch.ones_like(n2), n2).double())
    ct = c / r
    w = torch.complex((a / r).expand_as(r), (b / r).expand_as(r))
    p = 1.0
    for k in range(m):
        p *= -(2 * k + 1)
    p0, p1 = torch.full_like(r, p), ct * (2 * m + 1) * p
    if l == m:
        p1 = p0
    for e in range(m + 2, l + 1):
        p0, p1 = p1, ((2 * e - 1) * ct * p1 - (e + m - 1) * p0) / (e - m)
    norm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
    y = (norm * p1) * w ** m if m else torch.complex(norm * p1, torch.zeros_like(p1))
    zero = (1.0 / math.sqrt(4 * math.pi)) if l == 0 else 0.0
    return torch.where(n2 == 0, torch.full_like(y, zero), y), n2


def _gamma64():
    phi = _phi64()
    return [[float(np.sum(phi * np.roll(phi, 1024 * i) * np.roll(phi, 1024 * j)) / 1024.0) for j in range(3)] for i in range(3)]


def _summands64(eps, lms, radii, J):
    """S_lm[i, j] = 4 pi / L^3 sum_x eps(x) sum_{l1, l2} Gamma3 a_lm^i(x - l1)
    a_{l,-m}^j(x - l2) for every (l, m), with a_{l,-m} = (-1)^(l+m) conj a_lm."""
    L = eps.shape[0]
    P, G = _power64(L), _gamma64()
    spec = torch.fft.fftn(eps.double())
    i = torch.arange(L, device=DEV)
    x = 2 * math.pi * torch.sqrt(torch.arange(3 * L * L + 1, device=DEV, dtype=torch.float64)) / L
    e = eps.double()
    out = []
    for l, m in lms:
        tabs = [_jl64(l, x * (r * L / BOX)) for r in radii]
        A = torch.empty((len(radii), L ** 3), device=DEV, dtype=torch.complex128)
        for xs in i.split(max(1, (1 << 22) // (L * L))):
            part = [0.0] * len(radii)
            for ia in (xs - L, xs):
                for ib in (i - L, i):
                    for ic in (i - L, i):
                        y, n2 = _ylm64(l, m, ia[:, None, None], ib[None, :, None], ic[None, None, :])
                        y = y * (P[ia.abs()][:, None, None] * P[ib.abs()][None, :, None] * P[ic.abs()][None, None, :])
                        for k, t in enumerate(tabs):
                            part[k] = part[k] + y * t[n2]
            for k in range(len(radii)):
                A[k].view(L, L, L)[xs] = part[k]
        for k in range(len(radii)):
            A[k] = torch.fft.ifftn(A[k].view(L, L, L) * spec).reshape(-1)
        Q = torch.empty_like(A)
        sign = (-1.0) ** (l + m)
        for k in range(len(radii)):
            a3 = sign * A[k].conj().view(L, L, L)
            q = torch.zeros_like(a3)
            for u in range(3):
                fx = sum(G[u][v] * torch.roll(a3, v, 0) for v in range(3))
                for s in range(3):
                    fy = sum(G[s][v] * torch.roll(fx, v, 1) for v in range(3))
                    for t in range(3):
                        q += torch.roll(e * sum(G[t][v] * torch.roll(fy, v, 2) for v in range(3)), (-u, -s, -t), (0, 1, 2))
            Q[k] = q.reshape(-1)
        out.append((A @ Q.T).cpu().numpy() * (4 * math.pi / L ** 3))
    return np.array(out)


def exact(case, seed):
    d, J, kind = _inputs(case, seed), case["J"], case["kind"]
    L = 1 << J
    if kind in ("project", "deposit"):
        return _deposit64(d["pos"], d["w"] / d["w"].sum(), J)
    if kind == "window":
        sf = L / BOX
        P, spec = _power64(L), torch.fft.rfftn(d["eps"].double())
        if case["type"] == "cylinder":
            A, B = _cyl64("cylinder", P, L, case["R"] * sf, case["d"] * sf)
            spec *= A[:, :, None] * B
        else:
            tab = _iso64(case["type"], case["R"] * sf, case["d"] * sf, L)
            for x in torch.arange(L, device=DEV).split(32):
                spec[x] *= _iso_kernel(tab, P, L, x)
        return torch.fft.irfftn(spec, s=(L, L, L))
    if kind == "pcf":
        return _pcf64(case, d)
    if kind == "terms":
        return _summands64(d["eps"], [(case["l"] + k, case["m"]) for k in range(2 if case["paired"] else 1)], _radii(case), J)
    if kind == "zeta":
        if 8 ** J * (case["lmax"] + 1) ** 2 * case["nr"] > 4e9:
            return None
        r, sf, eps = _radii(case), L / BOX, d["eps"].double()
        rho = float(eps.sum().item()) / L ** 3
        lms = [(l, m) for l in range(case["lmax"] + 1) for m in range(l + 1)]
        S = dict(zip(lms, _summands64(eps - rho, lms, r, J)))
        at = [(i, j) for i in range(len(r)) for j in range(len(r))] if case["grid"] else [(0, 1)]
        ddd = np.array([[(-1) ** l * (S[l, 0][i, j] + sum((-1) ** m * 2 * S[l, m][i, j].real for m in range(1, l + 1))).real
                         for l in range(case["lmax"] + 1)] for i, j in at])
        rrr = np.zeros_like(ddd)
        rrr[:, 0] = rho ** 3
        return {"delta_ddd_l": ddd * sf ** 9, "rrr_l": rrr * sf ** 9, "zeta_l": ddd / rho ** 3}
    if kind == "triplets":
        out = []
        n1 = _density64(d["eps"], d["centers"])
        for o in d["offsets"]:
            o = torch.as_tensor(o, device=DEV)
            out.append(float(sum((n1 * _density64(d["eps"], d["centers"] + q[:3]) * _density64(d["eps"], d["centers"] + q[3:]))
                                 .sum() for q in o).item()))
        return np.array(out)
    return _density64(d["eps"], d["pos"] * (L / BOX)).cpu().numpy()
