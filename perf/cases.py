"""Performance cases: the work a user of this framework has it do, through its public entry points.

Five kinds, over the sizes of the repository's decks, tests and benchmark workloads:
  block  the column/wavelength loop on device arrays (Engine.solve_block_device);
  host   the same loop on host arrays, as the deck driver and the Fortran binding call it
         (Engine.solve_block);
  batch  a ragged batch replayed as a CUDA graph (Batch.run);
  post   the quantities derived from a solved block: intensities, optical depth and
         photosphere, wavelength-integrated emergent flux.
Atmospheres (rho and T along z in [-5e15, 5e15] cm):
  isothermal  Gaussian density with a floor at one temperature (the grey deck);
  agn         Gaussian density times a lognormal perturbation per cell, Gaussian temperature on a
              2000 K floor; rho0 drawn from [1e-11, 1e-7] g/cm^3 where "rho0" is 0;
  warm        as agn with a temperature that falls smoothly from the midplane to the boundary and
              stays above the floor, so that no two neighbouring levels share a temperature; the
              sample AGN deck's density floor;
  turbulent   Athena-style: independent lognormal turbulence of density and pressure, T = p/rho.
"""
import math

import numpy as np
import torch

Z0, Z1 = -5e15, 5e15
H, T_MID, T_FLOOR, RHO_FLOOR = 1.496e14, 6.1e4, 2000.0, 1e-24
FULLY_IONIZED_T, SIGMA_GREY = 2e4, 0.4
REFERENCE, LAMBDA_FASTEST = 0, 1
FIELDS = ("U", "kappa", "V", "Vtop", "Vbot")
PLANES = ("Vtop", "Vbot")


def _block(name, nx, ny, nz, nw, form, layout="reference", atmosphere="agn", rho0=1e-9, fields=True, grey=False):
    return {"name": name, "kind": "block", "nx": nx, "ny": ny, "nz": nz, "nw": nw, "form": form, "layout": layout,
            "atmosphere": atmosphere, "rho0": rho0, "fields": fields, "grey": grey}


def listed():
    return [
        # the sample grey deck: one column of ten levels, one wavelength; nothing but latency
        _block("grey_deck", 1, 1, 10, 1, "plain", atmosphere="isothermal", grey=True),
        # the sample Athena deck's block, host arrays in and out, as the drop-in driver calls it
        {"name": "athena_deck_host", "kind": "host", "nx": 31, "ny": 32, "nz": 33, "nw": 5, "form": "plain",
         "atmosphere": "turbulent", "rho0": 1e-9, "grey": False},
        # a handful of columns at full resolution: a look at one region of a snapshot, FP64 without
        # the reference's cancellation; far fewer items than the GPU has threads
        _block("few_columns_stable", 4, 4, 500, 250, "stable", atmosphere="turbulent"),
        # a chunk of the AGN grid, the reference's arithmetic, device-native layout
        _block("agn_plain", 48, 64, 512, 256, "plain", layout="lambda_fastest"),
        # the same grid on the mixed form
        _block("agn_mixed", 64, 64, 512, 256, "mixed", layout="lambda_fastest"),
        # a warm disk on ragged sizes with outputs in the reference's layout (the default)
        _block("warm_plain_reference", 40, 45, 500, 250, "plain", atmosphere="warm"),
        # the AGN grid on the mixed form in the reference's layout
        _block("agn_mixed_reference", 40, 40, 512, 256, "mixed"),
        # a serving job: emergent fluxes only, the precision grid's depth and wavelengths
        _block("flux_only_mixed", 32, 32, 1024, 512, "mixed", rho0=0.0, fields=False),
        # ragged turbulent columns in one launch, both precisions and both layouts
        {"name": "batch_mixed", "kind": "batch", "ncol": 1024, "nz_lo": 64, "nz_hi": 2048, "nw_lo": 32, "nw_hi": 1024,
         "shape_seed": 4, "form": "mixed", "layout": "lambda_fastest"},
        {"name": "batch_plain_reference", "kind": "batch", "ncol": 400, "nz_lo": 64, "nz_hi": 2048, "nw_lo": 32,
         "nw_hi": 1024, "shape_seed": 5, "form": "plain", "layout": "reference"},
        # grey transfer through a whole snapshot: one wavelength per column
        _block("grey_snapshot", 128, 128, 512, 1, "plain", atmosphere="turbulent", grey=True),
        # what analysis scripts derive from a solved block: I+ and I-, optical depth, photosphere,
        # bolometric flux
        dict(_block("products_reference", 28, 30, 500, 200, "plain"), kind="post"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choices(["block", "grey", "host", "batch", "post"], [10, 2, 2, 4, 2])[0]
    form = rng.choice(["plain", "stable", "mixed"])
    layout = rng.choice(["reference", "lambda_fastest"])
    atmosphere = rng.choice(["agn", "warm", "turbulent"])
    rho0 = rng.choice([0.0, 1e-9])
    if kind == "batch":
        return {"kind": "batch", "ncol": _log_int(rng, 1, 400), "nz_lo": _log_int(rng, 8, 64),
                "nz_hi": _log_int(rng, 128, 2048), "nw_lo": _log_int(rng, 1, 32), "nw_hi": _log_int(rng, 64, 1024),
                "shape_seed": rng.randrange(1 << 30), "form": form, "layout": layout}
    if kind == "grey":
        nx, ny, nz = _log_int(rng, 1, 160), _log_int(rng, 1, 160), _log_int(rng, 8, 1024)
        form = rng.choice(["plain", "stable"])
        c = _block("", nx, ny, nz, 1, form, layout, rng.choice(["isothermal", "turbulent"]), rho0, True, True)
    elif kind == "host":
        nx, ny, nz, nw = _log_int(rng, 1, 40), _log_int(rng, 1, 40), _log_int(rng, 10, 128), _log_int(rng, 1, 32)
        c = {"kind": "host", "nx": nx, "ny": ny, "nz": nz, "nw": nw, "form": form, "atmosphere": atmosphere,
             "rho0": rho0, "grey": False}
    else:
        cap = 1.5e8 if kind == "block" else 5e7
        while True:
            nx, ny = _log_int(rng, 1, 128), _log_int(rng, 1, 128)
            nz, nw = _log_int(rng, 10, 1024), _log_int(rng, 1, 512)
            if nx * ny * nz * nw <= cap:
                break
        c = _block("", nx, ny, nz, nw, form, layout, atmosphere, rho0, rng.random() < 0.75)
        c["kind"] = kind
    c.pop("name", None)
    return c


# ---- inputs -----------------------------------------------------------------------------

def _waves(nw):
    return np.logspace(2.0, 5.0, nw) if nw > 1 else np.array([5000.0])


def _rho0(case, gen, device):
    if case["rho0"] > 0.0:
        return case["rho0"]
    return float(10.0 ** (-11.0 + 4.0 * torch.rand((), generator=gen, device=device, dtype=torch.float64)))


def _atmosphere(kind, z, rho0, gen):
    """rho and T of the cells at heights z (any shape)."""
    def normal():
        return torch.randn(z.shape, generator=gen, device=z.device, dtype=torch.float64)

    g = torch.exp(-0.5 * (z / H) ** 2)
    if kind == "isothermal":
        return (rho0 * g).clamp(min=RHO_FLOOR) * 10.0 ** (0.05 * normal()), torch.full_like(z, T_FLOOR)
    if kind == "turbulent":
        rho = (rho0 * g).clamp(min=RHO_FLOOR) * 10.0 ** (0.5 * normal())
        k_cgs, m_u, mu = 1.380649e-16, 1.66053906660e-24, 0.6
        p = (rho0 * k_cgs * T_MID / (mu * m_u)) * g * torch.exp(-0.5 * (z / 2.5e14) ** 2) * 10.0 ** (0.5 * normal())
        return rho, (mu * m_u * p / (rho * k_cgs)).clamp(min=T_FLOOR)
    sigma_t, floor = (2.1e15, 1e-15) if kind == "warm" else (2.5e14, RHO_FLOOR)
    t = (T_MID * torch.exp(-0.5 * (z / sigma_t) ** 2)).clamp(min=T_FLOOR)
    return (rho0 * g).clamp(min=floor) * 10.0 ** (0.3 * normal()), t


def _block_inputs(case, seed, device):
    gen = torch.Generator(device=device).manual_seed(seed)
    rho0 = _rho0(case, gen, device)
    dz = (Z1 - Z0) / (case["nz"] - 1)
    z = Z0 + dz * torch.arange(case["nz"], device=device, dtype=torch.float64)
    rho, t = _atmosphere(case["atmosphere"], z.expand(case["nx"], case["ny"], -1).contiguous(), rho0, gen)
    return rho.contiguous(), t.contiguous(), dz


def _batch_shape(case):
    rng = np.random.default_rng(case["shape_seed"])

    def sizes(lo, hi):
        return np.clip(np.floor(np.exp(rng.uniform(math.log(lo), math.log(hi + 1), case["ncol"]))), lo, hi).astype(np.int64)

    return sizes(case["nz_lo"], case["nz_hi"]), sizes(case["nw_lo"], case["nw_hi"])


def _batch_inputs(case, seed, device):
    nz, nw = _batch_shape(case)
    gen = torch.Generator(device=device).manual_seed(seed)
    n = torch.from_numpy(nz).to(device)
    dz = (Z1 - Z0) / (n - 1).to(torch.float64)
    start = torch.cumsum(n, 0) - n
    col = torch.repeat_interleave(torch.arange(len(nz), device=device), n)
    z = Z0 + (torch.arange(int(n.sum()), device=device) - start[col]).to(torch.float64) * dz[col]
    rho, t = _atmosphere("turbulent", z, 1e-9, gen)
    return nz, nw, dz, rho, t


def _post_inputs(case, seed, device):
    """Arrays as a solve leaves them: U falling off over decades, fluxes of both signs, opacities
    whose optical depth crosses 1 within the column."""
    rho, _, dz = _block_inputs(case, seed, device)
    gen = torch.Generator(device=device).manual_seed(seed + 1)
    nx, ny, nz, nw = (case[k] for k in ("nx", "ny", "nz", "nw"))
    ref = case["layout"] == "reference"

    def field(rows):
        shape = (nw, nx, ny, rows) if ref else (rows, nx * ny, nw)
        return torch.randn(shape, generator=gen, device=device, dtype=torch.float64)

    u = 10.0 ** (2.0 * field(nz + 6) - 6.0)
    v = field(nz) * 1e-6
    kappa = 10.0 ** (field(nz) - 8.0)
    plane = torch.randn((nw, nx, ny), generator=gen, device=device, dtype=torch.float64).abs()
    return rho, dz, u, v, kappa, plane


def _shapes(case, nw):
    cols, nz = case["nx"] * case["ny"], case["nz"]
    if case.get("layout") == "lambda_fastest":
        u, f = (nz + 6, cols, nw), (nz, cols, nw)
    else:
        u, f = (nw, case["nx"], case["ny"], nz + 6), (nw, case["nx"], case["ny"], nz)
    p = (nw, case["nx"], case["ny"])
    return {"U": u, "kappa": f, "V": f, "Vtop": p, "Vbot": p}


def prepare(case, seed):
    from ocotillo_b200 import Engine
    eng = Engine(0)
    layout = LAMBDA_FASTEST if case.get("layout") == "lambda_fastest" else REFERENCE
    st = {"case": case, "eng": eng, "layout": layout}
    if case["kind"] == "batch":
        nz, nw, dz, rho, t = _batch_inputs(case, seed, "cuda")
        grids, off, pos, waves = {}, [], 0, []
        for w in nw.tolist():
            if w not in grids:
                grids[w] = pos
                waves.append(_waves(w))
                pos += w
            off.append(grids[w])
        b = eng.batch(nz, nw, dz.cpu().numpy(), np.concatenate(waves), np.array(off), layout=layout,
                      fully_ionized_T=FULLY_IONIZED_T, form=case["form"])
        st["batch"], st["out"] = b, b.alloc()
        b.bind(rho, t, st["out"])
        return st
    if not case["grey"]:
        eng.set_wavelengths(_waves(case["nw"]))
    if case["kind"] == "host":
        rho, t, dz = _block_inputs(case, seed, "cpu")
        st.update(rho=rho.numpy(), T=t.numpy(), dz=dz)
        return st
    if case["kind"] == "post":
        rho, dz, u, v, kappa, plane = _post_inputs(case, seed, "cuda")
        out = {k: torch.empty_like(v) for k in ("Ip", "Im", "tau")}
        out["photo"] = torch.empty(plane.shape, dtype=torch.int32, device="cuda")
        out["F"] = torch.empty(plane.shape[1:], dtype=torch.float64, device="cuda")
        st.update(rho=rho, dz=dz, U=u, V=v, kappa=kappa, plane=plane, out=out)
        return st
    rho, t, dz = _block_inputs(case, seed, "cuda")
    shapes = _shapes(case, case["nw"])
    st.update(rho=rho, T=t, dz=dz, out={k: torch.empty(shapes[k], dtype=torch.float64, device="cuda")
                                        for k in (FIELDS if case["fields"] else PLANES)})
    return st


def run(st):
    case, eng = st["case"], st["eng"]
    if case["kind"] == "batch":
        st["batch"].run()
        return st["out"]
    if case["kind"] == "host":
        out = eng.solve_block(st["rho"], st["T"], st["dz"], fully_ionized_T=FULLY_IONIZED_T, form=case["form"],
                              allow_zero_pivot=True)
        return {k: out[k] for k in FIELDS}
    if case["kind"] == "post":
        out, shape = st["out"], (case["nx"], case["ny"], case["nz"])
        eng.intensities_device(st["U"], st["V"], shape, case["nw"], out, layout=st["layout"])
        eng.optical_depth_device(st["kappa"], st["rho"], st["dz"], 1.0, out["tau"], out["photo"], layout=st["layout"])
        eng.integrated_flux_device(st["plane"], shape, out=out["F"])
        return out
    return eng.solve_block_device(st["rho"], st["T"], st["dz"], st["out"], fully_ionized_T=FULLY_IONIZED_T,
                                  lgrey=case["grey"], sigma_grey=SIGMA_GREY, form=case["form"], layout=st["layout"])


# Additions and multiplications of one (z, wavelength) point: Saha, opacities, coefficients,
# elimination, back-substitution and flux; grey transfer has no opacity sums.
_FLOPS, _FLOPS_GREY = 97, 45


def work(case):
    if case["kind"] == "batch":
        nz, nw = _batch_shape(case)
        points, cells, items = int((nz * nw).sum()), int(nz.sum()), int(nw.sum())
        return {"bytes": 8 * (2 * cells + 3 * points + 6 * items + 2 * items), "flops": _FLOPS * points}
    cells, items = case["nx"] * case["ny"] * case["nz"], case["nx"] * case["ny"] * case["nw"]
    points = items * case["nz"]
    if case["kind"] == "post":
        return {"bytes": 8 * (cells + 6 * points + items + case["nx"] * case["ny"]) + 4 * items,
                "flops": 5 * points + 2 * items}
    fields = case["kind"] == "host" or case["fields"]
    return {"bytes": 8 * (2 * cells + (3 * points + 6 * items if fields else 0) + 2 * items),
            "flops": (_FLOPS_GREY if case["grey"] else _FLOPS) * points}


# ---- the same quantities in plain 64-bit torch ---------------------------------------------

_C, _HP, _K, _KEV, _RY = 2.99792458e10, 6.62607015e-27, 1.380649e-16, 8.617333262145179e-05, 2.1798741e-11
_MP, _AE = 1.67262192369e-24, 0.6648e-24
_LOG10E = math.log10(math.e)


def _opacity(rho, t, wa):
    """kappa, 1 - albedo and S, broadcast over cells (rho, t) and wavelengths wa (Angstrom)."""
    iev = float.fromhex("0x1.b369160866803p+3")  # hydrogen ionization energy of the free-free factor, eV
    c_ion = (_MP / rho) * (2414683039571967.0 * t ** 1.5 * torch.exp(-(13.6 / t) / _KEV))
    x = 0.5 * (torch.sqrt(c_ion * c_ion + 4.0 * c_ion) - c_ion)
    x = torch.where(t > FULLY_IONIZED_T, torch.ones_like(x), x)
    n = rho / _MP
    nii = x * n
    ni = n - nii
    ionf = ni / (ni + nii)
    theta = 5040.0 / t
    lgt = torch.log10(theta)
    wcm = wa * 1e-8
    nu = _C / wcm
    stim = 1.0 - 10.0 ** (-(1.2398e4 / wa) * theta)
    # H bound-free: six levels and the rest as an integral
    s = torch.zeros_like(theta * wa)
    for q in range(1, 7):
        lam_n = q * q * (_HP * _C / _RY)
        e2 = (wcm / lam_n - 1.0) ** 2
        gaunt = 1.0 - (0.17285714285714285 * (1.0 - e2)) * (q * (1.0 + e2)) ** (-2.0 / 3.0)
        gaunt = torch.where(wcm <= lam_n, gaunt, torch.zeros_like(gaunt))
        s = s + gaunt / q ** 3 * torch.exp(-_RY * (1.0 - 1.0 / (q * q)) / (_K * t))
    unsold = 0.5 * _K * t / _RY * (torch.exp(-_RY * (1.0 - 1.0 / 36.0) / (_K * t)) - torch.exp(-_RY / (_K * t)))
    kabs = 1.0449e-26 * stim * ionf * wa ** 3 * (unsold + s)
    del s
    # H- bound-free and free-free
    hm = 4.158e-10 * (nii * _K * t) * theta ** 2.5 * 10.0 ** (0.754 * theta)
    a = (1.99654, -1.18267e-6, 2.62423e-7, -4.40524e-11, 3.23992e-15, -1.39568e-19, 2.78701e-24)
    sc = sum(1e-17 * c * wa ** i for i, c in enumerate(a))
    kabs = kabs + hm * stim * ionf * torch.where(wa < 16000.0, sc, torch.zeros_like(sc))
    b = ((-2.276300, -1.685000, 0.766610, -0.053356, 0.0), (15.28270, -9.284600, 1.993810, -0.142631, 0.0),
         (-197.789, 190.266, -67.9775, 10.6913, -0.62515))
    lw = torch.log10(wa)
    f = [sum(c * lw ** j for j, c in enumerate(row)) for row in b]
    kabs = kabs + ionf * nii * _K * t * 10.0 ** (f[0] + f[1] * lgt + f[2] * lgt * lgt - 26.0)
    esc = _AE * nii / n
    kabs = kabs / _MP
    kr = kabs + esc / _MP
    op = kr * rho
    neutral = (1.0 - x) > 1e-2
    gff = 1.0 + 0.3456 * (wa * 1.0968e-3) ** (-1.0 / 3.0) * (_LOG10E / theta * wa / 1.2398e4 + 0.5)
    kff = stim * ionf * 1.0443e-26 * wa ** 3 * gff * (0.5 * _LOG10E / theta / iev * 10.0 ** (-theta * iev)) / _MP
    gaunt = torch.log(torch.exp(5.960 - math.sqrt(3.0) / math.pi * torch.log(nu * 1e-9 * (t * 1e-4) ** -1.5)) + math.e)
    lnq = torch.log(nii * n) - 0.5 * torch.log(t) - 3.0 * torch.log(nu) + torch.log(-torch.expm1(-(_HP * nu / _K) / t))
    kb = 369234910.67735046 * torch.exp(lnq) * gaunt
    del gaunt, lnq, gff, stim
    op_i = op + kb
    extra = torch.where(neutral, kff, op_i / rho)
    op = torch.where(neutral, op + (kr + kff) * rho, op_i)
    kabs, kr = kabs + extra, kr + extra
    damping = (_HP * _C / _K / t / wcm).clamp(max=308.0)
    return op, kabs / kr, (2.0 * _HP * _C * _C / wcm ** 5) / torch.expm1(damping)


def _transfer(op, oma, src, dz, nz):
    """U (with three ghost levels each side), kappa and V as [z, item]; nz levels per item
    (rows beyond an item's are padding), dz per item.  The tridiagonal system is eliminated in
    difference form, whose terms are all positive."""
    rows, items = op.shape
    dev = op.device
    k = torch.arange(rows, device=dev)[:, None]
    it = torch.arange(items, device=dev)
    top, pad = k == nz - 1, k >= nz
    kh = 0.5 * (op[1:] + op[:-1])
    a, c = torch.zeros_like(op), torch.zeros_like(op)
    a[1:] = op[1:] ** 2 / kh
    c[:-1] = op[:-1] ** 2 / kh
    e = dz * dz * op ** 3 * oma
    d = src * e
    edge = 0.25 * dz * dz * op * oma
    end = top | (k == 0)
    a = torch.where(top, op, a)
    c = torch.where(k == 0, op, torch.where(top, torch.zeros_like(c), c))
    e = torch.where(end, (dz + edge) * op * op, e)
    d = torch.where(end, src * edge * op * op, d)
    del edge, kh
    for x, v in ((a, 0.0), (c, 1.0), (e, 0.0), (d, 0.0)):
        x.masked_fill_(pad, v)
    u, q, g = torch.zeros_like(op), torch.zeros_like(op), torch.zeros_like(op)
    h = e[0]
    u[0] = d[0] / (c[0] + h)
    for j in range(1, rows):
        r = 1.0 / (c[j - 1] + h)
        q[j - 1] = h * r
        g[j] = c[j - 1] * r
        h = torch.addcmul(e[j], a[j], q[j - 1])
        u[j] = torch.addcmul(d[j], a[j], u[j - 1]) / (c[j] + h)
    del a, c, e, d
    diff = torch.zeros_like(op)
    for j in range(rows - 2, -1, -1):
        diff[j] = u[j] - q[j] * u[j + 1]
        u[j] += g[j + 1] * u[j + 1]
    del q, g
    ext = torch.zeros((rows + 5, items), dtype=op.dtype, device=dev)  # row k + 3: level k minus level k + 1
    ext[3:rows + 2] = diff[:rows - 1]
    full = torch.zeros((rows + 6, items), dtype=op.dtype, device=dev)
    full[3:rows + 3] = u
    for i in range(3):
        ext[2 - i] = diff[i]
        ext[nz + 2 + i, it] = diff[nz - 2 - i, it]
        full[2 - i] = 2.0 * u[0] - u[i + 1]
        full[nz + 3 + i, it] = 2.0 * u[nz - 1, it] - u[nz - 2 - i, it]
    s1 = ext[2:rows + 2] + ext[3:rows + 3]
    s2 = s1 + ext[1:rows + 1] + ext[4:rows + 4]
    s3 = s2 + ext[0:rows] + ext[5:rows + 5]
    v = (45.0 * s1 - 9.0 * s2 + s3) / 60.0 / dz / op
    return full, op, v


def _exact_block(case, rho, t, dz):
    nz, nw, cols = case["nz"], case["nw"], case["nx"] * case["ny"]
    dev = rho.device
    wa = torch.from_numpy(_waves(nw)).to(dev)
    keep = case["kind"] == "host" or case["fields"]
    rows = {"U": nz + 6, "kappa": nz, "V": nz}
    out = {k: torch.empty((r, cols, nw), dtype=torch.float64, device=dev) for k, r in rows.items() if keep}
    planes = {k: torch.empty((cols, nw), dtype=torch.float64, device=dev) for k in PLANES}
    step = max(1, int(4e7) // (nz * nw))
    for c0 in range(0, cols, step):
        r, tt = (x.reshape(cols, nz)[c0:c0 + step].t()[:, :, None] for x in (rho, t))
        m = r.shape[1]
        if case["grey"]:
            alpha = 3.68e22 * tt ** -3.5 * r
            op, oma, src = (alpha + SIGMA_GREY) * r, alpha / (alpha + SIGMA_GREY), 5.6703744191844314e-05 * tt ** 4
        else:
            op, oma, src = _opacity(r, tt, wa)
        args = (x.expand(nz, m, nw).reshape(nz, m * nw) for x in (op, oma, src))
        u, kap, v = _transfer(*args, dz, torch.full((m * nw,), nz, device=dev))
        for k, x in (("U", u), ("kappa", kap), ("V", v)):
            if keep:
                out[k][:, c0:c0 + m] = x.view(-1, m, nw)
        planes["Vtop"][c0:c0 + m], planes["Vbot"][c0:c0 + m] = v[nz - 1].view(m, nw), v[0].view(m, nw)
    if case.get("layout") != "lambda_fastest":
        for k in out:
            out[k] = out[k].permute(2, 1, 0).reshape(nw, case["nx"], case["ny"], -1)
    out.update({k: x.t().reshape(nw, case["nx"], case["ny"]) for k, x in planes.items()})
    return out


def _exact_batch(case, seed):
    nz, nw, dz, rho, t = _batch_inputs(case, seed, "cuda")
    dev = rho.device
    col0 = np.cumsum(nz) - nz
    waves = {w: torch.from_numpy(_waves(w)).to(dev) for w in set(nw.tolist())}
    parts = {k: [None] * len(nz) for k in FIELDS}
    order = np.argsort(-nz, kind="stable")
    at = 0
    while at < len(order):  # columns of similar depth together, padded to the deepest
        deep, grp, items = int(nz[order[at]]), [], 0
        while at < len(order) and (not grp or (nz[order[at]] * 5 >= deep * 4 and (items + nw[order[at]]) * deep <= 4e7)):
            grp.append(int(order[at]))
            items += int(nw[order[at]])
            at += 1
        ops = [torch.ones((deep, items), dtype=torch.float64, device=dev) for _ in range(3)]
        pos = 0
        for i in grp:
            cells = slice(int(col0[i]), int(col0[i] + nz[i]))
            for dst, x in zip(ops, _opacity(rho[cells, None], t[cells, None], waves[int(nw[i])])):
                dst[:int(nz[i]), pos:pos + int(nw[i])] = x
            pos += int(nw[i])
        idx = torch.tensor(grp, device=dev)
        per = torch.from_numpy(nw[grp]).to(dev)
        levels = torch.repeat_interleave(torch.from_numpy(nz[grp]).to(dev), per)
        u, kap, v = _transfer(*ops, torch.repeat_interleave(dz[idx], per), levels)
        pos = 0
        for i in grp:
            n, w = int(nz[i]), int(nw[i])
            s = slice(pos, pos + w)
            for k, x in (("U", u[:n + 6, s]), ("kappa", kap[:n, s]), ("V", v[:n, s])):
                parts[k][i] = (x if case["layout"] == "lambda_fastest" else x.t()).reshape(-1).clone()
            parts["Vtop"][i], parts["Vbot"][i] = v[n - 1, s].clone(), v[0, s].clone()
            pos += w
    return {k: torch.cat(x) for k, x in parts.items()}


def exact(case, seed):
    if case["kind"] == "batch":
        return _exact_batch(case, seed)
    if case["kind"] == "host":
        rho, t, dz = _block_inputs(case, seed, "cpu")
        out = _exact_block(case, rho, t, dz)
        return {k: out[k].numpy() for k in FIELDS}
    if case["kind"] == "post":
        rho, dz, u, v, kappa, plane = _post_inputs(case, seed, "cuda")
        cells = case["nx"] * case["ny"]
        if case["layout"] == "reference":
            inner = u[..., 3:-3]
            tau = torch.cumsum(kappa * rho * dz, dim=-1)
        else:
            inner = u[3:-3]
            tau = torch.cumsum(kappa * rho.reshape(cells, -1).t()[:, :, None] * dz, dim=0)
        wa = torch.from_numpy(_waves(case["nw"])).to(u.device) * 1e-8
        flux = torch.trapezoid(plane, wa, dim=0) if case["nw"] > 1 else torch.zeros_like(plane[0])
        return {"Ip": inner + v, "Im": inner - v, "tau": tau, "photo": None, "F": flux}
    rho, t, dz = _block_inputs(case, seed, "cuda")
    return _exact_block(case, rho, t, dz)
