"""Performance cases of the boundary-element library: what a user has it do,
through its public entry points, over the sizes it is used at.

  listed()          the named cases
  draw(rng)         another case of the same ranges
  prepare(case, s)  the inputs of a case: a host mesh, frequencies, motion
                    fields, headings and cotangents, made from the seed
  run(state)        one call of the entry point
  work(case)        the bytes and operations a call cannot do without
  exact(case, s)    the same outputs from plain torch in 64 bits

Every call runs with the library's defaults (the process-wide context, mixed
precision to a residual of 1e-10 in the batched calls, FP64 in the single
ones).  Meshes are hemispheres, pairs of them and the WaveBot buoy with the
radius, the position and the frequencies varied by the seed.
"""
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch

RHO, G = 1000.0, 9.81


def _package():
    """The library (its folder's name has a dot, so it is loaded by path)."""
    name = "marinehydro_b200"
    if name not in sys.modules:
        folder = pathlib.Path(__file__).resolve().parents[1] / "marinehydro.jl_b200"
        spec = importlib.util.spec_from_file_location(name, folder / "__init__.py",
                                                      submodule_search_locations=[str(folder)])
        module = importlib.util.module_from_spec(spec)
        sys.modules[name] = module
        spec.loader.exec_module(module)
    return sys.modules[name]


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------

def _case(name, call, shape, nt, nphi, wave="delhommeau", direct=True, n_omega=1, n_dof=1, n_beta=0, radius=1.0):
    return dict(name=name, call=call, shape=shape, nt=nt, nphi=nphi, wave=wave, direct=direct, n_omega=n_omega,
                n_dof=n_dof, n_beta=n_beta, radius=radius)


def listed():
    return [
        # one coefficient of a coarse hemisphere: what a script or an optimiser calls point by point
        _case("radiation_50p", "radiation", "hemisphere", 10, 10, "wu"),
        # one diffraction force at an ordinary resolution, in the FP64 the call defaults to
        _case("diffraction_800p", "diffraction", "hemisphere", 40, 40, "wu", n_beta=1),
        # the influence matrices themselves, brought to the host (studies of the discretisation)
        _case("assemble_570p", "assemble", "hemisphere", 30, 38, "wu"),
        # a small body with all six motions and a heading over a coarse sweep
        _case("coefficients_200p_6dof", "batch", "hemisphere", 20, 20, n_omega=20, n_dof=6, n_beta=1),
        # the WaveBot at its default resolution: six motions, two headings, the default Green function
        _case("coefficients_wavebot_6dof", "batch", "wavebot", 0, 72, "wu", n_omega=16, n_dof=6, n_beta=2, radius=0.88),
        # a full sweep of one body at fine resolution
        _case("sweep_2048p_64w", "batch", "hemisphere", 64, 64, n_omega=64, n_dof=2, n_beta=1),
        # a finer, larger body with an odd number of panels, by the indirect method
        _case("sweep_2997p_24w", "batch", "hemisphere", 53, 111, direct=False, n_omega=24, n_dof=1, n_beta=1, radius=1.8),
        # two bodies some radii apart: pairs far from each other in wavelengths
        _case("two_bodies_1456p_32w", "batch", "pair", 26, 56, n_omega=32, n_dof=2, n_beta=1),
        # gradients of a full sweep with respect to the mesh, the frequencies and the motions
        _case("gradient_2048p_64w", "vjp", "hemisphere", 64, 64, n_omega=64, n_dof=2, n_beta=1),
        # one step of a two-body layout optimisation at one frequency
        _case("gradient_two_bodies_2048p", "vjp", "pair", 32, 64, "wu", direct=False, n_omega=1, n_dof=2, n_beta=1),
        # gradients of a coarse body with an odd number of panels
        _case("gradient_243p_12w", "vjp", "hemisphere", 17, 27, n_omega=12, n_dof=1, n_beta=1, radius=1.7),
        # a design study: coefficients and their derivatives along the radius
        _case("radius_870p_16w", "jvp", "hemisphere", 29, 58, n_omega=16, n_dof=1, radius=1.4),
    ]


def draw(rng):
    call = rng.choice(["radiation", "diffraction", "assemble", "batch", "batch", "batch", "vjp", "vjp", "jvp"])
    # (no mesh gradient on the buoy: its flat bottom has coplanar panels, where the closed form of
    # the panel integral takes the sign of a rounding error and has no derivative along the normal)
    shape = rng.choice(["hemisphere", "hemisphere", "hemisphere", "pair", "hemisphere" if call == "vjp" else "wavebot"])
    wave = rng.choice(["wu", "delhommeau", "delhommeau"]) if call in ("batch", "vjp", "jvp") else "wu"
    most = {"radiation": 900, "diffraction": 900, "assemble": 900, "batch": 2600, "vjp": 2000, "jvp": 1300}[call]
    panels = math.exp(rng.uniform(math.log(40), math.log(most)))
    if shape == "wavebot":
        nt, nphi = 0, max(5, round(panels / 17))
    else:
        one = panels / (2 if shape == "pair" else 1)
        bands = max(2, round(math.sqrt(one / rng.uniform(1.5, 3.0))))
        nt, nphi = 2 * bands - rng.randrange(2), max(6, round(one / bands))
    case = _case("", call, shape, nt, nphi, wave, True)
    if call in ("batch", "vjp", "jvp"):
        n = _panels(case)
        room = 0.5 * 64 * 2048.0 ** 2 / n ** 2 / (3 if call != "batch" else 1)
        case.update(direct=rng.random() < 0.7, n_dof=rng.choice([1, 2, 3, 6] if call == "batch" else [1, 2]),
                    n_omega=max(1, min(int(math.exp(rng.uniform(0.0, math.log(96)))), int(room))),
                    n_beta=rng.choice([0, 1, 1, 2] if call == "batch" else [0, 1]))
    elif call == "diffraction":
        case.update(n_beta=1)
    case.update(radius=round(0.88 if shape == "wavebot" else rng.uniform(0.6, 2.0), 3))
    del case["name"]
    return case


def _panels(case):
    bands = (case["nt"] + 1) // 2
    return 17 * case["nphi"] if case["shape"] == "wavebot" else bands * case["nphi"] * (2 if case["shape"] == "pair" else 1)


def work(case):
    """Bytes: the inputs and outputs as the caller holds them.  Operations
    (real): per pair the two Rankine terms (far field), per pair and
    frequency the wave term and the entries of S and D, then the
    factorisation (8/3 n^3) and the products and substitutions of every
    right-hand side; a reverse or forward derivative repeats the pair work
    and the substitutions."""
    n, w, d, b = _panels(case), case["n_omega"], case["n_dof"], case["n_beta"]
    call = case["call"]
    geom = 8.0 * n * 30
    pair = 60.0 * n * n + 120.0 * n * n * w
    if call == "assemble":
        return {"bytes": geom + 32.0 * n * n, "flops": pair}
    q = {"radiation": 1, "diffraction": 1}.get(call, d + b)
    solve = w * (8.0 / 3.0 * n ** 3 + 24.0 * n * n * q)
    out = 16.0 * w * (d * d + 2 * d * b)
    if call in ("radiation", "diffraction", "batch"):
        return {"bytes": geom + 24.0 * n * d + out, "flops": pair + solve}
    if call == "vjp":
        return {"bytes": 2 * (geom + 24.0 * n * d) + 2 * out, "flops": 2 * pair + solve + w * 32.0 * n * n * q}
    return {"bytes": 2 * geom + 24.0 * n * d + 2 * out, "flops": 2 * pair + solve + w * 32.0 * n * n * q}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------

def _panel_fields(verts, faces, first_vertex_radius=False):
    v = verts[faces]
    a, b, c, d = v[:, 0], v[:, 1], v[:, 2], v[:, 3]
    c1, c2 = np.cross(b - a, c - a), np.cross(c - a, d - a)
    a1, a2 = 0.5 * np.linalg.norm(c1, axis=1), 0.5 * np.linalg.norm(c2, axis=1)
    centers = ((a + b + c) / 3 * a1[:, None] + (a + c + d) / 3 * a2[:, None]) / (a1 + a2)[:, None]
    normals = c1 / np.linalg.norm(c1, axis=1)[:, None]
    reach = np.linalg.norm(v - centers[:, None, :], axis=2)
    return dict(vertices=verts, faces=faces, centers=centers, normals=normals, areas=a1 + a2,
                radii=reach[:, 0].copy() if first_vertex_radius else reach.max(axis=1))


def _revolved(profile, nphi):
    """Vertices and faces of a profile of (r, z) points from the waterline
    down, the last one on the axis, revolved with nphi sectors."""
    phi = 2 * np.pi * np.arange(nphi) / nphi
    rings = len(profile) - 1
    r, z = profile[:-1, 0], profile[:-1, 1]
    verts = np.concatenate([np.stack([r[:, None] * np.cos(phi), r[:, None] * np.sin(phi),
                                      np.repeat(z[:, None], nphi, 1)], axis=2).reshape(-1, 3),
                            [[0.0, 0.0, profile[-1, 1]]]])
    ring, s = np.repeat(np.arange(rings), nphi), np.tile(np.arange(nphi), rings)
    s2, last = (s + 1) % nphi, ring + 1 == rings
    a, d, pole = ring * nphi + s, ring * nphi + s2, rings * nphi
    faces = np.stack([a, np.where(last, pole, a + nphi), np.where(last, d, d + nphi), d], axis=1).astype(np.int64)
    return verts, faces


def _inputs(case, seed):
    """The arrays of a case, from the seed alone."""
    rng = np.random.default_rng(int(seed))
    radius = case["radius"] * rng.uniform(0.97, 1.03)
    where = np.array([rng.uniform(-1, 1), rng.uniform(-1, 1), 0.0])
    if case["shape"] == "wavebot":
        tall, cone, low = 0.16 * rng.uniform(0.9, 1.1), 0.37 * rng.uniform(0.9, 1.1), 0.35 * rng.uniform(0.9, 1.1)
        prof = [(radius, -tall * j / 4) for j in range(5)]
        prof += [(radius + (low - radius) * j / 9, -tall - cone * j / 9) for j in range(1, 10)]
        prof += [(low * (1 - j / 4), -tall - cone) for j in range(1, 5)]
        verts, faces = _revolved(np.array(prof), case["nphi"])
    else:
        bands = (case["nt"] + 1) // 2
        t = 0.5 * np.pi * np.arange(bands + 1) / bands
        verts, faces = _revolved(np.stack([radius * np.cos(t), -radius * np.sin(t)], axis=1), case["nphi"])
    verts = verts + where
    if case["shape"] == "pair":
        far = np.array([radius * rng.uniform(3.5, 5.0), 0.0, 0.0])
        verts, faces = np.concatenate([verts, verts + far]), np.concatenate([faces, faces + len(verts)])
    x = _panel_fields(verts, faces, case["shape"] == "wavebot")
    n, w, d, b = len(faces), case["n_omega"], case["n_dof"], case["n_beta"]
    x["omegas"] = np.linspace(0.3, 3.0, w) * rng.uniform(0.97, 1.03) if w > 1 else np.array([rng.uniform(0.9, 1.6)])
    x["betas"] = rng.uniform(0, np.pi, b)
    motions = np.zeros((d, n, 3))
    if case["shape"] == "pair":  # each body heaves by itself, then surges
        half = n // 2
        for q in range(d):
            rows = slice(0, half) if q % 2 == 0 else slice(half, n)
            motions[q, rows, (2, 0, 1)[(q // 2) % 3]] = 1.0
    else:  # heave, surge, sway, then the rotations about the body's centre
        for q in range(d):
            if q < 3:
                motions[q, :, (2, 0, 1)[q]] = 1.0
            else:
                axis = np.zeros(3)
                axis[(1, 0, 2)[q - 3]] = 1.0
                motions[q] = np.cross(axis, x["centers"] - where)
    x["dofs"] = motions
    if case["call"] == "vjp":
        x["bar_A"], x["bar_B"] = rng.standard_normal((2, d, d, w))
        x["bar_F"] = rng.standard_normal((d, w, b)) + 1j * rng.standard_normal((d, w, b))
        x["bar_K"] = rng.standard_normal((d, w, b)) + 1j * rng.standard_normal((d, w, b))
    if case["call"] == "jvp":  # along the size of the body, about its centre
        size = (verts - where) / radius, (x["centers"] - where) / radius
        x["t_vertices"], x["t_centers"] = size
        x["t_areas"] = 2 * x["areas"] / radius
    return x


def prepare(case, seed):
    mh = _package()
    x = _inputs(case, seed)
    mesh = mh.Mesh(x["vertices"], x["faces"], x["centers"], x["normals"], x["areas"], x["radii"])
    mh.default_context()
    waves = {"wu": mh.GFWu(), "delhommeau": mh.ExactGuevelDelhommeau()}
    state = dict(case=case, mesh=mesh, x=x, dofs=list(x["dofs"]),
                 options=dict(green_functions=(mh.Rankine(), mh.RankineReflected(), waves[case["wave"]]),
                              direct=case["direct"]))
    if case["call"] == "jvp":
        state["tangent"] = mh.MeshTangent(x["t_vertices"], x["t_centers"], np.zeros_like(x["normals"]), x["t_areas"],
                                          x["radii"] / case["radius"])
    return state


def run(state):
    mh, case, mesh, x, kw = _package(), state["case"], state["mesh"], state["x"], state["options"]
    call = case["call"]
    if call == "radiation":
        return mh.calculate_radiation_forces(mesh, [0.0, 0.0, 1.0], x["omegas"][0], **kw)
    if call == "diffraction":
        return np.array([mh.DiffractionForce(mesh, x["omegas"][0], [0.0, 0.0, 1.0], beta=x["betas"][0], **kw)])
    if call == "assemble":
        return mh.assemble_matrices(kw["green_functions"], mesh, x["omegas"][0] ** 2 / G, direct=kw["direct"])
    if call == "batch":
        return mh.hydro_batch(mesh, x["omegas"], state["dofs"], x["betas"], **kw)[:4]
    if call == "vjp":
        r = mh.hydro_batch_vjp(mesh, x["omegas"], state["dofs"], x["betas"], x["bar_A"], x["bar_B"], x["bar_F"],
                               x["bar_K"], **kw)
        return dict(A=r.added_mass, B=r.damping, F=r.diffraction, K=r.froude_krylov, vertices=r.mesh.vertices,
                    centers=r.mesh.centers, normals=r.mesh.normals, areas=r.mesh.areas, omegas=r.omegas,
                    dofs=list(r.dofs))
    r = mh.hydro_batch_jvp(mesh, x["omegas"], state["dofs"], x["betas"], state["tangent"], **kw)
    return dict(A=r.added_mass, B=r.damping, F=r.diffraction, K=r.froude_krylov, dA=r.d_added_mass, dB=r.d_damping,
                dF=r.d_diffraction, dK=r.d_froude_krylov)


# --------------------------------------------------------------------------
# the same outputs in plain torch, 64 bits, differentiable both ways
# --------------------------------------------------------------------------

class _Known(torch.autograd.Function):
    """f(x) with a derivative that is known as a value."""

    @staticmethod
    def forward(ctx, x, value, slope):
        ctx.save_for_backward(slope)
        ctx.save_for_forward(slope)
        return value.clone()

    @staticmethod
    def backward(ctx, g):
        return g * ctx.saved_tensors[0], None, None

    @staticmethod
    def jvp(ctx, t, *_):
        return t * ctx.saved_tensors[0]


def _series(x):
    """J0, J1, Y0, Y1 and the Struve functions H0, H1 by their power series
    (x up to about 12; x = 0 is read as 1e-30 in the logarithm)."""
    q, pi = -0.25 * x * x, math.pi
    j0, s0 = torch.ones_like(x), torch.zeros_like(x)
    j1, s1 = torch.ones_like(x), torch.ones_like(x)
    h0, h1 = x * (2 / pi), x * x * (2 / pi / 3)
    a, b, t0, t1, harm = j0, j1, h0, h1, 0.0
    for k in range(1, 60):
        harm += 1.0 / k
        a, b = a * q / k ** 2, b * q / (k * (k + 1))
        t0, t1 = -t0 * x * x / (2 * k + 1) ** 2, -t1 * x * x / ((2 * k + 1) * (2 * k + 3))
        j0, s0 = j0 + a, s0 - harm * a
        j1, s1 = j1 + b, s1 + (2 * harm + 1.0 / (k + 1)) * b
        h0, h1 = h0 + t0, h1 + t1
    j1 = 0.5 * x * j1
    safe = torch.clamp(x, min=1e-30)
    log = torch.log(0.5 * safe) + 0.57721566490153286061
    y0 = (2 / pi) * (log * j0 + s0)
    y1 = (2 / pi) * log * j1 - (2 / pi) / safe - (0.5 / pi) * x * s1
    return j0, j1, y0, y1, h0, h1


def _bessel(x):
    """J0, J1 and, at x > 0 (0 elsewhere), Y0, Y1, with their derivatives."""
    v = x.detach()
    j0, j1, y0, y1 = _series(v)[:4]
    on = v > 0
    safe = torch.where(on, v, torch.ones_like(v))
    dj1 = torch.where(on, j0 - j1 / safe, torch.full_like(v, 0.5))
    y0, y1 = torch.where(on, y0, torch.zeros_like(v)), torch.where(on, y1, torch.zeros_like(v))
    return (_Known.apply(x, j0, -j1), _Known.apply(x, j1, dj1), _Known.apply(x, y0, -y1),
            _Known.apply(x, y1, y0 - y1 / safe))


def _poly(t, *c):
    r = torch.full_like(t, c[-1])
    for v in reversed(c[:-1]):
        r = v + r * t
    return r


def _wu(r, z):
    """G, dG/dr, dG/dz (real and imaginary parts) of Wu's closed-form approximation."""
    d = torch.sqrt(r * r + z * z)
    alpha, beta, rho, ev = -z / d, r / d, d / (1 + d), torch.exp(z)
    fa = _poly(rho, 1.21, -13.328, 215.896, -1763.96, 8418.94, -24314.21, 42002.57, -41592.9, 21859.0, -4838.6)
    fb = _poly(rho, 0.938, 5.737, -67.92, 796.534, -4780.77, 17137.74, -36618.81, 44894.06, -29030.24, 7671.22)
    fc = _poly(rho, 1.268, -9.747, 209.653, -1397.89, 5155.67, -9844.35, 9136.4, -3272.62)
    fd = _poly(rho, 0.632, -40.97, 667.16, -6072.07, 31127.39, -96293.05, 181856.75, -205690.43, 128170.2, -33744.6)
    da = _poly(rho, 2.948, -24.53, 249.69, -754.85, -1187.71, 16370.75, -48811.41, 68220.87, -46688.0, 12622.25)
    db = _poly(rho, 1.11, 2.894, -76.765, 1565.35, -11336.19, 44270.15, -97014.11, 118879.26, -76209.82, 19923.28)
    dc = _poly(rho, 14.19, -148.24, 847.8, -2318.58, 3168.35, -1590.27)
    cube, d3 = rho * (1 - rho) ** 3, 1 + d ** 3
    lp = cube * ((1 - beta) * fa - beta * fb - alpha * fc / (1 + 6 * alpha * rho * (1 - rho)) + beta * (1 - beta) * fd)
    pp = ev * (torch.log(0.5 * (d - z)) + 0.5772156649 - 2 * d * d) + d * d - z
    l0 = 2 * pp / d3 + 2 * lp
    lsp = cube * (beta * da - (1 - alpha) * db + beta * (1 - beta) * rho * (1 - 2 * rho) * dc)
    ps = (beta + r) / (d - z) - 2 * beta + 2 * ev * d - r
    ls = 2 * ps / d3 - 4 * torch.exp(-d) * (1 - beta) * (1 + d / d3) + 2 * lsp
    j0, j1, y0, y1 = _bessel(r)
    small = r <= 3.0
    t, yy = r / 3, (r / 3) ** 2
    u = (3 / torch.where(small, torch.full_like(r, 4.0), r))
    uu = u * u
    h0 = torch.where(small, t * _poly(yy, 1.909859164, -1.909855001, 0.687514637, -0.126164557, 0.013828813, -0.000876918),
                     2 * _poly(uu, 0.99999906, 4.77228920, 3.85542044, 0.32303607)
                     / (3 * math.pi / u * _poly(uu, 1.0, 4.88331068, 4.28957333, 0.52120508)) + y0)
    h1 = torch.where(small, yy * _poly(yy, 1.909859286, -1.145914713, 0.294656958, -0.042070508, 0.003785727, -0.000207183),
                     2 * _poly(uu, 1.00000004, 3.92205313, 2.64893033, 0.27450895)
                     / (math.pi * _poly(uu, 1.0, 3.81095112, 2.26216956, 0.10885141)) + y1)
    g, gi = -l0 - 2 * math.pi * h0 * ev, 2 * math.pi * j0 * ev
    return (g, gi), (-ls - 2 * math.pi * (2 / math.pi - h1) * ev, -2 * math.pi * j1 * ev), (g + 2 / d, gi)


_NODES = np.polynomial.legendre.leggauss(110)


class _WaveG(torch.autograd.Function):
    """Re G, Im G, Re G_r, Im G_r of the infinite-depth wave term, from
    Newman's form of the principal-value integral: with X = r, Y = -z,
    Re G = -pi e^-Y (H0 + Y0)(X) - 2 int_0^Y e^(t-Y) / sqrt(X^2 + t^2) dt,
    the integral over t = X sinh s by Gauss-Legendre nodes."""

    @staticmethod
    def forward(ctx, r, z):
        y = -z
        x = torch.maximum(r, 1e-12 * y)
        top, decay = torch.asinh(y / x), torch.exp(z)
        i0, i1 = torch.zeros_like(x), torch.zeros_like(x)
        for u, w in zip(*_NODES):
            s = 0.5 * (u + 1) * top
            sh = torch.sinh(s)
            e = torch.exp(x * sh - y)
            i0 += (0.5 * w) * e
            i1 += (0.5 * w) * e / (1 + sh * sh)
        j0, j1, y0, y1, h0, h1 = _series(x)
        g = -math.pi * decay * (h0 + y0) - 2 * top * i0
        gr = -math.pi * decay * (2 / math.pi - h1 - y1) + 2 * top * i1 / x
        gi, gri = 2 * math.pi * decay * j0, -2 * math.pi * decay * j1
        gr = torch.where(r > 0, gr, torch.zeros_like(gr))
        ctx.save_for_backward(r, z, g, gi, gr, gri)
        ctx.save_for_forward(r, z, g, gi, gr, gri)
        return g, gi, gr, gri

    @staticmethod
    def _slopes(ctx):
        r, z, g, gi, gr, gri = ctx.saved_tensors
        d = torch.sqrt(r * r + z * z)
        on = r > 0
        safe = torch.where(on, r, torch.ones_like(r))
        gz = g + 2 / d
        gzz = gz - 2 * z / d ** 3  # and G_rr = -G_r / r - G_zz (harmonic)
        grr, grri = -gr / safe - gzz, -gri / safe - gi
        return (gr, gz), (gri, gi), (torch.where(on, grr, -gzz / 2), gr - 2 * r / d ** 3), (torch.where(on, grri, -gi / 2), gri)

    @staticmethod
    def backward(ctx, *up):
        s = _WaveG._slopes(ctx)
        return sum(u * a for u, (a, _) in zip(up, s)), sum(u * b for u, (_, b) in zip(up, s))

    @staticmethod
    def jvp(ctx, tr, tz):
        return tuple(tr * a + tz * b for a, b in _WaveG._slopes(ctx))


def _wave(kind, r, z):
    if kind == "wu":
        return _wu(r, z)
    g, gi, gr, gri = _WaveG.apply(r, z)
    return (g, gi), (gr, gri), (g + 2 / torch.sqrt(r * r + z * z), gi)


def _dot(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _rankine(px, m):
    """Integral of 1/r over panel j seen from point i and its gradient with
    respect to the panel's position: point source beyond seven radii, the
    closed form of a flat polygon within."""
    n = len(m["radii"])
    c = m["centers"].T
    rb = [px[q][:, None] - c[q][None, :] for q in range(3)]
    r2 = _dot(rb, rb)
    near = torch.sqrt(r2.detach()) <= 7 * m["radii"][None, :]
    r = torch.sqrt(torch.where(near, torch.ones_like(r2), r2))
    keep = (~near).to(r.dtype)
    one = keep * m["areas"][None, :] / r
    grad = [one * rb[q] / (r * r) for q in range(3)]
    i, j = torch.nonzero(near, as_tuple=True)
    x = [px[q][i] for q in range(3)]
    nv = [m["normals"][j, q] for q in range(3)]
    rad = m["radii"][j]
    gz = _dot([x[q] - c[q][j] for q in range(3)], nv)
    agz, sg = torch.abs(gz), torch.sign(gz.detach())
    use = agz.detach() >= 1e-4 * rad
    v = m["vertices"][m["faces"][j]]
    out, og = 0.0, [0.0, 0.0, 0.0]
    to = [[x[q] - v[:, a, q] for q in range(3)] for a in range(4)]
    rr = [torch.sqrt(_dot(t, t)) for t in to]
    for a in range(4):
        b = (a + 1) % 4
        e = [v[:, b, q] - v[:, a, q] for q in range(3)]
        l2 = _dot(e, e)
        live = torch.sqrt(l2.detach()) >= 1e-3 * rad
        ln = torch.sqrt(torch.where(live, l2, torch.ones_like(l2)))
        u = [e[q] / ln for q in range(3)]
        yx = [nv[1] * u[2] - nv[2] * u[1], nv[2] * u[0] - nv[0] * u[2], nv[0] * u[1] - nv[1] * u[0]]
        gy = _dot(to[a], yx)
        s = rr[a] + rr[b]
        s = torch.where(live, s, s + 2.0)
        ant, dnt = 2 * gy * ln, s * s - ln * ln + 2 * agz * s
        anl, dnl = s + ln, s - ln
        lg = torch.log(anl / dnl)
        at = torch.where(use, torch.atan2(ant, dnt), torch.zeros_like(ant))
        mask = live.to(ln.dtype)
        out = out + mask * (torch.where(gy.detach().abs() > 1e-5, gy * lg, torch.zeros_like(gy)) - 2 * agz * at)
        qq, den = gy * (dnl - anl) / (anl * dnl), ant * ant + dnt * dnt
        for q in range(3):
            dl = to[b][q] / rr[b] + to[a][q] / rr[a]
            dn = 2 * (s + agz) * dl + 2 * sg * s * nv[q]
            g = lg * yx[q] - 2 * sg * at * nv[q] + qq * dl - 2 * agz * (2 * ln * yx[q] * dnt - dn * ant) / den
            og[q] = og[q] - mask * g
    full = lambda t: torch.zeros((n, n), dtype=t.dtype, device=t.device).index_put((i, j), t)  # noqa: E731
    return one + full(out), [grad[q] + full(og[q]) for q in range(3)]


def _still(m, direct):
    """The parts of S and D that do not depend on the frequency."""
    x = m["centers"].T
    way = 1.0 if direct else -1.0
    s1, g1 = _rankine(x, m)
    s2, g2 = _rankine([x[0], x[1], -x[2]], m)
    nn = [m["normals"][:, q][None, :] if direct else m["normals"][:, q][:, None] for q in range(3)]
    g = [way * (g1[0] + g2[0]), way * (g1[1] + g2[1]), way * g1[2] + g2[2]]
    eye = torch.eye(len(m["radii"]), dtype=s1.dtype, device=s1.device)
    return -(s1 + s2) / (4 * math.pi), 0.5 * eye - _dot(nn, g) / (4 * math.pi)


def _matrices(m, k, still, kind, direct):
    c = m["centers"].T
    dx, dy = c[0][:, None] - c[0][None, :], c[1][:, None] - c[1][None, :]
    h2 = dx * dx + dy * dy
    on = (h2.detach() > 0)
    r = k * torch.where(on, torch.sqrt(torch.where(on, h2, torch.ones_like(h2))), torch.zeros_like(h2))
    z = k * (c[2][:, None] + c[2][None, :])
    g, gr, gz = _wave(kind, r, z)
    far = r.detach() > 1e-6
    f = torch.where(far, k * k / torch.where(far, r, torch.ones_like(r)), torch.zeros_like(r)) * (-1.0 if direct else 1.0)
    nn = [m["normals"][:, q][None, :] if direct else m["normals"][:, q][:, None] for q in range(3)]
    ka = k * m["areas"][None, :] / (4 * math.pi)
    side, up = f * (nn[0] * dx + nn[1] * dy), k * nn[2]
    s = torch.complex(still[0] - ka * g[0], -ka * g[1])
    d = torch.complex(still[1] - ka * (side * gr[0] + up * gz[0]), -ka * (side * gr[1] + up * gz[1]))
    return s, d


def _one(m, w, still, kind, direct, dofs, betas):
    """Forces at one frequency: F (influenced, right-hand side), FK (influenced, heading)."""
    k = w * w / G
    s, d = _matrices(m, k, still, kind, direct)
    nd = _dot([m["normals"][:, q] for q in range(3)], [dofs[:, :, q] for q in range(3)])  # (dof, panel)
    c = m["centers"].T
    rhs, waves = [torch.complex(torch.zeros_like(nd), -w * nd)], []
    for beta in betas:
        cb, sb = math.cos(beta), math.sin(beta)
        phase, decay = k * (c[0] * cb + c[1] * sb), torch.exp(k * c[2])
        e = torch.complex(torch.cos(phase), torch.sin(phase)) * decay
        vn = (G * k / w) * e * torch.complex(m["normals"][:, 0] * cb + m["normals"][:, 1] * sb, -m["normals"][:, 2])
        rhs.append(-vn[None])
        waves.append(RHO * G * e)
    b = torch.cat(rhs).T
    phi = torch.linalg.solve(d, s @ b) if direct else s @ torch.linalg.solve(d, b)
    wgt = -(nd * m["areas"][None, :])
    wc = torch.complex(wgt, torch.zeros_like(wgt))
    f = wc @ (1j * RHO * w * phi)
    fk = wc @ torch.stack(waves, dim=1) if waves else torch.zeros((len(dofs), 0), dtype=f.dtype, device=f.device)
    return f, fk


def _outputs(fs, fks, omegas, d):
    f, fk = torch.stack(fs, dim=2), torch.stack(fks, dim=1)  # (dof, rhs, w), (dof, w, beta)
    a, b = f[:, :d].real / omegas ** 2, f[:, :d].imag / omegas
    return a, b, f[:, d:].transpose(1, 2), fk


def exact(case, seed):
    x = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    names = ("vertices", "centers", "normals", "areas")
    put = lambda a: torch.tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
    m = {q: put(x[q]) for q in (*names, "radii", "faces")}
    call, kind, direct, d = case["call"], case["wave"], case["direct"], case["n_dof"]
    dofs, omegas, betas = put(x["dofs"]), put(x["omegas"]), list(x["betas"])
    host = lambda t: t.detach().resolve_conj().cpu().numpy()  # noqa: E731
    if call == "assemble":
        s, dd = _matrices(m, omegas[0] ** 2 / G, _still(m, direct), kind, direct)
        return host(s), host(dd)
    if call in ("radiation", "diffraction"):
        heave = torch.zeros((1, *m["centers"].shape), dtype=torch.float64, device=dev)
        heave[:, :, 2] = 1.0
        f, _ = _one(m, omegas[0], _still(m, direct), kind, direct, heave, betas if call == "diffraction" else [])
        if call == "diffraction":
            return host(f[0, 1:2])
        return host(torch.stack([f[0, 0].real / omegas[0] ** 2, f[0, 0].imag / omegas[0]]))
    if call == "batch":
        still = _still(m, direct)
        got = [_one(m, w, still, kind, direct, dofs, betas) for w in omegas]
        return tuple(host(t) for t in _outputs([g[0] for g in got], [g[1] for g in got], omegas, d))
    if call == "jvp":
        fw = torch.autograd.forward_ad
        with fw.dual_level():
            for q in ("vertices", "centers", "areas"):
                m[q] = fw.make_dual(m[q], put(x["t_" + q]))
            still = _still(m, direct)
            got = [_one(m, w, still, kind, direct, dofs, betas) for w in omegas]
            two = [fw.unpack_dual(t) for t in _outputs([g[0] for g in got], [g[1] for g in got], omegas, d)]
        out = {q: host(t.primal) for q, t in zip("ABFK", two)}
        out.update({"d" + q: host(torch.zeros_like(t.primal) if t.tangent is None else t.tangent) for q, t in zip("ABFK", two)})
        return out
    for q in names:
        m[q].requires_grad_()
    dofs.requires_grad_()
    omegas.requires_grad_()
    still = _still(m, direct)
    loose = [t.detach().requires_grad_() for t in still]
    bars = [put(x[q]) for q in ("bar_A", "bar_B", "bar_F", "bar_K")]
    fs, fks = [], []
    for z in range(case["n_omega"]):  # a frequency at a time, so that one frequency's graph is held
        f, fk = _one(m, omegas[z], loose, kind, direct, dofs, betas)
        a, b, ff, kk = _outputs([f], [fk], omegas[z:z + 1], d)
        total = (a * bars[0][:, :, z:z + 1]).sum() + (b * bars[1][:, :, z:z + 1]).sum()
        for out, bar in ((ff, bars[2][:, z:z + 1]), (kk, bars[3][:, z:z + 1])):
            total = total + (out.real * bar.real + out.imag * bar.imag).sum()
        total.backward()
        fs.append(f.detach())
        fks.append(fk.detach())
    torch.autograd.backward(still, [t.grad for t in loose])
    out = {q: host(t) for q, t in zip("ABFK", _outputs(fs, fks, omegas.detach(), d))}
    out.update({q: host(m[q].grad) for q in names})
    out.update(omegas=host(omegas.grad), dofs=list(host(dofs.grad)))
    return out
