"""The workloads whose speed this library is held to: what a user steps, through the public Python
binding and the C ABI, over the sizes, operators, responses and precisions of the configurations,
tests and benchmark.

A pass advances a scenario (or a batch of them) by a number of time steps and reads the whole state
back: the nine fields of both blocks and, with friction, the slip and state of the fault, in the
precision the scenario computes in.  Scenarios start from a seeded wave field that fills the
blocks, as in the middle of a run, so that absorbing layers, memory variables and the return map
have work to do.

`exact` is a plain FP64 solver of the same equations: summation-by-parts differences in flux form
on a general curvilinear grid, penalty boundary conditions, absorbing layers, friction,
viscoplasticity, attenuation and the five-stage low-storage Runge-Kutta scheme.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "waveqlab3d-gh_gb300"))

import wql  # noqa: E402

RHO, CS, CP = 2.67, 3.464, 6.0
DEV = "cuda"
_ctx = None


def context():
    global _ctx
    if _ctx is None:
        _ctx = wql.Context(0)
    return _ctx


# ------------------------------------------------------------------ cases ----

def case(name, mesh, nq1, nq2, nr, ns, steps, precision="fp32c", op="traditional", order=6, pml=0, fault="locked",
         response="elastic", hetero=False, source=False, members=0):
    c = dict(mesh=mesh, nq1=nq1, nq2=nq2, nr=nr, ns=ns, steps=steps, precision=precision, op=op, order=order, pml=pml,
             fault=fault, response=response, hetero=hetero, source=source, members=members)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest run in use: the CPU-sized benchmark problem (2 x 41^3, slip weakening), where launches and
        # latency count
        case("small_sw", "cartesian", 41, 41, 41, 41, 200, fault="sw"),
        # the same class of problem in the FP64 parity mode, on a curvilinear grid of odd extents
        case("fp64_curv_sw", "curvilinear", 67, 59, 71, 73, 20, precision="fp64", fault="sw"),
        # FP64 with absorbing layers on a heterogeneous Cartesian grid
        case("fp64_cart_pml", "cartesian", 75, 75, 81, 77, 16, precision="fp64", pml=10, hetero=True),
        # a served request: point source, stations and a heterogeneous medium in a locked Cartesian pair
        case("request", "cartesian", 76, 75, 150, 150, 60, hetero=True, source=True),
        # an ordinary rupture on a rough fault under topography, odd extents
        case("rough_sw", "curvilinear", 101, 93, 107, 113, 60, fault="sw"),
        # the headline benchmark: 2 x 201^3 curvilinear, rate-and-state friction
        case("rate_state", "curvilinear", 201, 201, 201, 201, 40, fault="rs"),
        # the largest: 2 x 401 x 201^2, 20-point absorbing layers, random medium, viscoplasticity
        case("plastic_pml", "curvilinear", 401, 401, 201, 201, 20, pml=20, fault="sw", response="plastic", hetero=True),
        # the upwind operators with absorbing layers and a point source, the absorbing-layer study's shape
        case("upwind_pml", "cartesian", 76, 76, 101, 151, 60, op="upwind", pml=12, source=True),
        # the same with attenuation
        case("upwind_anelastic", "cartesian", 76, 76, 101, 151, 40, op="upwind", pml=12, response="anelastic",
             source=True),
        # a table operator (upwind-DRP), as an operator study runs it
        case("drp", "cartesian", 76, 76, 101, 91, 20, op="upwind_drp", order=6, source=True),
        # an ensemble of uneven ruptures advanced as one batch, alternately flat and rough, 10-point layers
        case("ensemble", "mixed", 64, 64, 64, 112, 15, pml=10, fault="sw", hetero=True, members=6),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["sw", "sw", "rs", "request", "plastic", "upwind", "anelastic", "fp64", "fp64_pml", "drp", "ensemble"])
    mesh = rng.choice(["cartesian", "curvilinear"])
    hetero = rng.random() < 0.5
    if kind in ("sw", "rs"):
        dims = [size(41, 200) for _ in range(4)]
        c = case(None, mesh if kind == "sw" else "curvilinear", *dims, 0, fault=kind, hetero=hetero,
                 pml=rng.choice([0, 10]))
    elif kind == "request":
        n = size(96, 200)
        c = case(None, "cartesian", n // 2 + 1, n - n // 2, n, n, 0, hetero=hetero, source=True)
    elif kind == "plastic":
        c = case(None, "curvilinear", size(80, 300), size(80, 300), size(80, 180), size(80, 180), 0,
                 pml=rng.randint(10, 20), fault="sw", response="plastic", hetero=hetero)
    elif kind in ("upwind", "anelastic"):
        c = case(None, mesh, size(51, 150), size(51, 150), size(60, 150), size(60, 150), 0, op="upwind",
                 pml=rng.choice([8, 12]), response="anelastic" if kind == "anelastic" else "elastic", source=True)
    elif kind in ("fp64", "fp64_pml"):
        c = case(None, mesh, size(41, 100), size(41, 100), size(41, 100), size(41, 100), 0, precision="fp64",
                 fault="sw" if kind == "fp64" else "locked", pml=10 if kind == "fp64_pml" else 0, hetero=hetero)
    elif kind == "drp":
        op, order = rng.choice([("upwind", 4), ("upwind", 7), ("upwind_drp", 4), ("upwind_drp", 6), ("upwind", 5)])
        c = case(None, "cartesian", size(41, 110), size(41, 110), size(41, 110), size(41, 110), 0, op=op, order=order,
                 source=True)
    else:
        lo = size(64, 96)
        c = case(None, "mixed", lo, lo, lo, lo + size(8, 48), 0, pml=10, fault="sw", hetero=hetero,
                 members=rng.randint(3, 8))
    # as many steps as keep a pass in the range of the listed ones
    rate = 3e7 if c["precision"] == "fp64" or kind == "drp" else (2e8 if kind == "anelastic" else 5e8)
    c["steps"] = max(8, min(60, int(rate / sum(points(m) for m in members(c)))))
    return c


def members(c):
    """The scenarios of a case: itself, or the members of its batch."""
    if not c["members"]:
        return [c]
    out = []
    for i in range(c["members"]):
        n = c["nr"] + (c["ns"] - c["nr"]) * i // max(1, c["members"] - 1)
        out.append(dict(c, mesh="curvilinear" if i % 2 else "cartesian", nq1=n, nq2=n, nr=n, ns=n, members=0,
                        hetero=c["hetero"] and i % 4 < 2))
    return out


def points(c):
    return (c["nq1"] + c["nq2"]) * c["nr"] * c["ns"]


def extents(c):
    """Spacing 0.1 km along r and s, blocks joined at x = 0, free surface at y = 0."""
    return 0.1 * (c["nq1"] - 1), 0.1 * (c["nq2"] - 1), 0.1 * (c["nr"] - 1), 0.1 * (c["ns"] - 1)


def time_step():
    return 0.5 * 0.1 / math.sqrt(CS * CS + CP * CP)


def pml_sides(c, b):
    """Absorbing layers on every outer side but the free surface: -q, +q, -r, +r, -s, +s."""
    on = c["pml"] > 0
    return [on and b == 0, on and b == 1, False, on, on, on]


def sw_params():
    return dict(fs=0.677, fd=0.525, Dc=0.4, s0=(-120.0, -120.0, -120.0, 0.0, 71.8, 0.0), amp=12.0, radius=1.5,
                rise=0.0)


def rs_params():
    return dict(a=0.008, b=0.012, V0=1e-6, f0=0.6, L=0.02, Vini=1e-12, s0=(-120.0, 0.0, -120.0, 0.0, 75.0, 0.0),
                amp=25.0, radius=1.5, rise=0.15)


def deck(c):
    """The case as the reference's namelist input."""
    x1, x2, y, z = extents(c)
    t = (c["steps"] * 1000 + 0.5) * time_step()
    coupling = {"locked": "locked", "sw": "slip-weakening_friction", "rs": "rate-and-state_friction"}[c["fault"]]
    problem = {"locked": "TPV5", "sw": "sw_param", "rs": "rs_param"}[c["fault"]]
    extra = ""
    if c["op"] != "traditional":
        extra += f",\n fd_type = '{c['op']}',\n order = {c['order']}"
    if c["response"] != "elastic":
        extra += f",\n response = '{c['response']}'"
    if c["response"] == "plastic":
        extra += ",\n plastic_model = 'scec'"
    wf = "T" if c["fault"] != "locked" and not c["members"] else "F"
    s = (f"&problem_list\n name = 'case',\n problem = '{problem}',\n nblocks = 2,\n t_final = {t!r},\n CFL = 0.5d0,\n"
         f" coupling = '{coupling}',\n type_of_mesh = '{c['mesh']}',\n w_stride = 10,\n w_fault = {wf}{extra} /\n&block_list\n")
    for b, (n, a, e) in enumerate(((c["nq1"], -x1, 0.0), (c["nq2"], 0.0, x2))):
        p = pml_sides(c, b)
        tf = ["T" if v else "F" for v in p]
        i = b + 1
        s += (f"btp({i})%nqrs = {n}, {c['nr']}, {c['ns']},\nbtp({i})%aqrs = {a!r}, 0.0, {-z / 2!r},\n"
              f"btp({i})%bqrs = {e!r}, {y!r}, {z / 2!r},\nbtp({i})%rho_s_p = {RHO!r}, {CS!r}, {CP!r},\n"
              f"btp({i})%lqrs = {1 - b}, 2, 1,\nbtp({i})%rqrs = {b}, 1, 1,\n")
        if c["pml"]:
            s += (f"btp({i})%pml_lqrs = {tf[0]}, {tf[2]}, {tf[4]},\nbtp({i})%pml_rqrs = {tf[1]}, {tf[3]}, {tf[5]},\n"
                  f"btp({i})%npml = {c['pml']},\n")
    s += " /\n"
    if c["fault"] != "locked":
        f = sw_params() if c["fault"] == "sw" else rs_params()
        keys = ("fs", "fd", "Dc") if c["fault"] == "sw" else ("a", "b", "V0", "f0", "L", "Vini")
        s += ("&fault_list\n " + ", ".join(f"{k} = {f[k]!r}" for k in keys) + ",\n s0 = " +
              ", ".join(repr(v) for v in f["s0"]) + f",\n nuc_amp = {f['amp']!r}, nuc_radius = {f['radius']!r}, "
              f"nuc_y = {y / 2!r}, nuc_z = 0.0, nuc_rise = {f['rise']!r},\n barrier_y = 1000.0, barrier_z = 1000.0 /\n")
    if c["response"] == "plastic":
        s += "&plastic_list\n cohesion = 0.5, friction = 0.75, Tv = 0.03 /\n"
    if c["response"] == "anelastic":
        s += "&anelastic_list\n c = 2.0,\n weight_exp = 0.6,\n fref = 1.0 /\n"
    if c["source"]:
        # a double couple off the grid points of block 1, order-2 delta, and 32 stations on the free surface
        s += ("&moment_list\n use_moment_tensor = T,\n order = 2 /\n!---begin:tensor_listU---\n" +
              "'gaussian' 20.0 0.1 " + " ".join(repr(v) for v in SOURCE_M) +
              f" {-0.437 * x1!r} {0.521 * y!r} {0.031 * z!r} 0\n!---end:tensor_listU---\n"
              "!---begin:tensor_listV---\n!---end:tensor_listV---\n"
              "&output_list\n output_seismograms = T /\n!---begin:station_list---\n")
        for k in range(32):
            s += f"{-x1 + (x1 + x2) * (k + 0.5) / 32!r} 0d0 {z * (((7 * k) % 32) / 32 - 0.48)!r}\n"
        s += "!---end:station_list---\n"
    return s


SOURCE_M = (0.1, -0.2, 0.1, 0.3, -0.4, 0.2)


# ----------------------------------------------------------------- inputs ----

def filtered_noise(shape, power, seed):
    """White noise shaped in Fourier space by `power(k^2)` (k in cycles per point), unit standard deviation."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    w = torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)
    k2 = 0.0
    for d, n in enumerate(shape):
        k = torch.fft.rfftfreq(n, device=DEV, dtype=torch.float64) if d == len(shape) - 1 else torch.fft.fftfreq(
            n, device=DEV, dtype=torch.float64)
        k2 = k2 + (k * k).reshape([-1 if e == d else 1 for e in range(len(shape))])
    f = torch.fft.irfftn(torch.fft.rfftn(w) * power(k2), s=shape)
    f = f - f.mean()
    return f / f.std()


def geometry(c, seed):
    """(fault offset (ns, nr), the two blocks' topography (ns, nq)) in km, or None on a Cartesian grid."""
    if c["mesh"] != "curvilinear":
        return None
    n = (c["ns"], c["nr"])
    rough = filtered_noise(n, lambda k2: torch.where((k2 > 0) & (k2 < 0.25), 1.0 / torch.clamp(k2, min=1e-4), 0.0), seed)
    topo = filtered_noise((c["ns"], c["nq1"] + c["nq2"] - 1), lambda k2: torch.exp(-k2 * (math.pi * 10.0) ** 2 / 2), seed + 1)
    # 1 % of the fault's length and 50 m of relief
    rough = rough * 0.005 * 0.1 * (max(n) - 1)
    topo = 0.05 * topo
    return rough, (topo[:, :c["nq1"]].contiguous(), topo[:, c["nq1"] - 1:].contiguous())


def medium(c, seed):
    """lambda, mu, rho of the two blocks, each (3, ns, nr, nq): homogeneous, or a von Karman medium (5 %)."""
    n = (c["ns"], c["nr"], c["nq1"] + c["nq2"] - 1)
    if c["hetero"]:
        p = 0.05 * filtered_noise(n, lambda k2: (1.0 + k2 * (2 * math.pi * 20.0) ** 2) ** -0.85, seed + 2)
        p = torch.clamp(p, -0.2, 0.2)
    else:
        p = torch.zeros(n, device=DEV, dtype=torch.float64)
    cp, cs = CP * (1 + p), CS * (1 + p)
    rho = 1.6612 * cp - 0.4721 * cp ** 2 + 0.0671 * cp ** 3 - 0.0043 * cp ** 4 + 0.000106 * cp ** 5 if c["hetero"] else RHO + p
    mu = rho * cs * cs
    m = torch.stack([rho * cp * cp - 2 * mu, mu, rho])
    return m[..., :c["nq1"]], m[..., c["nq1"] - 1:]


def wave(c, b, seed):
    """The starting field of a block, (9, ns, nr, nq): plane-wave products of 12 to 40 points' length, about
    0.02 m/s and 0.3 MPa; with friction it fades towards the fault, which starts at rest."""
    g = torch.Generator().manual_seed(seed * 2 + b)
    n = (c["ns"], c["nr"], c["nq1"] if b == 0 else c["nq2"])
    out = torch.zeros((9,) + n, dtype=torch.float64, device=DEV)
    for comp in range(9):
        for _ in range(3):
            ax = []
            for d in range(3):
                length, phase = 12 + 28 * torch.rand((), generator=g).item(), 6.28 * torch.rand((), generator=g).item()
                ax.append(torch.sin(torch.arange(n[d], dtype=torch.float64, device=DEV) * (2 * math.pi / length) + phase))
            amp = (0.02 if comp < 3 else 0.3) * (0.5 + torch.rand((), generator=g).item())
            out[comp] += amp * ax[0][:, None, None] * ax[1][None, :, None] * ax[2][None, None, :]
    if c["fault"] != "locked":
        d = torch.arange(n[2], dtype=torch.float64, device=DEV)
        d = (n[2] - 1 - d) if b == 0 else d
        out *= 1 - torch.exp(-(d / 8) ** 2)
    return out


class State:
    pass


def prepare_one(c, seed):
    S = State()
    S.case = c
    f64 = c["precision"] == "fp64"
    media = {}
    geo = geometry(c, seed)
    if geo is not None:
        media["fault_offset"] = geo[0].cpu().numpy().ravel()
        media["topo_offset"] = tuple(t.cpu().numpy().ravel() for t in geo[1])
    if c["hetero"]:
        blocks = [m.cpu().numpy() for m in medium(c, seed)]
        for k, key in enumerate(("lam", "mu", "rho")):
            media[key] = tuple(m[k].ravel() for m in blocks)
    S.scn = wql.Scenario(context(), text=deck(c), precision=wql.FP64 if f64 else wql.FP32C, media=media or None)
    # the buffers that a program which takes snapshots keeps: pinned staging of one component and the
    # snapshot itself, in the precision of the run
    S.out, big = [], 0
    for b in range(2):
        w = wave(c, b, seed).cpu().numpy()
        for k in range(9):
            S.scn.set_field(b, k, w[k])
        n = w.shape[1:]
        big = max(big, n[0] * n[1] * n[2])
        dt = torch.float64 if f64 else torch.float32
        S.out.append([torch.zeros((3,) + n, dtype=dt), torch.zeros((6,) + n, dtype=dt)])
    S.stage = torch.zeros(big, dtype=torch.float64, pin_memory=True)
    return S


def prepare(c, seed):
    S = State()
    S.steps = c["steps"]
    S.parts = [prepare_one(m, seed + 1000 * i) for i, m in enumerate(members(c))]
    S.batch = None
    if c["members"]:
        S.batch = wql.Batch(context())
        for p in S.parts:
            S.batch.add(p.scn)
    return S


# -------------------------------------------------------------------- run ----

def snapshot(p):
    """The state of one scenario: per block the velocities and the stresses, and with friction the slip of both
    fault copies (strike, dip, total) and, under rate and state, the state variable."""
    L, f64 = wql.lib(), p.case["precision"] == "fp64"
    for b in range(2):
        for k in range(9):
            dst = p.out[b][0][k] if k < 3 else p.out[b][1][k - 3]
            src = p.stage[:dst.numel()]
            if L.wql_get_field(p.scn.h, b, k, ctypes.c_void_p(src.data_ptr())):
                raise RuntimeError("wql_get_field failed")
            dst.copy_(src.view(dst.shape))
    got = [p.out[0][0], p.out[0][1], p.out[1][0], p.out[1][1]]
    dt = np.float64 if f64 else np.float32
    if p.case["fault"] != "locked":
        got.append(np.stack([p.scn.iface(k, w) for k in range(2) for w in (1, 2, 3)]).astype(dt))
    if p.case["fault"] == "rs":
        got.append(np.stack([p.scn.iface(k, 4) for k in range(2)]).astype(dt))
    return got


def run(S):
    if S.batch is not None:
        S.batch.step(S.steps)
    else:
        S.parts[0].scn.step(S.steps)
    return [snapshot(p) for p in S.parts]


# ------------------------------------------------------------------- work ----

def work(c):
    """Per point and stage: the fields and rates read and written, the compensation (FP32C: 2 bytes), and the
    coefficients read; per absorbing-layer point and side the nine auxiliary fields and rates read and written; with
    attenuation 24 memory variables and rates read and written.  Once per pass the state is read out."""
    by, fl = 0.0, 0.0
    for m in members(c):
        w = 8 if m["precision"] == "fp64" else 4
        n = points(m)
        per = (36 + (13 if m["mesh"] == "curvilinear" else 3)) * w + (36 if w == 4 else 0)
        flops = 420 if m["mesh"] == "curvilinear" else 260
        if m["response"] == "anelastic":
            per += (96 + 1) * w
            flops += 250
        if m["response"] == "plastic":
            per += 13 * w / 5
            flops += 60 / 5
        slab = 0
        for b, nq in enumerate((m["nq1"], m["nq2"])):
            p = pml_sides(m, b)
            slab += m["pml"] * (nq * m["ns"] * (p[2] + p[3]) + nq * m["nr"] * (p[4] + p[5]) + m["nr"] * m["ns"] * (p[0] + p[1]))
        by += 5 * m["steps"] * (n * per + slab * 36 * w) + 9 * n * w
        fl += 5 * m["steps"] * (n * flops + slab * 120)
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------------------ exact ----

SBP = ((-1.582533518939116, 2.033378678700676, -0.141512858744873, -0.450398306578272, 0.104488069284042, 0.036577936277544),
       (-0.462059195631158, 0.0, 0.287258622978251, 0.258816087376832, -0.069112065532624, -0.014903449191300),
       (0.071247104721830, -0.636451095137907, 0.0, 0.606235523609147, -0.022902190275815, -0.018129342917256),
       (0.114713313798970, -0.290087484386815, -0.306681191361148, 0.0, 0.520262285050482, -0.051642265516119,
        0.013435342414630),
       (-0.036210680656541, 0.105400944933782, 0.015764336127392, -0.707905442575989, 0.0, 0.769199413962647,
        -0.164529643265203, 0.018281071473911),
       (-0.011398193015050, 0.020437334208704, 0.011220896474665, 0.063183694641876, -0.691649024426814, 0.0,
        0.739709139060752, -0.147941827812150, 0.016437980868017))
UP = ((-1.593253459452621, 2.093702214477299, -0.275607596716317, -0.302855902188632, 0.023993033880123, 0.054021710000147),
      (-0.460835552271137, -0.029551468764759, 0.393228064437077, 0.105980141988699, 0.030739159126096, -0.039560344515975),
      (0.096333139747688, -0.629259919521358, -0.306540940575249, 1.258766829227482, -0.589452745232692, 0.197069524204597,
       -0.026915887850467),
      (0.0925965903611, -0.240558007429252, -0.243684445410829, -0.318292975073623, 0.946962507015985, -0.330443502642251,
       0.106765523632994, -0.013345690454124),
      (-0.015609194255155, 0.033485250803205, 0.041897570295664, -0.450132219590077, -0.593528379527062, 1.406282074938901,
       -0.550950133911491, 0.146920035709731, -0.018365004463716),
      (-0.0161631016574, 0.040531470682718, -0.00533856744421, -0.025427590054054, -0.357460227911152, -0.572337434946968,
       1.313958528183954, -0.492734448068983, 0.131395852818395, -0.016424481602299))
UM = ((-1.58018369620741, 2.039450367044345, -0.189297839436616, -0.366971721882124, 0.044953974933765, 0.05204891554804),
      (-0.473094335557797, 0.029551468764759, 0.279404147185598, 0.215422101432619, -0.021790841692085, -0.029492540133095),
      (0.140255933237354, -0.88560840157053, 0.306540940575249, 0.491468255323896, -0.061405392278187, 0.008748664712219),
      (0.076418487423426, -0.11834612889915, -0.624133691970994, 0.318292975073623, 0.327107204245208, 0.020661154127888),
      (-0.008331008040049, -0.047235828122731, 0.402190050630647, -1.303115093827634, 0.593528379527062, 0.399693508760138,
       -0.036730008927433),
      (-0.016775726857039, 0.054367610816546, -0.120254802392339, 0.406675342006739, -1.257688453771463, 0.572337434946968,
       0.394187558455186, -0.032848963204599))
CENTRAL = {-3: -1 / 60, -2: 0.15, -1: -0.75, 1: 0.75, 2: -0.15, 3: 1 / 60}
FORWARD = dict(zip(range(-2, 5), (1 / 30, -2 / 5, -7 / 12, 4 / 3, -1 / 2, 2 / 15, -1 / 60)))
BACKWARD = {-o: -w for o, w in FORWARD.items()}
RK_A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
        -1275806237668 / 842570457699)
RK_B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
        3134564353537 / 4481467310338, 2277821191437 / 14882151754819)
RK_C = (0.0, 1432997174477 / 9575080441755, 2526269341429 / 6820363962896, 2006345519317 / 3224310063776,
        2802321613138 / 2924317926251)


def diff(u, axis, op):
    """First derivative along axis (0 q, 1 r, 2 s) of (..., s, r, q) arrays, index spacing 1/(n-1); op 'c', '+', '-'."""
    left, right, inner = {"c": (SBP, SBP, CENTRAL), "+": (UP, UM, FORWARD), "-": (UM, UP, BACKWARD)}[op]
    d = u.dim() - 1 - axis
    n = u.shape[d]
    out = torch.empty_like(u)
    mid = out.narrow(d, 6, n - 12)
    mid.zero_()
    for o, w in inner.items():
        mid.add_(u.narrow(d, 6 + o, n - 12), alpha=w)
    for i in range(6):
        a, z = out.select(d, i), out.select(d, n - 1 - i)
        a.zero_()
        z.zero_()
        for k, w in enumerate(left[i]):
            a.add_(u.select(d, k), alpha=w)
        for k, w in enumerate(right[i]):
            z.add_(u.select(d, n - 1 - k), alpha=-w)
    return out.mul_(n - 1)


SIG = ((3, 6, 7), (6, 4, 8), (7, 8, 5))


class Block:
    """One block of the plain solver."""

    def __init__(s, c, b, seed):
        s.c, s.b, s.up = c, b, c["op"] == "upwind"
        s.dp, s.dm = ("+", "-") if s.up else ("c", "c")
        nq, nr, ns = (c["nq1"], c["nq2"])[b], c["nr"], c["ns"]
        s.n = (nq, nr, ns)
        x1, x2, y, z = extents(c)
        r = [torch.arange(k, dtype=torch.float64, device=DEV) / (k - 1) for k in s.n]
        one = torch.ones((ns, nr, nq), dtype=torch.float64, device=DEV)
        X = [one * ((-x1 + x1 * r[0]) if b == 0 else x2 * r[0]), one * (y * r[1])[None, :, None],
             one * (-z / 2 + z * r[2])[:, None, None]]
        s.fault_y = X[1][:, :, -1 if b == 0 else 0].clone()
        s.fault_z = X[2][:, :, -1 if b == 0 else 0].clone()
        geo = geometry(c, seed)
        if geo is not None:
            X[0] += geo[0][:, :, None] * (r[0] if b == 0 else 1 - r[0])
            X[1] += geo[1][b][:, None, :] * (1 - r[1])[None, :, None]
            s.fault_y = X[1][:, :, -1 if b == 0 else 0].clone()
        # grid[j][d]: derivative of coordinate j along axis d (central rows); metric m[j][d] of xi_d along x_j
        G = [[diff(X[j], d, "c") for d in range(3)] for j in range(3)]
        J = (G[0][0] * (G[1][1] * G[2][2] - G[2][1] * G[1][2]) - G[1][0] * (G[0][1] * G[2][2] - G[2][1] * G[0][2]) +
             G[2][0] * (G[0][1] * G[1][2] - G[1][1] * G[0][2]))
        s.m = [[None] * 3 for _ in range(3)]
        for j in range(3):
            j1, j2 = (j + 1) % 3, (j + 2) % 3
            for d in range(3):
                d1, d2 = (d + 1) % 3, (d + 2) % 3
                s.m[j][d] = (G[j1][d1] * G[j2][d2] - G[j2][d1] * G[j1][d2]) / J
        s.J = J
        lam, mu, rho = (v.contiguous() for v in medium(c, seed)[b])
        if c["response"] == "anelastic":
            lo, hi = 1 / (2 * math.pi * 15.0), 200.0 / (2 * math.pi * 0.08)
            s.tau = [math.exp(math.log(lo) + (2 * k - 1) / 16 * (math.log(hi) - math.log(lo))) for k in range(1, 5)]
            s.w = (0.0336, 0.6873, 0.8767, 1.5202)
            s.qs = 1 / (2.0 * torch.sqrt(mu / rho))
            vS = sum(w / (((2 * math.pi) ** 2 * t * t + 1) / s.qs) for w, t in zip(s.w, s.tau))
            vP = sum(w / (((2 * math.pi) ** 2 * t * t + 1) / (0.5 * s.qs)) for w, t in zip(s.w, s.tau))
            M = (lam + 2 * mu) / (1 - vP)
            mu = mu / (1 - vS)
            lam = M - 2 * mu
            s.eta = torch.zeros((24,) + tuple(J.shape), dtype=torch.float64, device=DEV)
            s.deta = torch.zeros_like(s.eta)
        s.lam, s.mu, s.rho = lam, mu, rho
        s.F = wave(c, b, seed)
        s.DF = torch.zeros_like(s.F)
        tau0 = 42300 / 13613 if s.up else 1 / 0.315949074074074
        s.tau_h = [tau0 * (k - 1) for k in s.n]
        s.bc = [1 - b, b, 2, 1, 1, 1]
        s.slabs = {side: None for side in range(6) if pml_sides(c, b)[side]}
        for side in s.slabs:
            shape = list(s.F.shape)
            shape[3 - side // 2] = c["pml"]
            s.slabs[side] = [torch.zeros(shape, dtype=torch.float64, device=DEV) for _ in range(2)]
        s.src = None

    def basis(s, axis, at):
        """Unit normal along the gradient of xi_axis and two tangents on one face, and |gradient|."""
        g = torch.stack([at(s.m[j][axis]) for j in range(3)])
        norm = g.pow(2).sum(0).sqrt()
        n = g / norm
        t = torch.zeros_like(n)
        t[2 if axis == 1 else 1] = 1.0
        m = t - (n * t).sum(0) * n
        m = m / m.pow(2).sum(0).sqrt()
        return n, m, torch.linalg.cross(n, m, dim=0), norm

    def boundary(s, side):
        """Characteristic outer penalty of one face: the rate term and the auxiliary-field term."""
        axis, hi = side // 2, side % 2
        at = lambda v: v.select(v.dim() - 1 - axis, -1 if hi else 0)  # noqa: E731
        n, m, l, norm = s.basis(axis, at)
        u = at(s.F)
        lam, mu, rho = at(s.lam), at(s.mu), at(s.rho)
        Zp, Zs = torch.sqrt((lam + 2 * mu) * rho), torch.sqrt(mu * rho)
        r = {1: 0.0, 2: 1.0}[s.bc[side]]
        sg = 1.0 if hi else -1.0
        T = torch.stack([n[0] * u[SIG[j][0]] + n[1] * u[SIG[j][1]] + n[2] * u[SIG[j][2]] for j in range(3)])
        p, q = 0.0, 0.0
        for e, Z in ((l, Zs), (m, Zs), (n, Zp)):
            v, t = (e * u[:3]).sum(0), (e * T).sum(0)
            p = p + e * (0.5 * ((1 - r) * Z * v + sg * (1 + r) * t))
            q = q + e * (0.5 * ((1 - r) * v + sg * (1 + r) * t / Z))
        ub = torch.stack([norm * p[0], norm * p[1], norm * p[2], sg * norm * n[0] * q[0], sg * norm * n[1] * q[1],
                          sg * norm * n[2] * q[2], sg * norm * (n[1] * q[0] + n[0] * q[1]),
                          sg * norm * (n[2] * q[0] + n[0] * q[2]), sg * norm * (n[2] * q[1] + n[1] * q[2])])
        tr = lam * (ub[3] + ub[4] + ub[5])
        sat = torch.cat([ub[:3] / rho, 2 * mu * ub[3:6] + tr, mu * ub[6:]])
        return at, s.tau_h[axis] * sat, s.tau_h[axis] * ub

    def strain(s):
        g = [[0.0] * 3 for _ in range(3)]
        for comp in range(3):
            for d in range(3):
                D = diff(s.F[comp], d, s.dp)
                for j in range(3):
                    g[comp][j] = g[comp][j] + s.m[j][d] * D
        return g

    def divergence(s, comp, axes):
        """(1/J) sum_d D_d(J sum_{j in axes} m_jd sigma_{comp,j})."""
        out = 0.0
        for d in range(3):
            f = sum(s.J * s.m[j][d] * s.F[SIG[comp][j]] for j in axes)
            out = out + diff(f, d, s.dm)
        return out / s.J

    def rates(s, A, Bdt, fault_sat, amp):
        c, F, DF = s.c, s.F, s.DF
        lam, mu = s.lam, s.mu
        g = s.strain()
        DF.mul_(A)
        for comp in range(3):
            DF[comp] += s.divergence(comp, (0, 1, 2)) / s.rho
        tr = lam * (g[0][0] + g[1][1] + g[2][2])
        for j in range(3):
            DF[3 + j] += tr + 2 * mu * g[j][j]
        DF[6] += mu * (g[0][1] + g[1][0])
        DF[7] += mu * (g[0][2] + g[2][0])
        DF[8] += mu * (g[1][2] + g[2][1])
        outer = {side: s.boundary(side) for side in range(6) if 1 <= s.bc[side] <= 3}
        for side, (at, sat, _) in outer.items():
            at(DF).sub_(sat)
        face = DF.select(3, -1 if s.b == 0 else 0)
        face.sub_(fault_sat)
        if s.src is not None:
            lo, delta = s.src
            for k in range(6):
                DF[3 + k][lo[2]:lo[2] + delta.shape[0], lo[1]:lo[1] + delta.shape[1], lo[0]:lo[0] + delta.shape[2]] -= (
                    amp * SOURCE_M[k] * delta)
        damped = [0.0] * 6
        for side, (Q, DQ) in s.slabs.items():
            axis, hi, np_ = side // 2, side % 2, c["pml"]
            d, n = 3 - axis, s.n[axis]
            lo = n - np_ if hi else 0
            cut = lambda v: v.narrow(v.dim() - 1 - axis, lo, np_)  # noqa: E731
            i = torch.arange(np_, dtype=torch.float64, device=DEV)
            off = i + 1 if hi else (i + 1 - np_ if axis == 2 else i - np_)
            damp = (3 * math.log(1000.0) * (off / np_).abs()).reshape([-1 if e == d - 1 else 1 for e in range(3)])
            l, m_ = cut(lam), cut(mu)
            part = cut(DF)
            for k in range(3):
                part[k] -= damp * Q[k] / cut(s.rho)
            t = l * (Q[3] + Q[4] + Q[5])
            for k in range(3):
                part[3 + k] -= damp * (t + 2 * m_ * Q[3 + k])
                part[6 + k] -= m_ * damp * Q[6 + k]
            if c["response"] == "anelastic":
                for k in range(6):
                    if not torch.is_tensor(damped[k]):
                        damped[k] = torch.zeros_like(s.J)
                for k in {0: (0, 3, 4), 1: (1, 3, 5), 2: (2, 4, 5)}[axis]:
                    cut(damped[k]).add_(damp * Q[3 + k])
            new = A * DQ - (damp + 1.0) * Q
            for comp in range(3):
                new[comp] += cut(s.divergence(comp, (axis,)))
            new[3 + axis] += cut(g[axis][axis])
            for o in range(3):
                if o != axis:
                    new[SIG[axis][o]] += cut(g[o][axis])
            if side in outer:
                new.select(d, np_ - 1 if hi else 0).sub_(outer[side][2])
            DQ.copy_(new)
        if c["response"] == "anelastic":
            e = [g[0][0], g[1][1], g[2][2], g[0][1] + g[1][0], g[0][2] + g[2][0], g[1][2] + g[2][1]]
            e = [a - b_ for a, b_ in zip(e, damped)]
            t = e[0] + e[1] + e[2]
            for k in range(6):
                DF[3 + k] -= s.eta[4 * k:4 * k + 4].sum(0)
                for i in range(4):
                    w = s.w[i]
                    f = w * mu * s.qs * e[k] * (2 if k < 3 else 1)
                    if k < 3:
                        f = f + w * ((lam + 2 * mu) * 0.5 * s.qs - 2 * mu * s.qs) * t
                    j = 4 * k + i
                    s.deta[j].mul_(A).add_((f - s.eta[j]) / s.tau[i])
            s.eta.add_(s.deta, alpha=Bdt)
        for Q, DQ in s.slabs.values():
            Q.add_(DQ, alpha=Bdt)

    def update(s, Bdt):
        s.F.add_(s.DF, alpha=Bdt)

    def plastic(s):
        """The scec return map outside the absorbing layers (uniform initial stress)."""
        w, p, n = s.c["pml"], pml_sides(s.c, s.b), s.n
        box = s.F[:, w * p[4]:n[2] - w * p[5], w * p[2]:n[1] - w * p[3], w * p[0]:n[0] - w * p[1]]
        s0 = sw_params()["s0"]
        a = [box[3 + k] + s0[k] for k in range(6)]
        mean = (a[0] + a[1] + a[2]) / 3
        J2 = ((a[0] - a[1]) ** 2 + (a[1] - a[2]) ** 2 + (a[2] - a[0]) ** 2) / 6 + a[3] ** 2 + a[4] ** 2 + a[5] ** 2
        tau, th = torch.sqrt(J2), math.atan(0.75)
        Y = torch.clamp(0.5 * math.cos(th) - mean * math.sin(th), min=0.0)
        e = math.exp(-time_step() / 0.03)
        r = torch.where(tau > Y, e + (1 - e) * Y / tau, 1.0)
        for k in range(6):
            sd = a[k] - mean if k < 3 else a[k]
            box[3 + k] = torch.where(tau > Y, (mean if k < 3 else 0.0) + r * sd - s0[k], box[3 + k])


class Fault:
    """The interface condition, one copy per block."""

    def __init__(s, c, B):
        s.c, s.B = c, B
        s.par = sw_params() if c["fault"] == "sw" else (rs_params() if c["fault"] == "rs" else None)
        nf = (c["ns"], c["nr"])
        s.S = torch.zeros((2, 4) + nf, dtype=torch.float64, device=DEV)
        s.DS = torch.zeros_like(s.S)
        s.W = torch.zeros((2,) + nf, dtype=torch.float64, device=DEV)
        s.DW = torch.zeros_like(s.W)
        s.at = [lambda v: v[..., -1], lambda v: v[..., 0]]
        s.geo, s.T0 = [], []
        for b in range(2):
            n, m, l, norm = B[b].basis(0, s.at[b])
            s.geo.append((n, m, l, norm))
            if s.par is None:
                continue
            p = s.par["s0"]
            ten = ((p[0], p[3], p[4]), (p[3], p[1], p[5]), (p[4], p[5], p[2]))
            t = torch.stack([sum(ten[i][j] * n[j] for j in range(3)) for i in range(3)])
            y, z = B[b].fault_y, B[b].fault_z
            T0 = [(n * t).sum(0), (m * t).sum(0), (l * t).sum(0)]
            if c["fault"] == "rs":
                r = s.par
                v = torch.log(2 * torch.sinh(T0[2] / (r["a"] * -T0[0])))
                th = r["L"] / r["V0"] * torch.exp((r["a"] * v - r["f0"] - r["a"] * math.log(r["Vini"] / r["V0"])) / r["b"])
                s.W[b] = r["f0"] + r["b"] * torch.log(r["V0"] / r["L"] * th)
            dy = y - 0.05 * (c["nr"] - 1)
            s.T0.append(T0 + [s.par["amp"] * torch.exp(-(dy * dy + z * z) / (2 * s.par["radius"] ** 2))])

    def slip_rate(s, b, Phi, eta, sn):
        """The rate-and-state slip rate: bisection in ln V, then Newton."""
        r, psi = s.par, s.W[b]
        a = r["a"] * sn / eta
        rhs = Phi / eta
        f = lambda u: torch.exp(u) + a * torch.asinh(torch.exp(u + psi / r["a"]) / (2 * r["V0"])) - rhs  # noqa: E731
        lo, hi = torch.full_like(Phi, -200.0), torch.log(rhs)
        for _ in range(60):
            mid = 0.5 * (lo + hi)
            up = f(mid) > 0
            lo, hi = torch.where(up, lo, mid), torch.where(up, mid, hi)
        u = hi
        for _ in range(3):
            w = torch.exp(u + psi / r["a"]) / (2 * r["V0"])
            u = u - f(u) / (torch.exp(u) + a * w / torch.sqrt(1 + w * w))
        return torch.exp(u)

    def ramp(s, t):
        """The nucleation patch's time function."""
        x = t / s.par["rise"] if s.par["rise"] else 1.0
        return 1.0 if x >= 1 else (math.exp((x - 1) ** 2 / (x * (x - 2))) if x > 0 else 0.0)

    def solve(s, A, Bdt, t):
        B, sat = s.B, []
        U = [s.at[b](B[b].F) for b in range(2)]
        mat = [[s.at[b](v) for v in (B[b].lam, B[b].mu, B[b].rho)] for b in range(2)]
        Z = [(torch.sqrt((l + 2 * m) * r), torch.sqrt(m * r)) for l, m, r in mat]
        for b in range(2):
            n, m, l, norm = s.geo[b]
            e = (n, m, l)
            rot = []
            for u in U:
                T = torch.stack([sum(n[j] * u[SIG[i][j]] for j in range(3)) for i in range(3)])
                rot.append(([(k * u[:3]).sum(0) for k in e], [(k * T).sum(0) for k in e]))
            (uv, ut), (vv, vt) = rot
            Zu, Zv = (Z[0][0], Z[0][1], Z[0][1]), (Z[1][0], Z[1][1], Z[1][1])
            p = [Zu[k] * uv[k] - ut[k] for k in range(3)]
            q = [Zv[k] * vv[k] + vt[k] for k in range(3)]
            eta = [1 / (1 / Zu[k] + 1 / Zv[k]) for k in range(3)]
            phi = [eta[k] * (q[k] / Zv[k] - p[k] / Zu[k]) for k in range(3)]
            hat, V = list(phi), [torch.zeros_like(phi[0])] * 3
            if s.par is not None:
                T0 = s.T0[b]
                Tl = T0[2] + T0[3] * s.ramp(t)
                f1, f2 = T0[1] + phi[1], Tl + phi[2]
                Phi = torch.sqrt(f1 * f1 + f2 * f2)
                sn = torch.clamp(-(T0[0] + phi[0]), min=0.0)
                if s.c["fault"] == "sw":
                    r = s.par
                    tau = sn * (r["fs"] - (r["fs"] - r["fd"]) * torch.clamp(s.S[b, 3], max=r["Dc"]) / r["Dc"])
                    rate = torch.clamp((Phi - tau) / eta[1], min=0.0)
                else:
                    r = s.par
                    rate = s.slip_rate(b, Phi, eta[1], sn)
                    s.DW[b] = A * s.DW[b] + (r["b"] * r["V0"] / r["L"] * torch.exp(-(s.W[b] - r["f0"]) / r["b"]) -
                                             rate * r["b"] / r["L"])
                V = [V[0], f1 * rate / Phi, f2 * rate / Phi]
                hat = [phi[0], f1 - eta[1] * V[1] - T0[1], f2 - eta[1] * V[2] - Tl]
            # hat velocities of the two sides: characteristics kept, traction continuous, given slip rate
            uh = [(q[k] - hat[k]) / Zv[k] - V[k] for k in range(3)]
            vh = [(p[k] + hat[k]) / Zu[k] + V[k] for k in range(3)]
            jump = [vh[k] - uh[k] for k in range(3)]
            s.DS[b, :3] = A * s.DS[b, :3] + torch.stack(jump)
            s.DS[b, 3] = A * s.DS[b, 3] + torch.sqrt(jump[1] ** 2 + jump[2] ** 2)
            own_v, own_t, hv = (uv, ut, uh) if b == 0 else (vv, vt, vh)
            sg = 1.0 if b == 0 else -1.0
            back = lambda a: sum(e[k] * a[k] for k in range(3))  # noqa: E731
            lam, mu, rho = mat[b]
            Zp, Zs = Z[b]
            # the reference weights the Cartesian components (x, y, z) of the basis by (Zp, Zs, Zs)
            E = torch.stack(e)
            Zk = torch.stack([Zp, Zs, Zs])
            M = torch.einsum("rkab,ckab,kab->rcab", E, E, Zk)
            Pm = torch.einsum("rkab,ckab,kab->rcab", E, E, 1 / Zk)
            dv, dt = back([x - h for x, h in zip(own_v, hv)]), back([x - h for x, h in zip(own_t, hat)])
            dch = 0.5 * (torch.einsum("rcab,cab->rab", M, dv) + sg * dt)
            rr = torch.einsum("rcab,cab->rab", Pm, dch)
            g = norm * n
            tr = lam * (g * rr).sum(0)
            out = torch.stack([norm / rho * dch[0], norm / rho * dch[1], norm / rho * dch[2]] +
                              [sg * (tr + 2 * mu * g[k] * rr[k]) for k in range(3)] +
                              [sg * mu * (g[1] * rr[0] + g[0] * rr[1]), sg * mu * (g[2] * rr[0] + g[0] * rr[2]),
                               sg * mu * (g[2] * rr[1] + g[1] * rr[2])])
            sat.append(B[b].tau_h[0] * out)
        s.S.add_(s.DS, alpha=Bdt)
        if s.c["fault"] == "rs":
            s.W.add_(s.DW, alpha=Bdt)
        return sat


def place_source(c, B):
    """The order-2 discrete delta of the case's source on block 1 (Cartesian grids)."""
    x1, _, y, z = extents(c)
    pos, n = (-0.437 * x1 + x1, 0.521 * y, 0.031 * z + z / 2), (c["nq1"], c["nr"], c["ns"])
    lo, w = [], []
    for d in range(3):
        h = 0.1
        i0 = min(n[d] - 1, int(math.floor(pos[d] / h + 0.5)))
        a = pos[d] / h - i0
        beta, gam, gap = (1 - 2 * a) / 4 + 0.25, (2 * a - 1) / 16, (2 * a + 1) / 16
        lo.append(i0 - 2)
        w.append(torch.tensor([-gam, beta + 3 * gam - gap, 1 - a - 2 * beta - 3 * gam + 3 * gap, a + beta + gam - 3 * gap,
                               gap], dtype=torch.float64, device=DEV) / h)
    B.src = (lo, w[2][:, None, None] * w[1][None, :, None] * w[0][None, None, :])


def exact_one(c, seed):
    B = [Block(c, b, seed) for b in range(2)]
    if c["source"]:
        place_source(c, B[0])
    fault = Fault(c, B)
    dt = time_step()
    for step in range(c["steps"]):
        for k in range(5):
            A, Bdt = RK_A[k], RK_B[k] * dt
            t = (step + RK_C[k]) * dt
            sat = fault.solve(A, Bdt, t)
            amp = 20.0 / math.sqrt(2 * math.pi) * math.exp(-(20.0 ** 2) * (t - 0.1) ** 2 / 2)
            for b in range(2):
                B[b].rates(A, Bdt, sat[b], amp)
            for b in range(2):
                B[b].update(Bdt)
                if c["response"] == "plastic" and k == 4:
                    B[b].plastic()
    out = [B[0].F[:3], B[0].F[3:], B[1].F[:3], B[1].F[3:]]
    if c["fault"] != "locked":
        out.append(fault.S[:, 1:].reshape(6, c["ns"], c["nr"]))
    if c["fault"] == "rs":
        out.append(fault.W)
    return out


def exact(c, seed):
    """None for the table operators, for sources on curvilinear grids (their delta follows the local spacing) and for
    runs of more than about 20 seconds."""
    if c["op"] != "traditional" and (c["op"], c["order"]) != ("upwind", 6):
        return None
    if c["source"] and c["mesh"] != "cartesian":
        return None
    if 5 * c["steps"] * sum(points(m) for m in members(c)) > 5e9:
        return None
    return [exact_one(m, seed + 1000 * i) for i, m in enumerate(members(c))]
