"""The work that a user of the transport library has it do, as timed cases.

A case names a structure, a phonon spectrum and one call of the C ABI's Python
mirror (p-trans_b200/abi.py): the gray transmission function that the Fortran
host calls once per mean free path (ptg_transmission), the whole kappa chain in
its three MFP modes (ptg_kappa), the path-reweighting derivatives
(ptg_adjoint) and a batch of screened structures (ptg_batch_run).  Both
precisions are in use: FP32 for production runs, FP64 for runs that have to
repeat the CPU solver's trajectories.  Sizes are those of this repository's configurations, tests and
benchmark, or lie between them.
"""
import importlib.util
import math
import os
import sys

import numpy as np

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "p-trans_b200")
_TWO_PI_THZ = 2.0 * math.pi * 1e12
_FMAX_THZ = 15.0


def _package():
    """The package of this repository (its folder's name is no identifier)."""
    if "ptrans_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location(
            "ptrans_b200", os.path.join(_PKG, "__init__.py"), submodule_search_locations=[_PKG])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["ptrans_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["ptrans_b200"]


def listed():
    return [
        # a first look at a structure: one gray mean free path, few phonons, so
        # launches, copies and the host's share count
        {"name": "gray_film_first_look", "op": "transmission", "structure": "film", "nholes": 3, "modes": 16,
         "nangle": 11, "np": 20, "mfp_nm": 100.0, "fp64": False},
        # the Fortran host's call: TransmissionFunction for one MFP of its loop,
        # every mode of a small table, in a short wide wire
        {"name": "gray_wire", "op": "transmission", "structure": "wire", "length": 200.0, "width": 200.0,
         "modes": 120, "nangle": 11, "np": 100, "mfp_nm": 150.0, "fp64": False},
        # the same in FP64 in a long wire, where the caller compares with the CPU solver
        {"name": "gray_wire_fp64", "op": "transmission", "structure": "wire", "length": 1000.0, "width": 100.0,
         "modes": 120, "nangle": 11, "np": 25, "mfp_nm": 150.0, "fp64": True},
        # the benchmark's workload: porous thin film, 2000 modes each at its own
        # bulk MFP, 64 bins, 10^7 phonons
        {"name": "film_kappa", "op": "kappa", "structure": "film", "nholes": 3, "modes": 2000, "nangle": 11,
         "np": 500, "mfp": "per_mode", "mfp_lo_nm": 1.0, "fp64": False},
        # a porous film in FP64 at a sample of the size that such checks use
        {"name": "film_kappa_fp64", "op": "kappa", "structure": "film", "nholes": 3, "modes": 2000, "nangle": 11,
         "np": 5, "mfp": "per_mode", "mfp_lo_nm": 5.0, "fp64": True},
        # the FP64 nanowire configuration (10^5 phonons, diffuse walls), at the
        # cross-section and length of the parity tests
        {"name": "wire_kappa_fp64", "op": "kappa", "structure": "wire", "length": 300.0, "width": 60.0,
         "modes": 2000, "nangle": 11, "np": 5, "mfp": "per_mode", "mfp_lo_nm": 2.0, "fp64": True},
        # the reference's default without a MeanFreePath key: ballistic phonons,
        # Matthiessen's rule; a finer angle grid and counts that divide by nothing
        {"name": "spheres_matthiessen", "op": "kappa", "structure": "spheres", "modes": 357, "nangle": 31,
         "np": 333, "mfp": "matthiessen", "mfp_lo_nm": 1.0, "fp64": False},
        # the reference's MeanFreePath grid with interpolation, in a polycrystal
        # whose facets let half of the phonons through
        {"name": "voronoi_grid", "op": "kappa", "structure": "voronoi", "grains": 5, "modes": 250, "nangle": 11,
         "np": 401, "mfp": "grid", "nmfp": 7, "mfp_lo_nm": 5.0, "fp64": False},
        # spheres and capped cylinders of random axes, each wall with its own
        # specularity: the composite configuration, the largest case
        {"name": "inclusions_kappa", "op": "kappa", "structure": "inclusions", "spheres": 64, "cylinders": 16,
         "modes": 4000, "nangle": 11, "np": 500, "mfp": "per_mode", "mfp_lo_nm": 1.0, "fp64": False},
        # grains as they come out of a mesher: about 43 000 triangles, a BVH per grain
        {"name": "mesh_kappa", "op": "kappa", "structure": "voronoi", "grains": 5, "tri_levels": 4, "modes": 1000,
         "nangle": 11, "np": 250, "mfp": "per_mode", "mfp_lo_nm": 2.0, "fp64": False},
        # screening: many porous films with uneven sample counts in one launch
        {"name": "films_batch", "op": "batch", "films": 64, "modes": 500, "nangle": 11, "samples_lo": 1e4,
         "samples_hi": 1e6, "mfp_lo_nm": 1.0},
        # derivatives with respect to every wall's specularity and the scattering rates
        {"name": "inclusions_adjoint", "op": "adjoint", "structure": "inclusions", "spheres": 12, "cylinders": 5,
         "modes": 400, "nangle": 11, "np": 250, "mfp": "per_mode", "mfp_lo_nm": 5.0, "fp64": False},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _log_int(rng, lo, hi):
    return int(round(_log_uniform(rng, lo, hi)))


def draw(rng):
    op = rng.choice(["transmission", "transmission", "kappa", "kappa", "kappa", "kappa", "batch", "adjoint"])
    nangle = rng.choice([5, 7, 11, 11, 21, 31])
    if op == "batch":
        films, modes = _log_int(rng, 3, 96), _log_int(rng, 50, 700)
        lo = _log_uniform(rng, 3e3, 1e5)
        return {"op": op, "films": films, "modes": modes, "nangle": nangle, "samples_lo": lo,
                "samples_hi": lo * _log_uniform(rng, 1.0, 10.0), "mfp_lo_nm": _log_uniform(rng, 1.0, 20.0)}
    structure = rng.choice(["film", "film", "wire", "spheres", "voronoi", "inclusions", "mesh"])
    c = {"op": op, "structure": structure, "nangle": nangle, "fp64": False}
    if structure == "film":
        c["nholes"] = rng.randint(1, 3)
    elif structure == "wire":
        c["length"] = float(rng.randint(100, 1000))
        c["width"] = float(rng.randint(40, 200))
    elif structure == "voronoi":
        c["grains"] = rng.randint(2, 9)
    elif structure == "inclusions":
        c["spheres"], c["cylinders"] = rng.randint(1, 64), rng.randint(1, 16)
    elif structure == "mesh":
        c["structure"], c["grains"], c["tri_levels"] = "voronoi", rng.randint(2, 6), rng.randint(1, 4)
    if op == "adjoint":
        total = _log_uniform(rng, 2e4, 1.5e6)
        c["mfp"], c["mfp_lo_nm"] = "per_mode", _log_uniform(rng, 3.0, 50.0)
    elif op == "transmission":
        total = _log_uniform(rng, 2e3, 2e6)
        c["mfp_nm"] = _log_uniform(rng, 20.0, 3000.0)
        c["fp64"] = "tri_levels" not in c and rng.random() < 0.4
        if c["fp64"]:
            total = min(total, 1e5)
    else:
        total = _log_uniform(rng, 2e4, 8e6)
        c["mfp"] = rng.choice(["per_mode", "per_mode", "grid", "matthiessen"])
        c["mfp_lo_nm"] = _log_uniform(rng, 2.0, 20.0)
        if c["mfp"] == "grid":
            c["nmfp"] = rng.randint(2, 9)
        # the plain FP64 runs are checks: small structures, few phonons
        if structure in ("film", "wire", "spheres") and rng.random() < 0.3:
            c["fp64"], total = True, min(total, 1e5)
            c["mfp_lo_nm"] = max(c["mfp_lo_nm"], 5.0)
            if structure == "wire":
                c["length"] = min(c["length"], 400.0)
    if "tri_levels" in c:
        total = min(total, 2e6)
    per_mode_tasks = (nangle - 1) * c.get("nmfp", 1)
    c["modes"] = _log_int(rng, 8, max(9, min(3000, total / per_mode_tasks / 3)))
    c["np"] = max(1, int(total / (c["modes"] * per_mode_tasks)))
    return c


# ---- inputs -------------------------------------------------------------------

def _model(case, seed):
    synth = _package().synth
    s = case["structure"]
    if s == "film":
        return synth.film_with_holes(lx=300.0, ly=300.0, lz=145.0, nholes=case["nholes"], radius=50.0, seed=seed)
    if s == "wire":
        return synth.nanowire(length=case["length"], width=case["width"], height=case["width"], p_side=0.0)
    if s == "spheres":
        # two transmitting inclusions, moved a little by the seed
        d = np.random.default_rng(seed).uniform(-5.0, 5.0, 6)
        return synth.spheres_in_box(l=200.0, centres=((70 + d[0], 90 + d[1], 100 + d[2]),
                                                      (140 + d[3], 110 + d[4], 90 + d[5])),
                                    radii=(30, 32), t=0.5, p=0.3, p_wall=0.2)
    if s == "voronoi":
        return synth.voronoi_box(case["grains"], box=(1000.0, 1000.0, 1000.0), seed=seed, trans=0.5, spec=0.0,
                                 p_wall=0.0, tri_levels=case.get("tri_levels", -1))
    return synth.spheres_cylinders_box(case["spheres"], case["cylinders"], seed=seed)


def _spectrum(case, seed):
    return _package().synth.spectrum(case["modes"], seed=seed, mfp_lo=case.get("mfp_lo_nm", 1.0) * 1e-9)


def _run(case, seed):
    A = _package().abi
    kind = {"per_mode": A.MFP_PER_MODE, "grid": A.MFP_GRID, "matthiessen": A.MFP_MATTHIESSEN}[case.get("mfp", "per_mode")]
    grid = np.geomspace(max(20.0, case["mfp_lo_nm"]), 5000.0, case["nmfp"]) if kind == A.MFP_GRID else None
    return A.make_run(kind_mfp=kind, nangle=case["nangle"], np_=case.get("np", 1), seed=seed + 1, mfp_grid=grid,
                      precision=A.PREC_FP64 if case.get("fp64") else A.PREC_FP32, temperature=300.0, nbins=64,
                      bin_omega=(0.0, _FMAX_THZ * _TWO_PI_THZ))


def prepare(case, seed):
    """The structure built and on the GPU (a handle, or a batch object), the
    spectrum and the run's description."""
    A, synth = _package().abi, _package().synth
    spec = _spectrum(case, seed)
    st = {"case": case, "seed": seed, "run": _run(case, seed)}
    if case["op"] == "batch":
        models, nps = synth.film_batch(case["films"], seed=seed, n_modes=case["modes"], nangle=case["nangle"],
                                       samples_lo=case["samples_lo"], samples_hi=case["samples_hi"])
        st["geometry"] = [A.GeomBuf(m) for m in models]
        st["batch"] = A.Batch([g.view for g in st["geometry"]], nps, [seed + 1 + i for i in range(len(models))],
                              [0] * len(models), spec, st["run"])
        return st
    st["geometry"] = A.GeomBuf(_model(case, seed))
    st["handle"] = A.Handle(st["geometry"].view, spec)
    return st


def run(st):
    A, case = _package().abi, st["case"]
    if case["op"] == "transmission":
        t, e = st["handle"].transmission(case["mfp_nm"], case["nangle"], case["np"], seed=st["seed"] + 1,
                                         precision=A.PREC_FP64 if case["fp64"] else A.PREC_FP32)
        return {"transmit": t, "stderr": e}
    if case["op"] == "adjoint":
        return _numbers(st["handle"].adjoint(st["run"]))
    if case["op"] == "batch":
        return _numbers(st["batch"].run(want_counts=True))
    return _numbers(st["handle"].kappa(st["run"], want_transmit=case["mfp"] == "grid", want_counts=True))


def _numbers(r):
    """A result's numbers: counts as signed integers, without the timings."""
    out = {}
    for k, v in r.items():
        if v is None or k in ("kernel_ms", "graph_ms"):
            continue
        out[k] = v.view(np.int64) if isinstance(v, np.ndarray) and v.dtype == np.uint64 else v
    return out


# ---- the work of a pass --------------------------------------------------------

def work(case):
    """Bytes: the spectrum and the geometry's records in, the tallies and
    results out.  Operations: 60 per free flight (a direction, a free path and
    a move), the flights being what a phonon of that mean free path takes: the
    mean path through a slab between absorbing faces is twice its length
    whatever the scattering (Cauchy), so 2 L / MFP intrinsic events, and a wall
    event every mean chord of the structure."""
    if case["op"] == "batch":
        lo, hi = case["samples_lo"], case["samples_hi"]
        samples = case["films"] * ((hi - lo) / math.log(hi / lo) if hi > lo * 1.001 else lo)
        length, chord, records, tasks = 250.0, 250.0, 14 * case["films"], case["films"]
        tasks *= case["modes"] * (case["nangle"] - 1)
    else:
        tasks = case["modes"] * (case["nangle"] - 1) * case.get("nmfp", 1)
        samples = tasks * case["np"]
        s = case["structure"]
        if s == "film":
            length, records = 300.0, 6 + 2 * case["nholes"]
            chord = 4.0 / (2.0 / 145.0 + case["nholes"] * 2.0 * math.pi * 50.0 / 300.0 ** 2)
        elif s == "wire":
            length, chord, records = case["length"], case["width"], 12
        elif s == "spheres":
            length, chord, records = 200.0, 4.0 / (4 / 200.0 + 2 * 4 * math.pi * 31.0 ** 2 / 200.0 ** 3), 10
        elif s == "voronoi":
            length, chord = 1000.0, 1000.0 / case["grains"] ** (1.0 / 3.0)
            records = 6 + 16 * case["grains"] * (6 * 4 ** case["tri_levels"] if "tri_levels" in case else 1)
        else:
            length, records = 1000.0, 6 + 2 * (case["spheres"] + case["cylinders"])
            chord = 4.0 / (4 / 1000.0 + (case["spheres"] * 4 * math.pi * 55.0 ** 2
                                         + case["cylinders"] * 2 * math.pi * 30.0 * 280.0) / 1000.0 ** 3)
    if case["op"] == "transmission":
        inverse_mfp = 1.0 / case["mfp_nm"]
    elif case.get("mfp", "per_mode") == "matthiessen":
        inverse_mfp = 0.0
    elif case.get("mfp") == "grid":
        inverse_mfp = float(np.mean(1.0 / np.geomspace(max(20.0, case["mfp_lo_nm"]), 5000.0, case["nmfp"])))
    else:  # log-uniform up to 10 um
        inverse_mfp = (1.0 / case["mfp_lo_nm"] - 1.0e-4) / math.log(1.0e4 / case["mfp_lo_nm"])
    flights = samples * (1.0 + 2.0 * length * (inverse_mfp + 1.0 / chord))
    if case["op"] == "adjoint":
        flights *= 2.0  # a forward pass and the replay of what got through
    moved = 5 * 8 * case["modes"] + 112 * records + 8 * tasks
    return {"bytes": float(moved), "flops": 60.0 * flights}


# ---- the same walk in 64 bits ----------------------------------------------------

def exact(case, seed):
    """The transmission function of a short gray wire, walked in 64 bits with
    numpy from the random numbers that the library documents (Philox4x32-10,
    counter = flight, block and sample).  An error of rounding grows with every
    wall event (by one over the cosine of incidence, and much faster behind a
    hole or a sphere), so only where a phonon meets few walls do two walks with
    the same numbers end alike and the tallies have a value to compare with.
    Elsewhere the tallies are one sample of a random result and have none;
    counts stay equal whole numbers there."""
    if case["op"] != "transmission" or case["structure"] != "wire":
        return None
    tasks = case["modes"] * (case["nangle"] - 1)
    if case["length"] > 1.5 * case["width"] or case["length"] > 4.0 * case["mfp_nm"] or tasks * case["np"] > 5e5:
        return None
    counts = _walk_wire((case["length"], case["width"], case["width"]), case["mfp_nm"], case["modes"],
                        case["nangle"], case["np"], seed + 1, case["fp64"])
    t = np.zeros(case["modes"] * case["nangle"])
    t[:tasks] = counts / case["np"]
    t = t.reshape(case["nangle"], case["modes"], 1).transpose(2, 1, 0)
    return {"transmit": t, "stderr": np.sqrt(t * (1.0 - t) / case["np"])}


def _philox(c0, c1, sample, seed):
    """Philox4x32-10 of counters (c0, c1, lo sample, hi sample), as four uint64 arrays of 32-bit words."""
    m = np.uint64(0xFFFFFFFF)
    s = np.uint64(32)
    c0, c1 = c0.astype(np.uint64), np.full(len(sample), c1, np.uint64)
    c2, c3 = sample & m, sample >> s
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c0, np.uint64(0xCD9E8D57) * c2
        c0, c1, c2, c3 = (p1 >> s) ^ c1 ^ np.uint64(k0), p1 & m, (p0 >> s) ^ c3 ^ np.uint64(k1), p0 & m
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _u52(a, b):
    return (((a << np.uint64(20)) | (b >> np.uint64(12))).astype(np.float64) + 0.5) * 2.0 ** -52


def _u23(a):
    return ((a & np.uint64(0x7FFFFF)).astype(np.float64) + 0.5) * 2.0 ** -23


def _walk_wire(box, mfp, modes, nangle, n, seed, fp64):
    """Transmitted counts per task of a box between two baths (x) with diffuse
    side walls.  FP64 runs draw 52-bit numbers, two a block; FP32 runs four of
    23 bits, and do not step off the wall that they left."""
    box = np.array(box)
    sample = np.arange(modes * (nangle - 1) * n, dtype=np.uint64)
    theta = (sample // np.uint64(modes * n)).astype(np.float64) / (nangle - 1) * (math.pi / 2.0)
    counts = np.zeros(modes * (nangle - 1), np.int64)
    zero = np.zeros(len(sample), np.uint64)
    if fp64:
        a, b = _philox(zero, 0, sample, seed), _philox(zero, 1, sample, seed)
        y, z, phi, free = _u52(a[0], a[1]), _u52(a[2], a[3]), _u52(b[0], b[1]), _u52(b[2], b[3])
    else:
        y, z, phi, free = (_u23(w) for w in _philox(zero, 0, sample, seed))
    pos = np.stack([np.zeros(len(sample)), y * box[1], z * box[2]])
    d = np.stack([np.cos(theta), np.sin(theta) * np.cos(2 * math.pi * phi), np.sin(theta) * np.sin(2 * math.pi * phi)])
    free = -mfp * np.log(free)
    flight = 0
    while len(sample):
        flight += 1
        f = np.full(len(sample), flight, np.uint64)
        with np.errstate(divide="ignore", invalid="ignore"):
            t = np.where(d > 0, (box[:, None] - pos) / d, np.where(d < 0, -pos / d, np.inf))
        ax = np.argmin(t, axis=0)
        dist = np.take_along_axis(t, ax[None], 0)[0]
        if not fp64:
            dist = np.maximum(dist, 0.0)
        up = np.take_along_axis(d, ax[None], 0)[0] > 0
        inside = free < dist
        out = ~inside & (ax == 0)
        through = out & up
        np.add.at(counts, (sample[through] // np.uint64(n)).astype(np.int64), 1)
        step = np.where(inside, free, dist)
        pos = pos + step * d
        r = _philox(f, 0, sample, seed)
        if fp64:
            u0, u1 = _u52(r[0], r[1]), _u52(r[2], r[3])
            r1, r2 = _philox(f, 1, sample, seed), _philox(f, 2, sample, seed)
            phi_wall, free_pp, free_wall = _u52(r1[0], r1[1]), _u52(r1[0], r1[1]), _u52(r2[2], r2[3])
            sin2 = u1
        else:
            u0, u1 = _u23(r[0]), _u23(r[1])
            sin2, phi_wall, free_pp = u1, _u23(r[2]), _u23(r[2])
            free_wall = _u23(_philox(f, 1, sample, seed)[1])
        # intrinsic event: an isotropic direction about x
        s = np.sqrt(1.0 - (2.0 * u0 - 1.0) ** 2)
        pp = np.stack([2.0 * u0 - 1.0, s * np.cos(2 * math.pi * u1), s * np.sin(2 * math.pi * u1)])
        # diffuse wall: Lambert about the inward normal, in the wall's frame (t1, t2, n)
        sa, ca = np.sqrt(sin2), np.sqrt(1.0 - sin2)
        a, b = sa * np.cos(2 * math.pi * phi_wall), sa * np.sin(2 * math.pi * phi_wall)
        sg = np.where(up, 1.0, -1.0)
        wall = np.where(ax == 1, np.stack([sg * b, -sg * ca, a]), np.stack([-a, -b, -sg * ca]))
        d = np.where(inside, pp, wall)
        if fp64:
            pos = pos + 1.0e-7 * d
        free = free - step
        spent = free < 1.0e-10
        free = np.where(spent, -mfp * np.log(np.where(inside, free_pp, free_wall)), free)
        keep = ~out
        sample, pos, d, free = sample[keep], pos[:, keep], d[:, keep], free[keep]
    return counts
