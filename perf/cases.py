"""Timed cases: the runs that a user of this engine makes, through its public calls.

A case is one tracking job as a GENESIS user sets it up: a beam and one or more
radiation fields of a given size, an undulator lattice, the arithmetic form (plain
FP64, or mixed with an FP32 field), the field solver and the options of the run. One
pass starts the job from its initial state, integrates it over its lattice steps and
reads back the slice diagnostics, the particles and the fields:

  restart "upload"  beam and field come from pinned host memory (load_beam / load_field),
                    as a run started from loaded arrays;
  restart "device"  the initial state is kept in a second handle and copied on the device
                    (copy_state_from), as scans and the learned closure restart a run;
  records "every"   every step's diagnostics (run_diag), as output at every step;
  records "end"     steps only (run, optionally as one captured graph), then one record.

The beams have the structure that quiet loading gives them (beamlets of four members
that share energy and transverse coordinates, phases spread over the bucket, shot
noise on top); they are made with torch from the seed alone, on the GPU, so that a
checker can make the same inputs. Sizes and physics are those of the benchmark and the
test cases: 4 x 110-period planar modules with FODO quadrupoles at aw 1.7, the helical
Example1 undulator, grids of 101 to 255 points over 1e-4 to 2e-4 m, 2048 to 16384
particles a slice.

The mixed form keeps its field, coordinates and energy offsets in FP32 and the library
hands them out widened to FP64; a program that keeps such a run's results keeps them in
FP32, and so do the mixed cases.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "genesis-1.3-version4_gb300"))
import g4gpu  # noqa: E402

GAMMA0 = 11357.82
EEV, VACIMP, QE, CLIGHT = 510998.95069, 376.73, 1.602176634e-19, 299792458.0
# planar: the benchmark's undulator at its resonant wavelength; offres: the same at the
# benchmark's own 1 A (2.26 slices of slippage a period); helical: Example1's, resonant
UNDULATORS = {
    "planar": dict(aw=1.7, lambdau=0.015, helical=0, kx=0.0, ky=1.0, lambda0=0.015 * (1 + 1.7 ** 2) / 2 / GAMMA0 ** 2),
    "offres": dict(aw=1.7, lambdau=0.015, helical=0, kx=0.0, ky=1.0, lambda0=1e-10),
    "helical": dict(aw=0.84853, lambdau=0.015, helical=1, kx=0.5, ky=0.5, lambda0=1e-10),
}
PERIODS, QUAD_K1, QUAD_L = 110, 1.5, 0.08  # periods a module, FODO quadrupole between modules


def _case(name, form, undulator, nslice, npart, ngrid, steps, *, gridmax=1e-4, solver="adi", harm="1", time_run=True,
          power=0.0, restart="upload", records="every", graph=False, shapes="", efield="", filtered=False, counts=False,
          members=1):
    return dict(name=name, form=form, undulator=undulator, nslice=nslice, npart=npart, ngrid=ngrid, steps=steps,
                gridmax=gridmax, solver=solver, harm=harm, time_run=time_run, power=power, restart=restart,
                records=records, graph=graph, shapes=shapes, efield=efield, filtered=filtered, counts=counts,
                members=members)


def listed():
    return [
        # one steady-state slice with a 5 kW seed, Example1 of the reference, reference
        # arithmetic: the smallest job, where launches and latency count
        _case("steady_fp64", "plain", "helical", 1, 8192, 255, 111, gridmax=2e-4, time_run=False, power=5e3),
        # the same kind of job in the mixed form, replayed as a captured graph (a taper or
        # detuning scan runs many of these)
        _case("steady_mixed", "mixed", "planar", 1, 8192, 151, 221, time_run=False, power=1e3, records="end", graph=True),
        # a short pulse of odd sizes in reference arithmetic, as tests and small studies run
        _case("pulse_fp64", "plain", "helical", 22, 2052, 101, 60, power=1e4),
        # part of the benchmark's window in reference arithmetic
        _case("window_fp64", "plain", "planar", 320, 8192, 151, 12),
        # an ordinary time-dependent window, mixed, every step's diagnostics
        _case("window_mixed", "mixed", "planar", 700, 8192, 151, 48, power=1e4, restart="device"),
        # the benchmark's whole window (4096 x 8192 from shot noise), launch shapes as the
        # tuner sets them on this card
        _case("sase_mixed", "mixed", "offres", 4096, 8192, 151, 48, restart="device", shapes="128 1024 0"),
        # a wide beam on Example1's grid of 255 points
        _case("wide_grid_mixed", "mixed", "helical", 300, 8192, 255, 40, gridmax=2e-4, power=5e3, restart="device",
              records="end"),
        # harmonics 1, 3 and 5 with the FFT field solver (the benchmark's harmonic window, a
        # quarter of its slices)
        _case("harmonics_fft_mixed", "mixed", "planar", 512, 16384, 255, 16, gridmax=2e-4, solver="fft", harm="1 3 5",
              power=1e3, restart="device", records="end"),
        # the FFT solver with the source filter, reference arithmetic
        _case("filtered_fft_fp64", "plain", "helical", 64, 4096, 128, 24, gridmax=2e-4, solver="fft", power=1e4,
              filtered=True),
        # space charge: one short-range mode and the long-range loss
        _case("space_charge_mixed", "mixed", "planar", 512, 8192, 151, 40, power=1e4, restart="device",
              efield="1 0 1"),
        # a one4one window: slices hold different numbers of particles
        _case("one4one_mixed", "mixed", "helical", 150, 6000, 117, 48, power=1e4, counts=True),
        # an ensemble of uneven runs advanced together (one graph launch for all)
        _case("ensemble_mixed", "mixed", "planar", 120, 4096, 151, 32, power=1e3, restart="device", records="end",
              members=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _quad(n):
    return max(4, n // 4 * 4)


def draw(rng):
    """One more job of the same kinds: the sizes of a kind spread over its range."""
    kind = rng.choice(["steady", "steady", "window_fp64", "window_mixed", "window_mixed", "wide", "fft_mixed", "fft_fp64",
                       "space_charge", "one4one", "ensemble"])
    pw = 10 ** rng.uniform(2.5, 4.5)
    if kind == "steady":
        form = rng.choice(["plain", "mixed"])
        return _drawn(form, rng.choice(["planar", "helical"]), rng.randint(1, 4), _quad(_log(rng, 1024, 16384)),
                      rng.randint(51, 255), rng.randint(40, 160), gridmax=rng.uniform(1e-4, 2e-4), time_run=False, power=pw,
                      records=rng.choice(["every", "end"]), graph=rng.random() < 0.5)
    if kind == "window_fp64":
        ns = _log(rng, 8, 320)
        return _drawn("plain", rng.choice(["planar", "helical"]), ns, _quad(_log(rng, 1024, 8192)), rng.randint(51, 255),
                      rng.randint(8, 12), gridmax=rng.uniform(1e-4, 2e-4), power=pw)
    if kind == "window_mixed":
        return _drawn("mixed", rng.choice(["planar", "offres", "helical"]), _log(rng, 24, 2048), _quad(_log(rng, 1024, 16384)),
                      rng.randint(61, 167), rng.randint(24, 48), gridmax=rng.uniform(1e-4, 2e-4),
                      power=rng.choice([0.0, pw]), restart="device", records=rng.choice(["every", "end"]))
    if kind == "wide":
        return _drawn("mixed", rng.choice(["planar", "helical"]), _log(rng, 16, 300), _quad(_log(rng, 2048, 16384)),
                      rng.randint(169, 401), rng.randint(16, 40), gridmax=rng.uniform(1.5e-4, 3e-4), power=pw,
                      restart="device", records=rng.choice(["every", "end"]))
    if kind == "fft_mixed":
        return _drawn("mixed", "planar", _log(rng, 16, 512), _quad(_log(rng, 2048, 16384)),
                      rng.choice([101, 120, 128, 151, 165, 200, 225, 243, 250, 255, 256]), rng.randint(8, 16), gridmax=2e-4,
                      solver="fft", harm=rng.choice(["1", "1 3", "1 3 5"]), power=pw, restart="device", records="end",
                      filtered=rng.random() < 0.3)
    if kind == "fft_fp64":
        return _drawn("plain", "helical", _log(rng, 8, 96), _quad(_log(rng, 1024, 8192)),
                      rng.choice([101, 125, 128, 151, 165, 180, 225, 255]), rng.randint(8, 24), gridmax=2e-4, solver="fft",
                      power=pw, filtered=rng.random() < 0.5)
    if kind == "space_charge":
        return _drawn("mixed", rng.choice(["planar", "helical"]), _log(rng, 16, 512), _quad(_log(rng, 1024, 8192)),
                      rng.randint(61, 167), rng.randint(16, 40), power=pw, restart="device",
                      efield=rng.choice(["1 0 1", "1 0 0", "2 1 1", "0 0 1"]))
    if kind == "one4one":
        return _drawn("mixed", "helical", _log(rng, 16, 256), rng.randint(500, 8000), rng.randint(61, 167),
                      rng.randint(16, 48), power=pw, counts=True)
    return _drawn("mixed", "planar", _log(rng, 24, 160), _quad(_log(rng, 2048, 6000)), rng.randint(81, 167),
                  rng.randint(16, 32), power=pw, restart="device", records="end", members=rng.randint(2, 6))


def _drawn(*a, **k):
    c = _case("", *a, **k)
    del c["name"]
    return c


# ---- inputs ------------------------------------------------------------------------


def _lattice(case, taper=0.0):
    """Per-step table of modules of PERIODS one-period steps with a quadrupole between
    them (alternating sign), `steps` rows of it, aw falling linearly by `taper`."""
    u = UNDULATORS[case["undulator"]]
    n, col = case["steps"], {k: i for i, k in enumerate(g4gpu.LAT_COLS)}
    ku = 2 * math.pi / u["lambdau"]
    t = np.zeros((n, g4gpu.LAT_NCOL))
    drift, z = 0.0, 0.0
    for i in range(n):
        r = t[i]
        r[col["z"]] = z
        if i % (PERIODS + 1) == PERIODS:
            r[col["qf"]] = QUAD_K1 if (i // (PERIODS + 1)) % 2 == 0 else -QUAD_K1
            r[col["dz"]] = QUAD_L
            drift += QUAD_L
        else:
            aw = u["aw"] * (1 - taper * i / max(n - 1, 1))
            r[col["aw"]], r[col["ku"]], r[col["helical"]] = aw, ku, u["helical"]
            r[col["kx"]], r[col["ky"]] = ku * ku * u["kx"], ku * ku * u["ky"]
            r[col["dz"]] = u["lambdau"]
            r[col["slip"]] = u["lambdau"] * (1 + aw * aw) / (2 * GAMMA0 ** 2 * u["lambda0"])
            if drift > 0:
                t[i - 1][col["slip"]] += math.floor(drift / 2 / GAMMA0 ** 2 / u["lambda0"]) + 1
                drift = 0.0
        z += r[col["dz"]]
    return t


def _members(case):
    """The runs of a case: the case itself, or an ensemble's members with uneven sizes."""
    out = []
    for m in range(case["members"]):
        c = dict(case)
        if case["members"] > 1:
            c["nslice"] = max(8, case["nslice"] * (m + 1) // 2 + 3 * m)
            c["npart"] = _quad(case["npart"] * (1 + m % 3) // 2)
            c["ngrid"] = case["ngrid"] if m % 2 == 0 else case["ngrid"] * 2 // 3
        out.append((c, 0.004 * m if case["members"] > 1 else 0.0))
    return out


def _inputs(case, seed):
    """Particles [ns][np][6], slice currents, particle counts (or None) and fields
    [ns][ngrid^2] of one run, FP64 on the GPU."""
    ns, npart, ng = case["nslice"], case["npart"], case["ngrid"]
    u = UNDULATORS[case["undulator"]]
    gen = torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 7919)
    f8 = dict(dtype=torch.float64, device="cuda")
    nb = 1 if case["counts"] else 4
    ngrp = npart // nb

    def normal():
        return torch.randn((ns, ngrp, 1), generator=gen, **f8)

    beam = torch.empty((ns, npart, 6), **f8)
    b = beam.view(ns, ngrp, nb, 6)
    sx = math.sqrt(0.4e-6 / GAMMA0 * 15.0)
    spx = math.sqrt(0.4e-6 * GAMMA0 / 15.0)
    b[..., 0] = GAMMA0 + 1.5 * normal()
    for k, s in ((2, sx), (3, sx), (4, spx), (5, spx)):
        b[..., k] = s * normal()
    if case["time_run"]:
        s = torch.arange(ns, **f8) / max(ns - 1, 1)
        cur = 3000.0 * torch.exp(-0.5 * ((s - 0.5) / 0.6) ** 2)
    else:
        cur = torch.full((ns,), 3000.0, **f8)
    two_pi = 2 * math.pi
    th = two_pi * torch.rand((ns, ngrp, 1), generator=gen, **f8) / nb
    th = th + two_pi * torch.arange(nb, **f8) / nb
    if nb > 1:
        # shot noise: a small kick at the fundamental for every beamlet
        ne = cur * u["lambda0"] / CLIGHT / QE / ngrp
        amp = torch.sqrt(-torch.log(torch.rand((ns, ngrp), generator=gen, **f8).clamp_min(1e-12)) / ne[:, None])
        phi = two_pi * torch.rand((ns, ngrp), generator=gen, **f8)
        th = th + (2 * amp)[..., None] * torch.sin(th + phi[..., None])
    b[..., 1] = th
    counts = None
    if case["counts"]:
        counts = torch.randint(max(1, npart // 3), npart + 1, (ns,), generator=gen, device="cuda").to(torch.int32)
    fields = []
    for k, h in enumerate(int(v) for v in case["harm"].split()):
        lam = u["lambda0"] / h
        dgrid, ks = 2 * case["gridmax"] / (ng - 1), two_pi / lam
        x = torch.linspace(-case["gridmax"], case["gridmax"], ng, **f8)
        w0 = 30e-6
        mode = torch.exp(-(x[None, :] ** 2 + x[:, None] ** 2) / w0 ** 2)
        mode = mode * torch.exp(1j * (0.3e5 * x[None, :] + 2e8 * x[:, None] ** 2))
        scl = dgrid * EEV / ks
        amp = math.sqrt(case["power"] / 10 ** k * VACIMP) / scl
        mode = mode * (amp / torch.linalg.vector_norm(mode))
        ph = torch.polar(0.5 + torch.rand(ns, generator=gen, **f8), 0.4 * torch.randn(ns, generator=gen, **f8))
        fields.append((ph[:, None] * mode.reshape(1, -1)).contiguous())
    return beam, cur, counts, fields


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def _config(c):
    return g4gpu.Config(nslice=c["nslice"], npart=c["npart"], ngrid=c["ngrid"], harm=[int(v) for v in c["harm"].split()],
                        gridmax=c["gridmax"], lambda0=UNDULATORS[c["undulator"]]["lambda0"], sample=1.0, gammaref=GAMMA0,
                        precision=g4gpu.MIXED if c["form"] == "mixed" else g4gpu.PLAIN,
                        solver=g4gpu.SOLVER_FFT if c["solver"] == "fft" else g4gpu.SOLVER_ADI,
                        source_filter=int(c["filtered"]), xcut=0.5, ycut=0.4, sigmoid=0.1, time_run=int(c["time_run"]),
                        device=torch.cuda.current_device())


def _efield(c):
    nz, nphi, lr = (int(v) for v in c["efield"].split())
    return dict(rmax=0.0, ngrid=100, nz=nz, nphi=nphi, longrange=bool(lr))


def prepare(case, seed):
    """Handles with their lattice, the initial state (pinned host arrays, or a second
    handle that holds it on the device) and the pinned arrays the results go to."""
    runs = _members(case)
    batch = g4gpu.Batch([_config(c) for c, _ in runs]) if len(runs) > 1 else None
    state = {"batch": batch, "case": case, "runs": []}
    for m, (c, taper) in enumerate(runs):
        beam, cur, counts, fields = _inputs(c, seed * 64 + m)
        h = batch.members[m] if batch else g4gpu.Handle(_config(c))
        lattice = _lattice(c, taper)
        h.set_lattice(lattice)
        if c["shapes"]:
            h.set_launch_shapes(*[int(v) for v in c["shapes"].split()])
        if c["graph"]:
            h.set_graph_mode(True)
        r = {"h": h, "beam_in": _pinned(beam), "cur_in": cur.cpu(), "counts": None if counts is None else counts.cpu().numpy(),
             "field_in": [_pinned(f) for f in fields]}
        mixed = c["form"] == "mixed"
        del beam, fields
        # the results' arrays; a restart from the device no longer needs the inputs' ones
        if c["restart"] == "device":
            r["start"] = g4gpu.Handle(_config(c))
            _load(r["start"], r)
            r["start"].synchronize()
            r["beam"], r["field"] = r.pop("beam_in"), r.pop("field_in")
        else:
            r["beam"] = torch.empty_like(r["beam_in"], pin_memory=True)
            r["field"] = [torch.empty_like(f, pin_memory=True) for f in r["field_in"]]
        if mixed:
            r["beam32"] = torch.empty_like(r["beam"], dtype=torch.float32)
            r["field32"] = [torch.empty_like(f, dtype=torch.complex64) for f in r["field"]]
        nrec = c["steps"] if c["records"] == "every" else 1
        nh = 1 if c["harm"] == "1" else 3
        r["nharm"] = nh
        r["records"] = (np.zeros((nrec, c["nslice"], len(g4gpu.DB_COLS) + 2 * nh)),
                        np.zeros((nrec, len(c["harm"].split()), c["nslice"], len(g4gpu.DF_COLS))))
        r["c"] = c
        state["runs"].append(r)
    torch.cuda.empty_cache()
    return state


def _load(h, r):
    if r["counts"] is not None:
        h.load_beam_counts(r["beam_in"].numpy(), r["cur_in"].numpy(), r["counts"])
    else:
        h.load_beam_ptr(r["beam_in"].data_ptr(), r["cur_in"].data_ptr())
    for k, f in enumerate(r["field_in"]):
        h.load_field_ptr(k, f.data_ptr())


def run(state):
    case = state["case"]
    for r in state["runs"]:
        h = r["h"]
        if "start" in r:
            h.copy_state_from(r["start"])
        else:
            _load(h, r)
        if case["efield"]:
            h.set_efield(**_efield(case))
    if state["batch"] is not None:
        state["batch"].run(0, case["steps"])
    out = []
    for r in state["runs"]:
        h = r["h"]
        if case["records"] == "every":
            bd, fd = h.run_diag(0, case["steps"], nharm=r["nharm"], out=r["records"])
        else:
            if state["batch"] is None:
                h.run(0, case["steps"])
            bd, fd = h.diag(r["nharm"])
        h.get_beam(r["beam"].numpy())
        beam, field = r["beam"], r["field"]
        for k, f in enumerate(field):
            h.get_field(k, f.numpy())
        if "beam32" in r:
            beam = r["beam32"].copy_(beam)
            field = [a.copy_(b) for a, b in zip(r["field32"], field)]
            bd, fd = bd.astype(np.float32), fd.astype(np.float32)
        out.append({"beam": {n: beam[..., i] for i, n in enumerate(("gamma", "theta", "x", "y", "px", "py"))},
                    "field": field, "beam_diag": bd, "field_diag": fd})
    return out


def work(case):
    """Bytes: the state over the host link (or from its device copy) and back, and every
    step's particles and fields read and written once (the state of a job is larger than
    what stays on chip from one step to the next, but for the smallest). Flops: per
    particle and field about 400 for the push and the deposition, per cell about 60 for
    the ADI sweeps or 10 log2(ngrid) for the two transforms of the FFT solver."""
    by = fl = 0.0
    for c, _ in _members(case):
        n, cells = c["nslice"] * c["npart"], c["nslice"] * c["ngrid"] ** 2 * len(c["harm"].split())
        pb, cb = (28, 8) if c["form"] == "mixed" else (48, 16)
        by += 2 * (48 * n + 16 * cells) + c["steps"] * 2 * (pb * n + cb * cells)
        per_cell = 60 if c["solver"] == "adi" else 20 * math.log2(c["ngrid"])
        fl += c["steps"] * (400.0 * n * len(c["harm"].split()) + per_cell * cells)
    return {"bytes": by, "flops": fl}


# ---- the same run in 64 bits, with torch alone -------------------------------------


def _bessel(n, x):
    """J_n(x) by the trapezoidal rule on its integral (spectrally exact)."""
    t = (np.arange(256) + 0.5) * math.pi / 256
    return float(np.mean(np.cos(n * t - x * np.sin(t))))


def _coupling(aw, helical, h):
    if helical:
        return aw if h == 1 else 0.0
    if h % 2 == 0:
        return 0.0
    xi = 0.5 * aw * aw / (1 + aw * aw) * h
    m = (h - 1) // 2
    return aw * (_bessel(m, xi) - _bessel(m + 1, xi)) * (-1) ** m


def _plane(q, dz, x, p, gz):
    if q == 0:
        return x + p * dz / gz, p
    foc = torch.sqrt(abs(q) / gz)
    c, s = (torch.cos(foc * dz), torch.sin(foc * dz)) if q > 0 else (torch.cosh(foc * dz), torch.sinh(foc * dz))
    return c * x + s / foc * p / gz, (-s if q > 0 else s) * foc * gz * x + c * p


def _half(step, dz, P):
    aw = step["aw"]
    bpar = math.sqrt(1 - (1 + aw * aw) / GAMMA0 ** 2)
    qx = step["qf"] * GAMMA0 + step["kx"] * aw * aw / GAMMA0 / bpar
    qy = -step["qf"] * GAMMA0 + step["ky"] * aw * aw / GAMMA0 / bpar
    gz = torch.sqrt(P["gamma"] ** 2 - 1 - aw * aw - P["px"] ** 2 - P["py"] ** 2)
    P["x"], P["px"] = _plane(qx, dz / 2, P["x"], P["px"], gz)
    P["y"], P["py"] = _plane(qy, dz / 2, P["y"], P["py"], gz)


def _cells(P, gm, ng):
    """Lower-left cell, its weights and who lies on the grid."""
    dg = 2 * gm / (ng - 1)
    on = (P["x"].abs() < gm) & (P["y"].abs() < gm)
    tx, ty = torch.where(on, (P["x"] + gm) / dg, 0.0), torch.where(on, (P["y"] + gm) / dg, 0.0)
    ix, iy = tx.floor().clamp(max=ng - 2), ty.floor().clamp(max=ng - 2)
    return on, (ix + iy * ng).long(), 1 - (tx - ix), 1 - (ty - iy)


def _corners(i, wx, wy, ng):
    return ((i, wx * wy), (i + 1, (1 - wx) * wy), (i + ng, wx * (1 - wy)), (i + ng + 1, (1 - wx) * (1 - wy)))


def _tridiag(r, c, dim):
    """(I - i c D) x = r along `dim`, D the second difference with zero ends, by Thomas."""
    r = r.movedim(dim, 0)
    n = r.shape[0]
    a, b = -1j * c, 1 + 2j * c
    cp, d = [a / b], [r[0] / b]
    for k in range(1, n):
        m = b - a * cp[k - 1]
        cp.append(a / m)
        d.append((r[k] - a * d[k - 1]) / m)
    for k in range(n - 2, -1, -1):
        d[k] = d[k] - cp[k] * d[k + 1]
    return torch.stack(d).movedim(0, dim).contiguous()


def _second(u, dim):
    z = torch.zeros_like(u.narrow(dim, 0, 1))
    n = u.shape[dim]
    return torch.cat([u.narrow(dim, 1, n - 1), z], dim) - 2 * u + torch.cat([z, u.narrow(dim, 0, n - 1)], dim)


def _space_charge(c, step, P, valid, cur, rmax, lam):
    ef = _efield(c)
    nz, nphi, ng = ef["nz"], ef["nphi"], ef["ngrid"]
    ns, npart = P["x"].shape
    aw, ks = step["aw"], 2 * math.pi / lam
    loss = torch.zeros(ns, dtype=torch.float64, device="cuda")
    sx, sy = P["x"].std(1, unbiased=False), P["y"].std(1, unbiased=False)
    if ef["longrange"]:
        size = sx * sy
        i = torch.arange(ns, dtype=torch.float64, device="cuda")
        ds = (i[None, :] - i[:, None]) * lam * GAMMA0 / math.sqrt(1 + aw * aw)
        co = 1 - torch.sqrt(ds * ds / (ds * ds + size[None, :]))
        scl = lam / math.pi / CLIGHT / 2 / 8.85e-12
        loss = (torch.sign(ds) * co * scl * cur[None, :] / size[None, :]).sum(1) / EEV
    ez = loss[:, None].expand(ns, npart).clone()
    if nz == 0:
        return ez, rmax
    tx, ty = P["x"] - P["x"].mean(1, keepdim=True), P["y"] - P["y"].mean(1, keepdim=True)
    rad = torch.sqrt(tx * tx + ty * ty)
    bound, ext = rad.amax(1).tolist(), []
    for v in bound:
        rmax = 1.5 * v if v > rmax else rmax
        ext.append(rmax)
    dr = (torch.tensor(ext, dtype=torch.float64, device="cuda") / (ng - 1))[:, None]
    bins = (rad / dr).floor().long().clamp(0, ng - 1)
    phase = torch.complex(tx / rad, ty / rad)
    j = torch.arange(ng, dtype=torch.float64, device="cuda")
    vol = math.pi * dr * dr * (2 * j + 1)[None, :]
    lo, up = 2 * math.pi * j, 2 * math.pi * (j + 1)
    up[-1] = 0
    rlog = torch.log((j + 1) / j.clamp(min=1))
    rlog[0] = 0.5
    coef = -GAMMA0 ** 2 / (1 + aw * aw) / ks / ks
    econ = (VACIMP / EEV * cur / ks / npart)[:, None]
    for m in range(-nphi, nphi + 1):
        mid = -lo - up - 2 * math.pi * m * m * rlog
        mid[-1] -= 2 * math.pi * ng
        for l in range(1, nz + 1):
            wave = phase ** m * torch.polar(torch.ones_like(rad), l * P["theta"])
            src = torch.zeros((ns, ng), dtype=torch.complex128, device="cuda")
            src.scatter_add_(1, bins, wave.conj())
            src = 1j * econ / l / vol * src
            cl, cm, cu = coef * lo / l / l / vol, 1 + coef * mid / l / l / vol, coef * up / l / l / vol
            g, e, bet = [None], [src[:, 0] / cm[:, 0]], cm[:, 0]
            for k in range(1, ng):
                g.append(cu[:, k - 1] / bet)
                bet = cm[:, k] - cl[:, k] * g[k]
                e.append((src[:, k] - cl[:, k] * e[k - 1]) / bet)
            for k in range(ng - 2, -1, -1):
                e[k] = e[k] - g[k + 1] * e[k + 1]
            ez += 2 * (wave * torch.stack(e, 1).gather(1, bins)).real
    return ez, rmax


def _beam_diag(P, valid, nh):
    """The record's beam columns in the library's order."""
    w = valid.double()
    n = w.sum(1)

    def mean(v):
        return (v * w).sum(1) / n

    def ext(v, big, small):
        return [torch.where(valid, v, big).amin(1), torch.where(valid, v, -small).amax(1)]

    g, x, y, px, py = (P[k] for k in ("gamma", "x", "y", "px", "py"))
    m = {k: mean(P[k]) for k in ("gamma", "x", "y", "px", "py")}

    def var(a, b):
        return mean((P[a] - m[a][:, None]) * (P[b] - m[b][:, None]))

    cols = [m["gamma"], var("gamma", "gamma").sqrt(), m["x"], var("x", "x").sqrt(), m["y"], var("y", "y").sqrt(), m["px"],
            m["py"]]
    ex = (var("x", "x") * var("px", "px") - var("x", "px") ** 2).sqrt()
    ey = (var("y", "y") * var("py", "py") - var("y", "py") ** 2).sqrt()
    cols += [ex, ey, var("x", "x") / ex * m["gamma"], var("y", "y") / ey * m["gamma"], -var("x", "px") / ex,
             -var("y", "py") / ey]
    for v in (x, px, y, py, g):
        cols += ext(v, 1e9, 1e9)
    for h in range(1, nh + 1):
        c, s = mean(torch.cos(h * P["theta"])), mean(torch.sin(h * P["theta"]))
        cols += [torch.hypot(c, s), torch.atan2(s, c)]
    return torch.stack(cols, 1)


def _field_diag(u, gm, lam, ng, first):
    ns, dg, ks = u.shape[0], 2 * gm / (ng - 1), 2 * math.pi / lam
    w = u.real ** 2 + u.imag ** 2
    k = torch.arange(ng, dtype=torch.float64, device="cuda") - 0.5 * (ng - 1)
    p = w.sum((1, 2))
    safe = torch.where(p > 0, p, 1.0)
    x1, x2 = (w * k).sum((1, 2)) / safe, (w * k * k).sum((1, 2)) / safe
    y1, y2 = (w * k[:, None]).sum((1, 2)) / safe, (w * (k * k)[:, None]).sum((1, 2)) / safe
    mid, far = u[:, ng // 2, ng // 2], u.sum((1, 2))
    cols = [p * (dg * EEV / ks) ** 2 / VACIMP, x1 * dg, (x2 - x1 * x1).abs().sqrt() * dg, y1 * dg,
            (y2 - y1 * y1).abs().sqrt() * dg, (mid.real ** 2 + mid.imag ** 2) * EEV * EEV / ks / ks / VACIMP,
            torch.atan2(mid.imag, mid.real), (far.real ** 2 + far.imag ** 2) * dg * dg, torch.atan2(far.imag, far.real)]
    return torch.roll(torch.stack(cols, 1), -first, 0)


def _exact_run(c, taper, seed):
    beam, cur, counts, F = _inputs(c, seed)
    ns, npart, ng = c["nslice"], c["npart"], c["ngrid"]
    u = UNDULATORS[c["undulator"]]
    harm, gm, lam0 = [int(v) for v in c["harm"].split()], c["gridmax"], u["lambda0"]
    names = ("gamma", "theta", "x", "y", "px", "py")
    P = {n: beam[..., i].clone() for i, n in enumerate(names)}
    valid = torch.ones((ns, npart), dtype=torch.bool, device="cuda")
    if counts is not None:
        valid = torch.arange(npart, device="cuda")[None, :] < counts[:, None]
    n_of = valid.sum(1).double()
    F = [f.view(ns, ng, ng) for f in F]
    first, acc, rmax = [0] * len(F), [0.0] * len(F), 0.0
    table = _lattice(c, taper)
    dgrid = 2 * gm / (ng - 1)
    nh = 1 if c["harm"] == "1" else 3
    bds, fds = [], []
    xks = 2 * math.pi / lam0
    for i in range(c["steps"]):
        step = dict(zip(g4gpu.LAT_COLS, table[i]))
        aw, dz = step["aw"], step["dz"]
        xku = step["ku"] if step["ku"] else xks * 0.5 / GAMMA0 ** 2
        fc = [_coupling(aw, u["helical"], h) if aw > 0 else 0.0 for h in harm]
        _half(step, dz, P)
        ez = 0.0
        if c["efield"]:
            ez, rmax = _space_charge(c, step, P, valid, cur, rmax, lam0)
        awl = 1 + 0.5 * (step["kx"] * P["x"] ** 2 + step["ky"] * P["y"] ** 2)
        bt = 1 + P["px"] ** 2 + P["py"] ** 2 + (aw * awl) ** 2
        on, cell, wx, wy = _cells(P, gm, ng)
        rows = torch.arange(ns, device="cuda")
        drive = []
        for k, h in enumerate(harm):
            f = F[k].view(ns, -1)[(rows + first[k]) % ns]
            v = sum(f.gather(1, j) * w for j, w in _corners(cell, wx, wy, ng))
            drive.append(torch.where(on, v.conj(), 0.0) * (fc[k] / (h * xks)) * awl)

        def ode(g, th):
            a = sum(d * torch.polar(torch.ones_like(th), -h * th) for d, h in zip(drive, harm))
            e = (bt - 2 / xks * a.real) / (g * g)
            s = torch.sqrt(1 - e)
            return a.imag / s / g - ez, xks * (1 - 1 / s) + xku

        g0, t0 = P["gamma"], P["theta"]
        a1, b1 = ode(g0, t0)
        a2, b2 = ode(g0 + dz / 2 * a1, t0 + dz / 2 * b1)
        a3, b3 = ode(g0 + dz / 2 * a2, t0 + dz / 2 * b2)
        a4, b4 = ode(g0 + dz * a3, t0 + dz * b3)
        P["gamma"] = g0 + dz / 6 * (a1 + 2 * a2 + 2 * a3 + a4)
        P["theta"] = t0 + dz / 6 * (b1 + 2 * b2 + 2 * b3 + b4)
        del a1, a2, a3, a4, b1, b2, b3, b4, drive
        _half(step, dz, P)
        if counts is not None:
            for k, n in enumerate(names):
                P[n] = torch.where(valid, P[n], beam[..., k])
        on, cell, wx, wy = _cells(P, gm, ng)
        for k, h in enumerate(harm):
            src = torch.zeros((ns, ng * ng), dtype=torch.complex128, device="cuda")
            if aw > 0 and h % 2 == 1:
                scl = fc[k] * VACIMP * cur * (h * xks) * dz / (4 * EEV * n_of * dgrid ** 2)
                part = torch.sqrt(1 + step["kx"] * P["x"] ** 2 + step["ky"] * P["y"] ** 2) * scl[:, None] / P["gamma"]
                part = torch.where(on & valid, part, 0.0)
                ph = torch.complex(torch.sin(h * P["theta"]) * part, torch.cos(h * P["theta"]) * part)
                flat = torch.view_as_real(src)
                for j, w in _corners(cell, wx, wy, ng):
                    v = torch.view_as_real(ph * w)
                    for q in (0, 1):
                        flat[..., q].scatter_add_(1, j, v[..., q].contiguous())
            slot = (rows + first[k]) % ns
            src = src.view(ns, ng, ng)
            if first[k]:
                moved = torch.empty_like(src)
                moved[slot] = src
                src = moved
            if c["solver"] == "adi":
                cs = 0.25 * dz / (h * xks * dgrid ** 2)
                r = F[k] + 1j * cs * _second(F[k], 1) + src
                v = _tridiag(r, cs, 2)
                r = v + 1j * cs * _second(v, 2) + src
                F[k] = _tridiag(r, cs, 1)
            else:
                q = torch.arange(ng, dtype=torch.float64, device="cuda") - 0.5 * (ng - 1)
                q = torch.roll(q, (ng + 1) // 2)  # value of index i stored at (i + (n + 1) / 2) % n
                r2 = q[None, :] ** 2 + q[:, None] ** 2
                prop = torch.polar(torch.ones_like(r2), -r2 * (2 * math.pi / ng / dgrid) ** 2 / 2 / (h * xks) * dz)
                if c["filtered"]:
                    rho = torch.sqrt((q[None, :] / ng / 0.5) ** 2 + (q[:, None] / ng / 0.4) ** 2)
                    sig = 1 / (1 + torch.exp((rho - 1) / 0.1))
                    F[k] = torch.fft.ifft2(torch.fft.fft2(F[k]) * prop + 2 * torch.fft.fft2(src) * sig)
                else:
                    F[k] = torch.fft.ifft2(torch.fft.fft2(F[k]) * prop) + 2 * src
            del src
        if c["time_run"]:
            for k in range(len(F)):
                acc[k] += step["slip"]
                while abs(acc[k]) > 0.8:
                    acc[k] -= 1.0
                    first[k] = (first[k] + ns - 1) % ns
                    F[k][first[k]] = 0
        if c["records"] == "every" or i == c["steps"] - 1:
            bds.append(_beam_diag(P, valid, nh))
            fds.append(torch.stack([_field_diag(f, gm, lam0 / h, ng, s) for f, h, s in zip(F, harm, first)]))
    bd, fd = torch.stack(bds), torch.stack(fds)
    if c["records"] == "end":
        bd, fd = bd[0], fd[0]
    return {"beam": {n: P[n] for n in names}, "field": [f.reshape(ns, ng * ng) for f in F], "beam_diag": bd, "field_diag": fd}


def exact(case, seed):
    """What run() returns for these inputs, in 64 bits with torch; None where that would
    take too long."""
    runs = _members(case)
    if sum(c["steps"] * (c["nslice"] * c["npart"] + 0.5 * c["nslice"] * c["ngrid"] ** 2) for c, _ in runs) > 4e9:
        return None
    return [_exact_run(c, taper, seed * 64 + m) for m, (c, taper) in enumerate(runs)]
