"""Performance cases: what a user of mosaic_gb300 has it compute.

Every case goes through a public entry point: one exposure from host arrays
(``beam.atomic_scattering_kinematic``), a staged scan (``BatchedScan.run``),
exact frames of a theta x chi scan by their indices
(``SurrogateScan.exact``), free-space propagation of a detector field
(``propagation.propagate``) and one training step of the scan surrogate's
networks (``MLP``). Sizes are those of the repository's
workloads, tests and benchmark, or scaled between them so that a pass stays
below about a second.

Inputs are made from the seed alone: seeded atomic displacements (the
workloads' thermal model), seeded alloy species, seeded beam and motor
offsets. ``exact`` restates each result in FP64 with plain torch where that
takes seconds.
"""
import math
import os

import numpy as np
import torch

import mosaic_gb300
from mosaic_gb300 import Detector, Stage, workloads
from mosaic_gb300 import beam as Beam
from mosaic_gb300.geometry import align_rotation
from mosaic_gb300.propagation import propagate
from mosaic_gb300.sample import ChunkedSample
from mosaic_gb300.scan import BatchedScan, frames_from_motors
from mosaic_gb300.surrogate import MLP, SurrogateScan

HC_EV_A = 12398.419843320026
R_E = 2.81794092e-15
LATTICE = {"cu": 3.615, "cuni": 3.615, "bumps": 3.615, "poly": 3.615, "nacl": 5.64}

# A crystal of ``cells`` unit cells a side (rocksalt: cells x cells x cells/4;
# polycrystal: a cube of ``cells`` lattice constants), its reflection at the
# detector's centre, and the switches of the scattering call.
EXPOSURE = dict(entry="exposure", sample="cu", cells=20, ny=128, nz=128, distance_m=1.0,
                pitch_um=55.0, energy=10000.0, polarization=True, decay=False, sigma=0.08,
                profile="uniform", analyser="off", accept_mrad=0.0, depth=False, fast=True)


def _exposure(name, **kw):
    return dict(EXPOSURE, name=name, **kw)


def listed():
    return [
        # a few hundred atoms on a small frame: what an interactive user or a
        # fitting loop calls thousands of times; latency and launches count
        _exposure("exposure_864_32x24", cells=6, ny=32, nz=24),
        # the CPU-runnable configuration at full size (fcc_cu_32k)
        _exposure("exposure_32k_128", cells=20),
        # a strip detector of odd sides, an alloy with a dilute species, a
        # Gaussian beam and spherical decay: nothing is a round number
        _exposure("exposure_alloy_55k_487x195", sample="cuni", cells=24, ny=487, nz=195,
                  decay=True, profile="gaussian"),
        # the depth-dependent incident field (complex amplitudes), 2M atoms
        _exposure("exposure_depth_nacl_2m_256", sample="nacl", cells=100, ny=256, nz=256, sigma=0.05,
                  depth=True),
        # the headline workload: 8.19M atoms x 512 x 512
        _exposure("exposure_nacl_8m_512", sample="nacl", cells=160, ny=512, nz=512, sigma=0.05),
        # grains at random orientations on the largest detector, near (0.5 m)
        _exposure("exposure_polycrystal_1024", sample="poly", cells=110, ny=1024, nz=1024,
                  distance_m=0.5, energy=12000.0, sigma=0.0),
        # an analyser crystal in front of the detector (top-hat acceptance)
        _exposure("exposure_tophat_256k_200x160", cells=40, ny=200, nz=160, analyser="top-hat",
                  accept_mrad=4.0),
        # the exact mode: the reference CPU kernel's FP64 arithmetic
        _exposure("exposure_fp64_32k_48x40", cells=20, ny=48, nz=40, fast=False),
        # a rocking scan of a strained crystal, staged once and run from the
        # device: frames of uneven regions of interest
        dict(name="scan_staged_500k_16", entry="scan", sample="bumps", cells=50, frames=16,
             rois="64,128,256,512", npix=512, span_deg=0.5),
        # frames of a 101 x 101 theta x chi scan asked for by index: geometry,
        # plan and sum, as intensities (the scan surrogate's exact frames)
        dict(name="scan_frames_500k_64x128", entry="frames", sample="bumps", cells=50, frames=64,
             grid=101, roi=128, npix=512, span_deg=0.3),
        # a detector field propagated 0.5 m and its intensity
        dict(name="propagate_2048x1500", entry="propagate", ny=2048, nz=1500, pitch_um=1.0, z_m=0.5),
        # one step (forward, loss, gradients) of the scan surrogate's two
        # networks on the 101 x 101 scan's training set
        dict(name="surrogate_step_2x1272", entry="surrogate", rows=1272, hidden=256, layers=4,
             n_in=72, n_out=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["exposure", "exposure", "exposure", "exposure", "exposure", "fp64", "tophat",
                       "scan", "frames", "propagate", "surrogate"])
    if kind in ("exposure", "fp64", "tophat"):
        sample = rng.choice(["cu", "cuni", "nacl", "poly"]) if kind == "exposure" else "cu"
        c = dict(EXPOSURE, sample=sample, polarization=rng.random() < 0.7, decay=rng.random() < 0.4,
                 profile=rng.choice(["uniform", "gaussian"]), energy=rng.choice([8000.0, 10000.0, 12000.0]))
        cells, side, budget = (6, 110), (16, 1024), 2.1e12
        if kind == "fp64":
            c.update(fast=False)
            cells, side, budget = (6, 24), (8, 128), 2e8
        if kind == "tophat":
            c.update(analyser="top-hat", accept_mrad=round(rng.uniform(1.0, 8.0), 2))
            cells, side, budget = (8, 60), (16, 400), 5e10
        c["distance_m"] = rng.choice([0.5, 1.0, 1.0, 2.0])
        if sample == "poly":
            c.update(cells=_log(rng, 20, 90), sigma=0.0)
        else:
            c.update(cells=_log(rng, *cells), sigma=round(rng.uniform(0.02, 0.1), 3))
        c["ny"] = _log(rng, *side)
        # up to four times wider or narrower than it is high
        c["nz"] = max(side[0], min(side[1], int(c["ny"] * math.exp(rng.uniform(-1.4, 1.4)))))
        if rng.random() < 0.4:          # whole 4 x 4 blocks, as most real detectors have
            c["ny"], c["nz"] = max(4, c["ny"] // 4 * 4), max(4, c["nz"] // 4 * 4)
        while _atoms(c) * c["ny"] * c["nz"] > budget:
            c["ny"], c["nz"] = max(8, int(c["ny"] * 0.8)), max(8, int(c["nz"] * 0.8))
        c["depth"] = kind == "exposure" and sample != "poly" and rng.random() < 0.2
        return c
    if kind == "scan":
        rois = rng.sample([24, 48, 64, 100, 128, 200, 256, 384], 3)
        return dict(entry="scan", sample="bumps", cells=_log(rng, 10, 50), frames=rng.randint(3, 20),
                    rois=",".join(str(r) for r in rois), npix=384, span_deg=round(rng.uniform(0.1, 0.8), 2))
    if kind == "frames":
        return dict(entry="frames", sample="bumps", cells=_log(rng, 10, 50), frames=rng.randint(2, 64),
                    grid=rng.choice([21, 61, 101]), roi=rng.choice([24, 50, 64, 96, 128]), npix=256,
                    span_deg=round(rng.uniform(0.1, 0.5), 2))
    if kind == "propagate":
        ny, nz = _log(rng, 100, 2048), _log(rng, 100, 2048)
        return dict(entry="propagate", ny=ny, nz=nz, pitch_um=rng.choice([1.0, 2.0, 5.0]),
                    z_m=round(rng.uniform(0.05, 1.0), 3))
    return dict(entry="surrogate", rows=_log(rng, 64, 2048), hidden=rng.choice([64, 128, 256]),
                layers=rng.randint(2, 4), n_in=rng.choice([40, 72]), n_out=rng.choice([16, 32, 64]))


def _atoms(c):
    n = c["cells"]
    if c["sample"] == "nacl":
        return 8 * (n // 4 * 4 or n) ** 2 * max(n // 4, 1)
    return 4 * n ** 3


# ----------------------------------------------------------------- samples
def _chunks(case, rng):
    """Host chunks [(positions float32 A, (codes, labels))], the Bragg angle
    at the detector's centre and the largest extent [A]."""
    kind, n, E = case["sample"], case["cells"], case.get("energy", 10000.0)
    a = LATTICE[kind]
    fcc = workloads.fcc_basis()
    if kind == "nacl":
        # screw dislocation along z, (002) with G along the line, in a 4 x 4
        # grid of chunks where it is large
        m = n // 4 * 4 or n
        w = workloads.nacl_screw_8m(cells=(m, m, max(n // 4, 1)), npix=4,
                                    chunk_grid=(4, 4) if n >= 16 else (1, 1))
        out = [(p, (c, lab)) for p, c, lab in w.sample._chunks]
        return out, workloads.bragg_theta(a / 2.0, E)
    theta = workloads.bragg_theta(a / math.sqrt(3.0), E)
    if kind == "poly":
        pos, _ = workloads.polycrystal_positions(n * a, 24, a, int(rng.integers(1 << 30)),
                                                 device="cuda")
        m = 1_000_000
        return [(pos[i:i + m], (np.zeros(len(pos[i:i + m]), np.uint8), np.array(["Cu"])))
                for i in range(0, len(pos), m)], theta
    if kind == "bumps":
        pos, _ = workloads.bump_field_crystal(n, a, seed=int(rng.integers(1 << 30)))
        return [(pos, (np.zeros(len(pos), np.uint8), np.array(["Cu"])))], theta
    pos = workloads.lattice(a, (n,) * 3, fcc)
    pos -= pos.mean(axis=0)
    pos = (pos @ align_rotation([1, 1, 1], [0, 0, 1]).T).astype(np.float32)
    codes, labels = np.zeros(len(pos), np.uint8), ["Cu"]
    if kind == "cuni":              # 30 % Ni and 0.2 % Ag on the fcc sites
        u = rng.random(len(pos))
        codes = (u < 0.3).astype(np.uint8) + 2 * (u > 0.998).astype(np.uint8)
        labels = ["Cu", "Ni", "Ag"]
    return [(pos, (codes, np.array(labels)))], theta


def _sample(case, seed):
    rng = np.random.default_rng([seed, 11])
    chunks, theta = _chunks(case, rng)
    sigma = case.get("sigma", 0.0)
    th = dict(sigma=sigma, max_displacement=1.0, seed=int(rng.integers(1 << 30))) if sigma else None
    s = ChunkedSample(chunks, thermal=th)
    for c in range(1, s.chunk_total + 1):       # the seeded draw, kept by the sample
        s.load_chunk_positions(c, copy=False)
    return s, theta, float(np.linalg.norm(s.dimensions))


def _setup(case, seed):
    sample, theta, diag = _sample(case, seed)
    rng = np.random.default_rng([seed, 12])
    npix = (case["ny"], case["nz"]) if "ny" in case else (case["npix"],) * 2
    det = Detector()
    pitch = case.get("pitch_um", 55.0) * 1e4
    det.create_detector(npix, (pitch, pitch))
    det.position_detector_absolute(case.get("distance_m", 1.0) * 1e10, 2 * theta, 0.0, degrees=False)
    st = Stage()
    # near, not on, the reflection: within a few hundredths of a degree
    st.set_motor_value("mu", theta + math.radians(0.02) * rng.uniform(-1, 1), degrees=False)
    B = Beam()
    size = max(1000.0, 2.5 * diag)
    waist = (0.5 * diag, 0.6 * diag) if case.get("profile") == "gaussian" else None
    B.create_beam(case.get("energy", 10000.0), beam_size=(size, size), beam_samples=(256, 256),
                  beam_profile=case.get("profile", "uniform"), gaussian_waist=waist,
                  pol_perp_rate=1.0)
    B._use_fast_kernel = bool(case.get("fast", True))
    return sample, det, st, B, theta, rng


def _scan_steps(case, theta, rng):
    n = case["frames"]
    off = np.radians(np.linspace(-case["span_deg"], case["span_deg"], n)) + \
        math.radians(0.01) * rng.uniform(-1, 1)
    rois = [int(r) for r in case["rois"].split(",")]
    steps = [dict(mu=theta + float(o), chi=float(math.radians(0.1 * rng.uniform(-1, 1)))) for o in off]
    return steps, [rois[i % len(rois)] for i in range(n)]


def _grid_scan(case, sample, det, st, B, theta, rng, kw):
    st.set_motor_value("mu", theta, degrees=False)
    offs = np.radians(np.linspace(-case["span_deg"], case["span_deg"], case["grid"]))
    sc = SurrogateScan(B, sample, det, st, offs, offs.copy(), roi=case["roi"], sc_kwargs=kw)
    idx = np.sort(rng.choice(case["grid"] ** 2, size=case["frames"], replace=False))
    return sc, idx


def _network_inputs(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 5)
    x = torch.rand((2, case["rows"], case["n_in"]), generator=g, device="cuda") * 2 - 1
    t = torch.randn((2, case["rows"], case["n_out"]), generator=g, device="cuda")
    w = torch.rand(case["n_out"], generator=g, device="cuda") + 0.5
    return x.bfloat16(), t, w


def _field(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 3)
    nz, ny = case["nz"], case["ny"]
    y = torch.linspace(-1, 1, ny, device="cuda", dtype=torch.float64)
    z = torch.linspace(-1, 1, nz, device="cuda", dtype=torch.float64)
    cy, cz, s, c = (torch.rand(4, generator=g, device="cuda", dtype=torch.float64) - 0.5).tolist()
    r2 = (y[None, :] - cy) ** 2 + (z[:, None] - cz) ** 2
    amp = torch.exp(-r2 * (4 + 2 * s)) + 0.05
    noise = torch.randn((nz, ny), generator=g, device="cuda", dtype=torch.float64)
    return torch.polar(amp, 6 * c * r2 + 0.1 * noise).to(torch.complex64)


def prepare(case, seed):
    entry = case["entry"]
    if entry == "propagate":
        return dict(entry=entry, field=_field(case, seed), d=case["pitch_um"] * 1e-6, z=case["z_m"],
                    wavelength=HC_EV_A / 10000.0 * 1e-10)
    if entry == "surrogate":
        X, T, w = _network_inputs(case, seed)
        net = MLP(case["n_in"], case["n_out"], case["hidden"], case["layers"], seed=seed % 100000, groups=2)
        return dict(entry=entry, net=net, X=X, T=T, w=w)
    sample, det, st, B, theta, rng = _setup(case, seed)
    kw = dict(apply_polarization=bool(case.get("polarization", True)),
              spherical_decay=bool(case.get("decay", False)), remove_forward=False)
    if entry == "exposure":
        if case["analyser"] != "off":
            kw.update(analyser_mode=case["analyser"],
                      analyser_acceptance_angle_rad=case["accept_mrad"] * 1e-3)
        if case["depth"]:
            kw["use_depth_ein"] = True
        return dict(entry=entry, args=(sample, det, st), beam=B, kw=kw)
    if entry == "scan":
        steps, rois = _scan_steps(case, theta, rng)
        frames = frames_from_motors(st, det, steps, rois)
        return dict(entry=entry, scan=BatchedScan(B, sample, frames, **kw))
    sc, idx = _grid_scan(case, sample, det, st, B, theta, rng, kw)
    sc.exact(idx[:1])               # stages the atoms, as a scan's first frame does
    return dict(entry=entry, scan=sc, idx=idx)


def run(state):
    entry = state["entry"]
    if entry == "exposure":
        sample, det, st = state["args"]
        return state["beam"].atomic_scattering_kinematic(sample, det, st, **state["kw"])
    if entry == "scan":
        # the frames' fields, kept as the exposures' result type
        out, _ = state["scan"].run()
        return torch.view_as_complex(out).to(torch.complex64)
    if entry == "frames":
        return state["scan"].exact(state["idx"])
    if entry == "propagate":
        E, I = propagate(state["field"], state["d"], state["d"], state["z"], state["wavelength"],
                         intensity=True)
        return [E, I]
    net = state["net"]
    acts, posts, Y = net.forward(state["X"])
    loss, G, Gb = net.mse(Y, state["T"], state["w"])
    dW, db = net.backward(acts, posts, G, Gb)
    return [Y, loss] + list(dW) + list(db)


def work(case):
    """Bytes: each input read once and each output written once. Flops of a
    scattering sum: the reference's exact mode adds every (atom, pixel) term
    (20 operations and more a term); otherwise the field only has to be right,
    and what no method can avoid is taken as that of a fast transform,
    20 (n + p) log2(n + p) for n atoms and p pixels."""
    entry = case["entry"]
    if entry == "propagate":
        p = case["ny"] * case["nz"]
        return {"bytes": p * (8 + 8 + 4), "flops": 10 * p * math.log2(p)}
    if entry == "surrogate":
        d = [case["n_in"]] + [case["hidden"]] * case["layers"] + [case["n_out"]]
        par = sum(a * b + b for a, b in zip(d[:-1], d[1:]))
        return {"bytes": 2 * (par * 6 + case["rows"] * (case["n_in"] * 2 + case["n_out"] * 8)),
                "flops": 2 * 6 * par * case["rows"]}
    n = _atoms(case)
    if entry == "exposure":
        p, out = case["ny"] * case["nz"], 8
    elif entry == "scan":
        rois = [int(r) for r in case["rois"].split(",")]
        p, out = sum(min(rois[i % len(rois)], case["npix"]) ** 2 for i in range(case["frames"])), 8
    else:
        p, out = case["frames"] * min(case["roi"], case["npix"]) ** 2, 4
    direct = entry == "exposure" and not case["fast"]
    return {"bytes": n * 13 + p * out, "flops": 20.0 * (n * p if direct else (n + p) * math.log2(n + p))}


def _terms(case):
    n = _atoms(case)
    if case["entry"] == "exposure":
        return float(n) * case["ny"] * case["nz"]
    if case["entry"] == "frames":
        return float(n) * case["frames"] * min(case["roi"], case["npix"]) ** 2
    rois = [int(r) for r in case["rois"].split(",")]
    return float(n) * sum(min(rois[i % len(rois)], case["npix"]) ** 2 for i in range(case["frames"]))


# ------------------------------------------------------------------- exact
EXACT_TERMS = 8e9       # FP64 terms that take about ten seconds


def _tables(labels, energy):
    """f0 coefficients and f' + i f'' from the bundled table file."""
    z = np.load(os.path.join(os.path.dirname(mosaic_gb300.__file__), "data", "dabax_subset.npz"))
    f0 = {str(k): r for k, r in zip(z["f0_keys"], z["f0_rows"])}
    off = np.concatenate([[0], np.cumsum(z["f1f2_len"])])
    key = [str(k) for k in z["f1f2_keys"]]
    out = []
    for el in labels:
        i = key.index(el)
        t = z["f1f2_rows"][off[i]:off[i + 1]]
        j = min(max(int(np.searchsorted(t[:, 0], energy)), 1), len(t) - 1)
        w = (energy - t[j - 1, 0]) / (t[j, 0] - t[j - 1, 0])
        f1, f2 = (t[j - 1, c] + (t[j, c] - t[j - 1, c]) * w for c in (1, 2))
        out.append((f0[el].astype(np.float64), complex(np.float32(f1), np.float32(f2))))
    return out


def _atoms_of(sample):
    pos = np.concatenate([sample.load_chunk_positions(c, copy=False) for c in range(1, sample.chunk_total + 1)])
    names = np.concatenate([sample.load_chunk_species(c) for c in range(1, sample.chunk_total + 1)])
    labels = sorted(set(names.tolist()))
    return pos, np.searchsorted(np.array(labels), names), labels


def _lab(pos, R, t):
    """float32 lab positions [A], products and sums rounded one by one (the
    stage transform is defined in float32)."""
    p = torch.as_tensor(pos, device="cuda")
    R, t = np.float32(R), np.float32(t)
    cols = []
    for r in range(3):
        acc = p[:, 0] * float(R[r, 0])
        for c in (1, 2):
            q = p[:, c] * float(R[r, c])
            acc = acc + q
        cols.append(acc + float(t[r]))
    return torch.stack(cols, 1)


def _sum64(a, species, amp, tabs, P, b, e, k, polarization, decay):
    """FP64 field at pixels P (n, 3) [m] of atoms a (m, 3) [m] with complex
    amplitudes: phase k (b.a + |P - a|). The factor is taken at each pixel's
    direction from the sample's origin: atoms within 1e-7 of the distance
    change it by about 1e-8."""
    dev = a.device
    R = torch.linalg.vector_norm(P, dim=1)
    u = P / R[:, None]
    bt = torch.as_tensor(b, device=dev, dtype=torch.float64)
    et = torch.as_tensor(e, device=dev, dtype=torch.float64)
    s2 = ((k * 0.25e-10 / math.pi) ** 2) * ((bt - u) ** 2).sum(1)
    scale = torch.ones_like(R)
    if polarization:
        scale = torch.sqrt(torch.clamp(1.0 - (u @ et) ** 2, 0.0, 1.0))   # fully polarised along e
    S = len(tabs)
    W = torch.zeros((a.shape[0], 2 * S), dtype=torch.float64, device=dev)
    rows = torch.arange(a.shape[0], device=dev)
    W[rows, species] = amp.real.double()
    W[rows, S + species] = amp.imag.double()
    a2, ba = (a * a).sum(1), a @ bt
    kap = k / (2 * math.pi)
    field = torch.zeros(P.shape[0], dtype=torch.complex128, device=dev)
    for p0 in range(0, P.shape[0], 8192):
        sl = slice(p0, p0 + 8192)
        C = torch.zeros((P[sl].shape[0], 2 * S), dtype=torch.float64, device=dev)
        D = torch.zeros_like(C)
        for a0 in range(0, a.shape[0], 8192):
            at = slice(a0, a0 + 8192)
            num = a2[None, at] - 2.0 * (P[sl] @ a[at].T)
            r = torch.sqrt((R[sl] ** 2)[:, None] + num)
            cyc = kap * (ba[None, at] + num / (r + R[sl, None]))
            w = W[at]
            if decay:           # R0 / r = 1 - (r - R0) / r
                g = (R[sl, None] / r)
            cyc -= torch.round(cyc)
            cyc *= 2 * math.pi
            cs, sn = torch.cos(cyc), torch.sin(cyc)
            if decay:
                cs, sn = cs * g, sn * g
            C += cs @ w
            D += sn @ w
        sums = torch.complex(C[:, :S] - D[:, S:], D[:, :S] + C[:, S:])
        for s, (f0, an) in enumerate(tabs):
            f = f0[5] + sum(f0[i] * torch.exp(-f0[6 + i] * s2[sl]) for i in range(5))
            field[sl] += sums[:, s] * torch.complex(f + an.real, torch.full_like(f, an.imag))
    ph = kap * R
    ph = 2 * math.pi * (ph - torch.round(ph))
    return R_E * field * scale * torch.polar(torch.ones_like(ph), ph)


def _incident(B, lab):
    """E0 bilinear at the atoms' (y, z); 0 outside the beam grid."""
    E0 = torch.as_tensor(B._beam_E0_map.astype(np.complex128), device=lab.device)
    iu = lab[:, 1].double() / B._beam_du + B._beam_uc
    iv = lab[:, 2].double() / B._beam_dv + B._beam_vc
    n, m = E0.shape
    inside = (iu >= 0) & (iu <= n - 1) & (iv >= 0) & (iv <= m - 1)
    i0, j0 = iu.clamp(0, n - 1).floor().long(), iv.clamp(0, m - 1).floor().long()
    i1, j1 = (i0 + 1).clamp(max=n - 1), (j0 + 1).clamp(max=m - 1)
    fu, fv = iu - i0, iv - j0
    v = E0[i0, j0] * ((1 - fu) * (1 - fv)) + E0[i0, j1] * ((1 - fu) * fv) + \
        E0[i1, j0] * (fu * (1 - fv)) + E0[i1, j1] * (fu * fv)
    return torch.where(inside, v, torch.zeros_like(v))


def _exact_propagate(case, seed):
    """Angular spectrum on the padded grid, FP64: edge padding to a power of
    two that holds the field and its diffraction spread on both sides."""
    E = _field(case, seed).to(torch.complex128)
    nz, ny, d, z, lam = case["nz"], case["ny"], case["pitch_um"] * 1e-6, case["z_m"], HC_EV_A / 10000.0 * 1e-10
    sr = min(lam / (2 * d), 0.999999)
    pad = math.ceil(1.1 * z * min(sr / math.sqrt(1 - sr * sr), 2.0) / d)
    n2 = [1 << (min(n + 2 * pad, 8192) - 1).bit_length() for n in (nz, ny)]
    if z > min(n * d * d / lam for n in n2):
        return None             # split into several steps
    iz = (torch.arange(n2[0], device="cuda") - (n2[0] - nz) // 2).clamp(0, nz - 1)
    iy = (torch.arange(n2[1], device="cuda") - (n2[1] - ny) // 2).clamp(0, ny - 1)
    F = torch.fft.fft2(E[iz][:, iy])
    k = 2 * math.pi / lam
    fz, fy = (2 * math.pi * torch.fft.fftfreq(n, d, dtype=torch.float64, device="cuda") for n in n2)
    kt2 = fz[:, None] ** 2 + fy[None, :] ** 2
    if float(kt2.max()) > k * k:
        return None
    ph = -z * kt2 / (torch.sqrt(k * k - kt2) + k)
    G = torch.fft.ifft2(F * torch.polar(torch.ones_like(ph), ph))
    z0, y0 = (n2[0] - nz) // 2, (n2[1] - ny) // 2
    out = G[z0:z0 + nz, y0:y0 + ny].contiguous()
    return [out, out.real ** 2 + out.imag ** 2]


def _exact_network(case, seed):
    X, T, w = _network_inputs(case, seed)
    net = MLP(case["n_in"], case["n_out"], case["hidden"], case["layers"], seed=seed % 100000, groups=2)
    Wt = [t.double() for t in net.Wb]
    bias = [t.double() for t in net.b]
    acts = [X.double()]
    for l, (W, b) in enumerate(zip(Wt, bias)):
        y = acts[-1] @ W.transpose(1, 2) + b[:, None, :]
        acts.append(y if l == len(Wt) - 1 else torch.relu(y))
    Y = acts[-1]
    diff, ww = Y - T.double(), w.double()
    n = Y[0].numel()
    loss = (ww * diff * diff).sum() / n
    g = 2 * ww * diff / n
    dW, db = [None] * len(Wt), [None] * len(Wt)
    for l in range(len(Wt) - 1, -1, -1):
        dW[l], db[l] = g.transpose(1, 2) @ acts[l], g.sum(1)
        g = (g @ Wt[l]) * (acts[l] > 0)
    return [Y, loss] + dW + db


def exact(case, seed):
    entry = case["entry"]
    if entry == "propagate":
        return _exact_propagate(case, seed)
    if entry == "surrogate":
        return _exact_network(case, seed)
    if entry == "exposure" and (case["analyser"] != "off" or case["depth"]):
        return None
    if _terms(case) > EXACT_TERMS:
        return None
    sample, det, st, B, theta, rng = _setup(case, seed)
    pos, species, labels = _atoms_of(sample)
    tabs = _tables(labels, B._energy)
    sp = torch.as_tensor(species, device="cuda")
    k = 2 * math.pi / (6.62607015e-34 / 1.602176634e-19 * 299792458 / B._energy)
    pol, decay = bool(case.get("polarization", True)), bool(case.get("decay", False))

    def pixels(coords):
        return torch.as_tensor(np.asarray(coords, np.float64).T / 1e10, device="cuda").contiguous()

    if entry == "exposure":
        lab = _lab(pos, st.rotation, st.translation)
        f = _sum64(lab.double() / 1e10, sp, _incident(B, lab), tabs, pixels(det.pixel_coordinates),
                   [1.0, 0, 0], [0, 1.0, 0], k, pol, decay)
        return f.reshape(case["nz"], case["ny"]).cpu().numpy()

    # scans: the atoms stay in the sample frame, the pixels, beam and
    # polarization direction move into it
    if entry == "scan":
        steps, rois = _scan_steps(case, theta, rng)
        frames = frames_from_motors(st, det, steps, rois)
    else:
        sc, idx = _grid_scan(case, sample, det, st, B, theta, rng, {})
        frames = frames_from_motors(st, det, [sc.steps[i] for i in idx], [case["roi"]] * len(idx))
    a = torch.as_tensor(pos, device="cuda").double() / 1e10
    amp = torch.ones(a.shape[0], dtype=torch.complex128, device="cuda")
    fields = []
    for fr in frames:
        R = np.asarray(fr.rotation, np.float64)
        P = R.T @ (np.asarray(fr.pixels, np.float64) - np.asarray(fr.translation, np.float64)[:, None])
        fields.append(_sum64(a, sp, amp, tabs, pixels(P), R.T @ np.array([1.0, 0, 0]),
                             R.T @ np.array([0, 1.0, 0]), k, pol, decay))
    if entry == "scan":
        return torch.cat(fields)
    f = torch.stack(fields)
    return f.real ** 2 + f.imag ** 2
