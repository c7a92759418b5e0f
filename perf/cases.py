"""Performance cases of the framework's public entry points, with 64-bit results beside them.

A case is a dict of plain values; its ``kind`` says which entry point a pass goes through:

* ``scan``: ``ScanPlan.run`` over a set of rotations on a plan that the program keeps (what a
  search spends its time in), at the transform shape (n0, n1, n2) with a t^3 template;
* ``search``: a whole ``scan_subsets`` call on host arrays (filters, plan, upload, scan,
  download) with ``MaxScoreOverRotations``;
* ``maps``: ``scan_subsets`` with an analyzer of the caller's own, which gets one score map
  per rotation;
* ``batch``: ``scan_batch`` over one tomogram and three templates, with filter objects;
* ``refine``: the differentiable score of many peaks, forward and backward;
* ``peaks``: ``PeakCallerMaximumFilter`` on a score map on the device.

Tomograms are noise with rotated copies of a blob template, as in ``bench.py``. A maximum over
rotations is returned as the score map. The index of the rotation that reached it comes back in
the ``search`` cases, whose threshold leaves the voxels around the copies: over whole noise maps
two rotations can tie within rounding, and which of them is named says nothing.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pytme_b200 as P
from pytme_b200 import refine as RF
from pytme_b200 import synthetic as syn
from pytme_b200.analyzer import MaxScoreOverRotations, PeakCallerMaximumFilter
from pytme_b200.batch import MatchJob, scan_batch
from pytme_b200.filters import Compose, CTFReconstructed, WedgeReconstructed
from pytme_b200.matching import next_fast_len, rigid_transform_matrices
from pytme_b200.scores import MATCHING_EXHAUSTIVE_REGISTER, ScanPlan

EPS = 1.1920928955078125e-07
BATCH_TEMPLATES = (24, 32, 40)


def listed():
    scan = dict(kind="scan", score="FLCSphericalMask", precision="fp32", order=1, filters=False,
                graph=False)
    return [
        # one small launch group of a particle-sized box: launches and latency
        dict(scan, name="scan_64_fp32", n0=64, n1=64, n2=64, t=16, rotations=8, batch=8),
        # a whole small search with the defaults: FP32, cubic rotation, the 30-degree set's size
        dict(kind="search", name="search_64_fp32", score="FLCSphericalMask", precision="fp32",
             order=3, n0=64, n1=64, n2=64, t=16, rotations=360, batch=32, threshold=0.4),
        # the headline workload: a full tomogram, mixed precision, eight launch groups
        dict(scan, name="scan_512x512x200_mixed", n0=512, n1=512, n2=200, t=48, rotations=256,
             batch=32, precision="mixed"),
        # FLC with template and target filters at power-of-two sizes, mixed precision
        dict(scan, name="flc_256x256x128_mixed", score="FLC", n0=256, n1=256, n2=128, t=32,
             rotations=128, batch=64, precision="mixed", filters=True),
        # the largest job of the uneven batch, FP32 with a template filter, graph replay
        dict(scan, name="scan_320x320x160_fp32", n0=320, n1=320, n2=160, t=40, rotations=128,
             batch=64, filters=True, graph=True),
        # jobs of the uneven batch as a user starts them: host arrays in, host arrays out
        dict(kind="batch", name="batch_160x160x128_fp32", n0=160, n1=160, n2=128, rotations=192,
             batch=64),
        # FLC on a tomogram whose axes are no powers of two, cubic rotation (the default)
        dict(scan, name="flc_240x240x120_fp32", score="FLC", n0=240, n1=240, n2=120, t=32,
             rotations=32, batch=16, order=3),
        # a 464 x 480 x 150 tomogram: the transform length 468 has the factor 13
        dict(scan, name="scan_468x480x150_mixed", n0=468, n1=480, n2=150, t=32, rotations=64,
             batch=32, precision="mixed"),
        # an analyzer that wants every rotation's map
        dict(kind="maps", name="maps_160x160x100_fp32", score="FLCSphericalMask", n0=160, n1=160,
             n2=100, t=24, rotations=16, batch=32),
        # refinement of 2048 candidate peaks with the CTF x wedge filter, all gradients
        dict(kind="refine", name="refine_2048x32_filtered", peaks=2048, t=32, n0=256, n1=256,
             n2=128, filters=True),
        # fewer peaks of a larger template without a filter
        dict(kind="refine", name="refine_512x48", peaks=512, t=48, n0=192, n1=192, n2=128,
             filters=False),
        # peak calling on the headline workload's score map
        dict(kind="peaks", name="peaks_512x512x200", n0=512, n1=512, n2=200, num_peaks=1000,
             min_distance=24),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["scan"] * 6 + ["search"] * 2 + ["maps", "batch", "refine", "refine",
                                                        "peaks"])
    if kind == "refine":
        t = _log(rng, 12, 48)
        return dict(kind=kind, peaks=min(_log(rng, 48, 2048), 2048 * 32 ** 3 // t ** 3), t=t,
                    n0=rng.randint(96, 256), n1=rng.randint(96, 256), n2=rng.randint(64, 160),
                    filters=rng.random() < 0.5)
    if kind == "peaks":
        return dict(kind=kind, n0=_log(rng, 96, 512), n1=_log(rng, 96, 512),
                    n2=_log(rng, 64, 200), num_peaks=_log(rng, 50, 2000),
                    min_distance=rng.randint(10, 32))
    if kind == "batch":
        return dict(kind=kind, n0=rng.randint(96, 256), n1=rng.randint(96, 256),
                    n2=rng.randint(80, 160), rotations=_log(rng, 16, 128),
                    batch=rng.choice([16, 32, 64]))
    n0, n1, n2 = _log(rng, 64, 400), _log(rng, 64, 400), _log(rng, 48, 200)
    t = min(_log(rng, 12, 48), min(n0, n1, n2) // 2)
    case = dict(kind=kind, score=rng.choice(["FLCSphericalMask"] * 3 + ["FLC"] * 2 + ["CC"]),
                n0=n0, n1=n1, n2=n2, t=t, batch=rng.choice([8, 16, 32, 64]))
    voxels = n0 * n1 * n2
    while case["batch"] * voxels > 800_000_000:
        case["batch"] //= 2
    most = max(4, 600_000_000 // voxels)
    if kind == "maps":
        return dict(case, rotations=min(_log(rng, 4, 24), most))
    case.update(precision=rng.choice(["fp32", "mixed"]), order=rng.choice([1, 3]),
                rotations=min(_log(rng, 6, 200), most))
    if kind == "search":  # the index map is returned: few strong copies above the threshold
        return dict(case, score="FLCSphericalMask", precision="fp32", threshold=0.4,
                    rotations=min(case["rotations"], 100))
    case.update(n0=next_fast_len(n0), n1=next_fast_len(n1), n2=next_fast_len(n2))
    return dict(case, filters=rng.random() < 0.5, graph=rng.random() < 0.5)


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _radial(shape, device="cuda"):
    """Frequency norm and the cosine-like coordinate of the tilt axis at an rfft shape."""
    f0, f1 = (torch.fft.fftfreq(n, dtype=torch.float64, device=device) for n in shape[:2])
    f2 = torch.fft.rfftfreq(shape[2], dtype=torch.float64, device=device)
    k = torch.sqrt(f0[:, None, None] ** 2 + f1[None, :, None] ** 2 + f2[None, None, :] ** 2)
    return k, f0[:, None, None].abs().expand_as(k), f2[None, None, :].expand_as(k)


def _wedge_array(shape):
    """A missing wedge of +-60 degrees about axis 1, zero frequency kept, float32."""
    k, f0, f2 = _radial(shape)
    w = (f2 <= f0 * math.tan(math.radians(60.0))).to(torch.float32)
    w[0, 0, 0] = 1.0
    return w


def _ctf_array(shape):
    """A phase-flipped CTF (3 um defocus, 6.8 A pixels, 300 kV) times the wedge, float32."""
    k = _radial(shape)[0] / 6.8
    phase = math.pi * 0.0197 * k ** 2 * (30000.0 - 0.5 * 2.7e7 * (0.0197 * k) ** 2)
    return torch.sin(phase + 0.07).abs().to(torch.float32) * _wedge_array(shape)


def _template(t, score, rng):
    """Blob template and its mask: dilated threshold for FLC, a ball otherwise (host arrays)."""
    tmpl = syn.blob_template(t, rng, n_blobs=6, sigma=1.5 * t / 16, radius=5.0 * t / 16)
    if score == "FLC":
        return tmpl, syn.dilated_threshold_mask(tmpl, 0.1, 2)
    return tmpl, syn.spherical_mask((t,) * 3, t / 2, center=((t - 1) / 2,) * 3)


def _tomogram(shape, tmpl, mask, rots, copies, snr, seed):
    """float32 noise on the device with ``copies`` rotated templates added at random places."""
    gen = _generator(seed)
    out = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
    amp = math.sqrt(snr / max(float(tmpl[mask > 0].var()), 1e-30))
    pick = np.random.default_rng(seed + 1)
    t = tmpl.shape[0]
    which = pick.integers(0, len(rots), copies)
    turned = _rotated(torch.as_tensor(tmpl, device="cuda", dtype=torch.float64),
                      _matrices(rots[which], t), 1)
    for c in range(copies):
        a = [int(pick.integers(0, max(1, n - t + 1))) for n in shape]
        box = tuple(slice(i, min(i + t, n)) for i, n in zip(a, shape))
        out[box] += (amp * turned[c])[tuple(slice(0, s.stop - s.start) for s in box)].float()
    return out


def _problem(case, seed):
    """Everything that ``prepare`` and ``exact`` share: (tomogram, template, mask, rotations)."""
    rng = np.random.default_rng(seed)
    tmpl, mask = _template(case["t"], case["score"], rng)
    rots = syn.random_rotation_matrices(case["rotations"], rng)
    strong = case["kind"] == "search"
    target = _tomogram((case["n0"], case["n1"], case["n2"]), tmpl, mask, rots,
                       4 if strong else 24, 3.0 if strong else 0.1, seed)
    return target, tmpl, mask, rots


def _refine_inputs(case, seed):
    rng = np.random.default_rng(seed)
    t, n = case["t"], case["peaks"]
    tmpl, mask = _template(t, "FLC", rng)
    shape = (case["n0"], case["n1"], case["n2"])
    target = _tomogram(shape, tmpl, mask, syn.random_rotation_matrices(40, rng), 40, 0.5, seed)
    angles = np.stack([rng.uniform(-180, 180, n), rng.uniform(5, 175, n),
                       rng.uniform(-180, 180, n)], -1).astype(np.float32)
    shifts = rng.uniform(-0.8, 0.8, (n, 3)).astype(np.float32)
    # a few boxes reach past the tomogram's edge, as peaks near the border do
    corners = np.stack([rng.integers(-2, s - t + 3, n) for s in shape], -1).astype(np.int32)
    weight = rng.uniform(0.5, 1.5, n).astype(np.float32)
    filt = _ctf_array((t, t, t)) if case["filters"] else None
    return target, tmpl, mask, angles, shifts, corners, weight, filt


def _score_map(case, seed):
    """A smooth positive map: box-filtered noise, as maxima of correlations look."""
    x = torch.randn((1, 1, case["n0"], case["n1"], case["n2"]), generator=_generator(seed),
                    device="cuda")
    for _ in range(2):
        x = torch.nn.functional.avg_pool3d(x, 5, stride=1, padding=2, count_include_pad=False)
    return (x[0, 0].abs() * 0.05).contiguous()


class Collect:
    """An analyzer of the caller's own: keeps every rotation's score map."""

    def __init__(self, **kwargs):
        pass

    def init_state(self):
        return []

    def __call__(self, state, scores, rotation_matrix, **kwargs):
        return state + [scores.clone()]

    def result(self, state, **kwargs):
        return state

    @classmethod
    def merge(cls, results, **kwargs):
        return results[0]


def _filter_objects(seed):
    rng = np.random.default_rng(seed)
    wedge = dict(angles=(float(rng.uniform(50, 65)),) * 2, opening_axis=2, tilt_axis=0,
                 create_continuous_wedge=True)
    ctf = dict(defocus_x=float(rng.uniform(15000, 45000)), amplitude_contrast=0.07,
               spherical_aberration=2.7e7, acceleration_voltage=300e3, sampling_rate=6.8,
               flip_phase=True)
    return (Compose([WedgeReconstructed(**wedge), CTFReconstructed(**ctf)]),
            Compose([WedgeReconstructed(**wedge)]))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "peaks":
        return dict(case=case, scores=_score_map(case, seed))
    if kind == "refine":
        target, tmpl, mask, ang, sh, cor, w, filt = _refine_inputs(case, seed)
        prob = RF.RefineProblem(target, tmpl, mask, template_filter=filt)
        dev = prob.target.device
        leaf = lambda x: torch.as_tensor(x, device=dev).requires_grad_(True)  # noqa: E731
        return dict(case=case, problem=prob, template=leaf(tmpl), angles=leaf(ang),
                    shifts=leaf(sh), corners=torch.as_tensor(cor, device=dev),
                    weight=torch.as_tensor(w, device=dev))
    if kind == "batch":
        rng = np.random.default_rng(seed)
        shape = (case["n0"], case["n1"], case["n2"])
        rots = syn.random_rotation_matrices(case["rotations"], rng)
        jobs, target = [], None
        tf, gf = _filter_objects(seed)
        for t in BATCH_TEMPLATES:
            tmpl, mask = _template(t, "FLCSphericalMask", rng)
            if target is None:
                target = _tomogram(shape, tmpl, mask, rots, 12, 0.1, seed).cpu().numpy()
            jobs.append(MatchJob(target=target, template=tmpl, mask=mask, rotations=rots,
                                 template_filter=tf, target_filter=gf, interpolation_order=1))
        return dict(case=case, jobs=jobs)
    target, tmpl, mask, rots = _problem(case, seed)
    if kind in ("search", "maps"):
        P.backend.change_backend("b200", precision=case.get("precision", "fp32"),
                                 rotation_batch=case["batch"])
        md = P.MatchingData(target.cpu().numpy(), tmpl)
        md.template_mask = mask
        md.rotations = rots
        return dict(case=case, data=md)
    fast = (case["n0"], case["n1"], case["n2"])
    plan = ScanPlan(case["score"], fast, tmpl.shape, precision=case["precision"],
                    batch=case["batch"])
    plan.set_graph(case["graph"])
    plan.set_template(np.ascontiguousarray(tmpl[::-1, ::-1, ::-1]),
                      np.ascontiguousarray(mask[::-1, ::-1, ::-1]),
                      _ctf_array(tmpl.shape) if case["filters"] else None)
    plan.set_interpolation(case["order"])
    plan.set_target(_filtered(target, _wedge_array(fast)).float() if case["filters"] else target)
    mats = torch.as_tensor(rigid_transform_matrices(rots, (np.asarray(tmpl.shape) - 1) / 2),
                           device="cuda")
    return dict(case=case, plan=plan, matrices=mats,
                scores=torch.empty(fast, dtype=torch.float32, device="cuda"),
                index=torch.empty(fast, dtype=torch.int32, device="cuda"))


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "scan":
        smax, sarg = state["scores"].fill_(0.0), state["index"].fill_(-1)
        state["plan"].run(state["matrices"], 0, smax, sarg)
        return smax
    if kind in ("search", "maps"):
        setup, scoring = MATCHING_EXHAUSTIVE_REGISTER[case["score"]]
        res = P.scan_subsets(
            state["data"], matching_score=scoring, matching_setup=setup,
            callback_class=MaxScoreOverRotations if kind == "search" else Collect,
            callback_class_args={"score_threshold": case["threshold"]} if kind == "search" else {},
            interpolation_order=case.get("order", 1))
        return {"scores": res[0], "index": res[2]} if kind == "search" else res
    if kind == "batch":
        return [s for s, _ in scan_batch(state["jobs"], precision="fp32",
                                         rotation_batch=case["batch"])]
    if kind == "refine":
        leaves = (state["template"], state["angles"], state["shifts"])
        s = RF.refine_score(state["problem"], state["corners"], state["angles"], state["shifts"],
                            template=state["template"])
        return (s.detach(),) + torch.autograd.grad((s * state["weight"]).sum(), leaves)
    pc = PeakCallerMaximumFilter(shape=tuple(state["scores"].shape), num_peaks=case["num_peaks"],
                                 min_distance=case["min_distance"])
    pos, rot, sc, det = pc(pc.init_state(), scores=state["scores"],
                           rotation_matrix=np.eye(3, dtype=np.float32))
    return {"positions": pos, "rotations": rot, "scores": sc, "details": det}


def work(case):
    """Inputs read once, outputs written once; the transforms' operations for the scans."""
    n = case["n0"] * case["n1"] * case["n2"]
    if case["kind"] == "peaks":  # running maxima: about three comparisons per axis and voxel
        return {"bytes": 4.0 * n, "flops": 9.0 * n}
    if case["kind"] == "refine":
        v = case["peaks"] * case["t"] ** 3
        # per voxel: two 7-lerp samples, coordinates and sums forward; twice that backward
        return {"bytes": 4.0 * min(n, v) + 12.0 * case["t"] ** 3, "flops": 200.0 * v}
    maps = len(BATCH_TEMPLATES) if case["kind"] == "batch" else 1
    lines = 3 if case.get("score") == "FLC" else 1  # inverse transforms per rotation
    flops = maps * case["rotations"] * lines * (2.5 * n * math.log2(n) + 3.0 * n)
    outs = case["rotations"] if case["kind"] == "maps" else 2 * maps
    return {"bytes": 4.0 * n * (1 + outs), "flops": flops}


# ------------------------------------------------------------------ results in 64 bits
def _matrices(rots, t):
    """float32 pull matrices about the template's centre, as the inputs of the rotation."""
    rot = np.ascontiguousarray(rots, dtype=np.float32)
    c = np.float32((t - 1) / 2)
    right = np.identity(4, dtype=np.float32)
    left = np.identity(4, dtype=np.float32)
    left[:3, 3], right[:3, 3] = c, -c
    m = np.zeros((len(rot), 4, 4), dtype=np.float32)
    m[:, :3, :3], m[:, 3, 3] = np.linalg.inv(rot), 1
    return torch.as_tensor((left @ m) @ right, device="cuda").double()


def _spline_coefficients(x):
    """Cubic B-spline coefficients with mirrored ends: the interpolation systems solved."""
    for axis in range(3):
        n = x.shape[axis]
        a = torch.zeros((n, n), dtype=torch.float64, device=x.device)
        i = torch.arange(n, device=x.device)
        a[i, i] = 4 / 6
        for d in (-1, 1):
            j = i + d
            j = torch.where(j < 0, -j, torch.where(j >= n, 2 * n - 2 - j, j))
            a.index_put_((i, j), torch.full((n,), 1 / 6, dtype=torch.float64, device=x.device),
                         accumulate=True)
        y = x.movedim(axis, 0).reshape(n, -1)
        x = torch.linalg.solve(a, y).reshape((n,) + tuple(x.movedim(axis, 0).shape[1:]))
        x = x.movedim(0, axis)
    return x.contiguous()


def _rotated(vol, mats, order, coefficients=True):
    """Pull interpolation of ``vol`` under each matrix; zero outside the volume."""
    n = vol.shape[0]
    dev = vol.device
    src = _spline_coefficients(vol) if order == 3 and coefficients else vol
    ax = torch.arange(n, device=dev, dtype=torch.float64)
    o = torch.meshgrid(ax, ax, ax, indexing="ij")
    flat, out = src.reshape(-1), []
    for m in mats.to(dev):
        acc, idx, wgt = None, [], []
        inside = torch.ones((n, n, n), dtype=torch.bool, device=dev)
        for a in range(3):
            c = m[a, 0] * o[0] + m[a, 1] * o[1] + m[a, 2] * o[2] + m[a, 3]
            inside &= (c >= 0) & (c <= n - 1)
            lo = torch.floor(c)
            f, lo = c - lo, lo.long()
            if order == 1:
                w = [1 - f, f]
                i = [lo.clamp(0, n - 1), (lo + 1).clamp(0, n - 1)]
            else:
                s = 1 - f
                w = [s ** 3 / 6, (3 * f ** 3 - 6 * f ** 2 + 4) / 6,
                     (3 * s ** 3 - 6 * s ** 2 + 4) / 6, f ** 3 / 6]
                i = [(lo + d) for d in (-1, 0, 1, 2)]
                i = [torch.where(j < 0, -j, torch.where(j >= n, 2 * n - 2 - j, j)).clamp(0, n - 1)
                     for j in i]
            idx.append(i)
            wgt.append(w)
        for p in range(len(idx[0])):
            for q in range(len(idx[1])):
                w01, i01 = wgt[0][p] * wgt[1][q], (idx[0][p] * n + idx[1][q]) * n
                for r in range(len(idx[2])):
                    term = w01 * wgt[2][r] * flat[i01 + idx[2][r]]
                    acc = term if acc is None else acc + term
        out.append(torch.where(inside, acc, torch.zeros_like(acc)))
    return torch.stack(out)


def _filtered(x, filt):
    return torch.fft.irfftn(torch.fft.rfftn(x.double()) * filt.double(), s=tuple(x.shape))


def _padded(x, shape):
    out = torch.zeros(shape, dtype=torch.float64, device=x.device)
    out[tuple(slice(0, min(a, b)) for a, b in zip(x.shape, shape))] = \
        x[tuple(slice(0, min(a, b)) for a, b in zip(x.shape, shape))]
    return out


def _exact_maps(case, target, tmpl, mask, rots, fast):
    """One 64-bit score map at the transform shape after another."""
    score, order, t = case["score"], case.get("order", 1), case["t"]
    f = _padded(target.double(), fast)
    if score != "CC":
        f = f - f.mean()
    spec = torch.fft.rfftn(f)
    spec2 = torch.fft.rfftn(f * f) if score != "CC" else None
    back = lambda s: torch.fft.irfftn(s, s=tuple(fast))  # noqa: E731
    flip = lambda a: torch.as_tensor(a[::-1, ::-1, ::-1].copy(), device="cuda").double()  # noqa: E731
    tm, mk = flip(tmpl), flip(mask)
    filt = _ctf_array(tmpl.shape) if case.get("filters") else None

    def deviation(m, n_obs):
        fm = torch.fft.rfftn(_padded(m, fast))
        e1, e2 = back(spec * fm) / n_obs, back(spec2 * fm) / n_obs
        sd = torch.sqrt((e2 - e1 * e1).clamp(min=0))
        return torch.where(sd < EPS, torch.ones_like(sd), sd) * n_obs

    den = deviation(mk, mk.sum()) if score == "FLCSphericalMask" else None
    for m in _matrices(rots, t):
        x = _rotated(tm, m[None], order)[0]
        if filt is not None:
            x = _filtered(x, filt)
        m_r = mk
        if score == "FLC":
            m_r = _rotated(mk, m[None], order, coefficients=False)[0]
            den = deviation(m_r, m_r.sum())
        if score != "CC":
            n_obs = m_r.sum()
            mean = (x * m_r).sum() / n_obs
            sd = torch.sqrt(((x * x * m_r).sum() / n_obs - mean * mean).clamp(min=0))
            x = (x - mean) / sd * m_r
        cc = back(spec * torch.fft.rfftn(_padded(x, fast)))
        yield cc if den is None else cc / den


def _exact_refine(case, seed):
    target, tmpl, mask, ang, sh, cor, weight, filt = _refine_inputs(case, seed)
    t = case["t"]
    dev = target.device
    f = target.double()
    mean = f.mean()
    d64 = lambda x: torch.as_tensor(np.ascontiguousarray(x), device=dev).double()  # noqa: E731
    template = d64(tmpl).requires_grad_(True)
    angles, shifts = d64(ang).requires_grad_(True), d64(sh).requires_grad_(True)
    w, corners, mk = d64(weight), torch.as_tensor(cor, device=dev).long(), d64(mask).reshape(-1)
    ax = torch.arange(t, device=dev)
    grid = torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), -1).reshape(-1, 3)
    c, size = (t - 1) / 2, torch.tensor(f.shape, device=dev)
    scores, step = [], max(1, (1 << 20) // t ** 3)
    for lo in range(0, case["peaks"], step):
        part = slice(lo, lo + step)
        a = angles[part] * (math.pi / 180)
        (ca, cb, cg), (sa, sb, sg) = torch.cos(a).T, torch.sin(a).T
        rot = torch.stack([
            torch.stack([cg * cb * ca - sg * sa, -cg * cb * sa - sg * ca, cg * sb], -1),
            torch.stack([sg * cb * ca + cg * sa, -sg * cb * sa + cg * ca, sg * sb], -1),
            torch.stack([-sb * ca, sb * sa, cb], -1)], -2)
        u = torch.einsum("pji,pvj->pvi", rot, grid.double() - c - shifts[part][:, None]) + c
        inside = ((u >= 0) & (u <= t - 1)).all(-1)
        base = torch.floor(u).detach()
        frac, base = u - base, base.long().clamp(0, t - 1)
        up = (base + 1).clamp(max=t - 1)
        tr, mr = 0.0, 0.0
        for q in range(8):
            i = [(up if (q >> (2 - k)) & 1 else base)[..., k] for k in range(3)]
            g = [frac[..., k] if (q >> (2 - k)) & 1 else 1 - frac[..., k] for k in range(3)]
            at, wq = (i[0] * t + i[1]) * t + i[2], g[0] * g[1] * g[2] * inside
            tr = tr + wq * template.reshape(-1)[at]
            mr = mr + wq * mk[at]
        if filt is not None:
            box = torch.fft.rfftn(tr.reshape(-1, t, t, t), dim=(1, 2, 3)) * filt.double()
            tr = torch.fft.irfftn(box, s=(t, t, t), dim=(1, 2, 3)).reshape(tr.shape)
        pos = corners[part][:, None] + grid
        ok = ((pos >= 0) & (pos < size)).all(-1)
        pos = torch.minimum(pos.clamp(min=0), size - 1)
        # outside the tomogram lies its raw zero
        box = f[pos[..., 0], pos[..., 1], pos[..., 2]] * ok - mean
        n = mr.sum(1)
        mu = (tr * mr).sum(1) / n
        sd_t = torch.sqrt((tr * tr * mr).sum(1) / n - mu * mu)
        e1, e2 = (box * mr).sum(1) / n, (box * box * mr).sum(1) / n
        sd_f = torch.sqrt((e2 - e1 * e1).clamp(min=0))
        sd_f = torch.where(sd_f < EPS, torch.ones_like(sd_f), sd_f)
        s = (((tr - mu[:, None]) * mr * box).sum(1)) / (sd_t * sd_f * n)
        (s * w[part]).sum().backward()
        scores.append(s.detach())
    return torch.cat(scores), template.grad, angles.grad, shifts.grad


def exact(case, seed):
    kind = case["kind"]
    if kind in ("peaks", "batch"):  # positions, and filters that the framework builds
        return None
    if kind == "refine":
        return _exact_refine(case, seed)
    target, tmpl, mask, rots = _problem(case, seed)
    shape = tuple(target.shape)
    if kind == "scan":
        if case["filters"]:  # the plan's input is the filtered float32 target
            target = _filtered(target, _wedge_array(shape)).float()
        best = torch.zeros(shape, dtype=torch.float64, device=target.device)
        for m in _exact_maps(case, target, tmpl, mask, rots, shape):
            best = torch.maximum(best, m)
        return best
    fast = tuple(next_fast_len(n) for n in shape)
    if kind == "maps":
        return list(_exact_maps(case, target, tmpl, mask, rots, fast))
    best = torch.full(fast, case["threshold"], dtype=torch.float64, device=target.device)
    for m in _exact_maps(case, target, tmpl, mask, rots, fast):
        best = torch.maximum(best, m)
    shift = 1 - case["t"] // 2 - case["t"] % 2
    best = torch.roll(best, (shift,) * 3, (0, 1, 2))
    return {"scores": best[:shape[0], :shape[1], :shape[2]], "index": None}
