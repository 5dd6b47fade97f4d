"""Performance cases: what users of this package run, over the sizes it is used at.

An EMC reconstruction is a loop of iterations over one dataset that stays on
the GPU, so most cases are one iteration (expand, maximize, compress) of one
Context from a given model and scaling.  The others are an iteration
restricted by the learned proposal, six datasets replayed as one CUDA graph,
and the step of a streaming user who uploads new patterns and reads the model
back.  Sizes are those of the workloads in emc_b200/workloads.py and of the
tests; the data are made here the way emc_synthesize makes them (|F|^2 of
point scatterers, uniformly random orientations, log-normal brightness,
Poisson counts), with torch so that they are quick to make.

A case is a dict of plain values:
  kind        iterate | topk | graph | step
  side        detector side in pixels == model side in voxels
  rot_n       refinement of the 600-cell rotation sampling
  patterns    number of diffraction patterns
  photons     mean photons per pattern
  beamstop    radius of the masked centre in pixels
  likelihood, interp, precision   options of emc_b200.Context
  start       "refined": a model on its way to convergence (sharp posteriors);
              "random": the uniform random model a reconstruction starts from
  stats       whether the program reads the iteration's statistics
  sides       (graph) the detector sides of the datasets
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import emc_b200 as E
from emc_b200 import proposal as PR

SIGMA = 0.4  # width of the gaussian likelihood, the reference's value and the default
FLOOR = 1e-10  # lower bound of the model inside the poisson logarithm, the default
SCATTERERS, OBJECT_RADIUS, SCALE_SIGMA = 40, 0.3, 0.5
EDGE_ANGLE = math.radians(30.0)  # scattering angle at the middle of the detector's edge
TOP_K, MAX_CELLS, AUDIT = 2048, 32, 64  # the learned proposal as the benchmark runs it


def _case(kind, side, rot_n, patterns, photons, beamstop, likelihood="poisson", interp="nearest",
          precision="mixed", start="refined", stats=False, sides=""):
    return dict(kind=kind, side=side, rot_n=rot_n, patterns=patterns, photons=float(photons),
                beamstop=float(beamstop), likelihood=likelihood, interp=interp,
                precision=precision, start=start, stats=stats, sides=sides)


def listed():
    out = {
        # the smallest problem, in the package's default options (FP32, gaussian,
        # nearest voxel): launches and host calls are its time
        "tiny16_fp32_gauss": _case("iterate", 16, 2, 64, 400, 1.5, "gauss", precision="fp32",
                                   stats=True),
        # the first iteration of a small reconstruction, from a random model
        "small32_mixed_poisson": _case("iterate", 32, 4, 256, 1000, 2, start="random", stats=True),
        # the workload the CPU programs are used at, in the default options
        "cpu32_fp32_gauss": _case("iterate", 32, 4, 1000, 1000, 0, "gauss", precision="fp32",
                                  stats=True),
        # the drop-in replacement of the reference at 64^3: FP32, gaussian
        "b200_64_fp32_gauss": _case("iterate", 64, 8, 10_000, 2000, 4, "gauss", precision="fp32"),
        # the same dataset as production runs it: mixed precision, poisson
        "b200_64_mixed_poisson": _case("iterate", 64, 8, 10_000, 2000, 4),
        # gaussian likelihood on the tensor cores: its posteriors stay broad, so
        # the slice sums are the dense contraction
        "batch80_mixed_gauss": _case("iterate", 80, 8, 8000, 500, 6, "gauss"),
        # trilinear slicing and insertion
        "batch96_mixed_trilinear": _case("iterate", 96, 9, 11_000, 500, 6, interp="trilinear"),
        # plain FP32 poisson at 128^3 (the accuracy reference of the mixed runs)
        "large128_fp32_poisson": _case("iterate", 128, 8, 2000, 500, 6, precision="fp32"),
        # the largest dataset of the batched workload: what a production
        # iteration at 128^3 is
        "batch128_mixed_poisson": _case("iterate", 128, 12, 20_000, 500, 6),
        # a proposed iteration at 128^3: candidate cells from the previous
        # posterior, the dense audit of sampled patterns
        "learned128_topk": _case("topk", 128, 12, 10_000, 500, 6),
        # six small datasets of different detectors replayed as one graph
        "small6_graph": _case("graph", 128, 4, 500, 500, 6, sides="48,64,80,96,112,128"),
        # a streaming step: photon lists, model and scaling uploaded from
        # pinned host memory, one iteration, model and scaling read back
        "step112_mixed_poisson": _case("step", 112, 10, 14_000, 500, 6),
    }
    return [dict(c, name=n) for n, c in out.items()]


def draw(rng):
    """One more case of the same ranges, at most as costly as the listed ones."""
    def log_uniform(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choices(["iterate", "topk", "graph", "step"], [7, 1, 1, 1])[0]
    precision = "fp32" if kind == "iterate" and rng.random() < 0.45 else "mixed"
    likelihood = "gauss" if rng.random() < (0.6 if precision == "fp32" else 0.25) else "poisson"
    interp = "trilinear" if rng.random() < 0.25 else "nearest"
    side = int(round(log_uniform(16, 128)))
    if kind in ("topk", "graph"):
        likelihood, interp = "poisson", "nearest"
    if kind == "topk":
        side = 2 * int(round(log_uniform(24, 64)))  # the features bin pixels 2 x 2
    # orientation sampling grows with the resolution
    rot_n = min(12, max(2, round(side / 9) + rng.choice([-1, 0, 1])))
    if kind == "topk":
        rot_n = max(rot_n, 6)  # several fine rotations per coarse cell
    beamstop = rng.choice([0.0, round(side * rng.uniform(0.03, 0.07), 2)])
    photons = round(log_uniform(200, 2000), 1)
    sides = ""
    if kind == "graph":
        k = rng.randint(2, 6)
        sides = ",".join(str(int(round(log_uniform(32, 128)))) for _ in range(k))
        side, rot_n = max(int(s) for s in sides.split(",")), rng.randint(3, 5)
    R, npa = _n_rotations(rot_n), side * side
    evals = {"fp32": 6.0e11, "mixed": 1.0e13}[precision] / npa
    evals = min(evals, {"fp32": 3.0e8, "mixed": 1.2e9}[precision])
    if kind == "graph":
        evals = 4.0e6
    top = {"topk": 10_000, "graph": 1000}.get(kind, 20_000)
    top = max(65, min(top, int(evals / R)))
    patterns = int(round(log_uniform(64, top)))
    return _case(kind, side, rot_n, patterns, photons, beamstop, likelihood, interp, precision,
                 start="random" if kind == "iterate" and rng.random() < 0.25 else "refined",
                 stats=kind == "iterate" and rng.random() < 0.5, sides=sides)


# ------------------------------------------------------------------- inputs --

@functools.lru_cache(maxsize=None)
def _rotations(n):
    return E.generate_rotations(n)


@functools.lru_cache(maxsize=None)
def _cell_rotations(n):
    """The sampling sorted by coarse cell: (q, w, cell, cells)."""
    return PR.sorted_rotations(*_rotations(n))


def _n_rotations(n):
    return _rotations(n)[0].shape[0]


@functools.lru_cache(maxsize=None)
def _geometry(side, beamstop):
    """Pixel coordinates on the Ewald sphere, in pixel units, and the mask."""
    i = np.arange(side) - side / 2.0 + 0.5
    px, py = np.meshgrid(i, i)
    pr = np.hypot(px, py)
    ang = np.arctan(pr * (math.tan(EDGE_ANGLE) / (side / 2)))
    z = np.where(pr > 0, (1 - np.cos(ang)) / np.maximum(np.sin(ang), 1e-30) * pr, 0.0)
    mask = (pr > beamstop).astype(np.int32)
    return [np.ascontiguousarray(a, np.float32).reshape(-1) for a in (px, py, z)] + [mask.reshape(-1)]


def _matrices(q):
    """Rotation matrices [n][9] of quaternions in their own precision."""
    a, b, c, d = q.unbind(1)
    aa, bb, cc, dd = a * a, b * b, c * c, d * d
    return torch.stack([aa + bb - cc - dd, 2 * b * c - 2 * a * d, 2 * b * d + 2 * a * c,
                        2 * b * c + 2 * a * d, aa - bb + cc - dd, 2 * c * d - 2 * a * b,
                        2 * b * d - 2 * a * c, 2 * c * d + 2 * a * b, aa - bb - cc + dd], 1)


def _positions(m, side, xyz):
    """Voxel positions side/2 + 0.5 + R c of every (rotation, pixel), each of
    the three [rotations][pixels].  Which voxel a pixel falls on is decided in
    single precision, so the steps are single-precision ones: products and
    sums of float32 values are formed in float64, where they are exact or very
    nearly so, and rounded once per fused multiply-add."""
    x, y, z = (t.double()[None, :] for t in xyz)
    m = m.double()

    def f32(t):
        return t.float().double()

    out = []
    for k in range(3):
        m0, m1, m2 = (m[:, 3 * k + i, None] for i in range(3))
        t = f32(m0 * x + f32(m1 * y + f32(m2 * z)))
        out.append((t + (side / 2 + 0.5)).float())
    return out


def _dataset(case, side, seed):
    """Everything one Context is given: geometry, rotations, counts (uint8 or
    int16 on the GPU), starting model and scaling."""
    g = torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + side)
    x, y, z, mask = _geometry(side, case["beamstop"])
    if case["kind"] == "topk":
        q, w, cell, cells = _cell_rotations(case["rot_n"])
    else:
        (q, w), cell, cells = _rotations(case["rot_n"]), None, 0
    N, npix = case["patterns"], side * side

    def rnd(*shape):
        return torch.rand(*shape, generator=g, device="cuda")

    # |F|^2 of point scatterers, voxel k centred at k - side/2 - 0.5
    pos = torch.randn(SCATTERERS, 3, generator=g, device="cuda")
    pos = pos / pos.norm(dim=1, keepdim=True) * rnd(SCATTERERS, 1) ** (1 / 3) * OBJECT_RADIUS * side
    k = torch.arange(side, device="cuda") - side / 2 - 0.5
    e = torch.exp(2j * math.pi / side * k[None, :, None] * pos.T[:, None, :])  # [3][side][scatterers]
    F = torch.einsum("zs,ys,xs->zyx", e[2], e[1], e[0])
    truth = (F.abs() ** 2).float()
    # photons: trilinear slices at uniformly random orientations
    u = rnd(N, 3)
    quat = torch.stack([(1 - u[:, 0]).sqrt() * torch.sin(2 * math.pi * u[:, 1]),
                        (1 - u[:, 0]).sqrt() * torch.cos(2 * math.pi * u[:, 1]),
                        u[:, 0].sqrt() * torch.sin(2 * math.pi * u[:, 2]),
                        u[:, 0].sqrt() * torch.cos(2 * math.pi * u[:, 2])], 1)
    scale = torch.exp(SCALE_SIGMA * torch.randn(N, generator=g, device="cuda") - SCALE_SIGMA ** 2 / 2)
    xyz = [torch.from_numpy(a).cuda() for a in (x, y, z)]
    on = torch.from_numpy(mask).cuda() != 0
    counts = torch.empty(N, npix, dtype=torch.int16, device="cuda")
    step = max(1, (1 << 25) // npix)
    for p0 in range(0, N, step):
        ps = _positions(_matrices(quat[p0:p0 + step]), side, xyz)
        grid = torch.stack(ps, -1) * (2.0 / (side - 1)) - 1
        s = torch.nn.functional.grid_sample(truth[None, None], grid[None, None], "bilinear",
                                            "zeros", True)[0, 0, 0]
        f = case["photons"] * scale[p0:p0 + step] / (s * on).sum(1).clamp_min(1e-20)
        counts[p0:p0 + step] = torch.poisson(s * f[:, None], generator=g).clamp_max(2048).short()
    if case["start"] == "random":
        model = rnd(side ** 3)
    else:
        m = truth.reshape(-1) * torch.exp(0.25 * torch.randn(side ** 3, generator=g, device="cuda"))
        model = m / m.mean()
    # photons of a pattern over the mean slice of the starting model
    probe = torch.from_numpy(q[:: max(1, len(q) // 64)]).cuda()
    wsum = float((_slices(model, _matrices(probe), side, xyz, "nearest") * on).sum(1).mean())
    scaling = ((counts * on).sum(1).float() / max(wsum, 1e-20)).clamp_min(1e-3)
    return dict(x=x, y=y, z=z, mask=mask, q=q, w=w, cell=cell, cells=cells, counts=counts,
                model=model, scaling=scaling, side=side)


def _slices(model, m, side, xyz, interp, dtype=torch.float32):
    """Slices [rotations][pixels] of the model: the nearest voxel inside
    1 <= k < side, or trilinear over the corners inside 0 <= k < side."""
    ps = _positions(m, side, xyz)
    if interp == "nearest":
        v, ok = _nearest(ps, side, 1)
        return model.to(dtype)[v] * ok
    out = 0
    for v, wt in _corners(ps, side):
        out = out + model.to(dtype)[v] * wt.to(dtype)
    return out


def _nearest(ps, side, lower):
    """Voxel index and whether it is inside (halves round away from zero)."""
    d = [p.double() for p in ps]
    k = [torch.trunc(p + torch.copysign(torch.full_like(p, 0.5), p)).long() for p in d]
    ok = functools.reduce(torch.logical_and, [(t >= lower) & (t < side) for t in k])
    return ((k[2] * side + k[1]) * side + k[0]) * ok, ok


def _corners(ps, side):
    base = [torch.floor(p) for p in ps]
    frac = [(p - b).double() for p, b in zip(ps, base)]
    for c in range(8):
        k = [b.long() + ((c >> i) & 1) for i, b in enumerate(base)]
        wt = 1.0
        for i in range(3):
            wt = wt * (frac[i] if (c >> i) & 1 else 1 - frac[i])
        ok = functools.reduce(torch.logical_and, [(t >= 0) & (t < side) for t in k])
        yield ((k[2] * side + k[1]) * side + k[0]) * ok, wt * ok


# -------------------------------------------------------------------- state --

class _Array:
    """A device buffer of a context; it keeps the context, which frees the
    buffer when it goes, for as long as a tensor made of it lives."""

    def __init__(self, owner, ptr, n):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (ptr, False),
                                         "version": 2, "strides": None}


def _view(ctx, which):
    """A context buffer as a CUDA tensor."""
    ptr, nbytes = ctx.device_buffer(which)
    return torch.as_tensor(_Array(ctx, ptr, nbytes // 4), device="cuda")


def _photon_lists(counts):
    """Non-zero pixels of every pattern as CSR lists in pinned host memory."""
    nz = counts != 0
    row = torch.zeros(counts.shape[0] + 1, dtype=torch.int64)
    row[1:] = nz.sum(1).cumsum(0).cpu()
    idx = nz.flatten().nonzero().flatten()
    pix = (idx % counts.shape[1]).int().cpu()
    val = counts.flatten()[idx].float().cpu()
    return [t.pin_memory().numpy() for t in (row, pix, val)]


class _Dataset:
    """One Context with its data set, and the model and scaling it starts from."""

    def __init__(self, case, side, seed):
        d = _dataset(case, side, seed)
        self.ctx = ctx = E.Context(side, case["patterns"], len(d["w"]), likelihood=case["likelihood"],
                                   interp=case["interp"], precision=case["precision"], sigma=SIGMA,
                                   poisson_floor=FLOOR)
        ctx.set_geometry(d["x"], d["y"], d["z"], d["mask"])
        ctx.set_rotations(d["q"], d["w"])
        self.lists = None
        if case["kind"] == "step" or case["photons"] < 0.2 * side * side:
            self.lists = _photon_lists(d["counts"])
            ctx.set_patterns_sparse(*self.lists)
        else:
            ctx.set_patterns(d["counts"].float().cpu().numpy())
        self.host_model = d["model"].cpu().pin_memory().numpy()
        self.host_scaling = d["scaling"].cpu().pin_memory().numpy()
        ctx.set_model(self.host_model)
        ctx.set_scaling(self.host_scaling)
        ctx.synchronize()
        self.model0, self.scaling0 = d["model"], d["scaling"]
        self.model, self.scaling = _view(ctx, E.BUF_MODEL), _view(ctx, E.BUF_SCALING)
        self.data = d if case["kind"] == "topk" else None

    def reset(self):
        """The starting model and scaling again (on the context's stream)."""
        self.model.copy_(self.model0)
        self.scaling.copy_(self.scaling0)


class _State:
    def __init__(self, case, seed):
        self.case = case
        sides = [int(s) for s in case["sides"].split(",")] if case["sides"] else [case["side"]]
        self.sets = [_Dataset(case, s, seed + 31 * i) for i, s in enumerate(sides)]
        self.batch = self.prop = self.log_keep = None
        if case["kind"] == "graph":
            self.batch = E.Batch([s.ctx for s in self.sets])
            self.batch.capture()
        ctx = self.sets[0].ctx
        self.stream = torch.cuda.ExternalStream(self.batch.stream if self.batch else ctx.stream)
        if case["kind"] == "topk":
            d = self.sets[0].data
            self.prop = PR.LearnedProposal(ctx, d["cell"], d["cells"])
            self.log_keep = _log_mass(case, d)
            self.sets[0].data = None
        torch.cuda.synchronize()
        torch.cuda.empty_cache()


def _log_mass(case, d):
    """Log-posterior mass of every coarse cell under the starting model: what
    the previous iteration leaves to the proposed one."""
    side = d["side"]
    on = torch.from_numpy(d["mask"]).cuda().nonzero().flatten()
    xyz = [torch.from_numpy(d[k]).cuda()[on] for k in "xyz"]
    K = d["counts"][:, on].float()
    m = _matrices(torch.from_numpy(d["q"]).cuda())
    out = torch.full((case["patterns"], d["cells"]), -math.inf, device="cuda")
    cell = d["cell"]
    for c in range(d["cells"]):
        r0, r1 = np.searchsorted(cell, [c, c + 1])
        if r1 > r0:
            S = _slices(d["model"], m[r0:r1], side, xyz, case["interp"])
            ll = K @ S.clamp_min(FLOOR).log().T - d["scaling"][:, None] * S.sum(1)
            out[:, c] = torch.logsumexp(ll.double(), 1)
    return (out.double() - torch.logsumexp(out.double(), 1, keepdim=True)).float().contiguous()


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    """One iteration from the starting model and scaling: the new model and
    scaling of every dataset (and the statistics where the program reads them)."""
    case, sets = state.case, state.sets
    ctx = sets[0].ctx
    if case["kind"] == "step":
        s = sets[0]
        ctx.set_patterns_sparse(*s.lists)
        ctx.set_model(s.host_model)
        ctx.set_scaling(s.host_scaling)
        ctx.iterate(stats=False)
        return [ctx.get_model(), ctx.get_scaling()]
    stats = None
    state.stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(state.stream):
        for s in sets:
            s.reset()
    if case["kind"] == "graph":
        state.batch.launch(1)
    elif case["kind"] == "topk":
        state.prop.iterate_topk(None, state.log_keep, top_k=TOP_K, max_cells=MAX_CELLS, audit=AUDIT)
    else:
        stats = ctx.iterate(stats=case["stats"])
    torch.cuda.current_stream().wait_stream(state.stream)
    out = [t for s in sets for t in (s.model, s.scaling)]
    if stats:
        out += [stats["sum_plogp"], stats["total_loglik"], stats["model_max"]]
    return out


# --------------------------------------------------------------------- work --

def work(case):
    """The photons, rotations, model and scaling once, and the log-likelihood of
    every (pattern, rotation) over the active pixels; with broad (gaussian)
    posteriors the slice sums are a second contraction of that size.  A
    proposed iteration evaluates a few per cent of the rotations."""
    sides = [int(s) for s in case["sides"].split(",")] if case["sides"] else [case["side"]]
    N, R = case["patterns"], _n_rotations(case["rot_n"])
    by = fl = 0.0
    for side in sides:
        npa = float(_geometry(side, case["beamstop"])[3].sum())
        share = min(1.0, TOP_K / R) if case["kind"] == "topk" else 1.0
        fl += 2.0 * N * R * npa * share * (2 if case["likelihood"] == "gauss" else 1)
        by += 8.0 * N * min(case["photons"], npa) + 20.0 * R + 12.0 * side ** 3 + 12.0 * N
    return {"bytes": by, "flops": fl}


# -------------------------------------------------------------------- exact --

def exact(case, seed):
    """The iteration in 64 bits, from its formulas.  None for a proposed
    iteration (its candidates are part of the method)."""
    if case["kind"] == "topk":
        return None
    sides = [int(s) for s in case["sides"].split(",")] if case["sides"] else [case["side"]]
    out, stats = [], None
    for i, side in enumerate(sides):
        model, scaling, stats = _exact_iteration(case, _dataset(case, side, seed + 31 * i))
        out += [model, scaling]
    torch.cuda.empty_cache()
    if case["kind"] == "iterate" and case["stats"]:
        out += stats
    return out


def _exact_iteration(case, d):
    side, poisson = d["side"], case["likelihood"] == "poisson"
    on = torch.from_numpy(d["mask"]).cuda().nonzero().flatten()
    xyz = [torch.from_numpy(d[k]).cuda()[on] for k in "xyz"]
    K = d["counts"][:, on].double()
    N, npa = K.shape
    m = _matrices(torch.from_numpy(d["q"]).cuda())
    w = torch.from_numpy(d["w"]).cuda().double()
    R = len(w)
    phi = d["scaling"].double()
    model = d["model"].double()
    inv = 1.0 / (2.0 * npa * SIGMA ** 2)
    step = max(1, (1 << 26) // npa)
    LL = torch.empty(R, N, dtype=torch.float64, device="cuda")
    stat = torch.empty(R, dtype=torch.float64, device="cuda")
    for r0 in range(0, R, step):
        S = _slices(model, m[r0:r0 + step], side, xyz, case["interp"], torch.float64)
        if poisson:
            stat[r0:r0 + step] = S.sum(1)
            LL[r0:r0 + step] = S.clamp_min(FLOOR).log() @ K.T
        else:
            stat[r0:r0 + step] = (S * S).sum(1)
            LL[r0:r0 + step] = S @ K.T
    if poisson:
        LL -= stat[:, None] * phi
        cross = None
    else:
        cross = LL.clone()
        LL.mul_(2 / phi).sub_(stat[:, None]).sub_((K * K).sum(1) / phi ** 2).mul_(inv)
    lse = torch.logsumexp(LL, 0)
    P = LL.sub_(lse).exp_()
    plogp = float(torch.xlogy(P, P).sum())
    if poisson:
        num, den = K.sum(1), P.T @ stat
    else:
        num, den = (K * K).sum(1), (P * cross).sum(0)
        del cross
    new = torch.where((num > 0) & (den > 0), num / den, phi)
    T = P.sum(1)
    Kphi = K / new[:, None]
    acc = torch.zeros(side ** 3, dtype=torch.float64, device="cuda")
    wgt = torch.zeros_like(acc)
    for r0 in range(0, R, step):
        t = T[r0:r0 + step]
        wt = torch.where(t > 1e-10, w[r0:r0 + step] * t, 0.0)[:, None]
        U = (P[r0:r0 + step] @ Kphi) / t.clamp_min(1e-300)[:, None]
        ps = _positions(m[r0:r0 + step], side, xyz)
        near = [_nearest(ps, side, 0)] if case["interp"] == "nearest" else _corners(ps, side)
        for v, c in near:
            c = (c * wt).double()
            acc.index_add_(0, v.flatten(), (c * U).flatten())
            wgt.index_add_(0, v.flatten(), c.flatten())
    out = torch.where(wgt > 0, acc / wgt.clamp_min(1e-300), 0.0)
    out /= out.mean()
    return out, new, [plogp, float(lse.sum()), float(out.max())]
