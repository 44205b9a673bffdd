"""The calls this framework is used for, with the sizes they are used at.

A user has a cortical surface (a closed mesh with the medial wall masked out), keeps one engine
per subject, and asks it for distance fields and per-vertex wiring metrics:

* `distance`  one FP64 field per call to host memory: what the reference's per-source loop does
              through the distance-engine plug-in;
* `fields`    several FP64 fields per call to host memory;
* `metrics`   the FP64 records (MSD, distance to boundary, radii, perimeters, samples) of host
              sources, host records back; one source is the interactive look at one vertex;
* `records`   the same, device-resident sources and records (the serving and sharding paths);
* `analysis`  `WiringAnalysis.compute_all_wiring_costs` of a set of vertices or, with
              count 0, of the whole cortex: the float32 arrays and sample rows that get saved;
* `subject`   one subject from its mesh: operators, ordering and factors built, then the
              whole-cortex analysis, as the batch runner does per subject.

Meshes are the repository's seeded folded icospheres, orders 4 (2.6k vertices) to 8 (655k), the
cap fraction giving the sizes in between. The scales are the batch runner's twelve or the
analysis' default six.
"""

import math

import numpy as np
import torch

from fastcorticalwiring_b200 import _lib
from fastcorticalwiring_b200 import mesh as M
from fastcorticalwiring_b200.analysis import WiringAnalysis
from fastcorticalwiring_b200.meshgen import folded_icosphere

DIFFUSION_MM = 0.7
POISSON_SHIFT = 1e-10


def _case(name, kind, level, count, precision="fp64", jitter=0.0, cap=0.10, scales="runner", between=3,
          boundary_cap=-1.0, robust=False, depth=4):
    c = dict(kind=kind, level=level, count=count, precision=precision, jitter=jitter, cap=cap, scales=scales,
             between=between, boundary_cap=boundary_cap, robust=robust, depth=depth)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the drop-in engine's call, on the smallest mesh in use and on the fsaverage-sized one
        _case("distance_L4", "distance", 4, 1),
        _case("distance_L7", "distance", 7, 1),
        # one vertex's metrics, interactively
        _case("metrics_one_L6", "metrics", 6, 1, jitter=0.2),
        # a few fields at once (a ragged block), kept on the host
        _case("fields_L5_37", "fields", 5, 37),
        # FP64 records on the device: one ragged block, and several blocks at full size
        _case("records_fp64_L5_1000", "records", 5, 1000, jitter=0.1),
        _case("records_fp64_L7_4096", "records", 7, 4096),
        # the float32 wiring maps: some vertices with the production (robust) operators, the
        # analysis' own scales and a boundary cap; whole small and medium surfaces; a large
        # share of the fsaverage-sized surface; a finer one than fsaverage
        _case("analysis_robust_L5_300", "analysis", 5, 300, "mixed", 0.1, scales="default", boundary_cap=0.05,
              robust=True),
        _case("analysis_L5_all", "analysis", 5, 0, "mixed"),
        _case("analysis_L6_all", "analysis", 6, 0, "mixed", 0.2),
        _case("analysis_L7_16384", "analysis", 7, 16384, "mixed"),
        _case("analysis_L8_2048", "analysis", 8, 2048, "mixed", depth=2),
        # a subject from its mesh to its maps
        _case("subject_L5", "subject", 5, 0, "mixed", 0.1),
    ]


def draw(rng):
    kind = rng.choice(["distance", "fields", "metrics", "records", "analysis", "analysis", "subject"])
    cap = round(rng.uniform(0.03, 0.6), 3)
    jitter = rng.choice([0.0, 0.1, 0.2])
    level = rng.choice([4, 5] if kind == "subject" else [4, 5, 6, 7])
    most = {"fields": 400, "metrics": 3000, "records": 4096}.get(kind, 8192)
    most = min(most, int(0.35 * _full_vertices(level)))
    count = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    between, scales = rng.choice([0, 1, 3, 3]), rng.choice(["runner", "default"])
    if kind == "distance":
        return _case("", kind, level, 1, "fp64", jitter, cap)
    if kind == "fields":
        return _case("", kind, level, count, "fp64", jitter, cap)
    if kind in ("metrics", "records"):
        return _case("", kind, level, count, "fp64", jitter, cap, scales, between)
    robust = kind == "analysis" and rng.random() < 0.25
    whole = kind == "subject" or (level <= 5 and rng.random() < 0.5)
    return _case("", kind, level, 0 if whole else count, rng.choice(["mixed", "mixed", "fp64"]), jitter, cap, scales,
                 between, rng.choice([-1.0, 0.05]), robust)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _full_vertices(level):
    return 10 * 4 ** level + 2


def _mesh(case, seed):
    # the finest order is folded by fewer harmonics: they are what making a mesh takes
    lmax = 12 if case["level"] < 8 else 6
    return folded_icosphere(case["level"], seed=seed, jitter=case["jitter"], cap_fraction=case["cap"], lmax=lmax)


def _analysis(case, m):
    a = WiringAnalysis(m.vertices, m.faces, m.cortex_mask, precision=case["precision"],
                       engine_kwargs=dict(use_robust=case["robust"], pipeline_depth=case["depth"]))
    a.quiet = True
    return a


_kept = {}  # the subject in hand: a program keeps one engine per subject and calls it many times


def _subject(case):
    key = tuple(case[k] for k in ("level", "jitter", "cap", "robust", "depth", "precision"))
    if key not in _kept:
        for a in _kept.values():
            a.distance_engine.engine.close()
        _kept.clear()
        _kept[key] = _analysis(case, _mesh(case, 1))
    return _kept[key]


def _scales(case):
    return M.RUNNER_SCALES if case["scales"] == "runner" else WiringAnalysis.DEFAULT_SCALES


def _chosen(case, seed, pm):
    """The sources of a call: cortical vertices in no particular order, each once."""
    n = min(max(1, case["count"]), pm.n_vertices)
    return np.random.default_rng([seed, 17]).permutation(pm.n_vertices)[:n].astype(np.int32)


def _own_mesh(case):
    """Whole-cortex calls on small meshes take another surface for another seed."""
    return case["kind"] == "subject" or (case["count"] == 0 and case["level"] <= 6)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("analysis", "subject"):
        s["rows"] = np.zeros((2, _sample_rows(case)), dtype=np.float32)
    if kind == "subject":
        return dict(s, mesh=_mesh(case, seed))
    a = s["analysis"] = _analysis(case, _mesh(case, seed)) if _own_mesh(case) else _subject(case)
    pm = a.mesh
    if case["count"] == 0:
        pm.bfs  # the analysis' source order, made once per surface
    src = _chosen(case, seed, pm)
    if kind == "analysis":
        s["vertices"] = None if case["count"] == 0 else [int(v) for v in pm.sub_to_orig[src]]
    else:
        s.update(sources=src, targets=pm.targets(_scales(case)))
    if kind == "records":
        s["sources"] = torch.from_numpy(src).cuda()
        s["out"] = torch.empty((src.size, _lib.metrics_stride(len(s["targets"]), case["between"])),
                               dtype=torch.float64, device="cuda")
    return s


def _sample_rows(case):
    """Entries that hold every sample of a call: flagged sources have none, so fewer are used."""
    sources = case["count"] or _full_vertices(case["level"])
    return sources * _lib.samples_capacity(len(_scales(case)), case["between"])


def _padded(flat, rows):
    rows[:flat.size] = flat
    rows[flat.size:] = 0.0
    return rows


def _wiring(a, case, rows, vertices=None):
    cap = case["boundary_cap"]
    a.compute_all_wiring_costs(scale=_scales(case), vertex_subset=vertices, n_samples_between_scales=case["between"],
                               boundary_cap_fraction=None if cap < 0 else cap)
    return dict(a.get_metric_arrays(), field_flag=a.field_flag, sample_indptr=a.sample_indptr,
                sample_radii=_padded(a.sample_radii_flat, rows[0]), sample_areas=_padded(a.sample_areas_flat, rows[1]))


def _columns(rec):
    """A record's parts: MSD, boundary distance and health; the Newton evaluations; the geometry."""
    return dict(summary=rec[:, :6], evaluations=rec[:, 6], geometry=rec[:, 7:])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "subject":
        m = state["mesh"]
        a = _analysis(case, m)
        out = _wiring(a, case, state["rows"])
        a.distance_engine.engine.close()
        return out
    a = state["analysis"]
    if kind == "analysis":
        return _wiring(a, case, state["rows"], state["vertices"])
    eng = a.distance_engine.engine
    src = state["sources"]
    if kind == "distance":
        return a.distance_engine.compute_distance(int(src[0]))
    if kind == "fields":
        return eng.compute_distances(src, precision=case["precision"])
    if kind == "metrics":
        return _columns(eng.compute_metrics(src, state["targets"], n_between=case["between"],
                                            precision=case["precision"]))
    eng.compute_metrics_device(src, state["targets"], case["between"], 1e-6, case["precision"], state["out"],
                               torch.cuda.current_stream().cuda_stream)
    return _columns(state["out"])


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    n = int((1.0 - case["cap"]) * _full_vertices(case["level"]))
    nf = 2 * n
    count = 1 if case["kind"] in ("distance",) else (case["count"] or n)
    # entries of one factor in a minimum-degree order of such a mesh
    nnz = n * max(10.0, 7.3 * math.log2(n) - 54.0)
    half = 4 if case["precision"] == "mixed" else 8
    scales = len(_scales(case))
    record = 8 * (7 + 2 * scales + 2 * (scales - 1) * case["between"])
    fields = case["kind"] in ("distance", "fields")
    out = count * (8 * n if fields else record)
    # both factors and the mesh read once, the results written once; per source the heat
    # backward and both Poisson sweeps, each face's unit gradient and its divergence
    flops = count * (3 * 2.0 * nnz + 60.0 * nf)
    if case["kind"] == "subject":  # both factorisations (a nested-dissection order's 10 n^1.5) and the FP32 one
        flops += 3 * 10.0 * n ** 1.5
    return {"bytes": float(nnz * (8 + half) + nf * 12 + n * 24 + out), "flops": float(flops)}


# ---------------------------------------------------------------------------
# the same quantities in 64 bits, from dense operators, in plain torch
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Dense:
    """Heat-method distances of a triangle mesh with dense factors (consistent operators)."""

    def __init__(self, V, F):
        dev = _dev()
        self.V = torch.as_tensor(V, dtype=torch.float64, device=dev)
        self.F = torch.as_tensor(np.asarray(F, np.int64), device=dev)
        V, F = self.V, self.F
        n = self.n = V.shape[0]
        p = [V[F[:, c]] for c in range(3)]
        normal = torch.linalg.cross(p[1] - p[0], p[2] - p[0])
        twice = normal.norm(dim=1)
        self.area = 0.5 * twice
        unit = normal / twice[:, None]
        # gradient of the hat function of corner c: the opposite edge turned by 90 degrees
        self.g = [torch.linalg.cross(unit, p[(c + 2) % 3] - p[(c + 1) % 3]) / twice[:, None] for c in range(3)]
        L = torch.zeros((n, n), dtype=torch.float64, device=dev)
        for i in range(3):
            for j in range(3):
                L.index_put_((F[:, i], F[:, j]), self.area * (self.g[i] * self.g[j]).sum(1), accumulate=True)
        self.mass = torch.zeros(n, dtype=torch.float64, device=dev)
        for c in range(3):
            self.mass.index_add_(0, F[:, c], self.area / 3.0)
        A = L * DIFFUSION_MM ** 2
        A.diagonal().add_(self.mass)
        self.heat = torch.linalg.cholesky(A)
        del A
        L.diagonal().add_(POISSON_SHIFT * self.mass)
        self.poisson = torch.linalg.cholesky(L)

    def distances(self, src):
        """k x n fields of the sources src."""
        src = torch.as_tensor(np.asarray(src, np.int64), device=self.V.device)
        k = src.numel()
        b = torch.zeros((self.n, k), dtype=torch.float64, device=self.V.device)
        b[src, torch.arange(k, device=b.device)] = 1.0
        u = torch.cholesky_solve(b, self.heat)
        F = self.F
        div = torch.zeros_like(u)
        for f0 in range(0, F.shape[0], 8192):
            f = slice(f0, f0 + 8192)
            u0 = u[F[f, 0]]
            d1, d2 = u[F[f, 1]] - u0, u[F[f, 2]] - u0
            grad = [d1 * self.g[1][f, c, None] + d2 * self.g[2][f, c, None] for c in range(3)]
            norm = torch.sqrt(grad[0] ** 2 + grad[1] ** 2 + grad[2] ** 2)
            s = torch.where(norm > 1e-300, -self.area[f, None] / norm, torch.zeros_like(norm))
            for c in range(3):
                div.index_add_(0, F[f, c], s * sum(grad[x] * self.g[c][f, x, None] for x in range(3)))
        phi = torch.cholesky_solve(div, self.poisson).T
        return phi - phi.gather(1, src[:, None])


class _Geometry:
    """Areas, level-set lengths and radii of linear fields on a mesh, k fields (rows of d) at once."""

    def __init__(self, V, F, d):
        p = [V[F[:, c]] for c in range(3)]
        e1, e2 = p[1] - p[0], p[2] - p[0]
        a11, a22, a12 = (e1 * e1).sum(1), (e2 * e2).sum(1), (e1 * e2).sum(1)
        det = a11 * a22 - a12 * a12
        self.area = 0.5 * torch.sqrt(det)
        c = [d[:, F[:, i]] for i in range(3)]
        al, be = c[1] - c[0], c[2] - c[0]
        self.slope = torch.sqrt((al * al * a22 - 2.0 * al * be * a12 + be * be * a11) / det)
        self.hi = torch.maximum(torch.maximum(c[0], c[1]), c[2])
        self.lo = torch.minimum(torch.minimum(c[0], c[1]), c[2])
        self.mi = torch.maximum(torch.minimum(c[0], c[1]), torch.minimum(torch.maximum(c[0], c[1]), c[2]))
        self.dmax = self.hi.max(1).values

    def at(self, r, perimeter=False):
        """Area of {d <= r[k]} and its derivative, or the length of the level set."""
        lo, mi, hi, A, r = self.lo, self.mi, self.hi, self.area, r[:, None]
        low = r < mi
        den = (hi - lo) * torch.where(low, mi - lo, hi - mi)
        z = torch.where(low, r - lo, hi - r)
        part = z * z / den
        inside = (r > lo) & (r < hi)
        da = torch.where(inside, 2.0 * A * z / den, 0.0)
        if perimeter:
            return (da * self.slope).sum(1)
        ar = torch.where(inside, A * torch.where(low, part, 1.0 - part), torch.where(r >= hi, A, 0.0))
        return ar.sum(1), da.sum(1)

    def radius(self, target):
        """r with area(r) = target: Newton kept in a bracket."""
        lo, hi = torch.zeros_like(self.dmax), self.dmax.clone()
        r = torch.minimum(torch.full_like(hi, math.sqrt(target / math.pi)), 0.5 * hi)
        for _ in range(60):
            a, da = self.at(r)
            err = a - target
            if bool((err.abs() <= 1e-12 * target).all()):
                break
            hi, lo = torch.where(err > 0, r, hi), torch.where(err > 0, lo, r)
            new = r - err / da
            r = torch.where((da > 0) & (new > lo) & (new < hi), new, 0.5 * (lo + hi))
        return r


def exact(case, seed):
    n = (1.0 - case["cap"]) * _full_vertices(case["level"])
    count = case["count"] or n
    if case["robust"] or n > 40000 or (case["kind"] not in ("distance", "fields") and count * 2 * n > 2e8):
        return None
    own = _own_mesh(case)
    m = _mesh(case, seed if own else 1)
    pm = M.prepare(m.vertices, m.faces, m.cortex_mask)
    kind = case["kind"]
    src = np.arange(pm.n_vertices) if case["count"] == 0 else _chosen(case, seed, pm)
    dense = _Dense(pm.V, pm.F)
    if kind in ("distance", "fields"):
        d = dense.distances(src)
        return d[0] if kind == "distance" else d
    dev = _dev()
    va = torch.as_tensor(pm.vertex_area, device=dev)
    bnd = torch.as_tensor(pm.boundary.astype(np.int64), device=dev)
    scales, m_ = _scales(case), case["between"]
    targets = pm.targets(scales)
    nt, ne = len(targets), (len(targets) - 1) * m_
    rec = torch.zeros((src.size, 7 + 2 * nt + 2 * ne), dtype=torch.float64, device=dev)
    step = max(1, int(2e7 // pm.n_faces))
    for k0 in range(0, src.size, 512):
        part = src[k0:k0 + 512]
        fields = dense.distances(part)
        for j0 in range(0, part.size, step):
            d = fields[j0:j0 + step]
            o = rec[k0 + j0:k0 + j0 + d.shape[0]]
            at = torch.as_tensor(part[j0:j0 + step].astype(np.int64), device=dev)
            valid = d > 1e-6
            o[:, 0] = torch.where(valid, d, 0.0).sum(1) / valid.sum(1)
            o[:, 1] = (torch.where(valid, d, 0.0) @ va) / (valid.double() @ va)
            o[:, 2] = d[:, bnd].min(1).values if bnd.numel() else math.inf
            h = pm.health_h
            chord = (dense.V[None] - dense.V[at][:, None]).norm(dim=2)
            o[:, 3] = (d < -h).double().mean(1)
            o[:, 4] = (d < 0.9 * chord - h).double().mean(1)
            bad = (o[:, 3] > 1e-3) | (o[:, 4] > 1e-3)
            o[:, 5] = bad.double()
            geo = _Geometry(dense.V, dense.F, d)
            for i, t in enumerate(targets):
                o[:, 7 + i] = r = geo.radius(float(t))
                o[:, 7 + nt + i] = geo.at(r, perimeter=True)
            for i in range(nt - 1):
                for j in range(m_):
                    l0, l1 = torch.log(o[:, 7 + i]), torch.log(o[:, 8 + i])
                    r = torch.exp(l0 + (j + 1.0) / (m_ + 1.0) * (l1 - l0))
                    o[:, 7 + 2 * nt + i * m_ + j] = r
                    o[:, 7 + 2 * nt + ne + i * m_ + j] = geo.at(r)[0]
            o[:, 7:][bad] = math.nan
    rec = rec.cpu().numpy()
    if kind in ("metrics", "records"):
        return dict(_columns(rec), evaluations=None)
    return _exact_arrays(case, pm, src, rec, scales, targets, nt, m_, ne)


def _exact_arrays(case, pm, src, rec, scales, targets, nt, m_, ne):
    """The analysis' arrays over the full mesh from the records."""
    n = pm.cortex_mask_full.shape[0]
    orig = pm.sub_to_orig[src]
    good = rec[:, 5] == 0.0

    def full(col):
        x = np.full(n, np.nan)
        x[orig[good]] = rec[good, col]
        return x

    out = dict(msd_unweighted=full(0), msd_weighted=full(1), dist_to_boundary=full(2), field_flag=None,
               sample_indptr=None, sample_radii=None, sample_areas=None)
    for i, s in enumerate(scales):
        token = WiringAnalysis.scale_token(s)
        out["radius_" + token], out["perimeter_" + token] = full(7 + i), full(7 + nt + i)
    if case["boundary_cap"] < 0:  # each row: the scales and the samples between them, by radius
        col_r, col_a = [], []
        for i in range(nt):
            col_r.append(rec[:, 7 + i])
            col_a.append(np.full(src.size, targets[i]))
            for j in range(m_ if i + 1 < nt else 0):
                col_r.append(rec[:, 7 + 2 * nt + i * m_ + j])
                col_a.append(rec[:, 7 + 2 * nt + ne + i * m_ + j])
        by = np.argsort(orig[good], kind="stable")
        for name, col in (("sample_radii", col_r), ("sample_areas", col_a)):
            out[name] = _padded(np.stack(col, 1)[good][by].reshape(-1), np.zeros(_sample_rows(case)))
    return out
