"""Performance cases of the estimator stage: what a renderer has the library do, from the smallest call
to the largest iteration, through the public entry points.

The kinds of call:

* ``host``: one whole iteration from host records (``EstimatorStage.run``): upload, build, evaluate,
  the per-call results and the image read back, as the drop-in in a CPU renderer makes it.
* ``stage``: build, clear, evaluate and the image, on records that are already on the device.
* ``iteration``: the same with the light and camera passes on the device in front.
* ``gradient``: forward and backward of the differentiable estimator (``autograd.render``).
* ``noalloc``: the allocation-free PP3D call (``upbp_pp3d_evaluate_noalloc``) on device arrays.

``exact`` restates the estimators in 64 bits with torch, every pair tested, for the cases small enough.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from smallupbp_b200 import abi, autograd, engine
from smallupbp_b200 import workload as W

MODES = {"plain": engine.MODE_PLAIN, "mixed": engine.MODE_MIXED}

BASE = dict(kind="stage", scene="cube", mode="mixed", width=128, height=128, light_paths=16384, radius=0.01,
            photon_beams="short", query_beams="long", knn_photons=0, knn_beams=0, grid_res=0, mis=True, bp2d=False,
            rays=0, beams=0)


def case(name, **kw):
    return dict(BASE, name=name, **kw)


def listed():
    long2 = dict(photon_beams="long", radius=0.005)
    return [
        # A preview or a unit test of the renderer: the library's default (plain FP32) mode, everything
        # from host memory.  Launches, uploads and synchronisations count here.
        case("host_cube24", kind="host", mode="plain", width=24, height=24, light_paths=1536, radius=0.02),
        # A host application without device memory of its own to give asks for PP3D only.
        case("noalloc_cube64", kind="noalloc", mode="plain", width=64, height=64, light_paths=87000),
        # The small configuration (cube128), with its SHORT photon beams.
        case("stage_cube128"),
        # VolLightTracer's estimators without MIS, SHORT beams on both sides, a ragged image, B-P2D on.
        case("stage_nomis_317x243", mis=False, bp2d=True, query_beams="short", width=317, height=243,
             light_paths=40000, radius=0.008),
        # Interactive quality: a quarter of the large cube, in mixed precision ...
        case("stage_cube512", width=512, height=512, light_paths=262144, **long2),
        # ... in the reference's own precision ...
        case("stage_cube512_plain", mode="plain", width=512, height=512, light_paths=262144, **long2),
        # ... with the reference's KNN radii (-r_initial_pb2d_knn, -r_initial_bb1d_knn) ...
        case("stage_cube512_knn", width=512, height=512, light_paths=262144, knn_photons=8, knn_beams=6, **long2),
        # ... and over the reference's own uniform beam grid (-gridres 64).
        case("stage_cube512_grid64", width=512, height=512, light_paths=262144, grid_res=64, **long2),
        # Inverse rendering: one forward and backward pass for a medium's parameters.
        case("gradient_cube256", kind="gradient", width=256, height=256, light_paths=65536),
        # Beam-beam geometry without any coherence between the rays (closest-approach stress).
        case("stage_stress300k", scene="stress", beams=300000, rays=300000, radius=0.002),
        # The production iteration: 1024 x 1024, a million light paths, LONG photon beams.
        case("stage_cube1024", width=1024, height=1024, light_paths=1048576, **long2),
        # The heavy-tailed scene: three nested media, two million light paths, the light and camera passes
        # on the device as well.
        case("iteration_boxes1024", kind="iteration", scene="boxes", width=1024, height=1024, light_paths=2097152,
             radius=0.005),
    ]


def log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "noalloc", "stage", "stage", "stage", "stage", "iteration", "gradient"])
    scene = rng.choice(["cube", "cube", "boxes"]) if kind != "noalloc" else "cube"
    if kind == "stage" and rng.random() < 0.15:
        scene = "stress"
    option = rng.choice(["", "", "plain", "knn", "grid", "nomis"]) if kind == "stage" and scene != "stress" else ""
    c = dict(BASE, kind=kind, scene=scene)
    largest = {"host": 200, "noalloc": 200, "gradient": 300}.get(kind) or \
        {"": 800, "plain": 500, "knn": 600, "grid": 500, "nomis": 317}[option]
    w = log_int(rng, 24, largest)
    c["width"], c["height"] = w, max(16, int(w * rng.uniform(0.6, 1.1)))
    # about as many light paths as pixels, as in every configuration here
    c["light_paths"] = max(512, int(w * c["height"] * rng.uniform(0.5, 1.3)))
    if kind == "noalloc":
        c["light_paths"] = min(c["light_paths"], 80000)
    c["radius"] = round(rng.uniform(0.004, 0.006) if w > 300 else rng.uniform(0.008, 0.02), 4)
    c["photon_beams"] = rng.choice(["short", "long"]) if scene == "cube" else "short"
    if kind in ("host", "noalloc") or option == "plain":
        c["mode"] = "plain"
    if scene == "stress":
        c["beams"], c["rays"], c["radius"] = log_int(rng, 20000, 400000), log_int(rng, 20000, 400000), 0.002
    if option == "knn":
        c["knn_photons"], c["knn_beams"] = rng.randint(3, 10), rng.randint(3, 8)
    if option == "grid":
        c["grid_res"] = rng.randint(24, 80)
    if option == "nomis":
        c["height"], c["light_paths"] = min(c["height"], 243), min(c["light_paths"], 40000)
        c["mis"], c["query_beams"], c["bp2d"] = False, rng.choice(["short", "long"]), rng.random() < 0.5
    return c


# ---------------------------------------------------------------------------------------------------- inputs

def scene_config(c, seed):
    kw = dict(photon_beam_type=W.LONG_BEAM if c["photon_beams"] == "long" else W.SHORT_BEAM,
              query_beam_type=W.LONG_BEAM if c["query_beams"] == "long" else W.SHORT_BEAM,
              pb2d_knn=c["knn_photons"], bb1d_knn=c["knn_beams"], seed=1234 + seed)
    if c["photon_beams"] == "long":
        kw["beam_length_cap"] = 2.0
    make = W.cube_scene if c["scene"] == "cube" else W.nested_boxes_scene
    return make(c["scene"], c["width"], c["height"], c["light_paths"], 6, c["radius"], **kw)


def host_records(c, seed):
    """The iteration's records as a renderer holds them on the host (deterministic in the seed)."""
    if c["scene"] == "stress":
        return W.beam_stress(c["beams"], c["rays"], radius=c["radius"], seed=1234 + seed)
    w = W.generate(scene_config(c, seed), 0)
    if c["mis"]:
        return w
    n = W.without_mis(w, W.PB2D | W.BB1D | (W.BP2D if c["bp2d"] else 0))
    if c["bp2d"]:  # B-P2D is evaluated at the camera vertices
        n.update({k: w[k] for k in w if k.startswith("pq_")})
    return n


def device_arrays(w):
    """The records of the allocation-free call in device memory, as upbp_gpu.h structs, and their owners."""
    keep = {k: torch.from_numpy(np.ascontiguousarray(v).view(np.uint8).reshape(-1)).cuda()
            for k, v in w.items() if k.startswith(("lv_", "pq_", "cam_"))}

    def p(name, ctype):
        return C.cast(C.c_void_p(keep[name].data_ptr()), ctype)

    lv = abi.LightVertices(
        n=len(w["lv_path_idx"]), position=p("lv_position", abi.f32p), throughput=p("lv_throughput", abi.f32p),
        dir_fix=p("lv_dir_fix", abi.f32p), cont_prob=p("lv_cont_prob", abi.f32p), path_idx=p("lv_path_idx", abi.i32p),
        path_length=p("lv_path_length", abi.i32p), medium_id=p("lv_medium_id", abi.i32p),
        flags=p("lv_flags", abi.u32p), mis=p("lv_mis", C.POINTER(abi.Mis)), n_paths=len(w["lv_path_ends"]),
        path_ends=p("lv_path_ends", abi.i32p))
    pq = abi.PointQueries(
        n=len(w["pq_path_length"]), position=p("pq_position", abi.f32p), dir_fix=p("pq_dir_fix", abi.f32p),
        medium_id=p("pq_medium_id", abi.i32p), path_length=p("pq_path_length", abi.i32p),
        throughput=p("pq_throughput", abi.f32p), pixel=p("pq_pixel", abi.i32p),
        cam_mis_begin=p("pq_cam_mis_begin", abi.i64p))
    cam = p("cam_mis", C.POINTER(abi.Mis))
    params = abi.Params.from_buffer_copy(np.ascontiguousarray(w["params"]).tobytes())
    media = (abi.Medium * len(w["media"])).from_buffer_copy(np.ascontiguousarray(w["media"]).tobytes())
    return params, media, lv, pq, cam, keep


def calls(c):
    """Room for the per-call results of any iteration: the number of calls varies with the seed."""
    return 6 * c["width"] * c["height"]


def prepare(c, seed):
    s = dict(case=c)
    if c["kind"] == "host":
        s["stage"], s["records"] = engine.EstimatorStage(0, MODES[c["mode"]]), host_records(c, seed)
        s["results"] = {e: np.zeros((calls(c), 3), np.float32) for e in ("pb2d", "bb1d", "pp3d")}
        s["results"]["counts"] = np.zeros((calls(c), 3), np.int64)
        return s
    if c["kind"] == "noalloc":
        w = host_records(c, seed)
        s["params"], s["media"], s["lv"], s["pq"], s["cam"], s["keep"] = device_arrays(w)
        s["out"] = torch.zeros(calls(c), 3, dtype=torch.float32, device="cuda")
        s["call"] = engine.lib().upbp_pp3d_evaluate_noalloc
        s["call"].restype = C.c_int
        s["call"].argtypes = [C.POINTER(abi.Params), C.POINTER(abi.Medium), C.c_int32, C.POINTER(abi.LightVertices),
                              C.POINTER(abi.Mis), C.POINTER(abi.PointQueries), abi.f32p, C.c_void_p]
        return s
    st = s["stage"] = engine.EstimatorStage(0, MODES[c["mode"]])
    if c["grid_res"]:
        st.set_bb1d_grid(c["grid_res"])
    if c["scene"] == "stress" or not c["mis"]:
        w = s["records"] = host_records(c, seed)
        structs = abi.make_structs(w)
        st.load(w, structs)
        st.set_queries(w, structs)
    else:
        s["config"] = scene_config(c, seed)
        st.trace(s["config"], 0)
        if c["kind"] == "iteration":
            s["iteration"] = 0
    if c["kind"] == "gradient":
        st.build()
        media, _ = W.stage_constants(s["config"], 0)
        s["media"], s["medium"] = media, len(media) - 1
        m = media[-1]
        kw = dict(dtype=torch.float32, device="cuda", requires_grad=True)
        s["theta"] = [torch.tensor([float(x) for x in m["absorption"]], **kw),
                      torch.tensor([float(x) for x in m["scattering"]], **kw),
                      torch.tensor(float(m["mean_cosine"]), **kw)]
        gen = torch.Generator().manual_seed(99 + seed)
        s["target"] = (torch.rand(st.pixels(), 3, generator=gen) * 0.5).cuda()
    s["image"] = torch.zeros(st.pixels(), 3, dtype=torch.float32, device="cuda")
    return s


# ---------------------------------------------------------------------------------------------------- the pass

def run(s):
    c = s["case"]
    if c["kind"] == "noalloc":
        rc = s["call"](C.byref(s["params"]), s["media"], len(s["media"]), C.byref(s["lv"]), s["cam"], C.byref(s["pq"]),
                       C.cast(C.c_void_p(s["out"].data_ptr()), abi.f32p),
                       C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise engine.UpbpError(rc, "upbp_pp3d_evaluate_noalloc")
        return {"pp3d": s["out"]}
    st = s["stage"]
    if c["kind"] == "host":
        st.run(s["records"])
        out, stats = s["results"], st.query_stats()
        pb2d, bb1d = st.segment_results()
        for k, (name, rgb) in enumerate((("pb2d", pb2d), ("bb1d", bb1d), ("pp3d", st.point_results()))):
            out[name][:len(rgb)] = rgb
            out["counts"][:len(rgb), k] = stats["count_" + name]
        return dict(out, image=st.image())
    if c["kind"] == "gradient":
        for t in s["theta"]:
            t.grad = None
        image = autograd.render(st, s["media"], s["medium"], *s["theta"])
        ((image - s["target"]) ** 2).sum().backward()
        return {"image": image.detach(), "gradients": [t.grad for t in s["theta"]]}
    if c["kind"] == "iteration":
        st.trace(s["config"], s["iteration"])
    st.build()
    st.clear_image()
    st.evaluate()
    st.read_image_into(s["image"].data_ptr())
    return {"image": s["image"]}


# ---------------------------------------------------------------------------------------------------- the work

def work(c):
    """Estimates from the scene's averages (the counts of an iteration are random): records read, results
    and image written, and about 120 operations for each accepted pair (transmittance, phase function,
    kernel, MIS weight).  A segment of length l crosses 2 r l D pi/4 beams at a beam length density D."""
    px, n, r = c["width"] * c["height"], c["light_paths"], c["radius"]
    if c["scene"] == "stress":
        rays, beams, lq, lb, photons, points = c["rays"], c["beams"], 0.5, 0.5, 0, 0
        n, px = 4096, 64 * 64
    elif c["scene"] == "cube":
        rays, photons, points = 0.83 * px, 0.47 * n, 0.23 * px
        beams, lq = 1.38 * n, 0.9
        lb = 0.6 if c["photon_beams"] == "long" else 0.4
    else:
        rays, photons, points, beams, lq, lb = 0.95 * px, 0.6 * n, 0.3 * px, 1.9 * n, 0.9, 0.25
    if c["kind"] == "noalloc":
        pairs, byts = points * photons * 4.2 * r ** 3, 140 * photons + 180 * points
        return {"bytes": byts, "flops": 120 * pairs}
    pairs = rays * beams * lb * 2 * r * lq * 0.785 + rays * photons * math.pi * r * r * lq
    byts = 136 * (photons + 0.3 * n) + 68 * beams + 190 * rays + 180 * points + 12 * px
    if c["kind"] == "iteration":
        byts = 2 * byts
    if c["kind"] == "gradient":
        return {"bytes": 2 * byts, "flops": (120 + 360) * pairs}
    return {"bytes": byts, "flops": 120 * pairs}


# ---------------------------------------------------------------------------------------------------- 64 bits

class Records:
    """A workload's arrays as float64 / int64 tensors, MIS records as one tensor per field."""

    def __init__(self, w):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.w, self.dev, self.t = w, dev, {}
        for k, v in w.items():
            if k in ("media", "params"):
                continue
            v = np.ascontiguousarray(v)
            if v.dtype.names:
                for f in v.dtype.names:
                    self.t[k + "." + f] = self.tensor(v[f])
            else:
                self.t[k] = self.tensor(v)
        self.p = {f: (int if w["params"][f].dtype.kind in "iu" else float)(w["params"][f][0])
                  for f in w["params"].dtype.names}
        m = w["media"]
        st32 = np.abs(m["absorption"]) + np.abs(m["scattering"])
        lowest = np.where(st32 > 0, st32, np.inf)
        self.index = self.tensor(np.where((st32 > 0).any(1), lowest.argmin(1), 0))
        self.st, self.ss = self.tensor(st32), self.tensor(np.abs(m["scattering"]))
        self.min_st = self.st.gather(1, self.index[:, None])[:, 0]
        self.g, self.cont = self.tensor(m["mean_cosine"]), self.tensor(m["continuation_prob"])
        self.mfp = 1.0 / self.st.max(1).values
        self.scat = (self.ss > 0).any(1)

    def tensor(self, a):
        a = np.ascontiguousarray(a)
        return torch.from_numpy(a.astype(np.float64 if a.dtype.kind == "f" else np.int64)).to(self.dev)

    def __getitem__(self, k):
        return self.t[k]

    def att(self, med, t):
        return torch.exp(-self.st[med] * t[:, None])

    def least(self, med, rgb):
        return rgb.gather(1, self.index[med][:, None])[:, 0]

    def phase(self, med, cos):
        """Henyey-Greenstein pdf for the cosine of the deflection, and the sine."""
        g = self.g[med]
        iso = torch.full_like(cos, 0.25 / math.pi)
        hg = 0.25 / math.pi * (1 - g * g) / (1 + g * g - 2 * g * cos).clamp_min(1e-30) ** 1.5
        return torch.where(g.abs() < 1e-3, iso, hg), (1 - cos * cos).clamp_min(0).sqrt()


MIS = ("pdf_a_inv", "rev_pdf_a", "rev_pdf_a_without_bsdf", "ray_sample_pdf_inv", "ray_sample_rev_pdf_inv",
       "ray_sample_pdfs_ratio", "ray_sample_rev_pdfs_ratio", "sin_theta", "cos_theta_out", "surf_factor",
       "pp3d_factor", "pb2d_factor", "bb1d_factor", "bb1d_beam_selection_pdf", "flags")


def records_at(R, name, i):
    i = i.clamp(0, max(0, len(R[name + ".flags"]) - 1))
    return {f: R[name + "." + f][i] for f in MIS}


def chosen(mask, a, b):
    return {f: torch.where(mask, a[f], b[f]) for f in MIS}


def merge_terms(R, m, usable, light):
    """Density ratios of the merging techniques at one vertex: all but BB1D, and BB1D."""
    p, t = R.p, R.p["techniques"]
    qlong, plong = p["query_beam_type"] == W.LONG_BEAM, p["photon_beam_type"] == W.LONG_BEAM
    qa = ("ray_sample_rev_pdf_inv" if qlong else "ray_sample_rev_pdfs_ratio") if light else \
         ("ray_sample_pdf_inv" if qlong else "ray_sample_pdfs_ratio")
    pa = ("ray_sample_pdf_inv" if plong else "ray_sample_pdfs_ratio") if light else \
         ("ray_sample_rev_pdf_inv" if plong else "ray_sample_rev_pdfs_ratio")
    other = torch.zeros_like(m["pdf_a_inv"])
    if t & W.SURF:
        other = other + m["surf_factor"] * usable
    if t & W.PP3D:
        other = other + m["pp3d_factor"]
    if t & W.PB2D:
        other = other + m["pb2d_factor"] * m[qa]
    bb = m["bb1d_factor"] * m["bb1d_beam_selection_pdf"] * m[qa] * m["sin_theta"] * m[pa]
    return other, torch.where((m["flags"] & W.MIS_IN_MEDIUM_WITH_BEAMS) != 0, bb, 0.0) if t & W.BB1D else 0.0 * bb


def camera_weight(R, L, first, at, last, ntl):
    """AccumulateCameraPathWeight: `first` the merged vertex, at(k) camera entry k, `last` its reverse pdf."""
    weight, product = torch.zeros_like(last), torch.ones_like(last)
    for i in range(int(L.max()) if len(L) else 0):
        on = i < L
        m = first if i == 0 else at(L - i)
        spec = (m["flags"] & W.MIS_IS_SPECULAR) != 0
        following = at(L - i - 1)
        next_spec = torch.where(i < L - 1, (following["flags"] & W.MIS_IS_SPECULAR) != 0, spec)
        rev = last if i == 0 else m["rev_pdf_a"] * (ntl if i == 1 else 1.0)
        usable = torch.ones_like(spec) if i == 0 else ~spec
        product = torch.where(on, product * rev, product)
        a, b = merge_terms(R, m, usable.double(), False)
        weight = weight + torch.where(on, product * (a + b), 0.0)
        product = torch.where(on, product * m["pdf_a_inv"], product)
        if R.p["techniques"] & W.BPT:
            weight = weight + torch.where(on & usable & ~next_spec, product, 0.0)
    return weight


def light_weight(R, path, length, first, at, last, ntl, beam):
    """AccumulateLightPathWeight: `first` the merged vertex (index 0), at(v) light vertex v."""
    ends = R["lv_path_ends"]
    start = torch.where(path == 0, 0, ends[(path - 1).clamp_min(0)])
    weight, product, on = torch.zeros_like(last), torch.ones_like(last), torch.ones_like(last, dtype=torch.bool)
    for i in range(int(length.max()) + 1 if len(length) else 0):
        v = start + length - i
        m = first if i == 0 else at(v)
        spec = (m["flags"] & W.MIS_IS_SPECULAR) != 0
        next_spec = torch.where(i < length, (at(v - 1)["flags"] & W.MIS_IS_SPECULAR) != 0, spec)
        rev = last if i == 0 else m["rev_pdf_a"] if i > 1 else ntl if beam else m["rev_pdf_a_without_bsdf"] * ntl
        on = on & (i <= length) & (rev != 0)
        product = torch.where(on, product * rev, product)
        usable = torch.ones_like(spec) if i == 0 else ~spec
        if i:
            a, b = merge_terms(R, m, usable.double(), True)
            weight = weight + torch.where(on, product * (a + b), 0.0)
        product = torch.where(on, product * m["pdf_a_inv"], product)
        if R.p["techniques"] & W.BPT:
            weight = weight + torch.where(on & usable & ~next_spec, product, 0.0)
    return weight


def merged_vertex(R, like, med, pdf_a_inv, ray_inv):
    z, one = torch.zeros_like(like), torch.ones_like(like)
    p = R.p
    return dict(pdf_a_inv=pdf_a_inv, rev_pdf_a=one, rev_pdf_a_without_bsdf=one, ray_sample_pdf_inv=ray_inv,
                ray_sample_rev_pdf_inv=one, ray_sample_pdfs_ratio=1 / R.min_st[med], ray_sample_rev_pdfs_ratio=z,
                sin_theta=z, cos_theta_out=z, surf_factor=z, pp3d_factor=one * p["mis_factor_pp3d"],
                pb2d_factor=one * p["mis_factor_pb2d"], bb1d_factor=one * p["mis_factor_bb1d"],
                bb1d_beam_selection_pdf=one, flags=torch.full_like(med, W.MIS_IN_MEDIUM_WITH_BEAMS))


def segments(R):
    """The segments of all queries in walk order, with what the earlier ones of the query pass on."""
    n = len(R["sq_flags"])
    slots = int(R["sq_seg_count"].max()) if n else 0
    att = torch.ones(n, 3, dtype=torch.float64, device=R.dev)
    pdf, rev = torch.ones_like(att[:, 0]), torch.ones_like(att[:, 0])
    short = R.p["query_beam_type"] == W.SHORT_BEAM
    lite, inside = (R["sq_flags"] & W.Q_LITE) != 0, (R["sq_flags"] & W.Q_ORIGIN_IN_MEDIUM) != 0
    for i in range(slots):
        q = torch.nonzero(R["sq_seg_count"] > i)[:, 0]
        s = R["sq_seg_begin"][q] + i
        med, lo, hi = R["seg_medium"][s], R["seg_dist_min"][s], R["seg_dist_max"][s]
        yield q, med, lo, hi, att[q], pdf[q], rev[q], torch.ones_like(med, dtype=torch.bool) & (inside[q] if i == 0 else False)
        a = R.att(med, hi - lo)
        low = R.least(med, a)
        att_full = R["seg_attenuation"][s] / (R["seg_pdf"][s][:, None] if short else 1.0)
        origin = inside[q] if i == 0 else torch.zeros_like(inside[q])
        rev_lite = torch.where(R.scat[med], torch.where(origin, R.min_st[med] * low, low), 1.0)
        pdf_lite = torch.where(R.scat[med], low, 1.0)
        att[q] = att[q] * torch.where(lite[q][:, None], a, att_full)
        pdf[q] = pdf[q] * torch.where(lite[q], pdf_lite, R["seg_pdf"][s])
        rev[q] = rev[q] * torch.where(lite[q], rev_lite, R["seg_rev_pdf"][s])


def query_camera(R, q, rsr):
    """Camera entries of a segment query's call, entry L-1 with the reverse pdf that the call sets."""
    L, begin = R["sq_path_length"][q], R["sq_cam_mis_begin"][q]

    def at(k):
        m = records_at(R, "cam_mis", begin + k)
        return dict(m, ray_sample_rev_pdf_inv=torch.where(k == L - 1, 1 / rsr, m["ray_sample_rev_pdf_inv"]))
    return L, at


def exact_pb2d(R):
    p, out = R.p, torch.zeros(len(R["sq_flags"]), 3, dtype=torch.float64, device=R.dev)
    mis, short = not p["techniques"] & W.NO_MIS, p["query_beam_type"] == W.SHORT_BEAM
    photon = torch.nonzero((R["lv_flags"] & W.LV_IN_MEDIUM) != 0)[:, 0]
    r2 = p["radius_pb2d"] ** 2
    for q, med, lo, hi, attn, pdf0, rev0, origin in segments(R):
        live = torch.nonzero(R.scat[med] & ((R["sq_flags"][q] & W.Q_PB2D) != 0))[:, 0]
        for rows in live.split(max(1, 40_000_000 // max(1, len(photon)))):
            o, d = R["sq_origin"][q[rows]], R["sq_direction"][q[rows]]
            x = R["lv_position"][photon]
            t = d @ x.T - (o * d).sum(1)[:, None]
            d2 = ((x ** 2).sum(1)[None] - 2 * o @ x.T + (o ** 2).sum(1)[:, None]) - t * t
            a, b = torch.nonzero((t > lo[rows][:, None]) & (t < hi[rows][:, None]) & (d2 < r2 + 1e-9), as_tuple=True)
            row, lv = rows[a], photon[b]
            qi, m, t = q[row], med[row], t[a, b]
            o, d, x = R["sq_origin"][qi], R["sq_direction"][qi], R["lv_position"][lv]
            d2 = ((o + d * t[:, None] - x) ** 2).sum(1)
            keep = d2 <= r2
            att = R.att(m, t - lo[row])
            low = R.least(m, att)
            phase, sin = R.phase(m, (R["lv_dir_fix"][lv] * d).sum(1))
            value = R["lv_throughput"][lv] * R.ss[m] * (att / (low[:, None] if short else 1.0)) \
                * (phase * (1 - d2 / r2) / (r2 * math.pi / 2))[:, None]
            if mis:
                pl = R["lv_path_length"][lv]
                L = R["sq_path_length"][qi]
                keep &= (pl + L <= p["max_path_length"]) & (pl + L >= p["min_path_length"])
                keep &= ~((L == 1) & (t < p["min_dist_to_med"]))
                rsp = R.min_st[m] * low * pdf0[row]
                rsr = torch.where(origin[row], R.min_st[m] * low, low) * rev0[row]
                cand = merged_vertex(R, t, m, R["sq_last_pdf_w_inv"][qi] * t * t / rsp, 1 / rsp)
                beams = R.mfp[m] > p["bb1d_min_mfp"]
                cand["flags"] = torch.where(beams, W.MIS_IN_MEDIUM_WITH_BEAMS, 0)
                has = bool(p["techniques"] & W.BB1D) and len(R["beam_length"]) > 0
                cand["bb1d_beam_selection_pdf"] = torch.full_like(t, 1.0 if has else 0.0)
                last = R.min_st[m] / p["mis_factor_pb2d"] if short else rsp / p["mis_factor_pb2d"]
                lvm = records_at(R, "lv_mis", lv)
                L, at = query_camera(R, qi, rsr)
                cand0 = dict(cand, sin_theta=sin, ray_sample_rev_pdf_inv=lvm["ray_sample_pdf_inv"],
                             ray_sample_rev_pdfs_ratio=lvm["ray_sample_pdfs_ratio"])
                wc = camera_weight(R, L, cand0, at, last, phase * R["lv_cont_prob"][lv] * rsr / (t * t))
                wl = light_weight(R, R["lv_path_idx"][lv], pl, lvm, lambda v: records_at(R, "lv_mis", v), last,
                                  phase * R.cont[m], False)
                value = value / (wl + wc)[:, None]
            out.index_add_(0, qi[keep], (attn[row] * value)[keep])
    return out


def exact_bb1d(R):
    p, out = R.p, torch.zeros(len(R["sq_flags"]), 3, dtype=torch.float64, device=R.dev)
    mis, short = not p["techniques"] & W.NO_MIS, p["query_beam_type"] == W.SHORT_BEAM
    r = p["radius_bb1d"]
    bo, bd, bl = R["beam_origin"], R["beam_direction"], R["beam_length"]
    moment, along = torch.linalg.cross(bd, bo), (bo * bd).sum(1)
    for q, med, lo, hi, attn, pdf0, rev0, origin in segments(R):
        live = torch.nonzero(R.scat[med] & ((R["sq_flags"][q] & W.Q_BB1D) != 0))[:, 0]
        for rows in live.split(max(1, 40_000_000 // max(1, len(bl)))):
            o, d = R["sq_origin"][q[rows]], R["sq_direction"][q[rows]]
            # the lines' distance from their Pluecker coordinates
            b = d @ bd.T
            ad = d @ moment.T + torch.linalg.cross(d, o) @ bd.T
            i, j = torch.nonzero((ad ** 2 < r * r * (1 - b * b) + 1e-9) &
                                 (med[rows][:, None] == R["beam_medium_id"][None]), as_tuple=True)
            row = rows[i]
            qi, m = q[row], med[row]
            o, d, o2, e = R["sq_origin"][qi], R["sq_direction"][qi], bo[j], bd[j]
            c = torch.linalg.cross(d, e)
            s2, b, w = (c * c).sum(1), (d * e).sum(1), o - o2
            den = (d * d).sum(1) * (e * e).sum(1) - b * b
            dw, ew = (d * w).sum(1), (e * w).sum(1)
            t1, t2 = (b * ew - (e * e).sum(1) * dw) / den, ((d * d).sum(1) * ew - b * dw) / den
            sin = s2.sqrt()
            dist = (w * c).sum(1).abs() / sin
            keep = (dist <= r) & (t1 > lo[row]) & (t1 < hi[row]) & (t2 > 0) & (t2 < bl[j]) & (den > 1e-5)
            row, qi, m, j, t1, t2, sin, dist, b = (v[keep] for v in (row, qi, m, j, t1, t2, sin, dist, b))
            bshort = (R["beam_flags"][j] & W.SHORT_BEAM) != 0
            qa, ba = R.att(m, t1 - lo[row]), R.att(m, t2)
            ql, bl_ = R.least(m, qa), R.least(m, ba)
            att = qa * ba / (ql[:, None] if short else 1.0) / torch.where(bshort, bl_, 1.0)[:, None]
            phase, _ = R.phase(m, -b)
            value = R["beam_throughput"][j] * R.ss[m] * att * (phase * (1 - dist ** 2 / r ** 2) * 3 / (4 * r * sin))[:, None]
            ok = torch.ones_like(bshort)
            if mis:
                v = R["beam_light_vertex"][j]
                pl, L = R["lv_path_length"][v], R["sq_path_length"][qi]
                ok &= (pl + 1 + L <= p["max_path_length"]) & (pl + 1 + L >= p["min_path_length"])
                ok &= ~((L == 1) & (t1 < p["min_dist_to_med"]))
                st = R.min_st[m]
                rsq, rrq = st * ql * pdf0[row], torch.where(origin[row], st * ql, ql) * rev0[row]
                inside = (R["beam_ray_sampling_flags"][j] & W.ORIGIN_IN_MEDIUM) != 0
                rsb = st * bl_ * R["beam_ray_sample_pdf"][j]
                rrb = torch.where(inside, st * bl_, bl_) * R["beam_ray_sample_rev_pdf"][j]
                cand = merged_vertex(R, t1, m, R["sq_last_pdf_w_inv"][qi] * t1 * t1 / rsq, 1 / rsq)
                finite = (R["lv_flags"][v] & W.LV_IS_FINITE) != 0
                d2b = torch.where(finite, t2 * t2, 1.0)
                brec = merged_vertex(R, t1, m, R["beam_last_pdf_w_inv"][j] * d2b / rsb, 1 / rsb)
                last = (st if short else rsq) * torch.where(bshort, st, rsb) / (p["mis_factor_bb1d"] * sin)
                lvm = records_at(R, "lv_mis", v)
                delta = W.MIS_ON_LIGHT_SOURCE | W.MIS_IS_DELTA
                ntl = torch.where((lvm["flags"] & delta) == delta, 0.0,
                                  phase * R.cont[m] * rrb * lvm["cos_theta_out"].abs() / d2b)
                L, at = query_camera(R, qi, rrq)
                cand0 = dict(cand, sin_theta=sin, ray_sample_rev_pdf_inv=1 / rsb, ray_sample_rev_pdfs_ratio=1 / st)
                wc = camera_weight(R, L, cand0, at, last, phase * R.cont[m] * rrq / (t1 * t1))

                def lights(k):
                    rec = records_at(R, "lv_mis", k)
                    return dict(rec, ray_sample_rev_pdf_inv=torch.where(k == v, 1 / rrb, rec["ray_sample_rev_pdf_inv"]))
                wl = light_weight(R, R["lv_path_idx"][v], pl + 1, brec, lights, last, ntl, True)
                value = value / (wl + wc)[:, None]
            out.index_add_(0, qi[ok], (attn[row] * value)[ok])
    return out


def exact_pp3d(R):
    p, out = R.p, torch.zeros(len(R["pq_pixel"]), 3, dtype=torch.float64, device=R.dev)
    photon = torch.nonzero((R["lv_flags"] & W.LV_IN_MEDIUM) != 0)[:, 0]
    if not len(photon) or not p["techniques"] & W.PP3D:
        return out
    r, cells = p["radius_pp3d"], max(1, p["hash_cells"])
    x32 = R["lv_position"][photon].float()
    low, high = x32.min(0).values, x32.max(0).values
    inv = torch.tensor(1.0, dtype=torch.float32) / (torch.tensor(r, dtype=torch.float32) * 2)
    inv = inv.to(R.dev)

    def bucket(c):  # the reference's hash of an integer cell
        c = c.long() & 0xffffffff
        h = [(c[..., k] * f) & 0xffffffff for k, f in enumerate((73856093, 19349663, 83492791))]
        return (h[0] ^ h[1] ^ h[2]) % cells
    home = bucket(torch.floor(inv * (x32 - low)))
    for rows in torch.arange(len(R["pq_pixel"]), device=R.dev).split(max(1, 40_000_000 // len(photon))):
        x = R["pq_position"][rows]
        i, j = torch.nonzero(torch.cdist(x, R["lv_position"][photon],
                                         compute_mode="donot_use_mm_for_euclid_dist") <= r, as_tuple=True)
        q, lv = rows[i], photon[j]
        x32q = R["pq_position"][q].float()
        cell = inv * (x32q - low)
        base = torch.floor(cell)
        step = torch.where(cell - base < 0.5, -1.0, 1.0)
        times = torch.zeros_like(q)  # a photon counts once for each of the eight cells with its bucket
        for k in range(8):
            pick = torch.tensor([k >> 2 & 1, k >> 1 & 1, k & 1], dtype=torch.float32, device=R.dev)
            times += bucket(base + pick * step) == home[j]
        times *= ((x32q >= low) & (x32q <= high)).all(1)
        m, L = R["pq_medium_id"][q], R["pq_path_length"][q]
        pl = R["lv_path_length"][lv]
        ok = ((R["lv_flags"][lv] & W.LV_CONNECTABLE) != 0) & (pl + L <= p["max_path_length"]) & \
            (pl + L >= p["min_path_length"])
        phase, sin = R.phase(m, -(R["lv_dir_fix"][lv] * R["pq_dir_fix"][q]).sum(1))
        lvm = records_at(R, "lv_mis", lv)
        last = 1 / lvm["pp3d_factor"]
        begin = R["pq_cam_mis_begin"][q]
        first = dict(records_at(R, "cam_mis", begin + L), sin_theta=sin,
                     ray_sample_rev_pdf_inv=lvm["ray_sample_pdf_inv"],
                     ray_sample_rev_pdfs_ratio=lvm["ray_sample_pdfs_ratio"])
        wc = camera_weight(R, L, first, lambda k: records_at(R, "cam_mis", begin + k), last,
                           phase * R["lv_cont_prob"][lv])
        wl = light_weight(R, R["lv_path_idx"][lv], pl, lvm, lambda v: records_at(R, "lv_mis", v), last,
                          phase * R.cont[m], False)
        value = R["lv_throughput"][lv] * R.ss[m] * (phase * times / (wl + wc))[:, None]
        out.index_add_(0, q[ok], value[ok])
    return out


def exact_bp2d(R):
    """Photon beams at the camera vertices with a 2-D kernel, MIS weight 1."""
    p, out = R.p, torch.zeros(len(R["pq_pixel"]), 3, dtype=torch.float64, device=R.dev)
    r2, bo, bd, bl = p["radius_bb1d"] ** 2, R["beam_origin"], R["beam_direction"], R["beam_length"]
    for q in torch.arange(len(out), device=R.dev).split(max(1, 40_000_000 // max(1, len(bl)))):
        x, m = R["pq_position"][q], R["pq_medium_id"][q]
        t = x @ bd.T - (bo * bd).sum(1)[None]
        d2 = (x ** 2).sum(1)[:, None] - 2 * x @ bo.T + (bo ** 2).sum(1)[None] - t * t
        i, j = torch.nonzero((t > 0) & (t < bl[None]) & (d2 < r2 + 1e-9) & (m[:, None] == R["beam_medium_id"][None]),
                             as_tuple=True)
        x, m, t = x[i], m[i], t[i, j]
        d2 = ((bo[j] + bd[j] * t[:, None] - x) ** 2).sum(1)
        att = R.att(m, t)
        free = torch.where((R["beam_flags"][j] & W.SHORT_BEAM) != 0, R.least(m, att), 1.0)
        phase, _ = R.phase(m, (R["pq_dir_fix"][q[i]] * bd[j]).sum(1))
        value = R["beam_throughput"][j] * R.ss[m] * att * (phase / free * (1 - d2 / r2) / (r2 * math.pi / 2))[:, None]
        keep = (d2 <= r2) & R.scat[m]
        out.index_add_(0, q[i][keep], value[keep])
    return out


def exact(c, seed):
    """The pass in 64 bits: image and per-call results where every pair can be tested, None elsewhere.
    Counts have no such value, nor has a gradient, a KNN radius or a walk over the reference's grid."""
    if c["kind"] not in ("host", "noalloc", "stage") or c["scene"] == "stress" or c["knn_photons"] or c["knn_beams"]:
        return None
    if c["grid_res"] or c["width"] * c["height"] * c["light_paths"] > 4e9:
        return None
    R = Records(host_records(c, seed))
    p = R.p

    def room(v):
        return torch.cat([v, torch.zeros(calls(c) - len(v), 3, dtype=v.dtype, device=v.device)])
    if c["kind"] == "noalloc":
        return {"pp3d": room(exact_pp3d(R))}
    pb2d, bb1d, pp3d = exact_pb2d(R), exact_bb1d(R), exact_pp3d(R)
    points = exact_bp2d(R) * p["norm_bb1d"] if c["bp2d"] else pp3d * p["norm_pp3d"]
    image = torch.zeros(p["image_width"] * p["image_height"], 3, dtype=torch.float64, device=R.dev)
    image.index_add_(0, R["sq_pixel"], R["sq_throughput"] * (p["norm_pb2d"] * pb2d + p["norm_bb1d"] * bb1d))
    if len(points):
        image.index_add_(0, R["pq_pixel"], R["pq_throughput"] * points)
    if c["kind"] == "stage":
        return {"image": image}
    return {"pb2d": room(pb2d), "bb1d": room(bb1d), "pp3d": room(pp3d), "image": image, "counts": None}
