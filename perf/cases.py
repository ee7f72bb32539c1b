"""The calls that programs make of this library, over the sizes they make them at.

A case is a dict of plain values; its "kind" says which program it stands for:

  tile     one panel step of a caller's own tile driver through tile_kernel.h
           (dgeqrt, dlarft, dlarfb, dtsqrt, dlarft, dssrfb) on device tiles
  qr       factorization and explicit Q of a square matrix resident on the GPU
  tall     factorization of a tall matrix and Q^T applied to right-hand sides
  ragged   a column-major matrix of any size: padded into tiles, factored, Q^T
           applied, R and Q^T b converted back
  dropin   the reference's main program: host arrays through Hybrid_tile_QR,
           Hybrid_make_Q and the Hybrid_dgemm check
  lstsq    least squares for several right-hand sides, refined in FP64
  apply    Q^T C and Q C with the reflectors of a factorization kept on its plan
  batch    one launch over many small matrices of uneven shapes, and Q^T c
"""
import ctypes
import math
import random

import numpy as np
import torch

import hybrid3_gb300 as H

F64 = torch.float64
PRECISION = {"fp64": H.HQR_PREC_FP64, "split": H.HQR_PREC_OZAKI, "fast": H.HQR_PREC_OZAKI_FAST,
             "fp32": H.HQR_PREC_FP32}


def listed():
    return [
        # a caller's own tile driver at the tile order of the split updates: the smallest call, and latency
        {"name": "tile_step_128", "kind": "tile", "nb": 128, "ib": 32},
        # a small square QR + Q, FP64: launches and latency
        {"name": "qr_fp64_256", "kind": "qr", "n": 256, "nb": 64, "ib": 16, "precision": "fp64"},
        # sizes that are multiples of nothing, column-major in and out
        {"name": "ragged_fp64_1000x615", "kind": "ragged", "m": 1000, "n": 615, "nrhs": 5, "nb": 96, "ib": 32,
         "precision": "fp64"},
        # the reference's main program on its CPU workload's size (n = 2048, NB 256, IB 32), host arrays
        {"name": "dropin_2048", "kind": "dropin", "n": 2048, "nb": 256, "ib": 32, "pinned": True},
        # plain FP64 on the GPU at the tile order of the FP64 workload
        {"name": "qr_fp64_4096", "kind": "qr", "n": 4096, "nb": 256, "ib": 32, "precision": "fp64"},
        # split precision where the panel chain, not the update work, sets the pace
        {"name": "qr_split_3072", "kind": "qr", "n": 3072, "nb": 128, "ib": 32, "precision": "split"},
        # the headline workload: split precision, n = 16384
        {"name": "qr_split_16384", "kind": "qr", "n": 16384, "nb": 128, "ib": 32, "precision": "split"},
        # tall and skinny, domain tree, a few right-hand sides
        {"name": "tall_split_32768x2048", "kind": "tall", "m": 32768, "n": 2048, "nb": 128, "ib": 32, "tree": 32,
         "ct": 1, "precision": "split"},
        # the least-squares workload: FP32-class factorization, augmented-system refinement, 16 right-hand sides
        {"name": "lstsq_fp32_32768x8192", "kind": "lstsq", "m": 32768, "n": 8192, "nrhs": 16, "kappa": 1e3,
         "precision": "fp32", "augmented": True, "steps": 2},
        # ill-conditioned least squares at FP64 level, one plain refinement step
        {"name": "lstsq_split_12288x3072", "kind": "lstsq", "m": 12288, "n": 3072, "nrhs": 16, "kappa": 1e6,
         "precision": "split", "augmented": False, "steps": 1},
        # Q applied in both directions with the kept reflectors (a Krylov or projection loop's inner call)
        {"name": "apply_split_8192x512", "kind": "apply", "n": 8192, "nb": 128, "ib": 32, "ct": 4,
         "precision": "split"},
        # many uneven matrices in one launch, the batched workload's shapes
        {"name": "batch_256", "kind": "batch", "count": 256, "mmax": 2048, "shape_seed": 20151130, "nrhs": 4,
         "nb": 96, "ib": 16},
    ]


def log_between(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def multiple(x, q):
    return max(q, int(round(x / q)) * q)


def draw(rng):
    kind = rng.choice(["tile", "qr", "qr", "qr", "tall", "ragged", "ragged", "dropin", "lstsq", "lstsq", "apply",
                       "batch"])
    if kind == "tile":
        nb = int(log_between(rng, 24, 256))
        return {"kind": kind, "nb": nb, "ib": rng.choice([8, 16, 32, max(8, nb // 3)])}
    if kind == "qr":
        if rng.random() < 0.5:
            nb, ib = rng.choice([(64, 16), (96, 16), (96, 32), (128, 32), (192, 32), (256, 32), (256, 64)])
            return {"kind": kind, "n": multiple(log_between(rng, 256, 4096), nb), "nb": nb, "ib": ib,
                    "precision": "fp64"}
        return {"kind": kind, "n": multiple(log_between(rng, 512, 12288), 128), "nb": 128,
                "ib": rng.choice([16, 32]), "precision": "split"}
    if kind == "tall":
        n = multiple(log_between(rng, 512, 4096), 128)
        split = rng.random() < 0.7
        rows = log_between(rng, 4, 24) * n
        m = multiple(min(rows, 65536 if split else 2.5e11 / (2.0 * n * n)), 128)
        return {"kind": kind, "m": max(m, n), "n": n, "nb": 128, "ib": 32, "tree": rng.choice([0, 8, 16, 32]),
                "ct": rng.choice([1, 1, 2]), "precision": "split" if split else "fp64"}
    if kind == "ragged":
        n = int(log_between(rng, 30, 1500))
        nb, ib = rng.choice([(64, 16), (64, 32), (96, 32), (128, 16), (128, 32)])
        return {"kind": kind, "m": int(n * log_between(rng, 1, 6)), "n": n, "nrhs": rng.choice([1, 3, 5, 16, 33]),
                "nb": nb, "ib": ib, "precision": "split" if nb == 128 and rng.random() < 0.5 else "fp64"}
    if kind == "dropin":
        nb, ib = rng.choice([(64, 16), (128, 32), (256, 32)])
        return {"kind": kind, "n": multiple(log_between(rng, 256, 3072), nb), "nb": nb, "ib": ib,
                "pinned": rng.random() < 0.5}
    if kind == "lstsq":
        n = multiple(log_between(rng, 256, 6144), 128)
        m = max(n, multiple(min(n * log_between(rng, 1.5, 8), 32768), 128))
        p = rng.choice(["split", "fast", "fp32"])
        return {"kind": kind, "m": m, "n": n, "nrhs": rng.choice([1, 4, 16, 16, 40]),
                "kappa": rng.choice([1e2, 1e3]) if p != "split" else rng.choice([1e3, 1e5]), "precision": p,
                "augmented": p != "split", "steps": 3 if p != "split" else 1}
    if kind == "apply":
        return {"kind": kind, "n": multiple(log_between(rng, 512, 8192), 128), "nb": 128, "ib": 32,
                "ct": rng.choice([1, 2, 4, 8]), "precision": rng.choice(["split", "split", "split", "fp64"])}
    nb, ib = rng.choice([(64, 16), (96, 16), (128, 16)])
    mmax = 32 * int(log_between(rng, 6, 64))
    return {"kind": kind, "count": int(log_between(rng, 32, 1e6 / mmax if mmax < 2000 else 400)), "mmax": mmax,
            "shape_seed": rng.randrange(1 << 20), "nrhs": rng.choice([1, 4, 16]), "nb": nb, "ib": ib}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def up(x, q):
    return -(-x // q) * q


def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (int(seed) + 1))
    return g


def uniform(g, *shape):
    """i.i.d. uniform[-1, 1): the workloads' entries, in whatever layout."""
    return torch.rand(*shape, dtype=F64, device="cuda", generator=g).mul_(2.0).sub_(1.0)


def to_tiles(A, nb):
    m, n = A.shape
    return A.reshape(m // nb, nb, n // nb, nb).permute(2, 0, 3, 1).contiguous().reshape(-1)


def from_tiles(t, m, n, nb):
    return t.reshape(n // nb, m // nb, nb, nb).permute(1, 3, 0, 2).reshape(m, n)


def haar(g, n):
    q, r = torch.linalg.qr(torch.randn(n, n, dtype=F64, device="cuda", generator=g))
    return q * torch.sign(torch.diagonal(r))


def conditioned(g, m, n, kappa):
    """m x n (n a multiple of 128): a uniform matrix with columns scaled geometrically to 1/kappa, mixed by a
    dense orthogonal matrix (a Kronecker product of two Haar factors: cheap to apply)."""
    A = uniform(g, m, n)
    A *= kappa ** (-torch.arange(n, dtype=F64, device="cuda") / max(n - 1, 1))
    A = (A.reshape(m * (n // 128), 128) @ haar(g, 128)).reshape(m, n // 128, 128)
    return torch.einsum("kab,ac->kcb", A, haar(g, n // 128)).reshape(m, n).contiguous()


def batch_shapes(case):
    """The batched workload's shapes: m in {64 .. mmax} step 32, n in {32 .. m} step 32."""
    r = random.Random(case["shape_seed"])
    m = [32 * r.randint(2, case["mmax"] // 32) for _ in range(case["count"])]
    return m, [32 * r.randint(1, x // 32) for x in m]


class PageLocked:
    """n doubles of the library's page-locked host memory; an array made of it keeps it alive."""

    def __init__(self, n):
        self.p = ctypes.c_void_p()
        H.check(H.lib().hqr_host_alloc(ctypes.byref(self.p), 8 * n), "hqr_host_alloc")
        self.__array_interface__ = {"shape": (n,), "typestr": "<f8", "data": (self.p.value, False), "version": 3}

    def __del__(self):
        if self.p:
            H.lib().hqr_host_free(self.p)


def host_array(n, pinned):
    a = np.asarray(PageLocked(n)) if pinned else np.empty(n)
    a[:] = 0.0
    return a


def inputs(case, seed):
    """The inputs that prepare() and exact() share, made from the seed alone."""
    g = generator(seed)
    k = case["kind"]
    if k == "tile":
        nb = case["nb"]
        return {x: uniform(g, nb, nb) for x in ("a11", "a12", "a21", "a22")}   # [column][row]
    if k in ("qr", "dropin"):
        return {"a": uniform(g, case["n"] * case["n"])}
    if k == "tall":
        return {"a": uniform(g, case["m"] * case["n"]), "c": uniform(g, case["m"] * case["ct"] * case["nb"])}
    if k == "ragged":
        return {"a": uniform(g, case["n"], case["m"]), "b": uniform(g, case["nrhs"], case["m"])}   # column-major
    if k == "lstsq":
        A = conditioned(g, case["m"], case["n"], case["kappa"])
        x = torch.randn(case["n"], case["nrhs"], dtype=F64, device="cuda", generator=g)
        b = A @ x + 1e-4 * torch.randn(case["m"], case["nrhs"], dtype=F64, device="cuda", generator=g)
        return {"a2d": A, "b": b.t().contiguous()}
    if k == "apply":
        return {"a": uniform(g, case["n"] * case["n"]), "c": uniform(g, case["n"] * case["ct"] * case["nb"])}
    m, n = batch_shapes(case)
    nb = case["nb"]
    # every matrix zero-padded to whole tiles, one after the other
    a, c, where, oa, oc = [], [], [], 0, 0
    for i in range(len(m)):
        mp, np_, cw = up(m[i], nb), up(n[i], nb), up(case["nrhs"], nb)
        A = torch.zeros(mp, np_, dtype=F64, device="cuda")
        A[:m[i], :n[i]] = uniform(g, m[i], n[i])
        C = torch.zeros(mp, cw, dtype=F64, device="cuda")
        C[:m[i], :case["nrhs"]] = uniform(g, m[i], case["nrhs"])
        a.append(to_tiles(A, nb))
        c.append(to_tiles(C, nb))
        where.append((mp, np_, oa, oc))
        oa += mp * np_
        oc += mp * cw
    return {"a": torch.cat(a), "c": torch.cat(c), "where": where}


# ---------------------------------------------------------------------------
# What a program has in hand before the call
# ---------------------------------------------------------------------------
def prepare(case, seed):
    H.lib().hqr_set_error_mode(H.HQR_ERRORS_RETURN)
    k, s = case["kind"], {"case": case}
    x = inputs(case, seed)
    new = lambda n: torch.zeros(n, dtype=F64, device="cuda")   # noqa: E731
    if k == "tile":
        nb = case["nb"]
        s.update(x, w={key: torch.empty_like(v) for key, v in x.items()}, tau=new(nb), tau2=new(nb), y=new(nb * nb),
                 **{t: new(nb * nb) for t in ("t1", "t2", "t3", "t4")})
    elif k == "qr":
        n, nb = case["n"], case["nb"]
        s.update(x, plan=H.Plan(n, n, nb, case["ib"], PRECISION[case["precision"]]), w=torch.empty_like(x["a"]),
                 tau=new((n // nb) ** 2 * nb), q=new(n * n))
    elif k == "tall":
        m, n, nb = case["m"], case["n"], case["nb"]
        s.update(x, plan=H.Plan(m, n, nb, case["ib"], PRECISION[case["precision"]]), w=torch.empty_like(x["a"]),
                 cw=torch.empty_like(x["c"]), tau=new((m // nb) * (n // nb) * nb))
        if case["tree"]:
            s["plan"].set_tree(case["tree"])
    elif k == "ragged":
        nb, ct = case["nb"], up(case["nrhs"], case["nb"]) // case["nb"]
        mp, np_ = up(case["m"], nb), up(case["n"], nb)
        s.update(x, plan=H.Plan(mp, np_, nb, case["ib"], PRECISION[case["precision"]]), w=new(mp * np_),
                 cw=new(mp * ct * nb), tau=new((mp // nb) * (np_ // nb) * nb), r=new(case["n"] * case["m"]),
                 qtb=new(case["nrhs"] * case["m"]), mp=mp, np=np_, ct=ct)
    elif k == "dropin":
        n, nb = case["n"], case["nb"]
        s["status"] = H.status(n, n, nb)
        s["a"] = x["a"].cpu().numpy()
        for key, size in (("ry", n * n), ("tau", (n // nb) ** 2 * nb), ("q", n * n), ("qr", n * n)):
            s[key] = host_array(size, case["pinned"])
    elif k == "lstsq":
        m, n = case["m"], case["n"]
        s.update(plan=H.Plan(m, n, 128, 32, PRECISION[case["precision"]]), a=to_tiles(x["a2d"], 128), b=x["b"],
                 x=new(case["nrhs"] * n).reshape(case["nrhs"], n))
    elif k == "apply":
        n, nb = case["n"], case["nb"]
        s.update(plan=H.Plan(n, n, nb, case["ib"], PRECISION[case["precision"]]), ry=x["a"], c=x["c"],
                 tau=new((n // nb) ** 2 * nb), qtc=torch.empty_like(x["c"]), back=torch.empty_like(x["c"]))
        H.check(H.lib().hqr_geqrf(s["plan"].h, s["ry"].data_ptr(), s["tau"].data_ptr(), None), "hqr_geqrf")
    else:
        nb, where = case["nb"], x["where"]
        s.update(a=x["a"], c=x["c"], w=torch.empty_like(x["a"]), cw=torch.empty_like(x["c"]))
        s["batch"] = H.Batch([t[0] for t in where], [t[1] for t in where], [nb] * len(where),
                             [case["ib"]] * len(where), max_nrhs=case["nrhs"])
        ot, tau_at = 0, []
        for mp, np_, _, _ in where:
            tau_at.append(ot)
            ot += (mp // nb) * (np_ // nb) * nb
        s["tau"] = new(ot)
        s["pa"] = [s["w"].data_ptr() + 8 * t[2] for t in where]
        s["pc"] = [s["cw"].data_ptr() + 8 * t[3] for t in where]
        s["pt"] = [s["tau"].data_ptr() + 8 * o for o in tau_at]
        # the right-hand sides' places in the tile grids: what a program reads of Q^T C
        at = []
        for mp, _, _, oc in where:
            for col in range(case["nrhs"]):
                tile = oc + torch.arange(mp // nb) * nb * nb + (col // nb) * mp * nb + (col % nb) * nb
                at.append((tile[:, None] + torch.arange(nb)[None, :]).reshape(-1))
        s["at"] = torch.cat(at).cuda()
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    L, case = H.lib(), s["case"]
    k = case["kind"]
    if k == "tile":
        nb, ib, w = case["nb"], case["ib"], s["w"]
        for key in w:
            w[key].copy_(s[key])
        torch.cuda.current_stream().synchronize()   # the tile calls run on a stream of their own
        a11, a12, a21, a22 = (w[key].data_ptr() for key in ("a11", "a12", "a21", "a22"))
        tau, tau2, y, t1, t2, t3, t4 = (s[key].data_ptr() for key in ("tau", "tau2", "y", "t1", "t2", "t3", "t4"))
        L.tile_dgeqrt(nb, nb, ib, a11, nb, tau, y, t1, nb, None)
        L.tile_dlarft(nb, nb, 1, y, nb, tau, t2, nb, None)
        L.tile_dlarfb(nb, nb, a12, nb, y, t2, nb, None)
        L.tile_dtsqrt(nb, nb, ib, a11, nb, a21, nb, tau2, t3, nb, None)
        L.tile_dlarft(nb, nb, 1, a21, nb, tau2, t4, nb, None)
        L.tile_dssrfb(nb, nb, a12, a22, nb, a21, t4, nb, None)
        H.check(L.hqr_last_error(), "tile kernels")
        return {"a11": w["a11"], "a12": w["a12"], "a21": w["a21"], "a22": w["a22"], "tau": s["tau"],
                "tau2": s["tau2"], "y": s["y"], "t2": s["t2"], "t4": s["t4"]}
    if k == "qr":
        s["w"].copy_(s["a"])
        h, w, tau, q = s["plan"].h, s["w"].data_ptr(), s["tau"].data_ptr(), s["q"].data_ptr()
        H.check(L.hqr_geqrf(h, w, tau, None), "hqr_geqrf")
        H.check(L.hqr_make_q(h, q, w, tau, 1, None), "hqr_make_q")
        return {"q": s["q"], "r": s["w"], "tau": s["tau"]}
    if k == "tall":
        s["w"].copy_(s["a"])
        s["cw"].copy_(s["c"])
        h, w, tau = s["plan"].h, s["w"].data_ptr(), s["tau"].data_ptr()
        H.check(L.hqr_geqrf(h, w, tau, None), "hqr_geqrf")
        H.check(L.hqr_ormqr_t(h, w, tau, s["cw"].data_ptr(), case["ct"], 1, None), "hqr_ormqr_t")
        return {"ry": s["w"], "tau": s["tau"], "qtc": s["cw"]}
    if k == "ragged":
        m, n, nrhs, nb = case["m"], case["n"], case["nrhs"], case["nb"]
        h, w, c, tau = s["plan"].h, s["w"].data_ptr(), s["cw"].data_ptr(), s["tau"].data_ptr()
        H.check(L.hqr_colmajor_to_tiles_padded(m, n, m, nb, s["a"].data_ptr(), w, None), "to tiles")
        H.check(L.hqr_colmajor_to_tiles_padded(m, nrhs, m, nb, s["b"].data_ptr(), c, None), "to tiles")
        H.check(L.hqr_geqrf(h, w, tau, None), "hqr_geqrf")
        H.check(L.hqr_ormqr_t(h, w, tau, c, s["ct"], 1, None), "hqr_ormqr_t")
        H.check(L.hqr_tiles_to_colmajor_padded(m, n, m, nb, w, s["r"].data_ptr(), None), "from tiles")
        H.check(L.hqr_tiles_to_colmajor_padded(m, nrhs, m, nb, c, s["qtb"].data_ptr(), None), "from tiles")
        return {"ry": s["r"], "tau": s["tau"], "qtb": s["qtb"]}
    if k == "dropin":
        dp = ctypes.POINTER(ctypes.c_double)
        ry, tau, q, qr = (s[key].ctypes.data_as(dp) for key in ("ry", "tau", "q", "qr"))
        st = ctypes.byref(s["status"])
        s["ry"][:] = s["a"]
        s["q"][:] = 0.0   # the caller's part of Hybrid_make_Q
        L.Hybrid_tile_QR(st, ry, tau, 0, 1, case["ib"])
        H.check(L.hqr_last_error(), "Hybrid_tile_QR")
        L.Hybrid_make_Q(st, q, ry, tau, 0, 1, case["ib"])
        H.check(L.hqr_last_error(), "Hybrid_make_Q")
        L.Hybrid_dgemm(st, q, ry, qr, 0, 1)
        H.check(L.hqr_last_error(), "Hybrid_dgemm")
        return {"q": s["q"], "r": s["ry"], "tau": s["tau"], "qr": s["qr"]}
    if k == "lstsq":
        res = s["plan"].lstsq(s["a"].data_ptr(), s["b"].data_ptr(), case["nrhs"], s["x"].data_ptr(),
                              refine_steps=case["steps"], augmented=case["augmented"])
        return {"x": s["x"], "residual": np.array(res)}
    if k == "apply":
        h, ry, tau, ct = s["plan"].h, s["ry"].data_ptr(), s["tau"].data_ptr(), case["ct"]
        s["qtc"].copy_(s["c"])
        H.check(L.hqr_ormqr_t(h, ry, tau, s["qtc"].data_ptr(), ct, 1, None), "hqr_ormqr_t")
        s["back"].copy_(s["qtc"])
        H.check(L.hqr_ormqr_n(h, ry, tau, s["back"].data_ptr(), ct, 1, None), "hqr_ormqr_n")
        return {"qtc": s["qtc"], "c": s["back"]}
    s["w"].copy_(s["a"])
    s["cw"].copy_(s["c"])
    s["batch"].geqrf(s["pa"], s["pt"], wait=False)
    s["batch"].ormqr_t(s["pa"], s["pt"], s["pc"], case["nrhs"], wait=False)
    s["batch"].status()
    return {"ry": s["w"], "tau": s["tau"], "qtc": s["cw"][s["at"]]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    k = case["kind"]
    qr = lambda m, n: 2.0 * m * n * n - 2.0 * n ** 3 / 3.0           # noqa: E731
    apply_ = lambda m, n, c: 4.0 * m * n * c - 2.0 * n * n * c       # noqa: E731  Q^T C or Q C, C m x c
    if k == "tile":
        nb = case["nb"]
        # QR of a tile, T, its application, QR of the pair, T, its application
        return {"bytes": 8.0 * (8 * nb * nb + 3 * nb * nb), "flops": (4 / 3 + 2 / 3 + 3 + 2 + 2 / 3 + 5) * nb ** 3}
    if k == "qr":
        n = case["n"]
        return {"bytes": 24.0 * n * n, "flops": 8.0 / 3 * n ** 3}
    if k == "dropin":
        n = case["n"]
        return {"bytes": 40.0 * n * n, "flops": 8.0 / 3 * n ** 3 + 2.0 * n ** 3}
    if k in ("tall", "ragged"):
        m, n = case["m"], case["n"]
        c = case["ct"] * case["nb"] if k == "tall" else case["nrhs"]
        mn = min(m, n)
        return {"bytes": 16.0 * m * (n + c), "flops": qr(max(m, n), mn) + apply_(m, mn, c)}
    if k == "lstsq":
        m, n, c = case["m"], case["n"], case["nrhs"]
        step = 4.0 * m * n * c * (2 if case["augmented"] else 1)     # products with A and applications of Q
        return {"bytes": 8.0 * (m * n + (m + n) * c), "flops": qr(m, n) + apply_(m, n, c) + case["steps"] * step}
    if k == "apply":
        n, c = case["n"], case["ct"] * case["nb"]
        return {"bytes": 8.0 * (n * n + 3.0 * n * c), "flops": 2 * apply_(n, n, c)}
    m, n = batch_shapes(case)
    c = case["nrhs"]
    return {"bytes": sum(16.0 * a * (b + c) for a, b in zip(m, n)),
            "flops": sum(qr(a, b) + apply_(a, b, c) for a, b in zip(m, n))}


# ---------------------------------------------------------------------------
# The same in plain torch and numpy, 64 bits
# ---------------------------------------------------------------------------
def tile_householder(A, nb):
    """The flat-tree tile QR of A (whole tiles), LAPACK reflectors: A is overwritten by R above the diagonal and
    the reflectors below it; returns the TAU array of the tile layout and the list of block reflectors."""
    mt, nt = A.shape[0] // nb, A.shape[1] // nb
    tau = torch.zeros(nt, mt, nb, dtype=F64, device=A.device)
    blocks = []
    for i in range(min(mt, nt)):
        ri, ci = slice(i * nb, (i + 1) * nb), slice(i * nb, (i + 1) * nb)
        for k in range(i, mt):
            rk = slice(k * nb, (k + 1) * nb)
            if k == i:
                f, t = torch.geqrf(A[ri, ci].contiguous())
                A[ri, ci] = f
            else:
                top = A[ri, ci].clone()
                f, t = torch.geqrf(torch.cat([torch.triu(top), A[rk, ci]]))
                A[ri, ci] = torch.triu(f[:nb]) + torch.tril(top, -1)
                A[rk, ci] = f[nb:]
            tau[i, k] = t
            blocks.append((ri, rk, f, t))
            if i + 1 < nt:
                apply_block(A[:, (i + 1) * nb:], blocks[-1])
    return tau.reshape(-1), blocks


def apply_block(C, block):
    ri, rk, f, t = block
    if ri == rk:
        C[ri] = torch.ormqr(f, t, C[ri].contiguous(), transpose=True)
    else:
        both = torch.ormqr(f, t, torch.cat([C[ri], C[rk]]), transpose=True)
        n = ri.stop - ri.start
        C[ri], C[rk] = both[:n], both[n:]


def tile_reference(x, nb, ib):
    """tile_kernel.h's conventions (beta = +||x||, T lower), unblocked, in numpy."""
    a11, a12, a21, a22 = (x[key].cpu().numpy().T.copy() for key in ("a11", "a12", "a21", "a22"))
    tau, tau2, y = np.zeros(nb), np.zeros(nb), np.zeros((nb, nb))
    for i in range(nb - 1):
        col = a11[i:, i].copy()
        beta = np.linalg.norm(col)
        head = col[0] - beta
        v = col / head
        v[0] = 1.0
        tau[i] = 2.0 * head * head / (head * head + col[1:] @ col[1:])
        a11[i:, i + 1:] -= tau[i] * np.outer(v, v @ a11[i:, i + 1:])
        a11[i, i], a11[i + 1:, i], y[i:, i] = beta, v[1:], v

    def lower_t(y, tau):
        t, g = np.diag(tau), y.T @ y
        for i in range(1, nb):
            t[i, :i] = -tau[i] * (t[:i, :i].T @ g[:i, i])
        return t

    t2 = lower_t(y, tau)
    a12 -= y @ (t2 @ (y.T @ a12))
    for i in range(nb):
        col = a21[:, i].copy()
        beta = math.hypot(a11[i, i], np.linalg.norm(col))
        head = a11[i, i] - beta
        v = col / head
        tau2[i] = 2.0 * head * head / (head * head + col @ col)
        d = tau2[i] * (a11[i, i + 1:] + v @ a21[:, i + 1:])
        a11[i, i + 1:] -= d
        a21[:, i + 1:] -= np.outer(v, d)
        a11[i, i], a21[:, i] = beta, v
    t4 = lower_t(a21, tau2)
    d = t4 @ (a12 + a21.T @ a22)
    a12 -= d
    a22 -= a21 @ d
    f = lambda z: np.ascontiguousarray(z.T)   # noqa: E731
    return {"a11": f(a11), "a12": f(a12), "a21": f(a21), "a22": f(a22), "tau": tau, "tau2": tau2,
            "y": f(y).reshape(-1), "t2": f(t2).reshape(-1), "t4": f(t4).reshape(-1)}


def exact(case, seed):
    k = case["kind"]
    if k == "tile":
        return tile_reference(inputs(case, seed), case["nb"], case["ib"])
    if k == "batch":
        return None   # a thousand small factorizations: too long one by one
    if k == "lstsq":
        m, n = case["m"], case["n"]
        if 2.0 * m * n * n > 2e12:
            return None
        x = inputs(case, seed)
        sol = torch.linalg.lstsq(x["a2d"], x["b"].t().contiguous()).solution
        res = torch.linalg.norm(x["b"].t() - x["a2d"] @ sol, dim=0)
        return {"x": sol.t().contiguous(), "residual": res.cpu().numpy()}
    if k == "apply":
        return {"qtc": None, "c": inputs(case, seed)["c"]}   # Q Q^T C = C
    nb = case["nb"]
    m = up(case.get("m", case["n"]), nb)
    n = up(case["n"], nb)
    mt, nt = m // nb, n // nb
    if case.get("tree") or mt * nt > 600 or m * n > 4096 * 4096:
        return None
    x = inputs(case, seed)
    if k == "ragged":
        A = torch.zeros(m, n, dtype=F64, device="cuda")
        A[:case["m"], :case["n"]] = x["a"].t()
        C = torch.zeros(m, case["nrhs"], dtype=F64, device="cuda")
        C[:case["m"]] = x["b"].t()
    else:
        A = from_tiles(x["a"], m, n, nb).contiguous()
        C = torch.eye(m, dtype=F64, device="cuda") if k != "tall" else from_tiles(x["c"], m, case["ct"] * nb, nb)
    C = C.contiguous()
    tau, blocks = tile_householder(A, nb)
    for b in blocks:
        apply_block(C, b)
    if k == "tall":
        return {"ry": to_tiles(A, nb), "tau": tau, "qtc": to_tiles(C, nb)}
    if k == "ragged":
        return {"ry": A[:case["m"], :case["n"]].t().contiguous().reshape(-1), "tau": tau,
                "qtb": C[:case["m"]].t().contiguous().reshape(-1)}
    out = {"q": to_tiles(C, nb), "r": to_tiles(torch.triu(A), nb), "tau": tau}
    if k == "dropin":
        out = {key: v.cpu().numpy() for key, v in out.items()}
        out["qr"] = x["a"].cpu().numpy()
    return out
