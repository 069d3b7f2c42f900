"""The work a user of this library has it do, as cases to be timed and compared: sizes, inputs, one pass, exact values.

A pass goes through the public entry points on device tensors, as a Gauss-Newton / Levenberg-Marquardt program calls
them once per iteration: the plan, the layout and the buffers are in hand, the block values are new. The scenes have the
shapes and distributions of this repository's own workloads (scenes.py, bench.py, the tests): cameras seen through a
window of neighbours, k = 2 + Geom observations per point, standard normal Jacobians with log-uniform column scales.

    reduce     reset_schur_sparse + reduce_schur_sparse, the elimination of the points into a sparse S
    backsub    backsubstitute, the way back: the points from the retained variables
    lm_dense   a whole small step on a dense S: reset, reduce, Cholesky, solve, back-substitution
    pcg        the iterative solve of a large sparse S to 1e-8
    cholesky   the dense reduced solve, factorisation and one right-hand side
    qr         reduce_qr + reduced_normal_sparse, the elimination from the Jacobian itself
    qr_lsmr    the Jacobian route solved without forming S: reduce_qr, LSMR, back-substitution
    batch      many uneven problems as one captured step
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def library():
    """This repository's package (its folder's name is not an identifier, so it is loaded by path)."""
    if "blsgpu" not in sys.modules:
        folder = ROOT / "blocklinearsystems.jl_b200"
        spec = importlib.util.spec_from_file_location("blsgpu", folder / "__init__.py", submodule_search_locations=[str(folder)])
        module = importlib.util.module_from_spec(spec)
        sys.modules["blsgpu"] = module
        spec.loader.exec_module(module)
    return sys.modules["blsgpu"]


# ----------------------------------------------------------------------------------------------------------------------
# Cases
# ----------------------------------------------------------------------------------------------------------------------
def scene(kind, cams, points, width, kmean, kcap, dtype, lam, r_dims="6", e_dims="3", scaled=False):
    return dict(kind=kind, cams=cams, points=points, width=width, kmean=kmean, kcap=kcap, dtype=dtype, lam=lam, r_dims=r_dims,
                e_dims=e_dims, scaled=scaled)


def listed():
    return [
        # a small problem in a loop (a local window of a SLAM system): the whole step counts, launches and waits first
        dict(scene("lm_dense", 50, 2000, 50, 5.0, 8, "f64", 1e-3), name="lm step dense 50x2000 f64"),
        # the ordinary bundle adjustment, mixed precision
        dict(scene("reduce", 1000, 200_000, 61, 6.0, 40, "f32", 1e-4), name="reduce 1000x200k f32"),
        # the same in double precision with the conditioning scales that the linear-system layer turns on
        dict(scene("reduce", 1000, 200_000, 61, 6.0, 40, "f64", 1e-4, scaled=True), name="reduce 1000x200k f64 scaled"),
        # the largest scene, the benchmark's default
        dict(scene("reduce", 10_000, 1_000_000, 121, 7.67, 60, "f32", 1e-5), name="reduce 10000x1M f32"),
        # cameras that calibrate themselves: pose and intrinsics, nine variables
        dict(scene("reduce", 803, 120_001, 41, 6.0, 30, "f32", 1e-4, r_dims="9"), name="reduce 9x3 803x120k f32"),
        # a ragged problem: calibrated and uncalibrated cameras, points and inverse depths
        dict(scene("reduce", 97, 7001, 31, 4.3, 20, "f64", 1e-3, r_dims="9,6", e_dims="3,1"), name="reduce mixed 97x7001 f64"),
        # the way back after the reduced solve
        dict(scene("backsub", 3000, 300_000, 121, 7.67, 60, "f32", 1e-5), name="backsub 3000x300k f32"),
        # the reduced solve of a large scene
        dict(scene("pcg", 5000, 250_000, 121, 7.67, 60, "f32", 1e-5), name="pcg 5000 cameras f32"),
        # the reduced solve of a dense S of a thousand cameras
        dict(kind="cholesky", n=6000, dtype="f64", name="cholesky 6000 f64"),
        # ill-conditioned problems go through the Jacobian
        dict(scene("qr", 500, 100_000, 41, 5.8, 16, "f32", 1e-6), name="qr 500x100k f32"),
        # the same without forming S, odd sizes, double precision
        dict(scene("qr_lsmr", 211, 31_007, 41, 5.8, 16, "f64", 1e-6), name="qr lsmr solve 211x31007 f64"),
        # many independent problems of uneven sizes per step
        dict(kind="batch", problems=24, cams=200, points=16_000, width=31, kmean=4.3, kcap=20, dtype="f32", name="batch of 24 f32"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["lm_dense", "reduce", "reduce", "reduce", "reduce", "backsub", "pcg", "cholesky", "qr", "qr_lsmr", "batch"])
    dtype = rng.choice(["f32", "f64"])
    lam = 10.0 ** rng.uniform(-6, -3)
    if kind == "cholesky":
        return dict(kind=kind, n=log(200, 6000), dtype=dtype)
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(4, 24), cams=log(20, 200), points=log(1000, 16_000), width=31, kmean=4.3, kcap=20,
                    dtype=dtype)
    if kind == "lm_dense":
        cams = log(8, 300)
        return scene(kind, cams, cams * rng.randint(20, 60), min(cams, 61), rng.uniform(3.0, 6.0), 8, dtype, lam)
    cams = log(40, 3000 if kind in ("reduce", "backsub", "pcg") else 400)
    points = cams * log(40, 200)
    width = min(cams, rng.choice([31, 41, 61, 121]))
    kmean, kcap = rng.uniform(3.5, 7.6), rng.choice([16, 20, 40])
    if kind in ("qr", "qr_lsmr"):
        return scene(kind, cams, points, width, min(kmean, 6.0), 16, dtype, lam)
    if kind == "reduce":
        r_dims, e_dims = rng.choice([("6", "3")] * 4 + [("9", "3"), ("9,6", "3,1"), ("7", "3"), ("6,3", "3,2")])
        if (r_dims, e_dims) != ("6", "3"):
            points = min(points, 120_000)
        return scene(kind, cams, points, width, kmean, kcap, dtype, lam, r_dims, e_dims, scaled=rng.random() < 0.4)
    return scene(kind, cams, points, width, kmean, kcap, dtype, lam)


# ----------------------------------------------------------------------------------------------------------------------
# Scenes, on the GPU
# ----------------------------------------------------------------------------------------------------------------------
def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def cycle(text, n):
    """n block sizes, the sizes of `text` in turn for cameras; see point_sizes for points."""
    d = [int(x) for x in text.split(",")]
    return torch.tensor(d, device="cuda").repeat((n + len(d) - 1) // len(d))[:n]


def point_sizes(text, n):
    """n block sizes in descending order, an equal share of each (eliminated blocks come grouped by size)."""
    d = sorted((int(x) for x in text.split(",")), reverse=True)
    return torch.tensor(d, device="cuda").repeat_interleave((n + len(d) - 1) // len(d))[:n]


def segment_sum(x, lengths):
    flat = torch.segment_reduce(x.reshape(x.shape[0], -1), "sum", lengths=lengths, axis=0)
    return flat.reshape((lengths.numel(),) + tuple(x.shape[1:]))


class Scene:
    """Which camera sees which point (couplings point by point, cameras ascending) and the Jacobian of two residual rows
    per observation, padded to the largest block sizes: Jc (n, 2, DR), Jp (n, 2, DE), r (n, 2), all float64."""

    def __init__(self, case, gen):
        nc, npt, width, kcap = case["cams"], case["points"], min(case["width"], case["cams"]), min(case["kcap"], case["width"], case["cams"])
        f8 = dict(dtype=torch.float64, device="cuda", generator=gen)
        graph = generator(7919 * nc + npt)   # who sees whom belongs to the case: a program's layout outlives its values
        g8 = dict(f8, generator=graph)
        self.nc, self.npt = nc, npt
        self.r_dims, self.e_dims = cycle(case.get("r_dims", "6"), nc), point_sizes(case.get("e_dims", "3"), npt)
        p = 1.0 / (case["kmean"] - 1.0)
        u = torch.rand(npt, **g8).clamp_(1e-300, 1.0)
        k = (2 + torch.floor(torch.log(u) / math.log1p(-p))).clamp_(2, kcap).long()
        first = (torch.rand(npt, **g8) * (nc - width + 1)).long().clamp_(0, nc - width)
        cams = []
        for a in range(0, npt, 1 << 18):
            score = torch.rand(min(1 << 18, npt - a), width, device="cuda", generator=graph)
            pick = score.topk(kcap, dim=1).indices + first[a:a + (1 << 18), None]
            keep = torch.arange(kcap, device="cuda")[None, :] < k[a:a + (1 << 18), None]
            pick = torch.where(keep, pick, nc).sort(dim=1).values
            cams.append(pick[pick < nc])
        self.cam = torch.cat(cams)
        self.k, self.n = k, self.cam.numel()
        self.ptr = torch.zeros(npt + 1, dtype=torch.long, device="cuda")
        self.ptr[1:] = k.cumsum(0)
        self.pt = torch.repeat_interleave(torch.arange(npt, device="cuda"), k)
        self.DR, self.DE = int(self.r_dims.max()), int(self.e_dims.max())
        self.rmask = torch.arange(self.DR, device="cuda")[None, :] < self.r_dims[:, None]   # cameras x DR
        self.emask = torch.arange(self.DE, device="cuda")[None, :] < self.e_dims[:, None]   # points x DE
        cs = 10.0 ** (2 * torch.rand(nc, self.DR, **f8) - 1) * self.rmask
        ps = 10.0 ** (torch.rand(npt, 1, **f8) - 1) * self.emask
        self.Jc = torch.randn(self.n, 2, self.DR, **f8) * cs[self.cam, None, :]
        self.Jp = torch.randn(self.n, 2, self.DE, **f8) * ps[self.pt, None, :]
        self.r = torch.randn(self.n, 2, **f8)

    def couplings(self):
        return self.ptr.cpu().numpy(), self.cam.cpu().numpy()

    def by_camera(self, x):
        """Per camera the sum of x over its observations, in their order."""
        order = torch.argsort(self.cam, stable=True)
        return segment_sum(x[order], torch.bincount(self.cam, minlength=self.nc))


class Hessian:
    """H = J'J, b = J'r of a scene, padded, every value rounded to the storage type and held in float64; Marquardt damping."""

    def __init__(self, case, sc):
        self.sc, self.lam = sc, case.get("lam", 1e-4)
        round_ = (lambda x: x.float().double()) if case["dtype"] == "f32" else (lambda x: x)
        self.E = round_(segment_sum(torch.einsum("nka,nkb->nab", sc.Jp, sc.Jp), sc.k))
        self.C = round_(torch.einsum("nkw,nks->nws", sc.Jc, sc.Jp))      # per coupling [w, s]: the stored d_e x d_r, column by column
        self.R = round_(sc.by_camera(torch.einsum("nka,nkb->nab", sc.Jc, sc.Jc)))
        self.b_e = segment_sum(torch.einsum("nks,nk->ns", sc.Jp, sc.r), sc.k)
        self.b_r = sc.by_camera(torch.einsum("nkw,nk->nw", sc.Jc, sc.r))
        self.sc_r = torch.diagonal(self.R, dim1=1, dim2=2).clone()
        self.sc_e = torch.diagonal(self.E, dim1=1, dim2=2).clone()
        self.s_r = self.s_e = None
        if case.get("scaled"):   # the nearest power of two to 1 / sqrt of the damped diagonal
            scale = lambda d: torch.exp2(torch.round(-0.5 * torch.log2(torch.where(d > 0, d, 1.0) * (1 + self.lam))))
            self.s_r, self.s_e = scale(self.sc_r), scale(self.sc_e)

    def flat(self, x, mask):
        return None if x is None else x[mask].contiguous()

    def arrays(self, dtype):
        """The block storage as the library takes it (without R, whose layout is the pattern's)."""
        sc = self.sc
        m = sc.emask[:, :, None] & sc.emask[:, None, :]
        mc = sc.rmask[sc.cam][:, :, None] & sc.emask[sc.pt][:, None, :]
        return dict(E=self.E[m].to(dtype), C=self.C[mc].to(dtype), b_r=self.flat(self.b_r, sc.rmask), b_e=self.flat(self.b_e, sc.emask),
                    sc_r=self.flat(self.sc_r, sc.rmask), sc_e=self.flat(self.sc_e, sc.emask), s_r=self.flat(self.s_r, sc.rmask),
                    s_e=self.flat(self.s_e, sc.emask))

    def R_on_pattern(self, st, pat, dtype):
        """The retained storage: the diagonal block of camera r is the last block of its column of the pattern."""
        sc = self.sc
        start = torch.from_numpy(pat.R_block_start[pat.block_colptr[1:] - 1]).cuda()
        i = torch.arange(sc.DR, device="cuda")
        at = start[:, None, None] + i[None, :, None] + sc.r_dims[:, None, None] * i[None, None, :]
        R = torch.zeros(pat.R_length, dtype=dtype, device="cuda")
        m = sc.rmask[:, :, None] & sc.rmask[:, None, :]
        R[at[m]] = self.R[m].to(dtype)
        return R

    def R_dense(self, dtype):
        sc = self.sc
        off = torch.cumsum(sc.r_dims, 0) - sc.r_dims
        nr = int(sc.r_dims.sum())
        i = torch.arange(sc.DR, device="cuda")
        at = (off[:, None, None] + i[None, :, None]) + nr * (off[:, None, None] + i[None, None, :])
        m = sc.rmask[:, :, None] & sc.rmask[:, None, :]
        R = torch.zeros(nr * nr, dtype=dtype, device="cuda")
        R[at[m]] = self.R[m].to(dtype)
        return R


# ----------------------------------------------------------------------------------------------------------------------
# Exact values: the elimination in float64 torch, block by block
# ----------------------------------------------------------------------------------------------------------------------
class Exact:
    """S (blocks of the upper pattern, S = R + lam diag(sc_r) - C' E^-1 C) and g = b_r - C' E^-1 b_e, scaled as given."""

    def __init__(self, h):
        sc, lam = h.sc, h.lam
        self.h, self.sc = h, sc
        one = torch.ones((), dtype=torch.float64, device="cuda")
        s_r = h.s_r if h.s_r is not None else one.expand_as(h.b_r)
        s_e = h.s_e if h.s_e is not None else one.expand_as(h.b_e)
        E = h.E * s_e[:, :, None] * s_e[:, None, :] + torch.diag_embed(lam * h.sc_e * s_e**2 + (~sc.emask).double())
        self.C = h.C * s_r[sc.cam][:, :, None] * s_e[sc.pt][:, None, :]
        self.Einv = inverse(E)
        self.z = torch.einsum("pab,pb->pa", self.Einv, h.b_e * s_e)
        self.g = h.b_r * s_r - sc.by_camera(torch.einsum("nws,ns->nw", self.C, self.z[sc.pt]))
        W = torch.einsum("nab,nwb->nwa", self.Einv[sc.pt], self.C)
        j = torch.arange(sc.n, device="cuda") - sc.ptr[sc.pt]
        ends = torch.cumsum(j + 1, 0)
        total = int(ends[-1])

        def chunks():
            a = 0
            while a < sc.n:
                done = int(ends[a - 1]) if a else 0
                b = int(torch.searchsorted(ends, done + (1 << 23), right=True))
                b = min(max(b, a + 1), sc.n)
                c2 = torch.repeat_interleave(torch.arange(a, b, device="cuda"), j[a:b] + 1)
                c1 = torch.arange(c2.numel(), device="cuda") + done - (ends[c2] - j[c2] - 1) + sc.ptr[sc.pt[c2]]
                yield c1, c2
                a = b

        keys = torch.arange(sc.nc, device="cuda") * (sc.nc + 1)
        for c1, c2 in chunks():
            keys = torch.unique(torch.cat([keys, sc.cam[c2] * sc.nc + sc.cam[c1]]))
        self.keys, self.npairs = keys, total
        B = torch.zeros(keys.numel(), sc.DR, sc.DR, dtype=torch.float64, device="cuda")
        for c1, c2 in chunks():
            slot = torch.searchsorted(keys, sc.cam[c2] * sc.nc + sc.cam[c1])
            B.index_add_(0, slot, torch.einsum("nas,nbs->nab", self.C[c1], W[c2]), alpha=-1.0)
        diag = torch.searchsorted(keys, torch.arange(sc.nc, device="cuda") * (sc.nc + 1))
        B[diag] += h.R * s_r[:, :, None] * s_r[:, None, :] + torch.diag_embed(lam * h.sc_r * s_r**2)
        self.r2, self.r1 = keys // sc.nc, keys % sc.nc
        self.B = B

    def csc(self):
        """The values of the upper block pattern's CSC: per camera its scalar columns, each over the column's blocks in
        ascending order; the lower triangles of the diagonal blocks are stored as zeros."""
        sc = self.sc
        d1, d2 = sc.r_dims[self.r1], sc.r_dims[self.r2]
        H = torch.zeros(sc.nc, dtype=torch.long, device="cuda").index_add_(0, self.r2, d1)
        first = torch.searchsorted(self.r2, self.r2)
        before = torch.cumsum(d1, 0) - d1
        base = torch.cumsum(H * sc.r_dims, 0) - H * sc.r_dims
        i = torch.arange(sc.DR, device="cuda")
        at = (base[self.r2] + before - before[first])[:, None, None] + i[None, :, None] + H[self.r2][:, None, None] * i[None, None, :]
        m = (i[None, :, None] < d1[:, None, None]) & (i[None, None, :] < d2[:, None, None])
        low = (self.r1 == self.r2)[:, None, None] & (i[None, :, None] > i[None, None, :])
        S = torch.zeros(int((H * sc.r_dims).sum()), dtype=torch.float64, device="cuda")
        S[at[m]] = torch.where(low, 0.0, self.B)[m]
        return S

    def dense(self):
        """S as a full symmetric matrix."""
        sc = self.sc
        off = torch.cumsum(sc.r_dims, 0) - sc.r_dims
        nr = int(sc.r_dims.sum())
        i = torch.arange(sc.DR, device="cuda")
        m = sc.rmask[self.r1][:, :, None] & sc.rmask[self.r2][:, None, :]
        row = (off[self.r1][:, None, None] + i[None, :, None]).expand_as(m)[m]
        col = (off[self.r2][:, None, None] + i[None, None, :]).expand_as(m)[m]
        S = torch.zeros(nr, nr, dtype=torch.float64, device="cuda")
        S[row, col] = self.B[m]
        return torch.triu(S) + torch.triu(S, 1).T

    def gradient(self):
        return self.g[self.sc.rmask]

    def points(self, x_r):
        """x_e = z - E^-1 C x_r."""
        sc = self.sc
        x = torch.zeros(sc.nc, sc.DR, dtype=torch.float64, device="cuda")
        x[sc.rmask] = x_r
        t = segment_sum(torch.einsum("nws,nw->ns", self.C, x[sc.cam]), sc.k)
        return (self.z - torch.einsum("pab,pb->pa", self.Einv, t))[sc.emask]


def inverse(E):
    """The inverse of each small symmetric positive definite block, from its Cholesky factor, in pieces."""
    return torch.cat([torch.cholesky_inverse(torch.linalg.cholesky(E[a:a + 100_000])) for a in range(0, E.shape[0], 100_000)])


def conjugate_gradients(ex, g):
    """S x = g to the last bits, S from its upper blocks, block-Jacobi preconditioned (exact value of the pcg cases)."""
    sc = ex.sc
    B = torch.where((ex.r1 == ex.r2)[:, None, None], torch.triu(ex.B) + torch.triu(ex.B, 1).transpose(1, 2), ex.B)
    off = ex.r1 != ex.r2
    D = inverse(B[~off])

    def mul(x):
        X = x.view(sc.nc, sc.DR)
        y = torch.zeros_like(X).index_add_(0, ex.r1, torch.einsum("nab,nb->na", B, X[ex.r2]))
        return y.index_add_(0, ex.r2[off], torch.einsum("nab,na->nb", B[off], X[ex.r1[off]])).reshape(-1)

    x = torch.zeros_like(g)
    r = g.clone()
    z = torch.einsum("nab,nb->na", D, r.view(sc.nc, sc.DR)).reshape(-1)
    p, rz = z.clone(), torch.dot(r, z)
    for _ in range(400):
        q = mul(p)
        a = rz / torch.dot(p, q)
        x += a * p
        r -= a * q
        if float(torch.linalg.vector_norm(r) / torch.linalg.vector_norm(g)) < 1e-15:
            break
        z = torch.einsum("nab,nb->na", D, r.view(sc.nc, sc.DR)).reshape(-1)
        new = torch.dot(r, z)
        p = z + (new / rz) * p
        rz = new
    return x


# ----------------------------------------------------------------------------------------------------------------------
# What a program has in hand, and one pass
# ----------------------------------------------------------------------------------------------------------------------
def structure_of(bls, sc):
    ptr, cam = sc.couplings()
    return bls.SchurStructure.positional(sc.r_dims.cpu().numpy(), sc.e_dims.cpu().numpy(), (ptr, cam))


def prepare(case, seed):
    bls = library()
    state = {"reduce": prepare_reduce, "backsub": prepare_backsub, "lm_dense": prepare_lm_dense, "pcg": prepare_pcg,
             "cholesky": prepare_cholesky, "qr": prepare_qr, "qr_lsmr": prepare_qr, "batch": prepare_batch}[case["kind"]](bls, case, seed)
    state.update(bls=bls, run=PASSES[case["kind"]])
    return state


def run(state):
    return state["run"](state)


def prepare_reduce(bls, case, seed):
    dt = DTYPES[case["dtype"]]
    h = Hessian(case, Scene(case, generator(seed)))
    st = structure_of(bls, h.sc)
    pat = bls.build_schur_pattern(st)
    s = h.arrays(dt)
    s.update(R=h.R_on_pattern(st, pat, dt), S=torch.zeros(pat.nnz, dtype=dt, device="cuda"),
             g=torch.zeros(st.nr, dtype=torch.float64, device="cuda"), st=st, pat=pat, lam=h.lam, ws=bls.SchurReductionWorkspace(st, pat))
    return s


def pass_reduce(s):
    bls, ws, pat = s["bls"], s["ws"], s["pat"]
    bls.reset_schur_sparse(s["S"], s["R"], ws.r_to_s_map, pat.diag_inds, s["sc_r"], s["lam"], ws, s["s_r"])
    ok = bls.reduce_schur_sparse(s["S"], s["g"], s["b_r"], s["b_e"], s["sc_e"], s["lam"], s["st"], s["E"], s["C"], pat.block_colptr,
                                 pat.block_rowval, pat.block_row_offsets, pat.col_heights, ws, s["s_r"], s["s_e"])
    return {"S": s["S"], "g": s["g"], "ok": ok}


def prepare_backsub(bls, case, seed):
    s = prepare_reduce(bls, case, seed)
    s["bls"] = bls
    pass_reduce(s)   # the reduction whose caches the back-substitution reads
    s["x_r"] = torch.randn(s["st"].nr, dtype=torch.float64, device="cuda", generator=generator(seed + 1))
    s["x_e"] = torch.zeros(s["st"].ne, dtype=torch.float64, device="cuda")
    return s


def pass_backsub(s):
    s["bls"].backsubstitute(s["x_e"], s["x_r"], s["st"], s["C"], s["ws"], s["s_r"], s["s_e"])
    return s["x_e"]


def prepare_lm_dense(bls, case, seed):
    dt = DTYPES[case["dtype"]]
    h = Hessian(case, Scene(case, generator(seed)))
    st = structure_of(bls, h.sc)
    s = h.arrays(dt)
    f8 = dict(dtype=torch.float64, device="cuda")
    s.update(R=h.R_dense(dt), S=torch.zeros(st.nr * st.nr, dtype=dt, device="cuda"), g=torch.zeros(st.nr, **f8), x_r=torch.zeros(st.nr, **f8),
             x_e=torch.zeros(st.ne, **f8), st=st, lam=h.lam, ws=bls.SchurReductionWorkspace(st), solver=bls.DenseCholesky(st.nr))
    return s


def pass_lm_dense(s):
    bls, ws = s["bls"], s["ws"]
    bls.reset_schur_dense(s["S"], s["R"], s["sc_r"], s["lam"], ws)
    ok = bls.reduce_schur_dense(s["S"], s["g"], s["b_r"], s["b_e"], s["sc_e"], s["lam"], s["st"], s["E"], s["C"], ws)
    ok = ok and s["solver"].factor(s["S"])
    s["solver"].solve(s["g"], s["x_r"])
    bls.backsubstitute(s["x_e"], s["x_r"], s["st"], s["C"], ws)
    return {"S": s["S"], "g": s["g"], "x_r": s["x_r"], "x_e": s["x_e"], "ok": ok}


def prepare_pcg(bls, case, seed):
    dt = DTYPES[case["dtype"]]
    sc = Scene(case, generator(seed))
    ex = Exact(Hessian(case, sc))
    st = structure_of(bls, sc)
    pat = bls.build_schur_pattern(st)
    return dict(S=ex.csc().to(dt), g=ex.gradient(), x=torch.zeros(st.nr, dtype=torch.float64, device="cuda"), ws=bls.PCGWorkspace(st, pat))


def pass_pcg(s):
    s["x"].zero_()
    x, res = s["ws"].solve(s["S"], s["g"], s["x"], tol=1e-8)
    return {"x": x, "converged": res.converged}


def prepare_cholesky(bls, case, seed):
    n, gen = case["n"], generator(seed)
    A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen)
    S = A @ A.T / n + torch.eye(n, dtype=torch.float64, device="cuda")
    S = ((S + S.T) / 2).to(DTYPES[case["dtype"]]).reshape(-1)
    return dict(S=S, n=n, g=torch.randn(n, dtype=torch.float64, device="cuda", generator=gen),
                x=torch.zeros(n, dtype=torch.float64, device="cuda"), solver=bls.DenseCholesky(n))


def pass_cholesky(s):
    ok = s["solver"].factor(s["S"])
    return {"x": s["solver"].solve(s["g"], s["x"]), "ok": ok}


def qr_tables(case, sc, jst, dt):
    """The raw tables: a point's two rows per observation, its cameras' columns first, its own three last; damping rows
    zero. Values rounded to the storage type."""
    st = jst.schur
    M = torch.from_numpy(jst.table_nrows).cuda()[sc.pt]
    ncol = torch.from_numpy(jst.table_ncols).cuda()[sc.pt] - 1
    base = torch.from_numpy(jst.raw_offsets[:-1].copy()).cuda()[sc.pt]
    col = torch.from_numpy(jst.entry_col).cuda()
    row = 2 * (torch.arange(sc.n, device="cuda") - sc.ptr[sc.pt])
    i2 = torch.arange(2, device="cuda")[None, :, None]
    data = torch.zeros(jst.raw_length, dtype=dt, device="cuda")
    for J, c0, d in ((sc.Jc, col, sc.DR), (sc.Jp, ncol - sc.DE, sc.DE)):
        at = (base + row)[:, None, None] + i2 + (c0[:, None, None] + torch.arange(d, device="cuda")) * M[:, None, None]
        data[at.reshape(-1)] = J.to(dt).reshape(-1)
    r = torch.zeros(jst.residual_length, dtype=torch.float64, device="cuda")
    at = (torch.from_numpy(jst.residual_offsets[:-1].copy()).cuda()[sc.pt] + row)[:, None] + torch.arange(2, device="cuda")
    r[at.reshape(-1)] = sc.r.reshape(-1)
    return data, r


def prepare_qr(bls, case, seed):
    dt = DTYPES[case["dtype"]]
    sc = Scene(case, generator(seed))
    jst = bls.SchurJacobianStructure.positional(structure_of(bls, sc), (2 * sc.k).cpu().numpy())
    pat = bls.build_schur_pattern(jst.schur, bls.free_block_pairs(jst))
    data, r = qr_tables(case, sc, jst, dt)
    f8 = dict(dtype=torch.float64, device="cuda")
    nr, ne = jst.schur.nr, jst.schur.ne
    return dict(J=bls.SchurBlockJacobian(jst, dt, data=data, r=r), ws=bls.QRReductionWorkspace(jst, pat, dt), pat=pat, lam=case["lam"],
                sc_e=torch.ones(ne, **f8), sc_r=torch.ones(nr, **f8), S=torch.zeros(pat.nnz, dtype=dt, device="cuda"), g=torch.zeros(nr, **f8),
                x_r=torch.zeros(nr, **f8), x_e=torch.zeros(ne, **f8))


def pass_qr(s):
    ok = s["bls"].reduce_qr(s["ws"], s["J"], s["sc_e"], s["lam"])
    s["bls"].reduced_normal_sparse(s["S"], s["g"], s["ws"], s["pat"])
    return {"S": s["S"], "g": s["g"], "ok": ok}


def pass_qr_lsmr(s):
    bls = s["bls"]
    ok = bls.reduce_qr(s["ws"], s["J"], s["sc_e"], s["lam"])
    res = bls.lsmr_reduced(s["x_r"], s["ws"], s["lam"], s["sc_r"])
    bls.qr_backsubstitute(s["x_e"], s["x_r"], s["ws"])
    return {"x_r": s["x_r"], "x_e": s["x_e"], "ok": ok and res.solved}


def batch_cases(case):
    """The problems of a batch: up to the stated cameras and points, down to a tenth of them."""
    rng = np.random.default_rng(case["cams"])
    for i in range(case["problems"]):
        f = rng.uniform(0.1, 1.0)
        cams = max(8, int(f * case["cams"]))
        points = max(20 * cams, int(rng.uniform(0.5, 1.0) * f * case["points"]))
        yield scene("reduce", cams, points, case["width"], case["kmean"], case["kcap"], case["dtype"], float(10 ** rng.uniform(-6, -2)))


def prepare_batch(bls, case, seed):
    problems, gen = [], generator(seed)
    host = lambda x: x.double().cpu().numpy()
    for c in batch_cases(case):
        h = Hessian(c, Scene(c, gen))
        st = structure_of(bls, h.sc)
        pat = bls.build_schur_pattern(st)
        a = h.arrays(torch.float64)
        problems.append(bls.scenes.HessianProblem(None, st, pat, False, host(a["E"]), host(a["C"]), host(h.R_on_pattern(st, pat, torch.float64)),
                                                  host(a["b_r"]), host(a["b_e"]), host(a["sc_r"]), host(a["sc_e"]), h.lam, h.sc.n))
    batch = bls.batch.BatchedReduction(problems, DTYPES[case["dtype"]])
    batch.autotune()
    batch.capture()
    return dict(batch=batch)


def pass_batch(s):
    b = s["batch"]
    b.step()
    return {"S": b.S, "g": b.g, "ok": b.ok()}


PASSES = {"reduce": pass_reduce, "backsub": pass_backsub, "lm_dense": pass_lm_dense, "pcg": pass_pcg, "cholesky": pass_cholesky,
          "qr": pass_qr, "qr_lsmr": pass_qr_lsmr, "batch": pass_batch}


# ----------------------------------------------------------------------------------------------------------------------
# Exact outputs
# ----------------------------------------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "cholesky":
        n, gen, dt = case["n"], generator(seed), DTYPES[case["dtype"]]
        A = torch.randn(n, n, dtype=torch.float64, device="cuda", generator=gen)
        S = A @ A.T / n + torch.eye(n, dtype=torch.float64, device="cuda")
        S = ((S + S.T) / 2).to(dt).double()
        g = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
        return {"x": torch.cholesky_solve(g[:, None], torch.linalg.cholesky(S))[:, 0], "ok": True}
    if kind == "batch":
        gen = generator(seed)
        ex = [Exact(Hessian(c, Scene(c, gen))) for c in batch_cases(case)]
        return {"S": torch.cat([e.csc() for e in ex]), "g": torch.cat([e.gradient() for e in ex]), "ok": True}
    sc = Scene(case, generator(seed))
    if kind in ("qr", "qr_lsmr"):
        dt = DTYPES[case["dtype"]]
        sc.Jc, sc.Jp = sc.Jc.to(dt).double(), sc.Jp.to(dt).double()
        h = Hessian(dict(case, dtype="f64"), sc)
        h.sc_e = torch.ones_like(h.sc_e)
        h.sc_r = torch.zeros_like(h.sc_r) if kind == "qr" else torch.ones_like(h.sc_r)
        ex = Exact(h)
        if kind == "qr":
            return {"S": ex.csc(), "g": ex.gradient(), "ok": True}
        x_r = solve_dense(ex)
        return {"x_r": x_r, "x_e": ex.points(x_r), "ok": True}
    h = Hessian(case, sc)
    ex = Exact(h)
    if kind == "reduce":
        return {"S": ex.csc(), "g": ex.gradient(), "ok": True}
    if kind == "backsub":
        nr = int(sc.r_dims.sum())
        return ex.points(torch.randn(nr, dtype=torch.float64, device="cuda", generator=generator(seed + 1)))
    if kind == "pcg":
        if case["dtype"] == "f32":
            ex.B = ex.B.float().double()
        return {"x": conjugate_gradients(ex, ex.gradient()), "converged": True}
    x_r = solve_dense(ex)   # lm_dense: S's lower triangle stays R's
    S = torch.triu(ex.dense()) + torch.tril(h.R_dense(torch.float64).view(len(x_r), -1), -1)
    return {"S": S.T.reshape(-1), "g": ex.gradient(), "x_r": x_r, "x_e": ex.points(x_r), "ok": True}


def solve_dense(ex):
    return torch.cholesky_solve(ex.gradient()[:, None], torch.linalg.cholesky(ex.dense()))[:, 0]


# ----------------------------------------------------------------------------------------------------------------------
# The bytes and operations a pass cannot do without
# ----------------------------------------------------------------------------------------------------------------------
def moments(case):
    """E[k] and E[k (k - 1)] of k = 2 + Geom(p), capped."""
    p, cap = 1.0 / (case["kmean"] - 1.0), min(case["kcap"], case["width"], case["cams"])
    k = np.arange(2, cap + 1)
    w = p * (1 - p) ** (k - 2.0)
    w[-1] += 1 - w.sum()
    return float((w * k).sum()), float((w * k * (k - 1)).sum())


def mean_square(text):
    d = [int(x) for x in text.split(",")]
    return sum(d) / len(d), sum(x * x for x in d) / len(d)


def work(case):
    kind, w = case["kind"], 4 if case["dtype"] == "f32" else 8
    if kind == "cholesky":
        n = case["n"]
        return {"bytes": w * n * n / 2 + 16 * n, "flops": n**3 / 3 + 2 * n * n}
    if kind == "batch":
        one = scene("reduce", case["cams"], case["points"], case["width"], case["kmean"], case["kcap"], case["dtype"], 1e-4)
        one = dict(one, cams=max(8, int(0.55 * case["cams"])), points=int(0.41 * case["points"]))
        return {k: case["problems"] * v for k, v in work(one).items()}
    k1, k2 = moments(case)
    nc, npt, nobs = case["cams"], case["points"], k1 * case["points"]
    dr, dr2 = mean_square(case["r_dims"])
    de, de2 = mean_square(case["e_dims"])
    blocks = min(nc * (min(case["width"], nc) - 1), k2 / 2 * npt) + nc
    nnz = dr * dr * blocks if kind != "lm_dense" else (dr * nc) ** 2 / 2
    points = npt * (w * de2 + 16 * de) + nobs * (w * dr * de + 4)     # E, b_e, scaling_e; C and its camera index
    pair = npt * (de2 * 6 + k1 * (2 * dr * de2 + 2 * dr * de) + k2 / 2 * 2 * dr * dr * de + k1 * dr2 * de)
    if kind == "reduce":
        return {"bytes": points + w * nnz + w * dr2 * nc + 24 * dr * nc, "flops": pair}
    if kind == "backsub":
        return {"bytes": nobs * (w * dr * de + 4) + npt * (8 * de2 + 16 * de) + 8 * dr * nc, "flops": npt * (2 * de2 + 2 * k1 * dr * de)}
    if kind == "lm_dense":
        n = dr * nc
        return {"bytes": points + 2 * w * n * n + 32 * n + 8 * de * npt, "flops": pair + n**3 / 3 + 2 * n * n}
    if kind == "pcg":   # S is read once at the least; six iterations are usual
        return {"bytes": w * nnz + 16 * dr * nc, "flops": 6 * 4 * nnz}
    cells = npt * (2 * k2 * dr + 2 * k1 * dr + 3 * k1 * dr + (2 * k1 + 3) * de)     # (2k + 3) x (6k + 3) per table
    flops = cells * 4 * de + (npt * k2 * dr * dr * k1 * 2 if kind == "qr" else 0)
    return {"bytes": cells * w + npt * 8 * (2 * k1 + 3 + de) + (w * nnz if kind == "qr" else 8 * de * npt), "flops": flops}
