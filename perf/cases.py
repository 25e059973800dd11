"""Performance cases of the field solve: what a user's program has the library do, through
the public entry points of srmg.multigrid (the Python mirror of the C ABI).

Each case is a dict of plain values; ``prepare`` builds its inputs and keeps what a program
keeps between calls (the tree's context and stream, the work fields, the network), ``run`` is
one pass, ``work`` the bytes and operations the pass cannot do without and ``exact`` the
same result in 64 bits from plain torch.

Trees and operators are those of the seeded generators in ``srmg.gen`` / ``srmg.gen3``; a
tree is built once per process and shared by every state on it, as a program does between
two refinements.
"""
import ctypes
import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "steamroller.jl_b200"))

from srmg import freebc as fbc  # noqa: E402
from srmg import gen, gen3  # noqa: E402
from srmg import multigrid as mg  # noqa: E402
from srmg import tree as t2  # noqa: E402
from srmg import tree3 as t3  # noqa: E402
from srmg.streamer import BC_DENSITY, BC_EXTRAPOLATE, E_BACKGROUND, MINIMAL  # noqa: E402

M, G, S = 16, 2, 20
OPS = {"laplacian": 0, "helmholtz": 1, "laplacian4": 2}
LAMBDAS = (1.5e2, 1.2e3, 9.0e3)  # screening constants of the three photoionization terms, 1/m
TRANSPORT = mg.Transport(**MINIMAL)


# ------------------------------------------------------------------------------ cases

def listed():
    return [
        # derivs!'s fixed pair of V-cycles on the reference's own small run (256 x 256 cells)
        dict(name="vcycle-uniform", kind="vcycle", tree="uniform", level=5, op="laplacian", geom=1, cycles=2,
             ndown=2, ntop=4, nup=2),
        # the same call on a developed, branched discharge of 10M leaf cells
        dict(name="vcycle-large", kind="vcycle", tree="branched", leaf=10_000_000, tree_seed=5, op="laplacian",
             geom=1, cycles=2, ndown=2, ntop=4, nup=2),
        # the tolerance-driven mixed-precision solve on the refined channel tree
        dict(name="solve-channel", kind="solve", tree="channel", leaf=1_500_000, tree_seed=2, op="laplacian",
             geom=1),
        # one stage's potential and its three photoionization terms as one batch
        dict(name="batch-stage", kind="batch", tree="channel", leaf=300_000, tree_seed=3, geom=1),
        # full multigrid from a zero potential: the start of a run on a refined tree
        dict(name="fmg-channel", kind="fmg", tree="channel", leaf=400_000, tree_seed=4, op="laplacian", geom=1,
             ndown=3, ntop=5, nup=3),
        # the compact order-4 discretisation (poisson_order = 4) on a refined tree
        dict(name="order4-channel", kind="vcycle", tree="box", base=6, extra=3, tree_seed=41, op="laplacian4",
             geom=1, cycles=2, ndown=2, ntop=4, nup=2),
        # three dimensions: a uniform octree at order 2, a refined one at order 4
        dict(name="octree-uniform", kind="vcycle3", tree="octree", level=4, refine=0, tree_seed=1, op="laplacian",
             cycles=1, ndown=2, ntop=4, nup=2),
        dict(name="octree-order4", kind="vcycle3", tree="octree", level=3, refine=3, tree_seed=1,
             op="laplacian4", cycles=1, ndown=2, ntop=4, nup=2),
        # everything of a derivs! stage around the solve, on the large tree
        dict(name="stage-large", kind="stage", tree="branched", leaf=10_000_000, tree_seed=5, geom=1),
        # free boundary sources of the refined channel tree (4096 points along the column)
        dict(name="freebc-channel", kind="freebc", tree="channel", leaf=1_500_000, tree_seed=2, level=9),
        # the warm-start network: a training pass over four trees' blocks, an inference pass
        dict(name="cnn-train", kind="cnn_train", samples=1024),
        dict(name="cnn-forward", kind="cnn_forward", samples=4096),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vcycle", "solve", "batch", "fmg", "order4", "octree", "stage", "freebc", "cnn_train",
                       "cnn_forward"])
    seed = rng.randrange(1, 1000)
    sweeps = rng.choice([(2, 4, 2), (3, 5, 3), (1, 4, 1)])
    sw = dict(ndown=sweeps[0], ntop=sweeps[1], nup=sweeps[2])
    op = rng.choice(["laplacian", "helmholtz"])
    if kind == "vcycle":
        return dict(kind="vcycle", tree="channel", leaf=_log(rng, 2e4, 4e6), tree_seed=seed, op=op,
                    geom=rng.choice([0, 1, 2]), cycles=rng.choice([1, 2, 3]), **sw)
    if kind == "solve":
        return dict(kind="solve", tree="channel", leaf=_log(rng, 2e4, 2e6), tree_seed=seed, op=op, geom=1)
    if kind == "batch":
        return dict(kind="batch", tree="channel", leaf=_log(rng, 2e4, 6e5), tree_seed=seed, geom=1)
    if kind == "fmg":
        return dict(kind="fmg", tree="channel", leaf=_log(rng, 2e4, 1.5e6), tree_seed=seed, op=op, geom=1, **sw)
    if kind == "order4":
        return dict(kind="vcycle", tree="box", base=rng.choice([3, 4, 5, 6]), extra=rng.choice([1, 2, 3]),
                    tree_seed=seed, op=rng.choice(["laplacian4", "laplacian4", "helmholtz"]),
                    geom=rng.choice([0, 1, 2]), cycles=rng.choice([1, 2]), **sw)
    if kind == "octree":
        level = rng.choice([2, 3, 4])
        return dict(kind="vcycle3", tree="octree", level=level, refine=0 if level == 4 else rng.choice([0, 1, 2, 3]),
                    tree_seed=seed, op=rng.choice(["laplacian", "helmholtz", "laplacian4"]), cycles=1, **sw)
    if kind == "stage":
        return dict(kind="stage", tree="channel", leaf=_log(rng, 1e5, 6e6), tree_seed=seed, geom=1)
    if kind == "freebc":
        return dict(kind="freebc", tree="channel", leaf=_log(rng, 1e5, 1.5e6), tree_seed=seed,
                    level=rng.choice([9, 10, 11]))
    return dict(kind=kind, samples=_log(rng, 48, 6000))


# ------------------------------------------------------------------------------ trees

class Plan:
    """A tree with its context and stream, and the templates its inputs are drawn around."""

    def __init__(self, D, tree, conn, s, h1, template):
        self.D, self.tree, self.conn, self.s, self.h1 = D, tree, conn, s, h1
        self.nblk = tree.nblocks_created
        self.template = torch.from_numpy(template).cuda()
        self.leaf = torch.from_numpy(_leaf_mask(tree, D)).cuda()
        self.ctx = mg.Context(0, D=D).set_tree(tree, conn)
        self.stream = torch.cuda.Stream()
        self.ctx.set_stream(self.stream.cuda_stream)
        self.keep = {}

    def field(self):
        return torch.zeros((self.nblk,) + (S,) * self.D, dtype=torch.float64, device="cuda")

    def cells(self):
        return [len(layer.index) * M ** self.D for layer in self.tree]


def _leaf_mask(tree, D):
    m = np.zeros((tree.nblocks_created,) + (S,) * D, dtype=bool)
    v = (slice(G, G + M),) * D
    for layer in tree:
        for c, blk in layer.index.items():
            if tree.isleaf(layer.level, c):
                m[(blk - 1,) + v] = True
    return m


@functools.lru_cache(maxsize=None)
def _plan(kind, *key):
    if kind == "uniform":
        tree = t2.Tree((1, 1), key[0])
        t2.populate(tree, key[0])
        p = gen.config1(seed=1) if key[0] == 5 else gen.make_problem(
            tree, lambda r, z, l, gi, gj: 1e20 * np.exp(-(r * r + (z - 6e-3) ** 2) / 2e-7), gen.poisson_scale())
        return Plan(2, p.tree, p.conn, p.s, p.h1, p.b)
    if kind == "channel":
        leaf, seed = key
        base = 5 if leaf >= 4e5 else 4 if leaf >= 6e4 else 3
        p = gen.config2(seed=seed, target_leaf=leaf, base_level=base)
        return Plan(2, p.tree, p.conn, p.s, p.h1, p.b)
    if kind == "branched":
        p = gen.config5(seed=key[1], target_leaf=key[0])
        return Plan(2, p.tree, p.conn, p.s, p.h1, p.b)
    if kind == "box":
        base, extra, seed = key
        p = gen.order4_problem(seed=seed, geom=gen.GEOM_CYL1, base_level=base, extra=extra)
        return Plan(2, p.tree, p.conn, p.s, p.h1, p.b)
    level, refine, seed, stencil = key
    tree = t3.Tree3((1, 1, 1), level + refine)
    t3.populate(tree, level)
    rng = np.random.default_rng(seed)
    c = tuple(int(x) for x in rng.integers(1, 2 ** (level - 1) + 1, size=3))
    for l in range(level, level + refine):  # refine towards one seeded corner, with nesting
        t3.refine_block(tree, l, c, t3.BOX3)
        c = tuple(2 * x - int(rng.integers(0, 2)) for x in c)
    tree.sync()
    conn = t3.connectivity(tree, t3.BOX3 if stencil == "box" else t3.STAR3)
    ctr = rng.uniform(0.3, 0.7, size=3)
    h1 = 1.0 / M
    p = gen3.make_problem3(tree, conn, lambda x, y, z: np.exp(
        -((x - ctr[0]) ** 2 + (y - ctr[1]) ** 2 + (z - ctr[2]) ** 2) / 0.02), h1 * h1, h1=h1)
    return Plan(3, tree, conn, h1 * h1, h1, p.b)


def plan(case):
    kind = case["tree"]
    if kind == "uniform":
        return _plan(kind, case["level"])
    if kind == "box":
        return _plan(kind, case["base"], case["extra"], case["tree_seed"])
    if kind == "octree":
        return _plan(kind, case["level"], case["refine"], case["tree_seed"],
                     "box" if case["op"] == "laplacian4" else "star")
    return _plan(kind, case["leaf"], case["tree_seed"])


def operator(case, P):
    """(s, descriptor, op, k2, geometry, boundary table) of a case's discretisation."""
    op = case.get("op", "laplacian")
    if P.D == 3:
        k2 = 30.0 if op == "helmholtz" else 0.0
        bc = t3.boundaryconditions(((-1, -1), (1, -1), (-1, 1)))
        return P.s, ("helmholtz", k2) if k2 else op, OPS[op], k2, 0, bc
    geom = case["geom"]
    bc = {0: t2.boundaryconditions(((-1, -1), (-1, -1))), 1: gen.BC_POISSON,
          2: t2.boundaryconditions(((-1, -1), (1, 1)))}[geom]
    if op == "helmholtz":
        k2 = LAMBDAS[1] ** 2
        return P.h1 * P.h1, ("helmholtz", k2), 1, k2, geom, bc
    return P.s, op, OPS[op], 0.0, geom, bc


# ----------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 13)
    return g


def _noise(P, seed, k=0):
    """Log-uniform +-0.1 dex per cell, as the generators' density noise."""
    r = torch.rand((P.nblk,) + (S,) * P.D, generator=_gen(seed + 1000003 * k), device="cuda", dtype=torch.float64)
    return 10.0 ** (0.2 * r - 0.1)


def restrict_full(P, f):
    """Parents become the means of their children (restrict_full!), 2D and 3D."""
    for l in range(len(P.tree), 1, -1):
        P.ctx.check(mg.lib().srmg_restrict_level_dev(P.ctx.handle, f.data_ptr(), P.nblk, l))
    P.ctx.synchronize()


def charge(P, seed, photo=False):
    """A right-hand side: the tree's charge, noisy per cell, or a photoionization source
    (positive, where the charge is), consistent over the levels."""
    t = P.template.abs() * 1e-3 if photo else P.template
    b = torch.where(P.leaf, t * _noise(P, seed), torch.zeros_like(t))
    torch.cuda.synchronize()
    restrict_full(P, b)
    return b


class State:
    pass


def prepare(case, seed):
    st = State()
    st.case, kind = case, case["kind"]
    if kind in ("cnn_train", "cnn_forward"):
        n = case["samples"]
        st.net = _net()
        g = _gen(seed)
        # smooth tiles of (previous correction, charge change), normalised as the packer does
        st.x = torch.randn((n, S * S, 2), generator=g, device="cuda").mul_(0.5).to(torch.bfloat16)
        st.t = 0.1 * torch.randn((n, M * M), generator=g, device="cuda")
        return st
    P = st.P = plan(case)
    if kind == "stage":
        v = (slice(None),) + (slice(G, G + M),) * 2
        zero = P.field()
        b = torch.where(P.leaf, P.template, zero)
        # a neutral conducting plasma where the charge is, over the background density
        st.ne = torch.where(P.leaf, (1e13 + 10.0 * b.abs()) * _noise(P, seed), zero)
        st.nion = torch.where(P.leaf, st.ne + b * _noise(P, seed, 1), zero)
        st.phi = P.field()
        st.phi[v] = 10.0 * torch.randn(st.phi[v].shape, generator=_gen(seed + 5), device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        for f in (st.ne, st.nion, st.phi):
            restrict_full(P, f)
        st.q, st.eabs, st.dne, st.dni, st.n1, st.n1i = (P.field() for _ in range(6))
        st.e, st.flux = (torch.zeros((P.nblk, 2, S + 1, S + 1), dtype=torch.float64, device="cuda") for _ in "ef")
        st.maxdt = torch.zeros(1, dtype=torch.float64, device="cuda")
        st.eb = np.array(E_BACKGROUND)
    elif kind == "freebc":
        key = ("freebc", case["level"])
        if key not in P.keep:
            P.keep[key] = fbc.kernel(1, case["level"], (1, 1), P.h1)
        n, _, _, f = P.keep[key]
        st.f = f
        mg.freebc_set(P.ctx, 1, case["level"], (1, 1), f)
        st.q0 = charge(P, seed)
        st.q, st.b = P.field(), torch.zeros(n, dtype=torch.float64, device="cuda")
        st.u = P.field()
        st.u[P.leaf] = 1.0
        st.u *= 1e3 * torch.randn(st.u.shape, generator=_gen(seed + 5), device="cuda", dtype=torch.float64)
        torch.cuda.synchronize()
        restrict_full(P, st.u)
    elif kind == "batch":
        if "batch" not in P.keep:
            items = [(P.ctx, P.s, "laplacian", gen.BC_POISSON)]
            items += [(P.ctx, P.h1 * P.h1, ("helmholtz", lam * lam), gen.BC_PHOTO) for lam in LAMBDAS]
            P.keep["batch"] = mg.Batch(items, case["geom"])
            P.keep["batch"].set_stream(P.stream.cuda_stream)
        st.batch = P.keep["batch"]
        st.b = [charge(P, seed)] + [charge(P, seed + 17 * j, photo=True) for j in (1, 2, 3)]
        st.u = [P.field() for _ in range(4)]
    else:
        st.b = charge(P, seed, photo=case["op"] == "helmholtz")
        st.u, st.r, st.u1 = P.field(), P.field(), P.field()
        st.s, st.disc, st.op, st.k2, st.geom, st.bc = operator(case, P)
    torch.cuda.synchronize()
    return st


@functools.lru_cache(maxsize=None)
def _net():
    return mg.Cnn(0, seed=5)


# -------------------------------------------------------------------------------- run

def run(st):
    return {"vcycle": _run_vcycle, "vcycle3": _run_vcycle, "fmg": _run_fmg, "solve": _run_solve,
            "batch": _run_batch, "stage": _run_stage, "freebc": _run_freebc, "cnn_train": _run_train,
            "cnn_forward": _run_forward}[st.case["kind"]](st)


def _sweeps(case):
    return {k: case[k] for k in ("ndown", "ntop", "nup")}


def _run_vcycle(st):
    with torch.cuda.stream(st.P.stream):
        mg.vcycle_(st.P.ctx, st.u, st.b, st.r, st.u1, st.s, st.geom, st.bc, st.disc, ncycles=st.case["cycles"],
                   **_sweeps(st.case))
    return {"u": st.u}


def _run_fmg(st):
    with torch.cuda.stream(st.P.stream):
        st.u.zero_()
        mg.fmg_(st.P.ctx, st.u, st.b, st.r, st.u1, st.s, st.geom, st.bc, st.disc, **_sweeps(st.case))
    return {"u": st.u}


def _run_solve(st):
    with torch.cuda.stream(st.P.stream):
        st.u.zero_()
        mg.solve(st.P.ctx, st.u, st.b, st.s, st.geom, st.bc, st.disc, tol=1e-8, mode=mg.MODE_MIXED, inner_cycles=3,
                 **mg.TUNED)
    return {"u": st.u}


def _run_batch(st):
    with torch.cuda.stream(st.P.stream):
        for u in st.u:
            u.zero_()
        st.batch.solve(st.u, st.b, tol=1e-8, mode=mg.MODE_MIXED, **mg.TUNED)
    return {"u": st.u}


def _run_stage(st):
    """derivs! (src/streamer.jl:292-366) without its solve, and the stage combination."""
    P, c, lib = st.P, st.P.ctx, mg.lib()
    h, n = P.h1, P.nblk
    with torch.cuda.stream(P.stream):
        mg.netcharge(c, st.q, st.ne, st.nion)
        mg.restrict_full_(c, st.q)
        mg.restrict_full_(c, st.ne)
        for l in range(1, len(P.tree) + 1):
            mg.fill_ghost_(c, st.ne, l, BC_DENSITY, mask=15)
            mg.fill_ghost_(c, st.phi, l, gen.BC_POISSON)
        mg.electric_field(c, st.e, st.eabs, st.phi, h, st.eb)
        for l in range(1, len(P.tree) + 1):
            mg.fill_ghost_(c, st.eabs, l, BC_EXTRAPOLATE)
        c.check(lib.srmg_streamer_flux_dev(c.handle, st.flux.data_ptr(), None, st.maxdt.data_ptr(), st.ne.data_ptr(),
                                           st.e.data_ptr(), st.eabs.data_ptr(), n, h, ctypes.byref(TRANSPORT)))
        c.check(lib.srmg_streamer_rates_dev(c.handle, st.dne.data_ptr(), st.dni.data_ptr(), st.ne.data_ptr(),
                                            st.eabs.data_ptr(), st.flux.data_ptr(), n, h, st.case["geom"],
                                            ctypes.byref(TRANSPORT)))
        for out, f, d in ((st.n1, st.ne, st.dne), (st.n1i, st.nion, st.dni)):
            c.check(lib.srmg_ssprk3_stage_dev(c.handle, out.data_ptr(), f.data_ptr(), d.data_ptr(), d.data_ptr(),
                                              d.data_ptr(), f.numel(), STAGE_DT, 1))
    return {"q": st.q, "e": st.e, "eabs": st.eabs, "flux": st.flux, "dne": st.dne, "dni": st.dni, "n1": st.n1,
            "n1i": st.n1i, "maxdt": st.maxdt}


STAGE_DT = 1e-13


def _run_freebc(st):
    with torch.cuda.stream(st.P.stream):
        st.q.copy_(st.q0)
        mg.freebc_(st.P.ctx, st.q, st.u, st.P.h1, st.P.s, st.b)
    return {"q": st.q, "b": st.b}


def _run_train(st):
    """learn.train's pass: forward, the loss gradient by the caller, backward."""
    y = st.net.forward_train(st.x)
    dy = (2.0 / y.numel()) * (y - st.t)
    grad = st.net.backward_step(dy, 0.0, want_grad=True)
    return {"y": y, "grad": grad}


def _run_forward(st):
    return {"y": st.net.forward(st.x)}


# ------------------------------------------------------------------------------- work

CNN_MACS = (9 * 2 * 32 + 4 * 9 * 32 * 32 + 9 * 32) * S * S  # per sample, every pixel of the tile


def work(case):
    kind = case["kind"]
    if kind == "cnn_forward":
        n = case["samples"]
        return {"bytes": n * (S * S * 4 + M * M * 4), "flops": 2 * n * CNN_MACS}
    if kind == "cnn_train":  # forward, input gradients, weight gradients
        n = case["samples"]
        return {"bytes": n * (S * S * 4 + 3 * M * M * 4), "flops": 6 * n * CNN_MACS}
    P = plan(case)
    cells = sum(P.cells())
    if kind == "stage":
        # ne, nion, phi read; q, e, eabs, flux, both rates and both stage densities written
        return {"bytes": 8 * cells * 13, "flops": 120 * cells}
    if kind == "freebc":
        n = M << (case["level"] - 1)
        return {"bytes": 16 * cells + 8 * 4 * n, "flops": 20 * n * math.log2(n)}
    if kind == "batch":
        return {"bytes": 4 * 16 * cells, "flops": 4 * 9 * 40 * cells}
    if kind == "solve":  # u and b in, u out; some nine V-cycles of work
        return {"bytes": 24 * cells, "flops": 9 * 40 * cells}
    # V-cycles: u and b read once, u and the FAS right-hand sides written once, each cycle
    cycles = case.get("cycles", 1)
    points = {("laplacian4", 2): 18, ("laplacian4", 3): 38}.get((case["op"], P.D), 2 * (2 * P.D + 1))
    sweeps = case["ndown"] + case["nup"] + 1.5
    return {"bytes": cycles * 32 * cells, "flops": cycles * sweeps * (points + 4) * cells}


# ------------------------------------------------- the same results in 64 bits, plain torch

class Blocks:
    """The block-tree operations on [nblk, 20^D] fields, vectorised over the edge lists."""

    def __init__(self, P):
        self.P, self.D, self.npts = P, P.D, S ** P.D
        self.strides = [S ** d for d in range(P.D)]
        self.valid = self._offsets([np.arange(G, G + M)] * P.D)
        self.blocks, self.coords = [], []
        for layer in P.tree:
            self.blocks.append(self._t([b - 1 for b in layer.index.values()]))
            self.coords.append(self._t(np.array(list(layer.index.keys()), dtype=np.int64).reshape(-1, P.D)))
        self.edges = [self._level(l) for l in range(len(P.tree))]
        self.kids = [self._children(l) for l in range(len(P.tree))]

    def _t(self, a):
        return torch.as_tensor(np.asarray(a, dtype=np.int64), device="cuda")

    def _offsets(self, axes):
        """Flat offsets of the product of per-dimension positions, dimension 1 fastest."""
        o = np.zeros(1, dtype=np.int64)
        for d in reversed(range(self.D)):
            o = (o[:, None] + self.strides[d] * np.asarray(axes[d])[None, :]).reshape(-1)
        return self._t(o)

    @staticmethod
    def _groups(rows, *fields):
        key = np.concatenate([rows[f] for f in fields], axis=1)
        uniq, inv = np.unique(key, axis=0, return_inverse=True)
        for k, u in enumerate(uniq):
            yield u, rows[inv.reshape(-1) == k]

    def _level(self, l):
        c, D = self.P.conn, self.D
        ghost = {-1: np.arange(2), 0: np.arange(G, G + M), 1: np.arange(18, 20)}
        copies, mirrors, interps = [], [], []
        if len(c.neighbor[l]):
            for f, rows in self._groups(c.neighbor[l], "face"):
                copies.append((self._t(rows["to"] - 1), self._offsets([ghost[-x] for x in f]),
                               self._t(rows["from"] - 1), self._offsets([ghost[-x] + M * x for x in f])))
        if len(c.boundary[l]):
            for k, rows in self._groups(c.boundary[l], "face", "bnd"):
                f, b = k[:D], k[D:]
                src = [(3 - ghost[-1]) if b[d] < 0 else (35 - ghost[1]) if b[d] > 0 else ghost[f[d]] for d in range(D)]
                mirrors.append((self._t(rows["block"] - 1), self._offsets([ghost[x] for x in f]), self._offsets(src),
                                sum((1 + int(b[d])) * 3 ** d for d in range(D))))
        if len(c.refboundary[l]):
            for k, rows in self._groups(c.refboundary[l], "face", "subblock"):
                f, sb = k[:D], k[D:]
                js, ii = [], []
                for d in range(D):
                    p = ghost[f[d]]
                    js.append(np.full(2, 1 + 8 * sb[d]) if f[d] < 0 else np.full(2, 2 + 8 * (sb[d] - 1)) if f[d] > 0
                              else 2 + 8 * (sb[d] - 1) + ((p - G) >> 1))
                    ii.append(p if f[d] < 0 else p - 18 if f[d] > 0 else (p - G) & 1)
                interps.append((self._t(rows["fine"] - 1), self._offsets([ghost[x] for x in f]),
                                self._t(rows["coarse"] - 1), self._offsets(js), self._sides(js, ii)))
        return copies, mirrors, interps

    def _sides(self, js, ii):
        """Offsets of the coarse neighbour along each dimension for every fine position."""
        out = []
        for d in range(self.D):
            ax = list(js)
            ax[d] = js[d] + 2 * ii[d] - 1
            out.append(self._offsets(ax))
        return out

    def _children(self, l):
        ch, out = self.P.conn.child[l], []
        if len(ch):
            p = np.arange(M)
            for sb, rows in self._groups(ch, "subblock"):
                js = [2 + 8 * (s - 1) + (p >> 1) for s in sb]
                co = [2 + 8 * (s - 1) + np.arange(8) for s in sb]
                fine = [self._offsets([G + 2 * np.arange(8) + ((k >> d) & 1) for d in range(self.D)])
                        for k in range(2 ** self.D)]
                out.append((self._t(rows["fine"] - 1), self._t(rows["coarse"] - 1), self._offsets(co), fine,
                            self._offsets(js), self._sides(js, [p & 1] * self.D)))
        return out

    def _interp(self, u, blk, js, sides):
        b = blk[:, None]
        v = (0.5 if self.D == 2 else 0.25) * u[b, js]
        for o in sides:
            v = v + 0.25 * u[b, o]
        return v

    def fill(self, u, l, bc, mask=7, copy_interp=False):
        copies, mirrors, interps = self.edges[l]
        if mask & 1:
            for to, dst, fr, src in copies:
                u[to[:, None], dst] = u[fr[:, None], src]
        if mask & 2:
            for blk, dst, src, k in mirrors:
                u[blk[:, None], dst] = float(bc[k]) * u[blk[:, None], src]
        if mask & 4:
            for fine, dst, coarse, js, sides in interps:
                u[fine[:, None], dst] = u[coarse[:, None], js] if copy_interp else self._interp(u, coarse, js, sides)

    def restrict(self, u, l):
        for fine, coarse, co, fo, _, _ in self.kids[l]:
            u[coarse[:, None], co] = sum(u[fine[:, None], o] for o in fo) / 2 ** self.D

    def lhs(self, u, l, blk, coords, cells, op):
        """L u at cells `cells` of blocks `blk` of level l, with the diagonal of L."""
        name, s, k2, geom = op
        b = blk[:, None]
        sl = s / 4 ** l

        def at(*d):
            return u[b, cells + sum(self.strides[i] * x for i, x in enumerate(d))]
        if self.D == 3:
            if name != "laplacian4":
                centre = -6.0 - (sl * k2 if name == "helmholtz" else 0.0)
                v = centre * at(0, 0, 0)
                for d in ((1, 0, 0), (0, 1, 0), (0, 0, 1)):
                    v = v + at(*d) + at(*(-x for x in d))
                return v, centre
            v = -24.0 * at(0, 0, 0)
            for d in t3.BOX3:
                nz = sum(1 for x in d if x)
                if nz < 3:
                    v = v + (2.0 if nz == 1 else 1.0) * at(*d)
            return v / 6.0, -4.0
        i = 0.0
        if geom:
            pos = (cells if geom == 1 else cells // S) % S
            i = (M * (coords[:, geom - 1] - 1)[:, None] + pos[None, :] - 1).double()
        q = 2.0 * i - 1.0
        am, ap = ((2 * i - 2) / q, 2 * i / q) if geom else (1.0, 1.0)
        if name != "laplacian4":
            centre = -4.0 - (sl * k2 if name == "helmholtz" else 0.0)
            wr = (am, ap) if geom == 1 else (1.0, 1.0)
            wz = (am, ap) if geom == 2 else (1.0, 1.0)
            return (wz[0] * at(0, -1) + wr[0] * at(-1, 0) + centre * at(0, 0) + wr[1] * at(1, 0)
                    + wz[1] * at(0, 1)), centre
        if geom:
            em = 4 * (-2 + 9 * i - 16 * i * i + 8 * i ** 3) / q ** 3
            ep = 4 * (1 + i - 8 * i * i + 8 * i ** 3) / q ** 3
            cc = -16 * (1 - 5 * i + 5 * i * i) / q ** 2
        else:
            em, ep, cc = 4.0, 4.0, -20.0
        v = cc * at(0, 0)
        for t in (-1, 1):  # along the axis (or the second dimension), then the radial sides
            a = (lambda r: at(r, t)) if geom != 2 else (lambda r: at(t, r))
            v = v + am * a(-1) + 4.0 * a(0) + ap * a(1)
        v = v + (em * at(-1, 0) + ep * at(1, 0) if geom != 2 else em * at(0, -1) + ep * at(0, 1))
        return v / 6.0, cc / 6.0

    def colours(self, name):
        o = self.valid
        p = [(o // s) % S for s in self.strides]
        if name != "laplacian4":
            par = sum(p) + self.D - 1
            return [o[(par & 1) == c] for c in (0, 1)]
        z = p[2] + 1 if self.D == 3 else 0
        return [o[(((p[0] ^ ((c >> 1) + z)) & 1) == 0) & (((p[1] ^ ((c & 1) + z)) & 1) == 0)] for c in range(4)]

    def smooth(self, u, b, l, n, op, bc, omega):
        blk, co = self.blocks[l], self.coords[l]
        for _ in range(n):
            for cells in self.colours(op[0]):
                v, diag = self.lhs(u, l, blk, co, cells, op)
                i = (blk[:, None], cells)
                u[i] = u[i] - omega * (v + (op[1] / 4 ** l) * b[i]) / diag
                self.fill(u, l, bc, 3)

    def coarse_rhs(self, u, b, l, op):
        """The FAS right-hand side of level l - 1 under level l's children."""
        r = torch.zeros_like(u)
        blk = self.blocks[l]
        v, _ = self.lhs(u, l, blk, self.coords[l], self.valid, op)
        r[blk[:, None], self.valid] = -(b[blk[:, None], self.valid] + v / (op[1] / 4 ** l))
        self.restrict(r, l)
        blk = self.blocks[l - 1]
        v, _ = self.lhs(u, l - 1, blk, self.coords[l - 1], self.valid, op)
        new = torch.zeros_like(u)
        new[blk[:, None], self.valid] = v / (op[1] / 4 ** (l - 1))
        for _, coarse, co, _, _, _ in self.kids[l]:
            i = (coarse[:, None], co)
            b[i] = -(r[i] + new[i])

    def finest(self):
        return max(l for l, b in enumerate(self.blocks) if len(b))

    def prolong(self, u, e, l):
        for fine, coarse, _, _, js, sides in self.kids[l]:
            i = (fine[:, None], self.valid)
            u[i] = self._interp(e, coarse, js, sides) + u[i]

    def vcycle(self, u, b, op, bc, sweeps, lmax=None, omega=1.0, top_omega=None):
        lmax = self.finest() if lmax is None else lmax
        old = {}
        for l in range(lmax, 0, -1):
            self.smooth(u, b, l, sweeps["ndown"], op, bc, omega)
            self.restrict(u, l)
            self.fill(u, l - 1, bc)
            old[l - 1] = u[self.blocks[l - 1]].clone()
            self.coarse_rhs(u, b, l, op)
        self.smooth(u, b, 0, sweeps["ntop"], op, bc, top_omega or omega)
        e = torch.zeros_like(u)
        for l in range(1, lmax + 1):
            blk = self.blocks[l - 1]
            e[blk] = u[blk] - old[l - 1]
            self.fill(e, l - 1, bc)
            self.prolong(u, e, l)
            self.fill(u, l, bc)
            self.smooth(u, b, l, sweeps["nup"], op, bc, omega)
            self.fill(u, l, bc)

    def fmg(self, u, b, op, bc, sweeps, omega=1.25):
        lmax = self.finest()
        for l in range(lmax, 0, -1):
            self.restrict(u, l)
            self.fill(u, l - 1, bc)
            self.coarse_rhs(u, b, l, op)
        e, old = torch.zeros_like(u), None
        for l in range(lmax + 1):
            # level l - 1's correction is against its value before its prolongation
            before = u[self.blocks[l]].clone()
            if l > 0:
                blk = self.blocks[l - 1]
                e[blk] = u[blk] - old
                self.fill(e, l - 1, bc)
                self.prolong(u, e, l)
            self.fill(u, l, bc)
            self.vcycle(u, b, op, bc, sweeps, l, omega)
            old = before
        return u

    def solution(self, b, op, bc, tol=1e-12):
        """The discrete solution: V-cycles with a well-converged coarsest level."""
        u, b = torch.zeros_like(b), b.clone()
        leaf = self.P.leaf.reshape(b.shape)
        last = math.inf
        for _ in range(60):
            before = u.clone()
            self.vcycle(u, b, op, bc, dict(ndown=2, ntop=40, nup=2), top_omega=1.75)
            step = float((u - before)[leaf].norm() / u[leaf].norm().clamp_min(1e-300))
            if step < tol or (step < 1e-10 and step > 0.8 * last):
                break
            last = step
        for l in range(self.finest(), 0, -1):
            self.restrict(u, l)
        for l in range(len(self.blocks)):
            self.fill(u, l, bc)
        return u


def exact(case, seed):
    kind = case["kind"]
    if kind in ("cnn_train", "cnn_forward"):
        return _exact_cnn(case, seed)
    st = prepare(case, seed)
    P = st.P
    if kind == "freebc":
        return _exact_freebc(st)
    X = Blocks(P)
    if kind == "stage":
        return _exact_stage(st, X)
    shape = (P.nblk,) + (S,) * P.D
    if kind == "batch":
        if P.nblk > 4000:
            return None
        terms = [(("laplacian", P.s, 0.0, case["geom"]), gen.BC_POISSON)]
        terms += [(("helmholtz", P.h1 * P.h1, lam * lam, case["geom"]), gen.BC_PHOTO) for lam in LAMBDAS]
        return {"u": [X.solution(b.reshape(P.nblk, -1), op, bc).reshape(shape) for b, (op, bc) in zip(st.b, terms)]}
    op = (case["op"], st.s, st.k2, st.geom)
    b = st.b.reshape(P.nblk, -1)
    if kind == "solve":
        return None if P.nblk > 12000 else {"u": X.solution(b, op, st.bc).reshape(shape)}
    u, b = torch.zeros_like(b), b.clone()
    if kind == "fmg":
        X.fmg(u, b, op, st.bc, case)
    else:
        for _ in range(case["cycles"]):
            X.vcycle(u, b, op, st.bc, case)
    return {"u": u.reshape(shape)}


def _exact_cnn(case, seed):
    st = prepare(case, seed)
    th = torch.from_numpy(st.net.get_params()).cuda()
    theta = th.to(torch.bfloat16).double()  # the packed weights; the biases stay FP32
    leaves, at, cin, layers = [], 0, 2, []
    for k in range(6):
        cout = 32 if k < 5 else 1
        w = theta[at:at + 9 * cout * cin].reshape(9, cout, cin).clone().requires_grad_(True)
        at += 9 * cout * cin
        bias = th[at:at + cout].double().clone().requires_grad_(True)
        at += cout
        leaves += [w, bias]
        layers.append((w, bias))
        cin = 32
    train = case["kind"] == "cnn_train"
    n, step, ys = case["samples"], 256, []
    for i in range(0, n, step):
        a = st.x[i:i + step].double().reshape(-1, S, S, 2).permute(0, 3, 1, 2)
        for k, (w, bias) in enumerate(layers):
            a = torch.nn.functional.conv2d(a, w.permute(1, 2, 0).reshape(w.shape[1], w.shape[2], 3, 3), bias, padding=1)
            a = torch.relu(a) if k < 5 else a
        y = a[:, 0, G:G + M, G:G + M].reshape(-1, M * M)
        ys.append(y.detach())
        if train:
            ((y - st.t[i:i + step].double()) ** 2).sum().div(n * M * M).backward()
    if not train:
        return {"y": torch.cat(ys)}
    return {"y": torch.cat(ys), "grad": torch.cat([p.grad.reshape(-1) for p in leaves]).cpu().numpy()}


def _exact_freebc(st):
    P, n, level = st.P, len(st.f), st.case["level"]
    u, q = st.u.cpu().numpy(), st.q0.cpu().numpy()
    outer = np.zeros(n)
    for l, layer in enumerate(P.tree):
        p = 2 ** (level - l - 1)
        for (cr, cz), blk in layer.index.items():
            if cr == layer.domain[0]:
                i0 = p * (cz - 1) * M
                outer[i0:i0 + p * M] = np.repeat(u[blk - 1, G:G + M, G + M - 1] / (P.h1 / 2 ** l), p)
    k = torch.arange(n, device="cuda")

    def dst(x, three):
        """FFTW's RODFT10 (DST-II) or RODFT01 (DST-III), by direct sums."""
        x, out = torch.as_tensor(x, device="cuda"), []
        for i in range(0, n, 1024):
            r = k[i:i + 1024, None]
            arg = (k[None, :] + 1) * (2 * r + 1) if three else (2 * k[None, :] + 1) * (r + 1)
            sn = torch.sin((math.pi / (2 * n)) * (arg % (4 * n)).double())
            if three:
                sn[:, n - 1] *= 0.5
            out.append(2.0 * (sn @ x))
        return torch.cat(out).cpu().numpy()

    b = dst(st.f * dst(outer, False), True) * P.h1 / 2 ** (level - 1) / 2
    for l, layer in enumerate(P.tree):
        p, sl = 2 ** (level - l - 1), P.s / 4 ** l
        for e in P.conn.boundary[l]:
            if tuple(e["face"]) != (1, 0):
                continue
            cr, cz = layer.coord[int(e["block"])]
            i0 = p * (cz - 1) * M
            q[e["block"] - 1, G:G + M, G + M - 1] += (2 * abs(1 + 1 / (2 * M * cr - 1)) / sl
                                                      * b[i0:i0 + p * M].reshape(M, p).mean(axis=1))
        for e in P.conn.refboundary[l]:
            cr, cz = layer.coord[int(e["fine"])]
            if cr != layer.domain[0]:
                continue
            d = int(e["face"][1])
            i = G + 1 if d == -1 else M + G
            j = (cz - 1) * M + i - G
            first = p * j if d == 1 else p * (j - 3) - 1
            J = (M * cr - 1) // 2 + 1
            q[e["fine"] - 1, i - 1, G + M - 1] += 0.5 * abs(1 + 1 / (2 * J - 1)) / sl * b[first:first + 2 * p].mean()
    return {"q": q, "b": b}


def _exact_stage(st, X):
    P, tr = st.P, MINIMAL
    n = P.nblk
    flat = lambda f: f.reshape(n, -1).clone()  # noqa: E731
    ne, nion, phi = flat(st.ne), flat(st.nion), flat(st.phi)
    zeros = lambda: torch.zeros_like(ne)  # noqa: E731
    q, eabs, dne, dni = zeros(), zeros(), zeros(), zeros()
    V = X.valid
    every = torch.cat([b for b in X.blocks])[:, None]
    q[every, V] = nion[every, V] - ne[every, V]
    for l in range(X.finest(), 0, -1):
        X.restrict(q, l)
        X.restrict(ne, l)
    for l in range(len(X.blocks)):
        X.fill(ne, l, BC_DENSITY, copy_interp=True)
        X.fill(phi, l, gen.BC_POISSON)
    e, flux = (torch.zeros((n, 2, (S + 1) ** 2), dtype=torch.float64, device="cuda") for _ in range(2))
    faces = [X._offsets([np.arange(G, G + M + 1), np.arange(G, G + M)]),
             X._offsets([np.arange(G, G + M), np.arange(G, G + M + 1)])]
    big = lambda o: o % S + (S + 1) * (o // S)  # noqa: E731  (offsets in the 21 x 21 layout)
    for l, blk in enumerate(X.blocks):
        h = P.h1 / 2 ** l
        i = blk[:, None]
        for d in (0, 1):
            o = faces[d]
            e[i, d, big(o)] = (phi[i, o - X.strides[d]] - phi[i, o]) / h + float(st.eb[d])
        s2 = sum((e[i, d, big(V)] + e[i, d, big(V + X.strides[d])]) ** 2 / 4 for d in (0, 1))
        eabs[i, V] = s2.sqrt()
    for l in range(len(X.blocks)):
        X.fill(eabs, l, BC_EXTRAPOLATE)
    maxdt = torch.full((1,), math.inf, dtype=torch.float64, device="cuda")
    leaf = [torch.as_tensor([b - 1 for c, b in layer.index.items() if P.tree.isleaf(layer.level, c)], dtype=torch.int64,
                            device="cuda") for layer in P.tree]
    for l, blk in enumerate(leaf):
        if not len(blk):
            continue
        h, i = P.h1 / 2 ** l, blk[:, None]
        for d in (0, 1):
            o, w = faces[d], X.strides[d]
            ev = (eabs[i, o] + eabs[i, o - w]) / 2
            v = -e[i, d, big(o)] * tr["mu"]
            neg = torch.signbit(v)
            nd = torch.where(neg, ne[i, o - w], ne[i, o])
            nu = torch.where(neg, ne[i, o], ne[i, o - w])
            nu2 = torch.where(neg, ne[i, o + w], ne[i, o - 2 * w])
            a, b = nu - nu2, nd - nu
            lim = torch.where((10 * a).abs() > (4 * b).abs(), b / 3 + a / 6, a)
            lim = torch.where(a.abs() > (4 * b).abs(), b, lim)
            lim = torch.where(a * b < 0, torch.zeros_like(a), lim)
            F = v * (nu + lim)
            maxwell = (gen.EPSILON_0 / gen.ELEMENTARY_CHARGE) * ev / F.abs()
            F = F + tr["D"] * (ne[i, o - w] - ne[i, o]) / h
            flux[i, d, big(o)] = F
            m = torch.minimum(h / v.abs(), maxwell).min().clamp_max(h * h / tr["D"] / 4)
            maxdt = torch.minimum(maxdt, m)
    for l in range(1, len(X.blocks)):
        for r in P.conn.refboundary[l]:
            f, sb = r["face"], r["subblock"]
            d = 0 if f[0] else 1
            up = f[d] > 0
            fn, cn, tan = (2 + M if up else 2), (2 if up else 2 + M), 2 + 8 * (int(sb[1 - d]) - 1)
            fine, coarse = (flux[int(r[k]) - 1, d].view(S + 1, S + 1) for k in ("fine", "coarse"))
            src = fine[G:G + M, fn] if d == 0 else fine[fn, G:G + M]
            mean = src.reshape(8, 2).sum(1) / 2
            if d == 0:
                coarse[tan:tan + 8, cn] = mean
            else:
                coarse[cn, tan:tan + 8] = mean
    for l, blk in enumerate(leaf):
        if not len(blk):
            continue
        h, i = P.h1 / 2 ** l, blk[:, None]
        E, n1 = eabs[i, V], ne[i, V]
        chem = tr["mu"] * E * n1 * (tr["ai"] * torch.exp(-tr["Ei"] / E) - tr["aa"] * torch.exp(-tr["Ea"] / E))
        dni[i, V] = chem
        cr = torch.as_tensor([P.tree[l].coord[int(b) + 1][0] for b in blk.cpu()], device="cuda")
        J = (M * (cr[:, None] - 1) + (V % S)[None, :] - 1).double()
        v = chem + (1 - 1 / (2 * J - 1)).abs() * flux[i, 0, big(V)] / h - (1 + 1 / (2 * J - 1)) * flux[i, 0, big(V + 1)] / h
        dne[i, V] = v + flux[i, 1, big(V)] / h - flux[i, 1, big(V + S)] / h
    shape = st.ne.shape
    out = {"q": q, "eabs": eabs, "dne": dne, "dni": dni, "n1": ne + dne * STAGE_DT, "n1i": nion + dni * STAGE_DT}
    out = {k: v.reshape(shape) for k, v in out.items()}
    return {**out, "e": e.reshape(st.e.shape), "flux": flux.reshape(st.e.shape), "maxdt": maxdt}
