"""The work a user of this framework has it do, as measured cases.

A case is one of these programs (its "kind"):

  eager     airfoil's outer iterations called loop by loop, every update's rms back on the host before the next
            call, as a generated OP2 main runs them; the device datasets are read in place afterwards
  graph     the same iteration (rotated: res_calc first, the next iteration's save_soln + adt_calc last) captured
            once as a CUDA graph and launched again and again
  residual  adt_calc, res_calc and bres_calc without an update: a residual evaluation
  jac       jac1 or jac2: res and update, the sum and the maximum back on the host after every update, or the
            iteration captured as a graph
  batch     a group of independent airfoil solves iterated together, every solve's q copied to the host
  solve     one airfoil solve through the C++ application from host arrays to host results: declarations,
            plans, iterations with the rms returned, q fetched
  plan      op_plan_core of res_calc on a newly declared mesh, every array of the plan in host memory

"cells" come as I x J of the NACA0012 C-mesh (3 I J cells); NN x NN is jac's grid.
"""
import ctypes as C
import math
import weakref

import numpy as np
import torch

from oplus2_matlab_b200 import api, apps, group
from oplus2_matlab_b200 import mesh as M

SEED = 20261203  # of the scrambled numberings and the mix of a batch
INDS = [0, 0, 1, 1, 2, 2, 3, 3]  # res_calc: x, q, adt read, res incremented


def listed():
    return [
        # the reference's own small mesh: launches, latency and the host's share of a loop call
        dict(name="eager 7k f32", kind="eager", I=40, J=60, scramble=False, f64=False, seq=False, coloured=False, n=40),
        # the headline configuration, called as an application calls it
        dict(name="eager 720k f32", kind="eager", I=400, J=600, scramble=False, f64=False, seq=False, coloured=False, n=20),
        # the largest configuration: 2.88M cells whose numbering has no locality (a mesh generator's output)
        dict(name="eager 2.88M scrambled f32", kind="eager", I=800, J=1200, scramble=True, f64=False, seq=False, coloured=False, n=4),
        # the verification mode: rms summed in the sequential back-end's order, bit for bit
        dict(name="eager 180k seq f32", kind="eager", I=200, J=300, scramble=False, f64=False, seq=True, coloured=False, n=4),
        # the reference's two-level colouring, in double precision, at the headline size
        dict(name="eager 720k coloured f64", kind="eager", I=400, J=600, scramble=False, f64=True, seq=False, coloured=True, n=5),
        # a captured iteration, double precision, a ragged size
        dict(name="graph 407k f64", kind="graph", I=301, J=451, scramble=False, f64=True, n=20),
        # residual evaluation of a ragged mesh (convergence monitor, outer nonlinear solver)
        dict(name="residual 281k f32", kind="residual", I=250, J=375, scramble=False, f64=False, n=8),
        # jac1 at its benchmark size, reductions returned after every update
        dict(name="jac1 512 eager", kind="jac", variant=1, NN=512, graph=False, n=40),
        # jac2 (double matrix, strided float vectors) captured, an odd size
        dict(name="jac2 385 graph", kind="jac", variant=2, NN=385, graph=True, n=40),
        # a mix of solves sharing the GPU
        dict(name="batch of 12 f32", kind="batch", count=12, cmin=20000, cmax=400000, f64=False, n=30),
        # a short solve of a small mesh, host arrays in and out: uploads and plan building count
        dict(name="solve 45k f32", kind="solve", I=100, J=150, scramble=False, f64=False, n=100),
        # the execution plan of the headline loop for a mesh of odd size
        dict(name="plan 406k", kind="plan", I=301, J=450, scramble=False, part_size=0),
    ]


def _dims(rng, lo, hi):
    """I, J of a C-mesh of lo..hi cells, log-uniform, sides between 1:3 and 3:1 of the usual aspect."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    j = math.sqrt(cells / 2.0) * math.exp(rng.uniform(-0.5, 0.5))
    return max(3, round(cells / (3.0 * j))), max(5, round(j))


def draw(rng):
    kind = rng.choice(["eager", "eager", "eager", "graph", "residual", "jac", "batch", "solve", "plan"])
    flip = lambda p: rng.random() < p  # noqa: E731
    if kind == "eager":
        seq, coloured, scramble = flip(0.25), flip(0.25), flip(0.25)
        top = 180e3 if seq else 300e3 if coloured and scramble else 800e3
        i, j = _dims(rng, 3e3, top)
        f64 = flip(0.4)
        most = int(12e6 / (3 * i * j * (2 if f64 else 1)))
        return dict(kind=kind, I=i, J=j, scramble=scramble, f64=f64, seq=seq, coloured=coloured,
                    n=rng.randint(2, 4) if seq else max(2, min(most, rng.randint(5, 20))))
    if kind == "graph":
        i, j = _dims(rng, 3e3, 800e3)
        f64 = flip(0.5)
        most = int(12e6 / (3 * i * j * (2 if f64 else 1)))
        return dict(kind=kind, I=i, J=j, scramble=flip(0.25), f64=f64, n=max(4, min(most, rng.randint(10, 40))))
    if kind == "residual":
        i, j = _dims(rng, 3e3, 1000e3)
        return dict(kind=kind, I=i, J=j, scramble=flip(0.25), f64=flip(0.4), n=rng.randint(4, 16))
    if kind == "jac":
        nn = round(math.exp(rng.uniform(math.log(20), math.log(900))))
        return dict(kind=kind, variant=rng.choice([1, 2]), NN=nn, graph=flip(0.5), n=2 * rng.randint(10, 30))
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(3, 12), cmin=rng.randint(4000, 20000), cmax=rng.randint(60000, 400000),
                    f64=flip(0.3), n=rng.randint(10, 40))
    i, j = _dims(rng, 5e3, 300e3)
    if kind == "solve":
        return dict(kind=kind, I=i, J=j, scramble=flip(0.2), f64=flip(0.4), n=rng.randint(30, 150))
    return dict(kind=kind, I=i, J=j, scramble=flip(0.2), part_size=rng.choice([0, 0, 128, 256]))


# ------------------------------------------------------------------ inputs

_meshes = {}


def _mesh(i, j, scramble=False):
    """The mesh a program has read from its grid file; the last few are kept."""
    key = (i, j, scramble)
    if key not in _meshes:
        while len(_meshes) >= 16:
            _meshes.pop(next(iter(_meshes)))
        _meshes[key] = M.naca0012(i, j, scramble=scramble)
    return _meshes[key]


def _real(case):
    return np.float64 if case.get("f64") else np.float32


def _q0(case, mesh, seed):
    """A flow field under way: the free stream with a small disturbance in every cell."""
    t = _real(case)
    qinf = np.asarray(apps.airfoil_consts(t)["qinf"], np.float64)
    noise = np.random.default_rng(seed).uniform(-0.01, 0.01, (mesh.ncell, 4))
    q = qinf * (1.0 + noise)
    q[:, 2] = qinf[1] * noise[:, 2]
    return q.astype(t)


def _jac_mesh(case, seed):
    m = M.jac(case["NN"], case["variant"])
    noise = np.random.default_rng(seed).uniform(0.0, 0.01, m.r.shape)
    m.r = (m.r + noise).astype(np.float32)
    return m


def _flows(case, seed):
    """(I, J, mach, alpha) of every solve of a batch: the sizes by the case, the flow conditions by the seed."""
    rng = np.random.default_rng(seed)
    sizes = group.draw_instances(case["count"], SEED, case["cmin"], case["cmax"])
    return [(i, j, rng.uniform(0.3, 0.7), rng.uniform(-2.0, 6.0)) for i, j, _, _ in sizes]


# ------------------------------------------------------------------- state

_live = set()  # states that hold declarations of the library


class _State:
    pass


def _gone(key, graphs):
    for g in graphs:
        api.lib().op2b_graph_destroy(g)
    _live.discard(key)


def _settings(deferred=False, seq=False, coloured=False):
    """How the loops run; the previous problems' declarations go when none of them is in use."""
    if not _live:
        api.op_exit()
    api.set_error_mode(api.ERRORS_RETURN)
    api.clear_error()
    api.set_strategy(api.STRATEGY_COLOURED if coloured else api.STRATEGY_GATHER)
    api.set_reduction(api.REDUCE_SEQ if seq else api.REDUCE_TREE)
    api.set_gbl_deferred(1 if deferred else 0)


def _begin(state, **how):
    _settings(**how)
    api.op_init()
    state.graphs = []
    _live.add(id(state))
    weakref.finalize(state, _gone, id(state), state.graphs)


def _ok():
    if api.last_error():
        raise RuntimeError(api.last_error())


class _Dev:
    def __init__(self, ptr, shape, f64):
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr="<f8" if f64 else "<f4", version=2)


def _view(dat):
    """A dataset's device copy, read in place."""
    d = dat.contents
    return torch.as_tensor(_Dev(d.data_d, (d.set.contents.size, d.dim), d.type == b"double"), device="cuda")


def _bind(name, set_, args):
    arr = (api.op_arg * len(args))(*args)
    return name.encode(), set_, len(args), arr


ROTATED = ("res_calc", "bres_calc", "update", "adt_calc", "res_calc", "bres_calc", "update", "save_soln", "adt_calc")


def prepare(case, seed):
    s = _State()
    s.case, kind = case, case["kind"]
    lib = api.lib()
    if kind in ("eager", "graph", "residual"):
        mesh = _mesh(case["I"], case["J"], case["scramble"])
        _begin(s, seq=case.get("seq", False), coloured=case.get("coloured", False))
        q = _q0(case, mesh, seed)
        s.app = apps.Airfoil(mesh, _real(case), state=dict(q=q, qold=q, res=np.zeros_like(q), adt=np.zeros((mesh.ncell, 1))))
        if kind == "graph":
            s.app.iteration()  # builds the plans
            s.app.loop("save_soln")
            s.app.loop("adt_calc")
            api.sync()
            lib.op2b_capture_begin(0)
            for name in ROTATED:
                s.app.loop(name)
            s.graph = lib.op2b_capture_end()
            _ok()
            s.graphs.append(s.graph)
    elif kind == "jac":
        _begin(s, deferred=case["graph"])
        s.app = apps.Jac(_jac_mesh(case, seed), case["variant"])
        s.calls = _bind("res", s.app.edges, s.app.res_args), _bind("update", s.app.nodes, s.app.upd_args)
        if case["graph"]:
            res, update = s.calls
            for call in (res, update, res):  # builds the plans
                lib.op2b_par_loop(*call)
            api.sync()
            lib.op2b_capture_begin(0)
            for call in (update, res, update, res):
                lib.op2b_par_loop(*call)
            s.graph = lib.op2b_capture_end()
            _ok()
            s.graphs.append(s.graph)
    elif kind == "batch":
        _settings()
        s.group = group.Group(_real(case))
        s.ids, s.q = [], []
        for i, j, mach, alpha in _flows(case, seed):
            mesh = _mesh(i, j)
            s.ids.append(s.group.add(mesh, mach, alpha, 1 << 18))
            s.q.append(torch.empty((mesh.ncell, 4), dtype=torch.float64 if case["f64"] else torch.float32, pin_memory=True).numpy())
        s.group.run(1)  # the solves join
        s.group.sync()
    elif kind == "solve":
        _settings()
        s.mesh = _mesh(case["I"], case["J"], case["scramble"])
        rng = np.random.default_rng(seed)
        s.mach, s.alpha = rng.uniform(0.3, 0.7), rng.uniform(-2.0, 6.0)
        s.q = torch.empty((s.mesh.ncell, 4), dtype=torch.float64 if case["f64"] else torch.float32, pin_memory=True).numpy()
    elif kind == "plan":
        _settings()
        mesh = _mesh(case["I"], case["J"], case["scramble"])
        # the plan of a mesh whose cells are numbered from another one: another seed's plan is another plan
        s.mesh, s.shift = mesh, 1 + seed % (mesh.ncell - 1)
        s.ecell = ((mesh.ecell + s.shift) % mesh.ncell).astype(np.int32)
        s.dats = [np.zeros((mesh.nnode, 2), np.float32)] + [np.zeros((mesh.ncell, d), np.float32) for d in (4, 1, 4)]
    return s


# --------------------------------------------------------------------- run

def _plan(s):
    if not _live:
        api.op_exit()  # the previous plan, and the arrays that were returned from it
    m = s.mesh
    api.op_init()
    nodes, edges, cells = (api.op_decl_set(n, k) for n, k in ((m.nnode, "nodes"), (m.nedge, "edges"), (m.ncell, "cells")))
    pedge = api.op_decl_map(edges, nodes, 2, m.edge, "pedge")
    pecell = api.op_decl_map(edges, cells, 2, s.ecell, "pecell")
    x, q, adt, res = (api.op_decl_dat(set_, a.shape[1], "float", a, k)
                      for set_, a, k in zip((nodes, cells, cells, cells), s.dats, ("p_x", "p_q", "p_adt", "p_res")))
    args = [api.op_arg_dat(x, 0, pedge, 2, "float", api.OP_READ), api.op_arg_dat(x, 1, pedge, 2, "float", api.OP_READ),
            api.op_arg_dat(q, 0, pecell, 4, "float", api.OP_READ), api.op_arg_dat(q, 1, pecell, 4, "float", api.OP_READ),
            api.op_arg_dat(adt, 0, pecell, 1, "float", api.OP_READ), api.op_arg_dat(adt, 1, pecell, 1, "float", api.OP_READ),
            api.op_arg_dat(res, 0, pecell, 4, "float", api.OP_INC), api.op_arg_dat(res, 1, pecell, 4, "float", api.OP_INC)]
    p = api.op_plan_core("res_calc", edges, s.case["part_size"], args, INDS)
    _ok()
    p, arr = p.contents, np.ctypeslib.as_array
    nb, ni, n = p.nblocks, p.ninds, m.nedge
    out = dict(nblocks=p.nblocks, ncolors=p.ncolors, nshared=p.nshared, nthrcol=arr(p.nthrcol, (nb,)), thrcol=arr(p.thrcol, (n,)),
               offset=arr(p.offset, (nb,)), nelems=arr(p.nelems, (nb,)), blkmap=arr(p.blkmap, (nb,)),
               ncolblk=arr(p.ncolblk, (p.ncolors,)), ind_offs=arr(p.ind_offs, (nb * ni,)), ind_sizes=arr(p.ind_sizes, (nb * ni,)))
    for k in range(ni):
        out["ind_maps%d" % k] = arr(p.ind_maps[k], (p.nindirect[k],))
    for k in range(len(INDS)):
        out["loc_maps%d" % k] = arr(p.loc_maps[k], (n,))
    return out


def run(s):
    case, kind = s.case, s.case["kind"]
    n, lib = case.get("n"), api.lib()
    if kind == "eager":
        rms = s.app.iterate(n)
        api.sync()
        return dict(q=_view(s.app.p_q), qold=_view(s.app.p_qold), res=_view(s.app.p_res), adt=_view(s.app.p_adt), rms=rms)
    if kind == "graph":
        for _ in range(n):
            lib.op2b_graph_launch(s.graph)
        s.app.rms[0] = 0
        api.sync()
        return dict(q=_view(s.app.p_q), qold=_view(s.app.p_qold), res=_view(s.app.p_res), adt=_view(s.app.p_adt), rms=s.app.rms.copy())
    if kind == "residual":
        for _ in range(n):
            for name in ("adt_calc", "res_calc", "bres_calc"):
                s.app.loop(name)
        api.sync()
        return dict(adt=_view(s.app.p_adt), res=_view(s.app.p_res))
    if kind == "jac":
        a, loop = s.app, lib.op2b_par_loop
        sums = []
        if case["graph"]:
            for _ in range(n // 2):
                lib.op2b_graph_launch(s.graph)
            a.u_sum[0] = a.u_max[0] = 0
            api.sync()
            sums.append((float(a.u_sum[0]), float(a.u_max[0])))
        else:
            res, update = s.calls
            for _ in range(n):
                loop(*res)
                a.u_sum[0] = a.u_max[0] = 0
                loop(*update)
                sums.append((float(a.u_sum[0]), float(a.u_max[0])))
            api.sync()
        return dict(u=_view(a.p_u), du=_view(a.p_du), sums=np.array(sums, np.float32))
    if kind == "batch":
        s.group.run(n)
        s.group.sync()
        return [s.group.fetch_q(k, q) for k, q in zip(s.ids, s.q)]
    if kind == "solve":
        q, rms, _ = group.plain_solve(s.mesh, s.mach, s.alpha, n, _real(case), q_out=s.q)
        return dict(q=q, rms=rms.astype(_real(case)))
    return _plan(s)


# -------------------------------------------------------------------- work

def _airfoil_work(cells, n, f64, updates=2):
    """n outer iterations of airfoil: per update, every map, the coordinates, q, qold and adt read once, q and adt
    written once; once an iteration, qold written."""
    w = 8 if f64 else 4
    per_update = 2 * 16 + 16 + 2 * w + (4 + 4 + 4) * w + (1 + 1) * w  # 2 edges a cell, 16 bytes of maps each; pcell; x; q; adt
    return dict(bytes=float(cells) * n * (updates * per_update + 4 * w), flops=float(cells) * n * updates * (2 * 64 + 64 + 16))


def work(case):
    kind, n = case["kind"], case.get("n", 1)
    w = 8 if case.get("f64") else 4
    cells = 3 * case["I"] * case["J"] if "I" in case else 0
    if kind in ("eager", "graph"):
        return _airfoil_work(cells, n, case["f64"])
    if kind == "residual":  # maps, x, q read; adt written and read; res read and written
        return dict(bytes=float(cells) * n * (2 * 16 + 16 + 2 * w + 4 * w + 2 * w + 8 * w), flops=float(cells) * n * (2 * 64 + 64))
    if kind == "jac":  # A, the map, u, du and r read; u and du written
        nodes = (case["NN"] - 1) ** 2
        a, strides = (4, 4 * (2 + 2 + 1)) if case["variant"] == 1 else (8, 4 * (2 + 2 + 1))
        return dict(bytes=float(nodes) * n * (5 * (8 + a) + strides), flops=float(nodes) * n * (5 * 3 + 6))
    if kind == "batch":
        total = sum(3 * i * j for i, j, _, _ in group.draw_instances(case["count"], SEED, case["cmin"], case["cmax"]))
        d = _airfoil_work(total, n, case["f64"])
        return dict(bytes=d["bytes"] + 4.0 * w * total, flops=d["flops"])
    if kind == "solve":
        d = _airfoil_work(cells, n, case["f64"])
        return dict(bytes=d["bytes"] + cells * (48.0 + 2 * w + 8 * w), flops=d["flops"])
    # plan: both maps in; per edge thread colours and eight local indices out, the targets of four datasets
    return dict(bytes=2.0 * cells * (16 + 4 + 16) + 4 * 4.0 * cells * 1.2, flops=0.0)


# ------------------------------------------------------------------- exact

class _Flow:
    """airfoil's loops in 64 bits, plain torch."""

    def __init__(self, mesh, q, real, qinf=None):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev).to(torch.float64)  # noqa: E731
        k = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev).to(torch.int64)  # noqa: E731
        c = apps.airfoil_consts(real)
        self.gam, self.gm1, self.cfl, self.eps = (float(c[n]) for n in ("gam", "gm1", "cfl", "eps"))
        self.qinf = f(np.asarray(c["qinf"] if qinf is None else qinf, np.float64))
        self.x, self.edge, self.ecell = f(mesh.x(real)), k(mesh.edge), k(mesh.ecell)
        self.bedge, self.becell, self.cell = k(mesh.bedge), k(mesh.becell.reshape(-1)), k(mesh.cell)
        self.wall = (k(mesh.bound.reshape(-1)) == 1).unsqueeze(1)
        self.q = f(q)
        self.qold = self.q.clone()
        self.res = torch.zeros_like(self.q)
        self.adt = torch.zeros(mesh.ncell, dtype=torch.float64, device=dev)
        self.sum = 0.0

    def save_soln(self):
        self.qold = self.q.clone()

    def adt_calc(self):
        q, x = self.q, self.x[self.cell]
        u, v = q[:, 1] / q[:, 0], q[:, 2] / q[:, 0]
        c = torch.sqrt(self.gam * self.gm1 * (q[:, 3] / q[:, 0] - 0.5 * (u * u + v * v)))
        d = torch.roll(x, -1, 1) - x
        s = (u[:, None] * d[:, :, 1] - v[:, None] * d[:, :, 0]).abs() + c[:, None] * torch.sqrt((d * d).sum(2))
        self.adt = s.sum(1) / self.cfl

    def _side(self, q, d):
        p = self.gm1 * (q[..., 3] - 0.5 * (q[..., 1] ** 2 + q[..., 2] ** 2) / q[..., 0])
        vol = (q[..., 1] * d[:, 1] - q[..., 2] * d[:, 0]) / q[..., 0]
        flux = torch.stack([vol * q[..., 0], vol * q[..., 1] + p * d[:, 1], vol * q[..., 2] - p * d[:, 0],
                            vol * (q[..., 3] + p)], 1)
        return p, flux

    def res_calc(self):
        c1, c2 = self.ecell[:, 0], self.ecell[:, 1]
        d = self.x[self.edge[:, 0]] - self.x[self.edge[:, 1]]
        q1, q2 = self.q[c1], self.q[c2]
        mu = 0.5 * (self.adt[c1] + self.adt[c2]) * self.eps
        f = 0.5 * (self._side(q1, d)[1] + self._side(q2, d)[1]) + mu[:, None] * (q1 - q2)
        self.res.index_add_(0, c1, f)
        self.res.index_add_(0, c2, -f)

    def bres_calc(self):
        c = self.becell
        d = self.x[self.bedge[:, 0]] - self.x[self.bedge[:, 1]]
        q = self.q[c]
        p, flux = self._side(q, d)
        far = 0.5 * (flux + self._side(self.qinf.expand_as(q), d)[1]) + (self.adt[c] * self.eps)[:, None] * (q - self.qinf)
        zero = torch.zeros_like(p)
        self.res.index_add_(0, c, torch.where(self.wall, torch.stack([zero, p * d[:, 1], -p * d[:, 0], zero], 1), far))

    def update(self):
        d = self.res / self.adt[:, None]
        self.q = self.qold - d
        self.res = torch.zeros_like(d)
        self.sum += float((d * d).sum())

    def iteration(self):
        self.save_soln()
        for _ in range(2):
            self.adt_calc()
            self.res_calc()
            self.bres_calc()
            self.sum = 0.0
            self.update()
        return math.sqrt(self.sum / self.q.shape[0])

    def out(self, **more):
        return dict(q=self.q, qold=self.qold, res=self.res, adt=self.adt[:, None], **more)


def _free_stream(mach, alpha_deg):
    """Free stream of a flow condition (pressure and density one), the constants as the applications declare them."""
    gam = float(np.float32(1.4))
    u, a = math.sqrt(gam) * float(np.float32(mach)), math.radians(float(np.float32(alpha_deg)))
    return [1.0, u * math.cos(a), u * math.sin(a), 1.0 / (gam - 1.0) + 0.5 * u * u]


def _solve_exact(case, mesh, mach, alpha, n):
    qinf = _free_stream(mach, alpha)
    f = _Flow(mesh, np.tile(qinf, (mesh.ncell, 1)), _real(case), qinf)
    return f, [f.iteration() for _ in range(n)]


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind in ("eager", "graph", "residual"):
        mesh = _mesh(case["I"], case["J"], case["scramble"])
        f = _Flow(mesh, _q0(case, mesh, seed), _real(case))
        if kind == "eager":
            return f.out(rms=np.array([f.iteration() for _ in range(n)]))
        if kind == "residual":
            for _ in range(n):
                f.adt_calc()
                f.res_calc()
                f.bres_calc()
            return dict(adt=f.adt[:, None], res=f.res)
        f.iteration()
        f.save_soln()
        f.adt_calc()
        for _ in range(n):
            f.sum = 0.0
            for name in ROTATED:
                getattr(f, name)()
        return f.out(rms=np.array([f.sum]))
    if kind == "jac":
        m, v = _jac_mesh(case, seed), case["variant"]
        col = lambda a, k: torch.as_tensor(np.ascontiguousarray(np.asarray(a, np.float64).reshape(k, -1)[:, 0]))  # noqa: E731
        A, r, p = col(m.A, m.nedge), col(m.r, m.nnode), torch.as_tensor(m.pp.astype(np.int64))
        u, du, sums = torch.zeros_like(r), torch.zeros_like(r), []

        def res():
            du.index_add_(0, p[:, 0], A * u[p[:, 1]])

        def update():
            u.add_(du + r)
            du.zero_()
            return float((u * u).sum()), max(0.0, float(u.max()))
        res()
        if case["graph"]:
            update()
            res()
        for k in range(n):
            sums.append(update())
            if case["graph"] or k + 1 < n:
                res()
        if case["graph"]:  # a launch holds two updates: both add to the sum, the larger maximum stays
            sums = [(sums[-2][0] + sums[-1][0], max(sums[-2][1], sums[-1][1]))]
        wide = lambda a, w: torch.stack([a] + [torch.zeros_like(a)] * (w - 1), 1)  # noqa: E731
        return dict(u=wide(u, v), du=wide(du, 1 if v == 1 else 3), sums=np.array(sums))
    if kind == "batch":
        out = []
        for i, j, mach, alpha in _flows(case, seed):
            out.append(_solve_exact(case, _mesh(i, j), mach, alpha, n + 1)[0].q)
        return out
    if kind == "solve":
        rng = np.random.default_rng(seed)
        mach, alpha = rng.uniform(0.3, 0.7), rng.uniform(-2.0, 6.0)
        f, rms = _solve_exact(case, _mesh(case["I"], case["J"], case["scramble"]), mach, alpha, n)
        return dict(q=f.q, rms=np.array(rms))
    return None
