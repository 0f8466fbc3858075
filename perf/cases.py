"""Performance cases: what users of this framework run, through its public entry points.

A case is a dict of plain values. Its "kind" is one of

  march    the Airfoil time march: a field goes onto the declared mesh, the five
           op_par_loops run for some iterations with rms/maxerr/errloc read back
           after every update, and q and adt come back in the declared order
  loops    an application whose loops have no hand-written kernel (compiled at run
           time from its kernel source): diffusion on a node graph -- an edge loop
           with indirect increments, a direct loop with OP_INC and OP_MAX globals,
           and a boundary loop with indirect OP_WRITE, all called every iteration
  batch    iterations of many Airfoil instances of uneven size solved together
  predict  the learned warm start's inference on a mesh: the graph network's
           forward pass and the decoding to q
  train    one training step of that network: forward, loss, backward, AdamW
  layer    one linear layer of its MLPs (op2b_gemm_bf16): the forward product with
           bias and SiLU, the backward product with SiLU', the weight gradient
  plan     op_plan_get_stage for res_calc on a declared mesh
  job      a whole solve from host arrays: op_init, declarations, op_renumber,
           iterations, op_fetch_data, op_exit

Meshes are the seeded channel-with-bump quad meshes of op2b.mesh, in the order the
generator numbers them ("natural"), shuffled ("random"), or shuffled and renumbered
by op_renumber ("rcm").
"""
import functools
import gc
import math
import os
import sys
import weakref

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "op2-common_b200"))
from op2b import gnn as G  # noqa: E402
from op2b import lib as L  # noqa: E402
from op2b import mesh as M  # noqa: E402
from op2b.airfoil import Airfoil  # noqa: E402
from op2b.batch import AirfoilBatch, sample_instances  # noqa: E402

W = G.WIDTH


def listed():
    return [
        # the smallest mesh of the smoke check: launches, waits and the call path itself
        dict(name="march_24x12_f64", kind="march", I=24, J=12, dtype="f64", order="rcm", iters=50),
        # a mid-size ragged mesh, about the reference's own new_grid scale
        dict(name="march_601x299_f64", kind="march", I=601, J=299, dtype="f64", order="rcm",
             iters=20),
        # the benchmark's mesh
        dict(name="march_2400x1200_f64", kind="march", I=2400, J=1200, dtype="f64", order="rcm",
             iters=20),
        # the same mesh in the mixed form (float storage, double update)
        dict(name="march_2400x1200_f32", kind="march", I=2400, J=1200, dtype="f32", order="rcm",
             iters=20),
        # an application that does not call op_renumber (the reference's airfoil_plain)
        dict(name="march_1201x601_natural", kind="march", I=1201, J=601, dtype="f64",
             order="natural", iters=10),
        # user kernels on a large node graph
        dict(name="loops_1201x599_f64", kind="loops", I=1201, J=599, dtype="f64", dim=4,
             order="rcm", iters=10),
        # sixteen instances of 10K to 100K cells in their generator's order (as the training
        # data of the learned warm start is solved), FP32 phase
        dict(name="batch_16", kind="batch", n=16, lo=10_000, hi=100_000, mesh=0, fp32=True,
             iters=20),
        # the warm start's prediction at the evaluation mesh's scale
        dict(name="predict_481x239", kind="predict", I=481, J=239),
        # the training step the shipped network was trained with
        dict(name="train_200x100_b8", kind="train", I=200, J=100, batch=8, steps=8),
        # the edge MLP's first layer over a minibatch's messages (ragged row count)
        dict(name="layer_silu_200001", kind="layer", op="silu", rows=200_001, k=384, n=128),
        # the colouring plan of a renumbered mesh
        dict(name="plan_601x299", kind="plan", I=601, J=299, part=256, staging=1, order="rcm"),
        # a short whole solve from host arrays
        dict(name="job_600x300", kind="job", I=600, J=300, iters=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ij(rng, lo, hi):
    """A mesh of lo to hi cells (log-uniform), one to three times as long as high."""
    c = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = rng.uniform(1.0, 3.0)
    J = max(4, int(math.sqrt(c / a)))
    return max(4, int(c / J)), J


def draw(rng):
    kind = rng.choice(["march", "march", "march", "march", "loops", "loops", "batch", "predict",
                       "train", "layer", "plan", "job"])
    if kind == "march":
        order = rng.choice(["rcm", "rcm", "natural", "random"])
        I, J = _ij(rng, 200, 700_000 if order != "rcm" else 2_800_000)
        return dict(kind=kind, I=I, J=J, dtype=rng.choice(["f64", "f64", "f32"]), order=order,
                    iters=rng.randint(5, 20))
    if kind == "loops":
        I, J = _ij(rng, 400, 700_000)
        return dict(kind=kind, I=I, J=J, dtype=rng.choice(["f64", "f32"]), dim=rng.randint(1, 4),
                    order=rng.choice(["rcm", "natural", "random"]), iters=rng.randint(3, 10))
    if kind == "batch":
        n = _log(rng, 2, 64)
        hi = min(100_000, 600_000 // n)
        return dict(kind=kind, n=n, lo=max(200, hi // 10), hi=hi, mesh=rng.randint(1, 999),
                    fp32=rng.random() < 0.6, iters=rng.randint(5, 20))
    if kind == "predict":
        I, J = _ij(rng, 400, 115_000)
        return dict(kind=kind, I=I, J=J)
    if kind == "train":
        I, J = _ij(rng, 200, 20_000)
        return dict(kind=kind, I=I, J=J, batch=rng.randint(1, 8), steps=rng.randint(2, 8))
    if kind == "layer":
        op = rng.choice(["silu", "dsilu", "dw"])
        rows = _log(rng, 500, 200_000)
        k = rng.choice([8, 16, 128, 256, 384]) if op != "dsilu" else 128
        if op == "dw":
            rows = max(8, rows // 8 * 8)
        return dict(kind=kind, op=op, rows=rows, k=k, n=128)
    I, J = _ij(rng, 400, 170_000)
    if kind == "plan":
        return dict(kind=kind, I=I, J=J, part=rng.choice([64, 128, 256]),
                    staging=rng.choice([1, 4]), order=rng.choice(["rcm", "natural", "random"]))
    return dict(kind=kind, I=I, J=J, iters=rng.randint(20, 100))


# ---------------------------------------------------------------- shared pieces

class State:
    """What a case keeps between passes."""

    def __init__(self, case):
        self.case = dict(case)


_states = weakref.WeakSet()  # states declared in the present session
_open = False


def _session():
    """A library session for a new state.  Sets, maps and dats live until op_exit, so a
    session that no state uses any more is closed first."""
    global _open
    gc.collect()
    if _open and not len(_states):
        L.op_exit()
        _open = False
    if not _open:
        L.op_init()
        _open = True


@functools.lru_cache(maxsize=2)
def _mesh(I, J, order):
    return M.channel_bump(I, J, seed=1, permute=order != "natural")


def _np_type(case):
    return np.float64 if case["dtype"] == "f64" else np.float32


def _field(mesh, seed):
    """A flow field near freestream: qinf with a smooth perturbation of a few per cent."""
    rng = np.random.default_rng(seed)
    cen = mesh.x[mesh.cell[:, 0]]
    q = np.empty((mesh.ncell, 4))
    for m, v in enumerate(M.airfoil_constants()["qinf"]):
        a, b, ph = rng.uniform(1.0, 4.0), rng.uniform(1.0, 4.0), rng.uniform(0.0, 6.0)
        q[:, m] = (v if v else 0.2) * (1.0 + 0.03 * np.sin(a * cen[:, 0] + b * cen[:, 1] + ph))
    q[:, 2] -= 0.2
    return q


def _ints(a):
    return torch.from_numpy(np.ascontiguousarray(a, np.int32)).cuda()


def _pack(dat, rows, buf):
    if L.load().op2b_dat_pack(dat, rows.data_ptr(), rows.numel(), buf.data_ptr()) != 0:
        raise L.Op2Error(L.last_error())


def _unpack(dat, rows, buf):
    if L.load().op2b_dat_unpack(dat, rows.data_ptr(), 0, rows.numel(), buf.data_ptr()) != 0:
        raise L.Op2Error(L.last_error())


# ---------------------------------------------------------------- march

def _march_prepare(case, seed, s):
    _session()
    mesh, dt = _mesh(case["I"], case["J"], case["order"]), _np_type(case)
    q0 = _field(mesh, seed).astype(dt)
    s.app = Airfoil(mesh, dtype=dt, q0=q0)
    if case["order"] == "rcm":
        s.app.renumber(stats=False)
    s.rows = _ints(L.set_permutation(s.app.cells))
    s.q0 = torch.from_numpy(q0).cuda()
    s.q, s.adt = torch.empty_like(s.q0), torch.empty_like(s.q0[:, :1])
    _states.add(s)


def _march_run(s):
    _unpack(s.app.p_q, s.rows, s.q0)
    hist = s.app.iterate(s.case["iters"])
    _pack(s.app.p_q, s.rows, s.q)
    _pack(s.app.p_adt, s.rows, s.adt)
    return dict(q=s.q, adt=s.adt, rms=np.array([h[0] for h in hist]),
                maxerr=np.array([h[1] for h in hist]),
                errloc=np.array([h[2] for h in hist], np.int32))


def _march_exact(mesh, q0, iters, qinf=None):
    """The march in float64 torch; returns q, adt and the rms/maxerr histories."""
    k = M.airfoil_constants()
    gam, gm1, cfl, eps = k["gam"], k["gm1"], k["cfl"], k["eps"]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    qinf = dev(np.asarray(k["qinf"] if qinf is None else qinf, np.float64))
    x = dev(mesh.x.astype(np.float64))
    cell, edge, ecell = dev(mesh.cell).long(), dev(mesh.edge).long(), dev(mesh.ecell).long()
    bedge, bcell = dev(mesh.bedge).long(), dev(mesh.becell).long()
    wall = (dev(mesh.bound) == 1)[:, None]
    d_cell = [x[cell[:, (i + 1) % 4]] - x[cell[:, i]] for i in range(4)]
    d_edge = x[edge[:, 0]] - x[edge[:, 1]]
    d_bedge = x[bedge[:, 0]] - x[bedge[:, 1]]
    c1, c2 = ecell[:, 0], ecell[:, 1]

    def side(q, d):
        """(pressure, flux of q through the face d) of one side"""
        ri = 1.0 / q[..., 0]
        p = gm1 * (q[..., 3] - 0.5 * ri * (q[..., 1] ** 2 + q[..., 2] ** 2))
        v = ri * (q[..., 1] * d[:, 1] - q[..., 2] * d[:, 0])
        f = torch.stack([v * q[..., 0], v * q[..., 1] + p * d[:, 1], v * q[..., 2] - p * d[:, 0],
                         v * (q[..., 3] + p)], dim=-1)
        return p, f

    q, rms_h, max_h = dev(q0.astype(np.float64)), [], []
    for _ in range(iters):
        qold = q
        for _k in range(2):
            ri = 1.0 / q[:, 0]
            u, v = ri * q[:, 1], ri * q[:, 2]
            c = torch.sqrt(gam * gm1 * (ri * q[:, 3] - 0.5 * (u * u + v * v)))
            adt = sum(torch.abs(u * d[:, 1] - v * d[:, 0]) + c * d.norm(dim=1)
                      for d in d_cell) / cfl
            res = torch.zeros_like(q)
            q1, q2 = q[c1], q[c2]
            mu = (0.5 * eps * (adt[c1] + adt[c2]))[:, None]
            f = 0.5 * (side(q1, d_edge)[1] + side(q2, d_edge)[1]) + mu * (q1 - q2)
            res.index_add_(0, c1, f)
            res.index_add_(0, c2, -f)
            qb = q[bcell]
            p, fb = side(qb, d_bedge)
            fi = side(qinf.expand_as(qb), d_bedge)[1]
            far = 0.5 * (fb + fi) + (eps * adt[bcell])[:, None] * (qb - qinf)
            zero = torch.zeros_like(p)
            atw = torch.stack([zero, p * d_bedge[:, 1], -p * d_bedge[:, 0], zero], dim=-1)
            res.index_add_(0, bcell, torch.where(wall, atw, far))
            dq = res / adt[:, None]
            q = qold - dq
        rms_h.append(math.sqrt(float((dq * dq).sum()) / mesh.ncell))
        max_h.append(float((dq * dq).max()))
    return q, adt[:, None], np.array(rms_h), np.array(max_h)


def _march_case_exact(case, seed):
    mesh, dt = _mesh(case["I"], case["J"], case["order"]), _np_type(case)
    stored = M.Mesh(**{**mesh.__dict__, "x": mesh.x.astype(dt)})
    q, adt, rms, big = _march_exact(stored, _field(mesh, seed).astype(dt), case["iters"])
    return dict(q=q, adt=adt, rms=rms, maxerr=big, errloc=None)


def _march_work(cells, edges, nodes, bedges, iters, word):
    """Per half iteration: q and qold read, q written, coordinates and maps read."""
    step = 12 * word * cells + 2 * word * nodes + 16 * cells + 16 * edges + 16 * bedges
    return dict(bytes=2.0 * iters * step, flops=2.0 * iters * (75 * cells + 60 * edges))


def _sizes(I, J):
    return I * J, (I - 1) * J + I * (J - 1), (I + 1) * (J + 1), 2 * (I + J)


# ---------------------------------------------------------------- loops

_KAPPA, _WALL = 0.2, 0.25
_LOOPS = """
inline void diff_flux_%(s)s(const %(t)s *x1, const %(t)s *x2, const %(t)s *u1, const %(t)s *u2,
                            %(t)s *d1, %(t)s *d2) {
  const %(t)s dx = x1[0] - x2[0], dy = x1[1] - x2[1];
  const %(t)s w = scale / (dx * dx + dy * dy);
  for (int k = 0; k < %(d)d; k++) {
    const %(t)s f = w * (u2[k] - u1[k]);
    d1[k] += f;
    d2[k] -= f;
  }
}
inline void diff_step_%(s)s(%(t)s *u, %(t)s *du, double *rms, %(t)s *umax) {
  for (int k = 0; k < %(d)d; k++) {
    const %(t)s del = du[k];
    u[k] += del;
    du[k] = 0;
    *rms += (double)del * (double)del;
    if (u[k] > *umax) *umax = u[k];
  }
}
inline void diff_wall_%(s)s(%(t)s *u1, %(t)s *u2, const int *bound) {
  if (*bound == 1)
    for (int k = 0; k < %(d)d; k++) {
      u1[k] = (%(t)s)%(w)r;
      u2[k] = (%(t)s)%(w)r;
    }
}
"""


def _loops_scale(case):
    """A step well inside the explicit scheme's stability bound on this mesh."""
    h = min(2.0 / case["I"], 0.95 / case["J"])
    return float(np.float32(_KAPPA * h * h / 4.0))


def _loops_u0(case, seed):
    mesh = _mesh(case["I"], case["J"], case["order"])
    rng = np.random.default_rng(seed)
    k = rng.uniform(1.0, 5.0, (2, case["dim"]))
    return (np.sin(mesh.x @ k) + 0.1 * rng.standard_normal((mesh.nnode, case["dim"]))).astype(
        _np_type(case))


def _loops_prepare(case, seed, s):
    _session()
    mesh, dt, D = _mesh(case["I"], case["J"], case["order"]), _np_type(case), case["dim"]
    t = "double" if dt is np.float64 else "float"
    tag = "%s%d" % (case["dtype"], D)
    text = _LOOPS % dict(s=tag, t=t, d=D, w=_WALL)
    for name in ("flux", "step", "wall"):
        L.register_kernel("diff_%s_%s" % (name, tag), text)
    nodes = L.op_decl_set(mesh.nnode, "nodes")
    edges = L.op_decl_set(mesh.nedge, "edges")
    bedges = L.op_decl_set(mesh.nbedge, "bedges")
    pedge = L.op_decl_map(edges, nodes, 2, mesh.edge, "pedge")
    pbedge = L.op_decl_map(bedges, nodes, 2, mesh.bedge, "pbedge")
    u0 = _loops_u0(case, seed)
    x = L.op_decl_dat(nodes, 2, t, mesh.x.astype(dt), "x")
    s.p_u = L.op_decl_dat(nodes, D, t, u0, "u")
    du = L.op_decl_dat(nodes, D, t, None, "du")
    bound = L.op_decl_dat(bedges, 1, "int", mesh.bound, "bound")
    L.op_decl_const(1, t, _loops_scale(case), "scale")
    if case["order"] == "rcm":
        L.op_renumber(pedge, stats=False)
    s.rows = _ints(L.set_permutation(nodes))
    s.u0 = torch.from_numpy(u0).cuda()
    s.u = torch.empty_like(s.u0)
    s.rms, s.umax = np.zeros(1), np.zeros(1, dt)
    A, R, INC = L.op_arg_dat, L.OP_READ, L.OP_INC
    s.loops = [
        ("diff_flux_" + tag, edges,
         [A(x, 0, pedge, 2, t, R), A(x, 1, pedge, 2, t, R), A(s.p_u, 0, pedge, D, t, R),
          A(s.p_u, 1, pedge, D, t, R), A(du, 0, pedge, D, t, INC), A(du, 1, pedge, D, t, INC)]),
        ("diff_step_" + tag, nodes,
         [A(s.p_u, -1, L.OP_ID, D, t, L.OP_RW), A(du, -1, L.OP_ID, D, t, L.OP_RW),
          L.op_arg_gbl(s.rms, 1, "double", INC), L.op_arg_gbl(s.umax, 1, t, L.OP_MAX)]),
        ("diff_wall_" + tag, bedges,
         [A(s.p_u, 0, pbedge, D, t, L.OP_WRITE), A(s.p_u, 1, pbedge, D, t, L.OP_WRITE),
          A(bound, -1, L.OP_ID, 1, "int", R)])]
    _states.add(s)


def _loops_run(s):
    _unpack(s.p_u, s.rows, s.u0)
    rms, umax = [], []
    for _ in range(s.case["iters"]):
        s.rms[0], s.umax[0] = 0.0, -1e30
        for name, set_, args in s.loops:
            L.op_par_loop(name, set_, *args)
        rms.append(float(s.rms[0]))
        umax.append(float(s.umax[0]))
    _pack(s.p_u, s.rows, s.u)
    return dict(u=s.u, rms=np.array(rms), umax=np.array(umax))


def _loops_exact(case, seed):
    mesh = _mesh(case["I"], case["J"], case["order"])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    x = dev(mesh.x.astype(_np_type(case)).astype(np.float64))
    e = dev(mesh.edge).long()
    wall = dev(np.unique(mesh.bedge[mesh.bound == 1])).long()
    w = (_loops_scale(case) / ((x[e[:, 0]] - x[e[:, 1]]) ** 2).sum(1))[:, None]
    u, rms, umax = dev(_loops_u0(case, seed).astype(np.float64)), [], []
    for _ in range(case["iters"]):
        f = w * (u[e[:, 1]] - u[e[:, 0]])
        du = torch.zeros_like(u).index_add_(0, e[:, 0], f).index_add_(0, e[:, 1], -f)
        u = u + du
        rms.append(float((du * du).sum()))
        umax.append(float(u.max()))
        u[wall] = _WALL
    return dict(u=u, rms=np.array(rms), umax=np.array(umax))


# ---------------------------------------------------------------- batch

def _batch_specs(case, seed):
    """The case's mesh sizes with the seed's flow conditions."""
    rng = np.random.default_rng(seed)
    specs = sample_instances(case["n"], seed=case["mesh"], cells=(case["lo"], case["hi"]))
    return [dict(s, mach=float(rng.uniform(0.3, 0.7)), alpha=float(rng.uniform(-4.0, 6.0)),
                 bump=float(rng.uniform(0.0, 0.1))) for s in specs]


def _batch_mesh(p):
    return M.channel_bump(p["I"], p["J"], seed=p["seed"], bump=p["bump"], permute=False)


def _batch_prepare(case, seed, s):
    _session()
    specs = _batch_specs(case, seed)
    s.b = AirfoilBatch(specs, fp32=case["fp32"], renumber=False,
                       meshes=[_batch_mesh(p) for p in specs])
    # no instance changes its phase within a pass
    for key, v in (("tol", 0.0), ("promote_tol", 0.0), ("max_iter", 2.0 ** 30),
                   ("stall_window", 2.0 ** 30)):
        s.b.set(key, v)
    s.dats = s.b.d32 if case["fp32"] else s.b.d64
    q0 = L.op_fetch_data_idx(s.dats.p_q, 0, s.b.mesh.ncell - 1)
    s.rows = _ints(L.set_permutation(s.b.sets[3]))
    s.q0 = torch.from_numpy(q0).cuda()
    s.q = torch.empty_like(s.q0)
    weakref.finalize(s, _batch_close, s.b)
    _states.add(s)


def _batch_close(b):
    if _open:
        b.close()


def _batch_run(s):
    _unpack(s.dats.p_q, s.rows, s.q0)
    s.b.run(s.case["iters"], check_every=100)
    _pack(s.dats.p_q, s.rows, s.q)
    return dict(q=s.q, rms=s.b.stats()["rms_last"])


def _batch_exact(case, seed):
    dt = np.float32 if case["fp32"] else np.float64
    qs, rms = [], []
    for p in _batch_specs(case, seed):
        mesh = _batch_mesh(p)
        mesh.x = mesh.x.astype(dt)
        qinf = M.airfoil_constants(mach=p["mach"], alpha_deg=p["alpha"])["qinf"]
        q0 = np.repeat(qinf[None], mesh.ncell, 0).astype(dt)
        q, _, r, _ = _march_exact(mesh, q0, case["iters"], qinf=qinf.astype(dt))
        qs.append(q)
        rms.append(r[-1])
    return dict(q=torch.cat(qs), rms=np.array(rms))


# ---------------------------------------------------------------- the graph network

def _flow(seed):
    rng = np.random.default_rng(seed)
    return dict(mach=float(rng.uniform(0.3, 0.7)), alpha=float(rng.uniform(-4.0, 6.0)),
                bump=float(rng.uniform(0.0, 0.1)))


def _shipped_net():
    return os.path.join(os.path.dirname(os.path.abspath(G.__file__)), "data",
                        "gnn_airfoil_200x100.npz")


def _features(mesh, f, g):
    bf = lambda a: torch.from_numpy(a).to(torch.bfloat16)
    return bf(G.node_features(mesh, f["mach"], f["alpha"], f["bump"])), bf(
        G.edge_features(mesh, g))


def _predict_inputs(case, seed):
    f = _flow(seed)
    mesh = M.channel_bump(case["I"], case["J"], seed=7, bump=f["bump"])
    g = G.cell_graph(mesh)
    return (f, g) + _features(mesh, f, g)


def _predict_prepare(case, seed, s):
    _session()
    f, g, ni, ei = _predict_inputs(case, seed)
    s.net = G.GraphNet.load(_shipped_net())
    s.dg, s.ni, s.ei = s.net.upload_graph(g), ni.cuda(), ei.cuda()
    s.ms = torch.from_numpy(s.net.norm).cuda()
    s.qinf = torch.from_numpy(M.airfoil_constants(mach=f["mach"], alpha_deg=f["alpha"])["qinf"])
    s.qinf = s.qinf.cuda()
    s.q = torch.empty(g["N"], 4, dtype=torch.float64, device="cuda")
    _states.add(s)


def _predict_run(s):
    out = s.net.forward(s.dg, s.ni, s.ei, train=False)
    G._call("op2b_gnn_decode_q", s.dg["N"], out.data_ptr(), G.OUT, s.ms.data_ptr(),
            s.qinf.data_ptr(), s.q.data_ptr(), s.net.stream)
    return dict(out=out, q=s.q)


def _net_exact(p, off, steps, g, ni, ei):
    """The network's output in float64 torch; p: the flat parameters (a tensor)."""
    dev = lambda a: torch.from_numpy(a).cuda().long()
    src, dst = dev(g["src"]), dev(g["dst"])

    def mlp(name, h):
        for i in range(3):
            w0, b0, kin, nout = off[(name, i)]
            h = h @ p[w0:b0].view(nout, kin).T + p[b0:b0 + nout]
            if i < 2:
                h = h * torch.sigmoid(h)
        return h

    h, e = mlp("enc_node", ni.cuda().double()), mlp("enc_edge", ei.cuda().double())
    for l in range(steps):
        e = e + mlp("edge%d" % l, torch.cat([e, h[src], h[dst]], 1))
        agg = torch.zeros_like(h).index_add(0, dst, e)
        h = h + mlp("node%d" % l, torch.cat([h, agg], 1))
    return mlp("dec", h)


def _predict_exact(case, seed):
    f, g, ni, ei = _predict_inputs(case, seed)
    z = np.load(_shipped_net())
    off, _ = G.offsets(G.layout(steps=int(z["steps"])))
    with torch.no_grad():
        out = _net_exact(torch.from_numpy(z["params"].astype(np.float64)).cuda(), off,
                         int(z["steps"]), g, ni, ei)
    norm = torch.from_numpy(z["norm"].astype(np.float64)).cuda()
    qinf = M.airfoil_constants(mach=f["mach"], alpha_deg=f["alpha"])["qinf"]
    q = torch.from_numpy(qinf).cuda() + norm[:4] + norm[4:] * out[:, :4]
    return dict(out=out, q=q)


def _train_inputs(case, seed):
    """A minibatch: `batch` flows on one mesh family member each, smooth targets."""
    rng = np.random.default_rng(seed)
    g, nis, eis, tgs = None, [], [], []
    for b in range(case["batch"]):
        f = _flow(int(rng.integers(1 << 30)))
        mesh = M.channel_bump(case["I"], case["J"], seed=0, bump=f["bump"], permute=False)
        g = g or G.cell_graph(mesh)
        ni, ei = _features(mesh, f, g)
        k = rng.uniform(0.5, 3.0, (2, 4))
        tg = np.sin(mesh.x[mesh.cell[:, 0]] @ k + rng.uniform(0, 6, 4)) + f["mach"]
        nis.append(ni)
        eis.append(ei)
        tgs.append(torch.from_numpy(tg.astype(np.float32)))
    return g, nis, eis, tgs


def _train_prepare(case, seed, s):
    _session()
    g, nis, eis, tgs = _train_inputs(case, seed)
    s.net = G.GraphNet(steps=case["steps"], seed=seed)
    s.dg = s.net.upload_graph(G.replicate_graph(g, case["batch"]))
    s.ni, s.ei, s.tg = (torch.cat(v).cuda() for v in (nis, eis, tgs))
    _states.add(s)


def _train_run(s):
    # the learning rate of the first warm-up step
    loss = s.net.loss_grad(s.dg, s.ni, s.ei, s.tg)
    grad = s.net.g.clone()
    s.net.step(1e-5, weight_decay=1e-5)
    return dict(loss=loss, grad=grad)


def _train_exact(case, seed):
    g, nis, eis, tgs = _train_inputs(case, seed)
    lay = G.layout(steps=case["steps"])
    off, _ = G.offsets(lay)
    p = torch.from_numpy(G.init_params(lay, seed).astype(np.float64)).cuda().requires_grad_()
    loss = 0.0
    for ni, ei, tg in zip(nis, eis, tgs):
        out = _net_exact(p, off, case["steps"], g, ni, ei)
        one = ((out[:, :4] - tg.cuda().double()) ** 2).sum() / (4.0 * g["N"] * case["batch"])
        one.backward()
        loss += float(one)
    return dict(loss=torch.tensor([loss], dtype=torch.float64), grad=p.grad)


def _net_work(N, E, steps, train):
    rows = {"n": N, "e": E}
    flops = 0.0
    for name, layers in G.layout(steps=steps):
        r = rows["e" if name.startswith("edge") or name == "enc_edge" else "n"]
        flops += sum(2.0 * r * k * n for k, n in layers)
    # the features in, the node and edge states out of each step and into the next
    io = 32.0 * N + 16.0 * E + 32.0 * N
    state = 2.0 * W * (N + E) * (steps + 1)
    params = G.offsets(G.layout(steps=steps))[1]
    if not train:
        return dict(bytes=io + 2 * state + 2 * params, flops=flops)
    # the states again in the backward pass, their gradients, the parameters and moments
    return dict(bytes=io + 3 * state + 4 * state + 30.0 * params, flops=3 * flops)


# ---------------------------------------------------------------- one layer

def _layer_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *shape: torch.randn(*shape, generator=gen, device="cuda")
    rows, k, n = case["rows"], case["k"], case["n"]
    bf = torch.bfloat16
    if case["op"] == "dw":     # dW[n][k] += sum over rows of dY[row][n] X[row][k]
        return dict(a=(0.1 * rnd(rows, n)).to(bf), b=rnd(rows, k).to(bf))
    if case["op"] == "dsilu":  # dX = (dY W) * silu'(Z)
        return dict(a=(0.1 * rnd(rows, n)).to(bf), b=(rnd(n, k) / math.sqrt(k)).to(bf),
                    z=rnd(rows, k).to(bf))
    return dict(a=rnd(rows, k).to(bf), b=(rnd(n, k) / math.sqrt(k)).to(bf), bias=0.1 * rnd(n))


def _layer_prepare(case, seed, s):
    _session()
    s.x = _layer_inputs(case, seed)
    rows, k, n = case["rows"], case["k"], case["n"]
    bf = torch.bfloat16
    if case["op"] == "dw":
        s.c = torch.zeros(n, k, device="cuda")
    elif case["op"] == "dsilu":
        s.c = torch.empty(rows, k, dtype=bf, device="cuda")
    else:
        s.c, s.z = (torch.empty(rows, n, dtype=bf, device="cuda") for _ in range(2))
    _states.add(s)


def _layer_run(s):
    rows, k, n = s.case["rows"], s.case["k"], s.case["n"]
    a, b, st = s.x["a"].data_ptr(), s.x["b"].data_ptr(), torch.cuda.current_stream().cuda_stream
    if s.case["op"] == "dw":
        G._call("op2b_gnn_memset", s.c.data_ptr(), 0, 4 * n * k, st)
        split = max(1, min(2 * 148 // ((k + 127) // 128), rows // 256))
        G._call("op2b_gemm_bf16", n, k, rows, a, 1, n, b, 1, k, s.c.data_ptr(), k,
                G.EPI_ATOMIC_F32, None, None, None, 0, split, 2, st)
        return s.c
    if s.case["op"] == "dsilu":
        G._call("op2b_gemm_bf16", rows, k, n, a, n, 1, b, 1, k, s.c.data_ptr(), k,
                G.EPI_SILU_GRAD_BF16, None, None, s.x["z"].data_ptr(), k, 1, 2, st)
        return s.c
    G._call("op2b_gemm_bf16", rows, n, k, a, k, 1, b, k, 1, s.c.data_ptr(), n,
            G.EPI_BIAS_SILU_BF16, s.x["bias"].data_ptr(), s.z.data_ptr(), None, 0, 1, 2, st)
    return dict(c=s.c, z=s.z)


def _layer_exact(case, seed):
    x = {k: v.double() for k, v in _layer_inputs(case, seed).items()}
    if case["op"] == "dw":
        return x["a"].T @ x["b"]
    if case["op"] == "dsilu":
        g = torch.sigmoid(x["z"])
        return (x["a"] @ x["b"]) * (g * (1.0 + x["z"] * (1.0 - g)))
    z = x["a"] @ x["b"].T + x["bias"]
    return dict(c=z * torch.sigmoid(z), z=z)


def _layer_work(case):
    r, k, n = case["rows"], case["k"], case["n"]
    if case["op"] == "dw":
        b = 2.0 * r * (n + k) + 4.0 * n * k
    elif case["op"] == "dsilu":
        b = 2.0 * r * (n + 2 * k) + 2.0 * n * k
    else:
        b = 2.0 * r * (k + 2 * n) + 2.0 * n * k
    return dict(bytes=b, flops=2.0 * r * k * n)


# ---------------------------------------------------------------- plan

def _plan_prepare(case, seed, s):
    _session()
    # the seed numbers the mesh; the plan depends on nothing else
    rng = np.random.default_rng(seed)
    mesh = _mesh(case["I"], case["J"], "natural")
    if case["order"] == "natural":  # the generator's order from another cell on
        r = int(rng.integers(mesh.ncell))
        roll = lambda n: (np.arange(n) + r) % n
        mesh = M.renumber_mesh(mesh, roll(mesh.nnode), roll(mesh.ncell), roll(mesh.nedge),
                               roll(mesh.nbedge))
    else:
        mesh = M.permute_mesh(mesh, rng)
    app = Airfoil(mesh)
    if case["order"] == "rcm":
        app.renumber(stats=False)
    s.app = app
    _states.add(s)


def _plan_run(s):
    L.load().op2b_plan_release_all()
    p = L.op_plan_get_stage("res_calc", s.app.edges, s.case["part"], s.app.a_res,
                            [0, 0, 1, 1, 2, 2, 3, 3], s.case["staging"])
    # lengths that depend on the colouring and the sharing are filled up with -1
    d, n = L.plan_arrays(p), s.app.mesh.nedge
    most = dict(ncolblk=d["nblocks"], nsharedCol=d["nblocks"], col_offsets=n + 2 * d["nblocks"])
    out = {}
    for k, v in d.items():
        m = 2 * n if k.startswith("ind_map") else most.get(k)
        if m is not None and len(v) < m:
            v = np.concatenate([v, np.full(m - len(v), -1, v.dtype)])
        out[k] = v
    return out


# ---------------------------------------------------------------- job

def _job_prepare(case, seed, s):
    global _open
    if _open:  # the job opens and closes its own session
        gc.collect()
        L.op_exit()
        _open = False
    s.mesh = _mesh(case["I"], case["J"], "random")
    s.q0 = _field(s.mesh, seed)


def _job_run(s):
    L.op_init()
    try:
        app = Airfoil(s.mesh, q0=s.q0)
        app.renumber(stats=False)
        hist = app.iterate(s.case["iters"])
        q = app.fetch_original()
    finally:
        L.op_exit()
    return dict(q=q, rms=np.array([h[0] for h in hist]), maxerr=np.array([h[1] for h in hist]))


def _job_exact(case, seed):
    mesh = _mesh(case["I"], case["J"], "random")
    q, _, rms, big = _march_exact(mesh, _field(mesh, seed), case["iters"])
    return dict(q=q, rms=rms, maxerr=big)


# ---------------------------------------------------------------- what measures a case

_PREPARE = dict(march=_march_prepare, loops=_loops_prepare, batch=_batch_prepare,
                predict=_predict_prepare, train=_train_prepare, layer=_layer_prepare,
                plan=_plan_prepare, job=_job_prepare)
_RUN = dict(march=_march_run, loops=_loops_run, batch=_batch_run, predict=_predict_run,
            train=_train_run, layer=_layer_run, plan=_plan_run, job=_job_run)
_EXACT = dict(march=_march_case_exact, loops=_loops_exact, batch=_batch_exact,
              predict=_predict_exact, train=_train_exact, layer=_layer_exact, job=_job_exact)


def prepare(case, seed):
    s = State(case)
    _PREPARE[case["kind"]](s.case, seed, s)
    return s


def run(state):
    return _RUN[state.case["kind"]](state)


def exact(case, seed):
    f = _EXACT.get(case["kind"])
    return f(case, seed) if f else None


def work(case):
    kind = case["kind"]
    if kind == "layer":
        return _layer_work(case)
    if kind == "batch":
        word, total = 4 if case["fp32"] else 8, dict(bytes=0.0, flops=0.0)
        for p in _batch_specs(case, 0):
            c, e, n, b = _sizes(p["I"], p["J"])
            w = _march_work(c, e, n, b, case["iters"], word)
            total = {k: total[k] + w[k] for k in total}
        return total
    c, e, n, b = _sizes(case["I"], case["J"])
    if kind == "march":
        return _march_work(c, e, n, b, case["iters"], 8 if case["dtype"] == "f64" else 4)
    if kind == "loops":
        # u and the coordinates read, u written, the maps read, every iteration
        word, D = 8 if case["dtype"] == "f64" else 4, case["dim"]
        per = word * n * (2 * D + 2) + 8.0 * e + 12.0 * b
        return dict(bytes=case["iters"] * per, flops=case["iters"] * (e * (6 + 4.0 * D)
                                                                      + 4.0 * D * n))
    if kind == "predict":
        return _net_work(c, 2 * e, 8, False)
    if kind == "train":
        return _net_work(c * case["batch"], 2 * e * case["batch"], case["steps"], True)
    if kind == "plan":
        # the map read; thread colours, element order and local maps written
        return dict(bytes=8.0 * e + 4.0 * e + 8.0 * 2 * e + 8.0 * c, flops=0.0)
    # job: the host arrays over once, the field back, and the iterations
    w = _march_work(c, e, n, b, case["iters"], 8)
    return dict(bytes=w["bytes"] + 16.0 * n + 48.0 * c + 16.0 * e + 16.0 * b + 32.0 * c,
                flops=w["flops"])
