"""What a program asks of the gather-scatter library, as cases that can be timed.

A case is a mesh (its node numbering), a field (type, components, layout) and
the calls made on them.  Meshes are generated here: boxes of hexahedra with
element-major local nodes, boxes split into tetrahedra, and mixes of uneven
boxes.  Fields are seeded.  `listed()` holds the cases that are always
measured, `draw()` gives more of the same ranges.

Kinds of calls:
  gs     GatherScatter in place on element-local fields.  A pass first fills the
         field as the element kernel before it would (a copy), then calls
         GatherScatter `calls` times, as a solver's smoother and the
         performance test of dawgs do; a repeated Add without the fill would
         run into infinities.
  c0     Scatter from the gathered vector to the element-local field, then
         Gather back: the frame of an operator applied to gathered vectors.
  batch  GatherScatters of many meshes in one tuned batched call, from a graph.
  setup  Setup of a mesh from host ids, then the first GatherScatter.
"""
import math

import numpy as np
import torch

from dawgs_gb300 import ogs

TYPES = {"f64": torch.float64, "f32": torch.float32, "i64": torch.int64, "i32": torch.int32}
SIZE = {"f64": 8, "f32": 4, "i64": 8, "i32": 4}
OPS = {"add": ogs.Add, "mul": ogs.Mul, "max": ogs.Max, "min": ogs.Min}
TRANS = {"sym": ogs.Sym, "notrans": ogs.NoTrans, "trans": ogs.Trans}
KUHN = ((0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0))


def listed():
    return [
        # the smallest ordinary call: a mesh of one subdomain, where launches and latency count
        _case("gs_f64_small", "gs", 10, 10, 10, 3, calls=4),
        # the usual size of a spectral-element rank at the usual degree
        _case("gs_f64_p7", "gs", 24, 24, 24, 7, calls=4),
        # the largest: a whole GPU's mesh at high degree
        _case("gs_f64_p15", "gs", 24, 24, 24, 15, calls=2),
        # integer reductions (node flags, owner ranks) on an odd box
        _case("gs_i64_max_odd", "gs", 23, 19, 17, 6, type="i64", op="max"),
        # an interleaved vector field on a mesh whose elements come in no order (a partitioner's output)
        _case("gs_f32_vec3_perm", "gs", 32, 32, 16, 5, type="f32", k=3, permute=True, calls=4),
        # eight separate scalar fields (species) at once on the same kind of mesh
        _case("gs_f64_many8_perm", "gs", 32, 32, 16, 5, k=8, many=True, permute=True, calls=2),
        # tetrahedra: vertices of degree up to 24 beside edges and faces
        _case("gs_f64_tet", "gs", 32, 32, 24, 3, tet=True, calls=4),
        # Signed ids with masked (zero) boundary nodes, summed to the owners only
        _case("gs_f64_masked_trans", "gs", 21, 18, 20, 7, k=2, kind="signed", mask=True, trans="trans", calls=4),
        # an operator on gathered vectors: Scatter, Gather
        _case("c0_f64_p7", "c0", 24, 24, 24, 7, kind="signed"),
        _case("c0_f32_vec3_perm", "c0", 32, 32, 16, 5, type="f32", k=3, kind="signed", permute=True),
        # many uneven meshes, one batched call
        _case("batch_256", "batch", 16, 16, 16, 7, meshes=256),
        # setup from the ids in host memory, and the first call
        _case("setup_p7", "setup", 24, 24, 24, 7),
    ]


def _case(name, do, nx, ny, nz, p, type="f64", op="add", k=1, many=False, kind="unsigned", trans="sym",
          permute=False, mask=False, tet=False, calls=1, meshes=1):
    return {"name": name, "do": do, "nx": nx, "ny": ny, "nz": nz, "p": p, "type": type, "op": op, "k": k,
            "many": many, "kind": kind, "trans": trans, "permute": permute, "mask": mask, "tet": tet,
            "calls": calls, "meshes": meshes}


def draw(rng):
    """A case of the ranges above: 60 thousand to 25 million values, degree 1 to 15, every type and op."""
    do = rng.choice(("gs", "gs", "gs", "gs", "c0", "c0", "batch", "setup"))
    if do == "batch":
        c = _case("", do, rng.randint(6, 16), rng.randint(6, 16), rng.randint(6, 16), rng.randint(3, 7),
                  type=rng.choice(("f64", "f32")), meshes=int(round(math.exp(rng.uniform(math.log(8), math.log(256))))))
        del c["name"]
        return c
    tet = do == "gs" and rng.random() < 0.2
    p = rng.randint(1, 4) if tet else rng.randint(1, 15)
    k = rng.choice((1, 1, 1, 2, 3, 5, 8)) if do != "setup" else 1
    per = 6 * _tet_nodes(p) if tet else (p + 1) ** 3
    low = max(6e4, 8.0 * per * k)
    values = math.exp(rng.uniform(math.log(low), math.log(max(2 * low, 2.5e7 if do != "setup" else 1e7))))
    side = (values / k / per) ** (1 / 3)
    nx = max(2, int(round(side * math.exp(rng.uniform(-0.4, 0.4)))))
    ny = max(2, int(round(side * math.exp(rng.uniform(-0.4, 0.4)))))
    nz = max(2, int(round(side * side * side / nx / ny)))
    typ = rng.choice(("f64", "f64", "f64", "f32", "f32", "i64", "i32"))
    op = rng.choice(("add", "add", "add", "max", "min", "mul"))
    kind = "signed" if do == "c0" else rng.choice(("unsigned", "unsigned", "signed"))
    c = _case("", do, nx, ny, nz, p, type=typ, op=op if do != "c0" else "add", k=k,
              many=do == "gs" and k > 1 and rng.random() < 0.4, kind=kind,
              trans=rng.choice(("sym", "trans", "notrans")) if do == "gs" and kind == "signed" else "sym",
              permute=not tet and rng.random() < 0.4, mask=rng.random() < 0.2, tet=tet,
              calls=rng.randint(1, 4) if do == "gs" and op == "add" else 1)
    del c["name"]
    return c


# ---- meshes: global ids of the local nodes, element-major ----

def _tet_nodes(p):
    return (p + 1) * (p + 2) * (p + 3) // 6


def _mesh_ids(c, seed):
    nx, ny, nz, p = c["nx"], c["ny"], c["nz"], c["p"]
    sx, sy, sz = nx * p + 1, ny * p + 1, nz * p + 1
    if c["tet"]:  # each cell cut into six tetrahedra along its diagonal
        off = []
        for perm in KUHN:
            for a in range(p + 1):
                for b in range(a + 1):
                    for d in range(b + 1):
                        x = [0, 0, 0]
                        x[perm[0]], x[perm[1]], x[perm[2]] = a, b, d
                        off.append(x)
        off = np.array(off, dtype=np.int64)
        i, j, l = off[:, 0], off[:, 1], off[:, 2]
    else:
        q = np.arange(p + 1, dtype=np.int64)
        l, j, i = (a.reshape(-1) for a in np.meshgrid(q, q, q, indexing="ij"))
    node = i + sx * (j + sy * l)
    K, J, I = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    base = (p * (I + sx * (J + sy * K.astype(np.int64)))).reshape(-1)
    if c["permute"]:
        base = np.random.RandomState(seed % 2**32).permutation(base)
    ids = base[:, None] + node[None, :]
    if c["mask"]:  # nodes on the boundary x = 0 take no part
        ids = np.where(ids % sx == 0, -1, ids)
    return (ids + 1).reshape(-1)


def _mix(c):
    """(nx, ny, nz, p) of a batch's meshes, uneven up to the case's sides and degree; a batch is the same for every seed."""
    r = np.random.RandomState(c["meshes"])
    return [(r.randint(2, c["nx"] + 1), r.randint(2, c["ny"] + 1), r.randint(2, c["nz"] + 1),
             r.randint(1, c["p"] + 1), r.randint(1, 5)) for _ in range(c["meshes"])]


def _batch_meshes(c):
    for nx, ny, nz, p, k in _mix(c):
        yield _case("", "gs", int(nx), int(ny), int(nz), int(p), type=c["type"], k=int(k))


def _values(n, c, seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + salt)
    t = TYPES[c["type"]]
    if not t.is_floating_point:
        return torch.randint(-2**30, 2**30, (n,), generator=g, device="cuda", dtype=t)
    v = torch.rand(n, generator=g, device="cuda", dtype=t)
    return v * 1.5 + 0.5 if c["op"] == "mul" else v * 2 - 1


# ---- the passes ----

def _handle(c, ids):
    kind = ogs.Signed if c["kind"] == "signed" else ogs.Unsigned
    return ogs.ogs_t().Setup(ids.size, ids, None, kind, ogs.Auto, c["kind"] == "signed")


def prepare(case, seed):
    c = case
    if c["do"] == "batch":
        handles = [_handle(m, _mesh_ids(m, seed)) for m in _batch_meshes(c)]
        ks = [m["k"] for m in _batch_meshes(c)]
        src = _values(sum(g.N * k for g, k in zip(handles, ks)), c, seed)
        q = src.clone()
        fields, at = [], 0
        for g, k in zip(handles, ks):
            fields.append(q[at:at + g.N * k])
            at += g.N * k
        b = ogs.ogs_batch_t([(g, f, k, OPS[c["op"]], ogs.Sym) for g, f, k in zip(handles, fields, ks)], graph=True)
        b.tune()
        return {"case": c, "batch": b, "handles": handles, "src": src, "q": q}
    ids = _mesh_ids(c, seed)
    if c["do"] == "setup":
        src = _values(ids.size, c, seed)
        return {"case": c, "ids": ids, "src": src, "q": torch.empty_like(src)}
    g = _handle(c, ids)
    if c["do"] == "c0":
        x = _values(g.Ngather * c["k"], c, seed)
        return {"case": c, "g": g, "x": x, "q": _values(g.N * c["k"], c, seed, 1), "r": torch.zeros_like(x)}
    src = _values(g.N * c["k"], c, seed)
    q = torch.empty_like(src)
    s = {"case": c, "g": g, "src": src, "q": q}
    if c["many"]:
        s["fields"] = list(q.view(c["k"], g.N).unbind(0))
    return s


def run(state):
    c = state["case"]
    if c["do"] == "c0":
        g = state["g"]
        g.Scatter(state["q"], state["x"], c["k"], ogs.NoTrans)
        g.Gather(state["r"], state["q"], c["k"], ogs.Add, ogs.Trans)
        return state["q"], state["r"]
    q = state["q"]
    if c["do"] == "setup":
        ids = state["ids"].copy() if c["kind"] == "signed" else state["ids"]  # Signed Setup rewrites the ids' signs
        g = _handle(c, ids)
        q.copy_(state["src"])
        g.GatherScatter(q, 1, OPS[c["op"]], ogs.Sym)
        return q, g.NgatherGlobal
    q.copy_(state["src"])
    if c["do"] == "batch":
        state["batch"].GatherScatter()
        return q
    g, op, trans = state["g"], OPS[c["op"]], TRANS[c["trans"]]
    for _ in range(c["calls"]):
        if c["many"]:
            g.GatherScatterMany(state["fields"], op, trans)
        else:
            g.GatherScatter(q, c["k"], op, trans)
    return q


# ---- what a pass cannot do without ----

def _counts(c):
    """(local nodes, nodes that take part, distinct ids)"""
    nx, ny, nz, p = c["nx"], c["ny"], c["nz"], c["p"]
    n = nx * ny * nz * (6 * _tet_nodes(p) if c["tet"] else (p + 1) ** 3)
    rows = (nx * p + 1) * (ny * p + 1) * (nz * p + 1)
    if not c["mask"]:
        return n, n, rows
    if c["tet"]:  # of a boundary cell: per tetrahedron with a face, an edge or a vertex on x = 0
        lost = sum((p + 1) * (p + 2) // 2 if perm[2] == 0 else p + 1 if perm[1] == 0 else 1 for perm in KUHN)
    else:
        lost = (p + 1) ** 2
    return n, n - ny * nz * lost, rows - (ny * p + 1) * (nz * p + 1)


def work(case):
    c = case
    if c["do"] == "batch":
        got = {"bytes": 0, "flops": 0}
        for m in _batch_meshes(c):
            w = work(dict(m, calls=1))
            got = {key: got[key] + w[key] for key in got}
        return got
    n, nnz, rows = _counts(c)
    field, index = n * c["k"] * SIZE[c["type"]], 4 * nnz
    if c["do"] == "c0":
        gathered = rows * c["k"] * SIZE[c["type"]]
        return {"bytes": 2 * (field + gathered + index), "flops": (nnz - rows) * c["k"]}
    # the fill, then each call reads the field and the map and writes the field
    one = 2 * field + index
    ids = 8 * n + index if c["do"] == "setup" else 0
    return {"bytes": 2 * field + c["calls"] * one + ids, "flops": c["calls"] * (nnz - rows) * c["k"]}


# ---- the same in 64 bits with torch alone ----

def _groups(ids):
    """Row of each taking-part node, rows numbered by first appearance; and those nodes."""
    t = torch.from_numpy(ids).cuda()
    at = torch.nonzero(t).view(-1)
    _, inv = torch.unique(t[at], return_inverse=True)
    rows = int(inv.max()) + 1
    first = torch.full((rows,), at.numel(), device="cuda", dtype=torch.int64)
    first.scatter_reduce_(0, inv, torch.arange(at.numel(), device="cuda"), "amin")
    rank = torch.empty_like(first)
    order = torch.argsort(first)
    rank[order] = torch.arange(rows, device="cuda")
    owner = torch.zeros(at.numel(), dtype=torch.bool, device="cuda")
    owner[first] = True
    return rank[inv], at, rows, owner


def _wide(v):
    return v.double() if v.is_floating_point() else v.long()


def _reduce(v, row, rows, op, typ):
    """v: [members, k], reduced over the members of each row."""
    if op == "add":
        return torch.zeros((rows, v.shape[1]), dtype=v.dtype, device="cuda").index_add_(0, row, v)
    big = {"f64": torch.finfo(torch.float64).max, "f32": torch.finfo(torch.float32).max,
           "i64": 2**63 - 1, "i32": 2**31 - 1}[typ]
    start, how = {"mul": (1, "prod"), "max": (-big, "amax"), "min": (big, "amin")}[op]
    out = torch.full((rows, v.shape[1]), start, dtype=v.dtype, device="cuda")
    return out.scatter_reduce_(0, row[:, None].expand_as(v), v, how)


def _exact_gs(c, ids, v, calls):
    """v: [nodes, k]"""
    row, at, rows, owner = _groups(ids)
    x = _wide(v)
    signed = c["kind"] == "signed"
    for _ in range(calls):
        m = x[at]
        if signed and c["trans"] == "notrans":  # folds the owners, writes every member
            s = _reduce(m[owner], row[owner], rows, c["op"], c["type"])
        else:
            s = _reduce(m, row, rows, c["op"], c["type"])
        if c["type"] == "i32":
            s = s.int().long()
        if signed and c["trans"] == "trans":  # folds every member, writes the owners
            x[at[owner]] = s[row[owner]]
        else:
            x[at] = s[row]
    return x


def exact(case, seed):
    c = case
    if c["do"] == "batch":
        metas = list(_batch_meshes(c))
        src = _values(sum(_counts(m)[0] * m["k"] for m in metas), c, seed)
        out, at = [], 0
        for m in metas:
            n = _counts(m)[0] * m["k"]
            out.append(_exact_gs(m, _mesh_ids(m, seed), src[at:at + n].view(-1, m["k"]), 1).reshape(-1))
            at += n
        return torch.cat(out)
    ids = _mesh_ids(c, seed)
    n, k = ids.size, c["k"]
    if c["do"] == "c0":
        row, at, rows, _ = _groups(ids)
        x, q = _wide(_values(rows * k, c, seed)).view(-1, k), _wide(_values(n * k, c, seed, 1)).view(-1, k)
        q[at] = x[row]
        return q.reshape(-1), _reduce(q[at], row, rows, "add", c["type"]).reshape(-1)
    v = _values(n * k, c, seed)
    if c["do"] == "setup":
        return _exact_gs(c, ids, v.view(-1, 1), 1).reshape(-1), _counts(c)[2]
    if c["many"]:
        return _exact_gs(c, ids, v.view(k, n).t(), c["calls"]).t().reshape(-1)
    return _exact_gs(c, ids, v.view(n, k), c["calls"]).reshape(-1)
