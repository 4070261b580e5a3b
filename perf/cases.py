"""Performance cases: what a program that uses this library has it do, over the range of
sizes, precisions and options it is used with.

Five kinds of work, each through the public entry points:

* ``fit``   -- ``reconstruct``: oriented points in, the implicit field (keys, per-level and
  cumulative coefficients, isovalue) out; the forward path, from a preview of a few thousand
  points to a depth-9 scan;
* ``train`` -- ``reconstruct_differentiable``, a loss on field values (and gradients), and the
  reverse pass onto positions and normals: one optimisation step of a shape-fitting loop;
* ``query`` -- ``Reconstruction.evaluate`` of a reconstructed field at many points;
* ``mesh``  -- ``extract_mesh`` of a reconstructed field;
* ``relax`` -- ``ops.relax_sliced``: the ordered Gauss-Seidel sweeps of one level on the
  caller's own sparse operator.

Clouds are seeded synthetic stand-ins for scans, made on the GPU: a uniform sphere, a noisy
torus, a bumpy sphere with tenfold varying density, and a smooth union of three tori with
outliers and flipped normals.
"""
import math

import torch

from warp_psr_b200 import ops, reconstruct, reconstruct_differentiable
from warp_psr_b200.meshing import extract_mesh

DEVICE = "cuda"


def listed():
    return [
        # A preview while scanning: a few thousand points; launches and host waits are all of it.
        dict(name="fit_2k_d5_f32", kind="fit", shape="sphere", points=2_011, depth=5, full_depth=3, point_weight=2.0,
             dtype="float32", precision="input"),
        # The reference's defaults (depth 6, full depth 3) on a small clean scan.
        dict(name="fit_20k_d6_f32", kind="fit", shape="sphere", points=20_000, depth=6, full_depth=3,
             point_weight=2.0, dtype="float32", precision="input"),
        # A usual object scan: noisy, screened, single precision.
        dict(name="fit_200k_d8_f32", kind="fit", shape="torus", points=199_999, depth=8, full_depth=4,
             point_weight=4.0, dtype="float32", precision="input"),
        # The same in double precision and unscreened (plain Poisson reconstruction).
        dict(name="fit_200k_d8_f64_psr", kind="fit", shape="torus", points=200_000, depth=8, full_depth=4,
             point_weight=0.0, dtype="float64", precision="input"),
        # A full scan at depth 9 in the mixed precision.
        dict(name="fit_800k_d9_mixed", kind="fit", shape="bumpy", points=800_000, depth=9, full_depth=4,
             point_weight=2.0, dtype="float32", precision="mixed"),
        # One step of fitting a small point set: many such steps make an optimisation.
        dict(name="train_5k_d6_f32", kind="train", shape="sphere", points=5_003, depth=6, full_depth=3,
             point_weight=2.0, dtype="float32", precision="input", queries=4_096, at_inputs=False),
        # Gradients in double precision, loss on the values at 50,000 queries and on the field's
        # gradients at the inputs.
        dict(name="train_100k_d7_f64", kind="train", shape="torus", points=100_000, depth=7, full_depth=3,
             point_weight=2.0, dtype="float64", precision="input", queries=50_000, at_inputs=True),
        # Solve and adjoint of the depth-9 scan.
        dict(name="train_800k_d9_mixed", kind="train", shape="bumpy", points=800_000, depth=9, full_depth=4,
             point_weight=2.0, dtype="float32", precision="mixed", queries=32, at_inputs=False),
        # Solve and adjoint at scale: depth 10, outliers, flipped normals.
        dict(name="train_3500k_d10_mixed", kind="train", shape="tori", points=3_500_000, depth=10, full_depth=5,
             point_weight=4.0, dtype="float32", precision="mixed", queries=32, at_inputs=False),
        # Sampling a field at arbitrary points (ray marching, distance-like queries).
        dict(name="query_1m_d8_f32", kind="query", shape="torus", points=200_000, depth=8, full_depth=4,
             point_weight=4.0, dtype="float32", precision="input", queries=1_000_003),
        # The surface as triangles, on a grid of unequal sides.
        dict(name="mesh_d8_f32", kind="mesh", shape="torus", points=200_000, depth=8, full_depth=4, point_weight=4.0,
             dtype="float32", precision="input", nx=301, ny=257, nz=129),
        # The ordered relaxation alone, on an operator of the caller's.
        dict(name="relax_d8_f32", kind="relax", depth=8, thickness=3.0, dtype="float32", iters=8),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fit", "fit", "fit", "train", "train", "query", "mesh", "relax"])
    if kind == "relax":
        return dict(kind="relax", depth=rng.randint(4, 9), thickness=round(rng.uniform(1.0, 4.0), 3),
                    dtype=rng.choice(["float32", "float64"]), iters=rng.choice([4, 8, 8, 11]))
    dtype, precision = rng.choice([("float32", "input"), ("float32", "input"), ("float64", "input"),
                                   ("float32", "mixed"), ("float64", "mixed")])
    # In double precision and for meshes and queries up to a million points, in the mixed
    # precision and plain float32 up to the scale workload's size.
    large = kind in ("fit", "train") and precision == "mixed"
    points = log_int(1_000, 3_000_000 if large else 1_000_000)
    # A scan's depth follows its density: about one to four points per finest surface cell.
    depth = max(4, min(10 if large else 9, int(math.log(points, 4)) - rng.choice([0, 0, 1])))
    case = dict(kind=kind, shape=rng.choice(["sphere", "torus", "bumpy", "tori"]), points=points, depth=depth,
                full_depth=min(depth, rng.choice([3, 3, 4, 4, 5 if depth >= 8 else 4])),
                point_weight=rng.choice([0.0, 2.0, 2.0, 4.0]), dtype=dtype, precision=precision)
    if rng.random() < 0.25:  # noisy scans: more samples per node
        case["samples_per_node"] = round(rng.uniform(1.0, 12.0), 2)
    if rng.random() < 0.2:
        case["iters"] = rng.choice([4, 6, 10])
    if rng.random() < 0.15:
        case["base_v_cycles"] = 2
    if rng.random() < 0.15:
        case["base_depth"] = rng.randint(0, case["full_depth"])
    if kind == "train":
        case["queries"] = log_int(32, 100_000)
        case["at_inputs"] = rng.random() < 0.3
    elif kind == "query":
        case["queries"] = log_int(1_000, 4_000_000)
    elif kind == "mesh":
        n = log_int(32, 300)
        case.update(nx=n + rng.randint(0, 17), ny=n + rng.randint(0, 17), nz=max(8, n - rng.randint(0, 17)))
    return case


# ------------------------------------------------------------------ inputs
def _unit(n, gen):
    u = torch.randn((n, 3), generator=gen, device=DEVICE, dtype=torch.float64)
    return u / u.norm(dim=1, keepdim=True)


def _torus(n, gen, R, r):
    """n points uniform by area on a torus around the z axis, with exact normals."""
    parts, have = [], 0
    while have < n:
        m = 2 * (n - have) + 1024
        uv = torch.rand((m, 3), generator=gen, device=DEVICE, dtype=torch.float64)
        uv = uv[uv[:, 2] < (R + r * torch.cos(2 * math.pi * uv[:, 1])) / (R + r)][:n - have, :2]
        parts.append(uv)
        have += len(uv)
    u, v = (2 * math.pi * torch.cat(parts)).unbind(1)
    nrm = torch.stack([torch.cos(v) * torch.cos(u), torch.cos(v) * torch.sin(u), torch.sin(v)], 1)
    ring = R * torch.stack([torch.cos(u), torch.sin(u), torch.zeros_like(u)], 1)
    return ring + r * nrm, nrm


def _bumpy(n, gen):
    """Star-shaped surface |x| = r(x / |x|), r = 1 + a few smooth waves; density varies tenfold."""
    k = 3.0 * torch.randn((6, 3), generator=gen, device=DEVICE, dtype=torch.float64)
    ph = 2 * math.pi * torch.rand((6,), generator=gen, device=DEVICE, dtype=torch.float64)
    kd = 2.5 * torch.randn((4, 3), generator=gen, device=DEVICE, dtype=torch.float64)
    parts, have = [], 0
    while have < n:
        u = _unit(4 * (n - have) + 4096, gen)
        s = torch.sin(u @ kd.T).mean(1)
        accept = 0.1 + 0.9 * (0.5 + 0.5 * s) ** 2
        u = u[torch.rand(len(u), generator=gen, device=DEVICE, dtype=torch.float64) < accept][:n - have]
        parts.append(u)
        have += len(u)
    u = torch.cat(parts)
    r = 1 + 0.03 * torch.sin(u @ k.T + ph).sum(1, keepdim=True)
    g = 0.03 * torch.cos(u @ k.T + ph) @ k               # gradient of r with respect to u
    nrm = u - (g - (g * u).sum(1, keepdim=True) * u) / r  # gradient of |x| - r(x / |x|)
    return r * u, nrm / nrm.norm(dim=1, keepdim=True)


def _tori(n, gen):
    """Union of three tori with jitter, 1% outliers in the bounding box and 2% flipped normals."""
    R, r, side = 0.6, 0.2, 0.9
    angle = torch.tensor([math.pi / 2 + 2 * math.pi / 3 * j for j in range(3)], device=DEVICE, dtype=torch.float64)
    centre = side / math.sqrt(3) * torch.stack([torch.cos(angle), torch.sin(angle), torch.zeros_like(angle)], 1)
    pp, nn, have = [], [], 0
    while have < n:
        m = int(1.6 * (n - have)) + 4096
        which = torch.randint(0, 3, (m,), generator=gen, device=DEVICE)
        p, nrm = _torus(m, gen, R, r)
        p = p + centre[which]
        keep = torch.ones(m, dtype=torch.bool, device=DEVICE)
        for j in range(3):
            q = p - centre[j]
            inside = (q[:, :2].norm(dim=1) - R) ** 2 + q[:, 2] ** 2 < r * r
            keep &= (which == j) | ~inside
        p, nrm = p[keep][:n - have], nrm[keep][:n - have]
        pp.append(p)
        nn.append(nrm)
        have += len(p)
    p, nrm = torch.cat(pp), torch.cat(nn)
    lo, hi = p.min(0).values, p.max(0).values
    p = p + 0.001 * (hi - lo).norm() * torch.randn((n, 3), generator=gen, device=DEVICE, dtype=torch.float64)
    t = torch.rand((n, 4), generator=gen, device=DEVICE, dtype=torch.float64)
    out = t[:, 3:] < 0.01
    p = torch.where(out, lo + (hi - lo) * t[:, :3], p)
    nrm = torch.where(out, _unit(n, gen), nrm)
    flip = torch.rand((n, 1), generator=gen, device=DEVICE, dtype=torch.float64) < 0.02
    return p, torch.where(flip, -nrm, nrm)


def _cloud(case, gen):
    n = case["points"]
    if case["shape"] == "sphere":
        p = _unit(n, gen)
        nrm = p.clone()
    elif case["shape"] == "torus":
        p, nrm = _torus(n, gen, 1.0, 0.35)
        p = p + 0.002 * 2.9 * torch.randn((n, 3), generator=gen, device=DEVICE, dtype=torch.float64)
        nrm = nrm + 0.05 * torch.randn((n, 3), generator=gen, device=DEVICE, dtype=torch.float64)
        nrm = nrm / nrm.norm(dim=1, keepdim=True)
    elif case["shape"] == "bumpy":
        p, nrm = _bumpy(n, gen)
    else:
        p, nrm = _tori(n, gen)
    dtype = getattr(torch, case["dtype"])
    return p.to(dtype).contiguous(), nrm.to(dtype).contiguous()


def _options(case):
    names = ("depth", "full_depth", "point_weight", "precision", "samples_per_node", "iters", "base_v_cycles",
             "base_depth")
    return {k: case[k] for k in names if k in case}


def _result_dtype(case):
    return torch.float64 if case["dtype"] == "float64" or case["precision"] == "mixed" else torch.float32


def _level(case, gen):
    """One level's ordered system: the nodes of a spherical shell on the depth-d grid, a
    27-point diagonally dominant operator over the present neighbours in CSR, b and x."""
    d = case["depth"]
    n = 1 << d
    g = torch.arange(n + 1, device=DEVICE)
    r = 0.41 * n
    nodes = []
    for x0 in range(0, n + 1, 64):
        gx = g[x0:x0 + 64]
        dist = (((gx - n / 2) ** 2)[:, None, None] + ((g - n / 2) ** 2)[None, :, None]
                + ((g - n / 2) ** 2)[None, None, :]).double().sqrt()
        at = ((dist - r).abs() <= case["thickness"]).nonzero()
        at[:, 0] += x0
        nodes.append(at)
    c = torch.cat(nodes)
    keys = (d << 48) | (c[:, 0] << 32) | (c[:, 1] << 16) | c[:, 2]
    offs = torch.tensor([(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)], device=DEVICE)
    q = c[:, None, :] + offs
    qk = (d << 48) | (q[..., 0] << 32) | (q[..., 1] << 16) | q[..., 2]
    pos = torch.searchsorted(keys, qk.reshape(-1)).clamp(max=len(keys) - 1)
    found = (keys[pos] == qk.reshape(-1)).reshape(-1, 27) & ((q >= 0) & (q <= n)).all(-1)
    # a stiffness-like row: random negative couplings, the diagonal above their sum
    v = -torch.rand((len(c), 27), generator=gen, device=DEVICE, dtype=torch.float64) * found
    v[:, 13] = 0.2 - v.sum(1) + v[:, 13]
    dtype = getattr(torch, case["dtype"])
    counts = found.sum(1)
    offsets = torch.zeros(len(c) + 1, dtype=torch.int32, device=DEVICE)
    offsets[1:] = counts.cumsum(0)
    b = torch.randn(len(c), generator=gen, device=DEVICE, dtype=torch.float64).to(dtype)
    x = torch.randn(len(c), generator=gen, device=DEVICE, dtype=torch.float64).to(dtype)
    return dict(keys=keys, offsets=offsets, columns=pos.reshape(-1, 27)[found].int(), values=v[found].to(dtype), b=b,
                x=x)


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))
    if case["kind"] == "relax":
        return dict(case=case, **_level(case, gen))
    p, nrm = _cloud(case, gen)
    state = dict(case=case, positions=p, normals=nrm)
    lo, hi = p.min(0).values, p.max(0).values
    # What a program keeps of a result it copies into arrays of its own, of a size fixed ahead:
    # the library's views hold the whole result (a tape of gigabytes) until they are dropped.
    dtype = _result_dtype(case)
    if case["kind"] in ("fit", "train"):
        size = 2 * int(_coefficients(case)) + 20_000
        state["out"] = dict(keys=torch.zeros(size, dtype=torch.int64, device=DEVICE),
                            coefficients=torch.zeros(size, dtype=dtype, device=DEVICE),
                            cumulative=torch.zeros(size, dtype=dtype, device=DEVICE))
    elif case["kind"] == "mesh":
        size = 12 * max(case["nx"], case["ny"], case["nz"]) ** 2 + 4096
        state["out"] = dict(vertices=torch.zeros((size, 3), dtype=dtype, device=DEVICE),
                            indices=torch.zeros(6 * size, dtype=torch.int32, device=DEVICE))
    if "queries" in case:
        t = torch.rand((case["queries"], 3), generator=gen, device=DEVICE, dtype=torch.float64)
        q = lo + (hi - lo) * t.to(p.dtype)
        if case["kind"] == "query":  # half of them near the surface
            m = case["queries"] // 2
            pick = torch.randint(0, case["points"], (m,), generator=gen, device=DEVICE)
            q[:m] = torch.minimum(torch.maximum(p[pick] + 0.01 * (q[:m] - p[pick]), lo), hi)
        state["queries"] = q.to(_result_dtype(case)).contiguous()
        state["seed"] = torch.randn(case["queries"], generator=gen, device=DEVICE, dtype=torch.float64).to(
            _result_dtype(case))
    if case["kind"] in ("query", "mesh"):
        state["field"] = reconstruct(p, nrm, **_options(case))
        pad = 0.02 * (hi - lo)
        state["bounds"] = ((lo - pad).tolist(), (hi + pad).tolist())
    return state


def _keep(out, **arrays):
    for name, a in arrays.items():
        out[name][:len(a)].copy_(a)
    return out


def run(state):
    case = state["case"]
    if case["kind"] == "fit":
        r = reconstruct(state["positions"], state["normals"], **_options(case))
        kept = _keep(state["out"], keys=r.field.keys, coefficients=r.field.coefficients,
                     cumulative=r.field.cumulative)
        return dict(kept, iso=r.iso_value, counts=r.metadata["basis_counts"])
    if case["kind"] == "train":
        p = state["positions"].detach().requires_grad_(True)
        n = state["normals"].detach().requires_grad_(True)
        r = reconstruct_differentiable(p, n, **_options(case))
        v, _, _ = r.evaluate(state["queries"], centered=True)
        loss = (v * v).sum() if case["at_inputs"] else (v * state["seed"]).sum()
        if case["at_inputs"]:
            _, g, _ = r.evaluate(p.to(v.dtype))
            loss = loss + 0.1 * (g * g).sum()
        loss.backward()
        kept = _keep(state["out"], keys=r.result.field.keys, coefficients=r.coefficients.detach(),
                     cumulative=r.cumulative.detach())
        return dict(kept, values=v.detach(), loss=loss.detach(), iso=r.iso_value.detach(), grad_positions=p.grad,
                    grad_normals=n.grad)
    if case["kind"] == "query":
        values, gradients, valid = state["field"].evaluate(state["queries"])
        return dict(values=values, gradients=gradients, valid=valid)
    if case["kind"] == "mesh":
        mesh = extract_mesh(state["field"], resolution=(case["nx"], case["ny"], case["nz"]), bounds=state["bounds"])
        return _keep(state["out"], vertices=mesh.vertices, indices=mesh.indices)
    x = state["x"].clone()
    return ops.relax_sliced(state["keys"], case["depth"], state["offsets"], state["columns"], state["values"],
                            state["b"], x, case["iters"])


# ------------------------------------------------------------------ what a pass cannot do without
def _coefficients(case):
    """About how many basis functions a reconstruction has: a band of a few cells around the
    surface on every level down to where the points are dense, the full grid above."""
    full = (2 ** case["full_depth"] + 1) ** 3
    return full + sum(min(COEFFICIENTS_PER_CELL * 4 ** d, COEFFICIENTS_PER_POINT * case["points"])
                      for d in range(case["full_depth"] + 1, case["depth"] + 1))


COEFFICIENTS_PER_CELL = 15   # times 4^depth: the surfaces here span most of the cube
COEFFICIENTS_PER_POINT = 12  # a lone point's splat makes about this many


def work(case):
    elem = 8 if case["dtype"] == "float64" else 4
    if case["kind"] == "relax":
        rows = 4 * math.pi * (0.41 * 2 ** case["depth"]) ** 2 * 2 * case["thickness"]
        # the operator (27 columns and values), keys, offsets, b and x once; 27 products a visit
        return dict(bytes=rows * (27 * (4 + elem) + 8 + 4 + 3 * elem), flops=rows * case["iters"] * 57.0)
    n, total = case["points"], _coefficients(case)
    out = 8 if _result_dtype(case) == torch.float64 else 4
    iters = case.get("iters", 8)
    if case["kind"] == "query":
        q = case["queries"]
        # three levels' eight coefficients a query, a few products each
        return dict(bytes=q * (3 * out + 4 * out + 4) + total * (8 + 2 * out), flops=q * 3 * 8 * 20.0)
    if case["kind"] == "mesh":
        nodes = case["nx"] * case["ny"] * case["nz"]
        triangles = 4.0 * max(case["nx"], case["ny"], case["nz"]) ** 2
        return dict(bytes=total * (8 + 2 * out) + triangles * (12 + 0.5 * 3 * out), flops=nodes * 3 * 8 * 8.0)
    # points and normals in; keys, coefficients and cumulative coefficients out; the sweeps'
    # products, and the operator's (27 entries a row, 8 screening points of 8 products)
    w = dict(bytes=2 * 3 * elem * n + total * (8 + 2 * out), flops=total * (iters * 57.0 + 27 * 8 + 8 * 8 * 6))
    if case["kind"] == "train":
        w["bytes"] += 2 * 3 * elem * n + total * out
        w["flops"] *= 3
    return w


def tolerance(case):
    single = case["dtype"] == "float32" and case.get("precision") != "mixed"
    if case["kind"] in ("query", "relax"):
        # against `exact`: 1e-6 in single, 1e-14 in double precision
        return {"rel": 5e-6, "max": 2e-3} if single else {"rel": 1e-12, "max": 1e-10}
    # Four times what a change of rounding was seen to do: single against double precision on
    # inputs of one tree (coefficients 3e-6, gradients 6e-6, largest 5e-5), mixed against
    # double (coefficients 5e-8, gradients 1e-7, largest 6e-6).  Keys and counts are exact.
    if single:
        return {"rel": 2.5e-5, "max": 2e-4, "differ": 0.0}
    if case["precision"] == "mixed":
        return {"rel": 4e-7, "max": 2.5e-5, "differ": 0.0}
    return {"rel": 1e-10, "max": 1e-8, "differ": 0.0}


# ------------------------------------------------------------------ 64-bit references
def exact(case, seed):
    """Query and relax: the same arithmetic in float64 with plain torch (a query's field is an
    input: the reconstruction that the program already holds).  A whole reconstruction, its
    reverse pass and its mesh have no reference of this kind that runs in seconds."""
    if case["kind"] == "relax":
        return _exact_relax(case, prepare(case, seed))
    if case["kind"] == "query":
        return _exact_query(prepare(case, seed))
    return None


def _exact_relax(case, state):
    d, iters = case["depth"], case["iters"]
    n, keys, m = 1 << d, state["keys"], len(state["keys"])
    cx, cy, cz = (keys >> 32) & 65535, (keys >> 16) & 65535, keys & 65535
    counts = (state["offsets"][1:] - state["offsets"][:-1]).long()
    slot = torch.arange(27, device=DEVICE)
    have = slot < counts[:, None]
    at = (state["offsets"][:-1].long()[:, None] + slot) * have
    cols = torch.where(have, state["columns"].long()[at], m)
    vals = torch.where(have, state["values"].double()[at], 0.0)
    diag = (vals * (cols == torch.arange(m, device=DEVICE)[:, None])).sum(1)
    order = torch.argsort(4 * cz + (cx & 1) + 2 * (cy & 1), stable=True)
    ends = torch.bincount(4 * cz + (cx & 1) + 2 * (cy & 1), minlength=4 * (n + 1)).cumsum(0).tolist()
    x = torch.cat([state["x"].double(), torch.zeros(1, device=DEVICE, dtype=torch.float64)])
    b = state["b"].double()
    groups = [order[(ends[g - 1] if g else 0):ends[g]] for g in range(4 * (n + 1))]
    parts = [(r, cols[r], vals[r], b[r], diag[r]) if len(r) else None for r in groups]
    # sweeps pipelined over the slices: the front moves down, each slice in the window in turn
    for front in range(n, -iters, -1):
        for z in range(max(front, 0), min(front + iters, n + 1)):
            for colour in range(4):
                part = parts[4 * z + colour]
                if part is not None:
                    r, c, v, rb, rd = part
                    x[r] = x[r] + (rb - (v * x[c]).sum(1)) / rd
    return x[:m]


def _exact_query(state):
    field = state["field"].field
    keys = field.keys
    coefficients, cumulative = field.coefficients.double(), field.cumulative.double()
    dtype = field.coefficients.dtype
    linear = torch.tensor(field.linear, device=DEVICE, dtype=dtype).reshape(3, 3)
    shift = torch.tensor(field.translation, device=DEVICE, dtype=dtype)
    # A query's place in the unit cube is taken in the field's precision, for it chooses the
    # cell (the gradient jumps from cell to cell); all that follows is in 64 bits.
    q = state["queries"][:, None, :] * linear
    p = (((q[..., 0] + q[..., 1]) + q[..., 2]) + shift).double()
    linear = linear.double()
    valid = ((p >= 0) & (p <= 1)).all(1)

    def find(d, c):
        k = (d << 48) | (c[..., 0] << 32) | (c[..., 1] << 16) | c[..., 2]
        pos = torch.searchsorted(keys, k.reshape(-1)).clamp(max=len(keys) - 1)
        return pos.reshape(k.shape), (keys[pos] == k.reshape(-1)).reshape(k.shape)

    leaf = torch.zeros(len(p), dtype=torch.int64, device=DEVICE)
    for d in range(field.depth + 1):
        n = 1 << d
        cell = ((p * n).ceil().long() - 1).clamp(0, n - 1)
        leaf = torch.where(find(d, cell)[1], d, leaf)
    p = torch.where(p == 0, 1e-6, torch.where(p == 1, 1 - 1e-6, p))
    corner = torch.tensor([(i, j, k) for i in (0, 1) for j in (0, 1) for k in (0, 1)], device=DEVICE)
    out = torch.zeros((len(p), 4), dtype=torch.float64, device=DEVICE)

    def add_level(which, d, coef):
        if not 0 <= d <= field.depth or not bool(which.any()):
            return
        n = 1 << d
        t = p[which] * n
        cell = (t.ceil().long() - 1).clamp(0, n - 1)
        base = t.floor().long()
        node = cell[:, None, :] + corner
        pos, found = find(d, node)
        c = coef[pos] * found * (node >= base[:, None, :]).all(-1)
        up = node > base[:, None, :]
        fr = (t - base)[:, None, :]
        h = torch.where(up, fr, 1 - fr)
        s = torch.where(up, 1.0, -1.0)
        out[which, 0] += (c * h.prod(-1)).sum(1)
        out[which, 1] += (c * n * s[..., 0] * h[..., 1] * h[..., 2]).sum(1)
        out[which, 2] += (c * n * h[..., 0] * s[..., 1] * h[..., 2]).sum(1)
        out[which, 3] += (c * n * h[..., 0] * h[..., 1] * s[..., 2]).sum(1)

    for d in range(field.depth + 1):
        which = leaf == d
        add_level(which, d, coefficients)
        add_level(which, d - 1, cumulative)
        add_level(which, d + 1, coefficients)
    out[~valid] = float("nan")
    return dict(values=out[:, 0], gradients=out[:, 1:] @ linear, valid=None)
