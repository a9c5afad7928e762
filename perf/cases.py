"""The work that is timed: a frame of hair, as a program using this library asks for it.

A program sets a groom's per-frame inputs (spheres, wind, root motion), advances the groom, or all of its
grooms together, and hands the control points on: in place to a renderer that reads device memory, exported
strand-major into the renderer's own buffer, read back to the host, or as tessellated render strands. Grooms
start as they do in a program, straight along the normals of their roots, and go on from frame to frame.
"""
import math

import numpy as np
import torch

from barbu_gb300 import abi, hairsim

DT = 1.0 / 60.0
FRAMES = 60  # the per-frame inputs repeat after one second


def listed():
    return [
        # The reference program's own hair: class Hair on the scalp mesh's 448 roots, 4 points a strand, the
        # shader's arithmetic, one moving head sphere. The smallest call: launch and latency.
        dict(name="scalp", kind="hair", strands=448, seed_lengths=1),
        # One character's groom: 4,096 x 16 over one moving sphere, default contract (bit exact).
        dict(_GROOM, name="plain", strands=4096, points=16, substeps=4, root="rigid", spheres=1),
        # A prop with odd sizes whose renderer keeps strand-major buffers: positions and velocities exported.
        dict(_GROOM, name="ragged", strands=50021, points=23, substeps=5, spheres=7, wind=True, root="rigid",
             deliver="export"),
        # The large groom under either contract.
        dict(_GROOM, name="large", strands=262144, points=32, substeps=8, spheres=16, wind=True, lengths=True),
        dict(_GROOM, name="large_fast", strands=262144, points=32, substeps=8, spheres=16, wind=True, lengths=True,
             contract="fast"),
        # The largest single groom: a million 64-point strands on a rigged body among 32 spheres.
        dict(_GROOM, name="skinned", strands=1048576, points=64, substeps=8, spheres=32, root="skinned",
             contract="fast"),
        # A scene of 64 uneven grooms advanced together, the headline workload.
        dict(_CROWD, name="crowd", grooms=64, lo=1024, hi=131072, substeps=8, contract="fast"),
        # A crowd in the distance: many small grooms, where a frame is launches and short kernels.
        dict(_CROWD, name="crowd_small", grooms=48, lo=256, hi=4096, substeps=4),
        # The shader's arithmetic on a full head of longer strands.
        dict(_GROOM, name="reference_mode", mode="reference", strands=100003, points=8, substeps=1, iterations=8,
             spheres=1),
        # A frame whose positions a host program consumes.
        dict(_GROOM, name="to_host", strands=65536, points=16, substeps=4, root="rigid", spheres=4, contract="fast",
             deliver="host"),
        # A frame and its render strands at the reference program's tessellation settings.
        dict(_GROOM, name="tess", strands=4096, points=16, substeps=4, root="rigid", spheres=1, roots="grid",
             deliver="tess", lines=2, subsegments=16),
    ]


_GROOM = dict(kind="groom", mode="dftl", substeps=4, iterations=1, contract="exact", root="pinned", roots="ball",
              spheres=1, wind=False, lengths=False, deliver="inplace")
_CROWD = dict(kind="crowd", sizes=3, substeps=8, contract="exact")


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["hair", "groom", "groom", "groom", "groom", "reference", "tess", "crowd"])
    if kind == "hair":
        return dict(kind="hair", strands=_log(rng, 100, 20000), seed_lengths=rng.randrange(1, 1000))
    if kind == "crowd":
        hi = _log(rng, 512, 32768)
        return dict(_CROWD, grooms=rng.randint(4, 64), lo=max(32, hi // 64), hi=hi, sizes=rng.randrange(1000),
                    substeps=rng.randint(2, 8), contract=rng.choice(["exact", "fast"]))
    if kind == "reference":
        return dict(_GROOM, mode="reference", strands=_log(rng, 200, 100000), points=rng.randint(3, 24), substeps=1,
                    iterations=8, spheres=rng.randint(0, 4), deliver=rng.choice(["inplace", "export", "host"]))
    if kind == "tess":
        side = rng.randint(12, 64)
        return dict(_GROOM, strands=side * side, points=rng.randint(4, 20), substeps=4, root="rigid", spheres=1,
                    roots="grid", deliver="tess", lines=rng.randint(1, 3), subsegments=rng.randint(4, 16))
    points = rng.choice([rng.randint(3, 64), 8, 16, 24, 32, 64])
    substeps = rng.randint(1, 12)
    strands = min(_log(rng, 300, 300000), 64000000 // (points * substeps))
    root = rng.choice(["pinned", "rigid", "skinned"])
    return dict(_GROOM, strands=strands, points=points, substeps=substeps,
                iterations=rng.choice([1, 1, 1, 1, 2]), contract=rng.choice(["exact", "fast"]), root=root,
                spheres=rng.choice([0, 1, 4, rng.randint(0, 32)]), wind=rng.random() < 0.5,
                lengths=rng.random() < 0.5, deliver=rng.choice(["inplace", "export", "host"]))


# ---- inputs -----------------------------------------------------------------

def _rng(seed, stream):
    return np.random.default_rng([seed % (1 << 31), stream])


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def _roots(case, seed):
    """Roots and their normals: on a ball, on a grid over a ball (for triangles), or round a limb."""
    ns, rng = case["strands"], _rng(seed, 1)
    if case.get("root") == "skinned":
        theta, y = rng.uniform(0, 2 * math.pi, ns), rng.uniform(0, 2, ns)
        n = np.stack([np.cos(theta), np.zeros(ns), np.sin(theta)], 1)
        return (n * 0.5 + np.stack([np.zeros(ns), y, np.zeros(ns)], 1)).astype(np.float32), n.astype(np.float32)
    if case.get("roots") == "grid":
        side = math.isqrt(ns)
        i = np.arange(ns)
        theta = ((i % side) + rng.uniform(0, 0.5, ns)) * (2 * math.pi / side)
        phi = ((i // side) + 0.75 + rng.uniform(-0.2, 0.2, ns)) * (math.pi / (side + 0.5))
        d = np.stack([np.sin(phi) * np.cos(theta), np.cos(phi), np.sin(phi) * np.sin(theta)], 1)
        return d.astype(np.float32), d.astype(np.float32)
    d = _unit(rng.standard_normal((ns, 3)))
    r = d + 0.03 * rng.uniform(-1, 1, (ns, 3)) if case.get("lengths") else d
    return r.astype(np.float32), d.astype(np.float32)


def _shell(k, rng, lo, hi):
    s = np.zeros((k, 4), np.float32)
    s[:, :3] = _unit(rng.standard_normal((k, 3))) * rng.uniform(lo, hi, (k, 1))
    s[:, 3] = rng.uniform(0.1, 0.4, k)
    return s


def _rigid_frames(rng):
    """Column-major transforms of a body that sways about an axis and moves to and fro."""
    x, y, z = _unit(rng.standard_normal(3))
    out = np.zeros((FRAMES, 16), np.float32)
    for f in range(FRAMES):
        a = 0.15 * math.sin(2 * math.pi * (f + 1) / FRAMES)
        c, s, q = math.cos(a), math.sin(a), 1 - math.cos(a)
        m = np.eye(4)
        m[:3, :3] = [[c + x * x * q, x * y * q - z * s, x * z * q + y * s],
                     [y * x * q + z * s, c + y * y * q, y * z * q - x * s],
                     [z * x * q - y * s, z * y * q + x * s, c + z * z * q]]
        m[:3, 3] = 0.2 * math.sin(2 * math.pi * (f + 1) / FRAMES) * np.array([z, x, y])
        out[f] = m.T.reshape(16)
    return out


def _bone_frames(rng):
    """Skinning matrices of a chain of 4 bones up a limb of height 2, each swaying by a few degrees."""
    joint, out = np.arange(4) * (2.0 / 3), np.zeros((FRAMES, 4, 16), np.float32)
    axes, speed = _unit(rng.standard_normal((4, 3))), rng.integers(1, 3, 4)
    for f in range(FRAMES):
        g = np.eye(4)
        for b in range(4):
            x, y, z = axes[b]
            a = 0.1 * math.sin(2 * math.pi * (f + 1) * speed[b] / FRAMES)
            c, s, q = math.cos(a), math.sin(a), 1 - math.cos(a)
            m = np.eye(4)
            m[:3, :3] = [[c + x * x * q, x * y * q - z * s, x * z * q + y * s],
                         [y * x * q + z * s, c + y * y * q, y * z * q - x * s],
                         [z * x * q - y * s, z * y * q + x * s, c + z * z * q]]
            m[1, 3] = joint[b] - (joint[b - 1] if b else 0.0)
            g = g @ m
            bind = np.eye(4)
            bind[1, 3] = -joint[b]
            out[f, b] = (g @ bind).T.reshape(16)
    return out


def _inputs(case, seed):
    """Everything one groom is given, as host arrays."""
    q = dict(case)
    q["roots_xyz"], q["normals"] = _roots(case, seed)
    rng = _rng(seed, 2)
    ns, k = case["strands"], case["spheres"]
    q["strand_seed"] = int(rng.integers(1, 1 << 30))
    q["length"] = rng.uniform(0.3, 0.8, ns).astype(np.float32) if case["lengths"] else None
    t = np.arange(1, FRAMES + 1) * DT
    q["winds"] = np.stack([1.5 * np.sin(2 * math.pi * t), 0 * t, 0.5 + 0 * t], 1).astype(np.float32)
    if case["root"] == "skinned":
        q["bones"] = _bone_frames(rng)
        h = q["roots_xyz"][:, 1].astype(np.float64) * 1.5
        lo = np.clip(np.floor(h).astype(np.int64), 0, 2)
        w = np.clip(h - lo, 0, 1)
        main, other = np.where(w >= 0.5, lo + 1, lo), np.where(w >= 0.5, lo, lo + 1)
        q["slots"] = np.stack([main, main, main, other], 1).astype(np.uint8)
        q["weights"] = np.zeros((ns, 3), np.float32)
        q["weights"][:, 0] = np.maximum(w, 1 - w)
        theta, y = rng.uniform(0, 2 * math.pi, k), rng.uniform(-0.3, 2, k)
        d, r = rng.uniform(0.7, 1.1, k), rng.uniform(0.1, 0.25, k)
        rest = np.stack([d * np.cos(theta), y, d * np.sin(theta), np.ones(k)], 1)
        bone = np.clip(np.rint(y * 1.5), 0, 3).astype(np.int64)
        m = q["bones"].astype(np.float64).reshape(FRAMES, 4, 4, 4)
        q["sphere"] = np.einsum("kj,fkji->fki", rest, m[:, bone]).astype(np.float32)
        q["sphere"][:, :, 3] = r
        return q
    m = _rigid_frames(rng) if case["root"] == "rigid" else np.tile(np.eye(4, dtype=np.float32).reshape(16), (FRAMES, 1))
    # One sphere is the head or body that the hair grows on; several are limbs and props around it.
    s = np.array([[0, 0, 0, 0.98]], np.float32) if k == 1 else _shell(k, rng, 1.0, 1.6)
    q["transforms"] = m
    q["sphere"] = np.tile(s, (FRAMES, 1, 1))
    if k == 1:  # it moves with the roots, or to and fro under pinned ones
        move = m[:, 12:15] if case["root"] == "rigid" else 0.05 * np.sin(2 * math.pi * t)[:, None] * [1, 0, 0]
        q["sphere"][:, 0, :3] += move.astype(np.float32)
    return q


def _crowd(case):
    """The sizes of a crowd's grooms, from the case alone."""
    rng = np.random.default_rng([case["sizes"], case["grooms"]])
    out = []
    for _ in range(case["grooms"]):
        ns = int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"])))))
        out.append(dict(_GROOM, strands=ns, points=int(rng.choice([8, 16, 24, 32])), substeps=case["substeps"],
                        contract=case["contract"], root="rigid", spheres=int(rng.integers(1, 17)), lengths=True))
    return out


def _hair(case):
    return dict(_GROOM, mode="reference", strands=case["strands"], points=4, substeps=1, iterations=8, spheres=1)


def _members(case, seed):
    if case["kind"] == "crowd":
        return [_inputs(c, seed * 1000 + g) for g, c in enumerate(_crowd(case))]
    q = _inputs(_hair(case) if case["kind"] == "hair" else case, seed)
    if case["kind"] == "hair":
        q["strand_seed"] = case["seed_lengths"]
    return [q]


def _faces(ns):
    side = math.isqrt(ns)
    i, j = np.meshgrid(np.arange(side - 1), np.arange(side), indexing="ij")
    a, b, c, d = i * side + j, i * side + (j + 1) % side, (i + 1) * side + j, (i + 1) * side + (j + 1) % side
    return np.concatenate([np.stack([a, b, c], -1).reshape(-1, 3), np.stack([b, d, c], -1).reshape(-1, 3)]).astype(np.uint32)


def _tess_inputs(q, seed):
    rng = _rng(seed, 3)
    return (_faces(q["strands"]), rng.uniform(-0.1, 0.1, (q["strands"], q["points"], 4)).astype(np.float32),
            rng.random(abi.HS_TESS_RANDOM_SIZE).astype(np.float32))


# ---- the program ------------------------------------------------------------

class _View:
    """Device memory of a groom as an array others can read in place; it keeps the groom (and its context) alive."""

    def __init__(self, groom, ptr, shape):
        self.groom = groom
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(ptr, False), strides=None, version=2)


def _in_place(groom):
    ptr, layout = groom.device_positions()
    whole = torch.as_tensor(_View(groom, ptr, (layout.points_per_strand, layout.strand_stride, 4)), device="cuda")
    return whole[:, :groom.nstrands]


def _groom(ctx, q):
    sim = (abi.sim_params_reference(1.45) if q["mode"] == "reference" else
           abi.sim_params_dftl(substeps=q["substeps"], damping=0.9, wind_jitter=0.2 if q["wind"] else 0.0,
                               iterations=q["iterations"],
                               root_mode={"pinned": abi.HS_ROOT_PINNED, "rigid": abi.HS_ROOT_RIGID,
                                          "skinned": abi.HS_ROOT_SKINNED}[q["root"]],
                               contract=abi.HS_CONTRACT_FAST if q["contract"] == "fast" else abi.HS_CONTRACT_EXACT))
    rule = abi.HS_LENGTH_REFERENCE if q["mode"] == "reference" else abi.HS_LENGTH_TOTAL
    strand = abi.strand_params(q["points"], rule, 0.5, 0.1 if q["mode"] == "reference" else 0.0, q["strand_seed"])
    g = ctx.groom(q["roots_xyz"], q["normals"], strand, sim, lengths=q["length"])
    if q["root"] == "skinned":
        g.set_skin(q["slots"], q["weights"])
    return g


def prepare(case, seed):
    members = _members(case, seed)
    s = dict(case=case, members=members, frame=0)
    if case["kind"] == "hair":
        hair = hairsim.Hair(seed=members[0]["strand_seed"])
        hair.init()
        hair.setup(members[0]["roots_xyz"], members[0]["normals"])
        s.update(hair=hair, ctx=hair.ctx, grooms=[hair.groom])
    else:
        ctx = hairsim.Context()
        s.update(ctx=ctx, grooms=[_groom(ctx, q) for q in members])
    if case["kind"] == "crowd":
        s["handles"] = s["ctx"].handles_of(s["grooms"])
        s["transforms"] = np.ascontiguousarray(np.stack([q["transforms"] for q in members], 1))
        for g, q in zip(s["grooms"], members):
            g.set_spheres(q["sphere"][0])
    s["views"] = [_in_place(g) for g in s["grooms"]]
    g, deliver = s["grooms"][0], case.get("deliver")
    if deliver == "export":
        s["out"] = [torch.empty((g.nstrands, g.npoints, 4), device="cuda") for _ in range(2)]
    elif deliver == "host":
        s["out"] = torch.empty((g.nstrands, g.npoints, 3), pin_memory=True).numpy()
    elif deliver == "tess":
        g.tess_setup(*_tess_inputs(members[0], seed))
        p = hairsim.tess_params_reference()
        p.nlines, p.nsubsegments = case["lines"], case["subsegments"]
        count = g.tess_stream(p)
        ptr, n = hairsim.C.c_void_p(), hairsim.C.c_uint64()
        hairsim.check(hairsim.lib().hs_tess_device(g.h, hairsim.C.byref(ptr), hairsim.C.byref(n)), "hs_tess_device")
        s.update(tess=p, out=torch.as_tensor(_View(g, ptr.value, (count, 4)), device="cuda"))
    return s


def run(s):
    f, case = s["frame"] % FRAMES, s["case"]
    s["frame"] += 1
    if case["kind"] == "hair":
        s["hair"].set_bounding_sphere(s["members"][0]["sphere"][f, 0])
        s["hair"].update(DT)
        return s["views"][0]
    if case["kind"] == "crowd":
        s["ctx"].set_root_transforms(s["grooms"], s["transforms"][f], handles=s["handles"])
        s["ctx"].update_many(s["grooms"], DT, handles=s["handles"])
        return s["views"]
    g, q = s["grooms"][0], s["members"][0]
    if case["root"] == "rigid":
        g.set_root_transform(q["transforms"][f])
    elif case["root"] == "skinned":
        g.set_bone_matrices(q["bones"][f])
    if case["spheres"]:
        g.set_spheres(q["sphere"][f])
    if case["wind"]:
        g.set_wind(q["winds"][f])
    g.update(DT)
    deliver = case["deliver"]
    if deliver == "export":
        for field, out in enumerate(s["out"]):
            g.export(out.data_ptr(), out.numel(), abi.HS_EXPORT_STRAND_MAJOR, field)
        return s["out"]
    if deliver == "host":
        return g.readback_xyz(s["out"])
    if deliver == "tess":
        g.tess_stream(s["tess"])
        return [s["out"], s["views"][0]]
    return s["views"][0]


def work(case):
    """Positions and velocities (float4 each) read and written once a frame, what is delivered besides written
    once; 42 operations a point, substep and iteration (prediction, link, velocity), sphere tests not counted."""
    if case["kind"] == "crowd":
        each = [work(c) for c in _crowd(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    c = _hair(case) if case["kind"] == "hair" else case
    points = c["strands"] * c["points"]
    w = {"bytes": 64 * points, "flops": 42 * points * c["substeps"] * c["iterations"]}
    if c["deliver"] == "export":
        w["bytes"] += 32 * points
    elif c["deliver"] == "host":
        w["bytes"] += 12 * points
    elif c["deliver"] == "tess":
        lines = 3 * len(_faces(c["strands"])) * (c["points"] - 1) * c["lines"]
        w["bytes"] += 32 * lines * c["subsegments"]
        w["flops"] += 90 * lines * (c["subsegments"] + 1)
    return w


# ---- the same frame in 64 bits ----------------------------------------------

def _hash(x):
    x = x.astype(np.uint64)
    m = np.uint64(0xffffffff)
    x ^= x >> np.uint64(16)
    x = (x * np.uint64(0x7feb352d)) & m
    x ^= x >> np.uint64(15)
    x = (x * np.uint64(0x846ca68b)) & m
    return x ^ (x >> np.uint64(16))


def _uniform(seed, stream, ns):
    """The documented per-strand hash in [0, 1) of the caller's strand index."""
    inner = _hash(np.array([(0x9E3779B9 * (stream + 1)) & 0xffffffff]))
    key = _hash(np.array([seed], np.uint64) ^ inner)
    return (_hash((np.arange(ns, dtype=np.uint64) + key) & np.uint64(0xffffffff)) >> np.uint64(8)).astype(np.float64) / 2.0**24


def _stored_order(roots):
    """Strands are stored along a Z-order curve over their roots, 10 bits an axis."""
    if len(roots) <= 32:
        return np.arange(len(roots))
    lo, hi = roots.min(0), roots.max(0)
    code = np.zeros(len(roots), np.int64)
    for a in range(3):
        ext = hi[a] - lo[a]
        t = (roots[:, a] - lo[a]) / ext if ext > 0 else np.zeros(len(roots), np.float32)
        c = np.clip(t * np.float32(1023), 0, 1023).astype(np.int64)
        for b in range(10):
            code |= ((c >> b) & 1) << (3 * b + a)
    return np.argsort(code, kind="stable")


def _start(q):
    """A groom's starting positions and rest lengths, rounded as the library rounds them: (points, strands, 3)."""
    n, ns, f = q["points"], q["strands"], np.float32
    if q["mode"] == "reference":
        rv = f(1) + f(0.1) * (f(1) - f(2) * _uniform(q["strand_seed"], 1, ns).astype(f))
        off = (np.arange(n).astype(f) * (f(0.5) / f(n)))[:, None] * rv[None]
        rest = off - np.concatenate([np.zeros((1, ns), f), off[:-1]])
    else:
        total = q["length"] if q["length"] is not None else np.full(ns, 0.5, f)
        seg = (total / f(n - 1)).astype(f)
        off = np.arange(n).astype(f)[:, None] * seg[None]
        rest = np.tile(seg, (n, 1))
        rest[0] = 0
    off, rest = (torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (off, rest))
    r, d = (torch.from_numpy(q[k]).cuda() for k in ("roots_xyz", "normals"))
    return (r[None] + off[:, :, None] * d[None]).double(), rest.double()


def _dual_quats(m):
    """Unit dual quaternions (real xyzw, dual xyzw) of small rotations with translations."""
    m = m.astype(np.float64).reshape(-1, 4, 4).transpose(0, 2, 1)
    out = np.zeros((len(m), 8))
    for b, a in enumerate(m):
        w = 0.5 * math.sqrt(a[0, 0] + a[1, 1] + a[2, 2] + 1)
        v = np.array([a[2, 1] - a[1, 2], a[0, 2] - a[2, 0], a[1, 0] - a[0, 1]]) / (4 * w)
        t = a[:3, 3]
        out[b] = [*v, w, *(0.5 * (w * t + np.cross(t, v))), -0.5 * (t @ v)]
    return out


def _targets(q, f):
    r = torch.from_numpy(q["roots_xyz"]).cuda().double()
    if q["root"] == "rigid":
        m = torch.from_numpy(q["transforms"][f].astype(np.float64).reshape(4, 4)).cuda()
        return r @ m[:3, :3] + m[3, :3]
    if q["root"] == "pinned":
        return r
    dq = torch.from_numpy(_dual_quats(q["bones"][f])).cuda()
    slot = torch.from_numpy(q["slots"].astype(np.int64)).cuda()
    w = torch.from_numpy(q["weights"]).cuda().double()
    w = torch.cat([w, 1 - w.sum(1, keepdim=True)], 1)
    at = dq[slot]  # (strands, 4, 8)
    sign = torch.sign((at[:, :, :4] * at[:, 3:, :4]).sum(-1))
    sign[:, 3] = 1
    blend = (at * (w * sign)[:, :, None]).sum(1)
    blend = blend / blend[:, :4].norm(dim=1, keepdim=True)
    a, aw, b, bw = blend[:, :3], blend[:, 3:4], blend[:, 4:7], blend[:, 7:8]
    cross = torch.linalg.cross
    v = r + 2 * cross(a, cross(a, r) + aw * r)
    return v + 2 * (aw * b - bw * a + cross(a, b))


def _push(p, v, mask, spheres, reflect):
    """Every point out of the spheres, in their order. spheres: (K, strands or 1, 4)."""
    for s in spheres:
        c, r = s[None, :, :3], s[None, :, 3]
        d = p - c
        d2 = (d * d).sum(-1)
        hit = ((d2 < r * r) & (r > 0) & mask).unsqueeze(-1)
        if not bool(hit.any()):
            continue
        nrm = d / d2.sqrt().unsqueeze(-1)
        p = torch.where(hit, c + r.unsqueeze(-1) * nrm, p)
        if reflect:
            v = torch.where(hit, v - 2 * (nrm * v).sum(-1, keepdim=True) * nrm, v)
    return p, v


def _frame64(q, x, rest, n, force, target, spheres):
    """One frame from rest of strands of up to len(x) points; n: each strand's own count."""
    N, S, reference = len(x), q["substeps"], q["mode"] == "reference"
    h = float(np.float32(np.float32(DT) / np.float32(S)))
    damping, scale = (float(np.float32(0.8)), float(np.float32(1.45))) if reference else (float(np.float32(0.9)), 1.0)
    j = torch.arange(N, device="cuda")[:, None]
    mask, tip = j < n[None], (j == n[None] - 1).unsqueeze(-1)
    v, x0, root = torch.zeros_like(x), x[0].clone(), x[0].clone()
    for k in range(S):
        old, p = x, x + h * v + h * h * force[None]
        p[0] = x0 + (k + 1) / S * (target - x0) if k + 1 < S else target
        move, root = p[0] - root, p[0].clone()
        for _ in range(q["iterations"]):
            corr = torch.zeros_like(p)
            for i in range(1, N):
                d = p[i] - p[i - 1]
                moved = p[i - 1] + (scale * rest[i]).unsqueeze(-1) * d / d.norm(dim=-1, keepdim=True)
                corr[i] = moved - p[i]
                p[i] = moved
            corr = torch.where(mask.unsqueeze(-1), corr, 0.0)
            shift = torch.cat([corr[1:], torch.zeros_like(corr[:1])])
            if reference:
                v = torch.where(tip, corr, damping * shift)
            q0 = p[0].clone()
            p, v = _push(p, v, mask, spheres, reference)
            p[0] = q0
        if not reference:
            v = (p - old - damping * torch.where(tip, 0.0, shift)) / h
        v[0] = move if reference else move / h
        x = p
    return x, v


def _force(q, f):
    g = torch.tensor([0.0, float(np.float32(-9.81)) * (20.0 if q["mode"] == "reference" else 1.0), 0.0], dtype=torch.float64)
    out = g.repeat(q["strands"], 1)
    if q["wind"]:
        j = 1 + float(np.float32(0.2)) * (1 - 2 * _uniform(q["strand_seed"], 2, q["strands"]))
        out = out + torch.from_numpy(j)[:, None] * torch.from_numpy(q["winds"][f]).double()
    return out.cuda()


def _tess64(case, x, faces, tangents, random):
    n, lines, sub = case["points"], case["lines"], case["subsegments"]
    f = torch.from_numpy(faces.astype(np.int64)).cuda()
    t = torch.from_numpy(tangents).cuda().double()[:, :, :3].transpose(0, 1) * float(np.float32(1.45))
    u = torch.arange(sub + 1, device="cuda", dtype=torch.float64) / sub
    basis = torch.stack([2 * u**3 - 3 * u**2 + 1, -2 * u**3 + 3 * u**2, u**3 - 2 * u**2 + u, u**3 - u**2], 1)
    curve = sum(basis[None, None, :, k, None] * y[:, :, None] for k, y in enumerate((x[:-1], x[1:], t[:-1], t[1:])))
    at = curve[:, f]  # (segments, faces, 3, sub + 1, 3)
    rel = ((torch.arange(n - 1, device="cuda", dtype=torch.float64) / n)[:, None] + u[None] / n).clamp(0, 1)
    rel = rel**3 * (10 + rel * (-15 + 6 * rel))
    out = torch.empty((3, len(faces), n - 1, lines, sub, 2, 4), dtype=torch.float64, device="cuda")
    for inst in range(3):
        for line in range(lines):
            r = int(np.float32(np.float32(line) / np.float32(lines)) * np.float32(40) + np.float32(inst)) % len(random)
            sx, sy = float(random[4 * r]), float(random[4 * r + 1])
            if np.float32(random[4 * r] + random[4 * r + 1]) > 1:
                sx, sy = 1 - max(sx, sy), min(max(sx, sy), sy)
            p = (at[:, :, 0] * sx + at[:, :, 1] * sy + at[:, :, 2] * (1 - sx - sy)).transpose(0, 1)
            for end in range(2):
                out[inst, :, :, line, :, end, :3] = p[:, :, end:end + sub]
                out[inst, :, :, line, :, end, 3] = rel[None, :, end:end + sub]
    return out.reshape(-1, 4)


def exact(case, seed):
    members = _members(case, seed)
    N = max(q["points"] for q in members)
    xs, rests, spheres, K = [], [], [], max(q["spheres"] for q in members)
    for q in members:
        x, rest = _start(q)
        more = N - q["points"]
        xs.append(torch.cat([x, x[-1:] + torch.arange(1, more + 1, device="cuda")[:, None, None]]) if more else x)
        rests.append(torch.cat([rest, torch.ones((more, q["strands"]), dtype=torch.float64, device="cuda")]) if more else rest)
        s = torch.from_numpy(np.concatenate([q["sphere"][0].reshape(-1, 4), np.zeros((K - q["spheres"], 4), np.float32)])).cuda().double()
        spheres.append(s[:, None].expand(K, q["strands"], 4) if len(members) > 1 else s[:, None])
    n = torch.cat([torch.full((q["strands"],), q["points"], device="cuda") for q in members])
    rest = torch.cat(rests, 1)
    x, v = _frame64(members[0], torch.cat(xs, 1), rest, n, torch.cat([_force(q, 0) for q in members]),
                    torch.cat([_targets(q, 0) for q in members]), torch.cat(spheres, 1))
    if case.get("deliver") == "host":
        return x.transpose(0, 1).cpu().numpy()
    pos, out, at = torch.cat([x, rest.unsqueeze(-1)], -1), [], 0
    if case.get("deliver") == "export":
        vel = torch.cat([v, torch.zeros_like(rest).unsqueeze(-1)], -1)
        return [pos.transpose(0, 1).contiguous(), vel.transpose(0, 1).contiguous()]
    for q in members:
        order = torch.from_numpy(_stored_order(q["roots_xyz"])).cuda()
        out.append(pos[:q["points"], at:at + q["strands"]][:, order])
        at += q["strands"]
    if case.get("deliver") == "tess":
        return [_tess64(case, x, *_tess_inputs(members[0], seed)), out[0]]
    return out if case["kind"] == "crowd" else out[0]
